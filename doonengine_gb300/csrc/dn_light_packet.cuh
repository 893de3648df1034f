/*
 * dn_light_packet.cuh -- the lighting update with ray fans traced as warp packets.
 *
 * Every lit voxel casts two fans of K rays from one point: K specular rays around its reflection
 * direction (voxelLighting.comp:83-146, each up to specBounceLimit segments) and K shadow rays around the
 * sun direction (D8).  A warp takes one work unit -- 16, 8 or 4 voxels of a request group (a group is 32
 * voxels of one chunk) -- and traces the fans of PK_POOL_FAN / K of its voxels at a time as one pool: the
 * pool's rays are numbered (specular fans first, then the shadow rays), and a lane whose ray has ended takes
 * the pool's next ray, so consecutive rays of a fan run side by side and the lanes of a warp walk nearly the
 * same cells (a fan's shadow rays are almost parallel, its specular rays share their origin and lobe).  The
 * specular directions of a whole pool are formed before its first ray, by full warps.  Ended segments are
 * shaded once `batch` lanes have one.  Each ray's contributions go to shared memory; when the pool is empty,
 * each sum of a voxel's lighting is formed by one lane walking its rays (and their segments) in ray order, so
 * every sum is accumulated in exactly the reference's order.  The kernel writes each voxel's specular
 * lighting and leaves its direct light for the diffuse kernel (path_loop,
 * dn_light_path.cuh), which traces the diffuse paths (numDiffuse per voxel, up to
 * diffuseBounceLimit segments each) as per-lane path streams over all request groups and finishes each voxel
 * as the reference's lighting main does (running average, clamps, voxelLighting.comp:238-288).
 *
 * Results, traversal side effects (requested / touched / visible flags) and counters are those of the
 * one-voxel-per-lane form (dn_light_stream.cuh): the same rays are traced with the same
 * operations; only the assignment of rays to lanes differs.
 *
 * Bound by issue and by load latency at 28 warps per SM.  Between segments a lane keeps only its ray's number:
 * what a bounce needs besides (multiplier, sky flag) is in the ray's shared-memory slot and two flag bits, and
 * the light of see-through voxels is in shared memory for the rays that meet one (TintT), so the kernel takes
 * 71 registers (72 for many maps) instead of 80.  Measured with the directions formed by full warps, the table-free sums (a lane
 * per component) and the three unit sizes, us per frame or call, before -> after: 64x32x64 map at 1080p, K = 32:
 * 14200 -> 12240; 16x16x16 at 640x360, K = 16: 661 -> 507; glass 2970 -> 2597; twelve maps batched
 * 15230 -> 12010; eight maps served 2259 -> 1459.
 */
#pragma once
#include "dn_light_stream.cuh"

namespace dn {

#ifndef DN_PACKET_MIN_BLOCKS
// 7 blocks of 4 warps per SM (71 registers; 72 for many maps, with 60 bytes of spills).  The 64x32x64 map, us per frame: 12440; 6 blocks 12800, 8 (64
// registers, spills, little L1 left) 12990
#define DN_PACKET_MIN_BLOCKS 7
#endif

// specBounceLimit handled here (the reference's default is 2); larger limits use the stream kernel.  A pooled ray
// keeps one contribution per segment, so there are builds for at most 2, 4 and 8 segments: 128-ray pools for 2,
// 64-ray pools for more.  Four lighting updates of a 16x12x16 map with limit 4, K = 16 and 4 paths per voxel, read
// back: 6.8 ms, 18.8 with the ray streams.
constexpr uint32_t PK_MAX_SPEC_SEGMENTS = 8;
__host__ __device__ constexpr uint32_t packet_segments(uint32_t specBounceLimit)
{
    return specBounceLimit <= 2u ? 2u : specBounceLimit <= 4u ? 4u : 8u;
}

// the build a launch takes: its segments, or 0 for the ray streams.  far: a map of it is far (dn_walk.cuh); there is one
// far build, for the reference's limit and below (a lighting update of a 1x2x262200 map, us: K = 16 89, ray streams 189;
// K = 64 119, 630; batched with four 16x12x16 maps, which the far build then lights too, 1352 a frame, 7300)
__host__ __device__ constexpr uint32_t packet_build(uint32_t specBounceLimit, bool far)
{
    return specBounceLimit <= (far ? 2u : PK_MAX_SPEC_SEGMENTS) ? packet_segments(specBounceLimit) : 0u;
}

// resident blocks the register allocation of a build must allow (8-segment pools take 34 KB per block)
constexpr int packet_blocks(uint32_t segs) { return segs <= 4u ? DN_PACKET_MIN_BLOCKS : 6; }

// per-voxel data of the warp's unit (shared memory, written by the voxel's lane)
struct PacketVoxel {
    f3 pos0, talbedo, refl;
    uint32_t tmat, flags;    // flags: 1 valid, 2 first sample, 4 specular pass, 8 diffuse passes
};
enum : uint32_t { PV_VALID = 1u, PV_FIRST = 2u, PV_SPEC = 4u, PV_DIFF = 8u };

// rays per fan kind in one pool (voxels per pool = PK_POOL_FAN / K): the pool's specular slots, shadow
// contributions and counts live in shared memory, 38 B per pooled ray.  Larger pools shorten the tail that a
// pool's longest rays leave; the shared memory they take comes out of L1 (the SM's 256 KB split).  Measured, us per
// frame of the 64x32x64 map (K = 32), of a 16x16x16 map (K = 16) and of twelve maps batched: 128 rays 12444, 513,
// 12750; 96 rays 12299, 537, 13388; 192 rays 14361, 542, 13659.
#ifndef DN_PK_POOL_FAN
#define DN_PK_POOL_FAN 128
#endif
constexpr uint32_t PK_POOL_FAN = DN_PK_POOL_FAN;
constexpr uint32_t PK_POOL_ALT = PK_POOL_FAN == 64u ? 128u : 64u;   // the batched autotuner's other pool size

// Work units: 16 voxels of a request group at a time while more than PK_MID voxels per warp of the launch are left in
// the queue, 8 down to PK_TAIL, then 4; 2 or 1 in a launch that has no more voxels than twice its warps or its warps.
// Large units have fewer pool tails, small ones spread the end of a launch.
// One size for all, us per frame of the 64x32x64 map, the 16x16x16 map, the glass map and twelve maps batched: 16 voxels
// 12336, 514, 2885, 12105; 8 voxels 12444, 513, 2685, 12750; 4 voxels 12675, 573, 2720, 14115; these three 12243, 507,
// 2597, 12014 (a middle of 128 or 256 voxels per warp, a tail of 4 or 16: within 2 %).
#ifndef DN_PK_MID
#define DN_PK_MID 192
#endif
#ifndef DN_PK_TAIL
#define DN_PK_TAIL 8
#endif
constexpr uint32_t PK_MID = DN_PK_MID, PK_TAIL = DN_PK_TAIL;
#ifndef DN_PK_VOX
#define DN_PK_VOX 16
#endif
constexpr uint32_t PK_VOXELS = DN_PK_VOX;

template <uint32_t POOL, uint32_t SEGS>
struct PacketWarpT {
    PacketVoxel v[PK_VOXELS];
    // a pooled specular ray's direction and its reciprocal until a lane takes the ray, then the contributions of its
    // segments; while segment b > 0 runs, its place holds the ray's multiplier
    float con[3 * SEGS][POOL];
    float sh[3][POOL];                          // shadow contribution of each pooled ray
    uint8_t ncon[POOL];                         // contributions of each specular ray
    uint8_t shHas[POOL];                        // the shadow ray was unoccluded
    uint8_t specList[PK_VOXELS], fanList[PK_VOXELS], firstList[PK_VOXELS];   // the pool's voxels by what they cast
    TintT<32> tint;
};

// sets up voxel (req, vlane) of the group (voxel_setup of dn_light_stream.cuh) and writes the outputs that no ray
// decides: zero for invalid slots and for light the voxel does not cast rays for
__device__ __forceinline__ void packet_setup(PacketVoxel& pv, uint32_t req, uint32_t vlane, const DevMap& m,
                                             const dn_light_params& p, const Material* mats, const uint32_t* reqs,
                                             const uint32_t* nsamples, float4* out)
{
    pv.flags = 0;
    const uint32_t word = reqs[req];
    const uint32_t tile = word >> 4, group = word & 15u;
    const uint32_t tw = __ldg(&m.tword[tile]);
    const uint32_t vn = group * 32u + vlane;
    const uint64_t o = ((uint64_t)req * 32u + vlane) * 2u;
    i3 cp; uint32_t li;
    const ChunkRec* rc = &m.rec[tw & SLOT_MASK];
    if ((tw >> 30) != 2u || vn >= __ldg(&rc->nvox) || !select_voxel(rc, vn, cp, li)) {
        out[o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        out[o + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    const i3 mp{__ldg(&rc->pos[0]), __ldg(&rc->pos[1]), __ldg(&rc->pos[2])};
    const uint2 w = __ldg(&m.vox[__ldg(&rc->voxBase) + vn]);
    const f3 tnormal = voxel_normal(w);
    pv.tmat = w.x >> 24;
    pv.talbedo = mk((float)((w.y >> 24) & 0xFF) * INV255, (float)((w.y >> 16) & 0xFF) * INV255,
                    (float)((w.y >> 8) & 0xFF) * INV255);
    const uint32_t samples = __ldg(&nsamples[tw & SLOT_MASK]);
    const bool first = (samples < p.maxDiffuse ? samples : p.maxDiffuse) == 0u;
    f3 rp;
    rp.x = INV_CHUNK * (float)cp.x + (float)mp.x + HALF_INV_CHUNK;
    rp.y = INV_CHUNK * (float)cp.y + (float)mp.y + HALF_INV_CHUNK;
    rp.z = INV_CHUNK * (float)cp.z + (float)mp.z + HALF_INV_CHUNK;
    const float off = HALF_INV_CHUNK - EPS;
    pv.pos0 = add(rp, muls(tnormal, off));
    const Material& tm = mats[pv.tmat];
    const f3 viewDir = sub(pv.pos0, mk(p.camPos[0], p.camPos[1], p.camPos[2]));
    // no specular segments (specBounceLimit 0): the sum stays zero
    const bool doSpec = tm.specular > 0.0f && dot(viewDir, tnormal) < 0.0f && tm.reflectType <= 1u && p.specBounceLimit > 0u;
    const bool doDiff = tm.specular < 1.0f;
    if (doSpec) pv.refl = reflect(normalize(viewDir), tnormal);
    if (!doDiff) out[o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!doSpec) out[o + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    pv.flags = PV_VALID | (first ? PV_FIRST : 0u) | (doSpec ? PV_SPEC : 0u) | (doDiff ? PV_DIFF : 0u);
}

// Unit u of a queue of nreq request groups: voxels [first, first + count) of group r; false when there is none.  The
// queue is five stretches, of units of 16, 8, 4, 2 and 1 voxels.  (Formed again for every unit: kept over the loop,
// the stretches' bounds cost the many-map kernel more spills than the 60 bytes it has.)
__device__ __forceinline__ bool packet_unit(uint32_t u, uint32_t nreq, uint32_t& r, uint32_t& first, uint32_t& count)
{
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    uint32_t from = 0;
#pragma unroll 1
    for (uint32_t i = 0; i < 5u; i++) {
        // voxels per warp of the launch that the next stretches take
        const uint32_t left = i == 0u ? PK_MID : i == 1u ? PK_TAIL : i == 2u ? (nreq * 16u <= warps ? 2u : 0u)
                            : i == 3u ? (nreq * 32u <= warps ? 1u : 0u) : 0u;
        const uint32_t after = warps * left / 32u, to = nreq > after ? nreq - after : 0u;
        const uint32_t units = (to - from) << (i + 1u);
        if (u < units) {
            count = 16u >> i;
            r = from + (u >> (i + 1u));
            first = (u & ((2u << i) - 1u)) * count;
            return true;
        }
        u -= units;
        from = to;
    }
    return false;
}

// The work units of one launch (a part of a request group).  Per unit: (1) the setup of its voxels; (2) pools of
// PK_POOL_FAN/K voxels (at least one): the directions of all its specular rays, by whole warps; then every ray of
// the specular fans, the shadow fans and the first-sample shadow rays is traced by whichever lane is free -- a lane
// takes the pool's next ray as soon as its own ended, the shading of ended specular segments runs once `batch` lanes
// have one, so no lane waits for the slowest ray of a fan; each ray's contributions go to shared memory, and when
// the pool is empty every voxel's sums are formed in the reference's order and written (its diffuse paths run in
// k_light_diffuse, which reads the direct light left in the voxel's diffuse slot).
template <bool MANY, uint32_t POOL, uint32_t SEGS, bool TINTED, bool FAR>
__device__ __forceinline__ void packet_loop(const StreamArgs* one, const BatchLightArgs* many, PacketWarpT<POOL, SEGS>& W)
{
    static_assert(SEGS >= 2u && POOL >= 64u, "a slot holds a direction and its reciprocal, a pool one voxel's rays");
    const uint32_t lane = lane_id_s();
    const uint32_t below = (1u << lane) - 1u;
    uint32_t nreq = 0;
    if constexpr (MANY) nreq = *(volatile const uint32_t*)&many->reqStart[many->nmaps];
    else nreq = *(volatile const uint32_t*)one->nreqPtr;
    uint32_t* const counter = MANY ? many->workCounter : one->workCounter;
    const uint32_t batch = MANY ? many->batch : one->batch;
    Counters c{0, 0, 0, 0, 0};
    uint32_t lit = 0;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(counter, 1u);
        u = __shfl_sync(0xFFFFFFFFu, u, 0);
        // unit u: voxels [first, first + count) of request group r
        uint32_t r, first, count;
        if (!packet_unit(u, nreq, r, first, count)) break;
        // the group's map (warp-uniform)
        const BatchLightMap* e = nullptr;
        uint32_t req = r;
        if constexpr (MANY) {
            uint32_t lo = 0, hi = many->nmaps;
            while (hi - lo > 1u) {
                const uint32_t mid = (lo + hi) >> 1;
                if (__ldg(&many->reqStart[mid]) <= r) lo = mid; else hi = mid;
            }
            e = &many->maps[lo];
            req = r - __ldg(&many->reqStart[lo]);
        }
        const DevMap& m = MANY ? e->m : one->m;
        const dn_light_params& p = MANY ? e->p : one->p;
        const Material* mats = MANY ? e->mats : one->gtab->mats;
        const float (*sdir)[3] = MANY ? e->sdir : one->gtab->sdir;
        const float (*sinv)[3] = MANY ? e->sinv : one->gtab->sinv;
        const float (*pts)[3] = MANY ? e->p.spherePts : one->gtab->pts;
        float4* out = MANY ? e->out : one->out;
        const uint32_t K = p.K;
        const uint32_t overK = (65536u + K - 1u) / K;   // q / K = q * overK >> 16 for every q < 1024 (K <= 64)

        uint32_t myFlags = 0;
        if (lane < count) {
            packet_setup(W.v[lane], req, first + lane, m, p, mats, MANY ? e->reqs : one->reqs, MANY ? e->nsamples : one->nsamples, out);
            myFlags = W.v[lane].flags;
        }
        lit += myFlags & PV_VALID;
        const uint32_t specMask = __ballot_sync(0xFFFFFFFFu, (myFlags & PV_SPEC) != 0u);
        const uint32_t diffMask = __ballot_sync(0xFFFFFFFFu, (myFlags & PV_DIFF) != 0u);
        const uint32_t firstMask = diffMask & __ballot_sync(0xFFFFFFFFu, (myFlags & PV_FIRST) != 0u);
        uint32_t todo = specMask | diffMask;

        Ray s;
        s.mode = RM_IDLE;
        uint32_t q = 0;       // the lane's ray: its number in the pool
        while (todo) {
            // the pool's voxels: the lowest perPool bits left; its rays: K per specular voxel, then K per fan voxel,
            // then one per first-sample voxel
            const uint32_t perPool = K < POOL ? POOL * overK >> 16 : 1u;
            const bool mine = ((todo >> lane) & 1u) && (uint32_t)__popc(todo & below) < perPool;
            const uint32_t poolMask = __ballot_sync(0xFFFFFFFFu, mine);
            todo &= ~poolMask;
            const uint32_t specs = poolMask & specMask, fans = poolMask & diffMask & ~firstMask, firsts = poolMask & firstMask;
            __syncwarp();   // the last pool's sums have been read
            if ((specs >> lane) & 1u) W.specList[__popc(specs & below)] = (uint8_t)lane;
            if ((fans >> lane) & 1u) W.fanList[__popc(fans & below)] = (uint8_t)lane;
            if ((firsts >> lane) & 1u) W.firstList[__popc(firsts & below)] = (uint8_t)lane;
            __syncwarp();
            const uint32_t nSpec = (uint32_t)__popc(specs) * K, nFan = (uint32_t)__popc(fans) * K;
            const uint32_t total = nSpec + nFan + (uint32_t)__popc(firsts);
            // specular directions (voxelLighting.comp:83-97) and their reciprocals, a ray per lane.  The fan's offsets
            // come from a table in memory: a warp reads up to 32 of them at once, which the launch's constant arguments
            // serve one after the other (64x32x64 map at 1080p 10981 -> 10854 us)
            for (uint32_t i = lane; i < nSpec; i += 32u) {
                const uint32_t j = i * overK >> 16, k = i - j * K;
                const PacketVoxel& pv = W.v[W.specList[j]];
                const f3 P = mk(pts[k][0], pts[k][1], pts[k][2]);
                const f3 d = adds(normalize(add(muls(pv.refl, (float)mats[pv.tmat].shininess), P)), EPS);
                const f3 inv = rcp3(d);
                W.con[0][i] = d.x; W.con[1][i] = d.y; W.con[2][i] = d.z;
                W.con[3][i] = inv.x; W.con[4][i] = inv.y; W.con[5][i] = inv.z;
            }
            __syncwarp();
            uint32_t next = 0;
            for (;;) {
                // lanes without a ray take the pool's next rays in order
                const unsigned need = __ballot_sync(0xFFFFFFFFu, s.mode == RM_IDLE);
                if (next < total && need) {
                    const uint32_t mineq = next + (uint32_t)__popc(need & below);
                    if (s.mode == RM_IDLE && mineq < total) {
                        q = mineq;
                        uint32_t vi;
                        f3 d, inv;
                        if (q < nSpec) {
                            vi = W.specList[q * overK >> 16];
                            d = mk(W.con[0][q], W.con[1][q], W.con[2][q]);
                            inv = mk(W.con[3][q], W.con[4][q], W.con[5][q]);
                        } else {
                            const uint32_t f = q - nSpec;
                            uint32_t k = 64u;
                            if (f < nFan) {
                                const uint32_t j = f * overK >> 16;
                                vi = W.fanList[j];
                                k = f - j * K;
                            } else {
                                vi = W.firstList[f - nFan];
                            }
                            d = mk(sdir[k][0], sdir[k][1], sdir[k][2]);
                            inv = mk(sinv[k][0], sinv[k][1], sinv[k][2]);
                        }
                        c.rays++;
                        ray_begin<FAR, TINTED>(s, m, W.v[vi].pos0, d, inv, false, c, W.tint, lane);
                    }
                    next = min(next + (uint32_t)__popc(need), total);
                }
                const unsigned live = __ballot_sync(0xFFFFFFFFu, s.mode != RM_IDLE);
                if (!live) break;
                // step until 'batch' lanes have an ended segment (or none is left stepping); the live lanes
                // do not change while stepping, so one vote per round tells both
                for (;;) {
                    const unsigned st = __ballot_sync(0xFFFFFFFFu, ray_stepping(s));
                    if (!st || (uint32_t)__popc(live & ~st) >= batch) break;
                    if (ray_stepping(s)) walk_round<FAR, TINTED>(s, m, mats, p.sunStrength, c, W.tint, lane);
                }
                // shade the ended segments
                if (s.mode == RM_IDLE || ray_stepping(s)) continue;
                const f3 sun = mk(p.sunStrength[0], p.sunStrength[1], p.sunStrength[2]);
                f3 cadd;
                float cmul;
                ray_tint<TINTED>(s, W.tint, lane, cadd, cmul);
                const bool hit = s.mode == RM_HIT;
                s.mode = RM_IDLE;
                if (q >= nSpec) {
                    // shadow_ray: an unoccluded ray adds sunStrength * colorMult + colorAdd
                    const uint32_t f = q - nSpec;
                    W.sh[0][f] = sun.x * cmul + cadd.x;
                    W.sh[1][f] = sun.y * cmul + cadd.y;
                    W.sh[2][f] = sun.z * cmul + cadd.z;
                    W.shHas[f] = hit ? 0 : 1;
                    continue;
                }
                // specular_ray body after step_map (voxelLighting.comp:98-144).  A bounced segment started at the
                // last hit position (its origin) and left the multiplier in con and its material's sky flag in s.flags
                const PacketVoxel& pv = W.v[W.specList[q * overK >> 16]];
                const uint32_t b = s.flags >> RF_BOUNCES, at = SEGS == 2u ? (b ? 3u : 0u) : 3u * b;
                const uint32_t in = SEGS == 2u ? 3u : at, up = SEGS == 2u ? 3u : at + 3u;   // this multiplier, the next one
                const f3 mult = b ? mk(W.con[in][q], W.con[in + 1u][q], W.con[in + 2u][q]) : pv.talbedo;
                bool more = false, add_ = true;
                f3 sc;
                if (hit) {
                    const f3 hpos = ray_hit_position<FAR>(s);
                    Voxel hv;
                    decompress(m, ray_hit_index(s, m), hv);
                    const i3 hp{f2i(hpos.x), f2i(hpos.y), f2i(hpos.z)};
                    if (in_map(m, hp)) {
                        uint8_t* vp = &m.tvis[map_index(m, hp)];
                        if (*vp == 0) *vp = 1;
                    }
                    const f3 d = vabs(sub(vfloor(muls(hpos, 8.0f)), vfloor(muls(s.pos, 8.0f))));
                    add_ = !(dot(d, d) <= 1.0f);
                    if (add_) {
                        const Material& hm = mats[hv.material];
                        const f3 hd = muls(hv.diff, 1.0f - hm.specular);
                        if (hm.emissive) {
                            sc.x = ((hv.albedo.x * p.emissiveStrength * cmul + cadd.x) * mult.x) * pv.talbedo.x;
                            sc.y = ((hv.albedo.y * p.emissiveStrength * cmul + cadd.y) * mult.y) * pv.talbedo.y;
                            sc.z = ((hv.albedo.z * p.emissiveStrength * cmul + cadd.z) * mult.z) * pv.talbedo.z;
                        } else {
                            const f3 hc = mul(hd, hv.albedo);
                            sc.x = (hc.x * cmul + cadd.x) * mult.x;
                            sc.y = (hc.y * cmul + cadd.y) * mult.y;
                            sc.z = (hc.z * cmul + cadd.z) * mult.z;
                            if (hm.specular != 0.0f && (SEGS == 2u ? !b && p.specBounceLimit > 1u : b + 1u < SEGS && b + 1u < p.specBounceLimit)) {
                                // the bounce
                                more = true;
                                W.con[up][q] = mult.x * (hv.albedo.x * cmul * hm.specular);
                                W.con[up + 1u][q] = mult.y * (hv.albedo.y * cmul * hm.specular);
                                W.con[up + 2u][q] = mult.z * (hv.albedo.z * cmul * hm.specular);
                                const f3 nd = reflect(s.dir, hv.normal);
                                ray_begin<FAR, TINTED>(s, m, hpos, nd, rcp3(nd), true, c, W.tint, lane);
                                s.flags |= ((SEGS == 2u ? 1u : b + 1u) << RF_BOUNCES) | (hm.reflectType == 1u ? RF_SKY : 0u);
                                c.rays++;
                            }
                        }
                    }
                } else if (dot(s.dir, mk(p.sunDir[0], p.sunDir[1], p.sunDir[2])) > 0.99f) {
                    sc.x = sun.x * cmul + cadd.x;
                    sc.y = sun.y * cmul + cadd.y;
                    sc.z = sun.z * cmul + cadd.z;
                } else {
                    const bool reflectsSky = b ? (s.flags & RF_SKY) != 0u : mats[pv.tmat].reflectType == 1u;
                    const f3 sky = reflectsSky ? sky_color(mk(p.skyBot[0], p.skyBot[1], p.skyBot[2]),
                                                           mk(p.skyTop[0], p.skyTop[1], p.skyTop[2]), s.dir) : sun;
                    sc.x = (sky.x * cmul + cadd.x) * mult.x;
                    sc.y = (sky.y * cmul + cadd.y) * mult.y;
                    sc.z = (sky.z * cmul + cadd.z) * mult.z;
                }
                if (add_) {
                    W.con[at][q] = sc.x; W.con[at + 1u][q] = sc.y; W.con[at + 2u][q] = sc.z;
                }
                if (!more) W.ncon[q] = (uint8_t)((SEGS == 2u ? (b ? 1u : 0u) : b) + (add_ ? 1u : 0u));
            }
            __syncwarp();
            // the pool's sums in the reference's order (ray, then segment), a component of a voxel's specular or
            // direct light per lane, written as the voxel's lighting (voxelLighting.comp:266-288, FP32)
            const uint32_t nSpecSums = (uint32_t)__popc(specs) * 3u, nFanSums = (uint32_t)__popc(fans) * 3u;
            const uint32_t nSums = nSpecSums + nFanSums + (uint32_t)__popc(firsts) * 3u;
            for (uint32_t i = lane; i < nSums; i += 32u) {
                float acc = 0.0f;
                if (i < nSpecSums) {
                    const uint32_t j = i / 3u, comp = i - 3u * j, v = W.specList[j];
                    for (uint32_t k = j * K; k < j * K + K; k++) {
                        const uint32_t n = W.ncon[k];
                        if (n > 0u) acc = acc + W.con[comp][k];
                        if (n > 1u) acc = acc + W.con[3u + comp][k];
                        if constexpr (SEGS > 2u)
                            for (uint32_t b = 2; b < n; b++) acc = acc + W.con[3u * b + comp][k];
                    }
                    acc = acc / (float)K;
                    float* o = (float*)&out[((uint64_t)req * 32u + first + v) * 2u + 1u];
                    o[comp] = gmin(gmax(acc, 0.0f), 1.0f);
                    if (comp == 0u) o[3] = 0.0f;
                } else {
                    const uint32_t i2 = i - nSpecSums;
                    const bool fan = i2 < nFanSums;
                    const uint32_t i3 = fan ? i2 : i2 - nFanSums, j = i3 / 3u, comp = i3 - 3u * j;
                    const uint32_t v = fan ? W.fanList[j] : W.firstList[j];
                    const uint32_t k0 = fan ? j * K : nFan + j, n = fan ? K : 1u;
                    for (uint32_t k = k0; k < k0 + n; k++)
                        if (W.shHas[k]) acc = acc + W.sh[comp][k];
                    acc = acc / (float)n;
                    float* o = (float*)&out[((uint64_t)req * 32u + first + v) * 2u];
                    o[comp] = acc;
                    if (comp == 0u) o[3] = 0.0f;
                }
            }
        }
        __syncwarp();   // the unit's voxels are read no more
    }
    flush_counters(MANY ? many->stats : one->stats, c, 0, lit);
}

} // namespace dn
