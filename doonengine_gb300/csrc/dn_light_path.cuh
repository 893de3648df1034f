/*
 * dn_light_path.cuh -- the diffuse paths of a lighting update (voxelLighting.comp:148-214, 238-288).
 *
 * The packet kernel (dn_light_packet.cuh) leaves each voxel's direct light in its diffuse output slot; this kernel
 * traces the voxel's numDiffuse paths of up to diffuseBounceLimit segments, forms the running average and replaces
 * the slot.  Every lane owns one voxel and walks its paths in the reference's order (launches of few voxels: see
 * path_share); a lane whose voxel is done takes the next one of its warp's window, so that a long path holds no other
 * lane.  The paths of a warp have nothing in
 * common, so the walk's rounds run with about a third of the lanes, and what a segment's end needs runs for all
 * waiting lanes at once when `batch` of them wait (or none is left stepping).
 *
 * The code between segments is one sequence -- finish, fetch, choose the direction, begin -- with each part in one
 * place: as branches of one advance function, with the direction and the ray's start inlined at three ends, the
 * kernel was 54 KB and waited for instructions a quarter of the time (2.7 of 10.9 cycles per instruction).
 * With this loop and voxels found by their partial counts, us per frame or call, before -> after: 23x11x37 map with 2
 * paths per voxel 575 -> 464; 16x16x16 map 520 -> 461; glass 2653 -> 2435; twelve maps batched 11806 -> 10142; 64x32x64
 * map at 1080p 12324 -> 11826.
 */
#pragma once
#include "dn_light_stream.cuh"

// 7 blocks of 4 warps per SM (68 registers, 71 and 72 with paths side by side); 6 and 8 within 1 %
#ifndef DN_DIFF_MIN_BLOCKS
#define DN_DIFF_MIN_BLOCKS 7
#endif

namespace dn {

// per-lane voxel and path (shared memory, touched between segments only; an odd number of words per lane)
struct PathJob {
    f3 pos0, tnormal, direct;
    f3 acc, carry, normal;       // the voxel's sum; the path's colour so far; the normal the next direction starts from
    uint32_t material;           // of the last hit
    uint32_t key, vidx, req, vlane;   // vlane: bits 0-4; bit 9: the lane has one path of the voxel, others the rest
    float indirect;              // weight of the lighting so far (0: the voxel's first sample)
    uint32_t b, i;               // bounce, path
    uint32_t draw;               // what the next direction's sphere point is drawn with (path_base)
};
static_assert(sizeof(PathJob) % 8 == 4, "odd number of words");

// The voxel's new diffuse lighting from its paths' sum (voxelLighting.comp:266-278, FP32)
__device__ __forceinline__ void path_write(const PathJob& j, const DevMap& m, const dn_light_params& p, float4* out)
{
    const float4 prev = __ldg(&m.diff[j.vidx]);
    const float den = j.indirect + (float)p.numDiffuse;
    const f3 d = mk((prev.x * j.indirect + j.acc.x) / den, (prev.y * j.indirect + j.acc.y) / den,
                    (prev.z * j.indirect + j.acc.z) / den);
    out[((uint64_t)j.req * 32u + (j.vlane & 31u)) * 2u] = make_float4(gmin(gmax(d.x, 0.0f), 1.0f), gmin(gmax(d.y, 0.0f), 1.0f),
                                                             gmin(gmax(d.z, 0.0f), 1.0f), 0.0f);
}

// Sets up voxel (req, vlane); false when the slot holds no voxel with diffuse paths, or its lighting needs no ray and
// is written here.
__device__ __forceinline__ bool path_setup(PathJob& j, uint32_t req, uint32_t vlane, const DevMap& m, const dn_light_params& p,
                                           const Material* mats, const uint32_t* reqs, const uint32_t* nsamples, float4* out)
{
    const uint32_t word = reqs[req];
    const uint32_t tile = word >> 4, group = word & 15u;
    const uint32_t tw = __ldg(&m.tword[tile]);
    const uint32_t vn = group * 32u + vlane;
    i3 cp; uint32_t li;
    const ChunkRec* rc = &m.rec[tw & SLOT_MASK];
    if ((tw >> 30) != 2u || vn >= __ldg(&rc->nvox) || !select_voxel(rc, vn, cp, li)) return false;
    const i3 mp{__ldg(&rc->pos[0]), __ldg(&rc->pos[1]), __ldg(&rc->pos[2])};
    j.req = req; j.vlane = vlane;
    j.vidx = __ldg(&rc->voxBase) + vn;
    const uint2 w = __ldg(&m.vox[j.vidx]);
    if (!(mats[w.x >> 24].specular < 1.0f)) return false;
    j.tnormal = voxel_normal(w);
    const uint32_t samples = __ldg(&nsamples[tw & SLOT_MASK]);
    j.indirect = (float)(samples < p.maxDiffuse ? samples : p.maxDiffuse);
    const uint32_t gx = (uint32_t)(mp.x * 8 + cp.x), gy = (uint32_t)(mp.y * 8 + cp.y), gz = (uint32_t)(mp.z * 8 + cp.z);
    j.key = rng_key(__float_as_uint(p.time), p.mapId, gx + (m.sx * 8u) * (gy + (m.sy * 8u) * gz));
    f3 rp;
    rp.x = INV_CHUNK * (float)cp.x + (float)mp.x + HALF_INV_CHUNK;
    rp.y = INV_CHUNK * (float)cp.y + (float)mp.y + HALF_INV_CHUNK;
    rp.z = INV_CHUNK * (float)cp.z + (float)mp.z + HALF_INV_CHUNK;
    const float off = HALF_INV_CHUNK - EPS;
    j.pos0 = add(rp, muls(j.tnormal, off));
    const float4 d = out[((uint64_t)req * 32u + vlane) * 2u];
    j.direct = mk(d.x, d.y, d.z);
    j.acc = mk(0.0f, 0.0f, 0.0f);
    j.i = 0;
    if (p.numDiffuse == 0u || p.diffuseBounceLimit == 0u) {
        const f3 amb = mk(p.ambient[0], p.ambient[1], p.ambient[2]);
        for (uint32_t i = 0; i < p.numDiffuse; i++) j.acc = add(add(j.acc, amb), j.direct);
        path_write(j, m, p, out);
        return false;
    }
    return true;
}

// What the path's next direction is formed from (voxelLighting.comp:160-168); last: the direction of the segment before
// it.  point: the direction takes a point of the unit sphere, drawn with j.draw; lobe: it is a reflection's.
__device__ __forceinline__ f3 path_base(PathJob& j, f3 last, const dn_light_params& p, const Material* mats, bool& point, bool& lobe)
{
    const bool rngSin = p.rngMode == 1u;
    const uint32_t at = j.i * 16u + j.b;
    const float seed = p.time * (float)(j.i + 1u);
    lobe = false;
    f3 base = j.normal;
    if (j.b > 0u) {
        const Material& hm = mats[j.material];
        const float r = rngSin ? srand1(seed + (float)p.diffuseBounceLimit + (float)j.b) : hrand(j.key, 2u, at << 8);
        lobe = (r + 1.0f) * 0.5f < hm.specular;
        if (lobe) base = muls(reflect(last, j.normal), (float)hm.shininess);
    }
    point = lobe || j.indirect != 0.0f;
    j.draw = rngSin ? __float_as_uint((lobe ? p.time : seed) + (float)j.b) : ((lobe ? 3u : 1u) << 28) ^ (at << 8);
    return base;
}

// Points of the unit sphere for the lanes with `need`: the first try inside it (sphere_hash, sphere_sin), found by the
// whole warp.  About half of the tries are inside, so a lane alone makes 1.9 tries, but a warp whose lanes each make
// their own runs until its unluckiest lane is done (5.5 tries for 24 lanes), and reflections' and other directions'
// loops ran one after the other: directions took 45 % of the kernel's instructions.  Here every lane makes one try per
// round and the lanes that still need a point share all 32: 24 lanes are done in three rounds.  jobs, order: the warp's.
// us per pass, before -> after: 16x16x16 map (two frames) 426 -> 405; four updates of a 16x12x16 map with 4 paths per
// voxel 5248 -> 4770; twelve maps batched 9413 -> 9104; 64x32x64 map at 1080p 11066 -> 10990.
__device__ __forceinline__ f3 warp_sphere_points(bool need, bool sine, const PathJob* jobs, uint8_t* order)
{
    const uint32_t lane = lane_id_s();
    f3 point = mk(0.0f, 0.0f, 0.0f);
#pragma unroll 1
    for (uint32_t tried = 0; tried < 64u;) {
        const uint32_t left = __ballot_sync(0xFFFFFFFFu, need);
        if (left == 0u) break;
        // 2^share lanes for each of the n points left
        const uint32_t n = (uint32_t)__popc(left), share = (uint32_t)__clz((int)(n - 1u)) - 27u;
        const uint32_t rank = (uint32_t)__popc(left & ((1u << lane) - 1u));
        if (need) order[rank] = (uint8_t)(lane | (sine ? 32u : 0u));
        __syncwarp();
        const uint32_t t = tried + (lane & ((1u << share) - 1u));
        f3 q = mk(0.0f, 0.0f, 0.0f);
        bool inside = false;
        if (lane >> share < n && t < 64u) {
            const uint32_t who = order[lane >> share];
            const PathJob& j = jobs[who & 31u];
            if (who & 32u) {
                float at = __uint_as_float(j.draw);
                for (uint32_t i = 0; i < t; i++) at = at + 1.0f;
                q = sphere_try_sin(at);
            } else {
                q = sphere_try_hash(j.key, j.draw ^ (3u * t), j.draw ^ (3u * t + 1u), j.draw ^ (3u * t + 2u));
            }
            inside = !(dot(q, q) >= 1.0f);
        }
        const uint32_t found = (__ballot_sync(0xFFFFFFFFu, inside) >> ((rank << share) & 31u)) & (0xFFFFFFFFu >> (32u - (1u << share)));
        const uint32_t from = found ? (rank << share) + (uint32_t)__ffs((int)found) - 1u : lane;
        const f3 got = mk(__shfl_sync(0xFFFFFFFFu, q.x, (int)from), __shfl_sync(0xFFFFFFFFu, q.y, (int)from),
                          __shfl_sync(0xFFFFFFFFu, q.z, (int)from));
        if (need && found) { point = got; need = false; }
        tried += 1u << share;
        __syncwarp();
    }
    return point;
}

// the map whose range of a queue holds r: starts[map] <= r < starts[map + 1]
__device__ __forceinline__ uint32_t window_map(const uint32_t* starts, uint32_t nmaps, uint32_t r)
{
    uint32_t lo = 0, hi = nmaps;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&starts[mid]) <= r) lo = mid; else hi = mid;
    }
    return lo;
}

// Paths side by side (SIDE).  In a launch of at most two voxels per lane (counted in whole groups, of which about two
// thirds hold voxels) a lane's paths, one after the other, would be the launch's length while other lanes have nothing to
// do; there a voxel takes several lanes, a path each, and when the paths of all a warp's voxels have ended one lane per
// voxel adds them up in order.  How many lanes: all its paths up to 32; 16 for more, which then takes several passes with
// the sum carried on (16 and not 32: 33 paths are 3 passes of two voxels at a time instead of 2 passes of one).  Each
// window of the queue is taken by its own map's rule, so maps with one path keep a lane per voxel beside others.
// SIDE 0: a lane per voxel; 1: no map of the launch has more than 32 paths; 2: passes too (they cost the others 2.7 %).
// us per lighting update, a lane per voxel -> side by side: 3x2x3 map (0.002 voxels per lane) 4 paths 76 -> 47, 32 353 ->
// 57, 64 673 -> 103; 12x8x12 (0.55) 4 397 -> 278, 17 1035 -> 630, 33 1804 -> 857; 22x12x22 (1.84) 2 599 -> 569, 17 1979 ->
// 1959, 32 3338 -> 2240, 33 3418 -> 2685.  Batched frames: twelve 5x4x6 maps, 32 paths on one and 1 on the others, 1360 ->
// 447, with 33 on all 2181 -> 1517; a 3x2x3 map with 4, 16 or 64 paths beside two 14x9x14 maps with one, 294, 507, 1345 ->
// 284, 290, 330.  The line lies at two voxels per lane because up to there no number of paths loses; above it those that
// leave lanes of a warp without a path do (28x12x28, 2.8: 17 paths 2757 -> 3088, 32 4570 -> 3554), and below it all would
// lose by a lower line (18x12x18, 1.25: 4 paths 479, a lane per voxel 603).
__host__ __device__ __forceinline__ uint32_t path_share(const dn_light_params& p)
{
    return p.numDiffuse < 2u || p.diffuseBounceLimit == 0u ? 1u : p.numDiffuse <= 32u ? p.numDiffuse : 16u;
}
__device__ __forceinline__ bool paths_side_by_side(uint32_t nreq, uint32_t lanes) { return nreq <= lanes / 16u; }

// a map's windows are 2^-result of a request group: as parts for all maps (window_parts), smaller where a window's paths
// would fill a warp more than once
__device__ __forceinline__ uint32_t share_parts(uint32_t parts, uint32_t share)
{
    while (parts < 5u && (32u >> parts) * share > 32u) parts++;
    return parts;
}

// The persistent loop of the launch: one map (one) or a queue over the requests of many maps (many), each lane then
// reading its voxel's map through that map's entry of the device table.  FAR: maps above FAR_SUM chunks (dn_walk.cuh).
template <bool MANY, bool TINTED, uint32_t SIDE, bool FAR>
__device__ __forceinline__ void path_loop(const StreamArgs* one, const BatchLightArgs* many, uint32_t nreq, PathJob& j,
                                          TintT<128>& tint, uint8_t* order)
{
    const uint32_t lane = lane_id_s(), col = threadIdx.x;
    const uint32_t batch = MANY ? many->batch : one->batch;
    uint32_t* const counter = (MANY ? many->workCounter : one->workCounter) + 1;
    uint32_t winMap = 0, winReq = 0, winNext = 32, winEnd = 32;   // warp-uniform voxel window: map, request, next voxel, end
    const uint32_t allParts = window_parts(nreq, gridDim.x * (blockDim.x / 32u));
    // the queue: windows of the maps one after the other
    const uint32_t* const starts = MANY ? (SIDE != 0u ? many->winStart : many->reqStart) : nullptr;
    auto mapParams = [&](uint32_t map) -> const dn_light_params& { if constexpr (MANY) return many->maps[map].p; else return one->p; };
    uint32_t winShare = 1, parts = allParts;   // SIDE > 0: the lanes a voxel of the window takes, and the window's part of a group
    if constexpr (!MANY && SIDE != 0u) { winShare = path_share(one->p); parts = share_parts(allParts, winShare); }
    uint32_t nwin = nreq << parts;
    if constexpr (MANY && SIDE != 0u) nwin = *(volatile const uint32_t*)&many->winStart[many->nmaps];
    // whether the window's voxels take several lanes (one map: all windows' do)
    auto shared = [&]() { return SIDE != 0u && (!MANY || winShare > 1u); };
    bool team = false;                 // the warp's lanes are on such voxels
    uint32_t first = 0;                // the first path of their pass (SIDE 2)
    uint32_t role = 0;                 // the lane's path in its voxel's pass, from 1 on; 0: none
    bool exhausted = false;
    const BatchLightMap* le = nullptr;
    if constexpr (MANY) le = &many->maps[0];
    auto M = [&]() -> const DevMap& { if constexpr (MANY) return le->m; else return one->m; };
    auto P = [&]() -> const dn_light_params& { if constexpr (MANY) return le->p; else return one->p; };
    auto MATS = [&]() -> const Material* { if constexpr (MANY) return le->mats; else return one->gtab->mats; };
    auto OUT = [&]() -> float4* { if constexpr (MANY) return le->out; else return one->out; };
    Ray s;
    s.mode = RM_IDLE;
    bool own = false, done = false;    // the lane has a voxel; no voxel is left for it
    Counters c{0, 0, 0, 0, 0};
    for (;;) {
        const unsigned waiting = __ballot_sync(0xFFFFFFFFu, !ray_stepping(s) && !done);
        const unsigned stepping = __ballot_sync(0xFFFFFFFFu, ray_stepping(s));
        if ((waiting | stepping) == 0u) break;
        bool go = stepping == 0u;
        if (shared() && (!MANY || team || winNext < winEnd)) {
            // lanes whose path is done wait for their voxel's others, or for the lanes that finish before the warp turns to
            // the window's voxels: the threshold is a share of the lanes at work
            const unsigned work = __ballot_sync(0xFFFFFFFFu, own);
            go = go || (uint32_t)__popc(work & ~stepping) * 32u >= batch * (uint32_t)__popc(work);
        } else {
            go = go || (uint32_t)__popc(waiting) >= batch;
        }
        if (go) {
            bool start = false;        // the lane's next segment starts
            f3 org = mk(0.0f, 0.0f, 0.0f);
            if (s.mode == RM_HIT || s.mode == RM_MISS) {
                // diffuse_ray body after step_map (voxelLighting.comp:176-201)
                f3 cadd;
                float cmul;
                ray_tint<TINTED>(s, tint, col, cadd, cmul);
                if (s.mode == RM_HIT) {
                    org = ray_hit_position<FAR>(s);
                    const uint2 w = __ldg(&M().vox[ray_hit_index(s, M())]);
                    const f3 albedo = mk((float)((w.y >> 24) & 0xFF) * INV255, (float)((w.y >> 16) & 0xFF) * INV255,
                                         (float)((w.y >> 8) & 0xFF) * INV255);
                    j.normal = voxel_normal(w);
                    j.material = w.x >> 24;
                    const f3 d = vabs(sub(vfloor(muls(j.pos0, 8.0f)), vfloor(muls(org, 8.0f))));
                    if (!(dot(d, d) < 1.0f)) {
                        if (MATS()[j.material].emissive) {
                            const float e = P().emissiveStrength;
                            j.acc.x = j.acc.x + j.carry.x * (albedo.x * e * cmul + cadd.x);
                            j.acc.y = j.acc.y + j.carry.y * (albedo.y * e * cmul + cadd.y);
                            j.acc.z = j.acc.z + j.carry.z * (albedo.z * e * cmul + cadd.z);
                        } else {
                            j.carry.x = j.carry.x * (albedo.x * cmul + cadd.x);
                            j.carry.y = j.carry.y * (albedo.y * cmul + cadd.y);
                            j.carry.z = j.carry.z * (albedo.z * cmul + cadd.z);
                            j.b++;
                            start = j.b < P().diffuseBounceLimit;
                        }
                    }
                } else {
                    const float k = gmax(dot(s.dir, mk(P().sunDir[0], P().sunDir[1], P().sunDir[2])), 0.0f);
                    j.acc.x = j.acc.x + (j.carry.x * k * P().sunStrength[0] * cmul + cadd.x);
                    j.acc.y = j.acc.y + (j.carry.y * k * P().sunStrength[1] * cmul + cadd.y);
                    j.acc.z = j.acc.z + (j.carry.z * k * P().sunStrength[2] * cmul + cadd.z);
                }
                s.mode = RM_IDLE;
                if (!start) {
                    if (SIDE != 0u && j.vlane >= 512u) {
                        own = false;
                    } else {
                        j.acc = add(j.acc, j.direct);
                        j.i++;
                        if (j.i >= P().numDiffuse) {
                            path_write(j, M(), P(), OUT());
                            own = false;
                        }
                    }
                }
            }
            if (SIDE != 0u && team && __ballot_sync(0xFFFFFFFFu, own) == 0u) {
                // a pass has ended: its paths are added to the voxels' sums in the reference's order.  (A path adds at most
                // one contribution; one without adds zero, which changes no sum.)  The sum is carried where the voxel's
                // second lane keeps the direct light, which only the first one needs.
                uint32_t paths = winShare;
                if constexpr (SIDE == 2u) paths = mapParams(winMap).numDiffuse;
                __syncwarp();
                if (role == 1u) {
                    f3 acc = mk(0.0f, 0.0f, 0.0f);
                    if (SIDE == 2u && first) acc = (&j)[1].direct;
                    const f3 amb = mk(P().ambient[0], P().ambient[1], P().ambient[2]);
                    const uint32_t n = SIDE == 2u ? min(winShare, paths - first) : winShare;
                    for (uint32_t i = 0; i < n; i++) acc = add(add(add(acc, amb), (&j)[i].acc), j.direct);
                    if (SIDE == 2u && first + winShare < paths) {
                        (&j)[1].direct = acc;
                    } else {
                        j.acc = acc;
                        path_write(j, M(), P(), OUT());
                    }
                }
                __syncwarp();
                team = false;
                if constexpr (SIDE == 2u) {
                    first += winShare;
                    team = first < paths;
                    if (team && role) {
                        j.acc = mk(0.0f, 0.0f, 0.0f);
                        j.i = first + role - 1u;
                        own = j.i < paths;
                    }
                }
                if (!team) role = 0;
            }
            // voxels for the lanes without one
            for (;;) {
                const unsigned need = __ballot_sync(0xFFFFFFFFu, !own && !done);
                if (need == 0u || (SIDE != 0u && team)) break;
                if (winNext >= winEnd) {
                    uint32_t r = 0;
                    if (!exhausted && lane == 0) r = atomicAdd(counter, 1u);
                    r = __shfl_sync(0xFFFFFFFFu, r, 0);
                    if (exhausted || r >= nwin) {
                        exhausted = true;
                        if (!own) done = true;
                        break;
                    }
                    if constexpr (MANY && SIDE != 0u) {
                        winMap = window_map(starts, many->nmaps, r);
                        r -= __ldg(&starts[winMap]);
                        winShare = path_share(mapParams(winMap));
                        parts = share_parts(allParts, winShare);
                    }
                    winNext = (r & ((1u << parts) - 1u)) << (5u - parts);
                    winEnd = winNext + (32u >> parts);
                    r >>= parts;
                    if constexpr (MANY && SIDE == 0u) {
                        winMap = window_map(starts, many->nmaps, r);
                        r -= __ldg(&starts[winMap]);
                    }
                    winReq = r;
                }
                if (shared()) {
                    if (need != 0xFFFFFFFFu) break;   // the lanes at work finish first
                    const uint32_t nvox = min(32u / winShare, winEnd - winNext), v = lane / winShare;
                    if (v < nvox) {
                        if constexpr (MANY) {
                            le = &many->maps[winMap];
                            own = path_setup(j, winReq, winNext + v, le->m, le->p, le->mats, le->reqs, le->nsamples, le->out);
                        } else {
                            own = path_setup(j, winReq, winNext + v, one->m, one->p, MATS(), one->reqs, one->nsamples, one->out);
                        }
                        if (own) {
                            role = lane - v * winShare + 1u;
                            j.i = role - 1u;
                            j.vlane |= 512u;
                        }
                    }
                    winNext += nvox;
                    first = 0;
                    team = __ballot_sync(0xFFFFFFFFu, own) != 0u;
                    continue;
                }
                const uint32_t rank = __popc(need & ((1u << lane) - 1u));
                if (!own && !done && winNext + rank < winEnd) {
                    if constexpr (MANY) {
                        le = &many->maps[winMap];
                        own = path_setup(j, winReq, winNext + rank, le->m, le->p, le->mats, le->reqs, le->nsamples, le->out);
                    } else {
                        own = path_setup(j, winReq, winNext + rank, one->m, one->p, MATS(), one->reqs, one->nsamples, one->out);
                    }
                }
                const uint32_t took = (uint32_t)__popc(need) < winEnd - winNext ? (uint32_t)__popc(need) : winEnd - winNext;
                winNext += took;
            }
            // the next segment: a bounce, or a path's first
            const bool begin = own && !ray_stepping(s);
            bool point = false, lobe = false;
            f3 base = mk(0.0f, 0.0f, 0.0f);
            if (begin) {
                if (!start) {
                    if (SIDE == 0u || j.vlane < 512u) j.acc = add(j.acc, mk(P().ambient[0], P().ambient[1], P().ambient[2]));
                    j.carry = mk(1.0f, 1.0f, 1.0f);
                    j.normal = adds(j.tnormal, EPS);
                    j.b = 0;
                    org = j.pos0;
                }
                base = path_base(j, s.dir, P(), MATS(), point, lobe);
            }
            const f3 rs = warp_sphere_points(point, P().rngMode == 1u, &j - lane, order);
            if (begin) {
                f3 d = normalize(point ? add(base, rs) : base);
                if (!lobe) d = adds(d, EPS);
                ray_begin<FAR, TINTED>(s, M(), org, d, rcp3(d), start, c, tint, col);
                c.rays++;
            }
        }
        if (ray_stepping(s)) walk_round<FAR, TINTED>(s, M(), MATS(), P().sunStrength, c, tint, col);
    }
    flush_counters(MANY ? many->stats : one->stats, c, 0, 0);
}

// the SIDE a map asks for
__host__ __device__ __forceinline__ uint32_t path_side(const dn_light_params& p)
{
    return path_share(p) == 1u ? 0u : p.numDiffuse <= 32u ? 1u : 2u;
}

// the loop a launch runs: with paths side by side or a lane per voxel
template <bool MANY, uint32_t SIDE, bool FAR>
__device__ __forceinline__ void path_launch(const StreamArgs* one, const BatchLightArgs* many, bool tinted, PathJob& j,
                                            TintT<128>& tint, uint8_t* order)
{
    const uint32_t nreq = MANY ? *(volatile const uint32_t*)&many->reqStart[many->nmaps] : *(volatile const uint32_t*)one->nreqPtr;
    if constexpr (SIDE != 0u) {
        if (paths_side_by_side(nreq, gridDim.x * blockDim.x)) {
            if (tinted) path_loop<MANY, true, SIDE, FAR>(one, many, nreq, j, tint, order);
            else path_loop<MANY, false, SIDE, FAR>(one, many, nreq, j, tint, order);
            return;
        }
    }
    if (FAR || tinted) path_loop<MANY, true, 0, FAR>(one, many, nreq, j, tint, order);
    else if constexpr (!FAR) path_loop<MANY, false, 0, false>(one, many, nreq, j, tint, order);
}

} // namespace dn
