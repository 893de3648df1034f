/*
 * dn_light_stream.cuh -- the lighting update as persistent per-lane ray streams.
 *
 * Every lane of a warp owns one voxel at a time and walks that voxel's ray
 * jobs in the reference's order (voxelLighting.comp:238-264):
 *   K specular rays (each up to specBounceLimit segments), then the direct
 *   light rays (K fixed shadow rays, or one along the sun on the first
 *   sample), then numDiffuse diffuse paths (each up to diffuseBounceLimit
 *   segments), then the running average and the write-out.
 * All lanes share one loop whose body is one round of each lane's current ray
 * segment (walk_round, dn_walk.cuh), so lanes on different rays, different jobs
 * or different voxels still execute together.  When a segment ends, the lane waits; the per-segment work
 * (shading the finished segment, choosing and setting up the next one,
 * finishing a voxel, fetching the next voxel) runs for all waiting lanes at
 * once when at least `batch` lanes wait (or no lane is still stepping).
 * Each lane accumulates its voxel's sums in exactly the order of the
 * reference loops, so results are bit-identical to the one-voxel-at-a-time
 * form; only the schedule differs.  Voxels are fetched one per lane from a
 * warp-local window over the request list, refilled with one atomic per
 * 32 voxels.
 */
#pragma once
#include "dn_internal.cuh"

namespace dn {

#ifndef DN_STREAM_MIN_BLOCKS
#define DN_STREAM_MIN_BLOCKS 4   // 4 blocks of 4 warps per SM (measured best: leaves L1 room for the tile map)
#endif

enum : uint32_t { PH_FETCH = 0, PH_SPEC = 1, PH_SHADOW = 2, PH_DIFF = 3, PH_FINAL = 4, PH_DONE = 5 };

struct StreamArgs {
    DevMap m;
    const uint32_t* reqs;
    uint32_t* workCounter;            // [2], DevState::work
    const uint32_t* nreqPtr;
    const uint32_t* nsamples;
    float4* out;
    unsigned long long* stats;
    uint32_t batch;
    dn_light_params p;
    const struct LightTables* gtab;   // the launch's materials and shadow directions (k_light_prep)
    const uint32_t* mixed;            // nonzero: a loaded chunk has see-through voxels (mark_opaque_cells)
};

struct MaterialTable { Material m[256]; };

// per-launch tables the lighting kernels read through L1: the materials and the shadow directions
struct LightTables {
    Material mats[256];
    float sdir[65][3];   // shadow directions k < K, [64]: the first-sample direction sunDir + EPS
    float sinv[65][3];
    float pts[64][3];    // the specular fan's offsets
};

__device__ __forceinline__ f3 rcp3(f3 d) { return mk(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)); }

// per-lane job state of the voxel being lit
struct Job {
    uint32_t phase, k, b, i;
    uint32_t req, vlane, vidx;      // request, lane within it, pool index of the voxel
    f3 pos0, tnormal, talbedo, refl;
    uint32_t tmat, key;
    float indirect;
    bool firstSample, doSpec, doDiff;
    f3 spec, direct, acc;           // acc: shadow sum, then diffuse sum
    f3 jA, jB, jC;                  // spec: mult, lastPos ; diffuse: nc, hitNormal, lastDir
    uint32_t jU;                    // spec: reflectType ; diffuse: material of the last hit
    uint32_t map;                   // many-map launches: the voxel's map
};

} // namespace dn

namespace dn {

__device__ __forceinline__ uint32_t lane_id_s()
{
    uint32_t l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
    return l;
}

struct StreamShared {
    Material mats[256];
    float sdir[65][3];   // shadow directions k < K, [64]: the first-sample direction sunDir + EPS
    float sinv[65][3];
};


// diffuse bounce direction (voxelLighting.comp:160-168)
__device__ __forceinline__ f3 diffuse_dir(const Job& j, const dn_light_params& p, const Material* mats, bool rngSin)
{
    const Material& hm = mats[j.jU];
    bool lobe = false;
    const float seed = p.time * (float)(j.i + 1u);
    if (j.b > 0) {
        const float r = rngSin ? srand1(seed + (float)p.diffuseBounceLimit + (float)j.b)
                               : hrand(j.key, 2u, (j.i * 16u + j.b) << 8);
        lobe = (r + 1.0f) * 0.5f < hm.specular;
    }
    if (lobe) {
        const f3 rs = rngSin ? sphere_sin(p.time + (float)j.b) : sphere_hash(j.key, 3u, j.i * 16u + j.b);
        return normalize(add(muls(reflect(j.jC, j.jB), (float)hm.shininess), rs));
    }
    if (j.firstSample) return adds(normalize(j.jB), EPS);
    const f3 rs = rngSin ? sphere_sin(seed + (float)j.b) : sphere_hash(j.key, 1u, j.i * 16u + j.b);
    return adds(normalize(add(j.jB, rs)), EPS);
}

// Consumes the finished segment (hitState 1 hit / 2 miss) and sets up the next segment of this lane's
// voxel; returns true when a segment was started.  Leaves the job in PH_FETCH when the voxel is done.
template <bool FAR>
__device__ __forceinline__ bool advance(Job& j, Ray& s, TintT<128>& tint, const DevMap& m, const dn_light_params& p,
                                        const Material* mats, const float (*sdir)[3], const float (*sinv)[3],
                                        float4* out, Counters& c, uint32_t& lit)
{
    const bool rngSin = p.rngMode == 1u;
    const f3 sun = mk(p.sunStrength[0], p.sunStrength[1], p.sunStrength[2]);
    const f3 sunDir = mk(p.sunDir[0], p.sunDir[1], p.sunDir[2]);
    if (s.mode == RM_HIT || s.mode == RM_MISS) {
        const bool hit = s.mode == RM_HIT;
        s.mode = RM_IDLE;
        Voxel hv;
        f3 hpos = s.pos, cadd;
        float cmul;
        ray_tint<true>(s, tint, threadIdx.x, cadd, cmul);
        if (hit) {
            hpos = ray_hit_position<FAR>(s);
            decompress(m, ray_hit_index(s, m), hv);
        }
        if (j.phase == PH_SPEC) {
            // specular_ray body after step_map (voxelLighting.comp:98-144)
            bool done = true;
            if (hit) {
                const i3 hp{f2i(hpos.x), f2i(hpos.y), f2i(hpos.z)};
                if (in_map(m, hp)) {
                    uint8_t* vp = &m.tvis[map_index(m, hp)];
                    if (*vp == 0) *vp = 1;
                }
                const f3 d = vabs(sub(vfloor(muls(hpos, 8.0f)), vfloor(muls(j.jB, 8.0f))));
                if (!(dot(d, d) <= 1.0f)) {
                    const Material& hm = mats[hv.material];
                    const f3 hd = muls(hv.diff, 1.0f - hm.specular);
                    if (hm.emissive) {
                        j.spec.x = j.spec.x + ((hv.albedo.x * p.emissiveStrength * cmul + cadd.x) * j.jA.x) * j.talbedo.x;
                        j.spec.y = j.spec.y + ((hv.albedo.y * p.emissiveStrength * cmul + cadd.y) * j.jA.y) * j.talbedo.y;
                        j.spec.z = j.spec.z + ((hv.albedo.z * p.emissiveStrength * cmul + cadd.z) * j.jA.z) * j.talbedo.z;
                    } else {
                        const f3 hc = mul(hd, hv.albedo);
                        j.spec.x = j.spec.x + (hc.x * cmul + cadd.x) * j.jA.x;
                        j.spec.y = j.spec.y + (hc.y * cmul + cadd.y) * j.jA.y;
                        j.spec.z = j.spec.z + (hc.z * cmul + cadd.z) * j.jA.z;
                        if (hm.specular != 0.0f) {
                            j.jA.x = j.jA.x * (hv.albedo.x * cmul * hm.specular);
                            j.jA.y = j.jA.y * (hv.albedo.y * cmul * hm.specular);
                            j.jA.z = j.jA.z * (hv.albedo.z * cmul * hm.specular);
                            j.jU = hm.reflectType;
                            j.jB = hpos;
                            const f3 nd = reflect(s.dir, hv.normal);
                            j.b++;
                            if (j.b < p.specBounceLimit) {
                                ray_begin<FAR, true>(s, m, hpos, nd, rcp3(nd), true, c, tint, threadIdx.x);   // next bounce
                                c.rays++;
                                return true;
                            }
                        }
                    }
                }
            } else if (dot(s.dir, sunDir) > 0.99f) {
                j.spec.x = j.spec.x + (sun.x * cmul + cadd.x);
                j.spec.y = j.spec.y + (sun.y * cmul + cadd.y);
                j.spec.z = j.spec.z + (sun.z * cmul + cadd.z);
            } else {
                const f3 sc = (j.jU == 1u) ? sky_color(mk(p.skyBot[0], p.skyBot[1], p.skyBot[2]),
                                                      mk(p.skyTop[0], p.skyTop[1], p.skyTop[2]), s.dir) : sun;
                j.spec.x = j.spec.x + (sc.x * cmul + cadd.x) * j.jA.x;
                j.spec.y = j.spec.y + (sc.y * cmul + cadd.y) * j.jA.y;
                j.spec.z = j.spec.z + (sc.z * cmul + cadd.z) * j.jA.z;
            }
            if (done) { j.k++; j.b = 0; }
        } else if (j.phase == PH_SHADOW) {
            if (!hit) {
                j.acc.x = j.acc.x + (sun.x * cmul + cadd.x);
                j.acc.y = j.acc.y + (sun.y * cmul + cadd.y);
                j.acc.z = j.acc.z + (sun.z * cmul + cadd.z);
            }
            j.k++;
        } else if (j.phase == PH_DIFF) {
            // diffuse_ray body after step_map (voxelLighting.comp:176-201)
            bool pathDone = true;
            if (hit) {
                j.jB = hv.normal;
                j.jU = hv.material;
                const f3 d = vabs(sub(vfloor(muls(j.pos0, 8.0f)), vfloor(muls(hpos, 8.0f))));
                if (!(dot(d, d) < 1.0f)) {
                    const Material& hm = mats[hv.material];
                    if (hm.emissive) {
                        j.acc.x = j.acc.x + j.jA.x * (hv.albedo.x * p.emissiveStrength * cmul + cadd.x);
                        j.acc.y = j.acc.y + j.jA.y * (hv.albedo.y * p.emissiveStrength * cmul + cadd.y);
                        j.acc.z = j.acc.z + j.jA.z * (hv.albedo.z * p.emissiveStrength * cmul + cadd.z);
                    } else {
                        j.jA.x = j.jA.x * (hv.albedo.x * cmul + cadd.x);
                        j.jA.y = j.jA.y * (hv.albedo.y * cmul + cadd.y);
                        j.jA.z = j.jA.z * (hv.albedo.z * cmul + cadd.z);
                        j.jC = s.dir;
                        j.b++;
                        if (j.b < p.diffuseBounceLimit) {
                            const f3 nd = diffuse_dir(j, p, mats, rngSin);
                            ray_begin<FAR, true>(s, m, hpos, nd, rcp3(nd), true, c, tint, threadIdx.x);
                            c.rays++;
                            return true;
                        }
                    }
                }
            } else {
                const float k = gmax(dot(s.dir, sunDir), 0.0f);
                j.acc.x = j.acc.x + (j.jA.x * k * sun.x * cmul + cadd.x);
                j.acc.y = j.acc.y + (j.jA.y * k * sun.y * cmul + cadd.y);
                j.acc.z = j.acc.z + (j.jA.z * k * sun.z * cmul + cadd.z);
            }
            if (pathDone) { j.acc = add(j.acc, j.direct); j.i++; j.b = 0; }
        }
    }
    // start the next segment of this voxel
    for (int guard = 0; guard < 8; guard++) {
        if (j.phase == PH_SPEC) {
            if (j.k < p.K) {
                if (p.specBounceLimit == 0u) { j.k++; continue; }
                const Material& tm = mats[j.tmat];
                j.b = 0; j.jA = j.talbedo; j.jB = j.pos0; j.jU = tm.reflectType;
                const f3 P = mk(p.spherePts[j.k][0], p.spherePts[j.k][1], p.spherePts[j.k][2]);
                const f3 sd = adds(normalize(add(muls(j.refl, (float)tm.shininess), P)), EPS);
                ray_begin<FAR, true>(s, m, j.pos0, sd, rcp3(sd), false, c, tint, threadIdx.x);
                c.rays++;
                return true;
            }
            j.spec = divs(j.spec, (float)p.K);
            j.phase = j.doDiff ? PH_SHADOW : PH_FINAL;
            j.k = 0;
            continue;
        }
        if (j.phase == PH_SHADOW) {
            const uint32_t n = j.firstSample ? 1u : p.K;
            if (j.k < n) {
                const uint32_t q = j.firstSample ? 64u : j.k;
                ray_begin<FAR, true>(s, m, j.pos0, mk(sdir[q][0], sdir[q][1], sdir[q][2]), mk(sinv[q][0], sinv[q][1], sinv[q][2]), false, c, tint, threadIdx.x);
                c.rays++;
                return true;
            }
            j.direct = divs(j.acc, (float)n);
            j.acc = mk(0.0f, 0.0f, 0.0f);
            j.phase = PH_DIFF;
            j.i = 0; j.b = 0;
            continue;
        }
        if (j.phase == PH_DIFF) {
            if (j.i < p.numDiffuse) {
                if (j.b == 0) {
                    const f3 amb = mk(p.ambient[0], p.ambient[1], p.ambient[2]);
                    j.acc = add(j.acc, amb);
                    if (p.diffuseBounceLimit == 0u) { j.acc = add(j.acc, j.direct); j.i++; continue; }
                    j.jA = mk(1.0f, 1.0f, 1.0f);
                    j.jB = adds(j.tnormal, EPS);
                    j.jC = mk(0.0f, 0.0f, 0.0f);
                    j.jU = j.tmat;
                }
                const f3 nd = diffuse_dir(j, p, mats, rngSin);
                ray_begin<FAR, true>(s, m, j.pos0, nd, rcp3(nd), false, c, tint, threadIdx.x);
                c.rays++;
                return true;
            }
            const float4 prev = __ldg(&m.diff[j.vidx]);
            const float den = j.indirect + (float)p.numDiffuse;
            j.acc.x = (prev.x * j.indirect + j.acc.x) / den;
            j.acc.y = (prev.y * j.indirect + j.acc.y) / den;
            j.acc.z = (prev.z * j.indirect + j.acc.z) / den;
            j.phase = PH_FINAL;
            continue;
        }
        if (j.phase == PH_FINAL) {
            const float4 outS = make_float4(gmin(gmax(j.spec.x, 0.0f), 1.0f), gmin(gmax(j.spec.y, 0.0f), 1.0f),
                                            gmin(gmax(j.spec.z, 0.0f), 1.0f), 0.0f);
            const float4 outD = make_float4(gmin(gmax(j.acc.x, 0.0f), 1.0f), gmin(gmax(j.acc.y, 0.0f), 1.0f),
                                            gmin(gmax(j.acc.z, 0.0f), 1.0f), 0.0f);
            const uint64_t o = ((uint64_t)j.req * 32u + j.vlane) * 2u;
            out[o] = outD;
            out[o + 1] = outS;
            lit++;
            j.phase = PH_FETCH;
        }
        return false;
    }
    return false;
}

// Sets up voxel (req, vlane); returns false (and writes zero outputs) when the slot holds no voxel.
__device__ __forceinline__ bool voxel_setup(Job& j, uint32_t req, uint32_t vlane, const DevMap& m, const dn_light_params& p,
                                            const Material* mats, const uint32_t* reqs, const uint32_t* nsamples, float4* out)
{
    j.req = req; j.vlane = vlane;
    const uint32_t word = reqs[req];
    const uint32_t tile = word >> 4, group = word & 15u;
    const uint32_t tw = __ldg(&m.tword[tile]);
    const uint32_t vn = group * 32u + vlane;
    i3 cp; uint32_t li;
    const ChunkRec* rc = &m.rec[tw & SLOT_MASK];
    if ((tw >> 30) != 2u || vn >= __ldg(&rc->nvox) || !select_voxel(rc, vn, cp, li)) {
        const uint64_t o = ((uint64_t)req * 32u + vlane) * 2u;
        out[o] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        out[o + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return false;
    }
    const i3 mp{__ldg(&rc->pos[0]), __ldg(&rc->pos[1]), __ldg(&rc->pos[2])};
    j.vidx = __ldg(&rc->voxBase) + vn;
    const uint2 w = __ldg(&m.vox[j.vidx]);
    j.tnormal = mk(((float)((w.x >> 16) & 0xFF) * INV255 - 0.5f) * 2.0f, ((float)((w.x >> 8) & 0xFF) * INV255 - 0.5f) * 2.0f,
                   ((float)(w.x & 0xFF) * INV255 - 0.5f) * 2.0f);
    j.tmat = w.x >> 24;
    j.talbedo = mk((float)((w.y >> 24) & 0xFF) * INV255, (float)((w.y >> 16) & 0xFF) * INV255,
                   (float)((w.y >> 8) & 0xFF) * INV255);
    const uint32_t samples = __ldg(&nsamples[tw & SLOT_MASK]);
    const uint32_t ns = samples < p.maxDiffuse ? samples : p.maxDiffuse;
    j.indirect = (float)ns;
    j.firstSample = (j.indirect == 0.0f);
    const uint32_t gx = (uint32_t)(mp.x * 8 + cp.x), gy = (uint32_t)(mp.y * 8 + cp.y), gz = (uint32_t)(mp.z * 8 + cp.z);
    j.key = rng_key(__float_as_uint(p.time), p.mapId, gx + (m.sx * 8u) * (gy + (m.sy * 8u) * gz));
    f3 rp;
    rp.x = INV_CHUNK * (float)cp.x + (float)mp.x + HALF_INV_CHUNK;
    rp.y = INV_CHUNK * (float)cp.y + (float)mp.y + HALF_INV_CHUNK;
    rp.z = INV_CHUNK * (float)cp.z + (float)mp.z + HALF_INV_CHUNK;
    const float off = HALF_INV_CHUNK - EPS;
    j.pos0 = add(rp, muls(j.tnormal, off));
    const Material& tm = mats[j.tmat];
    j.doDiff = tm.specular < 1.0f;
    const f3 viewDir = sub(j.pos0, mk(p.camPos[0], p.camPos[1], p.camPos[2]));
    j.doSpec = tm.specular > 0.0f && dot(viewDir, j.tnormal) < 0.0f && tm.reflectType <= 1u;
    if (j.doSpec) j.refl = reflect(normalize(viewDir), j.tnormal);
    j.spec = mk(0.0f, 0.0f, 0.0f); j.acc = j.spec; j.direct = j.spec;
    j.k = 0; j.b = 0; j.i = 0;
    j.phase = j.doSpec ? PH_SPEC : (j.doDiff ? PH_SHADOW : PH_FINAL);
    return true;
}

// ------------------------------------------------------------ launches

// one map of a many-map lighting launch (device memory, written by the host and by k_batch_prep)
struct BatchLightMap {
    DevMap m;
    const uint32_t* reqs;
    const uint32_t* nsamples;
    float4* out;
    uint32_t* nreqPtr;          // the map's request count (clamped by k_batch_prep)
    uint64_t reqCap;
    dn_light_params p;
    const Material* mats;       // the map's 256 materials
    OpaqueSet opaque;           // those that are opaque
    float4* diffOut;            // committed lighting and sample counts (k_commit_batch)
    float4* specOut;
    uint32_t* samplesOut;
    float sdir[65][3];          // shadow directions of this map (k_batch_prep)
    float sinv[65][3];
};

struct BatchLightArgs {
    BatchLightMap* maps;
    const uint32_t* reqStart;   // [nmaps + 1]: first request of each map in the launch's queue
    const uint32_t* winStart;   // [nmaps + 1]: first window of each map where paths run side by side (dn_light_path.cuh)
    uint32_t nmaps;
    uint32_t* workCounter;
    unsigned long long* stats;
    uint32_t batch;
    uint32_t* mixed;            // nonzero: a loaded chunk of a map has see-through voxels (mark_opaque_cells)
};

// shadow directions normalize(sunDir * softness + P_k) + EPS (k < K) and sunDir + EPS ([64]) with reciprocals
__device__ __forceinline__ void shadow_dir(const dn_light_params& p, int k, float* d3, float* i3)
{
    const f3 sd = mk(p.sunDir[0], p.sunDir[1], p.sunDir[2]);
    f3 d;
    if (k == 64) d = adds(sd, EPS);
    else if ((uint32_t)k < p.K) {
        const f3 P = mk(p.spherePts[k][0], p.spherePts[k][1], p.spherePts[k][2]);
        d = adds(normalize(add(muls(sd, p.shadowSoftness), P)), EPS);
    } else d = mk(1.0f, 1.0f, 1.0f);
    d3[0] = d.x; d3[1] = d.y; d3[2] = d.z;
    i3[0] = __frcp_rn(d.x); i3[1] = __frcp_rn(d.y); i3[2] = __frcp_rn(d.z);
}

// A warp's window into the queue is a whole request group, or a part of one (2^-result) when the launch has fewer
// groups than warps: its few voxels then run on all SMs, and one waits for fewer others.
__device__ __forceinline__ uint32_t window_parts(uint32_t nreq, uint32_t warps)
{
    uint32_t parts = 0;
    while (parts < 5u && (nreq << (parts + 1u)) <= warps) parts++;
    return parts;
}

// The persistent loop of a lighting launch.  MANY = false: one map whose arguments live in the launch's
// parameter space (one) and whose materials and shadow directions were staged into sh.  MANY = true: a
// queue over the requests of many maps (many); each lane reads its current voxel's map, parameters,
// materials and shadow directions from that map's entry of the device table.  FAR: maps above FAR_SUM chunks
// (dn_walk.cuh).
template <bool MANY, bool FAR>
__device__ __forceinline__ void stream_loop(const StreamArgs* one, const BatchLightArgs* many, const StreamShared* sh,
                                            Job& j, TintT<128>& tint)
{
    const uint32_t lane = lane_id_s();
    const uint32_t batch = MANY ? many->batch : one->batch;
    uint32_t nreq = 0;
    if constexpr (MANY) nreq = *(volatile const uint32_t*)&many->reqStart[many->nmaps];
    else nreq = *(volatile const uint32_t*)one->nreqPtr;
    uint32_t* const counter = MANY ? many->workCounter : one->workCounter;
    uint32_t winMap = 0, winReq = 0, winNext = 32, winEnd = 32;   // warp-uniform voxel window: map, request, next voxel, end
    const uint32_t parts = window_parts(nreq, gridDim.x * (blockDim.x / 32u));
    bool exhausted = false;
    j.phase = PH_FETCH;
    j.map = 0;
    // the lane's current map (MANY only), read through its table entry: a register copy of the map's
    // arguments spilled 228 bytes per thread, and the pointer measured +1.2 % on the 64-map workload
    const BatchLightMap* le = nullptr;
    uint32_t lmi = 0xFFFFFFFFu;
    if constexpr (MANY) { le = &many->maps[0]; lmi = 0; }
    auto M = [&]() -> const DevMap& { if constexpr (MANY) return le->m; else return one->m; };
    auto P = [&]() -> const dn_light_params& { if constexpr (MANY) return le->p; else return one->p; };
    auto MATS = [&]() -> const Material* {
        if constexpr (MANY) return le->mats;
        else return sh->mats;
    };
    Ray s;
    s.mode = RM_IDLE;
    Counters c{0, 0, 0, 0, 0};
    uint32_t lit = 0;
    while (true) {
        const unsigned waiting = __ballot_sync(0xFFFFFFFFu, !ray_stepping(s) && j.phase != PH_DONE);
        const unsigned stepping = __ballot_sync(0xFFFFFFFFu, ray_stepping(s));
        if (waiting == 0u && stepping == 0u) break;
        if (stepping == 0u || (uint32_t)__popc(waiting) >= batch) {
            for (int round = 0; round < 4; round++) {
                // warp-cooperative voxel fetch for lanes whose voxel is done
                for (int guard = 0; guard < 64; guard++) {
                    const unsigned need = __ballot_sync(0xFFFFFFFFu, j.phase == PH_FETCH);
                    if (need == 0u) break;
                    if (winNext >= winEnd) {
                        uint32_t r = 0;
                        if (!exhausted && lane == 0) r = atomicAdd(counter, 1u);
                        r = __shfl_sync(0xFFFFFFFFu, r, 0);
                        if (exhausted || r >= nreq << parts) {
                            exhausted = true;
                            if (j.phase == PH_FETCH) j.phase = PH_DONE;
                            break;
                        }
                        winNext = (r & ((1u << parts) - 1u)) << (5u - parts);
                        winEnd = winNext + (32u >> parts);
                        r >>= parts;
                        if constexpr (MANY) {
                            // the map whose request range holds r: reqStart[map] <= r < reqStart[map + 1]
                            uint32_t lo = 0, hi = many->nmaps;
                            while (hi - lo > 1u) {
                                const uint32_t mid = (lo + hi) >> 1;
                                if (__ldg(&many->reqStart[mid]) <= r) lo = mid; else hi = mid;
                            }
                            winMap = lo;
                            winReq = r - __ldg(&many->reqStart[lo]);
                        } else {
                            winReq = r;
                        }
                    }
                    const uint32_t rank = __popc(need & ((1u << lane) - 1u));
                    if (j.phase == PH_FETCH && winNext + rank < winEnd) {
                        if constexpr (MANY) {
                            const BatchLightMap& e = many->maps[winMap];
                            if (winMap != lmi) { le = &e; lmi = winMap; }
                            j.map = winMap;
                            voxel_setup(j, winReq, winNext + rank, e.m, e.p, e.mats, e.reqs, e.nsamples, e.out);
                        } else {
                            voxel_setup(j, winReq, winNext + rank, one->m, one->p, MATS(), one->reqs, one->nsamples,
                                                  one->out);
                        }
                    }
                    const uint32_t took = (uint32_t)__popc(need) < winEnd - winNext ? (uint32_t)__popc(need) : winEnd - winNext;
                    winNext += took;
                }
                // shade the finished segment and set up the next one (or finish the voxel)
                if (!ray_stepping(s) && j.phase != PH_DONE && j.phase != PH_FETCH) {
                    if constexpr (MANY) {
                        if (j.map != lmi) { le = &many->maps[j.map]; lmi = j.map; }
                        advance<FAR>(j, s, tint, le->m, le->p, le->mats, le->sdir, le->sinv, le->out, c, lit);
                    } else {
                        advance<FAR>(j, s, tint, one->m, one->p, sh->mats, sh->sdir, sh->sinv, one->out, c, lit);
                    }
                }
                if (__ballot_sync(0xFFFFFFFFu, j.phase == PH_FETCH) == 0u) break;
            }
        }
        if (ray_stepping(s)) walk_round<FAR, true>(s, M(), MATS(), P().sunStrength, c, tint, threadIdx.x);
    }
    flush_counters(MANY ? many->stats : one->stats, c, 0, lit);
}

} // namespace dn
