/*
 * dn_walk.cuh -- the lighting rays' walk through the map: the two-level DDA of voxelShared.comp:300-475
 * (refraction off) as rounds of a chunk-level loop, a chunk entry and a voxel-level loop.
 *
 * A warp calls walk_round for its lanes' rays until enough of them have ended.  In one round a lane at the
 * chunk level takes up to WALK_OUT cells, a lane that reached a loaded chunk enters it, and a lane in a chunk
 * walks it until a voxel stops it or it leaves (at most 22 cells).  Each loop body is one DDA step and one occupancy test and nothing else, so the lanes in it run together however
 * their rays differ, and the rare paths (entering, leaving, voxels of see-through chunks, the map's border)
 * run once per round for all lanes that need them.
 *
 * What makes the bodies short:
 *  - the 2-bit tile map has a border (walk grid below): a ray that leaves the map reads state 1 there, so
 *    no step compares coordinates;
 *  - the smallest of the three side distances is formed once and the stepped axes are those that equal it
 *    (x <= min(y, z) holds exactly when x equals the minimum of all three);
 *  - at the voxel level one float per lane holds the cell's index and the steps left on each axis as small
 *    integers above 2^23, so that a step adds one constant per axis on the FMA pipe and both the word address
 *    and the exit test read the float's bits.
 * Measured against one loop whose body took a step at either level, with the entry, the exit and the segment's
 * end as branches of it (10.6 issue slots per 32 cells of one lane): frames of the 64x32x64 map (1080p, K = 32)
 * 24.2 -> 14.9 ms, of a 16x16x16 map (640x360, K = 16) 0.98 -> 0.70 ms.  Bound by issue and by the latency of the
 * loads in the loops (60 % of the issue slots used, 10 of 32 lanes per step).
 *
 * Every float operation on side distances, positions and directions is the reference's, in its order.
 *
 * D16's cell cap cannot be reached here: without refraction every step moves at least one axis one cell
 * towards the map's border, so a segment visits at most sx + sy + sz chunk cells and 22 voxel cells in each,
 * below the cap of 256 * (sx + sy + sz) + 4096.
 */
#pragma once
#include "dn_device.cuh"

namespace dn {

// Chunk cells a lane may take per round: rays that cross open sky would hold the others.  Voxel cells are not
// limited.  Measured on the 64x32x64 map (1080p, K = 32; ms per frame): 8 chunk cells 15.49, 6 15.62, 12 15.58, 4
// 16.51 and 16 16.93; voxel cells limited to 16 15.52, 8 16.31, 4 17.45.
#ifndef DN_WALK_OUT
#define DN_WALK_OUT 8
#endif

enum : uint32_t {
    RM_IDLE = 0,          // no segment
    RM_OUTER = 1,         // at the chunk level, the current cell is done: step next
    RM_ENTER = 2,         // at a loaded chunk's cell (2), or one whose materials are all opaque (3): enter it
    RM_ENTER_OPAQUE = 3,
    RM_INNER = 4,         // in a chunk, the current voxel cell is done: step next
    RM_HIT = 5,           // ended on a voxel
    RM_MISS = 6           // left the map
};
enum : uint32_t { RF_REQUESTED = 1u, RF_IGNORE = 2u, RF_OPAQUE = 4u };

struct Ray {
    f3 pos, dir, delta;      // origin, direction, |1 / direction|
    f3 oside; i3 cell; float olast;   // chunk level: side distances, cell, their minimum before the last step
    f3 side; float last, v;  // voxel level: the same; v codes the cell and the steps left (voxel_code)
    uint32_t slot;           // record of the entered chunk
    uint32_t mode, flags;
    f3 cadd; float cmul;     // light of the see-through voxels crossed
    uint32_t lastId, lastAt; // the last see-through voxel's identity, and the lane's voxel-cell count there
};

__device__ __forceinline__ bool ray_stepping(const Ray& r) { return r.mode - RM_OUTER < 4u; }

// 1.5 * 2^23: a float in [2^23, 2^24) holds a small integer, negative ones included, in its low mantissa bits
constexpr float CODE_BASE = 12582912.0f;
// exit bits of the voxel code: bit 3 of each 4-bit steps-left field
constexpr uint32_t CODE_EXIT = 0x888u << 10;

__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// the first side distance of one axis (init_DDA, voxelShared.comp:305): sg is +-1, fl the cell's coordinate
__device__ __forceinline__ float side0(float sg, float fl, float p, float delta)
{
    return (sg * (fl - p) + sg * 0.5f + 0.5f) * delta;
}

// the state of chunk cell (x, y, z), border cells included (DevMap::tbits)
__device__ __forceinline__ uint32_t walk_state(const DevMap& m, int32_t x, int32_t y, int32_t z)
{
    const uint32_t q = m.w0 + 2u * (uint32_t)x + (uint32_t)y * m.w1 + (uint32_t)z * m.w2;
    return (__ldg(&m.tbits[q >> 5]) >> (q & 31u)) & 3u;
}

// a ray at an unloaded chunk's cell requests it, once per segment
__device__ __forceinline__ void ray_request(Ray& r, const DevMap& m)
{
    if (r.flags & RF_REQUESTED) return;
    uint8_t* q = &m.treq[map_index(m, r.cell)];
    if (*q == 0) *q = 1;
    r.flags |= RF_REQUESTED;
}

// Starts a segment (step_map's set-up, voxelShared.comp:421-433, first voxel ignored).  keep: a bounce of the
// same ray job, which keeps the transparency state (D13).
__device__ __forceinline__ void ray_begin(Ray& r, const DevMap& m, f3 pos, f3 dir, f3 inv, bool keep, Counters& c)
{
    r.pos = pos; r.dir = dir; r.delta = vabs(inv);
    r.cadd = mk(0.0f, 0.0f, 0.0f);
    r.cmul = 1.0f;
    if (!keep) { r.lastId = 255u; r.lastAt = 0xFFFFFFFFu; }
    r.flags = 0;
    r.olast = 0.0f;
    const f3 fl = vfloor(pos);
    if (!finite_dir(inv)) {
        // D16: a zero or NaN direction component traverses nothing
        count_degenerate(m);
        r.mode = RM_MISS;
        return;
    }
    if (!(fl.x >= 0.0f && fl.y >= 0.0f && fl.z >= 0.0f && fl.x < (float)m.sx && fl.y < (float)m.sy && fl.z < (float)m.sz)) {
        r.mode = RM_MISS;
        return;
    }
    r.cell.x = (int32_t)fl.x; r.cell.y = (int32_t)fl.y; r.cell.z = (int32_t)fl.z;
    r.oside.x = side0(copysignf(1.0f, dir.x), fl.x, pos.x, r.delta.x);
    r.oside.y = side0(copysignf(1.0f, dir.y), fl.y, pos.y, r.delta.y);
    r.oside.z = side0(copysignf(1.0f, dir.z), fl.z, pos.z, r.delta.z);
    const uint32_t st = walk_state(m, r.cell.x, r.cell.y, r.cell.z);
    if (st >= 2u) {
        r.mode = st;
        r.flags = RF_IGNORE;
        return;
    }
    c.outer++;
    if (st == 1u) ray_request(r, m);
    r.mode = RM_OUTER;
}

// one round: see the file comment
__device__ __forceinline__ void walk_round(Ray& r, const DevMap& m, const Material* mats, const float* sunStrength,
                                           Counters& c)
{
    const float sgx = copysignf(1.0f, r.dir.x), sgy = copysignf(1.0f, r.dir.y), sgz = copysignf(1.0f, r.dir.z);
    if (r.mode == RM_OUTER) {
        const int32_t ix = r.dir.x < 0.0f ? -1 : 1, iy = r.dir.y < 0.0f ? -1 : 1, iz = r.dir.z < 0.0f ? -1 : 1;
        uint32_t st = 0, k = 0;
        float mn;
        do {
            mn = min3f(r.oside.x, r.oside.y, r.oside.z);
            const bool px = r.oside.x <= mn, py = r.oside.y <= mn, pz = r.oside.z <= mn;
            if (px) { r.oside.x = r.oside.x + r.delta.x; r.cell.x += ix; }
            if (py) { r.oside.y = r.oside.y + r.delta.y; r.cell.y += iy; }
            if (pz) { r.oside.z = r.oside.z + r.delta.z; r.cell.z += iz; }
            st = walk_state(m, r.cell.x, r.cell.y, r.cell.z);
            k++;
        } while (st == 0u && k < (uint32_t)DN_WALK_OUT);
        r.olast = mn;
        c.outer += st ? k - 1u : k;
        if (st == 1u) {
            if ((uint32_t)r.cell.x < m.sx && (uint32_t)r.cell.y < m.sy && (uint32_t)r.cell.z < m.sz) {
                c.outer++;
                ray_request(r, m);
            } else {
                r.mode = RM_MISS;
            }
        } else if (st >= 2u) {
            r.mode = st;
        }
    }
    bool occ = false;
    if (r.mode == RM_ENTER || r.mode == RM_ENTER_OPAQUE) {
        // voxelShared.comp:441-449: the entry point, clamped into the chunk
        const uint32_t t = map_index(m, r.cell);
        r.slot = __ldg(&m.tword[t]) & SLOT_MASK;
        if (m.ttouch[t] == 0) m.ttouch[t] = 1;
        c.outer++;
        c.entered++;
        c.inner++;
        const float tt = r.olast - EPS;
        const f3 up = add(r.pos, muls(r.dir, tt));
        f3 cp = mk((up.x - (float)r.cell.x) * 8.0f, (up.y - (float)r.cell.y) * 8.0f, (up.z - (float)r.cell.z) * 8.0f);
        const float lo = EPS, hi_ = 8.0f - EPS;
        // cp is finite (a finite origin and direction), so fminf / fmaxf give GLSL clamp's values
        cp.x = fminf(fmaxf(cp.x, lo), hi_); cp.y = fminf(fmaxf(cp.y, lo), hi_); cp.z = fminf(fmaxf(cp.z, lo), hi_);
        const f3 fl = vfloor(cp);
        r.side.x = side0(sgx, fl.x, cp.x, r.delta.x);
        r.side.y = side0(sgy, fl.y, cp.y, r.delta.y);
        r.side.z = side0(sgz, fl.z, cp.z, r.delta.z);
        r.last = 0.0f;
        // index x + 8y + 64z below bit 10; above it the steps left on each axis (7 - x upwards, x downwards) in
        // 4-bit fields, whose top bit appears when the axis leaves the chunk.  All exact in a float.
        const f3 left = mk(3.5f - sgx * (fl.x - 3.5f), 3.5f - sgy * (fl.y - 3.5f), 3.5f - sgz * (fl.z - 3.5f));
        r.v = CODE_BASE + (fl.x + 8.0f * fl.y + 64.0f * fl.z) + 1024.0f * (left.x + 16.0f * left.y + 256.0f * left.z);
        const uint32_t op = r.mode == RM_ENTER_OPAQUE ? RF_OPAQUE : 0u;
        if (!(r.flags & RF_IGNORE)) {
            const uint32_t b = __float_as_uint(r.v);
            occ = (__ldg(&m.rec[r.slot].mask[(b >> 5) & 15u]) >> (b & 31u)) & 1u;
        }
        r.flags = (r.flags & RF_REQUESTED) | op;
        r.mode = RM_INNER;
    }
    if (r.mode == RM_INNER) {
        const uint32_t* mask = m.rec[r.slot].mask;
        bool out = false;
        if (!occ) {
            const float cx = sgx - 1024.0f, cy = 8.0f * sgy - 16384.0f, cz = 64.0f * sgz - 262144.0f;
            uint32_t k = 0;
            do {
                const float mn = min3f(r.side.x, r.side.y, r.side.z);
                const bool px = r.side.x <= mn, py = r.side.y <= mn, pz = r.side.z <= mn;
                r.last = mn;
                if (px) { r.side.x = r.side.x + r.delta.x; r.v = r.v + cx; }
                if (py) { r.side.y = r.side.y + r.delta.y; r.v = r.v + cy; }
                if (pz) { r.side.z = r.side.z + r.delta.z; r.v = r.v + cz; }
                const uint32_t b = __float_as_uint(r.v);
                out = (b & CODE_EXIT) != 0u;
                if (out) break;
                occ = (__funnelshift_r(__ldg(&mask[(b >> 5) & 15u]), 0u, b)) & 1u;
                k++;
            } while (!occ);
            c.inner += k;
        }
        if (out) {
            r.mode = RM_OUTER;   // the chunk was crossed: the chunk level steps next
        } else if (occ) {
            c.hits++;
            // whether the voxel cell before this one was see-through (no empty voxel cell in between)
            const bool run = r.lastAt + 1u == c.inner;
            bool opaque = (r.flags & RF_OPAQUE) != 0u;
            if (!opaque) {
                const ChunkRec* rc = &m.rec[r.slot];
                const uint32_t vi = __ldg(&rc->voxBase) + vox_rank(rc, __float_as_uint(r.v) & 511u);
                const uint2 vw = __ldg(&m.vox[vi]);
                const uint32_t material = vw.x >> 24;
                const Material& mat = mats[material];
                opaque = mat.opacity == 1.0f;
                if (!opaque) {
                    const uint32_t thisID = (vw.y & 0xFFFFFF00u) | material;
                    if ((run ? r.lastId : 255u) != thisID) {
                        const f3 alb = mk((float)((vw.y >> 24) & 0xFF) * INV255, (float)((vw.y >> 16) & 0xFF) * INV255,
                                          (float)((vw.y >> 8) & 0xFF) * INV255);
                        const float k = r.cmul * mat.opacity;
                        r.cadd.x = r.cadd.x + k * alb.x * sunStrength[0];
                        r.cadd.y = r.cadd.y + k * alb.y * sunStrength[1];
                        r.cadd.z = r.cadd.z + k * alb.z * sunStrength[2];
                        r.cmul = r.cmul * (1.0f - mat.opacity);
                        r.lastId = thisID;
                    }
                    r.lastAt = c.inner;
                }
            }
            if (opaque) {
                r.mode = RM_HIT;
                if (run) r.lastAt = c.inner;   // a bounce goes on from this cell with the same state
            }
        }
    }
}

// the pool index of the voxel a ray ended on (RM_HIT)
__device__ __forceinline__ uint32_t ray_hit_index(const Ray& r, const DevMap& m)
{
    const ChunkRec* rc = &m.rec[r.slot];
    return __ldg(&rc->voxBase) + vox_rank(rc, __float_as_uint(r.v) & 511u);
}

// the hit position (voxelShared.comp:362-364) of a ray that ended on a voxel; its entry point is formed again
// from the chunk-level state, which the walk inside the chunk leaves as it was
__device__ __forceinline__ f3 ray_hit_position(const Ray& r)
{
    const float tt = r.olast - EPS;
    const f3 up = add(r.pos, muls(r.dir, tt));
    const f3 cell = mk((float)r.cell.x, (float)r.cell.y, (float)r.cell.z);
    f3 cp = mk((up.x - cell.x) * 8.0f, (up.y - cell.y) * 8.0f, (up.z - cell.z) * 8.0f);
    const float lo = EPS, hi_ = 8.0f - EPS;
    cp.x = fminf(fmaxf(cp.x, lo), hi_); cp.y = fminf(fmaxf(cp.y, lo), hi_); cp.z = fminf(fmaxf(cp.z, lo), hi_);
    const float t = r.last + EPS;
    return add(cell, muls(add(cp, muls(r.dir, t)), INV_CHUNK));
}

} // namespace dn
