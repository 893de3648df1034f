/*
 * dn_walk.cuh -- the lighting rays' walk through the map: the two-level DDA of voxelShared.comp:300-475
 * (refraction off) as rounds of a chunk-level loop, a chunk entry and a voxel-level loop.
 *
 * A warp calls walk_round for its lanes' rays until enough of them have ended.  In one round a lane at the
 * chunk level takes up to WALK_OUT cells, a lane that reached a loaded chunk enters it, and a lane in a chunk
 * walks it until a voxel stops it or it leaves (at most 22 cells).  Each loop body is one DDA step and one
 * occupancy test and nothing else, so the lanes in it run together however their rays differ, and the rare paths
 * (entering, leaving, voxels of see-through chunks, the map's border) run once per round for all lanes that need them.
 *
 * What makes the bodies short:
 *  - the 2-bit tile map has a border (walk grid below): a ray that leaves the map reads state 1 there, so
 *    no step compares coordinates;
 *  - the smallest of the three side distances is formed once and the stepped axes are those that equal it
 *    (x <= min(y, z) holds exactly when x equals the minimum of all three);
 *  - cells are coded as small integers above 2^23 in floats, so that a step adds one constant per stepped axis on
 *    the FMA pipe, the integer work reads the floats' bits, and a cell's coordinates as floats (a chunk entry
 *    needs them) are one subtraction away.  At the chunk level one float per axis; at the voxel level one for
 *    all, holding the cell's index and the steps left on each axis (voxel_code).  Per chunk-level step 20.7
 *    instructions, 8.3 of them on the half-rate ALU pipe, and 35.8 cycles of a scheduler; with integer
 *    coordinates 23.7, 12.3 and 43.7 (a loop over an empty grid, 6 blocks of 128 threads per SM).  (One float
 *    or integer for the chunk level's cell takes fewer instructions still, but recovering its coordinates sits in
 *    front of the two dependent loads of a chunk entry: 8 % slower on the 64x32x64 map.)
 * Measured against one loop whose body took a step at either level, with the entry, the exit and the segment's
 * end as branches of it (10.6 issue slots per 32 cells of one lane): frames of the 64x32x64 map (1080p, K = 32)
 * 24.2 -> 14.9 ms, of a 16x16x16 map (640x360, K = 16) 0.98 -> 0.70 ms.  Bound by issue and by the latency of the
 * loads in the loops (60 % of the issue slots used, 10 of 32 lanes per step).
 *
 * Every float operation on side distances, positions and directions is the reference's, in its order.
 *
 * TINTED: the launch has a map with a loaded chunk that is not all opaque.  Without one every occupied voxel ends the
 * ray, and the loops are compiled without see-through voxels: the lighting kernels hold both and a launch runs the one
 * its preparation found right (us a pass, before -> after: 16x16x16 map 444 -> 424, 23x11x37 438 -> 422, 64x32x64
 * at 1080p 11322 -> 11063, twelve maps batched 9884 -> 9415; glass unchanged).
 *
 * Maps of more than FAR_SUM chunks along their three axes together (FAR): coordinates are integers, and D16's
 * cap is checked.  In smaller ones a segment cannot reach it: without refraction every step moves at least one
 * axis one cell towards the map's border, so a segment visits at most sx + sy + sz chunk cells and 22 voxel cells
 * in each, below the cap of 256 * (sx + sy + sz) + 4096 (and 2^23).
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
enum : uint32_t { RF_REQUESTED = 1u, RF_IGNORE = 2u, RF_OPAQUE = 4u, RF_TINT = 8u,
                  RF_SKY = 16u };           // the packet kernel's, as the bits from RF_BOUNCES on
constexpr uint32_t RF_BOUNCES = 8;            // the ray's segments before this one

struct Ray {
    f3 pos, dir, delta;      // origin, direction, |1 / direction|
    f3 oside, cell; float olast;      // chunk level: side distances, coded cell, their minimum before the last step
    f3 side; float last, v;  // voxel level: the same; v codes the cell and the steps left (voxel_code)
    uint32_t slot;           // record of the entered chunk
    uint32_t mode, flags;
    uint32_t seg;            // FAR: cells visited by the segment
};

// What see-through voxels did to a lane's ray, in shared memory (one column per lane): most rays meet none, and
// the six registers buy a third more resident warps.  Valid while the ray's RF_TINT is set.
template <int LANES>
struct TintT {
    float add[3][LANES], mul[LANES];            // light gained, and the share that still passes
    uint32_t lastId[LANES], lastAt[LANES];      // the last see-through voxel's identity, and the lane's voxel-cell count there
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

// the first side distance of one axis, (s * (fl - p) + s * 0.5 + 0.5) * delta of init_DDA (voxelShared.comp:305): sg is
// +-1, so both products are exact and one fma rounds as their sum does; fl is the cell's coordinate
__device__ __forceinline__ float side0(float sg, float fl, float p, float delta)
{
    return (__fmaf_rn(sg, fl - p, sg * 0.5f) + 0.5f) * delta;
}

// The code of voxel cell fl of a chunk: index x + 8y + 64z below bit 10; above it the steps left on each axis
// (7 - x upwards, x downwards) in 4-bit fields, whose top bit appears when the axis leaves the chunk.  A step
// along an axis adds voxel_steps' constant.  All exact in a float.
__device__ __forceinline__ f3 voxel_steps(f3 sg)
{
    return mk(sg.x - 1024.0f, __fmaf_rn(sg.y, 8.0f, -16384.0f), __fmaf_rn(sg.z, 64.0f, -262144.0f));
}
// CODE_BASE + x + 8y + 64z + 1024 * (left.x + 16 left.y + 256 left.z) with left = 3.5 + 3.5 s - s * fl, sorted by fl
__device__ __forceinline__ float voxel_code(f3 sg, f3 fl)
{
    const float base = __fmaf_rn(sg.x, 3584.0f, __fmaf_rn(sg.y, 57344.0f, __fmaf_rn(sg.z, 917504.0f, CODE_BASE + 978432.0f)));
    return __fmaf_rn(fl.x, __fmaf_rn(sg.x, -1024.0f, 1.0f),
                     __fmaf_rn(fl.y, __fmaf_rn(sg.y, -16384.0f, 8.0f), __fmaf_rn(fl.z, __fmaf_rn(sg.z, -262144.0f, 64.0f), base)));
}

// Chunk cells: CODE_BASE + 2x, CODE_BASE + y, CODE_BASE + z; FAR: the integers x, y, z in the floats' bits.
constexpr uint32_t FAR_SUM = 1u << 18;
constexpr uint32_t CODE_BITS = 0x4B400000u;   // CODE_BASE's bits

template <bool FAR>
__device__ __forceinline__ f3 cell_code(f3 fl)
{
    if constexpr (FAR) return mk(__int_as_float(f2i(fl.x)), __int_as_float(f2i(fl.y)), __int_as_float(f2i(fl.z)));
    return mk(__fmaf_rn(2.0f, fl.x, CODE_BASE), CODE_BASE + fl.y, CODE_BASE + fl.z);
}
// the coordinates of a coded cell
template <bool FAR>
__device__ __forceinline__ f3 cell_pos(f3 c)
{
    if constexpr (FAR) return mk((float)__float_as_int(c.x), (float)__float_as_int(c.y), (float)__float_as_int(c.z));
    return mk((c.x - CODE_BASE) * 0.5f, c.y - CODE_BASE, c.z - CODE_BASE);
}
template <bool FAR>
__device__ __forceinline__ i3 cell_ints(f3 c)
{
    i3 p{__float_as_int(c.x), __float_as_int(c.y), __float_as_int(c.z)};
    if constexpr (!FAR) {
        p.x = (p.x - (int32_t)CODE_BITS) >> 1; p.y -= (int32_t)CODE_BITS; p.z -= (int32_t)CODE_BITS;
    }
    return p;
}
// the tile of a map cell
template <bool FAR>
__device__ __forceinline__ uint32_t cell_tile(const DevMap& m, f3 c)
{
    if constexpr (FAR) return map_index(m, cell_ints<FAR>(c));
    return (__float_as_uint(c.x) >> 1) + __float_as_uint(c.y) * m.sx + __float_as_uint(c.z) * m.sxy + m.tk;
}
// what a step adds to a coded cell
template <bool FAR>
__device__ __forceinline__ f3 cell_steps(f3 sg)
{
    if constexpr (FAR) return mk(__int_as_float(sg.x < 0.0f ? -1 : 1), __int_as_float(sg.y < 0.0f ? -1 : 1), __int_as_float(sg.z < 0.0f ? -1 : 1));
    return mk(2.0f * sg.x, sg.y, sg.z);
}
template <bool FAR>
__device__ __forceinline__ float cell_add(float c, float d)
{
    if constexpr (FAR) return __int_as_float(__float_as_int(c) + __float_as_int(d));
    return c + d;
}
// the place of a cell's state in the walk grid (wk takes the codes' CODE_BITS back), and the state, border cells included
template <bool FAR>
__device__ __forceinline__ uint32_t cell_bit(const DevMap& m, f3 c)
{
    const uint32_t x = __float_as_uint(c.x), y = __float_as_uint(c.y), z = __float_as_uint(c.z);
    return (FAR ? 2u * x + m.w0 : x + m.wk) + y * m.w1 + z * m.w2;
}
__device__ __forceinline__ uint32_t grid_state(const DevMap& m, uint32_t q)
{
    return __funnelshift_r(__ldg(&m.tbits[q >> 5]), 0u, q) & 3u;
}
template <bool FAR>
__device__ __forceinline__ uint32_t cell_state(const DevMap& m, f3 c) { return grid_state(m, cell_bit<FAR>(m, c)); }

// whether whole coordinates fl are a cell of the map
__device__ __forceinline__ bool inside_map(const DevMap& m, f3 fl)
{
    return min3f(fl.x, fl.y, fl.z) >= 0.0f && fl.x < (float)m.sx && fl.y < (float)m.sy && fl.z < (float)m.sz;
}

// whether the coded voxel of a record is occupied
__device__ __forceinline__ bool voxel_occupied(const ChunkRec* rec, float v)
{
    const uint32_t b = __float_as_uint(v);
    return __funnelshift_r(__ldg(&rec->mask[(b >> 5) & 15u]), 0u, b) & 1u;
}

// Entering a loaded chunk (voxelShared.comp:441-449): the entry point, clamped into the chunk.  It is finite (a
// finite origin and direction), so fminf / fmaxf give GLSL clamp's values.
__device__ __forceinline__ f3 chunk_entry(f3 pos, f3 dir, float olast, f3 cell)
{
    const float tt = olast - EPS;
    const f3 up = add(pos, muls(dir, tt));
    f3 cp = mk((up.x - cell.x) * 8.0f, (up.y - cell.y) * 8.0f, (up.z - cell.z) * 8.0f);
    const float lo = EPS, hi = 8.0f - EPS;
    cp.x = fminf(fmaxf(cp.x, lo), hi); cp.y = fminf(fmaxf(cp.y, lo), hi); cp.z = fminf(fmaxf(cp.z, lo), hi);
    return cp;
}

// a ray at an unloaded chunk's cell requests it, once per segment
__device__ __forceinline__ void ray_request(Ray& r, const DevMap& m, i3 cell)
{
    if (r.flags & RF_REQUESTED) return;
    uint8_t* q = &m.treq[map_index(m, cell)];
    if (*q == 0) *q = 1;
    r.flags |= RF_REQUESTED;
}

// Starts a segment (step_map's set-up, voxelShared.comp:421-433, first voxel ignored).  keep: a bounce of the
// same ray job, which keeps the transparency state (D13).
template <bool FAR, bool TINTED, class Tint>
__device__ __forceinline__ void ray_begin(Ray& r, const DevMap& m, f3 pos, f3 dir, f3 inv, bool keep, Counters& c, Tint& t,
                                          uint32_t col)
{
    r.pos = pos; r.dir = dir; r.delta = vabs(inv);
    r.flags = TINTED && keep ? r.flags & RF_TINT : 0u;
    if (TINTED && r.flags) { t.add[0][col] = 0.0f; t.add[1][col] = 0.0f; t.add[2][col] = 0.0f; t.mul[col] = 1.0f; }
    r.seg = 0;
    r.olast = 0.0f;
    const f3 fl = vfloor(pos);
    if (!finite_dir(inv)) {
        // D16: a zero or NaN direction component traverses nothing
        count_degenerate(m);
        r.mode = RM_MISS;
        return;
    }
    if (!inside_map(m, fl)) {
        r.mode = RM_MISS;
        return;
    }
    r.cell = cell_code<FAR>(fl);
    r.oside.x = side0(copysignf(1.0f, dir.x), fl.x, pos.x, r.delta.x);
    r.oside.y = side0(copysignf(1.0f, dir.y), fl.y, pos.y, r.delta.y);
    r.oside.z = side0(copysignf(1.0f, dir.z), fl.z, pos.z, r.delta.z);
    const uint32_t st = cell_state<FAR>(m, r.cell);
    if (st >= 2u) {
        r.mode = st;
        r.flags |= RF_IGNORE;
        return;
    }
    c.outer++;
    r.seg = 1;
    if (st == 1u) ray_request(r, m, cell_ints<FAR>(r.cell));
    r.mode = RM_OUTER;
}

// one round: see the file comment
template <bool FAR, bool TINTED, class Tint>
__device__ __forceinline__ void walk_round(Ray& r, const DevMap& m, const Material* mats, const float* sunStrength,
                                           Counters& c, Tint& t, uint32_t col)
{
    const f3 sg = mk(copysignf(1.0f, r.dir.x), copysignf(1.0f, r.dir.y), copysignf(1.0f, r.dir.z));
    // FAR: counts k visited cells at a level; false (the segment ends as a miss, D16) when the cap comes before the last
    auto visit = [&](uint32_t& count, uint32_t k) {
        if (FAR && r.seg + k > m.stepCap) { count += m.stepCap - r.seg; r.mode = RM_MISS; return false; }
        if (FAR) r.seg += k;
        count += k;
        return true;
    };
    if (r.mode == RM_OUTER) {
        const f3 d = cell_steps<FAR>(sg);
        uint32_t st = 0, k = 0;
        float mn;
        do {
            mn = min3f(r.oside.x, r.oside.y, r.oside.z);
            const bool px = r.oside.x <= mn, py = r.oside.y <= mn, pz = r.oside.z <= mn;
            if (px) { r.oside.x = r.oside.x + r.delta.x; r.cell.x = cell_add<FAR>(r.cell.x, d.x); }
            if (py) { r.oside.y = r.oside.y + r.delta.y; r.cell.y = cell_add<FAR>(r.cell.y, d.y); }
            if (pz) { r.oside.z = r.oside.z + r.delta.z; r.cell.z = cell_add<FAR>(r.cell.z, d.z); }
            st = cell_state<FAR>(m, r.cell);
            k++;
        } while (st == 0u && k < (uint32_t)DN_WALK_OUT);
        r.olast = mn;
        if (visit(c.outer, st ? k - 1u : k)) {
            if (st == 1u) {
                const i3 cell = cell_ints<FAR>(r.cell);
                if (!in_map(m, cell)) r.mode = RM_MISS;
                else if (visit(c.outer, 1u)) ray_request(r, m, cell);
            } else if (st >= 2u) {
                r.mode = st;
            }
        }
    }
    bool occ = false;
    if ((r.mode == RM_ENTER || r.mode == RM_ENTER_OPAQUE) && visit(c.outer, 1u)) {
        const uint32_t tile = cell_tile<FAR>(m, r.cell);
        r.slot = __ldg(&m.tword[tile]) & SLOT_MASK;
        if (m.ttouch[tile] == 0) m.ttouch[tile] = 1;
        c.entered++;
        const f3 cp = chunk_entry(r.pos, r.dir, r.olast, cell_pos<FAR>(r.cell));
        const f3 fl = vfloor(cp);
        r.side.x = side0(sg.x, fl.x, cp.x, r.delta.x);
        r.side.y = side0(sg.y, fl.y, cp.y, r.delta.y);
        r.side.z = side0(sg.z, fl.z, cp.z, r.delta.z);
        r.last = 0.0f;
        r.v = voxel_code(sg, fl);
        const uint32_t op = r.mode == RM_ENTER_OPAQUE ? RF_OPAQUE : 0u;
        if (!(r.flags & RF_IGNORE)) occ = voxel_occupied(&m.rec[r.slot], r.v);
        r.flags = (r.flags & ~(RF_IGNORE | RF_OPAQUE)) | op;
        r.mode = RM_INNER;
        visit(c.inner, 1u);
    }
    if (r.mode == RM_INNER) {
        const ChunkRec* rec = &m.rec[r.slot];
        bool out = false;
        if (!occ) {
            const f3 d = voxel_steps(sg);
            uint32_t k = 0;
            do {
                const float mn = min3f(r.side.x, r.side.y, r.side.z);
                const bool px = r.side.x <= mn, py = r.side.y <= mn, pz = r.side.z <= mn;
                r.last = mn;
                if (px) { r.side.x = r.side.x + r.delta.x; r.v = r.v + d.x; }
                if (py) { r.side.y = r.side.y + r.delta.y; r.v = r.v + d.y; }
                if (pz) { r.side.z = r.side.z + r.delta.z; r.v = r.v + d.z; }
                out = (__float_as_uint(r.v) & CODE_EXIT) != 0u;
                if (out) break;
                occ = voxel_occupied(rec, r.v);
                k++;
            } while (!occ);
            if (!visit(c.inner, k)) return;
        }
        if (out) {
            r.mode = RM_OUTER;   // the chunk was crossed: the chunk level steps next
        } else if (occ) {
            c.hits++;
            if constexpr (!TINTED) {
                r.mode = RM_HIT;
                return;
            }
            // whether the voxel cell before this one was see-through (no empty voxel cell in between)
            const bool tinted = (r.flags & RF_TINT) != 0u;
            const bool run = tinted && t.lastAt[col] + 1u == c.inner;
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
                    if (!tinted) {
                        t.add[0][col] = 0.0f; t.add[1][col] = 0.0f; t.add[2][col] = 0.0f; t.mul[col] = 1.0f;
                        r.flags |= RF_TINT;
                    }
                    if (!run || t.lastId[col] != thisID) {
                        const f3 alb = mk((float)((vw.y >> 24) & 0xFF) * INV255, (float)((vw.y >> 16) & 0xFF) * INV255,
                                          (float)((vw.y >> 8) & 0xFF) * INV255);
                        const float mul = t.mul[col];
                        const float k = mul * mat.opacity;
                        t.add[0][col] = t.add[0][col] + k * alb.x * sunStrength[0];
                        t.add[1][col] = t.add[1][col] + k * alb.y * sunStrength[1];
                        t.add[2][col] = t.add[2][col] + k * alb.z * sunStrength[2];
                        t.mul[col] = mul * (1.0f - mat.opacity);
                        t.lastId[col] = thisID;
                    }
                    t.lastAt[col] = c.inner;
                }
            }
            if (opaque) {
                r.mode = RM_HIT;
                if (run) t.lastAt[col] = c.inner;   // a bounce goes on from this cell with the same state
            }
        }
    }
}

// the light a ray gained from see-through voxels, and the share that still passes
template <bool TINTED, class Tint>
__device__ __forceinline__ void ray_tint(const Ray& r, const Tint& t, uint32_t col, f3& add, float& mul)
{
    add = mk(0.0f, 0.0f, 0.0f);
    mul = 1.0f;
    if (TINTED && (r.flags & RF_TINT)) { add = mk(t.add[0][col], t.add[1][col], t.add[2][col]); mul = t.mul[col]; }
}

// the pool index of the voxel a ray ended on (RM_HIT)
__device__ __forceinline__ uint32_t ray_hit_index(const Ray& r, const DevMap& m)
{
    const ChunkRec* rc = &m.rec[r.slot];
    return __ldg(&rc->voxBase) + vox_rank(rc, __float_as_uint(r.v) & 511u);
}

// the hit position (voxelShared.comp:362-364) of a ray that ended on a voxel; its entry point is formed again
// from the chunk-level state, which the walk inside the chunk leaves as it was
template <bool FAR>
__device__ __forceinline__ f3 ray_hit_position(const Ray& r)
{
    const f3 cell = cell_pos<FAR>(r.cell);
    const f3 cp = chunk_entry(r.pos, r.dir, r.olast, cell);
    const float t = r.last + EPS;
    return add(cell, muls(add(cp, muls(r.dir, t)), INV_CHUNK));
}

// ---------------------------------------------------------------- primary rays
//
// The draw's walk: one ray per lane from start to end, see-through voxels refracting it (step_map and step_chunk,
// voxelShared.comp:328-475, first voxel not ignored).  The loops are those of the lighting rays; only where the ray is
// inside a see-through voxel does it take one cell at a time, because the first empty cell behind refracts it.
// Neighbouring pixels' rays walk nearly the same cells, so a round has no limit on its chunk cells; but the lanes of a
// warp meet before each entry and after the walk (with returns from within the loops, a counting build found entries run
// by 13 lanes and shading by 8 of 32; they meet at 28 and 31 now).  Which axes the last step took -- the hit's normal --
// is not kept per step, which cost each loop four or five instructions of 26: how far the step moved says it, and is
// looked at once, at the hit.  1080p of the 64x32x64 map 300 -> 283 us, 257x143 12.2 -> 11.3, 639x400 41.7 -> 35.2,
// 960x540 with glass 127 -> 110.
//
// Bound by issue and the ALU pipe.  What a pixel does once costs as much as its steps (about 1200 instructions at a
// hit against 60 cells of 24), so the border normal, which only a ray that has not stepped needs, is formed where
// it is read, and the hit's chunk comes from the walk instead of three divisions of its tile.  Measured with the
// materials read from the launch's arguments (a copy of all 256 in each block's shared memory before) and one
// atomic per counter and block: a 1080p draw of the 64x32x64 map 612 -> 324 us, a 257x143 draw 16.7 -> 11.6 us,
// edited frames at 720p 294 -> 181 us.

__device__ __forceinline__ uint32_t step_axes(bool x, bool y, bool z) { return (x ? 1u : 0u) | (y ? 2u : 0u) | (z ? 4u : 0u); }

// normal_AABB, voxelShared.comp:276-284: the map's face at the point where a ray entered it
static __device__ __noinline__ f3 border_normal(f3 mapMax, f3 pos)
{
    const f3 cc = muls(add(mk(0.0f, 0.0f, 0.0f), mapMax), 0.5f);
    const f3 pp = sub(pos, cc);
    const f3 dd = muls(sub(mapMax, mk(0.0f, 0.0f, 0.0f)), 0.5f);
    const float bias = 1.0f + EPS;
    const f3 q = mk(pp.x / dd.x * bias, pp.y / dd.y * bias, pp.z / dd.z * bias);
    return normalize(mk(truncf(q.x), truncf(q.y), truncf(q.z)));
}

// the axes of a chunk-level step (bits 0-2) by how far it moved in the walk grid: no two sets of axes move alike, for w1 >= 4
// and w2 >= 2 * w1
__device__ __forceinline__ uint32_t grid_axes(const DevMap& m, f3 sg, uint32_t moved)
{
    const uint32_t x = sg.x < 0.0f ? 0u - 2u : 2u, y = sg.y < 0.0f ? 0u - m.w1 : m.w1, z = sg.z < 0.0f ? 0u - m.w2 : m.w2;
    uint32_t axes = 0;
#pragma unroll
    for (uint32_t a = 1; a < 8u; a++)
        if (moved == ((a & 1u) ? x : 0u) + ((a & 2u) ? y : 0u) + ((a & 4u) ? z : 0u)) axes = a;
    return axes;
}
// the axes of a voxel-level step by what it took from the voxel code: 1024, 16384 and 262144 less at most 73
__device__ __forceinline__ uint32_t voxel_axes(uint32_t moved)
{
    const uint32_t t = (moved + 512u) >> 10;
    return (t & 1u) | ((t >> 3) & 2u) | ((t >> 6) & 4u);
}

struct PrimaryHit { i3 cell; uint32_t local, voxel; };   // chunk, x + 8y + 64z in it, pool index

// The whole warp calls it; live: the lane has a ray.  pos, dir, inv: where the ray starts in the map, its direction and
// reciprocal; pos and dir become the hit's, or dir that of leaving the map.  normal: the hit's.
template <bool FAR>
__device__ __forceinline__ bool trace_primary(bool live, const DevMap& m, const Material* mats, f3 sunStrength, f3 org, f3& pos,
                                              f3& dir, f3 inv, float maxDepth, f3& normal, f3& cadd, float& cmul,
                                              PrimaryHit& hit, Counters& c)
{
    cadd = mk(0.0f, 0.0f, 0.0f);
    cmul = 1.0f;
    bool found = false;
    if (live) {
        c.rays++;
        if (!finite_dir(inv)) { count_degenerate(m); live = false; }
    }
    f3 fl = vfloor(pos);
    live = live && inside_map(m, fl);
    f3 delta = vabs(inv);
    f3 sg = mk(copysignf(1.0f, dir.x), copysignf(1.0f, dir.y), copysignf(1.0f, dir.z));
    f3 cell = cell_code<FAR>(fl);
    f3 oside = mk(side0(sg.x, fl.x, pos.x, delta.x), side0(sg.y, fl.y, pos.y, delta.y), side0(sg.z, fl.z, pos.z, delta.z));
    float olast = 0.0f, v = 0.0f;
    uint32_t lastId = 255u;
    float lastRefract = 1.0f;
    bool requested = false;
    // The hit normal is iterate_DDA's output of the last step (voxelShared.comp:316), before any step the map's
    // border; it is formed where it is read.  axes: the last step's (bits 0-2), or 8 no step yet, 16 and 32 a chunk-level
    // and a voxel-level step that moved by `moved`, 0 formed.
    uint32_t axes = 8u, moved = 0;
    auto settle = [&]() {
        if (axes & 8u) normal = border_normal(mk((float)m.sx, (float)m.sy, (float)m.sz), pos);
        if (axes & 16u) axes = grid_axes(m, sg, moved);
        if (axes & 32u) axes = voxel_axes(moved);
        if (axes & 7u) normal = mk(((axes & 1u) ? 1.0f : 0.0f) * -sg.x, ((axes & 2u) ? 1.0f : 0.0f) * -sg.y,
                                   ((axes & 4u) ? 1.0f : 0.0f) * -sg.z);
        axes = 0;
    };
    // the step that follows a refraction, from cell coordinates fl: they may lie outside the chunk or the map
    auto turn_step = [&](f3& side, float& last) {
        last = min3f(side.x, side.y, side.z);
        const bool px = side.x <= last, py = side.y <= last, pz = side.z <= last;
        if (px) { side.x = side.x + delta.x; fl.x = fl.x + sg.x; }
        if (py) { side.y = side.y + delta.y; fl.y = fl.y + sg.y; }
        if (pz) { side.z = side.z + delta.z; fl.z = fl.z + sg.z; }
        axes = step_axes(px, py, pz);
    };
    uint32_t st = 0;
    if (live) st = cell_state<FAR>(m, cell);
    // D16's cap on the cells visited, of both levels
    auto room = [&]() { return c.outer + c.inner < m.stepCap; };
    while (__any_sync(0xFFFFFFFFu, live)) {
        // a live lane is at a chunk cell of the map, its state in st
        live = live && room();
        if (live) c.outer++;
        bool step = true;      // the chunk level steps on from this cell
        __syncwarp();
        if (live && st >= 2u) {
            c.entered++;
            const uint32_t tile = cell_tile<FAR>(m, cell);
            const ChunkRec* rec = &m.rec[__ldg(&m.tword[tile]) & SLOT_MASK];
            if (m.ttouch[tile] == 0) m.ttouch[tile] = 1;
            f3 cp = chunk_entry(pos, dir, olast, cell_pos<FAR>(cell));
            fl = vfloor(cp);
            f3 side = mk(side0(sg.x, fl.x, cp.x, delta.x), side0(sg.y, fl.y, cp.y, delta.y), side0(sg.z, fl.z, cp.z, delta.z));
            float last = 0.0f;
            v = voxel_code(sg, fl);
            bool refracted = false, out = false;
            bool occ = false;
            live = room();
            if (live) {
                c.inner++;
                occ = voxel_occupied(rec, v);
            }
            while (live) {
                // at a visited voxel cell of the chunk
                bool turned = false;
                if (occ) {
                    const uint32_t li = __float_as_uint(v) & 511u;
                    const uint32_t idx = __ldg(&rec->voxBase) + vox_rank(rec, li);
                    const uint2 w = __ldg(&m.vox[idx]);
                    const Material& mat = mats[w.x >> 24];
                    c.hits++;
                    if (mat.opacity == 1.0f) {
                        settle();
                        const float t = last + EPS;
                        cp = add(cp, muls(dir, t));
                        pos = add(cell_pos<FAR>(cell), muls(cp, INV_CHUNK));
                        hit.voxel = idx;
                        found = true;
                        live = false;
                        break;
                    }
                    const uint32_t thisId = (w.y & 0xFFFFFF00u) | (w.x >> 24);
                    hit.voxel = idx;
                    if (lastId != thisId) {
                        f3 cur = add(cp, muls(dir, last));
                        cur = add(cell_pos<FAR>(cell), muls(cur, INV_CHUNK));
                        const f3 to = sub(cur, org);
                        if (maxDepth < 0.0f || dot(to, to) < maxDepth * maxDepth) {
                            const f3 alb = mk((float)((w.y >> 24) & 0xFF) * INV255, (float)((w.y >> 16) & 0xFF) * INV255,
                                              (float)((w.y >> 8) & 0xFF) * INV255);
                            const float k = cmul * mat.opacity;
                            cadd.x = cadd.x + k * alb.x * sunStrength.x;
                            cadd.y = cadd.y + k * alb.y * sunStrength.y;
                            cadd.z = cadd.z + k * alb.z * sunStrength.z;
                            cmul = cmul * (1.0f - mat.opacity);
                        }
                        if (last > 0.0f) {
                            turned = true;
                            cp = add(cp, muls(dir, last + EPS));
                            settle();
                            const f3 vn = voxel_normal(w);
                            const f3 n = (dot(vn, dir) < 0.0f) ? normalize(vn) : normal;
                            dir = refract(dir, n, lastRefract / mat.refractIndex);
                        }
                        lastId = thisId;
                        lastRefract = mat.refractIndex;
                    }
                } else if (lastId != 255u) {
                    // out of the see-through voxel (hit.voxel) into an empty cell
                    turned = true;
                    cp = add(cp, muls(dir, last + EPS));
                    const f3 old = dir;
                    const f3 vn = voxel_normal(__ldg(&m.vox[hit.voxel]));
                    const f3 nn = mk(-vn.x, -vn.y, -vn.z);
                    settle();
                    const f3 n = (dot(nn, dir) < 0.0f) ? normalize(nn) : normal;
                    dir = refract(dir, n, lastRefract);
                    if (dir.x == 0.0f && dir.y == 0.0f && dir.z == 0.0f) dir = old;
                    lastId = 255u;
                    lastRefract = 1.0f;
                }
                if (turned) {
                    // the DDA starts again at the turning point, then steps
                    refracted = true;
                    inv = mk(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
                    if (!finite_dir(inv)) { count_degenerate(m); live = false; break; }
                    delta = vabs(inv);
                    sg = mk(copysignf(1.0f, dir.x), copysignf(1.0f, dir.y), copysignf(1.0f, dir.z));
                    fl = vfloor(cp);
                    side = mk(side0(sg.x, fl.x, cp.x, delta.x), side0(sg.y, fl.y, cp.y, delta.y),
                              side0(sg.z, fl.z, cp.z, delta.z));
                    turn_step(side, last);
                    out = !(fl.x >= 0.0f && fl.y >= 0.0f && fl.z >= 0.0f && fl.x < 8.0f && fl.y < 8.0f && fl.z < 8.0f);
                    if (out) break;
                    v = voxel_code(sg, fl);
                    live = room();
                    if (!live) break;
                    c.inner++;
                    occ = voxel_occupied(rec, v);
                    continue;
                }
                const f3 d = voxel_steps(sg);
                const bool one = lastId != 255u;
                uint32_t k = 0;
                float before;
                do {
                    before = v;
                    last = min3f(side.x, side.y, side.z);
                    const bool px = side.x <= last, py = side.y <= last, pz = side.z <= last;
                    if (px) { side.x = side.x + delta.x; v = v + d.x; }
                    if (py) { side.y = side.y + delta.y; v = v + d.y; }
                    if (pz) { side.z = side.z + delta.z; v = v + d.z; }
                    out = (__float_as_uint(v) & CODE_EXIT) != 0u;
                    if (out) break;
                    occ = voxel_occupied(rec, v);
                    k++;
                } while (!occ && !one);
                axes = 32u;
                moved = __float_as_uint(before) - __float_as_uint(v);
                // D16: a segment that reaches the cap ends in the middle of a run
                c.inner += k;
                if (c.outer + c.inner > m.stepCap) { c.inner = m.stepCap - c.outer; live = false; }
                if (out) break;
            }
            if (live && refracted) {
                // the chunk-level DDA starts again at the last turning point, then steps
                pos = add(cell_pos<FAR>(cell), muls(cp, INV_CHUNK));
                fl = vfloor(pos);
                oside = mk(side0(sg.x, fl.x, pos.x, delta.x), side0(sg.y, fl.y, pos.y, delta.y),
                           side0(sg.z, fl.z, pos.z, delta.z));
                turn_step(oside, olast);
                live = inside_map(m, fl);
                if (live) {
                    cell = cell_code<FAR>(fl);
                    st = cell_state<FAR>(m, cell);
                    step = false;
                }
            }
        } else if (live && st == 1u && !requested) {
            uint8_t* p = &m.treq[map_index(m, cell_ints<FAR>(cell))];
            if (*p == 0) *p = 1;
            requested = true;
        }
        __syncwarp();
        if (live && step) {
            const f3 d = cell_steps<FAR>(sg);
            uint32_t k = 0, before, at = cell_bit<FAR>(m, cell);
            do {
                before = at;
                olast = min3f(oside.x, oside.y, oside.z);
                const bool px = oside.x <= olast, py = oside.y <= olast, pz = oside.z <= olast;
                if (px) { oside.x = oside.x + delta.x; cell.x = cell_add<FAR>(cell.x, d.x); }
                if (py) { oside.y = oside.y + delta.y; cell.y = cell_add<FAR>(cell.y, d.y); }
                if (pz) { oside.z = oside.z + delta.z; cell.z = cell_add<FAR>(cell.z, d.z); }
                at = cell_bit<FAR>(m, cell);
                st = grid_state(m, at);
                k++;
            } while (st == 0u);
            k--;
            axes = 16u;
            moved = at - before;
            c.outer += k;
            if (c.outer + c.inner > m.stepCap) { c.outer = m.stepCap - c.inner; live = false; }
            if (st == 1u && !in_map(m, cell_ints<FAR>(cell))) live = false;
        }
        __syncwarp();
    }
    hit.cell = cell_ints<FAR>(cell);
    hit.local = __float_as_uint(v) & 511u;
    return found;
}

} // namespace dn
