/*
 * dn_device.cuh -- device-side traversal and shading for sm_103a.
 *
 * The two-level chunk-skipping DDA (voxelShared.comp:300-475), the lighting
 * rays (voxelLighting.comp:65-288) and the primary-ray shading
 * (voxelDraw.comp:24-147), written for CUDA.  Every floating-point expression
 * keeps the reference's operation order and this file is compiled with
 * --fmad=false and IEEE division / square root, so a ray takes exactly the
 * same steps as on the host and hit voxels match bit for bit.
 *
 * Deterministic semantics (shared with the CPU oracle, numbered as there):
 *   D1 lighting reads last frame's committed lighting, new values are
 *      committed by a second kernel; D2 sample count snapshotted per launch;
 *   D3 FP32 lighting; D4 visible / requested / touched are per-tile bytes
 *      written with idempotent stores; D5 per-ray integer-hash RNG (or the
 *      reference's sin-fract with a deterministic sine); D6 bounded
 *      rejection sampling; D8 K fixed direct / specular rays; D9 emissive
 *      strength; D11 no FMA, IEEE div/sqrt, GLSL built-ins by their
 *      specification formulas; D13 transparency state fresh per ray job;
 *      D14 face code and global hit index.
 */
#pragma once
#include <stdint.h>
#include <cuda_runtime.h>

namespace dn {

constexpr float EPS = 0.0001f;            // voxelShared.comp:7
constexpr float INV_CHUNK = 0.125f;       // voxelShared.comp:4
constexpr float HALF_INV_CHUNK = 0.0625f; // voxelShared.comp:5
constexpr float INV255 = 0.00392156862f;  // voxelShared.comp:249-253
constexpr uint32_t SLOT_MASK = 0x3FFFFFFFu;

struct f3 { float x, y, z; };
struct i3 { int32_t x, y, z; };

__device__ __forceinline__ f3 mk(float x, float y, float z) { f3 r; r.x = x; r.y = y; r.z = z; return r; }
__device__ __forceinline__ f3 add(f3 a, f3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ f3 mul(f3 a, f3 b) { return mk(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ f3 muls(f3 a, float s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ f3 adds(f3 a, float s) { return mk(a.x + s, a.y + s, a.z + s); }
__device__ __forceinline__ f3 divs(f3 a, float s) { return mk(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// GLSL min/max: min(x, y) = y < x ? y : x; max(x, y) = x < y ? y : x
__device__ __forceinline__ float gmin(float x, float y) { return (y < x) ? y : x; }
__device__ __forceinline__ float gmax(float x, float y) { return (x < y) ? y : x; }
__device__ __forceinline__ float gsign(float x) { return (x > 0.0f) ? 1.0f : ((x < 0.0f) ? -1.0f : 0.0f); }
__device__ __forceinline__ f3 normalize(f3 v) { float l = sqrtf(dot(v, v)); return divs(v, l); }
__device__ __forceinline__ f3 vabs(f3 v) { return mk(fabsf(v.x), fabsf(v.y), fabsf(v.z)); }
__device__ __forceinline__ f3 vfloor(f3 v) { return mk(floorf(v.x), floorf(v.y), floorf(v.z)); }
__device__ __forceinline__ f3 reflect(f3 I, f3 N) { float t = 2.0f * dot(N, I); return sub(I, muls(N, t)); }
__device__ __forceinline__ f3 refract(f3 I, f3 N, float eta)
{
    float d = dot(N, I);
    float k = 1.0f - eta * eta * (1.0f - d * d);
    if (k < 0.0f) return mk(0.0f, 0.0f, 0.0f);
    float s = eta * d + sqrtf(k);
    return sub(muls(I, eta), muls(N, s));
}
// float -> int32 towards zero with saturation, NaN -> 0: PTX defines cvt.rzi.s32.f32 so for every float (C's cast and
// __float2int_rz are undefined outside the range, which det_sin of a large argument and positions far off reach)
__device__ __forceinline__ int32_t f2i(float x)
{
    int32_t i;
    asm("cvt.rzi.s32.f32 %0, %1;" : "=r"(i) : "f"(x));
    return i;
}

// ---------------------------------------------------------------- RNG (D5)

__device__ __forceinline__ uint32_t hash32(uint32_t x)
{
    // 32-bit integer finaliser ("lowbias32", C. Wellons' hash-prospector)
    x ^= x >> 16; x *= 0x7feb352du;
    x ^= x >> 15; x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}
__device__ __forceinline__ uint32_t rng_key(uint32_t seed, uint32_t mapId, uint32_t voxel)
{
    return hash32(seed ^ hash32(voxel ^ hash32(mapId + 0x632be5abu)));
}
__device__ __forceinline__ float hash_unit(uint32_t key, uint32_t x)
{
    uint32_t h = hash32(key ^ hash32(x));
    return (float)(h >> 8) * (1.0f / 8388608.0f) - 1.0f;
}
__device__ __forceinline__ float hrand(uint32_t key, uint32_t stream, uint32_t idx) { return hash_unit(key, (stream << 28) ^ idx); }
// deterministic sine: Cody-Waite reduction by pi/2 and Taylor polynomials on [-pi/4, pi/4]
__device__ __forceinline__ float det_sin(float x)
{
    const float P1 = 1.5703125f, P2 = 4.837512969970703125e-4f, P3 = 7.549790126404332e-8f;
    float kf = floorf(x * 0.636619746685028076f + 0.5f);
    float r = ((x - kf * P1) - kf * P2) - kf * P3;
    float r2 = r * r;
    int32_t q = f2i(kf) & 3;
    float s = r + r * r2 * (-0.16666667163372040f + r2 * (0.0083333337679505f +
              r2 * (-0.00019841270113829523f + r2 * 2.7557318844628753e-06f)));
    float c = 1.0f + r2 * (-0.5f + r2 * (0.0416666679084301f + r2 * (-0.0013888889225199819f +
              r2 * (2.4801587642286904e-05f + r2 * -2.755731998149713e-07f))));
    return q == 0 ? s : (q == 1 ? c : (q == 2 ? -s : -c));
}
__device__ __forceinline__ float srand1(float s) { float v = det_sin(s) * 43758.5453f; return (v - floorf(v)) * 2.0f - 1.0f; }
__device__ __forceinline__ f3 sphere_try_sin(float s) { return mk(srand1(s), srand1(s * 2.0f), srand1(s * 3.0f)); }
static __device__ __noinline__ f3 sphere_sin(float seed)
{
#pragma unroll 1
    for (int t = 0; t < 64; t++) {
        float s = seed;
        seed = seed + 1.0f;
        f3 p = sphere_try_sin(s);
        if (dot(p, p) >= 1.0f) continue;
        return p;
    }
    return mk(0.0f, 0.0f, 0.0f);
}
// a point of the cube from the hashes of three numbers (hrand's of one stream)
__device__ __forceinline__ f3 sphere_try_hash(uint32_t key, uint32_t x, uint32_t y, uint32_t z)
{
    return mk(hash_unit(key, x), hash_unit(key, y), hash_unit(key, z));
}
__device__ __forceinline__ f3 sphere_hash(uint32_t key, uint32_t stream, uint32_t base)
{
    // not unrolled: half the tries succeed, and 64 copies of the body are tens of KB of code
#pragma unroll 1
    for (uint32_t t = 0; t < 64; t++) {
        uint32_t i = (base << 8) | (3u * t);
        f3 p = mk(hrand(key, stream, i), hrand(key, stream, i + 1u), hrand(key, stream, i + 2u));
        if (dot(p, p) >= 1.0f) continue;
        return p;
    }
    return mk(0.0f, 0.0f, 0.0f);
}

// ------------------------------------------------------------ map layout

// chunk record, 128 B: occupancy mask (bit x + 8*(y + 8*z)), partial counts, voxel count, position, pool base,
// and the set of materials its voxels use (bit m of matSet[m >> 5]; written when the chunk is staged)
struct __align__(128) ChunkRec {
    uint32_t mask[16];
    uint32_t partial[3];
    uint32_t nvox;
    int32_t pos[3];
    uint32_t voxBase;
    uint32_t matSet[8];
};

struct Material {             // 32 B, DNmaterial
    float pad0, pad1;
    uint32_t emissive;
    float opacity, refractIndex, specular;
    uint32_t reflectType, shininess;
};

struct Counters {             // per-thread traversal counters
    uint32_t rays, outer, entered, inner, hits;
};

struct DevMap {
    uint32_t sx, sy, sz;
    uint32_t stepCap;                    // D16: cells a primary ray may visit
    const uint32_t* __restrict__ tword;  // state << 30 | slot
    // walk grid: 2 bits per chunk cell of the map and of a border one cell thick: 0 absent, 1 unloaded or
    // border, 2 loaded, 3 loaded and opaque (during lighting).  Cell (x, y, z) is at bit
    // w0 + 2x + y * w1 + z * w2; a row's border cell also starts the next row, a plane's border row the next plane
    const uint32_t* __restrict__ tbits;
    uint32_t w0, w1, w2;
    uint32_t wk, tk, sxy;                // coded cells (dn_walk.cuh): w0 and tile 0 less what the codes add; sx * sy
    uint8_t* treq;
    uint8_t* ttouch;
    uint8_t* tvis;
    const ChunkRec* __restrict__ rec;
    const uint2* __restrict__ vox;       // normal word, linear albedo word
    const float4* __restrict__ diff;
    const float4* __restrict__ spec;
    unsigned long long* degen;           // D16: segments ended at once for a degenerate direction (counter)
};

struct Voxel { f3 normal; uint32_t material; f3 albedo; f3 spec; f3 diff; };

__device__ __forceinline__ bool in_map(const DevMap& m, i3 p)
{
    return p.x >= 0 && p.y >= 0 && p.z >= 0 && (uint32_t)p.x < m.sx && (uint32_t)p.y < m.sy && (uint32_t)p.z < m.sz;
}
__device__ __forceinline__ uint32_t map_index(const DevMap& m, i3 p)
{
    return (uint32_t)p.x + m.sx * ((uint32_t)p.y + m.sy * (uint32_t)p.z);
}

// rank of voxel li among the set bits (get_voxel_index, voxelShared.comp:150-169): its quarter of the mask and the
// partial counts as two 16-byte loads that do not wait for one another, no loop over words
__device__ __forceinline__ uint32_t vox_rank(const ChunkRec* r, uint32_t li)
{
    const uint32_t w = li >> 5, quarter = w >> 2, in = w & 3u;
    const uint4 m = __ldg((const uint4*)&r->mask[quarter * 4u]);
    const uint4 p = __ldg((const uint4*)r->partial);   // partial[3], nvox
    uint32_t n = quarter == 0u ? 0u : quarter == 1u ? p.x : quarter == 2u ? p.y : p.z;
    const uint32_t own = in == 0u ? m.x : in == 1u ? m.y : in == 2u ? m.z : m.w;
    n += in > 0u ? __popc(m.x) : 0;
    n += in > 1u ? __popc(m.y) : 0;
    n += in > 2u ? __popc(m.z) : 0;
    return n + __popc(own & ((1u << (li & 31)) - 1u));
}

__device__ __forceinline__ f3 voxel_normal(uint2 w)
{
    return mk(((float)((w.x >> 16) & 0xFF) * INV255 - 0.5f) * 2.0f, ((float)((w.x >> 8) & 0xFF) * INV255 - 0.5f) * 2.0f,
              ((float)(w.x & 0xFF) * INV255 - 0.5f) * 2.0f);
}

__device__ __forceinline__ void decompress(const DevMap& m, uint32_t idx, Voxel& v)
{
    // decompress_voxel, voxelShared.comp:236-256, FP32 lighting
    uint2 w = __ldg(&m.vox[idx]);
    v.normal = mk(((float)((w.x >> 16) & 0xFF) * INV255 - 0.5f) * 2.0f,
                  ((float)((w.x >> 8) & 0xFF) * INV255 - 0.5f) * 2.0f,
                  ((float)(w.x & 0xFF) * INV255 - 0.5f) * 2.0f);
    v.material = w.x >> 24;
    v.albedo = mk((float)((w.y >> 24) & 0xFF) * INV255, (float)((w.y >> 16) & 0xFF) * INV255,
                  (float)((w.y >> 8) & 0xFF) * INV255);
    float4 d = __ldg(&m.diff[idx]);
    float4 s = __ldg(&m.spec[idx]);
    v.diff = mk(d.x, d.y, d.z);
    v.spec = mk(s.x, s.y, s.z);
}

// D16: a traversal segment whose direction has a zero or NaN component -- its reciprocal is then infinite
// or NaN -- traverses nothing and ends at once as a miss (counted in DevMap::degen).  The reference's side
// distances become NaN after one step of such a ray (0 * inf), after which no axis may be stepped again and
// its loops (voxelShared.comp:339, 435) never end; reflect() without an added EPSILON
// (voxelLighting.comp:132, 163) produces such directions.  With a finite direction every DDA step advances
// one axis monotonically (at most sx+sy+sz chunk cells and 24 voxel cells per chunk entered); the cell cap
// below ends only repeated refraction inside transparent voxels (the draw).
__device__ __forceinline__ bool finite_dir(f3 inv) { return isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z); }
__device__ __forceinline__ void count_degenerate(const DevMap& m) { if (m.degen) atomicAdd(m.degen, 1ull); }

__device__ __forceinline__ f3 sky_color(f3 bot, f3 top, f3 dir)
{
    // voxelShared.comp:289-295 gradient branch; mix(x, y, a) = x*(1-a) + y*a
    float a = dir.y * 0.5f + 1.0f;
    return mk(bot.x * (1.0f - a) + top.x * a, bot.y * (1.0f - a) + top.y * a, bot.z * (1.0f - a) + top.z * a);
}

// n-th set bit of a chunk mask -> local position; false if n >= popcount.  The partial counts name the quarter of the
// mask, a binary search over popcounts the bit in its word.
__device__ __forceinline__ bool select_voxel(const ChunkRec* r, uint32_t n, i3& out, uint32_t& li)
{
    const uint32_t p0 = __ldg(&r->partial[0]), p1 = __ldg(&r->partial[1]), p2 = __ldg(&r->partial[2]);
    uint32_t w = 0, count = 0;
    if (n >= p2) { w = 12; count = p2; }
    else if (n >= p1) { w = 8; count = p1; }
    else if (n >= p0) { w = 4; count = p0; }
    const uint4 q = __ldg((const uint4*)&r->mask[w]);
    uint32_t bits = q.x, c = (uint32_t)__popc(q.x);
    if (n - count >= c) { count += c; w++; bits = q.y; c = (uint32_t)__popc(q.y); }
    if (n - count >= c) { count += c; w++; bits = q.z; c = (uint32_t)__popc(q.z); }
    if (n - count >= c) { count += c; w++; bits = q.w; c = (uint32_t)__popc(q.w); }
    uint32_t k = n - count, b = 0;
    if (k >= c) return false;
#pragma unroll
    for (uint32_t s = 16; s > 0; s >>= 1) {
        const uint32_t low = (uint32_t)__popc((bits >> b) & ((1u << s) - 1u));
        if (k >= low) { k -= low; b += s; }
    }
    li = w * 32u + b;
    out.x = (int32_t)(li & 7u); out.y = (int32_t)((li >> 3) & 7u); out.z = (int32_t)(li >> 6);
    return true;
}

} // namespace dn
