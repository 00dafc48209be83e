// svo_trace.cuh -- hierarchical DDA through the one-bit SVO (device side).
//
// The reference traverses its pointer octree with a 5-deep stack and a 32^3
// leaf DDA (svo_functions.inc:1-329, CPU form tg_sparse_voxel_octree.c:558-740).
// Here the same voxel set is traversed over the occupancy levels of the new
// storage: cells of 2^g voxels for g = L-1, ..., 9, 7, 5 (every other level
// of the block pyramid), g = 3 and 2 (sub-block masks of each 32^3 block),
// then single voxels.  An occupied cell is entered (descend), an empty one is
// left through its nearest face (one step), and leaving the parent cell
// ascends.  The operations are exactly rounded, in the order of the CPU
// oracle (oracle/oracle_gi.c: oracle_trace), so hits, distances and face
// normals are bit-identical.
#pragma once

#include "tgx_internal.cuh"

struct SvoDev
{
    float mn[3];
    uint32_t L, B, NL;
    const uint32_t* table;
    const uint32_t* pool;
    const uint32_t* sub;     // per slot 32 words: 4^3-cell mask (0-15), 8^3-cell mask (16-17)
    const uint32_t* occ;
    const uint16_t* mat;
    uint32_t occ_off[16];    // word offset of each pyramid level (level 0 = 32^3 blocks), zero padded
};

// log2 of the cell size of traversal level li: 0, 2, 3, 5, 7, 9, ... capped at L-1
__host__ __device__ __forceinline__ uint32_t svo_level_log2(uint32_t L, uint32_t li)
{
    return li == 0 ? 0u : li <= 2 ? li + 1u : min(2u * li - 1u, L - 1u);
}

__host__ __device__ __forceinline__ uint32_t svo_n_levels(uint32_t L)
{
    uint32_t n = 4;
    while (svo_level_log2(L, n - 1) < L - 1) n++;
    return n;
}

// byte offset, after the pyramid words, of the device copy of the level offsets (16-byte aligned)
inline uint64_t svo_occ_off_bytes(uint64_t occ_words) { return (occ_words * 4 + 15) & ~(uint64_t)15; }

inline SvoDev svo_dev(const tgx_svo* s)
{
    SvoDev d;
    d.mn[0] = s->mn[0]; d.mn[1] = s->mn[1]; d.mn[2] = s->mn[2];
    d.L = s->L; d.B = s->B; d.NL = svo_n_levels(s->L);
    d.table = s->d_table; d.pool = s->d_pool; d.sub = s->d_sub; d.occ = s->d_occ; d.mat = s->d_mat;
    for (int i = 0; i < 16; i++) d.occ_off[i] = i < 10 ? (uint32_t)s->occ_off[i] : 0u;
    return d;
}

__device__ __forceinline__ uint32_t svo_material(const SvoDev& s, int32_t cx, int32_t cy, int32_t cz)
{
    if (!s.mat) return 0;
    const uint32_t bx = (uint32_t)cx >> 5, by = (uint32_t)cy >> 5, bz = (uint32_t)cz >> 5;
    const uint32_t tv = __ldg(&s.table[((uint64_t)bz * s.B + by) * s.B + bx]);
    if (!tv) return 0;
    const uint32_t v = ((uint32_t)cz & 31u) * 1024u + ((uint32_t)cy & 31u) * 32u + ((uint32_t)cx & 31u);
    return s.mat[(uint64_t)(tv - 1) * 32768u + v];
}

// The cell of coordinate p at cells of size 1/inv_size, a point on a cell
// border going to the lower cell when the ray steps down, clamped to
// [lo, hi].  For |x| < 2^30 (always, for rays inside the cube) the floor is an
// exact integer and the clamp is done on integers; NaN and larger values take
// the float form, whose results the integer form equals wherever both apply.
__device__ __forceinline__ int32_t svo_cell_at(float p, float inv_size, int32_t step, int32_t lo, int32_t hi)
{
    const float x = xmul(p, inv_size);
    float f = floorf(x);
    if (fabsf(x) < 1073741824.0f) {
        const int32_t c = (int32_t)f - ((step < 0 && x == f) ? 1 : 0);
        return min(max(c, lo), hi);
    }
    if (step < 0 && x == f) f = xsub(f, 1.0f);
    int32_t c = (int32_t)f;
    if (f < (float)lo) c = lo;
    if (f > (float)hi) c = hi;
    return c;
}

// Occupancy bit of cell c (grid coordinates at log2 size g); tv is the slot +
// 1 of the 32^3 block holding c, needed below the block level (g < 5).
__device__ __forceinline__ bool svo_occupied(const SvoDev& s, const uint32_t* occ_off, uint32_t g, const int32_t c[3],
                                             uint32_t tv)
{
    const bool sub = g < 5u;
    const uint32_t m = sub ? (32u >> g) : (s.B >> (g - 5u));
    const uint32_t mk = sub ? m - 1u : 0xffffffffu;
    const uint32_t v = (((uint32_t)c[2] & mk) * m + ((uint32_t)c[1] & mk)) * m + ((uint32_t)c[0] & mk);
    const uint32_t* base = !sub ? s.occ + occ_off[(g - 5u) & 15u]
                         : g == 0 ? s.pool + (uint64_t)(tv - 1u) * 1024u
                                  : s.sub + (uint64_t)(tv - 1u) * 32u + (g == 3 ? 16u : 0u);
    return (__ldg(&base[v >> 5]) >> (v & 31u)) & 1u;
}

// The general traversal of one ray, start to end, in the oracle's own form:
// top-down from the root, one level or one cell per iteration, float
// coordinates.  It takes every ray; the persistent kernels send it the few
// whose numbers the fast form below cannot hold (svo_ray_is_plain).
// Returns 1 on hit, 0 on a miss, -1 when max_steps ran out.
static __device__ __noinline__ int svo_trace_general(const SvoDev& s, const float* o, const float* d, uint32_t max_steps,
                                                     float* out_t, int32_t* c, int32_t* out_axis, uint32_t* out_steps)
{
    const float E = (float)(1u << s.L);
    float og[3], inv[3];
    int32_t st[3];
    for (int a = 0; a < 3; a++) {
        og[a] = xsub(o[a], s.mn[a]);
        st[a] = d[a] > 0.0f ? 1 : d[a] < 0.0f ? -1 : 0;
        inv[a] = st[a] ? xdiv(1.0f, d[a]) : 0.0f;
    }
    *out_steps = 0;
    *out_axis = -1;
    *out_t = 0.0f;
    c[0] = c[1] = c[2] = 0;
    if (!st[0] && !st[1] && !st[2]) return 0;
    float t0 = F32_MIN_TG, t1 = F32_MAX_TG;
    int32_t entry_axis = -1;
    for (int a = 0; a < 3; a++) {
        if (!st[a]) {
            if (og[a] < 0.0f || og[a] >= E) return 0;
            continue;
        }
        const float ta = xmul(xsub(0.0f, og[a]), inv[a]);
        const float tb = xmul(xsub(E, og[a]), inv[a]);
        const float tn = ta < tb ? ta : tb;
        const float tf = ta < tb ? tb : ta;
        if (tn > t0) { t0 = tn; entry_axis = a; }
        if (tf < t1) t1 = tf;
    }
    float t = t0 > 0.0f ? t0 : 0.0f;
    if (!(t < t1)) return 0;
    *out_axis = t0 > 0.0f ? entry_axis : -1;
    uint32_t li = s.NL - 1u, g = s.L - 1u, tv = 0;
    for (int a = 0; a < 3; a++)
        c[a] = svo_cell_at(xadd(og[a], xmul(t, d[a])), __int_as_float((int)((127u - g) << 23)), st[a], 0, (1 << (s.L - g)) - 1);
    for (uint32_t steps = 0; steps < max_steps;) {
        *out_steps = ++steps;
        *out_t = t;
        if (svo_occupied(s, s.occ_off, g, c, tv)) {
            if (li == 0) return 1;
            if (g == 5u) tv = __ldg(&s.table[((uint64_t)c[2] * s.B + (uint64_t)c[1]) * s.B + (uint64_t)c[0]]);
            const uint32_t gc = svo_level_log2(s.L, --li), sh = g - gc;
            g = gc;
            for (int a = 0; a < 3; a++) {
                const int32_t lo = c[a] << sh, hi = lo + (1 << sh) - 1;
                c[a] = svo_cell_at(xadd(og[a], xmul(t, d[a])), __int_as_float((int)((127u - g) << 23)), st[a], lo, hi);
            }
            continue;
        }
        const float size = (float)(1u << g);
        float tn[3];
        for (int a = 0; a < 3; a++)
            tn[a] = st[a] != 0 ? xmul(xsub(xmul((float)(c[a] + ((st[a] + 1) >> 1)), size), og[a]), inv[a]) : F32_MAX_TG;
        int am = 0;
        if (tn[1] < tn[am]) am = 1;
        if (tn[2] < tn[am]) am = 2;
        if (tn[am] > t) t = tn[am];
        *out_axis = am;
        int32_t prev = c[am];
        c[am] += st[am];
        int32_t cur = c[am];
        if (cur < 0 || cur >= (1 << (s.L - g))) return 0;
        while (li < s.NL - 1u) {   // ascend to the level whose parent the step stayed in
            const uint32_t gp = svo_level_log2(s.L, li + 1u), sh = gp - g;
            if ((prev >> sh) == (cur >> sh)) break;
            prev >>= sh; cur >>= sh;
            c[0] >>= sh; c[1] >>= sh; c[2] >>= sh;
            li++;
            g = gp;
        }
    }
    return -1;
}

// ---------------------------------------------------------------------------
// The fast form: the same cells, distances and step counts with about a third
// of the instructions per step.
//
// Mirrored axes.  On an axis the ray goes down, coordinates are counted from
// the far side: cell v' = E - 1 - v (one XOR with E - 1), origin -og, direction
// |d|.  Rounding to nearest is symmetric, so the mirrored products and sums are
// the negated or equal originals, bit for bit, and every axis steps up: the
// face a ray leaves through is always the next cell's first voxel, and the cube
// is left when a coordinate reaches E.
//
// One coordinate for all levels.  v' is a voxel coordinate inside the current
// cell of any size; the cell is v' without its low g bits.  Point location at
// voxel resolution, clamped to the current cell, gives the children of every
// finer level by masking, because floor(p / 2^g) = floor(floor(p) / 2^g) and
// clamping commutes with the shift.  A descent is therefore just "one level
// finer"; only a step locates a point.
//
// Integers in floats.  v' is kept as the bit pattern of 1.5 * 2^23 + v'
// (kMagic | v'): as a float its sums with whole numbers below 2^22 are exact,
// and p + 1.5 * 2^23 rounded down is the floor of p in place (mirrored, the
// lower-cell rule for a point on a border included), with no conversion
// instruction.  This holds for |p| < 2^22, hence svo_ray_is_plain.
//
// Step ahead of the word.  An iteration computes the step that an empty cell
// takes while the cell's occupancy word is on its way, and selects by the bit at
// the end: the chain of one ray, which decides the time of a small batch, is
// shorter by the load, and the lanes that descend no longer diverge from the
// ones that step (branching on the bit first: GI frame 1397 us, million rays
// 328, two frames of an update 932; selecting: 1358, 312, 918).
//
// Bound by instruction issue (about 95 instructions an iteration for a warp).
// Both launches of a 1-bounce 4-spp 1080p frame over the 512-object scene:
// 2.25 ms with both moves computed for every cell in float coordinates, 1.63 ms
// in this form; a million random rays through its 4096^3 SVO 0.84 -> 0.32 ms
// (together with the queue below instead of one thread per ray).
// ---------------------------------------------------------------------------

constexpr uint32_t kMagic = 0x4B400000u;           // 1.5 * 2^23
constexpr float kMagicF = 12582912.0f;
constexpr int kTraceRunning = -2;

struct RayState
{
    float og[3], d[3], inv[3];   // mirrored origin, |d|, |1 / d| (2^127 where d = 0: that axis is never the nearest)
    float off[3];                // kMagicF, plus E on mirrored axes
    uint32_t flip[3];            // all ones on mirrored axes, else 0
    uint32_t v[3];               // kMagic | mirrored voxel coordinate
    float t;
    int32_t last_axis;
    uint32_t lo, steps;          // level * sizeof(LevelDesc), steps used
    uint32_t tv;                 // slot + 1 of the 32^3 block the levels below 32 are inside
};

// A ray parked between its set-up and its DDA: 64 bytes, four 16-byte shared
// loads.  The mirrored axes are the sign bits of v; the level, the last axis
// and the few steps used so far share a word.
struct alignas(16) ParkedRay
{
    float og[3], d[3], inv[3];
    uint32_t v[3];
    float t;
    uint32_t tv, item;
    uint32_t misc;               // lo | (last_axis + 1) << 16 | steps << 24
};
static_assert(sizeof(ParkedRay) == 64, "four 16-byte shared loads");

__device__ __forceinline__ void svo_park(ParkedRay* p, const RayState& r, uint32_t item)
{
    uint4* q = reinterpret_cast<uint4*>(p);
    const uint32_t m = 0x80000000u;
    q[0] = make_uint4(__float_as_uint(r.og[0]), __float_as_uint(r.og[1]), __float_as_uint(r.og[2]), __float_as_uint(r.d[0]));
    q[1] = make_uint4(__float_as_uint(r.d[1]), __float_as_uint(r.d[2]), __float_as_uint(r.inv[0]), __float_as_uint(r.inv[1]));
    q[2] = make_uint4(__float_as_uint(r.inv[2]), r.v[0] | (r.flip[0] & m), r.v[1] | (r.flip[1] & m), r.v[2] | (r.flip[2] & m));
    q[3] = make_uint4(__float_as_uint(r.t), r.tv, item, r.lo | (uint32_t)(r.last_axis + 1) << 16 | r.steps << 24);
}

__device__ __forceinline__ void svo_unpark(const ParkedRay* p, float E, RayState& r, uint32_t& item)
{
    const uint4* q = reinterpret_cast<const uint4*>(p);
    const uint4 a = q[0], b = q[1], c = q[2], e = q[3];
    r.og[0] = __uint_as_float(a.x); r.og[1] = __uint_as_float(a.y); r.og[2] = __uint_as_float(a.z);
    r.d[0] = __uint_as_float(a.w); r.d[1] = __uint_as_float(b.x); r.d[2] = __uint_as_float(b.y);
    r.inv[0] = __uint_as_float(b.z); r.inv[1] = __uint_as_float(b.w); r.inv[2] = __uint_as_float(c.x);
    const uint32_t v[3] = {c.y, c.z, c.w};
#pragma unroll
    for (int i = 0; i < 3; i++) {
        r.flip[i] = (uint32_t)((int32_t)v[i] >> 31);
        r.off[i] = r.flip[i] ? kMagicF + E : kMagicF;
        r.v[i] = v[i] & 0x7fffffffu;
    }
    r.t = __uint_as_float(e.x);
    r.tv = e.y;
    item = e.z;
    r.lo = e.w & 0xffffu;
    r.last_axis = (int32_t)((e.w >> 16) & 0xffu) - 1;
    r.steps = e.w >> 24;
}

// One traversal level: where its occupancy bits are and how a voxel
// coordinate indexes them.  Built per launch in shared memory; a step reads it
// with two 16-byte loads.
struct alignas(16) LevelDesc
{
    uint64_t base;     // address of the occupancy words; for g < 5 of those of slot + 1 = 0
    uint32_t stride;   // bytes per block slot (g < 5), else 0
    uint32_t m;        // cells per axis of the indexed array
    uint32_t mk;       // the bits of a voxel coordinate that index it
    uint32_t low;      // 2^g - 1
    uint32_t g;        // log2 of the cell size
    uint32_t pad;
};
static_assert(sizeof(LevelDesc) == 32, "two 16-byte shared loads");
constexpr uint32_t kAscend = 32;   // ascend[p]: p = trailing zeros of the coordinate stepped to (kMagic's end at 22)

// The level a step ascends to and that level's low mask.  p is the highest
// coordinate bit the step changed (the carry of the increment, i.e. the
// trailing zeros of the new coordinate): the lowest level whose parent's cells
// are larger than 2^p, or the root level.  The same level as the
// one-level-at-a-time climb (tests/test_trace_ascend.py).
__host__ __device__ __forceinline__ uint32_t svo_ascend_level(uint32_t L, uint32_t NL, uint32_t p)
{
    uint32_t li = 0;
    while (li < NL - 1u && svo_level_log2(L, li + 1u) < p + 1u) li++;
    return li;
}

struct TraceTables
{
    LevelDesc lv[16];
    uint2 ascend[kAscend];   // level * sizeof(LevelDesc), low mask
};

// Fills the tables for SVO s, the first warp of the block; the caller synchronises.
__device__ __forceinline__ void svo_level_tables(const SvoDev& s, TraceTables& tb)
{
    const uint32_t i = threadIdx.x;
    if (i >= kAscend) return;
    LevelDesc d = {};
    if (i < s.NL) {
        const uint32_t g = svo_level_log2(s.L, i);
        d.g = g;
        d.low = (1u << g) - 1u;
        if (g >= 5u) {
            uint32_t off = 0;
#pragma unroll
            for (uint32_t k = 0; k < 16u; k++) off = k == g - 5u ? s.occ_off[k] : off;   // no indexed copy of the parameter
            d.base = (uint64_t)(s.occ + off);
            d.m = s.B >> (g - 5u);
            d.mk = ((1u << s.L) - 1u) & ~d.low;
        } else {
            d.stride = g == 0u ? 4096u : 128u;
            d.base = (uint64_t)(g == 0u ? s.pool : s.sub + (g == 3u ? 16u : 0u)) - d.stride;
            d.m = 32u >> g;
            d.mk = 31u & ~d.low;
        }
    }
    if (i < 16u) tb.lv[i] = d;
    const uint32_t up = svo_ascend_level(s.L, s.NL, i);
    tb.ascend[i] = make_uint2(up * (uint32_t)sizeof(LevelDesc), (1u << svo_level_log2(s.L, up)) - 1u);
}

__device__ __forceinline__ LevelDesc svo_level(const TraceTables& tb, uint32_t lo)   // lo: level * sizeof(LevelDesc)
{
    const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(tb.lv) + lo);
    const uint4 a = q[0], b = q[1];
    LevelDesc d;
    d.base = (uint64_t)a.y << 32 | a.x;
    d.stride = a.z; d.m = a.w;
    d.mk = b.x; d.low = b.y; d.g = b.z; d.pad = 0;
    return d;
}

// The bit index of the cell of voxel coordinate (x, y, z) in level ld's words
// (bits of the coordinates outside the level's mask are ignored), and its word.
__device__ __forceinline__ uint32_t svo_level_index(const LevelDesc& ld, uint32_t x, uint32_t y, uint32_t z)
{
    return (((z & ld.mk) * ld.m + (y & ld.mk)) * ld.m + (x & ld.mk)) >> ld.g;
}
__device__ __forceinline__ uint32_t svo_level_word(const LevelDesc& ld, uint32_t i, uint32_t tv)
{
    return __ldg(reinterpret_cast<const uint32_t*>(ld.base + (uint64_t)tv * ld.stride) + (i >> 5));
}
__device__ __forceinline__ bool svo_level_bit(const LevelDesc& ld, uint32_t x, uint32_t y, uint32_t z, uint32_t tv)
{
    const uint32_t i = svo_level_index(ld, x, y, z);
    return __funnelshift_r(svo_level_word(ld, i, tv), 0u, i) & 1u;   // the shift takes i mod 32
}

// Whether the fast form holds the ray: finite numbers, an origin within 2^20
// voxels of the cube's corner (so that every point of the ray inside the cube
// stays far inside +-2^22), and direction components that are zero or at least
// 2^-60 (their reciprocals stay below the 2^127 that stands for a zero's).
__device__ __forceinline__ bool svo_ray_is_plain(const float og[3], const float d[3])
{
    bool ok = true;
#pragma unroll
    for (int a = 0; a < 3; a++)
        ok = ok && fabsf(og[a]) <= 1048576.0f && fabsf(d[a]) <= 3.0e38f && (d[a] == 0.0f || fabsf(d[a]) >= 8.6736174e-19f);
    return ok;
}

// Sets up a ray.  Returns kTraceRunning when the DDA has to run, else the
// result (0: the ray misses the SVO cube or has no direction; 1: the entry
// voxel is set; and whatever the general form gives a ray that is not plain).
// r.v holds real, not mirrored, coordinates when it returns 1.
//
// The DDA starts where the top-down descent from the root would first find an
// empty cell, found bottom-up instead: the entry point's voxel, then its
// ancestors (the cell of every level that holds the point is the voxel's
// coordinates shifted right, with the same boundary rule) until an occupied
// one.  The descent's iterations are counted into r.steps as if they had
// run, so every result and the step budget stay those of the top-down walk.
__device__ __forceinline__ int svo_trace_begin(const SvoDev& s, const TraceTables& tb, const float o[3], const float d[3],
                                               uint32_t max_steps, RayState& r)
{
    const float E = (float)(1u << s.L);
    float og[3];
#pragma unroll
    for (int a = 0; a < 3; a++) og[a] = xsub(o[a], s.mn[a]);
    r.steps = 0;
    r.tv = 0;
    r.t = 0.0f;
    r.last_axis = -1;
    r.v[0] = r.v[1] = r.v[2] = 0;
    if (!svo_ray_is_plain(og, d)) {
        const float oo[3] = {o[0], o[1], o[2]}, dd[3] = {d[0], d[1], d[2]};
        int32_t c[3];
        const int res = svo_trace_general(s, oo, dd, max_steps, &r.t, c, &r.last_axis, &r.steps);
        r.v[0] = (uint32_t)c[0]; r.v[1] = (uint32_t)c[1]; r.v[2] = (uint32_t)c[2];
        return res;
    }
    if (d[0] == 0.0f && d[1] == 0.0f && d[2] == 0.0f) return 0;
    float t0 = F32_MIN_TG, t1 = F32_MAX_TG;
    int32_t entry_axis = -1;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const bool neg = d[a] < 0.0f;
        const float inv = d[a] != 0.0f ? xdiv(1.0f, d[a]) : 0.0f;
        r.flip[a] = neg ? 0xffffffffu : 0u;
        r.off[a] = neg ? kMagicF + E : kMagicF;
        r.og[a] = neg ? -og[a] : og[a];
        r.d[a] = fabsf(d[a]);
        r.inv[a] = d[a] != 0.0f ? fabsf(inv) : 1.7014118e38f;
        if (d[a] == 0.0f) {
            if (og[a] < 0.0f || og[a] >= E) return 0;
            continue;
        }
        const float ta = xmul(xsub(0.0f, og[a]), inv);
        const float tb = xmul(xsub(E, og[a]), inv);
        const float tn = ta < tb ? ta : tb;
        const float tf = ta < tb ? tb : ta;
        if (tn > t0) { t0 = tn; entry_axis = a; }
        if (tf < t1) t1 = tf;
    }
    r.t = t0 > 0.0f ? t0 : 0.0f;
    if (!(r.t < t1)) return 0;
    r.last_axis = t0 > 0.0f ? entry_axis : -1;
    r.lo = (s.NL - 1u) * (uint32_t)sizeof(LevelDesc);
    uint32_t cv[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const float p = xadd(r.og[a], xmul(r.t, r.d[a]));
        const int32_t at = __float_as_int(__fadd_rd(p, r.off[a]));
        r.v[a] = (uint32_t)min(max(at, (int32_t)kMagic), (int32_t)(kMagic + (1u << s.L) - 1u));
        cv[a] = (r.v[a] ^ r.flip[a]) & ((1u << s.L) - 1u);
    }
    if (max_steps < s.NL) return kTraceRunning;   // the budget could run out inside the descent: run it
    const uint32_t tv = __ldg(&s.table[((uint64_t)(cv[2] >> 5) * s.B + (uint64_t)(cv[1] >> 5)) * s.B + (uint64_t)(cv[0] >> 5)]);
    // coarsest empty level holding the point (-1: the voxel itself is set): the
    // levels below the lowest occupied one.  All levels' bits are loaded at once
    // (at most 8 levels for L <= 14) rather than one level per dependent step.
    uint32_t occ_mask = 0;
#pragma unroll
    for (uint32_t li = 0; li < 8u; li++) {
        if (li >= s.NL) break;   // the same in every lane
        const LevelDesc ld = svo_level(tb, li * (uint32_t)sizeof(LevelDesc));
        if (ld.g < 5u && tv == 0u) continue;   // below an unallocated block: empty
        if (svo_level_bit(ld, cv[0], cv[1], cv[2], tv)) occ_mask |= 1u << li;
    }
    const int32_t e = occ_mask ? __ffs((int)occ_mask) - 2 : (int32_t)s.NL - 1;
    if (e < 0) {   // the descent reaches the voxel: NL iterations, a hit
        r.steps = s.NL;
        r.v[0] = cv[0]; r.v[1] = cv[1]; r.v[2] = cv[2];
        return 1;
    }
    r.lo = (uint32_t)e * (uint32_t)sizeof(LevelDesc);
    r.tv = tv;
    r.steps = s.NL - 1u - (uint32_t)e;
    return kTraceRunning;
}

// v = min(a, b) and v = max(v, a) unless `keep`: one predicated instruction each,
// where a selection would be a second one (GI frame 1355 -> 1334 us, with the four
// places of the traversal's loop).
__device__ __forceinline__ void min_unless(bool keep, uint32_t& v, uint32_t a, uint32_t b)
{
    asm("{\n .reg .pred p;\n setp.eq.u32 p, %1, 0;\n @p min.s32 %0, %2, %3;\n}" : "+r"(v) : "r"((uint32_t)keep), "r"(a), "r"(b));
}
__device__ __forceinline__ void max_unless(bool keep, float& v, float a)
{
    asm("{\n .reg .pred p;\n setp.eq.u32 p, %1, 0;\n @p max.f32 %0, %0, %2;\n}" : "+f"(v) : "r"((uint32_t)keep), "f"(a));
}

// Runs at most n iterations of the DDA of a ray (each is one step of the
// max_steps budget: one level down into an occupied cell, or one cell on).
// Returns kTraceRunning, 1 on hit (r.t, r.v real coordinates, r.last_axis), 0
// on miss, -1 when max_steps ran out.  The loop has one exit and its body only
// nested ifs, so the lanes of a warp meet again after every iteration; with
// early returns they drifted apart (20 of 32 lanes per instruction).
__device__ __forceinline__ int svo_trace_run(const SvoDev& s, const TraceTables& tb, RayState& r, uint32_t max_steps,
                                             uint32_t n)
{
    const uint32_t extent = 1u << s.L;
    uint32_t last = min(n, max_steps - r.steps);   // the ray's iterations of this round (r.steps <= max_steps)
    int res = kTraceRunning;
    for (uint32_t k = 0; k < n; k++) {
        if (k < last) {
            const LevelDesc ld = svo_level(tb, r.lo);
            const uint32_t x = r.v[0] ^ r.flip[0], y = r.v[1] ^ r.flip[1], z = r.v[2] ^ r.flip[2];
            const uint32_t i = svo_level_index(ld, x, y, z);
            const uint32_t word = svo_level_word(ld, i, r.tv);
            // While the word is on its way: the step that an empty cell takes.  The distance to
            // the next cell on every axis: its first voxel w, less the origin, times 1 / d
            uint32_t w[3], nv[3], hi[3];
            float tn[3];
#pragma unroll
            for (int a = 0; a < 3; a++) {
                w[a] = (r.v[a] | ld.low) + 1u;
                tn[a] = xmul(xsub(xsub(__uint_as_float(w[a]), r.off[a]), r.og[a]), r.inv[a]);
            }
            const bool a1 = tn[1] < tn[0];
            const float t01 = fminf(tn[0], tn[1]);
            const bool a2 = tn[2] < t01;
            const uint32_t ws = a2 ? w[2] : a1 ? w[1] : w[0];
            // a step out of the cube also runs to the end (its level and point are not used)
            const uint2 up = tb.ascend[__popc(~ws & (ws - 1u))];
            const float to = fminf(t01, tn[2]), t = fmaxf(r.t, to);   // no NaN, and r.t is never -0
            // the point in the new cell: located at voxel resolution, clamped to the cell
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const bool moved = a == 2 ? a2 : a == 1 ? a1 && !a2 : !a1 && !a2;
                const int32_t lo = (int32_t)((moved ? w[a] : r.v[a]) & ~up.y);
                const int32_t at = __float_as_int(__fadd_rd(xadd(r.og[a], xmul(t, r.d[a])), r.off[a]));
                nv[a] = (uint32_t)max(at, lo);
                hi[a] = (uint32_t)lo | up.y;
            }
            const bool set = __funnelshift_r(word, 0u, i) & 1u;   // the shift takes i mod 32
            const uint32_t lo0 = r.lo;
#pragma unroll
            for (int a = 0; a < 3; a++) min_unless(set, r.v[a], nv[a], hi[a]);
            max_unless(set, r.t, to);
            r.last_axis = set ? r.last_axis : a2 ? 2 : a1 ? 1 : 0;
            r.lo = set ? lo0 - (uint32_t)sizeof(LevelDesc) : up.x;
            if (set) {
                if (lo0 == 0u) {
                    r.v[0] = x & (extent - 1u); r.v[1] = y & (extent - 1u); r.v[2] = z & (extent - 1u);
                    res = 1;
                    last = k + 1u;
                } else if (ld.g == 5u) {   // entering a 32^3 block: its slot
                    r.tv = __ldg(&s.table[((uint64_t)((z & (extent - 1u)) >> 5) * s.B + ((y & (extent - 1u)) >> 5)) * s.B +
                                          ((x & (extent - 1u)) >> 5)]);
                }
            } else if (ws & extent) {
                res = 0;
                last = k + 1u;
            }
        }
    }
    r.steps += last;
    return res == kTraceRunning && r.steps >= max_steps ? -1 : res;
}

// ---------------------------------------------------------------------------
// Persistent traversal of n rays.  io.load(i, o, d) reads ray i, io.store(i,
// res, t, c, axis) writes its result (c: grid voxel).  No CTA waits on another:
// a CTA that starts after the queue is drained exits at once.
//
// A warp sets rays up 32 at a time, one per lane, and parks the ones whose
// DDA has to run in a per-warp ring of 64 states in shared memory; a lane
// whose ray ended takes the next parked state.  The set-up (entry slab, the
// bottom-up start) then runs on full warps instead of on the few lanes that
// happen to need a ray at a refill.  A warp's first 32 rays are its own by
// index; the queue hands out what lies beyond all warps' first ones, so a list
// that fits the grid touches no counter (it need not be zeroed then).
// ---------------------------------------------------------------------------
constexpr uint32_t kTraceWarps = 4;     // 128 threads
// 72 registers, 7 CTAs per SM: bounds of 8 (64 registers, 32 bytes of spill) and
// 6 CTAs measured 5 % and 4 % slower on a 1080p GI frame (2.00 and 1.97 ms against 1.90)
constexpr uint32_t kTraceCtas = 7;
constexpr uint32_t kRing = 64;          // parked states per warp
// Rounds once no ray is left to take are longer by this factor: a refill has nothing
// to give, and the longest rays decide the time (two frames of an update 903 -> 887
// us, million rays 306 -> 302; 8 the same, 32: 893 and 304).
constexpr uint32_t kTailFactor = 4;

template <class IO>
__device__ __forceinline__ void svo_trace_queue(const SvoDev& s, const IO& io, uint32_t n, uint32_t max_steps,
                                                uint32_t steps_per_round, uint32_t* __restrict__ queue,
                                                uint32_t* __restrict__ exhausted, unsigned long long* __restrict__ work)
{
    __shared__ TraceTables tb;
    __shared__ ParkedRay ring[kTraceWarps][kRing];
    svo_level_tables(s, tb);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t n_first = gridDim.x * kTraceWarps * 32u;   // rays handed out by index
    uint32_t first = (blockIdx.x * kTraceWarps + w) * 32u;
    const float E = (float)(1u << s.L);
    RayState r;
    uint32_t item = 0;
    bool have = false;
    uint32_t head = 0, count = 0;   // the warp's ring (warp-uniform)
    bool own = true, drained = false;   // the warp's first rays are still to be set up; the queue is exhausted
    uint32_t done_steps = 0, done_rays = 0;   // this lane's finished rays and their DDA steps
    auto store = [&](uint32_t i, int res, const RayState& q) {
        const int32_t c[3] = {(int32_t)q.v[0], (int32_t)q.v[1], (int32_t)q.v[2]};
        io.store(i, res, q.t, c, q.last_axis);
        done_steps += q.steps;
        done_rays++;
        if (res < 0) atomicAdd(exhausted, 1u);
    };
    for (;;) {
        const uint32_t need_mask = __ballot_sync(0xffffffffu, !have);
        const uint32_t n_need = (uint32_t)__popc(need_mask);
        // set up rays, 32 at a time, until the ring can serve every idle lane
        while (n_need && count < n_need && !drained) {
            uint64_t base = first;
            if (own) {
                own = false;
                drained = n <= n_first;
            } else {
                uint32_t q = 0;
                if (lane == 0) q = atomicAdd(queue, 32u);
                base = (uint64_t)n_first + __shfl_sync(0xffffffffu, q, 0);
                drained = base + 32u >= n;
            }
            const uint32_t it = (uint32_t)base + lane;
            bool running = false;
            RayState rs;
            if (base + lane < n) {
                float o[3], d[3];
                io.load(it, o, d);
                const int res = svo_trace_begin(s, tb, o, d, max_steps, rs);
                running = res == kTraceRunning;
                if (!running) store(it, res, rs);
            }
            const uint32_t run_mask = __ballot_sync(0xffffffffu, running);
            if (running) {
                const uint32_t slot = (head + count + (uint32_t)__popc(run_mask & lt_mask)) & (kRing - 1u);
                svo_park(&ring[w][slot], rs, it);
            }
            count += (uint32_t)__popc(run_mask);
            __syncwarp();
        }
        // idle lanes take parked states in lane order
        const uint32_t take = min(n_need, count);
        if (!have) {
            const uint32_t rank = (uint32_t)__popc(need_mask & lt_mask);
            if (rank < take) {
                const uint32_t slot = (head + rank) & (kRing - 1u);
                svo_unpark(&ring[w][slot], E, r, item);
                have = true;
            }
        }
        head = (head + take) & (kRing - 1u);
        count -= take;
        __syncwarp();
        if (!__any_sync(0xffffffffu, have) && drained && count == 0) break;
        if (have) {
            // nothing left to take: the lanes run on by themselves
            const int res = svo_trace_run(s, tb, r, max_steps, drained && count == 0 ? kTailFactor * steps_per_round : steps_per_round);
            if (res != kTraceRunning) {
                store(item, res, r);
                have = false;
            }
        }
    }
    if (!work) return;
    // the frame's traversal work: one pair of 64-bit atomics per warp
    unsigned long long ws = done_steps, wr = done_rays;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        ws += __shfl_down_sync(0xffffffffu, ws, o);
        wr += __shfl_down_sync(0xffffffffu, wr, o);
    }
    if (lane == 0 && wr) {
        atomicAdd(&work[0], ws);
        atomicAdd(&work[1], wr);
    }
}
