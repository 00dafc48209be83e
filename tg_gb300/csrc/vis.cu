// vis.cu -- visibility-buffer pass.
//
// Replaces tg's instanced cluster-box raster (visibility.vert:19-26 with
// cluster_functions.inc:1-38), its fragment-shader DDA (visibility.frag:22-207)
// and the clear pass (clear.comp:15-21) with a binned compute pass:
//
//   1. k_vis_cluster_setup  one thread per (view, cluster pointer): drops
//      clusters outside the frustum or beyond the far plane (bounding
//      sphere, then box corners) and empty clusters, computes a conservative
//      screen-tile rectangle and a lower bound of the packed depth, and
//      appends a 32-byte record.
//   2. k_vis_count          per record: the ws2ms matrix and the camera
//      position in cluster space exactly as the shader does (one thread per
//      record), and its counts per (tile, depth bucket) (a half-warp per record).
//   3. k_vis_prefix         per tile: offsets of its depth buckets; per 256
//                           tiles: their sum and class histogram, also added
//                           up over 64 such groups.
//   4. k_vis_finalize       per 256 tiles: the tiles' offsets and places in the
//                           launch order (heaviest class first), from those sums.
//   5. k_vis_bin_fill       a half-warp per record, a warp per 256 tiles of the
//                           records of many: an 8-byte reference into each of
//                           its (tile, bucket) bins, so every tile's references
//                           are contiguous and run near to far; tiles without
//                           entries are cleared.
//   6. k_vis_tiles          one CTA per tile (heaviest first), one thread per
//      pixel (k_vis_tiles_groups: several, for frames of few tiles): batches of
//      the tile's entries (record and 64-byte bitmask) are gathered by cp.async
//      on an mbarrier;
//      each warp drops, 32 at a time, the entries that none of its pixels can
//      take; every pixel skips entries whose depth bound cannot beat its word and
//      rejects clear misses with a conservative reciprocal slab test; the
//      surviving (pixel, cluster) pairs are compacted by warp ballot and run
//      the shader's exact ray/box test and DDA on full warps, keeping each
//      pixel's minimum packed depth|pointer|voxel word (shared atomicMin);
//      every pixel is written once.
//      k_vis_tiles_queue is the persistent form over many jobs' tiles.
//
// Every pair evaluates the same binary32 operations in the same order as the
// CPU oracle's transcription of visibility.frag, so the buffer is bit-exact.

#include "graph_bins.h"
#include "tgx_internal.cuh"

#include <climits>
#include <cmath>
#include <type_traits>
#include <mutex>
#include <vector>

namespace {

constexpr uint32_t kCluster = 8;
constexpr uint32_t kMaxDdaSteps = 64;      // the 8^3 DDA needs at most 22
constexpr uint32_t kMaxBuckets = 32;       // depth buckets per tile at the finest setting (half an octave each)

struct alignas(16) VisRecord
{
    float    ox, oy, oz;        // camera position in cluster space (visibility.frag:66)
    uint32_t cluster_idx;
    uint32_t object_idx;
    uint32_t d24_lb;            // lower bound of the 24-bit depth field any pixel can get from it
    uint32_t cluster_pointer;
    uint32_t view;
};
static_assert(sizeof(VisRecord) == 32, "record layout");

enum Counter { C_RECORDS = 0, C_ENTRIES = 1, C_DDA_OVERRUN = 2, C_OVERFLOW = 3, C_TILE_QUEUE = 4, C_NONEMPTY = 5,
               C_CHUNKS = 6, C_COUNT = 8 };

// One (tile, cluster) pair as the tile kernel stages it: the record and the
// cluster's 64-byte bitmask.  The tile's bin holds only where the two are (a
// TileRef); the copies into shared memory gather them.
struct alignas(16) TileEntry
{
    VisRecord rec;
    uint32_t bits[16];
};
static_assert(sizeof(TileEntry) == 96, "entry layout");
struct alignas(8) TileRef
{
    uint32_t record, cluster_idx;
};

// A record's tile rectangle: x = tx0 | ty0 << 16, y = tx1 | ty1 << 16 (at most
// 4095 tiles a side); bit 31 of y: the record's tiles are in the chunk list.
constexpr uint32_t kListed = 0x80000000u;
struct TileRect
{
    uint32_t tx0, ty0, w, n;    // first tile, tiles per row, tiles
};
__device__ __forceinline__ TileRect tile_rect(uint2 r)
{
    TileRect t;
    t.tx0 = r.x & 0xffffu;
    t.ty0 = r.x >> 16;
    t.w = (r.y & 0xffffu) - t.tx0 + 1u;
    t.n = t.w * (((r.y & ~kListed) >> 16) - t.ty0 + 1u);
    return t;
}

// Records of more than kHalfWarpTiles tiles are cut into chunks of kChunkTiles,
// a list of (record, first tile) that the counting and the binning pass spread
// over the GPU, a warp per chunk; the others take a half-warp each.  A cluster
// next to the camera covers every tile: a half-warp alone was at 129,600 of them
// for 6 ms.  A record whose chunks find no room in the list goes the other way.
constexpr uint32_t kHalfWarpTiles = 64, kChunkTiles = 256;
// work counters of the tile kernel's counting variant (tgx_vis_work, same order)
enum Work { W_PAIRS = 0, W_DEPTH_SKIPS, W_DIR_SETUPS, W_SLAB_MISSES, W_SURE_HITS, W_EXACT_TESTS, W_DDAS, W_DDA_STEPS,
            W_HITS, W_BATCHES, W_COUNT };
constexpr uint32_t kOrderClasses = 32;     // tiles are launched heaviest class (log2 of bin count) first

// bucket of a depth key: one per power of two of the 24-bit depth, keys < 512 share bucket 0
// Depth buckets of a tile's entries: key = the 24-bit depth field's lower
// bound.  Keys below 512 share the first bucket; above, every half octave of
// the key is a fine bucket (0..31), and a frame uses 32 >> bshift buckets
// (bshift 0, 1 or 2: 32, 16 or 8 buckets, i.e. half, one or two octaves each).
__device__ __forceinline__ uint32_t depth_bucket(uint32_t key, uint32_t bshift)
{
    if (key < 512u) return 0u;
    const uint32_t l = 31u - (uint32_t)__clz(key);   // 9..23
    const uint32_t fine = 2u * (l - 8u) + ((key >> (l - 1u)) & 1u);
    return fine >> bshift;
}
// the smallest key of bucket b
__device__ __forceinline__ uint32_t bucket_lo(uint32_t b, uint32_t bshift)
{
    const uint32_t f = b << bshift;
    return f == 0u ? 0u : (f & 1u) ? (3u << ((f >> 1) + 7u)) : (1u << ((f >> 1) + 8u));
}

// p / tile_w for a pixel p < 512 of a tile (make_view_const: ceil(2^20 / tile_w))
__device__ __forceinline__ uint32_t tile_row(const ViewConst& vc, uint32_t p) { return (p * vc.tile_w_rcp) >> 20; }

// pixel `pix` of the tile at `place` (tile x | y << 16)
__device__ __forceinline__ void tile_pixel_place(const ViewConst& vc, uint32_t place, uint32_t pix, uint32_t& px, uint32_t& py)
{
    const uint32_t row = tile_row(vc, pix);
    px = (place & 0xffffu) * vc.tile_w + pix - row * vc.tile_w;
    py = (place >> 16) * vc.tile_h + row;
}

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool pred)
{
    const uint32_t mask = __ballot_sync(0xffffffffu, pred);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t base = 0;
    if (mask) {
        const int leader = __ffs(mask) - 1;
        if ((int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
        base = __shfl_sync(0xffffffffu, base, leader);
    }
    return base + __popc(mask & ((1u << lane) - 1u));
}

// ---------------------------------------------------------------------------
// 1. per-cluster setup
// ---------------------------------------------------------------------------

// kPacked: the scene's per-pointer table gives each pointer's object and
// whether its cluster is empty (one load beside the pointer's own, instead of
// the chain pointer -> owner -> bitmask); without it (the entry point that
// allocates nothing) the owner and the bitmask are read.
// kInline: the views and outputs of a frame of few views come as an argument;
// the first CTA stores them in the tables the later passes read.
constexpr uint32_t kInlineViews = 8;
struct InlineViews
{
    ViewConst views[kInlineViews];
    unsigned long long* outs[kInlineViews];
};
struct NoViews {};

template <bool kPacked, class Inline>
__global__ void __launch_bounds__(256, 4) k_vis_cluster_setup(
    const tgx_object* __restrict__ objects, const uint32_t* __restrict__ cluster_pointers,
    const uint32_t* __restrict__ c2o, const uint32_t* __restrict__ bits, const uint32_t* __restrict__ cp_obj,
    uint32_t n_cp, const __grid_constant__ Inline inl, ViewConst* views, unsigned long long** outs, uint32_t n_views,
    VisRecord* __restrict__ records, uint2* __restrict__ rects, uint32_t record_capacity, uint32_t* __restrict__ counters,
    uint32_t* __restrict__ zero, uint32_t n_zero, uint2* __restrict__ chunks, uint32_t chunk_cap,
    tgx_dev_status* __restrict__ status)
{
    pdl_wait();
    const uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // the (tile, bucket) counts start at zero; k_vis_count runs after this kernel
    for (uint64_t i = gid; i < n_zero; i += (uint64_t)gridDim.x * blockDim.x) zero[i] = 0u;
    constexpr bool kInline = !std::is_same<Inline, NoViews>::value;
    if constexpr (kInline) {
        if (blockIdx.x == 0) {
            constexpr uint32_t kWords = sizeof(ViewConst) / 4u;
            for (uint32_t i = threadIdx.x; i < n_views * kWords; i += blockDim.x)
                reinterpret_cast<uint32_t*>(views)[i] = reinterpret_cast<const uint32_t*>(inl.views)[i];
            if (threadIdx.x < n_views) outs[threadIdx.x] = inl.outs[threadIdx.x];
        }
    }
    const uint32_t v = (uint32_t)(gid / n_cp);
    const uint32_t cp = (uint32_t)(gid % n_cp);
    bool keep = false;
    VisRecord rec = {};
    uint32_t tx0 = 0, ty0 = 0, tx1 = 0, ty1 = 0;
    if (v < n_views) {
        const ViewConst* table = views;
        if constexpr (kInline) table = inl.views;
        const ViewConst& vc = table[v];
        const uint32_t ci = cluster_pointers[cp];
        const uint32_t po = kPacked ? cp_obj[cp] : 0u;
        if (!kPacked || !(po >> 31)) {   // bit 31: the cluster has no set voxel
            bool oi_cull = false;
            const uint32_t oi = kPacked ? po : c2o[ci];
            const tgx_object& od = objects[oi];
            const uint32_t nx = od.n_cluster_pointers_per_dim[0], ny = od.n_cluster_pointers_per_dim[1];
            const uint32_t rel = cp - od.first_cluster_pointer;
            const uint32_t rx = rel % nx, ry = (rel / nx) % ny, rz = rel / (nx * ny);
            const float offx = (float)(rx * kCluster), offy = (float)(ry * kCluster), offz = (float)(rz * kCluster);
            const float half = xmul((float)kCluster, 0.5f);
            const float ohx = xmul(half, (float)od.n_cluster_pointers_per_dim[0]);
            const float ohy = xmul(half, (float)od.n_cluster_pointers_per_dim[1]);
            const float ohz = xmul(half, (float)od.n_cluster_pointers_per_dim[2]);
            // the box's corner 0 relative to the camera and its three edges (8 voxels
            // along each rotated axis); corner k = base + (k&1) ex + (k&2) ey + (k&4) ez.
            // Rounding differs from a per-corner transform by ulps, far inside the
            // cull's slack (0.05 + 1e-5 |p|) and the rectangle's 2-pixel margin.
            float base[3], ex[3], ey[3], ez[3];
            {
                const float lx = offx - ohx, ly = offy - ohy, lz = offz - ohz;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const float r0 = od.rotation[r], r1 = od.rotation[4 + r], r2 = od.rotation[8 + r];
                    base[r] = r0 * lx + r1 * ly + r2 * lz + od.translation[r] - vc.cam[r];
                    ex[r] = 8.0f * r0; ey[r] = 8.0f * r1; ez[r] = 8.0f * r2;
                }
            }

            // ---- bounding-sphere cull against the side planes and the far plane ----
            {
                float q[3];
#pragma unroll
                for (int r = 0; r < 3; r++) q[r] = base[r] + 0.5f * (ex[r] + ey[r] + ez[r]);
                const float rad = 6.9283f + 0.05f + 1e-5f * (fabsf(q[0]) + fabsf(q[1]) + fabsf(q[2]));
                const float dist = sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
                bool out = dist - rad > vc.far_plane * 1.0001f;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    out |= vc.planes[3 * k] * q[0] + vc.planes[3 * k + 1] * q[1] + vc.planes[3 * k + 2] * q[2] < -rad;
                if (out) oi_cull = true;
            }

            if (!kPacked && !oi_cull) {
                // a cluster without set bits never writes (its DDA finds nothing)
                const uint4* w = reinterpret_cast<const uint4*>(bits + (uint64_t)ci * 16u);
                const uint4 a = w[0], b = w[1], c = w[2], d = w[3];
                oi_cull = !(a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w | c.x | c.y | c.z | c.w | d.x | d.y | d.z | d.w);
            }
            if (!oi_cull) {
            // ---- culling and conservative screen rectangle (never exact-critical: widened) ----
            float fxmin = 1e30f, fxmax = -1e30f, fymin = 1e30f, fymax = -1e30f;
            bool full = false, any_front = false;
            bool inside0 = false, inside1 = false, inside2 = false, inside3 = false;
            float cxw = 0.0f, cyw = 0.0f, czw = 0.0f;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                float p[3];
#pragma unroll
                for (int r = 0; r < 3; r++)
                    p[r] = base[r] + ((k & 1) ? ex[r] : 0.0f) + ((k & 2) ? ey[r] : 0.0f) + ((k & 4) ? ez[r] : 0.0f);
                cxw += p[0]; cyw += p[1]; czw += p[2];
                const float depth = p[0] * vc.fwd[0] + p[1] * vc.fwd[1] + p[2] * vc.fwd[2];
                if (depth > -0.5f) any_front = true;
                const float slack = -(0.05f + 1e-5f * (fabsf(p[0]) + fabsf(p[1]) + fabsf(p[2])));
                inside0 |= vc.planes[0] * p[0] + vc.planes[1] * p[1] + vc.planes[2] * p[2] > slack;
                inside1 |= vc.planes[3] * p[0] + vc.planes[4] * p[1] + vc.planes[5] * p[2] > slack;
                inside2 |= vc.planes[6] * p[0] + vc.planes[7] * p[1] + vc.planes[8] * p[2] > slack;
                inside3 |= vc.planes[9] * p[0] + vc.planes[10] * p[1] + vc.planes[11] * p[2] > slack;
                const float s = vc.inv_basis[0] * p[0] + vc.inv_basis[1] * p[1] + vc.inv_basis[2] * p[2];
                if (depth < 0.5f || s <= 0.0f) { full = true; continue; }
                const float fa = (vc.inv_basis[3] * p[0] + vc.inv_basis[4] * p[1] + vc.inv_basis[5] * p[2]) / s;
                const float fb = (vc.inv_basis[6] * p[0] + vc.inv_basis[7] * p[1] + vc.inv_basis[8] * p[2]) / s;
                fxmin = fminf(fxmin, fa); fxmax = fmaxf(fxmax, fa);
                fymin = fminf(fymin, fb); fymax = fmaxf(fymax, fb);
            }
            // lower bound of the distance from the camera to any point of the box
            const float cdist = sqrtf(cxw * cxw + cyw * cyw + czw * czw) * 0.125f;
            const float lb = fmaxf(0.0f, cdist * (1.0f - 1e-5f) - 6.9283f - 0.01f);
            const float lbq = lb / vc.far_plane;
            if (any_front && inside0 && inside1 && inside2 && inside3 && lbq <= 1.0001f) {
                const float W = (float)vc.width, H = (float)vc.height;
                float x0, x1, y0, y1;
                if (full) {
                    x0 = 0.0f; y0 = 0.0f; x1 = W - 1.0f; y1 = H - 1.0f;
                } else {
                    const float m = 2.0f;   // pixels of slack for the float projection
                    x0 = fxmin * W - 0.5f - m; x1 = fxmax * W - 0.5f + m;
                    y0 = (1.0f - fymax) * H - 0.5f - m; y1 = (1.0f - fymin) * H - 0.5f + m;
                }
                if (!(x1 < 0.0f || y1 < 0.0f || x0 > W - 1.0f || y0 > H - 1.0f)) {
                    const int ix0 = max(0, (int)floorf(x0)), iy0 = max(0, (int)floorf(y0));
                    const int ix1 = min((int)vc.width - 1, (int)ceilf(x1));
                    const int iy1 = min((int)vc.height - 1, (int)ceilf(y1));
                    if (ix0 <= ix1 && iy0 <= iy1) {
                        keep = true;
                        tx0 = (uint32_t)ix0 / vc.tile_w; ty0 = (uint32_t)iy0 / vc.tile_h;
                        tx1 = (uint32_t)ix1 / vc.tile_w; ty1 = (uint32_t)iy1 / vc.tile_h;
                    }
                }
            }
            if (keep) {
                // the exact cluster-space origin is computed by k_vis_count
                rec.cluster_idx = ci;
                rec.cluster_pointer = cp;
                rec.object_idx = oi;
                const float k24 = fminf(lbq, 1.0f) * 16777215.0f;
                rec.d24_lb = k24 >= 2.0f ? (uint32_t)k24 - 1u : 0u;
                rec.view = v;
            }
            }
        }
    }
    const uint32_t slot = warp_append(&counters[C_RECORDS], keep);
    if (!keep) return;
    if (slot >= record_capacity) {
        dev_error(status, TGX_ERR_CAPACITY, 1, slot);
        return;
    }
    records[slot] = rec;
    uint32_t listed = 0u;
    const uint32_t n = (tx1 - tx0 + 1u) * (ty1 - ty0 + 1u);
    if (n > kHalfWarpTiles) {
        const uint32_t n_chunks = (n + kChunkTiles - 1u) / kChunkTiles;
        const uint32_t first = atomicAdd(&counters[C_CHUNKS], n_chunks);
        const bool room = first <= chunk_cap && n_chunks <= chunk_cap - first;
        for (uint32_t k = 0; k < n_chunks && first + k < chunk_cap && first + k >= first; k++)
            chunks[first + k] = make_uint2(room ? slot : 0xffffffffu, k * kChunkTiles);
        if (room) listed = kListed;
    }
    rects[slot] = make_uint2(tx0 | (ty0 << 16), tx1 | (ty1 << 16) | listed);
}

// ---------------------------------------------------------------------------
// 2. per record: the exact ws2ms and ray origin (visibility.frag:57-66), one
//    thread per record; then its per-(tile, bucket) counts, a warp per listed
//    chunk and a half-warp per other record (records span ~17 tiles on average)
//    with the lanes over the tiles.  The loops write different fields and
//    buffers; the cull kept apart runs at high occupancy.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_vis_count(VisRecord* __restrict__ records, const uint2* __restrict__ rects,
                                                  const uint32_t* __restrict__ counters, uint32_t record_capacity,
                                                  const tgx_object* __restrict__ objects,
                                                  const ViewConst* __restrict__ views,
                                                  uint32_t* __restrict__ bucket_cnt, uint32_t n_tiles,
                                                  uint32_t bshift, const uint2* __restrict__ chunks, uint32_t chunk_cap)
{
    pdl_wait();
    const uint32_t n = min(counters[C_RECORDS], record_capacity);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        VisRecord& rec = records[i];
        const tgx_object& od = objects[rec.object_idx];
        const ViewConst& vc = views[rec.view];
        const uint32_t nx = od.n_cluster_pointers_per_dim[0], ny = od.n_cluster_pointers_per_dim[1];
        const uint32_t rel = rec.cluster_pointer - od.first_cluster_pointer;
        const float offx = (float)((rel % nx) * kCluster), offy = (float)(((rel / nx) % ny) * kCluster);
        const float offz = (float)((rel / (nx * ny)) * kCluster);
        const float half = xmul((float)kCluster, 0.5f);
        float rot[16], m0[16], m1[16], m2[16], m3[16], ws2ms[16];
#pragma unroll
        for (int k = 0; k < 16; k++) rot[k] = od.rotation[k];
        dm4_translate(-od.translation[0], -od.translation[1], -od.translation[2], m0);
        dm4_inverse(rot, m1);
        dm4_translate(xmul(half, (float)od.n_cluster_pointers_per_dim[0]), xmul(half, (float)od.n_cluster_pointers_per_dim[1]),
                      xmul(half, (float)od.n_cluster_pointers_per_dim[2]), m2);
        dm4_translate(-offx, -offy, -offz, m3);
        dm4_mul(m3, m2, ws2ms);
        dm4_mul(ws2ms, m1, ws2ms);
        dm4_mul(ws2ms, m0, ws2ms);
        float o[3];
        dm4_mulv4(ws2ms, vc.cam[0], vc.cam[1], vc.cam[2], 1.0f, o);
        rec.ox = o[0]; rec.oy = o[1]; rec.oz = o[2];
    }
    auto count = [&](uint32_t i, const TileRect& t, uint32_t k) {
        const ViewConst& vc = views[records[i].view];
        const uint32_t tile = vc.tile_base + (t.ty0 + k / t.w) * vc.tiles_x + t.tx0 + k % t.w;
        atomicAdd(&bucket_cnt[depth_bucket(records[i].d24_lb, bshift) * n_tiles + tile], 1u);
    };
    const uint32_t n_chunks = min(counters[C_CHUNKS], chunk_cap);
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < n_chunks; c += (gridDim.x * blockDim.x) >> 5) {
        const uint2 ch = chunks[c];
        if (ch.x >= n) continue;
        const TileRect t = tile_rect(rects[ch.x]);
        const uint32_t end = min(t.n, ch.y + kChunkTiles);
        for (uint32_t k = ch.y + (threadIdx.x & 31u); k < end; k += 32u) count(ch.x, t, k);
    }
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; i < n; i += (gridDim.x * blockDim.x) >> 4) {
        const uint2 r = rects[i];
        if (r.y & kListed) continue;
        const TileRect t = tile_rect(r);
        for (uint32_t k = threadIdx.x & 15u; k < t.n; k += 16u) count(i, t, k);
    }
}

// ---------------------------------------------------------------------------
// 3. per-tile bucket offsets (one thread per tile, bucket-major = coalesced),
//    and per CTA of 256 tiles: the sum of the tile totals and the histogram
//    of tile classes (groups = [n_ctas][kGroupWords]: the sum, then the classes),
//    added to those of its 64 CTAs (supers, zero before, the same layout)
// ---------------------------------------------------------------------------

constexpr uint32_t kScanTiles = 256;   // tiles per CTA of the prefix and finalize kernels
constexpr uint32_t kSuperGroups = 64;  // CTAs whose sums are added up
constexpr uint32_t kGroupWords = 1 + kOrderClasses;

__host__ __device__ constexpr uint32_t scan_groups(uint32_t n_tiles) { return (n_tiles + kScanTiles - 1) / kScanTiles; }
__host__ __device__ constexpr uint32_t scan_supers(uint32_t n_tiles)
{
    return (scan_groups(n_tiles) + kSuperGroups - 1) / kSuperGroups;
}

__device__ __forceinline__ uint32_t tile_class(uint32_t total) { return total ? 32u - __clz(total) : 0u; }

template <uint32_t kBuckets>
__global__ void __launch_bounds__(kScanTiles) k_vis_prefix(uint32_t* __restrict__ bucket_cnt,
                                                          uint32_t* __restrict__ tile_total, uint32_t n_tiles,
                                                          uint32_t* __restrict__ groups, uint32_t* __restrict__ supers)
{
    __shared__ uint32_t cls[kOrderClasses];
    __shared__ uint32_t wsum[kScanTiles / 32];
    if (threadIdx.x < kOrderClasses) cls[threadIdx.x] = 0;
    pdl_wait();
    __syncthreads();
    const uint32_t t = blockIdx.x * kScanTiles + threadIdx.x;
    uint32_t run = 0;
    if (t < n_tiles) {
        uint32_t c[kBuckets];   // all loads first: the stores below must not wait on them one by one
#pragma unroll
        for (uint32_t b = 0; b < kBuckets; b++) c[b] = bucket_cnt[b * n_tiles + t];
#pragma unroll
        for (uint32_t b = 0; b < kBuckets; b++) {
            bucket_cnt[b * n_tiles + t] = run;   // becomes the fill cursor
            run += c[b];
        }
        tile_total[t] = run;
        atomicAdd(&cls[tile_class(run)], 1u);
    }
    uint32_t sum = run;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31u) == 0) wsum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x < kGroupWords) {
        uint32_t v = 0;
        if (threadIdx.x == 0)
#pragma unroll
            for (uint32_t w = 0; w < kScanTiles / 32; w++) v += wsum[w];
        else v = cls[threadIdx.x - 1];
        groups[blockIdx.x * kGroupWords + threadIdx.x] = v;
        if (v) atomicAdd(&supers[blockIdx.x / kSuperGroups * kGroupWords + threadIdx.x], v);
    }
}

// ---------------------------------------------------------------------------
// 4. per CTA of 256 tiles: every tile's offset and place in the launch order
//    (heaviest class first).  Its base and class cursors come from the sums of
//    all supers and of the groups before it in its own.
//    (One CTA that scanned all groups' sums first took 104 us at 3488 groups;
//    reading every group's sums in every CTA 10 us at 507, 7 at 127.)
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(kScanTiles) k_vis_finalize(const uint32_t* __restrict__ tile_total, uint32_t n_tiles,
                                                            const uint32_t* __restrict__ groups,
                                                            const uint32_t* __restrict__ supers,
                                                            uint32_t* __restrict__ tile_off,
                                                            uint4* __restrict__ slot_info, uint32_t bin_capacity,
                                                            uint32_t* __restrict__ counters,
                                                            uint32_t* __restrict__ next_counters,
                                                            const ViewConst* __restrict__ views, uint32_t n_views)
{
    constexpr uint32_t kWarps = kScanTiles / 32;
    __shared__ uint32_t cur[kOrderClasses];
    __shared__ uint32_t part_tot[kWarps][kOrderClasses], part_pre[kWarps][kOrderClasses];
    __shared__ uint32_t red_pre[kWarps], red_all[kWarps], wsum[kWarps];
    const uint32_t g = blockIdx.x, lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t sg = g / kSuperGroups, n_supers = scan_supers(n_tiles);
    const uint32_t t = g * kScanTiles + threadIdx.x;
    const bool valid = t < n_tiles;
    // the tile's view and place in it; the view table is older than the kernels
    // before, whose end need not be awaited for it
    uint32_t view = 0, place = 0;
    if (valid) {
        uint32_t hi = n_views - 1;   // the last view whose first tile is <= t
        while (view < hi) {
            const uint32_t mid = (view + hi + 1) >> 1;
            if (__ldcg(&views[mid].tile_base) <= t) view = mid; else hi = mid - 1;
        }
        const uint32_t lt = t - __ldcg(&views[view].tile_base), tiles_x = __ldcg(&views[view].tiles_x);
        place = lt % tiles_x | (lt / tiles_x) << 16;
    }
    pdl_wait();
    // this group's base (the sums before it) and the frame's total
    uint32_t pre = 0, all = 0;
    for (uint32_t i = threadIdx.x; i < n_supers; i += kScanTiles) {
        const uint32_t v = supers[i * kGroupWords];
        all += v;
        pre += i < sg ? v : 0u;
    }
    const uint32_t own = sg * kSuperGroups + threadIdx.x;   // kSuperGroups <= kScanTiles
    if (own < g) pre += groups[own * kGroupWords];
    // per class (lane): its count over all groups and over the groups before this one
    uint32_t ct = 0, cp = 0;
    for (uint32_t b = wid; b < n_supers; b += kWarps) {
        const uint32_t v = supers[b * kGroupWords + 1u + lane];
        ct += v;
        cp += b < sg ? v : 0u;
    }
    for (uint32_t b = sg * kSuperGroups + wid; b < g; b += kWarps) cp += groups[b * kGroupWords + 1u + lane];
    part_tot[wid][lane] = ct;
    part_pre[wid][lane] = cp;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pre += __shfl_xor_sync(0xffffffffu, pre, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    if (lane == 0) { red_pre[wid] = pre; red_all[wid] = all; }
    // the tiles' totals, scanned within each warp
    const uint32_t x = valid ? tile_total[t] : 0u;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    if (wid == 0) {   // class bases, heaviest class first, plus this group's share before it
        uint32_t tot = 0, before = 0;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; w++) { tot += part_tot[w][lane]; before += part_pre[w][lane]; }
        uint32_t suffix = tot;   // classes lane .. 31
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_down_sync(0xffffffffu, suffix, o);
            if (lane + o < 32) suffix += y;
        }
        cur[lane] = suffix - tot + before;
        if (g == 0 && lane == 0) counters[C_NONEMPTY] = n_tiles - tot;   // class 0: the tiles without entries
    }
    __syncthreads();
    uint32_t base = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; w++) { base += red_pre[w]; total += red_all[w]; }
    if (g == 0 && threadIdx.x == 0) {
        counters[C_ENTRIES] = total;
        counters[C_OVERFLOW] = total > bin_capacity ? 1u : 0u;
    }
    if (g == 0 && next_counters && threadIdx.x < C_COUNT) next_counters[threadIdx.x] = 0u;   // the next frame's
    for (uint32_t w = 0; w < wid; w++) base += wsum[w];
    if (valid) {
        const uint32_t off = base + incl - x;
        tile_off[t] = off;
        slot_info[atomicAdd(&cur[tile_class(x)], 1u)] = make_uint4(view, off, x, place);
    }
}

// ---------------------------------------------------------------------------
// 5. bin fill: as in the count, a warp per listed chunk and a half-warp per
//    other record, a lane per tile, which takes the next place of the tile's
//    bucket and writes the 8-byte reference there.  (Writing the 96-byte entry
//    itself took 26 us at 1080p, 512 objects, and 210 us for 7.3 M entries;
//    the tile kernel gathers it as quickly from the record as from a copy.)
//    Then a warp per tile without entries clears it, unless that is left to the
//    tile kernel, which spreads writes to host memory over its time.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_vis_bin_fill(const VisRecord* __restrict__ records,
                                                     const uint2* __restrict__ rects,
                                                     const uint32_t* __restrict__ counters,
                                                     const ViewConst* __restrict__ views,
                                                     const uint32_t* __restrict__ tile_off,
                                                     uint32_t* __restrict__ cursor, TileRef* __restrict__ refs,
                                                     uint32_t n_tiles, uint32_t bin_capacity, uint32_t bshift,
                                                     const uint2* __restrict__ chunks, uint32_t chunk_cap,
                                                     const uint4* __restrict__ slot_info,
                                                     unsigned long long* const* __restrict__ outs, uint32_t clear,
                                                     tgx_dev_status* __restrict__ status)
{
    pdl_wait();
    // after an overflow the tile kernel scans all records instead
    const uint32_t n = counters[C_OVERFLOW] ? 0u : counters[C_RECORDS];
    // tiles k, k + step, ... below end of record i, four at a time so that their atomics are in flight together
    auto fill = [&](uint32_t i, const TileRect& t, uint32_t k, uint32_t end, uint32_t step) {
        const VisRecord& rec = records[i];
        const ViewConst& vc = views[rec.view];
        const uint32_t row = depth_bucket(rec.d24_lb, bshift) * n_tiles;
        const uint32_t base = vc.tile_base + t.ty0 * vc.tiles_x + t.tx0;
        const TileRef ref = {i, rec.cluster_idx};
        for (; k < end; k += 4u * step) {
            uint32_t pos[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) {
                const uint32_t kj = k + j * step;
                if (kj >= end) continue;
                const uint32_t tile = base + (kj / t.w) * vc.tiles_x + kj % t.w;
                pos[j] = tile_off[tile] + atomicAdd(&cursor[row + tile], 1u);
            }
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) {
                if (k + j * step >= end) continue;
                if (pos[j] >= bin_capacity) dev_error(status, TGX_ERR_DEVICE_FAULT, 3, pos[j]);
                else refs[pos[j]] = ref;
            }
        }
    };
    const uint32_t n_chunks = min(counters[C_CHUNKS], chunk_cap);
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < n_chunks; c += (gridDim.x * blockDim.x) >> 5) {
        const uint2 ch = chunks[c];
        if (ch.x >= n) continue;
        const TileRect t = tile_rect(rects[ch.x]);
        fill(ch.x, t, ch.y + (threadIdx.x & 31u), min(t.n, ch.y + kChunkTiles), 32u);
    }
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 4; i < n; i += (gridDim.x * blockDim.x) >> 4) {
        const uint2 r = rects[i];
        if (r.y & kListed) continue;
        const TileRect t = tile_rect(r);
        fill(i, t, threadIdx.x & 15u, t.n, 16u);
    }
    if (!clear) return;
    for (uint32_t slot = counters[C_NONEMPTY] + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); slot < n_tiles;
         slot += (gridDim.x * blockDim.x) >> 5) {
        const uint4 si = slot_info[slot];
        const ViewConst& vc = views[si.x];
        unsigned long long* const out = outs[si.x];
        for (uint32_t p = threadIdx.x & 31u; p < vc.tile_w * vc.tile_h; p += 32u) {
            uint32_t px, py;
            tile_pixel_place(vc, si.w, p, px, py);
            if (px < vc.width && py < vc.height) out[(size_t)py * vc.width + px] = ULLONG_MAX;
        }
    }
}

// ---------------------------------------------------------------------------
// 6. per-tile ray/cluster evaluation
// ---------------------------------------------------------------------------

// min and max that give NaN when either operand is NaN
__device__ __forceinline__ float min_nan(float a, float b)
{
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float max_nan(float a, float b)
{
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// gmax(gmax(q0, q1), q2) of the near-plane quotients q_i = (p_i - o_i) / d_i
// (F32_MIN when d_i is 0 or NaN), each an exactly rounded division, as the slab
// test and the voxel entry of visibility.frag compute them.  The maximum is
// located first with the correctly rounded reciprocals r_i (NaN when d_i is 0;
// RN(n * RN(1/d)) is within 2^-23 + 2^-24 relative of the exact quotient); when
// the largest approximation beats the next by more than 4e-6 of their
// magnitudes, and these are far from underflow and overflow, only that axis is
// divided, since its exact quotient is then surely the largest and the maximum
// of distinct values does not depend on the comparison order.  Otherwise (near
// ties, a direction component of 0 or NaN) all three are divided.
__device__ __forceinline__ float max_near_quot(float ox, float oy, float oz, float dx, float dy, float dz, float rx,
                                               float ry, float rz, float px, float py, float pz)
{
    const float nx = xsub(px, ox), ny = xsub(py, oy), nz = xsub(pz, oz);
    const float ax = xmul(nx, rx), ay = xmul(ny, ry), az = xmul(nz, rz);
    const float top = max_nan(max_nan(ax, ay), az);
    const float next = fmaxf(fminf(ax, ay), fminf(fmaxf(ax, ay), az));
    const float mag = fabsf(top) + fabsf(next);
    if (next < top - 4e-6f * mag && mag >= 1e-30f && mag <= 1e30f) {
        const bool x = ax == top, y = ay == top;
        return xdiv(x ? nx : y ? ny : nz, x ? dx : y ? dy : dz);
    }
    const float qx = dx > 0.0f || dx < 0.0f ? xdiv(nx, dx) : F32_MIN_TG;
    const float qy = dy > 0.0f || dy < 0.0f ? xdiv(ny, dy) : F32_MIN_TG;
    const float qz = dz > 0.0f || dz < 0.0f ? xdiv(nz, dz) : F32_MIN_TG;
    return gmax(gmax(qx, qy), qz);
}

// Floats of small integers and back by the bits of 2^23 + i: an addition each,
// where a conversion runs at a quarter of the rate.
constexpr float kTwo23 = 8388608.0f;
__device__ __forceinline__ float small_float(uint32_t i) { return __uint_as_float(0x4b000000u | i) - kTwo23; }
// min(max(floor(h), 0), 7), 0 for NaN
__device__ __forceinline__ uint32_t voxel_coord(float h)
{
    return __float_as_uint(__fadd_rz(fminf(fmaxf(h, 0.0f), 7.0f), kTwo23)) & 7u;
}

// The DDA's place in one word: bits 0..8 the voxel index; per axis the steps left
// before the border, 3 bits and a guard that the step past it sets (12..15,
// 16..19, 20..23); from bit 24 the steps taken, bit 30 at kMaxDdaSteps.
constexpr uint32_t kDdaLeft = 1u << 15 | 1u << 19 | 1u << 23, kDdaOverrun = 1u << 30;
static_assert(kMaxDdaSteps == 64, "bit 30 of the DDA's word");

// One axis' start: its distance, its step distance and what a step adds to the
// word.  For d < 0 the distances are those of the mirrored axis: (h - x) / -d.
__device__ __forceinline__ void dda_axis(float d, float r, float h, uint32_t x, float enter, uint32_t shift, uint32_t stride, float& tm,
                                         float& td, uint32_t& inc, uint32_t& place)
{
    const float xf = small_float(x);
    const bool pos = d > 0.0f;
    const float t = xadd(enter, xdiv(pos ? xsub(xf + 1.0f, h) : xsub(h, xf), fabsf(d)));
    const bool moves = pos || d < 0.0f;
    tm = moves ? t : F32_MAX_TG;
    td = moves ? fabsf(r) : F32_MAX_TG;
    inc = (1u << 24) + (moves ? (pos ? stride : 0u - stride) - (1u << shift) : 0u);
    place += (x * stride) + ((pos ? 7u - x : x) << shift);
}

// One (pixel, cluster) fragment of visibility.frag:78-207 given the cluster-space
// ray (o, d), the correctly rounded reciprocals (ix, iy, iz) of its direction
// components (NaN where one is 0) and the cluster's 16 bit words.  Returns the packed
// word or ~0.  The DDA's per-axis steps 1/|d| are |ix| etc. exactly: a
// correctly rounded 1/(-d) is the negated 1/d.  The first voxel is tested
// before the DDA's start distances are computed: a hit there never reads them.
// 2^-k when f = 2^k with 2^-k a normal float, else 0.  For such f,
// RN(v * 2^-k) equals RN(v / f) for every v: both round the same exact real
// once (zeros, infinities and subnormal results included; a NaN stays a NaN).
__device__ __forceinline__ float pow2_reciprocal(float f)
{
    const uint32_t b = __float_as_uint(f);
    const uint32_t e = b >> 23;   // sign 0 and biased exponent
    return (b & 0x7fffffu) == 0u && e >= 1u && e <= 253u ? __uint_as_float((254u - e) << 23) : 0.0f;
}

template <bool kCount = false>
__device__ __forceinline__ unsigned long long vis_pair(float ox, float oy, float oz, float dx, float dy, float dz,
                                                       float ix, float iy, float iz, bool sure_hit,
                                                       const uint32_t* __restrict__ w, uint32_t cluster_pointer,
                                                       float far_plane, float far_rcp, uint32_t* overrun,
                                                       uint32_t* work = nullptr)
{
    float enter;
    if (sure_hit) {
        // the box test surely passes: only the entry distance is needed, and of
        // each axis only the near-plane quotient can be ray_aabb's minimum
        enter = max_near_quot(ox, oy, oz, dx, dy, dz, ix, iy, iz, dx > 0.0f ? 0.0f : 8.0f, dy > 0.0f ? 0.0f : 8.0f,
                              dz > 0.0f ? 0.0f : 8.0f);
    } else {
        float exit_;
        if (!ray_aabb(ox, oy, oz, dx, dy, dz, 0.0f, 0.0f, 0.0f, 8.0f, 8.0f, 8.0f, enter, exit_)) return ULLONG_MAX;
        // a ray parallel to a slab it does not cross is never rasterised
        if ((dx == 0.0f && (ox < 0.0f || ox > 8.0f)) || (dy == 0.0f && (oy < 0.0f || oy > 8.0f)) ||
            (dz == 0.0f && (oz < 0.0f || oz > 8.0f)))
            return ULLONG_MAX;
    }
    if (kCount) work[W_DDAS]++;
    const bool ent = enter > 0.0f;
    const float hx = ent ? xadd(ox, xmul(enter, dx)) : ox;
    const float hy = ent ? xadd(oy, xmul(enter, dy)) : oy;
    const float hz = ent ? xadd(oz, xmul(enter, dz)) : oz;
    const uint32_t x = voxel_coord(hx), y = voxel_coord(hy), z = voxel_coord(hz);
    uint32_t rvi = 64u * z + 8u * y + x;
    if (kCount) work[W_DDA_STEPS]++;
    if (!((w[rvi >> 5] >> (rvi & 31u)) & 1u)) {
        float tmx, tmy, tmz, tdx, tdy, tdz;
        uint32_t incx, incy, incz, place = 1u << 24;
        dda_axis(dx, ix, hx, x, enter, 12u, 1u, tmx, tdx, incx, place);
        dda_axis(dy, iy, hy, y, enter, 16u, 8u, tmy, tdy, incy, place);
        dda_axis(dz, iz, hz, z, enter, 20u, 64u, tmz, tdz, incz, place);
        for (;;) {
            // the nearer of x and y (y unless x is less), z unless that is less
            const bool x_first = tmx < tmy;
            const bool xy_first = (x_first ? tmx : tmy) < tmz;
            const bool step_x = xy_first && x_first, step_y = xy_first && !x_first;
            tmx = step_x ? xadd(tmx, tdx) : tmx;
            tmy = step_y ? xadd(tmy, tdy) : tmy;
            tmz = xy_first ? tmz : xadd(tmz, tdz);
            place += step_x ? incx : step_y ? incy : incz;
            if (place & kDdaLeft) return ULLONG_MAX;
            if (kCount) work[W_DDA_STEPS]++;
            if ((w[(place >> 5) & 15u] >> (place & 31u)) & 1u) break;
            if (place & kDdaOverrun) {
                atomicAdd(overrun, 1u);
                return ULLONG_MAX;
            }
        }
        rvi = place & 511u;
    }
    if (kCount) work[W_HITS]++;
    // entry distance of the voxel box (visibility.frag:155): only the near-plane
    // quotient of each axis can be the maximum, since (vmin-o)/d <= (vmax-o)/d for d>0
    const float ve = max_near_quot(ox, oy, oz, dx, dy, dz, ix, iy, iz, small_float((rvi & 7u) + (dx > 0.0f ? 0u : 1u)),
                                   small_float(((rvi >> 3) & 7u) + (dy > 0.0f ? 0u : 1u)),
                                   small_float((rvi >> 6) + (dz > 0.0f ? 0u : 1u)));
    // a power-of-two far plane (far_rcp != 0) divides by one exact product
    const float depth = gmax(0.0f, far_rcp != 0.0f ? xmul(ve, far_rcp) : xdiv(ve, far_plane));
    if (!(depth <= 1.0f)) return ULLONG_MAX;
    const unsigned long long d24 = __float2uint_rz(xmul(depth, 16777215.0f));   // < 2^24
    return (d24 << 40) | ((unsigned long long)cluster_pointer << 9) | (unsigned long long)rvi;
}

// Conservative classification of the exact box test of vis_pair: kMiss or
// kHit only when the exact test surely gives that answer, else kUnsure.  Slab
// distances use a correctly rounded reciprocal (error < 2 ulp against the
// exact quotient of the same numerator); an answer is given only with a 1e-5
// relative margin.  A zero direction component comes with a NaN reciprocal
// (tile_batch): that, a NaN origin and distances that overflow leave NaN or
// infinity in the comparisons, which all fail then, and the exact test decides.
enum SlabClass { kMiss = 0, kUnsure = 1, kHit = 2 };
__device__ __forceinline__ int slab_class(float ox, float oy, float oz, float ix, float iy, float iz)
{
    const float ax = -ox * ix, bx = (8.0f - ox) * ix;
    const float ay = -oy * iy, by = (8.0f - oy) * iy;
    const float az = -oz * iz, bz = (8.0f - oz) * iz;
    const float en = max_nan(max_nan(min_nan(ax, bx), min_nan(ay, by)), min_nan(az, bz));
    const float ex = min_nan(min_nan(max_nan(ax, bx), max_nan(ay, by)), max_nan(az, bz));
    const float tol = 1e-5f * (fabsf(en) + fabsf(ex)) + 1e-30f;
    if (ex < -tol || en > ex + 2.0f * tol) return kMiss;
    if (ex > tol && en < ex - 2.0f * tol) return kHit;
    return kUnsure;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// One job's tile inputs: a scene's records and bins for its views.
struct TileJob
{
    const VisRecord* records;
    const uint2* rects;
    const TileRef* refs;         // the bins, tile after tile
    const uint4* slot_info;      // per launch slot (heavy first): view, first entry, entry count, tile x | y << 16
    const ViewConst* views;
    const uint32_t* bits;
    const float* inv_rot;
    unsigned long long* const* outs;
    uint32_t* counters;
    uint32_t* host_counters;     // pinned host memory for the frame's entry count and overflow flag, or null
    uint32_t n_tiles;
    uint32_t cleared;            // tiles without entries are done (k_vis_bin_fill)
    uint32_t first;              // the job's first item in a multi-job work queue
    unsigned long long* work;    // W_COUNT work counters (counting variant of the tile kernel only)
    uint32_t bshift;             // depth buckets: 32 >> bshift
    uint32_t batch;              // entries per staged batch (1..kBatch)
    uint32_t drain;              // live pairs a warp collects before its lanes run their DDAs (1..32)
    uint32_t extra_tx;           // bytes the first batch's barrier expects that nobody copies: 0, or 64
                                 // under TGX_FLAG_TEST_LOST_COPY (its wait then runs out)
    uint32_t interleave;         // k_vis_tiles: spread the tiles without entries evenly over the launch
                                 // (outputs in host memory), instead of launching them last
};

// Shared memory of a tile CTA (dynamic, tile_smem_bytes(threads)):
//   the mbarrier of the copies and a gather count;
//   the staged batch: up to kBatch of the tile's 96-byte entries;
//   every pixel's best packed word so far (the pair lanes' atomicMin target);
//   per warp, a ring of kQueue live (pixel, entry) pairs waiting for a lane:
//   the pixel's cluster-space direction and reciprocals and the packed
//   lane | entry << 5 | sure_hit << 13.
constexpr uint32_t kBatch = 48;                      // entries per staged batch
constexpr uint32_t kQueue = 64;                      // ring entries per warp (an entry adds at most 32)
constexpr uint32_t kWarpRays = 7 * kQueue;           // then the bounds of the warp's rays (warp_rays): 6 floats
constexpr uint32_t kQueueWords = kWarpRays + 8;      // the ring: 6 float arrays + the packed word
constexpr uint32_t kSmBar = 0, kSmN = 12, kSmLost = 16, kSmBars = 24;   // kSmLost: two words; kSmBars: kStages - 1 more mbarriers
constexpr uint32_t kSmStage = 128;                   // 16-byte aligned copy target
constexpr uint32_t kStages = 2;                      // stages of a tile with several groups of threads (vis_tile_groups)
// With several groups of threads a batch is up to four times as large: a group walks
// every kGroups-th entry, and the chain of a heavy tile is its batches (8x8 tiles at
// 480x270, 512 objects, 8 groups: 62 us with batches of 48, 49 with 192, 48 with 384;
// 16x16, 4 groups: 153 and 103; 2 groups gain 3 % from 96 and lose from 192).
__host__ __device__ constexpr uint32_t batch_factor(uint32_t groups) { return groups < 4u ? groups : 4u; }
static_assert(kBatch * 4u <= 256u, "an entry's index is 8 bits of a ring entry's packed word");
__host__ __device__ constexpr uint32_t tile_best_off(uint32_t groups)
{
    return kSmStage + (groups > 1u ? kStages : 1u) * batch_factor(groups) * kBatch * (uint32_t)sizeof(TileEntry);
}
__host__ __device__ constexpr uint32_t tile_smem_bytes(uint32_t pixels, uint32_t groups = 1u)
{
    return tile_best_off(groups) + 8u * pixels + (pixels * groups / 32u) * kQueueWords * 4u;
}

struct TileSm
{
    unsigned char* p;
    uint32_t best_off, pixels;
    __device__ __forceinline__ uint32_t bar() const { return smem_addr(p + kSmBar); }
    // mbarrier of stage i (stage 0's is that of the single-stage tiles)
    __device__ __forceinline__ uint32_t bar(uint32_t i) const { return smem_addr(p + (i ? kSmBars + 8u * (i - 1u) : kSmBar)); }
    // whether a wait of batch j ran out: batches take turns with two words, as a warp may be on the
    // next batch while another one reads this one's
    __device__ __forceinline__ volatile uint32_t& lost(uint32_t j) const { return *(volatile uint32_t*)(p + kSmLost + 4u * (j & 1u)); }
    __device__ __forceinline__ uint32_t& n() const { return *(uint32_t*)(p + kSmN); }
    __device__ __forceinline__ TileEntry* stage() const { return (TileEntry*)(p + kSmStage); }
    __device__ __forceinline__ unsigned long long* best() const { return (unsigned long long*)(p + best_off); }
    __device__ __forceinline__ uint32_t* queue(uint32_t warp) const
    {
        return (uint32_t*)(p + best_off + 8u * pixels) + warp * kQueueWords;
    }
};

template <uint32_t kGroups = 1>
__device__ __forceinline__ TileSm tile_sm()
{
    extern __shared__ __align__(128) unsigned char tile_dyn_smem[];
    return TileSm{tile_dyn_smem, tile_best_off(kGroups), blockDim.x / kGroups};
}

__device__ __forceinline__ void tile_smem_init(const TileSm& sm)
{
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(sm.bar()), "r"(blockDim.x));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

__device__ __forceinline__ void copy16(uint32_t to, const char* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(to), "l"(from) : "memory");
}

// Entries first .. first + n - 1 of the job's bins gathered to dst, a thread per
// entry: its reference, then 32 bytes of the record and 64 of the bitmask.
// (Spreading an entry's six copies over lanes: 106.7 to 108.6 us against 106.5
// at 1080p, 512 objects.)  Every thread of the CTA arrives once on the mbarrier
// at bar when its own copies have landed; `extra` more bytes are expected under
// the lost-copy test.
__device__ __forceinline__ void stage_entries(const TileJob& J, uint32_t bar, const TileEntry* dst, uint32_t first, uint32_t n,
                                              uint32_t extra)
{
    for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
        const TileRef ref = J.refs[first + e];
        const char* rec = reinterpret_cast<const char*>(J.records + ref.record);
        const char* bits = reinterpret_cast<const char*>(J.bits + (uint64_t)ref.cluster_idx * 16u);
        const uint32_t to = smem_addr(dst + e);
#pragma unroll
        for (uint32_t q = 0; q < 2u; q++) copy16(to + 16u * q, rec + 16u * q);
#pragma unroll
        for (uint32_t q = 0; q < 4u; q++) copy16(to + 32u + 16u * q, bits + 16u * q);
    }
    if (extra && threadIdx.x == 0)
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(extra) : "memory");
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(bar) : "memory");
}
// this thread's copies have landed
__device__ __forceinline__ void own_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A thread's pixel of a tile: its place, its world ray, its nearest depth so
// far and the cluster-space direction of the last object it met.
struct TilePixel
{
    uint32_t px, py;
    bool valid;
    float dws[3];
    float far_plane, far_rcp;
    uint32_t best_d24, cur_obj;
    float dx, dy, dz, ix, iy, iz;
    uint32_t qh;                 // the warp's ring: first pending entry (warp-uniform)
};

__device__ __forceinline__ void tile_pixel(const ViewConst& vc, uint32_t place, uint32_t pix, TilePixel& P)
{
    tile_pixel_place(vc, place, pix, P.px, P.py);
    P.valid = P.px < vc.width && P.py < vc.height;
    P.far_plane = vc.far_plane;
    P.far_rcp = pow2_reciprocal(vc.far_plane);
    // pixel ray in world space (visibility.frag:29-33,68; mix per GLSL 8.3)
    const float fx = xdiv(xadd((float)P.px, 0.5f), (float)vc.width);
    const float fy = xsub(1.0f, xdiv(xadd((float)P.py, 0.5f), (float)vc.height));
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float a = xadd(xmul(vc.bl[i], xsub(1.0f, fy)), xmul(vc.tl[i], fy));
        const float b = xadd(xmul(vc.br[i], xsub(1.0f, fy)), xmul(vc.tr[i], fy));
        P.dws[i] = xadd(xmul(a, xsub(1.0f, fx)), xmul(b, fx));
    }
    P.best_d24 = 0xffffffu;
    P.cur_obj = 0xffffffffu;
    P.dx = P.dy = P.dz = P.ix = P.iy = P.iz = 0.0f;
    P.qh = 0u;
}

// the warp's minimum and maximum, NaN when some lane holds one
__device__ __forceinline__ float warp_min(float x)
{
    float r;
    asm volatile("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float warp_max(float x)
{
    float r;
    asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// Bounds of the warp's world rays (its pixels inside the view) for warp_may_hit:
// per axis the middle and half the spread, the latter widened by 1e-5 of itself
// and 2e-6 of the middle; NaN when some ray is.
__device__ __forceinline__ void warp_rays(const TilePixel& P, float* __restrict__ bounds)
{
    const float inf = __int_as_float(0x7f800000);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float lo = warp_min(P.valid ? P.dws[i] : inf), hi = warp_max(P.valid ? P.dws[i] : -inf);
        const float mid = 0.5f * (lo + hi);
        if ((threadIdx.x & 31u) == 0u) {
            bounds[i] = mid;
            bounds[4 + i] = 0.5f * (hi - lo) * 1.00001f + 2e-6f * fabsf(mid);
        }
    }
    __syncwarp();
}

// Whether some ray of the warp can meet entry E's cube, one entry per lane: false
// only when the exact test surely fails for each of them.  The rays' directions
// in cluster space lie in m +- h per axis.  A line along u misses the cube of
// half edge 4 around c (from its origin) when for two axes j, k
// |u_j c_k - u_k c_j| > 4 (|u_j| + |u_k|); here the left side is taken at m and
// what it can lose over the spread is added on the right.  The margins: 2e-6 of
// the summed magnitudes on each direction (three products, two sums and a
// normalisation round by less than 3e-7), 1e-5 on the cube and its distance
// (the exact test's quotients differ from the real ones by less than 3e-7).
// NaN fails the comparison, hence keeps the entry; so do directions whose
// squares could underflow or overflow in the normalisation.
__device__ __forceinline__ bool warp_may_hit(const TileEntry& E, const float* __restrict__ bounds, const float* __restrict__ inv_rot)
{
    const float* L = inv_rot + 9u * E.rec.object_idx;
    const float mx = bounds[0], my = bounds[1], mz = bounds[2];
    const float hx = bounds[4], hy = bounds[5], hz = bounds[6];
    float u[3], s[3], c[3], a[3];
    const float4 oc = *reinterpret_cast<const float4*>(&E.rec.ox);
    const float o[3] = {oc.x, oc.y, oc.z};
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float l0 = L[3 * i], l1 = L[3 * i + 1], l2 = L[3 * i + 2];
        u[i] = __fmaf_rn(l0, mx, __fmaf_rn(l1, my, l2 * mz));
        s[i] = __fmaf_rn(fabsf(l0), hx, __fmaf_rn(fabsf(l1), hy, fabsf(l2) * hz));
        c[i] = 4.0f - o[i];
        a[i] = __fmaf_rn(1e-5f, fabsf(c[i]), 4.001f);
    }
    bool miss = false;
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int k = (j + 1) % 3;
        const float d = __fmaf_rn(u[j], c[k], -(u[k] * c[j]));
        // the spread's share, and the cube's (with its margin) at the largest |u|
        const float r = __fmaf_rn(s[j], fabsf(c[k]) + a[k], s[k] * (fabsf(c[j]) + a[j])) +
                        __fmaf_rn(fabsf(u[j]), a[k], fabsf(u[k]) * a[j]);
        miss |= fabsf(d) > r;
    }
    const float low = fmaxf(fmaxf(fabsf(u[0]), fabsf(u[1])), fabsf(u[2]));
    return !miss || !(low > 1e-15f && low + fmaxf(fmaxf(s[0], s[1]), s[2]) < 1e15f);
}

// Entries k0, k0 + kStep, ... of a staged batch of n.  First a lane looks at one
// entry each for the whole warp: entries that no pixel of the warp can take (its
// farthest word is nearer than the entry's depth bound, or no ray can meet its
// cube, warp_may_hit) are dropped 32 at a time.  The others every lane walks
// for its own pixel, nearest first (the depth skip, the cluster-space direction
// once per object, the conservative slab test); the pairs that survive are compacted by
// warp ballot into the warp's ring q; whenever it holds J.drain, all 32 lanes
// take one pair each and run the exact entry test and the voxel DDA (vis_pair),
// folding the result into the pixel's word (best: the warp's first pixel's)
// with a shared-memory atomicMin.  The ring is drained at the end.
//
// The tile kernel is bound by instruction issue (72 % of the slots at 1080p, 32
// warps per SM).  512 objects at 1920x1080, 8x8 tiles: 145 us and 124 M warp
// instructions with every entry walked by every warp; 126 us and 105 M with the
// look ahead (it leaves about half of the walks); 103 us with the divisions,
// conversions and branches of vis_pair reduced; 90 us with the entries of a look
// ahead walked nearest first (a bucket, an octave of depth, holds them in any
// order: 2.8 M pairs evaluated before, 2.0 M now); 88 with the first pairs
// evaluated early.
template <bool kCount, uint32_t kStep>
__device__ __forceinline__ void tile_batch(const TileJob& J, const TileEntry* const E, uint32_t k0, const uint32_t n, TilePixel& P,
                                           uint32_t* const q, unsigned long long* const best, uint32_t* work)
{
    const uint32_t lane = threadIdx.x & 31u;
    // half as many as long as some pixel has no word: the first ones rule out the most
    uint32_t drain = J.drain;
    float* const qf = (float*)q;
    uint32_t qn = 0;           // pending entries (warp-uniform)
    uint32_t todo = 0;         // of the 32 entries before `next`, those to walk (warp-uniform)
    uint32_t lb = 0;           // depth bound of the lane's entry among them
    for (uint32_t next = k0;;) {
        if (todo == 0u && next < n) {
            const uint32_t farthest = __reduce_max_sync(0xffffffffu, P.valid ? P.best_d24 : 0u);
            drain = farthest == 0xffffffu ? (J.drain + 1u) >> 1 : J.drain;
            const uint32_t e = next + kStep * lane;
            bool keep = e < n;
            if (keep) {
                lb = E[e].rec.d24_lb;
                keep = farthest >= lb && warp_may_hit(E[e], qf + kWarpRays, J.inv_rot);
            }
            todo = __ballot_sync(0xffffffffu, keep);
            if (kCount && P.valid) {
                for (uint32_t i = 0, k = next; i < 32u && k < n; i++, k += kStep)
                    if (!((todo >> i) & 1u)) {
                        if (P.best_d24 < E[k].rec.d24_lb) work[W_DEPTH_SKIPS]++;
                        else { work[W_PAIRS]++; work[W_SLAB_MISSES]++; }
                    }
            }
            next += 32u * kStep;
        }
        if (todo) {
            // the nearest of them: the entries of a bucket come in no order
            const uint32_t j = __reduce_min_sync(0xffffffffu, (todo >> lane) & 1u ? lb << 5 | lane : 0xffffffffu) & 31u;
            const uint32_t k = next - kStep * (32u - j);
            todo &= ~(1u << j);
            bool live = false, sure = false;
            const uint2 ol = *reinterpret_cast<const uint2*>(&E[k].rec.object_idx);   // object, depth bound
            if (P.valid) {
                if (P.best_d24 < ol.y) {   // cannot produce a smaller word
                    if (kCount) work[W_DEPTH_SKIPS]++;
                } else {
                    if (kCount) work[W_PAIRS]++;
                    if (ol.x != P.cur_obj) {
                        // normalize((ws2ms * v4(dir, 0)).xyz) (visibility.frag:69) with the
                        // object's shared linear part (see k_object_setup)
                        if (kCount) work[W_DIR_SETUPS]++;
                        P.cur_obj = ol.x;
                        const float* L = J.inv_rot + 9u * ol.x;
                        const float ux = xadd(xadd(xmul(P.dws[0], L[0]), xmul(P.dws[1], L[1])), xmul(P.dws[2], L[2]));
                        const float uy = xadd(xadd(xmul(P.dws[0], L[3]), xmul(P.dws[1], L[4])), xmul(P.dws[2], L[5]));
                        const float uz = xadd(xadd(xmul(P.dws[0], L[6]), xmul(P.dws[1], L[7])), xmul(P.dws[2], L[8]));
                        const float mag = xsqrt(xadd(xadd(xmul(ux, ux), xmul(uy, uy)), xmul(uz, uz)));
                        P.dx = xdiv(ux, mag); P.dy = xdiv(uy, mag); P.dz = xdiv(uz, mag);
                        const float nan = __int_as_float(0x7fffffff);
                        P.ix = P.dx != 0.0f ? __frcp_rn(P.dx) : nan;
                        P.iy = P.dy != 0.0f ? __frcp_rn(P.dy) : nan;
                        P.iz = P.dz != 0.0f ? __frcp_rn(P.dz) : nan;
                    }
                    const float4 o = *reinterpret_cast<const float4*>(&E[k].rec.ox);
                    const int sc = slab_class(o.x, o.y, o.z, P.ix, P.iy, P.iz);
                    live = sc != kMiss;
                    sure = sc == kHit;
                    if (kCount) work[sc == kMiss ? W_SLAB_MISSES : sc == kHit ? W_SURE_HITS : W_EXACT_TESTS]++;
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, live);
            if (live) {
                const uint32_t e = (P.qh + qn + __popc(m & ((1u << lane) - 1u))) & (kQueue - 1u);
                qf[0 * kQueue + e] = P.dx; qf[1 * kQueue + e] = P.dy; qf[2 * kQueue + e] = P.dz;
                qf[3 * kQueue + e] = P.ix; qf[4 * kQueue + e] = P.iy; qf[5 * kQueue + e] = P.iz;
                q[6 * kQueue + e] = lane | (k << 5) | ((uint32_t)sure << 13);
            }
            qn += __popc(m);
        }
        if (qn < drain && (todo || next < n)) continue;
        if (qn == 0u) break;   // nothing to walk and nothing pending
        // one pair per lane: the exact test and the DDA; the word goes to its pixel
        const uint32_t take = min(qn, 32u);
        __syncwarp();
        if (lane < take) {
            const uint32_t e = (P.qh + lane) & (kQueue - 1u);
            const uint32_t pk = q[6 * kQueue + e];
            const TileEntry& te = E[(pk >> 5) & 255u];
            const float4 o = *reinterpret_cast<const float4*>(&te.rec.ox);
            const unsigned long long w = vis_pair<kCount>(
                o.x, o.y, o.z, qf[0 * kQueue + e], qf[1 * kQueue + e], qf[2 * kQueue + e],
                qf[3 * kQueue + e], qf[4 * kQueue + e], qf[5 * kQueue + e], (pk >> 13) != 0u, te.bits,
                te.rec.cluster_pointer, P.far_plane, P.far_rcp, &J.counters[C_DDA_OVERRUN], work);
            // the minimum of 64 bits is a compare-and-swap loop: only where it can lower the word
            unsigned long long* const word = best + (pk & 31u);
            if (w < *(volatile unsigned long long*)word) atomicMin(word, w);
        }
        P.qh = (P.qh + take) & (kQueue - 1u);
        qn -= take;
        __syncwarp();
        P.best_d24 = min(P.best_d24, (uint32_t)(best[lane] >> 40));
        if (!kCount && todo) {   // entries that the words found so far rule out
            const uint32_t farthest = __reduce_max_sync(0xffffffffu, P.valid ? P.best_d24 : 0u);
            todo &= __ballot_sync(0xffffffffu, farthest >= lb);
            drain = farthest == 0xffffffu ? (J.drain + 1u) >> 1 : J.drain;
        }
    }
}

// the index of a slot's tile among all views' (what an error names)
__device__ __forceinline__ uint32_t tile_index(const ViewConst& vc, uint32_t place)
{
    return vc.tile_base + (place >> 16) * vc.tiles_x + (place & 0xffffu);
}

// A tile without entries: only cleared (no ray set-up, no barrier), unless it is already.
__device__ __forceinline__ void clear_tile(const TileJob& J, const uint4& si, uint32_t pix)
{
    if (J.cleared) return;
    const ViewConst& vc = J.views[si.x];
    uint32_t px, py;
    tile_pixel_place(vc, si.w, pix, px, py);
    if (px < vc.width && py < vc.height) J.outs[si.x][(size_t)py * vc.width + px] = ULLONG_MAX;
}

// Of records base .. base + m - 1, those of the view whose tile rectangle holds
// tile (tx, ty), copied into the stage (count in sm.n()).  All threads of the CTA.
__device__ __forceinline__ void gather_records(const TileJob& J, uint32_t base, uint32_t m, uint32_t view, uint32_t tx,
                                               uint32_t ty, const TileSm& sm)
{
    for (uint32_t k = threadIdx.x; k < m; k += blockDim.x) {
        const uint32_t r = base + k;
        const uint2 qr = J.rects[r];
        const uint2 q1 = make_uint2(qr.y & 0xffffu, (qr.y & ~kListed) >> 16);
        if (J.records[r].view == view && tx >= (qr.x & 0xffffu) && tx <= q1.x && ty >= (qr.x >> 16) && ty <= q1.y) {
            TileEntry& te = sm.stage()[atomicAdd(&sm.n(), 1u)];
            te.rec = J.records[r];
#pragma unroll
            for (int w = 0; w < 16; w++) te.bits[w] = J.bits[(uint64_t)te.rec.cluster_idx * 16u + w];
        }
    }
}

// Tile `slot` (in the job's heavy-first order) of one job: every pixel's
// nearest packed word over the entries binned to the tile.  `phase` is the
// parity of the mbarrier that the CTA's copies arrive on, carried across tiles.
// Returns false (the same in every thread) when a batch's copies did not complete
// in time: the status word then holds TGX_ERR_TIMEOUT, the CTA has issued no
// further copy, every thread's own have landed and it has written its pixels'
// words so far; it must not stage another tile.  With kNoCopies the entries are
// gathered without the mbarrier, as after an overflow.
//
// The tile's entries (sorted near to far by depth bucket) arrive kBatch at a
// time (stage_entries); the first copies are issued before the pixels' rays are
// set up, so the two overlap.  Per batch every lane walks the entries for its own pixel: the
// depth skip, the cluster-space direction (once per object), and the
// conservative slab test.  The pairs that survive are compacted by warp
// ballot into the warp's ring; whenever it holds 32, all 32 lanes take one
// pair each and run the exact entry test and the voxel DDA (vis_pair),
// folding the result into the pixel's word with a shared-memory atomicMin.
// The ring is drained at the end of each batch.  The minimum over a pixel's
// pairs does not depend on the order they are evaluated in (every word is
// distinct), so the buffer is the same bits as one DDA per pair in order.
template <bool kCount = false, bool kNoCopies = false>
__device__ __forceinline__ bool vis_tile(const TileJob& J, uint32_t slot, const TileSm& sm, uint32_t& phase,
                                         tgx_dev_status* __restrict__ status)
{
    uint32_t work[W_COUNT];
    if (kCount) {
#pragma unroll
        for (int i = 0; i < W_COUNT; i++) work[i] = 0u;
    }
    __syncthreads();   // the CTA's previous tile is done with the shared state
    const uint4 si = J.slot_info[slot];   // one load: the tile and its entry range
    // bins overflowed this frame: gather every record whose tile rectangle holds the tile (slow, exact)
    const bool scan_all = kNoCopies || J.counters[C_OVERFLOW] != 0u;
    const uint32_t begin = scan_all ? 0u : si.y;
    const uint32_t end = scan_all ? J.counters[C_RECORDS] : si.y + si.z;
    if (si.z == 0u) {   // the same in every thread
        clear_tile(J, si, threadIdx.x);
        return true;
    }
    const TileEntry* const E = sm.stage();
    if (!scan_all) stage_entries(J, sm.bar(), E, begin, min(J.batch, end - begin), J.extra_tx);
    sm.best()[threadIdx.x] = ULLONG_MAX;   // read by the thread's own warp, after warp_rays' barrier
    const uint32_t view = si.x;
    const ViewConst& vc = J.views[view];
    TilePixel P;
    tile_pixel(vc, si.w, threadIdx.x, P);
    const uint32_t tx = si.w & 0xffffu, ty = si.w >> 16;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t* const q = sm.queue(warp);
    unsigned long long* const best0 = sm.best() + (warp << 5);
    warp_rays(P, (float*)q + kWarpRays);

    bool lost = false;      // a wait for a batch's copy ran out (the same in every lane of a warp)
    for (uint32_t base = begin; base < end;) {
        uint32_t n;
        if (!scan_all) {
            n = min(J.batch, end - base);
            if (base != begin) {
                // the previous batch is fully consumed; after a lost copy nobody stages another
                if (__syncthreads_or(lost)) break;
                stage_entries(J, sm.bar(), E, base, n, 0u);
            }
            base += n;
            lost = __any_sync(0xffffffffu, !mbar_wait_bounded(sm.bar(), phase));
            phase ^= 1u;
            if (lost) continue;
        } else {
            // keep the records of this view whose tile rectangle holds this tile, copied into the stage
            __syncthreads();
            if (threadIdx.x == 0) sm.n() = 0;
            __syncthreads();
            const uint32_t m = min(J.batch, end - base);
            gather_records(J, base, m, view, tx, ty, sm);
            base += m;
            __syncthreads();
            n = sm.n();
            if (n == 0) continue;
        }
        if (kCount && P.valid) work[W_BATCHES]++;
        tile_batch<kCount, 1>(J, E, 0u, n, P, q, best0, work);
        // every pixel already nearer than the rest of the (bucket-sorted) entries: the tile is done
        if (!scan_all && base < end) {
            const uint32_t lo = bucket_lo(depth_bucket(E[n - 1].rec.d24_lb, J.bshift), J.bshift);
            if (__syncthreads_and(!P.valid || P.best_d24 < lo)) break;
        }
    }
    const unsigned long long best = sm.best()[threadIdx.x];
    if (__syncthreads_or(lost)) {
        // a batch's copies did not complete: report it, let this thread's own
        // land before the CTA is gone, and write the words found so far
        if (threadIdx.x == 0) dev_error(status, TGX_ERR_TIMEOUT, 5, tile_index(vc, si.w));
        own_copies_wait();
        if (P.valid) J.outs[view][(size_t)P.py * vc.width + P.px] = best;
        return false;
    }
    if (P.valid) J.outs[view][(size_t)P.py * vc.width + P.px] = best;
    if (kCount) {
        // per warp: sum the lanes' counters, one 64-bit atomic each
#pragma unroll
        for (int i = 0; i < W_COUNT; i++) {
            unsigned long long v = work[i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0u && v) atomicAdd(&J.work[i], v);
        }
    }
    return true;
}

// A tile with kGroups threads per pixel: group g of the CTA's threads covers all
// of the tile's pixels and takes entries g, g + kGroups, ... of every batch, all
// folding into the pixels' one set of words.  A frame whose tiles do not fill
// the GPU takes as long as its heaviest tile, a chain of dependent batches;
// more warps per tile shorten that chain.  Batches alternate between two stages,
// each refilled as soon as its batch is consumed.  The words are the same bits:
// the minimum does not depend on which group finds it.  One tile per CTA: the
// mbarriers' phases start at zero.
template <uint32_t kGroups>
__device__ __forceinline__ void vis_tile_groups(const TileJob& J, uint32_t slot, const TileSm& sm,
                                                tgx_dev_status* __restrict__ status)
{
    const uint32_t n_pix = blockDim.x / kGroups;
    const uint32_t grp = threadIdx.x / n_pix, pix = threadIdx.x - grp * n_pix;
    const uint4 si = J.slot_info[slot];
    // bins overflowed this frame: gather every record whose tile rectangle holds the tile (slow, exact)
    const bool scan_all = J.counters[C_OVERFLOW] != 0u;
    if (si.z == 0u) {
        if (grp == 0u) clear_tile(J, si, pix);
        return;
    }
    const uint32_t batch = J.batch * batch_factor(kGroups);
    const uint32_t n_batches = scan_all ? 0u : (si.z + batch - 1u) / batch;
    auto stage_of = [&](uint32_t j) { return sm.stage() + (j % kStages) * kBatch * batch_factor(kGroups); };
    auto stage = [&](uint32_t j) {   // batch j, in order
        const uint32_t first = j * batch;
        stage_entries(J, sm.bar(j % kStages), stage_of(j), si.y + first, min(batch, si.z - first), j == 0u ? J.extra_tx : 0u);
    };
    for (uint32_t j = 0; j < min(n_batches, kStages); j++) stage(j);
    if (threadIdx.x < 2u) sm.lost(threadIdx.x) = 0u;
    if (grp == 0u) sm.best()[pix] = ULLONG_MAX;
    __syncthreads();
    const uint32_t view = si.x;
    const ViewConst& vc = J.views[view];
    TilePixel P;
    tile_pixel(vc, si.w, pix, P);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t* const q = sm.queue(threadIdx.x >> 5);
    unsigned long long* const best0 = sm.best() + (pix & ~31u);
    warp_rays(P, (float*)q + kWarpRays);
    uint32_t j = 0;
    bool lost = false;
    while (j < n_batches) {
        const uint32_t n = min(batch, si.z - j * batch);
        const TileEntry* const E = stage_of(j);
        const bool late = __any_sync(0xffffffffu, !mbar_wait_bounded(sm.bar(j % kStages), (j / kStages) & 1u));
        uint32_t lo = 0u;
        if (late) {
            if (lane == 0) sm.lost(j) = 1u;
        } else {
            P.best_d24 = min(P.best_d24, (uint32_t)(best0[lane] >> 40));   // the other groups' words too
            tile_batch<false, kGroups>(J, E, grp, n, P, q, best0, nullptr);
            lo = bucket_lo(depth_bucket(E[n - 1].rec.d24_lb, J.bshift), J.bshift);
        }
        // the batch is consumed; every pixel already nearer than the rest of the (bucket-sorted) entries: done
        const bool done = __syncthreads_and(!P.valid || P.best_d24 < lo);
        lost = sm.lost(j) != 0u;
        j++;
        if (done || lost) break;
        if (j + kStages - 1u < n_batches) stage(j + kStages - 1u);
    }
    own_copies_wait();   // none may land after the CTA is gone
    if (threadIdx.x == 0 && lost) dev_error(status, TGX_ERR_TIMEOUT, 5, tile_index(vc, si.w));
    if (scan_all) {
        const uint32_t tx = si.w & 0xffffu, ty = si.w >> 16;
        const uint32_t n_rec = J.counters[C_RECORDS];
        for (uint32_t base = 0; base < n_rec; base += J.batch) {
            __syncthreads();
            if (threadIdx.x == 0) sm.n() = 0;
            __syncthreads();
            gather_records(J, base, min(J.batch, n_rec - base), view, tx, ty, sm);
            __syncthreads();
            tile_batch<false, kGroups>(J, sm.stage(), grp, sm.n(), P, q, best0, nullptr);
        }
    }
    __syncthreads();
    if (P.valid && grp == 0u) J.outs[view][(size_t)P.py * vc.width + P.px] = sm.best()[pix];
}

// The slot (heavy-first order, the tiles without entries last) that CTA b of
// t takes.  With interleave (outputs in host memory), the n non-empty tiles keep
// their order but the e = t - n empty ones are spread over the first f = 3/2 e
// CTAs, two of three: there the heavy tiles write little, and at the end the
// light ones fill the link by themselves.  Among the first f, CTA b is the
// c(b)-th non-empty one when c(b + 1) > c(b), with c(b) = floor(b (f - e) / f),
// else the (b - c(b))-th empty one.  Both maps are bijections of [0, t).  Frame of
// 512 objects at 1920x1080 to pinned memory: 148.1 us with the empty tiles
// spread over the whole launch, 145.2 at 2 of 3 (or 3 of 5), 148.4 at 4 of 5,
// 163 with all of them first.
__device__ __forceinline__ uint32_t tile_slot(uint32_t b, uint32_t t, uint32_t n, bool interleave)
{
    if (!interleave || n >= t) return b;
    const uint32_t e = t - n, f = (uint32_t)min((uint64_t)t, (uint64_t)e * 3u / 2u);
    if (b >= f) return b - e;
    const uint32_t c0 = (uint32_t)((uint64_t)b * (f - e) / f), c1 = (uint32_t)((uint64_t)(b + 1) * (f - e) / f);
    return c1 > c0 ? c0 : n + (b - c0);
}

// The totals the host sizes the next frame by, written while the frame's first tile starts.
__device__ __forceinline__ void publish_totals(const TileJob& J)
{
    if (blockIdx.x == 0 && threadIdx.x == 0 && J.host_counters) {
        J.host_counters[C_ENTRIES] = J.counters[C_ENTRIES];
        J.host_counters[C_OVERFLOW] = J.counters[C_OVERFLOW];
    }
}

// One CTA per tile of one job.  Instantiated per block size (= tile pixels) so the
// register budget can be bounded for the occupancy each size needs.
template <int kThreads, int kMinBlocks, bool kCount = false>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_vis_tiles(TileJob J, tgx_dev_status* __restrict__ status)
{
    const TileSm sm = tile_sm();
    tile_smem_init(sm);
    pdl_wait();
    publish_totals(J);
    uint32_t phase = 0;
    const uint32_t slot = J.interleave ? tile_slot(blockIdx.x, J.n_tiles, J.counters[C_NONEMPTY], true) : blockIdx.x;
    vis_tile<kCount>(J, slot, sm, phase, status);
}

// kGroups threads per pixel: kThreads = kGroups * the tile's pixels.
template <int kThreads, uint32_t kGroups>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) k_vis_tiles_groups(TileJob J, tgx_dev_status* __restrict__ status)
{
    const TileSm sm = tile_sm<kGroups>();
    tile_smem_init(sm);
    if (threadIdx.x == 0) {
#pragma unroll
        for (uint32_t i = 1; i < kStages; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(sm.bar(i)), "r"(blockDim.x));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_wait();
    publish_totals(J);
    __syncthreads();   // every thread arrives on the mbarriers
    const uint32_t slot = J.interleave ? tile_slot(blockIdx.x, J.n_tiles, J.counters[C_NONEMPTY], true) : blockIdx.x;
    vis_tile_groups<kGroups>(J, slot, sm, status);
}

// A CTA of the queue that lost a batch's copies still has the item that it drew
// meanwhile (thread 0's), which no other one takes: it renders that one without
// copies, and draws no more.  A function of its own: within the loop it took 1.4 %
// of a batch of 20 views (registers).
__device__ __noinline__ void vis_queue_last(const TileJob* jobs, uint32_t n_jobs, uint32_t total, uint32_t item, TileJob* job,
                                            uint32_t* slot, tgx_dev_status* status)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        *slot = 0xffffffffu;
        if (item < total) {
            uint32_t k = 0;   // the last job whose first item is <= item
            while (k + 1u < n_jobs && jobs[k + 1u].first <= item) k++;
            *job = jobs[k];
            if (item - job->first < job->counters[C_NONEMPTY]) *slot = item - job->first;
        }
    }
    __syncthreads();
    uint32_t phase = 0;
    if (*slot != 0xffffffffu) vis_tile<false, true>(*job, *slot, tile_sm(), phase, status);
}

// Persistent form over several jobs (scenes, each with its views): CTAs take
// tiles from one work queue in job order, each job's tiles heavy-first and those
// without entries passed over, until all jobs' tiles are done.  One thread per pixel
// whatever the jobs' sizes: several (vis_groups) are for the launches of a single
// frame or job, so small views of several jobs take as long as their heaviest tile.
template <int kThreads, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) k_vis_tiles_queue(const TileJob* __restrict__ jobs,
                                                                          uint32_t n_jobs, uint32_t total,
                                                                          uint32_t* __restrict__ queue,
                                                                          tgx_dev_status* __restrict__ status)
{
    const TileSm sm = tile_sm();
    __shared__ TileJob s_job;
    __shared__ uint32_t s_slot;
    tile_smem_init(sm);
    uint32_t phase = 0;
    // thread 0: the next item, drawn while the tile before it runs; the current job and its tiles with entries
    uint32_t item = threadIdx.x == 0 ? atomicAdd(queue, 1u) : 0u, job = 0xffffffffu, with_entries = 0;
    for (;;) {
        __syncthreads();   // the previous tile is done with s_job
        if (threadIdx.x == 0) {
            s_slot = 0xffffffffu;
            while (item < total) {
                uint32_t lo = 0, hi = n_jobs - 1;   // the last job whose first item is <= item
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1) >> 1;
                    if (jobs[mid].first <= item) lo = mid; else hi = mid - 1;
                }
                if (lo != job) {
                    job = lo;
                    s_job = jobs[lo];
                    with_entries = s_job.counters[C_NONEMPTY];
                }
                const uint32_t slot = item - s_job.first;
                // the job's other tiles are cleared: on to the next job's
                if (slot >= with_entries) atomicMax(queue, s_job.first + s_job.n_tiles);
                item = atomicAdd(queue, 1u);
                if (slot < with_entries) {
                    s_slot = slot;
                    break;
                }
            }
        }
        __syncthreads();
        if (s_slot == 0xffffffffu) return;
        if (!vis_tile(s_job, s_slot, sm, phase, status)) break;   // its staging barrier is not reusable
    }
    vis_queue_last(jobs, n_jobs, total, item, &s_job, &s_slot, status);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static void make_view_const(const tgx_view& v, uint32_t tile_w, uint32_t tile_h, uint32_t tile_base, ViewConst& c)
{
    memset(&c, 0, sizeof(c));
    for (int i = 0; i < 3; i++) {
        c.cam[i] = v.camera[i];
        c.bl[i] = v.ray_bl[i]; c.br[i] = v.ray_br[i]; c.tr[i] = v.ray_tr[i]; c.tl[i] = v.ray_tl[i];
    }
    c.far_plane = v.far_plane;
    c.width = v.width;
    c.height = v.height;
    c.tile_w = tile_w;
    c.tile_h = tile_h;
    c.tile_w_rcp = ((1u << 20) + tile_w - 1) / tile_w;
    c.tiles_x = (v.width + tile_w - 1) / tile_w;
    c.tiles_y = (v.height + tile_h - 1) / tile_h;
    c.tile_base = tile_base;
    // affine corner-ray model d(fx, fy) = bl + fx (br - bl) + fy (tl - bl):
    // p = s * d  <=>  (s, s fx, s fy) = B^-1 p with B = [bl | br-bl | tl-bl]
    double B[3][3];
    for (int i = 0; i < 3; i++) {
        B[i][0] = v.ray_bl[i];
        B[i][1] = (double)v.ray_br[i] - v.ray_bl[i];
        B[i][2] = (double)v.ray_tl[i] - v.ray_bl[i];
    }
    const double det = B[0][0] * (B[1][1] * B[2][2] - B[1][2] * B[2][1]) - B[0][1] * (B[1][0] * B[2][2] - B[1][2] * B[2][0]) +
                       B[0][2] * (B[1][0] * B[2][1] - B[1][1] * B[2][0]);
    const double inv[9] = {
        (B[1][1] * B[2][2] - B[1][2] * B[2][1]) / det, (B[0][2] * B[2][1] - B[0][1] * B[2][2]) / det,
        (B[0][1] * B[1][2] - B[0][2] * B[1][1]) / det, (B[1][2] * B[2][0] - B[1][0] * B[2][2]) / det,
        (B[0][0] * B[2][2] - B[0][2] * B[2][0]) / det, (B[0][2] * B[1][0] - B[0][0] * B[1][2]) / det,
        (B[1][0] * B[2][1] - B[1][1] * B[2][0]) / det, (B[0][1] * B[2][0] - B[0][0] * B[2][1]) / det,
        (B[0][0] * B[1][1] - B[0][1] * B[1][0]) / det};
    for (int i = 0; i < 9; i++) c.inv_basis[i] = (float)inv[i];
    double f[3], fl = 0.0;
    for (int i = 0; i < 3; i++) {
        f[i] = 0.25 * ((double)v.ray_bl[i] + v.ray_br[i] + v.ray_tr[i] + v.ray_tl[i]);
        fl += f[i] * f[i];
    }
    fl = sqrt(fl);
    for (int i = 0; i < 3; i++) c.fwd[i] = (float)(f[i] / fl);
    // side planes through the camera, spanned by adjacent corner rays, normals pointing inward
    const float* cr[4] = {v.ray_bl, v.ray_br, v.ray_tr, v.ray_tl};
    for (int k = 0; k < 4; k++) {
        const float* a = cr[k];
        const float* b = cr[(k + 1) % 4];
        double n[3] = {(double)a[1] * b[2] - (double)a[2] * b[1], (double)a[2] * b[0] - (double)a[0] * b[2],
                       (double)a[0] * b[1] - (double)a[1] * b[0]};
        const double sgn = n[0] * f[0] + n[1] * f[1] + n[2] * f[2] < 0 ? -1.0 : 1.0;
        const double l = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
        for (int i = 0; i < 3; i++) c.planes[3 * k + i] = (float)(sgn * n[i] / l);
    }
}

static tgx_status check_views(const tgx_view* views, uint32_t n_views, uint32_t tile_w, uint32_t tile_h)
{
    if (!views || n_views == 0 || n_views > 65535) { tgx_set_error("views: NULL or count %u out of range", n_views); return TGX_ERR_INVALID_ARGUMENT; }
    for (uint32_t i = 0; i < n_views; i++) {
        const tgx_view& v = views[i];
        if (v.width == 0 || v.height == 0 || (v.width + tile_w - 1) / tile_w > 4095 || (v.height + tile_h - 1) / tile_h > 4095) {
            tgx_set_error("view %u: size %ux%u out of range", i, v.width, v.height);
            return TGX_ERR_INVALID_ARGUMENT;
        }
        if (!(v.far_plane > 0.0f)) { tgx_set_error("view %u: far plane must be > 0", i); return TGX_ERR_INVALID_ARGUMENT; }
    }
    return TGX_OK;
}

// Scratch of one visibility frame (context buffers, or a frame graph's own).
struct VisScratch
{
    VisRecord* records;
    uint2* rects;
    uint32_t rec_cap;
    uint32_t* counters;
    uint32_t* next_counters = nullptr;   // cleared on the way, for the next frame (null: `counters` are cleared first)
    uint32_t* host_counters = nullptr;
    uint32_t* supers;          // directly before bucket_cnt: both start at zero
    uint32_t* bucket_cnt;
    uint32_t* tile_total;
    uint32_t* groups;
    uint32_t* tile_off;
    uint4* slot_info;
    TileRef* refs;
    uint32_t bin_capacity;     // references
    uint2* chunks;             // chunk list of the records of many tiles
    uint32_t chunk_cap;
};

// places of the chunk list: a frame lists about entries / kChunkTiles + (records of many tiles)
static uint32_t vis_chunk_cap(uint32_t n_tiles) { return std::max<uint32_t>(1u << 16, n_tiles); }

// bytes of the tile-sized part of the scratch
// (the bucket arrays are sized for the finest setting, kMaxBuckets per tile)
static size_t vis_tile_bytes(uint32_t n_tiles)
{
    return ((size_t)scan_supers(n_tiles) * kGroupWords + (size_t)n_tiles * (kMaxBuckets + 1) + (size_t)scan_groups(n_tiles) * kGroupWords) * 4 +
           8 + (size_t)vis_chunk_cap(n_tiles) * sizeof(uint2);
}

// bytes of the tile offsets (n_tiles + 1 words, padded to 16 bytes) and the slot records
static size_t vis_off_bytes(uint32_t n_tiles)
{
    return (size_t)((n_tiles + 4u) & ~3u) * 4 + (size_t)n_tiles * sizeof(uint4);
}

static void vis_carve_tiles(VisScratch& w, uint32_t* tile_cnt, uint32_t* tile_off, uint32_t n_tiles)
{
    w.supers = tile_cnt;
    w.bucket_cnt = w.supers + (size_t)scan_supers(n_tiles) * kGroupWords;
    w.tile_total = w.bucket_cnt + (size_t)n_tiles * kMaxBuckets;
    w.groups = w.tile_total + n_tiles;
    const size_t words = (size_t)(w.groups - tile_cnt) + (size_t)scan_groups(n_tiles) * kGroupWords;
    w.chunks = reinterpret_cast<uint2*>(tile_cnt + ((words + 1) & ~(size_t)1));
    w.chunk_cap = vis_chunk_cap(n_tiles);
    w.tile_off = tile_off;
    w.slot_info = reinterpret_cast<uint4*>(w.tile_off + ((n_tiles + 4u) & ~3u));
}

enum VisPhase { VIS_ALL = 0, VIS_TO_SCAN = 1, VIS_FROM_BINS = 2, VIS_NO_TILES = 3 };

static TileJob tile_job(const tgx_ctx* c, const tgx_scene* s, const ViewConst* d_vc, unsigned long long* const* d_outs,
                        uint32_t n_views, uint32_t n_tiles, const VisScratch& w)
{
    TileJob J;
    J.bshift = c->vis_bshift;
    J.batch = c->vis_batch;
    J.drain = c->vis_drain;
    J.records = w.records;
    J.rects = w.rects;
    J.refs = w.refs;
    J.slot_info = w.slot_info;
    J.views = d_vc;
    J.bits = s->d_bits;
    J.inv_rot = s->d_inv_rot;
    J.outs = d_outs;
    J.counters = w.counters;
    J.host_counters = w.host_counters;
    J.n_tiles = n_tiles;
    J.cleared = 1;
    J.first = 0;
    J.work = nullptr;
    J.extra_tx = 0;
    J.interleave = 0;
    return J;
}

// Threads per pixel of the tile launch: the largest power of two, up to 8 and
// 1024 threads a CTA, that keeps the launch within 12 (two) or 8 (four, eight)
// times 1024 threads per SM, as many as the kernels' 64 registers let run.  Below
// that the time is the heaviest tile's chain of batches, above it the sum of all
// tiles' work, which grows with the threads.  Tile kernel over the 512-object
// scene, 8x8 tiles, 1 / 2 / 4 / 8 threads per pixel, on 152 SMs: 480x270 130 / 72 /
// 50 / 49 us, 560x315 116 / 66 / 47 / 57, 640x480 80 / 51 / 50 / 75, 800x450 81 / 53 /
// 58 / 89, 1120x630 68 / 61 / 88 / 147, 1280x720 66 / 70 / 107 / 181, 1920x1080 88 /
// 123 / 200 / 360; 16x16 tiles, 1 / 2 / 4: 640x360 200 / 108 / 76, 800x450 155 / 84 /
// 88, 1280x720 100 / 97 / 151; 64 objects, 8x8: 640x360 31 / 22 / 18 / 21, 853x479
// 25 / 20 / 18 / 29.
// How far the heaviest tile stands out differs from frame to frame, so near a line
// either side can be the better one: at 1280x720 two threads lose 4 us in the frame
// above and win in others (whole frames, one / two threads: 512 objects, 8x8, two
// seeds 88 / 93 and 71 / 64, 16x16 120 / 117 and 90 / 76; 256 objects, 8x8 79 / 79.5
// and 49 / 47, 16x16 88 / 91 and 59 / 47; 64 objects, 8x8 37 / 33, 16x16 44 / 35).
// The entries of an earlier frame would not tell: it may be any other scene's.
static uint32_t vis_groups(const tgx_ctx* c, uint32_t pixels, uint32_t n_tiles)
{
    const uint64_t unit = 1024ull * (uint64_t)c->num_sms;
    uint32_t g = 1;
    while (g < 8u && pixels * g * 2u <= 1024u && (uint64_t)n_tiles * pixels * g * 2u <= (g == 1u ? 12u : 8u) * unit) g *= 2u;
    return g;
}

// The launches of one frame (n_views views of scene s, view table d_vc / d_outs
// on the device): all of them, or the part up to the tile scan, or the rest.
static tgx_status vis_launch(tgx_ctx* c, const tgx_scene* s, ViewConst* d_vc, unsigned long long** d_outs,
                             uint32_t n_views, uint32_t n_tiles, const VisScratch& w, int phase = VIS_ALL,
                             bool interleave = false, const InlineViews* views = nullptr)
{
    const uint64_t n_pairs = (uint64_t)s->n_cluster_pointers * n_views;
    const uint32_t n_scan_ctas = scan_groups(n_tiles);
    const uint32_t warp_grid = (uint32_t)c->num_sms * 8;
    const uint32_t bshift = c->vis_bshift;
    if (phase != VIS_FROM_BINS) {
        if (!w.next_counters) TGX_CUDA(cudaMemsetAsync(w.counters, 0, C_COUNT * sizeof(uint32_t), c->stream));
        const uint32_t setup_blocks = (uint32_t)((n_pairs + 255) / 256);
#define SETUP(type, inl)                                                                                               \
        TGX_LAUNCH_PDL(c, TR_VIS_SETUP, setup_blocks, 256, 0, (k_vis_cluster_setup<true, type>),                           \
                   s->d_objects, s->d_cluster_pointers, s->d_c2o, s->d_bits, s->d_cp_obj, s->n_cluster_pointers, inl,  \
                   d_vc, d_outs, n_views, w.records, w.rects, w.rec_cap, w.counters, w.supers,                         \
                   scan_supers(n_tiles) * kGroupWords + n_tiles * (kMaxBuckets >> bshift), w.chunks, w.chunk_cap, c->d_status)
        if (views) SETUP(InlineViews, *views);
        else SETUP(NoViews, NoViews{});
#undef SETUP
        // each pass is a programmatic dependent of the one before
        TGX_LAUNCH_PDL(c, TR_VIS_COUNT, warp_grid, 256, 0, k_vis_count, w.records, w.rects, w.counters, w.rec_cap,
                       s->d_objects, d_vc, w.bucket_cnt, n_tiles, bshift, w.chunks, w.chunk_cap);
#define PREFIX_ARGS w.bucket_cnt, w.tile_total, n_tiles, w.groups, w.supers
        if (bshift == 0) TGX_LAUNCH_PDL(c, TR_VIS_PREFIX, n_scan_ctas, kScanTiles, 0, k_vis_prefix<32>, PREFIX_ARGS);
        else if (bshift == 1) TGX_LAUNCH_PDL(c, TR_VIS_PREFIX, n_scan_ctas, kScanTiles, 0, k_vis_prefix<16>, PREFIX_ARGS);
        else TGX_LAUNCH_PDL(c, TR_VIS_PREFIX, n_scan_ctas, kScanTiles, 0, k_vis_prefix<8>, PREFIX_ARGS);
#undef PREFIX_ARGS
        TGX_LAUNCH_PDL(c, TR_VIS_SCAN, n_scan_ctas, kScanTiles, 0, k_vis_finalize, w.tile_total, n_tiles, w.groups, w.supers,
                       w.tile_off, w.slot_info, w.bin_capacity, w.counters, w.next_counters, d_vc, n_views);
    }
    if (phase == VIS_TO_SCAN) return TGX_OK;
    TGX_LAUNCH_PDL(c, TR_VIS_BIN, warp_grid, 256, 0, k_vis_bin_fill,
                   w.records, w.rects, w.counters, d_vc, w.tile_off, w.bucket_cnt, w.refs,
                   n_tiles, w.bin_capacity, bshift, w.chunks, w.chunk_cap, w.slot_info, d_outs, interleave ? 0u : 1u, c->d_status);
    if (phase == VIS_NO_TILES) return TGX_OK;
    TileJob J = tile_job(c, s, d_vc, d_outs, n_views, n_tiles, w);
    J.interleave = interleave ? 1u : 0u;
    J.cleared = interleave ? 0u : 1u;
    if (c->flags & TGX_FLAG_TEST_LOST_COPY) J.extra_tx = 64u;
    const uint32_t threads = c->tile_w * c->tile_h, smem = tile_smem_bytes(threads);
    if (c->vis_count_work) {
        // the counting variant (tgx_vis_count_work): same results, plus the work counters
        TGX_TRY(devbuf_reserve(c->vis_work, W_COUNT * sizeof(unsigned long long)));
        J.work = (unsigned long long*)c->vis_work.ptr;
        TGX_CUDA(cudaMemsetAsync(J.work, 0, W_COUNT * sizeof(unsigned long long), c->stream));
        if (threads == 64) TGX_LAUNCH(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<64, 16, true>), J, c->d_status);
        else if (threads == 128) TGX_LAUNCH(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<128, 10, true>), J, c->d_status);
        else if (threads == 256) TGX_LAUNCH(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<256, 5, true>), J, c->d_status);
        else TGX_LAUNCH(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<512, 2, true>), J, c->d_status);
        return TGX_OK;
    }
    // (the fallthrough: 1 thread per pixel, and the pixel counts that are no power of two from 64 to 512)
    const uint32_t groups = vis_groups(c, threads, n_tiles);
#define TILE_GROUPS(px, g)                                                                                      \
    if (threads == (px) && groups == (g)) {                                                                     \
        TGX_LAUNCH_PDL(c, TR_VIS_TILES, n_tiles, (px) * (g), tile_smem_bytes((px), (g)),                        \
                       (k_vis_tiles_groups<(px) * (g), (g)>), J, c->d_status);                                  \
        return TGX_OK;                                                                                          \
    }
    TILE_GROUPS(64, 2) TILE_GROUPS(64, 4) TILE_GROUPS(64, 8)
    TILE_GROUPS(128, 2) TILE_GROUPS(128, 4) TILE_GROUPS(128, 8)
    TILE_GROUPS(256, 2) TILE_GROUPS(256, 4)
    TILE_GROUPS(512, 2)
#undef TILE_GROUPS
    if (threads == 64) TGX_LAUNCH_PDL(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<64, 16>), J, c->d_status);
    else if (threads == 128) TGX_LAUNCH_PDL(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<128, 10>), J, c->d_status);
    else if (threads == 256) TGX_LAUNCH_PDL(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<256, 5>), J, c->d_status);
    else TGX_LAUNCH_PDL(c, TR_VIS_TILES, n_tiles, threads, smem, (k_vis_tiles<512, 2>), J, c->d_status);
    return TGX_OK;
}

// Once per context, with its device current: the persistent tile kernel's
// resident CTAs for the context's tile size (an occupancy query, so it is made
// outside any stream capture).
template <int kThreads, int kMinBlocks>
static uint32_t vis_queue_per_sm()
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_vis_tiles_queue<kThreads, kMinBlocks>, kThreads,
                                                      tile_smem_bytes(kThreads)) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    return (uint32_t)per_sm;
}

tgx_status vis_prepare_device(tgx_ctx* c)
{
    const uint32_t threads = c->tile_w * c->tile_h;
    const uint32_t per_sm = threads == 64 ? vis_queue_per_sm<64, 16>() : threads == 128 ? vis_queue_per_sm<128, 10>()
                          : threads == 256 ? vis_queue_per_sm<256, 5>() : vis_queue_per_sm<512, 2>();
    c->vis_tile_ctas = (uint32_t)c->num_sms * per_sm;
    // several threads per pixel take more dynamic shared memory than a launch gets by default
#define BIG_SMEM(px, g) \
    TGX_CUDA(cudaFuncSetAttribute(k_vis_tiles_groups<(px) * (g), (g)>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                  (int)tile_smem_bytes((px), (g))))
    BIG_SMEM(64, 2); BIG_SMEM(64, 4); BIG_SMEM(64, 8);
    BIG_SMEM(128, 2); BIG_SMEM(128, 4); BIG_SMEM(128, 8);
    BIG_SMEM(256, 2); BIG_SMEM(256, 4); BIG_SMEM(512, 2);
#undef BIG_SMEM
    return TGX_OK;
}

// The tile stage of several jobs as one persistent launch over a work queue
// (d_jobs: the jobs' TileJob records with their first queue items; d_queue
// zeroed here).
static tgx_status vis_launch_queue(tgx_ctx* c, const TileJob* d_jobs, uint32_t n_jobs, uint32_t total, uint32_t* d_queue)
{
    TGX_CUDA(cudaMemsetAsync(d_queue, 0, 4, c->stream));
    const uint32_t threads = c->tile_w * c->tile_h, smem = tile_smem_bytes(threads);
    const uint32_t grid = std::max(1u, std::min(c->vis_tile_ctas, total));
#define QUEUE_ARGS d_jobs, n_jobs, total, d_queue, c->d_status
    if (threads == 64) TGX_LAUNCH(c, TR_VIS_TILES, grid, threads, smem, (k_vis_tiles_queue<64, 16>), QUEUE_ARGS);
    else if (threads == 128) TGX_LAUNCH(c, TR_VIS_TILES, grid, threads, smem, (k_vis_tiles_queue<128, 10>), QUEUE_ARGS);
    else if (threads == 256) TGX_LAUNCH(c, TR_VIS_TILES, grid, threads, smem, (k_vis_tiles_queue<256, 5>), QUEUE_ARGS);
    else TGX_LAUNCH(c, TR_VIS_TILES, grid, threads, smem, (k_vis_tiles_queue<512, 2>), QUEUE_ARGS);
#undef QUEUE_ARGS
    return TGX_OK;
}

// host view table: ViewConst per view (tile bases) and the output pointer table
static std::vector<unsigned char> vis_view_table(tgx_ctx* c, const tgx_view* views, uint32_t n_views,
                                                 uint64_t* const* d_visbuf, uint32_t& n_tiles, size_t& ptr_off)
{
    std::vector<ViewConst> vcs(n_views);
    n_tiles = 0;
    for (uint32_t i = 0; i < n_views; i++) {
        make_view_const(views[i], c->tile_w, c->tile_h, n_tiles, vcs[i]);
        n_tiles += vcs[i].tiles_x * vcs[i].tiles_y;
    }
    const size_t vc_bytes = n_views * sizeof(ViewConst);
    ptr_off = (vc_bytes + 15) & ~(size_t)15;
    std::vector<unsigned char> stage(ptr_off + n_views * sizeof(void*));
    memcpy(stage.data(), vcs.data(), vc_bytes);
    memcpy(stage.data() + ptr_off, d_visbuf, n_views * sizeof(void*));
    return stage;
}

tgx_status vis_render_device(tgx_ctx* c, const tgx_scene* s, const tgx_view* views, uint32_t n_views,
                             uint64_t* const* d_visbuf, bool host_out)
{
    if (!c || !s || !d_visbuf) { tgx_set_error("tgx_vis_render: NULL argument"); return TGX_ERR_INVALID_ARGUMENT; }
    TGX_TRY(check_views(views, n_views, c->tile_w, c->tile_h));
    for (uint32_t i = 0; i < n_views; i++)
        if (!d_visbuf[i]) { tgx_set_error("tgx_vis_render: output %u is NULL", i); return TGX_ERR_INVALID_ARGUMENT; }
    TGX_CUDA(cudaSetDevice(c->device));

    // View constants and output pointers: up to kInlineViews go with the first
    // kernel as its argument, more are copied from pageable memory (staged by
    // the driver, no sync).  A small frame is a chain of short dependent kernels;
    // a copy or a memset in it costs as much as one of them (256x256 frame of a
    // small scene 37.3 us with a copy, a memset and the counters' copy back, 31.4
    // without; 512 objects at 1920x1080 with shading 148.6 and 137.9).
    uint32_t n_tiles = 0;
    size_t ptr_off = 0;
    const std::vector<unsigned char> stage = vis_view_table(c, views, n_views, d_visbuf, n_tiles, ptr_off);
    TGX_TRY(devbuf_reserve(c->vis_views, stage.size()));
    ViewConst* d_vc = (ViewConst*)c->vis_views.ptr;
    unsigned long long** d_outs = (unsigned long long**)((char*)c->vis_views.ptr + ptr_off);
    InlineViews inl;
    const bool few = n_views <= kInlineViews;
    if (few) {
        memcpy(inl.views, stage.data(), n_views * sizeof(ViewConst));
        memcpy(inl.outs, stage.data() + ptr_off, n_views * sizeof(void*));
    } else {
        TGX_CUDA(cudaMemcpyAsync(c->vis_views.ptr, stage.data(), stage.size(), cudaMemcpyHostToDevice, c->stream));
    }

    // Bin capacity.  Grown from earlier frames' totals, read back without
    // waiting.  A frame that could outgrow what is known (the first one, one
    // with more tiles or (view, cluster) pairs than before, or the one after an
    // overflow) is sized exactly instead: the host reads this frame's total
    // after the tile scan, once.  A frame that still overflows is rendered
    // correctly, but slowly, by the tile kernel's record scan.
    const uint64_t n_pairs = (uint64_t)s->n_cluster_pointers * n_views;
    if (n_pairs > 0xffffffffull) { tgx_set_error("too many (view, cluster) pairs"); return TGX_ERR_CAPACITY; }
    VisScratch w;
    bool exact = false;
    constexpr size_t kEntry = sizeof(TileRef);
    if (c->flags & TGX_FLAG_MIN_BIN_CAPACITY) {
        TGX_TRY(devbuf_reserve(c->vis_bins, 64 * kEntry));
        w.bin_capacity = 64;
    } else {
        exact = c->vis_last_tiles == 0 || n_tiles > c->vis_last_tiles || n_pairs > c->vis_last_pairs;
        if (c->vis_done && cudaEventQuery(c->vis_done) == cudaSuccess) {
            const uint32_t* hc = (const uint32_t*)c->h_vis_counters;
            if (hc[C_OVERFLOW]) exact = true;
            if ((size_t)hc[C_ENTRIES] * 2 > c->vis_bins.bytes / kEntry)
                TGX_TRY(devbuf_reserve(c->vis_bins, (size_t)hc[C_ENTRIES] * 2 * kEntry));
        }
        cudaGetLastError();
        TGX_TRY(devbuf_reserve(c->vis_bins, std::max<size_t>((size_t)n_tiles * 128, (size_t)1 << 20) * kEntry));
        w.bin_capacity = (uint32_t)std::min<size_t>(c->vis_bins.bytes / kEntry, 0xffffffffu);
    }
    w.rec_cap = (uint32_t)n_pairs;
    TGX_TRY(devbuf_reserve(c->vis_records, (size_t)w.rec_cap * (sizeof(VisRecord) + sizeof(uint2))));
    // Two sets of counters take turns: each frame's finalize kernel clears the
    // other set.  A set that may not be clear (the first frames, or a frame that
    // was not launched whole) is cleared by a memset.  So is the third set, which
    // frames use that a caller captures: their graph may run between any others.
    TGX_TRY(devbuf_reserve(c->vis_counters, 3 * C_COUNT * sizeof(uint32_t)));
    TGX_TRY(devbuf_reserve(c->vis_tile_cnt, vis_tile_bytes(n_tiles)));
    TGX_TRY(devbuf_reserve(c->vis_tile_off, vis_off_bytes(n_tiles)));
    w.records = (VisRecord*)c->vis_records.ptr;
    w.rects = (uint2*)(w.records + w.rec_cap);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    TGX_CUDA(cudaStreamIsCapturing(c->stream, &capture));
    const bool captured = capture != cudaStreamCaptureStatusNone;
    const uint32_t set = captured ? 2u : c->vis_counter_set == 0u ? 1u : 0u;
    uint32_t* const sets = (uint32_t*)c->vis_counters.ptr;
    w.counters = sets + set * C_COUNT;
    w.host_counters = (uint32_t*)c->h_vis_counters;
    if (!captured) {
        w.next_counters = sets + (set ^ 1u) * C_COUNT;
        if (!c->vis_counters_clear[set])
            TGX_CUDA(cudaMemsetAsync(w.counters, 0, C_COUNT * sizeof(uint32_t), c->stream));
        c->vis_counters_clear[0] = c->vis_counters_clear[1] = false;
    }
    c->vis_counter_set = set;
    w.refs = (TileRef*)c->vis_bins.ptr;
    vis_carve_tiles(w, (uint32_t*)c->vis_tile_cnt.ptr, (uint32_t*)c->vis_tile_off.ptr, n_tiles);
    if (!exact) {
        TGX_TRY(vis_launch(c, s, d_vc, d_outs, n_views, n_tiles, w, VIS_ALL, host_out, few ? &inl : nullptr));
    } else {
        TGX_TRY(vis_launch(c, s, d_vc, d_outs, n_views, n_tiles, w, VIS_TO_SCAN, host_out, few ? &inl : nullptr));
        TGX_CUDA(cudaMemcpyAsync(c->h_vis_counters, w.counters, C_COUNT * sizeof(uint32_t), cudaMemcpyDeviceToHost, c->stream));
        TGX_CUDA(cudaStreamSynchronize(c->stream));
        const uint32_t entries = ((const uint32_t*)c->h_vis_counters)[C_ENTRIES];
        if (entries > w.bin_capacity) {
            TGX_TRY(devbuf_reserve(c->vis_bins, (size_t)entries * kEntry));
            w.refs = (TileRef*)c->vis_bins.ptr;
            w.bin_capacity = (uint32_t)std::min<size_t>(c->vis_bins.bytes / kEntry, 0xffffffffu);
            if (entries <= w.bin_capacity) TGX_CUDA(cudaMemsetAsync(w.counters + C_OVERFLOW, 0, 4, c->stream));
        }
        TGX_TRY(vis_launch(c, s, d_vc, d_outs, n_views, n_tiles, w, VIS_FROM_BINS, host_out));
    }
    c->vis_last_tiles = n_tiles;
    c->vis_last_pairs = n_pairs;
    if (!captured) c->vis_counters_clear[set ^ 1u] = true;
    // the tile kernel wrote this frame's totals to pinned memory, read by the next call without waiting
    if (!c->vis_done) TGX_CUDA(cudaEventCreateWithFlags(&c->vis_done, cudaEventDisableTiming));
    TGX_CUDA(cudaEventRecord(c->vis_done, c->stream));
    return TGX_OK;
}

// ---------------------------------------------------------------------------
// batched frames: the visibility passes of many jobs captured as one CUDA graph
// ---------------------------------------------------------------------------

struct tgx_frame_graph
{
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    void* d_mem = nullptr;                       // view tables, then the shared scratch
    struct Job
    {
        const tgx_scene* scene;
        std::vector<tgx_view> views;             // resolutions fixed at capture
        std::vector<uint64_t*> outs;
        size_t table_off, ptr_off;
        uint32_t n_tiles;
        uint64_t rec_cap, bin_cap;               // this job's own scratch
        size_t scratch_off;
    };
    std::vector<Job> jobs;
    uint32_t kernels = 0;
};

static void frame_graph_free(tgx_frame_graph* g)
{
    if (!g) return;
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    cudaFree(g->d_mem);
    delete g;
}

extern "C" tgx_status tgx_frame_graph_create(tgx_ctx* c, const tgx_vis_job* jobs, uint32_t n_jobs,
                                             tgx_frame_graph** out)
{
    if (!c || !jobs || !n_jobs || !out) { tgx_set_error("tgx_frame_graph_create: NULL argument"); return TGX_ERR_INVALID_ARGUMENT; }
    *out = nullptr;
    TGX_CUDA(cudaSetDevice(c->device));
    tgx_frame_graph* g = new (std::nothrow) tgx_frame_graph();
    if (!g) return TGX_ERR_OUT_OF_MEMORY;
    auto fail = [&](tgx_status st) { cudaStreamSynchronize(c->stream); frame_graph_free(g); return st; };
    // sizes, and one uncaptured frame per job to size its bins
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    size_t table_bytes = 0, scratch_bytes = 0;
    uint32_t total_tiles = 0;
    std::vector<std::vector<unsigned char>> tables(n_jobs);
    auto job_bytes = [&](const tgx_frame_graph::Job& job) {
        return al((size_t)job.rec_cap * (sizeof(VisRecord) + sizeof(uint2))) + 256 + al(vis_tile_bytes(job.n_tiles)) +
               al(vis_off_bytes(job.n_tiles)) + al((size_t)job.bin_cap * sizeof(TileRef));
    };
    for (uint32_t j = 0; j < n_jobs; j++) {
        const tgx_vis_job& jb = jobs[j];
        if (!jb.scene || !jb.views || !jb.d_visbuf || !jb.n_views) {
            tgx_set_error("tgx_frame_graph_create: job %u has a NULL member or no views", j);
            return fail(TGX_ERR_INVALID_ARGUMENT);
        }
        tgx_status st = vis_render_device(c, jb.scene, jb.views, jb.n_views, jb.d_visbuf);
        if (st != TGX_OK) return fail(st);
        if (cudaStreamSynchronize(c->stream) != cudaSuccess) { tgx_set_error("tgx_frame_graph_create: frame failed"); return fail(TGX_ERR_CUDA); }
        const uint32_t entries = ((const uint32_t*)c->h_vis_counters)[C_ENTRIES];
        tgx_frame_graph::Job job;
        job.scene = jb.scene;
        job.views.assign(jb.views, jb.views + jb.n_views);
        job.outs.assign(jb.d_visbuf, jb.d_visbuf + jb.n_views);
        tables[j] = vis_view_table(c, jb.views, jb.n_views, jb.d_visbuf, job.n_tiles, job.ptr_off);
        job.table_off = table_bytes;
        table_bytes += al(tables[j].size());
        job.rec_cap = (uint64_t)jb.scene->n_cluster_pointers * jb.n_views;
        if (!graph_bin_capacity(job.n_tiles, entries, &job.bin_cap) || job.rec_cap > 0xffffffffull ||
            (uint64_t)total_tiles + job.n_tiles > 0xffffffffull) {
            tgx_set_error("tgx_frame_graph_create: job %u has too many (view, cluster) pairs or tiles", j);
            return fail(TGX_ERR_CAPACITY);
        }
        total_tiles += job.n_tiles;
        job.scratch_off = scratch_bytes;
        scratch_bytes += job_bytes(job);
        g->jobs.push_back(std::move(job));
    }
    const size_t jobs_off = table_bytes + scratch_bytes;
    const size_t total = jobs_off + al((size_t)n_jobs * sizeof(TileJob)) + 256;
    if (tgx_malloc(&g->d_mem, total) != cudaSuccess) {
        tgx_set_error("tgx_frame_graph_create: out of device memory (%zu bytes)", total);
        return fail(TGX_ERR_OUT_OF_MEMORY);
    }
    char* base = (char*)g->d_mem;
    for (uint32_t j = 0; j < n_jobs; j++)
        if (cudaMemcpy(base + g->jobs[j].table_off, tables[j].data(), tables[j].size(), cudaMemcpyHostToDevice) != cudaSuccess) {
            tgx_set_error("tgx_frame_graph_create: view table upload failed");
            return fail(TGX_ERR_CUDA);
        }
    // each job's own scratch, so the jobs' sorting passes can run side by side
    std::vector<VisScratch> ws(n_jobs);
    std::vector<TileJob> tjobs(n_jobs);
    for (uint32_t j = 0; j < n_jobs; j++) {
        const tgx_frame_graph::Job& job = g->jobs[j];
        VisScratch& w = ws[j];
        char* p = base + table_bytes + job.scratch_off;
        w.records = (VisRecord*)p;
        w.rec_cap = (uint32_t)job.rec_cap;
        w.rects = (uint2*)(w.records + job.rec_cap);
        p += al((size_t)job.rec_cap * (sizeof(VisRecord) + sizeof(uint2)));
        w.counters = (uint32_t*)p;
        p += 256;
        uint32_t* tile_cnt = (uint32_t*)p;
        p += al(vis_tile_bytes(job.n_tiles));
        uint32_t* tile_off = (uint32_t*)p;
        p += al(vis_off_bytes(job.n_tiles));
        w.refs = (TileRef*)p;
        w.bin_capacity = (uint32_t)job.bin_cap;
        vis_carve_tiles(w, tile_cnt, tile_off, job.n_tiles);
        ViewConst* d_vc = (ViewConst*)(base + job.table_off);
        unsigned long long** d_outs = (unsigned long long**)(base + job.table_off + job.ptr_off);
        tjobs[j] = tile_job(c, job.scene, d_vc, d_outs, (uint32_t)job.views.size(), job.n_tiles, w);
        tjobs[j].first = j ? tjobs[j - 1].first + g->jobs[j - 1].n_tiles : 0u;
        if (j == 0 && (c->flags & TGX_FLAG_TEST_LOST_COPY)) tjobs[j].extra_tx = 64u;
    }
    TileJob* d_jobs = (TileJob*)(base + jobs_off);
    uint32_t* d_queue = (uint32_t*)(base + jobs_off + al((size_t)n_jobs * sizeof(TileJob)));
    if (cudaMemcpy(d_jobs, tjobs.data(), n_jobs * sizeof(TileJob), cudaMemcpyHostToDevice) != cudaSuccess) {
        tgx_set_error("tgx_frame_graph_create: job table upload failed");
        return fail(TGX_ERR_CUDA);
    }
    // side streams and events for the fork and join inside the capture
    const uint32_t n_side = std::min<uint32_t>(n_jobs, 8u);
    std::vector<cudaStream_t> side(n_side, nullptr);
    std::vector<cudaEvent_t> done(n_jobs, nullptr);
    cudaEvent_t fork = nullptr;
    auto release = [&]() {
        for (cudaStream_t q : side) if (q) cudaStreamDestroy(q);
        for (cudaEvent_t e : done) if (e) cudaEventDestroy(e);
        if (fork) cudaEventDestroy(fork);
    };
    bool ok = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess;
    for (uint32_t k = 0; k < n_side && ok; k++) ok = cudaStreamCreateWithFlags(&side[k], cudaStreamNonBlocking) == cudaSuccess;
    for (uint32_t j = 0; j < n_jobs && ok; j++) ok = cudaEventCreateWithFlags(&done[j], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        release();
        tgx_set_error("tgx_frame_graph_create: stream or event creation failed");
        return fail(TGX_ERR_CUDA);
    }
    // capture (no trace events inside the graph): every job's passes up to the
    // bins on its side stream, then one persistent tile launch over all jobs
    const bool tracing = c->trace.enabled;
    c->trace.enabled = false;
    const uint64_t launches0 = c->launches;
    cudaStream_t main_stream = c->stream;
    if (cudaStreamBeginCapture(main_stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        c->trace.enabled = tracing;
        release();
        tgx_set_error("tgx_frame_graph_create: stream capture refused (%s)", cudaGetErrorString(cudaGetLastError()));
        return fail(TGX_ERR_CUDA);
    }
    tgx_status st = TGX_OK;
    if (n_jobs == 1) {
        // one job: its passes and its own tile launch, no fork
        const tgx_frame_graph::Job& job = g->jobs[0];
        ViewConst* d_vc = (ViewConst*)(base + job.table_off);
        unsigned long long** d_outs = (unsigned long long**)(base + job.table_off + job.ptr_off);
        st = vis_launch(c, job.scene, d_vc, d_outs, (uint32_t)job.views.size(), job.n_tiles, ws[0], VIS_ALL);
        goto captured;
    }
    if (cudaEventRecord(fork, main_stream) != cudaSuccess) st = TGX_ERR_CUDA;
    for (uint32_t k = 0; k < n_side && st == TGX_OK; k++)
        if (cudaStreamWaitEvent(side[k], fork, 0) != cudaSuccess) st = TGX_ERR_CUDA;
    for (uint32_t j = 0; j < n_jobs && st == TGX_OK; j++) {
        const tgx_frame_graph::Job& job = g->jobs[j];
        c->stream = side[j % n_side];
        ViewConst* d_vc = (ViewConst*)(base + job.table_off);
        unsigned long long** d_outs = (unsigned long long**)(base + job.table_off + job.ptr_off);
        st = vis_launch(c, job.scene, d_vc, d_outs, (uint32_t)job.views.size(), job.n_tiles, ws[j], VIS_NO_TILES);
        if (st == TGX_OK && cudaEventRecord(done[j], c->stream) != cudaSuccess) st = TGX_ERR_CUDA;
    }
    c->stream = main_stream;
    for (uint32_t j = 0; j < n_jobs && st == TGX_OK; j++)
        if (cudaStreamWaitEvent(main_stream, done[j], 0) != cudaSuccess) st = TGX_ERR_CUDA;
    if (st == TGX_OK) st = vis_launch_queue(c, d_jobs, n_jobs, total_tiles, d_queue);
captured:
    const cudaError_t ce = cudaStreamEndCapture(c->stream, &g->graph);
    release();
    c->trace.enabled = tracing;
    g->kernels = (uint32_t)(c->launches - launches0);
    c->launches = launches0;
    if (st != TGX_OK) return fail(st);
    if (ce != cudaSuccess || cudaGraphInstantiate(&g->exec, g->graph, 0) != cudaSuccess) {
        tgx_set_error("tgx_frame_graph_create: graph capture failed (%s)", cudaGetErrorString(cudaGetLastError()));
        return fail(TGX_ERR_CUDA);
    }
    *out = g;
    return TGX_OK;
}

extern "C" tgx_status tgx_frame_graph_launch(tgx_ctx* c, tgx_frame_graph* g)
{
    if (!c || !g) return TGX_ERR_INVALID_ARGUMENT;
    TGX_CUDA(cudaGraphLaunch(g->exec, c->stream));
    c->launches += g->kernels;
    return TGX_OK;
}

extern "C" tgx_status tgx_frame_graph_set_views(tgx_ctx* c, tgx_frame_graph* g, uint32_t job, const tgx_view* views)
{
    if (!c || !g || !views || job >= g->jobs.size()) return TGX_ERR_INVALID_ARGUMENT;
    tgx_frame_graph::Job& jb = g->jobs[job];
    const uint32_t n = (uint32_t)jb.views.size();
    for (uint32_t i = 0; i < n; i++)
        if (views[i].width != jb.views[i].width || views[i].height != jb.views[i].height) {
            tgx_set_error("tgx_frame_graph_set_views: view %u changes its resolution", i);
            return TGX_ERR_INVALID_ARGUMENT;
        }
    TGX_TRY(check_views(views, n, c->tile_w, c->tile_h));
    uint32_t n_tiles = 0;
    size_t ptr_off = 0;
    const std::vector<unsigned char> t = vis_view_table(c, views, n, jb.outs.data(), n_tiles, ptr_off);
    // the pinned-free staging copy is ordered on the stream before the next launch
    TGX_CUDA(cudaMemcpyAsync((char*)g->d_mem + jb.table_off, t.data(), t.size(), cudaMemcpyHostToDevice, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    jb.views.assign(views, views + n);
    return TGX_OK;
}

extern "C" uint32_t tgx_frame_graph_kernels(const tgx_frame_graph* g) { return g ? g->kernels : 0u; }

extern "C" void tgx_frame_graph_destroy(tgx_ctx* c, tgx_frame_graph* g)
{
    if (c) cudaStreamSynchronize(c->stream);
    frame_graph_free(g);
}

extern "C" tgx_status tgx_vis_render(tgx_ctx* c, const tgx_scene* s, const tgx_view* views, uint32_t n_views,
                                     uint64_t* const* d_visbuf)
{
    return vis_render_device(c, s, views, n_views, d_visbuf);
}

// The device address of pinned (page-locked, mapped) host memory, or null for
// any other pointer.  The tile kernel stores each pixel once, so it can write
// a pinned host buffer directly over the CPU-GPU link, hidden under its own
// work, instead of through a device buffer and a copy.
static uint64_t* mapped_host(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost && a.devicePointer ? (uint64_t*)a.devicePointer : nullptr;
}

// whether some output of a host-buffer render is written in host memory directly
static bool any_mapped(const std::vector<bool>& staged)
{
    for (bool st : staged)
        if (!st) return true;
    return false;
}

// Output pointers of a host-buffer render: pinned buffers directly, the rest
// in `stage` (device memory, `staged` entries) for a copy afterwards.
static tgx_status host_outputs(tgx_ctx* c, const tgx_view* views, uint32_t n_views, uint64_t* const* h_visbuf,
                               DevBuf& stage, std::vector<uint64_t*>& dptr, std::vector<bool>& staged, const char* who)
{
    size_t total = 0;
    std::vector<size_t> offs(n_views);
    dptr.assign(n_views, nullptr);
    staged.assign(n_views, false);
    for (uint32_t i = 0; i < n_views; i++) {
        if (!h_visbuf[i]) { tgx_set_error("%s: output %u is NULL", who, i); return TGX_ERR_INVALID_ARGUMENT; }
        dptr[i] = mapped_host(h_visbuf[i]);
        if (dptr[i]) continue;
        staged[i] = true;
        offs[i] = total;
        total += (size_t)views[i].width * views[i].height;
    }
    if (total) TGX_TRY(devbuf_reserve(stage, total * 8));
    for (uint32_t i = 0; i < n_views; i++)
        if (staged[i]) dptr[i] = (uint64_t*)stage.ptr + offs[i];
    return TGX_OK;
}

extern "C" tgx_status tgx_vis_render_host(tgx_ctx* c, const tgx_scene* s, const tgx_view* views, uint32_t n_views,
                                          uint64_t* const* h_visbuf)
{
    if (!c || !s || !h_visbuf) { tgx_set_error("tgx_vis_render_host: NULL argument"); return TGX_ERR_INVALID_ARGUMENT; }
    TGX_TRY(check_views(views, n_views, c->tile_w, c->tile_h));
    TGX_CUDA(cudaSetDevice(c->device));
    std::vector<uint64_t*> dptr;
    std::vector<bool> staged;
    TGX_TRY(host_outputs(c, views, n_views, h_visbuf, c->host_stage, dptr, staged, "tgx_vis_render_host"));
    TGX_TRY(vis_render_device(c, s, views, n_views, dptr.data(), any_mapped(staged)));
    for (uint32_t i = 0; i < n_views; i++)
        if (staged[i])
            TGX_CUDA(cudaMemcpyAsync(h_visbuf[i], dptr[i], (size_t)views[i].width * views[i].height * 8,
                                     cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    return TGX_OK;
}

// Pinned host buffers are written by the render itself.  Other buffers go
// through two device copies that alternate between frames: frame k renders
// into copy k % 2 on the context stream once frame k-2's copy out of it is
// done (an event wait on the device, not the host), then the copy stream
// takes it to the host while frame k+1 renders into the other copy.
extern "C" tgx_status tgx_vis_render_host_async(tgx_ctx* c, const tgx_scene* s, const tgx_view* views,
                                                uint32_t n_views, uint64_t* const* h_visbuf)
{
    if (!c || !s || !h_visbuf) {
        tgx_set_error("tgx_vis_render_host_async: NULL argument");
        return TGX_ERR_INVALID_ARGUMENT;
    }
    TGX_TRY(check_views(views, n_views, c->tile_w, c->tile_h));
    TGX_CUDA(cudaSetDevice(c->device));
    if (!c->copy_stream) {
        TGX_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
        for (int i = 0; i < 2; i++) {
            TGX_CUDA(cudaEventCreateWithFlags(&c->host_rendered[i], cudaEventDisableTiming));
            TGX_CUDA(cudaEventCreateWithFlags(&c->host_copied[i], cudaEventDisableTiming));
        }
    }
    const uint32_t slot = (uint32_t)(c->host_issued & 1u);
    // the copy two frames back reads this slot: the render waits for it on the device
    TGX_CUDA(cudaStreamWaitEvent(c->stream, c->host_copied[slot], 0));
    std::vector<uint64_t*> dptr;
    std::vector<bool> staged;
    TGX_TRY(host_outputs(c, views, n_views, h_visbuf, c->host_slot[slot], dptr, staged, "tgx_vis_render_host_async"));
    TGX_TRY(vis_render_device(c, s, views, n_views, dptr.data(), any_mapped(staged)));
    TGX_CUDA(cudaEventRecord(c->host_rendered[slot], c->stream));
    TGX_CUDA(cudaStreamWaitEvent(c->copy_stream, c->host_rendered[slot], 0));
    for (uint32_t i = 0; i < n_views; i++)
        if (staged[i])
            TGX_CUDA(cudaMemcpyAsync(h_visbuf[i], dptr[i], (size_t)views[i].width * views[i].height * 8,
                                     cudaMemcpyDeviceToHost, c->copy_stream));
    // marks the frame done: after its copies, or after its render when it wrote the host directly
    TGX_CUDA(cudaEventRecord(c->host_copied[slot], c->copy_stream));
    c->host_issued++;
    return TGX_OK;
}

extern "C" tgx_status tgx_vis_host_wait(tgx_ctx* c, uint32_t max_in_flight)
{
    if (!c) { tgx_set_error("tgx_vis_host_wait: NULL context"); return TGX_ERR_INVALID_ARGUMENT; }
    while (c->host_issued - c->host_done > max_in_flight) {
        // copies complete in issue order; the slot's event is that of its latest frame
        TGX_CUDA(cudaEventSynchronize(c->host_copied[c->host_done & 1u]));
        c->host_done++;
    }
    return TGX_OK;
}

extern "C" tgx_status tgx_vis_get_stats(tgx_ctx* c, tgx_vis_stats* out)
{
    if (!c || !out) return TGX_ERR_INVALID_ARGUMENT;
    memset(out, 0, sizeof(*out));
    if (!c->vis_counters.ptr) return TGX_OK;
    uint32_t h[C_COUNT];
    TGX_CUDA(cudaMemcpyAsync(c->h_counter, (uint32_t*)c->vis_counters.ptr + c->vis_counter_set * C_COUNT, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    memcpy(h, c->h_counter, sizeof(h));
    out->visible_clusters = h[C_RECORDS];
    out->bin_entries = h[C_ENTRIES];
    out->dda_overruns = h[C_DDA_OVERRUN];
    out->tiles = c->vis_last_tiles;
    return TGX_OK;
}

extern "C" tgx_status tgx_set_vis_tuning(tgx_ctx* c, uint32_t depth_buckets, uint32_t batch, uint32_t drain)
{
    if (!c) return TGX_ERR_INVALID_ARGUMENT;
    const uint32_t nb = depth_buckets ? depth_buckets : 16u, bt = batch ? batch : kBatch, dr = drain ? drain : 32u;
    if ((nb != 8 && nb != 16 && nb != 32) || bt > kBatch || dr > 32) {
        tgx_set_error("tgx_set_vis_tuning: depth buckets %u (8, 16 or 32), batch %u (1..%u), drain %u (1..32)", nb, bt,
                      kBatch, dr);
        return TGX_ERR_INVALID_ARGUMENT;
    }
    c->vis_bshift = nb == 32 ? 0u : nb == 16 ? 1u : 2u;
    c->vis_batch = bt;
    c->vis_drain = dr;
    return TGX_OK;
}

extern "C" tgx_status tgx_vis_count_work(tgx_ctx* c, int enable)
{
    if (!c) return TGX_ERR_INVALID_ARGUMENT;
    c->vis_count_work = enable != 0;
    return TGX_OK;
}

extern "C" tgx_status tgx_vis_get_work(tgx_ctx* c, tgx_vis_work* out)
{
    if (!c || !out) return TGX_ERR_INVALID_ARGUMENT;
    memset(out, 0, sizeof(*out));
    if (!c->vis_work.ptr) return TGX_OK;
    static_assert(sizeof(tgx_vis_work) == W_COUNT * sizeof(uint64_t), "tgx_vis_work layout");
    TGX_CUDA(cudaMemcpyAsync(out, c->vis_work.ptr, sizeof(*out), cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    return TGX_OK;
}

// ---------------------------------------------------------------------------
// Visibility render without any allocation (tgx_vis_render_noalloc).
//
// For callers that cannot allocate device memory at all: code running under an
// allocator they do not own (a host application with a fixed memory budget, or
// a plugin whose host forbids cudaMalloc), or code that must not trigger the
// implicit device synchronisation a cudaMalloc/cudaFree can cause.  All the
// scratch of the pass lives in one file-scope device array of fixed size,
// created when the library is loaded on a device and kept until the process
// exits.  The caller passes the scene arrays and the output buffer, both in
// device memory.
// ---------------------------------------------------------------------------

namespace {

constexpr uint32_t kNaMaxObjects = 65536;
constexpr uint32_t kNaMaxClusterPointers = 1u << 19;
constexpr uint32_t kNaMaxTiles = 32768;      // 16x16 tiles: up to 3840x2160
constexpr uint32_t kNaBins = 1u << 18;       // (tile, cluster) entries; more take the exact record-scan path
constexpr uint32_t kNaTile = 16;

constexpr size_t na_align(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kNaCounters = 0;
constexpr size_t kNaStatus = kNaCounters + 256;
constexpr size_t kNaViews = kNaStatus + 256;
constexpr size_t kNaInvRot = kNaViews + na_align(sizeof(ViewConst) + 16);
constexpr size_t kNaRecords = kNaInvRot + na_align((size_t)kNaMaxObjects * 9 * 4);
constexpr size_t kNaRects = kNaRecords + na_align((size_t)kNaMaxClusterPointers * sizeof(VisRecord));
constexpr size_t kNaSupers = kNaRects + na_align((size_t)kNaMaxClusterPointers * 8);   // the last words before the counts
constexpr size_t kNaBucketCnt = kNaSupers + na_align((size_t)scan_supers(kNaMaxTiles) * kGroupWords * 4);
constexpr uint32_t kNaBuckets = 16;          // depth buckets per tile (bucket shift 1)
constexpr size_t kNaTileTotal = kNaBucketCnt + na_align((size_t)kNaMaxTiles * kNaBuckets * 4);
constexpr size_t kNaGroups = kNaTileTotal + na_align((size_t)kNaMaxTiles * 4);
constexpr size_t kNaTileOff = kNaGroups + na_align((size_t)scan_groups(kNaMaxTiles) * kGroupWords * 4);
constexpr size_t kNaSlotInfo = kNaTileOff + na_align(((size_t)kNaMaxTiles + 4) * 4);
constexpr size_t kNaBinsOff = kNaSlotInfo + na_align((size_t)kNaMaxTiles * 16);
constexpr uint32_t kNaChunks = 1u << 16;
constexpr size_t kNaChunkOff = kNaBinsOff + na_align((size_t)kNaBins * sizeof(TileRef));
constexpr size_t kNaBytes = kNaChunkOff + na_align((size_t)kNaChunks * sizeof(uint2));   // about 28 MiB

// The scratch.  In host code this name is only a host-side stand-in: its
// device address is taken with cudaGetSymbolAddress below.
static __device__ __align__(256) unsigned char g_vis_noalloc_scratch[kNaBytes];

// The call's set-up on the device, so that no host buffer is read after the
// call returns: the first CTA writes the view constants and the output
// pointer (both passed by value) and zeroes the counters and the status
// word; every thread writes one object's 3x3 of inverse(rotation), as
// k_object_setup computes it at upload.
__global__ void __launch_bounds__(128) k_vis_noalloc_setup(ViewConst vc, unsigned long long* visbuf,
                                                          ViewConst* __restrict__ d_vc,
                                                          unsigned long long** __restrict__ d_outs,
                                                          uint32_t* __restrict__ counters,
                                                          tgx_dev_status* __restrict__ status,
                                                          const tgx_object* __restrict__ objs, uint32_t n,
                                                          float* __restrict__ inv_rot)
{
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            *d_vc = vc;
            *d_outs = visbuf;
            status->code = 0u;
            status->where = 0u;
            status->detail = 0ull;
        }
        if (threadIdx.x < 64) counters[threadIdx.x] = 0u;
    }
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float rot[16], inv[16];
#pragma unroll
    for (int k = 0; k < 16; k++) rot[k] = objs[i].rotation[k];
    dm4_inverse(rot, inv);
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) inv_rot[9 * i + 3 * r + c] = DM(inv, r, c);
}

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
void* g_na_ptr[kNaMaxDevices] = {};

// Device address of the scratch on the current device, looked up once per device.
tgx_status na_scratch(int device, unsigned char** out)
{
    if (device < 0 || device >= kNaMaxDevices) {
        tgx_set_error("tgx_vis_render_noalloc: device %d out of range", device);
        return TGX_ERR_INVALID_ARGUMENT;
    }
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_ptr[device]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_vis_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            tgx_set_error("tgx_vis_render_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
            return TGX_ERR_CUDA;
        }
        g_na_ptr[device] = p;
    }
    *out = (unsigned char*)g_na_ptr[device];
    return TGX_OK;
}

#define NA_LAUNCH(grid, block, kernel, ...)                                                        \
    do {                                                                                           \
        kernel<<<(grid), (block), 0, st>>>(__VA_ARGS__);                                           \
        const cudaError_t le_ = cudaGetLastError();                                                \
        if (le_ != cudaSuccess) {                                                                  \
            tgx_set_error("tgx_vis_render_noalloc: launch of %s failed: %s", #kernel,              \
                          cudaGetErrorString(le_));                                                \
            return TGX_ERR_CUDA;                                                                   \
        }                                                                                          \
    } while (0)

}  // namespace

extern "C" tgx_status tgx_vis_render_noalloc(void* stream, const tgx_object* d_objects, uint32_t n_objects,
                                             const uint32_t* d_cluster_pointers, uint32_t n_cluster_pointers,
                                             const uint32_t* d_cluster_idx_to_object_idx,
                                             const uint32_t* d_voxel_bits, const tgx_view* view, uint64_t* d_visbuf,
                                             tgx_device_error* out_error)
{
    if (!d_objects || !d_cluster_pointers || !d_cluster_idx_to_object_idx || !d_voxel_bits || !view || !d_visbuf) {
        tgx_set_error("tgx_vis_render_noalloc: NULL argument");
        return TGX_ERR_INVALID_ARGUMENT;
    }
    if (n_objects == 0 || n_objects > kNaMaxObjects) {
        tgx_set_error("tgx_vis_render_noalloc: %u objects, the fixed scratch holds 1..%u", n_objects, kNaMaxObjects);
        return TGX_ERR_CAPACITY;
    }
    if (n_cluster_pointers == 0 || n_cluster_pointers > kNaMaxClusterPointers) {
        tgx_set_error("tgx_vis_render_noalloc: %u cluster pointers, the fixed scratch holds 1..%u", n_cluster_pointers,
                      kNaMaxClusterPointers);
        return TGX_ERR_CAPACITY;
    }
    TGX_TRY(check_views(view, 1, kNaTile, kNaTile));
    ViewConst vc;
    make_view_const(*view, kNaTile, kNaTile, 0, vc);
    const uint32_t n_tiles = vc.tiles_x * vc.tiles_y;
    if (n_tiles > kNaMaxTiles) {
        tgx_set_error("tgx_vis_render_noalloc: %ux%u needs %u tiles of 16x16, the fixed scratch holds %u", view->width,
                      view->height, n_tiles, kNaMaxTiles);
        return TGX_ERR_CAPACITY;
    }
    int device = 0;
    TGX_CUDA(cudaGetDevice(&device));
    unsigned char* base = nullptr;
    TGX_TRY(na_scratch(device, &base));
    cudaStream_t st = (cudaStream_t)stream;

    uint32_t* counters = (uint32_t*)(base + kNaCounters);
    tgx_dev_status* status = (tgx_dev_status*)(base + kNaStatus);
    ViewConst* d_vc = (ViewConst*)(base + kNaViews);
    unsigned long long** d_outs = (unsigned long long**)(base + kNaViews + ((sizeof(ViewConst) + 15) & ~(size_t)15));
    float* inv_rot = (float*)(base + kNaInvRot);
    VisRecord* records = (VisRecord*)(base + kNaRecords);
    uint2* rects = (uint2*)(base + kNaRects);
    uint32_t* bucket_cnt = (uint32_t*)(base + kNaBucketCnt);
    uint32_t* supers = bucket_cnt - scan_supers(n_tiles) * kGroupWords;
    uint32_t* tile_total = (uint32_t*)(base + kNaTileTotal);
    uint32_t* groups = (uint32_t*)(base + kNaGroups);
    uint32_t* tile_off = (uint32_t*)(base + kNaTileOff);
    uint4* slot_info = (uint4*)(base + kNaSlotInfo);
    TileRef* refs = (TileRef*)(base + kNaBinsOff);
    uint2* chunks = (uint2*)(base + kNaChunkOff);

    int sms = 0;
    TGX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    const uint32_t warp_grid = (uint32_t)sms * 8;
    // what must start at zero (counters, status) is cleared by the set-up kernel;
    // everything else is written before it is read
    NA_LAUNCH((n_objects + 127) / 128, 128, k_vis_noalloc_setup, vc, (unsigned long long*)d_visbuf, d_vc, d_outs,
              counters, status, d_objects, n_objects, inv_rot);
    NA_LAUNCH((n_cluster_pointers + 255) / 256, 256, (k_vis_cluster_setup<false, NoViews>), d_objects, d_cluster_pointers,
              d_cluster_idx_to_object_idx, d_voxel_bits, (const uint32_t*)nullptr, n_cluster_pointers, NoViews{}, d_vc,
              d_outs, 1u, records, rects, kNaMaxClusterPointers, counters, supers,
              scan_supers(n_tiles) * kGroupWords + n_tiles * kNaBuckets, chunks, kNaChunks,
              status);
    NA_LAUNCH(warp_grid, 256, k_vis_count, records, rects, counters, kNaMaxClusterPointers, d_objects, d_vc, bucket_cnt,
              n_tiles, 1u, chunks, kNaChunks);
    const uint32_t n_scan_ctas = scan_groups(n_tiles);
    NA_LAUNCH(n_scan_ctas, kScanTiles, k_vis_prefix<kNaBuckets>, bucket_cnt, tile_total, n_tiles, groups, supers);
    NA_LAUNCH(n_scan_ctas, kScanTiles, k_vis_finalize, tile_total, n_tiles, groups, supers, tile_off, slot_info, kNaBins,
              counters, (uint32_t*)nullptr, d_vc, 1u);
    NA_LAUNCH(warp_grid, 256, k_vis_bin_fill, records, rects, counters, d_vc, tile_off, bucket_cnt, refs,
              n_tiles, kNaBins, 1u, chunks, kNaChunks, slot_info, d_outs, 1u, status);
    TileJob J;
    J.records = records;
    J.rects = rects;
    J.refs = refs;
    J.slot_info = slot_info;
    J.views = d_vc;
    J.bits = d_voxel_bits;
    J.inv_rot = inv_rot;
    J.outs = d_outs;
    J.counters = counters;
    J.host_counters = nullptr;
    J.n_tiles = n_tiles;
    J.cleared = 1;
    J.first = 0;
    J.work = nullptr;
    J.extra_tx = 0;
    J.interleave = 0;
    J.bshift = 1;
    J.batch = kBatch;
    J.drain = 32;
    k_vis_tiles<256, 5><<<n_tiles, kNaTile * kNaTile, tile_smem_bytes(kNaTile * kNaTile), st>>>(J, status);
    if (const cudaError_t le = cudaGetLastError(); le != cudaSuccess) {
        tgx_set_error("tgx_vis_render_noalloc: launch of k_vis_tiles failed: %s", cudaGetErrorString(le));
        return TGX_ERR_CUDA;
    }
    if (out_error) {
        tgx_dev_status hs;
        TGX_CUDA(cudaMemcpyAsync(&hs, status, sizeof(hs), cudaMemcpyDeviceToHost, st));
        TGX_CUDA(cudaStreamSynchronize(st));
        out_error->code = hs.code;
        out_error->where = hs.where;
        out_error->detail = hs.detail;
        if (hs.code) return (tgx_status)hs.code;
    }
    return TGX_OK;
}
#undef NA_LAUNCH
