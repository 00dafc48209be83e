// svo.cu -- one-bit SVO build on the GPU.
//
// Replaces tg's recursive single-threaded CPU builder tg_svo_create
// (tg_sparse_voxel_octree.c:466-542) with data-parallel passes that set exactly the
// same world voxels:
//
//   1. k_svo_candidates  one thread per cluster pointer: drops empty clusters
//      (:515-531) and lists the cluster with every 32^3 block that its world box
//      can touch (in an update: every dirty one).
//      k_svo_test_pairs  one thread per listed pair: the reference's OBB/AABB test
//      (tg_physics.c:226-392) on the nodes on the path from the root's children
//      down to the block, with the node boxes and ws2ms matrix of
//      tg__construct_inner_node (:319-397), except where it surely passes.  The
//      block of a pair that passes is marked in the dense block table.
//   2. k_svo_alloc       gives every marked block a slot in the block pool.
//   3. k_svo_pair_count, _ranges, _fill: the pairs grouped by block, a record of
//      corners and range for each.
//      k_svo_voxelize    one CTA per marked block, or four (8 layers each) when
//      few are marked; a warp per pair: the leaf voxelisation of
//      tg__construct_leaf_node (:102-317) -- corner lerp, [0,8)^3 test, bit
//      fetch -- into the block's image (and material grid) in shared memory,
//      written out whole and coalesced, with no global atomics; and inside each
//      block one bit per non-empty 4^3 and 8^3 cell (the sub-block levels the
//      traversal steps through before single voxels).
//      k_svo_publish     the slots go into the block table.
//   4. k_svo_pyramid     one bit per non-empty block and per non-empty node of
//      every coarser level.
//
// An update marks the blocks that moved objects touched or touch
// (k_svo_mark_dirty), frees their slots (k_svo_release_dirty) and runs the same
// passes over these blocks.
//
// The node encoding of the reference (u16 relative child pointers, 64-entry
// leaf lists) is not kept; the voxel set is.  Side length 2^6 .. 2^14.

#include "svo_trace.cuh"

#include <algorithm>
#include <vector>

namespace {

constexpr uint32_t kBlockSide = 32;
constexpr uint32_t kBlockWords = 1024;
// Table entries: 0 without a block, slot + 1 of one; with kMarked, a block that the
// pass under way builds: kMark until it has a slot, then kMarked | its place in the
// list of marked blocks, until k_svo_publish.
constexpr uint32_t kMarked = 0x80000000u;
constexpr uint32_t kMark = 0xffffffffu;
constexpr uint32_t kNoBlock = 0xffffffffu;   // block of a candidate pair that failed its test
constexpr uint32_t kWarpsPerVoxCta = 16;

struct SvoPair
{
    uint32_t cluster_pointer;
    uint32_t block;
};

enum SvoCounter { S_PAIRS = 0, S_MARKED = 1, S_SLOTS = 2, S_NONEMPTY = 3, S_FREED = 4, S_MOVED = 5, S_CAND = 6, S_COUNT = 8 };

struct dv3 { float x, y, z; };

__device__ __forceinline__ void cluster_offsets(const tgx_object& od, uint32_t rel, float off[3], float ohe[3])
{
    const uint32_t nx = od.n_cluster_pointers_per_dim[0], ny = od.n_cluster_pointers_per_dim[1];
    off[0] = (float)((rel % nx) * 8u);
    off[1] = (float)(((rel / nx) % ny) * 8u);
    off[2] = (float)((rel / (nx * ny)) * 8u);
    const float h = 4.0f;   // (f32)(TG_N_PRIMITIVES_PER_CLUSTER_CUBE_ROOT / 2)
    ohe[0] = xmul((float)od.n_cluster_pointers_per_dim[0], h);
    ohe[1] = xmul((float)od.n_cluster_pointers_per_dim[1], h);
    ohe[2] = xmul((float)od.n_cluster_pointers_per_dim[2], h);
}

// tg_world_space_to_cluster_model_space (tg_sparse_voxel_octree.c:23-60)
__device__ __forceinline__ void svo_ws2ms(const tgx_object& od, uint32_t rel, float* out)
{
    float off[3], ohe[3], rot[16], m1[16], m2[16], m3[16], m4[16];
    cluster_offsets(od, rel, off, ohe);
#pragma unroll
    for (int k = 0; k < 16; k++) rot[k] = od.rotation[k];
    dm4_translate(-od.translation[0], -od.translation[1], -od.translation[2], m1);
    dm4_inverse(rot, m2);
    dm4_translate(ohe[0], ohe[1], ohe[2], m3);
    dm4_translate(-off[0], -off[1], -off[2], m4);
    dm4_mul(m4, m3, out);
    dm4_mul(out, m2, out);
    dm4_mul(out, m1, out);
}

// tg_cluster_model_space_to_world_space (tg_sparse_voxel_octree.c:62-100)
__device__ __forceinline__ void svo_cs2ws(const tgx_object& od, uint32_t rel, float* out)
{
    float off[3], ohe[3], rot[16], m1[16], m2[16], m4[16];
    cluster_offsets(od, rel, off, ohe);
#pragma unroll
    for (int k = 0; k < 16; k++) rot[k] = od.rotation[k];
    dm4_translate(off[0], off[1], off[2], m1);
    dm4_translate(-ohe[0], -ohe[1], -ohe[2], m2);
    dm4_translate(od.translation[0], od.translation[1], od.translation[2], m4);
    dm4_mul(m4, rot, out);
    dm4_mul(out, m2, out);
    dm4_mul(out, m1, out);
}

__device__ __forceinline__ dv3 mulv4p(const float* m, float x, float y, float z)
{
    float r[3];
    dm4_mulv4(m, x, y, z, 1.0f, r);
    return dv3{r[0], r[1], r[2]};
}

__device__ __forceinline__ float dot3(dv3 a, dv3 b) { return xadd(xadd(xmul(a.x, b.x), xmul(a.y, b.y)), xmul(a.z, b.z)); }
__device__ __forceinline__ float mag3(dv3 a) { return xsqrt(dot3(a, a)); }
__device__ __forceinline__ dv3 sub3(dv3 a, dv3 b) { return dv3{xsub(a.x, b.x), xsub(a.y, b.y), xsub(a.z, b.z)}; }
__device__ __forceinline__ dv3 normalized3(dv3 a)
{
    const float m = mag3(a);
    return dv3{xdiv(a.x, m), xdiv(a.y, m), xdiv(a.z, m)};
}

// tg_intersect_aabb_obb_ignore_contact (tg_physics.c:226-392) with the AABB
// [0,8]^3 (the cluster) and the OBB given by its 8 corners (a block).
__device__ __forceinline__ bool aabb_obb(const dv3* c)
{
    const float mx = 8.0f;
    bool sep;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].x <= 0.0f;
    if (sep) return false;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].x >= mx;
    if (sep) return false;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].y <= 0.0f;
    if (sep) return false;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].y >= mx;
    if (sep) return false;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].z <= 0.0f;
    if (sep) return false;
    sep = true;
#pragma unroll
    for (int i = 0; i < 8; i++) sep &= c[i].z >= mx;
    if (sep) return false;

    const dv3 nxp = normalized3(sub3(c[1], c[0]));
    const dv3 nyp = normalized3(sub3(c[2], c[0]));
    const dv3 nzp = normalized3(sub3(c[4], c[0]));
    const dv3 nrm[6] = {dv3{-nxp.x, -nxp.y, -nxp.z}, nxp, dv3{-nyp.x, -nyp.y, -nyp.z}, nyp,
                        dv3{-nzp.x, -nzp.y, -nzp.z}, nzp};
    const float l0 = mag3(c[0]);
    const float l1 = mag3(c[7]);
    const dv3 n0 = l0 == 0.0f ? dv3{0.0f, 0.0f, 0.0f} : dv3{xdiv(c[0].x, l0), xdiv(c[0].y, l0), xdiv(c[0].z, l0)};
    const dv3 n1 = l1 == 0.0f ? dv3{0.0f, 0.0f, 0.0f} : dv3{xdiv(c[7].x, l1), xdiv(c[7].y, l1), xdiv(c[7].z, l1)};
    float dist[6];
    dist[0] = xmul(l0, dot3(n0, nrm[0]));
    dist[1] = xmul(l1, dot3(n1, nrm[1]));
    dist[2] = xmul(l0, dot3(n0, nrm[2]));
    dist[3] = xmul(l1, dot3(n1, nrm[3]));
    dist[4] = xmul(l0, dot3(n0, nrm[4]));
    dist[5] = xmul(l1, dot3(n1, nrm[5]));
#pragma unroll
    for (int p = 0; p < 6; p++) {
        sep = true;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const dv3 pt = dv3{(k & 1) ? mx : 0.0f, (k & 2) ? mx : 0.0f, (k & 4) ? mx : 0.0f};
            sep &= xsub(dot3(nrm[p], pt), dist[p]) >= 0.0f;
        }
        if (sep) return false;
    }
    return true;
}

// ---------------------------------------------------------------------------
// 1. candidates
// ---------------------------------------------------------------------------

// The blocks the conservative world box of a cluster reaches (clamped to the
// cube); false when it misses the cube.  lo, hi: the box.
__device__ __forceinline__ bool cluster_blocks(const tgx_object& od, uint32_t rel, const float mn[3], uint32_t B,
                                               float lo[3], float hi[3], int b0[3], int b1[3])
{
    float off[3], ohe[3];
    cluster_offsets(od, rel, off, ohe);
#pragma unroll
    for (int r = 0; r < 3; r++) { lo[r] = 1e30f; hi[r] = -1e30f; }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float lx = off[0] + ((k & 1) ? 8.0f : 0.0f) - ohe[0];
        const float ly = off[1] + ((k & 2) ? 8.0f : 0.0f) - ohe[1];
        const float lz = off[2] + ((k & 4) ? 8.0f : 0.0f) - ohe[2];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const float p = DM(od.rotation, r, 0) * lx + DM(od.rotation, r, 1) * ly + DM(od.rotation, r, 2) * lz +
                            od.translation[r];
            lo[r] = fminf(lo[r], p);
            hi[r] = fmaxf(hi[r], p);
        }
    }
    bool some = true;
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float slack = 0.5f + 1e-5f * fabsf(lo[r]) + 1e-5f * fabsf(hi[r]);
        b0[r] = max((int)floorf((lo[r] - slack - mn[r]) / 32.0f), 0);
        b1[r] = min((int)floorf((hi[r] + slack - mn[r]) / 32.0f), (int)B - 1);
        some = some && b0[r] <= b1[r];
    }
    return some;
}

// Every (cluster, block) pair whose block the cluster's conservative box
// reaches, one thread per cluster pointer, appended by one atomic per warp.  The
// tests of a pair are long (seven levels at 4096^3), so they run in a kernel of
// their own with a thread per pair: with a thread per cluster a warp took as
// long as its cluster with the most blocks.  Emptiness comes with the object in
// cp_obj instead of from the 64-byte bitmask.
__global__ void __launch_bounds__(128) k_svo_candidates(const tgx_object* __restrict__ objects,
                                                       const uint32_t* __restrict__ cp_obj, uint32_t n_cp, float mnx,
                                                       float mny, float mnz, uint32_t B, SvoPair* __restrict__ pairs,
                                                       uint32_t pair_capacity, uint32_t* __restrict__ counters,
                                                       tgx_dev_status* __restrict__ status,
                                                       const uint32_t* __restrict__ dirty /* null: every block; else a bit per block */)
{
    pdl_wait();
    const uint32_t cp = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const float mn[3] = {mnx, mny, mnz};
    float lo[3], hi[3];
    int b0[3] = {0, 0, 0}, b1[3] = {-1, -1, -1};
    const uint32_t po = cp < n_cp ? cp_obj[cp] : 0x80000000u;
    bool some = false;
    if (!(po >> 31)) {   // some set voxel
        const tgx_object& od = objects[po];
        some = cluster_blocks(od, cp - od.first_cluster_pointer, mn, B, lo, hi, b0, b1);
    }
    const uint32_t nx = some ? (uint32_t)(b1[0] - b0[0] + 1) : 0u, ny = some ? (uint32_t)(b1[1] - b0[1] + 1) : 0u;
    const uint32_t total = some ? nx * ny * (uint32_t)(b1[2] - b0[2] + 1) : 0u;
    auto block = [&](uint32_t k) {
        const uint32_t q = k / nx, x = k - q * nx, z = q / ny, y = q - z * ny;
        return (((uint32_t)b0[2] + z) * B + (uint32_t)b0[1] + y) * B + (uint32_t)b0[0] + x;
    };
    uint32_t n = total;
    if (dirty) {
        n = 0;
        for (uint32_t k = 0; k < total; k++) {
            const uint32_t blk = block(k);
            n += (dirty[blk >> 5] >> (blk & 31u)) & 1u;
        }
    }
    uint32_t incl = n;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    uint32_t base = 0;
    if (lane == 31u && incl) base = atomicAdd(&counters[S_CAND], incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - n;
    if (n == 0u) return;
    if ((uint64_t)base + n > pair_capacity) dev_error(status, TGX_ERR_CAPACITY, 11, base);
    for (uint32_t k = 0; k < total; k++) {
        const uint32_t blk = block(k);
        if (dirty && !((dirty[blk >> 5] >> (blk & 31u)) & 1u)) continue;
        if (base < pair_capacity) pairs[base] = SvoPair{cp, blk};
        base++;
    }
}

// The reference's test of every candidate pair, a thread each: a pair that fails
// gets the block ~0, one that passes marks its block (and lists it the first
// time).  Bound by instruction issue.  A node that holds the cluster's world box
// with a margin surely passes: no axis can separate them, and the margin
// (1 + 2e-5 of the coordinates) is far above the test's rounding.  Most levels of
// most paths are like that (a cluster's box lies inside its cell of 2^k voxels in
// all but about 45 / 2^k of the cases), so their tests are left out.  That needs a
// matrix that is a rotation to 10^-5 and node corners that are exact; other
// objects run every test: it takes a node's edges for the normals of its faces,
// and where they meet at other angles it separates clusters well inside a large
// node.  With all products of columns within 10^-5 a face leans by less than
// 2 x 3 10^-5 x 8192 = 0.5 over a node's side, half the margin (10^-3 leant by 16
// at 2^14 and kept clusters that the test drops).
// 386k clusters at 4096^3, both kernels: 90 us, against 385 with every test and a
// thread per cluster; with a dirty map (8 moved objects) 83 -> 27 us.
__global__ void __launch_bounds__(128) k_svo_test_pairs(
    const tgx_object* __restrict__ objects, const float4* __restrict__ inv, const uint32_t* __restrict__ cp_obj, float mnx,
    float mny, float mnz, uint32_t L, uint32_t B, uint32_t* __restrict__ table, SvoPair* __restrict__ pairs,
    uint32_t* __restrict__ marked, uint32_t pair_capacity, uint32_t* __restrict__ counters)
{
    pdl_wait();
    const uint32_t n = min(counters[S_CAND], pair_capacity), lane = threadIdx.x & 31u;
    const float mn[3] = {mnx, mny, mnz};
    const float ext = (float)(1u << L);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < n; i0 += stride) {
        const uint32_t i = i0 + lane;
        bool pass = i < n;
        uint32_t blk = 0;
        if (pass) {
            const SvoPair pr = pairs[i];
            blk = pr.block;
            const uint32_t bx = blk % B, by = (blk / B) % B, bz = blk / (B * B);
            const uint32_t po = cp_obj[pr.cluster_pointer];
            const tgx_object& od = objects[po];
            const uint32_t rel = pr.cluster_pointer - od.first_cluster_pointer;
            float lo[3], hi[3], ws2ms[16];
            int b0[3], b1[3];
            cluster_blocks(od, rel, mn, B, lo, hi, b0, b1);
            const float4 c0 = inv[4u * po], c1 = inv[4u * po + 1u], c2 = inv[4u * po + 2u], c3 = inv[4u * po + 3u];
            if (c0.x == c0.x) {
                float off[3], ohe[3];
                cluster_offsets(od, rel, off, ohe);
                const float s3[3] = {xadd(ohe[0], -off[0]), xadd(ohe[1], -off[1]), xadd(ohe[2], -off[2])};
                dm4_ws2ms(c0, c1, c2, c3, s3, od.translation, ws2ms);
            } else {
                svo_ws2ms(od, rel, ws2ms);
            }
            // whether nodes around the cluster can be passed without the test, and the margin they need
            bool skip = od.rotation[15] == 1.0f;
            float margin = 0.0f;
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float* p = od.rotation + 4 * r;
#pragma unroll
                for (int j = 0; j <= r; j++) {
                    const float* q = od.rotation + 4 * j;
                    skip = skip && fabsf(p[0] * q[0] + p[1] * q[1] + p[2] * q[2] - (r == j ? 1.0f : 0.0f)) <= 1e-5f;
                }
                // the last column and row are those of a rotation; node corners below 2^24 are exact
                skip = skip && p[3] == 0.0f && od.rotation[12 + r] == 0.0f && fabsf(mn[r]) + ext <= 16777216.0f;
                margin = fmaxf(margin, 1.0f + 2e-5f * (fabsf(lo[r]) + fabsf(hi[r]) + fabsf(mn[r]) + ext + fabsf(od.translation[r])));
            }
            // walk the reference's recursion from the root to this block
            dv3 pmin = dv3{mnx, mny, mnz};
            dv3 pmax = dv3{xadd(mnx, ext), xadd(mny, ext), xadd(mnz, ext)};
            for (int lev = (int)L - 1; lev >= 5; lev--) {
                const dv3 ce = dv3{xmul(xsub(pmax.x, pmin.x), 0.5f), xmul(xsub(pmax.y, pmin.y), 0.5f),
                                   xmul(xsub(pmax.z, pmin.z), 0.5f)};
                const uint32_t sh = (uint32_t)lev - 5;
                const uint32_t cx = (bx >> sh) & 1u, cy = (by >> sh) & 1u, cz = (bz >> sh) & 1u;
                pmin = dv3{xadd(pmin.x, xmul((float)cx, ce.x)), xadd(pmin.y, xmul((float)cy, ce.y)),
                           xadd(pmin.z, xmul((float)cz, ce.z))};
                pmax = dv3{xadd(pmin.x, ce.x), xadd(pmin.y, ce.y), xadd(pmin.z, ce.z)};
                const bool holds = skip && lo[0] - margin >= pmin.x && lo[1] - margin >= pmin.y && lo[2] - margin >= pmin.z &&
                                   hi[0] + margin <= pmax.x && hi[1] + margin <= pmax.y && hi[2] + margin <= pmax.z;
                if (pass && !holds) {
                    dv3 bc[8];
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        bc[k] = mulv4p(ws2ms, (k & 1) ? pmax.x : pmin.x, (k & 2) ? pmax.y : pmin.y,
                                       (k & 4) ? pmax.z : pmin.z);
                    pass = aabb_obb(bc);
                }
            }
            if (!pass) pairs[i].block = kNoBlock;
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, pass);
        if (lane == 0u && mask) atomicAdd(&counters[S_PAIRS], (uint32_t)__popc(mask));
        // a read before the swap: most blocks are marked by an earlier pair
        if (pass && *(volatile uint32_t*)&table[blk] == 0u && atomicCAS(&table[blk], 0u, kMark) == 0u)
            marked[atomicAdd(&counters[S_MARKED], 1u)] = blk;   // no more blocks than pairs: the list holds them
    }
}

// ---------------------------------------------------------------------------
// 2. slot allocation
// ---------------------------------------------------------------------------

// Marked block m of n takes a slot from the end of the free list first
// (free[n_free-1], free[n_free-2], ...), then fresh slots from `next_slot` on.
// The table entry holds m, marked, until k_svo_publish puts the slot there: the
// passes between group the pairs by m.
__global__ void __launch_bounds__(256) k_svo_alloc(uint32_t* __restrict__ table, const uint32_t* __restrict__ marked,
                                                  uint32_t n, const uint32_t* __restrict__ free_list, uint32_t n_free,
                                                  uint32_t next_slot, uint32_t* __restrict__ slots,
                                                  uint32_t* __restrict__ slot_block, uint32_t* __restrict__ nonempty,
                                                  uint32_t* __restrict__ cnt)
{
    pdl_wait();
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    const uint32_t blk = marked[m];
    const uint32_t slot = m < n_free ? free_list[n_free - 1u - m] : next_slot + (m - n_free);
    table[blk] = kMarked | m;
    slots[m] = slot;
    slot_block[slot] = blk;
    nonempty[slot] = 0u;
    cnt[m] = 0u;
}

// ---------------------------------------------------------------------------
// 3. voxelisation: one warp per (cluster, block) pair
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t trim_u32(float v) { return v > 0.0f ? (uint32_t)v : 0u; }

// max of a 16-bit code in place in shared memory (CAS on the containing word)
__device__ __forceinline__ void smem_max_u16(uint32_t* words, uint32_t idx, uint32_t val)
{
    uint32_t* base = words + (idx >> 1);
    const uint32_t shift = (idx & 1u) ? 16u : 0u;
    uint32_t old = *base;
    for (int guard = 0; guard < 1 << 20; guard++) {
        if (((old >> shift) & 0xffffu) >= val) return;
        const uint32_t nv = (old & ~(0xffffu << shift)) | (val << shift);
        const uint32_t prev = atomicCAS(base, old, nv);
        if (prev == old) return;
        old = prev;
    }
}

// 3a. the n candidates that passed grouped by their (marked) block: counts, a
// range each, placement.
// The order of the ranges is free, so a block's range comes from a counter
// (one atomic per warp) instead of a scan.
__global__ void __launch_bounds__(256) k_svo_pair_count(const SvoPair* __restrict__ pairs, uint32_t n,
                                                       const uint32_t* __restrict__ table, uint32_t* __restrict__ cnt)
{
    pdl_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t blk = pairs[i].block;
        if (blk != kNoBlock) atomicAdd(&cnt[table[blk] & ~kMarked], 1u);
    }
}

__global__ void __launch_bounds__(256) k_svo_pair_ranges(const uint32_t* __restrict__ cnt, uint32_t n,
                                                        uint32_t* __restrict__ total, uint32_t* __restrict__ off,
                                                        uint32_t* __restrict__ cursor)
{
    pdl_wait();
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const uint32_t c = m < n ? cnt[m] : 0u;
    uint32_t incl = c;
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    uint32_t base = 0;
    if (lane == 31u && incl) base = atomicAdd(total, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (m < n) off[m] = cursor[m] = base + incl - c;
}

// 3b. voxelisation: one CTA per marked block.  Its warps take the block's
// (cluster, block) pairs; every set voxel goes into the CTA's shared image of
// the block and its material code into the shared material grid, then the
// block is written out whole, coalesced, with no global atomics.

// A pair as its warp reads it: the block's corners in cluster space and the
// voxel range of the block that the cluster can touch -- the trimmed range of
// tg__construct_leaf_node (tg_sparse_voxel_octree.c:180-226).
struct alignas(16) PairRec
{
    float bc[24];                // the 8 corners (x, y, z), corner k = (k & 1, k & 2, k & 4)
    uint32_t lo, hi;             // x0 | y0 << 8 | z0 << 16 and x1 | y1 << 8 | z1 << 16
    uint32_t ci, lut;            // cluster index; the object's LUT << 8, bit 31: not plain (below)
};
static_assert(sizeof(PairRec) == 112, "seven 16-byte shared loads");

// `plain`: the block side is exactly 32 (min not so large that min + extent rounds)
// and no corner coordinate is NaN or beyond 10^6, which the row loop's arithmetic
// needs.  A pair whose trimmed range is empty has lo = hi = 0.
__device__ __forceinline__ void pair_setup(const tgx_object* __restrict__ objects,
                                           const uint32_t* __restrict__ cluster_pointers,
                                           const uint32_t* __restrict__ c2o, const SvoPair& pr, float mnx, float mny,
                                           float mnz, uint32_t B, PairRec* __restrict__ out)
{
    const uint32_t cp = pr.cluster_pointer;
    const uint32_t ci = cluster_pointers[cp];
    const tgx_object& od = objects[c2o[ci]];
    const uint32_t rel = cp - od.first_cluster_pointer;
    const uint32_t bx = pr.block % B, by = (pr.block / B) % B, bz = pr.block / (B * B);
    // block box: same values the recursion produces (exact powers of two)
    const dv3 pmin = dv3{xadd(mnx, (float)(bx * kBlockSide)), xadd(mny, (float)(by * kBlockSide)),
                         xadd(mnz, (float)(bz * kBlockSide))};
    const dv3 pmax = dv3{xadd(pmin.x, 32.0f), xadd(pmin.y, 32.0f), xadd(pmin.z, 32.0f)};
    const dv3 pext = sub3(pmax, pmin);
    float cs2ws[16], ws2cs[16];
    svo_cs2ws(od, rel, cs2ws);
    dv3 cw[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
        cw[k] = mulv4p(cs2ws, (k & 1) ? 8.0f : 0.0f, (k & 2) ? 8.0f : 0.0f, (k & 4) ? 8.0f : 0.0f);
    // :180-194 -- note corner 2 twice, corner 3 never
    auto vmin = [](dv3 p, dv3 q) { return dv3{p.x < q.x ? p.x : q.x, p.y < q.y ? p.y : q.y, p.z < q.z ? p.z : q.z}; };
    auto vmax = [](dv3 p, dv3 q) { return dv3{p.x > q.x ? p.x : q.x, p.y > q.y ? p.y : q.y, p.z > q.z ? p.z : q.z}; };
    const dv3 min_c = vmin(vmin(vmin(cw[0], cw[1]), vmin(cw[2], cw[2])), vmin(vmin(cw[4], cw[6]), vmin(cw[5], cw[7])));
    const dv3 max_c = vmax(vmax(vmax(cw[0], cw[1]), vmax(cw[2], cw[2])), vmax(vmax(cw[4], cw[6]), vmax(cw[5], cw[7])));
    const dv3 tmin = vmax(pmin, dv3{floorf(min_c.x), floorf(min_c.y), floorf(min_c.z)});
    const dv3 tmax = vmin(pmax, dv3{ceilf(max_c.x), ceilf(max_c.y), ceilf(max_c.z)});
    const uint32_t x0 = trim_u32(xsub(tmin.x, pmin.x)), y0 = trim_u32(xsub(tmin.y, pmin.y));
    const uint32_t x1 = trim_u32(xsub(tmax.x, pmin.x)), y1 = trim_u32(xsub(tmax.y, pmin.y));
    const uint32_t z0 = trim_u32(xsub(tmin.z, pmin.z)), z1 = trim_u32(xsub(tmax.z, pmin.z));
    float4* const q4 = reinterpret_cast<float4*>(out);
    if (x0 >= x1 || y0 >= y1 || z0 >= z1) {
        q4[6] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
    dm4_inverse(cs2ws, ws2cs);
    float bc[24];
    bool plain = pext.x == 32.0f && pext.y == 32.0f && pext.z == 32.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const dv3 c = mulv4p(ws2cs, (q & 1) ? pmax.x : pmin.x, (q & 2) ? pmax.y : pmin.y, (q & 4) ? pmax.z : pmin.z);
        bc[3 * q] = c.x; bc[3 * q + 1] = c.y; bc[3 * q + 2] = c.z;
        plain = plain && fabsf(c.x) <= 1e6f && fabsf(c.y) <= 1e6f && fabsf(c.z) <= 1e6f;
    }
#pragma unroll
    for (int q = 0; q < 6; q++) q4[q] = make_float4(bc[4 * q], bc[4 * q + 1], bc[4 * q + 2], bc[4 * q + 3]);
    reinterpret_cast<uint4*>(out)[6] = make_uint4(x0 | y0 << 8 | z0 << 16, x1 | y1 << 8 | z1 << 16, ci,
                                                  ((od.lut_idx << 8) & 0x7fffffffu) | (plain ? 0u : 0x80000000u));
}

// The pairs' records, those of a block side by side: a thread per pair.
__global__ void __launch_bounds__(128) k_svo_pair_fill(const SvoPair* __restrict__ pairs, uint32_t n,
                                                      const uint32_t* __restrict__ table, uint32_t* __restrict__ cursor,
                                                      const tgx_object* __restrict__ objects,
                                                      const uint32_t* __restrict__ cluster_pointers,
                                                      const uint32_t* __restrict__ c2o, float mnx, float mny, float mnz,
                                                      uint32_t B, PairRec* __restrict__ recs)
{
    pdl_wait();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const SvoPair pr = pairs[i];
        if (pr.block == kNoBlock) continue;
        pair_setup(objects, cluster_pointers, c2o, pr, mnx, mny, mnz, B, recs + atomicAdd(&cursor[table[pr.block] & ~kMarked], 1u));
    }
}

// The z- and y-lerps of tg__construct_leaf_node for row (iy, iz) of a block:
// the row's two ends p0, p1 in cluster space (they depend on the row only)
__device__ __forceinline__ void row_ends(const float* bc, float ty, float tz, float p0[3], float p1[3])
{
    const float omtz = xsub(1.0f, tz), omty = xsub(1.0f, ty);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float z0 = xadd(xmul(omtz, bc[c]), xmul(tz, bc[12 + c]));
        const float z1 = xadd(xmul(omtz, bc[3 + c]), xmul(tz, bc[15 + c]));
        const float z2 = xadd(xmul(omtz, bc[6 + c]), xmul(tz, bc[18 + c]));
        const float z3 = xadd(xmul(omtz, bc[9 + c]), xmul(tz, bc[21 + c]));
        p0[c] = xadd(xmul(omty, z0), xmul(ty, z2));
        p1[c] = xadd(xmul(omty, z1), xmul(ty, z3));
    }
}

// A pair that is not plain (see pair_setup), by one warp: conversions, block sides
// that round, NaN coordinates (which pass the range test and read voxel 0 of
// their axis), each voxel merged by itself.
template <bool kMat>
__device__ __noinline__ void voxelize_any(const float* bc, uint32_t x0, uint32_t x1, uint32_t y0, uint32_t z0, uint32_t ny,
                                          uint32_t rows, float rny, uint32_t lut, const uint32_t* cw, const uint8_t* cm,
                                          float mnx, float mny, float mnz, uint32_t B, uint32_t block, uint32_t word0,
                                          uint32_t n_words, uint32_t* img, uint32_t* smat)
{
    const uint32_t bx = block % B, by = (block / B) % B, bz = block / (B * B);
    const float px = xadd(mnx, (float)(bx * kBlockSide)), py = xadd(mny, (float)(by * kBlockSide)),
                pz = xadd(mnz, (float)(bz * kBlockSide));
    const dv3 pext = dv3{xsub(xadd(px, 32.0f), px), xsub(xadd(py, 32.0f), py), xsub(xadd(pz, 32.0f), pz)};
    for (uint32_t row = threadIdx.x & 31u; row < rows; row += 32) {
        const uint32_t q = (uint32_t)(((float)row + 0.5f) * rny);
        const uint32_t iy = y0 + (row - q * ny), iz = z0 + q;
        float p0[3], p1[3];
        row_ends(bc, xdiv(xadd((float)iy, 0.5f), pext.y), xdiv(xadd((float)iz, 0.5f), pext.z), p0, p1);
        const float row_base = xadd(xmul(xmul(pext.x, pext.y), (float)iz), xmul(pext.x, (float)iy));
        for (uint32_t ix = x0; ix < x1; ix++) {
            const float tx = xdiv(xadd((float)ix, 0.5f), pext.x);
            const float omtx = xsub(1.0f, tx);
            const float cx = xadd(xmul(omtx, p0[0]), xmul(tx, p1[0]));
            const float cy = xadd(xmul(omtx, p0[1]), xmul(tx, p1[1]));
            const float cz = xadd(xmul(omtx, p0[2]), xmul(tx, p1[2]));
            if (cx < 0.0f || cx >= 8.0f || cy < 0.0f || cy >= 8.0f || cz < 0.0f || cz >= 8.0f) continue;
            const uint32_t rvi = 64u * (uint32_t)cz + 8u * (uint32_t)cy + (uint32_t)cx;
            if (!(cw[rvi >> 5] & (1u << (rvi & 31u)))) continue;
            const uint32_t bvi = (uint32_t)xadd(row_base, (float)ix);
            if ((bvi >> 5) - word0 >= n_words) continue;   // a side that rounds above 32
            atomicOr(&img[(bvi >> 5) - word0], 1u << (bvi & 31u));
            if (kMat) smem_max_u16(smat, bvi - word0 * 32u, ((lut | cm[rvi]) + 1u) & 0xffffu);
        }
    }
}

// The masks of the 4^3 and 8^3 cells of 8 layers of a block (layers 8 u .. 8 u + 7,
// rows: their bit words), by one warp (lane y reads the rows (y, z)).  Sets
// *nonempty (zero before) when they hold a voxel.
__device__ __forceinline__ void layer_masks(const uint32_t* rows, uint32_t u, uint32_t* __restrict__ sb,
                                            uint32_t* __restrict__ nonempty)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t n4[2] = {0u, 0u};   // per 4 layers: which 4-voxel x-groups of row y hold a voxel
#pragma unroll
    for (int z = 0; z < 8; z++) {
        const uint32_t row = rows[z * 32 + lane];
        uint32_t f = row | row >> 1;
        f = (f | f >> 2) & 0x11111111u;   // bit 4 gx: some of the group's four voxels
        f = (f | f >> 3) & 0x03030303u;   // gather the eight bits
        f = (f | f >> 6) & 0x000f000fu;
        n4[z >> 2] |= (f | f >> 12) & 0xffu;
    }
    if (__any_sync(0xffffffffu, (n4[0] | n4[1]) != 0u) && lane == 0u) *nonempty = 1u;
    // 4^3 cells: bit ((cz * 8 + cy) * 8 + cx), cy = lane / 4
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t b = n4[h];
        b |= __shfl_xor_sync(0xffffffffu, b, 1);
        b |= __shfl_xor_sync(0xffffffffu, b, 2);
        uint32_t w = (lane & 3u) == 0u ? b << (((lane >> 2) & 3u) * 8u) : 0u;
        w |= __shfl_xor_sync(0xffffffffu, w, 4);
        w |= __shfl_xor_sync(0xffffffffu, w, 8);
        if ((lane & 15u) == 0u) sb[(2u * u + h) * 2u + (lane >> 4)] = w;
    }
    // 8^3 cells: bit ((cz * 4 + cy) * 4 + cx), cy = lane / 8: 16 bits for cz = u
    const uint32_t b = n4[0] | n4[1];
    uint32_t c3 = 0;
#pragma unroll
    for (int cx = 0; cx < 4; cx++) c3 |= ((b >> (2 * cx)) & 3u) ? (1u << cx) : 0u;
    c3 |= __shfl_xor_sync(0xffffffffu, c3, 1);
    c3 |= __shfl_xor_sync(0xffffffffu, c3, 2);
    c3 |= __shfl_xor_sync(0xffffffffu, c3, 4);
    uint32_t w8 = (lane & 7u) == 0u ? c3 << ((lane >> 3) * 4u) : 0u;
    w8 |= __shfl_xor_sync(0xffffffffu, w8, 8);
    w8 |= __shfl_xor_sync(0xffffffffu, w8, 16);
    if (lane == 0) reinterpret_cast<uint16_t*>(sb + 16)[u] = (uint16_t)w8;
}

// Bound by instruction issue.  The pairs are taken kVoxRound at a time: their
// records (k_svo_pair_fill: matrices, trimmed range, corners) are copied to
// shared memory, their voxel counts sorted by a warp bitonic sort per 32,
// heaviest first; then the warps take pairs in that order from a shared counter,
// the next one whenever they finish one.  Within a pair, a lane takes a row
// (iy, iz) of the range: the z- and y-lerps once per row; the x-lerp, the
// [0, 8)^3 test and the bit fetch per voxel, floor and range test in the bits of
// c + 1.5 * 2^23 rounded down (no conversion); the row's bits in one atomicOr on
// its word of the image.  Material codes are stored plainly.  A voxel that two
// pairs set (objects that overlap) needs the larger code: the second atomicOr
// finds its bit, marks it in s_conf, and blocks with marks go over their pairs
// once more for those voxels alone, with a 16-bit max.  The order of the pairs
// changes no bit.
// 512 objects, 4096^3, 565k pairs in 18.4k blocks: 2350 us with a warp per pair
// doing its set-up, 1430 with a lane per pair in the CTA's first warp (the
// others waited for it), 1245 with the records made by the pass that groups the
// pairs (29 us, 13 before).  Loading the next pair's bits ahead into registers:
// 1460 (spills); into L1: no change.
constexpr uint32_t kVoxRound = 128;     // pairs in shared memory at a time

template <bool kMat, uint32_t kSlabs>
__global__ void __launch_bounds__(32 * kWarpsPerVoxCta, 2) k_svo_voxelize(
    const uint32_t* __restrict__ bits, const PairRec* __restrict__ recs, const uint32_t* __restrict__ off,
    const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ marked, const uint32_t* __restrict__ slots,
    uint32_t* __restrict__ pool, uint32_t* __restrict__ sub, uint32_t* __restrict__ nonempty,
    const uint8_t* __restrict__ material, uint16_t* __restrict__ mat_pool, float mnx, float mny, float mnz, uint32_t B)
{
    pdl_wait();
    constexpr uint32_t kLayers = 32u / kSlabs, kWords = kBlockWords / kSlabs;
    extern __shared__ __align__(16) uint32_t s_blk[];   // the slab's bit words, then 16 words of u16 codes for each
    __shared__ PairRec s_rec[kVoxRound];
    __shared__ uint32_t s_cw[kWarpsPerVoxCta][16];       // each warp's current cluster bits
    __shared__ uint4 s_cm[kMat ? kWarpsPerVoxCta : 1][32];  // and its 512 material bytes
    __shared__ uint32_t s_conf[kMat ? kWords : 1];       // voxels more than one pair set
    __shared__ uint8_t s_order[kVoxRound];               // per chunk of 32: the round's pairs, heaviest first (255: none)
    __shared__ uint32_t s_next;                          // the next entry of s_order to take
    uint32_t* img = s_blk;
    uint16_t* smat = reinterpret_cast<uint16_t*>(s_blk + kWords);
    const uint32_t m = blockIdx.x / kSlabs, slab0 = (blockIdx.x % kSlabs) * kLayers;   // the slab's first layer
    const uint32_t slot = slots[m];
    const uint32_t pb = off[m], pe = pb + cnt[m];   // at least one pair
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    // the end of a pair's layers inside the slab (whole blocks: as the record has it)
    auto slab_end = [&](uint32_t z1) { return kSlabs == 1u ? z1 : min(z1, slab0 + kLayers); };
    bool again = false;                  // the pass over the doubly set voxels (the same in every thread)
    for (;;) {
        bool conflict = false;           // this thread met a doubly set voxel
        for (uint32_t r0 = pb; r0 < pe; r0 += kVoxRound) {
            const uint32_t np = min(kVoxRound, pe - r0);
            const uint32_t n_chunks = (np + 31u) / 32u;
            __syncthreads();   // the previous round's records are consumed
            if (wid < n_chunks) {
                const uint32_t i = wid * 32u + lane;
                // key: voxel count in the slab (pairs past the end sort last); value: pair in the round
                int32_t key = -1;
                uint32_t idx = i;
                if (i < np) {
                    const uint2 range = *reinterpret_cast<const uint2*>(&recs[r0 + i].lo);
                    const uint32_t x = (range.y & 255u) - (range.x & 255u), y = ((range.y >> 8) & 255u) - ((range.x >> 8) & 255u);
                    const uint32_t z0 = max(range.x >> 16, slab0), z1 = slab_end(range.y >> 16);
                    key = z0 < z1 ? (int32_t)(x * y * (z1 - z0)) : 0;
                }
                // ascending bitonic sort over the warp's 32 lanes
#pragma unroll
                for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
                    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                        const int32_t ok = __shfl_xor_sync(0xffffffffu, key, j);
                        const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, j);
                        const bool lower = (lane & j) == 0u, asc = (lane & k) == 0u;
                        const bool take = (asc == lower) ? (ok < key) : (ok > key);
                        if (take) { key = ok; idx = oi; }
                    }
                }
                // descending rank 31 - lane; pairs without voxels are left out
                s_order[wid * 32u + (31u - lane)] = (uint8_t)(key > 0 ? idx : 255u);
            }
            for (uint32_t k = threadIdx.x; k < np * 7u; k += blockDim.x)
                reinterpret_cast<uint4*>(s_rec)[k] = reinterpret_cast<const uint4*>(recs + r0)[k];
            if (r0 == pb && !again) {   // clear the block
                for (uint32_t k = threadIdx.x; k < kWords * (kMat ? 17u : 1u) / 4u; k += blockDim.x)
                    reinterpret_cast<uint4*>(s_blk)[k] = make_uint4(0u, 0u, 0u, 0u);
                if (kMat)
                    for (uint32_t k = threadIdx.x; k < kWords; k += blockDim.x) s_conf[k] = 0u;
            }
            if (threadIdx.x == 0) s_next = 0u;
            __syncthreads();
            for (;;) {
                uint32_t item = 0;
                if (lane == 0) item = atomicAdd(&s_next, 1u);
                item = __shfl_sync(0xffffffffu, item, 0);
                if (item >= n_chunks * 32u) break;
                const uint32_t k = s_order[item];
                if (k == 255u) continue;
                float bc[24];
                const float4* rq = reinterpret_cast<const float4*>(&s_rec[k]);
#pragma unroll
                for (int q = 0; q < 6; q++) {
                    const float4 t = rq[q];
                    bc[4 * q] = t.x; bc[4 * q + 1] = t.y; bc[4 * q + 2] = t.z; bc[4 * q + 3] = t.w;
                }
                const uint4 rm = *reinterpret_cast<const uint4*>(&s_rec[k].lo);
                const uint32_t x0 = rm.x & 255u, y0 = (rm.x >> 8) & 255u, z0 = max(rm.x >> 16, slab0);
                const uint32_t x1 = rm.y & 255u, ny = ((rm.y >> 8) & 255u) - y0, nz = slab_end(rm.y >> 16) - z0;
                const uint32_t lut = rm.w & 0x7fffffffu;   // << 8 already
                // the cluster's 16 bit words and 512 material bytes
                __syncwarp();
                if (lane < 16) s_cw[wid][lane] = bits[(uint64_t)rm.z * 16u + lane];
                if (kMat) s_cm[wid][lane] = reinterpret_cast<const uint4*>(material + (uint64_t)rm.z * 512u)[lane];
                __syncwarp();
                const uint32_t* cw = s_cw[wid];
                const uint8_t* cm = reinterpret_cast<const uint8_t*>(s_cm[wid]);
                // row -> (iy, iz) without integer division: row < 2^10 and ny <= 32, so
                // (row + 0.5) / ny lies at least 0.5 / ny from an integer while the float
                // product's error stays far below that
                const uint32_t rows = ny * nz;
                const float rny = 1.0f / (float)ny;
                if (rm.w >> 31) {
                    // (again as well: it only takes maxima)
                    voxelize_any<kMat>(bc, x0, x1, y0, z0, ny, rows, rny, lut, cw, cm, mnx, mny, mnz, B,
                                       marked[m], slab0 * 32u, kWords, img, s_blk + kWords);
                    continue;
                }
                for (uint32_t row = lane; row < rows; row += 32) {
                    const uint32_t q = (uint32_t)(((float)row + 0.5f) * rny);
                    const uint32_t iy = y0 + (row - q * ny), iz = z0 + q;
                    const uint32_t word = (iz - slab0) * 32u + iy;   // the row's word of the image
                    uint32_t want = 0xffffffffu;
                    if (again) {
                        want = s_conf[word];
                        if (!want) continue;
                    }
                    // (i + 0.5) / 32 is an exact scaling: the reciprocal multiply gives the same bits
                    float p0[3], p1[3];
                    row_ends(bc, xmul(xadd((float)iy, 0.5f), 0.03125f), xmul(xadd((float)iz, 0.5f), 0.03125f), p0, p1);
                    // tx = (ix + 0.5) / 32 is a multiple of 2^-6 below 1, so adding 1/32 per voxel is exact
                    float tx = xmul(xadd((float)x0, 0.5f), 0.03125f);
                    uint16_t* const codes = smat + word * 32u;
                    uint32_t mask = 0;
                    for (uint32_t ix = x0; ix < x1; ix++, tx = xadd(tx, 0.03125f)) {
                        const float omtx = xsub(1.0f, tx);
                        uint32_t f[3];   // bits of 1.5 * 2^23 + floor(c)
#pragma unroll
                        for (int c = 0; c < 3; c++)
                            f[c] = __float_as_uint(__fadd_rd(xadd(xmul(omtx, p0[c]), xmul(tx, p1[c])), 12582912.0f));
                        if (((f[0] | f[1] | f[2]) & ~7u) != 0x4B400000u) continue;   // some floor outside 0..7
                        const uint32_t rvi = (64u * f[2] + 8u * f[1] + f[0]) & 511u;
                        if (!((cw[rvi >> 5] >> (rvi & 31u)) & 1u)) continue;
                        if (!again) {
                            mask |= 1u << ix;
                            if (kMat) codes[ix] = (uint16_t)((lut | cm[rvi]) + 1u);
                        } else if ((want >> ix) & 1u) {
                            smem_max_u16(s_blk + kWords, word * 32u + ix, ((lut | cm[rvi]) + 1u) & 0xffffu);
                        }
                    }
                    if (mask) {
                        if (kMat) {
                            const uint32_t twice = atomicOr(&img[word], mask) & mask;
                            if (twice) { atomicOr(&s_conf[word], twice); conflict = true; }
                        } else {
                            atomicOr(&img[word], mask);
                        }
                    }
                }
            }
        }
        if (!kMat || again || !__syncthreads_or(conflict)) break;
        // doubly set voxels: forget their codes, then take the maximum over the pairs
        for (uint32_t w = wid; w < kWords; w += kWarpsPerVoxCta)
            if ((s_conf[w] >> lane) & 1u) smat[w * 32u + lane] = 0u;
        again = true;
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(pool + (uint64_t)slot * kBlockWords + slab0 * 32u);
    for (uint32_t k = threadIdx.x; k < kWords / 4u; k += blockDim.x) dst[k] = reinterpret_cast<const uint4*>(img)[k];
    if (kMat) {
        uint4* md = reinterpret_cast<uint4*>(mat_pool + (uint64_t)slot * 32768u + slab0 * 1024u);
        for (uint32_t k = threadIdx.x; k < kWords * 4u; k += blockDim.x) md[k] = reinterpret_cast<const uint4*>(smat)[k];
    }
    // the occupancy masks of every 8 layers, from the image while it is here
    if (wid < 4u / kSlabs) layer_masks(img + wid * 256u, slab0 / 8u + wid, sub + (uint64_t)slot * 32u, &nonempty[slot]);
}

// ---------------------------------------------------------------------------
// 4. occupancy pyramid
// ---------------------------------------------------------------------------

// The slots of the marked blocks go into the table.
__global__ void __launch_bounds__(256) k_svo_publish(uint32_t* __restrict__ table, const uint32_t* __restrict__ marked,
                                                    const uint32_t* __restrict__ slots, uint32_t n)
{
    pdl_wait();
    const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) table[marked[m]] = slots[m] + 1u;
}

// One thread per slot: a slot whose block holds a voxel sets its bit level by
// level up to the first one that is set already (whoever set that one goes on
// to the coarser ones), so the few words of the coarse levels do not take an
// atomic from every block.  The words are zero before.
__global__ void __launch_bounds__(256) k_svo_pyramid(const uint32_t* __restrict__ slot_block, uint32_t n_slots,
                                                    const uint32_t* __restrict__ nonempty, uint32_t* occ,
                                                    const uint64_t* __restrict__ occ_off, uint32_t n_levels, uint32_t B,
                                                    uint32_t* __restrict__ counters)
{
    pdl_wait();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t i = slot < n_slots ? slot_block[slot] : 0xffffffffu;
    const bool any = i != 0xffffffffu && nonempty[slot] != 0u;
    const uint32_t mask = __ballot_sync(0xffffffffu, any);
    if ((threadIdx.x & 31u) == 0u && mask) atomicAdd(&counters[S_NONEMPTY], (uint32_t)__popc(mask));
    if (!any) return;
    const uint32_t bx = i % B, by = (i / B) % B, bz = i / (B * B);
    for (uint32_t s = 0; s < n_levels; s++) {
        const uint32_t n = B >> s;
        const uint64_t idx = ((uint64_t)(bz >> s) * n + (by >> s)) * n + (bx >> s);
        uint32_t* w = &occ[occ_off[s] + (idx >> 5)];
        const uint32_t bit = 1u << (idx & 31u);
        if ((*(volatile uint32_t*)w & bit) || (atomicOr(w, bit) & bit)) break;
    }
}

// ---------------------------------------------------------------------------
// incremental update: blocks a moved object covered before or covers now
// ---------------------------------------------------------------------------

// Conservative world box of every non-empty cluster of one object -- the box
// k_svo_candidates selects blocks with -- marked into the dirty-block map (a
// bit per block).  The CTAs of a grid column share the object's clusters.
__device__ void mark_object_blocks(const tgx_object& od, const uint32_t* __restrict__ cp_obj, const float mn[3], uint32_t B,
                                   uint32_t* __restrict__ dirty)
{
    const uint32_t n = od.n_cluster_pointers_per_dim[0] * od.n_cluster_pointers_per_dim[1] * od.n_cluster_pointers_per_dim[2];
    for (uint32_t rel = blockIdx.y * blockDim.x + threadIdx.x; rel < n; rel += gridDim.y * blockDim.x) {
        if (cp_obj[od.first_cluster_pointer + rel] >> 31) continue;   // no set voxel
        float lo[3], hi[3];
        int b0[3], b1[3];
        if (!cluster_blocks(od, rel, mn, B, lo, hi, b0, b1)) continue;
        for (int bz = b0[2]; bz <= b1[2]; bz++)
            for (int by = b0[1]; by <= b1[1]; by++)
                for (int bx = b0[0]; bx <= b1[0]; bx++) {
                    const uint32_t blk = ((uint32_t)bz * B + (uint32_t)by) * B + (uint32_t)bx;
                    atomicOr(&dirty[blk >> 5], 1u << (blk & 31u));
                }
    }
}

__device__ __forceinline__ bool same_record(const tgx_object& x, const tgx_object& y)
{
    const uint32_t* a = reinterpret_cast<const uint32_t*>(&x);
    const uint32_t* b = reinterpret_cast<const uint32_t*>(&y);
    bool same = true;
#pragma unroll
    for (int k = 0; k < (int)(sizeof(tgx_object) / 4); k++) same &= a[k] == b[k];
    return same;
}

// A grid column per object: when the scene's record differs from the one the
// SVO was built from, the blocks its clusters touched before (old record) and
// touch now (new record) become dirty.
__global__ void __launch_bounds__(128) k_svo_mark_dirty(const tgx_object* __restrict__ cur,
                                                       const tgx_object* __restrict__ built,
                                                       const uint32_t* __restrict__ cp_obj, float mnx, float mny,
                                                       float mnz, uint32_t B, uint32_t* __restrict__ dirty)
{
    pdl_wait();
    const tgx_object now = cur[blockIdx.x], was = built[blockIdx.x];
    if (same_record(now, was)) return;
    const float mn[3] = {mnx, mny, mnz};
    mark_object_blocks(was, cp_obj, mn, B, dirty);
    mark_object_blocks(now, cp_obj, mn, B, dirty);
}

// Every dirty block that holds a slot gives it back: the table entry is emptied
// and the slot goes on the free list (a thread per 32 blocks of the map).
// k_svo_candidates re-marks the block if any cluster still reaches it, and what
// a slot holds is written whole before it is used again.  Moved objects are
// counted and their records taken over, a thread each.
__global__ void __launch_bounds__(256) k_svo_release_dirty(uint32_t* __restrict__ table, uint64_t n_words,
                                                          const uint32_t* __restrict__ dirty, uint64_t n_table,
                                                          uint32_t* __restrict__ nonempty, uint32_t* __restrict__ slot_block,
                                                          uint32_t* __restrict__ free_tail,
                                                          const tgx_object* __restrict__ cur, tgx_object* __restrict__ built,
                                                          uint32_t n_objects, uint32_t* __restrict__ counters)
{
    pdl_wait();
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = t; w < n_words; w += stride) {
        uint32_t m = dirty[w];
        while (m) {
            const uint64_t i = w * 32u + (uint32_t)(__ffs((int)m) - 1);
            m &= m - 1u;
            const uint32_t tv = i < n_table ? table[i] : 0u;
            if (tv == 0u) continue;
            nonempty[tv - 1u] = 0u;
            slot_block[tv - 1u] = 0xffffffffu;
            table[i] = 0u;
            free_tail[atomicAdd(&counters[S_FREED], 1u)] = tv - 1u;
        }
    }
    for (uint64_t o = t; o < n_objects; o += stride) {
        const tgx_object now = cur[o];
        if (same_record(now, built[o])) continue;
        built[o] = now;
        atomicAdd(&counters[S_MOVED], 1u);
    }
}

// Table entries still marked after an overflowed candidate pass, or an update that
// failed, go back to empty.
__global__ void __launch_bounds__(256) k_svo_unmark(uint32_t* __restrict__ table, uint64_t n_table)
{
    pdl_wait();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_table; i += (uint64_t)gridDim.x * blockDim.x)
        if (table[i] & kMarked) table[i] = 0u;
}

// ... and the slots that it gave to blocks are nobody's: the pyramid pass goes by
// slots, and a traversal that its bits led into a block without an entry would
// read before the pool.
__global__ void __launch_bounds__(256) k_svo_drop_slots(const uint32_t* __restrict__ table, uint32_t n_slots,
                                                       uint32_t* __restrict__ slot_block, uint32_t* __restrict__ nonempty)
{
    pdl_wait();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n_slots) return;
    const uint32_t blk = slot_block[slot];
    if (blk == 0xffffffffu || table[blk] == slot + 1u) return;
    slot_block[slot] = 0xffffffffu;
    nonempty[slot] = 0u;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// The counters are an ordinary allocation, and the first to go: their cudaFree
// waits for all work on the device (other contexts may still traverse the SVO),
// which that of a pool array does not.  cudaDeviceSynchronize would wait too, but
// it fails, and ends the capture, while another thread captures a stream.
static void svo_free(tgx_svo* s)
{
    if (!s) return;
    cudaFree(s->d_counters);
    cudaFree(s->d_table);
    cudaFree(s->d_pool);
    cudaFree(s->d_sub);
    cudaFree(s->d_occ);
    cudaFree(s->d_nonempty);
    cudaFree(s->d_mat);
    cudaFree(s->d_free);
    cudaFree(s->d_slot_block);
    cudaFree(s->d_objs);
    delete s;
}

// An SVO's arrays come from a memory pool of the context that builds it, which
// keeps up to kSvoPoolKeep bytes of freed arrays for the next build and gives the
// rest back; these go with the context (an array still in use keeps its part
// alive), or sooner: on tgx_trim, and when an allocation of any context finds
// no room (tgx_malloc).  A build of 18.4k blocks with materials (1.3 GB) and its free
// took 1.1 ms in the driver's allocator beside 1.9 ms of GPU work.  That is saved
// where a context builds again after it closed an SVO; its first build still pays
// for the memory (first and later passes of a build, a frame and the free: 3.04 and
// 1.73 ms).  Nothing waits when a pool array is freed: svo_free and
// svo_resize_slots do before.
constexpr uint64_t kSvoPoolKeep = 4ull << 30;

static cudaError_t svo_malloc(tgx_ctx* c, void** p, uint64_t bytes)
{
    if (!c->svo_pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = c->device;
        cudaMemPool_t pool = nullptr;
        if (const cudaError_t e = cudaMemPoolCreate(&pool, &props); e != cudaSuccess) return e;
        uint64_t keep = kSvoPoolKeep;
        if (const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep); e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        c->svo_pool = pool;
        svo_pool_opened(pool);
    }
    const uint64_t n = std::max<uint64_t>(bytes, 1);
    cudaError_t e = cudaMallocFromPoolAsync(p, n, c->svo_pool, c->stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        svo_pools_trim();
        e = cudaMallocFromPoolAsync(p, n, c->svo_pool, c->stream);
    }
    return e;
}

// The pair storage: pairs, then as many words for the list of the marked blocks.
constexpr uint64_t kPairBytes = sizeof(SvoPair) + 4;
static uint32_t* svo_marked(tgx_ctx* c)
{
    return (uint32_t*)((SvoPair*)c->svo_pairs.ptr + c->svo_pairs.bytes / kPairBytes);
}

static uint64_t svo_device_bytes(const tgx_svo* s)
{
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    return n_table * 4 + (uint64_t)s->pool_cap * (kBlockWords * 4 + 128 + 4 + 4 + 4 + (s->d_mat ? 65536 : 0)) +
           s->occ_words * 4 + (uint64_t)s->n_objects * sizeof(tgx_object);
}

// Per-slot arrays (pool, sub masks, non-empty flags, free list, block indices,
// materials) sized for `cap` slots; the first `keep` slots are carried over.  The
// rest of the small arrays start zero (no block: ~0); pool and material slots are written whole
// by the voxeliser before anything reads them.
static tgx_status svo_resize_slots(tgx_ctx* c, tgx_svo* s, uint32_t cap, uint32_t keep, bool materials)
{
    struct Arr { void** p; uint64_t per_slot; };
    void* mat = s->d_mat;
    Arr arrs[6] = {{(void**)&s->d_pool, kBlockWords * 4}, {(void**)&s->d_sub, 128}, {(void**)&s->d_nonempty, 4},
                   {(void**)&s->d_free, 4}, {(void**)&s->d_slot_block, 4}, {&mat, 65536}};
    const int n_arr = materials ? 6 : 5;
    void *fresh[6] = {}, *wait = nullptr;
    for (int a = 0; a < n_arr; a++)
        if (svo_malloc(c, &fresh[a], (uint64_t)cap * arrs[a].per_slot) != cudaSuccess ||
            (a == 0 && s->d_pool && tgx_malloc(&wait, 256) != cudaSuccess)) {
            for (int k = 0; k <= a; k++) cudaFree(fresh[k]);
            cudaFree(wait);
            cudaGetLastError();
            tgx_set_error("tgx_svo: out of device memory for %u blocks", cap);
            return TGX_ERR_OUT_OF_MEMORY;
        }
    for (int a = 0; a < n_arr; a++) {
        const uint64_t kept = (uint64_t)keep * arrs[a].per_slot, total = (uint64_t)cap * arrs[a].per_slot;
        if (kept) TGX_CUDA(cudaMemcpyAsync(fresh[a], *arrs[a].p, kept, cudaMemcpyDeviceToDevice, c->stream));
        if (a != 0 && a != 5) TGX_CUDA(cudaMemsetAsync((char*)fresh[a] + kept, a == 4 ? 0xff : 0, total - kept, c->stream));
    }
    if (s->d_pool) {
        TGX_CUDA(cudaStreamSynchronize(c->stream));
        cudaFree(wait);   // for every stream, as in svo_free
    }
    for (int a = 0; a < n_arr; a++) {
        cudaFree(*arrs[a].p);
        *arrs[a].p = fresh[a];
    }
    s->d_mat = (uint16_t*)mat;
    s->pool_cap = cap;
    return TGX_OK;
}

// Candidate pass over every cluster pointer (only blocks marked in `dirty` when
// it is given), with the pair storage grown to the exact count and the pass
// rerun once when the first estimate was short.  The list of the marked blocks
// follows the pairs.  Leaves the counters on the host.
static tgx_status svo_candidates(tgx_ctx* c, tgx_svo* s, const tgx_scene* sc, const uint32_t* dirty, uint64_t cap)
{
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    uint32_t* counters = s->d_counters;
    for (int attempt = 0; attempt < 2; attempt++) {
        TGX_TRY(devbuf_reserve(c->svo_pairs, cap * kPairBytes));
        cap = c->svo_pairs.bytes / kPairBytes;   // svo_marked() places the list by the buffer's size
        TGX_CUDA(cudaMemsetAsync(counters + S_PAIRS, 0, 2 * 4, c->stream));   // pairs, marks
        TGX_CUDA(cudaMemsetAsync(counters + S_CAND, 0, 4, c->stream));
        if (sc->n_cluster_pointers) {
            const uint32_t cap32 = (uint32_t)std::min<uint64_t>(cap, 0xffffffffu);
            TGX_LAUNCH_PDL(c, TR_SVO_CANDIDATES, (sc->n_cluster_pointers + 127) / 128, 128, 0, k_svo_candidates, sc->d_objects,
                       sc->d_cp_obj, sc->n_cluster_pointers, s->mn[0], s->mn[1], s->mn[2], s->B, (SvoPair*)c->svo_pairs.ptr,
                       cap32, counters, c->d_status, dirty);
            TGX_LAUNCH_PDL(c, TR_SVO_CANDIDATES, (uint32_t)c->num_sms * 16, 128, 0, k_svo_test_pairs, sc->d_objects, sc->d_inv,
                       sc->d_cp_obj, s->mn[0], s->mn[1], s->mn[2], s->L, s->B, s->d_table, (SvoPair*)c->svo_pairs.ptr,
                       svo_marked(c), cap32, counters);
        }
        if (cudaMemcpyAsync(c->h_counter, counters, S_COUNT * 4, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
            cudaStreamSynchronize(c->stream) != cudaSuccess) {
            tgx_set_error("tgx_svo: %s", cudaGetErrorString(cudaGetLastError()));
            return TGX_ERR_CUDA;
        }
        const uint32_t n_cand = ((uint32_t*)c->h_counter)[S_CAND];
        if (n_cand <= cap) return TGX_OK;
        // the capacity error recorded by the first attempt is expected; clear it and the marks it left
        TGX_CUDA(cudaMemsetAsync(c->d_status, 0, sizeof(tgx_dev_status), c->stream));
        const uint32_t grid = (uint32_t)std::min<uint64_t>((n_table + 255) / 256, (uint64_t)c->num_sms * 32);
        TGX_LAUNCH_PDL(c, TR_SVO_ALLOC, grid, 256, 0, k_svo_unmark, s->d_table, n_table);
        cap = (uint64_t)n_cand + 1024;
    }
    tgx_set_error("tgx_svo: pair count grew between two identical passes");
    return TGX_ERR_CAPACITY;
}

// Zeroes the pyramid, and the counts of pair ranges handed out and of non-empty blocks.
static tgx_status svo_clear_pyramid(tgx_ctx* c, tgx_svo* s)
{
    TGX_CUDA(cudaMemsetAsync(s->d_counters + S_SLOTS, 0, 2 * 4, c->stream));
    TGX_CUDA(cudaMemsetAsync(s->d_occ, 0, s->occ_words * 4, c->stream));
    return TGX_OK;
}

// The occupancy pyramid of the blocks of n_slots slots, over zeroes.
static tgx_status svo_pyramid(tgx_ctx* c, tgx_svo* s, uint32_t n_slots)
{
    if (n_slots)
        TGX_LAUNCH_PDL(c, TR_SVO_PYRAMID, (n_slots + 255) / 256, 256, 0, k_svo_pyramid, s->d_slot_block, n_slots, s->d_nonempty,
                   s->d_occ, (const uint64_t*)((char*)s->d_occ + svo_occ_off_bytes(s->occ_words)), s->n_levels, s->B,
                   s->d_counters);
    return TGX_OK;
}

// Slots for the n_marked marked blocks, voxelisation of the pairs, and the
// occupancy pyramid of all n_slots slots (cleared first).
static tgx_status svo_fill(tgx_ctx* c, tgx_svo* s, const tgx_scene* sc, uint32_t n_cand, uint32_t n_marked,
                           uint32_t n_free, uint32_t next_slot, uint32_t n_slots)
{
    uint32_t* counters = s->d_counters;
    const size_t sort_bytes = (size_t)n_marked * 4 * 4 + (size_t)s->n_pairs * sizeof(PairRec) + 64;
    TGX_TRY(devbuf_reserve(c->svo_sort, sort_bytes));
    TGX_TRY(svo_clear_pyramid(c, s));
    if (n_marked) {
        // group the pairs by marked block: counts, ranges, placement
        const uint32_t* marked = svo_marked(c);
        uint32_t* cnt = (uint32_t*)c->svo_sort.ptr;
        uint32_t *off = cnt + n_marked, *cursor = off + n_marked, *slots = cursor + n_marked;
        PairRec* recs = (PairRec*)(((uintptr_t)(slots + n_marked) + 15) & ~(uintptr_t)15);
        const uint32_t mgrid = (n_marked + 255) / 256;
        const uint32_t pgrid = (uint32_t)std::min<uint64_t>(((uint64_t)n_cand + 255) / 256, (uint64_t)c->num_sms * 16);
        TGX_LAUNCH_PDL(c, TR_SVO_ALLOC, mgrid, 256, 0, k_svo_alloc, s->d_table, marked, n_marked, s->d_free, n_free, next_slot,
                   slots, s->d_slot_block, s->d_nonempty, cnt);
        TGX_LAUNCH_PDL(c, TR_SVO_VOXELIZE, pgrid, 256, 0, k_svo_pair_count, (const SvoPair*)c->svo_pairs.ptr, n_cand,
                   s->d_table, cnt);
        TGX_LAUNCH_PDL(c, TR_SVO_VOXELIZE, mgrid, 256, 0, k_svo_pair_ranges, cnt, n_marked, counters + S_SLOTS, off, cursor);
        TGX_LAUNCH_PDL(c, TR_SVO_VOXELIZE, (uint32_t)std::min<uint64_t>(((uint64_t)n_cand + 127) / 128, (uint64_t)c->num_sms * 32),
                       128, 0, k_svo_pair_fill, (const SvoPair*)c->svo_pairs.ptr, n_cand, s->d_table, cursor, sc->d_objects,
                       sc->d_cluster_pointers, sc->d_c2o, s->mn[0], s->mn[1], s->mn[2], s->B, recs);
        // one CTA per marked block, or four (8 layers each) when there are so few blocks
        // that the heaviest ones (up to 190 pairs against 30 on average) would decide the
        // time: 280 blocks of an update 222 -> 98 us; 18.4k blocks took 1430 us whole and 2560 split
        // (and only where every block's side is exactly 32, so that a voxel's index stays in its layers)
        bool split = (uint64_t)n_marked < (uint64_t)c->num_sms * 16u;
        for (int i = 0; i < 3; i++) split = split && fabsf(s->mn[i]) + (float)(1u << s->L) <= 16777216.0f;
#define VOXELIZE(mat, slabs)                                                                                          \
        do {                                                                                                          \
            const uint32_t smem = kBlockWords / (slabs) * ((mat) ? 17u : 1u) * 4u;                                     \
            TGX_CUDA(cudaFuncSetAttribute(k_svo_voxelize<mat, slabs>, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                                          (int)smem));                                                                \
            TGX_LAUNCH_PDL(c, TR_SVO_VOXELIZE, n_marked * (slabs), 32 * kWarpsPerVoxCta, smem, (k_svo_voxelize<mat, slabs>), \
                       sc->d_bits, recs, off, cnt, marked, slots, s->d_pool,                                           \
                       s->d_sub, s->d_nonempty, sc->d_material, s->d_mat, s->mn[0], s->mn[1], s->mn[2], s->B);         \
        } while (0)
        if (s->d_mat && split) VOXELIZE(true, 4);
        else if (s->d_mat) VOXELIZE(true, 1);
        else if (split) VOXELIZE(false, 4);
        else VOXELIZE(false, 1);
#undef VOXELIZE
        if (c->flags & TGX_FLAG_TEST_FAILED_FILL) {
            tgx_set_error("tgx_svo: TGX_FLAG_TEST_FAILED_FILL");
            return TGX_ERR_CUDA;
        }
        TGX_LAUNCH_PDL(c, TR_SVO_PYRAMID, mgrid, 256, 0, k_svo_publish, s->d_table, marked, slots, n_marked);
    }
    return svo_pyramid(c, s, n_slots);
}

// After an update that failed with `why`: the blocks that no moved object touches
// stay, with a pyramid of their own.  No mark stays in the table (a traversal would
// take it for a slot), and the slots that were freed or given out are free.
static tgx_status svo_drop_update(tgx_ctx* c, tgx_svo* s, tgx_status why)
{
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((n_table + 255) / 256, (uint64_t)c->num_sms * 32);
    TGX_LAUNCH_PDL(c, TR_SVO_ALLOC, grid, 256, 0, k_svo_unmark, s->d_table, n_table);
    TGX_LAUNCH_PDL(c, TR_SVO_ALLOC, (s->pool_cap + 255) / 256, 256, 0, k_svo_drop_slots, s->d_table, s->pool_cap,
                   s->d_slot_block, s->d_nonempty);
    TGX_TRY(svo_clear_pyramid(c, s));
    TGX_TRY(svo_pyramid(c, s, s->n_slots));
    TGX_CUDA(cudaMemcpyAsync(c->h_counter, s->d_counters, S_COUNT * 4, cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    const uint32_t n_freed = ((const uint32_t*)c->h_counter)[S_FREED];
    s->n_free += n_freed;
    s->n_blocks -= n_freed;
    return why;
}

extern "C" tgx_status tgx_svo_build(tgx_ctx* c, const tgx_scene* sc, const float* mn, uint32_t L, tgx_svo** out)
{
    return tgx_svo_build_flags(c, sc, mn, L, 0u, out);
}

extern "C" tgx_status tgx_svo_build_flags(tgx_ctx* c, const tgx_scene* sc, const float* mn, uint32_t L, uint32_t flags,
                                          tgx_svo** out)
{
    if (flags & ~TGX_SVO_NO_MATERIALS) { tgx_set_error("tgx_svo_build: unknown flags %u", flags); return TGX_ERR_INVALID_ARGUMENT; }
    if (!c || !sc || !mn || !out) { tgx_set_error("tgx_svo_build: NULL argument"); return TGX_ERR_INVALID_ARGUMENT; }
    *out = nullptr;
    if (L < 6 || L > 14) { tgx_set_error("tgx_svo_build: extent_log2 %u outside 6..14", L); return TGX_ERR_INVALID_ARGUMENT; }
    for (int i = 0; i < 3; i++)
        if (!(fabsf(mn[i]) <= 16777216.0f) || mn[i] != floorf(mn[i])) {
            tgx_set_error("tgx_svo_build: min must be integral and |min| <= 2^24");
            return TGX_ERR_INVALID_ARGUMENT;
        }
    TGX_CUDA(cudaSetDevice(c->device));
    tgx_svo* s = new (std::nothrow) tgx_svo();
    if (!s) return TGX_ERR_OUT_OF_MEMORY;
    s->mn[0] = mn[0]; s->mn[1] = mn[1]; s->mn[2] = mn[2];
    s->L = L;
    s->B = 1u << (L - 5);
    s->n_objects = sc->n_objects;
    s->n_cluster_pointers = sc->n_cluster_pointers;
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    s->n_levels = L - 5 + 1;
    uint64_t occ_words = 0;
    for (uint32_t l = 0; l < s->n_levels; l++) {
        const uint64_t n = (uint64_t)(s->B >> l);
        s->occ_off[l] = occ_words;
        occ_words += (n * n * n + 31) / 32;
    }
    s->occ_words = occ_words;

    auto fail = [&](tgx_status st) { cudaStreamSynchronize(c->stream); svo_free(s); return st; };
    if (svo_malloc(c, (void**)&s->d_table, n_table * 4) != cudaSuccess ||
        svo_malloc(c, (void**)&s->d_occ, occ_words * 4 + 128) != cudaSuccess ||
        tgx_malloc((void**)&s->d_counters, S_COUNT * 4) != cudaSuccess ||
        svo_malloc(c, (void**)&s->d_objs, std::max<uint64_t>(1, (uint64_t)sc->n_objects) * sizeof(tgx_object)) != cudaSuccess) {
        cudaGetLastError();
        tgx_set_error("tgx_svo_build: out of device memory for the block table");
        return fail(TGX_ERR_OUT_OF_MEMORY);
    }
    if (cudaMemsetAsync(s->d_table, 0, n_table * 4, c->stream) != cudaSuccess ||
        cudaMemsetAsync(s->d_counters, 0, S_COUNT * 4, c->stream) != cudaSuccess ||
        (sc->n_objects && cudaMemcpyAsync(s->d_objs, sc->d_objects, (uint64_t)sc->n_objects * sizeof(tgx_object),
                                          cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess) ||
        cudaMemcpyAsync((char*)s->d_occ + svo_occ_off_bytes(occ_words), s->occ_off, sizeof(s->occ_off), cudaMemcpyHostToDevice,
                        c->stream) != cudaSuccess) {
        tgx_set_error("tgx_svo_build: memset failed");
        return fail(TGX_ERR_CUDA);
    }
    tgx_status st;
    // pair storage: start from a per-cluster estimate, retry once with the exact count
    if ((st = svo_candidates(c, s, sc, nullptr, std::max<uint64_t>(1024, (uint64_t)sc->n_cluster_pointers * 4))) != TGX_OK)
        return fail(st);
    const uint32_t* hc = (const uint32_t*)c->h_counter;
    s->n_pairs = hc[S_PAIRS];
    s->n_blocks = hc[S_MARKED];
    const uint32_t n_cand = hc[S_CAND];
    s->n_slots = s->n_blocks;
    const bool materials = sc->d_material && sc->d_luts && !(flags & TGX_SVO_NO_MATERIALS);
    if ((st = svo_resize_slots(c, s, std::max(s->n_blocks, 1u), 0, materials)) != TGX_OK) return fail(st);
    if ((st = svo_fill(c, s, sc, n_cand, s->n_blocks, 0, 0, s->n_slots)) != TGX_OK) return fail(st);
    s->device_bytes = svo_device_bytes(s);
    *out = s;
    return TGX_OK;
}

extern "C" tgx_status tgx_svo_update(tgx_ctx* c, tgx_svo* s, const tgx_scene* sc, uint32_t* out_n_moved)
{
    if (!c || !s || !sc) { tgx_set_error("tgx_svo_update: NULL argument"); return TGX_ERR_INVALID_ARGUMENT; }
    if (sc->n_objects != s->n_objects || sc->n_cluster_pointers != s->n_cluster_pointers) {
        tgx_set_error("tgx_svo_update: the scene has %u objects / %u cluster pointers, the SVO was built from %u / %u",
                      sc->n_objects, sc->n_cluster_pointers, s->n_objects, s->n_cluster_pointers);
        return TGX_ERR_INVALID_ARGUMENT;
    }
    if (out_n_moved) *out_n_moved = 0;
    if (sc->n_objects == 0) return TGX_OK;
    TGX_CUDA(cudaSetDevice(c->device));
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    const uint64_t n_words = (n_table + 31) / 32;
    TGX_TRY(devbuf_reserve(c->svo_scratch, n_words * 4));
    uint32_t* dirty = (uint32_t*)c->svo_scratch.ptr;
    uint32_t* counters = s->d_counters;
    TGX_CUDA(cudaMemsetAsync(dirty, 0, n_words * 4, c->stream));
    TGX_CUDA(cudaMemsetAsync(counters + S_FREED, 0, 2 * 4, c->stream));   // freed, moved
    TGX_LAUNCH_PDL(c, TR_SVO_CANDIDATES, dim3(sc->n_objects, 8), 128, 0, k_svo_mark_dirty, sc->d_objects, s->d_objs,
               sc->d_cp_obj, s->mn[0], s->mn[1], s->mn[2], s->B, dirty);
    const uint64_t items = std::max<uint64_t>(n_words, sc->n_objects);
    const uint32_t wgrid = (uint32_t)std::min<uint64_t>((items + 255) / 256, (uint64_t)c->num_sms * 16);
    TGX_LAUNCH_PDL(c, TR_SVO_ALLOC, wgrid, 256, 0, k_svo_release_dirty, s->d_table, n_words, dirty, n_table, s->d_nonempty,
               s->d_slot_block, s->d_free + s->n_free, sc->d_objects, s->d_objs, sc->n_objects, counters);
    // pairs of the dirty blocks, into the pair storage the last build left (grown when short)
    tgx_status st = svo_candidates(c, s, sc, dirty, std::max<uint64_t>(1024, c->svo_pairs.bytes / kPairBytes));
    if (st != TGX_OK) return svo_drop_update(c, s, st);
    const uint32_t* hc = (const uint32_t*)c->h_counter;
    const uint32_t n_moved = hc[S_MOVED], n_freed = hc[S_FREED], n_marked = hc[S_MARKED], hc_pairs = hc[S_PAIRS], n_cand = hc[S_CAND];
    if (out_n_moved) *out_n_moved = n_moved;
    if (n_moved == 0) return TGX_OK;
    const uint32_t n_free = s->n_free + n_freed;
    const uint32_t fresh = n_marked > n_free ? n_marked - n_free : 0u;
    const uint32_t need = s->n_slots + fresh;
    if (need > s->pool_cap) st = svo_resize_slots(c, s, need + need / 4 + 64, s->n_slots, s->d_mat != nullptr);
    s->n_pairs = hc_pairs;
    if (st == TGX_OK) st = svo_fill(c, s, sc, n_cand, n_marked, n_free, s->n_slots, need);
    if (st != TGX_OK) return svo_drop_update(c, s, st);
    s->n_free = n_free - (n_marked - fresh);
    s->n_slots = need;
    s->n_blocks = s->n_blocks - n_freed + n_marked;
    s->device_bytes = svo_device_bytes(s);
    return TGX_OK;
}

extern "C" void tgx_svo_destroy(tgx_ctx* c, tgx_svo* s)
{
    if (c) cudaStreamSynchronize(c->stream);
    svo_free(s);
}

extern "C" tgx_status tgx_svo_get_info(tgx_ctx* c, const tgx_svo* s, tgx_svo_info* out)
{
    if (!c || !s || !out) return TGX_ERR_INVALID_ARGUMENT;
    TGX_CUDA(cudaMemcpyAsync(c->h_counter, s->d_counters, S_COUNT * 4, cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    out->min[0] = s->mn[0]; out->min[1] = s->mn[1]; out->min[2] = s->mn[2];
    out->extent_log2 = s->L;
    out->blocks_per_axis = s->B;
    out->n_blocks = s->n_blocks;
    out->n_nonempty_blocks = ((const uint32_t*)c->h_counter)[S_NONEMPTY];
    out->n_pairs = s->n_pairs;
    out->device_bytes = s->device_bytes;
    return TGX_OK;
}

extern "C" tgx_status tgx_svo_download(tgx_ctx* c, const tgx_svo* s, int32_t* out_xyz, uint32_t* out_words,
                                       uint32_t capacity, uint32_t* out_n)
{
    if (!c || !s || !out_n) return TGX_ERR_INVALID_ARGUMENT;
    const uint64_t n_table = (uint64_t)s->B * s->B * s->B;
    std::vector<uint32_t> table(n_table), nonempty(std::max(s->n_slots, 1u));
    TGX_CUDA(cudaMemcpyAsync(table.data(), s->d_table, n_table * 4, cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaMemcpyAsync(nonempty.data(), s->d_nonempty, nonempty.size() * 4, cudaMemcpyDeviceToHost, c->stream));
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    uint32_t n = 0;
    for (uint64_t i = 0; i < n_table; i++) {
        const uint32_t tv = table[i];
        if (!tv || !nonempty[tv - 1]) continue;
        if (n < capacity) {
            if (out_xyz) {
                out_xyz[3 * n + 0] = (int32_t)(s->mn[0] + (float)((i % s->B) * kBlockSide));
                out_xyz[3 * n + 1] = (int32_t)(s->mn[1] + (float)(((i / s->B) % s->B) * kBlockSide));
                out_xyz[3 * n + 2] = (int32_t)(s->mn[2] + (float)((i / ((uint64_t)s->B * s->B)) * kBlockSide));
            }
            if (out_words)
                TGX_CUDA(cudaMemcpyAsync(out_words + (uint64_t)n * kBlockWords, s->d_pool + (uint64_t)(tv - 1) * kBlockWords,
                                         kBlockWords * 4, cudaMemcpyDeviceToHost, c->stream));
        }
        n++;
    }
    TGX_CUDA(cudaStreamSynchronize(c->stream));
    *out_n = n;
    return TGX_OK;
}

namespace {

// A caller's ray batch: origins and directions in, distance and world voxel out.
struct RayArrays
{
    const float *o, *d;
    float* t;
    int32_t* voxel;
    int32_t mn[3];
    __device__ __forceinline__ void load(uint32_t i, float oi[3], float di[3]) const
    {
        const size_t k = 3 * (size_t)i;
#pragma unroll
        for (int a = 0; a < 3; a++) { oi[a] = o[k + a]; di[a] = d[k + a]; }
    }
    __device__ __forceinline__ void store(uint32_t i, int res, float ti, const int32_t c[3], int32_t) const
    {
        const size_t k = 3 * (size_t)i;
        t[i] = res == 1 ? ti : F32_MAX_TG;
#pragma unroll
        for (int a = 0; a < 3; a++) voxel[k + a] = res == 1 ? c[a] + mn[a] : 0;
    }
};

__global__ void __launch_bounds__(32 * kTraceWarps, kTraceCtas) k_svo_trace(const __grid_constant__ SvoDev s, uint32_t n, RayArrays io,
                                                               uint32_t max_steps, uint32_t steps_per_round,
                                                               uint32_t* __restrict__ queue,
                                                               uint32_t* __restrict__ n_exhausted)
{
    svo_trace_queue(s, io, n, max_steps, steps_per_round, queue, n_exhausted, nullptr);
}

}  // namespace

extern "C" tgx_status tgx_svo_trace(tgx_ctx* c, const tgx_svo* s, uint32_t n, const float* d_o, const float* d_d,
                                    uint32_t max_steps, float* d_t, int32_t* d_voxel)
{
    if (!c || !s || (n && (!d_o || !d_d || !d_t || !d_voxel))) {
        tgx_set_error("tgx_svo_trace: NULL argument");
        return TGX_ERR_INVALID_ARGUMENT;
    }
    if (n == 0) return TGX_OK;
    TGX_TRY(devbuf_reserve(c->svo_counters, S_COUNT * 4 + 64));
    uint32_t* exhausted = (uint32_t*)c->svo_counters.ptr + S_COUNT;
    uint32_t* queue = exhausted + 1;
    if (!c->svo_trace_ctas) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_svo_trace, 32 * kTraceWarps, 0) != cudaSuccess || per_sm < 1) {
            cudaGetLastError();
            per_sm = 1;
        }
        c->svo_trace_ctas = (uint32_t)(c->num_sms * per_sm);
    }
    const uint32_t per_cta = 32 * kTraceWarps;
    const uint32_t grid = std::min(c->svo_trace_ctas, (n - 1) / per_cta + 1);
    // the queue counter is read only when the rays outnumber the launch's lanes
    if ((uint64_t)grid * per_cta < n) TGX_CUDA(cudaMemsetAsync(queue, 0, 4, c->stream));
    const RayArrays io = {d_o, d_d, d_t, d_voxel, {(int32_t)s->mn[0], (int32_t)s->mn[1], (int32_t)s->mn[2]}};
    TGX_LAUNCH(c, TR_SVO_TRACE, grid, per_cta, 0, k_svo_trace, svo_dev(s), n, io, max_steps, c->trace_steps_per_round,
               queue, exhausted);
    return TGX_OK;
}
