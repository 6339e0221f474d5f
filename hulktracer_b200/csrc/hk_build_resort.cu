// hk_build_resort.cu -- the reference's per-node re-sampling SAH builder
// (--treeType=SAH: KDTreeCPU::buildKDTreeSAH / buildNodeSAH,
// HulkEngine/src/KDTreeSAH.cpp:9-244) on the GPU, one level at a time.
//
// The reference recurses depth-first; every node takes every sample-th
// polygon of its own list, clips the triangle's bounds to the node box, makes
// one co-planar candidate (clipped extent <= FLT_EPSILON) or a begin and an
// end candidate per axis, sorts each axis, and sweeps the sorted values with
// running counts (below += previous group's co-planar + begin counts;
// co-planar = previous group's co-planar count; above -= this group's
// co-planar + end counts; the first group starts from list size / sample).
// Nodes are independent, so here all nodes of a level are processed at once:
//
//   keys     one 64-bit key per candidate slot: segment (node x 3 + axis),
//            the value as an order-preserving integer, the marker; each
//            segment occupies a fixed range (two slots per sampled polygon,
//            an unused slot sorts last in its segment)
//   sort     LSD radix sort of the level's keys, 8 bits per pass (so each
//            segment ends up sorted in place)
//   sweep    the running counts of the sequential sweep are prefix sums over
//            the sorted keys, taken with device-wide scans and read back at
//            every group of equal values; each group's SAH cost is computed
//            with the reference's float expression and the first minimum in
//            sweep order (axis, then value) wins through a 64-bit atomicMin
//            of (cost, key position)
//   split    checkPolygonToAAPlane by vertex coordinates on every polygon of
//            a split node; a stable partition (scans) writes the next level's
//            lists in the reference's list order, below child then above
//
// A level is nine launches (more while segments are long enough for the radix
// sort): every scan is one single-pass kernel that computes what it sums (the
// candidate counts, the group heads, the decisions, the classification) as it
// loads it, sizes that the host needs for the next level come back in one
// read, and launches in between take theirs from device memory. Three launches
// per scan and two reads per level took 5.1 ms for 59,280 triangles.
//
// The output is the compact tree the traversal kernels read (child pairs in
// breadth-first order: below, above; an absent child is an empty leaf cell),
// with the ropes and cell boxes of every cell. It is the tree of the
// reference's builder in the layout hk_tree_import makes of it.
#include <algorithm>
#include <cfloat>
#include <string>

#include "hk_common.cuh"
#include "hk_resort.h"
#include "hk_scan.cuh"

namespace hk {

template <class T>
cudaError_t RBuf<T>::ensure(size_t n) {
    if (n <= cap && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    const size_t c = n < 16 ? 16 : n + n / 4;
    cudaError_t e = cudaMalloc((void **)&p, c * sizeof(T));
    if (e == cudaSuccess) cap = c;
    return e;
}

template <class T>
void RBuf<T>::release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
}

namespace {

typedef unsigned long long u64;

// grow an output array keeping its first `keep` elements
template <class T>
cudaError_t grow_keep(RBuf<T> &b, size_t n, size_t keep, cudaStream_t st) {
    if (n <= b.cap && b.p) return cudaSuccess;
    const size_t c = n + n / 2 + 64;
    T *q = nullptr;
    cudaError_t e = cudaMalloc((void **)&q, c * sizeof(T));
    if (e != cudaSuccess) return e;
    if (b.p && keep) {
        e = cudaMemcpyAsync(q, b.p, keep * sizeof(T), cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) {
            cudaFree(q);
            return e;
        }
        cudaStreamSynchronize(st);
    }
    if (b.p) cudaFree(b.p);
    b.p = q;
    b.cap = c;
    return cudaSuccess;
}

// ---------------------------------------------------------------- scans ----
constexpr int kScanNT = 256;    // threads per scan tile
constexpr int kScanItems = 4;   // elements per thread
constexpr uint32_t kScanTile = kScanNT * kScanItems;
// polls before a wait gives up (error word). A short limit is raised: a tile's
// predecessor publishes within microseconds of its start, 64K polls are tens of
// milliseconds
constexpr uint32_t kScanSpins = 1u << 22, kScanSpinsMin = 1u << 16;

// tile states of a scan and its ticket; every scan of a build has a tag and a
// ticket of its own
struct ScanPtrs {
    uint32_t *flags, *ticket, *err;
    uint4 *aggs, *incls;   // uint2 scans use their first half
    uint32_t tag, spin_limit;
    uint32_t withhold;     // test aid: tile 0 publishes under an old tag, so that no tile sees it
};

// one scan: op.count() elements, op.load(i) -> Item, op.value(Item) -> T,
// op.apply(i, exclusive prefix, Item), op.finish(total) by one thread.
// A wait that runs out leaves prefixes that are too small, never too large, so
// this scan's own stores stay in range; what they index (key ranges, places of
// nodes and references) no longer fits together, so every later kernel of the
// build returns at once on the error word, which the host reads at the level's
// end.
template <class Op>
__global__ void __launch_bounds__(kScanNT) k_r_scan(Op op, ScanPtrs sp) {
    using T = typename Op::T;
    __shared__ T sw[kScanNT / 32];
    __shared__ T s_excl;
    __shared__ uint32_t s_tile, s_err;
    const uint32_t n = op.count();
    const uint32_t ntiles = n ? (n + kScanTile - 1) / kScanTile : 1u;
    T *aggs = reinterpret_cast<T *>(sp.aggs), *incls = reinterpret_cast<T *>(sp.incls);
    for (;;) {
        if (threadIdx.x == 0) {
            s_err = __ldcg(sp.err);
            s_tile = atomicAdd(sp.ticket, 1u);
        }
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= ntiles || s_err) break;
        const uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
        typename Op::Item it[kScanItems];
        T v[kScanItems], s = vzero<T>();
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            v[k] = vzero<T>();
            if (base + k < n) {
                it[k] = op.load(base + k);
                v[k] = op.value(it[k]);
            }
            s = vadd(s, v[k]);
        }
        T tot;
        const T ex = block_excl<kScanNT>(s, sw, tot);
        const uint32_t tag = sp.withhold && tile == 0 ? sp.tag - 1u : sp.tag;
        tile_prefix(tile, tot, tag, sp.flags, aggs, incls, &s_excl, sp.err, sp.spin_limit);
        T pre = vadd(s_excl, ex);
#pragma unroll
        for (int k = 0; k < kScanItems; k++) {
            if (base + k < n) op.apply(base + k, pre, it[k]);
            pre = vadd(pre, v[k]);
        }
        if (tile == ntiles - 1 && threadIdx.x == 0) op.finish(vadd(s_excl, tot));
        __syncthreads();
    }
}

// ----------------------------------------------------------- radix sort ----
constexpr int kRT = 256;                     // threads per sort tile
constexpr int kRI = 4;                       // keys per thread
// 1024 keys per tile: the levels that need this sort have few keys per SM, and
// a tile's rounds follow one another (4096 keys: 22 us a pass for 70,000 keys)
constexpr uint32_t kTile = kRT * kRI;

__global__ void __launch_bounds__(kRT) k_rs_hist(const u64 *__restrict__ keys, const uint32_t *__restrict__ nkeys,
                                                 int shift, uint32_t ntiles, uint32_t *hist,
                                                 const uint32_t *__restrict__ err) {
    __shared__ uint32_t h[256];
    const uint32_t n = *nkeys;
    if (*err) return;   // (uniform: only scans set it)
    h[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kTile;
    for (int r = 0; r < kRI; r++) {
        const size_t i = base + (size_t)r * kRT + threadIdx.x;
        if (i < n) atomicAdd(&h[(uint32_t)(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// exclusive prefix of the tiles' counts, digit by digit
struct RsScanOp {
    using T = uint2;
    using Item = uint32_t;
    uint32_t *hist;
    uint32_t n;
    __device__ uint32_t count() const { return n; }
    __device__ Item load(uint32_t i) const { return hist[i]; }
    __device__ T value(const Item &it) const { return make_uint2(it, 0); }
    __device__ void apply(uint32_t i, T pre, const Item &) const { hist[i] = pre.x; }
    __device__ void finish(T) const {}
};

// stable scatter: within a tile keys are ranked in index order (rounds of
// 256 consecutive keys; warps in order; lanes by __match_any_sync)
__global__ void __launch_bounds__(kRT) k_rs_scatter(const u64 *__restrict__ in, u64 *__restrict__ out,
                                                    const uint32_t *__restrict__ nkeys, int shift, uint32_t ntiles,
                                                    const uint32_t *__restrict__ offs,
                                                    const uint32_t *__restrict__ err) {
    __shared__ uint32_t run[256];
    __shared__ uint32_t wc[kRT / 32][256];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, n = *nkeys;
    if (*err) return;
    run[threadIdx.x] = 0;
    const size_t base = (size_t)blockIdx.x * kTile;
    for (int r = 0; r < kRI; r++) {
        for (uint32_t q = threadIdx.x; q < (kRT / 32) * 256; q += kRT) (&wc[0][0])[q] = 0;
        __syncthreads();
        const size_t i = base + (size_t)r * kRT + threadIdx.x;
        const bool have = i < n;
        const u64 k = have ? in[i] : 0ull;
        const uint32_t d = have ? ((uint32_t)(k >> shift) & 255u) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, d);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        if (have && lane == (uint32_t)(__ffs(peers) - 1)) wc[w][d] = __popc(peers);
        __syncthreads();
        size_t dst = 0;
        if (have) {
            uint32_t pre = 0;
            for (uint32_t q = 0; q < w; q++) pre += wc[q][d];
            dst = (size_t)offs[(size_t)d * ntiles + blockIdx.x] + run[d] + pre + rank;
        }
        __syncthreads();
        uint32_t tot = 0;
        for (int q = 0; q < kRT / 32; q++) tot += wc[q][threadIdx.x];
        run[threadIdx.x] += tot;
        if (have) out[dst] = k;
        __syncthreads();
    }
}

// ------------------------------------------------------------- helpers ----
constexpr uint32_t kNone = 3u;      // marker of an unused key slot
constexpr uint32_t kDecLeaf = 3u;   // decision: leaf (else the split axis)

__device__ __forceinline__ float c3(const float4 &v, uint32_t a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
__device__ __forceinline__ void s3(float4 &v, uint32_t a, float x) {
    if (a == 0) v.x = x;
    else if (a == 1) v.y = x;
    else v.z = x;
}
// _mm_min_ps / _mm_max_ps lanes
__device__ __forceinline__ float mnf(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float mxf(float a, float b) { return a > b ? a : b; }

__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ u64 make_key(uint32_t seg, float v, uint32_t marker) {
    return ((u64)seg << 34) | ((u64)f2o(v) << 2) | marker;
}
__device__ __forceinline__ float key_value(u64 k) { return o2f((uint32_t)(k >> 2)); }
__device__ __forceinline__ uint32_t lo32(u64 x) { return (uint32_t)x; }
__device__ __forceinline__ uint32_t hi32(u64 x) { return (uint32_t)(x >> 32); }

// sizes that a level leaves for the host (and, SK_MAXCNT, the next level's
// largest node that has candidates)
enum { SK_JUNCTIONS = 0, SK_REFS, SK_LEAFREFS, SK_MAXCNT, SK_ERR, SK_WORDS };

struct LevelPtrs {
    // this level
    uint32_t n;
    const float4 *lo, *hi;
    const float *surf;
    const uint32_t *off, *cnt, *ropes, *refs, *ref_node;
    // scratch
    uint32_t *koff, *jrank, *loff, *efirst, *decision, *gfirst;
    float *plane, *surf_lo, *surf_hi;
    u64 *best, *keys;
    uint4 *sweep;       // per key: begins and co-planars, co-planars, ends, groups before it
    uint2 *rscan;       // per reference: references that go below / above before it
    uint32_t *sizes;    // SK_*
    // next level
    float4 *nlo, *nhi;
    float *nsurf;
    uint32_t *noff, *ncnt, *nropes, *nrefs, *nref_node;
    // output
    uint2 *nodes;
    uint32_t *out_refs, *out_ropes;
    float4 *out_cbox;
    uint32_t cbase, nbase, rbase;
    ResortParams p;
    uint32_t depth;
};

// a scan of this build gave up waiting (the same for every thread of a kernel
// that is no scan): the kernel does nothing. Read beside the kernel's first loads.
__device__ __forceinline__ bool r_aborted(const LevelPtrs &L) { return L.sizes[SK_ERR] != 0; }

__device__ __forceinline__ bool forced_leaf(const LevelPtrs &L, uint32_t c, uint32_t depth) {
    return c == 0 || c <= L.p.leaf_size || depth >= L.p.max_depth;
}

// candidate slots of every node: six per sampled polygon
struct InitOp {
    using T = uint2;
    using Item = uint32_t;
    LevelPtrs L;
    __device__ uint32_t count() const { return L.n; }
    __device__ Item load(uint32_t i) const {
        const uint32_t c = L.cnt[i];
        L.best[i] = ~0ull;
        L.efirst[3 * (size_t)i] = L.efirst[3 * (size_t)i + 1] = L.efirst[3 * (size_t)i + 2] = 0;
        return forced_leaf(L, c, L.depth) ? 0u : 6u * ((c + L.p.sample - 1) / L.p.sample);
    }
    __device__ T value(const Item &it) const { return make_uint2(it, 0); }
    __device__ void apply(uint32_t i, T pre, const Item &) const { L.koff[i] = pre.x; }
    __device__ void finish(T tot) const { L.koff[L.n] = tot.x; }
};

// KDTreeSAH.cpp:51-82: candidates of the sampled polygons
__global__ void k_r_emit(LevelPtrs L, const float4 *__restrict__ V, const uint4 *__restrict__ T) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x, Q = L.koff[L.n] / 6u;
    if (r_aborted(L) || q >= Q) return;
    uint32_t a = 0, b = L.n;   // node: koff[i] / 6 <= q < koff[i + 1] / 6
    while (a < b) {
        const uint32_t m = (a + b) >> 1;
        if (L.koff[m + 1] / 6u <= q) a = m + 1;
        else b = m;
    }
    const uint32_t i = a;
    const uint32_t s = (L.koff[i + 1] - L.koff[i]) / 6u, j = q - L.koff[i] / 6u;
    const uint32_t poly = L.refs[L.off[i] + j * L.p.sample];
    const uint4 t = T[poly];
    const float4 p1 = V[t.x], p2 = V[t.y], p3 = V[t.z];
    const float4 bl = L.lo[i], bh = L.hi[i];
#pragma unroll
    for (uint32_t ax = 0; ax < 3; ax++) {
        float lo = mnf(mnf(c3(p1, ax), c3(p2, ax)), c3(p3, ax));
        float hi = mxf(mxf(c3(p1, ax), c3(p2, ax)), c3(p3, ax));
        lo = mxf(lo, c3(bl, ax));
        hi = mnf(hi, c3(bh, ax));
        const uint32_t seg = 3 * i + ax;
        const size_t k = (size_t)L.koff[i] + (size_t)ax * 2 * s + 2 * (size_t)j;
        if (fabsf(__fsub_rn(lo, hi)) <= FLT_EPSILON) {
            L.keys[k] = make_key(seg, lo, 1);
            L.keys[k + 1] = ((u64)seg << 34) | (0xffffffffull << 2) | kNone;
        } else {
            L.keys[k] = make_key(seg, lo, 0);
            L.keys[k + 1] = make_key(seg, hi, 2);
        }
    }
}

__device__ __forceinline__ void seg_range(const LevelPtrs &L, uint32_t seg, uint32_t &i, uint32_t &ax, uint32_t &s0,
                                          uint32_t &s1) {
    i = seg / 3;
    ax = seg - 3 * i;
    const uint32_t s = (L.koff[i + 1] - L.koff[i]) / 6u;
    s0 = L.koff[i] + ax * 2 * s;
    s1 = s0 + 2 * s;
}

// Levels whose candidate segments are all short sort each segment on its own
// instead of the whole level: a warp in registers up to kSegWarpMax keys
// (8 per lane), a CTA in shared memory up to kSegCtaMax. Segments hold their
// keys in fixed ranges, so either way every segment ends up sorted in place.
constexpr uint32_t kSegWarpMax = 256, kSegCtaMax = 4096;

template <int RJ>
__device__ __forceinline__ void reg_exchange(u64 (&x)[kSegWarpMax / 32], uint32_t nr, uint32_t lane, uint32_t k) {
#pragma unroll
    for (int r = 0; r < (int)(kSegWarpMax / 32); r++) {
        if ((r & RJ) || (uint32_t)r >= nr) continue;
        const bool up = (((uint32_t)r * 32u + lane) & k) == 0;
        const u64 a = x[r], b = x[r | RJ];
        if ((a > b) == up) {
            x[r] = b;
            x[r | RJ] = a;
        }
    }
}

__global__ void k_seg_sort_warp(LevelPtrs L, uint32_t nseg) {
    const uint32_t lane = threadIdx.x & 31u, seg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (seg >= nseg) return;   // uniform over the warp
    uint32_t i, ax, s0, s1;
    seg_range(L, seg, i, ax, s0, s1);
    const uint32_t n = s1 - s0;
    if (r_aborted(L) || n <= 1 || n > kSegWarpMax) return;
    uint32_t n2 = 1;
    while (n2 < n) n2 <<= 1;
    const uint32_t nr = (n2 + 31u) >> 5;
    u64 x[kSegWarpMax / 32];
#pragma unroll
    for (int r = 0; r < (int)(kSegWarpMax / 32); r++) {
        const uint32_t e = (uint32_t)r * 32u + lane;
        x[r] = e < n ? L.keys[s0 + e] : ~0ull;
    }
    for (uint32_t k = 2; k <= n2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                // partners in the lane's own registers (compile-time indices)
                if (j == 32) reg_exchange<1>(x, nr, lane, k);
                else if (j == 64) reg_exchange<2>(x, nr, lane, k);
                else reg_exchange<4>(x, nr, lane, k);
            } else {
                const bool lower = (lane & j) == 0;
#pragma unroll
                for (int r = 0; r < (int)(kSegWarpMax / 32); r++) {
                    if ((uint32_t)r >= nr) continue;
                    const u64 o = __shfl_xor_sync(0xffffffffu, x[r], (int)j);
                    const bool up = (((uint32_t)r * 32u + lane) & k) == 0;
                    const u64 mn = x[r] < o ? x[r] : o, mx = x[r] < o ? o : x[r];
                    x[r] = (lower == up) ? mn : mx;
                }
            }
        }
#pragma unroll
    for (int r = 0; r < (int)(kSegWarpMax / 32); r++) {
        const uint32_t e = (uint32_t)r * 32u + lane;
        if (e < n) L.keys[s0 + e] = x[r];
    }
}

__global__ void __launch_bounds__(256) k_seg_sort_cta(LevelPtrs L, uint32_t nseg) {
    __shared__ u64 sk[kSegCtaMax];
    if (r_aborted(L)) return;
    for (uint32_t seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
        uint32_t i, ax, s0, s1;
        seg_range(L, seg, i, ax, s0, s1);
        const uint32_t n = s1 - s0;
        if (n <= kSegWarpMax || n > kSegCtaMax) continue;   // uniform over the CTA
        uint32_t n2 = 1;
        while (n2 < n) n2 <<= 1;
        for (uint32_t e = threadIdx.x; e < n2; e += blockDim.x) sk[e] = e < n ? L.keys[s0 + e] : ~0ull;
        __syncthreads();
        for (uint32_t k = 2; k <= n2; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t e = threadIdx.x; e < n2; e += blockDim.x) {
                    const uint32_t p = e ^ j;
                    if (p > e) {
                        const bool up = (e & k) == 0;
                        const u64 a = sk[e], b = sk[p];
                        if ((a > b) == up) {
                            sk[e] = b;
                            sk[p] = a;
                        }
                    }
                }
                __syncthreads();
            }
        for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) L.keys[s0 + e] = sk[e];
        __syncthreads();
    }
}

// group heads and the counters the sweep accumulates
struct SweepOp {
    using T = uint4;
    using Item = uint4;
    LevelPtrs L;
    __device__ uint32_t count() const { return L.koff[L.n]; }
    __device__ Item load(uint32_t p) const {
        const u64 k = L.keys[p];
        const uint32_t m = (uint32_t)k & 3u;
        if (m == kNone) return make_uint4(0, 0, 0, 0);
        uint32_t i, ax, s0, s1;
        seg_range(L, (uint32_t)(k >> 34), i, ax, s0, s1);
        const float v = key_value(k);
        const bool head = p == s0 || !(key_value(L.keys[p - 1]) == v);
        // ends in the segment's first group are never subtracted (:164-169)
        if (m == 2 && key_value(L.keys[s0]) == v) atomicAdd(&L.efirst[(uint32_t)(k >> 34)], 1u);
        return make_uint4(m != 2 ? 1u : 0u, m == 1 ? 1u : 0u, m == 2 ? 1u : 0u, head ? 1u : 0u);
    }
    __device__ T value(const Item &it) const { return it; }
    __device__ void apply(uint32_t p, T pre, const Item &it) const {
        L.sweep[p] = pre;
        if (it.w) L.gfirst[pre.w] = p;
    }
    __device__ void finish(T tot) const {
        const uint32_t K = L.koff[L.n];
        L.sweep[K] = tot;
        L.gfirst[tot.w] = K;
    }
};

// (cost, key position) of the group that starts at key p, or ~0 when p
// starts no group or its cost is not below FLT_MAX
__device__ u64 r_group_cost(const LevelPtrs &L, uint32_t p) {
    const uint4 at = L.sweep[p];
    const uint32_t g = at.w;
    if (L.sweep[p + 1].w == g) return ~0ull;   // not a group head
    const u64 k = L.keys[p];
    const uint32_t seg = (uint32_t)(k >> 34);
    uint32_t i, ax, s0, s1;
    seg_range(L, seg, i, ax, s0, s1);
    const uint4 first = L.sweep[s0], last = L.sweep[s1];
    const uint32_t real_end = s0 + (last.x - first.x) + (last.z - first.z);
    const uint32_t nxt = L.gfirst[g + 1];
    const uint32_t l1 = nxt < real_end ? nxt : real_end;
    const uint4 end = L.sweep[l1];
    const uint32_t cop = p == s0 ? end.y - at.y : at.y - L.sweep[L.gfirst[g - 1]].y;
    const uint32_t below = at.x - first.x;
    const uint32_t N = L.cnt[i] / L.p.sample;
    const uint32_t above = N - (end.y - first.y) - ((end.z - first.z) - L.efirst[seg]);
    const float v = key_value(k);
    const float4 bl = L.lo[i], bh = L.hi[i];
    const float dim[3] = {__fsub_rn(bh.x, bl.x), __fsub_rn(bh.y, bl.y), __fsub_rn(bh.z, bl.z)};
    const float x = dim[(ax + 1) % 3], y = dim[(ax + 2) % 3];
    const float xpy = __fadd_rn(x, y), area = __fmul_rn(x, y);
    const float upper = __fadd_rn(area, __fmul_rn(__fsub_rn(c3(bh, ax), v), xpy));
    const float lower = __fadd_rn(area, __fmul_rn(__fsub_rn(v, c3(bl, ax)), xpy));
    const float cb = __fmul_rn(lower, (float)below), ca = __fmul_rn(upper, (float)above);
    const float ci = __fmul_rn(area, (float)cop);
    const float inv = __fdiv_rn(1.0f, L.surf[i]);
    const float score =
        __fadd_rn(L.p.ct, __fmul_rn(L.p.ci, __fmul_rn(__fadd_rn(__fadd_rn(ci, cb), ca), inv)));
    return score < FLT_MAX ? ((u64)f2o(score) << 32) | p : ~0ull;
}

// the SAH of every group (KDTreeSAH.cpp:147-175); the node's minimum of
// (cost, position) is taken over the warp first (keys are sorted by node, so
// a warp's lanes span few nodes), then with one atomicMin per node and warp
__global__ void k_r_cost(LevelPtrs L) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x, K = L.koff[L.n];
    const uint32_t lane = threadIdx.x & 31u;
    if (r_aborted(L)) return;
    u64 packed = ~0ull;
    uint32_t node = 0xffffffffu;
    if (p < K) {
        node = (uint32_t)(L.keys[p] >> 34) / 3u;
        packed = r_group_cost(L, p);
    }
    // segmented minimum over runs of equal node in lane order
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const u64 o = __shfl_down_sync(0xffffffffu, packed, off);
        const uint32_t on = __shfl_down_sync(0xffffffffu, node, off);
        if (lane + off < 32 && on == node && o < packed) packed = o;
    }
    const uint32_t prev = __shfl_up_sync(0xffffffffu, node, 1);
    const bool first = lane == 0 || prev != node;
    if (p < K && first && packed != ~0ull) atomicMin(&L.best[node], packed);
}


// leaf test (KDTreeSAH.cpp:186-191) and the split's child surfaces; ranks of
// the junctions and the leaves' places
struct DecideOp {
    using T = uint2;
    using Item = uint2;   // (junction, leaf references)
    LevelPtrs L;
    __device__ uint32_t count() const { return L.n; }
    __device__ Item load(uint32_t i) const {
        const uint32_t c = L.cnt[i];
        const u64 b = L.best[i];
        bool leaf = forced_leaf(L, c, L.depth) || b == ~0ull;
        if (!leaf) {
            const float score = o2f(hi32(b));
            const float leafcost = __fmul_rn(L.p.ci, (float)(c / L.p.sample));
            leaf = score >= leafcost;
        }
        if (leaf) {
            L.decision[i] = kDecLeaf;
            return make_uint2(0, c);
        }
        const u64 k = L.keys[lo32(b)];
        const uint32_t ax = (uint32_t)(k >> 34) % 3u;
        const float v = key_value(k);
        const float4 bl = L.lo[i], bh = L.hi[i];
        const float dim[3] = {__fsub_rn(bh.x, bl.x), __fsub_rn(bh.y, bl.y), __fsub_rn(bh.z, bl.z)};
        const float x = dim[(ax + 1) % 3], y = dim[(ax + 2) % 3];
        const float xpy = __fadd_rn(x, y), area = __fmul_rn(x, y);
        L.surf_hi[i] = __fadd_rn(area, __fmul_rn(__fsub_rn(c3(bh, ax), v), xpy));
        L.surf_lo[i] = __fadd_rn(area, __fmul_rn(__fsub_rn(v, c3(bl, ax)), xpy));
        L.plane[i] = v;
        L.decision[i] = ax;
        return make_uint2(1, 0);
    }
    __device__ T value(const Item &it) const { return it; }
    __device__ void apply(uint32_t i, T pre, const Item &) const {
        L.jrank[i] = pre.x;
        L.loff[i] = pre.y;
    }
    __device__ void finish(T tot) const {
        L.sizes[SK_JUNCTIONS] = tot.x;
        L.sizes[SK_LEAFREFS] = tot.y;
        L.sizes[SK_MAXCNT] = 0;   // k_r_nodes takes the maximum
    }
};

// KDTreeCPU::checkPolygonToAAPlane (KDTreeCPU.cpp:450-477) on the polygons of
// split nodes: (goes below, goes above)
struct ClassifyOp {
    using T = uint2;
    using Item = uint2;
    LevelPtrs L;
    uint32_t R;
    const float4 *V;
    const uint4 *Tr;
    __device__ uint32_t count() const { return R; }
    __device__ Item load(uint32_t q) const {
        const uint32_t i = L.ref_node[q];
        const uint32_t d = L.decision[i];
        if (d == kDecLeaf) return make_uint2(0, 0);
        const float v = L.plane[i];
        const uint4 t = Tr[L.refs[q]];
        const float a = c3(V[t.x], d), b = c3(V[t.y], d), c = c3(V[t.z], d);
        const bool cop = (a == v) & (b == v) & (c == v);
        const bool above = (a >= v) & (b >= v) & (c >= v);
        const bool below = (a <= v) & (b <= v) & (c <= v);
        // below, intersecting, co-planar; above, intersecting, co-planar
        return make_uint2(cop || !above ? 1u : 0u, cop || above || !below ? 1u : 0u);
    }
    __device__ T value(const Item &it) const { return it; }
    __device__ void apply(uint32_t q, T pre, const Item &) const { L.rscan[q] = pre; }
    __device__ void finish(T tot) const {
        L.rscan[R] = tot;
        L.sizes[SK_REFS] = tot.x + tot.y;
    }
};

// cells of this level, and the next level's nodes
__device__ __forceinline__ uint32_t r_node(const LevelPtrs &L, uint32_t i) {
    const uint32_t cell = L.cbase + i;
    const uint32_t c = L.cnt[i], d = L.decision[i];
    const float4 bl = L.lo[i], bh = L.hi[i];
    for (int f = 0; f < 6; f++) L.out_ropes[6 * (size_t)cell + f] = L.ropes[6 * (size_t)i + f];
    L.out_cbox[2 * (size_t)cell] = make_float4(bl.x, bl.y, bl.z, 0.0f);
    L.out_cbox[2 * (size_t)cell + 1] = make_float4(bh.x, bh.y, bh.z, 0.0f);
    if (d == kDecLeaf) {
        L.nodes[cell] = c ? make_uint2(((L.rbase + L.loff[i]) << 2) | kLeafTag, c) : make_uint2(kLeafTag, 0u);
        return 0;
    }
    const uint32_t k = L.jrank[i], pair = L.nbase + 2 * k;
    const float v = L.plane[i];
    L.nodes[cell] = make_uint2((pair << 2) | d, __float_as_uint(v));
    const uint2 r0 = L.rscan[L.off[i]], r1 = L.rscan[L.off[i] + c];
    const uint32_t cB = r1.x - r0.x, cA = r1.y - r0.y;
    const uint32_t oB = r0.x + r0.y;
    // below child (pair), above child (pair + 1)
    float4 hB = bh, lA = bl;
    s3(hB, d, v);
    s3(lA, d, v);
    L.nlo[2 * k] = bl;
    L.nhi[2 * k] = hB;
    L.nlo[2 * k + 1] = lA;
    L.nhi[2 * k + 1] = bh;
    L.nsurf[2 * k] = L.surf_lo[i];
    L.nsurf[2 * k + 1] = L.surf_hi[i];
    L.noff[2 * k] = oB;
    L.ncnt[2 * k] = cB;
    L.noff[2 * k + 1] = oB + cB;
    L.ncnt[2 * k + 1] = cA;
    for (int f = 0; f < 6; f++) {
        const uint32_t r = L.ropes[6 * (size_t)i + f];
        L.nropes[12 * (size_t)k + f] = r;
        L.nropes[12 * (size_t)k + 6 + f] = r;
    }
    L.nropes[12 * (size_t)k + 2 * d + 1] = pair + 1;
    L.nropes[12 * (size_t)k + 6 + 2 * d] = pair;
    const uint32_t sB = forced_leaf(L, cB, L.depth + 1) ? 0u : cB, sA = forced_leaf(L, cA, L.depth + 1) ? 0u : cA;
    return max(sB, sA);
}

__global__ void k_r_nodes(LevelPtrs L) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (r_aborted(L)) return;
    // the largest child with candidates
    const uint32_t m = __reduce_max_sync(0xffffffffu, i < L.n ? r_node(L, i) : 0u);
    if (m && (threadIdx.x & 31u) == 0) atomicMax(&L.sizes[SK_MAXCNT], m);
}

// leaf references out; split references into the next level (stable)
__global__ void k_r_scatter(LevelPtrs L, uint32_t R) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= R) return;
    const uint32_t i = L.ref_node[q];
    const uint32_t ref = L.refs[q];
    if (L.decision[i] == kDecLeaf) {
        L.out_refs[L.rbase + L.loff[i] + (q - L.off[i])] = ref;
        return;
    }
    const uint32_t k = L.jrank[i];
    const uint2 rq = L.rscan[q], rn = L.rscan[q + 1], r0 = L.rscan[L.off[i]], r1 = L.rscan[L.off[i] + L.cnt[i]];
    const uint32_t oB = r0.x + r0.y, cB = r1.x - r0.x;
    if (rn.x != rq.x) {
        const uint32_t dst = oB + (rq.x - r0.x);
        L.nrefs[dst] = ref;
        L.nref_node[dst] = 2 * k;
    }
    if (rn.y != rq.y) {
        const uint32_t dst = oB + cB + (rq.y - r0.y);
        L.nrefs[dst] = ref;
        L.nref_node[dst] = 2 * k + 1;
    }
}

// level 0: the root over every polygon (its box and half surface, getHalfBox-
// Surface, SharedFunctions.hpp:40-44, from the host), and the padding cell 1
struct RootPtrs {
    float4 *lo, *hi;
    float *surf;
    uint32_t *off, *cnt, *ropes, *refs, *ref_node;
    uint2 *nodes;
    uint32_t *out_ropes;
    float4 *out_cbox;
};
__global__ void k_r_root(RootPtrs P, float4 lo, float4 hi, float half, uint32_t nt) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nt) {
        P.refs[i] = i;
        P.ref_node[i] = 0;
    }
    if (i < 6) {
        P.ropes[i] = 0xffffffffu;
        P.out_ropes[6 + i] = 0xffffffffu;
    }
    if (i < 2) P.out_cbox[2 + i] = make_float4(0, 0, 0, 0);
    if (i == 0) {
        P.lo[0] = lo;
        P.hi[0] = hi;
        P.surf[0] = half;
        P.off[0] = 0;
        P.cnt[0] = nt;
        P.nodes[1] = make_uint2(kLeafTag, 0u);
    }
}

inline unsigned blocks(uint32_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t) ? (unsigned)((n + t - 1) / t) : 1u; }

}  // namespace

void ResortState::release() {
    for (int b = 0; b < 2; b++) {
        lo[b].release();
        hi[b].release();
        surf[b].release();
        off[b].release();
        cnt[b].release();
        ropes[b].release();
        refs[b].release();
        ref_node[b].release();
        keys[b].release();
    }
    koff.release();
    jrank.release();
    loff.release();
    efirst.release();
    decision.release();
    plane.release();
    surf_lo.release();
    surf_hi.release();
    best.release();
    sweep.release();
    rscan.release();
    hist.release();
    gfirst.release();
    scan_flags.release();
    scan_agg.release();
    scan_incl.release();
    tickets.release();
    sizes.release();
    if (host_sizes) cudaFreeHost(host_sizes);
    host_sizes = nullptr;
    nodes.release();
    out_refs.release();
    out_ropes.release();
    out_cbox.release();
}

#define RS_CHECK(x)                                                 \
    do {                                                            \
        cudaError_t e_ = (x);                                       \
        if (e_ != cudaSuccess) {                                    \
            if (err) *err = std::string(#x) + ": " + cudaGetErrorString(e_); \
            return HK_E_CUDA;                                       \
        }                                                           \
    } while (0)

// the tile states of a scan of up to n elements, and its tag and ticket
static cudaError_t scan_begin(ResortState &S, const ResortParams &p, size_t n, bool withhold, uint32_t &next_ticket,
                              ScanPtrs &sp, cudaStream_t st) {
    const size_t tiles = n / kScanTile + 2;
    if (tiles > std::min({S.scan_flags.cap, S.scan_agg.cap, S.scan_incl.cap})) {
        // the flags last: while they have a capacity all three stand and they
        // are cleared, also for the next build after a failure here
        S.scan_flags.release();
        cudaError_t e = S.scan_agg.ensure(tiles);
        if (e == cudaSuccess) e = S.scan_incl.ensure(tiles);
        if (e == cudaSuccess) e = S.scan_flags.ensure(tiles);
        if (e == cudaSuccess) {
            e = cudaMemsetAsync(S.scan_flags.p, 0, S.scan_flags.cap * 4, st);
            if (e != cudaSuccess) S.scan_flags.release();
        }
        if (e != cudaSuccess) return e;
    }
    S.scan_tag = (S.scan_tag + 1u) & 0x3fffffffu;
    sp = ScanPtrs{S.scan_flags.p, S.tickets.p + next_ticket++, S.sizes.p + SK_ERR, S.scan_agg.p, S.scan_incl.p,
                  S.scan_tag, p.spin_limit ? std::max(p.spin_limit, kScanSpinsMin) : kScanSpins, withhold ? 1u : 0u};
    return cudaSuccess;
}

template <class Op>
static cudaError_t scan(ResortState &S, const ResortParams &p, const Op &op, size_t n, bool withhold,
                        uint32_t &next_ticket, cudaStream_t st) {
    ScanPtrs sp;
    cudaError_t e = scan_begin(S, p, n, withhold, next_ticket, sp, st);
    if (e != cudaSuccess) return e;
    // a CTA per tile up to four per SM
    const unsigned grid = (unsigned)std::min<size_t>(n / kScanTile + 1, (size_t)p.sm_count * 4);
    k_r_scan<Op><<<grid, kScanNT, 0, st>>>(op, sp);
    return cudaGetLastError();
}

hk_status resort_build(ResortState &S, const ResortParams &p, const float4 *verts, const uint4 *tris, uint32_t nt,
                       const float *hbox, cudaStream_t st, std::string *err) {
    if (p.sample == 0 || p.max_depth > 64) {
        if (err) *err = "sample must be >= 1 and max_depth <= 64";
        return HK_E_ILLEGAL_INPUT;
    }
    // level 0: the root (cell 0) over every polygon; cell 1 is padding
    // cells [cbase, cbase + n) hold the current level; `written` cells exist
    uint32_t n = 1, R = nt, cbase = 0, rbase = 0, written = 2, depth = 0;
    // four scans a level and at most eight radix passes (34 + 30 key bits)
    constexpr uint32_t kTickets = 66 * 12;
    RS_CHECK(S.lo[0].ensure(1));
    RS_CHECK(S.hi[0].ensure(1));
    RS_CHECK(S.surf[0].ensure(1));
    RS_CHECK(S.off[0].ensure(1));
    RS_CHECK(S.cnt[0].ensure(1));
    RS_CHECK(S.ropes[0].ensure(6));
    RS_CHECK(S.refs[0].ensure(R));
    RS_CHECK(S.ref_node[0].ensure(R));
    RS_CHECK(S.sizes.ensure(SK_WORDS));
    RS_CHECK(S.tickets.ensure(kTickets));
    RS_CHECK(grow_keep(S.nodes, 2, 0, st));
    RS_CHECK(grow_keep(S.out_ropes, 12, 0, st));
    RS_CHECK(grow_keep(S.out_cbox, 4, 0, st));
    RS_CHECK(grow_keep(S.out_refs, 1, 0, st));
    if (!S.host_sizes) RS_CHECK(cudaHostAlloc((void **)&S.host_sizes, SK_WORDS * 4, cudaHostAllocDefault));
    RS_CHECK(cudaMemsetAsync(S.sizes.p, 0, SK_WORDS * 4, st));
    RS_CHECK(cudaMemsetAsync(S.tickets.p, 0, kTickets * 4, st));
    uint32_t next_ticket = 0;
    {
        const float sx = hbox[4] - hbox[0], sy = hbox[5] - hbox[1], sz = hbox[6] - hbox[2];
        const RootPtrs P{S.lo[0].p, S.hi[0].p, S.surf[0].p, S.off[0].p, S.cnt[0].p, S.ropes[0].p,
                         S.refs[0].p, S.ref_node[0].p, S.nodes.p, S.out_ropes.p, S.out_cbox.p};
        k_r_root<<<blocks(std::max<uint32_t>(R, 6)), 256, 0, st>>>(
            P, make_float4(hbox[0], hbox[1], hbox[2], hbox[3]), make_float4(hbox[4], hbox[5], hbox[6], hbox[7]),
            sx * sy + sz * sy + sx * sz, nt);
    }
    // the largest node with candidates (forced_leaf)
    uint32_t maxcnt = (nt <= p.leaf_size || p.max_depth == 0) ? 0u : nt;
    for (uint32_t level = 0; n > 0; level++) {
        const int cur = level & 1, nxt = cur ^ 1;
        const bool hold = (p.debug_flags & 1u) && level >= 1;
        depth = level;
        // per-node scratch
        RS_CHECK(S.koff.ensure((size_t)n + 1));
        RS_CHECK(S.jrank.ensure(n));
        RS_CHECK(S.loff.ensure(n));
        RS_CHECK(S.efirst.ensure(3 * (size_t)n));
        RS_CHECK(S.decision.ensure(n));
        RS_CHECK(S.plane.ensure(n));
        RS_CHECK(S.surf_lo.ensure(n));
        RS_CHECK(S.surf_hi.ensure(n));
        RS_CHECK(S.best.ensure(n));
        RS_CHECK(S.rscan.ensure((size_t)R + 1));
        // candidate slots: six per sampled polygon, at least one per node
        const uint64_t Q = maxcnt ? (uint64_t)R / p.sample + std::min(n, R) : 0u;
        if (6 * Q >= 0xfffffff0ull) {
            if (err) *err = "more candidate slots than 32 bits index";
            return HK_E_CAPACITY;
        }
        const uint32_t K = (uint32_t)(6 * Q);   // at most; the actual count stays on the device
        RS_CHECK(S.keys[0].ensure(K ? K : 1));
        RS_CHECK(S.keys[1].ensure(K ? K : 1));
        RS_CHECK(S.sweep.ensure((size_t)K + 1));
        RS_CHECK(S.gfirst.ensure((size_t)K + 2));
        // this level's cells in the output; the next level has at most 2 n nodes
        RS_CHECK(grow_keep(S.nodes, (size_t)cbase + n, written, st));
        RS_CHECK(grow_keep(S.out_ropes, 6 * ((size_t)cbase + n), 6 * (size_t)written, st));
        RS_CHECK(grow_keep(S.out_cbox, 2 * ((size_t)cbase + n), 2 * (size_t)written, st));
        const size_t n2max = std::min<size_t>(2 * (size_t)n, 2 * (size_t)R);
        RS_CHECK(S.lo[nxt].ensure(n2max));
        RS_CHECK(S.hi[nxt].ensure(n2max));
        RS_CHECK(S.surf[nxt].ensure(n2max));
        RS_CHECK(S.off[nxt].ensure(n2max));
        RS_CHECK(S.cnt[nxt].ensure(n2max));
        RS_CHECK(S.ropes[nxt].ensure(6 * n2max));
        LevelPtrs L;
        memset(&L, 0, sizeof L);
        L.n = n;
        L.lo = S.lo[cur].p;
        L.hi = S.hi[cur].p;
        L.surf = S.surf[cur].p;
        L.off = S.off[cur].p;
        L.cnt = S.cnt[cur].p;
        L.ropes = S.ropes[cur].p;
        L.refs = S.refs[cur].p;
        L.ref_node = S.ref_node[cur].p;
        L.koff = S.koff.p;
        L.jrank = S.jrank.p;
        L.loff = S.loff.p;
        L.efirst = S.efirst.p;
        L.decision = S.decision.p;
        L.plane = S.plane.p;
        L.surf_lo = S.surf_lo.p;
        L.surf_hi = S.surf_hi.p;
        L.best = S.best.p;
        L.sweep = S.sweep.p;
        L.gfirst = S.gfirst.p;
        L.rscan = S.rscan.p;
        L.sizes = S.sizes.p;
        L.nlo = S.lo[nxt].p;
        L.nhi = S.hi[nxt].p;
        L.nsurf = S.surf[nxt].p;
        L.noff = S.off[nxt].p;
        L.ncnt = S.cnt[nxt].p;
        L.nropes = S.ropes[nxt].p;
        L.nodes = S.nodes.p;
        L.out_ropes = S.out_ropes.p;
        L.out_cbox = S.out_cbox.p;
        L.p = p;
        L.depth = level;
        L.cbase = cbase;
        L.nbase = level == 0 ? 2u : cbase + n;   // the next level's first cell
        L.rbase = rbase;
        // 1. candidates
        int kc = 0;
        L.keys = S.keys[kc].p;
        RS_CHECK(scan(S, p, InitOp{L}, n, hold, next_ticket, st));
        if (K) {
            k_r_emit<<<blocks(K / 6), 256, 0, st>>>(L, verts, tris);
            // 2. sort by (segment, value, marker)
            const uint32_t maxseg = 2 * ((maxcnt + p.sample - 1) / p.sample);
            if (maxseg <= kSegCtaMax) {
                const uint32_t nseg = 3 * n;
                k_seg_sort_warp<<<(unsigned)(((size_t)nseg * 32 + 255) / 256), 256, 0, st>>>(L, nseg);
                if (maxseg > kSegWarpMax) k_seg_sort_cta<<<std::min<uint32_t>(nseg, p.sm_count * 8u), 256, 0, st>>>(L, nseg);
            } else {
                uint32_t segbits = 1;
                while (segbits < 30 && (1ull << segbits) < 3ull * n) segbits++;
                const int nbits = 34 + (int)segbits;
                const uint32_t ntiles = (K + kTile - 1) / kTile;
                RS_CHECK(S.hist.ensure(256 * (size_t)ntiles));
                for (int shift = 0; shift < nbits; shift += 8) {
                    k_rs_hist<<<ntiles, kRT, 0, st>>>(S.keys[kc].p, L.koff + n, shift, ntiles, S.hist.p,
                                                     L.sizes + SK_ERR);
                    RS_CHECK(scan(S, p, RsScanOp{S.hist.p, 256 * ntiles}, 256 * (size_t)ntiles, hold, next_ticket, st));
                    k_rs_scatter<<<ntiles, kRT, 0, st>>>(S.keys[kc].p, S.keys[kc ^ 1].p, L.koff + n, shift, ntiles,
                                                         S.hist.p, L.sizes + SK_ERR);
                    kc ^= 1;
                }
            }
            L.keys = S.keys[kc].p;
            // 3. sweep
            RS_CHECK(scan(S, p, SweepOp{L}, K, false, next_ticket, st));
            k_r_cost<<<blocks(K), 256, 0, st>>>(L);
        }
        // 4. decisions, ranks, leaf offsets; classification; cells and nodes
        RS_CHECK(scan(S, p, DecideOp{L}, n, hold, next_ticket, st));
        RS_CHECK(scan(S, p, ClassifyOp{L, R, verts, tris}, R, false, next_ticket, st));
        k_r_nodes<<<blocks(n), 256, 0, st>>>(L);
        RS_CHECK(cudaGetLastError());
        RS_CHECK(cudaMemcpyAsync(S.host_sizes, S.sizes.p, SK_WORDS * 4, cudaMemcpyDeviceToHost, st));
        RS_CHECK(cudaStreamSynchronize(st));
        if (S.host_sizes[SK_ERR]) {
            if (err) *err = "a scan's wait ran out";
            return HK_E_DEVICE_TIMEOUT;
        }
        const uint32_t J = S.host_sizes[SK_JUNCTIONS], R2 = S.host_sizes[SK_REFS], Lrefs = S.host_sizes[SK_LEAFREFS];
        maxcnt = S.host_sizes[SK_MAXCNT];
        // 5. leaf references, the next level's lists
        RS_CHECK(grow_keep(S.out_refs, (size_t)rbase + Lrefs, rbase, st));
        RS_CHECK(S.refs[nxt].ensure(R2));
        RS_CHECK(S.ref_node[nxt].ensure(R2));
        L.out_refs = S.out_refs.p;
        L.nrefs = S.refs[nxt].p;
        L.nref_node = S.ref_node[nxt].p;
        k_r_scatter<<<blocks(R), 256, 0, st>>>(L, R);
        RS_CHECK(cudaGetLastError());
        written = L.nbase;
        cbase = L.nbase;
        rbase += Lrefs;
        n = 2 * J;
        R = R2;
    }
    RS_CHECK(cudaStreamSynchronize(st));
    S.nn = written;
    S.nr = rbase;
    S.depth = depth;
    return HK_OK;
}

template struct RBuf<float4>;
template struct RBuf<float>;
template struct RBuf<uint32_t>;
template struct RBuf<u64>;
template struct RBuf<uint2>;
template struct RBuf<uint4>;

}  // namespace hk
