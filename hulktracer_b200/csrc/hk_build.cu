// hk_build.cu -- GPU KD-tree builder: exact binned SAH (sm_100a).
//
// Breadth-first and level-synchronous for nodes of more than 32 references:
// two launches per level in the binned mode (k_decide, k_plan_refs), three
// with exact_max or the proposer (k_hist on a second stream beside k_small,
// then k_plan_refs; the proposer adds its chain after k_hist); smaller nodes
// are deferred subtrees (below; hk_config subtree_max / subtree_depth /
// level_streams choose the layout). Splits are searched over 32 bins per
// axis, or, with exact_max (32..1024), over every clipped reference bound for
// nodes of at most exact_max references (one warp up to 128, one CTA above):
//   work      large nodes (> 256 references, or > 32 in a level of few
//             references): one CTA per chunk of up to 1024 references builds
//             shared-memory histograms (3 axes x {lo bin, hi bin,
//             flat-on-plane}) of the clipped reference bounds; a node of one
//             chunk is decided from them (one warp: scans over the 32 bins,
//             exact cost at the 31 planes per axis, argmin), the chunks of a
//             larger one are added up in global memory and the CTA that
//             finishes the last decides. Small nodes: one warp per node,
//             warp-private histogram, same SAH (up to 32 references counted
//             plane by plane, without a histogram). Every decision is also
//             tallied into the level totals (leaf refs, splits, next-level
//             nodes, child refs) that the capacity guard needs.
//   [learn]   learned mode: nodes of 33..1024 references get the binned SAH
//             and their histogram features in k_hist (a warp each up to 256
//             references); then k_learn runs the tensor-core MLP on them
//             (128-row tiles) and takes the top-k (axis, bin) proposals, and
//             k_refine_warp / k_refine_cta cost every clipped reference bound
//             inside the proposed bins exactly (the exact SAH restricted to
//             those bins); the cheaper of that and the binned optimum splits
//             the node
//   plan      single-pass scan over nodes (decoupled look-back): leaf
//             reference offsets, child pairs, next-level slots, child
//             reference offsets; emits compact node entries, cells and ropes,
//             next-level node records and the next level's large-node
//             chunks. The guard (the whole level stops splitting on overflow)
//             is decided from the tallies before anything is emitted.
//   refs      single-pass scan of the below/above flags of every reference,
//             fused with the stable partition into the next level and the
//             leaf reference list.
//   subtrees  a decidable node of 2..32 references is not split by the
//             levels: it is recorded (with its references) as a deferred
//             root. After the last level one warp per root builds its whole
//             subtree depth first in registers (one reference per lane, the
//             node's references a lane mask, the same SAH), a scan over the
//             subtrees' sizes places them after the levels' nodes and leaf
//             references, and a last pass moves them there. On the 200k-triangle
//             animated frame, deferring at any depth, 94% of the split
//             decisions are taken this way.
// Every kernel reads its work size from device memory, so the whole build is
// a fixed launch sequence (graph-capturable, no host round trips). Look-back
// waits are bounded: a wait that runs out sets an error bit and the build
// reports failure instead of hanging.
//
// The algorithm is restated serially in the CPU oracle (hko_build_binned); the
// two produce identical trees. The plane / bin / cost arithmetic below is
// written with explicit IEEE round-to-nearest intrinsics for that reason.
#include <algorithm>
#include <cstdio>
#include <type_traits>

#include "hk_build.h"
#include "hk_common.cuh"
#include "hk_internal.h"
#include "hk_mlp_tc.cuh"
#include "hk_mlp_tile.cuh"
#include "hk_scan.cuh"

namespace hk {

constexpr uint32_t kBins = 32;
constexpr uint32_t kSmall = 256;     // nodes with <= kSmall refs: one warp per node
constexpr uint32_t kChunk = 1024;    // most refs per histogram CTA of a large node (4 per thread)
constexpr uint32_t kChunkMin = 256;
constexpr uint32_t kWarpExact = 32;  // exact-SAH nodes up to this size: one warp, in registers
constexpr uint32_t kLearnMax = 1024; // learned mode: nodes of kWarpExact + 1 .. kLearnMax refs are proposer rows
constexpr uint32_t kHist = 3 * 3 * kBins;
static_assert(kHist % 4 == 0 && kHist / 4 > 64 && kHist / 4 <= 96, "k_small clears its histogram with 16-byte stores");
constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr uint32_t kTile = kScanThreads * kScanItems;
constexpr int kPlanItems = 1;                                 // nodes per thread of a plan tile
constexpr uint32_t kPlanTile = kScanThreads * kPlanItems;

// ---------------------------------------------------------------------------
// scan value types: uint2 (reference below/above flags; subtree sizes) and U7
// (node plan: leaf refs, splits, next-level nodes, child refs, below child
// refs, deferred-subtree refs, deferred-subtree roots)
// ---------------------------------------------------------------------------
struct U7 {
    uint32_t x, y, z, w, v, d, e;
};
__device__ __forceinline__ U7 vadd(U7 a, U7 b) {
    return U7{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w, a.v + b.v, a.d + b.d, a.e + b.e};
}
__device__ __forceinline__ U7 vsub(U7 a, U7 b) {
    return U7{a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w, a.v - b.v, a.d - b.d, a.e - b.e};
}
template <> __device__ __forceinline__ U7 vzero<U7>() { return U7{0, 0, 0, 0, 0, 0, 0}; }
__device__ __forceinline__ U7 shfl_up(U7 v, int d) {
    return U7{__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d),
              __shfl_up_sync(0xffffffffu, v.z, d), __shfl_up_sync(0xffffffffu, v.w, d),
              __shfl_up_sync(0xffffffffu, v.v, d), __shfl_up_sync(0xffffffffu, v.d, d),
              __shfl_up_sync(0xffffffffu, v.e, d)};
}
__device__ __forceinline__ U7 shfl_xor(U7 v, int d) {
    return U7{__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d),
              __shfl_xor_sync(0xffffffffu, v.z, d), __shfl_xor_sync(0xffffffffu, v.w, d),
              __shfl_xor_sync(0xffffffffu, v.v, d), __shfl_xor_sync(0xffffffffu, v.d, d),
              __shfl_xor_sync(0xffffffffu, v.e, d)};
}
__device__ __forceinline__ U7 ldcg(const U7 *p) {
    const uint32_t *q = reinterpret_cast<const uint32_t *>(p);
    return U7{__ldcg(q), __ldcg(q + 1), __ldcg(q + 2), __ldcg(q + 3), __ldcg(q + 4), __ldcg(q + 5), __ldcg(q + 6)};
}

// ---------------------------------------------------------------------------
// single-pass scans (hk_scan.cuh). The tag is build epoch x 64 + level. A wait
// that runs out (the build's spin limit, kSpinLimit polls by default) counts
// the tile as zero; every later kernel of the build then returns at once
// (level_aborted), so the inconsistent level is never read.
// ---------------------------------------------------------------------------
constexpr uint32_t kSpinLimit = 1u << 22;
// error bits after which the build's data may be inconsistent: a wait ran
// out (4), a partition / decision count mismatch (8), a plan bound (16)
constexpr uint32_t kErrAbort = 4u | 8u | 16u | kErrTensorWait;

// Kernels launched as programmatic dependents (launch_pdl) start before their
// predecessor in the stream has finished; this waits until it has, with its
// writes visible. Without the launch attribute it returns at once.
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The reference tiles' flags carry their values: two 64-bit words, each with
// the flag in its upper half and a count (below, above) in its lower half, so
// one load gives both and no fence stands between them. A word is read whole;
// two words that differ in their flags are a record between two writes.
__device__ __forceinline__ void ref_publish(ulonglong2 *rec, uint32_t flag, uint2 v) {
    const unsigned long long f = (unsigned long long)flag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(rec), "l"(f | v.x), "l"(f | v.y) : "memory");
}
__device__ __forceinline__ uint32_t ref_poll(const ulonglong2 *rec, uint32_t tag, uint2 &v) {
    unsigned long long x, y;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(rec) : "memory");
    v = make_uint2((uint32_t)x, (uint32_t)y);
    const uint32_t f = (uint32_t)(x >> 32);
    return f == (uint32_t)(y >> 32) && (f >> 2) == tag ? f & 3u : 0u;
}

__device__ __forceinline__ uint2 ref_lookback(const ulonglong2 *recs, uint32_t tile, uint32_t tag, uint32_t *err,
                                              uint32_t spin_limit) {
    const int lane = threadIdx.x & 31;
    uint2 excl = make_uint2(0, 0);
    int32_t p = (int32_t)tile - 1;
    for (;;) {
        const int32_t q = p - lane;
        uint2 v = make_uint2(0, 0);
        uint32_t st = 2;    // before tile 0: zero
        const int stop = lookback_window([&] { return q >= 0 ? st = ref_poll(recs + q, tag, v) : st; }, err, spin_limit);
        if (lane > stop || !st) v = make_uint2(0, 0);
        excl.x += __reduce_add_sync(0xffffffffu, v.x);
        excl.y += __reduce_add_sync(0xffffffffu, v.y);
        if (stop < 32) break;
        p -= 32;
    }
    return excl;
}

// Op: T (scan value), Item (what load caches for apply), Ctx (per-CTA
// constants), kItems (consecutive elements per thread); load(i) -> Item,
// value(Item) -> T, apply_first / apply(i, exclusive prefix, Item, Ctx),
// err(). One tile of a single-pass scan: load, block scan, publish the
// aggregate, look back for the tile's exclusive prefix, then apply_first every
// element with its global prefix, run between() (all threads), and apply every
// element.
template <class Op, class Between>
__device__ __forceinline__ void scan_tile(const Op &op, uint32_t tile, uint32_t n, uint32_t tag,
                                          const typename Op::Ctx &cx, uint32_t *flags, typename Op::T *aggs,
                                          typename Op::T *incls, typename Op::T *sh, typename Op::T &s_excl,
                                          const Between &between) {
    using T = typename Op::T;
    constexpr int kItems = Op::kItems;
    constexpr uint32_t kTileN = kScanThreads * kItems;
    const uint32_t base = tile * kTileN + threadIdx.x * kItems;
    typename Op::Item it[kItems];
    T s = vzero<T>();
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        it[k] = op.load(base + k < n ? base + k : 0xffffffffu, cx);
        s = vadd(s, op.value(it[k]));
    }
    T tot;
    const T ex = block_excl<kScanThreads>(s, sh, tot);
    tile_prefix(tile, tot, tag, flags, aggs, incls, &s_excl, op.err(), op.A.spin_limit);
    const T pre0 = vadd(s_excl, ex);
    T pre = pre0;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        if (base + k < n) op.apply_first(base + k, pre, it[k], cx);
        pre = vadd(pre, op.value(it[k]));
    }
    between();
    pre = pre0;
#pragma unroll
    for (int k = 0; k < kItems; k++) {
        if (base + k < n) op.apply(base + k, pre, it[k], cx);
        pre = vadd(pre, op.value(it[k]));
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// exact-order helpers shared with the oracle restatement
// ---------------------------------------------------------------------------
__device__ __forceinline__ float mxf(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float mnf(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float c3(float4 v, uint32_t a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
__device__ __forceinline__ void s3(float4 &v, uint32_t a, float x) {
    if (a == 0) v.x = x;
    else if (a == 1) v.y = x;
    else v.z = x;
}

// p_k = min + ext * (k / bins)
__device__ __forceinline__ float plane_k(float blo, float ext, uint32_t k) {
    return __fadd_rn(blo, __fmul_rn(ext, __fmul_rn((float)k, 0.03125f)));
}

__device__ __forceinline__ float surf(float4 lo, float4 hi) {
    float sx = __fsub_rn(hi.x, lo.x), sy = __fsub_rn(hi.y, lo.y), sz = __fsub_rn(hi.z, lo.z);
    return __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(sx, sy), __fmul_rn(sz, sy)), __fmul_rn(sx, sz)));
}

// bins of a clipped interval [lo, hi] on one axis: p_b <= lo < p_{b+1},
// p_c < hi <= p_{c+1}; on = the interval is flat and lies on plane b
__device__ __forceinline__ void bin_interval(float lo, float hi, float blo, float ext, float inv, int &b, int &c,
                                             bool &on) {
    b = __float2int_rz(__fmul_rn(__fsub_rn(lo, blo), inv));
    b = b < 0 ? 0 : (b > (int)kBins - 1 ? (int)kBins - 1 : b);
    while (b > 0 && lo < plane_k(blo, ext, b)) b--;
    while (b < (int)kBins - 1 && lo >= plane_k(blo, ext, b + 1)) b++;
    c = __float2int_rz(__fmul_rn(__fsub_rn(hi, blo), inv));
    c = c < 0 ? 0 : (c > (int)kBins - 1 ? (int)kBins - 1 : c);
    while (c > 0 && hi <= plane_k(blo, ext, c)) c--;
    while (c < (int)kBins - 1 && hi > plane_k(blo, ext, c + 1)) c++;
    on = (lo == hi) && b >= 1 && lo == plane_k(blo, ext, b);
}

// bins per unit length of the node on each axis (32 / extent). It only seeds
// bin_interval's first guess, whose corrections end on the one bin b with
// p_b <= lo < p_{b+1} from any start in [0, 31], so a fast division serves.
__device__ __forceinline__ float4 bin_scale(float4 blo, float4 bhi) {
    float4 r;
    r.x = __fdividef(32.0f, __fsub_rn(bhi.x, blo.x));
    r.y = __fdividef(32.0f, __fsub_rn(bhi.y, blo.y));
    r.z = __fdividef(32.0f, __fsub_rn(bhi.z, blo.z));
    r.w = 0.0f;
    return r;
}

// histogram contribution of one reference (shared-memory counters); inv3 =
// bin_scale(blo, bhi)
__device__ __forceinline__ void hist_ref(uint32_t *H, float4 tlo, float4 thi, float4 blo, float4 bhi, float4 inv3) {
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        float l = c3(blo, a), h = c3(bhi, a);
        float ext = __fsub_rn(h, l);
        if (!(ext > 0.0f)) continue;
        float inv = c3(inv3, a);
        float lo = mxf(c3(tlo, a), l), hi = mnf(c3(thi, a), h);
        int b, c;
        bool on;
        bin_interval(lo, hi, l, ext, inv, b, c, on);
        atomicAdd(&H[a * 96 + b], 1u);
        atomicAdd(&H[a * 96 + 32 + c], 1u);
        if (on) atomicAdd(&H[a * 96 + 64 + b], 1u);
    }
}

// The node's planes p_k (k = 1..31) of each axis in P[a * kPlaneRow + k], so the
// bin corrections read them instead of recomputing them (the same values),
// between -inf (k = 0) and +inf (k = 32): one warp or threads of a CTA; the
// caller syncs before reading.
constexpr uint32_t kPlaneRow = kBins + 1;
constexpr uint32_t kPlanes = (3 * kPlaneRow + 3) & ~3u;
// a warp's scratch for one node: histogram and plane table, or the packed
// bounds of at most 32 references
constexpr uint32_t kWarpScratch = kHist + kPlanes;
// one axis (a warp)
__device__ __forceinline__ void node_planes_row(float *P, uint32_t a, float4 blo, float4 bhi) {
    const uint32_t lane = threadIdx.x & 31u;
    const float l = c3(blo, a);
    P[a * kPlaneRow + lane] = lane ? plane_k(l, __fsub_rn(c3(bhi, a), l), lane) : -kInf;
    if (lane == 0) P[a * kPlaneRow + kBins] = kInf;
}
__device__ __forceinline__ void node_planes_warp(float *P, float4 blo, float4 bhi) {
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) node_planes_row(P, a, blo, bhi);
}
__device__ __forceinline__ void node_planes_cta(float *P, float4 blo, float4 bhi) {
    if (threadIdx.x < 96) node_planes_row(P, threadIdx.x >> 5, blo, bhi);
}

// bin_interval with the planes of the axis read from Pa
__device__ __forceinline__ void bin_interval_tab(float lo, float hi, float blo, float inv, const float *Pa, int &b,
                                                 int &c, bool &on) {
    b = __float2int_rz(__fmul_rn(__fsub_rn(lo, blo), inv));
    b = b < 0 ? 0 : (b > (int)kBins - 1 ? (int)kBins - 1 : b);
    while (b > 0 && lo < Pa[b]) b--;
    while (b < (int)kBins - 1 && lo >= Pa[b + 1]) b++;
    c = __float2int_rz(__fmul_rn(__fsub_rn(hi, blo), inv));
    c = c < 0 ? 0 : (c > (int)kBins - 1 ? (int)kBins - 1 : c);
    while (c > 0 && hi <= Pa[c]) c--;
    while (c < (int)kBins - 1 && hi > Pa[c + 1]) c++;
    on = (lo == hi) && b >= 1 && lo == Pa[b];
}

// A reference's bins on the axes with extent, with the node's plane table P
// (node_planes_*); lanes that do not `have` one get some bin. A first guess of
// a bin is all but always right, so the six bins are checked together, without
// a branch between their twelve plane reads; a reference with any wrong guess
// takes the walk. (Two loops of dependent reads per bin before: a frame of 1M
// triangles 2,989 us against 2,817, one of 3.5k 547 against 524.)
__device__ __forceinline__ void ref_bins(float4 tlo, float4 thi, float4 blo, float4 bhi, float4 inv3, const float *P,
                                         bool have, int (&b)[3], int (&c)[3], bool (&on)[3]) {
    bool good = true;
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        const float l = c3(blo, a), h = c3(bhi, a), inv = c3(inv3, a);
        const float lo = mxf(c3(tlo, a), l), hi = mnf(c3(thi, a), h);
        const float *Pa = P + a * kPlaneRow;
        b[a] = min(max(__float2int_rz(__fmul_rn(__fsub_rn(lo, l), inv)), 0), (int)kBins - 1);
        c[a] = min(max(__float2int_rz(__fmul_rn(__fsub_rn(hi, l), inv)), 0), (int)kBins - 1);
        const float b0 = Pa[b[a]], b1 = Pa[b[a] + 1], c0 = Pa[c[a]], c1 = Pa[c[a] + 1];
        good = good && (!(__fsub_rn(h, l) > 0.0f) || (lo >= b0 && lo < b1 && hi > c0 && hi <= c1));
        on[a] = lo == hi && b[a] >= 1 && lo == b0;
    }
    if (have && !good) {
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float l = c3(blo, a), h = c3(bhi, a);
            bin_interval_tab(mxf(c3(tlo, a), l), mnf(c3(thi, a), h), l, c3(inv3, a), P + a * kPlaneRow, b[a], c[a], on[a]);
        }
    }
}

// hist_ref with the node's plane table
__device__ __forceinline__ void hist_ref_tab(uint32_t *H, float4 tlo, float4 thi, float4 blo, float4 bhi, float4 inv3,
                                             const float *P) {
    int b[3], c[3];
    bool on[3];
    ref_bins(tlo, thi, blo, bhi, inv3, P, true, b, c, on);
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        if (!(__fsub_rn(c3(bhi, a), c3(blo, a)) > 0.0f)) continue;   // uniform
        atomicAdd(&H[a * 96 + b[a]], 1u);
        atomicAdd(&H[a * 96 + 32 + c[a]], 1u);
        if (on[a]) atomicAdd(&H[a * 96 + 64 + b[a]], 1u);
    }
}

struct Decision {
    int axis;
    float plane;
    uint32_t nb, na;
    float cost;
    int bin;      // plane index k of the chosen plane
};

// Warp-wide SAH over the node's histograms (all 32 lanes call it): lane k
// costs plane k of every axis, keeps its cheapest, and one warp argmin over
// (cost, axis, plane) picks the first minimum in (axis, plane) order, as the
// serial loop does. Below / above counts come from exclusive scans over the
// bins (packed 16 + 16 bits when the node has fewer than 65536 references).
template <class HistPtr>
__device__ Decision sah_warp(HistPtr H, float4 blo, float4 bhi, uint32_t cnt, float ct, float ci) {
    const uint32_t lane = threadIdx.x & 31u;
    const float A = surf(blo, bhi);
    const bool packed = cnt < 65536u;
    float mc = kInf;
    uint32_t mkey = 0xffffffffu, m_nb = 0, m_na = 0;
    float m_pk = 0.0f;
    uint32_t hist[9];   // every counter of the lane loaded together
#pragma unroll
    for (uint32_t k = 0; k < 9; k++) hist[k] = H[k * 32 + lane];
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        const float l = c3(blo, a), h = c3(bhi, a);
        const float ext = __fsub_rn(h, l);
        if (!(ext > 0.0f)) continue;
        const uint32_t hlo = hist[3 * a], hhi = hist[3 * a + 1];
        uint32_t slo, shi;
        if (packed) {
            uint32_t v = hlo | (hhi << 16);
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, v, d);
                if ((int)lane >= d) v += u;
            }
            slo = v & 0xffffu;
            shi = v >> 16;
        } else {
            slo = hlo;
            shi = hhi;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, slo, d), w = __shfl_up_sync(0xffffffffu, shi, d);
                if ((int)lane >= d) {
                    slo += u;
                    shi += w;
                }
            }
        }
        const uint32_t below = slo - hlo;          // sum_{b < k} hlo[b]
        const uint32_t above = cnt - (shi - hhi);  // sum_{c >= k} hhi[c]
        const uint32_t on = hist[3 * a + 2];
        const float pk = plane_k(l, ext, lane);
        const float pk1 = __shfl_down_sync(0xffffffffu, pk, 1);   // plane k + 1 (lane 31: unused)
        const bool valid = lane >= 1 && pk > l && pk < h && (lane == 31 || pk < pk1);
        if (!valid) continue;
        const uint32_t nb = below + on, na = above + on;
        float4 bb = bhi, ba = blo;
        s3(bb, a, pk);
        s3(ba, a, pk);
        const float sb = surf(blo, bb), sa = surf(ba, bhi);
        const float cost =
            __fadd_rn(ct, __fmul_rn(ci, __fdiv_rn(__fadd_rn(__fmul_rn(sb, (float)nb), __fmul_rn(sa, (float)na)), A)));
        if (cost < mc) {   // NaN / inf never win; an earlier axis keeps ties
            mc = cost;
            mkey = a * 32u + lane;
            m_nb = nb;
            m_na = na;
            m_pk = pk;
        }
    }
    // argmin over (cost, axis, plane): costs are +0 .. +inf (ct >= 0, ci > 0,
    // surfaces and counts >= 0; NaN never replaced kInf), so their bit
    // patterns order as the values do: the least cost, then the least key
    const uint32_t cbits = __float_as_uint(mc);
    const uint32_t mbits = __reduce_min_sync(0xffffffffu, cbits);
    const uint32_t bk = __reduce_min_sync(0xffffffffu, cbits == mbits ? mkey : 0xffffffffu);
    const float bc = __uint_as_float(mbits);
    Decision best{-1, 0.0f, 0, 0, kInf, 0};
    const uint32_t src = bk & 31u;
    const float pk = __shfl_sync(0xffffffffu, m_pk, src);
    const uint32_t nb = __shfl_sync(0xffffffffu, m_nb, src), na = __shfl_sync(0xffffffffu, m_na, src);
    if (bc < kInf) {
        best.axis = (int)(bk >> 5);
        best.plane = pk;
        best.nb = nb;
        best.na = na;
        best.cost = bc;
        best.bin = (int)src;
    }
    if (best.axis >= 0 && !(best.cost < __fmul_rn(ci, (float)cnt))) best.axis = -1;
    return best;
}

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
struct LevelArgs {
    // triangle bounds, 32 bytes (one memory sector) each: {lo.x, hi.x, lo.y,
    // hi.y}, {lo.z, hi.z, -, -}
    const float4 *tb;
    uint32_t wave;          // four CTAs per SM
    // the level's nodes and references, ping-pong by level parity: level L
    // reads buffer L & 1 and writes the other (the accessors below)
    float4 *lo_buf[2], *hi_buf[2];
    uint4 *info_buf[2];
    uint32_t *refs_buf[2], *ref_node_buf[2];
    int32_t *axis;
    float *plane;
    uint2 *cnt;
    float4 *split;          // per node: axis (int bits, -1 = leaf), plane, node min / max on the axis
    uint4 *scat;            // per node: where its references go (written by the plan scan)
    uint4 *chunks;          // large rank, node slot, first reference, end
    uint32_t *medium_slot;
    uint32_t *hist;
    uint32_t *done;
    uint2 *out_nodes;
    uint32_t *out_refs;
    uint32_t *out_ropes;
    float4 *out_cbox;
    BuildCounters *ctr;
    LevelCounters *lc, *nlc;
    uint32_t *err;
    uint32_t *epoch;        // build counter (k_root increments it)
    uint32_t level;
    float ct, ci;
    uint32_t max_depth, leaf_size;
    uint32_t cap_refs, cap_nodes, cap_level, cap_large, cap_chunks, cap_medium;
    uint32_t exact_max;     // 0: binned everywhere; else nodes <= exact_max refs take the exact SAH
    // learned proposer
    int learned, record;
    uint32_t *learn_slot;   // proposer row -> node slot
    LearnBin *learn_bin;    // proposer row -> binned decision
    uint2 *learn_prop;      // proposer row -> proposed bins, one byte each (0xff: none)
    float *feat;            // proposer row -> features
    int32_t *prop_log;      // optional: compact node -> its 8 proposed bins
    uint32_t cap_learn;
    MlpDevice mlp;
    float *rec_X;
    int32_t *rec_y;
    uint32_t *rec_rows, rec_cap;
    float fallback_ratio;
    uint32_t topk;
    uint32_t spin_limit;       // polls before a bounded wait gives up
    uint32_t withhold_level;   // test aid: at this level plan tile 0 never publishes its done flag
    // deferred subtrees: a decidable node of 2..defer (<= kDeferMax)
    // references is recorded (d_root: compact index, reference offset, count,
    // depth; d_lo / d_hi: its cell; defer_refs: its references) and built
    // after the levels; 0: none
    uint32_t defer;
    uint32_t defer_level;      // the first level whose nodes may be deferred
    uint4 *d_root;
    float4 *d_lo, *d_hi;
    uint32_t *defer_refs;
    uint32_t cap_defer;
    uint32_t *sc_rec;          // subtree scratch node slots, 16 words each (SubWord)
    uint4 *sc_ref;             // subtree scratch reference slots: (subtree, local index, triangle, -)
    uint32_t cap_sc_nodes, cap_sc_refs;
    uint2 *st_cnt, *st_root, *st_base;   // per subtree: (nodes, refs), root entry, place

    // (selects rather than indexing: a copy of the struct whose level changes
    // stays in registers)
    __device__ __forceinline__ bool odd() const { return (level & 1u) != 0; }
    __device__ __forceinline__ float4 *n_lo() const { return odd() ? lo_buf[1] : lo_buf[0]; }
    __device__ __forceinline__ float4 *n_hi() const { return odd() ? hi_buf[1] : hi_buf[0]; }
    __device__ __forceinline__ uint4 *n_info() const { return odd() ? info_buf[1] : info_buf[0]; }
    __device__ __forceinline__ uint32_t *refs() const { return odd() ? refs_buf[1] : refs_buf[0]; }
    __device__ __forceinline__ uint32_t *ref_node() const { return odd() ? ref_node_buf[1] : ref_node_buf[0]; }
    __device__ __forceinline__ float4 *nx_lo() const { return odd() ? lo_buf[0] : lo_buf[1]; }
    __device__ __forceinline__ float4 *nx_hi() const { return odd() ? hi_buf[0] : hi_buf[1]; }
    __device__ __forceinline__ uint4 *nx_info() const { return odd() ? info_buf[0] : info_buf[1]; }
    __device__ __forceinline__ uint32_t *nx_refs() const { return odd() ? refs_buf[0] : refs_buf[1]; }
    __device__ __forceinline__ uint32_t *nx_ref_node() const { return odd() ? ref_node_buf[0] : ref_node_buf[1]; }
};

// true (on every thread of the CTA alike) when an earlier kernel of this build
// hit an error after which its data may be inconsistent; the kernel then does
// nothing. Called after wait_prior_grid by every thread. (Loads that a kernel
// issues before it overlap the error word's.)
__device__ __forceinline__ bool level_aborted(const LevelArgs &A) {
    return __syncthreads_or((int)(__ldcg(A.err) & kErrAbort)) != 0;
}

__device__ __forceinline__ void load_bounds(const LevelArgs &A, uint32_t tri, float4 &lo, float4 &hi) {
    const float4 a = A.tb[2 * (size_t)tri], b = A.tb[2 * (size_t)tri + 1];
    lo = make_float4(a.x, a.z, b.x, 0.0f);
    hi = make_float4(a.y, a.w, b.y, 0.0f);
}
// one axis: (lo, hi)
__device__ __forceinline__ float2 load_bounds_axis(const LevelArgs &A, uint32_t tri, uint32_t axis) {
    return reinterpret_cast<const float2 *>(A.tb)[4 * (size_t)tri + axis];
}

__device__ __forceinline__ bool decidable(const LevelArgs &A, uint32_t cnt) {
    return cnt > A.leaf_size && A.level < A.max_depth;
}

// classes of a splittable node by its reference count: small (one warp,
// k_small), medium (exact SAH, one CTA, when exact_max reaches it) and large
// (chunked binned histograms, or the proposer). is_exact: above a warp's 32
// references and within exact_max
__device__ __forceinline__ bool is_exact(const LevelArgs &A, uint32_t c) {
    return A.exact_max >= kWarpExact && c > kWarpExact && c <= A.exact_max;
}
// learned mode: a proposer row (33..1024 references)
__device__ __forceinline__ bool is_learn(const LevelArgs &A, uint32_t c) {
    return A.learned && c > kWarpExact && c <= kLearnMax;
}
// ... whose histogram one warp builds (in the medium list; larger ones are chunks)
__device__ __forceinline__ bool is_row_warp(const LevelArgs &A, uint32_t c) { return is_learn(A, c) && c <= kSmall; }
// (nodes of up to kExactWarp references are one warp's work too, unless
// training rows are recorded, which the CTA does)
constexpr uint32_t kExactWarp = 128;
__device__ __forceinline__ bool is_medium(const LevelArgs &A, uint32_t c) {
    return (is_exact(A, c) && (c > kExactWarp || A.record)) || is_row_warp(A, c);
}
// large: k_hist's chunked histograms (in learned mode the proposer rows too, so
// that the proposer's chain needs nothing from k_small)
// A node of 33..256 references is a warp's work where a level has many of them
// and a CTA's chunk where it has few: one warp takes 8 us more for it (levels
// of up to 0 / 32k / 64k / 128k references: a frame of 3.5k triangles 529 / 519 /
// 519 / 519 us, of 24k 945 / 922 / 917 / 915, of 200k 1,656 / 1,652 / 1,654 / 1,653).
constexpr uint32_t kFewRefs = 131072;
__device__ __forceinline__ bool is_large(const LevelArgs &A, uint32_t c, uint32_t refs) {
    return (c > (refs <= kFewRefs ? kWarpExact : kSmall) || is_learn(A, c)) && !is_exact(A, c) && !is_row_warp(A, c);
}
// References per chunk of a node of more than kChunk references, in a level
// of `refs` references: small enough that the level's chunks fill k_decide's
// one wave of four CTAs per SM (A.wave), since a chunk of 256 takes 1.5 us less
// than one of 1024 and the levels of small scenes have few of them. A node of
// up to kChunk is one chunk: it then needs no sum in global memory.
__device__ __forceinline__ uint32_t chunk_refs(const LevelArgs &A, uint32_t refs) {
    // (refs / A.wave up to 256, up to 512)
    return refs < (kChunkMin + 1) * A.wave ? kChunkMin
                                           : (refs < (2 * kChunkMin + 1) * A.wave ? 2 * kChunkMin : kChunk);
}
__device__ __forceinline__ uint32_t node_chunks(uint32_t c, uint32_t per) {
    return c <= kChunk ? 1u : (c + per - 1) / per;
}
// a decidable node of 2..A.defer references roots a deferred subtree
constexpr uint32_t kDeferMax = 32;   // one reference per lane
constexpr int kDeferAxis = -2;       // the decision that records a deferred root
__device__ __forceinline__ bool is_deferred(const LevelArgs &A, uint32_t c) {
    return c >= 2 && c <= A.defer && A.level >= A.defer_level;
}

// the build's counters zeroed, the triangles' bounds, and the root node and
// references of level 0; a root that is a large node is the first of them (one launch: a memset and two kernels cost a small scene 5 us more)
static_assert(sizeof(BuildCounters) % 4 == 0, "cleared word by word");
__global__ void __launch_bounds__(256) k_root(LevelArgs A, const float *box, const float4 *__restrict__ V,
                                              const uint4 *__restrict__ T, uint32_t nt, float4 *__restrict__ tb) {
    const bool dec = nt > A.leaf_size && A.max_depth > 0;
    const bool medium = dec && is_medium(A, nt);
    const bool large = dec && is_large(A, nt, nt);
    const uint32_t per = nt <= kChunk ? kChunk : chunk_refs(A, nt), nch = large ? node_chunks(nt, per) : 0u;
    if (blockIdx.x == 0) {
        uint32_t *w = reinterpret_cast<uint32_t *>(A.ctr);
        for (uint32_t i = threadIdx.x; i < sizeof(BuildCounters) / 4; i += blockDim.x) w[i] = 0;
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *A.epoch += 1u;
        LevelCounters *l0 = &A.ctr->lvl[0];
        l0->nodes = 1;
        l0->refs = nt;
        l0->nodes_total = 2;
        l0->leafrefs_total = 0;
        l0->n_large = large ? 1u : 0u;
        l0->n_chunks = nch;
        l0->n_medium = medium ? 1u : 0u;
        if (medium) A.medium_slot[0] = 0;
        // level 0's node buffers (A.level is 0)
        A.n_lo()[0] = make_float4(box[0], box[1], box[2], 0.0f);
        A.n_hi()[0] = make_float4(box[4], box[5], box[6], 0.0f);
        A.n_info()[0] = make_uint4(0, nt, 0, 0);
        A.out_nodes[1] = make_uint2(kLeafTag, 0);
        A.out_nodes[0] = make_uint2(kLeafTag, 0);
        // root cell = scene box, no ropes (every face is the scene boundary)
        A.out_cbox[0] = make_float4(box[0], box[1], box[2], 0.0f);
        A.out_cbox[1] = make_float4(box[4], box[5], box[6], 0.0f);
        for (int f = 0; f < 6; f++) A.out_ropes[f] = 0xffffffffu;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        uint4 t = T[i];
        float4 a = V[t.x], b = V[t.y], c = V[t.z];
        tb[2 * (size_t)i] = make_float4(mnf(mnf(a.x, b.x), c.x), mxf(mxf(a.x, b.x), c.x), mnf(mnf(a.y, b.y), c.y),
                                        mxf(mxf(a.y, b.y), c.y));
        tb[2 * (size_t)i + 1] = make_float4(mnf(mnf(a.z, b.z), c.z), mxf(mxf(a.z, b.z), c.z), 0.0f, 0.0f);
        A.refs()[i] = i;
        A.ref_node()[i] = 0;
    }
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nch; k += gridDim.x * blockDim.x)
        A.chunks[k] = make_uint4(0, 0, k * per, min(nt, (k + 1) * per));
}



// level totals of the decisions (what the capacity guard needs), kept per
// thread and flushed once per CTA
struct Tally {
    uint32_t leafrefs = 0, leafnodes = 0, splits = 0, next = 0, childrefs = 0, deferrefs = 0, defernodes = 0;
    __device__ void add(const Decision &d, uint32_t cnt) {
        if (d.axis == kDeferAxis) {
            deferrefs += cnt;
            defernodes += 1;
        } else if (d.axis < 0) {
            leafrefs += cnt;
            leafnodes += cnt ? 1u : 0u;
        } else {
            splits += 1;
            next += (d.nb > 0 ? 1u : 0u) + (d.na > 0 ? 1u : 0u);
            childrefs += d.nb + d.na;
        }
    }
};

// all threads of the CTA call it once, at the end of the kernel
constexpr int kTallies = 7;
__device__ void tally_flush(const LevelArgs &A, const Tally &t, uint32_t *sh) {
    if (threadIdx.x < kTallies) sh[threadIdx.x] = 0;
    __syncthreads();
    if (t.leafrefs) atomicAdd(&sh[0], t.leafrefs);
    if (t.leafnodes) atomicAdd(&sh[1], t.leafnodes);
    if (t.splits) atomicAdd(&sh[2], t.splits);
    if (t.next) atomicAdd(&sh[3], t.next);
    if (t.childrefs) atomicAdd(&sh[4], t.childrefs);
    if (t.deferrefs) atomicAdd(&sh[5], t.deferrefs);
    if (t.defernodes) atomicAdd(&sh[6], t.defernodes);
    __syncthreads();
    // t_leafrefs .. t_defernodes are consecutive fields of LevelCounters
    if (threadIdx.x < kTallies && sh[threadIdx.x]) atomicAdd(&A.lc->t_leafrefs + threadIdx.x, sh[threadIdx.x]);
}

// the node's bounds blo / bhi, when the caller has them
__device__ __forceinline__ void write_decision(const LevelArgs &A, uint32_t s, const Decision &d, float4 blo,
                                              float4 bhi) {
    A.axis[s] = d.axis;
    A.plane[s] = d.plane;
    A.cnt[s] = make_uint2(d.nb, d.na);
    // the partition's view of the decision in one 16-byte record
    float l = 0.0f, h = 0.0f;
    if (d.axis >= 0) {
        l = c3(blo, (uint32_t)d.axis);
        h = c3(bhi, (uint32_t)d.axis);
    }
    A.split[s] = make_float4(__int_as_float(d.axis), d.plane, l, h);
}

__device__ __forceinline__ void write_decision(const LevelArgs &A, uint32_t s, const Decision &d) {
    if (d.axis >= 0) write_decision(A, s, d, A.n_lo()[s], A.n_hi()[s]);
    else write_decision(A, s, d, make_float4(0, 0, 0, 0), make_float4(0, 0, 0, 0));
}

// global histogram read past L1 (other CTAs wrote it with atomics)
struct GHist {
    const uint32_t *p;
    __device__ uint32_t operator[](uint32_t i) const { return __ldcg(p + i); }
};

// ---------------------------------------------------------------------------
// proposer features of one node (one warp), from the node's binned histogram
// (the counts the binned SAH itself uses, exact integers, so every kernel that
// builds the histogram gives the same features): per axis the 32 lower-bound
// bin counts and the 32 upper-bound bin counts as fractions of the node's
// references (192), the extents over the largest extent (3), depth /
// max_depth, references / 1024, 3 zeros = 200.
// ---------------------------------------------------------------------------
template <class HistPtr>
__device__ void hist_features(HistPtr H, uint32_t cnt, float4 blo, float4 bhi, uint32_t level, uint32_t max_depth,
                              float *out) {
    const uint32_t lane = threadIdx.x & 31u;
    const float inv = cnt ? 1.0f / (float)cnt : 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < 6; k++) {
        const uint32_t i = lane + 32u * k;                 // 0..191
        const uint32_t a = i >> 6, j = i & 63u;
        out[i] = (float)H[a * 96 + j] * inv;               // j < 32: lower-bound bins, else upper-bound bins
    }
    if (lane == 0) {
        const float ex = bhi.x - blo.x, ey = bhi.y - blo.y, ez = bhi.z - blo.z;
        const float m = fmaxf(ex, fmaxf(ey, ez));
        const float im = m > 0.0f ? 1.0f / m : 0.0f;
        out[192] = ex * im;
        out[193] = ey * im;
        out[194] = ez * im;
        out[195] = (float)level / (float)max_depth;
        out[196] = (float)cnt * (1.0f / 1024.0f);
        out[197] = out[198] = out[199] = 0.0f;
    }
    __syncwarp();
}

// training label of an exactly searched node: axis * 32 + the bin b of the
// chosen plane p on its axis (p_b <= p < p_{b+1}, p_k = min + ext * k / 32)
__device__ __forceinline__ int32_t exact_label(int axis, float p, float4 blo, float4 bhi) {
    const float l = c3(blo, (uint32_t)axis), h = c3(bhi, (uint32_t)axis), ext = __fsub_rn(h, l);
    int b = __float2int_rz(__fmul_rn(__fsub_rn(p, l), __fdividef(32.0f, ext)));
    b = b < 0 ? 0 : (b > (int)kBins - 1 ? (int)kBins - 1 : b);
    while (b > 0 && p < plane_k(l, ext, (uint32_t)b)) b--;
    while (b < (int)kBins - 1 && p >= plane_k(l, ext, (uint32_t)b + 1)) b++;
    return axis * 32 + b;
}

// ---------------------------------------------------------------------------
// exact SAH (no reference counterpart; the oracle restates it): every clipped
// reference bound on every axis with a positive extent is a candidate plane p
// (+0.0f turns a -0 bound into +0), with
//   below = #(lo < p) + #(flat at p),  above = #(hi > p) + #(flat at p)
// -- the partition's own classification; the lowest cost wins, ties to the lower
// axis, then the lower plane, as in the oracle's loop.
// ---------------------------------------------------------------------------
// Nodes of at most 32 references, one warp, one reference per lane. A plane p
// strictly inside the node needs no clipped bounds (lo < p says the same of
// the triangle's own bound), and a reference flat on an axis (lo == hi == v)
// goes below for v <= p and above for v >= p, which the bounds one step
// outside v say with the plain comparisons. So with lane_bounds' values
//   below(p) = #(lo < p),  above(p) = #(hi > p)
// hold for every plane either search costs, and the partition is the same two
// comparisons.
__device__ __forceinline__ void lane_bounds(float4 &lo, float4 &hi) {
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        // a NaN bound clips to the node's side
        const float l = fmaxf(c3(lo, a), -kInf), h = fminf(c3(hi, a), kInf);
        s3(lo, a, l == h ? nextafterf(l, -kInf) : l);
        s3(hi, a, l == h ? nextafterf(h, kInf) : h);
    }
}

// a warp's scratch: the bounds of a node's references, packed (the set lanes
// in order), 32 values per axis and side: lane_bounds' values, then the
// triangles' own (the exact search's candidates)
constexpr uint32_t kLaneScratch = 12 * 32;
static_assert(kLaneScratch <= kWarpScratch && kWarpScratch % 4 == 0, "the packed bounds fit a warp's scratch");

// the set lanes' bounds (rank: the lane's place among them, c of them) to S,
// padded to a multiple of four with references that no plane counts
template <bool EXACT>
__device__ __forceinline__ void lanes_pack(float *S, bool in, uint32_t rank, uint32_t c, float4 tlo, float4 thi,
                                           float4 nlo, float4 nhi) {
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();   // the previous node's readers are done
    if (in) {
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            S[(2 * a) * 32 + rank] = c3(nlo, a);
            S[(2 * a + 1) * 32 + rank] = c3(nhi, a);
            if (EXACT) {
                S[(6 + 2 * a) * 32 + rank] = c3(tlo, a);
                S[(7 + 2 * a) * 32 + rank] = c3(thi, a);
            }
        }
    }
    if (lane >= c && lane < ((c + 3u) & ~3u)) {
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            S[(2 * a) * 32 + lane] = kInf;
            S[(2 * a + 1) * 32 + lane] = -kInf;
        }
    }
    __syncwarp();
}

// surface times references of nb references in a below cell that is db long on
// axis a and na in an above cell that is da long, of a node with extents ext
__device__ __forceinline__ float bounds_num(uint32_t a, float db, float da, float4 ext, float nb, float na) {
    const float bx = a == 0 ? db : ext.x, by = a == 1 ? db : ext.y, bz = a == 2 ? db : ext.z;
    const float ax = a == 0 ? da : ext.x, ay = a == 1 ? da : ext.y, az = a == 2 ? da : ext.z;
    const float sb =
        __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(bx, by), __fmul_rn(bz, by)), __fmul_rn(bx, bz)));
    const float sa =
        __fmul_rn(2.0f, __fadd_rn(__fadd_rn(__fmul_rn(ax, ay), __fmul_rn(az, ay)), __fmul_rn(ax, az)));
    return __fadd_rn(__fmul_rn(sb, nb), __fmul_rn(sa, na));
}
// ... and the cost, Anode the node's surface
__device__ __forceinline__ float bounds_cost(uint32_t a, float db, float da, float4 ext, float Anode, float nb,
                                             float na, float ct, float ci) {
    return __fadd_rn(ct, __fmul_rn(ci, __fdiv_rn(bounds_num(a, db, da, ext, nb, na), Anode)));
}
// ... split at the plane pk
__device__ __forceinline__ float plane_cost(uint32_t a, float pk, float l, float h, float4 ext, float Anode, float nb,
                                            float na, float ct, float ci) {
    return bounds_cost(a, __fsub_rn(pk, l), __fsub_rn(h, pk), ext, Anode, nb, na, ct, ci);
}

// 1 where a < b, else 0
__device__ __forceinline__ float f_less(float a, float b) {
    float r;
    asm("set.lt.f32.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// the binned SAH of a packed node: lane k counts and costs plane k of every
// axis (sah_warp's planes, counts and argmin). Counting c references takes
// about 14 instructions each; a histogram costs about 350 whatever c is
// (clearing, bins, atomics, scans), and the subtree pass's nodes hold 9
// references on average.
// (COUNTS: also the winner's counts, which the subtree pass does not need; the
// counts are kept as floats, which hold them exactly and cost needs)
template <bool COUNTS>
__device__ __forceinline__ Decision sah_lanes_binned(const float *S, uint32_t c, float4 blo, float4 bhi, float ct,
                                                     float ci) {
    const uint32_t lane = threadIdx.x & 31u;
    const float Anode = surf(blo, bhi);
    const float4 ext = make_float4(__fsub_rn(bhi.x, blo.x), __fsub_rn(bhi.y, blo.y), __fsub_rn(bhi.z, blo.z), 0.0f);
    float pk[3], nb[3] = {0, 0, 0}, na[3] = {0, 0, 0};
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) pk[a] = plane_k(c3(blo, a), c3(ext, a), lane);
    for (uint32_t i = 0; i < c; i += 4) {
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float4 L = *reinterpret_cast<const float4 *>(S + (2 * a) * 32 + i);
            const float4 H = *reinterpret_cast<const float4 *>(S + (2 * a + 1) * 32 + i);
            nb[a] += f_less(L.x, pk[a]);
            na[a] += f_less(pk[a], H.x);
            nb[a] += f_less(L.y, pk[a]);
            na[a] += f_less(pk[a], H.y);
            nb[a] += f_less(L.z, pk[a]);
            na[a] += f_less(pk[a], H.z);
            nb[a] += f_less(L.w, pk[a]);
            na[a] += f_less(pk[a], H.w);
        }
    }
    if (!COUNTS) {
        // cost = ct + ci (num / Anode) does not fall as num rises, so the least
        // numerator has the least cost, and a numerator above it by one part in
        // 100,000 a greater one after rounding, as long as the cost is not above
        // 8 times its second term: one division instead of three per lane (a
        // frame of 200k triangles 1,594 -> 1,576 us, of 1M 2,665 -> 2,640); near
        // ties and unusual magnitudes go on below
        float num[3];
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float l = c3(blo, a), h = c3(bhi, a);
            const float pk1 = __shfl_down_sync(0xffffffffu, pk[a], 1);
            const bool ok = c3(ext, a) > 0.0f && lane >= 1 && pk[a] > l && pk[a] < h && (lane == 31 || pk[a] < pk1);
            num[a] = ok ? bounds_num(a, __fsub_rn(pk[a], l), __fsub_rn(h, pk[a]), ext, nb[a], na[a]) : kInf;
        }
        const float nmin = __uint_as_float(
            __reduce_min_sync(0xffffffffu, __float_as_uint(fminf(fminf(num[0], num[1]), num[2]))));
        const float q = __fdiv_rn(nmin, Anode), m = __fmul_rn(ci, q), cost = __fadd_rn(ct, m);
        if (nmin >= 1e-30f && q >= 1e-30f && m >= 1e-30f && fabsf(cost) <= __fmul_rn(8.0f, m) && cost < kInf) {
            const float thr = __fmul_rn(nmin, 1.00001f);
            const uint32_t v0 = __ballot_sync(0xffffffffu, num[0] <= thr), v1 = __ballot_sync(0xffffffffu, num[1] <= thr),
                           v2 = __ballot_sync(0xffffffffu, num[2] <= thr);
            if (__popc(v0) + __popc(v1) + __popc(v2) == 1) {
                const int ax = v0 ? 0 : (v1 ? 1 : 2);
                const int src = __ffs(v0 | v1 | v2) - 1;
                const float p = __shfl_sync(0xffffffffu, v0 ? pk[0] : (v1 ? pk[1] : pk[2]), src);
                const bool split = cost < __fmul_rn(ci, (float)c);
                return Decision{split ? ax : -1, p, 0, 0, cost, src};
            }
        }
    }
    float mc = kInf, m_pk = 0.0f;
    uint32_t mkey = 0xffffffffu, m_n = 0;
#pragma unroll
    for (uint32_t a = 0; a < 3; a++) {
        const float l = c3(blo, a), h = c3(bhi, a);
        if (!(c3(ext, a) > 0.0f)) continue;
        const float pk1 = __shfl_down_sync(0xffffffffu, pk[a], 1);   // plane k + 1 (lane 31: unused)
        if (!(lane >= 1 && pk[a] > l && pk[a] < h && (lane == 31 || pk[a] < pk1))) continue;
        const float cost = plane_cost(a, pk[a], l, h, ext, Anode, nb[a], na[a], ct, ci);
        if (cost < mc) {   // NaN / inf never win; an earlier axis keeps ties
            mc = cost;
            mkey = a * 32u + lane;
            if (COUNTS) m_n = (uint32_t)nb[a] | ((uint32_t)na[a] << 16);
            m_pk = pk[a];
        }
    }
    // as in sah_warp: the least cost, then the least key
    const uint32_t cbits = __float_as_uint(mc);
    const uint32_t mbits = __reduce_min_sync(0xffffffffu, cbits);
    const uint32_t bk = __reduce_min_sync(0xffffffffu, cbits == mbits ? mkey : 0xffffffffu);
    const float bc = __uint_as_float(mbits);
    Decision best{-1, 0.0f, 0, 0, kInf, 0};
    const uint32_t src = bk & 31u;
    const float p = __shfl_sync(0xffffffffu, m_pk, src);
    const uint32_t n = COUNTS ? __shfl_sync(0xffffffffu, m_n, src) : 0u;
    if (bc < kInf) best = Decision{(int)(bk >> 5), p, n & 0xffffu, n >> 16, bc, (int)src};
    if (best.axis >= 0 && !(best.cost < __fmul_rn(ci, (float)c))) best.axis = -1;
    return best;
}

// the lane of the warp with the least (cost, axis, plane); costs are +0 ..
// +inf, so their bits order as they do
__device__ __forceinline__ uint32_t warp_argmin(float cost, uint32_t ax, float pk) {
    const uint32_t mbits = __reduce_min_sync(0xffffffffu, __float_as_uint(cost));
    bool win = __float_as_uint(cost) == mbits;
    const uint32_t bax = __reduce_min_sync(0xffffffffu, win ? ax : 0xffffffffu);
    win = win && ax == bax;
    const uint32_t pb = __float_as_uint(pk), po = (pb & 0x80000000u) ? ~pb : (pb | 0x80000000u);
    const uint32_t bpo = __reduce_min_sync(0xffffffffu, win ? po : 0xffffffffu);
    return (__ffs(__ballot_sync(0xffffffffu, win && po == bpo)) - 1u) & 31u;
}

// the exact SAH of a packed node: candidate q of 6 c (axis, side, reference)
// is taken by lane q % 32, which counts the references below and above it;
// two sorts per axis and a binary search per candidate and list cost four
// times as much at the subtree pass's 9 references per node
template <bool COUNTS>
__device__ __forceinline__ Decision sah_lanes_exact(const float *S, uint32_t c, float4 blo, float4 bhi, float ct,
                                                    float ci) {
    const uint32_t lane = threadIdx.x & 31u;
    const float Anode = surf(blo, bhi);
    const float4 ext = make_float4(__fsub_rn(bhi.x, blo.x), __fsub_rn(bhi.y, blo.y), __fsub_rn(bhi.z, blo.z), 0.0f);
    float mc = kInf, m_pk = 0.0f;
    uint32_t m_ax = 3, m_n = 0;
    for (uint32_t q0 = 0; q0 < 6 * c; q0 += 32) {
        const uint32_t q = min(q0 + lane, 6 * c - 1);   // (a repeated candidate changes nothing)
        const uint32_t a = (q >= 2 * c ? 1u : 0u) + (q >= 4 * c ? 1u : 0u), j = q - 2 * a * c;
        const float x = S[(6 + 2 * a + (j >= c ? 1u : 0u)) * 32 + (j >= c ? j - c : j)];
        const float pk = __fadd_rn(x, 0.0f);
        const float l = c3(blo, a), h = c3(bhi, a);
        float nb = 0.0f, na = 0.0f;
        const float *Sl = S + 64 * a, *Sh = Sl + 32;
        for (uint32_t i = 0; i < c; i += 4) {
            const float4 L = *reinterpret_cast<const float4 *>(Sl + i);
            const float4 H = *reinterpret_cast<const float4 *>(Sh + i);
            nb += f_less(L.x, pk);
            na += f_less(pk, H.x);
            nb += f_less(L.y, pk);
            na += f_less(pk, H.y);
            nb += f_less(L.z, pk);
            na += f_less(pk, H.z);
            nb += f_less(L.w, pk);
            na += f_less(pk, H.w);
        }
        // (an axis without extent has no plane strictly inside)
        if (!(pk > l && pk < h)) continue;
        const float cost = plane_cost(a, pk, l, h, ext, Anode, nb, na, ct, ci);
        if (cost < mc || (cost == mc && a == m_ax && pk < m_pk)) {   // a rises with q
            mc = cost;
            m_ax = a;
            m_pk = pk;
            if (COUNTS) m_n = (uint32_t)nb | ((uint32_t)na << 16);
        }
    }
    // (equal keys are the same plane with the same counts)
    const uint32_t src = warp_argmin(mc, m_ax, m_pk);
    mc = __shfl_sync(0xffffffffu, mc, src);
    m_ax = __shfl_sync(0xffffffffu, m_ax, src);
    m_pk = __shfl_sync(0xffffffffu, m_pk, src);
    if (COUNTS) m_n = __shfl_sync(0xffffffffu, m_n, src);
    Decision best{-1, 0.0f, 0, 0, kInf, 0};
    if (mc < kInf) best = Decision{(int)m_ax, m_pk, m_n & 0xffffu, m_n >> 16, mc, 0};
    if (best.axis >= 0 && !(best.cost < __fmul_rn(ci, (float)c))) best.axis = -1;
    return best;
}

// a node of at most 32 references of the level, one per lane
template <bool EXACT>
__device__ __forceinline__ Decision sah_warp32(const LevelArgs &A, float *S, uint4 info, float4 blo, float4 bhi) {
    const uint32_t lane = threadIdx.x & 31u, c = info.y;
    float4 tlo = make_float4(0, 0, 0, 0), thi = tlo;
    if (lane < c) {
        const uint32_t tri = A.refs()[info.x + lane];
        load_bounds(A, tri, tlo, thi);
    }
    float4 nlo = tlo, nhi = thi;
    lane_bounds(nlo, nhi);
    lanes_pack<EXACT>(S, lane < c, lane, c, tlo, thi, nlo, nhi);
    return EXACT ? sah_lanes_exact<true>(S, c, blo, bhi, A.ct, A.ci)
                 : sah_lanes_binned<true>(S, c, blo, bhi, A.ct, A.ci);
}

// Exact SAH of a node of more than 32 references by a group of NT threads (a
// warp: up to 128 references; a CTA of 256: up to 1024), without sorting.
//   1. every clipped bound strictly inside the node goes to its bin's bucket
//      (32 bins per axis, a counting sort on the bins); bounds at the node's
//      sides only count;
//   2. a bin's candidates cannot cost less than its lower bound: the count
//      below and the below surface at the bin's lower edge, the count above
//      and the above surface at its upper edge. Every operation of the cost
//      is monotonic in these four, rounded or not, so the bound holds for the
//      rounded costs exactly;
//   3. the candidates of each axis's bin of least bound are costed (each
//      counts the bounds of its own bin's two buckets), then those of every
//      bin whose bound is not above the cost found.
// A 200k-triangle frame's 25,000 such nodes cost two rounds of few candidates
// each instead of three sorts and 6 binary searches per reference: 2,358 us of
// bitonic sorts (one CTA per node) before.
// A bound flat on its axis is kept one step outside its value (lane_bounds)
// and flagged; a flat bound equal to a bin's edge lies in another bin's bucket
// and is added from `on`.
template <uint32_t NT>
struct ExactSmem {
    static constexpr uint32_t kCap = 4 * NT;
    // bin counts, then the buckets' cursors ([axis * 64 + side * 32 + bin]),
    // then the candidates of the selected bins before each bin (97)
    uint32_t H[196];
    uint32_t S[6 * 33];        // per axis and side: bounds in the bins before
    uint32_t on[3 * 32];       // flat bounds on the bin's lower plane
    float P[kPlanes];          // planes
    uint32_t clip[6];          // bounds at (or past) the node's side
    uint32_t best;             // least cost so far (bits)
    uint32_t flat[6 * kCap / 32];
    float B[6 * kCap];         // buckets
    uint32_t w_cost[NT / 32], w_ax[NT / 32], w_nb[NT / 32], w_na[NT / 32];
    float w_pk[NT / 32];
};

template <uint32_t NT>
__device__ __forceinline__ void group_sync() {
    if (NT == 32) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ bool refine_better(float c, uint32_t a, float p, float bc, uint32_t ba, float bp) {
    return c < bc || (c == bc && (a < ba || (a == ba && p < bp)));
}

// the group's least (cost, axis, plane) with its counts, on every thread (S:
// shared memory with the arrays w_cost .. w_pk)
template <uint32_t NT, class Smem>
__device__ __forceinline__ void group_argmin(Smem &S, float &mc, uint32_t &m_ax, float &m_pk, uint32_t &m_nb,
                                             uint32_t &m_na) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t src = warp_argmin(mc, m_ax, m_pk);
    if (NT > 32) {
        if (lane == src) {
            const uint32_t w = threadIdx.x >> 5;
            S.w_cost[w] = __float_as_uint(mc);
            S.w_ax[w] = m_ax;
            S.w_pk[w] = m_pk;
            S.w_nb[w] = m_nb;
            S.w_na[w] = m_na;
        }
        __syncthreads();
        const uint32_t w = min(lane, NT / 32 - 1);
        mc = __uint_as_float(S.w_cost[w]);
        m_ax = S.w_ax[w];
        m_pk = S.w_pk[w];
        m_nb = S.w_nb[w];
        m_na = S.w_na[w];
        src = warp_argmin(mc, m_ax, m_pk);
    }
    mc = __shfl_sync(0xffffffffu, mc, src);
    m_ax = __shfl_sync(0xffffffffu, m_ax, src);
    m_pk = __shfl_sync(0xffffffffu, m_pk, src);
    m_nb = __shfl_sync(0xffffffffu, m_nb, src);
    m_na = __shfl_sync(0xffffffffu, m_na, src);
}

template <uint32_t NT>
__device__ Decision sah_exact_group(const LevelArgs &A, uint4 info, float4 blo, float4 bhi, ExactSmem<NT> &S) {
    constexpr uint32_t kCap = ExactSmem<NT>::kCap;
    const uint32_t lane = threadIdx.x & 31u, tid = NT == 32 ? lane : threadIdx.x;
    const uint32_t cnt = info.y;
    const float Anode = surf(blo, bhi);
    const float4 ext = make_float4(__fsub_rn(bhi.x, blo.x), __fsub_rn(bhi.y, blo.y), __fsub_rn(bhi.z, blo.z), 0.0f);
    group_sync<NT>();   // the previous node's readers are done
    for (uint32_t i = tid; i < 192; i += NT) S.H[i] = 0;
    for (uint32_t i = tid; i < 96; i += NT) {
        const uint32_t a = i >> 5;
        S.on[i] = 0;
        S.P[a * kPlaneRow + (i & 31u)] = (i & 31u) ? plane_k(c3(blo, a), c3(ext, a), i & 31u) : -kInf;
        if ((i & 31u) == 31) S.P[a * kPlaneRow + kBins] = kInf;
    }
    for (uint32_t i = tid; i < 6 * kCap / 32; i += NT) S.flat[i] = 0;
    if (tid < 6) S.clip[tid] = 0;
    if (tid == 6) S.best = __float_as_uint(kInf);
    // the thread's references, all loads issued together
    float4 tlo[4], thi[4];
    uint32_t tri[4], bins[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t r = tid + NT * k;
        tri[k] = r < cnt ? A.refs()[info.x + r] : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (tri[k] != 0xffffffffu) load_bounds(A, tri[k], tlo[k], thi[k]);
    group_sync<NT>();
    // 1. bins (5 bits each, lo then hi per axis), counts
    const float4 inv3 = bin_scale(blo, bhi);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (NT * k >= cnt) break;   // uniform
        const bool have = tri[k] != 0xffffffffu;
        if (!have) tlo[k] = bhi, thi[k] = blo;
        uint32_t w = 0;
        int bs[3], cs[3];
        bool ons[3];
        ref_bins(tlo[k], thi[k], blo, bhi, inv3, S.P, have, bs, cs, ons);
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float l = c3(blo, a), h = c3(bhi, a);
            if (!(c3(ext, a) > 0.0f)) continue;   // uniform
            const float lo = mxf(c3(tlo[k], a), l), hi = mnf(c3(thi[k], a), h);
            const int b = bs[a], c = cs[a];
            const bool on = ons[a];
            w |= ((uint32_t)b << (10 * a)) | ((uint32_t)c << (10 * a + 5));
            const uint32_t ml = __ballot_sync(0xffffffffu, have && !(lo > l));
            const uint32_t mh = __ballot_sync(0xffffffffu, have && !(hi < h));
            if (lane == 0) {
                if (ml) atomicAdd(&S.clip[2 * a], (uint32_t)__popc(ml));
                if (mh) atomicAdd(&S.clip[2 * a + 1], (uint32_t)__popc(mh));
            }
            if (have && lo > l) atomicAdd(&S.H[a * 64 + b], 1u);
            if (have && hi < h) atomicAdd(&S.H[a * 64 + 32 + c], 1u);
            if (have && on) atomicAdd(&S.on[a * 32 + b], 1u);
        }
        bins[k] = w;
    }
    group_sync<NT>();
    // the buckets' places
    for (uint32_t r = NT == 32 ? 0u : (tid >> 5); r < 6; r += NT / 32) {
        const uint32_t v = S.H[r * 32 + lane];
        uint32_t inc = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
            if ((int)lane >= d) inc += u;
        }
        S.S[r * 33 + lane] = S.H[r * 32 + lane] = inc - v;
        if (lane == 31) S.S[r * 33 + 32] = inc;
    }
    group_sync<NT>();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (tri[k] == 0xffffffffu) continue;
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float l = c3(blo, a), h = c3(bhi, a);
            if (!(c3(ext, a) > 0.0f)) continue;
            const float lo = mxf(c3(tlo[k], a), l), hi = mnf(c3(thi[k], a), h);
            const bool fl = lo == hi;
            if (lo > l) {
                const uint32_t pos = atomicAdd(&S.H[a * 64 + ((bins[k] >> (10 * a)) & 31u)], 1u);
                S.B[2 * a * kCap + pos] = fl ? nextafterf(lo, -kInf) : lo;
                if (fl) atomicOr(&S.flat[(2 * a * kCap + pos) >> 5], 1u << (pos & 31u));
            }
            if (hi < h) {
                const uint32_t pos = atomicAdd(&S.H[a * 64 + 32 + ((bins[k] >> (10 * a + 5)) & 31u)], 1u);
                S.B[(2 * a + 1) * kCap + pos] = fl ? nextafterf(hi, kInf) : hi;
                if (fl) atomicOr(&S.flat[((2 * a + 1) * kCap + pos) >> 5], 1u << (pos & 31u));
            }
        }
    }
    group_sync<NT>();
    // 2. the bins' lower bounds (one warp, lane = bin)
    float lb[3];
    uint32_t nc[3], taken = 0;
    float mc = kInf, m_pk = 0.0f;
    uint32_t m_ax = 3, m_nb = 0, m_na = 0;
    if (tid < 32) {
#pragma unroll
        for (uint32_t a = 0; a < 3; a++) {
            const float l = c3(blo, a), h = c3(bhi, a);
            const uint32_t *Sl = S.S + 2 * a * 33, *Sh = Sl + 33;
            nc[a] = Sl[lane + 1] - Sl[lane] + Sh[lane + 1] - Sh[lane];
            const float e0 = lane == 0 ? l : S.P[a * kPlaneRow + lane], e1 = lane == 31 ? h : S.P[a * kPlaneRow + lane + 1];
            lb[a] = bounds_cost(a, __fsub_rn(e0, l), __fsub_rn(h, e1), ext, Anode,
                                (float)(S.clip[2 * a] + Sl[lane]),
                                (float)(S.clip[2 * a + 1] + Sh[32] - Sh[lane + 1]), A.ct, A.ci);
        }
    }
    // 3. two rounds
    for (int round = 0; round < 2; round++) {
        if (tid < 32) {
            uint32_t base = 0;
            const float limit = __uint_as_float(S.best);
#pragma unroll
            for (uint32_t a = 0; a < 3; a++) {
                bool sel = nc[a] != 0;
                if (round == 0) {
                    // the least bound of the axis (bounds are not negative)
                    const uint32_t bits = sel ? __float_as_uint(lb[a]) : 0xffffffffu;
                    const uint32_t m = __reduce_min_sync(0xffffffffu, bits);
                    sel = sel && bits == m;
                    if (sel) taken |= 1u << a;
                } else {
                    sel = sel && !((taken >> a) & 1u) && !(lb[a] > limit);
                }
                const uint32_t v = sel ? nc[a] : 0u;
                uint32_t inc = v;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
                    if ((int)lane >= d) inc += u;
                }
                S.H[a * 32 + lane] = base + inc - v;
                base += __shfl_sync(0xffffffffu, inc, 31);
            }
            if (lane == 0) S.H[96] = base;
        }
        group_sync<NT>();
        const uint32_t M = S.H[96];
        for (uint32_t q = tid; q < M; q += NT) {
            uint32_t i = 0, n = 96;   // the last bin with H[i] <= q
            while (n > 1) {
                const uint32_t m = n >> 1;
                if (S.H[i + m] <= q) i += m;
                n -= m;
            }
            const uint32_t a = i >> 5, j = i & 31u;
            const uint32_t *Sl = S.S + 2 * a * 33, *Sh = Sl + 33;
            const uint32_t l0 = Sl[j], l1 = Sl[j + 1], h0 = Sh[j], h1 = Sh[j + 1];
            const float *Bl = S.B + 2 * a * kCap, *Bh = Bl + kCap;
            const uint32_t t = q - S.H[i];
            const bool side = t >= l1 - l0;
            const uint32_t pos = side ? h0 + t - (l1 - l0) : l0 + t;
            float x = side ? Bh[pos] : Bl[pos];
            if ((S.flat[((2 * a + (side ? 1u : 0u)) * kCap + pos) >> 5] >> (pos & 31u)) & 1u)
                x = nextafterf(x, side ? -kInf : kInf);
            const float pk = __fadd_rn(x, 0.0f), l = c3(blo, a), h = c3(bhi, a);
            if (!(pk > l && pk < h)) continue;
            uint32_t nb = S.clip[2 * a] + l0, na = S.clip[2 * a + 1] + Sh[32] - h1;
            for (uint32_t k = l0; k < l1; k++) nb += Bl[k] < pk ? 1u : 0u;
            for (uint32_t k = h0; k < h1; k++) na += Bh[k] > pk ? 1u : 0u;
            const float *Pa = S.P + a * kPlaneRow;
            if (!side) {
                if (j >= 1 && pk == Pa[j]) na += S.on[a * 32 + j];
            } else if (j < 31 && pk == Pa[j + 1]) {
                uint32_t b = j + 1;   // the bin whose bucket holds lower bounds equal to pk
                while (b < 31 && Pa[b + 1] <= pk) b++;
                nb += S.on[a * 32 + b];
            }
            const float cost = plane_cost(a, pk, l, h, ext, Anode, (float)nb, (float)na, A.ct, A.ci);
            if (refine_better(cost, a, pk, mc, m_ax, m_pk)) {
                mc = cost;
                m_ax = a;
                m_pk = pk;
                m_nb = nb;
                m_na = na;
            }
        }
        __syncwarp();
        const uint32_t wb = __reduce_min_sync(0xffffffffu, __float_as_uint(mc));
        if (lane == 0) atomicMin(&S.best, wb);
        group_sync<NT>();
    }
    group_argmin<NT>(S, mc, m_ax, m_pk, m_nb, m_na);
    Decision best{-1, 0.0f, 0, 0, kInf, 0};
    if (mc < kInf) best = Decision{(int)m_ax, m_pk, m_nb, m_na, mc, 0};
    if (best.axis >= 0 && !(best.cost < __fmul_rn(A.ci, (float)cnt))) best.axis = -1;
    return best;
}

// the binned SAH of a large node from its complete histogram (one warp): a
// proposer row keeps the binned decision and the features for k_refine_cta /
// k_refine_warp, every other node is decided here
template <class HistPtr>
__device__ __forceinline__ void finish_large(const LevelArgs &A, uint32_t s, const uint4 &info, float4 blo,
                                             float4 bhi, HistPtr H, Tally &tally) {
    const uint32_t lane = threadIdx.x & 31u;
    const Decision d = sah_warp(H, blo, bhi, info.y, A.ct, A.ci);
    if (is_learn(A, info.y)) {
        uint32_t row = 0;
        if (lane == 0) row = atomicAdd(&A.lc->n_learn, 1u);
        row = __shfl_sync(0xffffffffu, row, 0);
        if (row < A.cap_learn) {
            if (lane == 0) {
                A.learn_slot[row] = s;
                A.learn_bin[row] = LearnBin{d.cost, d.plane, d.axis, d.nb, d.na, {info.y, 0, 0}};
            }
            hist_features(H, info.y, blo, bhi, A.level, A.max_depth, A.feat + (size_t)row * 200);
            return;
        }
    }
    if (lane == 0) {
        write_decision(A, s, d);
        tally.add(d, info.y);
    }
}

// a small-node warp's shared memory (16-byte aligned in an array of them: the
// scratch is cleared and read 16 bytes at a time)
template <bool EXACT>
union alignas(16) WarpSmem {
    uint32_t scratch[kWarpScratch];
};
template <>
union alignas(16) WarpSmem<true> {
    uint32_t scratch[kWarpScratch];
    ExactSmem<32> exact;
};
static_assert(sizeof(WarpSmem<false>) % 16 == 0 && sizeof(WarpSmem<true>) % 16 == 0, "16-byte accesses");

// the binned histogram of a node by one warp: kPass references per lane and
// pass, their loads issued together
template <int kPass>
__device__ __forceinline__ void warp_hist(const LevelArgs &A, uint32_t *Hw, float *Pw, uint4 info, float4 blo,
                                          float4 bhi) {
    const uint32_t lane = threadIdx.x & 31u, cnt = info.y;
    __syncwarp();   // the previous node's readers are done
    {
        // 288 counters = 72 16-byte stores
        uint4 *H4 = reinterpret_cast<uint4 *>(Hw);
        H4[lane] = make_uint4(0, 0, 0, 0);
        H4[lane + 32] = make_uint4(0, 0, 0, 0);
        if (lane < kHist / 4 - 64) H4[lane + 64] = make_uint4(0, 0, 0, 0);
    }
    node_planes_warp(Pw, blo, bhi);
    __syncwarp();
    const float4 inv3 = bin_scale(blo, bhi);
    for (uint32_t base = 0; base < cnt; base += 32 * kPass) {
        uint32_t tri[kPass];
        float4 tlo[kPass], thi[kPass];
#pragma unroll
        for (int k = 0; k < kPass; k++) {
            const uint32_t r = base + 32u * k + lane;
            tri[k] = r < cnt ? A.refs()[info.x + r] : 0xffffffffu;
        }
#pragma unroll
        for (int k = 0; k < kPass; k++)
            if (tri[k] != 0xffffffffu) load_bounds(A, tri[k], tlo[k], thi[k]);
#pragma unroll
        for (int k = 0; k < kPass; k++) {
            if (base + 32u * k >= cnt) break;   // uniform across the warp
            if (tri[k] != 0xffffffffu) hist_ref_tab(Hw, tlo[k], thi[k], blo, bhi, inv3, Pw);
        }
    }
    __syncwarp();
}

// shared memory of a CTA's large-node work
struct HistSmem {
    uint32_t H[kHist];
    float P[kPlanes];
    int last;
};

// k_hist's work for one level (every CTA of the grid calls it): the chunks of
// the large nodes and, with MEDIUM, the medium nodes (exact SAH, XS)
enum : int { kHistChunks = 0, kHistExact = 1, kHistRows = 2 };
// what a CTA's large-node work starts from, loaded before the kernel's first
// barrier (the record of its first chunk is read whether the level has it or not)
struct HistStart {
    uint4 ck;
    uint32_t nch, nmed, nodes;
};
template <bool MEDIUM>
__device__ __forceinline__ HistStart hist_start(const LevelArgs &A) {
    return HistStart{__ldcg(A.chunks + min(blockIdx.x, A.cap_chunks - 1)), min(__ldcg(&A.lc->n_chunks), A.cap_chunks),
                     MEDIUM ? min(__ldcg(&A.lc->n_medium), A.cap_medium) : 0u, __ldcg(&A.lc->nodes)};
}

template <bool MEDIUM, uint32_t NT>
__device__ __forceinline__ void hist_body(const LevelArgs &A, const HistStart &hs, HistSmem &SH, ExactSmem<256> *XSp,
                                          Tally &tally) {
    uint32_t *H = SH.H;
    int &s_last = SH.last;
    const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t nch = hs.nch, nmed = hs.nmed, nodes = hs.nodes;
    for (uint32_t item = blockIdx.x; item < nch + nmed; item += gridDim.x) {
        if (MEDIUM && item >= nch) {
            // a medium node: the exact SAH in this CTA
            const uint32_t s = A.medium_slot[item - nch];
            if (s >= nodes) continue;
            const uint4 info = A.n_info()[s];
            const float4 blo = A.n_lo()[s], bhi = A.n_hi()[s];
            const Decision d = sah_exact_group<256>(A, info, blo, bhi, *XSp);
            if (threadIdx.x == 0) {
                write_decision(A, s, d);
                tally.add(d, info.y);
            }
            if (A.record && d.axis >= 0 && info.y <= kLearnMax) {
                // a training row: the node's binned histogram as features, the
                // bin of the exact plane as label (every thread holds d)
                for (uint32_t i = threadIdx.x; i < kHist; i += blockDim.x) H[i] = 0;
                __syncthreads();
                const float4 inv3 = bin_scale(blo, bhi);
                for (uint32_t r = info.x + threadIdx.x; r < info.x + info.y; r += blockDim.x) {
                    const uint32_t tri = A.refs()[r];
                    float4 tlo, thi;
                    load_bounds(A, tri, tlo, thi);
                    hist_ref(H, tlo, thi, blo, bhi, inv3);
                }
                __syncthreads();
                if (wib == 0) {
                    uint32_t row = 0;
                    if (lane == 0) row = atomicAdd(A.rec_rows, 1u);
                    row = __shfl_sync(0xffffffffu, row, 0);
                    if (row < A.rec_cap) {
                        hist_features(H, info.y, blo, bhi, A.level, A.max_depth, A.rec_X + (size_t)row * 200);
                        if (lane == 0) A.rec_y[row] = exact_label(d.axis, d.plane, blo, bhi);
                    }
                }
                __syncthreads();
            }
            continue;
        }
        const uint4 ck = item == blockIdx.x ? hs.ck : A.chunks[item];
        const uint32_t rank = ck.x, s = ck.y, r0 = ck.z, r1 = ck.w;
        if (rank >= A.cap_large || s >= nodes) continue;   // uniform per CTA
        const uint4 info = A.n_info()[s];
        const float4 blo = A.n_lo()[s], bhi = A.n_hi()[s];
        for (uint32_t i = threadIdx.x; i < kHist; i += blockDim.x) H[i] = 0;
        node_planes_cta(SH.P, blo, bhi);
        __syncthreads();
        const float4 inv3 = bin_scale(blo, bhi);
        for (uint32_t q0 = r0; q0 < r1; q0 += 4 * NT) {
            // four references a thread, their bounds loaded together
            constexpr int kPer = 4;
            uint32_t tri[kPer];
            float4 tlo[kPer], thi[kPer];
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const uint32_t r = q0 + threadIdx.x + NT * k;
                tri[k] = r < r1 ? A.refs()[r] : 0xffffffffu;
            }
#pragma unroll
            for (int k = 0; k < kPer; k++)
                if (tri[k] != 0xffffffffu) load_bounds(A, tri[k], tlo[k], thi[k]);
#pragma unroll
            for (int k = 0; k < kPer; k++)
                if (tri[k] != 0xffffffffu) hist_ref_tab(H, tlo[k], thi[k], blo, bhi, inv3, SH.P);
        }
        __syncthreads();
        if (info.y <= kChunk) {
            // the node's only chunk: its histogram is complete in shared memory
            if (wib == 0) finish_large(A, s, info, blo, bhi, H, tally);
            __syncthreads();
            continue;
        }
        uint32_t *G = A.hist + (size_t)rank * kHist;
        for (uint32_t i = threadIdx.x; i < kHist; i += blockDim.x)
            if (H[i]) atomicAdd(&G[i], H[i]);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t nchunks = node_chunks(info.y, chunk_refs(A, A.lc->refs));
            s_last = (atomicAdd(&A.done[rank], 1u) == nchunks - 1) ? 1 : 0;
        }
        __syncthreads();
        if (s_last && wib == 0) {
            __threadfence();
            finish_large(A, s, info, blo, bhi, GHist{G}, tally);
            // clean the histogram and the done counter for the next level
            __syncwarp();
            for (uint32_t i = lane; i < kHist; i += 32) G[i] = 0;
            if (lane == 0) A.done[rank] = 0;
        }
        __syncthreads();
    }
}

// k_hist: the chunks alone, with the exact search of the medium nodes, or (learned
// mode) with the proposer rows of up to 256 references, a warp each, the CTAs
// without chunks first
template <int MODE>
__global__ void __launch_bounds__(256, MODE == kHistRows ? 4 : 3) k_hist(LevelArgs A) {
    union Smem {
        HistSmem hist;
        std::conditional_t<MODE == kHistRows, WarpSmem<false>, uint32_t> rows[8];
    };
    __shared__ __align__(16) Smem SH;
    __shared__ std::conditional_t<MODE == kHistExact, ExactSmem<256>, uint32_t> XS;
    __shared__ uint32_t s_tally[kTallies];
    const HistStart hs = hist_start<MODE != kHistChunks>(A);
    if (level_aborted(A)) return;
    Tally tally;
    if constexpr (MODE == kHistExact) hist_body<true, 256>(A, hs, SH.hist, &XS, tally);
    else hist_body<false, 256>(A, HistStart{hs.ck, hs.nch, 0u, hs.nodes}, SH.hist, nullptr, tally);
    if constexpr (MODE == kHistRows) {
        __syncthreads();
        const uint32_t wib = threadIdx.x >> 5;
        for (uint32_t k = (gridDim.x - 1 - blockIdx.x) * 8 + wib; k < hs.nmed; k += gridDim.x * 8) {
            const uint32_t s = A.medium_slot[k];
            if (s >= hs.nodes) continue;
            const uint4 info = A.n_info()[s];
            const float4 blo = A.n_lo()[s], bhi = A.n_hi()[s];
            uint32_t *Hw = SH.rows[wib].scratch;
            warp_hist<4>(A, Hw, reinterpret_cast<float *>(Hw + kHist), info, blo, bhi);
            finish_large(A, s, info, blo, bhi, Hw, tally);
        }
    }
    tally_flush(A, tally, s_tally);
}

// Small nodes (not splittable, or splittable and neither medium nor large):
// one warp per node; the exact SAH in registers for nodes of at most 32
// references when exact_max >= 32 or in learned mode (the WARP_EXACT
// instantiations), else counts per plane up to 32 references and a
// warp-private histogram + the binned SAH above.
template <bool WARP_EXACT, bool LEARNED>
__device__ __forceinline__ void small_body(const LevelArgs &A, WarpSmem<WARP_EXACT && !LEARNED> *WSp, Tally &tally,
                                           uint32_t cta) {
    const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t nodes = A.lc->nodes, refs = A.lc->refs;
    const uint32_t nw = blockDim.x >> 5, ngroups = (nodes + nw - 1) / nw;
    for (uint32_t g = cta; g < ngroups; g += gridDim.x) {
        const uint32_t s = g * nw + wib;
        if (s >= nodes) continue;
        const uint4 info = A.n_info()[s];
        const float4 blo = A.n_lo()[s], bhi = A.n_hi()[s];   // (with the record: one round trip)
        const uint32_t cnt = info.y;
        const bool dec = decidable(A, cnt);
        if (dec && (is_large(A, cnt, refs) || is_medium(A, cnt))) continue;   // k_hist
        if (!dec || is_deferred(A, cnt)) {
            // a leaf, or the root of a subtree built after the levels
            if (lane == 0) {
                const Decision leaf{dec ? kDeferAxis : -1, 0.0f, 0, 0, kInf, 0};
                write_decision(A, s, leaf);
                tally.add(leaf, cnt);
            }
            continue;
        }
        Decision d;
        if (LEARNED || cnt <= kWarpExact) {
            // (learned mode: larger nodes are k_hist's)
            d = sah_warp32<WARP_EXACT>(A, reinterpret_cast<float *>(WSp[wib].scratch), info, blo, bhi);
        } else if (WARP_EXACT && !LEARNED && is_exact(A, cnt)) {
            if constexpr (WARP_EXACT && !LEARNED) d = sah_exact_group<32>(A, info, blo, bhi, WSp[wib].exact);
        } else {
            // (one reference per lane and pass in the exact instantiation, which
            // has few nodes here and no registers to spare)
            uint32_t *Hw = WSp[wib].scratch;
            warp_hist<WARP_EXACT ? 1 : 4>(A, Hw, reinterpret_cast<float *>(Hw + kHist), info, blo, bhi);
            d = sah_warp(Hw, blo, bhi, cnt, A.ct, A.ci);
        }
        if (lane == 0) {
            write_decision(A, s, d, blo, bhi);
            tally.add(d, cnt);
        }
        __syncwarp();
    }
}

template <bool WARP_EXACT, bool LEARNED>
__global__ void __launch_bounds__(256, LEARNED ? 5 : 4) k_small(LevelArgs A) {
    __shared__ __align__(16) WarpSmem<WARP_EXACT && !LEARNED> WS[8];
    __shared__ uint32_t s_tally[kTallies];
    wait_prior_grid();
    if (level_aborted(A)) return;
    Tally tally;
    small_body<WARP_EXACT, LEARNED>(A, WS, tally, blockIdx.x);
    tally_flush(A, tally, s_tally);
}

// Binned mode (no medium nodes, no proposer): a level's large-node chunks and
// small nodes in one launch on the build's stream, PDL-chained to the plan
// (no second stream, no fork and join per level)
// (1,024 threads per SM: a CTA's other warps wait while one costs a large
// node's planes, so the many nodes of large scenes go to CTAs of 128 threads,
// the few of small ones to CTAs of 256. A frame of 1M triangles 2,714 us with
// 128, 2,778 with 256, 2,746 with 64; 200k 1,638, 1,640 and 1,661; 24k 935 with
// 128 and 928 with 256)
template <uint32_t NT>
union DecideSmem {
    HistSmem hist;
    WarpSmem<false> small[NT / 32];
};

template <uint32_t NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_decide(LevelArgs A) {
    __shared__ __align__(16) DecideSmem<NT> sm;
    __shared__ uint32_t s_tally[kTallies];
    wait_prior_grid();
    const HistStart hs = hist_start<false>(A);
    if (level_aborted(A)) return;
    Tally tally;
    hist_body<false, NT>(A, hs, sm.hist, nullptr, tally);
    __syncthreads();
    // the last CTAs take the first node groups: the first ones have the chunks
    small_body<false, false>(A, sm.small, tally, gridDim.x - 1 - blockIdx.x);
    tally_flush(A, tally, s_tally);
}

constexpr int kLearnMaxK = 8;
// list capacity per (proposal, list): the largest power of two whose 3 k-fold
// is at most 2,048 (128 for k = 4). A bin with a longer list is not costed, so
// the rule is part of the result (the oracle has the same)
constexpr uint32_t kLearnScratch = 2048;
__host__ __device__ constexpr uint32_t learn_list_cap(uint32_t K) {
    uint32_t c = 1;
    while (2 * c * 3 * K <= kLearnScratch) c *= 2;
    return c;
}
// ---------------------------------------------------------------------------
// learned split search (no reference counterpart), two launches per level.
// k_learn: the network on the level's proposer rows (tcgen05: 128-row tiles,
// hk_mlp_tc.cuh; else mma.sync: 64-row tiles, hk_mlp_tile.cuh), then per row
// the top-k valid bins by logit (ties to the lower index; an axis of zero
// extent has no valid bin), one byte each (axis * 32 + bin, 0xff: none) in
// learn_prop.
// ---------------------------------------------------------------------------
template <bool TC>
__global__ void __launch_bounds__(256, 1) k_learn(LevelArgs A) {
    extern __shared__ __align__(1024) unsigned char learn_smem[];
    constexpr uint32_t kRows = TC ? (uint32_t)kTcRows : (uint32_t)kTileRows;
    wait_prior_grid();
    if (level_aborted(A)) return;
    const uint32_t rows = min(A.lc->n_learn, A.cap_learn);
    if (blockIdx.x * kRows >= rows) return;   // no tile: no TMEM taken (the CTA takes part in no barrier)
    const TileSmem S = tile_smem(learn_smem);
    const TcSmem T = tc_smem(learn_smem);
    uint32_t tmem = 0, g = 0;
    if (TC) tmem = tc_setup(T);
    const uint32_t K = A.topk < (uint32_t)kLearnMaxK ? (A.topk ? A.topk : 1u) : (uint32_t)kLearnMaxK;
    const float *logits = TC ? T.logits : S.logits;
    for (uint32_t row0 = blockIdx.x * kRows; row0 < rows; row0 += gridDim.x * kRows) {
        if constexpr (TC) {
            if (!tc_tile_forward(A.mlp, A.feat, row0, rows, T, tmem, g, A.err)) break;
        } else {
            tile_forward(A.mlp, A.feat, row0, rows, S);
        }
        // one thread per row (rr = threadIdx.x): a row's candidates are the
        // bins of its node's axes of nonzero extent, a NaN logit counting as
        // -inf, taken as the logits' bits in an order-preserving unsigned form
        // (-inf maps to 0x007fffff; an empty slot holds 0, below every
        // candidate). The candidates pass in index order through a sorted
        // list of NS slots, a candidate moving ahead of a slot only when its
        // key is strictly greater: the k best by (logit, then the lower index).
        constexpr uint32_t kStride = TC ? kTcLogitStride : (uint32_t)kMlpOut;
        const uint32_t rr = threadIdx.x;
        if (rr < kRows && row0 + rr < rows) {
            const uint32_t row = row0 + rr;
            const uint32_t slot = A.learn_slot[row];
            const float4 blo = A.n_lo()[slot], bhi = A.n_hi()[slot];
            const float *Lg = logits + rr * kStride;
            uint32_t tk[kLearnMaxK], tix[kLearnMaxK];
#pragma unroll
            for (int i = 0; i < kLearnMaxK; i++) tk[i] = 0u, tix[i] = 0xffu;
            auto select = [&](auto ns_tag) {
                constexpr int NS = decltype(ns_tag)::value;
#pragma unroll
                for (uint32_t j = 0; j < 3; j++) {
                    if (!(__fsub_rn(c3(bhi, j), c3(blo, j)) > 0.0f)) continue;
#pragma unroll 4
                    for (uint32_t k = 0; k < 32; k++) {
                        float x = Lg[32u * j + k];
                        if (x != x) x = -INFINITY;
                        if (x == 0.0f) x = 0.0f;   // -0 ties with +0, as the values compare
                        const uint32_t u = __float_as_uint(x);
                        uint32_t key = (u & 0x80000000u) ? ~u : (u | 0x80000000u), c = 32u * j + k;
#pragma unroll
                        for (int i = 0; i < NS; i++) {
                            const bool sw = key > tk[i];
                            const uint32_t k2 = sw ? tk[i] : key, c2 = sw ? tix[i] : c;
                            tk[i] = sw ? key : tk[i];
                            tix[i] = sw ? c : tix[i];
                            key = k2;
                            c = c2;
                        }
                    }
                }
            };
            if (K <= 4) select(std::integral_constant<int, 4>{});
            else select(std::integral_constant<int, kLearnMaxK>{});
            uint32_t packed[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
            for (uint32_t r = 0; r < (uint32_t)kLearnMaxK; r++)
                if (r < K && tk[r] != 0u) {
                    const uint32_t sh = 8u * (r & 3u);
                    packed[r >> 2] = (packed[r >> 2] & ~(0xffu << sh)) | (tix[r] << sh);
                }
            A.learn_prop[row] = make_uint2(packed[0], packed[1]);
            if (A.prop_log) {
                const uint32_t cidx = A.n_info()[slot].z;
                if (cidx < A.cap_nodes)
#pragma unroll
                    for (uint32_t r = 0; r < 8; r++) {
                        const uint32_t bb = (packed[r >> 2] >> (8u * (r & 3u))) & 0xffu;
                        A.prop_log[(size_t)cidx * 8 + r] = bb == 0xffu ? -1 : (int32_t)bb;
                    }
            }
        }
        __syncthreads();   // the logits are rewritten by the next tile
    }
    if (TC) tc_teardown(tmem);
}

// ---------------------------------------------------------------------------
// k_refine_warp, k_refine_cta: the exact search of a proposer row's proposed
// bins by a group of NT threads -- a warp for rows of up to kRefineWarpMax
// references, a CTA for larger ones, each kernel grid-striding over the level's
// rows and leaving the other's.
//   1. per proposed bin (axis a, bin b, the closed interval [P0, P1] =
//      [p_b, p_{b+1}] with p_0 the node's minimum and p_32 its maximum) the
//      references whose clipped lower bound lies below P0 and those whose
//      clipped upper bound lies above P1 are counted, and the lower and upper
//      bounds inside are listed in shared memory (in any order; a bound flat
//      on its axis one step outside its value and flagged, lane_bounds);
//   2. every listed bound p strictly inside the node is a candidate -- the
//      exact SAH's candidates that fall in the bin -- with
//        below = #(lo < P0) + #(listed lo < p),
//        above = #(hi > P1) + #(listed hi > p),
//      the exact SAH's own counts; the threads share the candidates, each
//      counts its bin's two lists, and the cheapest by (cost, axis, plane) wins
//      (equal keys are the same plane with the same counts). The lists hold a
//      32nd of the node's bounds: sorting them and searching the sorted lists
//      took 650 + 524 us of a 200k-triangle learned build;
//   3. that plane is taken unless it costs more than fallback_ratio x the
//      binned optimum found for the node (then the binned plane); the usual
//      leaf test follows.
// A bin whose lists overflow their capacity (learn_list_cap) is not costed.
// ---------------------------------------------------------------------------
constexpr uint32_t kRefineWarpMax = 128;   // rows up to this many references: one warp each
constexpr uint32_t kRefineLists = 1280;    // most floats in the lists: 2 K learn_list_cap(K), K = 5
static_assert(2 * 1 * learn_list_cap(1) <= kRefineLists && 2 * 2 * learn_list_cap(2) <= kRefineLists &&
                  2 * 3 * learn_list_cap(3) <= kRefineLists && 2 * 4 * learn_list_cap(4) <= kRefineLists &&
                  2 * 5 * learn_list_cap(5) <= kRefineLists && 2 * 6 * learn_list_cap(6) <= kRefineLists &&
                  2 * 7 * learn_list_cap(7) <= kRefineLists && 2 * 8 * learn_list_cap(8) <= kRefineLists,
              "the lists of every K fit");

template <uint32_t NT>
struct RefineSmem {
    uint32_t n[2 * kLearnMaxK];                 // listed lower, upper bounds per proposal
    uint32_t bl[kLearnMaxK], ab[kLearnMaxK];    // references below P0, above P1
    uint32_t flat[kRefineLists / 32];
    float lists[kRefineLists];
    uint32_t w_cost[NT / 32], w_ax[NT / 32], w_nb[NT / 32], w_na[NT / 32];
    float w_pk[NT / 32];
};

// the group's row: its decision, and whether the proposal was taken
template <uint32_t NT>
__device__ __forceinline__ Decision refine_group(const LevelArgs &A, uint32_t row, const LearnBin &lb, uint32_t s,
                                                 uint4 info, float4 blo, float4 bhi, RefineSmem<NT> &S, bool &take) {
    const uint32_t lane = threadIdx.x & 31u, tid = NT == 32 ? lane : threadIdx.x;
    const uint32_t cnt = info.y;
    const uint32_t K = A.topk < (uint32_t)kLearnMaxK ? (A.topk ? A.topk : 1u) : (uint32_t)kLearnMaxK;
    const uint32_t cap = learn_list_cap(K);
    const uint2 pp = A.learn_prop[row];
    const float4 ext = make_float4(__fsub_rn(bhi.x, blo.x), __fsub_rn(bhi.y, blo.y), __fsub_rn(bhi.z, blo.z), 0.0f);
    const float Anode = surf(blo, bhi);
    // (axis << 5) | bin of proposal i, or 0xff: none (no later one either)
    auto proposal = [&](uint32_t i) { return i < K ? ((i < 4 ? pp.x : pp.y) >> (8u * (i & 3u))) & 0xffu : 0xffu; };
    group_sync<NT>();   // the previous row's readers are done
    if (tid < 2 * kLearnMaxK) S.n[tid] = 0;
    if (tid < kLearnMaxK) S.bl[tid] = S.ab[tid] = 0;
    for (uint32_t i = tid; i < kRefineLists / 32; i += NT) S.flat[i] = 0;
    // the thread's references, all loads issued together
    float4 tlo[4], thi[4];
    uint32_t tri[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t r = tid + NT * k;
        tri[k] = r < cnt ? A.refs()[info.x + r] : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (tri[k] != 0xffffffffu) load_bounds(A, tri[k], tlo[k], thi[k]);
    group_sync<NT>();
    // 1. counts and lists
    for (uint32_t i = 0; i < (uint32_t)kLearnMaxK; i++) {
        const uint32_t b8 = proposal(i);
        if (b8 == 0xffu) break;
        const uint32_t a = b8 >> 5, b = b8 & 31u;
        const float l = c3(blo, a), h = c3(bhi, a);
        const float p0 = b == 0 ? l : plane_k(l, c3(ext, a), b);
        const float p1 = b == kBins - 1 ? h : plane_k(l, c3(ext, a), b + 1);
        float *Ls = S.lists + 2 * i * cap, *Hs = Ls + cap;
        uint32_t bl = 0, ab = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (tri[k] == 0xffffffffu) continue;
            const float lo = mxf(c3(tlo[k], a), l), hi = mnf(c3(thi[k], a), h);
            bl += lo < p0 ? 1u : 0u;
            ab += hi > p1 ? 1u : 0u;
            const bool fl = lo == hi;
            if (p0 <= lo && lo <= p1) {
                const uint32_t pos = atomicAdd(&S.n[2 * i], 1u);
                if (pos < cap) {
                    Ls[pos] = fl ? nextafterf(lo, -kInf) : lo;
                    if (fl) atomicOr(&S.flat[(2 * i * cap + pos) >> 5], 1u << ((2 * i * cap + pos) & 31u));
                }
            }
            if (p0 <= hi && hi <= p1) {
                const uint32_t pos = atomicAdd(&S.n[2 * i + 1], 1u);
                if (pos < cap) {
                    Hs[pos] = fl ? nextafterf(hi, kInf) : hi;
                    if (fl) atomicOr(&S.flat[((2 * i + 1) * cap + pos) >> 5], 1u << (((2 * i + 1) * cap + pos) & 31u));
                }
            }
        }
        bl = __reduce_add_sync(0xffffffffu, bl);
        ab = __reduce_add_sync(0xffffffffu, ab);
        if (lane == 0) {
            if (bl) atomicAdd(&S.bl[i], bl);
            if (ab) atomicAdd(&S.ab[i], ab);
        }
    }
    group_sync<NT>();
    // 2. the candidates of every proposal that did not overflow, numbered
    // proposal by proposal
    float mc = kInf, m_pk = 0.0f;
    uint32_t m_ax = 3, m_nb = 0, m_na = 0;
    for (uint32_t q = tid;; q += NT) {
        uint32_t i = 0, t = q, nl = 0, nh = 0, b8 = 0xffu;
        for (; i < (uint32_t)kLearnMaxK; i++) {
            b8 = proposal(i);
            if (b8 == 0xffu) break;
            nl = S.n[2 * i];
            nh = S.n[2 * i + 1];
            if (nl > cap || nh > cap) continue;   // not costed
            if (t < nl + nh) break;
            t -= nl + nh;
        }
        if (i == (uint32_t)kLearnMaxK || b8 == 0xffu) break;
        const uint32_t a = b8 >> 5;
        const float l = c3(blo, a), h = c3(bhi, a);
        const float *Ls = S.lists + 2 * i * cap, *Hs = Ls + cap;
        const bool side = t >= nl;
        const uint32_t at = 2 * i * cap + (side ? cap + t - nl : t);
        float x = S.lists[at];
        if ((S.flat[at >> 5] >> (at & 31u)) & 1u) x = nextafterf(x, side ? -kInf : kInf);
        if (!(x > l && x < h)) continue;
        const float pk = __fadd_rn(x, 0.0f);
        uint32_t nb = S.bl[i], na = S.ab[i];
        for (uint32_t k = 0; k < nl; k++) nb += Ls[k] < pk ? 1u : 0u;
        for (uint32_t k = 0; k < nh; k++) na += Hs[k] > pk ? 1u : 0u;
        const float cost = plane_cost(a, pk, l, h, ext, Anode, (float)nb, (float)na, A.ct, A.ci);
        if (refine_better(cost, a, pk, mc, m_ax, m_pk)) {
            mc = cost;
            m_ax = a;
            m_pk = pk;
            m_nb = nb;
            m_na = na;
        }
    }
    __syncwarp();
    group_argmin<NT>(S, mc, m_ax, m_pk, m_nb, m_na);
    // 3. the proposal's plane, or the binned optimum
    take = mc < kInf && mc <= __fmul_rn(A.fallback_ratio, lb.cost);
    if (!take) return Decision{lb.axis, lb.plane, lb.nb, lb.na, lb.cost, 0};
    Decision d{(int)m_ax, m_pk, m_nb, m_na, mc, 0};
    if (!(mc < __fmul_rn(A.ci, (float)cnt))) d.axis = -1;
    return d;
}

template <uint32_t NT>
__device__ __forceinline__ void refine_rows(const LevelArgs &A, RefineSmem<NT> *SM) {
    __shared__ uint32_t s_tally[kTallies];
    __shared__ uint32_t s_stat[2];
    if (level_aborted(A)) return;
    Tally tally;
    uint32_t n_learned = 0, n_fallback = 0;
    constexpr uint32_t kGroups = 256 / NT;
    const uint32_t g = threadIdx.x / NT;
    const uint32_t rows = min(A.lc->n_learn, A.cap_learn);
    for (uint32_t row = blockIdx.x * kGroups + g; row < rows; row += gridDim.x * kGroups) {
        const LearnBin lb = A.learn_bin[row];
        if ((lb.pad[0] <= kRefineWarpMax) != (NT == 32)) continue;   // the other kernel's row (uniform over the group)
        const uint32_t s = A.learn_slot[row];
        const uint4 info = A.n_info()[s];
        const float4 blo = A.n_lo()[s], bhi = A.n_hi()[s];
        bool take;
        const Decision d = refine_group<NT>(A, row, lb, s, info, blo, bhi, SM[g], take);
        if (threadIdx.x % NT == 0) {
            write_decision(A, s, d, blo, bhi);
            tally.add(d, info.y);
            if (take) n_learned++;
            else n_fallback++;
        }
    }
    __syncthreads();
    if (threadIdx.x < 2) s_stat[threadIdx.x] = 0;
    __syncthreads();
    if (n_learned) atomicAdd(&s_stat[0], n_learned);
    if (n_fallback) atomicAdd(&s_stat[1], n_fallback);
    __syncthreads();
    if (threadIdx.x == 0 && s_stat[0]) atomicAdd(&A.ctr->learned_nodes, s_stat[0]);
    if (threadIdx.x == 1 && s_stat[1]) atomicAdd(&A.ctr->fallback_nodes, s_stat[1]);
    tally_flush(A, tally, s_tally);
}

__global__ void __launch_bounds__(256, 3) k_refine_cta(LevelArgs A) {
    __shared__ RefineSmem<256> S;
    wait_prior_grid();
    refine_rows<256>(A, &S);
}

__global__ void __launch_bounds__(256, 3) k_refine_warp(LevelArgs A) {
    __shared__ RefineSmem<32> S[8];
    wait_prior_grid();
    refine_rows<32>(A, S);
}

// ---------------------------------------------------------------------------
// plan: single-pass scan over the level's nodes of (leaf refs, splits,
// next-level nodes, child refs, below child refs); the guard is decided from
// the decision tallies, block 0 writes the next level's counters, and every
// node emits its compact entry, its children's cells / ropes / next-level
// records and the next level's large-node chunks.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t level_tag(const LevelArgs &A) {
    return (*A.epoch * 64u + A.level) & 0x3fffffffu;
}

// the capacity guard: true when splitting this level would overflow
__device__ __forceinline__ bool level_over(const LevelArgs &A) {
    const LevelCounters *l = A.lc;
    const uint64_t child_refs = l->t_childrefs, splits = l->t_splits;
    // deferred-subtree references count as leaf references (a root that
    // cannot be expanded stays a leaf)
    const uint64_t leaf_refs = (uint64_t)l->t_leafrefs + l->t_deferrefs;
    return child_refs > A.cap_refs ||
           (uint64_t)l->leafrefs_total + l->defer_refs_total + leaf_refs + child_refs > A.cap_refs ||
           (uint64_t)l->nodes_total + 2 * splits > A.cap_nodes || l->t_next > A.cap_level;
}

// a child of count c (from reference start) in next-level slot ns: large nodes take a rank and
// their chunks (few per level, so plain atomics)
__device__ void child_setup(const LevelArgs &A, uint32_t ns, uint32_t start, uint32_t c) {
    const bool dec = c > A.leaf_size && A.level + 1 < A.max_depth;
    if (dec && is_medium(A, c)) {
        const uint32_t m = atomicAdd(&A.nlc->n_medium, 1u);
        if (m < A.cap_medium) A.medium_slot[m] = ns;
        else atomicOr(A.err, 2u);
        return;
    }
    const uint32_t refs = A.lc->t_childrefs;
    if (!(dec && is_large(A, c, refs))) return;
    const uint32_t per = c <= kChunk ? kChunk : chunk_refs(A, refs), nch = node_chunks(c, per);
    const uint32_t rank = atomicAdd(&A.nlc->n_large, 1u);
    const uint32_t first = atomicAdd(&A.nlc->n_chunks, nch);
    if (rank >= A.cap_large || first + nch > A.cap_chunks) {
        atomicOr(A.err, 2u);
        return;
    }
    for (uint32_t k = 0; k < nch; k++)
        A.chunks[first + k] = make_uint4(rank, ns, start + k * per, start + min(c, (k + 1) * per));
}

struct PlanCtx {
    uint32_t stop, nodes_total, leafrefs_total, defer_refs_total, defer_nodes_total;
};

struct PlanItem {
    uint4 info;     // start, count, compact index
    uint2 cnt;      // below, above
    int axis;
};

struct PlanOp {
    using T = U7;
    using Item = PlanItem;
    using Ctx = PlanCtx;
    static constexpr int kItems = kPlanItems;
    LevelArgs A;
    __device__ uint32_t count() const { return A.lc->nodes; }
    __device__ uint32_t tag() const { return level_tag(A); }
    __device__ uint32_t *err() const { return A.err; }
    __device__ Ctx ctx() const {
        const LevelCounters *l = A.lc;
        return Ctx{level_over(A) ? 1u : 0u, l->nodes_total, l->leafrefs_total, l->defer_refs_total,
                   l->defer_nodes_total};
    }
    // the next level's counters (one thread of the launch)
    __device__ void next_level(const Ctx &cx) const {
        LevelCounters *l = A.lc, *nx = A.nlc;
        const bool over = cx.stop != 0;
        l->stop = over ? 1u : 0u;
        if (over) A.ctr->capacity_hit = 1;
        nx->nodes = over ? 0u : l->t_next;
        nx->refs = over ? 0u : l->t_childrefs;
        nx->nodes_total = cx.nodes_total + (over ? 0u : 2u * l->t_splits);
        nx->leafrefs_total = cx.leafrefs_total + (over ? l->refs : l->t_leafrefs);
        nx->defer_refs_total = cx.defer_refs_total + (over ? 0u : l->t_deferrefs);
        nx->defer_nodes_total = cx.defer_nodes_total + (over ? 0u : l->t_defernodes);
        A.ctr->leaves += over ? l->nodes : l->t_leafnodes;
        if (!over && l->t_next) A.ctr->depth = A.level + 1;
    }
    __device__ Item load(uint32_t s, const Ctx &) const {
        if (s == 0xffffffffu) return Item{make_uint4(0, 0, 0, 0), make_uint2(0, 0), -1};
        return Item{A.n_info()[s], A.cnt[s], A.axis[s]};
    }
    __device__ T value(const Item &it) const {
        if (it.axis == kDeferAxis) return U7{0, 0, 0, 0, 0, it.info.y, 1};
        if (it.axis < 0) return U7{it.info.y, 0, 0, 0, 0, 0, 0};
        const uint2 c = it.cnt;
        return U7{0, 1, (c.x > 0 ? 1u : 0u) + (c.y > 0 ? 1u : 0u), c.x + c.y, c.x, 0, 0};
    }
    // where the node's references go (what the reference tiles wait for)
    __device__ void apply_first(uint32_t s, U7 pl, const Item &it, const Ctx &cx) const {
        const uint4 info = it.info;
        if (info.z >= A.cap_nodes) return;   // apply flags it
        if (!cx.stop && it.axis == kDeferAxis) {
            // reference r of this deferred root goes to defer_refs[off - start + r]
            const uint32_t off = cx.defer_refs_total + pl.d;
            A.scat[s] = make_uint4(off - info.x, 0, 0, 2u);
        } else if (cx.stop || it.axis < 0) {
            // reference r of this leaf goes to out_refs[off - start + r]
            const uint32_t off = cx.leafrefs_total + (cx.stop ? info.x : pl.x);
            A.scat[s] = make_uint4(off - info.x, 0, 0, 0);
        } else {
            // the node's below references go to nx_refs[pl.w ..), its above ones
            // right after them, each in its order within the node (its rank among
            // the node's flagged references), as next-level slots pl.z and pl.z +
            // (cnt.x > 0); w = above count << 2 | has-below << 1 | split
            const uint2 c2 = it.cnt;
            A.scat[s] = make_uint4(pl.w, pl.w + c2.x, pl.z, (c2.y << 2) | 1u | (c2.x ? 2u : 0u));
        }
    }
    // the node's compact entry, its children's cells / ropes / records
    __device__ void apply(uint32_t s, U7 pl, const Item &it, const Ctx &cx) const {
        const uint4 info = it.info;
        const int ax = cx.stop ? -1 : it.axis;
        if (info.z >= A.cap_nodes) {
            atomicOr(A.err, 16u);
            return;
        }
        if (ax == kDeferAxis) {
            // the subtree pass writes the node's entry; its cell and ropes are
            // already written (by its parent's plan)
            const uint32_t did = cx.defer_nodes_total + pl.e;
            if (did < A.cap_defer) {
                A.d_root[did] = make_uint4(info.z, cx.defer_refs_total + pl.d, info.y, A.level);
                A.d_lo[did] = A.n_lo()[s];
                A.d_hi[did] = A.n_hi()[s];
            } else {
                atomicOr(A.err, 2u);
            }
            return;
        }
        if (ax < 0) {
            const uint32_t off = cx.leafrefs_total + (cx.stop ? info.x : pl.x);
            A.out_nodes[info.z] = make_uint2((off << 2) | kLeafTag, info.y);
            return;
        }
        const uint32_t pair = cx.nodes_total + 2 * pl.y;
        const uint2 ct = it.cnt;
        // the tallies that passed the guard and this scan sum the same
        // decisions; these checks only keep an inconsistent level in bounds
        if ((uint64_t)pair + 1 >= A.cap_nodes ||
            (uint64_t)pl.z + (ct.x ? 1u : 0u) + (ct.y ? 1u : 0u) > A.cap_level) {
            atomicOr(A.err, 16u);
            return;
        }
        const float p = A.plane[s];
        const float4 lo = A.n_lo()[s], hi = A.n_hi()[s];
        uint32_t r[6];
        {
            // the parent's ropes: 6 words at a 24-byte stride (8-byte aligned)
            const uint2 *pr2 = reinterpret_cast<const uint2 *>(A.out_ropes + 6 * (size_t)info.z);
            const uint2 a0 = pr2[0], a1 = pr2[1], a2 = pr2[2];
            r[0] = a0.x; r[1] = a0.y; r[2] = a1.x; r[3] = a1.y; r[4] = a2.x; r[5] = a2.y;
        }
        A.out_nodes[info.z] = make_uint2((pair << 2) | (uint32_t)ax, __float_as_uint(p));
        uint32_t ns = pl.z;
        const uint32_t co = pl.w;
        {
            // cells and ropes of both children: the parent's ropes, with the
            // face on the split plane pointing at the sibling
            float4 bh = hi, al = lo;
            s3(bh, ax, p);
            s3(al, ax, p);
            A.out_cbox[2 * (size_t)pair] = lo;
            A.out_cbox[2 * (size_t)pair + 1] = bh;
            A.out_cbox[2 * (size_t)pair + 2] = al;
            A.out_cbox[2 * (size_t)pair + 3] = hi;
            uint32_t rb[6], ra[6];
#pragma unroll
            for (int f = 0; f < 6; f++) {
                rb[f] = f == 2 * ax + 1 ? pair + 1 : r[f];
                ra[f] = f == 2 * ax ? pair : r[f];
            }
            // the pair's 12 rope words start at 24 * pair bytes, pair even
            // (nodes_total starts at 2 and grows by pairs): 16-byte aligned
            uint4 *dst = reinterpret_cast<uint4 *>(A.out_ropes + 6 * (size_t)pair);
            dst[0] = make_uint4(rb[0], rb[1], rb[2], rb[3]);
            dst[1] = make_uint4(rb[4], rb[5], ra[0], ra[1]);
            dst[2] = make_uint4(ra[2], ra[3], ra[4], ra[5]);
        }
        if (ct.x) {
            float4 h2 = hi;
            s3(h2, ax, p);
            A.nx_lo()[ns] = lo;
            A.nx_hi()[ns] = h2;
            A.nx_info()[ns] = make_uint4(co, ct.x, pair, 0);
            child_setup(A, ns, co, ct.x);
            ns++;
        } else {
            A.out_nodes[pair] = make_uint2(kLeafTag, 0);
        }
        if (ct.y) {
            float4 l2 = lo;
            s3(l2, ax, p);
            A.nx_lo()[ns] = l2;
            A.nx_hi()[ns] = hi;
            A.nx_info()[ns] = make_uint4(co + ct.x, ct.y, pair + 1, 0);
            child_setup(A, ns, co + ct.x, ct.y);
        } else {
            A.out_nodes[pair + 1] = make_uint2(kLeafTag, 0);
        }
    }
};

// refs: single-pass scan of the below / above flags, segmented by node, fused
// with the stable partition: a reference's rank among its node's below (above)
// references, added to where the plan scan put the node's children, is its
// place in the next level.
struct RefItem {
    uint2 f;        // below / above flags
    uint32_t s;     // node slot
    uint32_t tri;
};

struct RefOp {
    using Item = RefItem;
    using Ctx = uint32_t;   // the level stopped splitting
    static constexpr int kItems = 4;
    LevelArgs A;
    // kItems references, one of each run of 32 from `base`, those before n:
    // every index load together, then every gather
    __device__ void load(uint32_t base, uint32_t n, const Ctx &stop, Item (&it)[kItems]) const {
        uint32_t node[kItems], tri[kItems];
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const bool in = base + 32u * k < n;
            node[k] = in ? A.ref_node()[base + 32u * k] : 0u;
            tri[k] = in ? A.refs()[base + 32u * k] : 0u;
        }
        float4 sp[kItems];
#pragma unroll
        for (int k = 0; k < kItems; k++)
            sp[k] = base + 32u * k < n ? A.split[node[k]] : make_float4(__int_as_float(-1), 0, 0, 0);
#pragma unroll
        for (int k = 0; k < kItems; k++) {
            const int ax = stop ? -1 : __float_as_int(sp[k].x);
            it[k] = Item{make_uint2(0, 0), node[k], tri[k]};
            if (ax < 0) continue;
            const float p = sp[k].y, l = sp[k].z, h = sp[k].w;
            const float2 b = load_bounds_axis(A, tri[k], (uint32_t)ax);
            const float lo = mxf(b.x, l), hi = mnf(b.y, h);
            const bool flat_on = (lo == hi) && lo == p;
            it[k].f = make_uint2((lo < p || flat_on) ? 1u : 0u, (hi > p || flat_on) ? 1u : 0u);
        }
    }
    // R: the reference's rank among its node's below / above references
    // sc: the node's destinations
    __device__ void apply(uint32_t r, uint2 R, const Item &it, const uint4 &sc) const {
        if (!(sc.w & 1u)) {
            const uint32_t off = sc.x + r;   // leaf, or a deferred root (w = 2)
            if (off < A.cap_refs) (sc.w & 2u ? A.defer_refs : A.out_refs)[off] = it.tri;
            else atomicOr(A.err, 2u);
            return;
        }
        if (it.f.x) {
            const uint32_t pos = sc.x + R.x;
            if (pos < A.cap_refs && R.x < sc.y - sc.x) {
                A.nx_refs()[pos] = it.tri;
                A.nx_ref_node()[pos] = sc.z;
            } else {
                atomicOr(A.err, 8u);
            }
        }
        if (it.f.y) {
            const uint32_t pos = sc.y + R.y;
            if (pos < A.cap_refs && R.y < (sc.w >> 2)) {
                A.nx_refs()[pos] = it.tri;
                A.nx_ref_node()[pos] = sc.z + ((sc.w & 2u) ? 1u : 0u);
            } else {
                atomicOr(A.err, 8u);
            }
        }
    }
};

// segmented scan values: the flag counts since the last node start, and
// whether a node starts in the span
struct SegV {
    uint2 v;
    uint32_t h;
};
__device__ __forceinline__ SegV seg_join(SegV a, SegV b) {   // a before b
    return SegV{b.h ? b.v : vadd(a.v, b.v), a.h | b.h};
}

struct RefTileSmem {
    SegV w_tot[kScanThreads / 32];
    uint2 carry;                          // the tile's first segment: flags in earlier tiles
    uint32_t first_node, last_node;       // nodes of the tile's references
    uint32_t wait_ok;
};

// One reference tile (kTile references; a warp's 128 are consecutive, a run of
// 32 per item, so ranks are ballots and population counts and a warp's stores
// of an item are runs too: four consecutive references per thread with shuffle
// scans took 1,707 us a 200k-triangle frame against 1,688). What bounds it is
// the chain of dependent loads and waits. The scan is segmented by node: a tile in which a node starts publishes its last
// segment's counts as complete (status 2) at once; only its first segment,
// when it continues a node of earlier tiles, needs the look-back, which ends at
// the tile where that node starts. One warp looks back while another waits
// (wait_plan(first, last node)) for the plan tiles of the tile's nodes; the
// scatter follows both.
template <class Wait>
__device__ void ref_tile(const RefOp &R, uint32_t rt, uint32_t nr, uint32_t tag, uint32_t stop, ulonglong2 *recs,
                         RefTileSmem &sh, const Wait &wait_plan) {
    const LevelArgs &A = R.A;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t r0 = rt * kTile;
    const uint32_t w0 = r0 + wid * (32u * kScanItems), base = w0 + lane;
    // node of the reference before the warp's first one
    uint32_t prev = (lane == 0 && w0 > 0 && w0 <= nr) ? A.ref_node()[w0 - 1] : 0xffffffffu;
    RefItem it[kScanItems];
    R.load(base, nr, stop, it);
    if (threadIdx.x == 0) sh.first_node = it[0].s;
    // rank of each item since the last node start in the warp (seen: there is one)
    uint2 rank[kScanItems];
    uint32_t seen = 0, starts = 0;
    SegV run{make_uint2(0, 0), 0u};
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        const uint32_t r = base + 32u * k;
        if (r == min(nr, r0 + kTile) - 1) sh.last_node = it[k].s;
        const uint32_t up = __shfl_up_sync(0xffffffffu, it[k].s, 1);
        if (lane) prev = up;
        const bool hd = r >= nr || it[k].s != prev;
        if (k == 0) starts = hd ? 1u : 0u;
        prev = __shfl_sync(0xffffffffu, it[k].s, 31);   // for lane 0 of the next item
        const uint32_t H = __ballot_sync(0xffffffffu, hd), B = __ballot_sync(0xffffffffu, it[k].f.x != 0);
        const uint32_t Ab = __ballot_sync(0xffffffffu, it[k].f.y != 0);
        const uint32_t below = (1u << lane) - 1u, hle = H & (below | (1u << lane));
        // the lanes before this one, from the last start on
        const uint32_t span = hle ? below & (0xffffffffu << (31 - __clz(hle))) : below;
        rank[k] = make_uint2(__popc(B & span), __popc(Ab & span));
        if (!hle) rank[k] = vadd(rank[k], run.v);
        if (hle || run.h) seen |= 1u << k;
        const uint32_t tail = H ? 0xffffffffu << (31 - __clz(H)) : 0xffffffffu;
        run = seg_join(run, SegV{make_uint2(__popc(B & tail), __popc(Ab & tail)), H ? 1u : 0u});
    }
    if (lane == 0) sh.w_tot[wid] = run;
    __syncthreads();
    SegV wp{make_uint2(0, 0), 0u}, tot{make_uint2(0, 0), 0u};
    for (uint32_t w = 0; w < kScanThreads / 32; w++) {
        if (w < wid) wp = seg_join(wp, sh.w_tot[w]);
        tot = seg_join(tot, sh.w_tot[w]);
    }
    if (threadIdx.x == 0) ref_publish(recs + rt, (tag << 2) | (tot.h ? 2u : 1u), tot.v);
    if (wid == 0) {
        // when the tile's first reference starts a node no earlier tile matters
        const uint2 c = __shfl_sync(0xffffffffu, starts, 0)
                            ? make_uint2(0, 0)
                            : ref_lookback(recs, rt, tag, A.err, A.spin_limit);
        if (threadIdx.x == 0) {
            if (!tot.h) ref_publish(recs + rt, (tag << 2) | 2u, vadd(c, tot.v));
            sh.carry = c;
        }
    } else if (wid == 1) {
        const bool ok = wait_plan(sh.first_node, sh.last_node);
        if (lane == 0) sh.wait_ok = ok ? 1u : 0u;
    }
    __syncthreads();
    if (!sh.wait_ok) return;   // uniform: the scatter needs the plan's destinations
    if (!wp.h) wp.v = vadd(wp.v, sh.carry);
    uint4 sc[kScanItems];   // written by plan tiles of this launch
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        sc[k] = base + 32u * k < nr ? __ldcg(A.scat + it[k].s) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + 32u * k < nr)
            R.apply(base + 32u * k, (seen >> k) & 1u ? rank[k] : vadd(rank[k], wp.v), it[k], sc[k]);
    __syncthreads();
}

// ---------------------------------------------------------------------------
// plan + refs of one level in one launch. Tickets 0 .. node tiles - 1 are plan
// tiles (kPlanTile nodes), the rest reference tiles (kTile refs). A plan tile
// publishes a done flag once its nodes' reference destinations are written,
// then emits the rest; a reference tile computes its flags, scans and looks
// back, then waits (bounded) for the plan tiles of its nodes (its references
// belong to a contiguous run of nodes) before it scatters. Plan tiles take
// their tickets before any reference tile and wait for nothing but earlier
// plan tiles, so every wait ends.
// ---------------------------------------------------------------------------
struct PlanSmem {
    U7 shp[kScanThreads / 32 + 1];
    U7 sxp;
    RefTileSmem shr_seg;
    uint32_t tile;
};

__device__ __forceinline__ void plan_refs_body(const LevelArgs &A, PlanSmem &SM, uint32_t *pflags, U7 *paggs,
                                               U7 *pincls, ulonglong2 *rrecs, uint32_t *pdone, uint32_t *ticket) {
    const PlanOp P{A};
    const RefOp R{A};
    // (the level's counters, read while the error word is)
    const uint32_t tag = level_tag(A);
    const PlanCtx pc = P.ctx();
    const uint32_t stop = pc.stop;              // the guard, decided from the tallies by every CTA
    const uint32_t nn = A.lc->nodes, nr = A.lc->refs;
    if (level_aborted(A)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) P.next_level(pc);
    const uint32_t ntn = (nn + kPlanTile - 1) / kPlanTile;
    const uint32_t ntr = (nr + kTile - 1) / kTile;
    // with a CTA per tile every CTA takes one ticket and the others none
    const bool single = ntn + ntr <= gridDim.x;
    if (single && blockIdx.x >= ntn + ntr) return;
    if (threadIdx.x == 0) SM.tile = atomicAdd(ticket, 1u);
    for (;;) {
        __syncthreads();
        const uint32_t t = SM.tile;
        if (t < ntn) {
            // the done flag follows the tile's reference destinations; the
            // rest of its emission overlaps the reference tiles' scatter
            scan_tile(P, t, nn, tag, pc, pflags, paggs, pincls, SM.shp, SM.sxp, [&] {
                __threadfence();
                __syncthreads();
                if (threadIdx.x == 0 && !(t == 0 && A.level == A.withhold_level))
                    *reinterpret_cast<volatile uint32_t *>(pdone + t) = tag;
            });
        } else if (t < ntn + ntr) {
            // true when every plan tile of the tile's nodes has published its
            // reference destinations (one warp, lane k at the k-th such plan
            // tile: a tile's references span at most kTile nodes); a wait that
            // runs out leaves the tile's scatter undone (error bit 4, the
            // build reports failure)
            static_assert(kTile / kPlanTile + 2 <= 32, "one lane per plan tile of a reference tile");
            auto wait_plan = [&](uint32_t first, uint32_t last) -> bool {
                const uint32_t k = first / kPlanTile + (threadIdx.x & 31u);
                const bool mine = k <= last / kPlanTile && k < ntn;
                for (uint32_t spins = 0;; spins++) {
                    const bool ready = !mine || __ldcv(pdone + k) == tag;
                    if (__ballot_sync(0xffffffffu, !ready) == 0) break;
                    if (spins >= A.spin_limit) {
                        if (!ready) atomicOr(A.err, 4u);
                        return false;
                    }
                    __nanosleep(32);
                }
                __threadfence();
                return true;
            };
            ref_tile(R, t - ntn, nr, tag, stop, rrecs, SM.shr_seg, wait_plan);
        } else {
            break;
        }
        if (single) break;
        if (threadIdx.x == 0) SM.tile = atomicAdd(ticket, 1u);
    }
}

// Four CTAs per SM, one resident wave: 64 registers keep the four references
// of a thread in flight without spills, and fewer CTAs take fewer tickets (six
// per SM: a 200k-triangle frame 1,631 us, a 1M one 2,764; five 1,610 and 2,701;
// four 1,602 and 2,678; three 1,645 and 2,762).
constexpr int kPlanGrid = 4;
__global__ void __launch_bounds__(kScanThreads, kPlanGrid) k_plan_refs(LevelArgs A, uint32_t *pflags, U7 *paggs, U7 *pincls,
                                                               ulonglong2 *rrecs, uint32_t *pdone, uint32_t *ticket) {
    __shared__ PlanSmem SM;
    wait_prior_grid();
    plan_refs_body(A, SM, pflags, paggs, pincls, rrecs, pdone, ticket);
}

// ---------------------------------------------------------------------------
// deferred subtrees. After the levels, one warp builds each subtree rooted at
// a recorded node of at most kDeferMax references, depth first, with one
// reference per lane (a node's references are a mask of the warp's lanes, in
// the root's order), deciding every node with the levels' SAH of at most 32
// references (sah_lanes_binned, or sah_lanes_exact). Nodes are numbered locally:
// a split takes the next pair of local indices (below, above); the below
// child is built next and the above child waits on a stack in shared memory.
// Nodes go to 64-byte scratch records (cell, ropes, entry, subtree and local
// index) and references to slots keyed (subtree, local index), handed out per
// warp in chunks. A single-pass scan over the subtrees' sizes places subtree
// i after the levels' nodes and leaf references and after subtrees 0 .. i-1,
// and the last pass moves every slot to its place. When the subtrees do not
// fit the node or reference capacity (or a scratch arena ran out), every root
// stays a leaf holding its references instead. The oracle's
// hko_build_binned restates this order.
// ---------------------------------------------------------------------------
constexpr uint32_t kLocalRope = 0x80000000u;   // a rope to a local index of the same subtree
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint32_t kScNodeChunk = 64;          // node slots per chunk (pairs never straddle)
constexpr uint32_t kScRefChunk = 256;          // reference slots per chunk
constexpr int kSubWarps = 8;

// entries of a warp's stack of waiting (above) children: one per depth below
// the root, an even count (the per-warp shared-memory regions stay 16-byte
// aligned)
__host__ __device__ constexpr uint32_t sub_stack_entries(uint32_t max_depth) { return (max_depth + 3u) & ~1u; }
// the words of a scratch record; on the stack of waiting children the record
// holds the child's lane mask, depth and scratch slot instead of the words
// after the slashes
enum SubWord : uint32_t {
    kWLo = 0,        // cell minimum, 3 words
    kWSub = 3,       // subtree / lane mask
    kWHi = 4,        // cell maximum, 3 words
    kWIndex = 7,     // local index / depth
    kWRope = 8,      // 6 words
    kWEntry = 14,    // the node's entry, 2 words / scratch slot
    kWords = 16
};

// per warp: the packed bounds (the exact search's candidates too), then the
// stack
__host__ __device__ constexpr size_t sub_warp_smem(uint32_t entries, bool exact) {
    return (exact ? kLaneScratch : kLaneScratch / 2) * 4 + (size_t)kWords * 4 * entries;
}

// a scratch entry moved to its place: child pairs and leaf starts shifted by
// the subtree's first node / reference; an empty cell keeps start 0
__device__ __forceinline__ uint2 sub_relocate(uint2 e, uint32_t nb, uint32_t rb) {
    if ((e.x & 3u) == kLeafTag) return e.y ? make_uint2((((e.x >> 2) + rb) << 2) | kLeafTag, e.y) : e;
    return make_uint2((((e.x >> 2) + nb) << 2) | (e.x & 3u), e.y);
}

// the rest of a warp's scratch chunk marked unused
__device__ __forceinline__ void sub_close_chunks(const LevelArgs &A, uint32_t nbase, uint32_t nused, uint32_t rbase,
                                                 uint32_t rused) {
    const uint32_t lane = threadIdx.x & 31u;
    if (nbase != kNoSlot)
        for (uint32_t k = nused + lane; k < kScNodeChunk; k += 32)
            A.sc_rec[(size_t)(nbase + k) * kWords + kWSub] = kNoSlot;
    if (rbase != kNoSlot)
        for (uint32_t k = rused + lane; k < kScRefChunk; k += 32) A.sc_ref[rbase + k] = make_uint4(kNoSlot, 0, 0, 0);
}

// a new chunk of `chunk` slots from the counter (all lanes; kNoSlot when the
// arena is spent)
__device__ __forceinline__ uint32_t sub_chunk(uint32_t *ctr, uint32_t chunk, uint32_t cap) {
    uint32_t b = 0;
    if ((threadIdx.x & 31u) == 0) b = atomicAdd(ctr, chunk);
    b = __shfl_sync(0xffffffffu, b, 0);
    return (uint64_t)b + chunk <= cap ? b : kNoSlot;
}

// true (CTA-uniform) when the build has any error bit: the subtree pass reads
// records and references that a capacity error may have left unwritten
__device__ __forceinline__ bool sub_aborted(const LevelArgs &A) {
    __shared__ uint32_t s_err;
    __syncthreads();
    if (threadIdx.x == 0) s_err = __ldcg(A.err);
    __syncthreads();
    return s_err != 0;
}

// The subtrees of roots A.lc->defer_nodes_total .. A.nlc->defer_nodes_total,
// one warp per subtree taken by ticket from A.lc (E stack entries per warp).
// Lane r holds reference r of the root. The current node's record is spread
// over the lanes too, word lane % 16 in each half of the warp: a split changes
// two words of each child's record (its cell's cut side, its rope across the
// plane), so the pair's records are one 128-byte store, the lower half's the
// below child, and the above child's stack entry one shared-memory store.
// Issue-bound (87% of issue slots): 576 warp instructions per SAH evaluation,
// 615,571 of them on the 200k-triangle frame, 398 us (806 and 599 us with a
// histogram per node and separate entry, cell and rope stores).
template <bool WARP_EXACT>
__global__ void __launch_bounds__(kSubWarps * 32, 4) k_subtree(LevelArgs A, uint32_t E) {
    extern __shared__ __align__(16) unsigned char sub_smem[];
    wait_prior_grid();
    if (sub_aborted(A)) return;
    const uint32_t wib = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    unsigned char *wbase = sub_smem + (size_t)wib * sub_warp_smem(E, WARP_EXACT);
    float *Sw = reinterpret_cast<float *>(wbase);
    uint32_t *stack = reinterpret_cast<uint32_t *>(wbase + sub_warp_smem(0, WARP_EXACT));
    const uint32_t r0 = min(A.lc->defer_nodes_total, A.cap_defer);
    const uint32_t r1 = min(A.nlc->defer_nodes_total, A.cap_defer);
    const uint32_t word = lane & 15u, child = lane >> 4;
    uint32_t nbase = kNoSlot, nused = kScNodeChunk, rbase = kNoSlot, rused = kScRefChunk;
    uint32_t leaves = 0, maxdepth = 0;
    bool dead = false;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = r0 + atomicAdd(&A.lc->sub_ticket, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        if (i >= r1 || dead) break;
        const uint4 rt = A.d_root[i];   // compact index, reference offset, count, depth
        float4 lo = A.d_lo[i], hi = A.d_hi[i];
        const uint32_t cnt0 = min(rt.z, 32u);
        if ((uint64_t)rt.y + cnt0 > A.cap_refs || rt.x >= A.cap_nodes) {
            dead = true;   // an inconsistent record: the roots stay leaves
            break;
        }
        uint32_t tri = 0;
        float4 tlo = make_float4(0, 0, 0, 0), thi = tlo;
        if (lane < cnt0) {
            tri = A.defer_refs[rt.y + lane];
            load_bounds(A, tri, tlo, thi);
        }
        float4 nlo = tlo, nhi = thi;
        lane_bounds(nlo, nhi);
        // the root's record words (cell and ropes)
        uint32_t rec = 0;
        if (word >= kWRope && word < kWRope + 6) rec = A.out_ropes[6 * (size_t)rt.x + word - kWRope];
        if (word < 3) rec = __float_as_uint(c3(lo, word));
        if (word >= kWHi && word < kWHi + 3) rec = __float_as_uint(c3(hi, word - kWHi));
        uint32_t mask = cnt0 >= 32 ? 0xffffffffu : ((1u << cnt0) - 1u);
        uint32_t depth = rt.w, slot = kNoSlot, sp = 0, npair = 0, nref = 0;
        uint2 root_entry = make_uint2(kLeafTag, 0);
        // a node's entry, written by the lanes that wrote its record
        auto put_entry = [&](uint2 entry) {
            if (slot == kNoSlot) root_entry = entry;
            else if ((lane | 1u) == ((slot & 1u) ? 31u : 15u))
                A.sc_rec[(size_t)slot * kWords + word] = (lane & 1u) ? entry.y : entry.x;
        };
        for (;;) {
            const bool in = (mask >> lane) & 1u;
            const uint32_t c = __popc(mask);
            Decision d{-1, 0.0f, 0, 0, kInf, 0};
            if (c > A.leaf_size && depth < A.max_depth) {
                lanes_pack<WARP_EXACT>(Sw, in, __popc(mask & ((1u << lane) - 1u)), c, tlo, thi, nlo, nhi);
                d = WARP_EXACT ? sah_lanes_exact<false>(Sw, c, lo, hi, A.ct, A.ci)
                               : sah_lanes_binned<false>(Sw, c, lo, hi, A.ct, A.ci);
            }
            if (d.axis < 0) {
                // a leaf: its references in the subtree's next local slots
                put_entry(make_uint2((nref << 2) | kLeafTag, c));
                if (rused + c > kScRefChunk) {
                    sub_close_chunks(A, kNoSlot, 0, rbase, rused);
                    rbase = sub_chunk(&A.ctr->sc_ref_ctr, kScRefChunk, A.cap_sc_refs);
                    rused = 0;
                    if (rbase == kNoSlot) {
                        dead = true;
                        break;
                    }
                }
                if (in) {
                    const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
                    A.sc_ref[rbase + rused + rank] = make_uint4(i, nref + rank, tri, 0);
                }
                rused += c;
                nref += c;
                leaves++;
            } else {
                const uint32_t ax = (uint32_t)d.axis;
                const float p = d.plane;
                const uint32_t pair = npair;
                npair += 2;
                put_entry(make_uint2((pair << 2) | ax, __float_as_uint(p)));
                // the partition of the levels (checkPolygonToAAPlane on the
                // clipped bounds, see lane_bounds), as lane masks
                const uint32_t bm = __ballot_sync(0xffffffffu, in && c3(nlo, ax) < p);
                const uint32_t am = __ballot_sync(0xffffffffu, in && c3(nhi, ax) > p);
                if (nused + 2 > kScNodeChunk) {
                    sub_close_chunks(A, nbase, nused, kNoSlot, 0);
                    nbase = sub_chunk(&A.ctr->sc_node_ctr, kScNodeChunk, A.cap_sc_nodes);
                    nused = 0;
                    if (nbase == kNoSlot) {
                        dead = true;
                        break;
                    }
                }
                const uint32_t sb = nbase + nused;   // even: chunks and pairs are
                nused += 2;
                // the children's records: the parent's, cut on the split's
                // side, with the rope across the plane at the sibling (the
                // entry of a child is that of an empty cell until it is decided)
                const uint32_t cut = __float_as_uint(p);
                const uint32_t recB =
                    word == kWHi + ax ? cut : (word == kWRope + 1 + 2 * ax ? kLocalRope | (pair + 1) : rec);
                const uint32_t recA = word == kWLo + ax ? cut : (word == kWRope + 2 * ax ? kLocalRope | pair : rec);
                const uint32_t mine = child ? recA : recB;
                uint32_t w = mine;
                if (word == kWSub) w = i;
                if (word == kWIndex) w = pair + child;
                if (word >= kWEntry) w = word == kWEntry ? kLeafTag : 0u;
                A.sc_rec[(size_t)sb * kWords + lane] = w;
                if (bm | am) maxdepth = max(maxdepth, depth + 1);
                if (am) {
                    if (sp >= E) {
                        dead = true;
                        break;
                    }
                    w = mine;
                    if (word == kWSub) w = am;
                    if (word == kWIndex) w = depth + 1;
                    if (word == kWEntry) w = sb + 1;
                    if (child) stack[sp * kWords + word] = w;
                    sp++;
                }
                if (bm) {
                    mask = bm;
                    s3(hi, ax, p);
                    depth++;
                    slot = sb;
                    rec = recB;
                    continue;
                }
            }
            if (sp == 0) break;
            __syncwarp();
            sp--;
            const uint32_t *e = stack + sp * kWords;
            const uint4 e0 = *reinterpret_cast<const uint4 *>(e), e1 = *reinterpret_cast<const uint4 *>(e + kWHi);
            slot = e[kWEntry];
            rec = e[word];
            __syncwarp();
            lo = make_float4(__uint_as_float(e0.x), __uint_as_float(e0.y), __uint_as_float(e0.z), 0.0f);
            hi = make_float4(__uint_as_float(e1.x), __uint_as_float(e1.y), __uint_as_float(e1.z), 0.0f);
            mask = e0.w;
            depth = e1.w;
        }
        if (!dead && lane == 0) {
            A.st_cnt[i] = make_uint2(npair, nref);
            A.st_root[i] = root_entry;
        }
    }
    if (dead) {
        if (lane == 0) atomicExch(&A.ctr->sub_overflow, 1u);
    } else {
        sub_close_chunks(A, nbase, nused, rbase, rused);
    }
    if (lane == 0 && leaves) {
        atomicAdd(&A.ctr->sub_leaves, leaves);
        atomicMax(&A.ctr->sub_depth, maxdepth);
    }
}

// subtree sizes -> places (exclusive prefix over the subtrees); the thread of
// the last subtree decides whether they fit and writes the build's totals
struct SubScanOp {
    using T = uint2;
    using Item = uint2;
    using Ctx = uint32_t;
    static constexpr int kItems = kScanItems;
    LevelArgs A;
    uint32_t n;
    __device__ uint32_t *err() const { return A.err; }
    __device__ Item load(uint32_t i, const Ctx &) const { return i == 0xffffffffu ? make_uint2(0, 0) : A.st_cnt[i]; }
    __device__ T value(const Item &it) const { return it; }
    __device__ void apply_first(uint32_t i, uint2 pre, const Item &, const Ctx &) const { A.st_base[i] = pre; }
    __device__ void apply(uint32_t i, uint2 pre, const Item &it, const Ctx &) const {
        if (i + 1 != n) return;
        LevelCounters *fin = A.lc;
        BuildCounters *c = A.ctr;
        const uint2 tot = vadd(pre, it);
        const uint32_t N0 = fin->nodes_total, R0 = fin->leafrefs_total;
        const bool fits = !c->sub_overflow && (uint64_t)N0 + tot.x <= A.cap_nodes &&
                          (uint64_t)R0 + tot.y <= A.cap_refs;
        c->sub_n0 = N0;
        c->sub_r0 = R0;
        c->sub_fits = fits ? 1u : 0u;
        if (fits) {
            fin->nodes_total = N0 + tot.x;
            fin->leafrefs_total = R0 + tot.y;
            c->sub_nodes = tot.x;
            c->sub_refs = tot.y;
            c->leaves += c->sub_leaves;
            c->depth = max(c->depth, c->sub_depth);
        } else {
            // every root a leaf over its references (they were counted as
            // leaf references by the levels' guard, so they fit)
            fin->leafrefs_total = R0 + fin->defer_refs_total;
            c->leaves += n;
            c->capacity_hit = 1;
        }
    }
};

__global__ void __launch_bounds__(kScanThreads) k_sub_scan(LevelArgs A, uint32_t *flags, uint2 *aggs,
                                                           uint2 *incls) {
    __shared__ uint2 sh[kScanThreads / 32 + 1];
    __shared__ uint2 sx;
    __shared__ uint32_t s_tile;
    wait_prior_grid();
    if (sub_aborted(A)) return;
    const uint32_t n = min(A.lc->defer_nodes_total, A.cap_defer);
    const uint32_t ntiles = (n + kTile - 1) / kTile;
    const SubScanOp op{A, n};
    const uint32_t tag = level_tag(A);
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&A.ctr->sub_ticket, 1u);
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= ntiles) break;
        scan_tile(op, t, n, tag, 0u, flags, aggs, incls, sh, sx, [] {});
    }
}

// every scratch slot to its place (or, when the subtrees do not fit, every
// root a leaf)
__global__ void __launch_bounds__(256) k_sub_place(LevelArgs A) {
    wait_prior_grid();
    if (sub_aborted(A)) return;
    const uint32_t n = min(A.lc->defer_nodes_total, A.cap_defer);
    if (n == 0) return;
    const BuildCounters *c = A.ctr;
    const uint32_t N0 = c->sub_n0, R0 = c->sub_r0;
    const uint32_t stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (!c->sub_fits) {
        for (uint32_t i = t0; i < n; i += stride) {
            const uint4 rt = A.d_root[i];
            A.out_nodes[rt.x] = make_uint2(((R0 + rt.y) << 2) | kLeafTag, rt.z);
        }
        const uint32_t nr = min(A.lc->defer_refs_total, A.cap_refs);
        for (uint32_t k = t0; k < nr; k += stride) {
            if ((uint64_t)R0 + k < A.cap_refs) A.out_refs[R0 + k] = A.defer_refs[k];
            else atomicOr(A.err, 2u);
        }
        return;
    }
    const uint32_t nsn = min(c->sc_node_ctr, A.cap_sc_nodes), nsr = min(c->sc_ref_ctr, A.cap_sc_refs);
    for (uint32_t j = t0; j < nsn; j += stride) {
        const uint4 *rec = reinterpret_cast<const uint4 *>(A.sc_rec + (size_t)j * kWords);
        const uint4 w0 = rec[0], w1 = rec[1], w2 = rec[2], w3 = rec[3];
        if (w0.w >= n) continue;  // an unused slot
        const uint2 base = A.st_base[w0.w];
        const uint32_t nb = N0 + base.x, g = nb + w1.w;
        if (g >= A.cap_nodes) {
            atomicOr(A.err, 16u);
            continue;
        }
        A.out_nodes[g] = sub_relocate(make_uint2(w3.z, w3.w), nb, R0 + base.y);
        A.out_cbox[2 * (size_t)g] =
            make_float4(__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z), 0.0f);
        A.out_cbox[2 * (size_t)g + 1] =
            make_float4(__uint_as_float(w1.x), __uint_as_float(w1.y), __uint_as_float(w1.z), 0.0f);
        auto rope = [&](uint32_t r) { return r != kNoSlot && (r & kLocalRope) ? nb + (r & ~kLocalRope) : r; };
        uint2 *dst = reinterpret_cast<uint2 *>(A.out_ropes + 6 * (size_t)g);   // 24 bytes a node: 8-byte aligned
        dst[0] = make_uint2(rope(w2.x), rope(w2.y));
        dst[1] = make_uint2(rope(w2.z), rope(w2.w));
        dst[2] = make_uint2(rope(w3.x), rope(w3.y));
    }
    for (uint32_t j = t0; j < nsr; j += stride) {
        const uint4 q = A.sc_ref[j];
        if (q.x >= n) continue;
        const uint32_t pos = R0 + A.st_base[q.x].y + q.y;
        if (pos < A.cap_refs) A.out_refs[pos] = q.z;
        else atomicOr(A.err, 16u);
    }
    for (uint32_t i = t0; i < n; i += stride) {
        const uint2 base = A.st_base[i];
        A.out_nodes[A.d_root[i].x] = sub_relocate(A.st_root[i], N0 + base.x, R0 + base.y);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// k_subtree's grid: four CTAs of kSubWarps warps per SM, one wave
static unsigned sub_grid(int sm_count) { return (unsigned)sm_count * 4u; }

// CTAs of a level kernel: at most per_sm per SM (one resident wave), and no
// more waves of one per SM than `ctas` fill. Every kernel here takes any grid;
// CTAs without work still cost their launch and exit (a scene of 3.5k
// triangles: 592 CTAs per k_decide 504 us a frame, 296 486), and too few cost
// more (24k triangles: 592 CTAs 910 us, 296 917).
static unsigned level_grid(int sm_count, unsigned per_sm, uint64_t ctas) {
    const uint64_t waves = (ctas + sm_count - 1) / sm_count;
    return (unsigned)sm_count * (unsigned)std::min<uint64_t>(std::max<uint64_t>(waves, 1), per_sm);
}

// a launch that may start while the stream's previous kernel finishes
// (programmatic stream serialization); the kernel calls wait_prior_grid()
// before it reads anything that kernel wrote
template <class... KArgs, class... Args>
static cudaError_t launch_pdl(void (*k)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                              Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

template <class T>
static cudaError_t dalloc(T *&p, size_t n) {
    if (p) cudaFree(p);
    p = nullptr;
    return cudaMalloc((void **)&p, std::max<size_t>(n, 1) * sizeof(T));
}

void build_release(BuildState &S) {
    auto f = [](auto *&p) {
        if (p) cudaFree((void *)p);
        p = nullptr;
    };
    f(S.tb);
    for (int k = 0; k < 2; k++) {
        f(S.n_lo[k]); f(S.n_hi[k]); f(S.n_info[k]); f(S.refs[k]); f(S.ref_node[k]);
    }
    f(S.d_axis); f(S.d_plane); f(S.d_cnt); f(S.d_split); f(S.d_scat);
    f(S.chunks); f(S.hist); f(S.done); f(S.medium_slot); f(S.learn_slot); f(S.learn_bin); f(S.learn_prop); f(S.feat); f(S.prop_log);
    f(S.plan_flags); f(S.ref_recs); f(S.plan_done); f(S.plan_agg); f(S.plan_incl); f(S.epoch);
    f(S.ctr); f(S.err);
    f(S.out_nodes); f(S.out_refs); f(S.out_ropes); f(S.out_cbox);
    f(S.d_root); f(S.d_lo); f(S.d_hi); f(S.defer_refs);
    f(S.sc_rec); f(S.sc_ref);
    f(S.st_cnt); f(S.st_root); f(S.st_base); f(S.sub_flags); f(S.sub_agg); f(S.sub_incl);
    S.cap_defer = S.cap_sc_nodes = S.cap_sc_refs = S.sub_tiles = 0;
    if (S.ev_fork) cudaEventDestroy(S.ev_fork);
    if (S.ev_join) cudaEventDestroy(S.ev_join);
    if (S.ev_learn) cudaEventDestroy(S.ev_learn);
    if (S.ev_join2) cudaEventDestroy(S.ev_join2);
    if (S.aux) cudaStreamDestroy(S.aux);
    if (S.aux2) cudaStreamDestroy(S.aux2);
    S.ev_fork = S.ev_join = S.ev_learn = S.ev_join2 = nullptr;
    S.aux = S.aux2 = nullptr;
    S.nt = S.cap_refs = S.cap_nodes = S.cap_level = 0;
    S.plan_tiles = S.ref_tiles = 0;
    S.active = false;
}

hk_status build_prepare(BuildState &S, const BuildParams &p, uint32_t nt, int sm_count) {
    // leaf starts and child-pair indices are stored shifted left by 2 bits
    const uint64_t kMaxIndex = (1ull << 30) - 64;
    if ((uint64_t)nt > kMaxIndex / 16) return HK_E_CAPACITY;
    uint32_t cap_refs = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(p.max_refs, nt), kMaxIndex);
    uint32_t cap_nodes = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(12ull * nt, 1024ull), kMaxIndex);
    S.p = p;
    S.sm_count = sm_count;
    if (S.ctr && S.nt == nt && S.cap_refs == cap_refs && S.cap_nodes == cap_nodes && p.max_depth <= S.alloc_depth) {
        if (p.prop_log && !S.prop_log && dalloc(S.prop_log, (size_t)S.cap_nodes * 8) != cudaSuccess) return HK_E_ALLOC;
        return HK_OK;
    }
    build_release(S);
    S.nt = nt;
    S.cap_refs = cap_refs;
    S.cap_nodes = cap_nodes;
    S.alloc_depth = p.max_depth;
    S.cap_level = std::min(cap_refs, cap_nodes) + 1;
    S.cap_large = cap_refs / (kWarpExact + 1) + 2;   // learned mode: every node above 32 references
    S.cap_chunks = cap_refs / kChunkMin + S.cap_large + 2;
    S.cap_medium = cap_refs / (kWarpExact + 1) + 2;
    S.cap_learn = cap_refs / (kWarpExact + 1) + 2;
    S.plan_tiles = S.cap_level / kPlanTile + 2;
    S.ref_tiles = cap_refs / kTile + 2;
    // a deferred root holds 2..32 references, all within the reference arena
    S.cap_defer = cap_refs / 2 + 2;
    // subtree scratch: the arenas' own capacities, plus one open chunk per
    // warp of k_subtree, plus the reference slots a chunk can leave unused at
    // its end (fewer than a 32-reference leaf, per 256)
    {
        const uint64_t warps = (uint64_t)sub_grid(sm_count) * kSubWarps;
        S.cap_sc_nodes = (uint32_t)std::min<uint64_t>((uint64_t)cap_nodes + warps * kScNodeChunk, kMaxIndex);
        S.cap_sc_refs =
            (uint32_t)std::min<uint64_t>((uint64_t)cap_refs + cap_refs / 7 + warps * kScRefChunk, kMaxIndex);
    }
    S.sub_tiles = S.cap_defer / kTile + 2;
    bool bad = false;
    bad |= dalloc(S.tb, 2 * (size_t)nt) != cudaSuccess;
    for (int k = 0; k < 2; k++) {
        bad |= dalloc(S.n_lo[k], S.cap_level) != cudaSuccess;
        bad |= dalloc(S.n_hi[k], S.cap_level) != cudaSuccess;
        bad |= dalloc(S.n_info[k], S.cap_level) != cudaSuccess;
        bad |= dalloc(S.refs[k], cap_refs) != cudaSuccess;
        bad |= dalloc(S.ref_node[k], cap_refs) != cudaSuccess;
    }
    bad |= dalloc(S.d_axis, S.cap_level) != cudaSuccess;
    bad |= dalloc(S.d_plane, S.cap_level) != cudaSuccess;
    bad |= dalloc(S.d_cnt, S.cap_level) != cudaSuccess;
    bad |= dalloc(S.d_split, S.cap_level) != cudaSuccess;
    bad |= dalloc(S.d_scat, S.cap_level) != cudaSuccess;
    bad |= dalloc(S.chunks, S.cap_chunks) != cudaSuccess;
    bad |= dalloc(S.hist, (size_t)S.cap_large * kHist) != cudaSuccess;
    bad |= dalloc(S.done, S.cap_large) != cudaSuccess;
    bad |= dalloc(S.medium_slot, S.cap_medium) != cudaSuccess;
    bad |= dalloc(S.learn_slot, S.cap_learn) != cudaSuccess;
    bad |= dalloc(S.learn_bin, S.cap_learn) != cudaSuccess;
    bad |= dalloc(S.learn_prop, S.cap_learn) != cudaSuccess;
    bad |= dalloc(S.feat, (size_t)S.cap_learn * kMlpIn) != cudaSuccess;
    if (p.prop_log) bad |= dalloc(S.prop_log, (size_t)cap_nodes * 8) != cudaSuccess;
    bad |= dalloc(S.plan_flags, S.plan_tiles) != cudaSuccess;
    bad |= dalloc(S.ref_recs, S.ref_tiles) != cudaSuccess;
    bad |= dalloc(S.plan_done, S.plan_tiles) != cudaSuccess;
    {
        U7 *pa = nullptr, *pi = nullptr;
        bad |= dalloc(pa, S.plan_tiles) != cudaSuccess;
        bad |= dalloc(pi, S.plan_tiles) != cudaSuccess;
        S.plan_agg = pa;
        S.plan_incl = pi;
    }
    bad |= dalloc(S.epoch, 1) != cudaSuccess;
    bad |= dalloc(S.ctr, 1) != cudaSuccess;
    bad |= dalloc(S.err, 1) != cudaSuccess;
    bad |= dalloc(S.out_nodes, cap_nodes) != cudaSuccess;
    bad |= dalloc(S.out_refs, cap_refs) != cudaSuccess;
    bad |= dalloc(S.out_ropes, (size_t)cap_nodes * 6) != cudaSuccess;
    bad |= dalloc(S.out_cbox, (size_t)cap_nodes * 2) != cudaSuccess;
    bad |= dalloc(S.d_root, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.d_lo, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.d_hi, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.defer_refs, cap_refs) != cudaSuccess;
    bad |= dalloc(S.sc_rec, (size_t)S.cap_sc_nodes * kWords) != cudaSuccess;
    bad |= dalloc(S.sc_ref, S.cap_sc_refs) != cudaSuccess;
    bad |= dalloc(S.st_cnt, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.st_root, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.st_base, S.cap_defer) != cudaSuccess;
    bad |= dalloc(S.sub_flags, S.sub_tiles) != cudaSuccess;
    bad |= dalloc(S.sub_agg, S.sub_tiles) != cudaSuccess;
    bad |= dalloc(S.sub_incl, S.sub_tiles) != cudaSuccess;
    bad |= cudaStreamCreateWithFlags(&S.aux, cudaStreamNonBlocking) != cudaSuccess;
    bad |= cudaEventCreateWithFlags(&S.ev_fork, cudaEventDisableTiming) != cudaSuccess;
    bad |= cudaEventCreateWithFlags(&S.ev_join, cudaEventDisableTiming) != cudaSuccess;
    bad |= cudaStreamCreateWithFlags(&S.aux2, cudaStreamNonBlocking) != cudaSuccess;
    bad |= cudaEventCreateWithFlags(&S.ev_learn, cudaEventDisableTiming) != cudaSuccess;
    bad |= cudaEventCreateWithFlags(&S.ev_join2, cudaEventDisableTiming) != cudaSuccess;
    if (bad) {
        build_release(S);
        return HK_E_ALLOC;
    }
    cudaMemset(S.err, 0, 4);
    cudaMemset(S.epoch, 0, 4);
    cudaMemset(S.hist, 0, (size_t)S.cap_large * kHist * sizeof(uint32_t));
    cudaMemset(S.done, 0, (size_t)S.cap_large * sizeof(uint32_t));
    cudaMemset(S.plan_flags, 0, (size_t)S.plan_tiles * 4);
    cudaMemset(S.ref_recs, 0, (size_t)S.ref_tiles * sizeof(ulonglong2));
    cudaMemset(S.plan_done, 0, (size_t)S.plan_tiles * 4);
    cudaMemset(S.sub_flags, 0, (size_t)S.sub_tiles * 4);

    cudaMemset(S.ctr, 0, sizeof(BuildCounters));
    // these run on the legacy stream, which does not order against the
    // context's own stream: every one is finished before a build may start
    if (cudaDeviceSynchronize() != cudaSuccess) return HK_E_ALLOC;
    return HK_OK;
}

hk_status build_ensure_outputs(BuildState &S, BuildOutputs *o) {
    if (!S.out_nodes || !S.out_refs) return HK_E_ALLOC;
    if (o) {
        o->nodes = S.out_nodes;
        o->refs = S.out_refs;
    }
    return HK_OK;
}

cudaError_t build_learn_setup() {
    static uint64_t attr_set = 0;   // the shared-memory opt-in is per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !((attr_set >> dev) & 1u)) {
        e = cudaFuncSetAttribute(k_learn<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_learn<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
        if (e != cudaSuccess) return e;
        if (dev < 64) attr_set |= 1ull << dev;
    }
    return cudaSuccess;
}

cudaError_t build_launch(BuildState &S, const float4 *verts, const uint4 *tris, uint32_t nt, const float *box,
                         cudaStream_t st) {
    const int G = S.sm_count * 4;
    LevelArgs A;
    memset(&A, 0, sizeof(A));
    A.tb = S.tb;
    A.wave = (uint32_t)G;
    A.axis = S.d_axis;
    A.plane = S.d_plane;
    A.cnt = S.d_cnt;
    A.split = S.d_split;
    A.scat = S.d_scat;
    A.chunks = S.chunks;
    A.hist = S.hist;
    A.done = S.done;
    A.out_nodes = S.out_nodes;
    A.out_refs = S.out_refs;
    A.out_ropes = S.out_ropes;
    A.out_cbox = S.out_cbox;
    A.ctr = S.ctr;
    A.err = S.err;
    A.epoch = S.epoch;
    A.ct = S.p.ct;
    A.ci = S.p.ci;
    A.max_depth = S.p.max_depth;
    A.leaf_size = S.p.leaf_size;
    A.cap_refs = S.cap_refs;
    A.cap_nodes = S.cap_nodes;
    A.cap_level = S.cap_level;
    A.cap_large = S.cap_large;
    A.cap_chunks = S.cap_chunks;
    A.cap_medium = S.cap_medium;
    A.medium_slot = S.medium_slot;
    A.learned = (S.p.mode == HK_BUILD_LEARNED) ? 1 : 0;
    // learned mode: nodes up to 32 references take the warp's exact SAH,
    // 33..1024 the proposer, larger ones the binned SAH (exact_max unused)
    A.exact_max = A.learned ? 0u : S.p.exact_max;
    A.record = (S.p.mode == HK_BUILD_BINNED && S.p.record && S.learn && S.learn->rec_X) ? 1 : 0;
    A.learn_slot = S.learn_slot;
    A.learn_bin = S.learn_bin;
    A.learn_prop = S.learn_prop;
    A.feat = S.feat;
    A.cap_learn = S.cap_learn;
    A.prop_log = (A.learned && S.p.prop_log) ? S.prop_log : nullptr;
    A.fallback_ratio = S.p.fallback_ratio;
    A.topk = S.p.topk;
    A.spin_limit = S.p.spin_limit ? S.p.spin_limit : kSpinLimit;
    A.withhold_level = (S.p.debug_flags & 1u) ? 1u : 0xffffffffu;
    A.defer = std::min<uint32_t>(S.p.defer, kDeferMax);
    A.defer_level = (S.p.defer_margin && S.p.defer_margin < S.p.max_depth) ? S.p.max_depth - S.p.defer_margin : 0u;
    A.d_root = S.d_root;
    A.d_lo = S.d_lo;
    A.d_hi = S.d_hi;
    A.defer_refs = S.defer_refs;
    A.cap_defer = S.cap_defer;
    A.sc_rec = S.sc_rec;
    A.sc_ref = S.sc_ref;
    A.cap_sc_nodes = S.cap_sc_nodes;
    A.cap_sc_refs = S.cap_sc_refs;
    A.st_cnt = S.st_cnt;
    A.st_root = S.st_root;
    A.st_base = S.st_base;
    if (S.learn) {
        A.rec_X = S.learn->rec_X;
        A.rec_y = S.learn->rec_y;
        A.rec_rows = S.learn->rec_rows;
        A.rec_cap = S.learn->rec_cap;
    }
    if (A.learned) {
        if (!(S.learn && S.learn->have_mlp)) return cudaErrorInvalidValue;
        A.mlp = S.learn->mlp;
        const cudaError_t e = build_learn_setup();
        if (e != cudaSuccess) return e;
    }
    if (A.prop_log) cudaMemsetAsync(A.prop_log, 0xff, (size_t)S.cap_nodes * 8 * sizeof(int32_t), st);
    // the per-rank histograms and done counters are zero here: zeroed at
    // allocation, cleaned by the kernel that used them, and zeroed again by
    // build_read_stats after a build that stopped on an error
    for (int k = 0; k < 2; k++) {
        A.lo_buf[k] = S.n_lo[k];
        A.hi_buf[k] = S.n_hi[k];
        A.info_buf[k] = S.n_info[k];
        A.refs_buf[k] = S.refs[k];
        A.ref_node_buf[k] = S.ref_node[k];
    }
    A.level = 0;
    k_root<<<std::min<unsigned>(G, nt / 256 + 1), 256, 0, st>>>(A, box, verts, tris, nt, S.tb);
    const bool exact_small = A.learned || A.exact_max >= kWarpExact;
    const uint32_t sub_E = sub_stack_entries(S.p.max_depth);
    const size_t sub_smem = kSubWarps * sub_warp_smem(sub_E, exact_small);
    // (a level's references are two to three times the triangles, its nodes of a
    // CTA each rarely below 64 references; a reference tile is 1,024 references)
    const unsigned g_nodes3 = level_grid(S.sm_count, 3, nt / 32), g_nodes4 = level_grid(S.sm_count, 4, nt / 32);
    const unsigned g_plan = level_grid(S.sm_count, kPlanGrid, nt / 256);
    const bool binned_only = !A.learned && A.exact_max == 0 && S.p.level_streams != 2;
    for (uint32_t L = 0; L <= S.p.max_depth; L++) {
        A.level = L;
        A.lc = &S.ctr->lvl[L];
        A.nlc = &S.ctr->lvl[L + 1];
        if (binned_only) {
            // one wave (four CTAs per SM resident), grid-stride over the work
            if (nt > kFewRefs) launch_pdl(k_decide<128>, S.sm_count * 8, 128, 0, st, A);
            else launch_pdl(k_decide<256>, g_nodes4, 256, 0, st, A);
            launch_pdl(k_plan_refs, g_plan, kScanThreads, 0, st, A, S.plan_flags,
                       static_cast<U7 *>(S.plan_agg), static_cast<U7 *>(S.plan_incl), S.ref_recs, S.plan_done,
                       &A.lc->plan_ticket);
            continue;
        }
        // large (and medium) nodes on the second stream, beside the small
        // nodes (independent nodes; both only add to the level tallies):
        // binned histograms, or the proposer's features, inference and costing
        cudaEventRecord(S.ev_fork, st);
        cudaStreamWaitEvent(S.aux, S.ev_fork, 0);
        // one wave: three (four) CTAs per SM resident
        if (A.learned) k_hist<kHistRows><<<g_nodes4, 256, 0, S.aux>>>(A);
        else if (A.exact_max >= kWarpExact) k_hist<kHistExact><<<g_nodes3, 256, 0, S.aux>>>(A);
        else k_hist<kHistChunks><<<g_nodes3, 256, 0, S.aux>>>(A);
        if (A.learned) {
            // the proposer's chain on the second stream after the histograms
            // (every proposer row comes from k_hist), beside the small nodes
            if (mlp_use_tcgen05() && A.mlp.tcw) launch_pdl(k_learn<true>, S.sm_count, 256, kTcSmem, S.aux, A);
            else launch_pdl(k_learn<false>, S.sm_count, 256, kTileSmem, S.aux, A);
            // the two costing kernels take disjoint rows (by reference count)
            // and only add to the tallies: the warp-costed rows on a third
            // stream, beside the CTA-costed ones
            cudaEventRecord(S.ev_learn, S.aux);
            cudaStreamWaitEvent(S.aux2, S.ev_learn, 0);
            k_refine_warp<<<g_nodes3, 256, 0, S.aux2>>>(A);
            cudaEventRecord(S.ev_join2, S.aux2);
            launch_pdl(k_refine_cta, g_nodes3, 256, 0, S.aux, A);
        }
        cudaEventRecord(S.ev_join, S.aux);
        if (A.learned) {
            launch_pdl(k_small<true, true>, level_grid(S.sm_count, 5, nt / 32), 256, 0, st, A);
        } else if (A.exact_max >= kWarpExact) {
            launch_pdl(k_small<true, false>, g_nodes4, 256, 0, st, A);
        } else {
            launch_pdl(k_small<false, false>, g_nodes4, 256, 0, st, A);
        }
        cudaStreamWaitEvent(st, S.ev_join, 0);
        if (A.learned) cudaStreamWaitEvent(st, S.ev_join2, 0);
        launch_pdl(k_plan_refs, g_plan, kScanThreads, 0, st, A, S.plan_flags, static_cast<U7 *>(S.plan_agg),
                   static_cast<U7 *>(S.plan_incl), S.ref_recs, S.plan_done, &A.lc->plan_ticket);
    }
    if (A.defer) {
        // every subtree (roots 0 .. the last level's total, tickets of level
        // 0's counter: the earliest roots, with the largest subtrees, first),
        // then their places and the final layout; tag level 63 keeps the
        // scan's flags apart from the levels'
        A.lc = &S.ctr->lvl[0];
        A.nlc = &S.ctr->lvl[S.p.max_depth + 1];
        const unsigned g_sub = std::min(g_nodes4, sub_grid(S.sm_count));
        if (exact_small)
            launch_pdl(k_subtree<true>, g_sub, kSubWarps * 32, sub_smem, st, A, sub_E);
        else
            launch_pdl(k_subtree<false>, g_sub, kSubWarps * 32, sub_smem, st, A, sub_E);
        A.level = 63;
        A.lc = &S.ctr->lvl[S.p.max_depth + 1];
        launch_pdl(k_sub_scan, std::min<unsigned>(S.sm_count * 2, nt / kTile + 1), kScanThreads, 0, st, A, S.sub_flags, S.sub_agg, S.sub_incl);
        launch_pdl(k_sub_place, level_grid(S.sm_count, 8, nt / 64), 256, 0, st, A);
    }
    S.active = true;
    S.last_level = S.p.max_depth + 1;
    return cudaGetLastError();
}

const uint32_t *build_nodes_total_ptr(const BuildState &S) {
    return &S.ctr->lvl[S.p.max_depth + 1].nodes_total;
}

hk_status build_read_stats(BuildState &S, cudaStream_t st, hk_tree_stats *out) {
    BuildCounters c;
    uint32_t err = 0;
    if (cudaMemcpyAsync(&c, S.ctr, sizeof(c), cudaMemcpyDeviceToHost, st) != cudaSuccess) return HK_E_CUDA;
    if (cudaMemcpyAsync(&err, S.err, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return HK_E_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return HK_E_CUDA;
    S.last_err = err;
    if (err) {
        cudaMemsetAsync(S.err, 0, 4, st);
        // a stopped build may leave partial histograms behind
        cudaMemsetAsync(S.hist, 0, (size_t)S.cap_large * kHist * sizeof(uint32_t), st);
        cudaMemsetAsync(S.done, 0, (size_t)S.cap_large * sizeof(uint32_t), st);
        if (err & (4u | kErrTensorWait)) return HK_E_DEVICE_TIMEOUT;   // a bounded wait ran out
        if (err & (8u | 16u)) return HK_E_BOUNDS;       // a partition / plan check fired
        return HK_E_CAPACITY;                           // an arena or list was too small
    }
    const LevelCounters &fin = c.lvl[S.last_level];
    out->nodes = fin.nodes_total;
    out->refs = fin.leafrefs_total;
    out->leaves = c.leaves;
    out->depth = c.depth;
    out->capacity_hit = c.capacity_hit;
    out->learned_nodes = c.learned_nodes;
    out->fallback_nodes = c.fallback_nodes;
    return HK_OK;
}

}  // namespace hk
