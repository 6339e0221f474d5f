// hk_scan.cuh -- single-pass scans with decoupled look-back: the parts that
// the builders share.
//
// Tiles are taken in order from an atomic ticket, so every tile a CTA waits
// for belongs to a CTA that is already running and publishes its aggregate
// without waiting. A tile's flag is (tag << 2) | status, status 1 = aggregate,
// 2 = inclusive prefix; the tag names the scan, so flags of earlier scans are
// stale and the flag arrays are never cleared. Waits are bounded: one that
// runs out sets error bit 4.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace hk {

// scan values: sums of counters, element by element
__device__ __forceinline__ uint2 vadd(uint2 a, uint2 b) { return make_uint2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ uint4 vadd(uint4 a, uint4 b) {
    return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ uint2 vsub(uint2 a, uint2 b) { return make_uint2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ uint4 vsub(uint4 a, uint4 b) {
    return make_uint4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
}
template <class T> __device__ __forceinline__ T vzero();
template <> __device__ __forceinline__ uint2 vzero<uint2>() { return make_uint2(0, 0); }
template <> __device__ __forceinline__ uint4 vzero<uint4>() { return make_uint4(0, 0, 0, 0); }
__device__ __forceinline__ uint2 shfl_up(uint2 v, int d) {
    return make_uint2(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ uint4 shfl_up(uint4 v, int d) {
    return make_uint4(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d),
                      __shfl_up_sync(0xffffffffu, v.z, d), __shfl_up_sync(0xffffffffu, v.w, d));
}
__device__ __forceinline__ uint2 shfl_xor(uint2 v, int d) {
    return make_uint2(__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ uint4 shfl_xor(uint4 v, int d) {
    return make_uint4(__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d),
                      __shfl_xor_sync(0xffffffffu, v.z, d), __shfl_xor_sync(0xffffffffu, v.w, d));
}
// loads past L1 (values other CTAs of the same kernel published)
__device__ __forceinline__ uint2 ldcg(const uint2 *p) { return __ldcg(p); }
__device__ __forceinline__ uint4 ldcg(const uint4 *p) { return __ldcg(p); }

// inclusive warp scan
template <class T>
__device__ __forceinline__ T warp_incl(T v) {
    const int lane = threadIdx.x & 31;
    for (int d = 1; d < 32; d <<= 1) {
        T u = shfl_up(v, d);
        if (lane >= d) v = vadd(v, u);
    }
    return v;
}

// exclusive block scan of one value per thread (NT threads); returns the
// thread's exclusive prefix and the block total
template <int NT, class T>
__device__ __forceinline__ T block_excl(T v, T *sh_warp, T &total) {
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = warp_incl(v);
    if (lane == 31) sh_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < NW ? sh_warp[lane] : vzero<T>();
        T wi = warp_incl(w);
        if (lane < NW) sh_warp[lane] = wi;
    }
    __syncthreads();
    T wbase = warp ? sh_warp[warp - 1] : vzero<T>();
    total = sh_warp[NW - 1];
    __syncthreads();
    return vadd(wbase, vsub(inc, v));
}

// One window of a look-back (a warp, lane k at the tile k before): poll()
// gives the lane's status (0: not published yet). The window is complete once
// every tile up to the nearest inclusive one has published, whatever the tiles
// behind it do: waiting for all 32 held every tile of a level until its 32
// predecessors had loaded their references (7 of a level's 20 us). Returns that
// nearest lane (32: none in the window); a wait that runs out sets error bit 4
// and ends the look-back at the first tile without a value.
template <class Poll>
__device__ __forceinline__ int lookback_window(const Poll &poll, uint32_t *err, uint32_t spin_limit) {
    for (uint32_t spins = 0;; spins++) {
        const uint32_t st = poll();
        const uint32_t m2 = __ballot_sync(0xffffffffu, st == 2u), m0 = __ballot_sync(0xffffffffu, st == 0u);
        const int stop = m2 ? __ffs(m2) - 1 : 32;
        const uint32_t need = stop >= 31 ? 0xffffffffu : (2u << stop) - 1u;
        if (!(m0 & need)) return stop;
        if (spins >= spin_limit) {
            if ((threadIdx.x & 31u) == 0) atomicOr(err, 4u);
            return __ffs(m0) - 1;
        }
        __nanosleep(32);
    }
}

template <class T>
__device__ T lookback(const uint32_t *flags, const T *aggs, const T *incls, uint32_t tile, uint32_t tag,
                      uint32_t *err, uint32_t spin_limit) {
    const int lane = threadIdx.x & 31;
    T excl = vzero<T>();
    int32_t p = (int32_t)tile - 1;
    for (;;) {
        const int32_t q = p - lane;
        uint32_t st = 2;    // before tile 0: an inclusive prefix of zero
        const int stop = lookback_window(
            [&] {
                if (q >= 0) {
                    const uint32_t f = __ldcv(flags + q);
                    st = (f >> 2) == tag ? f & 3u : 0u;
                }
                return st;
            },
            err, spin_limit);
        __threadfence();
        T v = vzero<T>();
        if (q >= 0 && lane <= stop && st) v = lane == stop ? ldcg(incls + q) : ldcg(aggs + q);
        for (int o = 16; o; o >>= 1) v = vadd(v, shfl_xor(v, o));
        excl = vadd(excl, v);
        if (stop < 32) break;
        p -= 32;
    }
    return excl;
}

// Publishes a tile's total (an inclusive prefix for tile 0) and, by the CTA's
// first warp, looks back for the prefix of the tiles before it; every thread
// of the CTA calls it, the result (in *s_excl) is for all after it returns.
template <class T>
__device__ __forceinline__ void tile_prefix(uint32_t tile, T tot, uint32_t tag, uint32_t *flags, T *aggs, T *incls,
                                            T *s_excl, uint32_t *err, uint32_t spin_limit) {
    if (threadIdx.x == 0) {
        if (tile == 0) incls[0] = tot;
        else aggs[tile] = tot;
        __threadfence();
        *reinterpret_cast<volatile uint32_t *>(flags + tile) = (tag << 2) | (tile == 0 ? 2u : 1u);
    }
    if (threadIdx.x < 32) {
        const T e = tile ? lookback(flags, aggs, incls, tile, tag, err, spin_limit) : vzero<T>();
        if (threadIdx.x == 0) {
            if (tile) {
                incls[tile] = vadd(e, tot);
                __threadfence();
                *reinterpret_cast<volatile uint32_t *>(flags + tile) = (tag << 2) | 2u;
            }
            *s_excl = e;
        }
    }
    __syncthreads();
}

}  // namespace hk
