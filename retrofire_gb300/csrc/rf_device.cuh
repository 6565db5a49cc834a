// rf_device.cuh — device helpers shared by the kernel translation units.
#ifndef RF_DEVICE_CUH
#define RF_DEVICE_CUH

#include <cuda_runtime.h>

#include "rf_exact.cuh"
#include "rf_internal.cuh"
#include "rf_kernels.cuh"

namespace rfd {
using namespace rfx;

// First in every kernel of a frame: wait for the kernel before it on the
// stream (launch_next; no wait otherwise), then let the one after it come up.
__device__ __forceinline__ void grid_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Largest i with key(i) <= x over a sorted array of n records.
template <class F>
__device__ __forceinline__ uint32_t upper_index(uint32_t n, uint32_t x, F key) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (key(mid) <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// upper_index by a whole warp for one x (all lanes call): 32 records are
// looked at a step, so 110,000 take four dependent loads instead of 17
// (vertex stage of 64 scenes with as many draws: 86 us with a binary search by
// one lane and a walk by each, 67 with these two; triangle lists 123 -> 118,
// both rasters 685 -> 664).
template <class F>
__device__ __forceinline__ uint32_t warp_find(uint32_t n, uint32_t x, F key) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) / 32u, at = lo + lane * step;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, lane == 0u || (at < hi && key(at) <= x));
        lo += (31u - __clz(b)) * step;  // (keys do not decrease: the lanes that hold are the first ones)
        hi = min(hi, lo + step);
    }
    return lo;
}

// upper_index for the 32 lanes of a warp whose x do not decrease with the
// lane (all lanes call): the search for lane 0's x, then each lane looks
// through the next records, 32 loaded at a time.
template <class F>
__device__ __forceinline__ uint32_t warp_upper_index(uint32_t n, uint32_t x, F key) {
    if (n <= 1u) return 0u;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = warp_find(n, __shfl_sync(0xFFFFFFFFu, x, 0), key), d = lo;
    for (;;) {
        const uint32_t k = lo + lane < n ? key(lo + lane) : 0xFFFFFFFFu;  // (no x is that large)
        uint32_t i = 0;  // the last of these records not above x
#pragma unroll
        for (uint32_t step = 16; step >= 1u; step >>= 1)
            if (__shfl_sync(0xFFFFFFFFu, k, i + step) <= x) i += step;
        if (__shfl_sync(0xFFFFFFFFu, k, 0) <= x) d = lo + i;
        if (!__any_sync(0xFFFFFFFFu, i == 31u)) return d;
        lo += 31u;
    }
}

// Position of the r-th set bit of v (r >= 1, at most popc(v)): halving
// search on popcounts.
__device__ __forceinline__ uint32_t nth_bit(uint32_t v, uint32_t r) {
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t w = 16; w >= 1; w >>= 1) {
        const uint32_t c = __popc(v & ((1u << w) - 1u));
        if (c < r) {
            r -= c;
            v >>= w;
            pos += w;
        }
    }
    return pos;
}
// The lane whose bits hold the k-th of all (incl: the lanes' inclusive
// counts; every lane calls).
__device__ __forceinline__ uint32_t lane_of(uint32_t incl, uint32_t k) {
    uint32_t L = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, L + step - 1u);
        if (v <= k) L += step;
    }
    return L & 31u;
}

// Warp-aggregated 64-bit counter add (all 32 lanes must call).
__device__ __forceinline__ void warp_add_u64(unsigned long long *dst, unsigned long long v,
                                             bool same_dst) {
    if (same_dst) {
        if (!__any_sync(0xFFFFFFFFu, (v >> 27) != 0ull)) {  // the sum fits 32 bits: one instruction
            v = __reduce_add_sync(0xFFFFFFFFu, (uint32_t)v);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
        }
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
    } else if (v) {
        atomicAdd(dst, v);
    }
}

// Row quantity r of half H after j scanlines (see HalfRuns): one of the two
// precomputed single-binade runs U, else the general loop from the second.
__device__ __forceinline__ float row_value(const HalfRec *__restrict__ H, const HalfRuns *__restrict__ U,
                                           int r, uint32_t j) {
    const uint32_t e0 = U->e0[r];
    if (j <= e0) return u2f(H->b0[r] + j * (uint32_t)U->i0[r]);
    const uint32_t j1 = j - e0 - 1u;
    if (j <= U->e1[r]) return u2f(U->b1[r] + j1 * (uint32_t)U->i1[r]);
    return seq_add_n(u2f(U->b1[r]), H->d[r], j1);
}

}  // namespace rfd

#endif
