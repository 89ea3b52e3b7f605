// The end of a two-phase reduction: the last block sums (or takes the maximum of) the blocks' partials in
// block order.  One thread that loaded each partial as it needed it took 75-140 us for the 1184 partials of a
// full grid, an L2 round trip per partial; here a warp loads 32 at a time, the next 32 under way, and the order
// of the additions stays.
#pragma once
#include <cuda_runtime.h>

namespace sw2 {

// p[0], p[stride], ... in order; all 32 lanes of one warp call it and get the result
__device__ __forceinline__ double ordered_sum(const double* p, int stride, int count) {
    const int lane = threadIdx.x & 31;
    double s = 0.0, next = lane < count ? __ldcg(p + (size_t)lane * stride) : 0.0;
    for (int base = 0; base < count; base += 32) {
        const double cur = next;
        const int k = base + 32 + lane;
        next = k < count ? __ldcg(p + (size_t)k * stride) : 0.0;
        const int here = count - base;
#pragma unroll
        for (int l = 0; l < 32; l++) {
            const double v = __shfl_sync(0xffffffffu, cur, l);
            if (l < here) s += v;
        }
    }
    return s;
}
// the largest of 0 and p[0], p[stride], ... (fmax: a NaN is passed over, as one by one)
__device__ __forceinline__ double warp_max(const double* p, int stride, int count) {
    double m = 0.0;
    for (int k = threadIdx.x & 31; k < count; k += 32) m = fmax(m, __ldcg(p + (size_t)k * stride));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

}  // namespace sw2
