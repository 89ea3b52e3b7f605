// The end of a two-phase reduction: the last block sums (or takes the maximum of) the blocks' partials in
// block order.  One thread that loaded each partial as it needed it took 75-140 us for the 1184 partials of a
// full grid, an L2 round trip per partial; here a warp loads 32 at a time, the next 32 under way, and the order
// of the additions stays.  The columns of a reduction are loaded together, and a grid of a few blocks makes only their
// additions: column by column and 32 additions at least, a block-Jacobi BiCGStab iteration on 105 nodes was 8 % slower
// than with the one thread (1.30 and 1.42 ms a solve; 1.28 now).
#pragma once
#include <cuda_runtime.h>

namespace sw2 {

// Column c < N of the partials p[4 k + c], k < count, for all 32 lanes of the one warp that calls it: the sum in order of k, or
// for the columns in the bit set MAXES the largest of 0 and the entries (fmax: a NaN is passed over, as one by one)
template <unsigned MAXES, int N>
__device__ __forceinline__ void reduce_partials(const double* p, int count, double (&out)[N]) {
    const int lane = threadIdx.x & 31;
    double next[N], cur[N];
    auto load = [&](int k) {
#pragma unroll
        for (int c = 0; c < N; c++) next[c] = k < count ? __ldcg(p + 4 * (size_t)k + c) : 0.0;
    };
    auto add = [&](int l) {
#pragma unroll
        for (int c = 0; c < N; c++)
            if (!(MAXES >> c & 1)) out[c] += __shfl_sync(0xffffffffu, cur[c], l);
    };
#pragma unroll
    for (int c = 0; c < N; c++) out[c] = 0.0;
    load(lane);
    for (int base = 0; base < count; base += 32) {
#pragma unroll
        for (int c = 0; c < N; c++) {
            cur[c] = next[c];
            if (MAXES >> c & 1) out[c] = fmax(out[c], cur[c]);
        }
        load(base + 32 + lane);
        if (count - base >= 32) {
#pragma unroll
            for (int l = 0; l < 32; l++) add(l);
        } else {
            for (int l = 0; l < count - base; l++) add(l);
        }
    }
#pragma unroll
    for (int c = 0; c < N; c++)
        if (MAXES >> c & 1) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) out[c] = fmax(out[c], __shfl_xor_sync(0xffffffffu, out[c], o));
        }
}

}  // namespace sw2
