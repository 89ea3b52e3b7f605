// Matrix passes over level 0 that stream the matrix through shared memory: y = A x (with row weights),
// r = b - A x, and the smoothing sweep y = x + w Dinv (b - A x).
//
// What bounds them: the FP32 values (63 per node) come from HBM once a pass, 0.71 GB for 2M nodes, 108 us at the
// measured copy rate.  Read directly by two lanes per node (k_amg_l0, k_spmv), every load instruction touches
// one line per node, a node's 252 bytes lying apart, and the L1 wavefronts (78 % busy), not HBM, set the time.  Here
// a CTA takes a tile of kTileNodes consecutive nodes, whose values, columns, smoother blocks and right-hand side
// are contiguous, copies them to shared memory (cp.async, 16 bytes a thread) and reads them there; only the gathers
// of x go through L1.  Nine CTAs an SM cover each other's copies: two stages in one CTA left room for three
// and took 231 us.  The row pointers are 9 x the slot pointers, so they are not read.  Lanes per node and the order of
// the sums are those of the kernels they stand in for, so the results are the same bits.
// 2M nodes: sweep 178 -> 138 us, product 162 -> 122 us; 500k nodes: 55 -> 42, 50 -> 37 us.  What is left above the copy
// rate is instructions (half the issue slots) and the latency of the gathers.
// In FP64 the tile is twice as large, fewer CTAs fit, and the direct kernels stay the faster ones (260 against 305 us).
//
// `rev` walks the tiles backwards.  Passes over the same matrix alternate the direction, so that a pass starts on
// what the last one left in L2 (126 MB): most of the matrix at 1M triangles, a sixth at 4M.
#include "sw2_launch.h"

namespace sw2 {

constexpr int kTileNodes = 64;
constexpr int kTileSlots = 8 * kTileNodes;   // tiles with more neighbour slots are read from global memory

struct TileStage {
    float v[9 * kTileSlots + 4];   // starts at the 16-byte boundary before the tile's first value
    int col[kTileSlots + 4];
    float D[9 * kTileNodes];
    float b[3 * kTileNodes];
};

// count entries of src from index first to shared memory, 16 bytes at a time from the 16-byte boundary at or before it
// (src itself is 16-byte aligned).  Unless it is the last tile, what the final piece reads past the range is the next
// tile's; the last tile's entries up to `limit` are read one by one at the end.
template <class T, int NT>
__device__ __forceinline__ void stage_range(T* dst, const T* src, int first, int count, int limit, bool last) {
    const int skew = first & 3, units = (skew + count + 3) >> 2;
    const T* from = src + (first - skew);
    if (!last) {
        for (int u = threadIdx.x; u < units; u += NT) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(dst + 4 * u);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from + 4 * u) : "memory");
        }
    } else {
        for (int e = threadIdx.x; e < skew + count; e += NT)
            if (first - skew + e < limit) dst[e] = from[e];
    }
}

// this lane's share of the three rows' sums: slots lane, lane + 2, ..
__device__ __forceinline__ void lane_sums(const float* v, const int* col, int deg, const float* __restrict__ x, int lane,
                                          double& y0, double& y1, double& y2) {
    const int len = 3 * deg;
#pragma unroll 2
    for (int j = lane; j < deg; j += 2) {
        const int c = col[j];
        const double x0 = x[3 * c], x1 = x[3 * c + 1], x2 = x[3 * c + 2];
        const float* v0 = v + 3 * j;
        y0 += (double)v0[0] * x0 + (double)v0[1] * x1 + (double)v0[2] * x2;
        const float* v1 = v0 + len;
        y1 += (double)v1[0] * x0 + (double)v1[1] * x1 + (double)v1[2] * x2;
        const float* v2 = v1 + len;
        y2 += (double)v2[0] * x0 + (double)v2[1] * x1 + (double)v2[2] * x2;
    }
}

template <int MODE>
__global__ void __launch_bounds__(2 * kTileNodes) k_tile_rows(BlockCSR A, const float* __restrict__ vals, const float* __restrict__ dinv,
                                                              const float* __restrict__ b, const float* __restrict__ x,
                                                              float* __restrict__ y, const double* __restrict__ rw, double w,
                                                                 int rev, const int* __restrict__ skip) {
    if (skip && *skip) return;
    constexpr int LANES = 2, NT = kTileNodes * LANES;
    static_assert(L0Lanes<float>::value == LANES && SpmvLanes<float>::value == LANES, "the lanes of the kernels it stands in for");
    __shared__ __align__(16) TileStage S;
    const int ntiles = (A.nnodes + kTileNodes - 1) / kTileNodes;
    const int lane = threadIdx.x & (LANES - 1), sub = threadIdx.x / LANES;
    const int nslots = A.nnz / 9;
    auto pointers = [&](int t, int& p0, int& p1, int& q0, int& q1) {   // slots of tile t and of this thread's node
        p0 = p1 = q0 = q1 = 0;
        if (t >= ntiles) return;
        const int a0 = (rev ? ntiles - 1 - t : t) * kTileNodes;
        p0 = A.bptr[a0];
        p1 = A.bptr[min(a0 + kTileNodes, A.nnodes)];
        if (a0 + sub < A.nnodes) { q0 = A.bptr[a0 + sub]; q1 = A.bptr[a0 + sub + 1]; }
    };
    int p0, p1, q0, q1;
    pointers(blockIdx.x, p0, p1, q0, q1);
#pragma unroll 1
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int a0 = (rev ? ntiles - 1 - t : t) * kTileNodes, cnt = min(kTileNodes, A.nnodes - a0);
        const bool staged = p1 - p0 <= kTileSlots, last = a0 + kTileNodes >= A.nnodes;
        if (staged) {
            stage_range<float, NT>(S.v, vals, 9 * p0, 9 * (p1 - p0), A.nnz, last);
            stage_range<int, NT>(S.col, A.bcol, p0, p1 - p0, nslots, last);
        }
        if (MODE == 1) stage_range<float, NT>(S.D, dinv, 9 * a0, 9 * cnt, 9 * A.nnodes, last);
        if (MODE != 2) stage_range<float, NT>(S.b, b, 3 * a0, 3 * cnt, 3 * A.nnodes, last);
        asm volatile("cp.async.commit_group;" ::: "memory");
        int np0, np1, nq0, nq1;   // of the next tile, one step before they are needed
        pointers(t + gridDim.x, np0, np1, nq0, nq1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const int a = a0 + sub;
        const bool valid = a < A.nnodes;
        double y0 = 0, y1 = 0, y2 = 0;
        if (staged) {
            const int sv = (9 * p0) & 3, sc = p0 & 3;
            lane_sums(S.v + sv + 9 * (q0 - p0), S.col + sc + (q0 - p0), q1 - q0, x, lane, y0, y1, y2);
        } else {
            lane_sums(vals + 9 * q0, A.bcol + q0, q1 - q0, x, lane, y0, y1, y2);
        }
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) {
            y0 += __shfl_xor_sync(0xffffffffu, y0, o);
            y1 += __shfl_xor_sync(0xffffffffu, y1, o);
            y2 += __shfl_xor_sync(0xffffffffu, y2, o);
        }
        if (lane == 0 && valid) {
            if (MODE == 2) {
                if (rw) {   // the product rounded to VT, then its row weights, as two passes would
                    y0 = (double)(float)y0 * rw[3 * a]; y1 = (double)(float)y1 * rw[3 * a + 1]; y2 = (double)(float)y2 * rw[3 * a + 2];
                }
                y[3 * a] = (float)y0; y[3 * a + 1] = (float)y1; y[3 * a + 2] = (float)y2;
            } else {
                const double r0 = (double)S.b[3 * sub] - y0, r1 = (double)S.b[3 * sub + 1] - y1, r2 = (double)S.b[3 * sub + 2] - y2;
                if (MODE == 0) {
                    y[3 * a] = (float)r0; y[3 * a + 1] = (float)r1; y[3 * a + 2] = (float)r2;
                } else {
                    const float* D = S.D + 9 * sub;
                    y[3 * a] = (float)((double)x[3 * a] + w * ((double)D[0] * r0 + (double)D[1] * r1 + (double)D[2] * r2));
                    y[3 * a + 1] = (float)((double)x[3 * a + 1] + w * ((double)D[3] * r0 + (double)D[4] * r1 + (double)D[5] * r2));
                    y[3 * a + 2] = (float)((double)x[3 * a + 2] + w * ((double)D[6] * r0 + (double)D[7] * r1 + (double)D[8] * r2));
                }
            }
        }
        __syncthreads();   // the next tile overwrites this one
        p0 = np0; p1 = np1; q0 = nq0; q1 = nq1;
    }
}

template <int MODE>
static void run_tiles(const BlockCSR& A, const float* vals, const float* dinv, const float* b, const float* x, float* y,
                      const double* rw, double w, int rev, const int* skip, cudaStream_t st) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tile_rows<MODE>, 2 * kTileNodes, 0) != cudaSuccess)
        return;   // the caller's error check reports it
    const int ntiles = (A.nnodes + kTileNodes - 1) / kTileNodes, most = sms * (per_sm > 0 ? per_sm : 1);
    k_tile_rows<MODE><<<ntiles < most ? ntiles : most, 2 * kTileNodes, 0, st>>>(A, vals, dinv, b, x, y, rw, w, rev, skip);
}
void tile_sweep(const BlockCSR& A, const float* vals, const float* dinv, const float* b, const float* x, float* y, double w,
                int rev, const int* skip, cudaStream_t st) {
    run_tiles<1>(A, vals, dinv, b, x, y, nullptr, w, rev, skip, st);
}
void tile_resid(const BlockCSR& A, const float* vals, const float* b, const float* x, float* r, int rev, const int* skip, cudaStream_t st) {
    run_tiles<0>(A, vals, nullptr, b, x, r, nullptr, 0.0, rev, skip, st);
}
void tile_product(const BlockCSR& A, const float* vals, const float* x, float* y, const double* rw, int rev, const int* skip, cudaStream_t st) {
    run_tiles<2>(A, vals, nullptr, nullptr, x, y, rw, 0.0, rev, skip, st);
}

}  // namespace sw2
