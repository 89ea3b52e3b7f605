// One cycle of right-preconditioned GMRES(m) on the scaled SW2 system, entirely
// on the device, so that a cycle is a few CUDA graph replays (kGmSegment steps each).
//
// Why next to the reference's BiCGStab: with an approximate multilevel
// preconditioner the preconditioned SW2 operator at large Courant numbers is far
// from normal, and BiCGStab's residual then swings by orders of magnitude (in
// FP32 it does not recover).  GMRES minimises the residual over the Krylov space,
// so it decreases monotonically; restarted from the true FP64 residual after each
// cycle it serves both the FP64 solve and the FP32 inner solve of the iterative
// refinement.
//
// A cycle from x = 0 on right-hand side r, minimising ||W (r - A M^-1 V y)||_2 for
// the row weights W = diag(rw):
//   beta = ||W r||_2, v_0 = W r / beta, g = beta e_0
//   for j < m:  w = W A M^-1 v_j ; h_{:,j} = V_j^T w (one multi-dot pass) ;
//               w -= V_j h_{:,j} ; h_{j+1,j} = ||w|| ; v_{j+1} = w / h_{j+1,j} ;
//               Givens rotation of column j ; stop when |g_{j+1}| <= rtol * beta
//   y = H^-1 g (k x k triangular), out = M^-1 (V_k y)
// Classical Gram-Schmidt keeps one pass over the basis per step; its dot products
// accumulate in FP64 whatever the basis precision.  The rotations and the
// triangular solve run in one thread (k <= kGmM).  Deterministic: fixed block
// order in every reduction, no atomics besides the last-block counter.
#include <cmath>
#include "sw2_launch.h"

namespace sw2 {

static int gm_grid(long n) {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0; cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    long need = (n + 255) / 256, cap = 4L * sms;
    if (cap > kMaxBlocks) cap = kMaxBlocks;
    return (int)(need < cap ? (need < 1 ? 1 : need) : cap);
}

// last block of the grid (thread 0) after every block published its partials
__device__ __forceinline__ bool gm_last_block(const GmresDev& G) {
    __shared__ bool is_last;
    __threadfence();   // every thread's partial writes are visible device-wide before the count
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int t = atomicInc(G.counter, gridDim.x - 1);
        is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    return is_last;
}

// 16-byte loads and stores of basis entries (4 floats or 2 doubles); the basis stride is a
// multiple of 4 entries, so every vector starts on a 16-byte boundary.
template <class VT> struct Quad { static constexpr int N = 16 / sizeof(VT); };
__device__ __forceinline__ void ld16(const float* p, float (&o)[4]) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
}
__device__ __forceinline__ void ld16(const double* p, double (&o)[2]) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(p));
    o[0] = t.x; o[1] = t.y;
}
__device__ __forceinline__ void ld16_rw(const float* p, float (&o)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
}
__device__ __forceinline__ void ld16_rw(const double* p, double (&o)[2]) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    o[0] = t.x; o[1] = t.y;
}
__device__ __forceinline__ void st16(float* p, const float (&o)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void st16(double* p, const double (&o)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
}

// In the last block, the sum of column col of the blocks' partials by all its threads
// (each thread a fixed stride of blocks, then the warp and block trees): the result in
// thread 0.  Every thread of the block calls it.
__device__ __forceinline__ double gm_sum_partials(const GmresDev& G, int col) {
    __shared__ double red[8];
    double t = 0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) t += __ldcg(G.partial + col * kMaxBlocks + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    double s = 0;
    if (threadIdx.x == 0)
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) s += red[k];
    return s;
}

// beta = ||r||_2 ; g = beta e_0 ; target = rtol * beta ; columns = 0
template <class VT>
__global__ void __launch_bounds__(256) k_gm_start(int n, const VT* __restrict__ r, const double* __restrict__ rw,
                                                  GmresDev G) {
    __shared__ double sh[8];
    double ss = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = (double)r[i] * rw[i];
        ss += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < 8; k++) t += sh[k];
        G.partial[blockIdx.x] = t;
    }
    if (!gm_last_block(G)) return;
    const double tsum = gm_sum_partials(G, 0);
    if (threadIdx.x == 0) {
        const double beta = sqrt(tsum);
        G.scal[0] = beta;
        G.scal[1] = G.scal[3] * beta;       // stopping target on |g_{j+1}|
        G.scal[2] = beta;
        for (int k = 0; k <= kGmM; k++) G.g[k] = 0.0;
        G.g[0] = beta;
        G.state[1] = 0;
        G.state[2] = isfinite(beta) ? 0 : 2;
        G.state[0] = (beta > 0.0 && isfinite(beta)) ? 0 : 1;
    }
}

template <class VT>
__global__ void k_gm_v0(int n, const VT* __restrict__ r, const double* __restrict__ rw, VT* __restrict__ v0, GmresDev G) {
    if (G.state[0]) return;
    const double inv = 1.0 / G.scal[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v0[i] = (VT)((double)r[i] * rw[i] * inv);
}

// h_k = v_k . w for k < nv (w = v_nv before orthogonalisation), into column j of H.
// A block takes kDotGroup basis vectors at a time: their 16-byte loads are issued together, and each thread keeps an accumulator
// for each.  A thread's elements and the reduction tree do not depend on the group, so every h_k is the same sum as with all
// accumulators in one thread; w comes from L2 for every group but the first.
// On a small mesh a block has one load per thread and vector, and what bounded it was its own end (a tree of 40 shuffles, a
// fence, a count) as one block per group, with the sum over the blocks left to one of all blocks, from partials a column's width
// apart: 19.6 us at 188k FP64 entries and 58 us at 1.5M FP32 ones (means over cycles of 30 and 50 steps), now 11.5
// and 44 us.  The eight trees share their shuffles: at each level a lane keeps half of the columns and hands the others to its
// partner, and each column's tree stays the same.
// Four blocks on an SM hold the whole grid (592 blocks) at once: with the three that its registers allowed freely the FP32
// case took 51 us.
constexpr int kDotGroup = 8;
constexpr int kDotLoads = 10;   // partials a lane loads at once: half of a full grid's 592 / 32
template <int O, int K>
__device__ __forceinline__ void dot_level(double* acc) {   // K columns -> K / 2, the upper ones where lane & O
    const bool up = threadIdx.x & O;
#pragma unroll
    for (int k = 0; k < K / 2; k++) {
        const double keep = up ? acc[k + K / 2] : acc[k], give = up ? acc[k] : acc[k + K / 2];
        acc[k] = keep + __shfl_xor_sync(0xffffffffu, give, O);
    }
}
template <class VT>
__global__ void __launch_bounds__(256, 4) k_gm_dots(int n, int nv, const VT* __restrict__ Vb, size_t ld, double* dst,
                                                 GmresDev G) {
    if (G.state[0]) return;
    __shared__ double sh[2][8][kDotGroup];
    const VT* w = Vb + (size_t)nv * ld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NQ = Quad<VT>::N;
    const int nq = n / NQ;
    for (int k0 = 0, turn = 0; k0 < nv; k0 += kDotGroup, turn ^= 1) {
        double acc[kDotGroup];
#pragma unroll
        for (int k = 0; k < kDotGroup; k++) acc[k] = 0.0;
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
            const size_t i = (size_t)q * NQ;
            VT wq[NQ];
            ld16_rw(w + i, wq);
            VT x[kDotGroup][NQ];
#pragma unroll
            for (int k = 0; k < kDotGroup; k++)
                if (k0 + k < nv) ld16(Vb + (size_t)(k0 + k) * ld + i, x[k]);
#pragma unroll
            for (int k = 0; k < kDotGroup; k++)
                if (k0 + k < nv) {
#pragma unroll
                    for (int c = 0; c < NQ; c++) acc[k] += (double)x[k][c] * (double)wq[c];
                }
        }
        for (int i = nq * NQ + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const double wi = w[i];
#pragma unroll
            for (int k = 0; k < kDotGroup; k++)
                if (k0 + k < nv) acc[k] += (double)Vb[(size_t)(k0 + k) * ld + i] * wi;
        }
        dot_level<16, 8>(acc);
        dot_level<8, 4>(acc);
        dot_level<4, 2>(acc);
        double v = acc[0];                          // column lane >> 2, bit by bit
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if ((lane & 3) == 0) sh[turn][warp][lane >> 2] = v;
        __syncthreads();
        if (threadIdx.x < kDotGroup && k0 + (int)threadIdx.x < nv) {
            double t = 0;
            for (int w8 = 0; w8 < 8; w8++) t += sh[turn][w8][threadIdx.x];
            G.partial[(k0 + threadIdx.x) * kMaxBlocks + blockIdx.x] = t;
        }
    }
    if (gm_last_block(G)) {   // warp w sums columns w, w + 8, ...; its lanes stride over the blocks
        for (int c = warp; c < nv; c += 8) {
            double t = 0;
            for (int b0 = lane; b0 < (int)gridDim.x; b0 += 32 * kDotLoads) {
                double p[kDotLoads];
#pragma unroll
                for (int u = 0; u < kDotLoads; u++) {
                    const int b = b0 + 32 * u;
                    p[u] = b < (int)gridDim.x ? __ldcg(G.partial + c * kMaxBlocks + b) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kDotLoads; u++)
                    if (b0 + 32 * u < (int)gridDim.x) t += p[u];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) dst[c] = t;
        }
    }
}

// First pass of classical Gram-Schmidt with re-orthogonalisation (CGS2): w -= sum_k h_k v_k, no norm.
template <class VT>
__global__ void __launch_bounds__(256) k_gm_sub(int n, int j, VT* __restrict__ Vb, size_t ld, GmresDev G) {
    if (G.state[0]) return;
    __shared__ double h[kGmM + 1];
    for (int k = threadIdx.x; k <= j; k += blockDim.x) h[k] = __ldcg(G.H + j * (kGmM + 1) + k);
    __syncthreads();
    VT* w = Vb + (size_t)(j + 1) * ld;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v = w[i];
        int k = 0;
        for (; k + 8 <= j + 1; k += 8) {
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = (double)Vb[(size_t)(k + u) * ld + i];
#pragma unroll
            for (int u = 0; u < 8; u++) v -= h[k + u] * x[u];
        }
        for (; k <= j; k++) v -= h[k] * (double)Vb[(size_t)k * ld + i];
        w[i] = (VT)v;
    }
}

// w -= sum_k h_k v_k ; h_{j+1,j} = ||w|| ; Givens rotation of column j ; convergence test.
// SECOND: the coefficients come from the re-orthogonalisation pass (G.H2) and are added to
// those of the first pass (column j of G.H) before the rotations.
template <class VT, bool SECOND>
__global__ void __launch_bounds__(256) k_gm_orth(int n, int j, VT* __restrict__ Vb, size_t ld, GmresDev G) {
    if (G.state[0]) return;
    __shared__ double sh[8];
    __shared__ double h[kGmM + 1];
    for (int k = threadIdx.x; k <= j; k += blockDim.x)
        h[k] = SECOND ? __ldcg(G.H2 + k) : __ldcg(G.H + j * (kGmM + 1) + k);
    __syncthreads();
    VT* w = Vb + (size_t)(j + 1) * ld;
    double ss = 0;
    constexpr int NQ = Quad<VT>::N;
    const int nq = n / NQ;
    // NQ consecutive entries per thread, eight 16-byte basis loads in flight, then the
    // updates of each entry in basis order (the same arithmetic per entry as one at a time)
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        const size_t i = (size_t)q * NQ;
        VT wq[NQ];
        ld16_rw(w + i, wq);
        double v[NQ];
#pragma unroll
        for (int c = 0; c < NQ; c++) v[c] = wq[c];
        int k = 0;
        for (; k + 8 <= j + 1; k += 8) {
            VT x[8][NQ];
#pragma unroll
            for (int u = 0; u < 8; u++) ld16(Vb + (size_t)(k + u) * ld + i, x[u]);
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int c = 0; c < NQ; c++) v[c] -= h[k + u] * (double)x[u][c];
        }
        for (; k <= j; k++) {
            VT x[NQ];
            ld16(Vb + (size_t)k * ld + i, x);
#pragma unroll
            for (int c = 0; c < NQ; c++) v[c] -= h[k] * (double)x[c];
        }
        VT o[NQ];
#pragma unroll
        for (int c = 0; c < NQ; c++) {
            o[c] = (VT)v[c];
            ss += (double)o[c] * (double)o[c];
        }
        st16(w + i, o);
    }
    for (int i = nq * NQ + blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v = w[i];
        for (int k = 0; k <= j; k++) v -= h[k] * (double)Vb[(size_t)k * ld + i];
        const VT vv = (VT)v;
        w[i] = vv;
        ss += (double)vv * (double)vv;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < 8; k++) t += sh[k];
        G.partial[blockIdx.x] = t;
    }
    if (!gm_last_block(G)) return;
    // the column and the earlier rotations in shared memory: one thread applies them in turn, and each step from
    // global memory was an L2 round trip (8.7 us a launch at 30 columns on a small mesh)
    __shared__ double cs[kGmM], sn[kGmM];
    double* col = G.H + j * (kGmM + 1);
    for (int k = threadIdx.x; k <= j; k += blockDim.x) {
        if (SECOND) h[k] = __ldcg(col + k) + h[k];
        if (k < j) { cs[k] = __ldcg(G.cs + k); sn[k] = __ldcg(G.sn + k); }
    }
    const double tsum = gm_sum_partials(G, 0);            // (synchronises the block)
    if (threadIdx.x == 0) {
        const double hn = sqrt(tsum);
        for (int k = 0; k < j; k++) {                 // earlier rotations
            const double a = h[k], b = h[k + 1];
            h[k] = cs[k] * a + sn[k] * b;
            h[k + 1] = -sn[k] * a + cs[k] * b;
        }
        const double a = h[j], b = hn;
        const double rr = hypot(a, b);
        const double c = rr > 0.0 ? a / rr : 1.0, s = rr > 0.0 ? b / rr : 0.0;
        G.cs[j] = c; G.sn[j] = s;
        h[j] = rr;
        col[j + 1] = 0.0;
        G.g[j + 1] = -s * G.g[j];
        G.g[j] = c * G.g[j];
        G.scal[4] = hn;
        G.scal[2] = fabs(G.g[j + 1]);
        G.state[1] = j + 1;
        if (!isfinite(rr) || !isfinite(hn)) { G.state[2] = 2; G.state[0] = 1; G.state[1] = j; }
        else if (rr == 0.0) { G.state[2] = 1; G.state[0] = 1; G.state[1] = j; }   // breakdown: drop column j
        else if (!(fabs(G.g[j + 1]) > G.scal[1]) || hn == 0.0) G.state[0] = 1;
    }
    __syncthreads();
    for (int k = threadIdx.x; k <= j; k += blockDim.x) col[k] = h[k];
}

template <class VT>
__global__ void k_gm_scale(int n, int j, VT* __restrict__ Vb, size_t ld, GmresDev G) {
    if (G.state[0]) return;
    const double inv = 1.0 / G.scal[4];
    VT* w = Vb + (size_t)(j + 1) * ld;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) w[i] = (VT)((double)w[i] * inv);
}

// y = H^-1 g on the k columns built (upper triangular after the rotations).  One thread substitutes, in the order
// of the columns; the rows it needs next are fetched into shared memory kSolveRows at a time by the block.
constexpr int kSolveRows = 16;
__global__ void __launch_bounds__(256) k_gm_solve(GmresDev G) {
    __shared__ double rows[kSolveRows][kGmM], y[kGmM];
    const int k = G.state[1];
    for (int top = k - 1; top >= 0; top -= kSolveRows) {
        const int low = top - kSolveRows + 1 > 0 ? top - kSolveRows + 1 : 0;
        __syncthreads();
        for (int e = threadIdx.x; e < (top - low + 1) * k; e += blockDim.x) {
            const int r = e % (top - low + 1), t = e / (top - low + 1);   // row low + r of column t
            if (t >= low + r) rows[r][t] = G.H[t * (kGmM + 1) + low + r];
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = top; i >= low; i--) {
                double s = G.g[i];
                for (int t = i + 1; t < k; t++) s -= rows[i - low][t] * y[t];
                const double d = rows[i - low][i];
                y[i] = d != 0.0 ? s / d : 0.0;
            }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < k; t += blockDim.x) G.y[t] = y[t];
    if (threadIdx.x == 0) G.state[0] = 0;   // let the final preconditioner apply run
}

// out = V_k y, 16 bytes per load and 8 basis vectors in flight (each entry's sum in basis order)
template <class VT>
__global__ void __launch_bounds__(256) k_gm_combine(int n, const VT* __restrict__ Vb, size_t ld, VT* __restrict__ out, GmresDev G) {
    __shared__ double y[kGmM];
    const int k = G.state[1];
    for (int t = threadIdx.x; t < k; t += blockDim.x) y[t] = G.y[t];
    __syncthreads();
    constexpr int NQ = Quad<VT>::N;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q * NQ < n; q += gridDim.x * blockDim.x) {
        const size_t i = (size_t)q * NQ;          // the basis is padded to whole 16-byte pieces; out is not
        double s[NQ];
#pragma unroll
        for (int c = 0; c < NQ; c++) s[c] = 0;
        int t = 0;
        for (; t + 8 <= k; t += 8) {
            VT x[8][NQ];
#pragma unroll
            for (int u = 0; u < 8; u++) ld16(Vb + (size_t)(t + u) * ld + i, x[u]);
#pragma unroll
            for (int u = 0; u < 8; u++)
#pragma unroll
                for (int c = 0; c < NQ; c++) s[c] += y[t + u] * (double)x[u][c];
        }
        for (; t < k; t++) {
            VT x[NQ];
            ld16(Vb + (size_t)t * ld + i, x);
#pragma unroll
            for (int c = 0; c < NQ; c++) s[c] += y[t] * (double)x[c];
        }
#pragma unroll
        for (int c = 0; c < NQ; c++)
            if (i + c < (size_t)n) out[i + c] = (VT)s[c];
    }
}

template <class VT>
void gmres_begin(int n, VT* Vb, const VT* rhs, const double* rw, const GmresDev& G, cudaStream_t st) {
    const int g = gm_grid(n);
    k_gm_start<VT><<<g, 256, 0, st>>>(n, rhs, rw, G);
    k_gm_v0<VT><<<g, 256, 0, st>>>(n, rhs, rw, Vb, G);
}
template <class VT>
void gmres_steps(const BlockCSR& A, const PrecondOp<VT>& P, const VT* vals, VT* Vb, size_t ld, VT* z, const double* rw,
                 const GmresDev& G, cudaStream_t st, int first, int last, bool reorth) {
    const int n = A.n, g = gm_grid(n);
    const int* done = G.state;
    for (int j = first; j < last; j++) {
        precond_apply<VT>(A, P, Vb + (size_t)j * ld, z, done, st);
        spmv_skip<VT>(A, vals, z, Vb + (size_t)(j + 1) * ld, rw, done, st);
        k_gm_dots<VT><<<g, 256, 0, st>>>(n, j + 1, Vb, ld, G.H + (size_t)j * (kGmM + 1), G);
        if (reorth) {
            k_gm_sub<VT><<<g, 256, 0, st>>>(n, j, Vb, ld, G);
            k_gm_dots<VT><<<g, 256, 0, st>>>(n, j + 1, Vb, ld, G.H2, G);
            k_gm_orth<VT, true><<<g, 256, 0, st>>>(n, j, Vb, ld, G);
        } else {
            k_gm_orth<VT, false><<<g, 256, 0, st>>>(n, j, Vb, ld, G);
        }
        k_gm_scale<VT><<<g, 256, 0, st>>>(n, j, Vb, ld, G);
    }
}
template <class VT>
void gmres_end(const BlockCSR& A, const PrecondOp<VT>& P, VT* Vb, size_t ld, VT* z, VT* out, const GmresDev& G, cudaStream_t st) {
    k_gm_solve<<<1, 256, 0, st>>>(G);
    k_gm_combine<VT><<<gm_grid(A.n), 256, 0, st>>>(A.n, Vb, ld, z, G);
    precond_apply<VT>(A, P, z, out, nullptr, st);
}
#define SW2_GMRES_INSTANCE(VT)                                                                                             \
    template void gmres_begin<VT>(int, VT*, const VT*, const double*, const GmresDev&, cudaStream_t);                      \
    template void gmres_steps<VT>(const BlockCSR&, const PrecondOp<VT>&, const VT*, VT*, size_t, VT*, const double*,       \
                                  const GmresDev&, cudaStream_t, int, int, bool);                                          \
    template void gmres_end<VT>(const BlockCSR&, const PrecondOp<VT>&, VT*, size_t, VT*, VT*, const GmresDev&, cudaStream_t);
SW2_GMRES_INSTANCE(double)
SW2_GMRES_INSTANCE(float)

}  // namespace sw2
