// Device code of the AMG levels that one thread-block cluster runs, with a cluster barrier between passes; what bounds
// them and why stands in amg_kernels.cu.
#pragma once
#include "sw2_launch.h"

namespace sw2 {

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() { int r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ int cluster_ctas() { int r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }

template <class VT> struct ClusterLevel {
    int n;
    const int *bptr, *bcol;            // node graph (level 0: neighbour slots)
    const int *agg, *mptr, *mem;       // link to the next coarser level
    const VT *val, *dinv;              // level 0: values in the CSR layout
    const VT* b;
    VT *x, *t;
};
template <class VT> struct ClusterArgs {
    int lo, nlev;                      // levels lo .. nlev-1 run in the kernel
    const int* indptr0;                // CSR rows of level 0 (used when lo == 0)
    const int* skip;
    const VT* op;                      // the coarsest level's operator, row-major
    VT* bc[kAmgMaxLevels];             // right-hand sides the kernel writes (levels past lo; the same as lev[l].b)
    ClusterLevel<VT> lev[kAmgMaxLevels];
};
struct Vec3 { double v0, v1, v2; };
template <class VT> __device__ __forceinline__ Vec3 ld3cg(const VT* p) { return Vec3{(double)__ldcg(p), (double)__ldcg(p + 1), (double)__ldcg(p + 2)}; }
template <class VT> __device__ __forceinline__ void st3(VT* p, double a, double b, double c) { p[0] = (VT)a; p[1] = (VT)b; p[2] = (VT)c; }

// lanes per node, as in k_amg_l0 (level 0) and k_amg_bsr
template <class VT, bool L0> struct RowLanes { static constexpr int value = L0 ? (sizeof(VT) == 4 ? 2 : 4) : (sizeof(VT) == 4 ? 4 : 8); };

// What a pass reads as x of node c: the vector itself, the first sweep w Dinv b, or the vector
// plus its aggregate's correction (each rounded to VT as when it is stored).
enum { X_PLAIN = 0, X_FIRST = 1, X_PROLONG = 2 };
template <class VT, int XK>
__device__ __forceinline__ Vec3 cluster_x(const ClusterLevel<VT>& L, const VT* x, const VT* xc, int c, double w) {
    if (XK == X_FIRST) {
        const Vec3 b = ld3cg(L.b + 3 * c);
        const VT* D = L.dinv + 9 * (size_t)c;
        return Vec3{(double)(VT)(w * ((double)D[0] * b.v0 + (double)D[1] * b.v1 + (double)D[2] * b.v2)),
                    (double)(VT)(w * ((double)D[3] * b.v0 + (double)D[4] * b.v1 + (double)D[5] * b.v2)),
                    (double)(VT)(w * ((double)D[6] * b.v0 + (double)D[7] * b.v1 + (double)D[8] * b.v2))};
    }
    Vec3 v = ld3cg(x + 3 * c);
    if (XK == X_PROLONG) {
        const Vec3 e = ld3cg(xc + 3 * L.agg[c]);
        v = Vec3{(double)(VT)(v.v0 + e.v0), (double)(VT)(v.v1 + e.v1), (double)(VT)(v.v2 + e.v2)};
    }
    return v;
}
// (A x) of node a by its lanes; every lane returns the sums
template <class VT, bool L0, int XK>
__device__ __forceinline__ Vec3 cluster_row(const ClusterLevel<VT>& L, const int* __restrict__ indptr0, const VT* x, const VT* xc,
                                            int a, bool valid, int lane, double w) {
    constexpr int LANES = RowLanes<VT, L0>::value;
    double y0 = 0, y1 = 0, y2 = 0;
    const int q0 = valid ? L.bptr[a] : 0, q1 = valid ? L.bptr[a + 1] : 0;
    const int rs = (L0 && valid) ? indptr0[3 * a] : 0, len = L0 ? 3 * (q1 - q0) : 3;
#pragma unroll 2
    for (int q = q0 + lane; q < q1; q += LANES) {
        const Vec3 xv = cluster_x<VT, XK>(L, x, xc, L.bcol[q], w);
        const VT* v = L0 ? L.val + rs + 3 * (q - q0) : L.val + 9 * (size_t)q;
        y0 += (double)v[0] * xv.v0 + (double)v[1] * xv.v1 + (double)v[2] * xv.v2;
        v += len;
        y1 += (double)v[0] * xv.v0 + (double)v[1] * xv.v1 + (double)v[2] * xv.v2;
        v += len;
        y2 += (double)v[0] * xv.v0 + (double)v[1] * xv.v1 + (double)v[2] * xv.v2;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        y2 += __shfl_xor_sync(0xffffffffu, y2, o);
    }
    return Vec3{y0, y1, y2};
}
// y = x + w Dinv (b - A x) over the level
template <class VT, bool L0, int XK>
__device__ __forceinline__ void cluster_sweep(const ClusterLevel<VT>& L, const int* indptr0, const VT* x, const VT* xc, VT* y,
                                              double w, int gwarp, int nwarps) {
    constexpr int LANES = RowLanes<VT, L0>::value, PER_WARP = 32 / LANES;
    const int lane = threadIdx.x & (LANES - 1), sub = (threadIdx.x & 31) / LANES;
    for (int base = gwarp * PER_WARP; base < L.n; base += nwarps * PER_WARP) {
        const int a = base + sub;
        const bool valid = a < L.n, out = valid && lane == 0;
        Vec3 b{0, 0, 0}, xa{0, 0, 0};
        double D[9];
        if (out) {                     // issued before the row's dependent loads
            b = ld3cg(L.b + 3 * a);
            xa = cluster_x<VT, XK>(L, x, xc, a, w);
#pragma unroll
            for (int e = 0; e < 9; e++) D[e] = L.dinv[9 * (size_t)a + e];
        }
        const Vec3 s = cluster_row<VT, L0, XK>(L, indptr0, x, xc, a, valid, lane, w);
        if (out) {
            const double r0 = b.v0 - s.v0, r1 = b.v1 - s.v1, r2 = b.v2 - s.v2;
            st3(y + 3 * a, xa.v0 + w * (D[0] * r0 + D[1] * r1 + D[2] * r2), xa.v1 + w * (D[3] * r0 + D[4] * r1 + D[5] * r2),
                xa.v2 + w * (D[6] * r0 + D[7] * r1 + D[8] * r2));
        }
    }
}
// bc[I] = sum over the members of aggregate I of b - A x (in member order, each residual rounded to VT)
template <class VT, bool L0>
__device__ __forceinline__ void cluster_restrict(const ClusterLevel<VT>& L, const int* indptr0, int nc, VT* bc, int gwarp, int nwarps) {
    constexpr int LANES = RowLanes<VT, L0>::value, PER_WARP = 32 / LANES;
    const int lane = threadIdx.x & (LANES - 1), sub = (threadIdx.x & 31) / LANES;
    for (int I = gwarp; I < nc; I += nwarps) {
        double s0 = 0, s1 = 0, s2 = 0;
        const int m0 = L.mptr[I], m1 = L.mptr[I + 1];
        for (int t = m0; t < m1; t += PER_WARP) {
            const bool valid = t + sub < m1;
            const int a = valid ? L.mem[t + sub] : 0;
            Vec3 b{0, 0, 0};
            if (valid) b = ld3cg(L.b + 3 * a);
            const Vec3 s = cluster_row<VT, L0, X_PLAIN>(L, indptr0, L.x, nullptr, a, valid, lane, 0.0);
            const double r0 = (double)(VT)(b.v0 - s.v0), r1 = (double)(VT)(b.v1 - s.v1), r2 = (double)(VT)(b.v2 - s.v2);
            const int cnt = m1 - t < PER_WARP ? m1 - t : PER_WARP;
#pragma unroll
            for (int k = 0; k < PER_WARP; k++) {
                const double a0 = __shfl_sync(0xffffffffu, r0, k * LANES), a1 = __shfl_sync(0xffffffffu, r1, k * LANES),
                             a2 = __shfl_sync(0xffffffffu, r2, k * LANES);
                if (k < cnt) { s0 += a0; s1 += a1; s2 += a2; }
            }
        }
        if ((threadIdx.x & 31) == 0) st3(bc + 3 * I, s0, s1, s2);
    }
}

template <class VT, bool L0>
__device__ __forceinline__ void cluster_down(const ClusterArgs<VT>& P, const ClusterLevel<VT>& L, int l, double w, int gwarp, int nwarps) {
    const int* ip = L0 ? P.indptr0 : nullptr;
    cluster_sweep<VT, L0, X_FIRST>(L, ip, nullptr, nullptr, L.x, w, gwarp, nwarps);
    cluster_sync();
    cluster_restrict<VT, L0>(L, ip, P.lev[l + 1].n, P.bc[l + 1], gwarp, nwarps);
    cluster_sync();
}
template <class VT, bool L0>
__device__ __forceinline__ void cluster_up(const ClusterArgs<VT>& P, const ClusterLevel<VT>& L, int l, double w, int gwarp, int nwarps) {
    const int* ip = L0 ? P.indptr0 : nullptr;
    cluster_sync();
    cluster_sweep<VT, L0, X_PROLONG>(L, ip, L.x, P.lev[l + 1].x, L.t, w, gwarp, nwarps);
    cluster_sync();
    cluster_sweep<VT, L0, X_PLAIN>(L, ip, L.t, nullptr, L.x, w, gwarp, nwarps);
}

// kAmgCoarseSweeps damped block-Jacobi sweeps from zero on the coarsest level, one thread per node (k_amg_coarsest's
// arithmetic).  A sweep is bound by the gathers of the iterate from shared memory: ~0.25 us for 150 nodes.
constexpr int kCoarsestRegBlocks = 8;   // blocks of a node kept in registers; further ones are read again each sweep
template <class VT>
__device__ __forceinline__ void coarsest_sweeps(const ClusterLevel<VT>& L, double w, double* xs) {
    const int i = threadIdx.x;
    const bool mine = i < L.n;
    const int q0 = mine ? L.bptr[i] : 0, deg = mine ? L.bptr[i + 1] - q0 : 0;
    double V[kCoarsestRegBlocks][9], D[9], b0 = 0, b1 = 0, b2 = 0, x0 = 0, x1 = 0, x2 = 0;
    int col[kCoarsestRegBlocks];
#pragma unroll
    for (int k = 0; k < kCoarsestRegBlocks; k++) {   // a missing block is a zero block of the node itself
        const bool has = k < deg;
        col[k] = has ? L.bcol[q0 + k] : (mine ? i : 0);
#pragma unroll
        for (int e = 0; e < 9; e++) V[k][e] = has ? (double)L.val[9 * (size_t)(q0 + k) + e] : 0.0;
    }
    if (mine) {
#pragma unroll
        for (int e = 0; e < 9; e++) D[e] = (double)L.dinv[9 * (size_t)i + e];
        const Vec3 b = ld3cg(L.b + 3 * i);
        b0 = b.v0; b1 = b.v1; b2 = b.v2;
        x0 = (double)(VT)(w * (D[0] * b0 + D[1] * b1 + D[2] * b2));
        x1 = (double)(VT)(w * (D[3] * b0 + D[4] * b1 + D[5] * b2));
        x2 = (double)(VT)(w * (D[6] * b0 + D[7] * b1 + D[8] * b2));
        xs[i] = x0; xs[kAmgCoarsest + i] = x1; xs[2 * kAmgCoarsest + i] = x2;
    }
    __syncthreads();
    for (int s = 1; s < kAmgCoarseSweeps; s++) {
        const double* x = xs + ((s & 1) ? 0 : 3 * kAmgCoarsest);
        double* y = xs + ((s & 1) ? 3 * kAmgCoarsest : 0);
        double r0 = b0, r1 = b1, r2 = b2;
#pragma unroll
        for (int k = 0; k < kCoarsestRegBlocks; k++) {
            const double a0 = x[col[k]], a1 = x[kAmgCoarsest + col[k]], a2 = x[2 * kAmgCoarsest + col[k]];
            r0 -= V[k][0] * a0 + V[k][1] * a1 + V[k][2] * a2;
            r1 -= V[k][3] * a0 + V[k][4] * a1 + V[k][5] * a2;
            r2 -= V[k][6] * a0 + V[k][7] * a1 + V[k][8] * a2;
        }
        for (int k = kCoarsestRegBlocks; k < deg; k++) {
            const int c = L.bcol[q0 + k];
            const VT* v = L.val + 9 * (size_t)(q0 + k);
            const double a0 = x[c], a1 = x[kAmgCoarsest + c], a2 = x[2 * kAmgCoarsest + c];
            r0 -= (double)v[0] * a0 + (double)v[1] * a1 + (double)v[2] * a2;
            r1 -= (double)v[3] * a0 + (double)v[4] * a1 + (double)v[5] * a2;
            r2 -= (double)v[6] * a0 + (double)v[7] * a1 + (double)v[8] * a2;
        }
        if (mine) {
            x0 = (double)(VT)(x0 + w * (D[0] * r0 + D[1] * r1 + D[2] * r2));
            x1 = (double)(VT)(x1 + w * (D[3] * r0 + D[4] * r1 + D[5] * r2));
            x2 = (double)(VT)(x2 + w * (D[6] * r0 + D[7] * r1 + D[8] * r2));
            y[i] = x0; y[kAmgCoarsest + i] = x1; y[2 * kAmgCoarsest + i] = x2;
        }
        __syncthreads();
    }
    if (mine) st3(L.x + 3 * i, x0, x1, x2);
}

// the operator's product, a warp per row
template <class VT>
__device__ __forceinline__ void coarsest_product(const ClusterLevel<VT>& L, const VT* __restrict__ op, double* bs, int gwarp, int nwarps) {
    const int m = 3 * L.n;
    for (int k = threadIdx.x; k < m; k += blockDim.x) bs[k] = (double)__ldcg(L.b + k);
    __syncthreads();
    for (int i = gwarp; i < m; i += nwarps) {
        const VT* row = op + (size_t)i * m;
        double s = 0;
#pragma unroll 8
        for (int k = threadIdx.x & 31; k < m; k += 32) s += (double)row[k] * bs[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) L.x[i] = (VT)s;
    }
}

// x <- V-cycle(b) on the levels lo .. of P, by the whole cluster.  OP: the coarsest solve by its operator, else by
// sweeps.  xs: 3 kAmgCoarsest (OP) or 6 kAmgCoarsest doubles of shared memory.  The last pass is not synchronised.
template <class VT, bool OP>
__device__ __forceinline__ void cluster_cycle(const ClusterArgs<VT>& P, const VT* b, VT* x, double w, double* xs) {
    static_assert(kAmgNu == 2, "the passes are two sweeps before and two after each coarse correction");
    const int gwarp = (cluster_rank() * blockDim.x + threadIdx.x) >> 5, nwarps = (cluster_ctas() * blockDim.x) >> 5;
    const int last = P.nlev - 1;
    auto level = [&](int l) {
        ClusterLevel<VT> L = P.lev[l];
        if (l == P.lo) { L.b = b; L.x = x; }
        return L;
    };
    for (int l = P.lo; l < last; l++) {
        const ClusterLevel<VT> L = level(l);
        if (l == 0) cluster_down<VT, true>(P, L, l, w, gwarp, nwarps);
        else cluster_down<VT, false>(P, L, l, w, gwarp, nwarps);
    }
    const ClusterLevel<VT> C = level(last);
    if (OP) coarsest_product<VT>(C, P.op, xs, gwarp, nwarps);
    else if (cluster_rank() == 0) coarsest_sweeps<VT>(C, w, xs);
    for (int l = last - 1; l >= P.lo; l--) {
        const ClusterLevel<VT> L = level(l);
        if (l == 0) cluster_up<VT, true>(P, L, l, w, gwarp, nwarps);
        else cluster_up<VT, false>(P, L, l, w, gwarp, nwarps);
    }
}

// the kernel's arguments for the levels lo .. of H (vals0: level-0 values)
template <class VT>
static inline ClusterArgs<VT> cluster_args(const BlockCSR& A, const AmgHost& H, int lo, const VT* vals0, const int* skip) {
    ClusterArgs<VT> P{};
    P.lo = lo; P.nlev = H.nlev; P.indptr0 = A.indptr; P.skip = skip; P.op = AmgBuf<VT>::coarsest(H);
    for (int l = lo; l < H.nlev; l++) {
        const AmgLevel& L = H.lev[l];
        ClusterLevel<VT>& D = P.lev[l];
        D.n = l ? L.n : A.nnodes;
        D.bptr = l ? L.bptr : A.bptr; D.bcol = l ? L.bcol : A.bcol;
        D.val = l ? AmgBuf<VT>::val(L) : vals0; D.dinv = l ? AmgBuf<VT>::dinv(L) : AmgBuf<VT>::dinv0(H);
        D.b = P.bc[l] = AmgBuf<VT>::b(L); D.x = AmgBuf<VT>::x(L); D.t = AmgBuf<VT>::t(L);
        if (l + 1 < H.nlev) { D.agg = H.link[l].agg; D.mptr = H.link[l].mptr; D.mem = H.link[l].mem; }
    }
    return P;
}
static inline cudaLaunchConfig_t cluster_config(int ctas, int threads, cudaLaunchAttribute* at, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(threads); cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = ctas; at->val.clusterDim.y = 1; at->val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cfg;
}
// whether one cluster of this size can be scheduled with the kernel
template <class K>
static inline bool cluster_schedulable(K kernel, int ctas, int threads, int smem = 0) {
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = cluster_config(ctas, threads, &at, nullptr);
    cfg.dynamicSmemBytes = smem;
    int fit = 0;
    const bool ok = (ctas <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                    cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();   // not schedulable
    return ok && fit > 0;
}

}  // namespace sw2
