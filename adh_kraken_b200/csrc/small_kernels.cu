// Krylov solves of small meshes (at most kClusterNodes nodes) as one kernel: a GMRES cycle, or a run of BiCGStab
// iterations, with its preconditioner (AMG V-cycle or multicolour block ILU(0)) in one thread-block cluster whose
// distributed shared memory holds the matrix, the hierarchy and the vectors.
//
// What bounds these solves is latency.  As launches an iteration on 1111 nodes took 45 us with the V-cycle in a cluster
// kernel of its own, and one kernel with its vectors in L2 was no faster (42 us): a pass that reads what other SMs have
// just written, and a barrier that waits for its stores to reach L2, cost ~4 us.  Here every CTA owns a run of nodes on every
// level (compact parts of the graph, small_order) and keeps their rows, smoother blocks and vector entries in shared
// memory, the rows of level 0 in registers.  Reading neighbours' entries from the owner's memory is no way out
// (3.7 cycles per scattered 8-byte load of an SM measured: 22 us an iteration); instead every CTA holds copies of the entries
// that its rows need from others (its halo), and whoever writes an entry also stores it into the copies.  A pass
// then reads its own memory alone, the cluster barrier after it waits for shared memory only (measured with 512 threads:
// 480 cycles, 1000 after 128 scattered stores to other CTAs, 1700 after one to global memory by every thread), and
// nothing but the right-hand side and the result goes through L2.  The measurements stand at small_solver_plan.
//
// Sums are per CTA, stored into every CTA's table and added by each in the same order after a barrier, so that all CTAs take
// the same decisions.  Vectors are held as doubles rounded to the Krylov precision VT wherever the kernels per step store
// them in it; products are accumulated in double.
#include <algorithm>
#include <cmath>
#include "amg_cluster.cuh"

namespace sw2 {

constexpr unsigned kElsewhere = 1u << 30;
constexpr int kSmallThreads = 512;
constexpr int kRowLanes = 4;                        // lanes per node
constexpr int kSmallCtas = 16;                      // a CTA owns at most 128 nodes: a node per kRowLanes threads
constexpr int kSlots = 8;                           // sums a BiCGStab iteration shares

// Byte offsets into the dynamic shared memory, the same in every CTA (a remote address is the owner's mapping of the
// local one); computed on the host (small_layout).
struct SmallLevelAt {
    int n, per;                                     // nodes, most nodes of a CTA
    int n0, own;                                    // this CTA's run (set in the kernel)
    unsigned val, D, b, x, t, r, node, ptr, col, dptr, dst, agg, mptr, mem;   // x, t: with the halo
};
struct SmallAt {
    int nlev;                                       // AMG levels (1: ILU only)
    SmallLevelAt lev[kAmgMaxLevels];
    unsigned lu, ludinv, lucol, luend, cptr, cnode;   // ILU: its slots with the lower neighbours first, nodes by colour
    unsigned op, table, part, vec, vlen, H, basis, scratch, h, hr, cs, sn, g;   // vec: the solver's own vectors, each vlen bytes
    int slots;                                      // table: [CTA][slots]
    SmallLevelPlan plan[kAmgMaxLevels];
    int kind, ncolors;                              // of the preconditioner, as SmallPrecond
    double w;
    const void* op_at;                              // the operator's rows in global memory
    int op_here, basis_here;                        // whether the operator's rows and the basis are in shared memory
    unsigned bytes;
};
template <class VT> struct SmallMatrix {
    int nnodes;
    const int *bptr, *bcol;
    const VT* vals;
};
template <class VT> struct SmallPrecond {
    int kind;                                       // 1: block ILU(0), 2: AMG
    ClusterArgs<VT> amg;                            // levels 0 ..
    const VT *lu, *dinv;                            // ILU factor in the CSR layout, inverted diagonal blocks
    const int* node_color;
};

extern __shared__ __align__(16) char small_sm[];
// The offsets stand in shared memory too: read as a kernel parameter by a function that is not inlined they are loads
// through L1, which every cluster barrier empties (3500 cycles a pass).
__shared__ SmallAt small_at;
template <class T> __device__ __forceinline__ T* at(unsigned off) { return reinterpret_cast<T*>(small_sm + off); }
// a double of CTA `rank`'s shared memory at byte offset off
__device__ __forceinline__ unsigned remote(unsigned off, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(small_sm) + off, r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ double ld_remote(unsigned a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void st_remote(unsigned a, double v) { asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
// entries of a node given as CTA << 16 | index there, with kElsewhere if that is another one
// component r of entry a of the vector at off, into the copies (push) or everywhere (put)
__device__ __forceinline__ void push(const SmallLevelAt& L, unsigned off, int a, int r, double v) {
    for (int q = at<int>(L.dptr)[a], q1 = at<int>(L.dptr)[a + 1]; q < q1; q++) {
        const unsigned d = at<unsigned>(L.dst)[q];
        st_remote(remote(off + 24 * (d & 0xffff) + 8 * r, d >> 16), v);
    }
}
__device__ __forceinline__ void put(const SmallLevelAt& L, unsigned off, int a, int r, double v) {
    at<double>(off)[3 * a + r] = v;
    push(L, off, a, r, v);
}
// f(node of this CTA, component) by the node's lanes; lanes without an entry repeat the last one with false
template <class F> __device__ __forceinline__ void own_entries(const SmallLevelAt& L, F f) {
    const int r = threadIdx.x & (kRowLanes - 1);
    for (int base = 0; base < L.own; base += kSmallThreads / kRowLanes) {
        const int a = base + threadIdx.x / kRowLanes;
        f(min(a, L.own - 1), min(r, 2), a < L.own && r < 3);
    }
}
template <class VT> __device__ __forceinline__ double rnd(double v) { return (double)(VT)v; }
// the kernels' first step
__device__ __forceinline__ void load_offsets(const SmallAt& P) {
    for (int i = threadIdx.x; i < (int)(sizeof(SmallAt) / 4); i += kSmallThreads) reinterpret_cast<int*>(&small_at)[i] = reinterpret_cast<const int*>(&P)[i];
    __syncthreads();
    if (threadIdx.x < P.nlev) {                     // run of CTA c: n c / ctas .. n (c + 1) / ctas
        SmallLevelAt& L = small_at.lev[threadIdx.x];
        L.n0 = L.n * cluster_rank() / kSmallCtas;
        L.own = L.n * (cluster_rank() + 1) / kSmallCtas - L.n0;
    }
    __syncthreads();
}

// the structure of this CTA's rows
__device__ __forceinline__ void load_rows(const SmallLevelAt& L, const SmallLevelPlan& G) {
    const int n0 = L.n0, own = L.own, q0 = G.ptr[n0], q1 = G.ptr[n0 + own], d0 = G.dptr[n0], d1 = G.dptr[n0 + own];
    for (int a = threadIdx.x; a <= own; a += kSmallThreads) {
        at<int>(L.ptr)[a] = G.ptr[n0 + a] - q0;
        at<int>(L.dptr)[a] = G.dptr[n0 + a] - d0;
        if (a < own) at<int>(L.node)[a] = G.node[n0 + a];
    }
    for (int q = threadIdx.x; q < q1 - q0; q += kSmallThreads) at<unsigned>(L.col)[q] = 24 * G.col[q0 + q];
    for (int q = threadIdx.x; q < d1 - d0; q += kSmallThreads) at<unsigned>(L.dst)[q] = G.dst[d0 + q];
    __syncthreads();
}
// block values of this CTA's rows, 8 lanes per node; slot: where each one goes, null for its own place
template <class VT>
__device__ __forceinline__ void load_values(const SmallLevelAt& L, const int* bptr, const VT* from, bool csr, unsigned to, const int* slot) {
    for (int a = threadIdx.x >> 3; a < L.own; a += kSmallThreads / 8) {
        const int s0 = bptr[at<int>(L.node)[a]], d0 = at<int>(L.ptr)[a], deg = at<int>(L.ptr)[a + 1] - d0;
        for (int k = threadIdx.x & 7; k < deg; k += 8) {
            const int d = slot ? slot[d0 + k] : d0 + k;
#pragma unroll
            for (int e = 0; e < 9; e++)
                at<double>(to)[9 * d + e] = (double)from[csr ? 9 * (size_t)s0 + (e / 3) * 3 * deg + 3 * k + e % 3 : 9 * (size_t)(s0 + k) + e];
        }
    }
}
template <class VT>
__device__ __forceinline__ void load_blocks(const SmallLevelAt& L, const VT* dinv, unsigned to) {
    for (int k = threadIdx.x; k < 9 * L.own; k += kSmallThreads) at<double>(to)[k] = (double)dinv[9 * (size_t)at<int>(L.node)[k / 9] + k % 9];
}
template <class VT>
__device__ void load_level(const SmallLevelAt& L, const SmallLevelAt& C, const SmallLevelPlan& G, const ClusterLevel<VT>& M, bool csr) {
    load_rows(L, G);
    load_values<VT>(L, M.bptr, M.val, csr, L.val, nullptr);
    load_blocks<VT>(L, M.dinv, L.D);
    for (int a = threadIdx.x; a < L.own; a += kSmallThreads) at<unsigned>(L.agg)[a] = G.agg[L.n0 + a];
    const int m0 = G.mptr[C.n0], m1 = G.mptr[C.n0 + C.own];
    for (int I = threadIdx.x; I <= C.own; I += kSmallThreads) at<int>(L.mptr)[I] = G.mptr[C.n0 + I] - m0;
    for (int k = threadIdx.x; k < m1 - m0; k += kSmallThreads) at<unsigned>(L.mem)[k] = G.mem[m0 + k];
}
// rows of level 0 alone (ILU), with the factor: of each node the slots of lower neighbours, then of the upper ones
template <class VT>
__device__ void load_ilu(const SmallAt& P, const SmallMatrix<VT>& A, const SmallPrecond<VT>& M) {
    const SmallLevelAt& L = P.lev[0];
    load_rows(L, P.plan[0]);
    load_values<VT>(L, A.bptr, A.vals, true, L.val, nullptr);
    load_blocks<VT>(L, M.dinv, P.ludinv);
    int *cptr = at<int>(P.cptr), *cnode = at<int>(P.cnode), *slot = at<int>(P.scratch);
    for (int c = threadIdx.x; c <= P.ncolors; c += kSmallThreads) {   // nodes by colour
        int k = 0;
        for (int a = 0; a < L.own; a++) k += M.node_color[at<int>(L.node)[a]] < c ? 1 : 0;
        cptr[c] = k;
        for (int a = 0; a < L.own; a++)
            if (M.node_color[at<int>(L.node)[a]] == c) cnode[k++] = a;
    }
    for (int a = threadIdx.x; a < L.own; a += kSmallThreads) {
        const int i = at<int>(L.node)[a], c = M.node_color[i], d0 = at<int>(L.ptr)[a], d1 = at<int>(L.ptr)[a + 1];
        const int* col = A.bcol + A.bptr[i] - d0;
        int lo = d0, up = d0;
        for (int d = d0; d < d1; d++) up += M.node_color[col[d]] < c ? 1 : 0;
        at<int>(P.luend)[2 * a] = up;
        for (int d = d0; d < d1; d++)
            if (M.node_color[col[d]] < c) { at<unsigned>(P.lucol)[lo] = at<unsigned>(L.col)[d]; slot[d] = lo++; }
            else if (M.node_color[col[d]] > c) { at<unsigned>(P.lucol)[up] = at<unsigned>(L.col)[d]; slot[d] = up++; }
        at<int>(P.luend)[2 * a + 1] = up;
        for (int d = d0; d < d1; d++)
            if (M.node_color[col[d]] == c) slot[d] = up++;   // the node itself: not read
    }
    __syncthreads();
    load_values<VT>(L, A.bptr, M.lu, true, P.lu, slot);
}

// component r of the row blocks' slots s0 .. s1 times the vector at off
__device__ __forceinline__ double row_sum(const double* val, const unsigned* col, int s0, int s1, int r, unsigned off) {
    const double* v = val + 9 * s0 + 3 * r;
    double y0 = 0, y1 = 0, y2 = 0;
#pragma unroll 4
    for (int s = s0; s < s1; s++, v += 9) {
        const double* x = at<double>(off + col[s]);
        y0 = fma(v[0], x[0], y0); y1 = fma(v[1], x[1], y1); y2 = fma(v[2], x[2], y2);
    }
    return y0 + y1 + y2;
}
__device__ __forceinline__ Vec3 of_node(double v) {   // the components that the node's lanes hold
    const int base = threadIdx.x & 31 & ~(kRowLanes - 1);
    return Vec3{__shfl_sync(0xffffffffu, v, base), __shfl_sync(0xffffffffu, v, base + 1), __shfl_sync(0xffffffffu, v, base + 2)};
}
__device__ __forceinline__ double dot3(const double* D, Vec3 v) { return fma(D[0], v.v0, fma(D[1], v.v1, D[2] * v.v2)); }
// f(node of this CTA, component, its row times the vector at off, whether it has one)
template <class F>
__device__ __forceinline__ void own_rows(const SmallLevelAt& L, unsigned off, F f) {
    own_entries(L, [&](int a, int r, bool valid) {
        const int* ptr = at<int>(L.ptr) + a;
        f(a, r, row_sum(at<double>(L.val), at<unsigned>(L.col), ptr[0], ptr[1], r, off), valid);
    });
}
// A thread's part of level 0: two slots of its node's row (further ones are read from shared memory) and component r of
// the smoother.  From shared memory alone a pass took 1200 cycles of its bandwidth, with them ~200.
struct Row0 {
    double v[2][9], D[3];
    unsigned x[2];                                  // the slots' entries; none: the node's own, times zero
    int a, r, more, end;                            // node, component (lane 3 repeats 2), further slots
    bool node, entry;                               // whether this thread has a node, and writes an entry
};
__device__ __forceinline__ Row0 load_row0(const SmallLevelAt& L, unsigned D) {
    Row0 R;
    const int lane = threadIdx.x & (kRowLanes - 1), a = threadIdx.x / kRowLanes;
    R.node = a < L.own;
    R.a = max(0, min(a, L.own - 1)); R.r = min(lane, 2);
    R.entry = R.node && lane < 3;
    const int s0 = R.node ? at<int>(L.ptr)[R.a] : 0;
    R.end = R.node ? at<int>(L.ptr)[R.a + 1] : 0;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int s = s0 + lane + kRowLanes * q;
        const bool has = s < R.end;
        R.x[q] = has ? at<unsigned>(L.col)[s] : 24u * R.a;
#pragma unroll
        for (int e = 0; e < 9; e++) R.v[q][e] = has ? at<double>(L.val)[9 * s + e] : 0.0;
    }
    R.more = s0 + lane + 2 * kRowLanes;
#pragma unroll
    for (int e = 0; e < 3; e++) R.D[e] = D && R.node ? at<double>(D)[9 * R.a + 3 * R.r + e] : 0.0;
    return R;
}
// the node's row times the vector at off, in all its lanes
__device__ __forceinline__ Vec3 row0(const SmallLevelAt& L, const Row0& R, unsigned off) {
    double y0 = 0, y1 = 0, y2 = 0;
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const double *x = at<double>(off + R.x[q]), x0 = x[0], x1 = x[1], x2 = x[2];
        y0 = fma(R.v[q][0], x0, y0); y1 = fma(R.v[q][3], x0, y1); y2 = fma(R.v[q][6], x0, y2);
        y0 = fma(R.v[q][1], x1, y0); y1 = fma(R.v[q][4], x1, y1); y2 = fma(R.v[q][7], x1, y2);
        y0 = fma(R.v[q][2], x2, y0); y1 = fma(R.v[q][5], x2, y1); y2 = fma(R.v[q][8], x2, y2);
    }
    for (int s = R.more; s < R.end; s += kRowLanes) {
        const double *x = at<double>(off + at<unsigned>(L.col)[s]), *v = at<double>(L.val) + 9 * s;
        y0 += dot3(v, Vec3{x[0], x[1], x[2]}); y1 += dot3(v + 3, Vec3{x[0], x[1], x[2]}); y2 += dot3(v + 6, Vec3{x[0], x[1], x[2]});
    }
    __syncwarp();
#pragma unroll
    for (int o = kRowLanes / 2; o > 0; o >>= 1) {
        y0 += __shfl_xor_sync(0xffffffffu, y0, o);
        y1 += __shfl_xor_sync(0xffffffffu, y1, o);
        y2 += __shfl_xor_sync(0xffffffffu, y2, o);
    }
    return Vec3{y0, y1, y2};
}
__device__ __forceinline__ double component(const Vec3& v, int r) { return r == 0 ? v.v0 : r == 1 ? v.v1 : v.v2; }
// level_pass of level 0
template <class VT, bool SMOOTH>
__device__ __forceinline__ void pass0(const SmallLevelAt& L, const Row0& R, unsigned b, unsigned x, unsigned y) {
    Vec3 s = row0(L, R, x);
    const double* bb = at<double>(b) + 3 * R.a;
    s = Vec3{bb[0] - s.v0, bb[1] - s.v1, bb[2] - s.v2};
    if (SMOOTH) {
        const double v = rnd<VT>(at<double>(x)[3 * R.a + R.r] + small_at.w * dot3(R.D, s));
        if (R.entry) put(L, y, R.a, R.r, v);
    } else if (R.entry) {
        at<double>(y)[3 * R.a + R.r] = rnd<VT>(component(s, R.r));
    }
    cluster_sync();
}
// y = x + w Dinv (b - A x), or with !SMOOTH y = b - A x; b, y: offsets of this CTA's entries
template <class VT, bool SMOOTH>
__device__ __noinline__ void level_pass(int l, unsigned b, unsigned x, unsigned y) {
    const SmallLevelAt& L = small_at.lev[l];
    own_rows(L, x, [&](int a, int r, double s, bool valid) {
        const double res = at<double>(b)[3 * a + r] - s;
        if (SMOOTH) {
            const double v = rnd<VT>(at<double>(x)[3 * a + r] + small_at.w * dot3(at<double>(L.D) + 9 * a + 3 * r, of_node(res)));
            if (valid) put(L, y, a, r, v);
        } else if (valid) {                         // the residual is read by the restriction alone
            at<double>(y)[3 * a + r] = rnd<VT>(res);
        }
    });
    cluster_sync();
}
// this CTA's run of a vector that every CTA holds whole, into the others: a warp per CTA
__device__ __forceinline__ void share_run(const SmallLevelAt& C, unsigned off) {
    __syncthreads();
    const int i0 = 3 * C.n0, cnt = 3 * C.own;
    for (int to = threadIdx.x >> 5; to < kSmallCtas; to += kSmallThreads / 32)
        if (to != cluster_rank())
            for (int i = threadIdx.x & 31; i < cnt; i += 32) st_remote(remote(off + 8 * (i0 + i), to), at<double>(off)[i0 + i]);
}
// y = M^-1 x on this CTA's entries at the offsets x and y (AMG: x is not y); every CTA's y is complete after it, its halo too
template <class VT>
__device__ __forceinline__ void small_apply(const Row0& R, unsigned x, unsigned y) {
    const SmallAt& P = small_at;
    const SmallLevelAt& L0 = P.lev[0];
    if (P.kind == 1) {
        for (int i = threadIdx.x; i < 3 * L0.own; i += kSmallThreads) at<double>(y)[i] = at<double>(x)[i];
        __syncthreads();
        const int r = min(threadIdx.x & (kRowLanes - 1), 2);
        for (int k = 0; k < 2 * P.ncolors; k++) {   // forward over the colours, then backward
            const bool fwd = k < P.ncolors;
            const int c = fwd ? k : 2 * P.ncolors - 1 - k, c0 = at<int>(P.cptr)[c], c1 = at<int>(P.cptr)[c + 1];
            for (int base = c0; base < c1; base += kSmallThreads / kRowLanes) {
                if (base + (int)(threadIdx.x & ~31u) / kRowLanes >= c1) break;   // (a whole warp)
                const int q = base + threadIdx.x / kRowLanes, a = at<int>(P.cnode)[min(q, c1 - 1)];
                const int* end = at<int>(P.luend) + 2 * a;
                const double s = fwd ? row_sum(at<double>(P.lu), at<unsigned>(P.lucol), at<int>(L0.ptr)[a], end[0], r, y)
                                     : row_sum(at<double>(P.lu), at<unsigned>(P.lucol), end[0], end[1], r, y);
                double v = at<double>(y)[3 * a + r] - s;
                if (!fwd) v = dot3(at<double>(P.ludinv) + 9 * a + 3 * r, of_node(v));
                __syncwarp();
                if (q < c1 && (threadIdx.x & (kRowLanes - 1)) < 3) put(L0, y, a, r, rnd<VT>(v));
            }
            cluster_sync();
        }
        return;
    }
    const int last = P.nlev - 1;
    auto first_sweep = [&](const SmallLevelAt& L, unsigned b) {   // t = w Dinv b
        own_entries(L, [&](int a, int r, bool valid) {
            const double* v = at<double>(b) + 3 * a;
            if (valid) put(L, L.t, a, r, rnd<VT>(P.w * dot3(at<double>(L.D) + 9 * a + 3 * r, Vec3{v[0], v[1], v[2]})));
        });
        cluster_sync();
    };
    if (R.entry) {                                  // first_sweep of level 0
        const double* v = at<double>(x) + 3 * R.a;
        put(L0, L0.t, R.a, R.r, rnd<VT>(P.w * dot3(R.D, Vec3{v[0], v[1], v[2]})));
    }
    cluster_sync();
    for (int l = 0; l < last; l++) {
        const SmallLevelAt &L = P.lev[l], &C = P.lev[l + 1];
        const unsigned b = l ? L.b : x, xl = l ? L.x : y;
        if (l == 0) {
            pass0<VT, true>(L, R, b, L.t, xl);
            pass0<VT, false>(L, R, b, xl, L.r);
        } else {
            level_pass<VT, true>(l, b, L.t, xl);
            level_pass<VT, false>(l, b, xl, L.r);
        }
        // restriction, 16 lanes per coarse node: 4 members times the components
        const int r = min(threadIdx.x & 3, 2), sub = threadIdx.x >> 2 & 3;
        const int* mptr = at<int>(L.mptr);
        for (int base = 0; base < C.own; base += kSmallThreads / 16) {
            const int I = base + (threadIdx.x >> 4), J = min(I, C.own - 1), k1 = mptr[J + 1];
            double s = 0;
#pragma unroll 2
            for (int k = mptr[J] + sub; k < k1; k += 4) {
                const unsigned m = at<unsigned>(L.mem)[k], o = L.r + 24 * (m & 0xffff) + 8 * r;
                s += m & kElsewhere ? ld_remote(remote(o, m >> 16 & 0xff)) : *at<double>(o);
            }
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            if (I < C.own && (threadIdx.x & 15) < 3) at<double>(C.b)[3 * (I + (l + 1 == last ? C.n0 : 0)) + r] = rnd<VT>(s);
        }
        if (l + 1 == last) {
            share_run(C, C.b);
            cluster_sync();
        } else {
            __syncthreads();
            first_sweep(C, C.b);
        }
    }
    {   // the coarsest level by its operator, two rows of this CTA's nodes to a warp
        const SmallLevelAt& C = P.lev[last];
        const int m = 3 * C.n, rows = 3 * C.own, lane = threadIdx.x & 31;
        const double* cb = at<double>(C.b);
        if (!P.op_here) {                           // (C.t) its columns keep the level's own order
            for (int k = threadIdx.x; k < m; k += kSmallThreads) at<double>(C.t)[3 * at<int>(C.node)[k / 3] + k % 3] = cb[k];
            __syncthreads();
            cb = at<double>(C.t);
        }
        for (int i = threadIdx.x >> 5; i < rows; i += kSmallThreads / 16) {
            const int i2 = min(i + kSmallThreads / 32, rows - 1);
            double s = 0, s2 = 0;
            if (P.op_here) {
                const VT *row = at<VT>(P.op) + (size_t)i * m, *row2 = at<VT>(P.op) + (size_t)i2 * m;
#pragma unroll 4
                for (int k = lane; k < m; k += 32) { s = fma((double)row[k], cb[k], s); s2 = fma((double)row2[k], cb[k], s2); }
            } else {
                auto from = [&](int r) { return static_cast<const VT*>(P.op_at) + (size_t)(3 * at<int>(C.node)[C.n0 + r / 3] + r % 3) * m; };
                const VT *row = from(i), *row2 = from(i2);
#pragma unroll 8
                for (int k = lane; k < m; k += 32) { s = fma((double)row[k], cb[k], s); s2 = fma((double)row2[k], cb[k], s2); }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                s += __shfl_xor_sync(0xffffffffu, s, o);
                s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            }
            if (lane == 0) {
                double* xc = at<double>(C.x) + 3 * C.n0;
                xc[i] = rnd<VT>(s);
                xc[i2] = rnd<VT>(s2);               // (the last row more than once, with the same value)
            }
        }
        share_run(C, C.x);
        cluster_sync();
    }
    for (int l = last - 1; l >= 0; l--) {
        const SmallLevelAt &L = P.lev[l], &C = P.lev[l + 1];
        const unsigned b = l ? L.b : x, xl = l ? L.x : y;
        own_entries(L, [&](int a, int r, bool valid) {
            const unsigned g = at<unsigned>(L.agg)[a], o = C.x + 24 * (g & 0xffff) + 8 * r;
            const double e = g & kElsewhere ? ld_remote(remote(o, g >> 16 & 0xff)) : *at<double>(o);
            if (valid) put(L, xl, a, r, rnd<VT>(at<double>(xl)[3 * a + r] + e));
        });
        cluster_sync();
        if (l == 0) {
            pass0<VT, true>(L, R, b, xl, L.t);
            pass0<VT, true>(L, R, b, L.t, xl);
        } else {
            level_pass<VT, true>(l, b, xl, L.t);
            level_pass<VT, true>(l, b, L.t, xl);
        }
    }
}
template <class VT>
__device__ void load_solver(const SmallAt& from, const SmallMatrix<VT>& A, const SmallPrecond<VT>& M) {
    load_offsets(from);
    const SmallAt& P = small_at;
    if (M.kind == 1) {
        load_ilu<VT>(P, A, M);
    } else {
        for (int l = 0; l < P.nlev - 1; l++) load_level<VT>(P.lev[l], P.lev[l + 1], P.plan[l], M.amg.lev[l], l == 0);
        const SmallLevelAt& C = P.lev[P.nlev - 1];
        const int m = 3 * C.n;
        const int* node = at<int>(C.node);
        for (int i = threadIdx.x; i < C.n; i += kSmallThreads) at<int>(C.node)[i] = P.plan[P.nlev - 1].node[i];
        __syncthreads();
        if (P.op_here)                              // rows and columns in the cluster's order
            for (int r = threadIdx.x >> 5; r < 3 * C.own; r += kSmallThreads / 32) {
                const VT* from = M.amg.op + (size_t)(3 * node[C.n0 + r / 3] + r % 3) * m;
                for (int k = threadIdx.x & 31; k < m; k += 32) at<VT>(P.op)[(size_t)r * m + k] = from[3 * node[k / 3] + k % 3];
            }
    }
}

// A CTA's share of a sum or maximum goes into every CTA's table; after the next cluster_sync every thread of every CTA
// gets the same result from table_sum / table_max (called by whole half warps, one slot each).
template <bool MAX>
__device__ __forceinline__ void publish(const SmallAt& P, int slot, double v) {
    double* sh = at<double>(P.part);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, v, o);
        v = MAX ? fmax(v, u) : v + u;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = threadIdx.x < kSmallThreads / 32 ? sh[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double u = __shfl_xor_sync(0xffffffffu, v, o);
            v = MAX ? fmax(v, u) : v + u;
        }
        if (threadIdx.x < kSmallCtas) st_remote(remote(P.table + 8 * (cluster_rank() * P.slots + slot), threadIdx.x), v);
    }
}
template <bool MAX>
__device__ __forceinline__ double table_total(const SmallAt& P, int slot) {
    const int k = threadIdx.x & 15;
    double v = k < kSmallCtas ? at<double>(P.table)[k * P.slots + slot] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, v, o);
        v = MAX ? fmax(v, u) : v + u;
    }
    return v;
}
__device__ __forceinline__ void publish_sum(const SmallAt& P, int slot, double v) { publish<false>(P, slot, v); }
__device__ __forceinline__ void publish_max(const SmallAt& P, int slot, double v) { publish<true>(P, slot, v); }
__device__ __forceinline__ double table_sum(const SmallAt& P, int slot) { return table_total<false>(P, slot); }
__device__ __forceinline__ double table_max(const SmallAt& P, int slot) { return table_total<true>(P, slot); }

// ---------------------------------------------------------------- one GMRES cycle (gmres_kernels.cu's steps)
template <class VT> struct SmallGmres {
    SmallAt at;
    SmallMatrix<VT> A;
    SmallPrecond<VT> P;
    VT* Vb; size_t ld;                              // basis in global memory, where it does not fit here
    const VT* rhs;
    VT* out;
    const double* rw;
    GmresDev G;
    int m;
};
template <class VT>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_gmres(const __grid_constant__ SmallGmres<VT> S) {
    __shared__ double s_hn;
    __shared__ int s_stop, s_cols, s_status, s_steps;   // s_stop: the same in every CTA
    const SmallAt& P = small_at;
    const GmresDev& G = S.G;
    load_solver<VT>(S.at, S.A, S.P);
    const int rank = cluster_rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i0 = 3 * P.lev[0].n0, cnt = 3 * P.lev[0].own, slot = S.m;   // slot of the norms
    auto id = [&](int i) { return 3 * at<int>(P.lev[0].node)[i / 3] + i % 3; };
    const unsigned own_len = 24u * P.lev[0].per, z_at = P.vec, v_at = z_at + P.vlen, w_at = v_at + own_len, rw_at = w_at + own_len;
    double *v = at<double>(v_at), *w = at<double>(w_at), *rw = at<double>(rw_at);
    double *h = at<double>(P.h), *hr = at<double>(P.hr), *cs = at<double>(P.cs), *sn = at<double>(P.sn), *g = at<double>(P.g);
    VT* basis = P.basis_here ? at<VT>(P.basis) : S.Vb + i0;   // vector k at k * ldb
    const size_t ldb = P.basis_here ? (size_t)3 * P.lev[0].per : S.ld;
    
    double ss = 0;
    for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
        rw[i] = S.rw[id(i)];
        w[i] = (double)S.rhs[id(i)] * rw[i];
        ss += w[i] * w[i];
    }
    cluster_sync();                                 // every CTA runs, and its shared memory is set up
    publish_sum(P, slot, ss);
    cluster_sync();
    const double beta = sqrt(table_sum(P, slot)), target = G.scal[3] * beta;
    if (threadIdx.x == 0) {
        g[0] = beta; s_cols = 0; s_steps = 0; s_status = isfinite(beta) ? 0 : 2;
        s_stop = (beta > 0.0 && isfinite(beta)) ? 0 : 1;
        if (rank == 0) { G.scal[0] = beta; G.scal[1] = target; G.scal[2] = beta; }
    }
    __syncthreads();
    if (!s_stop) {
        const double inv = 1.0 / beta;
        for (int i = threadIdx.x; i < cnt; i += kSmallThreads) { v[i] = rnd<VT>(w[i] * inv); basis[i] = (VT)v[i]; }
    }
    __syncthreads();
    const Row0 R = load_row0(P.lev[0], S.P.kind == 2 ? P.lev[0].D : 0u);
    for (int j = 0;; j++) {
        const bool last = j == S.m || s_stop;       // the cycle's end: v = V y
        if (last) {
            const int k = s_cols;
            cluster_sync();                         // all of H is there
            if (warp == 0) {                        // y = H^-1 g, column by column, by every CTA for itself
                for (int t = lane; t < k; t += 32) h[t] = g[t];
                __syncwarp();
                for (int i = k - 1; i >= 0; i--) {
                    const unsigned col = remote(P.H + 8 * (i >> 4) * S.m, (i & (kSmallCtas - 1)));
                    const double d = ld_remote(col + 8 * i), yi = d != 0.0 ? h[i] / d : 0.0;
                    for (int t = lane; t < i; t += 32) h[t] -= ld_remote(col + 8 * t) * yi;
                    __syncwarp();
                    if (lane == 0) h[i] = yi;
                    __syncwarp();
                }
                if (rank == 0 && lane == 0) {
                    if (s_steps > 0) { G.scal[2] = fabs(g[s_steps]); G.scal[4] = s_hn; }
                    G.state[0] = 0; G.state[1] = k; G.state[2] = s_status;
                }
            }
            __syncthreads();
            for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
                double t = 0;
#pragma unroll 8
                for (int q = 0; q < k; q++) t = fma(h[q], (double)basis[(size_t)q * ldb + i], t);
                v[i] = rnd<VT>(t);
            }
        }
        __syncthreads();                            // v is complete in this CTA
        small_apply<VT>(R, v_at, z_at);
        if (last) break;
        {   // w = rw o (A z), rounded as the separate passes round it
            const Vec3 t = row0(P.lev[0], R, z_at);
            if (R.entry) w[3 * R.a + R.r] = rnd<VT>(rnd<VT>(component(t, R.r)) * rw[3 * R.a + R.r]);
        }
        __syncthreads();
        for (int k = warp; k <= j; k += kSmallThreads / 32) {   // this CTA's share of v_k . w
            const VT* vk = basis + (size_t)k * ldb;
            double t = 0;
#pragma unroll 4
            for (int i = lane; i < cnt; i += 32) t = fma((double)vk[i], w[i], t);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane < kSmallCtas) st_remote(remote(P.table + 8 * (rank * P.slots + k), lane), t);
        }
        cluster_sync();
        for (int base = 2 * warp; base <= j; base += kSmallThreads / 16) {
            const int k = base + (lane >> 4);
            const double t = table_sum(P, min(k, j));
            if ((lane & 15) == 0 && k <= j) h[k] = t;
        }
        __syncthreads();
        if (threadIdx.x == kSmallThreads - 32) {    // meanwhile every CTA turns the column by the earlier rotations
            double a = h[0];
#pragma unroll 4
            for (int k = 0; k < j; k++) {
                const double b = h[k + 1];
                hr[k] = cs[k] * a + sn[k] * b;
                a = -sn[k] * a + cs[k] * b;
            }
            hr[j] = a;
        }
        ss = 0;
        for (int i = threadIdx.x; i < cnt; i += kSmallThreads) {
            double x = w[i];
#pragma unroll 8
            for (int k = 0; k <= j; k++) x = fma(-h[k], (double)basis[(size_t)k * ldb + i], x);
            x = rnd<VT>(x);
            w[i] = x;
            ss += x * x;
        }
        publish_sum(P, slot, ss);
        cluster_sync();
        const double hn = sqrt(table_sum(P, slot)), inv = 1.0 / hn;
        if (threadIdx.x == 0) {
            const double a = hr[j], b = hn, rr = hypot(a, b);
            const double c = rr > 0.0 ? a / rr : 1.0, s = rr > 0.0 ? b / rr : 0.0;
            cs[j] = c; sn[j] = s; hr[j] = rr;
            const double gj = g[j], gn = -s * gj;
            g[j] = c * gj; g[j + 1] = gn;
            s_cols = j + 1;
            if (!isfinite(rr) || !isfinite(hn)) { s_status = 2; s_stop = 1; s_cols = j; }
            else if (rr == 0.0) { s_status = 1; s_stop = 1; s_cols = j; }   // breakdown: drop column j
            else if (!(fabs(gn) > target) || hn == 0.0) s_stop = 1;
            s_hn = hn; s_steps = j + 1;
        }
        __syncthreads();
        if (rank == (j & (kSmallCtas - 1)))             // the columns of H go round the CTAs
            for (int k = threadIdx.x; k <= j; k += kSmallThreads) at<double>(P.H)[(j >> 4) * S.m + k] = hr[k];
        if (!s_stop && j + 1 < S.m) {
            VT* next = basis + (size_t)(j + 1) * ldb;
            for (int i = threadIdx.x; i < cnt; i += kSmallThreads) { v[i] = rnd<VT>(w[i] * inv); next[i] = (VT)v[i]; }
        }
    }
    for (int i = threadIdx.x; i < cnt; i += kSmallThreads) S.out[id(i)] = (VT)at<double>(z_at)[i];
    cluster_sync();
}

// ---------------------------------------------------------------- BiCGStab (la_kernels.cu's recurrences)
template <class VT> struct SmallBicg {
    SmallAt at;
    SmallMatrix<VT> A;
    SmallPrecond<VT> P;
    KrylovVecs<VT> V;
    KrylovScalars* S;
    int right, first, iterations;                   // first: start a solve; iterations of this launch
};
template <class VT>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_bicg(const __grid_constant__ SmallBicg<VT> B) {
    const SmallAt& P = small_at;
    const KrylovVecs<VT>& V = B.V;
    load_solver<VT>(B.at, B.A, B.P);
    const int rank = cluster_rank();
    const int cnt = 3 * P.lev[0].own;
    auto id = [&](int i) { return 3 * at<int>(P.lev[0].node)[i / 3] + i % 3; };
    auto off = [&](int k) { return P.vec + k * P.vlen; };
    const unsigned x_at = off(0), r_at = off(1), p_at = off(2), q_at = off(3), s_at = off(4), Ap_at = off(5), As_at = off(6), z_at = off(7), b_at = off(8);
    double *x = at<double>(x_at), *r = at<double>(r_at), *p = at<double>(p_at), *q = at<double>(q_at), *sv = at<double>(s_at),
           *Ap = at<double>(Ap_at), *As = at<double>(As_at), *b = at<double>(b_at);
    auto own = [&](auto f) { for (int i = threadIdx.x; i < cnt; i += kSmallThreads) f(i); };
    
    own([&](int i) {
        const int g = id(i);
        b[i] = (double)V.b[g];
        if (!B.first) {
            x[i] = (double)V.x[g]; r[i] = (double)V.r[g]; p[i] = (double)V.p[g]; q[i] = (double)V.q[g];
            Ap[i] = (double)V.Ap[g];
        }
    });
    cluster_sync();                                 // every CTA's shared memory is set up
    // a vector that apply takes, after its entries are written
    auto ready = [&](unsigned src) {
        __syncthreads();
        if (B.right) return;
        own_entries(P.lev[0], [&](int a, int r, bool valid) { if (valid) push(P.lev[0], src, a, r, at<double>(src)[3 * a + r]); });
        cluster_sync();
    };
    const Row0 R = load_row0(P.lev[0], B.P.kind == 2 ? P.lev[0].D : 0u);
    auto times_A = [&](unsigned src, unsigned dst) {   // complete in this CTA
        const Vec3 t = row0(P.lev[0], R, src);
        if (R.entry) at<double>(dst)[3 * R.a + R.r] = rnd<VT>(component(t, R.r));
        __syncthreads();
    };
    KrylovScalars s = *B.S;                         // the same in every thread
    // Every phase applies A M^-1 (right) or M^-1 A (left) to a vector: x of a start, p and s of an iteration.  A left
    // preconditioned start first takes M^-1 b.
    enum { RHS, START, P_HALF, S_HALF };
    int phase = !B.first ? P_HALF : B.right ? START : RHS, k = 0;
    if (B.first) own([&](int i) { x[i] = b[i]; });
    while (phase < P_HALF || (k < B.iterations && !s.done)) {
        const unsigned src = phase == START ? x_at : phase == P_HALF ? p_at : s_at;
        const unsigned dst = phase == START ? r_at : phase == P_HALF ? Ap_at : As_at;
        if (phase != RHS) {
            ready(src);
            if (!B.right) times_A(src, dst);
        }
        const unsigned to = B.right ? z_at : phase == RHS ? b_at : dst;
        small_apply<VT>(R, B.right ? src : to, to);
        if (B.right) times_A(z_at, dst);
        if (phase == RHS) {
            own([&](int i) { x[i] = b[i]; });
            phase = START;
        } else if (phase == START) {
            double rmax = 0, bmax = 0, rr = 0;
            own([&](int i) {
                const VT t = (VT)b[i] + (VT)-1 * (VT)r[i];
                r[i] = q[i] = p[i] = (double)t; Ap[i] = 0;
                rmax = fmax(rmax, fabs((double)t)); bmax = fmax(bmax, fabs(b[i]));
                rr += (double)t * (double)t;
            });
            publish_max(P, 0, rmax); publish_max(P, 1, bmax); publish_sum(P, 2, rr);
            cluster_sync();
            s.rnorm = table_max(P, 0); s.bnorm = table_max(P, 1); s.rho = table_sum(P, 2);
            s.rhop = 1.0; s.alpha = 1.0; s.omega = 1.0; s.beta = 0.0; s.it = 0; s.status = 0;
            s.done = (s.rnorm > (s.tol + s.bnorm * s.rtol)) ? 0 : 1;
            if (!isfinite(s.rnorm) || !isfinite(s.rho)) { s.status = 2; s.done = 1; }
            phase = P_HALF;
        } else if (phase == P_HALF) {
            double qa = 0;
            own([&](int i) { qa += q[i] * Ap[i]; });
            publish_sum(P, 3, qa);
            cluster_sync();
            s.gamma = table_sum(P, 3);
            if (s.gamma == 0.0 || !isfinite(s.gamma)) { s.status = 1; s.done = 1; break; }
            s.alpha = s.rho / s.gamma;
            const VT alpha = (VT)s.alpha;
            own([&](int i) { sv[i] = (double)((VT)r[i] + -alpha * (VT)Ap[i]); });
            phase = S_HALF;
        } else {
            double ss = 0, aa = 0, aq = 0;
            own([&](int i) { ss += As[i] * sv[i]; aa += As[i] * As[i]; aq += As[i] * q[i]; });
            publish_sum(P, 4, ss); publish_sum(P, 5, aa); publish_sum(P, 6, aq);
            cluster_sync();
            const double a = table_sum(P, 4), bb = table_sum(P, 5), c = table_sum(P, 6);
            if (bb == 0.0) { s.omega = 0.0; s.status = 3; }
            else {
                const double om = a / bb;
                const double rho_new = -1.0 * om * c;
                const double beta = (rho_new * s.alpha) / (s.rho * om);
                if (om == 0.0 || rho_new == 0.0 || !isfinite(om) || !isfinite(beta)) {
                    s.omega = 0.0; s.status = 5;    // breakdown: take the half step x += alpha p, then stop
                } else {
                    s.omega = om; s.rhop = s.rho; s.rho = rho_new; s.beta = beta;
                }
            }
            const bool s_zero = s.status == 3 || s.status == 5;
            const VT alpha = (VT)s.alpha, omega = (VT)s.omega, beta = (VT)s.beta;
            double rmax = 0;
            own([&](int i) {
                VT xi = (VT)x[i] + alpha * (VT)p[i];
                VT ri;
                if (s_zero) {
                    ri = (VT)sv[i];
                } else {
                    xi = xi + omega * (VT)sv[i];
                    ri = (VT)sv[i] + -omega * (VT)As[i];
                    VT pi = (VT)p[i] + -omega * (VT)Ap[i];
                    pi = pi * beta;
                    p[i] = (double)(pi + (VT)1 * ri);
                }
                x[i] = (double)xi; r[i] = (double)ri;
                rmax = fmax(rmax, fabs((double)ri));
            });
            publish_max(P, 7, rmax);
            cluster_sync();
            s.rnorm = table_max(P, 7);
            s.it += 1;
            if (s.status == 3) { s.status = 0; s.done = 1; }
            if (s.status == 5) { s.status = 1; s.done = 1; }
            if (!(s.rnorm > (s.tol + s.bnorm * s.rtol)) || s.it >= s.max_it) s.done = 1;
            if (!isfinite(s.rnorm)) { s.status = 2; s.done = 1; }
            phase = P_HALF;
            k++;
        }
    }
    own([&](int i) {
        const int g = id(i);
        V.x[g] = (VT)x[i]; V.r[g] = (VT)r[i]; V.p[g] = (VT)p[i]; V.q[g] = (VT)q[i]; V.Ap[g] = (VT)Ap[i];
        V.b[g] = (VT)b[i];
    });
    cluster_sync();                                 // no CTA leaves while another reads its memory, or its scalars
    if (rank == 0 && threadIdx.x == 0) *B.S = s;
}

// ---------------------------------------------------------------- host side
template <class VT>
static SmallPrecond<VT> small_precond(const BlockCSR& A, const PrecondOp<VT>& op) {
    SmallPrecond<VT> P{};
    P.kind = op.kind;
    if (op.kind == 2) {
        P.amg = cluster_args<VT>(A, *op.amg, 0, op.vals, nullptr);
    } else {
        P.lu = op.lu; P.dinv = op.dinv; P.node_color = op.ilu->view.node_color;
    }
    return P;
}
// Places everything in shared memory; bytes > limit: it does not fit.  basis: the GMRES restart
// length, 0 for BiCGStab.
template <class VT>
static SmallAt small_layout(const BlockCSR& A, const PrecondOp<VT>& op, const SmallPlan& S, int basis) {
    SmallAt P{};
    unsigned top = 0;
    auto take = [&](size_t bytes) { const unsigned o = top; top += (unsigned)((bytes + 15) & ~(size_t)15); return o; };
    P.nlev = op.kind == 2 ? op.amg->nlev : 1;
    P.kind = op.kind; P.w = kAmgOmega;
    if (op.kind == 1) P.ncolors = op.ilu->ncolors;
    if (op.kind == 2) P.op_at = sizeof(VT) == 8 ? (const void*)op.amg->cl.op64 : (const void*)op.amg->cl.op32;
    for (int l = 0; l < P.nlev; l++) {
        SmallLevelAt& L = P.lev[l];
        L.n = l ? op.amg->lev[l].n : A.nnodes;
        P.plan[l] = S.lev[l];
        L.per = (L.n + S.ctas - 1) / S.ctas;
        const size_t whole = 24 * (size_t)(L.per + P.plan[l].halo);
        const bool coarsest = l > 0 && l == P.nlev - 1;   // every CTA holds all of it, and none has its rows
        if (l > 0) { L.b = take(24 * (size_t)(coarsest ? L.n : L.per)); L.x = take(coarsest ? 24 * (size_t)L.n : whole); }
        L.node = take(4 * (size_t)(coarsest ? L.n : L.per));
        if (coarsest) break;
        const int slots = P.plan[l].slots;
        L.val = take(72 * (size_t)slots); L.col = take(4 * (size_t)slots); L.ptr = take(4 * (size_t)(L.per + 1));
        L.dptr = take(4 * (size_t)(L.per + 1)); L.dst = take(4 * (size_t)P.plan[l].push);
        if (op.kind != 2) break;
        L.D = take(72 * (size_t)L.per); L.t = take(whole); L.r = take(24 * (size_t)L.per);
        const int nc = op.amg->lev[l + 1].n;
        L.agg = take(4 * (size_t)L.per); L.mptr = take(4 * (size_t)((nc + S.ctas - 1) / S.ctas + 1));
        L.mem = take(4 * (size_t)P.plan[l].members);
    }
    if (op.kind == 1) {
        const int per = P.lev[0].per, slots = P.plan[0].slots;
        P.lu = take(72 * (size_t)slots); P.ludinv = take(72 * (size_t)per); P.lucol = take(4 * (size_t)slots); P.luend = take(8 * (size_t)per);
        P.cptr = take(4 * (size_t)(P.ncolors + 1)); P.cnode = take(4 * (size_t)per);
        P.scratch = take(4 * (size_t)slots);        // while the factor is loaded
    }
    P.slots = basis ? basis + 1 : kSlots;
    P.table = take(8 * (size_t)P.slots * S.ctas); P.part = take(8 * (kSmallThreads / 32));
    P.vlen = (unsigned)(24 * (P.lev[0].per + P.plan[0].halo));
    P.vec = take(basis ? P.vlen + 72 * (size_t)P.lev[0].per : P.vlen * (size_t)9);   // GMRES: z, and three without a halo
    const size_t m = basis;
    if (basis) {
        P.H = take(8 * m * ((m + S.ctas - 1) / S.ctas));
        P.h = take(8 * m); P.hr = take(8 * (m + 1)); P.cs = take(8 * m); P.sn = take(8 * m); P.g = take(8 * (m + 1));
    }
    const unsigned limit = (unsigned)S.smem;
    if (op.kind == 2) {                             // the operator's rows, if they fit; read through L2 otherwise
        const SmallLevelAt& C = P.lev[P.nlev - 1];
        const size_t bytes = 9 * (size_t)C.per * C.n * sizeof(VT);
        if (top + bytes <= limit) { P.op = take(bytes); P.op_here = 1; }
        else P.lev[P.nlev - 1].t = take(24 * (size_t)C.n);
    }
    if (basis) {
        const size_t bytes = 3 * (size_t)P.lev[0].per * basis * sizeof(VT);
        if (top + bytes <= limit) { P.basis = take(bytes); P.basis_here = 1; }
    }
    P.bytes = top;
    return P;
}
// How a level's rows lie in a cluster of `ctas` CTAs: CTA c owns the places n c / ctas .. n (c + 1) / ctas of an order.
static int run_start(int n, int c, int ctas) { return (int)((long)n * c / ctas); }
static int run_owner(int n, int i, int ctas) { return (int)(((long)(i + 1) * ctas - 1) / n); }
// An order of the nodes in which these runs are compact: the graph halved again and again, each time at the middle of a
// breadth-first order from a far node.
std::vector<int> small_order(const std::vector<int>& bptr, const std::vector<int>& bcol, int n, int ctas) {
    std::vector<int> order(n), part(n, 0), seen(n, 0);
    for (int i = 0; i < n; i++) order[i] = i;
    int stamp = 0, parts = 0;
    auto breadth_first = [&](std::vector<int>& nodes, int first) {
        std::vector<int> out;
        const int p = part[nodes[0]];
        stamp++;
        auto visit = [&](int i) { if (part[i] == p && seen[i] != stamp) { seen[i] = stamp; out.push_back(i); } };
        visit(first);
        for (size_t k = 0, rest = 0; out.size() < nodes.size(); k++) {
            while (k == out.size()) visit(nodes[rest++]);   // the next component
            for (int q = bptr[out[k]]; q < bptr[out[k] + 1]; q++) visit(bcol[q]);
        }
        nodes = out;
    };
    for (int step = ctas; step > 1; step /= 2)
        for (int c = 0; c < ctas; c += step) {
            const int i0 = run_start(n, c, ctas), mid = run_start(n, c + step / 2, ctas), i1 = run_start(n, c + step, ctas);
            if (i1 == i0) continue;
            std::vector<int> nodes(order.begin() + i0, order.begin() + i1);
            breadth_first(nodes, nodes[0]);
            for (int k = 0; k < 2; k++) breadth_first(nodes, nodes.back());
            std::copy(nodes.begin(), nodes.end(), order.begin() + i0);
            parts++;
            for (int i = mid; i < i1; i++) part[order[i]] = parts;
        }
    return order;
}
// and of the coarser level's, by the mean place of their members
std::vector<int> small_coarse_order(const std::vector<int>& fine, const std::vector<int>& agg, int nc) {
    std::vector<double> place(nc, 0), members(nc, 0);
    for (size_t k = 0; k < fine.size(); k++) { place[agg[fine[k]]] += (double)k; members[agg[fine[k]]] += 1; }
    std::vector<int> order(nc);
    for (int i = 0; i < nc; i++) { order[i] = i; place[i] /= std::max(1.0, members[i]); }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return place[a] < place[b]; });
    return order;
}
static std::vector<int> places(const std::vector<int>& order) {
    std::vector<int> at(order.size());
    for (size_t k = 0; k < order.size(); k++) at[order[k]] = (int)k;
    return at;
}
SmallHostLevel small_level_plan(const std::vector<int>& bptr, const std::vector<int>& bcol, const std::vector<int>& order, int ctas) {
    SmallHostLevel H;
    const int n = (int)order.size(), per = (n + ctas - 1) / ctas;
    const std::vector<int> place = places(order);
    H.node = order;
    H.ptr.assign(1, 0);
    for (int k = 0; k < n; k++) {
        for (int q = bptr[order[k]]; q < bptr[order[k] + 1]; q++) H.col.push_back(place[bcol[q]]);
        H.ptr.push_back((int)H.col.size());
    }
    std::vector<std::vector<int>> copies(n);        // CTA << 16 | index of the copies of each node
    for (int c = 0; c < ctas; c++) {
        const int n0 = run_start(n, c, ctas), n1 = run_start(n, c + 1, ctas);
        std::vector<int> halo;
        for (int q = H.ptr[n0]; q < H.ptr[n1]; q++)
            if (H.col[q] < n0 || H.col[q] >= n1) halo.push_back(H.col[q]);
        std::sort(halo.begin(), halo.end());
        halo.erase(std::unique(halo.begin(), halo.end()), halo.end());
        for (size_t k = 0; k < halo.size(); k++) copies[halo[k]].push_back(c << 16 | (per + (int)k));
        for (int q = H.ptr[n0]; q < H.ptr[n1]; q++) {
            int& j = H.col[q];
            j = j >= n0 && j < n1 ? j - n0 : per + (int)(std::lower_bound(halo.begin(), halo.end(), j) - halo.begin());
        }
        H.halo = std::max(H.halo, (int)halo.size());
        H.slots = std::max(H.slots, H.ptr[n1] - H.ptr[n0]);
    }
    H.dptr.assign(1, 0);
    for (int k = 0; k < n; k++) {
        H.dst.insert(H.dst.end(), copies[k].begin(), copies[k].end());
        H.dptr.push_back((int)H.dst.size());
    }
    for (int c = 0; c < ctas; c++)
        H.push = std::max(H.push, H.dptr[run_start(n, c + 1, ctas)] - H.dptr[run_start(n, c, ctas)]);
    return H;
}
// The links of a level to the next coarser one (to the coarsest, which every CTA holds whole: plain indices).
SmallHostLink small_link_plan(const std::vector<int>& agg, const std::vector<int>& mptr, const std::vector<int>& mem,
                              const std::vector<int>& order, const std::vector<int>& coarse, bool coarsest, int ctas) {
    SmallHostLink H;
    const int n = (int)order.size(), nc = (int)coarse.size();
    const std::vector<int> place = places(order), cplace = places(coarse);
    auto at = [&](int k, int of, int me) {
        const int o = run_owner(of, k, ctas);
        return o << 16 | (k - run_start(of, o, ctas)) | (o != me ? (int)kElsewhere : 0);
    };
    for (int k = 0; k < n; k++) {
        const int I = cplace[agg[order[k]]];
        H.agg.push_back(coarsest ? I : at(I, nc, run_owner(n, k, ctas)));
    }
    H.mptr.assign(1, 0);
    for (int k = 0; k < nc; k++) {
        for (int q = mptr[coarse[k]]; q < mptr[coarse[k] + 1]; q++) H.mem.push_back(at(place[mem[q]], n, run_owner(nc, k, ctas)));
        H.mptr.push_back((int)H.mem.size());
    }
    for (int c = 0; c < ctas; c++) H.members = std::max(H.members, H.mptr[run_start(nc, c + 1, ctas)] - H.mptr[run_start(nc, c, ctas)]);
    return H;
}
template <class VT>
bool small_solver_takes(const BlockCSR& A, const PrecondOp<VT>& op, const SmallPlan& S, int basis) {
    if (S.ctas <= 0 || A.nnodes > kClusterNodes || op.mixed) return false;
    if (op.kind == 2 && !(op.amg->cl.ctas == S.ctas && op.amg->cl.lo == 0 && op.amg->nlev > 1 && op.amg->patch.mode == 0)) return false;
    if (op.kind != 1 && op.kind != 2) return false;
    return (long)small_layout<VT>(A, op, S, basis).bytes <= S.smem;
}
// A plan for the current device, ctas 0 where no such cluster can be scheduled.  Measured in FP64, general kernels ->
// here: 14 GMRES(30) cycles with AMG on the 1111-node flume 17.4 -> 5.6 ms (14 us an iteration, of which ~8 are the cluster
// barriers); a BiCGStab solve with ILU there 2.54 -> 0.82 ms; one with AMG on 576 nodes 0.86 -> 0.33 ms.
// A whole Newton solve is 1.4 (20 nodes) to 3.4 times faster at every size up to 2048 nodes, with either preconditioner, both
// methods and precisions and randomly numbered nodes, so the line is what the CTAs hold: 128 nodes each.
SmallPlan small_solver_plan(int smem_limit) {
    SmallPlan S;
    S.smem = smem_limit - 1024 - (int)sizeof(SmallAt);                 // the kernels' static shared memory
    auto ready = [&](auto kernel, int ctas) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S.smem) != cudaSuccess) { cudaGetLastError(); return false; }
        return cluster_schedulable(kernel, ctas, kSmallThreads, S.smem);
    };
    if (ready(k_small_gmres<double>, kSmallCtas) && ready(k_small_gmres<float>, kSmallCtas) && ready(k_small_bicg<double>, kSmallCtas) &&
        ready(k_small_bicg<float>, kSmallCtas))
        S.ctas = kSmallCtas;
    return S;
}
template <class VT>
void small_gmres_cycle(const BlockCSR& A, const PrecondOp<VT>& op, const VT* vals, VT* Vb, size_t ld, const VT* rhs, VT* out,
                       const double* rw, const GmresDev& G, int m, const SmallPlan& plan, cudaStream_t st) {
    SmallGmres<VT> S{small_layout<VT>(A, op, plan, m), SmallMatrix<VT>{A.nnodes, A.bptr, A.bcol, vals}, small_precond<VT>(A, op),
                     Vb, ld, rhs, out, rw, G, m};
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = cluster_config(plan.ctas, kSmallThreads, &at, st);
    cfg.dynamicSmemBytes = S.at.bytes;
    cudaLaunchKernelEx(&cfg, k_small_gmres<VT>, S);
}
template <class VT>
void small_bicg(const BlockCSR& A, const PrecondOp<VT>& op, const KrylovVecs<VT>& V, KrylovScalars* S, bool first, int iterations,
                const SmallPlan& plan, cudaStream_t st) {
    SmallBicg<VT> B{small_layout<VT>(A, op, plan, 0), SmallMatrix<VT>{A.nnodes, A.bptr, A.bcol, V.vals}, small_precond<VT>(A, op), V, S,
                    op.right ? 1 : 0, first ? 1 : 0, iterations};
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = cluster_config(plan.ctas, kSmallThreads, &at, st);
    cfg.dynamicSmemBytes = B.at.bytes;
    cudaLaunchKernelEx(&cfg, k_small_bicg<VT>, B);
}
#define SW2_SMALL_INSTANCE(VT)                                                                                                 \
    template bool small_solver_takes<VT>(const BlockCSR&, const PrecondOp<VT>&, const SmallPlan&, int);                        \
    template void small_gmres_cycle<VT>(const BlockCSR&, const PrecondOp<VT>&, const VT*, VT*, size_t, const VT*, VT*,         \
                                        const double*, const GmresDev&, int, const SmallPlan&, cudaStream_t);                  \
    template void small_bicg<VT>(const BlockCSR&, const PrecondOp<VT>&, const KrylovVecs<VT>&, KrylovScalars*, bool, int,      \
                                 const SmallPlan&, cudaStream_t);
SW2_SMALL_INSTANCE(double)
SW2_SMALL_INSTANCE(float)

}  // namespace sw2
