// Message-passing network over the mesh's node graph that predicts the next SW2
// time step (the Newton initial guess), with its training kernels.
//
// Per node i (H = 64 hidden features):
//   e0   = SiLU(W0 f_i + b0)                              f_i: 8 normalised inputs
//   for l = 1..3:
//     X_l = [e | mean_j e_j | sum_j wx_ij (e_j - e_i) | sum_j wy_ij (e_j - e_i)]   (4H)
//     e  <- e + SiLU(W_l X_l + b_l)
//   y    = S S (Wd e + bd)                                 3 outputs (normalised correction)
// where S is the neighbourhood mean (self included) that keeps the correction smooth.
// with wx_ij = (x_j - x_i) / (L deg_i) over the mesh edges (L = mean edge length):
// the mean and the two edge-weighted differences let a layer see values and
// first differences of its neighbourhood in both directions.
//
// Weights are stored in BF16 and converted to FP32 in shared memory; every sum
// accumulates in FP32.  The node graph is symmetric, so the backward pass of the
// aggregation is again a gather over each node's neighbours (the reverse slot of
// each edge is precomputed): no atomics, and training is deterministic.
// Weight gradients reduce per block into partial sums that a second kernel adds in
// block order.
//
// The dense layers run on the FP32 cores: 33 kFLOP per node and layer, 0.22 ms for 500k nodes at
// the chip's FP32 rate (the neighbour gathers of the same nodes take 0.17 ms).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace {

constexpr int H = 64;
constexpr int MAXIN = 4 * H;

struct Graph {
    int n;
    const int* indptr;      // [n+1]
    const int* nbr;         // [nnz] neighbour node of each slot
    const int* rev;         // [nnz] slot of the reverse edge (in the neighbour's list)
    const float* wx;        // [nnz] (x_j - x_i) / (L deg_i)
    const float* wy;
    const float* inv_deg;   // [n]
    const float* swx;       // [n] sum_j wx_ij
    const float* swy;
};

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z) {
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// X[i] = [E_i, mean E_j, sum wx (E_j - E_i), sum wy (E_j - E_i)]; one warp per node, 2 features per lane
__global__ void k_agg_fwd(Graph g, const float* __restrict__ E, float* __restrict__ X) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= g.n) return;
    const int i = warp;
    const float2 ei = reinterpret_cast<const float2*>(E + (size_t)i * H)[lane];
    float2 a = {0, 0}, gx = {0, 0}, gy = {0, 0};
    for (int s = g.indptr[i]; s < g.indptr[i + 1]; s++) {
        const int j = g.nbr[s];
        const float2 ej = reinterpret_cast<const float2*>(E + (size_t)j * H)[lane];
        const float wx = g.wx[s], wy = g.wy[s];
        a.x += ej.x; a.y += ej.y;
        gx.x += wx * (ej.x - ei.x); gx.y += wx * (ej.y - ei.y);
        gy.x += wy * (ej.x - ei.x); gy.y += wy * (ej.y - ei.y);
    }
    const float d = g.inv_deg[i];
    float2* xo = reinterpret_cast<float2*>(X + (size_t)i * MAXIN);
    xo[lane] = ei;
    xo[32 + lane] = make_float2(a.x * d, a.y * d);
    xo[64 + lane] = gx;
    xo[96 + lane] = gy;
}

// dE[j] += dX_e[j] + sum_{i in N(j)} (dA_i / deg_i + wx_ij dGx_i + wy_ij dGy_i) - swx_j dGx_j - swy_j dGy_j
__global__ void k_agg_bwd(Graph g, const float* __restrict__ dX, float* __restrict__ dE) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= g.n) return;
    const int j = warp;
    const float2* xj = reinterpret_cast<const float2*>(dX + (size_t)j * MAXIN);
    float2 acc = xj[lane];
    const float2 gxj = xj[64 + lane], gyj = xj[96 + lane];
    acc.x -= g.swx[j] * gxj.x + g.swy[j] * gyj.x;
    acc.y -= g.swx[j] * gxj.y + g.swy[j] * gyj.y;
    for (int s = g.indptr[j]; s < g.indptr[j + 1]; s++) {
        const int i = g.nbr[s], r = g.rev[s];        // slot r of node i points to j
        const float2* xi = reinterpret_cast<const float2*>(dX + (size_t)i * MAXIN);
        const float2 da = xi[32 + lane], dgx = xi[64 + lane], dgy = xi[96 + lane];
        const float di = g.inv_deg[i], wx = g.wx[r], wy = g.wy[r];
        acc.x += da.x * di + wx * dgx.x + wy * dgy.x;
        acc.y += da.y * di + wx * dgx.y + wy * dgy.y;
    }
    float2* o = reinterpret_cast<float2*>(dE + (size_t)j * H);
    float2 cur = o[lane];
    cur.x += acc.x; cur.y += acc.y;
    o[lane] = cur;
}

// ---------------------------------------------------------------- dense layers
// Three products over the nodes: forward X W^T, backward dZ W, and the weight gradient dZ^T X.  They run on the FP32
// cores with every sum in the order of its index (k, o or node), so the results do not depend on the tiling.
// What bounds a straightforward form is shared memory: one weight and one input read per multiply-add or two kept the
// 500k-node layer (256 -> 64) at 4.2 ms, 16 % of the FP32 rate.  Here a thread owns 4 outputs x 8 nodes (or 4 x 4
// weights), so that 12 16-byte shared reads feed 128 multiply-adds, the weights stay in shared memory while a CTA walks
// over its tiles, and the next piece of X is fetched (cp.async) while this one is multiplied.
// Times before and after: 256 -> 64 forward at 500k nodes 4.2 -> 0.50 ms; at 125k nodes all layers of a training pass
// forward 3.70 -> 0.47, input gradients 1.83 -> 0.69, weight gradients 4.47 -> 0.46 ms.
constexpr int DENSE_THREADS = 256;
constexpr int CHUNK = 32;             // inputs of X staged at a time
constexpr int LDA = CHUNK + 4;        // padded row: 16-byte aligned, rows 4 banks apart

__device__ __forceinline__ void cp16(float* dst, const float* src, bool on) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = on ? 16 : 0;    // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// 4 consecutive floats to shared memory: asynchronously where the source is 16-byte aligned, else one by one
__device__ __forceinline__ void stage4(float* dst, const float* src, bool on, int vec) {
    if (vec) { cp16(dst, src, on); return; }
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) v = make_float4(src[0], src[1], src[2], src[3]);
    *reinterpret_cast<float4*>(dst) = v;
}
__device__ __forceinline__ void put4(float* dst, const float (&v)[4], int count, int vec) {
    if (vec && count >= 4) { *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]); return; }
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (q < count) dst[q] = v[q];
}

// acc[i][q] += sum over r of A[node i][r] B[r][4 outputs], r in order, four at a time; node i is 16 rows after node i-1
template <int NPT>
__device__ __forceinline__ void tile_fma(float (&acc)[NPT][4], const float* A, int lda, const float* B, int ldb, int count) {
    for (int r = 0; r < count; r += 4) {
        float4 w[4];
#pragma unroll
        for (int c = 0; c < 4; c++) w[c] = *reinterpret_cast<const float4*>(B + (r + c) * ldb);
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const float4 x = *reinterpret_cast<const float4*>(A + i * 16 * lda + r);
            const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                acc[i][0] += w[c].x * xs[c]; acc[i][1] += w[c].y * xs[c];
                acc[i][2] += w[c].z * xs[c]; acc[i][3] += w[c].w * xs[c];
            }
        }
    }
}

// bit 0: X, bit 1: outputs and R, bit 2: W may be read or written 16 bytes at a time
enum { VEC_X = 1, VEC_OUT = 2, VEC_W = 4, VEC_IN = 8 };

// Y = act(W X + b) (+ R): W [out][in] BF16 -> shared FP32 [in][64]; 16 NPT nodes per tile, thread t: outputs
// 4 (t % 16) .. + 3 of nodes t / 16 + 16 i
template <int NPT>
__global__ void __launch_bounds__(DENSE_THREADS, 2) k_dense_fwd(int n, int in, int out, const __nv_bfloat16* __restrict__ W,
                                                                const float* __restrict__ b, const float* __restrict__ X,
                                                                const float* __restrict__ R, int act, float* __restrict__ Z,
                                                                float* __restrict__ Y, int vec) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TN = 16 * NPT;
    float* Ws = sm;                   // [in][64]
    float* Xs = sm + in * H;          // [2][TN][LDA]
    const int ntiles = (n + TN - 1) / TN, nch = (in + CHUNK - 1) / CHUNK;
    const int mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int total = mine * nch;
    auto fetch = [&](int it) {
        const int base = (blockIdx.x + (it / nch) * gridDim.x) * TN, k0 = (it % nch) * CHUNK;
        const int w4 = (in - k0 < CHUNK ? in - k0 : CHUNK) / 4;
        float* dst = Xs + (it & 1) * TN * LDA;
        for (int t = threadIdx.x; t < TN * w4; t += DENSE_THREADS) {
            const int r = t / w4, c = 4 * (t - r * w4), node = base + r;
            const bool on = node < n;
            stage4(dst + r * LDA + c, X + (size_t)(on ? node : 0) * in + k0 + c, on, vec & VEC_X);
        }
        cp_commit();
    };
    if (total > 0) fetch(0);
    if (vec & VEC_W) {                // 8 inputs of an output at a time, lanes along the outputs
        for (int t = threadIdx.x; t < (in / 8) * H; t += DENSE_THREADS) {
            const int o = t % H, k = 8 * (t / H);
            const uint4 u = o < out ? *reinterpret_cast<const uint4*>(W + (size_t)o * in + k) : make_uint4(0, 0, 0, 0);
            const unsigned p[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                Ws[(k + 2 * c) * H + o] = __uint_as_float(p[c] << 16);
                Ws[(k + 2 * c + 1) * H + o] = __uint_as_float(p[c] & 0xffff0000u);
            }
        }
    } else {
        for (int t = threadIdx.x; t < in * H; t += DENSE_THREADS) {
            const int k = t / H, o = t % H;
            Ws[t] = o < out ? __bfloat162float(W[(size_t)o * in + k]) : 0.0f;
        }
    }
    const int ng = threadIdx.x >> 4, o0 = (threadIdx.x & 15) * 4;
    float acc[NPT][4];
    for (int it = 0; it < total; it++) {
        const int ch = it % nch, k0 = ch * CHUNK;
        if (it + 1 < total) { fetch(it + 1); cp_wait<1>(); }
        else cp_wait<0>();
        __syncthreads();
        if (ch == 0) {
#pragma unroll
            for (int i = 0; i < NPT; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] = 0.0f;
        }
        tile_fma<NPT>(acc, Xs + (it & 1) * TN * LDA + ng * LDA, LDA, Ws + k0 * H + o0, H, in - k0 < CHUNK ? in - k0 : CHUNK);
        __syncthreads();              // the next fetch overwrites this buffer
        if (ch < nch - 1 || o0 >= out) continue;
        const int base = (blockIdx.x + (it / nch) * gridDim.x) * TN;
        float bias[4];
#pragma unroll
        for (int q = 0; q < 4; q++) bias[q] = o0 + q < out ? b[o0 + q] : 0.0f;
#pragma unroll
        for (int i = 0; i < NPT; i++) {
            const int node = base + ng + 16 * i;
            if (node >= n) continue;
            const size_t at = (size_t)node * out + o0;
            float z[4], y[4];
#pragma unroll
            for (int q = 0; q < 4; q++) { z[q] = acc[i][q] + bias[q]; y[q] = act ? silu(z[q]) : z[q]; }
            if (Z) put4(Z + at, z, out - o0, vec & VEC_OUT);
            if (R) {
                if (vec & VEC_OUT) {
                    const float4 r = *reinterpret_cast<const float4*>(R + at);
                    y[0] += r.x; y[1] += r.y; y[2] += r.z; y[3] += r.w;
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (o0 + q < out) y[q] += R[at + q];
                }
            }
            put4(Y + at, y, out - o0, vec & VEC_OUT);
        }
    }
}

// The forward pass to a few outputs (the decoder, 64 -> 3): bound by reading X, so a thread per node with the tile's X
// in shared memory
constexpr int NARROW = 4, NARROW_NODES = 128;
__global__ void __launch_bounds__(NARROW_NODES) k_dense_narrow(int n, int in, int out, const __nv_bfloat16* __restrict__ W,
                                                               const float* __restrict__ b, const float* __restrict__ X,
                                                               const float* __restrict__ R, int act, float* __restrict__ Z,
                                                               float* __restrict__ Y) {
    extern __shared__ __align__(16) float sm[];
    float* Ws = sm;                   // [in][NARROW]
    float* Xs = sm + in * NARROW;     // [NARROW_NODES][in + 1]
    const int base = blockIdx.x * NARROW_NODES, ldx = in + 1;
    for (int t = threadIdx.x; t < in * NARROW; t += NARROW_NODES) {
        const int k = t / NARROW, o = t % NARROW;
        Ws[t] = o < out ? __bfloat162float(W[(size_t)o * in + k]) : 0.0f;
    }
    for (int t = threadIdx.x; t < NARROW_NODES * in; t += NARROW_NODES) {
        const int r = t / in, k = t - r * in;
        Xs[r * ldx + k] = base + r < n ? X[(size_t)base * in + t] : 0.0f;
    }
    __syncthreads();
    const int node = base + threadIdx.x;
    if (node >= n) return;
    float acc[NARROW] = {0.0f, 0.0f, 0.0f, 0.0f};
    const float* xr = Xs + threadIdx.x * ldx;
#pragma unroll 8
    for (int k = 0; k < in; k++) {
        const float4 w = reinterpret_cast<const float4*>(Ws)[k];
        const float x = xr[k];
        acc[0] += w.x * x; acc[1] += w.y * x; acc[2] += w.z * x; acc[3] += w.w * x;
    }
#pragma unroll
    for (int o = 0; o < NARROW; o++) {
        if (o >= out) break;
        const size_t at = (size_t)node * out + o;
        const float z = acc[o] + b[o];
        if (Z) Z[at] = z;
        float y = act ? silu(z) : z;
        if (R) y += R[at];
        Y[at] = y;
    }
}

// dZ = dY * act'(Z), then dX = W^T dZ (dX may be null): the tile's dZ in shared memory, 64 inputs at a time; thread t:
// inputs 4 (t % 16) .. + 3 of nodes t / 16 + 16 i
template <int NPT>
__global__ void __launch_bounds__(DENSE_THREADS, 2) k_dense_bwd_x(int n, int in, int out, const __nv_bfloat16* __restrict__ W,
                                                                  const float* __restrict__ Z, const float* __restrict__ dY,
                                                                  int act, float* __restrict__ dZ, float* __restrict__ dX,
                                                                  int vec) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TN = 16 * NPT, LDD = H + 4;
    float* Ws = sm;                   // [out4][in], rows past out zero
    const int out4 = (out + 3) & ~3;
    float* Ds = sm + out4 * in;       // [TN][LDD]
    if (dX)
        for (int t = threadIdx.x; t < out4 * in; t += DENSE_THREADS) Ws[t] = t < out * in ? __bfloat162float(W[t]) : 0.0f;
    const int ntiles = (n + TN - 1) / TN;
    const int ng = threadIdx.x >> 4, j0 = (threadIdx.x & 15) * 4;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int base = tile * TN;
        __syncthreads();              // the last tile's products are done with Ds
        if (vec & VEC_IN) {
            // 16 bytes of dY and of Z per load, four of each under way: one value at a time their latency was a third
            // of the kernel (138 us, now 92, mean over the five layers of a gradient at 126k nodes)
            const int out_q = out >> 2;
#pragma unroll 4
            for (int t = threadIdx.x; t < TN * out_q; t += DENSE_THREADS) {
                const int r = t / out_q, o = 4 * (t - r * out_q), node = base + r;
                float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (node < n) {
                    const size_t idx = (size_t)node * out + o;
                    d = *reinterpret_cast<const float4*>(dY + idx);
                    if (act) {
                        const float4 z = *reinterpret_cast<const float4*>(Z + idx);
                        d.x *= dsilu(z.x); d.y *= dsilu(z.y); d.z *= dsilu(z.z); d.w *= dsilu(z.w);
                    }
                    *reinterpret_cast<float4*>(dZ + idx) = d;
                }
                *reinterpret_cast<float4*>(Ds + r * LDD + o) = d;
            }
        } else {
            for (int t = threadIdx.x; t < TN * out4; t += DENSE_THREADS) {
                const int r = t / out4, o = t - r * out4, node = base + r;
                float d = 0.0f;
                if (node < n && o < out) {
                    const size_t idx = (size_t)node * out + o;
                    d = dY[idx];
                    if (act) d *= dsilu(Z[idx]);
                    dZ[idx] = d;
                }
                Ds[r * LDD + o] = d;
            }
        }
        __syncthreads();
        if (!dX) continue;
        for (int k0 = 0; k0 + j0 < in; k0 += H) {
            float acc[NPT][4];
#pragma unroll
            for (int i = 0; i < NPT; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[i][q] = 0.0f;
            tile_fma<NPT>(acc, Ds + ng * LDD, LDD, Ws + k0 + j0, in, out4);
#pragma unroll
            for (int i = 0; i < NPT; i++) {
                const int node = base + ng + 16 * i;
                if (node < n) put4(dX + (size_t)node * in + k0 + j0, acc[i], 4, vec & VEC_OUT);
            }
        }
    }
}

// partial dW[o][k] and db[o] over a chunk of nodes, summed in node order: blockIdx.x the chunk, blockIdx.y 64 inputs;
// thread t: outputs 4 (t / 16) .. + 3 x inputs 4 (t % 16) .. + 3, 32 nodes staged at a time
constexpr int WNODES = 32;
__global__ void __launch_bounds__(DENSE_THREADS) k_dense_bwd_w(int n, int in, int out, int nodes_per_block,
                                                               const float* __restrict__ X, const float* __restrict__ dZ,
                                                               float* __restrict__ part, int vec) {
    __shared__ __align__(16) float Xs[2][WNODES][H], Ds[2][WNODES][H];
    const int k0 = blockIdx.y * H, nk = in - k0 < H ? in - k0 : H;
    const long first = (long)blockIdx.x * nodes_per_block;
    const int n0 = (int)first, n1 = (int)(first + nodes_per_block < n ? first + nodes_per_block : n);
    const int oq = (threadIdx.x >> 4) * 4, kq = (threadIdx.x & 15) * 4;
    const int steps = (n1 - n0 + WNODES - 1) / WNODES;
    auto fetch = [&](int s) {
        const int buf = s & 1, base = n0 + s * WNODES;
        for (int t = threadIdx.x; t < WNODES * (H / 4); t += DENSE_THREADS) {
            const int r = t / (H / 4), c = 4 * (t % (H / 4)), node = base + r;
            const bool on = node < n1;
            const size_t at = (size_t)(on ? node : n0);
            stage4(&Xs[buf][r][c], X + at * in + k0 + (c < nk ? c : 0), on && c < nk, vec & VEC_X);
            if (vec & VEC_OUT) stage4(&Ds[buf][r][c], dZ + at * out + (c < out ? c : 0), on && c < out, 1);
            else
                for (int q = 0; q < 4; q++) Ds[buf][r][c + q] = on && c + q < out ? dZ[at * out + c + q] : 0.0f;
        }
        cp_commit();
    };
    float acc[4][4], bacc[4];
#pragma unroll
    for (int o = 0; o < 4; o++) {
        bacc[o] = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; k++) acc[o][k] = 0.0f;
    }
    fetch(0);
    for (int s = 0; s < steps; s++) {
        if (s + 1 < steps) { fetch(s + 1); cp_wait<1>(); }
        else cp_wait<0>();
        __syncthreads();
        const int buf = s & 1, cnt = n1 - n0 - s * WNODES < WNODES ? n1 - n0 - s * WNODES : WNODES;
        if (oq < out) {
#pragma unroll 4
            for (int r = 0; r < cnt; r++) {
                const float4 d = *reinterpret_cast<const float4*>(&Ds[buf][r][oq]), x = *reinterpret_cast<const float4*>(&Xs[buf][r][kq]);
                const float dv[4] = {d.x, d.y, d.z, d.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int o = 0; o < 4; o++) {
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[o][k] += dv[o] * xv[k];
                    bacc[o] += dv[o];
                }
            }
        }
        __syncthreads();
    }
    float* p = part + (size_t)blockIdx.x * (out * in + out);
#pragma unroll
    for (int o = 0; o < 4; o++) {
        if (oq + o >= out) break;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (kq + k < nk) p[(oq + o) * in + k0 + kq + k] = acc[o][k];
        if (blockIdx.y == 0 && kq == 0) p[out * in + oq + o] = bacc[o];
    }
}

// g[c] = sum over blocks of part[blk][c] (fixed block order)
__global__ void k_reduce_parts(int nparts, int count, const float* __restrict__ part, float* __restrict__ g) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= count) return;
    float s = 0.0f;
    int p = 0;
    for (; p + 16 <= nparts; p += 16) {   // 16 loads in flight, added in block order
        float v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = part[(size_t)(p + q) * count + c];
#pragma unroll
        for (int q = 0; q < 16; q++) s += v[q];
    }
    for (; p < nparts; p++) s += part[(size_t)p * count + c];
    g[c] = s;
}

// Adam on the FP32 master weights, then their BF16 copy
__global__ void k_adam(int count, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, __nv_bfloat16* __restrict__ wb, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi; v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    wb[i] = __float2bfloat16(wi);
}

__global__ void k_to_bf16(int count, const float* __restrict__ w, __nv_bfloat16* __restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) wb[i] = __float2bfloat16(w[i]);
}

// Inputs f_i (8) from the FP64 state: [h, u, v, dh, du, dv, z, wet] normalised by (mu, sd)
__global__ void k_features(int n, const double* __restrict__ sol, const double* __restrict__ sol_prev,
                           const double* __restrict__ z, const float* __restrict__ mu, const float* __restrict__ sd,
                           float* __restrict__ F) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f[8];
    for (int v = 0; v < 3; v++) {
        f[v] = (float)sol[3 * i + v];
        f[3 + v] = (float)(sol[3 * i + v] - sol_prev[3 * i + v]);
    }
    f[6] = (float)z[i];
    f[7] = sol[3 * i] > 0.0 ? 1.0f : 0.0f;
    for (int c = 0; c < 8; c++) F[(size_t)i * 8 + c] = (f[c] - mu[c]) / sd[c];
}

// targets: T = (sol_next - sol - (sol - sol_prev)) / scale  -- the correction to linear extrapolation;
// M = 1 where the guess will use the network (h > min_depth now and next), else 0
__global__ void k_targets(int n, const double* __restrict__ sol_next, const double* __restrict__ sol,
                          const double* __restrict__ sol_prev, const float* __restrict__ scale, double min_depth,
                          float* __restrict__ T, float* __restrict__ M) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int v = 0; v < 3; v++) {
        const int d = 3 * i + v;
        T[d] = (float)((sol_next[d] - 2.0 * sol[d] + sol_prev[d]) / (double)scale[v]);
    }
    M[i] = (sol[3 * i] > min_depth && sol_next[3 * i] > min_depth) ? 1.0f : 0.0f;
}

// 3-channel neighbourhood mean (self included): Ys_i = (Y_i + sum_j Y_j) / (deg_i + 1).  Smooths the
// network's correction so that its errors stay smooth: the SW2 residual differentiates the guess, and
// node-to-node noise in it costs more residual than the same error spread smoothly.
__global__ void k_smooth3(Graph g, const float* __restrict__ Y, float* __restrict__ Ys) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    float a = Y[3 * i], b = Y[3 * i + 1], c = Y[3 * i + 2];
    for (int s = g.indptr[i]; s < g.indptr[i + 1]; s++) {
        const int j = g.nbr[s];
        a += Y[3 * j]; b += Y[3 * j + 1]; c += Y[3 * j + 2];
    }
    const float w = 1.0f / (float)(g.indptr[i + 1] - g.indptr[i] + 1);
    Ys[3 * i] = a * w; Ys[3 * i + 1] = b * w; Ys[3 * i + 2] = c * w;
}
// adjoint: dY_j = dYs_j / (deg_j + 1) + sum_{i in N(j)} dYs_i / (deg_i + 1)
__global__ void k_smooth3_adj(Graph g, const float* __restrict__ dYs, float* __restrict__ dY) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= g.n) return;
    const float wj = 1.0f / (float)(g.indptr[j + 1] - g.indptr[j] + 1);
    float a = dYs[3 * j] * wj, b = dYs[3 * j + 1] * wj, c = dYs[3 * j + 2] * wj;
    for (int s = g.indptr[j]; s < g.indptr[j + 1]; s++) {
        const int i = g.nbr[s];
        const float wi = 1.0f / (float)(g.indptr[i + 1] - g.indptr[i] + 1);
        a += dYs[3 * i] * wi; b += dYs[3 * i + 1] * wi; c += dYs[3 * i + 2] * wi;
    }
    dY[3 * j] = a; dY[3 * j + 1] = b; dY[3 * j + 2] = c;
}

// loss partials and dY = 2 M (Y - T) / count over the node mask M (1: the node counts)
__global__ void __launch_bounds__(256) k_mse(int n3, const float* __restrict__ Y, const float* __restrict__ T,
                                             const float* __restrict__ M, float inv_count, float* __restrict__ dY,
                                             float* __restrict__ part) {
    __shared__ float sh[8];
    float s = 0.0f;
    for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < n3; d += gridDim.x * blockDim.x) {
        const float e = (Y[d] - T[d]) * M[d / 3];
        s += e * e;
        dY[d] = 2.0f * e * inv_count;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < 8; w++) t += sh[w];
        part[blockIdx.x] = t * inv_count;
    }
}

// guess = sol + (sol - sol_prev) + scale * Y   (FP64 out), per node; a node that is
// shallow now or would be shallow in the guess (h <= min_depth) keeps sol: the
// guess must not move the wet/dry front, which the residual punishes hardest
__global__ void k_apply_guess(int n, const double* __restrict__ sol, const double* __restrict__ sol_prev,
                              const float* __restrict__ Y, const float* __restrict__ scale, double min_depth,
                              double* __restrict__ guess) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double g[3];
    for (int v = 0; v < 3; v++)
        g[v] = 2.0 * sol[3 * i + v] - sol_prev[3 * i + v] + (double)scale[v] * (double)Y[3 * i + v];
    const bool keep = !(sol[3 * i] > min_depth) || !(g[0] > min_depth);
    for (int v = 0; v < 3; v++) guess[3 * i + v] = keep ? sol[3 * i + v] : g[v];
}

inline int nb(long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ C ABI (include/adh_sw2_gnn.h)
extern "C" {

static Graph mk(int n, const int* indptr, const int* nbr, const int* rev, const float* wx, const float* wy,
                const float* inv_deg, const float* swx, const float* swy) {
    return Graph{n, indptr, nbr, rev, wx, wy, inv_deg, swx, swy};
}

int sw2n_agg_fwd(int n, const int* indptr, const int* nbr, const int* rev, const float* wx, const float* wy,
                 const float* inv_deg, const float* swx, const float* swy, const float* E, float* X, void* stream) {
    if (n <= 0 || !E || !X) return -1;
    k_agg_fwd<<<nb(32L * n, 256), 256, 0, (cudaStream_t)stream>>>(mk(n, indptr, nbr, rev, wx, wy, inv_deg, swx, swy), E, X);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_agg_bwd(int n, const int* indptr, const int* nbr, const int* rev, const float* wx, const float* wy,
                 const float* inv_deg, const float* swx, const float* swy, const float* dX, float* dE, void* stream) {
    if (n <= 0 || !dX || !dE) return -1;
    k_agg_bwd<<<nb(32L * n, 256), 256, 0, (cudaStream_t)stream>>>(mk(n, indptr, nbr, rev, wx, wy, inv_deg, swx, swy), dX, dE);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
static int num_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}
static bool dense_sizes(int in, int out) { return in > 0 && in <= MAXIN && out > 0 && out <= H && in % 4 == 0; }
extern "C++" {
// Allows a launch of `smem` bytes.  What is set is always `most`, the kernel's need at the widest layer: the attribute is the
// kernel's, not the launch's, and a thread that set its own smaller need would have another's launch refused.
template <class K> static bool dense_attr(K kernel, size_t smem, size_t most) {
    return smem <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess;
}
static constexpr size_t fwd_smem(int in, int npt) { return sizeof(float) * ((size_t)in * H + 2 * 16 * (size_t)npt * LDA); }
static constexpr size_t bwd_smem(int in, int out, int npt) { return sizeof(float) * ((size_t)((out + 3) & ~3) * in + (size_t)16 * npt * (H + 4)); }
static constexpr size_t narrow_smem(int in) { return sizeof(float) * ((size_t)in * NARROW + (size_t)NARROW_NODES * (in + 1)); }
}
// Tiles of 128 nodes, or of 16, which spread a small graph over more SMs, but read shared memory three times as often for a
// multiply-add.  The line is where the two cross: one wide tile for two SMs where the products weigh (256 -> 64 forward, 16 and
// 128 nodes: 26.8 and 28.8 us at 6000, 37.0 and 28.8 at 10,000, 56 and 29 at 18,900; with gradients 42 and 44, 58 and 52, 79 and 56),
// one per SM in narrow layers (8 -> 64 forward: 6.3 and 9.3 us at 6000, 8.3 and 9.4 at 14,000, 10.3 and 9.4 at 18,900, 13.5 and
// 10.4 at 30,000).
static bool wide_tiles(int n, int in, int sms) { return (long)n >= (in > H ? 64L : 128L) * sms; }

extern "C++" {
template <int NPT>
static int run_dense_fwd(int n, int in, int out, const __nv_bfloat16* W, const float* b, const float* X, const float* R, int act,
                         float* Z, float* Y, int vec, int sms, cudaStream_t st) {
    const size_t smem = fwd_smem(in, NPT);
    const int tiles = nb(n, 16 * NPT), grid = tiles < 2 * sms ? tiles : 2 * sms;
    if (!dense_attr(k_dense_fwd<NPT>, smem, fwd_smem(MAXIN, NPT))) return -2;
    k_dense_fwd<NPT><<<grid, DENSE_THREADS, smem, st>>>(n, in, out, W, b, X, R, act, Z, Y, vec);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
}
int sw2n_dense_fwd(int n, int in, int out, const void* W_bf16, const float* b, const float* X, const float* R, int act,
                   float* Z, float* Y, void* stream) {
    if (n <= 0 || !dense_sizes(in, out) || !W_bf16 || !b || !X || !Y) return -1;
    const __nv_bfloat16* W = (const __nv_bfloat16*)W_bf16;
    cudaStream_t st = (cudaStream_t)stream;
    if (out <= NARROW) {
        const size_t smem = narrow_smem(in);
        if (!dense_attr(k_dense_narrow, smem, narrow_smem(MAXIN))) return -2;
        k_dense_narrow<<<nb(n, NARROW_NODES), NARROW_NODES, smem, st>>>(n, in, out, W, b, X, R, act, Z, Y);
        return cudaGetLastError() == cudaSuccess ? 0 : -2;
    }
    const int vec = (aligned16(X) ? VEC_X : 0) | (out % 4 == 0 && aligned16(Y) && aligned16(Z) && aligned16(R) ? VEC_OUT : 0) |
                    (in % 8 == 0 && aligned16(W) ? VEC_W : 0);
    const int sms = num_sms();
    return wide_tiles(n, in, sms) ? run_dense_fwd<8>(n, in, out, W, b, X, R, act, Z, Y, vec, sms, st)
                              : run_dense_fwd<1>(n, in, out, W, b, X, R, act, Z, Y, vec, sms, st);
}

extern "C++" {
template <int NPT>
static bool run_dense_bwd_x(int n, int in, int out, const __nv_bfloat16* W, const float* Z, const float* dY, int act, float* dZ,
                            float* dX, int vec, int sms, cudaStream_t st) {
    const size_t smem = bwd_smem(in, out, NPT);
    const int tiles = nb(n, 16 * NPT), grid = tiles < 2 * sms ? tiles : 2 * sms;
    if (!dense_attr(k_dense_bwd_x<NPT>, smem, bwd_smem(MAXIN, H, NPT))) return false;
    k_dense_bwd_x<NPT><<<grid, DENSE_THREADS, smem, st>>>(n, in, out, W, Z, dY, act, dZ, dX, vec);
    return true;
}
}
// backward of a dense layer: dZ (out) = dY * act'(Z); dX = W^T dZ (if dX); gW [out*in + out] = (dW, db)
// summed over nodes; part must hold nparts * (out*in + out) floats with nparts = ceil(n / nodes_per_block)
int sw2n_dense_bwd(int n, int in, int out, const void* W_bf16, const float* X, const float* Z, const float* dY, int act,
                   float* dZ, float* dX, int nodes_per_block, float* part, float* gW, void* stream) {
    if (n <= 0 || !dense_sizes(in, out) || nodes_per_block <= 0 || !dZ || !part || !gW) return -1;
    cudaStream_t st = (cudaStream_t)stream;
    const __nv_bfloat16* W = (const __nv_bfloat16*)W_bf16;
    const int sms = num_sms(), vx = (aligned16(dX) ? VEC_OUT : 0) |
                                         (out % 4 == 0 && aligned16(dY) && aligned16(Z) && aligned16(dZ) ? VEC_IN : 0);
    const bool ok = wide_tiles(n, in, sms) ? run_dense_bwd_x<8>(n, in, out, W, Z, dY, act, dZ, dX, vx, sms, st)
                                       : run_dense_bwd_x<1>(n, in, out, W, Z, dY, act, dZ, dX, vx, sms, st);
    if (!ok) return -2;
    const int nparts = nb(n, nodes_per_block);
    const int vec = (aligned16(X) ? VEC_X : 0) | (out % 4 == 0 && aligned16(dZ) ? VEC_OUT : 0);
    k_dense_bwd_w<<<dim3(nparts, nb(in, H)), DENSE_THREADS, 0, st>>>(n, in, out, nodes_per_block, X, dZ, part, vec);
    const int count = out * in + out;
    k_reduce_parts<<<nb(count, 128), 128, 0, st>>>(nparts, count, part, gW);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_adam(int count, float* w, const float* g, float* m, float* v, void* w_bf16, float lr, float b1, float b2,
              float eps, int t, void* stream) {
    if (count <= 0 || t <= 0) return -1;
    float c1 = 1.0f, c2 = 1.0f, p1 = 1.0f, p2 = 1.0f;
    for (int k = 0; k < t && k < 100000; k++) { p1 *= b1; p2 *= b2; }
    c1 = 1.0f - p1; c2 = 1.0f - p2;
    k_adam<<<nb(count, 256), 256, 0, (cudaStream_t)stream>>>(count, w, g, m, v, (__nv_bfloat16*)w_bf16, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_to_bf16(int count, const float* w, void* w_bf16, void* stream) {
    if (count <= 0) return -1;
    k_to_bf16<<<nb(count, 256), 256, 0, (cudaStream_t)stream>>>(count, w, (__nv_bfloat16*)w_bf16);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_features(int n, const double* sol, const double* sol_prev, const double* z, const float* mu, const float* sd,
                  float* F, void* stream) {
    if (n <= 0) return -1;
    k_features<<<nb(n, 256), 256, 0, (cudaStream_t)stream>>>(n, sol, sol_prev, z, mu, sd, F);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_targets(int n, const double* sol_next, const double* sol, const double* sol_prev, const float* scale,
                 double min_depth, float* T, float* M, void* stream) {
    if (n <= 0) return -1;
    k_targets<<<nb(n, 256), 256, 0, (cudaStream_t)stream>>>(n, sol_next, sol, sol_prev, scale, min_depth, T, M);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// part must hold 148*4 floats; the loss is the sum of part[0 .. returned count)
int sw2n_mse(int n, const float* Y, const float* T, const float* M, float* dY, float* part, void* stream) {
    if (n <= 0) return -1;
    const int blocks = 148 * 4;
    k_mse<<<blocks, 256, 0, (cudaStream_t)stream>>>(3 * n, Y, T, M, 1.0f / (3.0f * n), dY, part);
    return cudaGetLastError() == cudaSuccess ? blocks : -2;
}

int sw2n_smooth3(int n, const int* indptr, const int* nbr, const float* Y, float* Ys, void* stream) {
    if (n <= 0 || !Y || !Ys || Y == Ys) return -1;
    Graph g{}; g.n = n; g.indptr = indptr; g.nbr = nbr;
    k_smooth3<<<nb(n, 256), 256, 0, (cudaStream_t)stream>>>(g, Y, Ys);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_smooth3_adj(int n, const int* indptr, const int* nbr, const float* dYs, float* dY, void* stream) {
    if (n <= 0 || !dYs || !dY || dYs == dY) return -1;
    Graph g{}; g.n = n; g.indptr = indptr; g.nbr = nbr;
    k_smooth3_adj<<<nb(n, 256), 256, 0, (cudaStream_t)stream>>>(g, dYs, dY);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int sw2n_apply_guess(int n, const double* sol, const double* sol_prev, const float* Y, const float* scale,
                     double min_depth, double* guess, void* stream) {
    if (n <= 0) return -1;
    k_apply_guess<<<nb(n, 256), 256, 0, (cudaStream_t)stream>>>(n, sol, sol_prev, Y, scale, min_depth, guess);
    return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // extern "C"
