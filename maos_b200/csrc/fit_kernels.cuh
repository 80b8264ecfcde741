// Kernels of the assembled DM fit (sparse plus low rank) for B200 (sm_100a).
//
// The reference's default GPU fit (cuda/solve.cu cusolve_sparse, cumuv_t)
// applies FR and FL as cuSPARSE csrmv plus two cuBLAS gemv per operator,
// one instance at a time.  Here:
//   k_lr_dot   t[b][q] = V_q' x_b (FP64 block partials, the last block to
//              arrive adds them in a fixed order)
//   k_spmv_lr  y_b = M x_b - U t_b, M in CSR as (column, value) pairs read
//              once per group of NI instances, optionally + p.Ap partials for
//              the CG.
// Inside the CG, k_cg_step (tomo_kernels.cuh) leaves t = V' p with the new p,
// so an iteration is two launches.  Every instance's sums are formed
// independently of the others (a warp per row, each lane holding NI instance
// sums, reduced over the warp), so results do not depend on which instances
// run together.
#pragma once
#include "tomo_kernels.cuh"

namespace mb {

// NI instances share a thread's E elements of every column of V.
// grid: (ceil(n / (kThreads * E)), ceil(nb / NI)); part [nb][nq][gridDim.x]; t [nb][kMaxLr]
template <int NI, int E>
__global__ void __launch_bounds__(kThreads)
k_lr_dot(const float *__restrict__ x, const float *__restrict__ V, int nq, long n, double *__restrict__ part,
         float *__restrict__ t, unsigned *__restrict__ cnt, int nb, const int *__restrict__ act) {
    pdl_enter();
    const int b0 = blockIdx.y * NI;
    bool on[NI];
    bool any = false;
#pragma unroll
    for (int u = 0; u < NI; u++) {
        on[u] = b0 + u < nb && !inactive(act, b0 + u);
        any |= on[u];
    }
    if (!any) return;
    __shared__ double sh[kThreads / 32][kMaxLr][NI];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long j0 = (long)blockIdx.x * (kThreads * E) + threadIdx.x;
    float xv[NI][E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const long j = j0 + e * kThreads;
#pragma unroll
        for (int u = 0; u < NI; u++) xv[u][e] = on[u] && j < n ? x[(size_t)(b0 + u) * n + j] : 0.f;
    }
#pragma unroll 2
    for (int q = 0; q < nq; q++) {
        float vv[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const long j = j0 + e * kThreads;
            vv[e] = j < n ? V[(size_t)q * n + j] : 0.f;
        }
        double v[NI];
#pragma unroll
        for (int u = 0; u < NI; u++) {
            v[u] = 0;
#pragma unroll
            for (int e = 0; e < E; e++) v[u] += (double)vv[e] * (double)xv[u][e];
        }
        const int at = warp_sum_many<NI>(v);
        if (lane % (32 / NI) == 0) sh[wid][q][at] = v[0];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nq * NI; e += kThreads) {
        const int q = e / NI, u = e - q * NI;
        double s = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; w++) s += sh[w][q][u];
        if (b0 + u < nb) part[((size_t)(b0 + u) * nq + q) * gridDim.x + blockIdx.x] = s;
    }
    if (last_block(cnt + b0, gridDim.x)) {
        for (int e = wid; e < nq * NI; e += kThreads / 32) {
            const int q = e / NI, u = e - q * NI;
            if (b0 + u >= nb || inactive(act, b0 + u)) continue;
            const double s = warp_sum_fresh(part + ((size_t)(b0 + u) * nq + q) * gridDim.x, gridDim.x);
            if (lane == 0) t[(size_t)(b0 + u) * kMaxLr + q] = (float)s;
        }
        if (threadIdx.x == 0) cnt[b0] = 0;
    }
}

// The NI instances of a group with their values of one index side by side:
// out[(group*n + j)*NI + q] = x[(group*NI + q)*n + j], 0 past the last
// instance.  grid: (ceil(n / kThreads), groups).
template <int NI>
__global__ void __launch_bounds__(kThreads)
k_interleave(const float *__restrict__ x, float *__restrict__ out, long n, int nb) {
    pdl_enter();
    const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int b0 = blockIdx.y * NI;
    float v[NI];
#pragma unroll
    for (int q = 0; q < NI; q++) v[q] = b0 + q < nb ? x[(size_t)(b0 + q) * n + j] : 0.f;
    float *o = out + ((size_t)blockIdx.y * n + j) * NI;
    if constexpr (NI % 4 == 0) {
#pragma unroll
        for (int q = 0; q < NI; q += 4)
            *reinterpret_cast<float4 *>(o + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    } else {
#pragma unroll
        for (int q = 0; q < NI; q++) o[q] = v[q];
    }
}

// The NI values of one column, the first ni of them real (IL: interleaved, one
// or two vector loads).
template <int NI, bool IL>
__device__ __forceinline__ void load_column(float (&v)[NI], const float *__restrict__ xb, int i, long ncol, int ni) {
    if constexpr (IL && NI % 4 == 0) {
        const float4 *p = reinterpret_cast<const float4 *>(xb + (size_t)i * NI);
#pragma unroll
        for (int q = 0; q < NI / 4; q++) {
            const float4 f = p[q];
            v[4 * q] = f.x, v[4 * q + 1] = f.y, v[4 * q + 2] = f.z, v[4 * q + 3] = f.w;
        }
    } else if constexpr (IL && NI == 2) {
        const float2 f = *reinterpret_cast<const float2 *>(xb + (size_t)i * NI);
        v[0] = f.x, v[1] = f.y;
    } else {
#pragma unroll
        for (int q = 0; q < NI; q++) v[q] = q < ni ? xb[(size_t)q * ncol + i] : 0.f;
    }
}

// y[b][i] = sum_e M[i][e] x[b][col_e] - sum_q U[q*nrow + i] t[b][q] (+ add[b][i]).
// IL: x is interleaved (k_interleave).  A row's columns are scattered over
// about ten cache lines per 32 of them, and each instance's gather pays for all
// of those; side by side, one gather serves the group (30 m, 256 instances: 222
// -> 153 us per launch).
// One warp takes kSpmvRows rows one after the other (the CTA's barriers, its
// p.Ap partial and its arrival are shared by them; four entries per lane are
// in flight); the NI sums are reduced over the warp by exchanging halves, so a
// row costs NI + 1 shuffles instead of 5 NI.
// grid: (ceil(nb/NI), ceil(nrow / kSpmvBlock)).
// With dot_part: the p.Ap partials (dot_x = p) per CTA, [nb][gridDim.y].
constexpr int kSpmvRows = 2;
constexpr int kSpmvBlock = kThreads / 32 * kSpmvRows;  // rows per CTA

template <int NI, bool IL>
__global__ void __launch_bounds__(kThreads)
k_spmv_lr(const int *__restrict__ rp, const GatherW *__restrict__ ent, int nrow, long ncol,
          const float *__restrict__ x, float *__restrict__ y, const float *__restrict__ U,
          const float *__restrict__ t, int nq, const float *__restrict__ add, const float *__restrict__ dot_x,
          double *__restrict__ dot_part, int nbatch, const int *__restrict__ act) {
    pdl_enter();
    const int b0 = blockIdx.x * NI;
    const int ni = min(NI, nbatch - b0);
    bool on[NI];
    bool any = false;
#pragma unroll
    for (int q = 0; q < NI; q++) {
        on[q] = q < ni && !inactive(act, b0 + q);
        any |= on[q];
    }
    if (!any) return;  // uniform over the instance group
    __shared__ double sh[kThreads / 32][NI];
    __shared__ float s_t[NI][kMaxLr];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int row0 = blockIdx.y * kSpmvBlock + wid;
    if (nq) {
        if (threadIdx.x < NI * kMaxLr) {
            const int u = threadIdx.x / kMaxLr;
            s_t[u][threadIdx.x % kMaxLr] = u < ni ? t[(size_t)(b0 + u) * kMaxLr + threadIdx.x % kMaxLr] : 0.f;
        }
        __syncthreads();
    }
    const float *xb = x + (size_t)b0 * ncol;
    double dv = 0.0;
    int inst = 0;  // the instance whose sum this lane holds after the reduction
    bool out = false;
#pragma unroll
    for (int rr = 0; rr < kSpmvRows; rr++) {
        const int row = row0 + rr * (kThreads / 32);
        if (row >= nrow) break;
        const float uv = lane < nq ? U[(size_t)lane * nrow + row] : 0.f;
        float acc[NI];
#pragma unroll
        for (int q = 0; q < NI; q++) acc[q] = 0.f;
        const int e1 = rp[row + 1];
        for (int e = rp[row] + lane; e < e1; e += 4 * 32) {
            GatherW g[4];
#pragma unroll
            for (int c = 0; c < 4; c++) g[c] = e + 32 * c < e1 ? ent[e + 32 * c] : GatherW{0, 0.f};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (e + 32 * c >= e1) break;
                float v[NI];
                load_column<NI, IL>(v, xb, g[c].i, ncol, ni);
#pragma unroll
                for (int q = 0; q < NI; q++) acc[q] += g[c].w * v[q];
            }
        }
        inst = warp_sum_many<NI>(acc);
        out = lane % (32 / NI) == 0 && inst < ni && !inactive(act, b0 + inst);
        float lr = 0.f;
        for (int q = 0; q < nq; q++) lr += __shfl_sync(0xffffffffu, uv, q) * s_t[inst][q];
        if (out) {
            const size_t o = (size_t)(b0 + inst) * nrow + row;
            float v = acc[0] - lr;
            if (add) v += add[o];
            y[o] = v;
            if (dot_part) dv += (double)v * (double)dot_x[o];
        }
    }
    if (!dot_part) return;  // uniform
    if (threadIdx.x < NI * (kThreads / 32)) sh[threadIdx.x / NI][threadIdx.x % NI] = 0.0;
    __syncthreads();
    if (out) sh[wid][inst] = dv;
    __syncthreads();
    if (threadIdx.x < ni) {  // instances past nbatch have no row in dot_part
        double s = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; w++) s += sh[w][threadIdx.x];
        dot_part[(size_t)(b0 + threadIdx.x) * gridDim.y + blockIdx.y] = s;
    }
}

}  // namespace mb
