// The quadratic surrogate as a differentiable function: forward, backward,
// the ridge refit's normal equations, an FP64 solve (LDL') and a
// gradient-ascent mutation step (include/csx_surrogate.h).
//
// Reference: brain/evolve.py:211-220 (features: [1 | genes | g_i g_j, j <= i
// < 16]) and :250-268 (refit_surrogate: numpy FP64 normal equations and
// solve); src/screen.zig:97-112 (the screen's score of the same features).
//
// Work sizes are small next to the screen: a refit table of 400,000 rows of
// 16 genes is 25.6 MB. The normal equations (nf(nf+1)/2 products per row) run on
// the tensor cores in fixed point (csx_gram.cuh), those of the full surface, and
// of tables for which FP64 sums are closer, on the FP64 pipe; everything else is
// a few hundred FP32 FMAs per row.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "csx_device.cuh"
#include "csx_screen.h"
#include "csx_surrogate.h"
#include "csx_tc.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kQuadGenes = 16;                             // the reference layouts' quadratic block
constexpr int kNQuad = kQuadGenes * (kQuadGenes + 1) / 2;  // 136
constexpr int kMaxLin = 29;
constexpr int kMinFeat = 1 + kQuadGenes + kNQuad;  // 153
constexpr int kMaxFeat = 1 + kMaxLin + kNQuad;     // 166
// The full surface (csx_screen.h): the quadratic block over all 29 genes.
constexpr int kNQuadFull = kMaxLin * (kMaxLin + 1) / 2;  // 435
constexpr int kFullFeat = 1 + kMaxLin + kNQuadFull;      // 465
constexpr int kFeatCap = kFullFeat;                      // stride of per-feature partial sums
constexpr int kRowThreads = 256;                   // rows per tile in the row kernels
constexpr int kPartBlocks = 152;                   // fixed: the reductions' summation order never changes
constexpr int kPartBlocksFull = 64;                // the same for the full layout's normal equations
constexpr int kGramRows = 32;                      // rows per Φ tile in the normal equations
constexpr int kGramBlk = 4;                        // each thread owns a 4×4 block of ΦᵀΦ
constexpr int kGramThreads = 1024;                 // 4×4 blocks per CTA (CTAs along y split the blocks)
constexpr int kSolveThreads = 256;

__host__ __device__ constexpr int tri(int i) { return i * (i + 1) / 2; }
__host__ __device__ constexpr int gram_nb(int nf) { return (nf + kGramBlk - 1) / kGramBlk; }
__host__ __device__ constexpr int gram_pairs(int nf) { return tri(gram_nb(nf)); }
constexpr int kGramFeatPadFull = gram_nb(kFullFeat) * kGramBlk;  // 468

// Coefficients as the row kernels read them: linear terms padded with zeros to
// 29, quadratic terms packed (i, j <= i) over the first QG genes (16: the
// reference's layouts; 29: the full surface).
template <int QG>
struct CoefT {
    float c0;
    float lin[kMaxLin];
    float q[QG * (QG + 1) / 2];
};

template <int P>
__device__ __forceinline__ float in_prec(float x) {
    if constexpr (P == CSX_SG_BF16) return __bfloat162float(__float2bfloat16_rn(x));
    return x;
}

template <int P, int QG>
__device__ void load_coef(CoefT<QG> &s, const float *coef, int ng) {
    constexpr int nq = QG * (QG + 1) / 2;
    for (int i = threadIdx.x; i < 1 + kMaxLin + nq; i += blockDim.x) {
        float v;
        if (i == 0) {
            v = coef[0];
        } else if (i <= kMaxLin) {
            v = (i <= ng) ? coef[i] : 0.0f;
        } else {
            v = coef[1 + ng + (i - 1 - kMaxLin)];
        }
        reinterpret_cast<float *>(&s)[i] = in_prec<P>(v);
    }
}

// Stage rows [r0, r0 + kRowThreads) of the gene table into shared memory
// (coalesced), row stride `st` (odd, so a thread-per-row read is conflict
// free). Eight loads are in flight per thread: one at a time, the 29 loads of
// a full tile cost 29 trips to memory, two thirds of the row kernels' time.
__device__ void stage_rows(float *tile, const float *genes, int64_t n, int ldg, int ng, int st, int64_t r0) {
    const int rows = static_cast<int>((n - r0 < kRowThreads) ? (n - r0) : kRowThreads);
    const int total = rows * ng, step = static_cast<int>(blockDim.x);
    const int dr = step / ng, dk = step - dr * ng;
    const float *src = genes + r0 * static_cast<int64_t>(ldg);
    int idx = threadIdx.x, r = idx / ng, k = idx - r * ng;
    while (idx < total) {
        float v[8];
        int at[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            at[u] = -1;
            if (idx < total) {
                v[u] = src[r * static_cast<int64_t>(ldg) + k];
                at[u] = r * st + k;
            }
            idx += step;
            r += dr;
            k += dk;
            if (k >= ng) {
                k -= ng;
                ++r;
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (at[u] >= 0) tile[at[u]] = v[u];
    }
}

template <int P>
__device__ __forceinline__ void read_row(float (&g)[kMaxLin], const float *tile, int st, int ng) {
#pragma unroll
    for (int k = 0; k < kMaxLin; ++k) g[k] = (k < ng) ? in_prec<P>(tile[threadIdx.x * st + k]) : 0.0f;
}

// FP32 score. The reference layouts: linear terms, then the quadratic rows.
// The full surface: csx_screen.h's defined FMA order (the screen's score).
template <int QG>
__device__ __forceinline__ float score_f32(const CoefT<QG> &c, const float (&g)[kMaxLin]) {
    if constexpr (QG == kMaxLin) {
        float r = c.c0;
#pragma unroll
        for (int k = 0; k < kMaxLin; ++k) {
            float t = c.lin[k];
#pragma unroll
            for (int l = 0; l <= k; ++l) t = __fmaf_rn(c.q[tri(k) + l], g[l], t);
            r = __fmaf_rn(g[k], t, r);
        }
        return r;
    } else {
        float s = c.c0;
#pragma unroll
        for (int k = 0; k < kMaxLin; ++k) s = __fmaf_rn(c.lin[k], g[k], s);
#pragma unroll
        for (int i = 0; i < QG; ++i) {
            float t = 0.0f;
#pragma unroll
            for (int j = 0; j <= i; ++j) t = __fmaf_rn(c.q[tri(i) + j], g[j], t);
            s = __fmaf_rn(t, g[i], s);
        }
        return s;
    }
}

// ∂score/∂g_k = lin_k + Σ_{j<=k} q_kj g_j + Σ_{i>=k} q_ik g_i (k < QG).
template <int QG>
__device__ __forceinline__ void grad_f32(const CoefT<QG> &c, const float (&g)[kMaxLin], float (&d)[kMaxLin]) {
#pragma unroll
    for (int k = 0; k < kMaxLin; ++k) d[k] = c.lin[k];
#pragma unroll
    for (int i = 0; i < QG; ++i) {
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            const float q = c.q[tri(i) + j];
            d[i] = __fmaf_rn(q, g[j], d[i]);
            d[j] = __fmaf_rn(q, g[i], d[j]);
        }
    }
}

__host__ __device__ inline int stride_for(int ng) { return ((ng + 1) & 1) ? ng + 1 : ng + 2; }  // odd, >= ng + 1

template <int P, int QG>
__global__ void __launch_bounds__(kRowThreads) sg_forward_kernel(const float *__restrict__ coef, int ng,
                                                                 const float *__restrict__ genes, int64_t n,
                                                                 int ldg, float *__restrict__ score) {
    __shared__ CoefT<QG> c;
    extern __shared__ float tile[];
    const int st = stride_for(ng);
    load_coef<P, QG>(c, coef, ng);
    for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kRowThreads; r0 < n;
         r0 += static_cast<int64_t>(gridDim.x) * kRowThreads) {
        __syncthreads();
        stage_rows(tile, genes, n, ldg, ng, st, r0);
        __syncthreads();
        if (r0 + threadIdx.x < n) {
            float g[kMaxLin];
            read_row<P>(g, tile, st, ng);
            score[r0 + threadIdx.x] = score_f32(c, g);
        }
    }
}

template <int QG>
__global__ void __launch_bounds__(kRowThreads) sg_forward_f64_kernel(const double *__restrict__ coef, int ng,
                                                                     const float *__restrict__ genes, int64_t n,
                                                                     int ldg, double *__restrict__ score) {
    constexpr int nq = QG * (QG + 1) / 2;
    __shared__ double lin[kMaxLin], q[nq], c0;
    extern __shared__ float tile[];
    const int st = stride_for(ng);
    for (int i = threadIdx.x; i < 1 + kMaxLin + nq; i += blockDim.x) {
        if (i == 0) c0 = coef[0];
        else if (i <= kMaxLin) lin[i - 1] = (i <= ng) ? coef[i] : 0.0;
        else q[i - 1 - kMaxLin] = coef[1 + ng + (i - 1 - kMaxLin)];
    }
    for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kRowThreads; r0 < n;
         r0 += static_cast<int64_t>(gridDim.x) * kRowThreads) {
        __syncthreads();
        stage_rows(tile, genes, n, ldg, ng, st, r0);
        __syncthreads();
        if (r0 + threadIdx.x < n) {
            double g[kMaxLin];
#pragma unroll
            for (int k = 0; k < kMaxLin; ++k) g[k] = (k < ng) ? static_cast<double>(tile[threadIdx.x * st + k]) : 0.0;
            double s = c0;
#pragma unroll
            for (int k = 0; k < kMaxLin; ++k) s = fma(lin[k], g[k], s);
#pragma unroll
            for (int i = 0; i < QG; ++i) {
                double t = 0.0;
#pragma unroll
                for (int j = 0; j <= i; ++j) t = fma(q[tri(i) + j], g[j], t);
                s = fma(t, g[i], s);
            }
            score[r0 + threadIdx.x] = s;
        }
    }
}

template <int P, int QG>
__global__ void __launch_bounds__(kRowThreads) sg_grad_genes_kernel(const float *__restrict__ coef, int ng,
                                                                    const float *__restrict__ genes, int64_t n,
                                                                    int ldg, const float *__restrict__ gout,
                                                                    float *__restrict__ dgenes) {
    __shared__ CoefT<QG> c;
    extern __shared__ float tile[];
    const int st = stride_for(ng);
    load_coef<P, QG>(c, coef, ng);
    for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kRowThreads; r0 < n;
         r0 += static_cast<int64_t>(gridDim.x) * kRowThreads) {
        __syncthreads();
        stage_rows(tile, genes, n, ldg, ng, st, r0);
        __syncthreads();
        const int64_t r = r0 + threadIdx.x;
        float d[kMaxLin];
        if (r < n) {
            float g[kMaxLin];
            read_row<P>(g, tile, st, ng);
            grad_f32(c, g, d);
            const float go = gout[r];
#pragma unroll
            for (int k = 0; k < kMaxLin; ++k) d[k] = (k < ng) ? __fmul_rn(go, d[k]) : 0.0f;
        }
        __syncthreads();
        // write back through the tile so that the global stores are coalesced
        if (r < n) {
#pragma unroll
            for (int k = 0; k < kMaxLin; ++k)
                if (k < ng) tile[threadIdx.x * st + k] = d[k];
        }
        __syncthreads();
        const int64_t rows = (n - r0 < kRowThreads) ? (n - r0) : kRowThreads;
        const int total = static_cast<int>(rows) * ldg;
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int rr = idx / ldg, k = idx - rr * ldg;
            dgenes[r0 * ldg + idx] = (k < ng) ? tile[rr * st + k] : 0.0f;
        }
    }
}

// Feature f as a product x[a]·x[b] over x = [g_0 .. g_{ng-1}, 1].
__device__ __forceinline__ void feature_pair(int f, int ng, int &a, int &b) {
    if (f == 0) {
        a = ng;
        b = ng;
    } else if (f <= ng) {
        a = f - 1;
        b = ng;
    } else {
        int q = f - 1 - ng, i = 0;
        while (tri(i + 1) <= q) ++i;
        a = i;
        b = q - tri(i);
    }
}

// Per-block partial sums of Σ_r gout_r Φ_f(g_r), FP64, thread f per feature.
// The rows of a tile are staged 64 at a time as FP64: x = [g, 1] and, for an
// FP32 gout, h = gout x (48 bits: exact), so that a feature's term is one
// FMA(h_a, x_b, sum), the same real product rounded once as FMA(gout, x_a x_b,
// sum). The FP64 pipe (two lanes per SM) bounds it: converting both genes and
// multiplying them per feature took four of its operations where one does
// (100,003 rows of 29 genes: 210 µs). An FP64 gout keeps FMA(gout, x_a x_b):
// gout x_a would round.
constexpr int kCoefRows = 64;

template <typename TG>
__global__ void __launch_bounds__(kRowThreads) sg_grad_coef_kernel(int ng, int nf, const float *__restrict__ genes,
                                                                   int64_t n, int ldg, const TG *__restrict__ gout,
                                                                   double *__restrict__ part) {
    constexpr int kPer = (kFeatCap + kRowThreads - 1) / kRowThreads;  // features per thread (2)
    constexpr bool kF32 = sizeof(TG) == 4;
    constexpr int kX = kMaxLin + 1;
    __shared__ double xs[kCoefRows][kX], hs[kF32 ? kCoefRows : 1][kX];
    __shared__ double go_s[kCoefRows];
    int a[kPer], b[kPer];
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
        a[m] = b[m] = 0;
        const int f = threadIdx.x + m * kRowThreads;
        if (f < nf) feature_pair(f, ng, a[m], b[m]);
    }
    double acc[kPer] = {};
    const int nx = ng + 1;
    for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * kRowThreads; t0 < n;
         t0 += static_cast<int64_t>(gridDim.x) * kRowThreads) {
        const int64_t t1 = t0 + kRowThreads < n ? t0 + kRowThreads : n;
        for (int64_t r0 = t0; r0 < t1; r0 += kCoefRows) {
            const int rows = static_cast<int>(t1 - r0 < kCoefRows ? t1 - r0 : kCoefRows);
            __syncthreads();
#pragma unroll 8
            for (int idx = threadIdx.x; idx < rows * nx; idx += kRowThreads) {
                const int r = idx / nx, k = idx - r * nx;
                const double x = k < ng ? static_cast<double>(genes[(r0 + r) * static_cast<int64_t>(ldg) + k]) : 1.0;
                xs[r][k] = x;
                if (kF32) hs[kF32 ? r : 0][k] = static_cast<double>(gout[r0 + r]) * x;
            }
            if (!kF32 && threadIdx.x < rows) go_s[threadIdx.x] = static_cast<double>(gout[r0 + threadIdx.x]);
            __syncthreads();
#pragma unroll
            for (int m = 0; m < kPer; ++m) {
                if (threadIdx.x + m * kRowThreads < nf) {
#pragma unroll 4
                    for (int r = 0; r < rows; ++r)
                        acc[m] = kF32 ? fma(hs[kF32 ? r : 0][a[m]], xs[r][b[m]], acc[m])
                                      : fma(go_s[r], xs[r][a[m]] * xs[r][b[m]], acc[m]);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
        const int f = threadIdx.x + m * kRowThreads;
        if (f < nf) part[static_cast<int64_t>(blockIdx.x) * kFeatCap + f] = acc[m];
    }
}

// Sums of `nparts` partial results: eight threads per entry take every eighth
// part, so that the loads of one entry overlap (one thread per entry waited
// for 152 loads in turn: 21 µs for 153 entries, 27 for the normal equations').
constexpr int kSumSplit = 8;

__device__ __forceinline__ double sum_parts(const double *__restrict__ p, int nparts, int64_t stride, bool live,
                                            double (*s)[32]) {
    double v = 0.0;
    if (live) {
#pragma unroll 4
        for (int q = threadIdx.y; q < nparts; q += kSumSplit) v += p[q * stride];
    }
    s[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y != 0) return 0.0;
#pragma unroll
    for (int y = 1; y < kSumSplit; ++y) v += s[y][threadIdx.x];
    return v;
}

template <typename T>
__global__ void __launch_bounds__(32 * kSumSplit) sg_sum_parts_kernel(const double *__restrict__ part, int nparts,
                                                                      int stride, int nf, T *__restrict__ out) {
    __shared__ double s[kSumSplit][32];
    const int f = blockIdx.x * 32 + threadIdx.x;
    const double v = sum_parts(part + f, nparts, stride, f < nf, s);
    if (threadIdx.y == 0 && f < nf) out[f] = static_cast<T>(v);
}

struct GramRange;
__device__ __forceinline__ bool gram_fixed(const GramRange *r, int ng);

// Normal equations in FP64 (the full surface, and the tables that csx_gram.cuh
// leaves): thread t of CTA column y owns the 4×4 block number
// y·1024 + t, (bi, bj) with bj <= bi, of ΦᵀΦ; CTA row x accumulates rows of
// its chunk. Column 0's threads t < nf also accumulate (Φᵀy)_t. Φ for
// kGramRows rows is staged in shared memory in FP64 (exact: a product of two
// f32 genes), featpad = 4·ceil(nf/4) features per row.
__global__ void __launch_bounds__(kGramThreads) sg_gram_kernel(int ng, int nf, const float *__restrict__ genes,
                                                               int64_t n, int ldg, const double *__restrict__ fit,
                                                               double *__restrict__ part_g,
                                                               double *__restrict__ part_r,
                                                               const GramRange *__restrict__ range) {
    if (range && gram_fixed(range, ng)) return;  // sg_gram_mma_kernel's table
    extern __shared__ double phi[];  // [kGramRows][featpad]
    __shared__ float gs[kGramRows][kMaxLin + 1];
    __shared__ double ys[kGramRows];
    __shared__ unsigned char fa[kGramFeatPadFull], fb[kGramFeatPadFull];  // feature f = x[fa]·x[fb]
    const int nb = gram_nb(nf), featpad = nb * kGramBlk;
    const int npairs = tri(nb);
    const int t = threadIdx.x;
    for (int f = t; f < nf; f += blockDim.x) {
        int a, b;
        feature_pair(f, ng, a, b);
        fa[f] = static_cast<unsigned char>(a);
        fb[f] = static_cast<unsigned char>(b);
    }
    const int pt = blockIdx.y * kGramThreads + t;  // this thread's block number
    int bi = 0;
    while (tri(bi + 1) <= pt) ++bi;
    const int bj = pt - tri(bi);
    const bool owner = pt < npairs;
    const bool rhs_here = blockIdx.y == 0 && t < nf && fit;
    double acc[kGramBlk][kGramBlk] = {};
    double racc = 0.0;
    const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = static_cast<int64_t>(blockIdx.x) * chunk;
    const int64_t hi = (lo + chunk < n) ? lo + chunk : n;
    for (int64_t r0 = lo; r0 < hi; r0 += kGramRows) {
        const int rows = static_cast<int>((hi - r0 < kGramRows) ? hi - r0 : kGramRows);
        __syncthreads();
        for (int idx = t; idx < rows * ng; idx += blockDim.x) {
            const int r = idx / ng, k = idx - r * ng;
            gs[r][k] = genes[(r0 + r) * static_cast<int64_t>(ldg) + k];
        }
        if (t < rows) {
            gs[t][ng] = 1.0f;
            ys[t] = fit ? fit[r0 + t] : 0.0;
        }
        __syncthreads();
        for (int idx = t; idx < kGramRows * featpad; idx += blockDim.x) {
            const int r = idx / featpad, f = idx - r * featpad;
            double v = 0.0;
            if (r < rows && f < nf) v = static_cast<double>(gs[r][fa[f]]) * static_cast<double>(gs[r][fb[f]]);
            phi[idx] = v;
        }
        __syncthreads();
        if (owner) {
            for (int r = 0; r < rows; ++r) {
                const double *pr = phi + r * featpad;
                double xa[kGramBlk], xb[kGramBlk];
#pragma unroll
                for (int u = 0; u < kGramBlk; ++u) {
                    xa[u] = pr[bi * kGramBlk + u];
                    xb[u] = pr[bj * kGramBlk + u];
                }
#pragma unroll
                for (int u = 0; u < kGramBlk; ++u)
#pragma unroll
                    for (int v = 0; v < kGramBlk; ++v) acc[u][v] = fma(xa[u], xb[v], acc[u][v]);
            }
        }
        if (rhs_here) {
            for (int r = 0; r < rows; ++r) racc = fma(ys[r], phi[r * featpad + t], racc);
        }
    }
    if (owner) {
        double *dst = part_g + (static_cast<int64_t>(blockIdx.x) * npairs + pt) * (kGramBlk * kGramBlk);
#pragma unroll
        for (int u = 0; u < kGramBlk; ++u)
#pragma unroll
            for (int v = 0; v < kGramBlk; ++v) dst[u * kGramBlk + v] = acc[u][v];
    }
    if (rhs_here) part_r[static_cast<int64_t>(blockIdx.x) * kFeatCap + t] = racc;
}

__global__ void __launch_bounds__(32 * kSumSplit) sg_gram_sum_kernel(const double *__restrict__ part_g, int nparts,
                                                                     int nf, double *__restrict__ gram) {
    __shared__ double sp[kSumSplit][32];
    const int64_t e = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;  // (pair, u, v)
    const int npairs = gram_pairs(nf);
    const int64_t total = static_cast<int64_t>(npairs) * kGramBlk * kGramBlk;
    const double s = sum_parts(part_g + e, nparts, total, e < total, sp);
    if (threadIdx.y != 0 || e >= total) return;
    const int t = static_cast<int>(e / (kGramBlk * kGramBlk)), uv = static_cast<int>(e % (kGramBlk * kGramBlk));
    const int u = uv / kGramBlk, v = uv - u * kGramBlk;
    int bi = 0;
    while (tri(bi + 1) <= t) ++bi;
    const int bj = t - tri(bi);
    const int a = bi * kGramBlk + u, b = bj * kGramBlk + v;
    if (a >= nf || b >= nf) return;
    gram[static_cast<int64_t>(a) * nf + b] = s;
    gram[static_cast<int64_t>(b) * nf + a] = s;
}

// (G + αI) w = rhs + α·prior, FP64, by a square-root-free Cholesky
// factorisation (L D Lᵀ) of the matrix with the right side as one more row: at
// the end that row holds D⁻¹ L⁻¹ (rhs + α·prior), and only Lᵀ w = that is left
// to solve. A cluster of eight CTAs holds the packed rows in shared memory, row
// i in CTA i mod 8, and takes four columns per step: every CTA sends its rows'
// four entries to all (distributed shared memory), all meet at the cluster's
// barrier, each factors the 4×4 diagonal block and the columns' entries for
// itself and updates its own rows.
//
// What bounds it is the chain of pivots: a reciprocal and a few dependent
// FP64 operations per column (no square root, no division per row), then the
// barrier per four columns; the updates run on eight SMs' FP64 pipes (two
// lanes each).
constexpr int kSolveCtas = 8;
constexpr int kSolveNb = 4;

__host__ __device__ constexpr int solve_rows(int n, int r) {  // rows r, r + 8, ... <= n (n is the right side)
    return r <= n ? (n - r) / kSolveCtas + 1 : 0;
}
// Doubles before local row q (global row r + 8 q, r + 8 q + 1 long).
__host__ __device__ constexpr int solve_off(int r, int q) { return q * (r + 1) + kSolveCtas * (q * (q - 1) / 2); }
constexpr size_t solve_smem(int n) {  // the largest CTA's rows, two column buffers, L's columns, the scales, the copy for n <= 166
    return (static_cast<size_t>(solve_off(kSolveCtas - 1, solve_rows(n, 0))) + 2ull * (n + 1) * kSolveNb +
            static_cast<size_t>(n + 1) * kSolveNb + 4ull * (kFullFeat + 1) + 2 + (n <= kMaxFeat ? static_cast<size_t>(tri(n)) : 0u)) *
           sizeof(double);
}

// The power of two that brings a diagonal entry d into [1, 4) when it
// multiplies its row and its column. Rows and columns scaled by powers of two
// leave every rounding as it is, and no product of two entries of a panel can
// overflow or vanish (unscaled, u_ak u_bk of a matrix of 1e-170 was 0).
__device__ __forceinline__ double solve_scale(double d) {
    const int64_t bits = __double_as_longlong(d);
    const int64_t e = bits >> 52;  // sign and biased exponent
    if (e < 0 || e == 2047 || bits == 0) return 1.0;  // not positive definite: reported below
    return __longlong_as_double((1023 - ((e - 1023) >> 1)) << 52);
}

// 1 / d for a pivot: a float reciprocal of the significand's leading bits and
// two Newton steps x += x (1 - m x), then the exponent: four dependent FP64
// operations of 64 cycles each, where the division takes 565 cycles. Within
// 2^-52 of 1 / d (the two steps square the seed's 2^-22 twice, which leaves the
// last one's rounding); the division otherwise (zero, negative, subnormal, infinite, NaN, or a reciprocal
// near underflow). The float parts are read off and put back by integer
// operations: the conversions run on the FP64 pipe too.
__device__ __forceinline__ double pivot_rcp(double d) {
    const int64_t bits = __double_as_longlong(d);
    const int64_t e = bits >> 52;  // sign and biased exponent
    if (e < 2 || e > 2040) return 1.0 / d;
    const double m = __longlong_as_double((bits & 0x000fffffffffffffll) | 0x3ff0000000000000ll);
    const float mf = __uint_as_float(0x3f800000u | static_cast<uint32_t>((bits >> 29) & 0x7fffffu));
    const uint32_t xf = __float_as_uint(__frcp_rn(mf));  // in (1/2, 1]
    double x = __longlong_as_double((static_cast<int64_t>(xf) << 29) + (static_cast<int64_t>(1023 - 127) << 52));
    x = fma(x, fma(-m, x, 1.0), x);
    x = fma(x, fma(-m, x, 1.0), x);
    return __longlong_as_double(__double_as_longlong(x) - ((e - 1023) << 52));
}

// Lᵀ w = z by one CTA, 32 unknowns at a time from the last: within a block one
// warp takes an unknown per step, one FMA for all 32 lanes; then every warp
// takes the block's unknowns off the ones before it, a warp per 32 of them and
// half of the block. `row(i)` is L's row i; y and the scales sc have n entries in
// shared memory.
template <class RowFn>
__device__ void back_substitute(int n, double *y, double (*half)[kFullFeat + 1], const double *sc, RowFn row,
                                double *__restrict__ w) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i0 = (n - 1) & ~31; i0 >= 0; i0 -= 32) {
        const int cnt = min(32, n - i0);
        if (warp == 0) {
            double z = lane < cnt ? y[i0 + lane] : 0.0;
            double l = lane < cnt - 1 ? row(i0 + cnt - 1)[i0 + lane] : 0.0;
            for (int k = cnt - 1; k > 0; --k) {
                const double nxt = lane < k - 1 ? row(i0 + k - 1)[i0 + lane] : 0.0;  // the next step's entries
                const double wk = __shfl_sync(0xffffffffu, z, k);
                if (lane < k) z = fma(-l, wk, z);
                l = nxt;
            }
            if (lane < cnt) {
                y[i0 + lane] = z;
                w[i0 + lane] = z * sc[i0 + lane];
            }
        }
        __syncthreads();
        const int groups = i0 >> 5;  // of 32 unknowns before the block
        for (int t = warp; t < 2 * groups; t += kSolveThreads / 32) {
            const int j = (t >> 1) * 32 + lane, h = t & 1;
            const int k1 = min(cnt, 16 * h + 16);
            double s = 0.0;
#pragma unroll 8
            for (int k = 16 * h; k < k1; ++k) s = fma(row(i0 + k)[j], y[i0 + k], s);
            half[h][j] = s;
        }
        __syncthreads();
        for (int j = tid; j < i0; j += kSolveThreads) y[j] -= half[0][j] + half[1][j];
        __syncthreads();
    }
}

__global__ void __cluster_dims__(kSolveCtas, 1, 1) __launch_bounds__(kSolveThreads)
    sg_ridge_solve_kernel(int n, const double *__restrict__ gram, const double *__restrict__ rhs, double alpha,
                          const double *__restrict__ prior, double *__restrict__ w, int *status) {
    extern __shared__ __align__(16) double sm[];  // the panels are written as double2
    __shared__ double s_l[kSolveNb][kSolveNb], s_r[kSolveNb];
    cg::cluster_group cluster = cg::this_cluster();
    const int r = static_cast<int>(cluster.block_rank());
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrows = solve_rows(n, r);
    double *A = sm;                                              // this CTA's packed rows
    double *P = sm + ((solve_off(kSolveCtas - 1, solve_rows(n, 0)) + 1) & ~1);  // two buffers of (n + 1) x 4 column entries
    double *Lc = P + 2 * (n + 1) * kSolveNb;                     // the step's columns of L, all rows
    double *zs = Lc + (n + 1) * kSolveNb;                        // the last solve's unknowns
    auto *half = reinterpret_cast<double(*)[kFullFeat + 1]>(zs + kFullFeat + 1);
    double *sc = zs + 3 * (kFullFeat + 1);                       // the rows' scales
    double *Lfull = zs + 4 * (kFullFeat + 1);                    // n <= 166: L in one CTA for the last solve
    for (int j = tid; j < n; j += kSolveThreads) sc[j] = solve_scale(gram[static_cast<int64_t>(j) * n + j] + alpha);
    __syncthreads();
    for (int q = warp; q < nrows; q += kSolveThreads / 32) {
        const int i = r + kSolveCtas * q;
        double *row = A + solve_off(r, q);
        for (int j = lane; j <= i; j += 32) {
            double v;
            if (i < n) v = (gram[static_cast<int64_t>(i) * n + j] + (i == j ? alpha : 0.0)) * sc[i] * sc[j];
            else v = j < n ? (rhs[j] + (prior ? alpha * prior[j] : 0.0)) * sc[j] : 0.0;
            row[j] = v;
        }
    }
    int bad = 0;  // thread 0's count is the one reported
    cluster.sync();  // own rows are in, and every CTA runs before another writes its shared memory
    for (int k0 = 0, buf = 0; k0 < n; k0 += kSolveNb, buf ^= 1) {
        const int nb = min(kSolveNb, n - k0);
        double *Pb = P + buf * (n + 1) * kSolveNb;
        // own rows' entries of the four columns to every CTA
        const int q0 = k0 > r ? (k0 - r + kSolveCtas - 1) / kSolveCtas : 0;  // first own row >= k0
        for (int e = tid; e < (nrows - q0) * 2 * kSolveCtas; e += kSolveThreads) {  // two columns each
            const int c = 2 * (e & 1), dst = (e >> 1) & (kSolveCtas - 1), q = q0 + (e >> 4);
            const int i = r + kSolveCtas * q;
            const double *src = A + solve_off(r, q) + k0 + c;
            double2 v = make_double2(0.0, 0.0);
            if (c < nb && k0 + c <= i) v.x = src[0];
            if (c + 1 < nb && k0 + c + 1 <= i) v.y = src[1];
            *reinterpret_cast<double2 *>(cluster.map_shared_rank(Pb, dst) + i * kSolveNb + c) = v;
        }
        cluster.sync();
        // The 4x4 diagonal block by one warp, lane 4a + b with entry (a, b):
        // an FP64 instruction takes its 64 cycles whether one lane or all are
        // active, so the block's updates of one column are one instruction.
        if (warp == 0) {
            const int a = (lane >> 2) & 3, b = lane & 3;
            double v = a >= b && a < nb ? Pb[(k0 + a) * kSolveNb + b] : (a == b ? 1.0 : 0.0);
            double rc = 0.0;  // lane (a, k): 1 / d_k
#pragma unroll
            for (int k = 0; k < kSolveNb; ++k) {
                const double d = __shfl_sync(0xffffffffu, v, 5 * k);
                // u_ak u_bk while the reciprocal is on its way
                const double uu = __shfl_sync(0xffffffffu, v, 4 * a + k) * __shfl_sync(0xffffffffu, v, 4 * b + k);
                if (!(d > 0.0) && bad == 0) bad = k0 + k + 1;
                const double r = pivot_rcp(d);
                if (b == k) rc = r;
                if (b > k && a >= b) v = fma(-uu, r, v);
            }
            const double l = v * rc;  // a > b: l_ab = u_ab / d_b
            if (lane < 16) {
                if (a > b) s_l[a][b] = l;
                if (a == b) s_r[a] = rc;
            }
        }
        __syncthreads();
        // the columns below: u (undivided) back into the buffer, l = u / d beside it
        for (int i = k0 + tid; i <= n; i += kSolveThreads) {
            double u[kSolveNb];
#pragma unroll
            for (int c = 0; c < kSolveNb; ++c) u[c] = (c < nb && k0 + c <= i) ? Pb[i * kSolveNb + c] : 0.0;
#pragma unroll
            for (int c = 1; c < kSolveNb; ++c)
#pragma unroll
                for (int m = 0; m < c; ++m) u[c] = fma(-u[m], s_l[c][m], u[c]);
#pragma unroll
            for (int c = 0; c < kSolveNb; ++c) {
                Pb[i * kSolveNb + c] = u[c];
                Lc[i * kSolveNb + c] = u[c] * s_r[c];
            }
        }
        __syncthreads();
        for (int q = q0 + warp; q < nrows; q += kSolveThreads / 32) {
            const int i = r + kSolveCtas * q;
            double *row = A + solve_off(r, q);
            if (lane < nb && k0 + lane < i) row[k0 + lane] = Lc[i * kSolveNb + lane];  // L's entries stay in the row
            const double u0 = Pb[i * kSolveNb], u1 = Pb[i * kSolveNb + 1], u2 = Pb[i * kSolveNb + 2],
                         u3 = Pb[i * kSolveNb + 3];
            const int jend = i < n ? i : n - 1;
            for (int j = k0 + kSolveNb + lane; j <= jend; j += 32) {
                double v = row[j];
                v = fma(-u0, Lc[j * kSolveNb], v);
                v = fma(-u1, Lc[j * kSolveNb + 1], v);
                v = fma(-u2, Lc[j * kSolveNb + 2], v);
                v = fma(-u3, Lc[j * kSolveNb + 3], v);
                row[j] = v;
            }
        }
        __syncthreads();
    }
    cluster.sync();  // every row of L is final
    if (r == 0) {
        if (__syncthreads_or(bad))  // no weights from a factorisation that failed
            for (int j = tid; j < n; j += kSolveThreads) sc[j] = __longlong_as_double(0x7ff8000000000000ll);
        const double *zrow = cluster.map_shared_rank(A, n % kSolveCtas) + solve_off(n % kSolveCtas, n / kSolveCtas);
        for (int j = tid; j < n; j += kSolveThreads) zs[j] = zrow[j];
        if (n <= kMaxFeat) {  // L into this CTA, then the solve on local rows
            for (int i = warp; i < n; i += kSolveThreads / 32) {
                const double *src = cluster.map_shared_rank(A, i % kSolveCtas) + solve_off(i % kSolveCtas, i / kSolveCtas);
                for (int j = lane; j < i; j += 32) Lfull[tri(i) + j] = src[j];
            }
            __syncthreads();
            back_substitute(n, zs, half, sc, [&](int i) { return Lfull + tri(i); }, w);
        } else {
            __syncthreads();
            back_substitute(
                n, zs, half, sc,
                [&](int i) {
                    return cluster.map_shared_rank(A, i % kSolveCtas) + solve_off(i % kSolveCtas, i / kSolveCtas);
                },
                w);
        }
        if (tid == 0) *status = bad;
    }
    cluster.sync();  // no CTA leaves while its rows are read
}

// The rows an ascent reads and writes (the same ones in place); columns ng..cols
// are copied where they differ.
struct AscendRows {
    const float *in;
    float *out;
    int ldi, ldo, cols;
};

template <int QG>
__global__ void __launch_bounds__(kRowThreads) sg_ascend_kernel(const float *__restrict__ coef, int ng, AscendRows R,
                                                                int64_t n, float eta, int steps,
                                                                float *__restrict__ score) {
    __shared__ CoefT<QG> c;
    extern __shared__ float tile[];
    const int st = stride_for(ng);
    load_coef<CSX_SG_FP32, QG>(c, coef, ng);
    for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kRowThreads; r0 < n;
         r0 += static_cast<int64_t>(gridDim.x) * kRowThreads) {
        __syncthreads();
        stage_rows(tile, R.in, n, R.ldi, ng, st, r0);
        __syncthreads();
        const int64_t r = r0 + threadIdx.x;
        if (r < n) {
            float g[kMaxLin], d[kMaxLin];
            read_row<CSX_SG_FP32>(g, tile, st, ng);
            for (int s = 0; s < steps; ++s) {
                // keep the coefficient loads inside the loop: hoisted, the full
                // surface's 435 quadratic terms would not fit in registers
                asm volatile("" ::: "memory");
                grad_f32(c, g, d);
#pragma unroll
                for (int k = 0; k < kMaxLin; ++k)
                    if (k < ng) g[k] = fmaxf(fminf(__fmaf_rn(eta, d[k], g[k]), 1.0f), 0.0f);
            }
            if (score) score[r] = score_f32(c, g);
#pragma unroll
            for (int k = 0; k < kMaxLin; ++k)
                if (k < ng) tile[threadIdx.x * st + k] = g[k];
        }
        __syncthreads();
        const int64_t rows = (n - r0 < kRowThreads) ? (n - r0) : kRowThreads;
        const int total = static_cast<int>(rows) * ng;
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int rr = idx / ng, k = idx - rr * ng;
            R.out[(r0 + rr) * static_cast<int64_t>(R.ldo) + k] = tile[rr * st + k];
        }
        if (R.in != R.out && R.cols > ng) {
            const int more = R.cols - ng;
            for (int idx = threadIdx.x; idx < static_cast<int>(rows) * more; idx += blockDim.x) {
                const int rr = idx / more, k = ng + idx - rr * more;
                R.out[(r0 + rr) * static_cast<int64_t>(R.ldo) + k] = R.in[(r0 + rr) * static_cast<int64_t>(R.ldi) + k];
            }
        }
    }
}

// The same for few rows: sixteen lanes per row, lane k with gene k (its
// gradient's 16 coefficients in registers) and gene 16 + k, the row's genes
// exchanged by shuffles. One thread per row leaves most SMs without work below
// some ten thousand rows (5,120 rows: 20 CTAs). The gradient is accumulated in
// grad_f32's order, the score by the row's first lane in score_f32's, so the
// results are the same bits.
constexpr int kLaneRows = 16;  // rows per CTA
constexpr int64_t kLaneMaxRows = 30000;

__global__ void __launch_bounds__(kLaneRows * 16) sg_ascend_lanes_kernel(const float *__restrict__ coef, int ng,
                                                                         AscendRows R, int64_t n, float eta,
                                                                         int steps, float *__restrict__ score) {
    __shared__ CoefT<kQuadGenes> c;
    __shared__ float fin[kLaneRows][kMaxLin + 3];
    const int k = threadIdx.x & 15, rr = threadIdx.x >> 4;
    const int64_t r = static_cast<int64_t>(blockIdx.x) * kLaneRows + rr;
    const float *src = R.in + (r < n ? r : 0) * static_cast<int64_t>(R.ldi);
    float g0 = src[k], g1 = k + 16 < ng ? src[k + 16] : 0.0f;
    load_coef<CSX_SG_FP32, kQuadGenes>(c, coef, ng);
    __syncthreads();
    float q[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) q[l] = l <= k ? c.q[tri(k) + l] : c.q[tri(l) + k];
    const float w0 = c.lin[k], w1 = k + 16 < kMaxLin ? c.lin[k + 16] : 0.0f;
    for (int s = 0; s < steps; ++s) {
        float d = w0;
#pragma unroll
        for (int l = 0; l < 16; ++l) {
            const float x = __shfl_sync(0xffffffffu, g0, l, 16);
            d = __fmaf_rn(q[l], x, d);
            if (l == k) d = __fmaf_rn(q[l], x, d);  // the square's derivative: its term twice
        }
        g0 = fmaxf(fminf(__fmaf_rn(eta, d, g0), 1.0f), 0.0f);
        g1 = fmaxf(fminf(__fmaf_rn(eta, w1, g1), 1.0f), 0.0f);
    }
    if (r < n) {
        float *row = R.out + r * static_cast<int64_t>(R.ldo);
        row[k] = g0;
        if (k + 16 < ng) row[k + 16] = g1;
        if (R.in != R.out)
            for (int m = ng + k; m < R.cols; m += 16) row[m] = src[m];
        fin[rr][k] = g0;
        if (k + 16 < kMaxLin) fin[rr][k + 16] = k + 16 < ng ? g1 : 0.0f;
    }
    __syncwarp();
    if (score && r < n && k == 0) {
        float g[kMaxLin];
#pragma unroll
        for (int m = 0; m < kMaxLin; ++m) g[m] = fin[rr][m];
        score[r] = score_f32(c, g);
    }
}

}  // namespace

#include "csx_gram.cuh"

namespace {

#define SG_CUDA(call)                                                                       \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess) {                                                            \
            std::fprintf(stderr, "csx: %s failed: %s\n", #call, cudaGetErrorString(e_));   \
            return e_ == cudaErrorMemoryAllocation ? CSX_ERR_OOM : CSX_ERR_CUDA;             \
        }                                                                                   \
    } while (0)

// nf -> genes: the reference layouts (153..166: 16-gene quadratic block, ng
// genes linear) or the full surface (465: 29 genes, all quadratic).
int check_layout(int nf, int ldg, int64_t n, int &ng) {
    if (n < 0) return CSX_ERR_BAD_ARGS;
    if (nf == kFullFeat) {
        ng = kMaxLin;
    } else {
        if (nf < kMinFeat || nf > kMaxFeat) return CSX_ERR_BAD_ARGS;
        ng = nf - 1 - kNQuad;
    }
    if (ldg < ng) return CSX_ERR_BAD_ARGS;
    return CSX_OK;
}

bool is_full(int nf) { return nf == kFullFeat; }

int row_grid(int64_t n) {
    const int64_t tiles = (n + kRowThreads - 1) / kRowThreads;
    const int64_t cap = 152 * 8;
    return static_cast<int>(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
}

size_t tile_bytes(int ng) { return static_cast<size_t>(kRowThreads) * stride_for(ng) * sizeof(float); }

int gram_parts(int nf) { return is_full(nf) ? kPartBlocksFull : kPartBlocks; }
size_t part_gram_bytes(int nf) {
    return static_cast<size_t>(gram_parts(nf)) * gram_pairs(nf) * kGramBlk * kGramBlk * sizeof(double);
}
static_assert(kGmPartBytes + 15 <= static_cast<size_t>(kPartBlocks) * gram_pairs(kMaxFeat) * kGramBlk * kGramBlk * sizeof(double),
              "the fixed-point sums end before part_r");
constexpr size_t kPartCoefBytes = static_cast<size_t>(kPartBlocks) * kFeatCap * sizeof(double);
size_t gram_smem(int nf) { return static_cast<size_t>(kGramRows) * gram_nb(nf) * kGramBlk * sizeof(double); }

int enable_smem() {  // on the current device, every call (cheap)
    SG_CUDA(cudaFuncSetAttribute(sg_ridge_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(std::max(solve_smem(kMaxFeat), solve_smem(kFullFeat)))));
    SG_CUDA(cudaFuncSetAttribute(sg_gram_mma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kGmSmem)));
    SG_CUDA(cudaFuncSetAttribute(sg_gram_mma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kGmSmem)));
    SG_CUDA(cudaFuncSetAttribute(sg_gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(gram_smem(kFullFeat))));
    return CSX_OK;
}

template <typename TG, typename TD>
int coef_grad(int ng, int nf, const float *genes, int64_t n, int ldg, const TG *gout, TD *dcoef, void *work,
              cudaStream_t s) {
    if (!dcoef) return CSX_OK;
    if (!work) return CSX_ERR_BAD_ARGS;
    auto *part = static_cast<double *>(work);
    const int grid = static_cast<int>(n > 0 ? ((n + kRowThreads - 1) / kRowThreads < kPartBlocks
                                                   ? (n + kRowThreads - 1) / kRowThreads
                                                   : kPartBlocks)
                                            : 1);
    sg_grad_coef_kernel<TG><<<grid, kRowThreads, 0, s>>>(ng, nf, genes, n, ldg, gout, part);
    SG_CUDA(cudaGetLastError());
    sg_sum_parts_kernel<<<(nf + 31) / 32, dim3(32, kSumSplit), 0, s>>>(part, grid, kFeatCap, nf, dcoef);
    SG_CUDA(cudaGetLastError());
    return CSX_OK;
}

}  // namespace

extern "C" {

uint64_t csx_sg_workspace_bytes(int nf) {
    const size_t g = is_full(nf) ? part_gram_bytes(kFullFeat) : part_gram_bytes(kMaxFeat);
    return static_cast<uint64_t>(g + kPartCoefBytes);
}

int csx_sg_forward(const float *d_coef, int nf, const float *d_genes, int64_t n, int ldg, int precision,
                   float *d_score, void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, ldg, n, ng)) return rc;
    if (n == 0) return CSX_OK;
    if (!d_coef || !d_genes || !d_score) return CSX_ERR_BAD_ARGS;
    auto s = static_cast<cudaStream_t>(stream);
    const int grid = row_grid(n);
    const size_t tb = tile_bytes(ng);
    if (precision == CSX_SG_FP32) {
        if (is_full(nf))
            sg_forward_kernel<CSX_SG_FP32, kMaxLin><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg, d_score);
        else
            sg_forward_kernel<CSX_SG_FP32, kQuadGenes><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                    d_score);
    } else if (precision == CSX_SG_BF16) {
        if (is_full(nf))
            sg_forward_kernel<CSX_SG_BF16, kMaxLin><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg, d_score);
        else
            sg_forward_kernel<CSX_SG_BF16, kQuadGenes><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                    d_score);
    } else {
        return CSX_ERR_BAD_ARGS;
    }
    SG_CUDA(cudaGetLastError());
    return CSX_OK;
}

int csx_sg_forward_f64(const double *d_coef, int nf, const float *d_genes, int64_t n, int ldg, double *d_score,
                       void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, ldg, n, ng)) return rc;
    if (n == 0) return CSX_OK;
    if (!d_coef || !d_genes || !d_score) return CSX_ERR_BAD_ARGS;
    auto s = static_cast<cudaStream_t>(stream);
    if (is_full(nf))
        sg_forward_f64_kernel<kMaxLin><<<row_grid(n), kRowThreads, tile_bytes(ng), s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                      d_score);
    else
        sg_forward_f64_kernel<kQuadGenes><<<row_grid(n), kRowThreads, tile_bytes(ng), s>>>(d_coef, ng, d_genes, n,
                                                                                         ldg, d_score);
    SG_CUDA(cudaGetLastError());
    return CSX_OK;
}

}  // extern "C"

namespace {

template <typename TD>
int sg_backward(const float *d_coef, int nf, const float *d_genes, int64_t n, int ldg, int precision,
                const float *d_gout, float *d_dgenes, TD *d_dcoef, void *d_work, void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, ldg, n, ng)) return rc;
    if (precision != CSX_SG_FP32 && precision != CSX_SG_BF16) return CSX_ERR_BAD_ARGS;
    if (n > 0 && (!d_genes || !d_gout || (d_dgenes && !d_coef))) return CSX_ERR_BAD_ARGS;
    auto s = static_cast<cudaStream_t>(stream);
    if (d_dgenes && n > 0) {
        const int grid = row_grid(n);
        const size_t tb = tile_bytes(ng);
        const bool full = is_full(nf);
        if (precision == CSX_SG_FP32 && full)
            sg_grad_genes_kernel<CSX_SG_FP32, kMaxLin><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                    d_gout, d_dgenes);
        else if (precision == CSX_SG_FP32)
            sg_grad_genes_kernel<CSX_SG_FP32, kQuadGenes><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                       d_gout, d_dgenes);
        else if (full)
            sg_grad_genes_kernel<CSX_SG_BF16, kMaxLin><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                    d_gout, d_dgenes);
        else
            sg_grad_genes_kernel<CSX_SG_BF16, kQuadGenes><<<grid, kRowThreads, tb, s>>>(d_coef, ng, d_genes, n, ldg,
                                                                                       d_gout, d_dgenes);
        SG_CUDA(cudaGetLastError());
    }
    return coef_grad(ng, nf, d_genes, n, ldg, d_gout, d_dcoef, d_work, s);
}

}  // namespace

extern "C" {

int csx_sg_backward(const float *d_coef, int nf, const float *d_genes, int64_t n, int ldg, int precision,
                    const float *d_gout, float *d_dgenes, double *d_dcoef, void *d_work, void *stream) {
    return sg_backward(d_coef, nf, d_genes, n, ldg, precision, d_gout, d_dgenes, d_dcoef, d_work, stream);
}

int csx_sg_backward_f32(const float *d_coef, int nf, const float *d_genes, int64_t n, int ldg, int precision,
                        const float *d_gout, float *d_dgenes, float *d_dcoef, void *d_work, void *stream) {
    return sg_backward(d_coef, nf, d_genes, n, ldg, precision, d_gout, d_dgenes, d_dcoef, d_work, stream);
}

int csx_sg_backward_coef_f64(int nf, const float *d_genes, int64_t n, int ldg, const double *d_gout, double *d_dcoef,
                             void *d_work, void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, ldg, n, ng)) return rc;
    if (n > 0 && (!d_genes || !d_gout)) return CSX_ERR_BAD_ARGS;
    return coef_grad(ng, nf, d_genes, n, ldg, d_gout, d_dcoef, d_work, static_cast<cudaStream_t>(stream));
}

int csx_sg_normal_equations(int nf, const float *d_genes, int64_t n, int ldg, const double *d_fit, double *d_gram,
                            double *d_rhs, void *d_work, void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, ldg, n, ng)) return rc;
    if (!d_gram || !d_work || (n > 0 && !d_genes) || (d_fit && !d_rhs)) return CSX_ERR_BAD_ARGS;
    if (int rc = enable_smem()) return rc;
    auto s = static_cast<cudaStream_t>(stream);
    auto *part_g = static_cast<double *>(d_work);
    auto *part_r = reinterpret_cast<double *>(static_cast<char *>(d_work) + part_gram_bytes(is_full(nf) ? kFullFeat
                                                                                                          : kMaxFeat));
    const int npairs = gram_pairs(nf);
    const int ycols = (npairs + kGramThreads - 1) / kGramThreads;
    const int threads = ycols > 1 ? kGramThreads : ((npairs > nf ? npairs : nf) + 31) / 32 * 32;
    const int64_t want = (n + kGramRows - 1) / kGramRows;
    const int cap = gram_parts(nf);
    const int grid = static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
    GramRange *range = nullptr;
    if (!is_full(nf)) {
        range = reinterpret_cast<GramRange *>(reinterpret_cast<char *>(part_r) + kPartCoefBytes - sizeof(GramRange));
        // 16-byte entries in a workspace that is only asked to hold doubles: from
        // its next such boundary (they take 11 of the 17 MB before part_r)
        auto *part = reinterpret_cast<longlong2 *>((reinterpret_cast<uintptr_t>(d_work) + 15) & ~uintptr_t{15});
        SG_CUDA(cudaMemsetAsync(range, 0, sizeof(GramRange), s));
        sg_range_kernel<<<static_cast<unsigned>(std::min<int64_t>(n / 64 + 1, 152 * 4)), 256, 0, s>>>(
            ng, d_genes, n, ldg, d_fit, range);
        SG_CUDA(cudaGetLastError());
        const int64_t drain = kGmRows * kGmDrain;
        const int chunks = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(kGmChunks, (n + drain - 1) / drain)));
        const bool stack = kPairRows + ng - 16 + 2 <= 64;
        (stack ? sg_gram_mma_kernel<true> : sg_gram_mma_kernel<false>)<<<dim3(chunks, kGmBlocks), kGmThreads, kGmSmem, s>>>(
            ng, nf, d_genes, n, ldg, d_fit, range, part);
        SG_CUDA(cudaGetLastError());
        const int total = tri(nf) + (d_fit ? nf : 0);
        double *rhs = d_fit ? d_rhs : nullptr;
        sg_gram_final_kernel<<<(total + 31) / 32, dim3(32, kSumSplit), 0, s>>>(
            ng, nf, chunks, kGmSmall * std::sqrt(static_cast<double>(n)), range, part, d_gram, rhs);
        SG_CUDA(cudaGetLastError());
        // these two leave at once where the fixed-point sums stand
        sg_gram_kernel<<<dim3(grid, ycols), threads, gram_smem(nf), s>>>(ng, nf, d_genes, n, ldg, d_fit, part_g, part_r,
                                                                        range);
        SG_CUDA(cudaGetLastError());
        sg_gram_fp64_final_kernel<<<(total + 31) / 32, dim3(32, kSumSplit), 0, s>>>(ng, nf, range, part_g, part_r, grid,
                                                                                   d_gram, rhs);
        SG_CUDA(cudaGetLastError());
        return CSX_OK;
    }
    sg_gram_kernel<<<dim3(grid, ycols), threads, gram_smem(nf), s>>>(ng, nf, d_genes, n, ldg, d_fit, part_g, part_r,
                                                                    nullptr);
    SG_CUDA(cudaGetLastError());
    const int64_t ne = static_cast<int64_t>(npairs) * kGramBlk * kGramBlk;
    sg_gram_sum_kernel<<<static_cast<unsigned>((ne + 31) / 32), dim3(32, kSumSplit), 0, s>>>(part_g, grid, nf, d_gram);
    SG_CUDA(cudaGetLastError());
    if (d_fit) {
        sg_sum_parts_kernel<<<(nf + 31) / 32, dim3(32, kSumSplit), 0, s>>>(part_r, grid, kFeatCap, nf, d_rhs);
        SG_CUDA(cudaGetLastError());
    }
    return CSX_OK;
}

int csx_sg_ridge_solve(int nf, const double *d_gram, const double *d_rhs, double alpha, const double *d_prior,
                       double *d_w, int *d_status, void *stream) {
    if (nf < 1 || (nf > kMaxFeat && nf != kFullFeat) || !d_gram || !d_rhs || !d_w || !d_status || !(alpha >= 0.0))
        return CSX_ERR_BAD_ARGS;
    if (int rc = enable_smem()) return rc;
    auto s = static_cast<cudaStream_t>(stream);
    sg_ridge_solve_kernel<<<kSolveCtas, kSolveThreads, solve_smem(nf), s>>>(nf, d_gram, d_rhs, alpha, d_prior, d_w,
                                                                            d_status);
    SG_CUDA(cudaGetLastError());
    return CSX_OK;
}

static int sg_ascend(const float *d_coef, int nf, const AscendRows &R, int64_t n, float eta, int steps,
                     float *d_score, void *stream) {
    int ng = 0;
    if (int rc = check_layout(nf, R.ldi < R.ldo ? R.ldi : R.ldo, n, ng)) return rc;
    if (steps < 0 || R.cols < ng || R.cols > R.ldi || R.cols > R.ldo) return CSX_ERR_BAD_ARGS;
    if (n == 0) return CSX_OK;
    if (!d_coef || !R.in || !R.out) return CSX_ERR_BAD_ARGS;
    auto s = static_cast<cudaStream_t>(stream);
    if (is_full(nf))
        sg_ascend_kernel<kMaxLin><<<row_grid(n), kRowThreads, tile_bytes(ng), s>>>(d_coef, ng, R, n, eta, steps, d_score);
    else if (n <= kLaneMaxRows)
        sg_ascend_lanes_kernel<<<static_cast<unsigned>((n + kLaneRows - 1) / kLaneRows), kLaneRows * 16, 0, s>>>(
            d_coef, ng, R, n, eta, steps, d_score);
    else
        sg_ascend_kernel<kQuadGenes><<<row_grid(n), kRowThreads, tile_bytes(ng), s>>>(d_coef, ng, R, n, eta, steps,
                                                                                     d_score);
    SG_CUDA(cudaGetLastError());
    return CSX_OK;
}

int csx_sg_ascend(const float *d_coef, int nf, float *d_genes, int64_t n, int ldg, float eta, int steps,
                  float *d_score, void *stream) {
    return sg_ascend(d_coef, nf, AscendRows{d_genes, d_genes, ldg, ldg, ldg}, n, eta, steps, d_score, stream);
}

int csx_sg_ascend_to(const float *d_coef, int nf, const float *d_genes, int64_t n, int ldg, int cols, float eta,
                     int steps, float *d_out, int ldo, float *d_score, void *stream) {
    return sg_ascend(d_coef, nf, AscendRows{d_genes, d_out, ldg, ldo, cols}, n, eta, steps, d_score, stream);
}

}  // extern "C"
