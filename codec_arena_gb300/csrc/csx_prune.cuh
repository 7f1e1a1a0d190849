// csx_prune.cuh — the pruning screen: a certified upper bound of each
// candidate's score from its parents and crossover bits, taken before its
// mutation draws, so that a candidate which cannot reach the top-K skips them.
// Part of csx_screen.cu's translation unit (included there, in order); not a
// standalone header.
//
// The reference scores every candidate in full (src/screen.zig:225-253: two
// parent draws, the immigrant test, 29 x (crossover bit + mutation unit), the
// jump test, Model.score). Here a candidate is judged in three steps, each only
// for what the one before could not rule out:
//   1. its four header draws (parents, immigrant, jump) and a table with an
//      upper bound of every parent pair, over all crossover masks;
//   2. its 16 crossover bits (and jump value): the bound of its own mask;
//   3. the full synthesis and the score in the reference's f32 order.
// A candidate is skipped only when its score is certainly below the K-th score
// of candidates already screened, so the survivors, their scores and the
// screened count are those of the reference's run.
//
// The bound. Gene k of a crossover candidate is g_k = clamp01(par_k + d_k)
// with par_k the parent's gene chosen by the crossover bit and |d_k| <=
// |sigma|; with y_k = clamp01(par_k) and s = |sigma| + 2^-24 (the rounding of
// par_k + d_k where it is not clamped), g_k lies in [max(0, y_k - s), min(1,
// y_k + s)]: a box of centre c_k and radius r_k (clamp01 is monotone and
// 1-Lipschitz). The surface is the quadratic
//   f(g) = 16 w0 + sum_k w_k g_k + sum_{j<=i<16} Q_ij g_i g_j,
// so with u = g - c over the first 16 genes:
//   f(g) = f(c) + grad f(c) . u + sum_{j<=i<16} Q_ij u_i u_j + tail
//        <= f(c) + sum_k |grad_k f(c)| r_k + sum_k d_k r_k^2 + tail
// for any d >= 0 with diag(d) - Q positive semidefinite (quad_diag: about half
// of sum_i max(Q_ii, 0) r_i^2 + sum_{j<i} |Q_ij| r_i r_j, which d_k = Q_kk +
// sum_{j != k} |Q_kj| / 2 gives, and the pairs the table leaves fall from 12 to
// 9% on the committed surface, from 30 to 23% on a seeded 153-term one).
// grad f(c) = w + Qs c (Qs = Q + Q^T); the tail sum_{k>=16} w_k g_k is taken at
// its largest over both parents' boxes. A jump to value v at gene j < 16 is a
// box of centre v and radius 0; past gene 15 it raises f by at most
// JumpBound::c[j]. The bounds are evaluated in f32; PruneConst::err covers
// their rounding and the reference order's (a candidate's f32 score is within
// gamma_35 * A of its real value), so a candidate is skipped only when
//   bound + err < K-th score.
//
// What bounds it: the instruction issue. One bound per candidate with its
// gradient on the tensor cores (787 instructions per candidate, 20 of its 36
// hashes) screened 2.65e9 candidates (64 elites, committed surface, sigma
// 0.12, top 256) in 63.7 ms; the pair table leaves four hashes for nine
// candidates in ten: 32.1 ms. 1e8 candidates of 96 elites: 3.09 -> 1.89 ms;
// 3.3e8 with a linear tail: 11.1 -> 4.4 ms.
#pragma once

namespace csx {

constexpr int kPruneMs = 3;  // order statistics each CTA publishes (publish_first)
// Candidates per thread between the CTA's barriers, and outer rounds between
// merges of a non-empty buffer.
constexpr int kPruneRounds = 64;
constexpr uint32_t kPruneMergeRounds = 4;
// Rounds without the bounds (screen_p_kernel): a warp whose CTA's queue is full
// within kPruneQuick candidates per thread was left a third or more of them; a
// round without is 2^1 .. 2^(kPruneDirect - 1) candidates per thread.
constexpr int kPruneQuick = 6;
constexpr uint32_t kPruneDirect = 8;
// kGolden's inverse modulo 2^64: a draw offset back from its state.
constexpr uint64_t golden_inverse() {
    uint64_t x = kGolden;  // correct to 3 bits; each Newton step doubles them
    for (int i = 0; i < 5; ++i) x *= 2 - kGolden * x;
    return x;
}
constexpr uint64_t kGoldenInv = golden_inverse();
static_assert(kGolden * kGoldenInv == 1, "inverse modulo 2^64");

struct PruneConst {
    float qs[16][16];  // Qs = Q + Q^T (Qs_kk = 2 Q_kk): grad of the quadratic block is Qs x
    float d[16];       // diag(d) - Q is positive semidefinite (quad_diag)
    float s;           // half-width of a gene's mutation box around its clamped parent gene
    float err;         // bound rounding + reference-order rounding, rounded up
};

struct PruneArgs : ScreenArgs {
    PruneConst pc;
    const uint32_t *box;  // ne x 16: each elite gene's mutation box, half2 (centre, radius)
    const float *u0;      // ne x ne: pair_bound_kernel's bound of every mask of a parent pair
    const float *t1;      // its bounds of the masks that agree on k1 genes: pair_index x 2^k1
    uint64_t goff[8];     // draw offset (x kGolden) of those genes' crossover bits
    uint32_t k1;
    const float *tmax;    // ne x ne: the linear tail's largest value over a pair (null without a tail)
    uint32_t *pub;        // kPruneMs x gridDim.x: okey of each CTA's m-th, 2m-th and 4m-th best entry
    uint32_t el_smem;     // 1: the elite table is copied to shared memory (prune_el_smem)
    uint32_t bm_words;    // words of the pair bitmap in shared memory (0: the pair table is read directly)
    uint32_t bm_period;   // rounds (outer) between its rebuilds, a power of two
};

// FP64 score of a queued candidate for the precision form, out of line. Its
// full synthesis, jump applied, is scored by the FFMA filter first (within
// ScreenArgs::err of the real score); only a candidate the filter cannot
// place below tlo = threshold - err is scored in FP64 (rounded to f32, which
// err covers as well): the FP64 pipe runs at a small fraction of the FP32
// rate. A filtered-out candidate returns -inf.
__device__ __noinline__ float prune_rescore64(const ScreenArgs *__restrict__ A, const float *el, uint64_t seed_t,
                                              uint64_t p, float tlo) {
    const CandHead h = cand_head(A->sc, seed_t, p);
    const float sf = synth_score<true, false, false, DevModel, true>(A->m, A->sc, el, seed_t, p, h, nullptr);
    if (sf < tlo) return -INFINITY;
    return static_cast<float>(score64_at<true>(&A->m, &A->sc, el, seed_t, p));  // out of line: own registers
}

// Score of a queued candidate: the reference's f32 order (out of line), or
// the precision form's FP64 score.
template <bool kFp64>
__device__ __forceinline__ float prune_rescore(const ScreenArgs *__restrict__ A, const float *el, uint64_t seed_t,
                                               uint64_t p, float tlo) {
    if (!kFp64) return exact_score_at<true>(A, el, seed_t, p);
    return prune_rescore64(A, el, seed_t, p, tlo);
}

// The filter's score of one candidate, its jump applied (within ScreenArgs::err of
// the real score), out of line: for the rounds that score without the bounds.
__device__ __noinline__ float filter_score_at(const ScreenArgs *__restrict__ A, const float *el, uint64_t seed_t,
                                              uint64_t p) {
    const CandHead h = cand_head(A->sc, seed_t, p);
    return synth_score<true, false, false, DevModel, true>(A->m, A->sc, el, seed_t, p, h, nullptr);
}

// The j-th largest (1-based) of v[0..n), by one warp (every lane calls):
// bisection on the 32-bit key, the largest x with #{v >= x} >= j.
__device__ __forceinline__ uint32_t warp_kth_largest(const uint32_t *v, uint32_t n, uint32_t j) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t prefix = 0;
    for (int b = 31; b >= 0; --b) {
        const uint32_t cand = prefix | (1u << b);
        uint32_t c = 0;
        for (uint32_t i = lane; i < n; i += 32) c += (v[i] >= cand) ? 1u : 0u;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= j) prefix = cand;
    }
    return prefix;
}

// The first of the list positions m, 2m, 4m that each CTA publishes: the
// smallest power of two of which the grid's CTAs can cover K (1 up to one
// survivor per CTA: the 1st, 2nd and 4th best; past four survivors per CTA m
// alone). With the 1st, 2nd and 4th whatever K, lists past four survivors per
// CTA had only a CTA's own threshold: 2,047 of 5e7 candidates scored 41% of them
// in 4.4 ms instead of 5% in 1.2 (full surface: 97% in 7.1, 16% in 3.5).
__device__ __forceinline__ uint32_t publish_first(uint32_t keep) {
    uint32_t m = 1;
    while (static_cast<uint64_t>(m) * gridDim.x < keep) m <<= 1;
    return m;
}

template <class Args>
__device__ __noinline__ void prune_merge(const Args *A, Entry *E, uint32_t *sel, uint32_t bn, unsigned int *s_buf_n,
                                         unsigned long long *s_t1, unsigned long long *s_t2, float *s_ts) {
    const uint32_t tid = threadIdx.x;
    cta_merge_top(E, A->kpad, A->sort_n, bn);
    if (tid == 0) {
        *s_buf_n = 0;
        const Entry kth = E[A->keep - 1];
        if (kth.k1 != 0ull) {
            *s_t1 = kth.k1;
            *s_t2 = kth.k2;
            const unsigned int ok = static_cast<unsigned int>(kth.k1 >> 32);
            *s_ts = okey_score(ok);
            atomicMax(&A->ctrl->gtau, ok);
        }
    }
    const uint32_t m0 = publish_first(A->keep);
    if (tid < kPruneMs && (m0 << tid) <= A->keep) {
        const unsigned int ok = static_cast<unsigned int>(E[(m0 << tid) - 1].k1 >> 32);
        if (ok != 0u) atomicMax(&A->pub[tid * gridDim.x + blockIdx.x], ok);
    }
    __syncthreads();
    if (tid < 32) {
        uint32_t best = 0;
        for (int mi = 0; mi < kPruneMs; ++mi) {
            const uint32_t m = m0 << mi, jm = (A->keep + m - 1) / m;
            if (m > A->keep || (mi > 0 && m > 4)) continue;
            const volatile uint32_t *src = A->pub + mi * gridDim.x;
            for (uint32_t i = tid; i < gridDim.x; i += 32) sel[i] = src[i];
            __syncwarp();
            best = max(best, warp_kth_largest(sel, gridDim.x, jm));
            __syncwarp();
        }
        if (tid == 0 && best != 0u) atomicMax(&A->ctrl->gtau, best);
    }
}

// ---- the parent pairs' bounds ------------------------------------------------------

// Each elite gene's mutation box [max(0, y - s), min(1, y + s)], y the
// clamped gene, as FP16 (centre, radius): the radius, rounded up, reaches both
// ends of the box from the rounded centre.
__global__ void prune_box_kernel(const float *__restrict__ tab, int ne, float s, uint32_t *__restrict__ box) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ne * 16) return;
    const float y = fmaxf(fminf(tab[(i >> 4) * kNtot + (i & 15)], 1.0f), 0.0f);  // +inf (NaN gene) -> 1
    const float lo = fmaxf(__fsub_rd(y, s), 0.0f), hi = fminf(__fadd_ru(y, s), 1.0f);
    const __half c = __float2half_rn(0.5f * (lo + hi));
    const float cf = __half2float(c);
    const __half r = __float2half_ru(fmaxf(__fsub_ru(hi, cf), __fsub_ru(cf, lo)));
    const __half2 h = __halves2half2(c, r);
    box[i] = *reinterpret_cast<const uint32_t *>(&h);
}

// Upper bounds of the real score of the crossover candidates of parents a, b
// (no jump), their own f32 rounding added: t1 over the masks that agree on the
// first k1 genes, u0 over all masks. The genes are taken in the order `perm`
// (the ones that matter most first); the masks of the first n_enum are
// enumerated and the others take the hull of both parents' boxes:
//   max over masks of [f(c) + sum |grad_k f(c)| r_k] + sum d_k r_k^2 + tail.
// A pair and its mirror have the same masks (complemented), so a <= b is
// evaluated once. A group of 2^(k1 - 5) x 16 threads takes a pair: each thread
// fixes genes 5..k1-1, takes every 16th value of the enumerated genes from k1
// on, and walks the first five in Gray order, where a flip updates the
// gradient by 16 FMAs and the value by two; its 32 maxima meet the other
// threads' in shared memory.
constexpr int kPairGray = 5;   // genes walked in Gray order per thread
constexpr int kPairUps = 16;   // threads that share the enumerated genes from k1 on
constexpr int kMaxMaskGenes = 8;

struct PairArgs {
    float qs[16][16];  // Qs in `perm` order
    float lin[16];     // linear weights in that order
    float d[16];       // PruneConst::d in that order
    float tl[kNtot - 16];
    float w16, s, err;
    const float *tab;
    const uint32_t *box;
    float *u0, *t1, *tmax;
    int ne, n_enum, k1, tail;
    uint8_t perm[16];
};

// Index of the unordered pair {a, b} among a <= b.
__host__ __device__ __forceinline__ uint32_t pair_index(uint32_t a, uint32_t b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    return hi * (hi + 1) / 2 + lo;
}

__global__ void __launch_bounds__(128, 3) pair_bound_kernel(const __grid_constant__ PairArgs A) {
    __shared__ uint32_t s_best[(128 / kPairUps) << kPairGray];  // okey of each pair's 2^k1 entries
    __shared__ uint32_t s_top[128 / kPairUps];
    const uint32_t tid = threadIdx.x;
    const uint32_t low_log2 = static_cast<uint32_t>(A.k1 - kPairGray);
    const uint32_t g_log2 = low_log2 + 4;  // threads per pair: 2^low x kPairUps
    const uint32_t slot = tid >> g_log2, sub = tid & ((1u << g_log2) - 1u);
    const uint32_t low = sub & ((1u << low_log2) - 1u), up = sub >> low_log2;
    const uint32_t n_slots = 128u >> g_log2;
    for (uint32_t i = tid; i < (n_slots << A.k1); i += 128) s_best[i] = 0u;
    if (tid < n_slots) s_top[tid] = 0u;
    __syncthreads();
    const uint32_t n_pairs = static_cast<uint32_t>(A.ne) * (A.ne + 1) / 2;
    const uint32_t pair = blockIdx.x * n_slots + slot;
    const bool mine = pair < n_pairs;
    uint32_t a = 0, b = 0;  // pair = b (b + 1) / 2 + a, a <= b
    if (mine) {
        b = static_cast<uint32_t>((sqrt(8.0 * pair + 1.0) - 1.0) * 0.5);
        while (b * (b + 1) / 2 > pair) --b;
        while ((b + 1) * (b + 2) / 2 <= pair) ++b;
        a = pair - b * (b + 1) / 2;
    }
    float c[16], r[16], d[16];  // centre under parent a (or the hull's), radius, centre of b minus centre of a
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const uint32_t wa = A.box[a * 16 + A.perm[q]], wb = A.box[b * 16 + A.perm[q]];
        const float2 fa = __half22float2(*reinterpret_cast<const __half2 *>(&wa));
        const float2 fb = __half22float2(*reinterpret_cast<const __half2 *>(&wb));
        if (q < A.n_enum) {
            c[q] = fa.x;
            d[q] = fb.x - fa.x;  // exact: FP16 values in [0, 1]
            r[q] = fmaxf(fa.y, fb.y);
        } else {
            const float lo = fminf(__fsub_rd(fa.x, fa.y), __fsub_rd(fb.x, fb.y));
            const float hi = fmaxf(__fadd_ru(fa.x, fa.y), __fadd_ru(fb.x, fb.y));
            c[q] = 0.5f * (lo + hi);
            d[q] = 0.0f;
            r[q] = fmaxf(__fsub_ru(hi, c[q]), __fsub_ru(c[q], lo));
        }
    }
    float best[1 << kPairGray];  // by the first five genes' mask
#pragma unroll
    for (int i = 0; i < (1 << kPairGray); ++i) best[i] = -INFINITY;
    const uint32_t n_up = mine ? 1u << (A.n_enum - A.k1) : 0u;
    for (uint32_t u = up; u < n_up; u += kPairUps) {
        const uint32_t hi = (u << low_log2) | low;  // genes 5.. of the mask
        float x[16], g[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            x[q] = c[q];
            if (q >= kPairGray && ((hi >> (q - kPairGray)) & 1u)) x[q] = c[q] + d[q];
            g[q] = A.lin[q];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k)
#pragma unroll
            for (int q = 0; q < 16; ++q) g[q] = __fmaf_rn(A.qs[k][q], x[k], g[q]);
        float f = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; ++q) f = __fmaf_rn(x[q], A.lin[q] + g[q], f);
        f = __fmaf_rn(0.5f, f, A.w16);
#pragma unroll
        for (int st = 0; st < (1 << kPairGray); ++st) {
            if (st > 0) {  // Gray code: flip gene ctz(st)
                const int q = (st & 1) ? 0 : (st & 2) ? 1 : (st & 4) ? 2 : (st & 8) ? 3 : 4;
                const bool back = ((st >> (q + 1)) & 1) != 0;  // the bit was set: return to parent a
                const float e = back ? -d[q] : d[q];
                f = __fmaf_rn(e, __fmaf_rn(0.5f * A.qs[q][q], e, g[q]), f);
#pragma unroll
                for (int k = 0; k < 16; ++k) g[k] = __fmaf_rn(A.qs[q][k], e, g[k]);
            }
            float v = f;
#pragma unroll
            for (int q = 0; q < 16; ++q) v = __fmaf_rn(fabsf(g[q]), r[q], v);
            best[st ^ (st >> 1)] = fmaxf(best[st ^ (st >> 1)], v);
        }
    }
    if (up < n_up) {
        float top = -INFINITY;
#pragma unroll
        for (int i = 0; i < (1 << kPairGray); ++i) {
            top = fmaxf(top, best[i]);
            atomicMax(&s_best[(slot << A.k1) + (low << kPairGray) + i], score_okey(best[i]));
        }
        atomicMax(&s_top[slot], score_okey(top));
    }
    __syncthreads();
    if (!mine) return;
    float q2 = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) q2 = __fmaf_ru(A.d[i], __fmul_ru(r[i], r[i]), q2);
    float tl = 0.0f;
    if (A.tail) {
#pragma unroll
        for (int k = 16; k < kNtot; ++k) {
            const float ya = fmaxf(fminf(A.tab[a * kNtot + k], 1.0f), 0.0f);
            const float yb = fmaxf(fminf(A.tab[b * kNtot + k], 1.0f), 0.0f);
            const float w = A.tl[k - 16];
            const float y = w >= 0.0f ? fminf(__fadd_ru(fmaxf(ya, yb), A.s), 1.0f)
                                      : fmaxf(__fsub_rd(fminf(ya, yb), A.s), 0.0f);
            tl = __fmaf_ru(w, y, tl);
        }
    }
    const float add = q2 + tl + A.err;
    for (uint32_t i = sub; i < (1u << A.k1); i += 1u << g_log2)
        A.t1[(static_cast<size_t>(pair) << A.k1) + i] = okey_score(s_best[(slot << A.k1) + i]) + add;
    if (sub == 0) {
        const float v = okey_score(s_top[slot]) + add;
        A.u0[a * A.ne + b] = v;
        A.u0[b * A.ne + a] = v;
        if (A.tail) {
            A.tmax[a * A.ne + b] = tl;
            A.tmax[b * A.ne + a] = tl;
        }
    }
}

// ---- the pruning screen ------------------------------------------------------------

// Per-warp queues: candidates whose parent pair the table cannot rule out,
// and those whose first k1 crossover bits cannot either (or that jump).
constexpr uint32_t kWqCap = 64;
struct WarpQueue {
    uint4 q1[kWqCap];   // splitmix64 state of the candidate's first draw, its index in the item,
    uint4 q2[kWqCap];   //   ea | eb << 11 | immigrant << 30 | jump << 31
    uint32_t i1[kWqCap], i2[kWqCap];  // its item
};

// A candidate by its header draws: parents, immigrant, jump, and the state of
// the next candidate's first draw (the jump test's draw ends a candidate without
// one).
struct PairHead {
    uint32_t ea, eb;
    bool imm, jump;
    uint64_t next;
};

__device__ __forceinline__ PairHead pair_head(const SynthConst &C, bool pow2, uint64_t s0) {
    PairHead h;
    const uint32_t xa = draw_hi(s0), xb = draw_hi(s0 + kGolden);
    if (pow2) {
        h.ea = xa & (C.ne - 1);
        h.eb = xb & (C.ne - 1);
    } else {
        h.ea = fastmod_u32(xa, C.ne_magic, C.ne);
        h.eb = fastmod_u32(xb, C.ne_magic, C.ne);
    }
    h.imm = (draw_vh(s0 + 2 * kGolden) >> 8) < C.imm_thr;
    const uint64_t sj = s0 + (h.imm ? 32u : 61u) * kGolden;
    h.jump = (draw_vh(sj) >> 8) < C.jump_thr;
    h.next = sj + (h.jump ? 3u : 1u) * kGolden;
    return h;
}

__device__ __forceinline__ uint32_t pair_meta(const PairHead &h) {
    return h.ea | (h.eb << 11) | (h.imm ? 1u << 30 : 0u) | (h.jump && !h.imm ? 1u << 31 : 0u);
}

// Whether the bound of the masks that agree with the candidate's first k1
// crossover bits, plus what its jump can add (a jump past gene 15 adds nothing
// without a tail), leaves it a chance at tlo.
__device__ __forceinline__ bool mask_passes(const PruneArgs &A, uint64_t s0, uint32_t meta, float tlo) {
    const uint32_t ea = meta & 2047u, eb = (meta >> 11) & 2047u;
    float jc = 0.0f;
    if (meta >> 31) jc = A.jb.c[draw_hi(s0 + 62 * kGolden) % 29u];
    uint32_t mask = 0;
#pragma unroll
    for (uint32_t k = 0; k < kMaxMaskGenes; ++k)
        if (k < A.k1) mask |= (draw_bitword(s0 + A.goff[k]) >> 31) << k;
    if (ea > eb) mask ^= (1u << A.k1) - 1u;
    const float b1 = A.t1[(static_cast<size_t>(pair_index(ea, eb)) << A.k1) + mask];
    return !(__fadd_ru(b1, jc) < tlo);
}

// The bound of one queued candidate from its 16 crossover bits (and its jump):
// f(c) + sum (|grad_k f(c)| + d_k r_k) r_k (+ the pair's tail).
// Elite e's boxes are bx[kStride e ..].
template <bool kTail, int kStride>
__device__ __forceinline__ float prune_bound(const PruneArgs &A, const uint32_t *__restrict__ bx, uint64_t s0,
                                             uint32_t meta) {
    const uint32_t ea = meta & 2047u, eb = (meta >> 11) & 2047u;
    const uint32_t *pa = bx + ea * kStride, *pb = bx + eb * kStride;
    uint32_t jidx = kNoJump;
    float jval = 0.0f;
    if (meta >> 31) {
        const uint64_t sj = s0 + 61 * kGolden;
        jidx = draw_hi(sj + kGolden) % 29u;
        jval = static_cast<float>(draw_vh(sj + 2 * kGolden) >> 8) * (1.0f / 16777216.0f);
    }
    uint64_t sb = s0 + 3 * kGolden;  // crossover bit draw of gene 0
    float g[16], c[16], r[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = A.m.wlin[j];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint32_t bw = draw_bitword(sb);
        sb += 2 * kGolden;
        const uint32_t w = ((static_cast<int32_t>(bw) < 0) ? pb : pa)[k];
        const float2 cr = __half22float2(*reinterpret_cast<const __half2 *>(&w));
        const bool j = jidx == static_cast<uint32_t>(k);
        c[k] = j ? jval : cr.x;
        r[k] = j ? 0.0f : cr.y;
#pragma unroll
        for (int q = 0; q < 16; ++q) g[q] = __fmaf_rn(A.pc.qs[k][q], c[k], g[q]);
    }
    float f2 = 0.0f, l1 = 0.0f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        f2 = __fmaf_rn(c[k], __fadd_rn(g[k], A.m.wlin[k]), f2);
        l1 = __fmaf_rn(__fmaf_rn(A.pc.d[k], r[k], fabsf(g[k])), r[k], l1);
    }
    float b = __fadd_rn(__fmaf_rn(0.5f, f2, A.m.w16), l1);
    if (kTail) b = __fadd_rn(b, __fadd_rn(A.tmax[ea * A.sc.ne + eb], jidx >= 16u ? A.jb.c[jidx] : 0.0f));
    return b;
}

// The pruning screen (persistent, dynamic items). Each thread walks its item's
// candidates by their four header draws alone (parents, immigrant, jump): the
// pair table rules out most of them. What it cannot rule out, immigrants and
// jumping candidates go to the warp's queue; when that holds a warp's worth,
// the warp draws their crossover bits and evaluates the candidate's own bound,
// and what passes goes to the CTA's queue for the full synthesis and the exact
// score (the filter form's queue).
// Pair bitmap: u0[pair] >= threshold as one bit per pair in shared memory; it
// is rebuilt as the threshold rises (a bit of an older threshold only passes
// more).
// Global threshold: besides the best CTA K-th score (Ctrl::gtau), every CTA
// publishes the keys of its m-th best entry, for three m (publish_first). If ceil(K / m) CTAs
// have published keys >= x, at least K distinct screened candidates score at
// least x, so the generation's K-th score is >= x; each published key only
// grows, so a stale read gives a lower, still valid, threshold. After each
// merge warp 0 takes the best such x and raises Ctrl::gtau to it.
// kFp64: the precision form's ranking -- queued candidates are scored in FP64
// and rank by that score rounded to f32 (the FP64 top-K; PruneConst::err
// covers the rounding of those scores too) -- instead of the reference's f32
// order.
// kFar: the box table stays in global memory (prune_bx_smem).
// Rounds without the bounds. Elites that are alike and score near the top (a run
// that screens its own survivors) leave the bounds little to rule out: every
// crossover of theirs lies within its mutation box of the threshold. The f32
// order's form then costs the bounds and the queue, 117 ms of 1e9 candidates
// where the unpruned kernel takes 32. So where most of a CTA's warps fill the
// queue at once (kPruneQuick) in two rounds in a row, each such round is followed
// by one that scores by the filter alone and queues what may reach the threshold, up to
// 128 candidates per thread: 46 ms (bounds that leave a third: 88 -> 46; 3e7
// candidates 4.2 -> 2.05). On elites of full spread nothing changed (2.65e9 22.3
// ms, 1e8 1.36). The FP64 form keeps its queue (the bounds cost it less beside its
// scores: 35 ms of 3e8 where its unpruned kernel takes 17 to 29; with these rounds
// 14, but 11.0 ms instead of 10.7 at 1e9 on elites of full spread).
template <bool kTail, bool kFp64, bool kFar>
__global__ void __launch_bounds__(kThreads, 3) screen_p_kernel(const __grid_constant__ PruneArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Entry *E = reinterpret_cast<Entry *>(smem_raw);
    WarpQueue *wqs = reinterpret_cast<WarpQueue *>(E + A.sort_n);
    // the elite table: only the queued candidates' full synthesis reads it;
    // in shared memory where that costs no CTA per SM, else through L1
    float *el_copy = reinterpret_cast<float *>(wqs + kThreads / 32);
    const float *el = A.el_smem ? el_copy : A.el;
    Pend *pend = reinterpret_cast<Pend *>(el_copy + (A.el_smem ? (A.sc.ne + 1) * kNtot : 0u));
    uint32_t *bx = reinterpret_cast<uint32_t *>(pend + kPendCap);
    uint32_t *bm = bx + (kFar ? 0u : A.sc.ne * 17);
    uint32_t *sel = bm + A.bm_words;
    __shared__ unsigned int s_buf_n, s_pend_n;
    __shared__ uint32_t s_quick, s_fails, s_direct;
    __shared__ unsigned long long s_t1, s_t2;
    __shared__ float s_ts;

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    WarpQueue &wq = wqs[warp];
    for (uint32_t i = tid; i < A.sort_n; i += kThreads) E[i] = Entry{0ull, 0ull};
    if (A.el_smem)
        for (uint32_t i = tid; i < (A.sc.ne + 1) * kNtot; i += kThreads) el_copy[i] = A.el[i];
    if (!kFar)
        for (uint32_t i = tid; i < A.sc.ne * 16; i += kThreads) bx[(i >> 4) * 17 + (i & 15u)] = A.box[i];
    for (uint32_t i = tid; i < A.bm_words; i += kThreads) bm[i] = 0xffffffffu;
    if (tid == 0) {
        s_buf_n = 0;
        s_pend_n = 0;
        s_quick = s_fails = s_direct = 0;
        s_t1 = 0;
        s_t2 = 0;
        s_ts = -INFINITY;
    }
    const unsigned int n_items = *reinterpret_cast<volatile unsigned int *>(&A.ctrl->n_items);
    __syncthreads();

    Entry *buf = E + A.kpad;
    uint32_t item = 0, left = 0, n_it = 0;
    uint64_t st = 0;  // state of the candidate's first draw
    uint32_t screened = 0, exact = 0;  // per thread: far below 2^32
    bool valid = false;
    auto start_item = [&]() {
        valid = item < n_items;
        n_it = left = 0;  // a thread without work counts down from 2^32 and never passes
        if (valid) {
            const Item it = A.items[item];
            st = stream_seed(A.seed, it.stream) + (it.draw0 + 1) * kGolden;
            n_it = left = it.n;
            screened += it.n;
            valid = left > 0;
        }
    };
    auto next_item = [&]() {
        item = gridDim.x * kThreads + atomicAdd(&A.ctrl->next_item, 1u);
        start_item();
    };
    item = A.ctrl->item_begin + tid * gridDim.x + blockIdx.x;  // the first: its place in the grid
    start_item();
    unsigned int gk = 0;
    uint32_t round = 0, n1 = 0, n2 = 0;  // n1, n2: the warp's queue lengths
    const uint32_t lt = (1u << lane) - 1u;
    const bool pow2 = (A.sc.ne & (A.sc.ne - 1)) == 0;
    // candidates the CTA's full queue could not take (one from either warp
    // queue); the warp pauses until the flush
    uint32_t n_def = 0;
    Pend def[2] = {{0u, 0u, 0u}, {0u, 0u, 0u}};
    auto push = [&](const uint4 &e, uint32_t itm) {
        const Item it = A.items[itm];
        const uint64_t s0 = (static_cast<uint64_t>(e.y) << 32) | e.x;
        const uint64_t draw = (s0 - stream_seed(A.seed, it.stream)) * kGoldenInv - 1;
        const Pend q{itm, e.z, static_cast<uint32_t>(draw - it.draw0)};
        const unsigned int ps = atomicAdd(&s_pend_n, 1u);
        if (ps < kPendCap) {
            pend[ps] = q;
        } else {
            if (n_def == 0) def[0] = q;
            else def[1] = q;
            ++n_def;
        }
    };

    auto rescore = [&](const Pend &q, float ts) {
        const Item it = A.items[q.item];
        const float s = prune_rescore<kFp64>(&A, el, stream_seed(A.seed, it.stream), it.draw0 + q.ddraw,
                                             __fsub_rd(ts, A.err));
        ++exact;
        if (s >= ts) {
            const unsigned long long k1 =
                (static_cast<unsigned long long>(score_okey(s)) << 32) | static_cast<unsigned int>(~q.item);
            const unsigned long long k2 = (static_cast<unsigned long long>(~q.dcand) << 32) | q.ddraw;
            buf[atomicAdd(&s_buf_n, 1u)] = Entry{k1, k2};  // score >= ts: ties with the K-th kept
        }
    };

    auto merge = [&](uint32_t bn) { prune_merge(&A, E, sel, bn, &s_buf_n, &s_t1, &s_t2, &s_ts); };

    for (;;) {
        __syncthreads();
        const unsigned int pn = min(s_pend_n, kPendCap);
        unsigned int bn = s_buf_n;  // nobody appends until after the next barrier
        if (!kFp64 && tid == 0) {  // whether the next round scores without the bounds (read behind the barriers below)
            const bool fail = s_quick > kThreads / 64 && (s_t1 != 0ull || gk != 0u);
            if (s_direct != 0u) {
                s_direct = 0;  // never two in a row: the rounds with the bounds drain the warps' queues
            } else {
                s_fails = fail ? min(s_fails + 1u, kPruneDirect) : 0u;
                s_direct = s_fails >= 2u ? 1u << (s_fails - 1u) : 0u;
            }
            s_quick = 0;
        }
        const int any = __syncthreads_or(valid || n_def > 0 || n1 + n2 > 0);
        const int any_def = __syncthreads_or(n_def > 0);
        // the queue is evaluated once it can employ every thread (or a thread
        // waits on it, or the work is done); a flush appends <= pn + 2 x 256 <= 1024
        if (pn >= kThreads || any_def || (!any && pn > 0)) {
            if (bn + kPendCap + 2 * kThreads > A.buf_cap) merge(bn);  // make room first
            float ts = s_ts;
            const unsigned int g = *reinterpret_cast<volatile unsigned int *>(&A.ctrl->gtau);
            if ((static_cast<unsigned long long>(g) << 32) > s_t1) ts = okey_score(g);
            for (uint32_t i = tid; i < pn; i += kThreads) rescore(pend[i], ts);
            for (uint32_t i = 0; i < n_def; ++i) rescore(i == 0 ? def[0] : def[1], ts);
            n_def = 0;
            __syncthreads();
            bn = s_buf_n;
            if (tid == 0) s_pend_n = 0;
            __syncthreads();
        }
        // merge when half full, and every kPruneMergeRounds rounds while the
        // buffer holds anything: the CTA's threshold and published keys then
        // follow the candidates it finds instead of waiting for a full buffer
        if (bn >= A.buf_cap / 2 || (bn > 0 && (!any || (round & (kPruneMergeRounds - 1)) == 0))) merge(bn);
        if (!any) break;
        float ts = s_ts;
        const unsigned long long t1 = s_t1;
        // one lane's reading for the whole warp: the ballots below stand under it
        gk = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile unsigned int *>(&A.ctrl->gtau), 0);
        if ((static_cast<unsigned long long>(gk) << 32) > t1) ts = okey_score(gk);
        const float tlo = __fsub_rd(ts, A.pc.err);
        // rebuild the bitmap: early on at rounds 1, 2, 4, ..., then every bm_period
        if (((round & (A.bm_period - 1)) == 0 || (round & (round - 1)) == 0) && tlo > -INFINITY) {
            for (uint32_t w = warp; w < A.bm_words; w += kThreads / 32) {
                const uint32_t i = w * 32 + lane;
                const bool on = i < A.sc.ne * A.sc.ne && !(A.u0[i] < tlo);
                const uint32_t bits = __ballot_sync(0xffffffffu, on);
                if (lane == 0) bm[w] = bits;
            }
            __syncwarp();
        }
        ++round;
        if (const uint32_t cnt = kFp64 ? 0u : s_direct; cnt != 0u && ts > -INFINITY) {
            const float td = __fsub_rd(ts, A.err);
#pragma unroll 1
            for (uint32_t i = 0; i < cnt && valid && n_def == 0; ++i) {
                const Item it = A.items[item];
                const uint64_t seed_t = stream_seed(A.seed, it.stream);
                const uint64_t p = (st - seed_t) * kGoldenInv - 1;
                if (!(filter_score_at(&A, el, seed_t, p) < td)) {
                    const Pend q{item, n_it - left, static_cast<uint32_t>(p - it.draw0)};
                    const unsigned int ps = atomicAdd(&s_pend_n, 1u);
                    if (ps < kPendCap) {
                        pend[ps] = q;
                    } else {
                        def[0] = q;
                        n_def = 1;
                    }
                }
                const bool imm = (draw_vh(st + 2 * kGolden) >> 8) < A.sc.imm_thr;
                const uint64_t sj = st + (imm ? 32u : 61u) * kGolden;
                st = sj + (((draw_vh(sj) >> 8) < A.sc.jump_thr) ? 3u : 1u) * kGolden;
                if (--left == 0) next_item();
            }
            continue;
        }
#pragma unroll 1
        for (int rr = 0; rr < kPruneRounds; ++rr) {
            const uint64_t s0 = st;
            const uint32_t itm = item, dcand = n_it - left;
            const PairHead h = pair_head(A.sc, pow2, s0);
            st = h.next;
            const uint32_t pi = h.ea * A.sc.ne + h.eb;
            const bool on = A.bm_words ? ((bm[pi >> 5] >> (pi & 31u)) & 1u) != 0u : !(A.u0[pi] < tlo);
            const bool pass = valid && (h.imm || h.jump || on);
            if (--left == 0) next_item();
            const uint32_t m = __ballot_sync(0xffffffffu, pass);
            if (pass) {
                const uint32_t slot = n1 + __popc(m & lt);
                wq.q1[slot] = make_uint4(static_cast<uint32_t>(s0), static_cast<uint32_t>(s0 >> 32), dcand, pair_meta(h));
                wq.i1[slot] = itm;
            }
            n1 += __popc(m);
            if (n1 < 32 && (n1 + n2 == 0 || __any_sync(0xffffffffu, valid))) continue;
            // a warp's worth (or, without work left, the rest) of the first queue: the first k1 bits
            __syncwarp();
            {
                const uint32_t nb = min(n1, 32u);
                n1 -= nb;
                bool to2 = false, immq = false;
                uint4 q = make_uint4(0u, 0u, 0u, 0u);
                uint32_t iq = 0;
                if (lane < nb) {
                    q = wq.q1[n1 + lane];
                    iq = wq.i1[n1 + lane];
                    const uint64_t sq = (static_cast<uint64_t>(q.y) << 32) | q.x;
                    immq = (q.w & (1u << 30)) != 0u;
                    to2 = !immq && mask_passes(A, sq, q.w, tlo);
                }
                if (immq) push(q, iq);  // immigrants are always scored
                const uint32_t m2 = __ballot_sync(0xffffffffu, to2);
                if (to2) {
                    const uint32_t slot = n2 + __popc(m2 & lt);
                    wq.q2[slot] = q;
                    wq.i2[slot] = iq;
                }
                n2 += __popc(m2);
            }
            // the second queue: each candidate's own bound
            if (n2 >= 32 || (n2 > 0 && n1 == 0 && !__any_sync(0xffffffffu, valid))) {
                __syncwarp();
                const uint32_t nb = min(n2, 32u);
                n2 -= nb;
                if (lane < nb) {
                    const uint4 q = wq.q2[n2 + lane];
                    const uint64_t sq = (static_cast<uint64_t>(q.y) << 32) | q.x;
                    const float f = kFar ? prune_bound<kTail, 16>(A, A.box, sq, q.w)
                                         : prune_bound<kTail, 17>(A, bx, sq, q.w);
                    if (!(f < tlo)) push(q, wq.i2[n2 + lane]);  // NaN: scored
                }
            }
            if (__any_sync(0xffffffffu, n_def > 0)) {
                if (!kFp64 && lane == 0 && rr < kPruneQuick) atomicAdd(&s_quick, 1u);
                break;
            }
        }
    }
    Entry *out = A.lists + static_cast<size_t>(blockIdx.x) * A.kpad;
    for (uint32_t i = tid; i < A.kpad; i += kThreads) out[i] = E[i];
    unsigned long long scr = screened, exa = exact;
    for (int o = 16; o > 0; o >>= 1) {
        scr += __shfl_down_sync(0xffffffffu, scr, o);
        exa += __shfl_down_sync(0xffffffffu, exa, o);
    }
    if (lane == 0) {
        atomicAdd(&A.ctrl->screened, scr);
        atomicAdd(&A.ctrl->exact_evals, exa);
    }
}

using PruneScreenFn = void (*)(PruneArgs);

// The pruning kernel of a plan: with a linear tail or not, ranking in the
// reference's f32 order or (the precision form) in FP64, the box table in
// shared memory or not.
template <bool kFar>
PruneScreenFn screen_p_pick(bool tail, bool fp64) {
    if (tail) return fp64 ? screen_p_kernel<true, true, kFar> : screen_p_kernel<true, false, kFar>;
    return fp64 ? screen_p_kernel<false, true, kFar> : screen_p_kernel<false, false, kFar>;
}
PruneScreenFn screen_p_fn(bool tail, bool fp64, bool bx_smem) {
    return bx_smem ? screen_p_pick<false>(tail, fp64) : screen_p_pick<true>(tail, fp64);
}

// Words of the pair bitmap for ne elites: one bit per pair up to 16 KB of
// shared memory (362 elites), past that the screen reads the table.
inline uint32_t prune_bm_words(int ne) {
    const uint64_t w = (static_cast<uint64_t>(ne) * ne + 31) / 32;
    return w <= 4096 ? static_cast<uint32_t>(w) : 0u;
}

// Whether the box table goes to shared memory: not beside lists of 4096 entries
// where the elites are more than the queues leave room for (1057 of them).
inline bool prune_bx_smem(uint32_t sort_n, int ne) { return sort_n < 8192 || ne <= 1024; }

// Shared memory of the pruning screen: the sort buffer, the warps' queues, the
// CTA's queue, the box table (prune_bx_smem), the pair bitmap and the selection scratch of the
// published keys (one per CTA, at most 3 CTAs per SM), with el_smem the elite
// table.
size_t prune_smem(uint32_t sort_n, int ne, int num_sms, bool el_smem) {
    return static_cast<size_t>(sort_n) * sizeof(Entry) + (kThreads / 32) * sizeof(WarpQueue) +
           kPendCap * sizeof(Pend) + (prune_bx_smem(sort_n, ne) ? static_cast<size_t>(ne) * 17 * sizeof(uint32_t) : 0) +
           prune_bm_words(ne) * sizeof(uint32_t) + 3ull * num_sms * sizeof(uint32_t) +
           (el_smem ? static_cast<size_t>(ne + 1) * kNtot * sizeof(float) : 0);
}

// PruneConst::d: d >= 0 with diag(d) - Qsym positive semidefinite (Qsym = Qs /
// 2, the symmetric form of Q) and a small sum, so that u' Q u <= sum d_k u_k^2.
// Row sums of |Qsym| dominate; scaled by the largest eigenvalue of
// diag(d)^-1/2 Qsym diag(d)^-1/2 they still do, and a few rounds move d towards
// the genes on which the eigenvector shows it binding. The eigenvalues come
// from power iteration and certify nothing: the d taken is the one whose
// diag(d) - Qsym passes a Cholesky factorisation with every pivot above 1e-6 of
// the matrix's largest entry (a double factorisation's error is below 1e-12 of
// it), raised by a hundredth until it does. About 100 N^2 multiply-adds.
template <int N>
void quad_diag(const float (&qs)[N][N], float (&out)[N]) {
    double S[N][N], dom[N], d[N], v[N], best[N], top = 0.0, best_sum = 0.0;
    for (int i = 0; i < N; ++i)
        for (int j = 0; j < N; ++j) {
            S[i][j] = 0.5 * static_cast<double>(qs[i][j]);
            top = std::max(top, std::fabs(S[i][j]));
        }
    if (top == 0.0) {
        for (int i = 0; i < N; ++i) out[i] = 0.0f;
        return;
    }
    for (int i = 0; i < N; ++i) {
        dom[i] = S[i][i];
        for (int j = 0; j < N; ++j)
            if (j != i) dom[i] += std::fabs(S[i][j]);
        dom[i] = std::max(dom[i], 1e-6 * top);
        best[i] = d[i] = dom[i];
        best_sum += dom[i];
        v[i] = 1.0 / std::sqrt(static_cast<double>(N));
    }
    for (int round = 0; round < 4; ++round) {
        double M[N][N], h[N], shift = 0.0, lam = 0.0;
        for (int i = 0; i < N; ++i) h[i] = 1.0 / std::sqrt(d[i]);
        for (int i = 0; i < N; ++i) {
            double row = 0.0;
            for (int j = 0; j < N; ++j) {
                M[i][j] = S[i][j] * h[i] * h[j];
                row += std::fabs(M[i][j]);
            }
            shift = std::max(shift, row);
        }
        for (int it = 0; it < 24; ++it) {  // power iteration, shifted so that the largest eigenvalue leads
            double w[N], n2 = 0.0;
            lam = 0.0;
            for (int i = 0; i < N; ++i) {
                double s = 0.0;
                for (int j = 0; j < N; ++j) s += M[i][j] * v[j];
                lam += s * v[i];
                w[i] = s + 0.5 * shift * v[i];
                n2 += w[i] * w[i];
            }
            if (!(n2 > 0.0)) break;
            const double inv = 1.0 / std::sqrt(n2);
            for (int i = 0; i < N; ++i) v[i] = w[i] * inv;
        }
        lam = std::max(lam, 1e-6);
        double sum = 0.0;
        for (int i = 0; i < N; ++i) sum += d[i] * lam;
        if (sum < best_sum) {
            best_sum = sum;
            for (int i = 0; i < N; ++i) best[i] = d[i] * lam;
        }
        const double eta = 0.5 / (1.0 + 0.3 * round);
        for (int i = 0; i < N; ++i)
            d[i] = std::max(d[i] * lam * std::pow((v[i] * v[i] + 0.01) / (d[i] * lam / sum + 0.01), eta), 1e-6 * top);
    }
    for (int tries = 0;; ++tries) {  // dom itself passes: rows dominated with room
        const bool last = tries == 64;
        const double up = std::pow(1.01, tries) * (1.0 + 1e-4);
        for (int i = 0; i < N; ++i) d[i] = (last ? dom[i] * 1.001 : best[i] * up) + 2e-6 * top;
        if (last) break;
        double L[N][N];
        bool ok = true;
        for (int k = 0; k < N && ok; ++k)
            for (int i = k; i < N; ++i) {
                double s = (i == k ? d[i] : 0.0) - S[i][k];
                for (int m = 0; m < k; ++m) s -= L[i][m] * L[k][m];
                if (i == k) {
                    if (!(s > 1e-6 * top)) {
                        ok = false;
                        break;
                    }
                    L[k][k] = std::sqrt(s);
                } else {
                    L[i][k] = s / L[k][k];
                }
            }
        if (ok) break;
    }
    for (int i = 0; i < N; ++i) out[i] = std::nextafter(static_cast<float>(d[i]), INFINITY);
}

// The bound's constants for a model whose filter bound is finite and a
// mutation width the fast delta form handles (PruneConst::d is set by the plan
// that prunes). *tail: some linear weight past gene 15 is nonzero. Returns
// false when the bound cannot be certified (non-finite sums).
bool make_prune(const csx_model &m, float sigma, PruneConst *pc, bool *tail) {
    const double s = std::min(std::fabs(static_cast<double>(sigma)) + std::ldexp(1.0, -24), 1.0);
    double qsum = 0.0, lsum = 0.0;
    bool tail_nz = false;
    for (int i = 0; i < 16; ++i)
        for (int j = 0; j <= i; ++j) qsum += std::fabs(static_cast<double>(m.w_quad[i * 16 + j]));
    for (int k = 0; k < kNtot; ++k) {
        const double w = static_cast<double>(m.w_lin[k]);
        lsum += std::fabs(w);
        if (k >= 16) tail_nz = tail_nz || w != 0.0;
    }
    for (int j = 0; j < 16; ++j)
        for (int k = 0; k < 16; ++k) {
            const float q = j >= k ? m.w_quad[j * 16 + k] : m.w_quad[k * 16 + j];
            pc->qs[j][k] = (j == k) ? 2.0f * q : q;  // exact: the weights are finite and below 1e30
        }
    const double up = 1.0 + std::ldexp(1.0, -20);
    const double u = std::ldexp(1.0, -24);
    auto gamma = [u](double n) { return n * u / (1.0 - n * u); };
    const double w16 = 16.0 * std::fabs(static_cast<double>(m.w0));
    // magnitudes the bound's f32 sums reach: sum d_k r_k^2 <= 2 qsum (r <= 1/2 + 2^-10, sum d <= 2.002 qsum)
    const double a_bound = w16 + 3.0 * lsum + 6.0 * qsum;
    const double a_ref = w16 + lsum + qsum;  // the reference order's (genes in [0, 1])
    const double err = (2.0 * gamma(64) * a_bound + gamma(35) * a_ref) * up + 1e-30;
    if (!std::isfinite(err) || err > 1e30) return false;
    pc->s = std::nextafter(static_cast<float>(s), INFINITY);
    pc->err = std::nextafter(static_cast<float>(err), INFINITY);
    *tail = tail_nz;
    return true;
}

// CTAs per SM of a pruning screen with this shared memory (228 KB per SM, 1 KB
// reserved per CTA; at most 3, its register limit).
inline int prune_fit(size_t smem) { return std::min(3, static_cast<int>((228u << 10) / (smem + 1024))); }

// Whether the elite table goes to shared memory: where it costs no CTA per SM
// (the queue's synthesis reads it).
inline bool prune_el_smem(uint32_t sort_n, int ne, int num_sms, size_t max_smem) {
    const size_t with = prune_smem(sort_n, ne, num_sms, true);
    return with + 1024 <= max_smem && prune_fit(with) >= prune_fit(prune_smem(sort_n, ne, num_sms, false));
}

// Masks the pair table enumerates per pair: 2^n_enum. One mask costs about 45
// instructions against some 150 per candidate of the screen, so the table is
// given one mask per eight candidates (at least five genes' masks, whatever the
// budget): 3-4% of the screen. All 16 genes at
// 2.65e9 candidates and 64 elites (2080 pairs); fewer genes loosen the bound
// (pairs left at the final threshold, committed surface: 8% with 16 genes
// enumerated, 10% with 10, 11% with 8, 14% with 6).
inline int pair_enum(uint64_t lambda, int ne) {
    const uint64_t pairs = static_cast<uint64_t>(ne) * (ne + 1) / 2;
    int k = kPairGray;
    while (k < 16 && (pairs << (k + 1)) <= lambda / 8) ++k;
    return k;
}

// Genes of the mask table: the enumerated ones but four (a pair's group of
// threads shares those), at most eight, fewer where the table would pass 64 MB,
// down to the five of a thread's Gray walk: 151 MB at the 1,536 elites that the
// library takes at most.
inline int pair_k1(int n_enum, int ne) {
    const uint64_t pairs = static_cast<uint64_t>(ne) * (ne + 1) / 2;
    int k = std::min(kMaxMaskGenes, std::max(kPairGray, n_enum - 4));
    while (k > kPairGray && (pairs << (k + 2)) > (64ull << 20)) --k;
    return k;
}

// Device scratch of the pair bounds: boxes, then u0, then (with a tail) tmax,
// then t1.
struct PairBufs {
    uint32_t *box = nullptr;
    float *u0 = nullptr, *tmax = nullptr, *t1 = nullptr;
    int n_enum = kPairGray, k1 = kPairGray;
};

// The 16 quadratic genes in descending order of their influence: the mean
// gradient over the unit box (the device call's elites are not on the host).
void gene_order(const csx_model &m, const PruneConst &pc, uint8_t (&perm)[16]) {
    double infl[16];
    for (int k = 0; k < 16; ++k) {
        double g = static_cast<double>(m.w_lin[k]);
        for (int j = 0; j < 16; ++j) g += 0.5 * static_cast<double>(pc.qs[k][j]);
        infl[k] = std::fabs(g);
        perm[k] = static_cast<uint8_t>(k);
    }
    std::stable_sort(perm, perm + 16, [&](uint8_t a, uint8_t b) { return infl[a] > infl[b]; });
}

// The pair table's arguments: the model in gene_order, and the table's own
// rounding.
PairArgs make_pair_args(const csx_model &m, const PruneConst &pc, int ne, bool tail,
                        const float *tab, const PairBufs &b) {
    PairArgs P{};
    double qsum = 0.0, lsum = 0.0;
    gene_order(m, pc, P.perm);
    for (int i = 0; i < 16; ++i) {
        P.lin[i] = m.w_lin[P.perm[i]];
        P.d[i] = pc.d[P.perm[i]];
        for (int j = 0; j < 16; ++j) {
            P.qs[i][j] = pc.qs[P.perm[i]][P.perm[j]];
            qsum += std::fabs(static_cast<double>(P.qs[i][j]));
        }
    }
    for (int k = 0; k < kNtot; ++k) lsum += std::fabs(static_cast<double>(m.w_lin[k]));
    for (int k = 16; k < kNtot; ++k) P.tl[k - 16] = m.w_lin[k];
    P.w16 = 16.0f * m.w0;
    P.s = pc.s;
    // rounding of the table's f32 sums: at most 16 + 31 + 31 + 16 + 20 roundings along any chain (the
    // gradient's FMAs and flips, the value's flips, the radius sum, the remainder and the tail), 128 with
    // room, over sums of magnitude at most w16 + 4 lsum + 4 qsum (Qs counted in full, radii at most 1)
    const double u = std::ldexp(1.0, -24), gam = 128 * u / (1.0 - 128 * u);
    const double e = 2.0 * gam * (std::fabs(static_cast<double>(P.w16)) + 4.0 * lsum + 4.0 * qsum) + 1e-30;
    P.err = std::nextafter(static_cast<float>(e * (1.0 + std::ldexp(1.0, -20))), INFINITY);
    P.tab = tab;
    P.box = b.box;
    P.u0 = b.u0;
    P.t1 = b.t1;
    P.tmax = b.tmax;
    P.tail = tail ? 1 : 0;
    P.ne = ne;
    P.n_enum = b.n_enum;
    P.k1 = b.k1;
    return P;
}

}  // namespace csx
