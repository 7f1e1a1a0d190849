// csx_prune_full.cuh — the pruning screen of the full quadratic surface (all
// 29 genes quadratic): a certified upper bound of each candidate from its
// parents and crossover bits, the bound's gradient on the tensor cores.
// Part of csx_screen.cu's translation unit (included there, in order); not a
// standalone header.
//
// The unpruned screen draws 58 values and spends 464 FMAs on every candidate
// (src/screen.zig:225-253's synthesis; the surface is this library's
// extension). Here a crossover candidate draws its 29 crossover bits, and with
// yh its clamped parent genes in FP16 and s the mutation half-width (2^-12 for
// the rounding of yh included),
//   f(g) <= f(yh) + s sum_k |grad_k f(yh)| + s^2 sum_k d_k,
// diag(d) - Q positive semidefinite (quad_diag), grad f(yh) = w + Qs yh. A jump
// at gene j puts its value in yh_j. Only what the bound leaves, and immigrants,
// are synthesised and scored. (A table over parent pairs, as the 16-gene
// surface has, rules out next to none of them here: seven genes in eight of 29
// would stay open.)
//
// Qs yh is a 29 x 29 product per candidate, 841 FMAs: each 128-thread group
// writes its candidates' yh as FP16 rows of a shared-memory tile and one thread
// issues tcgen05.mma (M 128, N 32, K 32, FP32 accumulation); every thread reads
// its own row back. Where the bound leaves more than half of a round's candidates
// (elites that are alike and near the top, as survivors screened again are; a
// threshold not yet settled), a CTA scores the next ones without it and tries
// again, after four such rounds in a row at growing distances. A round that tries
// again takes a quarter of the candidates: its queue is full within two or three
// per thread. 2.65e8 candidates whose elites are the survivors of a screen: 28.0
// ms with every candidate queued and fetched back, 19.6 so (16.5 unpruned: the
// coefficients come from shared memory here, and with them as constants in this
// kernel its other rounds spill, 11.9 ms instead of 11.3 on uniform elites); 5e7:
// 6.6 ms, 4.5 so, 3.5 unpruned.
//
// What bounds it is the instruction issue, 33 hashes first. 2.65e8 candidates
// of 64 uniform elites, a seeded N(0, 0.1) surface, sigma 0.12, top 256: 16.5
// ms unpruned, 10.9 here (5.2% scored, 1% of it immigrants); 5e7: 2.6 ms.
#pragma once

namespace csx {

constexpr int kFtStride = 30;        // halfs per elite row: 15 words, odd
constexpr uint32_t kFtTile = 8192;   // a group's X tile: 128 rows x 32 halfs
constexpr uint32_t kFtB = 2048;      // the B tile: 32 x 32 halfs
constexpr int kFtRounds = 16;        // candidates per thread between the CTA's barriers
constexpr uint32_t kFtProbe = 32;    // most outer rounds between probes of the bound while it is off

// Qs 2^-e in FP16 (e places the largest entry in [2^14, 2^15)), K-major core
// matrices of 8 rows x 16 bytes, LBO 128, SBO 512.
struct FullPrune {
    alignas(16) uint16_t btile[kFtB / 2];
    float dscale;  // 2^e
    float s;       // half-width around the FP16 centre, rounded up
    float c0;      // s^2 sum d_k, rounded up
    float err;     // rounding of the bound, of its FP16 gradient and of the score's FMA order
};

struct FullPruneArgs : FullScreenArgs {
    FullPrune fp;
    uint32_t *pub;
    uint32_t sel_cap;
    uint32_t el_smem;
};

__device__ __forceinline__ void tc_mma_acc(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u)
        : "memory");
}

// The full surface's coefficients in shared memory, row k = [w_k, Q_k0 .. Q_kk]
// from a 16-byte boundary.
__host__ __device__ constexpr int ft_row(int k) {
    int o = 0;
    for (int j = 0; j < k; ++j) o += (j + 2 + 3) / 4 * 4;
    return o;
}
constexpr int kFtCoef = ft_row(kNtot);

// The score of the candidate at p, out of line and with the coefficients from
// shared memory (16 bytes to every lane at once): in line it spilled, and
// through the kernel's arguments each coefficient was a load of its own: a
// screen that scored every candidate took 26.7 and 30.3 ms at 2.65e8 where the
// unpruned kernel takes 16.5.
__device__ __forceinline__ float full_score(const SynthConst &C, float w0, uint32_t coef, const float *el,
                                            uint64_t seed_t, uint64_t p, const CandHead &h) {
    GeneSource S = gene_source(C, el, seed_t, p, h);
    float G[kNtot];
    float R = w0;
#pragma unroll
    for (int k = 0; k < kNtot; ++k) {
        float g = next_gene<true>(S, k);
        g = (static_cast<uint32_t>(k) == h.jidx) ? h.jval : g;
        G[k] = g;
        float t = 0.0f;
#pragma unroll
        for (int c = 0; c < (k + 2 + 3) / 4; ++c) {
            float q[4];
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(q[0]), "=f"(q[1]), "=f"(q[2]), "=f"(q[3])
                         : "r"(coef + 4u * static_cast<uint32_t>(ft_row(k) + 4 * c)));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = 4 * c + e;  // w_k, then Q_k,i-1
                if (i == 0) t = q[0];
                else if (i <= k + 1) t = __fmaf_rn(q[e], G[i - 1], t);
            }
        }
        R = __fmaf_rn(g, t, R);
    }
    return R;
}
__device__ __noinline__ float full_score_at(const SynthConst *__restrict__ C, float w0, uint32_t coef, const float *el,
                                            uint64_t seed_t, uint64_t p) {
    const CandHead h = cand_head(*C, seed_t, p);
    return full_score(*C, w0, coef, el, seed_t, p, h);
}

// A round without the bound, out of line: kFtRounds candidates of the thread's
// items scored, the ones at the threshold ts or above to the CTA's queue.
struct DirectRound {  // a thread's place among its items, and the candidate the full queue did not take
    uint64_t st;
    uint32_t item, left, n_it, screened, exact, n_def;
    bool valid;
    Pend def;
};
__device__ __noinline__ void full_direct(const FullPruneArgs *__restrict__ A, const float *el, uint32_t coef,
                                         Pend *pend, unsigned int *s_pend_n, float ts, DirectRound *place) {
    if (!place->valid) return;
    const uint32_t n_items = A->ctrl->n_items;
    DirectRound d = *place;
    Item it = A->items[d.item];
    uint64_t seed_t = stream_seed(A->seed, it.stream);
    uint64_t p = (d.st - seed_t) * kGoldenInv - 1;
#pragma unroll 1
    for (int r = 0; r < kFtRounds && d.n_def == 0; ++r) {
        const CandHead h = cand_head(A->sc, seed_t, p);
        ++d.exact;
        if (full_score(A->sc, A->fm.w0, coef, el, seed_t, p, h) >= ts) {
            const Pend q{d.item, d.n_it - d.left, static_cast<uint32_t>(p - it.draw0)};
            const unsigned int slot = atomicAdd(s_pend_n, 1u);
            if (slot < kPendCap) {
                pend[slot] = q;
            } else {
                d.def = q;
                d.n_def = 1;
            }
        }
        p += h.len;
        if (--d.left == 0) {
            d.item = gridDim.x * kThreads + atomicAdd(&A->ctrl->next_item, 1u);
            d.n_it = 0;
            d.valid = d.item < n_items;
            if (!d.valid) break;
            it = A->items[d.item];
            seed_t = stream_seed(A->seed, it.stream);
            p = it.draw0;
            d.n_it = d.left = it.n;
            d.screened += it.n;
            d.valid = it.n > 0;
            if (!d.valid) break;
        }
    }
    d.st = seed_t + (p + 1) * kGolden;
    *place = d;
}

// One round of a 128-thread group: row `row` of its tile <- pk (32 halfs), one
// MMA pair. Returns false when the wait gave up; then the group stops its MMAs
// together (tcp_round's give-up path).
__device__ __forceinline__ bool ft_round(TcGroup &g, const uint32_t (&pk)[16], uint32_t row, volatile uint32_t *gbad,
                                         volatile uint32_t *fail_phase) {
    const uint32_t a = g.xs + (row >> 3) * 512u + (row & 7u) * 16u;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + 128u * c), "r"(pk[4 * c]),
                     "r"(pk[4 * c + 1]), "r"(pk[4 * c + 2]), "r"(pk[4 * c + 3])
                     : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    if (g.bar_id == 1)
        asm volatile("bar.sync 1, 128;" ::: "memory");
    else
        asm volatile("bar.sync 2, 128;" ::: "memory");
    if (*gbad != 0u) return true;
    if (g.issuer) {
        tc_fence_after();
        tc_mma_acc(g.tmem_d, g.adesc, g.bdesc, g.idesc, false);
        tc_mma_acc(g.tmem_d, g.adesc + (256u >> 4), g.bdesc + (256u >> 4), g.idesc, true);  // genes 16..31
        tc_commit(g.mbar);
    }
    const bool ok = mbar_wait(g.mbar, g.phase);
    if (!ok) {
        *fail_phase = g.phase;
        *gbad = 1u;
    }
    g.phase ^= 1u;
    tc_fence_after();
    return ok;
}

__global__ void __launch_bounds__(kThreads, 3) screen_ft_kernel(const __grid_constant__ FullPruneArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Entry *E = reinterpret_cast<Entry *>(smem_raw);
    float *el_copy = reinterpret_cast<float *>(E + A.sort_n);
    const float *el = A.el_smem ? el_copy : A.el;
    float *coef = el_copy + (A.el_smem ? ((A.sc.ne + 1) * kNtot + 3u) & ~3u : 0u);
    Pend *pend = reinterpret_cast<Pend *>(coef + kFtCoef);
    uint32_t *sel = reinterpret_cast<uint32_t *>(pend + kPendCap);
    uint16_t *yt = reinterpret_cast<uint16_t *>(sel + A.sel_cap);
    __shared__ __align__(8) unsigned long long s_mbar[2];
    __shared__ uint32_t s_tbase;
    __shared__ unsigned int s_buf_n, s_pend_n, s_passed, s_seen;
    __shared__ uint32_t s_gbad[2], s_fail_phase[2];
    __shared__ unsigned long long s_t1, s_t2;
    __shared__ float s_ts;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, grp = warp >> 2;
    const uint32_t base = smem_u32(smem_raw);
    const uint32_t xs0 = (smem_u32(yt + A.sc.ne * kFtStride) + 1023u) & ~1023u;
    const uint32_t bts = xs0 + 2u * kFtTile;
    for (uint32_t i = tid; i < A.sort_n; i += kThreads) E[i] = Entry{0ull, 0ull};
    if (A.el_smem)
        for (uint32_t i = tid; i < (A.sc.ne + 1) * kNtot; i += kThreads) el_copy[i] = A.el[i];
    for (uint32_t i = tid; i < A.sc.ne * kNtot; i += kThreads) {
        const uint32_t r = i / kNtot, k = i - r * kNtot;
        yt[r * kFtStride + k] = __half_as_ushort(__float2half_rn(fmaxf(fminf(A.el[i], 1.0f), 0.0f)));
    }
    for (uint32_t i = tid; i < 30u * 30u; i += kThreads) {  // row k's entry 0 is w_k, entry j + 1 is Q_kj
        const uint32_t k = i / 30u, e = i - k * 30u;
        if (k < kNtot && e <= k + 1u) {
            uint32_t o = 0;
            for (uint32_t j = 0; j < k; ++j) o += (j + 5u) / 4u * 4u;
            coef[o + e] = e == 0 ? A.fm.wlin[k] : A.fm.wq[k * (k + 1u) / 2u + e - 1u];
        }
    }
    for (uint32_t i = tid; i < kFtB / 4; i += kThreads)
        reinterpret_cast<uint32_t *>(smem_raw + (bts - base))[i] = reinterpret_cast<const uint32_t *>(A.fp.btile)[i];
    if (warp == 0) tc_alloc(smem_u32(&s_tbase), 64);
    if (tid == 0) {
        mbar_init(smem_u32(&s_mbar[0]), 1);
        mbar_init(smem_u32(&s_mbar[1]), 1);
        s_buf_n = s_pend_n = s_passed = s_seen = 0;
        s_gbad[0] = s_gbad[1] = 0;
        s_fail_phase[0] = s_fail_phase[1] = 0;
        s_t1 = 0;
        s_t2 = 0;
        s_ts = -INFINITY;
    }
    const unsigned int n_items = *reinterpret_cast<volatile unsigned int *>(&A.ctrl->n_items);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    TcGroup tg;
    tg.xs = xs0 + grp * kFtTile;
    tg.mbar = smem_u32(&s_mbar[grp]);
    tg.tmem_d = s_tbase + 32u * grp;
    tg.tmem_ld = s_tbase + ((32u * (warp & 3u)) << 16) + 32u * grp;
    tg.adesc = tc_sdesc(tg.xs, 128, 512);
    tg.bdesc = tc_sdesc(bts, 128, 512);
    tg.idesc = (1u << 4) | ((32u >> 3) << 17) | ((128u >> 4) << 24);  // FP16 x FP16 -> FP32, N 32, M 128
    tg.bar_id = 1u + grp;
    tg.phase = 0;
    tg.issuer = (tid & 127u) == 0;
    bool tc_ok = true;

    Entry *buf = E + A.kpad;
    uint32_t item = 0, left = 0, n_it = 0;
    uint64_t st = 0;
    uint32_t screened = 0, exact = 0;
    bool valid = false;
    auto start_item = [&]() {
        valid = item < n_items;
        n_it = left = 0;
        if (valid) {
            const Item it = A.items[item];
            st = stream_seed(A.seed, it.stream) + (it.draw0 + 1) * kGolden;
            n_it = left = it.n;
            screened += it.n;
            valid = left > 0;
        }
    };
    item = A.ctrl->item_begin + tid * gridDim.x + blockIdx.x;  // the first: its place in the grid
    start_item();
    unsigned int gk = 0;
    uint32_t round = 0, off_until = 0, fails = 0;  // rounds below off_until pass everything on
    const bool pow2 = (A.sc.ne & (A.sc.ne - 1)) == 0;
    bool has_def = false;  // holds a candidate the full queue could not take; pauses until the flush
    Pend def{0u, 0u, 0u};

    auto rescore = [&](const Pend &q, float ts) {
        const Item it = A.items[q.item];
        const float s = full_score_at(&A.sc, A.fm.w0, smem_u32(coef), el, stream_seed(A.seed, it.stream),
                                      it.draw0 + q.ddraw);
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
        // a group whose tensor-core wait gave up ends the CTA's screening
        const int stop = (s_gbad[0] | s_gbad[1]) != 0u;
        // the bound left more than half of the last round: off for a round (the
        // threshold has yet to settle), after the fourth time in a row for ever longer
        if (s_passed * 2 > s_seen) {
            ++fails;
            off_until = round + (fails <= 4 ? 1u : min(1u << (fails - 4), kFtProbe));
            fails = min(fails, 24u);
        } else if (s_seen > 0) {
            fails = 0;
        }
        const int any = __syncthreads_or((valid || has_def) && !stop);
        const int any_def = __syncthreads_or(has_def);
        if (tid == 0) s_passed = s_seen = 0;
        if (pn >= kThreads || any_def || (!any && pn > 0)) {
            if (bn + kPendCap + kThreads > A.buf_cap) merge(bn);  // make room first
            float ts = s_ts;
            const unsigned int g = *reinterpret_cast<volatile unsigned int *>(&A.ctrl->gtau);
            if ((static_cast<unsigned long long>(g) << 32) > s_t1) ts = okey_score(g);
            for (uint32_t i = tid;; i += kThreads) {
                Pend q;
                if (i < pn) {
                    q = pend[i];
                } else if (has_def) {
                    q = def;
                    has_def = false;
                } else {
                    break;
                }
                rescore(q, ts);
            }
            __syncthreads();
            bn = s_buf_n;
            if (tid == 0) s_pend_n = 0;
            __syncthreads();
        }
        if (bn >= A.buf_cap / 2 || (bn > 0 && (!any || (round & 3u) == 0))) merge(bn);
        if (!any) break;
        float ts = s_ts;
        gk = *reinterpret_cast<volatile unsigned int *>(&A.ctrl->gtau);
        if ((static_cast<unsigned long long>(gk) << 32) > s_t1) ts = okey_score(gk);
        const float tlo = __fsub_rd(ts, A.fp.err);
        // the same in every thread (the group's barriers need it): gk may differ
        // between threads. The barrier also orders s_passed / s_seen's zeros.
        const bool settled = __syncthreads_or(ts > -INFINITY) != 0;
        const bool on = settled && round >= off_until;
        ++round;
        // tried again, a short round
        const int r0 = on && fails > 1 ? kFtRounds - kFtRounds / 4 : 0;
        if (!on && settled) {
            DirectRound d{st, item, left, n_it, screened, exact, 0u, valid, {0u, 0u, 0u}};
            full_direct(&A, el, smem_u32(coef), pend, &s_pend_n, ts, &d);
            st = d.st;
            item = d.item;
            left = d.left;
            n_it = d.n_it;
            screened = d.screened;
            exact = d.exact;
            valid = d.valid;
            has_def = d.n_def != 0u;
            def = d.def;
            continue;
        }
        uint32_t passed = 0, seen = 0;
#pragma unroll 1
        for (int r = r0; r < kFtRounds; ++r) {
            const bool act = valid && !has_def;
            const uint64_t s0 = st;
            const PairHead h = pair_head(A.sc, pow2, s0);
            bool pass = act;
            if (on) {
                uint32_t pk[16];
                const uint16_t *ya = yt + h.ea * kFtStride, *yb = yt + h.eb * kFtStride;
                uint64_t sb = s0 + 3 * kGolden;  // crossover bit draw of gene 0
#pragma unroll
                for (int k = 0; k < 32; k += 2) {
                    uint32_t lo = 0, hi = 0;
                    if (k < kNtot) {
                        lo = ((static_cast<int32_t>(draw_bitword(sb)) < 0) ? yb : ya)[k];
                        sb += 2 * kGolden;
                    }
                    if (k + 1 < kNtot) {
                        hi = ((static_cast<int32_t>(draw_bitword(sb)) < 0) ? yb : ya)[k + 1];
                        sb += 2 * kGolden;
                    }
                    pk[k >> 1] = lo | (hi << 16);
                }
                if (h.jump && !h.imm) {  // the jump's value in its gene's place (rounded as the genes are)
                    const uint32_t j = draw_hi(s0 + 62 * kGolden) % 29u;
                    const float v = static_cast<float>(draw_vh(s0 + 63 * kGolden) >> 8) * (1.0f / 16777216.0f);
                    const uint32_t hv = __half_as_ushort(__float2half_rn(v));
#pragma unroll
                    for (int k = 0; k < 15; ++k)
                        if (static_cast<uint32_t>(k) == j >> 1)
                            pk[k] = (j & 1u) ? (pk[k] & 0xffffu) | (hv << 16) : (pk[k] & 0xffff0000u) | hv;
                }
                if (!act)
#pragma unroll
                    for (int k = 0; k < 16; ++k) pk[k] = 0u;
                if (!ft_round(tg, pk, tid & 127u, &s_gbad[grp], &s_fail_phase[grp])) tc_ok = false;
                float f2 = 0.0f, l1 = 0.0f;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float d[16];
                    tc_ld16(tg.tmem_ld + 16u * half, d);
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        const int q = 16 * half + k;
                        if (q < kNtot) {
                            const float2 yh = __half22float2(*reinterpret_cast<const __half2 *>(&pk[q >> 1]));
                            const float g = __fmaf_rn(d[k], A.fp.dscale, A.fm.wlin[q]);
                            l1 = __fadd_rn(l1, fabsf(g));
                            f2 = __fmaf_rn((q & 1) ? yh.y : yh.x, __fadd_rn(g, A.fm.wlin[q]), f2);
                        }
                    }
                }
                const float b = __fadd_rn(__fmaf_rn(A.fp.s, l1, __fmaf_rn(0.5f, f2, A.fm.w0)), A.fp.c0);
                pass = act && (h.imm || !(b < tlo));  // immigrants are always scored; a NaN bound is never trusted
                seen += act ? 1u : 0u;
                passed += pass ? 1u : 0u;
            }
            if (pass) {
                const unsigned int slot = atomicAdd(&s_pend_n, 1u);
                const Item it = A.items[item];
                const uint64_t draw = (s0 - stream_seed(A.seed, it.stream)) * kGoldenInv - 1;
                const Pend q{item, n_it - left, static_cast<uint32_t>(draw - it.draw0)};
                if (slot < kPendCap) {
                    pend[slot] = q;
                } else {
                    has_def = true;
                    def = q;
                }
            }
            if (act) {
                st = h.next;
                if (--left == 0) {
                    item = gridDim.x * kThreads + atomicAdd(&A.ctrl->next_item, 1u);
                    start_item();
                }
            }
        }
        if (on) {
            atomicAdd(&s_seen, seen);
            atomicAdd(&s_passed, passed);
        }
    }
    Entry *out = A.lists + static_cast<size_t>(blockIdx.x) * A.kpad;
    for (uint32_t i = tid; i < A.kpad; i += kThreads) out[i] = E[i];
    unsigned long long scr = screened, exa = exact;
    for (int o = 16; o > 0; o >>= 1) {
        scr += __shfl_down_sync(0xffffffffu, scr, o);
        exa += __shfl_down_sync(0xffffffffu, exa, o);
    }
    if ((tid & 31) == 0) {
        atomicAdd(&A.ctrl->screened, scr);
        atomicAdd(&A.ctrl->exact_evals, exa);
    }
    if (!tc_ok) atomicOr(&A.ctrl->err, kErrTc);
    __syncthreads();
    if (s_gbad[grp] != 0u && tg.issuer) (void)mbar_wait(tg.mbar, s_fail_phase[grp]);  // bounded
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tc_dealloc(s_tbase, 64);
}

// Shared memory: the sort buffer, the coefficients, the queue, the selection scratch, the FP16
// parent table, two X tiles and the B tile (1 KB aligned), with el_smem the
// elite table.
size_t full_prune_smem(uint32_t sort_n, int ne, int num_sms, bool el_smem) {
    return static_cast<size_t>(sort_n) * sizeof(Entry) + kPendCap * sizeof(Pend) + 3ull * num_sms * sizeof(uint32_t) +
           static_cast<size_t>(ne) * kFtStride * sizeof(uint16_t) + 1024 + 2 * kFtTile + kFtB +
           (kFtCoef + (el_smem ? static_cast<size_t>(ne + 1) * kNtot + 3 : 0)) * sizeof(float);
}

// The bound's constants; false when they cannot be certified (weights too large
// or not finite, an exponent out of range).
//
// Rounding. Qs 2^-e rounds to FP16 by dq_kj (computed here); with the MMA's
// exact products and an FP32 accumulation taken as losing at most 2^-18 of its
// absolute sum, |2^e D_k - (Qs yh)_k| <= eps_k = sum_j (dq_kj + 2^-18 (|Qs_kj| +
// dq_kj)), which raises the bound by at most (s + 1/2) sum eps_k. The bound's
// own f32 sums (at most 64 roundings along a chain, over magnitudes of |w0| + 3
// sum |w| + 6 sum |Q|) and the score's FMA order (each term at most 59
// roundings, over |w0| + sum |w| + sum |Q|) are covered by gamma_64 twice.
bool make_full_prune(const csx_model_full &m, float sigma, FullPrune *t) {
    double qs[29][29], qsum = 0.0, lsum = 0.0, qmax = 0.0;
    float qf[29][29], d[29];
    for (int i = 0; i < kNtot; ++i) {
        lsum += std::fabs(static_cast<double>(m.w_lin[i]));
        for (int j = 0; j <= i; ++j) {
            const float q = m.w_quad[i * (i + 1) / 2 + j];
            qsum += std::fabs(static_cast<double>(q));
            qf[i][j] = qf[j][i] = i == j ? 2.0f * q : q;
        }
    }
    const double w0 = std::fabs(static_cast<double>(m.w0)), a_ref = w0 + lsum + qsum;
    if (!std::isfinite(a_ref) || a_ref > 1e30) return false;
    for (int i = 0; i < kNtot; ++i)
        for (int j = 0; j < kNtot; ++j) {
            qs[i][j] = static_cast<double>(qf[i][j]);
            qmax = std::max(qmax, std::fabs(qs[i][j]));
        }
    int e = 0;
    if (qmax > 0.0) {
        e = std::ilogb(qmax) + 1 - 15;
        if (e < -126 || e > 127) return false;
    }
    double eps = 0.0;
    std::memset(t->btile, 0, sizeof(t->btile));
    for (int n = 0; n < kNtot; ++n)
        for (int k = 0; k < kNtot; ++k) {
            const __half h = __float2half_rn(static_cast<float>(std::ldexp(qs[n][k], -e)));
            const double back = std::ldexp(static_cast<double>(__half2float(h)), e);
            if (!std::isfinite(back)) return false;
            const double dq = std::fabs(back - qs[n][k]);
            eps += dq + std::ldexp(1.0, -18) * (std::fabs(qs[n][k]) + dq);
            const int off = (n >> 3) * 512 + (k >> 3) * 128 + (n & 7) * 16 + (k & 7) * 2;
            t->btile[off / 2] = *reinterpret_cast<const uint16_t *>(&h);
        }
    // Whether the bound can rule out much: its mean slack s sum |grad_k| + c0
    // against the score's spread over uniform genes (s.d. from the gradient at
    // the centre and the products' variances). The K-th score lies some five
    // s.d. up: at a slack of 2 the bound leaves under 1% of the candidates (ten
    // seeded surfaces at sigma 0.12), at 3.6 to 4.1 it leaves 7 to 27% (sigma
    // 0.2), at 6 nearly all, where the unpruned kernel is faster (16.5 ms
    // against 25 at 2.65e8 with every candidate scored).
    double var = 0.0, slack = 0.0;
    const double s0 = std::min(std::fabs(static_cast<double>(sigma)), 1.0);
    for (int k = 0; k < kNtot; ++k) {
        double a = static_cast<double>(m.w_lin[k]), v = 0.0;
        for (int j = 0; j < kNtot; ++j) {
            a += 0.5 * qs[k][j];
            v += qs[k][j] * qs[k][j] / 12.0;
            if (j < k) var += qs[k][j] * qs[k][j] / 144.0;
        }
        var += a * a / 12.0 + 0.25 * qs[k][k] * qs[k][k] / 180.0;
        slack += 0.8 * s0 * std::sqrt(a * a + v);
    }
    quad_diag<kNtot>(qf, d);
    double dsum = 0.0;
    for (int k = 0; k < kNtot; ++k) dsum += static_cast<double>(d[k]);
    const double up = 1.0 + std::ldexp(1.0, -20), u = std::ldexp(1.0, -24), g64 = 64 * u / (1.0 - 64 * u);
    const double s = std::min(std::fabs(static_cast<double>(sigma)) + std::ldexp(1.0, -24), 1.0) + std::ldexp(1.0, -12);
    const double c0 = s * s * dsum * up;
    if (slack + c0 > 3.2 * std::sqrt(var)) return false;
    const double a_bound = w0 + 3.0 * lsum + 6.0 * qsum + c0;
    const double err = (2.0 * g64 * a_bound + g64 * a_ref + (s + 0.5) * eps) * up + 1e-30;
    if (!std::isfinite(err) || err > 1e30 || !std::isfinite(c0)) return false;
    t->dscale = std::ldexp(1.0f, e);
    t->s = std::nextafter(static_cast<float>(s), INFINITY);
    t->c0 = std::nextafter(static_cast<float>(c0), INFINITY);
    t->err = std::nextafter(static_cast<float>(err), INFINITY);
    return true;
}

}  // namespace csx
