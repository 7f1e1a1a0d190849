// csx_ties.cuh — exact tie order: the device half of the replay of a
// stream's heap (src/screen.zig:151-193,306-319).
// Part of csx_screen.cu's translation unit (included there, in order); not a
// standalone header.
//
// The reference keeps each stream's top-K in a binary min-heap that rejects a
// candidate scoring <= its root, then stable-sorts the concatenated heap
// arrays by score. Candidates with exactly equal f32 scores from one stream
// therefore rank by their final heap-array positions, and at the K-th score
// the heap's history decides which of them survive. The screen ranks ties
// by (stream, index) instead; for the streams where that can differ the host
// replays the stream's heap (csx_screen.cu, fix_ties) from the candidates
// these kernels collect.
#pragma once

namespace csx {

// A candidate of the replayed stream: its stream-local index, first draw and
// reference-order score.
struct TieHit {
    uint64_t index, draw;
    float score;
    uint32_t pad_;
};

// Every candidate of stream `stream` with stream-local index in [a, b) whose
// score exceeds thr (all of them when `all`), appended to out (at most cap;
// *count counts every append, so a count above cap reports an overflow).
// One thread per work item of the generation; items of other streams or
// ranges return at once.
template <bool kFastDelta, class Args>
__global__ void tie_collect_kernel(const __grid_constant__ Args A, uint64_t n_items, uint32_t stream, uint64_t a,
                                   uint64_t b, float thr, int all, TieHit *__restrict__ out,
                                   unsigned int *__restrict__ count, unsigned int cap) {
    const uint64_t seed_t = stream_seed(A.seed, stream);
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_items;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const Item it = A.items[i];
        if (it.stream != stream || it.idx0 >= b || it.idx0 + it.n <= a) continue;
        uint64_t p = it.draw0;
        for (uint32_t c = 0; c < it.n; ++c) {
            const uint64_t idx = it.idx0 + c;
            if (idx >= b) break;
            const CandHead h = cand_head(A.sc, seed_t, p);
            if (idx >= a) {
                const float s = cand_score<kFastDelta>(A, A.el, seed_t, p, h);
                if (all || s > thr) {
                    const unsigned int slot = atomicAdd(count, 1u);
                    if (slot < cap) out[slot] = TieHit{idx, p, s, 0u};
                }
            }
            p += h.len;
        }
    }
}

// The same for a generation the pruning screen ran, whose pair tables are still
// there: only candidates that the pair's and the mask's bounds leave a chance
// above thr are scored, a warp's worth at a time. Scoring every candidate of a
// stream took 12.3 ms where a 2.65e9 generation held one tie. count[0]: hits;
// count[1]: candidates scored (where that is most of a chunk, the host goes on
// without the tables: elites that are alike and near the top, 1e9 candidates
// replayed in 97 ms with them throughout, 72 so).
constexpr uint32_t kTieQueue = 64;

__global__ void __launch_bounds__(256) tie_collect_pruned_kernel(const __grid_constant__ PruneArgs A, uint64_t n_items,
                                                                 uint32_t stream, uint64_t a, uint64_t b, float thr,
                                                                 TieHit *__restrict__ out,
                                                                 unsigned int *__restrict__ count, unsigned int cap) {
    __shared__ uint64_t q_st[8][kTieQueue], q_idx[8][kTieQueue], r_st[8][kTieQueue], r_idx[8][kTieQueue];
    __shared__ uint32_t q_meta[8][kTieQueue];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint64_t seed_t = stream_seed(A.seed, stream);
    const bool pow2 = (A.sc.ne & (A.sc.ne - 1)) == 0;
    const float tlo = __fsub_rd(thr, A.pc.err);
    uint32_t n1 = 0, n2 = 0;  // queued after the pair's test (q), after the mask's (r)
    uint32_t scored = 0;      // by this lane
    auto score = [&](uint64_t st, uint64_t idx) {
        const uint64_t p = (st - seed_t) * kGoldenInv - 1;
        const float s = exact_score_at<true>(&A, A.el, seed_t, p);
        ++scored;
        if (s > thr) {
            const unsigned int slot = atomicAdd(count, 1u);
            if (slot < cap) out[slot] = TieHit{idx, p, s, 0u};
        }
    };
    auto drain = [&](bool all) {
        while (n1 >= 32 || (all && n1 > 0)) {
            __syncwarp();
            const uint32_t nb = min(n1, 32u);
            n1 -= nb;
            bool pass = false;
            uint64_t st = 0, idx = 0;
            if (lane < nb) {
                st = q_st[warp][n1 + lane];
                idx = q_idx[warp][n1 + lane];
                const uint32_t meta = q_meta[warp][n1 + lane];
                pass = (meta & (1u << 30)) != 0u || mask_passes(A, st, meta, tlo);
            }
            const uint32_t m = __ballot_sync(0xffffffffu, pass);
            if (pass) {
                r_st[warp][n2 + __popc(m & lt)] = st;
                r_idx[warp][n2 + __popc(m & lt)] = idx;
            }
            n2 += __popc(m);
            if (n2 >= 32) {
                __syncwarp();
                n2 -= 32;
                score(r_st[warp][n2 + lane], r_idx[warp][n2 + lane]);
            }
        }
        if (all && n2 > 0) {
            __syncwarp();
            if (lane < n2) score(r_st[warp][lane], r_idx[warp][lane]);
            n2 = 0;
        }
        __syncwarp();
    };
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t w0 = static_cast<uint64_t>(blockIdx.x) * blockDim.x + warp * 32; w0 < n_items; w0 += stride) {
        const uint64_t i = w0 + lane;
        uint32_t left = 0;
        uint64_t st = 0, idx = 0;
        if (i < n_items) {
            const Item it = A.items[i];
            if (it.stream == stream && it.idx0 < b && it.idx0 + it.n > a) {
                left = static_cast<uint32_t>(min(static_cast<uint64_t>(it.n), b - it.idx0));
                st = seed_t + (it.draw0 + 1) * kGolden;
                idx = it.idx0;
            }
        }
        while (__any_sync(0xffffffffu, left > 0)) {
            const PairHead h = pair_head(A.sc, pow2, st);
            const bool pass = left > 0 && idx >= a && (h.imm || h.jump || !(A.u0[h.ea * A.sc.ne + h.eb] < tlo));
            const uint32_t m = __ballot_sync(0xffffffffu, pass);
            if (pass) {
                const uint32_t slot = n1 + __popc(m & lt);
                q_st[warp][slot] = st;
                q_idx[warp][slot] = idx;
                q_meta[warp][slot] = pair_meta(h);
            }
            n1 += __popc(m);
            if (n1 >= 32) drain(false);
            if (left > 0) {
                st = h.next;
                ++idx;
                --left;
            }
        }
    }
    drain(true);
    scored = __reduce_add_sync(0xffffffffu, scored);
    if (lane == 0 && scored) atomicAdd(count + 1, scored);
}

// Survivor records of the candidates at (stream, draw, index): genes and
// lineage regenerated, the score in the reference's order (the full
// surface's with FullScreenArgs).
template <bool kFastDelta, class Model>
__device__ void tie_regen_one(const Model &m, const SynthConst &sc, uint64_t seed, const float *el,
                              const unsigned long long *ids, const unsigned int *tribes, const TieHit &t,
                              uint64_t stream, csx_survivor *o) {
    const uint64_t seed_t = stream_seed(seed, stream);
    const CandHead h = cand_head(sc, seed_t, t.draw);
    float genes[kNtot];
    const float s = cand_genes<kFastDelta>(m, sc, el, seed_t, t.draw, h, genes);
    csx_survivor v;
    v.score = s;
    v.tribe = tribes[h.ea];
    v.pa = ids[h.ea];
    v.pb = ids[h.eb];
    v.stream = stream;
    v.index = t.index;
    v.draw = t.draw;
#pragma unroll
    for (int k = 0; k < kNtot; ++k) v.g[k] = genes[k];
    v.reserved = 0;
    *o = v;
}

template <bool kFastDelta>
__global__ void tie_regen_kernel(const __grid_constant__ ScreenArgs A, const TieHit *__restrict__ hits,
                                 const uint64_t *__restrict__ streams, uint32_t n,
                                 const unsigned long long *__restrict__ ids, const unsigned int *__restrict__ tribes,
                                 csx_survivor *__restrict__ out) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) tie_regen_one<kFastDelta>(A.m, A.sc, A.seed, A.el, ids, tribes, hits[q], streams[q], out + q);
}

template <bool kFastDelta>
__global__ void tie_regen_full_kernel(const __grid_constant__ FullScreenArgs A, const TieHit *__restrict__ hits,
                                      const uint64_t *__restrict__ streams, uint32_t n,
                                      const unsigned long long *__restrict__ ids,
                                      const unsigned int *__restrict__ tribes, csx_survivor *__restrict__ out) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) tie_regen_one<kFastDelta>(A.fm, A.sc, A.seed, A.el, ids, tribes, hits[q], streams[q], out + q);
}

}  // namespace csx
