// csx_dense.cuh — item building for small generations: every draw is hashed
// once and blocks of draws are mapped entry to exit, so that no thread walks
// a long chain.
// Part of csx_screen.cu's translation unit (included there, in order); not a
// standalone header.
//
// A candidate starting at draw p has its immigrant test at p + 2 and its jump
// test at p + 32 (immigrant) or p + 61, and is 33, 35, 62 or 64 draws long
// (src/screen.zig:225-250), so a chain of candidates enters a block of draws
// at one of its first 64 draws and leaves it into one of the next block's
// first 64. Both tests of a draw are the top 24 bits of one hash. A block's
// map (exit and candidate count of each of the 64 entries) needs no knowledge
// of where the truth enters; maps compose, and the truth enters stream t's
// first block at 0. Blocks are the work items.
//
// Against the walk of csx_pipeline.cuh this hashes 62 draws per candidate
// instead of two tests, but its longest chain is the composition (some tens
// of shared-memory steps) where the walk's is a segment and the link's the
// rarest of the chain meetings (tens of thousands of candidates on one warp).
// What bounds it is issue: the hashes, and 64 chains per block. Items of 8 to
// 16 candidates also put more of the screen's threads to work. At 2e5
// candidates (T = 4) items 0.50 -> 0.057 ms and screen 0.29 -> 0.14; at 1e6
// items 0.70 -> 0.147 and screen 0.29 -> 0.16.
#pragma once

namespace csx {

constexpr uint32_t kDenseGroup = 32;  // blocks per group: one CTA maps and composes them
// A group's scratch in the checkpoint array, in 8-byte words: its blocks' maps
// (64 x 16 bits each) and its own map (64 x 32 bits).
constexpr uint32_t kDenseWords = kDenseGroup * 64 * 2 / 8 + 64 * 4 / 8;
constexpr uint32_t kDenseTile = 512;  // groups composed per step of a stream's CTA

struct DenseGeom {
    uint32_t b_log2;  // draws per block
    uint32_t gps;     // groups per stream
};

// Maps of one group's blocks and of the group: entry e -> exit | count << 6.
__global__ void __launch_bounds__(256) dense_map_kernel(SynthConst sc, StreamGeom g, DenseGeom d,
                                                        uint64_t *__restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t B = 1u << d.b_log2, n_draws = kDenseGroup * B + 64, words = n_draws / 32;
    uint32_t *imm = reinterpret_cast<uint32_t *>(smem_raw), *jmp = imm + words;
    uint16_t *maps = reinterpret_cast<uint16_t *>(jmp + words);
    const uint32_t gid = blockIdx.x, tl = gid / d.gps, gi = gid - tl * d.gps;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t first = static_cast<uint64_t>(gi) * kDenseGroup * B;
    uint64_t st = stream_seed(g.seed, g.t0 + tl) + (first + tid + 1) * kGolden;
    for (uint32_t w = warp; w < words; w += 8) {  // warp w's lanes take draws 32 w .. 32 w + 31
        const uint32_t k24 = draw_vh(st) >> 8;
        st += 256 * kGolden;
        const uint32_t bi = __ballot_sync(0xffffffffu, k24 < sc.imm_thr);
        const uint32_t bj = __ballot_sync(0xffffffffu, k24 < sc.jump_thr);
        if (lane == 0) {
            imm[w] = bi;
            jmp[w] = bj;
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < kDenseGroup * 64; i += 256) {
        const uint32_t b0 = (i >> 6) * B, end = b0 + B;
        uint32_t p = b0 + (i & 63u), n = 0;
        while (p < end) {
            const uint32_t qi = p + 2;
            const bool im = (imm[qi >> 5] >> (qi & 31u)) & 1u;
            const uint32_t qj = p + (im ? 32u : 61u);
            const bool ju = (jmp[qj >> 5] >> (qj & 31u)) & 1u;
            p = qj + (ju ? 3u : 1u);
            ++n;
        }
        maps[i] = static_cast<uint16_t>((p - end) | (n << 6));  // at most B / 33 + 1 candidates
    }
    __syncthreads();
    uint64_t *dst = scratch + static_cast<uint64_t>(gid) * kDenseWords;
    for (uint32_t i = tid; i < kDenseGroup * 64 * 2 / 16; i += 256)
        reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(maps)[i];
    if (tid < 64) {
        uint32_t e = tid, n = 0;
        for (uint32_t b = 0; b < kDenseGroup; ++b) {
            const uint32_t m = maps[b * 64 + e];
            n += m >> 6;
            e = m & 63u;
        }
        reinterpret_cast<uint32_t *>(dst + kDenseGroup * 16)[tid] = e | (n << 6);
    }
}

// One CTA per stream: the truth's entry and index at every group, and each
// group's item count (its blocks with a candidate of the stream's my). The
// groups of a tile compose in sixteen chunks in parallel; one thread carries
// the truth over the chunks, and sixteen threads carry it inside them.
__global__ void __launch_bounds__(1024) dense_chain_kernel(StreamGeom g, DenseGeom d,
                                                           const uint64_t *__restrict__ scratch,
                                                           SegOut *__restrict__ outs, Ctrl *__restrict__ ctrl) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *tile = reinterpret_cast<uint32_t *>(smem_raw);  // kDenseTile x 64
    __shared__ uint32_t cmap[16][64];
    __shared__ uint32_t s_e[17];
    __shared__ uint64_t s_i[17];
    __shared__ uint32_t s_end_e, s_end_g;
    __shared__ uint64_t s_end_i;
    const uint32_t tl = blockIdx.x, tid = threadIdx.x;
    const uint64_t my = g.t0 + tl == g.T - 1 ? g.my_last : g.per;
    const uint64_t *src = scratch + static_cast<uint64_t>(tl) * d.gps * kDenseWords;
    SegOut *out = outs + static_cast<uint64_t>(tl) * d.gps;
    const uint64_t gdraws = static_cast<uint64_t>(kDenseGroup) << d.b_log2;
    if (tid == 0) {
        s_e[16] = 0;
        s_i[16] = 0;
        s_end_g = 0xffffffffu;
    }
    for (uint32_t base = 0; base < d.gps; base += kDenseTile) {
        const uint32_t n = min(kDenseTile, d.gps - base), cs = (n + 15) / 16;
        __syncthreads();
        for (uint32_t i = tid; i < n * 64; i += 1024)
            tile[i] = reinterpret_cast<const uint32_t *>(src + static_cast<uint64_t>(base + (i >> 6)) * kDenseWords +
                                                         kDenseGroup * 16)[i & 63u];
        __syncthreads();
        {
            const uint32_t c = tid >> 6, j1 = min(n, (c + 1) * cs);
            uint32_t e = tid & 63u, cnt = 0;
            for (uint32_t j = c * cs; j < j1; ++j) {
                const uint32_t m = tile[j * 64 + e];
                cnt += m >> 6;
                e = m & 63u;
            }
            cmap[c][tid & 63u] = e | (cnt << 6);
        }
        __syncthreads();
        if (tid == 0) {
            uint32_t e = s_e[16];
            uint64_t idx = s_i[16];
            for (int c = 0; c < 16; ++c) {
                s_e[c] = e;
                s_i[c] = idx;
                const uint32_t m = cmap[c][e];
                idx += m >> 6;
                e = m & 63u;
            }
            s_e[16] = e;
            s_i[16] = idx;
        }
        __syncthreads();
        if (tid < 16) {
            uint32_t e = s_e[tid];
            uint64_t idx = s_i[tid];
            const uint32_t j1 = min(n, (tid + 1) * cs);
            for (uint32_t j = tid * cs; j < j1; ++j) {
                const uint32_t m = tile[j * 64 + e], cnt = m >> 6;
                SegOut o;
                o.pos = (base + j) * gdraws + e;
                o.I = idx;
                o.lo = 0;
                o.cnt = idx < my ? static_cast<uint32_t>(min(static_cast<uint64_t>(cnt), my - idx)) : 0u;
                o.nitems = idx < my ? kDenseGroup : 0u;
                if (idx < my && idx + cnt > my) {  // the stream ends inside this group (one thread sees it)
                    s_end_e = e;
                    s_end_i = idx;
                    s_end_g = base + j;
                }
                out[base + j] = o;
                idx += cnt;
                e = m & 63u;
            }
        }
    }
    __syncthreads();
    if (s_end_g != 0xffffffffu) {
        const uint16_t *bm = reinterpret_cast<const uint16_t *>(src + static_cast<uint64_t>(s_end_g) * kDenseWords);
        uint16_t *m16 = reinterpret_cast<uint16_t *>(smem_raw);
        for (uint32_t i = tid; i < kDenseGroup * 64; i += 1024) m16[i] = bm[i];
        __syncthreads();
        if (tid == 0) {
            uint32_t e = s_end_e, nb = 0;
            for (uint64_t idx = s_end_i; idx < my; ++nb) {
                const uint32_t m = m16[nb * 64 + e];
                idx += m >> 6;
                e = m & 63u;
            }
            out[s_end_g].nitems = nb;
        }
    }
    if (tid == 0 && s_i[16] < my) atomicOr(&ctrl->err, kErrAssemble);
}

// One warp per group: the truth through its blocks' maps, one item per block.
__global__ void __launch_bounds__(128) dense_emit_kernel(StreamGeom g, DenseGeom d,
                                                         const uint64_t *__restrict__ scratch,
                                                         const SegOut *__restrict__ outs,
                                                         const uint32_t *__restrict__ off, Item *__restrict__ items,
                                                         const Ctrl *__restrict__ ctrl) {
    __shared__ __align__(16) uint16_t maps[4][kDenseGroup * 64];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint64_t gid = static_cast<uint64_t>(blockIdx.x) * 4 + w;
    if (gid >= g.n_seg || ctrl->err) return;  // whole warps
    const SegOut o = outs[gid];
    if (o.nitems == 0) return;
    const uint4 *src = reinterpret_cast<const uint4 *>(scratch + gid * kDenseWords);
    for (uint32_t i = lane; i < kDenseGroup * 64 * 2 / 16; i += 32) reinterpret_cast<uint4 *>(maps[w])[i] = src[i];
    __syncwarp();
    const uint64_t tl = gid / d.gps;
    const uint64_t gdraws = static_cast<uint64_t>(kDenseGroup) << d.b_log2;
    const uint64_t gstart = (gid - tl * d.gps) * gdraws;
    uint32_t e = static_cast<uint32_t>(o.pos - gstart), n = 0, my_e = 0, my_n = 0, my_c = 0;
    for (uint32_t b = 0; b < kDenseGroup; ++b) {  // every lane follows the same chain
        const uint32_t m = maps[w][b * 64 + e];
        if (b == lane) {
            my_e = e;
            my_n = n;
            my_c = m >> 6;
        }
        n += m >> 6;
        e = m & 63u;
    }
    if (lane < o.nitems) {
        Item it;
        it.draw0 = gstart + (static_cast<uint64_t>(lane) << d.b_log2) + my_e;
        it.idx0 = o.I + my_n;
        it.stream = static_cast<uint32_t>(g.t0 + tl);
        it.n = min(my_c, o.cnt - my_n);
        items[off[gid] + lane] = it;
    }
}

}  // namespace csx
