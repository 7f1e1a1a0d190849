// csx_gram.cuh — the refit's normal equations ΦᵀΦ and Φᵀy on the tensor
// cores, in fixed point: each row's products to 8.1 x 2^-56 of the product of
// their variables' largest values. Tables with an entry for which FP64 sums
// would be closer are left to the FP64 kernel.
// Part of csx_surrogate.cu's translation unit (included there); not a
// standalone header.
//
// Reference: brain/evolve.py:250-268 (numpy FP64 normal equations of the
// features [1 | genes | g_i g_j, j <= i < 16]).
//
// The FP64 pipe of this GPU does two multiply-adds per SM and clock, so the
// 11781 products per row (153 features) took 8.8 ms at 400,000 rows at that
// pipe's full rate. Here each feature value is a 56-bit integer cut into
// seven signed 8-bit digits, held as FP16 (exact), and
//   Σ_r φ φ' = Σ_{i+j<=6} 2^(-14-8(i+j)) Σ_r d_i d'_j + (digits past the seventh)
// is 28 FP16 MMAs per pair of tiles with FP32 accumulation in tensor memory.
// A digit product is at most 2^14 and at most seven of them share an
// accumulator, so 128 rows stay below 2^24 and the accumulation is exact;
// then the accumulators are added to 64-bit integers. The digits and partial
// sums are integers: the result does not depend on any order. (Splitting FP64
// products over low-precision exact products: Ozaki, Ogita, Oishi, Rump 2012,
// "Error-free transformations of matrix multiplication".)
//
// Rows of the MMA. An entry of ΦᵀΦ is a sum of products of four variables of
// x = [g_0 .. g_15, 1] (or of one of the linear-only genes and a feature).
// With the 17 variables in three parts, two of any four lie in the same part:
// every entry is (a pair inside a part) x (a feature). So 57 rows (6·7/2 +
// 6·7/2 + 5·6/2 pairs), the linear-only genes and y are multiplied with all
// features, instead of all features with all.
//
// Scale. Gene a's values are at most 2^E_a (E_a from a pass over the table);
// a gene is its 24-bit significand and its exponent below E_a, a product of
// two genes a 48-bit integer shifted by both and rounded to 2^-55 of
// 2^(E_a+E_b). A table with an infinite or NaN entry is left to the FP64
// kernel.
//
// Small entries. The rounding is relative to the scale 2^(E_a+E_b+E_c+E_d) of
// an entry Σ_r φ φ', not to the entry: two genes that are never large together
// leave products of 1e-9 with 25 bits, and their squares with eight. The
// errors of n rows (8.1 x 2^-56 of the scale at most each; by chance their
// sum's s.d. is about sqrt(n) 2^-57 of it) are below the 2^-54 of the last
// rounding of an FP64 sum where the entry's magnitude Σ_r |φ φ'| is at least
// sqrt(n) / 8 of its scale. So every entry is held against that line
// (kGmSmall): where one of them, or one of Φᵀy by the sum of φ |y| (a row of
// its own), is below, the FP64 kernel takes the table. A sum whose terms cancel
// (genes of both signs) can only be taken for small. Largest error over the
// entries, in units of 2^-53 of the entry, fixed point / FP64 sums, emulated at
// 4,999 rows: uniform genes 1.0/3.3, a population 1.1/3.3, its genes and 1%
// immigrants 1.1/3.0; two genes of which one is 100 times smaller in every
// row 615/3.0, 1e4 times 4e5/3.2. Such a table takes the FP64 kernel's time and
// the fixed point's: 400,000 rows of 16 genes 9.5 ms instead of 0.69, 4,999 of
// 29 0.20 instead of 0.054. The check costs the others 2 to 16 us (two launches
// that leave at once, and from 22 genes on one digit per A tile).
#pragma once

namespace {

constexpr int kDigits = 7;
constexpr int kGmRows = 32;       // table rows per stage
// Stages between drains: 128 rows keep the FP32 sums exact where seven digit
// products share an accumulator, 256 where four do (stacked digits).
constexpr int kGmDrain = 4;
constexpr int kGmN = 64;          // features per column block
constexpr int kGmBlocks = 3;      // column blocks (166 features at most)
constexpr int kGmChunks = 50;     // row chunks: 150 CTAs
constexpr int kGmOutRows = 72;    // pair rows (57) + linear-only genes (13) + y + |y|
constexpr int kGmTasks = 544;     // digit tasks per stage, one per thread: 136 values x 4 groups of 8 rows
constexpr int kGmThreads = kGmTasks + 32;  // and a warp that issues the MMAs (it waits where their queue is full)
constexpr double kGmSmall = 0.125;  // an entry's magnitude over sqrt(n) scales from which fixed point is taken
constexpr int kGmVars = 32;       // variables per row: g_0..g_15, 1, linear-only genes
constexpr uint32_t kGmA = 128 * kGmRows * 2, kGmB = kGmN * kGmRows * 2;  // bytes of one digit's tiles
constexpr uint32_t kGmBuf = kDigits * (kGmA + kGmB);
constexpr size_t kGmPartBytes = static_cast<size_t>(kGmChunks) * kGmBlocks * kGmOutRows * kGmN * sizeof(longlong2);
constexpr size_t kGmSmem = 1024 + 2 * kGmBuf + kGmRows * (kGmVars - 1) * sizeof(int2) + kGmRows * sizeof(int64_t);

// What the range pass leaves: the largest |value| of each gene (as f32 bits)
// and of y (as FP64 bits); the flag of a wait that gave up, and of a table with
// an entry too small beside its scale.
struct GramRange {
    unsigned long long ymax;
    uint32_t gmax[kMaxLin];
    uint32_t err;
    uint32_t small;
};

__device__ __forceinline__ bool gram_finite(const GramRange *r, int ng) {
    bool ok = (r->ymax >> 52) < 2047;
    for (int k = 0; k < ng; ++k) ok = ok && (r->gmax[k] >> 23) < 255;
    return ok;
}

// Whether the fixed-point sums stand (known once sg_gram_final_kernel is through).
__device__ __forceinline__ bool gram_fixed(const GramRange *r, int ng) { return r->small == 0 && gram_finite(r, ng); }

// E with |x| <= 2^E for every |x| whose f32 bits are at most `bits`.
__device__ __forceinline__ int range_exp(uint32_t bits) {
    if (bits == 0) return 0;
    const int e = static_cast<int>(bits >> 23);
    if (e == 0) return 32 - __clz(bits - 1) - 149;  // subnormal: bits x 2^-149
    return e - 127 + ((bits & 0x7fffffu) ? 1 : 0);
}
__device__ __forceinline__ int range_exp64(unsigned long long bits) {
    if (bits == 0) return 0;
    const int e = static_cast<int>(bits >> 52);
    if (e == 0) return -1022;
    return e - 1023 + ((bits & 0xfffffffffffffull) ? 1 : 0);
}

__global__ void __launch_bounds__(256) sg_range_kernel(int ng, const float *__restrict__ genes, int64_t n, int ldg,
                                                       const double *__restrict__ fit, GramRange *__restrict__ out) {
    // eight rows in flight per warp; up to 16 genes two rows per load (the lane's
    // upper half takes the second)
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int two = ng <= 16 ? 1 : 0, col = two ? lane & 15 : lane, sub = two ? lane >> 4 : 0;
    const int64_t step = nw << two;
    uint32_t m = 0;
    unsigned long long my = 0;
#pragma unroll 8
    for (int64_t r = (w0 << two) + sub; r < n; r += step)
        if (col < ng) m = max(m, __float_as_uint(genes[r * ldg + col]) & 0x7fffffffu);
    if (fit) {
#pragma unroll 4
        for (int64_t r = w0 * 32 + lane; r < n; r += nw * 32)
            my = max(my, static_cast<unsigned long long>(__double_as_longlong(fit[r])) & 0x7fffffffffffffffull);
        for (int o = 16; o > 0; o >>= 1) my = max(my, __shfl_xor_sync(0xffffffffu, my, o));
    }
    if (two) m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
    // one update per CTA and column: an update per warp spent 65 us on the 30
    // addresses at 400,000 rows
    __shared__ uint32_t sm[8][32];
    __shared__ unsigned long long sy[8];
    const int warp = threadIdx.x >> 5;
    sm[warp][lane] = m;
    if (lane == 31) sy[warp] = my;
    __syncthreads();
    if (warp == 0) {
        for (int w = 1; w < 8; ++w) m = max(m, sm[w][lane]);
        if (lane < ng) atomicMax(&out->gmax[lane], m);
        if (lane == 31) {
            for (int w = 1; w < 8; ++w) my = max(my, sy[w]);
            atomicMax(&out->ymax, my);
        }
    }
}

// Pair rows: part of variable v (17 of them, 16 = the constant 1), and the row
// of the pair {a, b} of one part.
__host__ __device__ __forceinline__ int var_part(int v) { return v < 6 ? 0 : v < 12 ? 1 : 2; }
__host__ __device__ __forceinline__ int pair_row(int a, int b) {
    const int p = var_part(a), hi = (a > b ? a : b) - 6 * p, lo = (a > b ? b : a) - 6 * p;
    return 21 * p + tri(hi) + lo;
}
constexpr int kPairRows = 57;

// Row q of the A side as a pair of variables (linear-only gene k is variable
// 17 + k - 16; its partner is the 1); y is (255, 255), |y| (253, 253).
__device__ __forceinline__ void gram_row_vars(int q, int ng, int &a, int &b) {
    if (q < kPairRows) {
        const int p = q < 21 ? 0 : q < 42 ? 1 : 2;
        int i = 0;
        while (tri(i + 1) <= q - 21 * p) ++i;
        a = 6 * p + i;
        b = 6 * p + (q - 21 * p - tri(i));
    } else if (q < kPairRows + ng - 16) {
        a = 17 + q - kPairRows;
        b = 16;
    } else {
        a = b = q == kPairRows + ng - 16 ? 255 : 253;
    }
}
// Feature f as a pair of variables, in the same numbering.
__device__ __forceinline__ void gram_feature_vars(int f, int ng, int &a, int &b) {
    feature_pair(f, ng, a, b);
    auto var = [ng](int x) { return x == ng ? 16 : x < 16 ? x : x + 1; };
    a = var(a);
    b = var(b);
}

__device__ __forceinline__ void gm_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc ? 1u : 0u)
        : "memory");
}

// The integer that v holds, |v| < 2^24, without the conversion unit (16 per SM
// and clock): its multiple of 4096 and the rest, each read off the significand.
__device__ __forceinline__ int exact_int(float v) {
    constexpr float kMagic = 12582912.0f;  // 1.5 x 2^23
    const float hm = __fmaf_rn(v, 1.0f / 4096.0f, kMagic);
    const float l = __fmaf_rn(__fsub_rn(hm, kMagic), -4096.0f, v);  // exact, |l| <= 2048
    const int h = __float_as_int(hm) - 0x4b400000, li = __float_as_int(__fadd_rn(l, kMagic)) - 0x4b400000;
    return h * 4096 + li;
}

// One CTA: the table rows of chunk blockIdx.x, the features of column block
// blockIdx.y. While a stage's MMAs run, the next stage's digits are made in the
// other buffer. part[(chunk, block)]: kGmOutRows x 64 x {hi, lo}; the chunk's
// sum is hi 2^-30 + lo 2^-62 of the row's times the feature's scale.
template <bool kStack>
__global__ void __launch_bounds__(kGmThreads, 1) sg_gram_mma_kernel(int ng, int nf, const float *__restrict__ genes,
                                                                   int64_t n, int ldg,
                                                                   const double *__restrict__ fit,
                                                                   GramRange *__restrict__ range,
                                                                   longlong2 *__restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long s_mbar[2];
    __shared__ uint32_t s_tbase, s_bad;
    __shared__ unsigned char s_va[kGmOutRows + kGmN], s_vb[kGmOutRows + kGmN];
    __shared__ int s_exp[kGmVars];
    if (!gram_finite(range, ng)) return;  // the FP64 kernel's table (every CTA alike)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t base = (csx::smem_u32(smem_raw) + 1023u) & ~1023u;
    unsigned char *bufs = smem_raw + (base - csx::smem_u32(smem_raw));
    int2 *vars = reinterpret_cast<int2 *>(bufs + 2 * kGmBuf);             // [row][kGmVars - 1]: significand, shift
    int64_t *yint = reinterpret_cast<int64_t *>(vars + kGmRows * (kGmVars - 1));  // y 2^(55 - E_y)
    const int n_rows = kPairRows + (ng - 16) + 2;                          // A rows in use
    const int f0 = blockIdx.y * kGmN, n_feat = min(kGmN, nf - f0);
    for (uint32_t i = tid; i < 2 * kGmBuf / 16; i += kGmThreads) reinterpret_cast<uint4 *>(bufs)[i] = uint4{0, 0, 0, 0};
    if (tid < kGmOutRows + kGmN) {
        int a = 254, b = 254;  // nothing there: the zeros stay
        if (tid < n_rows) gram_row_vars(tid, ng, a, b);
        else if (tid >= kGmOutRows && tid - kGmOutRows < n_feat) gram_feature_vars(f0 + tid - kGmOutRows, ng, a, b);
        s_va[tid] = static_cast<unsigned char>(a);
        s_vb[tid] = static_cast<unsigned char>(b);
    }
    if (tid < ng) s_exp[tid] = range_exp(range->gmax[tid]);
    if (warp == 0) csx::tc_alloc(csx::smem_u32(&s_tbase), 512);
    if (tid == 0) {
        csx::mbar_init(csx::smem_u32(&s_mbar[0]), 1);
        csx::mbar_init(csx::smem_u32(&s_mbar[1]), 1);
        s_bad = 0;
    }
    csx::tc_fence_before();
    __syncthreads();
    csx::tc_fence_after();
    const uint32_t tmem = s_tbase;
    const int y_exp = range_exp64(range->ymax);
    const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = static_cast<int64_t>(blockIdx.x) * chunk, hi = min(n, lo + chunk);
    const int stages = hi > lo ? static_cast<int>((hi - lo + kGmRows - 1) / kGmRows) : 0;

    // A stage's raw values, loaded a stage ahead of their use: thread tid takes
    // row tid / 16, genes tid % 16 and 16 + tid % 16 (the first 512 threads),
    // the last 32 threads y.
    const int lr = tid >> 4, lk = tid & 15;
    uint32_t x0 = 0, x1 = 0;
    unsigned long long xy = 0;
    auto load = [&](int t) {
        const int64_t r0 = lo + static_cast<int64_t>(t) * kGmRows;
        x0 = x1 = 0;
        xy = 0;
        if (tid < 512) {
            if (t < stages && r0 + lr < hi) {
                const float *src = genes + (r0 + lr) * static_cast<int64_t>(ldg);
                x0 = __float_as_uint(src[lk]);
                if (lk + 16 < ng) x1 = __float_as_uint(src[lk + 16]);
            }
        } else if (tid < kGmTasks && t < stages && fit && r0 + (tid - 512) < hi) {
            xy = static_cast<unsigned long long>(__double_as_longlong(fit[r0 + (tid - 512)]));
        }
    };
    // significand (bit 23 leading, 5 bits up) and exponent below the gene's largest
    auto split = [&](uint32_t x, int k) {
        int e = static_cast<int>((x >> 23) & 255u);
        int m = static_cast<int>((x & 0x7fffffu) | (e ? 0x800000u : 0u));
        if (e == 0) {  // subnormal or zero: the leading bit up to bit 23
            const int up = m ? __clz(m) - 8 : 0;
            m <<= up;
            e = 1 - up;
        }
        return make_int2(((x >> 31) ? -m : m) * 32, m ? s_exp[k] - (e - 127) : 0);
    };

    // the stage's variables, then its digits into buffer t & 1
    auto make = [&](int t) {
        const int64_t r0 = lo + static_cast<int64_t>(t) * kGmRows;
        if (tid < 512) {
            vars[lr * (kGmVars - 1) + lk] = split(x0, lk);
            if (lk + 16 < ng) vars[lr * (kGmVars - 1) + lk + 17] = split(x1, lk + 16);
            if (lk == 15) vars[lr * (kGmVars - 1) + 16] = make_int2(r0 + lr < hi ? 0x800000 * 32 : 0, 0);
        } else if (tid < kGmTasks) {  // y 2^(55 - E_y), rounded: its 53-bit significand 3 bits up, shifted by its exponent
            const int e = static_cast<int>((xy >> 52) & 2047u);
            int64_t m = static_cast<int64_t>((xy & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull)) << 4;
            if (xy >> 63) m = -m;
            const int sh = m ? max(0, min(63, y_exp - ((e ? e : 1) - 1023))) : 0;
            yint[tid - 512] = ((m >> sh) + 1) >> 1;
        }
        load(t + 1);
        // the digit warps alone: the issuing warp is still waiting on the MMA queue
        if (tid < kGmTasks) asm volatile("bar.sync 1, %0;" ::"n"(kGmTasks) : "memory");
        unsigned char *buf = bufs + (t & 1) * kGmBuf;
        constexpr int kF = kGmOutRows + kGmN;
        static_assert(kF * (kGmRows / 8) == kGmTasks, "one task per thread");
        const int kg = tid / kF, f = tid - kg * kF;
        const uint32_t a = tid < kGmTasks ? s_va[f] : 254u, b = tid < kGmTasks ? s_vb[f] : 254u;
        if (a != 254u) {
            uint32_t w[8][2];  // the integers, every digit offset by 128
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int r = kg * 8 + e;
                int64_t v;
                if (a == 255u || a == 253u) {
                    const int64_t yi = yint[r];
                    v = (a == 253u && yi < 0 ? -yi : yi) + 0x0080808080808080ll;
                } else {
                    const int2 va = vars[r * (kGmVars - 1) + a], vb = vars[r * (kGmVars - 1) + b];
                    const int64_t p = static_cast<int64_t>(va.x) * vb.x;  // the product, 10 bits up
                    v = ((p >> min(va.y + vb.y, 63)) + (1 + 2 * 0x0080808080808080ll)) >> 1;
                }
                w[e][0] = static_cast<uint32_t>(v);
                w[e][1] = static_cast<uint32_t>(v >> 32);
            }
            const int row = f < kGmOutRows ? f : f - kGmOutRows;
            unsigned char *dst = buf + (f < kGmOutRows ? 0u : kDigits * kGmA) + (row >> 3) * (kGmRows * 16) +
                                 kg * 128 + (row & 7) * 16;
            const bool is_a = f < kGmOutRows;
#pragma unroll
            for (int i = 0; i < kDigits; ++i) {  // digit i: byte 6 - i (the first with what lies above it)
                constexpr int kTop = 0;
                const int byte = 6 - i;
                uint32_t h[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t x = w[2 * e][byte >> 2], y = w[2 * e + 1][byte >> 2];
                    uint32_t t2;
                    if (i == kTop) {
                        t2 = __byte_perm(x, y, 0x7632) & 0x03ff03ffu;
                    } else {
                        const uint32_t c = byte & 3;
                        t2 = __byte_perm(x, y, ((4 + c) << 8) | c) & 0x00ff00ffu;
                    }
                    t2 |= 0x64006400u;  // FP16 1024 + byte
                    const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
                    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&t2), off);
                    h[e] = *reinterpret_cast<const uint32_t *>(&d);
                }
                const uint32_t at = !is_a ? i * kGmB
                                    : kStack ? (i >> 1) * kGmA + (i & 1) * (64 / 8) * (kGmRows * 16) : i * kGmA;
                *reinterpret_cast<uint4 *>(dst + at) = make_uint4(h[0], h[1], h[2], h[3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        csx::tc_fence_before();
        __syncthreads();
    };

    constexpr int kDrain = kStack ? 2 * kGmDrain : kGmDrain;
    constexpr uint32_t idesc = (1u << 4) | ((kGmN >> 3) << 17) | ((128u >> 4) << 24);  // FP16 x FP16 -> FP32
    int64_t acc_hi[16], acc_lo[16];  // warps 0..15: lane quarter warp % 4, 16 columns
#pragma unroll
    for (int c = 0; c < 16; ++c) acc_hi[c] = acc_lo[c] = 0;
    uint32_t phase[2] = {0u, 0u};
    bool ok = true;
    load(0);
    if (stages > 0) make(0);
    for (int t = 0; t < stages; ++t) {
        const bool first = t % kDrain == 0;
        if (tid == kGmTasks && s_bad == 0) {
            csx::tc_fence_after();
            const uint32_t a0 = base + (t & 1) * kGmBuf, b0 = a0 + kDigits * kGmA;
            // consecutive MMAs go to different accumulators
            for (int ks = 0; ks < kGmRows / 16; ++ks)
                for (int i = 0; i < kDigits; i += kStack ? 2 : 1)
                    for (int j = 0; i + j < kDigits; ++j)
                        gm_mma(tmem + (i + j) * kGmN,
                               csx::tc_sdesc(a0 + (kStack ? i >> 1 : i) * kGmA + ks * 256, 128, kGmRows * 16),
                               csx::tc_sdesc(b0 + j * kGmB + ks * 256, 128, kGmRows * 16), idesc,
                               !(first && i == 0 && ks == 0));
            csx::tc_commit(csx::smem_u32(&s_mbar[t & 1]));
        }
        __syncwarp();
        // the other buffer's MMAs (stage t - 1) were waited for below
        if (t + 1 < stages) make(t + 1);
        if (ok && !csx::mbar_wait(csx::smem_u32(&s_mbar[t & 1]), phase[t & 1])) {
            ok = false;
            s_bad = 1;
        }
        phase[t & 1] ^= 1u;
        csx::tc_fence_after();
        if (__syncthreads_or(!ok)) {  // a wait gave up: every thread leaves together
            ok = false;
            break;
        }
        if (t % kDrain == kDrain - 1 || t + 1 == stages) {
            const uint32_t ta = tmem + ((32u * (warp & 3)) << 16) + 16u * (warp >> 2);
            if (warp < 16) {
#pragma unroll
                for (int s = 0; s < kDigits; ++s) {
                    float r[16];
                    csx::tc_ld16(ta + s * kGmN, r);
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const int v = s & 1 ? exact_int(r[c]) : __float2int_rn(r[c]);
                        if (s < 3) acc_hi[c] += static_cast<int64_t>(v) * (1 << (8 * (2 - s)));
                        else acc_lo[c] += static_cast<int64_t>(v) * (1 << (8 * (6 - s)));
                    }
                }
#pragma unroll
                for (int c = 0; c < 16; ++c) {  // lo counts 2^-32 of hi's unit: what passes 32 bits moves up
                    acc_hi[c] += acc_lo[c] >> 32;
                    acc_lo[c] &= 0xffffffffll;
                }
            }
            csx::tc_fence_before();
            __syncthreads();
            csx::tc_fence_after();
        }
    }
    const int row = 32 * (warp & 3) + lane;
    if (kStack) {  // the rows above carry 2^-8 (their last 8 bits lie past 2^-62 and are dropped)
        longlong2 *up = reinterpret_cast<longlong2 *>(bufs);  // no MMA reads the buffers any more
        __syncthreads();
        if (warp < 16 && row >= 64)
#pragma unroll
            for (int c = 0; c < 16; ++c) up[(row - 64) * kGmN + 16 * (warp >> 2) + c] = make_longlong2(acc_hi[c], acc_lo[c]);
        __syncthreads();
        if (warp < 16 && row < 64) {
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const longlong2 u = up[row * kGmN + 16 * (warp >> 2) + c];
                acc_hi[c] += u.x >> 8;
                acc_lo[c] += ((u.x & 255) << 24) + (u.y >> 8);
            }
        }
    }
    if (warp < 16 && row < kGmOutRows) {
        longlong2 *dst = part + ((static_cast<int64_t>(blockIdx.x) * kGmBlocks + blockIdx.y) * kGmOutRows + row) * kGmN +
                         16 * (warp >> 2);
#pragma unroll
        for (int c = 0; c < 16; ++c) dst[c] = make_longlong2(acc_hi[c], acc_lo[c]);
    }
    if (!ok && tid == 0) {
        atomicOr(&range->err, 1u);
        // bounded: the MMAs of the wait that gave up still read the buffers
        (void)csx::mbar_wait(csx::smem_u32(&s_mbar[0]), phase[0] ^ 1u);
        (void)csx::mbar_wait(csx::smem_u32(&s_mbar[1]), phase[1] ^ 1u);
    }
    csx::tc_fence_before();
    __syncthreads();
    csx::tc_fence_after();
    if (warp == 0) csx::tc_dealloc(tmem, 512);
}

// Entry e of the packed lower triangle of ΦᵀΦ (i, j <= i), then of Φᵀy (i).
struct GramEntry {
    int i, j;
    bool live, right;
};
__device__ __forceinline__ GramEntry gram_entry(int nf, bool has_rhs) {
    const int e = blockIdx.x * 32 + threadIdx.x, n_gram = tri(nf);
    GramEntry r{0, 0, e < n_gram + (has_rhs ? nf : 0), e >= n_gram};
    if (!r.live) return r;
    if (r.right) {
        r.i = e - n_gram;
        return r;
    }
    r.i = static_cast<int>((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
    while (tri(r.i) > e) --r.i;
    while (tri(r.i + 1) <= e) ++r.i;
    r.j = e - tri(r.i);
    return r;
}
__device__ __forceinline__ void gram_store(const GramEntry &e, int nf, double v, double *gram, double *rhs) {
    if (e.right) {
        rhs[e.i] = v;
    } else {
        gram[static_cast<int64_t>(e.i) * nf + e.j] = v;
        gram[static_cast<int64_t>(e.j) * nf + e.i] = v;
    }
}

// Which row and feature of the MMA an entry is, the chunks' sums (eight threads
// per entry), its scale, and whether it is too small beside that.
__global__ void __launch_bounds__(32 * kSumSplit) sg_gram_final_kernel(int ng, int nf, int chunks, double small,
                                                                       GramRange *__restrict__ range,
                                                                       const longlong2 *__restrict__ part,
                                                                       double *__restrict__ gram,
                                                                       double *__restrict__ rhs) {
    __shared__ long long sh[kSumSplit][32], sl[kSumSplit][32];
    if (!gram_finite(range, ng)) return;
    const int y = threadIdx.y;
    const GramEntry en = gram_entry(nf, rhs != nullptr);
    int row = 0, col = 0, ex = 0;
    bool zero = false;  // a factor that is zero throughout: the sum is exact
    if (en.live) {
        auto expo = [&](int x) {
            if (x == 16) return 0;
            const uint32_t m = range->gmax[x < 16 ? x : x - 1];
            zero = zero || m == 0;
            return range_exp(m);
        };
        auto feature = [ng](int u, int w) {  // of two variables of the 17
            const int hi2 = u > w ? u : w, lo2 = u > w ? w : u;
            return hi2 < 16 ? 1 + ng + tri(hi2) + lo2 : lo2 < 16 ? 1 + lo2 : 0;
        };
        int a, b;
        gram_feature_vars(en.i, ng, a, b);
        ex = expo(a) + expo(b);
        if (en.right) {
            row = kPairRows + ng - 16;
            col = en.i;
            ex += range_exp64(range->ymax);
            zero = zero || range->ymax == 0;
        } else {
            int c, d;
            gram_feature_vars(en.j, ng, c, d);
            ex += expo(c) + expo(d);
            auto same = [](int u, int w) { return var_part(u) == var_part(w); };
            if (a > 16 || b > 16) row = kPairRows + (a > 16 ? a : b) - 17, col = en.j;
            else if (c > 16 || d > 16) row = kPairRows + (c > 16 ? c : d) - 17, col = en.i;
            else if (same(a, b)) row = pair_row(a, b), col = en.j;
            else if (same(c, d)) row = pair_row(c, d), col = en.i;
            else if (same(a, c)) row = pair_row(a, c), col = feature(b, d);
            else if (same(a, d)) row = pair_row(a, d), col = feature(b, c);
            else if (same(b, c)) row = pair_row(b, c), col = feature(a, d);
            else row = pair_row(b, d), col = feature(a, c);
        }
    }
    long long h = 0, l = 0, m = 0;  // m: the |y| row's high part
    if (en.live) {
        const longlong2 *src = part + (static_cast<int64_t>(col / kGmN) * kGmOutRows + row) * kGmN + col % kGmN;
        const int64_t step = static_cast<int64_t>(kGmBlocks) * kGmOutRows * kGmN;
#pragma unroll 4
        for (int q = y; q < chunks; q += kSumSplit) {
            const longlong2 x = src[q * step];
            h += x.x;
            l += x.y;
        }
        if (en.right)
            for (int q = y; q < chunks; q += kSumSplit) m += src[q * step + kGmN].x;
    }
    sh[y][threadIdx.x] = h;
    sl[y][threadIdx.x] = l;
    __syncthreads();
    if (y == 0) {
#pragma unroll
        for (int q = 1; q < kSumSplit; ++q) {
            h += sh[q][threadIdx.x];
            l += sl[q][threadIdx.x];
        }
    }
    __syncthreads();
    sh[y][threadIdx.x] = m;
    __syncthreads();
    if (!en.live || y != 0) return;
#pragma unroll
    for (int q = 1; q < kSumSplit; ++q) m += sh[q][threadIdx.x];
    // a scaled feature is Σ_i d_i 2^(-7-8i): the sum is Σ_s v_s 2^(-14-8s)
    const double f = (static_cast<double>(h) + scalbn(static_cast<double>(l), -32)) * 0x1p-30;  // in scales
    const double mag = en.right ? static_cast<double>(m) * 0x1p-30 : f;
    if (!zero && fabs(mag) < small) range->small = 1u;
    double v = scalbn(f, ex);
    if (range->err) v = __longlong_as_double(0x7ff8000000000000ll);  // a wait gave up: no result
    gram_store(en, nf, v, gram, rhs);
}

// The same from the FP64 kernel's parts, where the fixed-point sums don't stand.
__global__ void __launch_bounds__(32 * kSumSplit) sg_gram_fp64_final_kernel(int ng, int nf,
                                                                            const GramRange *__restrict__ range,
                                                                            const double *__restrict__ part_g,
                                                                            const double *__restrict__ part_r,
                                                                            int nparts, double *__restrict__ gram,
                                                                            double *__restrict__ rhs) {
    __shared__ double sp[kSumSplit][32];
    if (gram_fixed(range, ng)) return;
    const GramEntry en = gram_entry(nf, rhs != nullptr);
    const int bi = en.i / kGramBlk, bj = en.j / kGramBlk;
    const double *src = en.right ? part_r + en.i
                                 : part_g + (tri(bi) + bj) * (kGramBlk * kGramBlk) + (en.i % kGramBlk) * kGramBlk +
                                       en.j % kGramBlk;
    const int64_t npairs = gram_pairs(nf);
    const double v = sum_parts(src, nparts, en.right ? kFeatCap : npairs * kGramBlk * kGramBlk, en.live, sp);
    if (en.live && threadIdx.y == 0) gram_store(en, nf, v, gram, rhs);
}

}  // namespace
