// Encode for 8-wide and 4-wide groups with many rows: tcgen05 products filter, exact fp32 decides, a thread owns a row.
//
// A block is four groups of 128 threads; a group has a tile of 128 rows of one (head, group of channels), thread = row =
// tensor-memory lane, and 128 tensor-memory columns.  Per stage and half of the 256 words one thread issues two
// tcgen05.mma steps of 16 columns each: ones against -|c|^2/2 in three fp16 parts, and the row's fp16 split (hi | lo)
// against (word | word), which leaves the scores t = r.c - |c|^2/2 in tensor memory (the distance is |r|^2 - 2t).  The thread
// keeps the largest score of every four neighbouring words; the fours within a margin of the row's maximum are
// re-evaluated in the library's exact arithmetic, nearly always one four.  No value crosses threads.
//
// The exact argmin is among the re-evaluated words (encode_tc.cu has the argument and the bound, 2^-15 (xx + cc_max) plus
// 2^-18 sqrt(cc_max) in units of t; the three fp16 parts of -|c|^2/2 add 2^-25, the kernel 2^-23).  Rows or words outside
// fp16's range, and a product that never arrived, re-evaluate every word.
//
// Blocks split the tiles of all (head, group) pairs evenly, span by span of 16384 rows, and bring a pair's tables in when they
// enter it, so the chip stays full whatever the number of pairs; a table costs about one tile's time.
//
// Bound by latency between the phases of a stage at 16 warps an SM.  4 x 8192 fp16 rows x 8 heads, 16 x 8, two
// stages, rows wanted: 320 us a side, against 572 us for the mma.sync kernel of encode_tc.cu.  Whitened (fp32 words, a third product a
// half): 3001 fp32 rows x 8 heads, 32 x 4, one stage 47 us against 125 for the fp32 scan of all words.
// (Words as fp32 pairs in copies without bank conflicts, two exact chains an instruction: 372 us where this takes 344, as look-ups are scarcer than
// issue slots.)
//
// Reference statements: src/jointkv/closed_loop_vq.py:52-76 (search), :343-395 (stage recursion),
// src/jointkv/cq_tac.py:86-105.

#include "common.cuh"
#include "narrow_plan.cuh"

namespace tacvq {

namespace narrow {

constexpr int kThreads = kRows * kGroups, kHalf = kMaxWords / 2;
constexpr size_t kWordBytes = kMaxWords * 32, kSeedBytes = kMaxWords * 32, kNormBytes = kMaxWords * 4;
constexpr size_t kStageBytes = kWordBytes + kSeedBytes + kNormBytes;  // (word | word), seeds, |word|^2
// fp32 words: their fp16 rounding takes the place of the words above; what it leaves follows, (low | 0), and the words themselves
template <int DSUB, bool EXACT32>
constexpr size_t kStage = EXACT32 ? kStageBytes + kWordBytes + kMaxWords * DSUB * 4 : kStageBytes;
constexpr size_t kABytes = kRows * 32;                                // a group's (hi | lo) rows
constexpr size_t kFixedBytes = (1 + kGroups) * kABytes + 256;         // ones, rows, barriers
constexpr int kMaxStages = 12;                                        // and the length of the queue of codes
static_assert(kMaxStages * (kStageBytes + 4) + kFixedBytes <= 227 * 1024, "one block's tables");

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// blocks in which a wait was given up; expected to stay 0
__device__ unsigned int g_timeouts = 0;

constexpr int kSpins = 1 << 17;
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity, int spins) {
    int done = 0;
#pragma unroll 1
    for (int spin = 0; spin < spins && !done; ++spin)
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.s32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// 32 or 16 columns; the registers are valid when it returns
__device__ __forceinline__ void tmem_load(float (&v)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]),
          "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]),
          "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_load(float (&v)[16], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]),
          "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(taddr)
        : "memory");
}
// K-major rows of 32 bytes with the 32-byte swizzle: start address / 16 in bits 0-13, 256 bytes between groups of 8 rows in
// bits 32-45, version 1 in bits 46-47, swizzle mode 6 in bits 61-63 (16-byte piece c of row r sits at c ^ ((r >> 2) & 1))
__device__ __forceinline__ uint64_t descriptor(uint32_t smem_addr) {
    return ((uint64_t)((256u >> 4) | (1u << 14) | (6u << 29)) << 32) | (((smem_addr & 0x3ffffu) >> 4) | (1u << 16));
}
// fp32 accumulator (bits 4-5), fp16 operands, K-major, N / 8 in bits 17-22, M / 16 in bits 24-28
constexpr uint32_t kMmaShape = (1u << 4) | ((uint32_t)(kHalf >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem), "l"(a), "l"(b), "r"(kMmaShape), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// acc = 2 acc + b, two at a time
__device__ __forceinline__ void double_add2(float &acc0, float &acc1, float b0, float b1) {
    asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%4, %4};\nmov.b64 c, {%2, %3};\nfma.rn.f32x2 a, a, b, c;\nmov.b64 {%0, %1}, a;\n}"
        : "+f"(acc0), "+f"(acc1) : "f"(b0), "f"(b1), "f"(2.0f));
}
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ void unpack8(const uint4 raw, float (&v)[8]) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    const __half2 h[4] = {__floats2half2_rn(v[0], v[1]), __floats2half2_rn(v[2], v[3]), __floats2half2_rn(v[4], v[5]),
                          __floats2half2_rn(v[6], v[7])};
    return *reinterpret_cast<const uint4 *>(h);
}

template <int DSUB>
__device__ __forceinline__ void load_word(float (&w)[8], const unsigned char *from) {
#pragma unroll
    for (int j = 0; j < DSUB; j += 4) *reinterpret_cast<float4 *>(w + j) = *reinterpret_cast<const float4 *>(from + j * 4);
}

// DSUB = 8, or 4 run as 8 with the upper four elements of rows and words held at zero: appending zeros changes neither the
// FMA chain of a dot product nor the left-to-right sum of squares.
// EXACT32: the words that decide are fp32 (transformed by a whitener); they are scored by three products, of the row's high and low
// halves with the word's high one and of the high halves with the word's low one, which drops 2^-21 |r||c| and, where the low halves
// are subnormal, 2^-22 |r|.  The rows of the reconstruction are summed from `plain`.
template <int DSUB, typename XT, bool EXACT32>
__global__ void __launch_bounds__(kThreads, 1)
encode_narrow_kernel(const XT *__restrict__ x, int64_t sxb, int64_t sxh, int64_t sxt, const void *__restrict__ tables_in,
                     const __half *__restrict__ plain, const float *__restrict__ sqnorm_in, uint8_t *__restrict__ codes, void *__restrict__ recon, int recon_dtype,
                     int B, int H, int T, int G, int S, int K, int64_t t0, int64_t T_cap, int vec_ok, int last_shift, int spins) {
    extern __shared__ __align__(1024) unsigned char smem[];
    // Columns of a load from tensor memory.  What is decided by them is registers: 32 at a time made the kernels keep part of a row's state in
    // local memory in every stage.  us, 32 / 16 columns, 32768 rows x 8 heads with rows: 16 x 2 x 8 fp16 441 / 344, 16 x 8 286 / 207, 32 x 4
    // 436 / 363; whitened 32 x 4, 3001 fp32 rows, with the whitening, 106 / 85.  fp32 rows of 8-wide words fit either way: 360 / 383, whitened 73 / 74.  (8 columns: 364
    // where 16 take 344; the next 16 asked for before these are looked at: 368.)
    constexpr int kColumns = DSUB == 8 && sizeof(XT) == 4 ? 32 : 16;
    constexpr size_t kStageBytes = kStage<DSUB, EXACT32>, kExactAt = narrow::kStageBytes + kWordBytes;
    const __half *tables = reinterpret_cast<const __half *>(tables_in);
    unsigned char *ones = smem + (size_t)S * kStageBytes, *misc = ones + (1 + kGroups) * kABytes;
    const uint32_t bars = smem_u32(misc);                               // [kGroups]
    uint32_t *in_flight = reinterpret_cast<uint32_t *>(misc + 32);      // [kGroups] phase of the last product asked for; 2: none
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(misc + 64);
    int *cc_tops = reinterpret_cast<int *>(misc + 128);                 // [S] largest |word|^2 as bits (they order like ints)
    const int tid = threadIdx.x, warp = tid >> 5;
    const int grp = warp >> 2, row = tid & (kRows - 1);
    const float inf = __int_as_float(0x7f800000);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)(kGroups * kHalf)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < kGroups; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8 * i) : "memory");
            in_flight[i] = 2u;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kRows * 2) {
        const int piece = (tid & 1) ^ ((tid >> 3) & 1);
        *reinterpret_cast<uint4 *>(ones + tid * 16) = piece == 0 ? make_uint4(0x3c003c00u, 0x00003c00u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tmem_slot) + (uint32_t)(grp * kHalf);
    const uint32_t my_scores = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    unsigned char *A = ones + (1 + grp) * kABytes;
    unsigned char *a_hi = A + row * 32 + ((row >> 2) & 1) * 16;
    const uint32_t bar = bars + 8 * grp;
    const int copy = ((tid >> 2) & 1) * 16;
    uint32_t phase = 0u;
    bool fail = false;
    // the scores of one half of a stage's words, once all rows are written and the previous scores are read
    auto issue = [&](const unsigned char *stage, int half) {
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(kRows) : "memory");
        if (row == 0 && !fail) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t words_a = smem_u32(stage) + half * (kHalf * 32);
            mma(tmem, descriptor(smem_u32(ones)), descriptor(words_a + (uint32_t)kWordBytes), 0u);
            mma(tmem, descriptor(smem_u32(A)), descriptor(words_a), 1u);
            if constexpr (EXACT32) mma(tmem, descriptor(smem_u32(A)), descriptor(words_a + (uint32_t)narrow::kStageBytes), 1u);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
            in_flight[grp] = phase;
        }
        __syncwarp();
    };

    const uint32_t rows = (uint32_t)B * (uint32_t)T;  // the launcher keeps B*T below 2^31
    const uint32_t tiles = (rows + kRows - 1) / kRows;
    const int pairs = H * G;

    // Spans of kSpan tiles are finished one after the other by all blocks: a row's neighbouring groups, which share its
    // sectors, are then read and written while the row is in L2.
#pragma unroll 1
    for (uint32_t span = 0; span < tiles; span += kSpan) {
    const uint32_t wide = min((uint32_t)kSpan, tiles - span);
    // Blocks get turns, a tile for every group of threads: where a block's part of a pair was any number of tiles, groups idled at its end.  With that
    // and spans of 64 tiles, us, 16 x 2 x 8 with rows, 32768 rows x 8 heads 344 / 325 (fp32 rows 359 / 318), 16384 rows 157 / 149; 32 x 4, 32768
    // rows 362 / 316.  Smaller units, and fewer blocks, for a call (or the end of one) of less than a span: narrow_plan.cuh.
    const uint32_t shift = wide == kSpan ? 2u : (uint32_t)last_shift, units = (wide + (1u << shift) - 1) >> shift;
    const int64_t work = (int64_t)pairs * units, end = work * (blockIdx.x + 1) / gridDim.x;
#pragma unroll 1
    for (int64_t at = work * blockIdx.x / gridDim.x; at < end;) {
        const int hg = (int)(at / units), h = hg / G, g = hg % G;
        const uint32_t unit0 = (uint32_t)(at - (int64_t)hg * units), mine = (uint32_t)min((int64_t)(units - unit0), end - at);
        const uint32_t tile0 = span + (unit0 << shift), tile1 = span + min(wide, (unit0 + mine) << shift);  // of this pair, for this block
        // ---- the pair's tables ----
        __syncthreads();  // the previous pair's are no longer read
        if (tid < S) cc_tops[tid] = 0;
        __syncthreads();
#pragma unroll 1
        for (int i = tid; i < S * kMaxWords; i += kThreads) {
            const int s = i / kMaxWords, k = i % kMaxWords;
            unsigned char *stage = smem + (size_t)s * kStageBytes;
            uint4 w = make_uint4(0u, 0u, 0u, 0u), low = w;
            float cc = inf;  // padding words can never be chosen
            if (k < K) {
                const int64_t word = (((int64_t)h * S + s) * G + g) * K + k;
                if constexpr (EXACT32) {
                    const float *from = reinterpret_cast<const float *>(tables_in) + word * DSUB;
                    float e[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, back[8];
#pragma unroll
                    for (int j = 0; j < DSUB; j += 4) *reinterpret_cast<float4 *>(e + j) = __ldg(reinterpret_cast<const float4 *>(from + j));
#pragma unroll
                    for (int j = 0; j < DSUB; j += 4) *reinterpret_cast<float4 *>(stage + kExactAt + (k * DSUB + j) * 4) = *reinterpret_cast<const float4 *>(e + j);
                    cc = sqnorm_in != nullptr ? sqnorm_in[word] : sqnorm_ordered<DSUB>([&](int j) { return e[j]; });
                    w = pack8(e);
                    unpack8(w, back);
#pragma unroll
                    for (int j = 0; j < 8; ++j) e[j] -= back[j];
                    low = pack8(e);
                } else if constexpr (DSUB == 8) {
                    w = __ldg(reinterpret_cast<const uint4 *>(tables + word * 8));
                } else {
                    const uint2 half_word = __ldg(reinterpret_cast<const uint2 *>(tables + word * 4));
                    w = make_uint4(half_word.x, half_word.y, 0u, 0u);
                }
                if constexpr (EXACT32) {
                } else if (sqnorm_in != nullptr) {
                    cc = sqnorm_in[word];
                } else {
                    float e[8];
                    unpack8(w, e);
                    cc = sqnorm_ordered<DSUB>([&](int j) { return e[j]; });
                }
                if (cc == cc) atomicMax(cc_tops + s, __float_as_int(cc));
            }
            *reinterpret_cast<uint4 *>(stage + k * 32) = w;
            *reinterpret_cast<uint4 *>(stage + k * 32 + 16) = w;
            if constexpr (EXACT32) {
                unsigned char *to = stage + narrow::kStageBytes + k * 32;
                *reinterpret_cast<uint4 *>(to + ((k >> 2) & 1) * 16) = low;
                *reinterpret_cast<uint4 *>(to + (((k >> 2) & 1) ^ 1) * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            const float t = -0.5f * cc;
            const __half p1 = __float2half_rn(t);
            const float r1 = k < K ? t - __half2float(p1) : 0.0f;
            const __half p2 = __float2half_rn(r1);
            const __half p3 = __float2half_rn(r1 - __half2float(p2));
            const __half2 parts[2] = {__halves2half2(p1, p2), __halves2half2(p3, __float2half_rn(0.0f))};
            const uint2 raw = *reinterpret_cast<const uint2 *>(parts);
            const int flip = (k >> 2) & 1;
            *reinterpret_cast<uint4 *>(stage + kWordBytes + k * 32 + flip * 16) = make_uint4(raw.x, raw.y, 0u, 0u);
            *reinterpret_cast<uint4 *>(stage + kWordBytes + k * 32 + (flip ^ 1) * 16) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<float *>(stage + kWordBytes + kSeedBytes + k * 4) = cc;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();

        // ---- the tiles, a group each; the next tile's row travels while this one is searched ----
        uint4 raw[sizeof(XT) / 2];
        uint32_t grow = (tile0 + grp) * kRows + row;
        uint32_t nb = grow / (uint32_t)T, nt = grow % (uint32_t)T;  // divided out once, then advanced by the stride
        auto fetch = [&](uint32_t tile) {
#pragma unroll
            for (int i = 0; i < (int)sizeof(XT) / 2; ++i) raw[i] = make_uint4(0u, 0u, 0u, 0u);
            if (tile >= tile1 || grow >= rows) return;
            const XT *src = x + (int64_t)nb * sxb + (int64_t)h * sxh + (int64_t)nt * sxt + (int64_t)g * DSUB;
            if (!vec_ok) {
                uint32_t w[4 * (sizeof(XT) / 2)] = {};
#pragma unroll
                for (int i = 0; i < DSUB; ++i) {
                    if constexpr (sizeof(XT) == 4) w[i] = __float_as_uint(src[i]);
                    else w[i / 2] |= (uint32_t)__half_as_ushort(src[i]) << (16 * (i & 1));
                }
#pragma unroll
                for (int i = 0; i < (int)sizeof(XT) / 2; ++i) raw[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
            } else if constexpr (DSUB * sizeof(XT) == 8) {
                const uint2 v = __ldg(reinterpret_cast<const uint2 *>(src));
                raw[0].x = v.x, raw[0].y = v.y;
            } else {
#pragma unroll
                for (int i = 0; i < (int)(DSUB * sizeof(XT)) / 16; ++i) raw[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
            }
        };
        fetch(tile0 + grp);
#pragma unroll 1
        for (uint32_t tile = tile0 + grp; tile < tile1; tile += kGroups) {
            float r[8];
            // not before this point: converted right after its load, the row would be waited for a trip early
#pragma unroll
            for (int i = 0; i < (int)sizeof(XT) / 2; ++i) asm volatile("" : "+r"(raw[i].x), "+r"(raw[i].y), "+r"(raw[i].z), "+r"(raw[i].w));
            if constexpr (sizeof(XT) == 2) {
                unpack8(raw[0], r);
            } else {
                r[0] = __uint_as_float(raw[0].x), r[1] = __uint_as_float(raw[0].y), r[2] = __uint_as_float(raw[0].z), r[3] = __uint_as_float(raw[0].w);
                r[4] = __uint_as_float(raw[1].x), r[5] = __uint_as_float(raw[1].y), r[6] = __uint_as_float(raw[1].z), r[7] = __uint_as_float(raw[1].w);
            }
            uint64_t picks = 0ull;
            uint32_t later = 0u;
            const uint32_t b = nb, t = nt;
            const bool live = grow < rows;
            grow += kGroups * kRows;
            nb += (kGroups * kRows) / (uint32_t)T;
            nt += (kGroups * kRows) % (uint32_t)T;
            if (nt >= (uint32_t)T) nt -= (uint32_t)T, ++nb;
            fetch(tile + kGroups);
            uint8_t *code_at = codes + (((int64_t)b * H + h) * T_cap + t0 + t) * ((int64_t)S * G) + g;

#pragma unroll 1
            for (int s = 0; s < S; ++s) {
                const unsigned char *stage = smem + (size_t)s * kStageBytes;
                const float *nrm = reinterpret_cast<const float *>(stage + kWordBytes + kSeedBytes);
                const float xx = sqnorm_ordered<8>([&](int i) { return r[i]; });
                {
                    const uint4 hi = pack8(r);
                    float back[8], rest[8];
                    unpack8(hi, back);
#pragma unroll
                    for (int i = 0; i < 8; ++i) rest[i] = r[i] - back[i];
                    *reinterpret_cast<uint4 *>(a_hi) = hi;
                    *reinterpret_cast<uint4 *>(A + row * 32 + (((row >> 2) & 1) ^ 1) * 16) = pack8(rest);
                }
                const float cc_top = __int_as_float(cc_tops[s]);
                float rough;
                asm("sqrt.approx.f32 %0, %1;" : "=f"(rough) : "f"(cc_top));
                float rough_row = 0.0f;
                if constexpr (EXACT32) asm("sqrt.approx.f32 %0, %1;" : "=f"(rough_row) : "f"(xx));
                const float margin = 3.0517578125e-05f * (xx + cc_top) + (EXACT32 ? 3.82e-06f * rough_row : 0.0f) + 3.82e-06f * rough + 1.1920929e-07f;

                // ---- half by half: the largest score of every four words, their largest, and the fours close to that.  The first half's
                // are looked at while the second half's product runs, against the first half's own maximum: at worst a few too many.
                float top = -inf, first_top = -inf;
                uint32_t low = 0u, high = 0u;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float top4[32];
                    if (half == 0) issue(stage, 0);
                    if (!fail && !bounded_wait(bar, phase, spins)) fail = true;
                    phase ^= 1u;
                    fail = __any_sync(0xffffffffu, fail);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < kHalf / kColumns; ++c) {
                        float v[kColumns];
                        tmem_load(v, my_scores + c * kColumns);
#pragma unroll
                        for (int p = 0; p < kColumns / 4; ++p) {
                            top4[c * (kColumns / 4) + p] = fmaxf(max3(v[4 * p], v[4 * p + 1], v[4 * p + 2]), v[4 * p + 3]);
                            asm volatile("" : "+f"(top4[c * (kColumns / 4) + p]));  // before the next columns are loaded: all of them at once do not fit
                        }
                    }
                    if (half == 0) issue(stage, 1);
                    float m0 = top4[0], m1 = top4[16];
#pragma unroll
                    for (int p = 1; p < 15; p += 2) m0 = max3(m0, top4[p], top4[p + 1]), m1 = max3(m1, top4[16 + p], top4[17 + p]);
                    top = fmaxf(top, max3(fmaxf(m0, m1), top4[15], top4[31]));
                    // Bits by saturating and doubling multiply-adds, 8 fours a chain.  No score lies less than 2^-60 above the limit, where it
                    // would count in part and disturb the bits below: products of fp16 values and their sums are multiples of 2^-48, and so
                    // is the limit, as the margin is at least 2^-23.
                    constexpr float kSteep = 1.152921504606846976e18f;  // 2^60
                    const float offset = (margin - top) * kSteep;
                    float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int i = 7; i >= 0; --i)
#pragma unroll
                        for (int c = 0; c < 4; c += 2)
                            double_add2(sum[c], sum[c + 1], fma_sat(top4[8 * c + i], kSteep, offset), fma_sat(top4[8 * c + 8 + i], kSteep, offset));
                    // sums below 2^16 show in the mantissa of 2^23 + sum
                    const uint32_t bits = __byte_perm(__float_as_uint(fmaf(sum[1], 256.0f, sum[0] + 8388608.0f)),
                                                      __float_as_uint(fmaf(sum[3], 256.0f, sum[2] + 8388608.0f)), 0x5410);
                    if (half == 0) low = bits, first_top = top;
                    else high = bits;
                }
                if (!(first_top >= top - margin)) low = 0u;
                // |r|^2 < 2^30 keeps every element below 2^15
                if (fail || !(xx < 1.0e9f) || !(cc_top < 1.3e5f) || !(top > -inf)) low = high = ~0u;

                // ---- exact re-evaluation.  A lane starts at word lane % 4 of its four and reads copy (lane / 4) % 2 of the words, so that
                // eight neighbouring lanes meet eight different 16-byte banks whatever their fours are ----
                float best = 3.402823466e38f;  // an infinite or NaN distance never wins, as in a scan for '<' from +inf
                int arg = 0x7fffffff;
                while ((low | high) != 0u) {
                    const int p = low != 0u ? __ffs((int)low) - 1 : 31 + __ffs((int)high);
                    if (low != 0u) low &= low - 1u;
                    else high &= high - 1u;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int k = 4 * p + ((j + tid) & 3);
                        float w[8];
                        if constexpr (EXACT32) load_word<DSUB>(w, stage + kExactAt + k * DSUB * 4);
                        else unpack8(*reinterpret_cast<const uint4 *>(stage + k * 32 + copy), w);
                        float dot = __fmaf_rn(r[0], w[0], 0.0f);
#pragma unroll
                        for (int i = 1; i < DSUB; ++i) dot = __fmaf_rn(r[i], w[i], dot);
                        const float dist = distance_expr(xx, nrm[k], dot);
                        if (dist < best || (dist == best && k < arg)) best = dist, arg = k;  // the lowest of a tie
                    }
                }
                __syncwarp();
                if (arg >= K) arg = 0;  // no distance was finite
                float sel[8];
                if constexpr (EXACT32) load_word<DSUB>(sel, stage + kExactAt + arg * DSUB * 4);
                else unpack8(*reinterpret_cast<const uint4 *>(stage + arg * 32 + copy), sel);
#pragma unroll
                for (int i = 0; i < DSUB; ++i) r[i] = __fsub_rn(r[i], sel[i]);
                picks = (picks >> 8) | ((uint64_t)(later & 255u) << 56);  // a queue of 12 bytes
                later = (later >> 8) | ((uint32_t)arg << 24);
                if (live) code_at[(int64_t)s * G] = (uint8_t)arg;
            }
            if (recon != nullptr && live) {
                float dec[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
                for (int s = 0; s < S; ++s) {  // stage s is byte 12 - S + s of the queue
                    const int byte = kMaxStages - S + s;
                    const int code = (int)((byte < 8 ? (uint32_t)(picks >> (8 * byte)) : later >> (8 * (byte - 8))) & 255u);
                    float w[8];
                    if constexpr (EXACT32) {
                        const __half *from = plain + ((((int64_t)h * S + s) * G + g) * K + code) * DSUB;
                        uint4 v = make_uint4(0u, 0u, 0u, 0u);
                        if constexpr (DSUB == 8) {
                            v = __ldg(reinterpret_cast<const uint4 *>(from));
                        } else {
                            const uint2 half_word = __ldg(reinterpret_cast<const uint2 *>(from));
                            v.x = half_word.x, v.y = half_word.y;
                        }
                        unpack8(v, w);
                    } else {
                        unpack8(*reinterpret_cast<const uint4 *>(smem + (size_t)s * kStageBytes + code * 32 + copy), w);
                    }
#pragma unroll
                    for (int i = 0; i < DSUB; ++i) dec[i] = __fadd_rn(dec[i], w[i]);
                }
                const int64_t o = (((int64_t)b * H + h) * T + t) * ((int64_t)G * DSUB) + (int64_t)g * DSUB;
                if (recon_dtype == TACVQ_F16) {
                    const uint4 out = pack8(dec);
                    if constexpr (DSUB == 8) *reinterpret_cast<uint4 *>((__half *)recon + o) = out;
                    else *reinterpret_cast<uint2 *>((__half *)recon + o) = make_uint2(out.x, out.y);
                } else {
                    *reinterpret_cast<float4 *>((float *)recon + o) = make_float4(dec[0], dec[1], dec[2], dec[3]);
                    if constexpr (DSUB == 8) *reinterpret_cast<float4 *>((float *)recon + o + 4) = make_float4(dec[4], dec[5], dec[6], dec[7]);
                }
            }
        }
        at += mine;
    }
    }
    if (__syncthreads_or(fail)) {  // each group's last product ends before the block's memory goes
        if (row == 0 && in_flight[grp] < 2u) bounded_wait(bar, in_flight[grp], kSpins);
        if (tid == 0) atomicAdd(&g_timeouts, 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        const uint32_t base = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"((uint32_t)(kGroups * kHalf)) : "memory");
    }
}

}  // namespace narrow

// Returns TACVQ_ERR_UNSUPPORTED when the geometry is not this kernel's.
int encode_narrow_launch(const EncodeArgs &a) {
    using namespace narrow;
    const int sub = a.D / a.G;
    if ((sub != 8 && sub != 4) || a.K > kMaxWords || a.S > kMaxStages) return TACVQ_ERR_UNSUPPORTED;
    if (a.tables_f32 && (a.x_dtype != TACVQ_F32 || (reinterpret_cast<uintptr_t>(a.recon_tables) & 15u) != 0)) return TACVQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a.tables) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    if (a.recon != nullptr && (reinterpret_cast<uintptr_t>(a.recon) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    const int64_t rows = (int64_t)a.B * a.T;
    if (rows >= (int64_t)1 << 31) return TACVQ_ERR_UNSUPPORTED;
    const int64_t tiles = (rows + kRows - 1) / kRows;
    const int elem = a.x_dtype == TACVQ_F16 ? 2 : 4, vec = sub * elem < 16 ? sub * elem : 16, per_vec = vec / elem;
    const int vec_ok = (reinterpret_cast<uintptr_t>(a.x) % vec) == 0 && a.sxb % per_vec == 0 && a.sxh % per_vec == 0 && a.sxt % per_vec == 0;
    const size_t stage = a.tables_f32 ? (sub == 8 ? kStage<8, true> : kStage<4, true>) : kStageBytes;
    const size_t smem = (size_t)a.S * stage + kFixedBytes + (size_t)a.S * 4;
    if (smem > 227 * 1024) return TACVQ_ERR_UNSUPPORTED;
    const Deal dealt = deal(tiles, (int64_t)a.H * a.G, 148);
    auto launch = [&](auto kernel, auto *xp) -> int {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kernel<<<(unsigned)dealt.blocks, kThreads, smem, a.stream>>>(xp, a.sxb, a.sxh, a.sxt, a.tables, a.recon_tables, a.sqnorm, a.codes, a.recon,
                                                               a.recon_dtype, a.B, a.H, a.T, a.G, a.S, a.K, a.t0, a.T_cap, vec_ok, dealt.shift,
                                                               a.wait_spins < 0 ? kSpins : a.wait_spins);
        return launch_status();
    };
    if (a.tables_f32) {
        if (sub == 8) return launch(encode_narrow_kernel<8, float, true>, (const float *)a.x);
        return launch(encode_narrow_kernel<4, float, true>, (const float *)a.x);
    }
    if (sub == 8) {
        if (a.x_dtype == TACVQ_F16) return launch(encode_narrow_kernel<8, __half, false>, (const __half *)a.x);
        return launch(encode_narrow_kernel<8, float, false>, (const float *)a.x);
    }
    if (a.x_dtype == TACVQ_F16) return launch(encode_narrow_kernel<4, __half, false>, (const __half *)a.x);
    return launch(encode_narrow_kernel<4, float, false>, (const float *)a.x);
}

int narrow_timeouts(unsigned int *out) { return (int)cudaMemcpyFromSymbol(out, narrow::g_timeouts, sizeof(unsigned int)); }

}  // namespace tacvq
