// Encode for 64- and 128-wide groups: the tensor core scores every word, exact fp32 decides.
//
// A block is one or two groups of 512 threads, each with its own tile of 128 rows of one (head, group of channels).
// Four threads share a row (tensor-memory lane): thread q holds the 8-element pieces q, q + 4, ... of the fp32 residual
// in registers and looks at words 64 q .. 64 q + 63.  Per stage a group
//   1. has its rows' fp16 rounding in shared memory (K-major panels, 128-byte swizzle) and one thread issue the
//      128 x 256 x d product with the stage's words (tcgen05.mma, fp32 accumulators in 256 tensor-memory columns); a
//      first step of 16 columns (A: ones, B: -|c|^2/2 in three fp16 parts) makes every sum the score
//      t = r.c - |c|^2/2, the distance being |r|^2 - 2t,
//   2. reads its scores twice: once for the row's maximum, once for the mask of words within a margin of it,
//   3. takes the only word of the mask; two or three words are scored in fp32, and where that leaves the best too close to
//      another, or where there are more, the row goes to shared memory and the library's exact chains decide,
//   4. subtracts the chosen word and writes the new fp16 row.
// The two groups share the word tables: resident for the block's life up to two stages, otherwise a ring of two
// that the group which leaves a stage last refills (words by TMA, norms by its warps).  While one group waits for its product the other one reads
// scores, which keeps the tensor core and the schedulers busy in turn.
//
// Margin (encode_tc.cu has the argument that twice the error bound E of a score keeps the exact argmin and its ties on
// the list).  E collects, with u = |r| max|c| and cc = max|c|^2: rounding the row to fp16, 2^-11 u (nothing for the
// first stage of fp16 rows); the exact chain, 2^-17 u; the tensor core's sums, at most nine steps that each lose
// 17 units of 2^-24 of a magnitude below u + cc / 2, so 2^-16.7 (u + cc / 2); the roundings of the distance,
// 2^-23 (|r|^2 + cc); the three fp16 parts of -|c|^2/2, 2^-25; rows that are subnormal in fp16, 2^-25 sqrt(d) max|c|.
// The kernel allows  (1.0625 * 2^-10, or 2^-14) u  +  2^-20 |r|^2  +  2^-15 cc  +  2^-18 max|c|  +  2^-23.
// With EXACT32 the words are fp32 (transformed by a whitener) and their fp16 rounding is scored: 2^-10 u more, and
// 2^-20 |r| for words that are subnormal in fp16; everything that decides reads the fp32 words.
// Rows or words outside fp16's range, and a product that never arrived, list every word.
//
// What bounds it: latency between the phases of a stage more than the tensor core (1152 cycles a tile and stage) or the
// issue slots, hence two tiles a block and four threads a row.  262144 fp16 rows x 8 heads, 128 wide, 2 stages: 807 us,
// against 1675 us for one tile of 128 rows a block with the residual in tensor memory.
//
// Reference statements: src/jointkv/closed_loop_vq.py:52-76 (search), :343-395 (stage recursion), :312-320, 384-390
// (whitened assignment).

#include <atomic>

#include "common.cuh"
#include "table_map.cuh"

namespace tacvq {

namespace wide {

constexpr int kRows = 128;          // rows per group of threads
constexpr int kShare = 4;           // threads per row
constexpr int kGroupThreads = kShare * kRows;
constexpr int kMaxGroups = 2;       // groups of threads per block
constexpr int kSeedBytes = kMaxWords * 32;  // 16 halves a word
constexpr int kOnesBytes = kRows * 32;

// blocks in which a wait was given up; read by tensor_memory_timeouts, expected to stay 0
__device__ unsigned int g_timeouts = 0;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
constexpr int kSpins = 1 << 17;
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity, int spins) {
    int done = 0;
#pragma unroll 1
    for (int spin = 0; spin < spins && !done; ++spin)
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.s32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// 16 columns; the registers are valid when it returns
__device__ __forceinline__ void tmem_load16(uint32_t (&v)[16], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
// Shared-memory operand descriptors of tcgen05.mma, K-major: start address / 16 in bits 0-13, leading offset (not used by
// swizzled layouts of one panel width) in bits 16-29, bytes / 16 between groups of 8 rows in bits 32-45, version 1 in bits
// 46-47, swizzle in bits 61-63 (2: 128-byte rows, 6: 32-byte rows).
__device__ __forceinline__ uint64_t panel_descriptor(uint32_t smem_addr) {
    return ((uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32) | (((smem_addr & 0x3ffffu) >> 4) | (1u << 16));
}
__device__ __forceinline__ uint64_t narrow_descriptor(uint32_t smem_addr) {
    return ((uint64_t)((256u >> 4) | (1u << 14) | (6u << 29)) << 32) | (((smem_addr & 0x3ffffu) >> 4) | (1u << 16));
}
// fp32 accumulator (bits 4-5), fp16 operands, K-major, N / 8 in bits 17-22, M / 16 in bits 24-28
constexpr uint32_t kMmaShape = (1u << 4) | ((uint32_t)(kMaxWords >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(tmem), "l"(a), "l"(b), "r"(kMmaShape), "r"(accumulate) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// two neighbouring fp32 values per instruction
__device__ __forceinline__ void sub2(float &a0, float &a1, float b0, float b1) {
    asm("{\n.reg .b64 a, b;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nadd.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}" : "+f"(a0), "+f"(a1) : "f"(-b0), "f"(-b1));
}
__device__ __forceinline__ void fma2(float &acc0, float &acc1, float a0, float a1, float b0, float b1) {
    asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%0, %1};\nfma.rn.f32x2 c, a, b, c;\nmov.b64 {%0, %1}, c;\n}"
        : "+f"(acc0), "+f"(acc1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
// acc = 2 acc + b
__device__ __forceinline__ void double_add2(float &acc0, float &acc1, float b0, float b1) {
    asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%4, %4};\nmov.b64 c, {%2, %3};\nfma.rn.f32x2 a, a, b, c;\nmov.b64 {%0, %1}, a;\n}"
        : "+f"(acc0), "+f"(acc1) : "f"(b0), "f"(b1), "f"(2.0f));
}
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// for margins, which have room for its 2^-22
__device__ __forceinline__ float rough_sqrt(float v) {
    float d;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ uint4 pack8(const float *v) {
    const __half2 h[4] = {__floats2half2_rn(v[0], v[1]), __floats2half2_rn(v[2], v[3]), __floats2half2_rn(v[4], v[5]),
                          __floats2half2_rn(v[6], v[7])};
    return *reinterpret_cast<const uint4 *>(h);
}
__device__ __forceinline__ void unpack8(const uint4 raw, float *v) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __half22float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// |word|^2 in the library's order, for callers that bring no norms: lane u of four neighbouring ones owns the eight running
// sums of set u, so that a word arrives in whole sectors, and all four return the total
template <int DSUB>
__device__ __forceinline__ float word_norm_by_four(const __half *__restrict__ word, int lane) {
    uint4 raw[DSUB / 32];
#pragma unroll
    for (int i = 0; i < DSUB / 32; ++i) raw[i] = __ldg(reinterpret_cast<const uint4 *>(word) + 4 * i + (lane & 3));
    float set[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < DSUB / 32; ++i) {
        float v[8];
        unpack8(raw[i], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) set[j] = __fadd_rn(set[j], __fmul_rn(v[j], v[j]));
    }
    float total = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        float sum = __shfl_sync(0xffffffffu, set[j], lane & 28);
#pragma unroll
        for (int u = 1; u < 4; ++u) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, set[j], (lane & 28) + u));
        total = j == 0 ? sum : __fadd_rn(total, sum);
    }
    return total;
}

// The same by one thread, with few registers: for words that did not arrive in time.
template <int DSUB>
__device__ __forceinline__ float word_norm_alone(const __half *__restrict__ word) {
    float total = 0.0f;
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        float mine = 0.0f;
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
            float set = 0.0f;
#pragma unroll 1
            for (int i = 8 * u + j; i < DSUB; i += 32) {
                const float v = __half2float(word[i]);
                set = __fadd_rn(set, __fmul_rn(v, v));
            }
            mine = u == 0 ? set : __fadd_rn(mine, set);
        }
        total = j == 0 ? mine : __fadd_rn(total, mine);
    }
    return total;
}

// A 16-byte load that is not moved ahead of others: for words that did not arrive in time, off the usual path.
__device__ __forceinline__ uint4 load_in_place(const __half *from) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(from) : "memory");
    return v;
}

// Which of a thread's 64 words a bit of its mask stands for: 16 columns take 16 bits, the even ones first.
__device__ __forceinline__ int word_of_bit(int bit) { return (bit & 48) | ((bit & 7) << 1) | ((bit >> 3) & 1); }

template <int DSUB>
struct Layout {
    static constexpr size_t kTabBytes = (size_t)kMaxWords * DSUB * 2;
    static constexpr size_t kRowBytes = (size_t)kRows * DSUB * 2;
    static constexpr size_t kTab = 0;                                    // [2] tables, swizzled panels
    static constexpr size_t kSeed = 2 * kTabBytes;                       // [2][256][16] half: -|c|^2/2 in three parts
    static constexpr size_t kOnes = kSeed + 2 * kSeedBytes;              // [128][16] half: 1, 1, 1, 0 ...
    static constexpr size_t kNrm = kOnes + kOnesBytes;                   // [2][256] float
    static constexpr size_t kMisc = kNrm + 2 * kMaxWords * 4;            // barriers, tensor-memory slot, largest norms
    static constexpr size_t kA = kMisc + 1024;                           // [2] fp16 rows, swizzled panels
    static constexpr size_t kTop = kA + kMaxGroups * kRowBytes;          // [2 groups][4 q][128] float: largest score; first dot product
    static constexpr size_t kXx = kTop + 2 * kGroupThreads * 4;          // the same: partial |r|^2; second dot product
    static constexpr size_t kInfo = kXx + 2 * kGroupThreads * 4;         // the same of u16: words listed, two of them
    static constexpr size_t kSlot = kInfo + 2 * kGroupThreads * 2;       // [2 groups][4 quads of warps] half a residual row
    static constexpr size_t kBytes = kSlot + 8 * (size_t)DSUB * 2;
    // half index of element e of a word or row: panels of 64 elements, 16-byte pieces swizzled by the row number
    template <int ROWS>
    __device__ static __forceinline__ int at(int r, int e) {
        return (e >> 6) * (ROWS * 64) + r * 64 + ((((e >> 3) & 7) ^ (r & 7)) << 3) + (e & 7);
    }
};

struct Args {
    const void *x;
    int64_t sxb, sxh, sxt;
    const __half *tables;    // scored words (fp16)
    const float *words32;    // EXACT32: the words that decide
    const __half *recon_tables;
    const float *sqnorm;     // |word|^2 of the deciding words; may be null for fp16 words
    uint8_t *codes;
    void *recon;
    int recon_dtype, B, H, T, G, S, K, vec_ok, use_map, spins;
    int64_t t0, T_cap;
};

// GROUPS = 1: one tile a block, for launches that leave no tile waiting; twice the registers per thread.
template <int DSUB, typename XT, bool EXACT32, int GROUPS>
__global__ void __launch_bounds__(GROUPS * kGroupThreads, 1)
encode_wide_kernel(const Args a, const __grid_constant__ CUtensorMap table_map) {
    using L = Layout<DSUB>;
    constexpr int kPieces = DSUB / 8, kOwn = kPieces / kShare;
    // Fp32 scores further apart than this many u tell which of two words the exact distances prefer.  Each word's share, in units of 2^-24 u: DSUB
    // roundings of the exact chain, DSUB / 8 + 3 of the score's sums, one where the norm is subtracted and one in the distance (twice u, but a score is half a
    // distance); a hundredth is left for the bound u itself, and the term of the norms is twice what it needs.  (3.2e-5, twice what is needed at 128, sent 1.8 times as many rows to the chains:
    // 849 us where it is 815, 16 whitened stages x 2048 rows 181 / 177.)
    constexpr float kClose = 1.01f * 2.0f * (DSUB + DSUB / 8 + 5) * 5.9604645e-8f;
    extern __shared__ __align__(1024) unsigned char smem[];
    __half *tabs = reinterpret_cast<__half *>(smem + L::kTab);
    float *nrms = reinterpret_cast<float *>(smem + L::kNrm);
    const uint32_t misc = smem_u32(smem + L::kMisc);
    const uint32_t full_bar = misc, mma_bar = misc + 16;  // [2] each
    unsigned int *left = reinterpret_cast<unsigned int *>(smem + L::kMisc + 64);  // [2][16]: groups that left a stage of this buffer, all uses together, per share
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L::kMisc + 48);
    uint32_t *in_flight = reinterpret_cast<uint32_t *>(smem + L::kMisc + 52);     // [2] phase of the last product asked for; 2: none
    float *cc_tops = reinterpret_cast<float *>(smem + L::kMisc + 192);            // [2][16]: largest norm of a share

    const int hg = blockIdx.y, h = hg / a.G, g = hg % a.G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = a.S, K = a.K;
    constexpr int groups = GROUPS;
    const uint32_t rows = (uint32_t)a.B * (uint32_t)a.T;  // the launcher keeps B*T below 2^31
    const uint32_t tiles = (rows + kRows - 1) / kRows;
    const float inf = __int_as_float(0x7f800000);
    const bool resident = S <= 2;
    // Warps that fill a stage's buffer, a share of the words each: four where the norms are there to be copied, all sixteen of a
    // group where they are computed.  (By four warps, four words at a time, that took longer than the stage: 192 rows of 8 heads,
    // 16 stages of 128, rows wanted: 290 us, so 115, with norms 92.)
    const int shares = a.sqnorm != nullptr ? 4 : 16;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)(groups * kMaxWords)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full_bar + 8 * i), "r"(shares) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mma_bar + 8 * i) : "memory");
            in_flight[i] = 2u;
        }
        for (int i = 0; i < 32; ++i) left[i] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < kRows * 2; i += blockDim.x) {  // 16-byte piece c of row r sits at piece c ^ ((r >> 2) & 1)
        const int r = i >> 1, piece = (i & 1) ^ ((r >> 2) & 1);
        *reinterpret_cast<uint4 *>(smem + L::kOnes + r * 32 + (i & 1) * 16) =
            piece == 0 ? make_uint4(0x3c003c00u, 0x00003c00u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
    const int64_t head_words = ((int64_t)h * S * a.G + g) * K;   // word 0 of stage 0; a stage is G * K words further
    const int64_t stage_words = (int64_t)a.G * K;
    const uint32_t trips = blockIdx.x * groups < tiles ? (tiles - blockIdx.x * groups + gridDim.x * groups - 1) / (gridDim.x * groups) : 0u;
    const uint32_t uses = resident ? (uint32_t)S : trips * (uint32_t)S;

    // one warp: the words of a stage by plain copies, and their norms
    auto copy_table = [&](int buf, int64_t first) {
        __half *tab = tabs + (size_t)buf * (L::kTabBytes / 2);
#pragma unroll 1
        for (int i = lane; i < kMaxWords * kPieces; i += 32) {
            const int k = i / kPieces, p = i % kPieces;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (k < K) v = *reinterpret_cast<const uint4 *>(a.tables + (first + k) * DSUB + p * 8);
            *reinterpret_cast<uint4 *>(tab + L::template at<kMaxWords>(k, p * 8)) = v;
        }
    };
    // the norms and seeds of a share of use u's words, by a warp; the first share's also fetches all the words by TMA (or plain
    // copies without a tensor map)
    // (`ahead`: norms of words k_begin + lane and 32 further that are in registers already)
    auto load_table = [&](uint32_t u, int share, const float *ahead) {
        const int s = (int)(u % (uint32_t)S), buf = (int)(u & 1u);
        const int64_t first = head_words + s * stage_words;
        if (share != 0) {
        } else if (a.use_map) {
            if (lane == 0) {
                asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(full_bar + 8 * buf), "r"((uint32_t)L::kTabBytes) : "memory");
#pragma unroll
                for (int panel = 0; panel < DSUB / 64; ++panel)
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(smem_u32(tabs) + (uint32_t)(buf * L::kTabBytes) + panel * (kMaxWords * 128)), "l"(&table_map), "r"(panel * 64),
                                 "r"((int)first), "r"(full_bar + 8 * buf) : "memory");
            }
        } else {
            copy_table(buf, first);
        }
        const int k_begin = share * (kMaxWords / shares), k_end = k_begin + kMaxWords / shares;
        float *nrm = nrms + buf * kMaxWords;
        if (ahead != nullptr) {
            nrm[k_begin + lane] = ahead[0];
            nrm[k_begin + 32 + lane] = ahead[1];
        } else if (a.sqnorm != nullptr) {
#pragma unroll 1
            for (int k = k_begin + lane; k < k_end; k += 32) nrm[k] = k < K ? __ldg(a.sqnorm + first + k) : inf;
        } else {
#pragma unroll 1
            for (int k0 = k_begin; k0 < k_end; k0 += 8) {
                const int k = k0 + (lane >> 2);
                const float v = word_norm_by_four<DSUB>(a.tables + (first + min(k, K - 1)) * DSUB, lane);
                if ((lane & 3) == 0) nrm[k] = k < K ? v : inf;
            }
        }
        __syncwarp();
        float top = 0.0f;
        unsigned char *seed = smem + L::kSeed + buf * kSeedBytes;
#pragma unroll 1
        for (int k = k_begin + lane; k < k_end; k += 32) {
            const float v = nrm[k];
            if (k < K && v == v) top = fmaxf(top, v);
            const float t = -0.5f * v;  // padding words: -inf, never within the margin
            const __half p1 = __float2half_rn(t);
            const float r1 = k < K ? t - __half2float(p1) : 0.0f;
            const __half p2 = __float2half_rn(r1);
            const __half p3 = __float2half_rn(r1 - __half2float(p2));
            const __half2 parts[2] = {__halves2half2(p1, p2), __halves2half2(p3, __float2half_rn(0.0f))};
            const uint2 raw = *reinterpret_cast<const uint2 *>(parts);
            const int flip = (k >> 2) & 1;
            *reinterpret_cast<uint4 *>(seed + k * 32 + flip * 16) = make_uint4(raw.x, raw.y, 0u, 0u);
            *reinterpret_cast<uint4 *>(seed + k * 32 + (flip ^ 1) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
        if (lane == 0) cc_tops[buf * 16 + share] = top;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full_bar + 8 * buf) : "memory");
    };
#pragma unroll 1
    for (int i = warp; i < 2 * shares; i += GROUPS * 16)
        if ((uint32_t)(i / shares) < uses) load_table((uint32_t)(i / shares), i % shares, nullptr);

    const int grp = warp >> 4, part = warp & 3, q = (warp >> 2) & 3;
    const int row = part * 32 + lane;                     // of the group's tile
    const int group_barrier = 1 + grp, quad_barrier = 3 + grp * 4 + part;
    auto sync_group = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group_barrier), "r"(kGroupThreads) : "memory"); };
    auto sync_quad = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(quad_barrier), "r"(128) : "memory"); };  // the four warps of 32 rows
    __half *A = reinterpret_cast<__half *>(smem + L::kA + grp * L::kRowBytes);
    float *tops = reinterpret_cast<float *>(smem + L::kTop) + grp * kGroupThreads + row;   // [q * kRows]: this row's four
    float *xxs = reinterpret_cast<float *>(smem + L::kXx) + grp * kGroupThreads + row;
    uint16_t *infos = reinterpret_cast<uint16_t *>(smem + L::kInfo) + grp * kGroupThreads + row;
    float *slot = reinterpret_cast<float *>(smem + L::kSlot) + (grp * 4 + part) * (DSUB / 2);
    const uint32_t scores = tmem_base + (uint32_t)(grp * kMaxWords + q * 64) + ((uint32_t)(part * 32) << 16);
    const uint32_t my_mma = mma_bar + 8 * grp;
    uint32_t mma_phase = 0u;
    bool fail = false;
    // fp32 vectors of 128, one a row, by the four warps of 32 rows together (whole lines): a thread gets its pieces of its row's.  In two halves,
    // for which the place of the fp16 rows is just large enough.
    auto fetch_fp32 = [&](unsigned long long mine, float *out) {
        constexpr int kAtOnce = 32 / kPieces, kEach = 8 / kAtOnce;
        uint4 v[2][kEach];
#pragma unroll
        for (int i = 0; i < kEach; ++i) {
            const unsigned long long from = __shfl_sync(0xffffffffu, mine, q * 8 + i * kAtOnce + lane / kPieces);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                v[half][i] = make_uint4(0u, 0u, 0u, 0u);
                if (from != 0ull) v[half][i] = __ldg(reinterpret_cast<const uint4 *>(from) + half * kPieces + lane % kPieces);
            }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (half == 1) sync_quad();
#pragma unroll
            for (int i = 0; i < kEach; ++i)
                *reinterpret_cast<uint4 *>(A + L::template at<kRows>(part * 32 + q * 8 + i * kAtOnce + lane / kPieces, (lane % kPieces) * 8)) = v[half][i];
            sync_quad();
#pragma unroll
            for (int m = half * (kOwn / 2); m < (half + 1) * (kOwn / 2); ++m)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    *reinterpret_cast<float4 *>(out + 8 * m + 4 * i) =
                        *reinterpret_cast<const float4 *>(A + L::template at<kRows>(row, (2 * (4 * m + q) + i - half * kPieces) * 8));
        }
        sync_quad();
    };
    // (batch entry, token) of this thread's row: divided out once, then advanced by the stride of the tiles
    const uint32_t step = gridDim.x * groups * kRows, step_b = step / (uint32_t)a.T, step_t = step % (uint32_t)a.T;
    uint32_t grow = (blockIdx.x * groups + grp) * kRows + row;
    uint32_t nb = grow / (uint32_t)a.T, nt = grow % (uint32_t)a.T;
#pragma unroll 1
    for (uint32_t trip = 0; trip < trips; ++trip, grow += step) {
        const bool live = grow < rows;
        const uint32_t rb = live ? nb : 0u, rt = live ? nt : 0u;
        nb += step_b;
        nt += step_t;
        if (nt >= (uint32_t)a.T) nt -= (uint32_t)a.T, ++nb;
        const XT *src = reinterpret_cast<const XT *>(a.x) + (int64_t)rb * a.sxb + (int64_t)h * a.sxh + (int64_t)rt * a.sxt + (int64_t)g * DSUB;
        uint8_t *code_at = a.codes + (((int64_t)rb * a.H + h) * a.T_cap + a.t0 + rt) * ((int64_t)S * a.G) + g;

        // ---- the row: fp32 into registers, fp16 rounding into shared memory ----
        float r[kOwn * 8];
        if constexpr (sizeof(XT) == 2) {
            // the four warps fetch their 32 rows together (whole sectors); a thread's pieces then come back from shared memory
            constexpr int kAtOnce = 32 / kPieces;
            const unsigned long long mine = live ? (unsigned long long)src : 0ull;
            if (a.vec_ok) {
                uint4 v[8 / kAtOnce];
#pragma unroll
                for (int i = 0; i < 8 / kAtOnce; ++i) {
                    const unsigned long long from = __shfl_sync(0xffffffffu, mine, q * 8 + i * kAtOnce + lane / kPieces);
                    v[i] = make_uint4(0u, 0u, 0u, 0u);
                    if (from != 0ull) v[i] = __ldg(reinterpret_cast<const uint4 *>(from) + lane % kPieces);
                }
#pragma unroll
                for (int i = 0; i < 8 / kAtOnce; ++i)
                    *reinterpret_cast<uint4 *>(A + L::template at<kRows>(part * 32 + q * 8 + i * kAtOnce + lane / kPieces, (lane % kPieces) * 8)) = v[i];
            } else {
#pragma unroll 1
                for (int i = q * 8; i < q * 8 + 8; ++i) {
                    const unsigned long long from = __shfl_sync(0xffffffffu, mine, i);
#pragma unroll 1
                    for (int e = lane; e < DSUB; e += 32)
                        A[L::template at<kRows>(part * 32 + i, e)] = from != 0ull ? reinterpret_cast<const __half *>(from)[e] : __float2half_rn(0.0f);
                }
            }
            sync_quad();
#pragma unroll
            for (int m = 0; m < kOwn; ++m) unpack8(*reinterpret_cast<const uint4 *>(A + L::template at<kRows>(row, (4 * m + q) * 8)), r + 8 * m);
        } else {
            if (DSUB == 128 && a.vec_ok) {
                // The same in two halves.  Against 32 bytes of its own row a thread, us: 65536 rows x 8 heads, two stages 318 / 288, 16 stages x
                // 2048 rows 109 / 103.  64 wide it is 181 / 183.
                fetch_fp32(live ? (unsigned long long)src : 0ull, r);
            } else {
#pragma unroll
                for (int m = 0; m < kOwn; ++m) {
                    const XT *piece = src + 8 * (4 * m + q);
                    if (live && a.vec_ok) {
                        *reinterpret_cast<float4 *>(r + 8 * m) = __ldg(reinterpret_cast<const float4 *>(piece));
                        *reinterpret_cast<float4 *>(r + 8 * m + 4) = __ldg(reinterpret_cast<const float4 *>(piece) + 1);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) r[8 * m + j] = live ? to_float<XT>(piece[j]) : 0.0f;
                    }
                }
            }
#pragma unroll
            for (int m = 0; m < kOwn; ++m) *reinterpret_cast<uint4 *>(A + L::template at<kRows>(row, (4 * m + q) * 8)) = pack8(r + 8 * m);
        }
        if (a.vec_ok && grow + step < rows && grow + step > grow) {  // the next tile's row on its way to L2
            const char *ahead = reinterpret_cast<const char *>(reinterpret_cast<const XT *>(a.x) + (int64_t)nb * a.sxb + (int64_t)h * a.sxh +
                                                               (int64_t)nt * a.sxt + (int64_t)g * DSUB);
            constexpr int kLines = (int)(DSUB * sizeof(XT)) / 128;
            if (q < kLines) asm volatile("prefetch.global.L2 [%0];" ::"l"(ahead + q * 128));
        }

#pragma unroll 1
        for (int s = 0; s < S; ++s) {
            const uint32_t u = resident ? (uint32_t)s : trip * (uint32_t)S + s;
            const int buf = (int)(u & 1u);
            const __half *tab = tabs + (size_t)buf * (L::kTabBytes / 2);
            const float *nrm = nrms + buf * kMaxWords;
            const int64_t first = head_words + s * stage_words;
            // One group a block: the norms of the next stage's words are asked for here and wait in registers, because the four warps
            // that fill its buffer hold up the other twelve meanwhile.
            float ahead[2] = {inf, inf};
            if constexpr (GROUPS == 1) {
                if (a.sqnorm != nullptr && q == 0 && !resident && u >= 1 && u + 1 < uses) {
                    const float *from = a.sqnorm + head_words + (int64_t)((u + 1) % (uint32_t)S) * stage_words;
                    const int k = part * 64 + lane;
                    if (k < K) ahead[0] = __ldg(from + k);
                    if (k + 32 < K) ahead[1] = __ldg(from + k + 32);
                }
            }
            {
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // |r|^2 for the margins; the exact one is taken where it decides
#pragma unroll
                for (int i = 0; i < kOwn * 8; i += 4) {
                    fma2(sum[0], sum[1], r[i], r[i + 1], r[i], r[i + 1]);
                    fma2(sum[2], sum[3], r[i + 2], r[i + 3], r[i + 2], r[i + 3]);
                }
                xxs[q * kRows] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            sync_group();  // the group's rows are written, its scores read, the previous stage's words no longer used
            // A warp that gives up (never seen) lists every word from here on and takes words and norms from global memory.  It writes
            // nothing to the ring and no longer counts as having left a stage: the other group may be working on the buffer's
            // previous use, which is then not refilled either, so that all warps end up this way.
            if (!fail && !bounded_wait(full_bar + 8 * buf, (u >> 1) & 1u, a.spins)) fail = true;
            fail = __any_sync(0xffffffffu, fail);
            // by a warp that refills no tables where four do: a thread is held up by the products that it asks for nearly until they are done (1300
            // clocks), a refill takes 1450.  By warp 0, one after the other, 16 stages x 2048 rows took 105 us, so 102; x 16384 rows 525 / 507.
            if ((warp & 15) == 15) {
                if (lane == 0 && !fail) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d0 = tmem_base + (uint32_t)grp * kMaxWords, a0 = smem_u32(A), b0 = smem_u32(tab);
                    mma(d0, narrow_descriptor(smem_u32(smem + L::kOnes)), narrow_descriptor(smem_u32(smem + L::kSeed + buf * kSeedBytes)), 0u);
#pragma unroll 1
                    for (int ks = 0; ks < DSUB / 16; ++ks)
                        mma(d0, panel_descriptor(a0 + (ks >> 2) * (kRows * 128) + (ks & 3) * 32),
                            panel_descriptor(b0 + (ks >> 2) * (kMaxWords * 128) + (ks & 3) * 32), 1u);
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(my_mma) : "memory");
                    in_flight[grp] = mma_phase;
                }
                __syncwarp();
            }
            // use u - 1 is left: the last group to leave it refills its buffer, a share per warp (where there are four, those of q = 0)
            if (q * 4 < shares && !resident && u >= 1 && u + 1 < uses && !fail) {
                unsigned int n = 0u;
                __threadfence_block();
                if (lane == 0) n = atomicAdd(left + ((u - 1) & 1u) * 16 + q * 4 + part, 1u) + 1u;
                __threadfence_block();
                n = __shfl_sync(0xffffffffu, n, 0);
                if (n % (unsigned int)groups == 0u) load_table(u + 1, q * 4 + part, GROUPS == 1 && a.sqnorm != nullptr ? ahead : nullptr);
            }
            const float xx = (xxs[0] + xxs[kRows]) + (xxs[2 * kRows] + xxs[3 * kRows]);
            const float *share_tops = cc_tops + buf * 16;
            float cc_top = fmaxf(fmaxf(share_tops[0], share_tops[1]), fmaxf(share_tops[2], share_tops[3]));
            if (shares != 4)
#pragma unroll 1
                for (int i = 4; i < shares; ++i) cc_top = fmaxf(cc_top, share_tops[i]);
            const float u_top = rough_sqrt(xx * cc_top);
            const float margin = (sizeof(XT) == 2 && s == 0 ? 6.103515625e-05f : EXACT32 ? 2.01416015625e-03f : 1.03759765625e-03f) * u_top +
                                 9.5367431640625e-07f * xx + 3.0517578125e-05f * cc_top + 3.814697265625e-06f * rough_sqrt(cc_top) +
                                 (EXACT32 ? 9.5367431640625e-07f * rough_sqrt(xx) : 0.0f) + 1.1920929e-07f;
            if (!fail && !bounded_wait(my_mma, mma_phase, a.spins)) fail = true;
            mma_phase ^= 1u;
            fail = __any_sync(0xffffffffu, fail);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

            // ---- the row's largest score ----
            float top = -inf;
#pragma unroll 2
            for (int c = 0; c < 4; ++c) {
                uint32_t v[16];
                tmem_load16(v, scores + c * 16);
                float m0 = top, m1 = -inf;
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    m0 = max3(m0, __uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                    m1 = max3(m1, __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                }
                top = fmaxf(m0, m1);
            }
            tops[q * kRows] = fail ? -inf : top;  // (what a warp that gave up has read says nothing, and must not raise the others' limit)
            sync_quad();
            top = fmaxf(fmaxf(tops[0], tops[kRows]), fmaxf(tops[2 * kRows], tops[3 * kRows]));
            // ---- the words close to it ----
            const bool all = fail || !(xx < 1.0e9f) || !(cc_top < 1.3e5f) || !(top > -inf);
            // No score lies less than 2^-60 above the limit, where it would count in part and disturb the bits below: products of fp16 values
            // and their sums are multiples of 2^-48, and so is the limit, as the margin is at least 2^-23.
            constexpr float kSteep = 1.152921504606846976e18f;  // 2^60
            const float offset = (margin - top) * kSteep;
            uint64_t mask = 0ull;
#pragma unroll 2
            for (int c = 0; c < 4; ++c) {
                uint32_t v[16];
                tmem_load16(v, scores + c * 16);
                // bit i: column 2i, bit 8 + i: column 2i + 1.  The sign of (v - limit) is made 0 or 1 by a saturating multiply-add and
                // shifted in by a doubling one, which leaves the integer pipe to the maxima.
                float even = 0.0f, odd = 0.0f;
#pragma unroll
                for (int i = 7; i >= 0; --i)
                    double_add2(even, odd, fma_sat(__uint_as_float(v[2 * i]), kSteep, offset), fma_sat(__uint_as_float(v[2 * i + 1]), kSteep, offset));
                const uint32_t hits = __float_as_uint(fmaf(odd, 256.0f, even + 8388608.0f)) & 0xffffu;  // sums below 2^16 show in the mantissa of 2^23 + sum
                mask = (mask >> 16) | ((uint64_t)hits << 48);
            }
            if (all) mask = ~0ull;
            {
                const int n = __popcll(mask);
                const uint64_t more = mask & (mask - 1ull);
                const int lowest = n > 0 ? word_of_bit(__ffsll((long long)mask) - 1) : 0, also = n > 1 ? word_of_bit(__ffsll((long long)more) - 1) : 0;
                infos[q * kRows] = (uint16_t)((min(n, 3) << 12) | (also << 6) | lowest);
            }
            sync_quad();
            // ---- the choice ----
            int n_words = 0, wa = 0, wb = 0, wc = 0;  // the last three listed, of the first two of every thread
            bool hidden = false;  // a thread lists more words than it tells
#pragma unroll
            for (int i = 0; i < kShare; ++i) {
                const int info = infos[i * kRows], n = info >> 12;
                n_words += n;
                hidden |= n > 2;
                if (n >= 1) wc = wb, wb = wa, wa = i * 64 + (info & 63);
                if (n >= 2) wc = wb, wb = wa, wa = i * 64 + ((info >> 6) & 63);
            }
            int pick = min(wa, K - 1);  // (a row past the end may have listed padding words)
            // (rows past the end are all alike: one that is undecided would be 32 in a row)
            bool undecided = live && n_words != 1;
            if (__any_sync(0xffffffffu, undecided)) {  // the same in the four warps
                // Two words (mostly all there are): their dot products once more in fp32, each thread over its part of the
                // row.  Further apart than kClose u and 2^-22 (|r|^2 + cc), for the roundings of the norms' and distances' sums, they
                // settle about 99 rows in 100.
                if (undecided) {
                    const int ka = min(wa, K - 1), kb = min(wb, K - 1);
                    float dots[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int m = 0; m < kOwn; ++m) {
                        const int e = 8 * (4 * m + q);
                        float c0[8], c1[8];
                        if constexpr (EXACT32) {
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                *reinterpret_cast<float4 *>(c0 + 4 * i) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + ka) * DSUB + e) + i);
                                *reinterpret_cast<float4 *>(c1 + 4 * i) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + kb) * DSUB + e) + i);
                            }
                        } else {
                            unpack8(*reinterpret_cast<const uint4 *>(tab + L::template at<kMaxWords>(ka, e)), c0);
                            unpack8(*reinterpret_cast<const uint4 *>(tab + L::template at<kMaxWords>(kb, e)), c1);
                        }
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            fma2(dots[0], dots[1], r[8 * m + j], r[8 * m + j + 1], c0[j], c0[j + 1]);
                            fma2(dots[2], dots[3], r[8 * m + j], r[8 * m + j + 1], c1[j], c1[j + 1]);
                        }
                    }
                    tops[q * kRows] = dots[0] + dots[1];
                    xxs[q * kRows] = dots[2] + dots[3];
                }
                sync_quad();
                const bool three = undecided && n_words == 3 && !hidden && max(max(wa, wb), wc) < K;
                float better = 0.0f;  // of the first two
                if ((undecided && n_words == 2 && max(wa, wb) < K) || three) {
                    const float ta = ((tops[0] + tops[kRows]) + (tops[2 * kRows] + tops[3 * kRows])) - 0.5f * nrm[wa];
                    const float tb = ((xxs[0] + xxs[kRows]) + (xxs[2 * kRows] + xxs[3 * kRows])) - 0.5f * nrm[wb];
                    pick = tb > ta ? wb : wa;
                    better = fmaxf(ta, tb);
                    undecided = !(fabsf(ta - tb) > kClose * u_top + 2.4e-7f * (xx + cc_top) + 1.0e-30f);
                }
                // The third word of a row, in a quarter of the stages of 32 whitened rows.  Left to the chains, which hold up the whole group, us:
                // 16 stages x 2048 rows 102 / 96, whitened 207 / 185, whitened 4 x 4096 rows 1144 / 1025.
                if (__any_sync(0xffffffffu, three)) {  // the same in the four warps
                    sync_quad();
                    if (three) {
                        float dots[2] = {0.0f, 0.0f};
#pragma unroll
                        for (int m = 0; m < kOwn; ++m) {
                            const int e = 8 * (4 * m + q);
                            float c0[8];
                            if constexpr (EXACT32) {
#pragma unroll
                                for (int i = 0; i < 2; ++i)
                                    *reinterpret_cast<float4 *>(c0 + 4 * i) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + wc) * DSUB + e) + i);
                            } else {
                                unpack8(*reinterpret_cast<const uint4 *>(tab + L::template at<kMaxWords>(wc, e)), c0);
                            }
#pragma unroll
                            for (int j = 0; j < 8; j += 2) fma2(dots[0], dots[1], r[8 * m + j], r[8 * m + j + 1], c0[j], c0[j + 1]);
                        }
                        tops[q * kRows] = dots[0] + dots[1];
                    }
                    sync_quad();
                    if (three) {
                        const float tc = ((tops[0] + tops[kRows]) + (tops[2 * kRows] + tops[3 * kRows])) - 0.5f * nrm[wc];
                        const float close = kClose * u_top + 2.4e-7f * (xx + cc_top) + 1.0e-30f;
                        if (tc > better + close) pick = wc, undecided = false;  // however close the other two are
                        else if (!(better > tc + close)) undecided = true;
                    }
                }
                sync_quad();  // all of it is read
                // ---- the exact chains of every listed word, one row after the other through shared memory ----
#pragma unroll 1
                for (uint32_t open = __ballot_sync(0xffffffffu, undecided); open != 0u; open &= open - 1u) {  // the same in the four warps
                    const int who = __ffs((int)open) - 1;
                    // the eight floats of piece p = 4m + q: where the fp16 row was (128 bytes a panel) for q < 2, else in the slot
                    float *fp16_row = reinterpret_cast<float *>(A + (part * 32 + who) * 64);
                    auto piece_at = [&](int owner, int m) {
                        const int i = (owner & 1) * kOwn + m;
                        return owner < 2 ? fp16_row + (i >> 2) * (kRows * 32) + (i & 3) * 8 : slot + i * 8;
                    };
                    if (lane == who) {
#pragma unroll
                        for (int m = 0; m < kOwn; ++m) {
                            float *dst = piece_at(q, m);
                            *reinterpret_cast<float4 *>(dst) = make_float4(r[8 * m], r[8 * m + 1], r[8 * m + 2], r[8 * m + 3]);
                            *reinterpret_cast<float4 *>(dst + 4) = make_float4(r[8 * m + 4], r[8 * m + 5], r[8 * m + 6], r[8 * m + 7]);
                        }
                    }
                    sync_quad();
                    // |r|^2 in the library's order: lane (set, j) takes running sum j of the set
                    float sum = 0.0f;
#pragma unroll
                    for (int m = 0; m < kOwn; ++m) {
                        const float e = piece_at(lane >> 3, m)[lane & 7];
                        sum = __fadd_rn(sum, __fmul_rn(e, e));
                    }
                    float exact = __shfl_sync(0xffffffffu, sum, lane & 7);
#pragma unroll
                    for (int other = 1; other < 4; ++other) exact = __fadd_rn(exact, __shfl_sync(0xffffffffu, sum, other * 8 + (lane & 7)));
                    sum = exact;
                    exact = __shfl_sync(0xffffffffu, sum, 0);
#pragma unroll
                    for (int j = 1; j < 8; ++j) exact = __fadd_rn(exact, __shfl_sync(0xffffffffu, sum, j));
                    // lane l of warp q: bits l and 32 + l of the warp's mask of this row
                    const uint32_t listed[2] = {__shfl_sync(0xffffffffu, (uint32_t)mask, who), __shfl_sync(0xffffffffu, (uint32_t)(mask >> 32), who)};
                    float best = inf;
                    int arg = 0x7fff;
#pragma unroll 1
                    for (int half = 0; half < 2; ++half) {
                        const int k = q * 64 + word_of_bit(half * 32 + lane);
                        if ((((half ? listed[1] : listed[0]) >> lane) & 1u) != 0u && k < K) {
                            float dot = 0.0f;
                            auto chain = [&](auto fetch) {
                                // words from L2, 16 whitened stages x 2048 rows: 181 us, two pieces at a time 185; with two groups a block four spill
#pragma unroll (EXACT32 && GROUPS == 1 ? 4 : 2)
                                for (int p = 0; p < kPieces; ++p) {
                                    const float *from = piece_at(p & 3, p >> 2);
                                    float e[8], w[8];
                                    *reinterpret_cast<float4 *>(e) = *reinterpret_cast<const float4 *>(from);
                                    *reinterpret_cast<float4 *>(e + 4) = *reinterpret_cast<const float4 *>(from + 4);
                                    fetch(8 * p, w);
#pragma unroll
                                    for (int j = 0; j < 8; ++j) dot = __fmaf_rn(e[j], w[j], dot);
                                }
                            };
                            if constexpr (EXACT32) {
                                chain([&](int e, float *w) {
                                    *reinterpret_cast<float4 *>(w) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + k) * DSUB + e));
                                    *reinterpret_cast<float4 *>(w + 4) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + k) * DSUB + e + 4));
                                });
                            } else if (!fail) {
                                chain([&](int e, float *w) { unpack8(*reinterpret_cast<const uint4 *>(tab + L::template at<kMaxWords>(k, e)), w); });
                            } else {
                                chain([&](int e, float *w) { unpack8(load_in_place(a.tables + (first + k) * DSUB + e), w); });
                            }
                            float cc = nrm[k];
                            if (fail) cc = a.sqnorm != nullptr ? __ldg(a.sqnorm + first + k) : word_norm_alone<DSUB>(a.tables + (first + k) * DSUB);
                            const float dist = distance_expr(exact, cc, dot);
                            if (dist < best) best = dist, arg = k;  // a lane's two words ascend
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int off = 16; off >= 1; off >>= 1) {
                        const float other = __shfl_xor_sync(0xffffffffu, best, off);
                        const int other_arg = __shfl_xor_sync(0xffffffffu, arg, off);
                        if (other < best || (other == best && other_arg < arg)) best = other, arg = other_arg;
                    }
                    if (lane == who) {
                        tops[q * kRows] = best;
                        infos[q * kRows] = (uint16_t)arg;
                    }
                    sync_quad();
                    if (lane == who) {
                        float least = inf;
                        pick = 0;  // where every distance was +inf or NaN
#pragma unroll
                        for (int i = 0; i < kShare; ++i)  // ascending words: the lowest of a tie
                            if (tops[i * kRows] < least) least = tops[i * kRows], pick = infos[i * kRows];
                    }
                }
            }

            // ---- update ----
            if (s + 1 < S) {
                auto subtract = [&](auto fetch) {
#pragma unroll
                    for (int m = 0; m < kOwn; ++m) {
                        const int e = 8 * (4 * m + q);
                        float c[8];
                        fetch(e, c);
#pragma unroll
                        for (int j = 0; j < 8; j += 2) sub2(r[8 * m + j], r[8 * m + j + 1], c[j], c[j + 1]);
                        *reinterpret_cast<uint4 *>(A + L::template at<kRows>(row, e)) = pack8(r + 8 * m);
                    }
                };
                if constexpr (EXACT32 && DSUB == 128 && GROUPS == 1) {
                    // 16 bytes of 32 words a load are 32 lines; the words of 32 rows together are 4 lines a load.  Whole calls, us, 16 stages x 2048
                    // fp16 rows x 8 heads with rows 217 / 206.  (With two groups a block another one hides it: 1154 / 1157 for 4 x 4096 rows.)
                    // A few rows have few lines, and the exchange costs more: one row, one head, 16 stages 69 / 77, nine rows 75 / 81.
                    float words[kOwn * 8];
                    const float *word = a.words32 + (first + pick) * DSUB;
                    if (__popc(__ballot_sync(0xffffffffu, live)) > 8) {  // the same in the four warps
                        fetch_fp32((unsigned long long)word, words);
                    } else if (live) {
#pragma unroll
                        for (int m = 0; m < kOwn; ++m)
#pragma unroll
                            for (int i = 0; i < 2; ++i) *reinterpret_cast<float4 *>(words + 8 * m + 4 * i) = __ldg(reinterpret_cast<const float4 *>(word + 8 * (4 * m + q)) + i);
                    } else {
#pragma unroll
                        for (int i = 0; i < kOwn * 8; ++i) words[i] = 0.0f;
                    }
#pragma unroll
                    for (int m = 0; m < kOwn; ++m) {
#pragma unroll
                        for (int j = 0; j < 8; j += 2) sub2(r[8 * m + j], r[8 * m + j + 1], words[8 * m + j], words[8 * m + j + 1]);
                        *reinterpret_cast<uint4 *>(A + L::template at<kRows>(row, 8 * (4 * m + q))) = pack8(r + 8 * m);
                    }
                } else if constexpr (EXACT32) {
                    subtract([&](int e, float *c) {
                        *reinterpret_cast<float4 *>(c) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + pick) * DSUB + e));
                        *reinterpret_cast<float4 *>(c + 4) = __ldg(reinterpret_cast<const float4 *>(a.words32 + (first + pick) * DSUB + e + 4));
                    });
                } else if (!fail) {
                    subtract([&](int e, float *c) { unpack8(*reinterpret_cast<const uint4 *>(tab + L::template at<kMaxWords>(pick, e)), c); });
                } else {
                    subtract([&](int e, float *c) { unpack8(load_in_place(a.tables + (first + pick) * DSUB + e), c); });
                }
            }
            if (live && q == 0) code_at[(int64_t)s * a.G] = (uint8_t)pick;
        }
        if (a.recon != nullptr) {
            // a warp per row: the sum of the plain words in stage order, whole sectors in and out
            // (all eight rows of a warp at once where a block has one tile and nothing hides the words' way from L2)
            constexpr int kEach = DSUB / 32, kTogether = GROUPS == 1 ? 8 : 4;
            const int64_t o = (((int64_t)rb * a.H + h) * a.T + rt) * ((int64_t)a.G * DSUB) + (int64_t)g * DSUB;
            const long long mine = live ? o : -1ll;
            const unsigned long long codes_at = (unsigned long long)code_at;
            __threadfence_block();
            sync_quad();  // the codes that the q = 0 warp stored are read by all four
#pragma unroll 1
            for (int r0 = q * 8; r0 < q * 8 + 8; r0 += kTogether) {
                float sum[kTogether][kEach];
#pragma unroll
                for (int i = 0; i < kTogether; ++i)
#pragma unroll
                    for (int j = 0; j < kEach; ++j) sum[i][j] = 0.0f;
#pragma unroll 1
                for (int s0 = 0; s0 < S; s0 += 32) {
                    int some[kTogether];  // lane: the code of stage s0 + lane
#pragma unroll
                    for (int i = 0; i < kTogether; ++i) {
                        const uint8_t *from = reinterpret_cast<const uint8_t *>(__shfl_sync(0xffffffffu, codes_at, r0 + i));
                        const bool there = __shfl_sync(0xffffffffu, mine, r0 + i) >= 0;
                        some[i] = 0;
                        if (there && s0 + lane < S) some[i] = __ldcg(from + (int64_t)(s0 + lane) * a.G);
                    }
                    const int n = min(32, S - s0);
#pragma unroll 2
                    for (int s = 0; s < n; ++s) {
                        const __half *words = a.recon_tables + (head_words + (s0 + s) * stage_words) * DSUB + lane * kEach;
#pragma unroll
                        for (int i = 0; i < kTogether; ++i) {
                            const int code = __shfl_sync(0xffffffffu, some[i], s);
                            __half raw[kEach];
                            if constexpr (kEach == 4) *reinterpret_cast<uint2 *>(raw) = __ldg(reinterpret_cast<const uint2 *>(words + (int64_t)code * DSUB));
                            else *reinterpret_cast<uint32_t *>(raw) = __ldg(reinterpret_cast<const uint32_t *>(words + (int64_t)code * DSUB));
#pragma unroll
                            for (int j = 0; j < kEach; ++j) sum[i][j] = __fadd_rn(sum[i][j], __half2float(raw[j]));
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < kTogether; ++i) {
                    const long long at = __shfl_sync(0xffffffffu, mine, r0 + i);
                    if (at < 0) continue;
                    if (a.recon_dtype == TACVQ_F16) {
                        __half out[kEach];
#pragma unroll
                        for (int j = 0; j < kEach; ++j) out[j] = __float2half_rn(sum[i][j]);
                        __half *dst = (__half *)a.recon + at + lane * kEach;
                        if constexpr (kEach == 4) *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(out);
                        else *reinterpret_cast<uint32_t *>(dst) = *reinterpret_cast<const uint32_t *>(out);
                    } else {
                        float *dst = (float *)a.recon + at + lane * kEach;
                        if constexpr (kEach == 4) *reinterpret_cast<float4 *>(dst) = make_float4(sum[i][0], sum[i][1], sum[i][2], sum[i][3]);
                        else *reinterpret_cast<float2 *>(dst) = make_float2(sum[i][0], sum[i][1]);
                    }
                }
            }
        }
        sync_quad();  // the rows' places in shared memory take the next tile
    }
    if (__syncthreads_or(fail)) {
        // what is still in flight ends before the block's memory goes: each group's last product, each buffer's last copy (a
        // warp that gave up since owes the barrier an arrival)
        if ((tid & (kGroupThreads - 1)) == 0 && in_flight[grp] < 2u) bounded_wait(my_mma, in_flight[grp], kSpins);
        if (tid == 0) {
            atomicAdd(&g_timeouts, 1u);
            for (uint32_t buf = 0; buf < 2 && buf < uses; ++buf) {
                const unsigned int copies = left[buf * 16] / (unsigned int)groups;  // after the first one
                for (int share = 1; share < shares; ++share)
                    if (left[buf * 16 + share] / (unsigned int)groups < copies)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full_bar + 8 * buf) : "memory");
                bounded_wait(full_bar + 8 * buf, copies & 1u, kSpins);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)(groups * kMaxWords)) : "memory");
}

// tensor maps that could not be made: counted with the time-outs, so that a run on plain copies shows up
static std::atomic<unsigned int> g_map_failures{0};

template <int DSUB, typename XT, bool EXACT32>
static int launch(const EncodeArgs &e, const __half *scored) {
    const int64_t rows = (int64_t)e.B * e.T;
    if (rows >= (int64_t)1 << 31) return TACVQ_ERR_UNSUPPORTED;
    const int64_t words = (int64_t)e.H * e.S * e.G * e.K;
    if (words >= (int64_t)1 << 31 || (int64_t)e.H * e.G > 65535) return TACVQ_ERR_UNSUPPORTED;
    if (e.recon != nullptr && (reinterpret_cast<uintptr_t>(e.recon) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    CUtensorMap map;
    const int use_map = make_table_map(&map, scored, words, DSUB);
    if (!use_map && words >= kMaxWords) g_map_failures.fetch_add(1u);
    const int per_vec = 16 / (int)sizeof(XT);
    const int vec_ok = (reinterpret_cast<uintptr_t>(e.x) & 15u) == 0 && e.sxb % per_vec == 0 && e.sxh % per_vec == 0 && e.sxt % per_vec == 0;
    // One tile a block while that leaves no tile waiting, else two; as many blocks as the chip runs at once, which then
    // walk over the tiles of their (head, group).
    const int units = e.H * e.G;
    const int64_t tiles = (rows + kRows - 1) / kRows;
    const int groups = tiles * units <= 148 ? 1 : kMaxGroups;
    constexpr size_t smem = Layout<DSUB>::kBytes;
    static_assert(smem <= 227 * 1024, "one block an SM");
    int64_t blocks = (tiles + groups - 1) / groups;
    const int64_t most = units < 148 ? 148 / units : 1;
    if (blocks > most) blocks = most;
    const Args a{e.x, e.sxb, e.sxh, e.sxt, scored, EXACT32 ? (const float *)e.tables : nullptr, e.recon_tables, e.sqnorm, e.codes, e.recon,
                 e.recon_dtype, e.B, e.H, e.T, e.G, e.S, e.K, vec_ok, use_map, e.wait_spins < 0 ? kSpins : e.wait_spins, e.t0, e.T_cap};
    auto kernel = groups == 1 ? encode_wide_kernel<DSUB, XT, EXACT32, 1> : encode_wide_kernel<DSUB, XT, EXACT32, kMaxGroups>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return (int)err;
    kernel<<<dim3((unsigned)blocks, (unsigned)units), groups * kGroupThreads, smem, e.stream>>>(a, map);
    return launch_status();
}

}  // namespace wide

// Returns TACVQ_ERR_UNSUPPORTED when the geometry is not this kernel's.
int encode_wide_launch(const EncodeArgs &e) {
    const int d = e.D / e.G;
    if ((d != 64 && d != 128) || e.K > kMaxWords || (reinterpret_cast<uintptr_t>(e.tables) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    if (e.tables_f32) {  // transformed words: they come with their fp16 rounding and norms, or not to this kernel
        if (e.filter_tables == nullptr || e.sqnorm == nullptr || e.x_dtype != TACVQ_F32 || (reinterpret_cast<uintptr_t>(e.recon_tables) & 15u) != 0)
            return TACVQ_ERR_UNSUPPORTED;
        return d == 128 ? wide::launch<128, float, true>(e, e.filter_tables) : wide::launch<64, float, true>(e, e.filter_tables);
    }
    const __half *tables = (const __half *)e.tables;
    if (e.x_dtype == TACVQ_F16) return d == 128 ? wide::launch<128, __half, false>(e, tables) : wide::launch<64, __half, false>(e, tables);
    return d == 128 ? wide::launch<128, float, false>(e, tables) : wide::launch<64, float, false>(e, tables);
}

int narrow_timeouts(unsigned int *out);
int few_timeouts(unsigned int *out);

// of all encode kernels that wait for products or copies
int tensor_memory_timeouts(unsigned int *out) {
    unsigned int narrow = 0, few = 0;
    int st = (int)cudaMemcpyFromSymbol(out, wide::g_timeouts, sizeof(unsigned int));
    if (st == 0) st = narrow_timeouts(&narrow);
    if (st == 0) st = few_timeouts(&few);
    if (st == 0) *out += wide::g_map_failures.load() + narrow + few;
    return st;
}

}  // namespace tacvq
