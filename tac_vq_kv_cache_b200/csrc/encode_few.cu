// Encode of a handful of rows (decode steps) for wide groups (d = 32, 64, 128; fp16 tables): one block per
// (side, head, group) and one, two or four rows, all stages in one launch, K and V together.
//
// What bounds it: with so few rows the arithmetic is nothing; the time is the serial chain of the stages.  The
// d-step fused-multiply-add chain that the library's order prescribes alone takes 700 cycles, so it is not run:
// the tensor cores score all 256 words against the residual (mma.sync, A = 16 words, B's eight columns = the fp16
// high and low halves of up to four residual rows, error 2^-22), and the word with the best score is the code
// unless another one lies within the margin below.  Then, for about one row-stage in 200, the block runs the exact
// chain for every word, a thread per word.  The tables of the next two stages (64 KB each at d = 128) arrive by
// TMA meanwhile, in 128-byte-swizzled panels, from which ldmatrix and a lane per word both read without conflicts;
// eight further warps compute the next stage's |c|^2 beside the search.
//
// Margin.  In units of t = r.c - |c|^2/2 (distance = |r|^2 - 2t): the exact chain rounds d times, at most
// 2^-17 |r||c| in all; the tensor core's fp32 accumulation at most 2^-16 |r||c|; the halves drop at most
// 2^-22 |r||c| + 2^-21 |c| (fp16 subnormals); the roundings of the distance expression are 2^-22 (|r|^2 + |c|^2).
// Two words are told apart if their scores differ by twice the sum; the kernel allows twice that again:
//   1.5 * 2^-14 |r| max|c| + 2^-20 (|r|^2 + max|c|^2) + 2^-18 max|c|.
//
// Measured, 8 KV heads, K and V of one decode step, device time: 16 stages x 128, batch 1: 140 us in two launches of the
// 128-row tile kernel of encode_tc_large.cu, 27 us here (1.3 us a stage: reading the 64 KB table from shared memory for the
// scores and again for |c|^2 is 0.6 us of it, the exchange of the votes and the update 0.5 us); 2 stages x 128, batch
// 16: 31 us before, 7.5 us here.  Running the exact chain in every stage instead of the scores: 33 us; a cluster of eight
// blocks with 32 words each: 87 us (a cluster barrier and the fetch of the winning word are 0.7 us a stage, and not
// all clusters are resident at once).
//
// Reference statements: src/jointkv/closed_loop_vq.py:52-76 (search), :343-395 (stage recursion).

#include <type_traits>

#include "common.cuh"
#include "table_map.cuh"

namespace tacvq {

namespace {

constexpr int kThreads = kMaxWords;  // a thread per word; as many threads again compute |c|^2 one stage ahead
constexpr int kWarps = kThreads / 32;
constexpr int kRing = 3;             // stages of tables in shared memory
constexpr int kSpins = 1 << 20;

// blocks in which a wait was given up; expected to stay 0
__device__ unsigned int g_timeouts = 0;

struct FewSide {
    const void *x;
    const __half *tables;
    const float *sqnorm;  // optional |word|^2
    uint8_t *codes;
    void *recon;
};

template <int DSUB, int R>
struct FewLayout {
    static constexpr int kPanel = DSUB < 64 ? DSUB : 64;                   // halves per panel row (64 or 128 bytes)
    static constexpr size_t kSlot = (size_t)kMaxWords * DSUB * 2;
    // the ring of tables (swizzled panels) comes first; behind it, as its length is a run-time value:
    static constexpr size_t kRes = 0;                                      // [R][DSUB] float: residual
    static constexpr size_t kDec = kRes + (size_t)R * DSUB * 4;            // [R][DSUB] float: sum of the words so far
    static constexpr size_t kParts = kDec + (size_t)R * DSUB * 4;          // [8][DSUB + 8] half: column r = high, 4 + r = low halves of row r
    static constexpr size_t kScore = kParts + (size_t)8 * (DSUB + 8) * 2;  // [R][256] float
    static constexpr size_t kVote = kScore + (size_t)R * kMaxWords * 4;    // [R][8] uint4: best, its word, second, largest |c|^2 per warp
    static constexpr size_t kNrm = kVote + (size_t)R * kWarps * 16;        // [2][256] float: |c|^2 of this and the next stage
    static constexpr size_t kBar = kNrm + 2 * kMaxWords * 4;               // [ring] mbarrier
    static constexpr size_t kTail = kBar + kRing * 8;
    static constexpr size_t bytes(int ring) { return 1024 + (size_t)ring * kSlot + kTail; }
    // byte offset of element e (a multiple of 8) of word k in a slot: the 16-byte pieces of a panel row are exclusive-ored
    // with the row (128-byte rows: row & 7; 64-byte rows: (row / 2) & 3), as the copy engine stores them
    __device__ static __forceinline__ int at(int k, int e) {
        if constexpr (DSUB >= 64) return (e >> 6) * (kMaxWords * 128) + k * 128 + ((((e >> 3) & 7) ^ (k & 7)) << 4) + (e & 7) * 2;
        else return k * 64 + ((((e >> 3) & 3) ^ ((k >> 1) & 3)) << 4) + (e & 7) * 2;
    }
};

// monotone map float -> uint32; NaN maps above everything
__device__ __forceinline__ uint32_t ordered_bits_of(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// |v|^2 in the library's order for d a multiple of 32 by eight neighbouring lanes (see common.cuh); all eight
// return the total.
template <int DSUB>
__device__ __forceinline__ float lanes8_sqnorm(const float *v, int lane) {
    const int j = lane & 7;
    float set[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < DSUB; i += 8) set[(i >> 3) & 3] = __fadd_rn(set[(i >> 3) & 3], __fmul_rn(v[i + j], v[i + j]));
    const float mine = __fadd_rn(__fadd_rn(__fadd_rn(set[0], set[1]), set[2]), set[3]);
    float sums[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sums[k] = __shfl_sync(0xffffffffu, mine, (lane & 24) + k);
    float total = sums[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) total = __fadd_rn(total, sums[k]);
    return total;
}

__device__ __forceinline__ void unpack_piece(const unsigned char *at, float (&c)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4 *>(at);
    const __half2 *hv = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(hv[j]);
        c[2 * j] = f.x;
        c[2 * j + 1] = f.y;
    }
}

// set + (a, b)^2 for a pair of elements, products and sums rounded separately
__device__ __forceinline__ void add_square2(unsigned long long &set, float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    asm("mul.rn.f32x2 %0, %0, %0;" : "+l"(v));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(set) : "l"(v));
}

// |c|^2 of one word in the library's order (common.cuh), by one thread
template <int DSUB, typename PieceOf>
__device__ __forceinline__ float word_sqnorm(PieceOf piece_of) {
    unsigned long long set[4][4];  // four sets of eight running sums, in pairs
#pragma unroll
    for (int i = 0; i < 16; ++i) set[i >> 2][i & 3] = 0ull;
#pragma unroll
    for (int i = 0; i < DSUB; i += 8) {
        float c[8];
        unpack_piece(piece_of(i), c);
#pragma unroll
        for (int j = 0; j < 4; ++j) add_square2(set[(i >> 3) & 3][j], c[2 * j], c[2 * j + 1]);
    }
    float total = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        unsigned long long sum = set[0][j];
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum) : "l"(set[1][j]));
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum) : "l"(set[2][j]));
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum) : "l"(set[3][j]));
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(sum));
        total = j == 0 ? lo : __fadd_rn(total, lo);
        total = __fadd_rn(total, hi);
    }
    return total;
}

__device__ __forceinline__ void searchers_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

}  // namespace

// R rows per block.  blockIdx.x = row block, .y = head * G + group, .z = side.
template <int DSUB, typename XT, int R>
__global__ void __launch_bounds__(2 * kThreads, 1)
encode_few_wide_kernel(FewSide first, FewSide second, int64_t sxb, int64_t sxh, int64_t sxt, int recon_dtype, int ring,
                       int32_t *__restrict__ seq_start, int32_t *__restrict__ seq_end, int start, int end, int B, int H, int T,
                       int G, int S, int K, int64_t t0, int64_t T_cap, int spins, const __grid_constant__ CUtensorMap first_map,
                       const __grid_constant__ CUtensorMap second_map) {
    using L = FewLayout<DSUB, R>;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    unsigned char *tab = smem_dyn + ((1024u - ((uint32_t)__cvta_generic_to_shared(smem_dyn) & 1023u)) & 1023u);
    unsigned char *smem = tab + (size_t)ring * L::kSlot;
    float *res = reinterpret_cast<float *>(smem + L::kRes);
    float *dec = reinterpret_cast<float *>(smem + L::kDec);
    __half *parts = reinterpret_cast<__half *>(smem + L::kParts);
    float *score = reinterpret_cast<float *>(smem + L::kScore);
    uint4 *vote = reinterpret_cast<uint4 *>(smem + L::kVote);
    float *nrm = reinterpret_cast<float *>(smem + L::kNrm);
    const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(smem + L::kBar);
    const uint32_t tab0 = (uint32_t)__cvta_generic_to_shared(tab);
    constexpr int PS = DSUB + 8;  // halves per column of `parts`: padded so that a fragment's columns differ in bank

    const int h = blockIdx.y / G, g = blockIdx.y % G;
    const bool is_second = blockIdx.z != 0;
    const FewSide side = is_second ? second : first;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows = B * T, row0 = blockIdx.x * R;
    const float inf = __int_as_float(0x7f800000);

    const __half *words = side.tables + ((int64_t)h * S * G + g) * K * DSUB;  // stage s is s * G * K words on
    const int64_t stage_halves = (int64_t)G * K * DSUB;
    auto request = [&](int s, int slot) {  // table of stage s, by one thread
        const uint32_t bar = bar0 + slot * 8, dst = tab0 + (uint32_t)(slot * L::kSlot);
        const int first_word = ((h * S + s) * G + g) * K;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)L::kSlot) : "memory");
#pragma unroll
        for (int panel = 0; panel < DSUB / L::kPanel; ++panel)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                             dst + panel * (kMaxWords * 128)),
                         "l"(is_second ? &second_map : &first_map), "r"(panel * 64), "r"(first_word), "r"(bar)
                         : "memory");
    };
    auto arrived = [&](int slot, int phase, int polls) {
        int ok = 0;
        for (int spin = 0; spin < polls && !ok; ++spin)  // bounded: on running out the stage reads global memory
            asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.s32 %0, 1, 0, p;\n}"
                         : "=r"(ok) : "r"(bar0 + slot * 8), "r"((uint32_t)phase) : "memory");
        return ok != 0;
    };
    if (seq_start != nullptr) start_after_previous_kernel();  // a decode step: its attention is next, and waits for this grid where it has to
    if (tid == 0) {
        for (int i = 0; i < ring; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + i * 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int s = 0; s < ring && s < 2; ++s) request(s, s);
    }
    if (seq_start != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
        for (int b = tid; b < B; b += 2 * kThreads) {
            seq_start[b] = start;
            seq_end[b] = end;
        }
    auto split = [&](int r, int e, float v) {
        const __half hi = __float2half_rn(v);
        parts[r * PS + e] = hi;
        parts[(4 + r) * PS + e] = __float2half_rn(v - __half2float(hi));
    };
    if constexpr (R < 4)  // columns without a row
        for (int i = tid; i < 8 * PS; i += 2 * kThreads)
            if (((i / PS) & 3) >= R) parts[i] = __float2half_rn(0.0f);
    for (int i = tid; i < R * DSUB; i += 2 * kThreads) {
        const int row = row0 + i / DSUB;
        float v = 0.0f;
        if (row < rows) {
            const int b = row / T, t = row % T;
            v = to_float<XT>(((const XT *)side.x)[(int64_t)b * sxb + (int64_t)h * sxh + (int64_t)t * sxt + (int64_t)g * DSUB + i % DSUB]);
        }
        res[i] = v;
        dec[i] = 0.0f;
        split(i / DSUB, i % DSUB, v);
    }
    uint8_t *code_at = nullptr;  // threads 0..R-1: their row's first code byte
    if (tid < R && row0 + tid < rows) {
        const int b = (row0 + tid) / T, t = (row0 + tid) % T;
        code_at = side.codes + (((int64_t)b * H + h) * T_cap + t0 + t) * ((int64_t)S * G) + g;
    }
    __syncthreads();  // mbarriers and rows

    const bool searcher = tid < kThreads;
    const int word = tid & (kThreads - 1);
    auto norm_stage = [&](int s, int slot, bool staged) {  // by the threads that do not search
        float v = inf;  // words past K can never be chosen
        if (word < K) {
            if (side.sqnorm != nullptr) v = side.sqnorm[(((int64_t)h * S + s) * G + g) * K + word];
            else if (staged) v = word_sqnorm<DSUB>([&](int e) { return tab + (size_t)slot * L::kSlot + L::at(word, e); });
            else v = word_sqnorm<DSUB>([&](int e) { return reinterpret_cast<const unsigned char *>(words + s * stage_halves + (int64_t)word * DSUB + e); });
        }
        nrm[(s & 1) * kMaxWords + word] = v;
    };
    if (!searcher) norm_stage(0, 0, __all_sync(0xffffffffu, arrived(0, 0, spins)));

    int requested = S < 2 ? S : 2;
    int slot = 0, phase = 0, next = ring > 2 ? 2 : 0;  // slot of stage s with its phase, slot of stage s + 2
    for (int s = 0; s < S; ++s) {
        const bool staged = __syncthreads_and(arrived(slot, phase, spins));  // also: norms of stage s and the previous update have settled
        if (!staged) spins = 0;  // a table did not arrive in time: no further one is asked for or waited for
        const int slot_now = slot;
        slot = slot + 1 == ring ? (phase ^= 1, 0) : slot + 1;
        if (!searcher) {
            if (s + 1 < S) norm_stage(s + 1, slot, __all_sync(0xffffffffu, arrived(slot, phase, spins)));
            continue;
        }
        const unsigned char *stage = tab + (size_t)slot_now * L::kSlot;
        const __half *plain = words + s * stage_halves;
        if (tid == 0 && s + 2 < S && spins != 0) {  // its slot was last read by the previous stage's update
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            request(s + 2, next);
            ++requested;
        }
        next = next + 1 == ring ? 0 : next + 1;
        auto piece_of = [&](int k, int e) {  // eight elements of word k
            return staged ? stage + L::at(k, e) : reinterpret_cast<const unsigned char *>(plain + (int64_t)k * DSUB + e);
        };
        const float cc = nrm[(s & 1) * kMaxWords + tid];

        // ---- scores of this warp's 32 words: two tiles of 16 words x 8 columns -----------------------------------
        float acc[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
        if (staged) {
#pragma unroll
            for (int ks = 0; ks < DSUB / 16; ++ks) {
                const __half *col = parts + (lane >> 2) * PS + ks * 16 + 2 * (lane & 3);
                const uint32_t b0 = *reinterpret_cast<const uint32_t *>(col), b1 = *reinterpret_cast<const uint32_t *>(col + 8);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    uint32_t a[4];
                    const uint32_t from = tab0 + (uint32_t)(slot_now * L::kSlot) + L::at(warp * 32 + m * 16 + (lane & 15), ks * 16 + (lane >> 4) * 8);
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(from));
                    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                        : "+f"(acc[m][0]), "+f"(acc[m][1]), "+f"(acc[m][2]), "+f"(acc[m][3])
                        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
                }
            }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // lane's columns 2 (lane % 4) + (i & 1); high and low meet across lanes 2 apart
                const float sum = acc[m][i] + __shfl_xor_sync(0xffffffffu, acc[m][i], 2);
                const int r = 2 * (lane & 1) + (i & 1);
                if ((lane & 2) == 0 && r < R) score[r * kMaxWords + warp * 32 + m * 16 + (i >> 1) * 8 + (lane >> 2)] = sum;
            }
        __syncwarp();
        float xx[R];
        {
            const float v = lanes8_sqnorm<DSUB>(res + ((lane >> 3) % R) * DSUB, lane);  // a group of eight lanes per row
#pragma unroll
            for (int r = 0; r < R; ++r) xx[r] = __shfl_sync(0xffffffffu, v, r * 8);
        }
        const uint32_t cc_top = __reduce_max_sync(0xffffffffu, tid < K ? __float_as_uint(cc) : 0u);  // a NaN or negative-looking one ranks high
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float t = __fmaf_rn(-0.5f, cc, score[r * kMaxWords + tid]);
            const uint32_t bits = ordered_bits_of(t);  // a NaN (as of an infinite product) becomes the best or the worst: seen below
            const uint32_t top = __reduce_max_sync(0xffffffffu, bits);
            const int w = __ffs((int)__ballot_sync(0xffffffffu, bits == top)) - 1;
            const uint32_t second = __reduce_max_sync(0xffffffffu, lane == w ? 0u : bits);
            if (lane == 0) vote[r * kWarps + warp] = make_uint4(top, (unsigned)(warp * 32 + w), second, cc_top);
        }
        searchers_barrier();
        // ---- every warp: the winner of each row (eight lanes a row) and whether the scores decide it ---------------
        int pick;
        {
            const int r = (lane >> 3) % R;
            uint4 v = vote[r * kWarps + (lane & 7)];
            if constexpr (R == 1) {  // whole-warp reductions: the four groups of eight lanes hold the same votes
                const uint32_t top = __reduce_max_sync(0xffffffffu, v.x);
                const int w = __ffs((int)__ballot_sync(0xffffffffu, v.x == top)) - 1;  // the lowest warp, hence the lowest word
                const uint32_t second = __reduce_max_sync(0xffffffffu, (lane & 7) == w ? v.z : v.x);
                v = make_uint4(top, __shfl_sync(0xffffffffu, v.y, w), second, __reduce_max_sync(0xffffffffu, v.w));
            } else {
#pragma unroll
                for (int off = 4; off >= 1; off >>= 1) {
                    const uint4 o = make_uint4(__shfl_xor_sync(0xffffffffu, v.x, off), __shfl_xor_sync(0xffffffffu, v.y, off),
                                               __shfl_xor_sync(0xffffffffu, v.z, off), __shfl_xor_sync(0xffffffffu, v.w, off));
                    const bool theirs = o.x > v.x || (o.x == v.x && o.y < v.y);
                    v = theirs ? make_uint4(o.x, o.y, max(o.z, v.x), max(o.w, v.w)) : make_uint4(v.x, v.y, max(v.z, o.x), max(o.w, v.w));
                }
            }
            pick = (int)v.y;
            float rr = xx[0];
#pragma unroll
            for (int q = 1; q < R; ++q) rr = r == q ? xx[q] : rr;
            auto value_of = [](uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); };
            const float cm = __uint_as_float(v.w), gap = value_of(v.x) - value_of(v.z);
            const float margin = 9.1552734375e-05f * sqrtf(rr * cm) + 9.5367431640625e-07f * (rr + cm) + 3.814697265625e-06f * sqrtf(cm);
            // residuals or words beyond fp16's comfort, or any NaN, are left to the exact chain
            const bool decided = staged && rr < 1073741824.0f && cm < 1073741824.0f && gap > margin;
            if (!__all_sync(0xffffffffu, decided)) {  // the same answer in every warp
                searchers_barrier();  // everybody has read the votes
                float dot[R];
#pragma unroll
                for (int q = 0; q < R; ++q) dot[q] = 0.0f;
#pragma unroll 4
                for (int i = 0; i < DSUB; i += 8) {
                    float c[8];
                    unpack_piece(piece_of(tid < K ? tid : 0, i), c);
#pragma unroll
                    for (int q = 0; q < R; ++q)
#pragma unroll
                        for (int j = 0; j < 8; ++j) dot[q] = __fmaf_rn(res[q * DSUB + i + j], c[j], dot[q]);
                }
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    const float dist = distance_expr(xx[q], cc, dot[q]);
                    // a NaN or infinite distance never wins, as in a strict '<' scan from +inf; + 0 makes -0 equal +0
                    const uint32_t bits = tid < K && dist < inf ? ordered_bits_of(dist + 0.0f) : 0xffffffffu;
                    const uint32_t low = __reduce_min_sync(0xffffffffu, bits);
                    const int w = __ffs((int)__ballot_sync(0xffffffffu, bits == low)) - 1;
                    if (lane == 0) vote[q * kWarps + warp] = make_uint4(low, (unsigned)(warp * 32 + w), 0u, 0u);
                }
                searchers_barrier();
                uint4 e = vote[r * kWarps + (lane & 7)];
#pragma unroll
                for (int off = 4; off >= 1; off >>= 1) {
                    const uint32_t ox = __shfl_xor_sync(0xffffffffu, e.x, off), oy = __shfl_xor_sync(0xffffffffu, e.y, off);
                    if (ox < e.x || (ox == e.x && oy < e.y)) {
                        e.x = ox;
                        e.y = oy;
                    }
                }
                pick = e.x == 0xffffffffu ? 0 : (int)e.y;
            }
        }
        // ---- update: subtract the chosen words ----------------------------------------------------------------------
#pragma unroll
        for (int base = 0; base < R * DSUB; base += kThreads) {
            const int i = base + tid, r = i / DSUB, e = i % DSUB;
            const int k = __shfl_sync(0xffffffffu, pick, (r & 3) * 8 & 31);
            if (i < R * DSUB) {
                const float f = __half2float(*reinterpret_cast<const __half *>(piece_of(k, e & ~7) + (e & 7) * 2));
                const float v = __fsub_rn(res[i], f);
                res[i] = v;
                dec[i] = __fadd_rn(dec[i], f);
                split(r, e, v);
            }
        }
        if (warp == 0) {
            const int k = __shfl_sync(0xffffffffu, pick, (lane & 3) * 8);
            if (code_at != nullptr) code_at[(int64_t)s * G] = (uint8_t)k;
        }
    }
    if (spins == 0 && tid == 0) {  // never seen: one more bounded wait, so that no copy outlives the block
        atomicAdd(&g_timeouts, 1u);
        for (int i = 0; i < ring && i < requested; ++i) arrived(i, ((requested - i + ring - 1) / ring - 1) & 1, kSpins);
    }
    if (side.recon != nullptr) {
        for (int i = tid; searcher && i < R * DSUB; i += kThreads) {  // each thread's own elements
            const int row = row0 + i / DSUB;
            if (row >= rows) continue;
            const int b = row / T, t = row % T;
            const int64_t at = (((int64_t)b * H + h) * T + t) * ((int64_t)G * DSUB) + (int64_t)g * DSUB + i % DSUB;
            if (recon_dtype == TACVQ_F16) store_as<__half>((__half *)side.recon + at, dec[i]);
            else store_as<float>((float *)side.recon + at, dec[i]);
        }
    }
}

template <int DSUB, typename XT>
static int launch_few(const FewSide &first, const FewSide &second, int sides, int64_t sxb, int64_t sxh, int64_t sxt, int recon_dtype,
                      int32_t *seq_start, int32_t *seq_end, int start, int end, int B, int H, int T, int G, int S, int K,
                      int64_t t0, int64_t T_cap, int spins, cudaStream_t stream) {
    const int64_t rows = (int64_t)B * T;
    const int ring = S < kRing ? S : kRing;
    CUtensorMap first_map, second_map;
    const int64_t all_words = (int64_t)H * S * G * K;
    if (!make_table_map(&first_map, first.tables, all_words, DSUB) || !make_table_map(&second_map, second.tables, all_words, DSUB))
        return TACVQ_ERR_UNSUPPORTED;
    auto go = [&](auto kernel, int per_block, size_t smem) -> int {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        dim3 grid((unsigned)((rows + per_block - 1) / per_block), (unsigned)(H * G), (unsigned)sides);
        const cudaError_t launched = launch_dependent(seq_start != nullptr, kernel, grid, dim3(2 * kThreads), smem, stream, first, second, sxb, sxh, sxt,
                                                      recon_dtype, ring, seq_start, seq_end, start, end, B, H, T, G, S, K, t0, T_cap,
                                                      spins < 0 ? kSpins : spins, first_map, second_map);
        return launched == cudaSuccess ? launch_status() : (int)launched;
    };
    // the fewest rows per block that keep the launch to about one block per SM
    const int64_t units = (int64_t)H * G * sides;
    if (rows * units <= 148) return go(encode_few_wide_kernel<DSUB, XT, 1>, 1, FewLayout<DSUB, 1>::bytes(ring));
    if (rows * units <= 2 * 148) return go(encode_few_wide_kernel<DSUB, XT, 2>, 2, FewLayout<DSUB, 2>::bytes(ring));
    return go(encode_few_wide_kernel<DSUB, XT, 4>, 4, FewLayout<DSUB, 4>::bytes(ring));
}

static bool few_wide_ok(const void *x, const void *tables, int x_dtype, int64_t rows, int K) {
    return rows > 0 && rows <= (1 << 20) && K <= kMaxWords && ((uintptr_t)tables & 15) == 0 &&
           ((uintptr_t)x % (x_dtype == TACVQ_F16 ? 2 : 4)) == 0;
}

template <typename XT>
static int dispatch_few(int d, const FewSide &first, const FewSide &second, int sides, int64_t sxb, int64_t sxh, int64_t sxt,
                        int recon_dtype, int32_t *seq_start, int32_t *seq_end, int start, int end, int B, int H, int T, int G,
                        int S, int K, int64_t t0, int64_t T_cap, int spins, cudaStream_t stream) {
    switch (d) {
#define TACVQ_CASE(N)                                                                                                             \
    case N:                                                                                                                       \
        return launch_few<N, XT>(first, second, sides, sxb, sxh, sxt, recon_dtype, seq_start, seq_end, start, end, B, H, T, G, S, \
                                 K, t0, T_cap, spins, stream);
        TACVQ_CASE(32)
        TACVQ_CASE(64)
        TACVQ_CASE(128)
#undef TACVQ_CASE
        default: return TACVQ_ERR_UNSUPPORTED;
    }
}

// One side (K or V rows of an append).
int encode_few_wide_launch(const EncodeArgs &a) {
    if (a.tables_f32 || !few_wide_ok(a.x, a.tables, a.x_dtype, (int64_t)a.B * a.T, a.K)) return TACVQ_ERR_UNSUPPORTED;
    const FewSide side = {a.x, (const __half *)a.tables, a.sqnorm, a.codes, a.recon};
    auto go = [&](auto *tag) {
        using XT = typename std::remove_pointer<decltype(tag)>::type;
        return dispatch_few<XT>(a.D / a.G, side, side, 1, a.sxb, a.sxh, a.sxt, a.recon_dtype, nullptr, nullptr, 0, 0, a.B, a.H, a.T,
                                a.G, a.S, a.K, a.t0, a.T_cap, a.wait_spins, a.stream);
    };
    return a.x_dtype == TACVQ_F16 ? go((__half *)nullptr) : go((float *)nullptr);
}

// Both sides of a decode step and the visible ranges.
int decode_prologue_wide_launch(const void *k_rows, const void *v_rows, int rows_dtype, int64_t sxb, int64_t sxh, int64_t sxt,
                                const __half *ktab, const __half *vtab, uint8_t *kcodes, uint8_t *vcodes, int32_t *seq_start,
                                int32_t *seq_end, int start, int end, int B, int H, int T, int D, int G, int S, int K, int64_t t0,
                                int64_t T_cap, cudaStream_t stream) {
    if (!few_wide_ok(k_rows, ktab, rows_dtype, (int64_t)B * T, K) || !few_wide_ok(v_rows, vtab, rows_dtype, 1, K)) return TACVQ_ERR_UNSUPPORTED;
    const FewSide first = {k_rows, ktab, nullptr, kcodes, nullptr}, second = {v_rows, vtab, nullptr, vcodes, nullptr};
    return rows_dtype == TACVQ_F16
               ? dispatch_few<__half>(D / G, first, second, 2, sxb, sxh, sxt, TACVQ_F16, seq_start, seq_end, start, end, B, H, T, G, S, K,
                                      t0, T_cap, -1, stream)
               : dispatch_few<float>(D / G, first, second, 2, sxb, sxh, sxt, TACVQ_F16, seq_start, seq_end, start, end, B, H, T, G, S, K,
                                     t0, T_cap, -1, stream);
}

int few_timeouts(unsigned int *out) { return (int)cudaMemcpyFromSymbol(out, g_timeouts, sizeof(unsigned int)); }

}  // namespace tacvq
