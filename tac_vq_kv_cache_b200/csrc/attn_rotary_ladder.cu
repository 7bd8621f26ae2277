// Attention over codes of PRE-rotary keys for deep ladders of full-width words (one group of 128 channels, 4 to 16 residual
// stages, 256 words): the layout the adapter is deployed with.
//
// What bounds it.  A token's K row is the sum of one 256-byte word per stage and so is its V row: 8 KB of words for 32 code
// bytes.  Fetched per token from L2 (attn_rotary_kernel) that traffic is everything: 86 us at 8 heads x 4096 tokens.  Here
//   keys    eight blocks of a cluster share a head's key tables, 16 channels each (8j .. 8j+7 and their rotary partners 64 +
//           8j ..), 128 KB of shared memory at 16 stages.  A block rebuilds its 16 channels of every token of the cluster
//           and leaves its part of the scores; the parts meet through distributed shared memory.
//   values  are never rebuilt: sum_t p_t sum_s word_s[code] = sum_s sum_w (sum of p_t over the tokens with code w) word_w,
//           so block j adds the weights of all tokens up by code for stages j and j + 8 and multiplies the two histograms with
//           these stages' words, each read once; the eight results are added through distributed shared memory.
//
// Pass K on the tensor cores.  A token's words are gathered by ldmatrix: lane l gives the address of stage l % 16, piece l / 16
// (8 channels), and the transposed 8x8 matrices are the A operand (row = channel, k = stage) of one m16n8k16 product whose
// B operand has ones in the token's column only: eight tokens add up into one accumulator, column = token, one fp32 sum per
// channel.  (With the words as B operand, 16 stages x 8 channels, it took two products a token and was bound by them:
// 34 k clocks for 4096 tokens.)  A code's 32 pieces lie in one 512-byte row with the stage deciding the bank, so every gather is
// free of conflicts for any codes.  The sums are rounded to fp16 (the reference's fp16 window), rotated in the fp16 arithmetic of
// apply_rotary_pos_emb, transposed by movmatrix, and the result is the A operand of the product with the query heads.
//
// In a decode step the ladder's new token takes longer to encode (16 stages one after the other on a few SMs) than everything
// here up to the scores of the old ones, so those go first and the kernel waits for the new codes where it needs them.  Codes are
// read from L2 (code_word, code_byte): a line of the first-level cache that was fetched for an old token before the wait may hold the
// place of the new one, and would still hold its old bytes after it.
//
// Weights enter the histograms as integers, because shared-memory integer adds are single instructions: a weight's multiple of
// 2^-19 goes to one bin and what that leaves, in units of 2^-38, to another, which keeps all 24 bits of a weight down to 2^-15.  The sums
// are exact.
//
// Where a cluster's time goes, us after its start, one row with 4096 tokens: tables there 5.5, scores of 64 SMs 27.5, parts exchanged 31.5, scores
// exchanged 36.0, histograms 40.2, end 44.1.  Scores travel in one exchange with the blocks' maxima, and every block takes the weights of all tokens
// itself, which saves one of four exchanges (2 us); sums in two chains of products and rotary rows in whole channel pairs take 1 us off the scores.
//
// A sum of 16 words by the tensor core is no further from the exact one than fp32 adds in order: over 2^20 sums of 4, 8, 12 and 16 normal values,
// of equal spread and falling by 0.9 and 0.6 a stage, 3.5e-10 to 9.3e-9 in the 2-norm against 3.5e-10 to 1.3e-8, and the same fp16
// value in every case.
//
// us a decode step of 16 stages and 8 KV heads, against attn_rotary_kernel: one row of 6144 tokens with a window of 4096 47 / 107, 600
// tokens 39 / 103 (27 are the new token's encode), 16384 tokens 117 / 232, 8 x 2000 154 / 225, 16 x 1000 184 / 228; ladder_plan.cuh has the sizes that
// are left to that kernel.  Tables, gathers and products are 16 stages wide for fewer stages too.
//
// Semantics replaced: experiments_followup_mistral/evaluate_mistral_longbench.py:112-122 including the rotary step
// (:113-118); the query arrives rotated at its own position and scaled.

#include <math.h>

#include <atomic>

#include "common.cuh"
#include "ladder_plan.cuh"

namespace tacvq {

namespace ladder {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kDim = 128, kWords = 256, kStages = 16, kSlices = 8, kHeads = 4;
constexpr int kRowBytes = kStages * 2 * 16;           // a code's words of all stages, this block's 16 channels
constexpr int kTabBytes = kWords * kRowBytes;         // 131072
constexpr int kScoreBytes = kChunk * kHeads * 4;      // parts of the scores, then scores, then per-warp sums
constexpr int kHistBytes = 2 * 2 * kWords * kHeads * 4;  // [multiples | rest][stage j or j + 8][word][head]
constexpr int kOutBytes = kSlices * 64 * 4;           // [source block][64 of the 512 outputs]
constexpr int kSmallFloats = kSlices * kHeads + 2 * kWarps * kHeads;  // maxima of the blocks, maxima and sums of the warps
constexpr int kSmemBytes = kTabBytes + kScoreBytes + kHistBytes + kOutBytes + kSmallFloats * 4;
static_assert(kWarps * kHeads * kDim * 4 <= kScoreBytes, "per-warp sums reuse the score area");
static_assert(kSmemBytes <= 227 * 1024, "");

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&d)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix(uint32_t v) {  // 8x8 halves transposed
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(v));
    return d;
}
__device__ __forceinline__ uint4 ldg_in_place(const void *p) {  // a load that stays where it is written
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// Code bytes as they are in L2, which is where the kernel before this one has left them by the time its end was waited for.  Not
// ld.global.nc: that is for memory which nobody writes while the kernel runs.
__device__ __forceinline__ uint32_t code_word(const uint8_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t code_byte(const uint8_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// all blocks of the cluster: writes before are seen by reads after, in every block's shared memory
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_block(uint32_t addr, int rank) {  // the same place in another block's shared memory
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_cluster4(uint32_t addr, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// 2^19, of which kChunk weights add up to 2^31 at most; adding the others rounds to an integer
constexpr float kFine = 524288.0f, kRound = 8388608.0f, kRoundSigned = 12582912.0f;

// Clusters of 8 blocks share the KV heads x B x splits items (a split of a row's visible tokens) evenly, head by head; a
// cluster loads the key tables when the head changes.
__global__ void __launch_bounds__(kThreads, 1)
attn_rotary_ladder_kernel(const __half *__restrict__ q, const uint8_t *kcodes, const uint8_t *vcodes,
                          const __half *__restrict__ ktab, const __half *__restrict__ vtab, const __half *__restrict__ rope,
                          const int32_t *seq_start, const int32_t *seq_end, float *__restrict__ part,
                          int B, int Hq, int Hkv, int S, int64_t T_cap, int splits, const LadderStep step) {
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *area = smem + kTabBytes;                              // scores, then weights, then sums
    uint32_t *hist = reinterpret_cast<uint32_t *>(area + kScoreBytes);
    float *out_s = reinterpret_cast<float *>(area + kScoreBytes + kHistBytes);
    float *top_s = out_s + kSlices * 64;  // [block][head]
    float *warp_top = top_s + kSlices * kHeads, *warp_sum = warp_top + kWarps * kHeads;
    const uint32_t tab_u32 = smem_u32(smem), area_u32 = smem_u32(area);

    const int slice = blockIdx.x % kSlices, cluster = blockIdx.x / kSlices, clusters = gridDim.x / kSlices;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rep = Hq / Hkv;
    const int64_t rows = (int64_t)B * Hq;
    const int r8 = lane >> 2, kq = lane & 3;

    // this lane's place in a code's row for the gather: stage lane % 16, piece lane / 16; byte lane % 4 of a code word -> bits 8..15
    const uint32_t k_base = tab_u32 + (lane >> 4) * (kStages * 16) + (lane & 15) * 16;
    const uint32_t k_sel = 0x4404u | ((uint32_t)(lane & 3) << 4);
    const int k_lane = (lane & 15) >> 2;  // which of a token's four code words
    const int words_per_token = S >> 2;
    const int f0 = slice * 8 + 2 * kq;    // this lane's channel pair of the query (and its partner 64 on)
    int loaded = -1;
    auto load_table = [&](int h) {  // word w of stage s, pieces 8j.. and 64 + 8j.., to byte w * 512 + piece * 256 + s * 16
        if (h == loaded) return;
        for (int idx = tid; idx < kWords * kStages * 2; idx += kThreads) {
            const int s = idx & (kStages - 1), piece = (idx >> 4) & 1, word = idx >> 5;
            const uint32_t to = tab_u32 + word * kRowBytes + piece * (kStages * 16) + s * 16;
            if (s < S) cp_async16(to, ktab + (((int64_t)h * S + s) * kWords + word) * kDim + piece * 64 + slice * 8);
            else asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(to), "r"(0u) : "memory");
        }
        loaded = h;
    };

    const int per_head = B * splits;
    const int64_t items = (int64_t)Hkv * per_head;
    const int item_begin = (int)(items * cluster / clusters), item_end = (int)(items * (cluster + 1) / clusters);
    load_table(item_begin / per_head);
    // A decode step's new codes come from the kernel before this one, and nothing else that is read here; without one, all may.
    bool waited = false;
    auto wait_once = [&]() {
        if (!waited) wait_for_previous_kernel();
        waited = true;
    };
    if (step.fresh == 0) wait_once();
    for (int item = item_begin; item < item_end; ++item) {
        const int h = item / per_head, b = item % per_head / splits, split = item % splits;
        const int lo_all = step.fresh != 0 ? step.start : seq_start ? max(seq_start[b], 0) : 0;
        const int hi_all = step.fresh != 0 ? step.end : seq_end ? min(seq_end[b], (int)T_cap) : (int)T_cap;
        const int n_all = hi_all > lo_all ? hi_all - lo_all : 0;
        const int per = min((n_all + splits - 1) / splits, kChunk);  // the split count is for the range that the launcher was told
        const int first = lo_all + split * per;
        const int n = max(min(first + per, lo_all + n_all) - first, 0);
        float *dst = part + ((int64_t)split * rows + (int64_t)b * Hq + h * rep) * (kDim + 2);
        if (n == 0) {  // the same for the whole cluster: the neutral state
            if (slice == 0)
                for (int i = tid; i < rep * (kDim + 2); i += kThreads) dst[i] = i % (kDim + 2) == 0 ? -INFINITY : 0.0f;
            continue;
        }
        const uint8_t *kc = kcodes + (((int64_t)b * Hkv + h) * T_cap + first) * S, *vc = vcodes + (((int64_t)b * Hkv + h) * T_cap + first) * S;
        const __half *rp = rope + (int64_t)first * kDim + slice * 8 + 2 * kq;
        const int old_tiles = step.fresh != 0 ? max(min(step.end - step.fresh - first, n), 0) >> 4 : (n + 15) >> 4;  // without a new token

        load_table(h);
        // ---- pass K: this block's part of the scores ------------------------------------------------------------------
        {
            uint32_t q0 = 0u, q1 = 0u;  // B operand: column r8 = head, k = this lane's channel pair, lower and upper
            if (r8 < rep) {
                const uint32_t *src = reinterpret_cast<const uint32_t *>(q + ((int64_t)b * Hq + h * rep + r8) * kDim + f0);
                q0 = __ldg(src);
                q1 = __ldg(src + 32);
            }
            const int tiles = (n + 15) >> 4;
            uint32_t cn[2], rn[2][2];  // code words of tokens 0-7 and 8-15 (lane = 4 x token + word); cosines and sines of token r8, channels 2kq, 2kq + 1
            auto fetch = [&](int tile) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int t = min(tile * 16 + u * 8 + r8, n - 1);
                    cn[u] = kq < words_per_token ? code_word(kc + (int64_t)t * S + 4 * kq) : 0u;
                    const uint32_t *turn = reinterpret_cast<const uint32_t *>(rp + (int64_t)t * kDim);
                    rn[u][0] = __ldg(turn);
                    rn[u][1] = __ldg(turn + 32);
                }
            };
            for (int i = tid; i < kHistBytes / 4; i += kThreads) hist[i] = 0u;
            if (old_tiles < tiles && warp >= old_tiles) wait_once();
            fetch(min(warp, tiles - 1));
            cp_async_wait_all();
            __syncthreads();  // tables; the sums of the item before have been read
            for (int tile = warp; tile < tiles; tile += kWarps) {
                const uint32_t code[2] = {cn[0], cn[1]};
                const uint32_t turn[2][2] = {{rn[0][0], rn[0][1]}, {rn[1][0], rn[1][1]}};
                if (tile + kWarps < tiles) {
                    if (tile + kWarps >= old_tiles) wait_once();
                    fetch(tile + kWarps);
                }
                uint32_t a[4];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    // all gathers before the first product: in turn, each would wait for the one before
                    uint32_t m[8][4];  // stages 0-7 and 8-15 of the lower channels, then of the upper ones
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const uint32_t at = prmt(__shfl_sync(0xffffffffu, code[u], t * 4 + k_lane), 0u, k_sel);
                        ldmatrix_x4_trans(m[t], k_base + at + at);
                    }
                    // channel r8 and its partner, tokens 2kq and 2kq + 1 of these eight; in two chains, which hold zeros for each other's tokens
                    float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f}, odd[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const uint32_t one = r8 == t ? 0x3c003c00u : 0u;
                        if (t & 1) mma16816(odd, m[t][0], m[t][2], m[t][1], m[t][3], one, one);
                        else mma16816(sum, m[t][0], m[t][2], m[t][1], m[t][3], one, one);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[i] += odd[i];
                    // The zeros in the other tokens' columns do not hide a word that is not finite (0 x inf): then every token's words
                    // are added without the others'.
                    if (__any_sync(0xffffffffu, !(fabsf((sum[0] + sum[1]) + (sum[2] + sum[3])) < INFINITY))) {
#pragma unroll 1
                        for (int j = 0; j < 4; ++j) {  // channel r8 or its partner of token 2kq + j % 2
                            float alone = 0.0f;
#pragma unroll 1
                            for (int st = 0; st < S; ++st) {
                                const uint32_t word = __shfl_sync(0xffffffffu, code[u], (2 * kq + (j & 1)) * 4 + (st >> 2)) >> (8 * (st & 3)) & 255u;
                                alone += __half2float(*reinterpret_cast<const __half *>(smem + word * kRowBytes + (j >> 1) * (kStages * 16) + st * 16 + r8 * 2));
                            }
                            sum[0] = j == 0 ? alone : sum[0], sum[1] = j == 1 ? alone : sum[1];
                            sum[2] = j == 2 ? alone : sum[2], sum[3] = j == 3 ? alone : sum[3];
                        }
                    }
                    // round, turn to row = token, k = channel; rotate (k cos + rotate_half(k) sin, products and sum in fp16)
                    const __half2 low = __floats2half2_rn(sum[0], sum[1]), high = __floats2half2_rn(sum[2], sum[3]);
                    const uint32_t lt = movmatrix(*reinterpret_cast<const uint32_t *>(&low)), ht = movmatrix(*reinterpret_cast<const uint32_t *>(&high));
                    const __half2 kl = *reinterpret_cast<const __half2 *>(&lt), kh = *reinterpret_cast<const __half2 *>(&ht);
                    const __half2 cosv = *reinterpret_cast<const __half2 *>(&turn[u][0]), sinv = *reinterpret_cast<const __half2 *>(&turn[u][1]);
                    const __half2 tl = __hadd2(__hmul2(kl, cosv), __hmul2(__hneg2(kh), sinv));
                    const __half2 th = __hadd2(__hmul2(kh, cosv), __hmul2(kl, sinv));
                    a[u] = *reinterpret_cast<const uint32_t *>(&tl);
                    a[2 + u] = *reinterpret_cast<const uint32_t *>(&th);
                }
                float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma16816(d, a[0], a[1], a[2], a[3], q0, q1);
                if (kq < 2) {  // columns 0..3: a token's four heads
                    float2 *score = reinterpret_cast<float2 *>(area) + (tile * 16 + r8) * 2 + kq;
                    score[0] = make_float2(d[0], d[1]);
                    score[16] = make_float2(d[2], d[3]);
                }
            }
        }
        // what the value side reads is on its way while the scores are exchanged: the codes of stages `slice` and `slice` + 8, and
        // these stages' words (a thread has 8 channels of every 32nd one)
        if (old_tiles < (n + 15) >> 4) wait_once();
        const int stages = slice + 8 < S ? 2 : slice < S ? 1 : 0, piece = tid & 15;
        uint32_t v_codes[kChunk / kThreads];
#pragma unroll
        for (int i = 0; i < kChunk / kThreads; ++i) {
            const int t = tid + i * kThreads;
            v_codes[i] = 0u;
            if (t < n && stages > 0) {
                v_codes[i] = code_byte(vc + (int64_t)t * S + slice);
                if (stages > 1) v_codes[i] |= code_byte(vc + (int64_t)t * S + slice + 8) << 8;
            }
        }
        uint4 v_words[2 * kWords / 32];
#pragma unroll
        for (int k = 0; k < 2 * kWords / 32; ++k)
            if (k < stages * (kWords / 32))
                v_words[k] = ldg_in_place(vtab + (((int64_t)h * S + slice + 8 * (k >> 3)) * kWords + (k & 7) * 32 + (tid >> 4)) * kDim + piece * 8);
        cluster_barrier();

        // ---- block j adds up the parts of its share of the tokens; scores and the share's maxima go to every block --------------
        {
            const int share = (n + kSlices - 1) / kSlices;  // at most kThreads
            const int t = slice * share + tid;
            float sc[kHeads] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            if (tid < share && t < n) {
                float4 v[kSlices];
#pragma unroll
                for (int k = 0; k < kSlices; ++k) v[k] = ld_cluster4(in_block(area_u32 + t * 16, k));
                float4 s = v[0];
#pragma unroll
                for (int k = 1; k < kSlices; ++k) s.x += v[k].x, s.y += v[k].y, s.z += v[k].z, s.w += v[k].w;
                sc[0] = s.x, sc[1] = s.y, sc[2] = s.z, sc[3] = s.w;
#pragma unroll
                for (int k = 0; k < kSlices; ++k) st_cluster4(in_block(area_u32 + t * 16, k), s);
            }
#pragma unroll
            for (int r = 0; r < kHeads; ++r) {
                float v = sc[r];
#pragma unroll
                for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
                if (lane == 0) warp_top[warp * kHeads + r] = v;
            }
            __syncthreads();
            if (tid < kSlices * kHeads) {  // this block's maximum of head tid % 4, to block tid / 4
                float v = warp_top[tid & 3];
                for (int w = 1; w < kWarps; ++w) v = fmaxf(v, warp_top[w * kHeads + (tid & 3)]);
                st_cluster(in_block(smem_u32(top_s + slice * kHeads + (tid & 3)), tid >> 2), v);
            }
            cluster_barrier();
        }

        // ---- weights by code, stages `slice` and `slice` + 8; every block takes the weights of all tokens, relative to the largest score of all --------
        float ref[kHeads], weight_sum[kHeads];
#pragma unroll
        for (int r = 0; r < kHeads; ++r) {
            float top = top_s[r];
#pragma unroll
            for (int k = 1; k < kSlices; ++k) top = fmaxf(top, top_s[k * kHeads + r]);
            ref[r] = top == -INFINITY ? 0.0f : top;  // a score of -inf weighs nothing, also where there is no other; NaN stays NaN
            weight_sum[r] = 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kChunk / kThreads; ++i) {
            const int t = tid + i * kThreads;
            if (t >= n) break;
            const float4 s4 = *reinterpret_cast<const float4 *>(area + t * 16);
            float p[kHeads] = {__expf(s4.x - ref[0]), __expf(s4.y - ref[1]), __expf(s4.z - ref[2]), __expf(s4.w - ref[3])};
#pragma unroll
            for (int r = 0; r < kHeads; ++r) weight_sum[r] += p[r];
            // lane l takes the heads in the order l, l + 1, ..: the 32 adds of an instruction spread over all banks
            if (lane & 1) {
                const float x = p[0];
                p[0] = p[1], p[1] = p[2], p[2] = p[3], p[3] = x;
            }
            if (lane & 2) {
                float x = p[0];
                p[0] = p[2], p[2] = x;
                x = p[1];
                p[1] = p[3], p[3] = x;
            }
            uint32_t w[kHeads], rest[kHeads];
#pragma unroll
            for (int r = 0; r < kHeads; ++r) {  // a NaN leaves some integer here; the sum of the weights spoils the result
                const float near = fmaf(p[r], kFine, kRound);
                w[r] = __float_as_uint(near) & 0x7fffffu;
                rest[r] = __float_as_uint(fmaf(fmaf(p[r], kFine, kRound - near), kFine, kRoundSigned)) - __float_as_uint(kRoundSigned);
            }
            for (int st = 0; st < stages; ++st) {
                uint32_t *bin = hist + (st * kWords + (v_codes[i] >> (8 * st) & 255u)) * kHeads;
#pragma unroll
                for (int r = 0; r < kHeads; ++r) {
                    atomicAdd(bin + ((r + lane) & 3), w[r]);
                    atomicAdd(bin + 2 * kWords * kHeads + ((r + lane) & 3), rest[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kHeads; ++r) {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) weight_sum[r] += __shfl_xor_sync(0xffffffffu, weight_sum[r], off);
            if (lane == 0) warp_sum[warp * kHeads + r] = weight_sum[r];
        }
        __syncthreads();

        // ---- histograms x words, all heads -----------------------------------------
        {
            float acc[kHeads][8];
#pragma unroll
            for (int r = 0; r < kHeads; ++r)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[r][i] = 0.0f;
#pragma unroll
            for (int k = 0; k < 2 * kWords / 32; ++k) {
                if (k >= stages * (kWords / 32)) break;
                const int st = k >> 3, word = (k & 7) * 32 + (tid >> 4);
                const uint4 w4 = *reinterpret_cast<const uint4 *>(hist + (st * kWords + word) * kHeads);
                const int4 s4 = *reinterpret_cast<const int4 *>(hist + ((2 + st) * kWords + word) * kHeads);
                if ((w4.x | w4.y | w4.z | w4.w | s4.x | s4.y | s4.z | s4.w) == 0u) continue;  // a word that nobody refers to may hold anything
                constexpr float kUnit = 1.0f / kFine, kRestUnit = 1.0f / (kFine * kFine);
                const float w[kHeads] = {fmaf((float)s4.x, kRestUnit, (float)w4.x * kUnit), fmaf((float)s4.y, kRestUnit, (float)w4.y * kUnit),
                                         fmaf((float)s4.z, kRestUnit, (float)w4.z * kUnit), fmaf((float)s4.w, kRestUnit, (float)w4.w * kUnit)};
                const __half2 *hp = reinterpret_cast<const __half2 *>(&v_words[k]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __half22float2(hp[i]);
#pragma unroll
                    for (int r = 0; r < kHeads; ++r) {
                        acc[r][2 * i] = fmaf(w[r], f.x, acc[r][2 * i]);
                        acc[r][2 * i + 1] = fmaf(w[r], f.y, acc[r][2 * i + 1]);
                    }
                }
            }
            float *sums = reinterpret_cast<float *>(area);  // [warp][head][channel]; every thread is done with the weights
#pragma unroll
            for (int r = 0; r < kHeads; ++r) {
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], 16);
                if (lane < 16) {
                    float4 *to = reinterpret_cast<float4 *>(sums + (warp * kHeads + r) * kDim + piece * 8);
                    to[0] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
                    to[1] = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
                }
            }
            __syncthreads();
            float v = 0.0f;  // output tid = head x 128 + channel
            for (int w = 0; w < kWarps; ++w) v += sums[w * (kHeads * kDim) + tid];
            st_cluster(in_block(smem_u32(out_s + slice * 64 + (tid & 63)), tid >> 6), v);
        }
        cluster_barrier();
        if (tid < 64) {  // outputs slice * 64 .. + 63
            const int o = slice * 64 + tid, r = o >> 7, channel = o & 127;
            float a = 0.0f, l = 0.0f, top = -INFINITY;
            for (int k = 0; k < kSlices; ++k) {
                a += out_s[k * 64 + tid];
                top = fmaxf(top, top_s[k * kHeads + r]);
            }
            for (int w = 0; w < kWarps; ++w) l += warp_sum[w * kHeads + r];
            if (l != l) a = l;
            // Scores of -inf alone: not the neutral state (a sum of 0).  The merge gives it no weight beside others and makes NaN of it alone.
            if (top == -INFINITY && l == 0.0f) l = 1.0f;
            if (r < rep) {
                dst[r * (kDim + 2) + 2 + channel] = a;
                if (channel == 0) {
                    dst[r * (kDim + 2)] = top;
                    dst[r * (kDim + 2) + 1] = l;
                }
            }
        }
    }
    cp_async_wait_all();  // no copy outlives the block
    wait_once();          // who waits for this grid may rely on the kernel before it too
}

}  // namespace ladder

bool attn_rotary_ladder_supported(int Hq, int Hkv, int D, int G, int S, int K) {
    const int rep = Hkv > 0 ? Hq / Hkv : 0;
    return D == 128 && G == 1 && K == 256 && S >= 4 && S <= 16 && S % 4 == 0 && (rep == 1 || rep == 2 || rep == 4);
}

// Partial states [split][B*Hq][2 + D] for attn_combine_kernel; *splits is how many (0: nothing was launched, the call is
// for the general kernel).
int attn_rotary_ladder_dispatch(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab, const __half *vtab,
                                const __half *rope, const int32_t *seq_start, const int32_t *seq_end, float *part, int B, int Hq,
                                int Hkv, int S, int64_t T_cap, int64_t visible, int sms, const LadderStep &step, int *splits, cudaStream_t stream) {
    using namespace ladder;
    *splits = 0;
    cudaError_t e = cudaFuncSetAttribute(attn_rotary_ladder_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSlices);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kSlices;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // clusters that fit the chip beside one another: 15 on a B200, whose GPCs differ in size
    static std::atomic<int> cached[64];
    int dev = 0, most = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) most = cached[dev].load(std::memory_order_relaxed);
    if (most == 0) {
        e = cudaOccupancyMaxActiveClusters(&most, attn_rotary_ladder_kernel, &cfg);
        if (e != cudaSuccess) return (int)e;
        if (most < 1) return TACVQ_OK;
        if (dev >= 0 && dev < 64) cached[dev].store(most, std::memory_order_relaxed);
    }
    const Plan dealt = plan(B, Hq, Hkv, S, T_cap, visible, sms, most);
    if (dealt.splits == 0) return TACVQ_OK;
    *splits = dealt.splits;
    cfg.gridDim = dim3((unsigned)(kSlices * dealt.clusters));
    cfg.numAttrs = step.fresh != 0 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, attn_rotary_ladder_kernel, q, kcodes, vcodes, ktab, vtab, rope, seq_start, seq_end, part, B, Hq, Hkv, S,
                           T_cap, *splits, step);
    return e == cudaSuccess ? launch_status() : (int)e;
}

}  // namespace tacvq
