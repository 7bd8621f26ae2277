// Attention over codes of PRE-rotary keys for the benchmark geometry (head_dim 128 = 16 groups x 8,
// two residual stages, 256 words), with both contractions on the tensor cores (mma.sync).
//
// A block serves one KV head, up to R batch rows and one range of positions, at most 6144 tokens in all, in two passes:
//   pass K   key tables (128 KB) in shared memory.  Four lanes share a token; lane j of them rebuilds groups j, j+4, j+8
//            and j+12 as fp16 (packed add of the two stages = the reference's fp16 window), which are exactly the
//            rotary partners c, c+64, rotates them with the cos/sin of the token's position, and the warp multiplies
//            8 tokens x 128 channels with the 4 query heads by four m16n8k16 products: rows 0-7 of the A
//            operand carry the lower 64 channels of the 8 tokens, rows 8-15 the upper 64, and the 8 columns
//            of the B operand are (4 heads) x (lower | upper query channels); the two halves of a score
//            meet through one shuffle.  fp32 scores go to shared memory.
//   softmax  maximum of every row and head, p = exp(score - max) as fp16 [row][head][token] over the score area.
//   pass V   value tables loaded over the key tables; P.V with
//            m16n8k8 products exactly as in the kernel without rotary step (attn_gsrq.cu): rows =
//            channels, columns = 4 heads x 2 visiting orders, contraction = tokens; value codes land by
//            cp.async and are handed out by ldmatrix.trans.
// All rows of a batch stand at the same positions, so the rows of a block share their cos/sin (256 bytes a position, eight
// times a token's codes): a warp keeps those of its 8 positions in registers and goes through the block's rows.  A chunk is as
// long as the score area allows, because each one copies both tables (2 x 128 KB).
//
// What bounds it: wavefronts of the L1/shared pipe and the latency between them at 16 warps.  A block of 4856 tokens, in clocks: tables,
// softmax and sums 20 k (29 k when scattered 16-byte cp.async filled the tables), pass K 50 k (10.3 a token, 6.2 of them wavefronts), pass V 25 k (5.2, of
// which 4.4 are look-ups).  us a decode step with 8 KV heads, 8 rows x 32768: 163 (180 with those copies).  Against a row and at most 4096 tokens a
// block, before: 8 rows x 32768 183 / 205, a window of 4096 of them 45 / 91, 2 x 65536 115 / 148.
//
// Every shared-memory gather is conflict-free for arbitrary codes: a code's 32 codewords lie in one
// 512-byte row, the position of (stage, group) inside the row decides the bank, and the lanes that are
// served together read different positions (the two tokens of a quarter warp take the stages in opposite
// order in pass K; the four token pairs visit (stage, group) in four orders in pass V).
//
// Semantics replaced: experiments_followup_mistral/evaluate_mistral_longbench.py:112-122 including the
// rotary step (:113-118).  Differences from that dense path, inside the 2e-3 tolerance: the rotation is
// a packed multiply and a fused multiply-add per channel pair (the reference rounds both products), and
// probabilities enter the P.V product as fp16.

#include "table_rows.cuh"

namespace tacvq {

namespace rotmma {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kDim = 128, kWords = 256, kRowBytes = 512;   // a code's 32 codewords
constexpr int kChunk = 6144;                               // tokens per block at most, over all its rows
constexpr int kTabBytes = kWords * kRowBytes;              // 131072
constexpr int kScoreBytes = kChunk * 4 * 4;                // fp32 [token][4 heads]
template <int R>
constexpr int kPositions = kChunk / R;                     // positions per block at most
template <int R>
constexpr int kProbStride = kPositions<R> * 2 + 16;        // bytes per row and head of the fp16 probabilities
constexpr int kVStagePerWarp = 1024;                       // one 32-token tile of value codes
constexpr int kRedFloats = kWarps * 4;
constexpr int kSmemBytes = kTabBytes + kScoreBytes + 2 * kRedFloats * 4 + 4 * 16;
static_assert(16 * kProbStride<4> + kWarps * kVStagePerWarp <= kScoreBytes, "probabilities and code staging reuse the score area");
static_assert(kSmemBytes <= 227 * 1024, "");
static_assert(kWarps * 32 * 32 * 4 <= kTabBytes, "merge scratch reuses the table area");

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&d)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(addr));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

template <int R>
__global__ void __launch_bounds__(kThreads, 1)
attn_rotary_mma_kernel(const __half *__restrict__ q, const uint8_t *kcodes, const uint8_t *vcodes,
                       const __half *__restrict__ ktab, const __half *__restrict__ vtab, const __half *__restrict__ rope,
                       const int32_t *seq_start, const int32_t *seq_end, float *__restrict__ part,
                       int B, int Hq, int Hkv, int64_t T_cap, int splits) {
    constexpr int kPos = kPositions<R>, kStride = kProbStride<R>;
    constexpr int kRowWarps = kWarps / R, kRowThreads = kThreads / R;  // softmax and pass V: warps of one batch row
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *tab_s = smem_raw;
    float *score_s = reinterpret_cast<float *>(smem_raw + kTabBytes);  // [R][kPos][4 heads]
    float *red_s = reinterpret_cast<float *>(smem_raw + kTabBytes + kScoreBytes);  // [2][warps][4]
    int4 *limit_s = reinterpret_cast<int4 *>(red_s + 2 * kRedFloats);  // per row: first and last + 1 visible token, both ends for code reads
    const uint32_t tab_u32 = smem_u32(tab_s), score_u32 = smem_u32(score_s);

    const int split = blockIdx.x, h = blockIdx.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rep = Hq / Hkv;  // 1, 2 or 4 query heads per KV head
    const int b0 = (int)((int64_t)blockIdx.z * B / gridDim.z), n_rows = (int)((int64_t)(blockIdx.z + 1) * B / gridDim.z) - b0;

    // A decode step's new codes and ranges come from the kernel before this one; the tables and the query do not.
    copy_table_rows<kWarps>(tab_u32, ktab + (size_t)h * 2 * 16 * kWords * 8, warp, lane);
    wait_for_previous_kernel();
    // positions that some row of the block sees, and this split's share of them
    int lo_all = 0x7fffffff, hi_all = 0;
    for (int r = 0; r < n_rows; ++r) {
        const int lo = seq_start ? max(seq_start[b0 + r], 0) : 0;
        const int hi = seq_end ? min(seq_end[b0 + r], (int)T_cap) : (int)T_cap;
        if (hi > lo) lo_all = min(lo_all, lo), hi_all = max(hi_all, hi);
    }
    const int n_all = hi_all > lo_all ? hi_all - lo_all : 0;
    const int per = min((n_all + splits - 1) / splits, kPos);  // the split count is for the range that the launcher was told
    const int chunk = n_all > 0 ? lo_all + split * per : 0;
    const int n = n_all > 0 ? max(min(chunk + per, hi_all) - chunk, 0) : 0;
    const int64_t rows = (int64_t)B * Hq;

    if (n <= 0) {  // an empty range contributes the neutral state
        for (int idx = tid; idx < n_rows * rep * (kDim + 2); idx += kThreads) {
            const int r = idx / (kDim + 2), col = idx % (kDim + 2);
            part[((int64_t)split * rows + (int64_t)(b0 + r / rep) * Hq + h * rep + r % rep) * (kDim + 2) + col] = col == 0 ? -INFINITY : 0.0f;
        }
        return;
    }
    const size_t row_step = (size_t)Hkv * (size_t)T_cap * 32;  // code bytes from one batch row to the next
    const size_t code_at = (((size_t)b0 * Hkv + h) * (size_t)T_cap + chunk) * 32;

    if (tid < n_rows) {
        const int lo = seq_start ? max(seq_start[b0 + tid], 0) : 0;
        const int hi = seq_end ? min(seq_end[b0 + tid], (int)T_cap) : (int)T_cap;
        const int first = max(lo - chunk, 0), end = min(hi - chunk, n);
        // a row without a token here reads the codes of some position of the chunk and drops them
        limit_s[tid] = first < end ? make_int4(first, end, first, end - 1) : make_int4(n, 0, 0, n - 1);
    }

    // ---- pass K ------------------------------------------------------------------------------------
    const int g8 = lane >> 2, j4 = lane & 3;
    {
        // B operand: column n = g8 is (head n & 3, channel half n >> 2); this lane's 16 channels of it, for every row
        uint32_t qf[R][8];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int head = g8 & 3, half = g8 >> 2;
            uint4 lo4 = make_uint4(0u, 0u, 0u, 0u), hi4 = lo4;
            if (head < rep && r < n_rows) {
                const uint4 *src = reinterpret_cast<const uint4 *>(q + ((size_t)(b0 + r) * Hq + h * rep + head) * kDim + half * 64 + 8 * j4);
                lo4 = __ldg(src);
                hi4 = __ldg(src + 4);
            }
            qf[r][0] = lo4.x, qf[r][1] = lo4.y, qf[r][2] = lo4.z, qf[r][3] = lo4.w;
            qf[r][4] = hi4.x, qf[r][5] = hi4.y, qf[r][6] = hi4.z, qf[r][7] = hi4.w;
        }
        // step (ci, sf) gathers group j + 4 ci of stage sf ^ (token parity), which lies 128 ci bytes behind that of ci = 0
        const int first_stage = g8 & 1;
        const uint32_t k_off[2] = {tab_u32 + word_place(first_stage, j4) * 16, tab_u32 + word_place(first_stage ^ 1, j4) * 16};
        const uint32_t k_sel = 0x4404u | ((uint32_t)j4 << 4);  // byte j of a word -> bits 8..15
        // a token's 32 code bytes: stage s at bytes 16s..16s+15; group j + 4 ci is byte j of word ci
        const uint8_t *kc = kcodes + code_at + first_stage * 16;
        const int other_stage = 16 - 32 * first_stage;
        const ptrdiff_t v_from_k = reinterpret_cast<intptr_t>(vcodes) - reinterpret_cast<intptr_t>(kcodes);
        const __half *rp = rope + (size_t)chunk * kDim + 8 * j4;

        const int trips = (n + 8 * kWarps - 1) / (8 * kWarps);
        uint4 cn[2], rn[4];
        int4 limit;
        auto fetch_codes = [&](int r, int local) {
            limit = limit_s[r];
            const int t = min(max(local, limit.z), limit.w);
            const uint8_t *src = kc + (size_t)r * row_step + (size_t)t * 32;
            cn[0] = *reinterpret_cast<const uint4 *>(src);
            cn[1] = *reinterpret_cast<const uint4 *>(src + other_stage);
            // to L2: the key codes two trips on, and the value codes of this one for pass V
            const int ahead = max(min(local + 16 * kWarps, limit.w), 0);
            if (j4 < 2) prefetch_l2(j4 == 0 ? kc + (size_t)r * row_step + (size_t)ahead * 32 : src + v_from_k);
        };
        auto fetch_rope = [&](int local) {
            const uint4 *cs = reinterpret_cast<const uint4 *>(rp + (size_t)min(local, n - 1) * kDim);
            rn[0] = __ldg(cs), rn[1] = __ldg(cs + 4);          // cosines of frequencies 8j .. and 32 + 8j ..
            rn[2] = __ldg(cs + 8), rn[3] = __ldg(cs + 12);     // sines
        };
        fetch_rope(warp * 8 + g8);
        __syncthreads();
        fetch_codes(0, warp * 8 + g8);
#pragma unroll 1
        for (int trip = 0; trip < trips; ++trip) {
            const int local = (trip * kWarps + warp) * 8 + g8;
            const uint32_t cosv[8] = {rn[0].x, rn[0].y, rn[0].z, rn[0].w, rn[1].x, rn[1].y, rn[1].z, rn[1].w};
            const uint32_t sinv[8] = {rn[2].x, rn[2].y, rn[2].z, rn[2].w, rn[3].x, rn[3].y, rn[3].z, rn[3].w};
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (r >= n_rows) break;
                const uint32_t first[4] = {cn[0].x, cn[0].y, cn[0].z, cn[0].w}, second[4] = {cn[1].x, cn[1].y, cn[1].z, cn[1].w};
                const bool seen = local >= limit.x && local < limit.y;
                if (r + 1 < n_rows && r + 1 < R) fetch_codes(r + 1, local);
                else if (trip + 1 < trips) fetch_codes(0, local + 8 * kWarps);
                float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (__any_sync(0xffffffffu, seen)) {
                    // first stage of this lane's order, then the other; the packed fp16 sum does not depend on the order
                    uint32_t k[4][4];
#pragma unroll
                    for (int ci = 0; ci < 4; ++ci) {
                        const uint32_t at0 = prmt(first[ci], 0u, k_sel), at1 = prmt(second[ci], 0u, k_sel);
                        const uint4 a = lds128(k_off[0] + at0 + at0 + ci * 128), b = lds128(k_off[1] + at1 + at1 + ci * 128);
                        k[ci][0] = hadd2(a.x, b.x), k[ci][1] = hadd2(a.y, b.y), k[ci][2] = hadd2(a.z, b.z), k[ci][3] = hadd2(a.w, b.w);
                    }
                    // k'_c = k_c cos - k_{c+64} sin ;  k'_{c+64} = k_{c+64} cos + k_c sin
                    uint32_t rl[8], rh[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t lo = k[i >> 2][i & 3], hi = k[2 + (i >> 2)][i & 3];
                        rl[i] = hfma2(hi ^ 0x80008000u, sinv[i], hmul2(lo, cosv[i]));
                        rh[i] = hfma2(lo, sinv[i], hmul2(hi, cosv[i]));
                    }
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        mma16816(d, rl[2 * ks], rh[2 * ks], rl[2 * ks + 1], rh[2 * ks + 1], qf[r][2 * ks], qf[r][2 * ks + 1]);
                }
                // rows 0-7 x columns 0-3 hold the lower halves of the scores (lanes j < 2), rows 8-15 x columns 4-7
                // the upper halves (lanes j >= 2)
                const float up0 = __shfl_xor_sync(0xffffffffu, d[2], 2), up1 = __shfl_xor_sync(0xffffffffu, d[3], 2);
                if (j4 < 2 && local < n)
                    *reinterpret_cast<float2 *>(score_s + ((size_t)r * kPos + local) * 4 + 2 * j4) =
                        seen ? make_float2(d[0] + up0, d[1] + up1) : make_float2(-INFINITY, -INFINITY);
            }
            if (trip + 1 < trips) fetch_rope(local + 8 * kWarps);
        }
    }
    __syncthreads();

    // ---- value tables; softmax over the block's tokens, kRowWarps warps a batch row ---
    copy_table_rows<kWarps>(tab_u32, vtab + (size_t)h * 2 * 16 * kWords * 8, warp, lane);
    const int n_pad = (n + 31) & ~31;
    const int row = warp / kRowWarps, row_warp = warp % kRowWarps;
    const bool row_live = row < n_rows;
    float m[4], l[4];
    {
        float4 sv[kPos / kRowThreads];
        float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int k = 0; k < kPos / kRowThreads; ++k) {
            const int i = row_warp * 32 + lane + k * kRowThreads;
            if (i < n && row_live) {
                sv[k] = *reinterpret_cast<const float4 *>(score_s + ((size_t)row * kPos + i) * 4);
                top[0] = fmaxf(top[0], sv[k].x), top[1] = fmaxf(top[1], sv[k].y), top[2] = fmaxf(top[2], sv[k].z), top[3] = fmaxf(top[3], sv[k].w);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], off));
            if (lane == 0) red_s[warp * 4 + r] = top[r];
        }
        __syncthreads();  // also: every thread holds its scores, the score area may be overwritten
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            m[r] = -INFINITY;
            for (int w = 0; w < kRowWarps; ++w) m[r] = fmaxf(m[r], red_s[(row * kRowWarps + w) * 4 + r]);
            l[r] = 0.0f;
        }
        __half *prob = reinterpret_cast<__half *>(score_s) + (size_t)row * 4 * (kStride / 2);
#pragma unroll
        for (int k = 0; k < kPos / kRowThreads; ++k) {
            const int i = row_warp * 32 + lane + k * kRowThreads;
            if (i < n_pad && row_live) {
                float p[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (i < n) {  // a token that the row does not see scored -inf: weight 0 as long as the row has a maximum
                    p[0] = __expf(sv[k].x - m[0]), p[1] = __expf(sv[k].y - m[1]), p[2] = __expf(sv[k].z - m[2]), p[3] = __expf(sv[k].w - m[3]);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    l[r] += p[r];
                    prob[(size_t)r * (kStride / 2) + i] = __float2half_rn(p[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], off);
            if (lane == 0) red_s[kRedFloats + warp * 4 + r] = l[r];
        }
    }

    // ---- pass V ------------------------------------------------------------------------------------
    const int r8 = lane >> 2, kq = lane & 3;
    uint32_t v_off[2][2], v_sel[2][2];
#pragma unroll
    for (int sp = 0; sp < 2; ++sp)
#pragma unroll
        for (int gsel = 0; gsel < 2; ++gsel) {
            const int s = sp ^ (kq & 1), gh = gsel ^ (kq >> 1);
            v_off[sp][gsel] = tab_u32 + word_place(s, 2 * r8 + gh) * 16;
        }
#pragma unroll
    for (int tk = 0; tk < 2; ++tk)
#pragma unroll
        for (int gsel = 0; gsel < 2; ++gsel) v_sel[tk][gsel] = 0x4404u | ((uint32_t)(tk * 2 + (gsel ^ (kq >> 1))) << 4);  // code byte -> bits 8..15
    const int b_head = r8 & 3;                       // B-operand column n = r8: head n & 3, visiting order n >> 2
    const bool b_valid = (r8 >> 2) == (kq >> 1);
    const uint32_t vstage_u32 = score_u32 + R * 4 * kStride + warp * kVStagePerWarp;
    // landing place of a token's two 16-byte stage halves: odd token pairs swap the halves (stage
    // order of the value look-ups), tokens 4..7 of every eight swap them once more so that the eight rows of an
    // ldmatrix tile cover all banks (a request takes sixteen tokens, two lanes a token: whole sectors)
    const uint32_t v_land = vstage_u32 + (lane >> 1) * 32 + ((((lane >> 2) ^ (lane >> 3) ^ lane) & 1) * 16);
    const uint32_t v_row0 = vstage_u32 + (8 * (lane >> 4) + (lane & 7)) * 32 + ((((lane >> 3) & 1) ^ ((lane >> 2) & 1)) * 16);
    const uint32_t p_read = score_u32 + (uint32_t)((row * 4 + b_head) * kStride + kq * 4);
    // a row that sees nothing of this chunk has no maximum and no weights
    const int4 own = row_live ? limit_s[row] : make_int4(0, 0, 0, 0);
    const int tiles = own.x < own.y ? n_pad >> 5 : 0;
    const uint8_t *vc = vcodes + code_at + (size_t)(row_live ? row : 0) * row_step;
    auto land_codes = [&](int tile) {
#pragma unroll
        for (int u = 0; u < 2; ++u)
            cp_async16(v_land + u * 512, vc + (size_t)min(max(tile * 32 + u * 16 + (lane >> 1), own.z), own.w) * 32 + (lane & 1) * 16);
    };

    float acc[8][4];
#pragma unroll
    for (int mm = 0; mm < 8; ++mm) acc[mm][0] = acc[mm][1] = acc[mm][2] = acc[mm][3] = 0.0f;
    __syncthreads();  // probabilities written; nobody reads scores any more
    if (row_warp < tiles) land_codes(row_warp);
    cp_async_wait_all();  // the first tile of codes
    __syncthreads();
    for (int tile = row_warp; tile < tiles; tile += kRowWarps) {
        uint32_t vm_lo[4], vm_hi[4];  // tokens 0..15 and 16..31 of the tile
        ldmatrix_x4_trans(vm_lo, v_row0);
        ldmatrix_x4_trans(vm_hi, v_row0 + 512);
        __syncwarp();
        if (tile + kRowWarps < tiles) land_codes(tile + kRowWarps);
        const uint32_t p_tile = p_read + (uint32_t)tile * 64;
#pragma unroll 1
        for (int a = 0; a < 2; ++a) {
            const uint32_t vm[4] = {a ? vm_hi[0] : vm_lo[0], a ? vm_hi[1] : vm_lo[1], a ? vm_hi[2] : vm_lo[2], a ? vm_hi[3] : vm_lo[3]};
#pragma unroll
            for (int ksl = 0; ksl < 2; ++ksl) {
                uint32_t b0 = 0u;
                if (b_valid) b0 = lds32(p_tile + (uint32_t)(a * 2 + ksl) * 16);
                uint4 sa[2], sb[2];
#pragma unroll
                for (int tk = 0; tk < 2; ++tk) {
                    uint4 gth[2][2];
#pragma unroll
                    for (int sp = 0; sp < 2; ++sp)
#pragma unroll
                        for (int gsel = 0; gsel < 2; ++gsel) {
                            const uint32_t code256 = prmt(vm[ksl * 2 + sp], 0u, v_sel[tk][gsel]);
                            gth[sp][gsel] = lds128(v_off[sp][gsel] + code256 + code256);
                        }
                    sa[tk] = make_uint4(hadd2(gth[0][0].x, gth[1][0].x), hadd2(gth[0][0].y, gth[1][0].y),
                                        hadd2(gth[0][0].z, gth[1][0].z), hadd2(gth[0][0].w, gth[1][0].w));
                    sb[tk] = make_uint4(hadd2(gth[0][1].x, gth[1][1].x), hadd2(gth[0][1].y, gth[1][1].y),
                                        hadd2(gth[0][1].z, gth[1][1].z), hadd2(gth[0][1].w, gth[1][1].w));
                }
                const uint32_t a0[4] = {sa[0].x, sa[0].y, sa[0].z, sa[0].w}, a1[4] = {sa[1].x, sa[1].y, sa[1].z, sa[1].w};
                const uint32_t c0[4] = {sb[0].x, sb[0].y, sb[0].z, sb[0].w}, c1[4] = {sb[1].x, sb[1].y, sb[1].z, sb[1].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    mma1688(acc[2 * i], prmt(a0[i], a1[i], 0x5410u), prmt(c0[i], c1[i], 0x5410u), b0);
                    mma1688(acc[2 * i + 1], prmt(a0[i], a1[i], 0x7632u), prmt(c0[i], c1[i], 0x7632u), b0);
                }
            }
        }
        cp_async_wait_all();
        __syncwarp();  // the next tile's codes have landed and are visible to the whole warp
    }

    // ---- sum the warps, write this split's partial state ------------------------------------------------
    __syncthreads();  // the value tables are no longer read
    float *wacc = reinterpret_cast<float *>(tab_s);  // [warps][8 products x 4 registers][32 lanes]
    {
        float *base = wacc + (size_t)warp * 1024 + lane;
#pragma unroll
        for (int mm = 0; mm < 8; ++mm) {
            base[(mm * 4 + 0) * 32] = acc[mm][0];
            base[(mm * 4 + 1) * 32] = acc[mm][1];
            base[(mm * 4 + 2) * 32] = acc[mm][2];
            base[(mm * 4 + 3) * 32] = acc[mm][3];
        }
    }
    __syncthreads();
    for (int oo = tid; oo < n_rows * 4 * kDim; oo += kThreads) {
        // output o of a row <-> (product mm, register j, lane of visiting order 0); its twin of order 1 is (mm, j^2, lane^2)
        const int br = oo >> 9, o = oo & 511;
        const int mm = o >> 6, j = (o >> 4) & 3, l16 = o & 15;
        const int src_r8 = l16 >> 1, src_kq = l16 & 1;
        const int lane0 = src_r8 * 4 + src_kq;
        const int r = 2 * src_kq + (j & 1);
        if (r >= rep) continue;
        const int dim = (2 * src_r8 + (j >> 1)) * 8 + mm;
        float asum = 0.0f;
        for (int w = br * kRowWarps; w < (br + 1) * kRowWarps; ++w) {
            const float *src = wacc + (size_t)w * 1024;
            asum += src[(mm * 4 + j) * 32 + lane0] + src[(mm * 4 + (j ^ 2)) * 32 + (lane0 ^ 2)];
        }
        float *dst = part + ((int64_t)split * rows + (int64_t)(b0 + br) * Hq + h * rep + r) * (kDim + 2);
        dst[2 + dim] = asum;
        if (dim == 0) {
            float top = -INFINITY, lsum = 0.0f;
            for (int w = br * kRowWarps; w < (br + 1) * kRowWarps; ++w) {
                top = fmaxf(top, red_s[w * 4 + r]);
                lsum += red_s[kRedFloats + w * 4 + r];
            }
            dst[0] = top;
            dst[1] = limit_s[br].x < limit_s[br].y ? lsum : 0.0f;  // without a token there is no maximum, and weights that mean nothing
        }
    }
}

// Rows a block, and splits of the positions, for `visible` positions a row.  One block per SM; a block costs its
// table copies and merge (kFixed) and its tokens, whose price falls with the rows that share a position's cos/sin; the pair with
// the least waves x block is taken.  Up to eight parts a row are merged in one round of loads, more take kMerge longer.  In clocks, from the
// measured kernel.  (Splits for the buffer instead of the visible range: 8 rows
// with 4096 of 30001 tokens visible 91 us a step against 45.)
struct Plan {
    int rows, splits;
};

inline Plan plan(int B, int Hkv, int64_t visible, int sms) {
    constexpr double kFixed = 14000.0, kMerge = 3000.0;
    Plan best = {0, 0};
    double least_cost = 0.0;
    for (int rows = 4; rows >= 1; rows >>= 1) {
        if (rows > 1 && B <= rows / 2) continue;  // fewer rows than that share a block
        const int groups = (B + rows - 1) / rows, share = (B + groups - 1) / groups;
        const double token = rows == 4 ? 19.0 : rows == 2 ? 20.0 : 22.0;
        const int64_t least = (visible + kChunk / rows - 1) / (kChunk / rows);
        for (int splits = least < 1 ? 1 : (int)(least > 65 ? 65 : least); splits <= 64; ++splits) {
            const int64_t per = (visible + splits - 1) / splits;
            const int64_t waves = ((int64_t)groups * Hkv * splits + sms - 1) / sms;
            const double cost = (double)waves * (kFixed + (double)(share * per) * token) + 40.0 * splits + (splits > 8 ? kMerge : 0.0);
            if (best.rows == 0 || cost < least_cost) least_cost = cost, best = {rows, splits};
            if (per * share <= 256) break;
        }
    }
    return best;
}

}  // namespace rotmma

bool attn_rotary_mma_supported(int Hq, int Hkv, int D, int G, int S, int K) {
    const int rep = Hkv > 0 ? Hq / Hkv : 0;
    return D == 128 && G == 16 && S == 2 && K == 256 && (rep == 1 || rep == 2 || rep == 4);
}

template <int R>
static int launch_rotary_mma(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab, const __half *vtab,
                             const __half *rope, const int32_t *seq_start, const int32_t *seq_end, float *part, int B, int Hq,
                             int Hkv, int64_t T_cap, int splits, bool after_prologue, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(rotmma::attn_rotary_mma_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, rotmma::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((unsigned)splits, (unsigned)Hkv, (unsigned)((B + R - 1) / R));
    e = launch_dependent(after_prologue, rotmma::attn_rotary_mma_kernel<R>, grid, dim3(rotmma::kThreads), rotmma::kSmemBytes, stream, q, kcodes,
                         vcodes, ktab, vtab, rope, seq_start, seq_end, part, B, Hq, Hkv, T_cap, splits);
    return e == cudaSuccess ? launch_status() : (int)e;
}

// Partial states [split][B*Hq][2 + D] for attn_combine_kernel; *splits is how many (0: `visible` positions are too many for
// the score areas of 64 splits, nothing was launched).  No row may see more than `visible` positions, nor may two rows of
// the batch together span more.
int attn_rotary_mma_dispatch(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab, const __half *vtab,
                             const __half *rope, const int32_t *seq_start, const int32_t *seq_end, float *part, int B, int Hq,
                             int Hkv, int64_t T_cap, int64_t visible, int sms, bool after_prologue, int *splits,
                             cudaStream_t stream) {
    const rotmma::Plan plan = rotmma::plan(B, Hkv, visible, sms);
    *splits = plan.splits;
    switch (plan.rows) {
        case 1: return launch_rotary_mma<1>(q, kcodes, vcodes, ktab, vtab, rope, seq_start, seq_end, part, B, Hq, Hkv, T_cap, plan.splits, after_prologue, stream);
        case 2: return launch_rotary_mma<2>(q, kcodes, vcodes, ktab, vtab, rope, seq_start, seq_end, part, B, Hq, Hkv, T_cap, plan.splits, after_prologue, stream);
        case 4: return launch_rotary_mma<4>(q, kcodes, vcodes, ktab, vtab, rope, seq_start, seq_end, part, B, Hq, Hkv, T_cap, plan.splits, after_prologue, stream);
        default: return TACVQ_OK;
    }
}

}  // namespace tacvq
