// Decode-step attention over codes for head_dim 128 and at most 32 code bytes a token and side ("slots": stage x group), one,
// two or four query heads per KV head, no rotary step: the reference's own ladders (tables [H,S,256,128]), two additive
// full-width codebooks, grouped codebooks of one stage.  (16 groups x 2 stages with four heads has a kernel of its own.)
//
// A block takes one (batch row, KV head, group of HEADS query heads) and a range of tokens:
//   scores   a table lut[code][slot] of the HEADS partial scores q . word, fp32, built once; a token's score is the sum of its
//            slots' entries.
//   values   no value row is rebuilt: sum_t p_t sum_slot word[slot][code] = sum_slot sum_code (sum of p_t over the tokens with that
//            code) word, so a token adds its weights to hist[code][slot] and the histogram meets the V words once, at the end.
//
// What bounds it is the shared-memory pipe, so both tables are laid out for it: a code's entries of all slots fill one 256-byte
// row, the slot decides the bank, and lanes that are served together work on different slots (lane l takes slot k XOR l at step k;
// with fewer than eight slots the table is there several times and neighbouring lanes use different copies).  In the histogram
// the heads rotate with the lane as well: the 32 adds of an instruction meet 32 banks, whatever the codes.  Against tables
// ordered [slot][code], where random codes collide (2.6 wavefronts a look-up instead of 1, 3.6 an add), that is what this kernel
// gains.
//
// Weights are added as integers, because shared-memory integer adds are single instructions (a float add is a compare-and-swap
// loop).  FINE: a weight's multiple of 2^-19 goes to one bin and what that leaves, in units of 2^-38, to another, which keeps all 24
// bits of a weight down to 2^-15 and costs two adds.  Otherwise weights from 2^-10 on are added in units of 2^-20, smaller ones in
// units of 2^-30 and in bins of their own, one add each; ladders of up to 16 full-width stages with four query heads are content
// with that, as their weights had 18 bits before. Integer sums are exact and the result does not depend on the order.  A weight is
// relative to a reference that lies a little (kHeadroom) above the largest score when it was last set; when a score exceeds it, or
// the bins could overflow, they are folded into fp32 sums that every thread keeps in registers.  (With the largest score itself as
// the reference, ten of the first sixteen segments set it anew.)
//
// us a decode step with 8 KV heads, against the kernels this one replaced (tables ordered [slot][code] for full-width words, rebuilt value
// rows for groups): 2 x 128, 16 rows x 16384 tokens 31.4 / 44.7; 16 x 128, 2 x 32768 78 / 142; 16 x 8, 8 x 32768 94 / 229; 32 x 4 164 / 309;
// 16 x 2 x 8 with two query heads a KV head 103 / 302, with one 141 / 296.  The second add of a weight is 18 us of the 94 and 14 of the 164.
//
// Short calls are bound by what a block does besides its tokens.  In clocks, one row of 100 tokens, 2 x 2 x 64: empty bins 1.6 k, score
// table 17 k, folding the bins once 2.7 k (8 k for one slot), V words 7 k.  The table is a tensor-core product for every width from 16
// on and has its query channels in registers below, bins are folded a row a warp, lanes take neighbouring words of 4 channels: us a call,
// one row, before / now: 2 x 2 x 64 with one head 19.7 / 13.0, 1 x 128 15.4 / 11.0, 16 x 8 18.4 / 15.9, 8 x 2 x 16 22.8 / 18.7; 16 rows of 300
// tokens, 32 x 4 43.2 / 34.2 a step.
//
// Semantics replaced: experiments_followup_mistral/evaluate_mistral_longbench.py:112-122 (no rotary step).  Differences from the
// dense path inside the 2e-3 tolerance: the V row is the exact sum of its words (the reference rounds that sum to fp16 once), a
// score is the sum of partial dot products (the reference rounds the rebuilt key to fp16 first).

#include <type_traits>

#include "common.cuh"

namespace tacvq {
namespace slots {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kDim = 128, kWords = 256, kRowBytes = 256;
constexpr unsigned kEarlyBlocks = 98;  // two thirds of a B200's 148 SMs: a third is free for a merge that starts early
constexpr int kAreaBytes = kWords * kRowBytes;  // score table; histogram of large weights; of small weights
// 4096 weights of at most 1 x kLarge, or of less than 2^-10 x kSmall, add up below 2^32
constexpr float kLarge = 1048575.0f, kSmall = 1073740800.0f, kBorder = 0.0009765625f;
constexpr float kFine = 524288.0f, kRound = 8388608.0f, kRoundSigned = 12582912.0f;  // 2^19; adding them rounds to an integer
constexpr float kHeadroom = 1.0f;  // natural-log units
constexpr int kQueryFloats = kDim * 4 + 32 * 4;  // [group][channel of the group, one more][head]
constexpr int kSmemBytes = 3 * kAreaBytes + (kQueryFloats + kWarps * 8 + 8) * 4;
static_assert(kWarps * 4 * kDim * 4 <= kAreaBytes, "the warps' sums reuse a histogram");

// P: the slots rounded up to a power of two
template <int P>
struct Shape {
    static constexpr int kHeads = P == 32 ? 2 : 4, kEntry = kHeads * 4;
    static constexpr int kSpread = P == 32 ? 16 : 8;                   // lanes served together
    static constexpr int kCopies = P < kSpread ? kSpread / P : 1;
    static constexpr int kCodeWords = P < 4 ? 1 : P / 4;
    static constexpr int kTokens = P >= 16 ? 2 : P == 8 ? 4 : 8;       // a thread's tokens of a segment
    static constexpr int kFold = 4096 * kCopies;                       // tokens after which the bins are folded: a copy takes 4096 weights
    static constexpr int kUsed = kCopies * P * kHeads;                 // words of a code's row that are used
    static constexpr int kBins = kUsed * kWords / kThreads;            // a thread's bins, of all copies
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ void add_shared(uint32_t addr, uint32_t v) { asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {  // two fp32 sums
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// a token's code bytes; slots that are a power of two have rows that one or two aligned loads fetch
template <int P, bool FULL>
__device__ __forceinline__ void load_codes(const uint8_t *p, int slots, uint32_t (&w)[Shape<P>::kCodeWords]) {
    if constexpr (!FULL || P == 1) {
#pragma unroll
        for (int i = 0; i < Shape<P>::kCodeWords; ++i) {
            w[i] = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (4 * i + j < P && 4 * i + j < slots) w[i] |= (uint32_t)p[4 * i + j] << (8 * j);
        }
    } else if constexpr (P == 2) {
        w[0] = *reinterpret_cast<const unsigned short *>(p);
    } else if constexpr (P == 4) {
        w[0] = *reinterpret_cast<const uint32_t *>(p);
    } else if constexpr (P == 8) {
        const uint2 v = *reinterpret_cast<const uint2 *>(p);
        w[0] = v.x, w[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < P / 16; ++i) {
            const uint4 v = reinterpret_cast<const uint4 *>(p)[i];
            w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
        }
    }
}
// words 4 slots apart, in the lane's order: word k becomes word k XOR x / 4 (the bytes follow by selector)
template <int NW>
__device__ __forceinline__ void permute_words(uint32_t (&w)[NW], int x) {
    if constexpr (NW >= 2) {
        if (x & 4) {
#pragma unroll
            for (int i = 0; i < NW; i += 2) {
                const uint32_t t = w[i];
                w[i] = w[i + 1], w[i + 1] = t;
            }
        }
    }
    if constexpr (NW >= 8) {
        if (x & 8) {
#pragma unroll
            for (int i = 0; i < NW; i += 4) {
                uint32_t t = w[i];
                w[i] = w[i + 2], w[i + 2] = t;
                t = w[i + 1];
                w[i + 1] = w[i + 3], w[i + 3] = t;
            }
        }
    }
}

// adds a token's weights w[r] (FINE: and rest[r] to the second bins) at offsets to[r], heads in the lane's order; ALL: none of the
// block's heads is missing
template <int P, bool FULL, bool FINE, bool ALL>
__device__ __forceinline__ void add_weights(const uint32_t (&codes)[Shape<P>::kCodeWords], const uint32_t (&w)[Shape<P>::kHeads],
                                            const uint32_t (&rest)[Shape<P>::kHeads], const uint32_t (&to)[Shape<P>::kHeads],
                                            const uint32_t (&sel)[4], uint32_t lane_xor, int x, int slots, int rot, int heads) {
    constexpr int H = Shape<P>::kHeads;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        if (!FULL && (k ^ x) >= slots) continue;
        const uint32_t at = (prmt(codes[k >> 2], 0u, sel[k & 3]) | (uint32_t)(k * Shape<P>::kEntry)) ^ lane_xor;
#pragma unroll
        for (int r = 0; r < H; ++r)
            if (ALL || ((r + rot) & (H - 1)) < heads) {
                add_shared(at + to[r], w[r]);
                if constexpr (FINE) add_shared(at + to[r] + kAreaBytes, rest[r]);
            }
    }
}

template <int P, bool FULL, bool FINE>
__global__ void __launch_bounds__(kThreads, 1)
attn_slots_kernel(const __half *__restrict__ q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *__restrict__ ktab,
                  const __half *__restrict__ vtab, const int32_t *seq_start, const int32_t *seq_end, float *__restrict__ part, __half *__restrict__ out,
                  float *__restrict__ state_out, int B, int Hq, int Hkv, int G, int S, int64_t T_cap, int splits) {
    using L = Shape<P>;
    constexpr int H = L::kHeads, NW = L::kCodeWords, NT = L::kTokens;
    extern __shared__ __align__(256) unsigned char smem[];
    float *q_s = reinterpret_cast<float *>(smem + 3 * kAreaBytes);
    float *red = q_s + kQueryFloats;  // [warps][H] maxima, [warps][H] sums
    const uint32_t hist = smem_u32(smem) + kAreaBytes;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rep = Hq / Hkv, head_groups = (rep + H - 1) / H;
    const int split = blockIdx.x, h = blockIdx.y / head_groups, b = blockIdx.z;
    const int head0 = h * rep + blockIdx.y % head_groups * H, heads = min(H, (h + 1) * rep - head0);
    const int d = kDim / G, slots = S * G;

    // ---- lane constants ---------------------------------------------------------------------------------------------
    const int x = lane & (P < L::kSpread ? P - 1 : L::kSpread - 1);           // slot order: slot k XOR x at step k
    const int copy = P < L::kSpread ? (lane & (L::kSpread - 1)) / P : 0;
    const uint32_t lane_xor = (uint32_t)(copy * P + x) * L::kEntry;
    const int rot = lane / L::kSpread;                                        // head order: head r + rot at step r
    uint32_t sel[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) sel[i] = 0x4404u | (uint32_t)((i ^ x) & 3) << 4;  // code byte -> bits 8..15
    const uint8_t *kc_row = kcodes + ((int64_t)b * Hkv + h) * T_cap * slots, *vc_row = vcodes + ((int64_t)b * Hkv + h) * T_cap * slots;

    // ---- score table, and empty bins ----------------------------------------------------------------------------------
#pragma unroll
    for (int i = tid; i < 2 * kWords * L::kUsed / 4; i += kThreads)
        *reinterpret_cast<uint4 *>(smem + kAreaBytes + i / (L::kUsed / 4) * kRowBytes + i % (L::kUsed / 4) * 16) = make_uint4(0u, 0u, 0u, 0u);
    auto put_entry = [&](int code, int slot, int pair, float first, float second) {  // heads 2 * pair and the next, every copy
#pragma unroll
        for (int u = 0; u < L::kCopies; ++u)
            *(reinterpret_cast<float2 *>(smem + code * kRowBytes + (u * P + slot) * L::kEntry) + pair) = make_float2(first, second);
    };
    const __half *q_rows = q + ((int64_t)b * Hq + head0) * kDim;
    if (d >= 16) {
        // tensor cores: A = 16 words, B = the heads; warp w takes words 16 w .. 16 w + 15 of every slot.  A lane's 16 bytes are channels
        // 32 c + 8 kq .. of its two words (8 bytes, channels 4 kq .., for words of 16), which makes them the operands of two
        // products (one) over a channel order that the query follows.  32 channels at a time, added in fp32: the tensor core cuts off what
        // it adds to a sum that is there.
        const int r8 = lane >> 2, kq = lane & 3;
        auto products = [&](auto width) {
            constexpr int D = decltype(width)::value, C = D / 32;
            uint4 qf[C];
            auto load_query = [&](int g) {
#pragma unroll
                for (int c = 0; c < C; ++c) qf[c] = r8 < heads ? __ldg(reinterpret_cast<const uint4 *>(q_rows + r8 * kDim + g * D + 32 * c + 8 * kq)) : make_uint4(0u, 0u, 0u, 0u);
            };
            if (G == 1) load_query(0);
#pragma unroll 2
            for (int slot = 0; slot < slots; ++slot) {
                const uint4 *row = reinterpret_cast<const uint4 *>(ktab + (((int64_t)h * slots + slot) * kWords + warp * 16 + r8) * D) + kq;
                if (G > 1) load_query(slot % G);
                uint4 a[C], c8[C];
#pragma unroll
                for (int c = 0; c < C; ++c) a[c] = __ldg(row + 4 * c), c8[c] = __ldg(row + D + 4 * c);
                float part[C][4];
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    part[c][0] = part[c][1] = part[c][2] = part[c][3] = 0.0f;
                    mma16816(part[c], a[c].x, c8[c].x, a[c].y, c8[c].y, qf[c].x, qf[c].y);
                    mma16816(part[c], a[c].z, c8[c].z, a[c].w, c8[c].w, qf[c].z, qf[c].w);
                }
#pragma unroll
                for (int step = 1; step < C; step *= 2)
#pragma unroll
                    for (int c = 0; c < C; c += 2 * step)
#pragma unroll
                        for (int i = 0; i < 4; ++i) part[c][i] += part[c + step][i];
                if (2 * kq < H) {
                    put_entry(warp * 16 + r8, slot, kq, part[0][0], part[0][1]);
                    put_entry(warp * 16 + r8 + 8, slot, kq, part[0][2], part[0][3]);
                }
            }
        };
        if (d == 128) products(std::integral_constant<int, 128>());
        else if (d == 64) products(std::integral_constant<int, 64>());
        else if (d == 32) products(std::integral_constant<int, 32>());
        else {
#pragma unroll 4
            for (int slot = 0; slot < slots; ++slot) {
                const uint2 *row = reinterpret_cast<const uint2 *>(ktab + (((int64_t)h * slots + slot) * kWords + warp * 16 + r8) * 16) + kq;
                const uint2 a = __ldg(row), c8 = __ldg(row + 8 * 4);
                const uint2 qf = r8 < heads ? __ldg(reinterpret_cast<const uint2 *>(q_rows + r8 * kDim + slot % G * 16) + kq) : make_uint2(0u, 0u);
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                mma16816(sum, a.x, c8.x, a.y, c8.y, qf.x, qf.y);
                if (2 * kq < H) {
                    put_entry(warp * 16 + r8, slot, kq, sum[0], sum[1]);
                    put_entry(warp * 16 + r8 + 8, slot, kq, sum[2], sum[3]);
                }
            }
        }
    } else if constexpr (P >= 16) {
        for (int i = tid; i < kDim * H; i += kThreads) {
            const int r = i / kDim, c = i % kDim;
            q_s[(c / d * (d + 1) + c % d) * H + r] = r < heads ? __half2float(q_rows[r * kDim + c]) : 0.0f;
        }
        __syncthreads();
        // neighbouring lanes take different slots (no conflicts where they write and where they read the query), the next
        // lanes neighbouring codes (whole sectors of the table); a thread stays with a slot and has the query's channels in registers
        constexpr int kNear = L::kSpread, kTrips = kNear * kWords / kThreads;
        auto entries = [&](auto width) {
            constexpr int C = decltype(width)::value;  // channels of a word
#pragma unroll 1
            for (int slot = tid % kNear; slot < (FULL ? P : slots); slot += kNear) {
                const __half *words = ktab + (((int64_t)h * slots + slot) * kWords + tid / kNear) * C;
                uint32_t raw[kTrips][C / 2];
#pragma unroll
                for (int i = 0; i < kTrips; ++i) {
                    const __half *word = words + i * (kThreads / kNear) * C;
                    if constexpr (C == 8) {
                        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(word));
                        raw[i][0] = v.x, raw[i][1] = v.y, raw[i][2] = v.z, raw[i][3] = v.w;
                    } else {
                        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(word));
                        raw[i][0] = v.x, raw[i][1] = v.y;
                    }
                }
                const float2 *qv = reinterpret_cast<const float2 *>(q_s + slot % G * (C + 1) * H);
                float qr[C][H];
#pragma unroll
                for (int e = 0; e < C; ++e)
#pragma unroll
                    for (int r = 0; r < H; r += 2) {
                        const float2 v = qv[(e * H + r) / 2];
                        qr[e][r] = v.x, qr[e][r + 1] = v.y;
                    }
#pragma unroll
                for (int i = 0; i < kTrips; ++i) {
                    float dot[H];
#pragma unroll
                    for (int r = 0; r < H; ++r) dot[r] = 0.0f;
#pragma unroll
                    for (int e = 0; e < C; ++e) {
                        const __half2 pair = *reinterpret_cast<const __half2 *>(&raw[i][e / 2]);
                        const float f = __half2float(e & 1 ? __high2half(pair) : __low2half(pair));
#pragma unroll
                        for (int r = 0; r < H; ++r) dot[r] = fmaf(qr[e][r], f, dot[r]);
                    }
#pragma unroll
                    for (int r = 0; r < H; r += 2) put_entry(tid / kNear + i * (kThreads / kNear), slot, r / 2, dot[r], dot[r + 1]);
                }
            }
        };
        if (d == 4) entries(std::integral_constant<int, 4>());
        else entries(std::integral_constant<int, 8>());
    }

    // A decode step's new codes and ranges come from the kernel before this one; the tables and the query do not.
    wait_for_previous_kernel();
    // us a step, always / never / so: 2 x 128, 8 rows x 16384 tokens 27.4 / 26.1 / 26.1; 16 x 2 x 8 with one head a KV head, 16 x 396 29.6 / 27.7 / 27.7,
    // 4 x 466 20.1 / 23.9 / 20.1.
    if (gridDim.x * gridDim.y * gridDim.z <= kEarlyBlocks) launch_dependents();
    const int lo_all = max(seq_start ? seq_start[b] : 0, 0);
    const int hi_all = min(seq_end ? seq_end[b] : (int)T_cap, (int)T_cap);
    const int n_all = hi_all > lo_all ? hi_all - lo_all : 0;
    const int per = (n_all + splits - 1) / splits;
    const int lo = lo_all + split * per;
    const int hi = min(lo + per, lo_all + n_all);
    uint32_t kc[NT][NW], vc[NT][NW];
    auto fetch = [&](const uint8_t *row, int base, uint32_t (&w)[NT][NW]) {  // tokens past the end repeat the last one
#pragma unroll
        for (int j = 0; j < NT; ++j) load_codes<P, FULL>(row + (int64_t)min(base + j * kThreads + tid, hi - 1) * slots, slots, w[j]);
    };
    if (lo < hi) {
        fetch(kc_row, lo, kc);
        fetch(vc_row, lo, vc);
    }
    __syncthreads();

    // ---- tokens, a segment of NT x 512 at a time ------------------------------------------------------------------------
    float m[H], l[H], sums[L::kBins];  // reference score, this thread's weights; its folded bins tid + 512 i of [code][copy][slot][head]
#pragma unroll
    for (int r = 0; r < H; ++r) m[r] = -INFINITY, l[r] = 0.0f;
#pragma unroll
    for (int i = 0; i < L::kBins; ++i) sums[i] = 0.0f;
    auto fold = [&](float f) {  // what is in the bins joins the sums, times f; the bins become empty
        constexpr int kAtOnce = 8;
#pragma unroll
        for (int i0 = 0; i0 < L::kBins; i0 += kAtOnce) {
            uint32_t large[kAtOnce], small[kAtOnce];
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const int bin = tid + (i0 + i) * kThreads, at = kAreaBytes + bin / L::kUsed * kRowBytes + bin % L::kUsed * 4;
                large[i] = *reinterpret_cast<uint32_t *>(smem + at);
                small[i] = *reinterpret_cast<uint32_t *>(smem + at + kAreaBytes);
            }
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const int bin = tid + (i0 + i) * kThreads, at = kAreaBytes + bin / L::kUsed * kRowBytes + bin % L::kUsed * 4;
                *reinterpret_cast<uint32_t *>(smem + at) = 0u;
                *reinterpret_cast<uint32_t *>(smem + at + kAreaBytes) = 0u;
                float v;
                if constexpr (FINE) v = fmaf((float)(int32_t)small[i], 1.0f / (kFine * kFine), (float)large[i] * (1.0f / kFine));
                else v = fmaf((float)small[i], 1.0f / kSmall, (float)large[i] * (1.0f / kLarge));
                sums[i0 + i] = (sums[i0 + i] + v) * f;
            }
        }
    };
    int pending = 0;
#pragma unroll 1
    for (int base = lo;; base += NT * kThreads) {
        const bool more = base < hi;
        float sc[NT][H];
        bool grow = false;
        if (more) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (j > 0 && base + j * kThreads >= hi) {  // nobody has a token here
#pragma unroll
                    for (int r = 0; r < H; ++r) sc[j][r] = -INFINITY;
                    continue;
                }
                permute_words<NW>(kc[j], x);
                // two heads an addition; several short sums have less rounding than a long one
                constexpr int kSums = P == 32 ? 4 : P >= 4 ? 2 : 1;
                unsigned long long part[kSums][H / 2], pair[H / 2];
#pragma unroll
                for (int r = 0; r < H / 2; ++r)
#pragma unroll
                    for (int i = 0; i < kSums; ++i) part[i][r] = 0ull;
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    if (!FULL && (k ^ x) >= slots) continue;
                    const unsigned char *entry = smem + ((prmt(kc[j][k >> 2], 0u, sel[k & 3]) | (uint32_t)(k * L::kEntry)) ^ lane_xor);
                    if constexpr (H == 4) {
                        const ulonglong2 e = *reinterpret_cast<const ulonglong2 *>(entry);
                        part[k % kSums][0] = add2(part[k % kSums][0], e.x);
                        part[k % kSums][1] = add2(part[k % kSums][1], e.y);
                    } else {
                        part[k % kSums][0] = add2(part[k % kSums][0], *reinterpret_cast<const unsigned long long *>(entry));
                    }
                }
#pragma unroll
                for (int r = 0; r < H / 2; ++r) {
                    pair[r] = part[0][r];
                    if constexpr (kSums == 2) pair[r] = add2(pair[r], part[1][r]);
                    if constexpr (kSums == 4) pair[r] = add2(add2(pair[r], part[1][r]), add2(part[2][r], part[3][r]));
                }
#pragma unroll
                for (int r = 0; r < H; ++r) {
                    sc[j][r] = __uint_as_float((uint32_t)(pair[r / 2] >> (32 * (r & 1))));
                    if (base + j * kThreads + tid >= hi) sc[j][r] = -INFINITY;
                    grow |= sc[j][r] > m[r];
                }
            }
            if (base + NT * kThreads < hi) fetch(kc_row, base + NT * kThreads, kc);
        }
        // every thread has added its weights of the segment before when this returns
        const bool grown = __syncthreads_or(grow);
        float mine = 1.0f;  // what a fold multiplies this thread's bins by, which are all of one head
        if (grown) {
#pragma unroll
            for (int r = 0; r < H; ++r) {
                float v = sc[0][r];
#pragma unroll
                for (int j = 1; j < NT; ++j) v = fmaxf(v, sc[j][r]);
#pragma unroll
                for (int off = 16; off >= 1; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
                if (lane == 0) red[warp * H + r] = v;
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < H; ++r) {
                float top = m[r];
                for (int w = 0; w < kWarps; ++w) top = fmaxf(top, red[w * H + r]);
                top = top > m[r] ? top + kHeadroom : m[r];
                const float f = top == -INFINITY ? 1.0f : __expf(m[r] - top);  // 0 for the first tokens
                m[r] = top;
                l[r] *= f;
                mine = (tid & (H - 1)) == r ? f : mine;
            }
        }
        if (grown || !more || pending + NT * kThreads > L::kFold) {
            if (pending > 0) fold(mine);
            pending = 0;
            __syncthreads();  // bins are empty, maxima are read
        }
        if (!more) break;
        pending += NT * kThreads;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            if (base + j * kThreads + tid >= hi) continue;
            permute_words<NW>(vc[j], x);
            uint32_t w[H], rest[H], to[H];
#pragma unroll
            for (int r = 0; r < H; ++r) {
                const float p = __expf(sc[j][r] - m[r]);
                l[r] += p;
                // to the nearest integer by adding 2^23 (a conversion runs at a quarter of the rate); a NaN's sum spoils the result
                if constexpr (FINE) {
                    const float near = fmaf(p, kFine, kRound);
                    w[r] = __float_as_uint(near) & 0x7fffffu;
                    rest[r] = __float_as_uint(fmaf(fmaf(p, kFine, kRound - near), kFine, kRoundSigned)) - __float_as_uint(kRoundSigned);
                    to[r] = hist + r * 4;
                } else {
                    const bool small = p < kBorder;
                    w[r] = __float_as_uint(fmaf(p, small ? kSmall : kLarge, kRound)) & 0x7fffffu;
                    rest[r] = 0u;
                    to[r] = hist + r * 4 + (small ? kAreaBytes : 0);
                }
            }
            if (rot & 1) {
                const uint32_t w0 = w[0], r0 = rest[0], t0 = to[0];
#pragma unroll
                for (int r = 0; r + 1 < H; ++r) w[r] = w[r + 1], rest[r] = rest[r + 1], to[r] = to[r + 1];
                w[H - 1] = w0, rest[H - 1] = r0, to[H - 1] = t0;
            }
            if constexpr (H == 4) {
                if (rot & 2) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t wr = w[r], rr = rest[r], tr = to[r];
                        w[r] = w[r + 2], rest[r] = rest[r + 2], to[r] = to[r + 2];
                        w[r + 2] = wr, rest[r + 2] = rr, to[r + 2] = tr;
                    }
                }
            }
            if (heads == H) add_weights<P, FULL, FINE, true>(vc[j], w, rest, to, sel, lane_xor, x, slots, rot, heads);
            else add_weights<P, FULL, FINE, false>(vc[j], w, rest, to, sel, lane_xor, x, slots, rot, heads);
        }
        if (base + NT * kThreads < hi) fetch(vc_row, base + NT * kThreads, vc);
    }
    // the score table is done with: its place takes the folded weights, [code][slot][head]; a row's copies are in neighbouring lanes
#pragma unroll
    for (int i = 0; i < L::kBins; ++i) {
        const int bin = tid + i * kThreads, col = bin % L::kUsed;
        if constexpr (L::kCopies > 1) {
#pragma unroll
            for (int off = P * H; off < L::kUsed; off *= 2) sums[i] += __shfl_xor_sync(0xffffffffu, sums[i], off);
        }
        if (col < P * H) *reinterpret_cast<float *>(smem + bin / L::kUsed * kRowBytes + col * 4) = sums[i];
    }
#pragma unroll
    for (int r = 0; r < H; ++r) {
        float v = l[r];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[kWarps * H + warp * H + r] = v;
    }
    __syncthreads();

    // ---- weights x V words: a thread has a piece of 8 channels (4, for words that short) of every 32nd (16th) word ---------
    float *warp_sums = reinterpret_cast<float *>(smem + kAreaBytes);  // [warp][H][128]
    auto product = [&](auto width) {
        constexpr int C = decltype(width)::value, kPieces = kDim / C, kSlices = kThreads / kPieces;
        // words of four channels: neighbouring lanes take the words of a sector, a warp eight groups (a group a lane would be 32 lines a load)
        const int piece = C == 4 ? (warp & 3) * 8 + (lane >> 2) : tid % kPieces, g = piece * C / d, off = piece * C % d;
        const int first = C == 4 ? (warp >> 2) * 4 + (lane & 3) : tid / kPieces;  // of this thread's words, kSlices apart
        float acc[H][C];
#pragma unroll
        for (int r = 0; r < H; ++r)
#pragma unroll
            for (int i = 0; i < C; ++i) acc[r][i] = 0.0f;
        for (int s = 0; s < S; ++s) {
            const __half *words = vtab + ((int64_t)h * slots + s * G + g) * kWords * d + off;
            const unsigned char *weights = smem + (s * G + g) * L::kEntry;
            constexpr int kTrips = kWords / kSlices, kAtOnce = 8;  // words of a thread; of them, on their way together
#pragma unroll 1
            for (int trip = 0; trip < kTrips; trip += kAtOnce) {
                uint32_t raw[kAtOnce][C / 2];
#pragma unroll
                for (int k = 0; k < kAtOnce; ++k) {
                    const __half *from = words + (first + (trip + k) * kSlices) * d;
                    if constexpr (C == 8) {
                        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(from));
                        raw[k][0] = v.x, raw[k][1] = v.y, raw[k][2] = v.z, raw[k][3] = v.w;
                    } else {
                        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(from));
                        raw[k][0] = v.x, raw[k][1] = v.y;
                    }
                }
#pragma unroll
                for (int k = 0; k < kAtOnce; ++k) {
                    float w[H];
                    bool used = false;  // a word that no token refers to may hold anything
#pragma unroll
                    for (int r = 0; r < H; r += 2) {
                        const float2 v = *reinterpret_cast<const float2 *>(weights + (first + (trip + k) * kSlices) * kRowBytes + r * 4);
                        w[r] = v.x, w[r + 1] = v.y;
                        used |= v.x != 0.0f || v.y != 0.0f;
                    }
#pragma unroll
                    for (int i = 0; i < C / 2; ++i) {
                        const uint32_t pair = used ? raw[k][i] : 0u;
                        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&pair));
#pragma unroll
                        for (int r = 0; r < H; ++r) {
                            acc[r][2 * i] = fmaf(w[r], f.x, acc[r][2 * i]);
                            acc[r][2 * i + 1] = fmaf(w[r], f.y, acc[r][2 * i + 1]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < H; ++r) {
#pragma unroll
            for (int i = 0; i < C; ++i) {
                if constexpr (C == 4) {
                    acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], 1);
                    acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], 2);
                } else {
                    acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], 16);
                }
            }
            if (C == 4 ? (lane & 3) == 0 : lane < 16) {
#pragma unroll
                for (int i = 0; i < C; i += 4)
                    *reinterpret_cast<float4 *>(warp_sums + (warp * H + r) * kDim + piece * C + i) = make_float4(acc[r][i], acc[r][i + 1], acc[r][i + 2], acc[r][i + 3]);
            }
        }
    };
    if (P == 32 && d == 4) product(std::integral_constant<int, P == 32 ? 4 : 8>());
    else product(std::integral_constant<int, 8>());
    __syncthreads();
    const int64_t rows = (int64_t)B * Hq;
    for (int o = tid; o < heads * kDim; o += kThreads) {
        const int r = o / kDim, channel = o % kDim;
        float lsum = 0.0f, asum = 0.0f;
        // words of four channels: a channel is in every fourth warp's sums
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            lsum += red[(kWarps + w) * H + r];
            if (P < 32 || d > 4 || w % 4 == channel / 32) asum += warp_sums[(w * H + r) * kDim + channel];
        }
        float top = m[0];
#pragma unroll
        for (int k = 1; k < H; ++k) top = r == k ? m[k] : top;
        // the state's reference is a score that was there, as exactly as fp32 has it: the sums follow what the subtraction gave
        const float ref = top - kHeadroom, back = top == -INFINITY ? 1.0f : expf(top - ref);
        top = ref;
        lsum *= back;
        asum *= back;
        const int64_t row = (int64_t)b * Hq + head0 + r;
        if (splits == 1) {  // the whole row was handled here: this is the result
            if (out) out[row * kDim + channel] = __float2half_rn(lsum == 0.0f ? 0.0f : asum / lsum);
            if (state_out) {
                float *dst = state_out + row * (kDim + 2);
                if (channel == 0) dst[0] = top, dst[1] = lsum;
                dst[2 + channel] = asum;
            }
        } else {
            float *dst = part + ((int64_t)split * rows + row) * (kDim + 2);
            if (channel == 0) dst[0] = top, dst[1] = lsum;
            dst[2 + channel] = asum;
        }
    }
}

template <int P, bool FINE>
static int launch(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab, const __half *vtab,
                  const int32_t *seq_start, const int32_t *seq_end, float *part, __half *out, float *state_out, int B, int Hq, int Hkv,
                  int G, int S, int64_t T_cap, int splits, bool after_prologue, cudaStream_t stream) {
    auto kernel = S * G == P ? attn_slots_kernel<P, true, FINE> : attn_slots_kernel<P, false, FINE>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    const int rep = Hq / Hkv, head_groups = (rep + Shape<P>::kHeads - 1) / Shape<P>::kHeads;
    dim3 grid((unsigned)splits, (unsigned)(Hkv * head_groups), (unsigned)B);
    e = launch_dependent(after_prologue, kernel, grid, dim3(kThreads), kSmemBytes, stream, q, kcodes, vcodes, ktab, vtab, seq_start, seq_end,
                         part, out, state_out, B, Hq, Hkv, G, S, T_cap, splits);
    return e == cudaSuccess ? launch_status() : (int)e;
}

}  // namespace slots

bool attn_slots_supported(int B, int Hq, int Hkv, int D, int G, int S, int K) {
    const int rep = Hkv > 0 ? Hq / Hkv : 0;
    return D == 128 && K == 256 && G <= 32 && S * G <= 32 && (rep == 1 || rep == 2 || rep == 4) && (int64_t)Hkv * 2 <= 65535 && B <= 65535;
}

// Blocks per (batch row, KV head): the count with the cheapest waves of one block an SM.  In clocks: a block pays for its tables
// (a head's K and V words from L2) and for its tokens; several blocks a row for the merge.  Against one block a pair as long as the pairs
// fill the chip, 2 x 128 and 2 rows of 500 tokens: 21 us a step, 27 before.
int attn_slots_splits(int B, int Hq, int Hkv, int G, int S, int64_t visible, int sms) {
    const int n = S * G, heads = n > 16 ? 2 : 4, rep = Hq / Hkv, slots = n > 16 ? 32 : n > 8 ? 16 : n > 4 ? 8 : 4;
    const int64_t pairs = (int64_t)B * Hkv * ((rep + heads - 1) / heads);
    const double fixed = 6000.0 + 4500.0 * S, token = 1.0 + 0.07 * slots * heads;
    int best = 1;
    double least_cost = 0.0;
    for (int splits = 1; splits <= 64; ++splits) {
        const int64_t per = (visible + splits - 1) / splits, waves = (pairs * splits + sms - 1) / sms;
        const double cost = (double)waves * (fixed + token * (double)per) + (splits > 1 ? 5000.0 + 30.0 * splits : 0.0);
        if (splits == 1 || cost < least_cost) least_cost = cost, best = splits;
        if (per <= 512) break;
    }
    return best;
}

// `after_prologue`: the launch before this one is the prologue of the same decode step, which lets this one start when everything before it has ended.
int attn_slots_dispatch(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab, const __half *vtab,
                        const int32_t *seq_start, const int32_t *seq_end, float *part, __half *out, float *state_out, int B, int Hq,
                        int Hkv, int G, int S, int64_t T_cap, int splits, bool after_prologue, cudaStream_t stream) {
#define TACVQ_LAUNCH(P, FINE)                                                                                                               \
    slots::launch<P, FINE>(q, kcodes, vcodes, ktab, vtab, seq_start, seq_end, part, out, state_out, B, Hq, Hkv, G, S, T_cap, splits, \
                           after_prologue, stream)
#define TACVQ_CASE(P) return coarse ? TACVQ_LAUNCH(P, false) : TACVQ_LAUNCH(P, true);
    const int n = S * G;
    const bool coarse = G == 1 && Hq == 4 * Hkv && n <= 16;
    if (n == 1) TACVQ_CASE(1)
    if (n == 2) TACVQ_CASE(2)
    if (n <= 4) TACVQ_CASE(4)
    if (n <= 8) TACVQ_CASE(8)
    if (n <= 16) TACVQ_CASE(16)
    return TACVQ_LAUNCH(32, true);
#undef TACVQ_CASE
#undef TACVQ_LAUNCH
}

}  // namespace tacvq
