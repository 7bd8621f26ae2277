// How attention over codes of pre-rotary keys is divided for full-width ladders, and which of its two kernels takes a call
// (host code; attn_rotary_ladder.cu, attn_rotary.cu).
#pragma once

#include <stdint.h>

namespace tacvq {

// Blocks of attn_rotary_kernel per (batch row, KV head): about four waves (two resident per SM), at least 256 tokens per block, at most 64 splits.
inline int rotary_splits(int B, int Hkv, int64_t T_cap, int sms) {
    const int64_t pairs = (int64_t)B * Hkv;
    int64_t splits = (8 * (int64_t)sms + pairs - 1) / pairs;
    const int64_t by_len = (T_cap + 255) / 256;
    if (splits > by_len) splits = by_len;
    if (splits > 64) splits = 64;
    if (splits < 1) splits = 1;
    return (int)splits;
}

namespace ladder {

constexpr int kChunk = 4096;  // tokens of a cluster at a time at most

struct Plan {
    int clusters, splits;  // splits = 0: the general kernel is quicker, or the visible range needs more than 64
};

// us of attn_rotary_kernel for a ladder: trips of 32 tokens through blocks that fetch every token's words from L2, two blocks an SM.
inline double general_us(int B, int Hq, int Hkv, int S, int64_t T_cap, int64_t visible, int sms) {
    const int splits = rotary_splits(B, Hkv, T_cap, sms), rep = Hq / Hkv;
    const int64_t blocks = (int64_t)splits * B * Hkv, trips = ((visible + splits - 1) / splits + 31) / 32;
    const double trip = rep == 4 ? 2.49 + 0.59 * S : rep == 2 ? 1.56 + 0.518 * S : 1.2 + 0.5 * S;
    return 7.0 + (double)((blocks + 2 * sms - 1) / (2 * sms)) * (double)trips * (blocks <= sms ? 0.8 * trip : trip);
}

// `most`: clusters that the chip holds beside one another.  The items (a split of a row's visible tokens) are dealt out in the cheapest way, in
// tokens: an item costs its barriers, histograms and products (kFixed) and its tokens, a change of head the table (kTable).
//
// The ladder kernel pays per item, the general one per token and stage, so many rows of few tokens and short ladders belong to the latter.  us a call,
// general / ladder kernel, 8 KV heads with four query heads each: 16 stages, 16 x 300 tokens 68 / 113, 4 x 2000 103 / 81, 1 x 600 75 / 22; 8 stages,
// 16 x 300 44 / 91, 8 x 2000 122 / 112; 4 stages, 4 x 2000 46 / 68, 1 x 600 34 / 16.  Both estimates are fitted to calls of 4 to 16
// stages, 1 to 16 rows and 300 to 16384 tokens (within 7 %).  The 4 us are what a decode step hides of the ladder kernel behind the encode of its token.
inline Plan plan(int B, int Hq, int Hkv, int S, int64_t T_cap, int64_t visible, int sms, int most) {
    constexpr double kFixed = 1500.0, kTable = 1500.0;
    const int64_t least = (visible + kChunk - 1) / kChunk;
    Plan best = {0, 0};
    double least_cost = 0.0, us = 0.0;
    for (int s = least < 1 ? 1 : (int)(least > 65 ? 65 : least); s <= 64; ++s) {
        const int64_t per = (visible + s - 1) / s, items = (int64_t)Hkv * B * s, per_head = (int64_t)B * s;
        const int64_t heads_at_once = most / Hkv;  // clusters a head, when every head has some
        const int64_t options[2] = {items < most ? items : most, heads_at_once > 0 ? Hkv * (heads_at_once < per_head ? heads_at_once : per_head) : 0};
        for (const int64_t c : options) {
            if (c < 1) continue;
            const int64_t rounds = (items + c - 1) / c;
            const int64_t tables = items % c == 0 && per_head % (items / c) == 0 ? 1 : 1 + (rounds + per_head - 2) / per_head;
            const double cost = (double)rounds * (kFixed + (double)per) + (double)tables * kTable + 20.0 * s;
            if (best.clusters == 0 || cost < least_cost) {
                least_cost = cost, best = {(int)c, s};
                us = 3.4 + (double)rounds * (5.5 + 0.265 * S + (double)per * (0.00686 + 0.000071 * S)) + 3.06 * (double)tables;
            }
        }
        if (per <= 256) break;
    }
    if (best.clusters == 0 || (int64_t)Hkv * B * best.splits > 0x7fffffff || us > general_us(B, Hq, Hkv, S, T_cap, visible, sms) + 4.0) return {0, 0};
    return best;
}

}  // namespace ladder
}  // namespace tacvq
