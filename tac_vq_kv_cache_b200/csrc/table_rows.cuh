// Tables of two stages x 16 groups of 8-wide words in shared memory, as the benchmark layout's kernels gather from them.
#pragma once

#include "common.cuh"

namespace tacvq {

// A code's 32 words fill one 512-byte row; a word's place in it decides its bank, whatever the code: stage * 4 + group % 4.
__device__ __forceinline__ int word_place(int stage, int group) { return (group >> 2) * 8 + stage * 4 + (group & 3); }

// A head's tables [stage][group][word][8] -> rows [word][place], by WARPS warps.  A warp takes 32 words of eight neighbouring places: whole
// lines in, a word a lane; the lanes then turn their eight pieces so that at every step eight neighbouring lanes store to eight
// different banks.  16-byte cp.async with scattered places go out one a clock, and less from all SMs at once: 8.9 k to 12 k clocks for a
// table, 2.9 k this way (a flat copy of 128 KB takes 1.7 k).
template <int WARPS>
__device__ __forceinline__ void copy_table_rows(uint32_t rows_u32, const __half *__restrict__ src, int warp, int lane) {
    constexpr int kUnits = 4 * (kMaxWords / 32) / WARPS;  // of a warp; all their words are asked for before the first is stored
    static_assert(kUnits * WARPS == 4 * (kMaxWords / 32), "");
    uint4 v[kUnits][8];
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
        const int unit = warp + i * WARPS, block = unit & 3, word = (unit >> 2) * 32 + lane;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = __ldg(reinterpret_cast<const uint4 *>(src) + ((j >> 2) * 16 + block * 4 + (j & 3)) * kMaxWords + word);
    }
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
        const int unit = warp + i * WARPS, block = unit & 3, word = (unit >> 2) * 32 + lane;
#pragma unroll
        for (int k = 1; k < 8; k <<= 1) {  // piece j becomes piece j + lane (mod 8)
            const bool turn = (lane & k) != 0;
            uint4 w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint4 a = v[i][j], b = v[i][(j + k) & 7];
                w[j] = make_uint4(turn ? b.x : a.x, turn ? b.y : a.y, turn ? b.z : a.z, turn ? b.w : a.w);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) v[i][j] = w[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(rows_u32 + word * 512 + (block * 8 + ((j + lane) & 7)) * 16), "r"(v[i][j].x),
                         "r"(v[i][j].y), "r"(v[i][j].z), "r"(v[i][j].w) : "memory");
    }
}

}  // namespace tacvq
