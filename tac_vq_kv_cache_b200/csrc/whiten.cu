// Whitened assignment geometry: transform rows and codewords once, before the search.
//
//   search_rows[b,h,t,g*d+i]   = sum_j W[h,g,i,j] * x[b,h,t,g*d+j]
//   search_tables[h,s,g,k,i]   = sum_j W[h,g,i,j] * tables[h,s,g,k,j]
// each as one fused-multiply-add chain over j ascending.  The encode kernels then search the
// transformed rows against the transformed words and subtract transformed words stage by stage,
// which is the reference's "transform once, subtract transformed codewords" recursion
// (src/jointkv/closed_loop_vq.py:312-320, 384-390; src/jointkv/cq_tac.py:80-85).
//
// Wide groups (d = 32, 64, 128) are a d x d product per row: a block keeps one (head, group) matrix,
// transposed, and a tile of rows in shared memory; a thread owns 4 outputs of several rows and
// walks j in order, four steps per 16-byte shared-memory load.  Narrow groups (d <= 16) cost d
// multiply-adds per output and stay one thread per output.

#include <type_traits>

#include "common.cuh"

namespace tacvq {

// ------------------------------------------------------------------------------------------------
// narrow groups: one thread = one output element
// ------------------------------------------------------------------------------------------------

template <typename XT>
__global__ void __launch_bounds__(256)
whiten_rows_kernel(const XT *__restrict__ x, int64_t sxb, int64_t sxh, int64_t sxt, const float *__restrict__ whitener,
                   float *__restrict__ out, int B, int H, int T, int D, int G) {
    const int d = D / G;
    const int64_t total = (int64_t)B * H * T * D;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int c = (int)(idx % D);
        const int64_t row = idx / D;
        const int t = (int)(row % T);
        const int64_t bh = row / T;
        const int h = (int)(bh % H);
        const int64_t b = bh / H;
        const int g = c / d, i = c % d;
        const XT *src = x + b * sxb + (int64_t)h * sxh + (int64_t)t * sxt + (int64_t)g * d;
        const float *w = whitener + (((int64_t)h * G + g) * d + i) * d;
        float acc = 0.0f;
        for (int j = 0; j < d; ++j) acc = __fmaf_rn(w[j], to_float<XT>(src[j]), acc);
        out[idx] = acc;
    }
}

__global__ void __launch_bounds__(256)
whiten_tables_kernel(const __half *__restrict__ tables, const float *__restrict__ whitener, float *__restrict__ out,
                     int H, int S, int G, int K, int d) {
    const int64_t total = (int64_t)H * S * G * K * d;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % d);
        const int64_t word = idx / d;  // ((h*S+s)*G+g)*K+k
        const int g = (int)((word / K) % G);
        const int h = (int)(word / ((int64_t)K * G * S));
        const float *w = whitener + (((int64_t)h * G + g) * d + i) * d;
        const __half *src = tables + word * d;
        float acc = 0.0f;
        for (int j = 0; j < d; ++j) acc = __fmaf_rn(__half2float(src[j]), w[j], acc);
        out[idx] = acc;
    }
}

// ------------------------------------------------------------------------------------------------
// wide groups: shared-memory tiles, 4 outputs x several rows per thread
// ------------------------------------------------------------------------------------------------

constexpr int kWideThreads = 256, kWideBlocks = 2 * 148;

// R rows a thread
template <int DSUB, int R>
struct WideLayout {
    static constexpr int kWStride = DSUB + 4;  // floats; rows of the transposed matrix stay 16-byte aligned, banks staggered
    static constexpr int kOutPerRow = DSUB / 4;                       // threads that share a row
    static constexpr int kRowGroups = kWideThreads / kOutPerRow;      // rows handled side by side
    static constexpr int kRows = R * kRowGroups;                      // of a tile
    static constexpr size_t kBytes = ((size_t)DSUB * kWStride + (size_t)kRows * DSUB) * sizeof(float);
};

struct WideArgs {
    const void *x;
    const __half *tables;
    const float *whitener;
    float *out_tables, *out_rows;
    int64_t sxb, sxh, sxt;
    uint32_t rows, words;  // B * T, S * K
    int H, T, D, G, S, K, vec_rows, vec_words;
};

// Tiles of a (head, group): its words', then its rows'.  The tiles of all of them are dealt out evenly to two blocks an SM, which keep
// the matrix while they stay with a (head, group).  Bound by the FMA pipe and the copies in front of it.  Against a launch for the words and one
// for the rows, a block and a copy of the matrix for every 64 of either, us a whole whitened encode of 8 heads, 128 wide: 16 stages, one row
// 137 / 116, 2048 rows 228 / 208; two stages, one row 41 / 25, 4000 rows 111 / 92, 16000 rows 340 / 288.
template <int DSUB, typename XT, int R>
__global__ void __launch_bounds__(kWideThreads, 2)
whiten_wide_kernel(const WideArgs a) {
    using L = WideLayout<DSUB, R>;
    extern __shared__ __align__(16) float wsm[];
    float *wt = wsm;                                  // [j][i] : W transposed
    float *xs = wsm + (size_t)DSUB * L::kWStride;     // [row][j]
    const int tid = threadIdx.x;
    const int i0 = (tid % L::kOutPerRow) * 4, rg = tid / L::kOutPerRow;
    const uint32_t word_tiles = (a.words + L::kRows - 1) / L::kRows, tiles = word_tiles + (a.rows + L::kRows - 1) / L::kRows;
    const int64_t work = (int64_t)a.H * a.G * tiles, end = work * (blockIdx.x + 1) / gridDim.x;
    int have = -1;
#pragma unroll 1
    for (int64_t at = work * blockIdx.x / gridDim.x; at < end; ++at) {
        const int hg = (int)(at / tiles), h = hg / a.G, g = hg % a.G;
        const uint32_t tile = (uint32_t)(at - (int64_t)hg * tiles);
        const bool is_words = tile < word_tiles;
        const uint32_t row0 = (is_words ? tile : tile - word_tiles) * L::kRows, count = (is_words ? a.words : a.rows) - row0;
        // element of the input and of the output where a row starts
        auto word_at = [&](uint32_t r) { return ((((int64_t)h * a.S + r / a.K) * a.G + g) * a.K + r % a.K) * DSUB; };
        auto row_in = [&](uint32_t r) { return (int64_t)(r / a.T) * a.sxb + (int64_t)h * a.sxh + (int64_t)(r % a.T) * a.sxt + (int64_t)g * DSUB; };
        auto row_out = [&](uint32_t r) { return (((int64_t)(r / a.T) * a.H + h) * a.T + r % a.T) * a.D + (int64_t)g * DSUB; };
        __syncthreads();  // the previous tile is read
        if (hg != have) {
            // four columns of a row of W per thread, neighbouring threads in neighbouring rows: the transposed stores miss each
            // other's banks
            const float *w = a.whitener + (int64_t)hg * DSUB * DSUB;
            for (int e = tid; e < DSUB * DSUB / 4; e += kWideThreads) {
                const int i = e % DSUB, j = (e / DSUB) * 4;
                const float4 v = __ldg(reinterpret_cast<const float4 *>(w + i * DSUB + j));
                wt[j * L::kWStride + i] = v.x;
                wt[(j + 1) * L::kWStride + i] = v.y;
                wt[(j + 2) * L::kWStride + i] = v.z;
                wt[(j + 3) * L::kWStride + i] = v.w;
            }
            have = hg;
        }
        auto bring = [&](const auto *src, uint32_t r, int j, int vec_ok) {
            using T = std::remove_cv_t<std::remove_pointer_t<decltype(src)>>;
            float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            if (r < count) {
                if (!vec_ok) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = to_float<T>(src[i]);
                } else if constexpr (sizeof(T) == 2) {
                    const uint4 raw = __ldg(reinterpret_cast<const uint4 *>(src));
                    const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __half22float2(h2[i]);
                        v[2 * i] = f.x, v[2 * i + 1] = f.y;
                    }
                } else {
                    *reinterpret_cast<float4 *>(v) = __ldg(reinterpret_cast<const float4 *>(src));
                    *reinterpret_cast<float4 *>(v + 4) = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                }
            }
            *reinterpret_cast<float4 *>(xs + r * DSUB + j) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4 *>(xs + r * DSUB + j + 4) = make_float4(v[4], v[5], v[6], v[7]);
        };
#pragma unroll
        for (int e = tid; e < L::kRows * DSUB / 8; e += kWideThreads) {
            const uint32_t r = e / (DSUB / 8);
            const int j = (e % (DSUB / 8)) * 8;
            if (is_words) bring(a.tables + word_at(row0 + r) + j, r, j, a.vec_words);
            else bring(reinterpret_cast<const XT *>(a.x) + row_in(row0 + r) + j, r, j, a.vec_rows);
        }
        __syncthreads();
        float acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) acc[r][ii] = 0.0f;
#pragma unroll 2
        for (int j4 = 0; j4 < DSUB; j4 += 4) {
            float4 wv[4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) wv[jj] = *reinterpret_cast<const float4 *>(wt + (j4 + jj) * L::kWStride + i0);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float4 xv = *reinterpret_cast<const float4 *>(xs + (rg + r * L::kRowGroups) * DSUB + j4);
                const float xj[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {  // j ascending for every output: the chain order of the scalar form
                    acc[r][0] = __fmaf_rn(wv[jj].x, xj[jj], acc[r][0]);
                    acc[r][1] = __fmaf_rn(wv[jj].y, xj[jj], acc[r][1]);
                    acc[r][2] = __fmaf_rn(wv[jj].z, xj[jj], acc[r][2]);
                    acc[r][3] = __fmaf_rn(wv[jj].w, xj[jj], acc[r][3]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t own = rg + r * L::kRowGroups, row = row0 + own;
            if (own < count) {
                float *to = is_words ? a.out_tables + word_at(row) : a.out_rows + row_out(row);
                *reinterpret_cast<float4 *>(to + i0) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
            }
        }
    }
}

// Rows a thread: what finishes first when the tiles go round two blocks an SM.  A tile costs its multiply-adds, or the wider of the
// shared-memory loads, which four rows a thread do not make up for; a turn more costs a copy.  Units of 128 x 4 multiply-adds an SM.  (Eight everywhere, 2048 rows and 4096 words of 8 heads: three
// turns of 64 rows instead of three of 56.)
template <int DSUB>
static int wide_rows_a_thread(const WideArgs &a) {
    int best = 8;
    int64_t least = -1;
    for (const int r : {8, 7, 6, 4}) {
        const int64_t tile = r * (kWideThreads / (DSUB / 4)), tiles = (a.words + tile - 1) / tile + (a.rows + tile - 1) / tile;
        const int64_t turns = (tiles * a.H * a.G + kWideBlocks - 1) / kWideBlocks;
        const int64_t cost = turns * ((4 * r > 16 + r ? 4 * r : 16 + r) + 2);
        if (least < 0 || cost < least) least = cost, best = r;
    }
    return best;
}

template <int DSUB, typename XT, int R>
static int launch_wide(const WideArgs &a, cudaStream_t stream) {
    using L = WideLayout<DSUB, R>;
    auto kernel = whiten_wide_kernel<DSUB, XT, R>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::kBytes);
    if (e != cudaSuccess) return (int)e;
    const int64_t tiles = (int64_t)a.H * a.G * ((a.words + L::kRows - 1) / L::kRows + (a.rows + L::kRows - 1) / L::kRows);
    kernel<<<(unsigned)(tiles < kWideBlocks ? tiles : kWideBlocks), kWideThreads, L::kBytes, stream>>>(a);
    return launch_status();
}

template <int DSUB, typename XT>
static int whiten_wide(const WideArgs &a, cudaStream_t stream) {
    switch (wide_rows_a_thread<DSUB>(a)) {
        case 4: return launch_wide<DSUB, XT, 4>(a, stream);
        case 6: return launch_wide<DSUB, XT, 6>(a, stream);
        case 7: return launch_wide<DSUB, XT, 7>(a, stream);
        default: return launch_wide<DSUB, XT, 8>(a, stream);
    }
}

int whiten_dispatch(const void *x, int x_dtype, int64_t sxb, int64_t sxh, int64_t sxt, const __half *tables,
                    const float *whitener, float *search_tables, float *search_rows, int B, int H, int T, int D, int G,
                    int S, int K, cudaStream_t stream) {
    const int d = D / G;
    // the tiled kernels read rows and matrices in 16-byte pieces
    const bool aligned = (((uintptr_t)search_rows | (uintptr_t)search_tables | (uintptr_t)whitener) & 15) == 0;
    if (aligned && (d == 128 || d == 64 || d == 32) && (int64_t)B * T <= 0x7fffffff) {
        const int per_vec = x_dtype == TACVQ_F16 ? 8 : 4;
        const int vec_rows = ((uintptr_t)x & 15) == 0 && sxb % per_vec == 0 && sxh % per_vec == 0 && sxt % per_vec == 0;
        const WideArgs a = {x, tables, whitener, search_tables, search_rows, sxb, sxh, sxt, (uint32_t)((int64_t)B * T), (uint32_t)(S * K),
                            H, T, D, G, S, K, vec_rows, ((uintptr_t)tables & 15) == 0};
        const bool half = x_dtype == TACVQ_F16;
        if (d == 128) return half ? whiten_wide<128, __half>(a, stream) : whiten_wide<128, float>(a, stream);
        if (d == 64) return half ? whiten_wide<64, __half>(a, stream) : whiten_wide<64, float>(a, stream);
        return half ? whiten_wide<32, __half>(a, stream) : whiten_wide<32, float>(a, stream);
    }
    const int64_t tt = (int64_t)H * S * G * K * d;
    int64_t blocks = (tt + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    whiten_tables_kernel<<<(unsigned)blocks, 256, 0, stream>>>(tables, whitener, search_tables, H, S, G, K, d);
    int st = launch_status();
    if (st != TACVQ_OK) return st;
    const int64_t rt = (int64_t)B * H * T * D;
    blocks = (rt + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    if (x_dtype == TACVQ_F16)
        whiten_rows_kernel<__half><<<(unsigned)blocks, 256, 0, stream>>>((const __half *)x, sxb, sxh, sxt, whitener, search_rows, B, H, T, D, G);
    else
        whiten_rows_kernel<float><<<(unsigned)blocks, 256, 0, stream>>>((const float *)x, sxb, sxh, sxt, whitener, search_rows, B, H, T, D, G);
    return launch_status();
}

// Transformed words (d a multiple of 32) for a search that filters on the tensor core: their fp16 rounding, and |word|^2 in
// the library's order, eight neighbouring lanes per word (lane j owns running sum j of each of the four sets).
__global__ void __launch_bounds__(256)
round_words_kernel(const float *__restrict__ words32, __half *__restrict__ words16, float *__restrict__ norms, int64_t words, int d) {
    const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, j = lane & 7;
    const int64_t word = slot >> 3;
    const int64_t at = (word < words ? word : words - 1) * d;  // spare lanes redo the last word
    float set[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int i = 0; i < d; i += 32) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float v = words32[at + i + 8 * u + j];
            if (word < words) words16[at + i + 8 * u + j] = __float2half_rn(v);
            set[u] = __fadd_rn(set[u], __fmul_rn(v, v));
        }
    }
    const float mine = __fadd_rn(__fadd_rn(__fadd_rn(set[0], set[1]), set[2]), set[3]);
    const int first = lane & 24;
    float total = __shfl_sync(0xffffffffu, mine, first);
#pragma unroll
    for (int k = 1; k < 8; ++k) total = __fadd_rn(total, __shfl_sync(0xffffffffu, mine, first + k));
    if (j == 0 && word < words) norms[word] = total;
}

int round_words_dispatch(const float *words32, __half *words16, float *norms, int64_t words, int d, cudaStream_t stream) {
    round_words_kernel<<<(unsigned)((words * 8 + 255) / 256), 256, 0, stream>>>(words32, words16, norms, words, d);
    return launch_status();
}

}  // namespace tacvq
