// Encode for 32-wide groups (fp16 tables): tensor cores filter, exact fp32 decides.
//
// Same idea as the 8-wide kernel in encode_tc.cu, shaped as a block-level GEMM.  A block owns 128
// rows of one (head, group).  Per stage it
//   1. keeps, next to the fp32 residual tile, its fp16 rounding in shared memory,
//   2. scores all 128 x 256 (row, word) pairs with mma.sync.m16n8k16 (ldmatrix fragments), each of 16 warps owning
//      32 rows x 64 words, the accumulators seeded with -|c|^2/2; a score is t = r.c - |c|^2/2 and the
//      distance is |r|^2 - 2t,
//   3. takes the row maxima over the four word quarters and lists every pair whose score lies within
//      a margin of its row's maximum,
//   4. re-evaluates the listed pairs in the library's exact fp32 order (one d-step FMA chain each,
//      one pair per thread) and keeps the lowest (distance, index) per row with a 64-bit shared atomicMin,
//   5. subtracts the chosen words from the fp32 residual tile and refreshes the fp16 copy.
// 64- and 128-wide groups have encode_wide.cu.
//
// Margin (see encode_tc.cu for the argument that a margin of twice the error bound keeps the exact
// argmin and everything tied with it on the list).  The fp16 rounding of the residual changes a dot
// product by at most 2^-11 sum |r_i c_i| <= 2^-11 |r| |c|; the tensor core's fp32 accumulation of the
// exact products, the exact chain's own roundings and the roundings of the distance expression add at
// most about 2^-17 (|r|^2 + |c|^2).  In units of t the kernel allows
//   1.25 * 2^-10 |r| max|c|  +  2^-14 (|r|^2 + max|c|^2)  +  2^-18 max|c|   (fp16 subnormals).
// On Gaussian data that lists about 1.07 words per row.  If the list overflows, or a residual is too
// large for fp16, the block re-evaluates every pair of that stage: slow, still exact.
//
// Reference statements: src/jointkv/closed_loop_vq.py:52-76 (search), :343-395 (stage recursion).

#include "common.cuh"

namespace tacvq {

namespace {

constexpr int kRows = 128;     // rows per block
constexpr int kThreads = 512;  // 16 warps = 4 row blocks of 32 x 4 word quarters of 64
constexpr int kListCap = 2048;

template <int DSUB>
struct TcLargeLayout {
    static constexpr int kHalfStride = DSUB + 8;  // halves: 16-byte rows that land on distinct banks for ldmatrix
    static constexpr int kResStride = DSUB + 4;   // floats
    static constexpr size_t kTab = 0;                                              // [256][kHalfStride] half
    static constexpr size_t kHi = kTab + (size_t)kMaxWords * kHalfStride * 2;      // [kRows][kHalfStride] half
    static constexpr size_t kRes = kHi + (size_t)kRows * kHalfStride * 2;          // [kRows][kResStride] float
    static constexpr size_t kNrm = kRes + (size_t)kRows * kResStride * 4;          // [256] float
    static constexpr size_t kSeed = kNrm + kMaxWords * 4;                          // [256] float: -|c|^2/2
    static constexpr size_t kXx = kSeed + kMaxWords * 4;                           // [kRows] float
    static constexpr size_t kRowMax = kXx + kRows * 4;                             // [4][kRows] float
    static constexpr size_t kThr = kRowMax + 4 * kRows * 4;                        // [kRows] float
    static constexpr size_t kBest = kThr + kRows * 4;                              // [kRows] u64
    static constexpr size_t kList = kBest + kRows * 8;                             // [kListCap] u16
    static constexpr size_t kMisc = kList + kListCap * 2;                          // count, big flag, cc_max
    static constexpr size_t kRowCnt = kMisc + 32;                                  // [kRows] int: listed words per row
    static constexpr size_t kHist = kRowCnt + kRows * 4;                           // [kRows][S] u8
    static constexpr size_t bytes(int S) { return kHist + (size_t)kRows * S; }
    // half index of element e of word k / of row r
    __device__ static __forceinline__ int tab_at(int k, int e) {
        return k * kHalfStride + e;
    }
    __device__ static __forceinline__ int hi_at(int r, int e) {
        return r * kHalfStride + e;
    }
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void *smem_ptr) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(smem_ptr);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

__device__ __forceinline__ void mma_acc_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// monotone map float -> uint32 (total order of the values, -0 below +0)
__device__ __forceinline__ uint32_t ordered_bits(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// |v|^2 of a d-vector (d a multiple of 32) by eight neighbouring lanes, in the library's order
// (four sets of eight running sums: element i goes to set (i/8)%4, sum i%8; per sum the sets are added
// ((0+1)+2)+3; the eight sums are added 0..7).  Lane j of the group owns sum j.  All eight return the total.
template <int DSUB, typename Load>
__device__ __forceinline__ float group8_sqnorm_ordered(Load at, int lane) {
    const int j = lane & 7;
    float set[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < DSUB; i += 8) {
        const float v = at(i + j);
        set[(i >> 3) & 3] = __fadd_rn(set[(i >> 3) & 3], __fmul_rn(v, v));
    }
    const float mine = __fadd_rn(__fadd_rn(__fadd_rn(set[0], set[1]), set[2]), set[3]);
    const int first = lane & 24;
    float total = __shfl_sync(0xffffffffu, mine, first);
#pragma unroll
    for (int k = 1; k < 8; ++k) total = __fadd_rn(total, __shfl_sync(0xffffffffu, mine, first + k));
    return total;
}

// four consecutive residual elements -> fp32 tile and its fp16 rounding; returns max |element|
__device__ __forceinline__ float store_residual4(float *res_at, __half *hi_at, const float4 v) {
    *reinterpret_cast<float4 *>(res_at) = v;
    __half2 h[2] = {__floats2half2_rn(v.x, v.y), __floats2half2_rn(v.z, v.w)};
    *reinterpret_cast<uint2 *>(hi_at) = *reinterpret_cast<const uint2 *>(h);
    return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
}

template <typename XT>
__device__ __forceinline__ float4 load4(const XT *src, bool vec);
template <>
__device__ __forceinline__ float4 load4<float>(const float *src, bool vec) {
    if (vec) return *reinterpret_cast<const float4 *>(src);
    return make_float4(src[0], src[1], src[2], src[3]);
}
template <>
__device__ __forceinline__ float4 load4<__half>(const __half *src, bool vec) {
    __half2 h[2];
    if (vec) {
        *reinterpret_cast<uint2 *>(h) = *reinterpret_cast<const uint2 *>(src);
    } else {
        h[0] = __halves2half2(src[0], src[1]);
        h[1] = __halves2half2(src[2], src[3]);
    }
    const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
    return make_float4(a.x, a.y, b.x, b.y);
}

}  // namespace

template <int DSUB, typename XT>
__global__ void __launch_bounds__(kThreads, 1)
encode_tc_large_kernel(const XT *__restrict__ x, int64_t sxb, int64_t sxh, int64_t sxt, const __half *__restrict__ tables,
                       const float *__restrict__ sqnorm_in, uint8_t *__restrict__ codes, void *__restrict__ recon,
                       int recon_dtype, int B, int H, int T, int G, int S, int K, int64_t t0, int64_t T_cap, int vec_ok) {
    using L = TcLargeLayout<DSUB>;
    constexpr int RS = L::kResStride;
    constexpr int kChunks = DSUB / 8;  // threads per row: each owns elements [4c, 4c+4) and [d/2 + 4c, d/2 + 4c + 4)
    constexpr int kPass = kThreads / kChunks;  // rows per pass over the tile
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half *tab = reinterpret_cast<__half *>(smem_raw + L::kTab);
    __half *hi = reinterpret_cast<__half *>(smem_raw + L::kHi);
    float *res = reinterpret_cast<float *>(smem_raw + L::kRes);
    float *nrm = reinterpret_cast<float *>(smem_raw + L::kNrm);
    float *seed = reinterpret_cast<float *>(smem_raw + L::kSeed);
    float *xxs = reinterpret_cast<float *>(smem_raw + L::kXx);
    float *rowmax = reinterpret_cast<float *>(smem_raw + L::kRowMax);
    float *thr = reinterpret_cast<float *>(smem_raw + L::kThr);
    unsigned long long *best = reinterpret_cast<unsigned long long *>(smem_raw + L::kBest);
    uint16_t *list = reinterpret_cast<uint16_t *>(smem_raw + L::kList);
    int *count = reinterpret_cast<int *>(smem_raw + L::kMisc);
    int *big = count + 1;  // some residual element of the coming stage does not fit fp16
    float *cc_max = reinterpret_cast<float *>(count + 2);
    int *rowcnt = reinterpret_cast<int *>(smem_raw + L::kRowCnt);
    uint8_t *hist = smem_raw + L::kHist;

    const int hg = blockIdx.y;
    const int h = hg / G, g = hg % G;
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, q = lane & 3;
    // row block (32 rows), word quarter (64 words)
    const int wr = warp >> 2, wq = warp & 3;
    const uint32_t rows = (uint32_t)B * (uint32_t)T;  // the launcher keeps B*T below 2^31
    const uint32_t tile = blockIdx.x * kRows;
    const int my_c = tid % kChunks, my_r = tid / kChunks;  // this thread's piece column and first row
    const float inf = __int_as_float(0x7f800000);

    uint8_t *code_at = nullptr;  // this row's first code byte (threads 0..kRows-1)
    if (tid < kRows && tile + tid < rows) {
        const uint32_t row = tile + tid;
        const uint32_t b = row / (uint32_t)T, t = row % (uint32_t)T;
        code_at = codes + (((int64_t)b * H + h) * T_cap + t0 + t) * ((int64_t)S * G) + g;
    }
    if (tid == 0) *big = 0;
    __syncthreads();
#pragma unroll
    for (int r = my_r; r < kRows; r += kPass) {
        const uint32_t row = tile + r;
        float4 v0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v1 = v0;
        if (row < rows) {
            const uint32_t b = row / (uint32_t)T, t = row % (uint32_t)T;
            const XT *src = x + (int64_t)b * sxb + (int64_t)h * sxh + (int64_t)t * sxt + (int64_t)g * DSUB + 4 * my_c;
            v0 = load4<XT>(src, vec_ok != 0);
            v1 = load4<XT>(src + DSUB / 2, vec_ok != 0);
        }
        const float top0 = store_residual4(res + r * RS + 4 * my_c, hi + L::hi_at(r, 4 * my_c), v0);
        const float top1 = store_residual4(res + r * RS + DSUB / 2 + 4 * my_c, hi + L::hi_at(r, DSUB / 2 + 4 * my_c), v1);
        if (!(fmaxf(top0, top1) < 32768.0f)) *big = 1;
    }

    for (int s = 0; s < S; ++s) {
        __syncthreads();  // residual tiles settled; the previous stage's table is no longer read
        const __half *src = tables + (((int64_t)h * S + s) * G + g) * (int64_t)K * DSUB;
        // caller-supplied word norms: fetched by the upper half of the block while the table is copied
        const int norm_k = tid - (kThreads - kMaxWords);
        float norm_v = inf;
        if (sqnorm_in != nullptr && norm_k >= 0 && norm_k < K) norm_v = sqnorm_in[(((int64_t)h * S + s) * G + g) * K + norm_k];
        if (tid == 0) {
            *count = 0;
            *cc_max = 0.0f;
        }
        for (int idx = tid; idx < kMaxWords * kChunks; idx += kThreads) {
            const int k = idx / kChunks, c = idx % kChunks;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (k < K) v = *reinterpret_cast<const uint4 *>(src + (int64_t)k * DSUB + c * 8);
            *reinterpret_cast<uint4 *>(tab + L::tab_at(k, c * 8)) = v;
        }
        __syncthreads();
        // |c|^2 per word and |r|^2 per row, eight lanes per vector (four vectors per warp and trip, placed so
        // that their loads miss each other's banks).  The largest |c|^2 is gathered with an integer atomic
        // maximum (non-negative floats order like their bit patterns).
        {
            float top = 0.0f;
            if (sqnorm_in == nullptr) {
#pragma unroll
                for (int it = 0; it < 4; ++it) {
                    const int k = warp * 16 + it * 4 + (lane >> 3);
                    float v = group8_sqnorm_ordered<DSUB>([&](int i) { return __half2float(tab[L::tab_at(k, i)]); }, lane);
                    if (k >= K) v = inf;  // padding words can never be chosen
                    else if (v == v) top = fmaxf(top, v);
                    if ((lane & 7) == 0) {
                        nrm[k] = v;
                        seed[k] = -0.5f * v;
                    }
                }
            } else if (norm_k >= 0) {
                nrm[norm_k] = norm_v;
                seed[norm_k] = -0.5f * norm_v;
                if (norm_k < K && norm_v == norm_v) top = norm_v;
            }
            if (sqnorm_in == nullptr || norm_k >= 0) {  // warp-uniform
#pragma unroll
                for (int off = 16; off >= 1; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
                if (lane == 0) atomicMax(reinterpret_cast<int *>(cc_max), __float_as_int(top));
            }
        }
        // Row norms in 32 trips of 4 rows.
        for (int trip = warp; trip < 32; trip += 16) {
            const int r = (trip >> 1) * 8 + (trip & 1) + 2 * (lane >> 3);
            const float v = group8_sqnorm_ordered<DSUB>([&](int i) { return res[r * RS + i]; }, lane);
            if ((lane & 7) == 0) {
                xxs[r] = v;
                best[r] = ~0ull;
                rowcnt[r] = 0;
            }
        }
        __syncthreads();

        // ---- approximate scores: 32 rows x 64 words per warp --------------------------------------
        float acc[2][8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const float2 sv = *reinterpret_cast<const float2 *>(seed + wq * 64 + n * 8 + 2 * q);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                acc[m][n][0] = sv.x;
                acc[m][n][1] = sv.y;
                acc[m][n][2] = sv.x;
                acc[m][n][3] = sv.y;
            }
        }
        {
            // ldmatrix lane addresses: A tiles are [16 rows][16 k], B tiles [16 words][16 k] (two n-tiles)
            const int a_row = wr * 32 + (lane & 15), a_col = (lane >> 4) * 8;
            const int b_row = wq * 64 + (lane & 7) + (lane >> 4) * 8, b_col = ((lane >> 3) & 1) * 8;
#pragma unroll 2
            for (int ks = 0; ks < DSUB / 16; ++ks) {
                uint32_t a[2][4];
#pragma unroll
                for (int m = 0; m < 2; ++m) ldmatrix_x4(a[m], hi + L::hi_at(a_row + m * 16, ks * 16 + a_col));
#pragma unroll
                for (int np = 0; np < 4; ++np) {
                    uint32_t bw[4];
                    ldmatrix_x4(bw, tab + L::tab_at(b_row + np * 16, ks * 16 + b_col));
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        mma_acc_16816(acc[m][2 * np], a[m], bw[0], bw[1]);
                        mma_acc_16816(acc[m][2 * np + 1], a[m], bw[2], bw[3]);
                    }
                }
            }
        }
        // row maxima over this warp's 64 words
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float top = fmaxf(acc[m][0][2 * half], acc[m][0][2 * half + 1]);
#pragma unroll
                for (int n = 1; n < 8; ++n) top = fmaxf(top, fmaxf(acc[m][n][2 * half], acc[m][n][2 * half + 1]));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
                top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
                if (q == 0) rowmax[wq * kRows + wr * 32 + m * 16 + half * 8 + gid] = top;
            }
        }
        __syncthreads();
        if (tid < kRows) {
            const float top = fmaxf(fmaxf(rowmax[tid], rowmax[kRows + tid]), fmaxf(rowmax[2 * kRows + tid], rowmax[3 * kRows + tid]));
            const float cm = *cc_max, xx = xxs[tid];
            const float margin = 1.220703125e-03f * sqrtf(xx * cm) + 6.103515625e-05f * (xx + cm) + 3.814697265625e-06f * sqrtf(cm);
            thr[tid] = (*big != 0) ? -inf : top - margin;
        }
        __syncthreads();
        if (tid == 0) *big = 0;  // read above; the update below raises it for the next stage
        // List the pairs within the margin.  Per row a thread shifts the sign of (score - limit) of its
        // 16 words into a word (first word ends at bit 15, set = below the limit); one atomic per warp
        // reserves the slots, then each thread walks its set bits.
        {
            uint32_t pass[2][2];
            int hits = 0;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float limit = thr[wr * 32 + m * 16 + half * 8 + gid];
                    uint32_t fail = 0u;
#pragma unroll
                    for (int n = 0; n < 8; ++n) {
                        fail = __funnelshift_l(__float_as_uint(acc[m][n][2 * half] - limit), fail, 1);
                        fail = __funnelshift_l(__float_as_uint(acc[m][n][2 * half + 1] - limit), fail, 1);
                    }
                    pass[m][half] = ~fail & 0xffffu;
                    hits += __popc(pass[m][half]);
                }
            }
            int before = hits;  // inclusive prefix over the warp
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, before, off);
                if (lane >= off) before += up;
            }
            int base = 0;
            if (lane == 31 && before > 0) base = atomicAdd(count, before);
            base = __shfl_sync(0xffffffffu, base, 31);
            int slot = base + before - hits;
#pragma unroll
            for (int m = 0; m < 2; ++m) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    uint32_t todo = pass[m][half];
                    const int r = wr * 32 + m * 16 + half * 8 + gid;
                    while (todo != 0u) {
                        const int bit = 31 - __clz(todo);
                        todo &= ~(1u << bit);
                        const int pos = 15 - bit;  // n * 2 + e
                        if (slot < kListCap) list[slot] = (uint16_t)((r << 8) | (wq * 64 + (pos >> 1) * 8 + 2 * q + (pos & 1)));
                        ++slot;
                        atomicAdd(rowcnt + r, 1);
                    }
                }
            }
        }
        __syncthreads();
        // ---- exact re-evaluation ------------------------------------------------------------------
        {
            const int listed = *count;
            const bool everything = listed > kListCap;
            const int work = everything ? kRows * K : listed;
            for (int i = tid; i < work; i += kThreads) {
                int r, k;
                if (everything) {
                    r = i / K, k = i % K;
                } else {
                    const int entry = list[i];
                    r = entry >> 8, k = entry & 255;
                }
                if (k >= K) continue;
                if (!everything && rowcnt[r] == 1) {  // the only word within the margin is the argmin
                    best[r] = (unsigned long long)k;
                    continue;
                }
                const float *rv = res + r * RS;
                float dot = 0.0f;
#pragma unroll 8
                for (int i8 = 0; i8 < DSUB; i8 += 8) {
                    const uint4 cw = *reinterpret_cast<const uint4 *>(tab + L::tab_at(k, i8));
                    const __half2 *c2 = reinterpret_cast<const __half2 *>(&cw);
                    const float4 r0 = *reinterpret_cast<const float4 *>(rv + i8);
                    const float4 r1 = *reinterpret_cast<const float4 *>(rv + i8 + 4);
                    float2 c;
                    c = __half22float2(c2[0]);
                    dot = __fmaf_rn(r0.x, c.x, dot);
                    dot = __fmaf_rn(r0.y, c.y, dot);
                    c = __half22float2(c2[1]);
                    dot = __fmaf_rn(r0.z, c.x, dot);
                    dot = __fmaf_rn(r0.w, c.y, dot);
                    c = __half22float2(c2[2]);
                    dot = __fmaf_rn(r1.x, c.x, dot);
                    dot = __fmaf_rn(r1.y, c.y, dot);
                    c = __half22float2(c2[3]);
                    dot = __fmaf_rn(r1.z, c.x, dot);
                    dot = __fmaf_rn(r1.w, c.y, dot);
                }
                const float dist = distance_expr(xxs[r], nrm[k], dot);
                if (dist < inf) {  // an infinite or NaN distance never wins, as in a strict '<' scan
                    const unsigned long long key = ((unsigned long long)ordered_bits(dist) << 32) | (unsigned)k;
                    atomicMin(best + r, key);
                }
            }
        }
        __syncthreads();
        // ---- update: subtract the chosen words, refresh the fp16 copy -------------------------------
#pragma unroll
        for (int r = my_r; r < kRows; r += kPass) {
            const unsigned long long key = best[r];
            const int pick = (key == ~0ull) ? 0 : (int)(key & 0xffffffffull);
            float top = 0.0f;
#pragma unroll
            for (int piece = 0; piece < 2; ++piece) {
                const int at = piece * (DSUB / 2) + 4 * my_c;
                __half2 c2[2];
                *reinterpret_cast<uint2 *>(c2) = *reinterpret_cast<const uint2 *>(tab + L::tab_at(pick, at));
                const float4 rv = *reinterpret_cast<const float4 *>(res + r * RS + at);
                const float2 w0 = __half22float2(c2[0]), w1 = __half22float2(c2[1]);
                const float4 nv = make_float4(__fsub_rn(rv.x, w0.x), __fsub_rn(rv.y, w0.y), __fsub_rn(rv.z, w1.x), __fsub_rn(rv.w, w1.y));
                top = fmaxf(top, store_residual4(res + r * RS + at, hi + L::hi_at(r, at), nv));
            }
            if (!(top < 32768.0f)) *big = 1;
        }
        if (tid < kRows) {
            const unsigned long long key = best[tid];
            const int pick = (key == ~0ull) ? 0 : (int)(key & 0xffffffffull);
            hist[tid * S + s] = (uint8_t)pick;
            if (code_at != nullptr) code_at[(int64_t)s * G] = (uint8_t)pick;
        }
    }

    if (recon != nullptr) {
        __syncthreads();
        // stage loop outermost: the gathers of a stage (this thread's rows and pieces) travel together
        constexpr int kMine = kRows / kPass;
        float4 sum[kMine][2];
#pragma unroll
        for (int i = 0; i < kMine; ++i) sum[i][0] = sum[i][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const __half *words = tables + ((int64_t)h * S * G + g) * (int64_t)K * DSUB + 4 * my_c;
        const int64_t stage_words = (int64_t)G * K * DSUB;
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
            uint2 raw[kMine][2];
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
                const __half *word = words + s * stage_words + (int64_t)hist[(my_r + i * kPass) * S + s] * DSUB;
                raw[i][0] = *reinterpret_cast<const uint2 *>(word);
                raw[i][1] = *reinterpret_cast<const uint2 *>(word + DSUB / 2);
            }
#pragma unroll
            for (int i = 0; i < kMine; ++i) {
#pragma unroll
                for (int piece = 0; piece < 2; ++piece) {
                    const __half2 *c2 = reinterpret_cast<const __half2 *>(&raw[i][piece]);
                    const float2 w0 = __half22float2(c2[0]), w1 = __half22float2(c2[1]);
                    float4 &acc = sum[i][piece];
                    acc = make_float4(__fadd_rn(acc.x, w0.x), __fadd_rn(acc.y, w0.y), __fadd_rn(acc.z, w1.x), __fadd_rn(acc.w, w1.y));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
            const uint32_t row = tile + my_r + i * kPass;
            if (row >= rows) continue;
            const uint32_t b = row / (uint32_t)T, t = row % (uint32_t)T;
#pragma unroll
            for (int piece = 0; piece < 2; ++piece) {
                const int at = piece * (DSUB / 2) + 4 * my_c;
                const int64_t o = (((int64_t)b * H + h) * T + t) * ((int64_t)G * DSUB) + (int64_t)g * DSUB + at;
                if (recon_dtype == TACVQ_F16) {
                    __half2 out[2] = {__floats2half2_rn(sum[i][piece].x, sum[i][piece].y), __floats2half2_rn(sum[i][piece].z, sum[i][piece].w)};
                    *reinterpret_cast<uint2 *>((__half *)recon + o) = *reinterpret_cast<const uint2 *>(out);
                } else {
                    *reinterpret_cast<float4 *>((float *)recon + o) = sum[i][piece];
                }
            }
        }
    }
}

// Returns TACVQ_ERR_UNSUPPORTED when the geometry is not this kernel's, so the caller can go on to
// the scalar kernels.
int encode_tc_large_launch(const EncodeArgs &a) {
    if (a.tables_f32 || a.K > kMaxWords || a.D / a.G != 32) return TACVQ_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(a.tables) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    constexpr int DSUB = 32;
    const size_t smem = TcLargeLayout<DSUB>::bytes(a.S);
    if (smem > 227 * 1024) return TACVQ_ERR_UNSUPPORTED;
    const int64_t rows = (int64_t)a.B * a.T;
    if (rows >= (int64_t)1 << 31) return TACVQ_ERR_UNSUPPORTED;
    if (a.recon != nullptr && (reinterpret_cast<uintptr_t>(a.recon) & 15u) != 0) return TACVQ_ERR_UNSUPPORTED;
    // 4-element vector loads of the states need an aligned base and strides that keep the alignment
    const size_t elem = a.x_dtype == TACVQ_F16 ? 2 : 4;
    const int vec_ok = (reinterpret_cast<uintptr_t>(a.x) % (4 * elem) == 0 && a.sxb % 4 == 0 && a.sxh % 4 == 0 && a.sxt % 4 == 0) ? 1 : 0;
    dim3 grid((unsigned)((rows + kRows - 1) / kRows), (unsigned)(a.H * a.G));
    auto launch = [&](auto kernel, auto *xp) -> int {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        kernel<<<grid, kThreads, smem, a.stream>>>(xp, a.sxb, a.sxh, a.sxt, (const __half *)a.tables, a.sqnorm, a.codes,
                                                   a.recon, a.recon_dtype, a.B, a.H, a.T, a.G, a.S, a.K, a.t0, a.T_cap, vec_ok);
        return launch_status();
    };
    if (a.x_dtype == TACVQ_F16) return launch(encode_tc_large_kernel<DSUB, __half>, (const __half *)a.x);
    return launch(encode_tc_large_kernel<DSUB, float>, (const float *)a.x);
}

}  // namespace tacvq
