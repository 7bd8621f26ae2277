// Attention over stored codes - geometry-generic kernel and the log-sum-exp merge.
//
// One block serves one (batch row, KV head, sequence split).  It first builds, for each of the
// REP query heads that share the KV head, a look-up table lut[r][code][slot] = q_r[group] . word
// (slot = stage*G + group), then scans its token range one token per warp step:
//     score_r = sum_slot lut[r][kcode[slot]][slot]            (lane = slot, warp reduction)
//     online softmax (running max m_r, sum l_r)
//     acc_r  += exp(score_r - m_r) * V_row                      (lane owns D/32 channels; the V row is
//                                                               rebuilt from its codes exactly as the
//                                                               reference stores it: fp32 stage sum
//                                                               rounded once to fp16)
// and finally merges its warps' states into one partial state per split.  A second kernel merges
// the splits.  This kernel is the fallback for every geometry; the (G=16,S=2,d=8) benchmark
// geometry has a specialised kernel in attn_gsrq.cu.
//
// Semantics replaced: experiments_followup_mistral/evaluate_mistral_longbench.py:112-122
// (dequantised window -> repeat_kv -> softmax(q K^T) V), without the rotary step.

#include "common.cuh"

namespace tacvq {

constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = kAttnThreads / 32;

template <int REP, int DPL>
__global__ void __launch_bounds__(kAttnThreads)
attn_generic_kernel(const __half *__restrict__ q, const uint8_t *__restrict__ kcodes,
                    const uint8_t *__restrict__ vcodes, const __half *__restrict__ ktab,
                    const __half *__restrict__ vtab, const int32_t *__restrict__ seq_start,
                    const int32_t *__restrict__ seq_end, float *__restrict__ part, int B, int Hq, int Hkv, int D, int G,
                    int S, int K, int64_t T_cap, int splits) {
    extern __shared__ __align__(16) float smem[];
    const int slots = S * G;
    const int d = D / G;
    float *lut = smem;  // [REP][K][slots]

    const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    // ---- look-up tables -------------------------------------------------------------------------
    for (int idx = tid; idx < slots * K; idx += kAttnThreads) {
        const int slot = idx % slots, k = idx / slots;  // slot fastest: conflict-free table writes
        const int s = slot / G, g = slot % G;
        const __half *w = ktab + ((((int64_t)h * S + s) * G + g) * K + k) * d;
        float dot[REP];
#pragma unroll
        for (int r = 0; r < REP; ++r) dot[r] = 0.0f;
        for (int i = 0; i < d; ++i) {
            const float c = __half2float(w[i]);
#pragma unroll
            for (int r = 0; r < REP; ++r)
                dot[r] = fmaf(__half2float(q[((int64_t)b * Hq + h * REP + r) * D + g * d + i]), c, dot[r]);
        }
#pragma unroll
        for (int r = 0; r < REP; ++r) lut[((size_t)r * K + k) * slots + slot] = dot[r];
    }
    __syncthreads();

    // ---- token range of this split ---------------------------------------------------------------
    const int lo_all = seq_start ? seq_start[b] : 0;
    const int hi_all = seq_end ? seq_end[b] : (int)T_cap;
    const int n_all = hi_all > lo_all ? hi_all - lo_all : 0;
    const int per = (n_all + splits - 1) / splits;
    const int lo = lo_all + split * per;
    const int hi = min(lo + per, lo_all + n_all);

    float m[REP], l[REP], acc[REP][DPL];
#pragma unroll
    for (int r = 0; r < REP; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[r][i] = 0.0f;
    }
    const int c0 = lane * DPL;
    const int vg = c0 / d, vi0 = c0 % d;
    const int64_t code_row = ((int64_t)b * Hkv + h) * T_cap;

    for (int t = lo + warp; t < hi; t += kAttnWarps) {
        const uint8_t *kc = kcodes + (code_row + t) * slots;
        const uint8_t *vc = vcodes + (code_row + t) * slots;
        float sc[REP];
#pragma unroll
        for (int r = 0; r < REP; ++r) sc[r] = 0.0f;
        for (int j = lane; j < slots; j += 32) {
            const int code = kc[j];
#pragma unroll
            for (int r = 0; r < REP; ++r) sc[r] += lut[((size_t)r * K + code) * slots + j];
        }
#pragma unroll
        for (int r = 0; r < REP; ++r) {
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) sc[r] += __shfl_xor_sync(0xffffffffu, sc[r], off);
        }
        float vrow[DPL];
#pragma unroll
        for (int i = 0; i < DPL; ++i) vrow[i] = 0.0f;
        for (int s = 0; s < S; ++s) {
            const int code = vc[s * G + vg];
            const __half *w = vtab + ((((int64_t)h * S + s) * G + vg) * K + code) * d + vi0;
#pragma unroll
            for (int i = 0; i < DPL; ++i) vrow[i] = __fadd_rn(vrow[i], __half2float(__ldg(w + i)));
        }
#pragma unroll
        for (int r = 0; r < REP; ++r) {
            if (sc[r] > m[r]) {
                const float scale = __expf(m[r] - sc[r]);  // exp(-inf) = 0 on the first token
                l[r] *= scale;
#pragma unroll
                for (int i = 0; i < DPL; ++i) acc[r][i] *= scale;
                m[r] = sc[r];
            }
            const float p = __expf(sc[r] - m[r]);
            l[r] += p;
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[r][i] = fmaf(p, __half2float(__float2half_rn(vrow[i])), acc[r][i]);
        }
    }

    // ---- merge the warps of this block -----------------------------------------------------------
    __syncthreads();  // LUT no longer needed: reuse its storage
    float *wm = smem;                          // [warps][REP]
    float *wl = wm + kAttnWarps * REP;         // [warps][REP]
    float *wacc = wl + kAttnWarps * REP;       // [warps][REP][D]
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < REP; ++r) {
            wm[warp * REP + r] = m[r];
            wl[warp * REP + r] = l[r];
        }
    }
#pragma unroll
    for (int r = 0; r < REP; ++r)
#pragma unroll
        for (int i = 0; i < DPL; ++i) wacc[((size_t)warp * REP + r) * D + c0 + i] = acc[r][i];
    __syncthreads();
    const int64_t rows = (int64_t)B * Hq;
    for (int idx = tid; idx < REP * (D + 2); idx += kAttnThreads) {
        const int r = idx / (D + 2), col = idx % (D + 2);
        float top = -INFINITY;
        for (int w = 0; w < kAttnWarps; ++w) top = fmaxf(top, wm[w * REP + r]);
        float sum = 0.0f;
        if (col == 0) {
            sum = top;
        } else {
            for (int w = 0; w < kAttnWarps; ++w) {
                const float mw = wm[w * REP + r];
                if (wl[w * REP + r] == 0.0f) continue;  // no token; a sum that is NaN spoils the others
                const float scale = __expf(mw - top);
                sum += scale * (col == 1 ? wl[w * REP + r] : wacc[((size_t)w * REP + r) * D + (col - 2)]);
            }
        }
        const int64_t row = (int64_t)b * Hq + h * REP + r;
        part[((int64_t)split * rows + row) * (D + 2) + col] = sum;
    }
}

// Merge n_parts states laid out [n_parts][rows][2+D]; one block per row.  What bounds it is the memory latency of a row's
// n_parts states, so nothing walks them one after the other: the threads take a part's (m, l) each and reduce, then groups
// of 128 threads (a thread per channel) take every groups-th part, up to eight loads in flight.  Up to eight parts are requested at
// once by every thread, which then needs no other: us a merge of 32 rows of eight parts 3.6 with the reduction, 2.5 one part after the other.
constexpr int kCombineLanes = 128, kCombineGroups = 8, kCombineFew = 8;

__global__ void __launch_bounds__(kCombineLanes * kCombineGroups)
attn_combine_kernel(const float *states, int n_parts, int64_t rows, int D, __half *__restrict__ out,
                    float *__restrict__ merged) {
    __shared__ float red[2 * kCombineLanes * kCombineGroups / 32];
    __shared__ float sums[kCombineGroups * kCombineLanes];
    const int64_t row = blockIdx.x;
    const int W = D + 2;
    const int64_t stride = rows * W;
    const float *own = states + row * W;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    wait_for_previous_kernel();
    launch_dependents();  // the next kernel may be scheduled; one that follows as a dependent waits for this grid itself
    if (n_parts <= kCombineFew) {
        for (int i = tid; i < D; i += blockDim.x) {
            float m[kCombineFew], part[kCombineFew], v[kCombineFew];
#pragma unroll
            for (int p = 0; p < kCombineFew; ++p) {
                const float *from = own + (p < n_parts ? p : 0) * stride;
                m[p] = from[0], part[p] = p < n_parts ? from[1] : 0.0f, v[p] = from[2 + i];
            }
            float top = m[0], l = 0.0f, a = 0.0f;
#pragma unroll
            for (int p = 1; p < kCombineFew; ++p) top = fmaxf(top, m[p]);
#pragma unroll
            for (int p = 0; p < kCombineFew; ++p) {
                if (part[p] == 0.0f) continue;  // no token there
                const float f = __expf(m[p] - top);
                l += f * part[p];
                if (m[p] != -INFINITY) a += f * v[p];
            }
            if (merged) {
                merged[row * W + 2 + i] = a;
                if (i == 0) merged[row * W] = top, merged[row * W + 1] = l;
            }
            if (out) out[row * D + i] = __float2half_rn(l == 0.0f ? 0.0f : a / l);
        }
        return;
    }
    float top = -INFINITY;
    for (int p = tid; p < n_parts; p += blockDim.x) top = fmaxf(top, own[p * stride]);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    if (lane == 0) red[warp] = top;
    __syncthreads();
    for (int w = 0; w < warps; ++w) top = fmaxf(top, red[w]);
    float l = 0.0f;
    for (int p = tid; p < n_parts; p += blockDim.x) {
        const float part = own[p * stride + 1];
        if (part != 0.0f) l += __expf(own[p * stride] - top) * part;  // 0: no token there
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    if (lane == 0) red[warps + warp] = l;
    __syncthreads();
    l = 0.0f;
    for (int w = 0; w < warps; ++w) l += red[warps + w];
    const int group = tid / kCombineLanes, groups = blockDim.x / kCombineLanes, at = tid % kCombineLanes;
    for (int base = 0; base < D; base += kCombineLanes) {
        const int i = base + at;
        float a = 0.0f;
        if (i < D) {
#pragma unroll 8
            for (int p = group; p < n_parts; p += groups) {
                const float m = own[p * stride], v = own[p * stride + 2 + i];
                if (m != -INFINITY) a += __expf(m - top) * v;
            }
        }
        sums[group * kCombineLanes + at] = a;
        __syncthreads();
        if (group == 0 && i < D) {
            for (int g = 1; g < groups; ++g) a += sums[g * kCombineLanes + at];
            if (merged) merged[row * W + 2 + i] = a;
            if (out) out[row * D + i] = __float2half_rn(l == 0.0f ? 0.0f : a / l);
        }
        __syncthreads();
    }
    if (merged && tid == 0) {
        merged[row * W] = top;
        merged[row * W + 1] = l;
    }
}

int attn_combine_dispatch(const float *states, int n_parts, __half *out, float *merged, int64_t rows, int D,
                          cudaStream_t stream) {
    if (rows == 0) return TACVQ_OK;
    // a group for every eight parts: more would have less than one round of loads each
    const int groups = n_parts > 8 * kCombineGroups ? kCombineGroups : n_parts > 8 ? (n_parts + 7) / 8 : 1;
    const cudaError_t e = launch_dependent(true, attn_combine_kernel, dim3((unsigned)rows), dim3(kCombineLanes * groups), 0, stream, states,
                                           n_parts, rows, D, out, merged);
    return e == cudaSuccess ? launch_status() : (int)e;
}

int attn_generic_splits(int B, int Hkv, int64_t T_cap, int sms) {
    const int pairs = B * Hkv;
    int splits = (2 * sms + pairs - 1) / pairs;
    const int64_t by_len = (T_cap + 255) / 256;
    if (splits > by_len) splits = (int)by_len;
    if (splits > 64) splits = 64;
    if (splits < 1) splits = 1;
    return splits;
}

size_t attn_generic_smem(int REP, int D, int G, int S, int K) {
    const size_t lut = (size_t)REP * K * S * G * sizeof(float);
    const size_t merge = ((size_t)2 * kAttnWarps * REP + (size_t)kAttnWarps * REP * D) * sizeof(float);
    return lut > merge ? lut : merge;
}

template <int REP, int DPL>
static int launch_generic(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab,
                          const __half *vtab, const int32_t *seq_start, const int32_t *seq_end, float *part, int B,
                          int Hq, int Hkv, int D, int G, int S, int K, int64_t T_cap, int splits, cudaStream_t stream) {
    const size_t smem = attn_generic_smem(REP, D, G, S, K);
    if (smem > 227 * 1024) return TACVQ_ERR_UNSUPPORTED;
    auto kernel = attn_generic_kernel<REP, DPL>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((unsigned)splits, (unsigned)Hkv, (unsigned)B);
    kernel<<<grid, kAttnThreads, smem, stream>>>(q, kcodes, vcodes, ktab, vtab, seq_start, seq_end, part, B, Hq, Hkv, D,
                                                 G, S, K, T_cap, splits);
    return launch_status();
}

template <int REP>
static int dispatch_dpl(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab,
                        const __half *vtab, const int32_t *seq_start, const int32_t *seq_end, float *part, int B,
                        int Hq, int Hkv, int D, int G, int S, int K, int64_t T_cap, int splits, cudaStream_t stream) {
#define TACVQ_CASE(N) \
    case N: return launch_generic<REP, N>(q, kcodes, vcodes, ktab, vtab, seq_start, seq_end, part, B, Hq, Hkv, D, G, S, K, T_cap, splits, stream);
    switch (D / 32) {
        TACVQ_CASE(1)
        TACVQ_CASE(2)
        TACVQ_CASE(4)
        TACVQ_CASE(8)
        default: return TACVQ_ERR_UNSUPPORTED;
    }
#undef TACVQ_CASE
}

int attn_generic_dispatch(const __half *q, const uint8_t *kcodes, const uint8_t *vcodes, const __half *ktab,
                          const __half *vtab, const int32_t *seq_start, const int32_t *seq_end, float *part, int B,
                          int Hq, int Hkv, int D, int G, int S, int K, int64_t T_cap, int splits, cudaStream_t stream) {
#define TACVQ_CASE(N) \
    case N: return dispatch_dpl<N>(q, kcodes, vcodes, ktab, vtab, seq_start, seq_end, part, B, Hq, Hkv, D, G, S, K, T_cap, splits, stream);
    switch (Hq / Hkv) {
        TACVQ_CASE(1)
        TACVQ_CASE(2)
        TACVQ_CASE(4)
        TACVQ_CASE(8)
        default: return TACVQ_ERR_UNSUPPORTED;
    }
#undef TACVQ_CASE
}

}  // namespace tacvq
