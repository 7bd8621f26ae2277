// Whether a stack of matrices is the identity: a whitener that is one leaves rows and words unchanged bit for bit.
#pragma once

#include "common.cuh"

namespace tacvq {

constexpr int kIdentityBlocks = 8, kIdentityThreads = 1024;

// A one belongs at every (n + 1)-th element of a matrix.  WIDE elements at a time; n is a multiple of WIDE.
template <int WIDE>
__device__ __forceinline__ bool differs_from_identity(const float *__restrict__ matrices, int64_t count, int n) {
    constexpr int kStep = kIdentityBlocks * kIdentityThreads * WIDE;
    const int size = n * n, every = n + 1;
    const int64_t elements = count * size;
    int64_t i = (int64_t)(blockIdx.x * kIdentityThreads + threadIdx.x) * WIDE;
    int at = (int)(i % size), place = at % every;  // in the matrix; past the last element that is a one
    const int at_step = kStep % size, place_step = at_step % every;
    bool differs = false;
#pragma unroll 4
    for (; i < elements; i += kStep) {
        const int one = place == 0 ? 0 : every - place;  // which of the next elements is on the diagonal
        float v[WIDE];
        if constexpr (WIDE == 4) *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(matrices + i);
        else v[0] = matrices[i];
#pragma unroll
        for (int j = 0; j < WIDE; ++j) differs |= !(v[j] == (one == j ? 1.0f : 0.0f));
        at += at_step, place += place_step;
        if (place >= every) place -= every;
        if (at >= size) at -= size, place = place == 0 ? every - 1 : place - 1;  // n * n is one more than a multiple of n + 1
    }
    return differs;
}

// One cluster, so that the answer needs no second launch and no memory that somebody has cleared: its first block says yes, and after a barrier of the
// cluster any block may say no.  Asked before the values of a training step are searched, which wait for it.  us from a graph, one block / eight / a comparison with
// torch.eye: 8 matrices of 128 x 128 7.9 / 3.1 / 14.6, 64 of them 52 / 9.1 / 15.1, 256 of 4 x 4 74 / 2.6 / 6.2.
__global__ void __cluster_dims__(kIdentityBlocks, 1, 1) __launch_bounds__(kIdentityThreads)
is_identity_kernel(const float *__restrict__ matrices, int64_t count, int n, uint8_t *answer) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *answer = 1;
    const bool wide = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(matrices) & 15) == 0;
    const bool differs = __syncthreads_or(wide ? differs_from_identity<4>(matrices, count, n) : differs_from_identity<1>(matrices, count, n));
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (differs && threadIdx.x == 0) *answer = 0;
}

inline int is_identity_launch(const float *matrices, int64_t count, int n, uint8_t *answer, cudaStream_t stream) {
    is_identity_kernel<<<kIdentityBlocks, kIdentityThreads, 0, stream>>>(matrices, count, n, answer);
    return launch_status();
}

}  // namespace tacvq
