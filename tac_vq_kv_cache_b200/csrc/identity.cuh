// Whether a stack of matrices is the identity: a whitener that is one leaves rows and words unchanged bit for bit.
#pragma once

#include "common.cuh"

namespace tacvq {

// One block, so that the answer needs no second launch: 8 matrices of 128 x 128 (512 KB, from L2) take it about as long as a launch.  A one
// belongs at every (n + 1)-th element of a matrix.
__global__ void __launch_bounds__(1024)
is_identity_kernel(const float *__restrict__ matrices, int64_t count, int n, uint8_t *__restrict__ answer) {
    const int size = n * n, every = n + 1;
    bool differs = false;
    if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(matrices) & 15) == 0) {
        const int ahead = 4 * 1024 % every;
        for (int64_t m = 0; m < count; ++m, matrices += size) {
            int place = (int)(4 * threadIdx.x) % every;
#pragma unroll 4
            for (int i = threadIdx.x; i < size / 4; i += 1024) {
                const float4 v = reinterpret_cast<const float4 *>(matrices)[i];
                const int one = place == 0 ? 0 : every - place;  // which of the four is on the diagonal, if one is
                differs |= !(v.x == (one == 0 ? 1.0f : 0.0f) && v.y == (one == 1 ? 1.0f : 0.0f) && v.z == (one == 2 ? 1.0f : 0.0f) && v.w == (one == 3 ? 1.0f : 0.0f));
                place += ahead;
                if (place >= every) place -= every;
            }
        }
    } else {
        const int ahead = 1024 % every;
        for (int64_t m = 0; m < count; ++m, matrices += size) {
            int place = (int)threadIdx.x % every;
#pragma unroll 4
            for (int i = threadIdx.x; i < size; i += 1024) {
                differs |= !(matrices[i] == (place == 0 ? 1.0f : 0.0f));
                place += ahead;
                if (place >= every) place -= every;
            }
        }
    }
    differs = __syncthreads_or(differs);
    if (threadIdx.x == 0) *answer = differs ? 0 : 1;
}

inline int is_identity_launch(const float *matrices, int64_t count, int n, uint8_t *answer, cudaStream_t stream) {
    is_identity_kernel<<<1, 1024, 0, stream>>>(matrices, count, n, answer);
    return launch_status();
}

}  // namespace tacvq
