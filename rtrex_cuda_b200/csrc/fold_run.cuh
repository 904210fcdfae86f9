// The ordered fold of a run of weights by one warp: acc + w[0] + w[1] + ... (or
// acc - w[0] - ...), one dependent double operation per weight, the same on
// every lane.  128 weights at a time go through shared memory, from which every
// lane reads them two per 16-byte broadcast load, with the next 128 in flight:
// 4.2 ns per weight, the latency of the dependent add (B200; a double
// shuffle per weight takes 15 ns).  A missing weight in the last step is +0.0,
// which changes no difference and no sum that is not -0.0.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rtr {

constexpr int kFoldStep = 128;

// sm: kFoldStep doubles of this warp, 16-byte aligned.
template <bool kSubtract>
__device__ __forceinline__ double fold_run(const double* __restrict__ w, int64_t n, double acc, double* sm)
{
    const int lane = threadIdx.x & 31;
    double v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = j * 32 + lane < n ? w[j * 32 + lane] : 0.0;
    for (int64_t b = 0; b < n; b += kFoldStep) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sm[j * 32 + lane] = v[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t i = b + kFoldStep + j * 32 + lane;
            v[j] = i < n ? w[i] : 0.0;
        }
        const double2* s2 = reinterpret_cast<const double2*>(sm);
        const int pairs = n - b < kFoldStep ? (int)(n - b + 31) / 32 * 16 : kFoldStep / 2;
        for (int q0 = 0; q0 < pairs; q0 += 16) {
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const double2 x = s2[q0 + q];
                acc = kSubtract ? acc - x.x : acc + x.x;
                acc = kSubtract ? acc - x.y : acc + x.y;
            }
        }
        __syncwarp();
    }
    return acc;
}

}  // namespace rtr
