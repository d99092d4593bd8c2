// Ordered sums on the device.
#pragma once

namespace mel {

// running sums of `n` terms t[k*stride] (k = 0..n-1) added in order to acc, eight loads in flight
// while eight are added
__device__ __forceinline__ double ordered_sum(double acc, const double* t, int n, int stride)
{
    double v[8], w[8];
    int k = 0;
    if (n >= 8) {
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = t[(size_t)j * stride];
        for (; k + 24 <= n; k += 16) {
#pragma unroll
            for (int j = 0; j < 8; j++) w[j] = t[(size_t)(k + 8 + j) * stride];
#pragma unroll
            for (int j = 0; j < 8; j++) acc += v[j];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = t[(size_t)(k + 16 + j) * stride];
#pragma unroll
            for (int j = 0; j < 8; j++) acc += w[j];
        }
#pragma unroll
        for (int j = 0; j < 8; j++) acc += v[j];
        k += 8;
    }
    for (; k + 4 <= n; k += 4) {
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = t[(size_t)(k + j) * stride];
#pragma unroll
        for (int j = 0; j < 4; j++) acc += w[j];
    }
    for (; k < n; k++) acc += t[(size_t)k * stride];
    return acc;
}

}  // namespace mel
