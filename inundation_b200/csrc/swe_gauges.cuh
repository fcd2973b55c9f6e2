// The gauges of a calibration after a step, by one CTA of 256 threads: the gauge kernel, and the
// persistent kernel's forward run.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "swe_common.cuh"

namespace swe {

// After step `done` of a run (1-based): record the gauges' depths (record = 1) or add their squared misfit to
// the loss. All threads; acc: a double per thread.
__device__ __forceinline__ void gauge_after_step(const swe_state_t &s, const swe_gauges_t &gg, int record, uint64_t done,
                                                 double *acc) {
    double sum = 0.0;
    if (done >= 1 && done <= gg.steps) {
        float *row = gg.obs + static_cast<size_t>(done - 1) * gg.count;
        for (uint32_t g = threadIdx.x; g < gg.count; g += kThreads) {
            const uint32_t c = gg.cells[g];
            const float H = s.h[c] + s.h_lo[c];
            if (record) {
                row[g] = H;
            } else {
                const double d = static_cast<double>(H) - static_cast<double>(row[g]);
                sum += d * d;
            }
        }
    }
    if (record) return;
    acc[threadIdx.x] = sum;
    __syncthreads();
    for (int w = kThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) acc[threadIdx.x] += acc[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *gg.loss += acc[0];
}

}  // namespace swe
