// Sampling CDFs on the device: the serial Kahan prefix sums of the host build, in parallel, with
// the host build's bits (k_kahan.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace wobgb {

// Bytes of device scratch launch_kahan_cdf needs for `arrays` (1 or 2) weight arrays of n entries.
size_t kahan_scratch_bytes(uint32_t n, int arrays);

// For each of the `arrays` weight arrays w[a] (device, n entries): cdf[a] = the Kahan prefix sums of
// w[a] in order, divided by the total and made nondecreasing, and totals[a] = the total, bit for bit
// what scene_build.cpp's kahan_cdf computes. scratch: kahan_scratch_bytes, 256-byte aligned.
cudaError_t launch_kahan_cdf(uint32_t n, int arrays, const float *const *w, float *const *cdf, float *totals,
                             void *scratch, cudaStream_t stream);

// Guide table (scene_build.cpp's build_guide) of a nondecreasing device CDF: G = guide_records(n)
// records of 4 words.
cudaError_t launch_guide(uint32_t n, uint32_t G, const float *cdf, uint32_t *rec, cudaStream_t stream);

}  // namespace wobgb
