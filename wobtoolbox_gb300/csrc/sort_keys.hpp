// Sort of 64-bit keys on the device (k_sort.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace wobgb {

// Entries the arrays of a sort of n keys hold: the next power of two (at least 1).
inline uint32_t sort_padded(uint32_t n) {
    uint32_t n2 = 1;
    while (n2 < n) n2 <<= 1;
    return n2;
}

// Sorts n2 (a power of two) device keys ascending, in place; with val (may be null) the entries are
// (key, val) pairs ordered by key, then val. Pad with the largest key (and val) to reach n2.
cudaError_t launch_sort_keys(uint32_t n2, uint64_t *key, uint32_t *val, cudaStream_t stream);

}  // namespace wobgb
