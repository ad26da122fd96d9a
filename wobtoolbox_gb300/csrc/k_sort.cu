// Bitonic sort of 64-bit keys, alone or with 32-bit values, for the Morton orders of a scene build and
// of the control variate's evaluation points.
//
// One launch per compare-exchange step (190 for 2^19 keys, 136 for 2^16) is bound by the launches: a
// step over keys that sit in the L2 takes as long as starting it, 2.9 us. Here a block sorts and
// merges tiles of kTile keys in shared memory, all steps of distance below kTile in one launch, and
// the longer steps go two to a launch with four keys a thread: 24 launches for 2^19 keys with values
// (0.79 -> 0.21 ms) and 11 for 2^16 without (0.40 -> 0.09 ms).
#include "sort_keys.hpp"

namespace wobgb {

namespace {

constexpr uint32_t kTile = 4096;  // 48 KB of shared memory with values
constexpr uint32_t kTileThreads = 1024;

template <bool kVals>
__device__ __forceinline__ void exchange(uint64_t &ka, uint32_t &va, uint64_t &kb, uint32_t &vb, bool up) {
    const bool greater = ka > kb || (kVals && ka == kb && va > vb);
    if (greater == up) {
        const uint64_t k = ka;
        ka = kb;
        kb = k;
        if (kVals) {
            const uint32_t v = va;
            va = vb;
            vb = v;
        }
    }
}

// Steps of distance below kTile: of the stages k = 2 .. kTile (kAll), or of stage k alone.
template <bool kVals, bool kAll>
__global__ void __launch_bounds__(kTileThreads) tile_kernel(uint32_t n2, uint32_t stage, uint64_t *key, uint32_t *val) {
    __shared__ uint64_t sk[kTile];
    __shared__ uint32_t sv[kVals ? kTile : 1];
    const uint32_t base = blockIdx.x * kTile, m = min(kTile, n2 - base);
    for (uint32_t i = threadIdx.x; i < m; i += kTileThreads) {
        sk[i] = key[base + i];
        if (kVals) sv[i] = val[base + i];
    }
    for (uint32_t k = kAll ? 2u : stage; k <= (kAll ? m : stage); k <<= 1) {
        for (uint32_t j = kAll ? k >> 1 : m >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < m / 2; t += kTileThreads) {
                const uint32_t i = 2 * t - (t & (j - 1)), l = i + j;  // t's bits with a zero inserted at j
                uint64_t ka = sk[i], kb = sk[l];
                uint32_t va = 0, vb = 0;
                if (kVals) {
                    va = sv[i];
                    vb = sv[l];
                }
                exchange<kVals>(ka, va, kb, vb, ((base + i) & k) == 0);
                sk[i] = ka;
                sk[l] = kb;
                if (kVals) {
                    sv[i] = va;
                    sv[l] = vb;
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < m; i += kTileThreads) {
        key[base + i] = sk[i];
        if (kVals) val[base + i] = sv[i];
    }
}

// Stage k's steps of distance 2 j and j: thread t takes the four keys j apart.
template <bool kVals>
__global__ void __launch_bounds__(256) two_steps_kernel(uint32_t n2, uint32_t j, uint32_t k, uint64_t *key, uint32_t *val) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= n2 / 4) return;
    const uint32_t i = (t & (j - 1)) | ((t & ~(j - 1)) << 2);
    const bool up = (i & k) == 0;
    uint64_t a[4];
    uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 4; q++) {
        a[q] = key[i + q * j];
        if (kVals) v[q] = val[i + q * j];
    }
    exchange<kVals>(a[0], v[0], a[2], v[2], up);
    exchange<kVals>(a[1], v[1], a[3], v[3], up);
    exchange<kVals>(a[0], v[0], a[1], v[1], up);
    exchange<kVals>(a[2], v[2], a[3], v[3], up);
#pragma unroll
    for (int q = 0; q < 4; q++) {
        key[i + q * j] = a[q];
        if (kVals) val[i + q * j] = v[q];
    }
}

template <bool kVals>
__global__ void __launch_bounds__(256) one_step_kernel(uint32_t n2, uint32_t j, uint32_t k, uint64_t *key, uint32_t *val) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= n2 / 2) return;
    const uint32_t i = (t & (j - 1)) | ((t & ~(j - 1)) << 1), l = i + j;
    uint64_t ka = key[i], kb = key[l];
    uint32_t va = kVals ? val[i] : 0u, vb = kVals ? val[l] : 0u;
    exchange<kVals>(ka, va, kb, vb, (i & k) == 0);
    key[i] = ka;
    key[l] = kb;
    if (kVals) {
        val[i] = va;
        val[l] = vb;
    }
}

template <bool kVals>
cudaError_t sort_impl(uint32_t n2, uint64_t *key, uint32_t *val, cudaStream_t st) {
    if (n2 < 2) return cudaSuccess;
    const uint32_t tiles = (n2 + kTile - 1) / kTile;
    tile_kernel<kVals, true><<<tiles, kTileThreads, 0, st>>>(n2, 0, key, val);
    for (uint32_t k = 2 * kTile; k <= n2 && k != 0; k <<= 1) {
        uint32_t j = k >> 1;
        while (j >= 2 * kTile) {
            two_steps_kernel<kVals><<<(n2 / 4 + 255) / 256, 256, 0, st>>>(n2, j >> 1, k, key, val);
            j >>= 2;
        }
        if (j >= kTile) one_step_kernel<kVals><<<(n2 / 2 + 255) / 256, 256, 0, st>>>(n2, j, k, key, val);
        tile_kernel<kVals, false><<<tiles, kTileThreads, 0, st>>>(n2, k, key, val);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sort_keys(uint32_t n2, uint64_t *key, uint32_t *val, cudaStream_t stream) {
    return val ? sort_impl<true>(n2, key, val, stream) : sort_impl<false>(n2, key, val, stream);
}

}  // namespace wobgb
