// Scene construction on the GPU from device arrays (no counterpart in the reference, whose
// SceneHost builds on the host, scene.cuh:264-299, with lbvh's build, scene.cuh:266).
//
// Produces the same packed records as build_host_scene (scene_build.cpp) -- element and 3D
// intersection records in storage order, area and |g| CDFs (Kahan prefix sums, normalised, made
// nondecreasing), guide tables, padded boxes -- with a different BVH topology: Morton codes of the
// element centroids, a bitonic sort of (code, caller index), a binary radix tree over the sorted
// codes (Karras, "Maximizing parallelism in the construction of BVHs, octrees, and k-d trees",
// HPG 2012), bottom-up boxes, and a collapse into the 4-wide layout (each wide node takes its binary
// node's two children, each expanded once more when it holds more than kLeafMax elements: the wide
// nodes are the binary nodes of even depth with more than kLeafMax elements, numbered in binary node
// order). Storage order is the sorted order, so every leaf is a contiguous range and a depth-first
// traversal with children in order still returns hits in storage order; hit sets do not depend on
// the topology. Nothing is read back before the end: the checks of the input, the node count, the
// depth and the totals come in one copy. The CDFs come from k_kahan.cu, whose prefix sums have the bits of the
// host build's serial ones, so the sampling tables are bit-identical to a host build over the same
// storage order.
#include "scene_build_gpu.hpp"

#include "kahan_scan.hpp"
#include "scene_host.hpp"
#include "scratch.hpp"
#include "sort_keys.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace wobgb {

namespace {

constexpr int kT = 256;

// order-preserving float <-> uint32 map (for atomicMin / atomicMax on floats)
__device__ __forceinline__ uint32_t ord(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float unord(uint32_t u) {
    const uint32_t v = (u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u;
    float f;
    std::memcpy(&f, &v, 4);
    return f;
}

constexpr uint32_t kBadTree = 64u;

struct Bounds {  // ordered-uint encodings
    uint32_t lo[3], hi[3], clo[3], chi[3], mag;
    uint32_t bad;            // bit 0 non-finite vertex, 1 normal, 2 data, 3 alpha, 4 type, 5 normal length, 6 tree
    uint32_t all_dirichlet;  // 1 until a non-Dirichlet element is seen
    uint32_t n_nodes, depth; // of the 4-wide tree
    float totals[2];         // area, |g|
};

// padding of the host build: 1e-5 (extent + max |coordinate|)
__host__ __device__ inline float box_pad(const Bounds &b, int dim) {
    float ext = 0.0f;
    for (int k = 0; k < dim; k++) {
        const float e = unord(b.hi[k]) - unord(b.lo[k]);
        ext = ext < e ? e : ext;
    }
    return 1e-5f * (ext + unord(b.mag)) + 1e-30f;
}

__device__ __forceinline__ bool finite_f(float x) { return isfinite(x); }

// The checks of the input, element boxes and the scene's bounds. The bounds are reduced over the block
// before the global atomics: one atomic an element and word on a handful of addresses took 0.35 ms
// for 327,680 triangles, one a block 0.02 ms.
template <int D>
__global__ void __launch_bounds__(kT) k_validate(uint32_t n, const float *__restrict__ verts,
                                                 const float *__restrict__ normals, const float *__restrict__ bvals,
                                                 const float *__restrict__ alphas, const int32_t *__restrict__ types,
                                                 float *__restrict__ box, Bounds *b) {
    constexpr int kWords = 4 * D + 1;  // per axis min lo, max hi, min c, max c; then max |coordinate|
    __shared__ uint32_t red[kT / 32][kWords];
    __shared__ uint32_t s_bad, s_other;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_bad = s_other = 0u;
    __syncthreads();
    uint32_t word[kWords];  // minima as complements, so that every word is a maximum
#pragma unroll
    for (int k = 0; k < kWords; k++) word[k] = 0u;
    if (i < n) {
        uint32_t bad = 0;
        const float *v = verts + (size_t)i * D * D;
        for (int k = 0; k < D * D; k++)
            if (!finite_f(v[k])) bad |= 1u;
        for (int k = 0; k < D; k++) {
            if (!finite_f(normals[(size_t)i * D + k])) bad |= 2u;
            if (!finite_f(bvals[(size_t)i * D + k])) bad |= 4u;
            if (alphas && !finite_f(alphas[(size_t)i * D + k])) bad |= 8u;
        }
        float q = 0.0f;
        for (int k = 0; k < D; k++) q += normals[(size_t)i * D + k] * normals[(size_t)i * D + k];
        if (!(q >= 0.25f && q <= 4.0f)) bad |= 32u;  // as the host build: normals far from unit length
        const int t = types[i];
        if (t < 0 || t > 2) bad |= 16u;
        if (bad) atomicOr(&s_bad, bad);
        if (t != 0) s_other = 1u;
        // element box, centroid (scene_build.cpp: lo / hi / s / dim, left to right)
        for (int k = D; k < 3; k++)
            box[(size_t)i * 9 + k] = box[(size_t)i * 9 + 3 + k] = box[(size_t)i * 9 + 6 + k] = 0.0f;
        float mag = 0.0f;
#pragma unroll
        for (int k = 0; k < D; k++) {
            float lo = v[k], hi = v[k], s = v[k];
            for (int j = 1; j < D; j++) {
                lo = fminf(lo, v[j * D + k]);
                hi = fmaxf(hi, v[j * D + k]);
                s = s + v[j * D + k];
            }
            const float c = s / (float)D;
            box[(size_t)i * 9 + k] = lo;
            box[(size_t)i * 9 + 3 + k] = hi;
            box[(size_t)i * 9 + 6 + k] = c;
            word[4 * k] = ~ord(lo);
            word[4 * k + 1] = ord(hi);
            word[4 * k + 2] = ~ord(c);
            word[4 * k + 3] = ord(c);
            mag = fmaxf(mag, fmaxf(fabsf(lo), fabsf(hi)));
        }
        word[4 * D] = ord(mag);
    }
#pragma unroll
    for (int k = 0; k < kWords; k++) {
        const uint32_t m = __reduce_max_sync(0xffffffffu, word[k]);
        if (lane == 0) red[warp][k] = m;
    }
    __syncthreads();
    if (threadIdx.x < kWords) {
        const int k = threadIdx.x, axis = k >> 2;
        uint32_t m = red[0][k];
        for (int w = 1; w < kT / 32; w++) m = max(m, red[w][k]);
        if (k == 4 * D) atomicMax(&b->mag, m);
        else if ((k & 3) == 0) atomicMin(&b->lo[axis], ~m);
        else if ((k & 3) == 1) atomicMax(&b->hi[axis], m);
        else if ((k & 3) == 2) atomicMin(&b->clo[axis], ~m);
        else atomicMax(&b->chi[axis], m);
    }
    if (threadIdx.x == 0) {
        if (s_bad) atomicOr(&b->bad, s_bad);
        if (s_other) atomicAnd(&b->all_dirichlet, 0u);
    }
}

__device__ __forceinline__ uint64_t spread21(uint64_t x) {  // 21 bits -> every third bit
    x &= 0x1FFFFFull;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}
__device__ __forceinline__ uint64_t spread32(uint64_t x) {  // 32 bits -> every second bit
    x &= 0xFFFFFFFFull;
    x = (x | (x << 16)) & 0x0000FFFF0000FFFFull;
    x = (x | (x << 8)) & 0x00FF00FF00FF00FFull;
    x = (x | (x << 4)) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | (x << 2)) & 0x3333333333333333ull;
    x = (x | (x << 1)) & 0x5555555555555555ull;
    return x;
}

template <int D>
__global__ void k_morton(uint32_t n, uint32_t n2, const float *__restrict__ box, const Bounds *b, uint64_t *key,
                         uint32_t *val) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n2) return;
    if (i >= n) {
        key[i] = ~0ull;
        val[i] = 0xFFFFFFFFu;
        return;
    }
    uint64_t q[3] = {0, 0, 0};
    const int bits = D == 3 ? 21 : 32;
    const double scale = (double)((1ull << bits) - 1);
    for (int k = 0; k < D; k++) {
        const double lo = (double)unord(b->clo[k]), hi = (double)unord(b->chi[k]);
        const double ext = hi - lo;
        const double x = ext > 0.0 ? ((double)box[(size_t)i * 9 + 6 + k] - lo) / ext : 0.0;
        q[k] = (uint64_t)fmin(fmax(x * scale, 0.0), scale);
    }
    key[i] = D == 3 ? (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2])
                    : (spread32(q[0]) << 1) | spread32(q[1]);
    val[i] = i;
}

// common-prefix length of the augmented keys (code, index) at sorted positions a and b
__device__ __forceinline__ int delta(const uint64_t *key, int64_t n, int64_t a, int64_t b) {
    if (b < 0 || b >= n) return -1;
    const uint64_t ka = key[a], kb = key[b];
    if (ka != kb) return __clzll((long long)(ka ^ kb));
    return 64 + __clz((int)((uint32_t)a ^ (uint32_t)b));
}

constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kNotWide = 0xFFFFFFFFu;

// Binary radix tree: internal node i has children child[2i], child[2i+1] (kLeafBit | sorted
// position for leaves) and covers sorted positions [first[i], last[i]].
__global__ void k_radix_tree(uint32_t n, const uint64_t *__restrict__ key, uint32_t *child, uint32_t *first,
                             uint32_t *last, uint32_t *parent_int, uint32_t *parent_leaf) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t N = n;
    if (i >= N - 1) return;
    const int d = (delta(key, N, i, i + 1) - delta(key, N, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(key, N, i, i - d);
    int64_t lmax = 2;
    while (delta(key, N, i, i + lmax * d) > dmin) lmax *= 2;
    int64_t l = 0;
    for (int64_t t = lmax / 2; t >= 1; t /= 2)
        if (delta(key, N, i, i + (l + t) * d) > dmin) l += t;
    const int64_t j = i + l * d;
    const int dnode = delta(key, N, i, j);
    int64_t s = 0, t = l;
    do {
        t = (t + 1) / 2;
        if (delta(key, N, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int64_t g = i + s * d + (d < 0 ? -1 : 0);
    const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
    const uint32_t left = (lo == g) ? (kLeafBit | (uint32_t)g) : (uint32_t)g;
    const uint32_t right = (hi == g + 1) ? (kLeafBit | (uint32_t)(g + 1)) : (uint32_t)(g + 1);
    child[2 * i] = left;
    child[2 * i + 1] = right;
    first[i] = (uint32_t)lo;
    last[i] = (uint32_t)hi;
    if (left & kLeafBit) parent_leaf[left & ~kLeafBit] = (uint32_t)i;
    else parent_int[left] = (uint32_t)i;
    if (right & kLeafBit) parent_leaf[right & ~kLeafBit] = (uint32_t)i;
    else parent_int[right] = (uint32_t)i;
}

// Boxes of the binary nodes, bottom-up: the second child to arrive at a parent writes its box.
// A climb is bounded by the tree height (at most 96 levels for 64-bit codes plus 32 index bits);
// a longer one can only come from a malformed tree and sets bit 6 of the error word.
__global__ void k_boxes(uint32_t n, int dim, const uint32_t *__restrict__ val, const float *__restrict__ ebox,
                        const uint32_t *__restrict__ child, const uint32_t *__restrict__ parent_int,
                        const uint32_t *__restrict__ parent_leaf, uint32_t *flags, float *ibox, Bounds *bd) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n || n < 2) return;
    const float pad = box_pad(*bd, dim);
    uint32_t node = parent_leaf[s];
    for (int level = 0;; level++) {
        if (level > 128 || node >= n - 1) {
            atomicOr(&bd->bad, kBadTree);
            return;
        }
        __threadfence();
        if (atomicAdd(&flags[node], 1u) == 0u) return;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int c = 0; c < 2; c++) {
            const uint32_t ch = child[2 * node + c];
            for (int k = 0; k < 3; k++) {
                float a, b;
                if (ch & kLeafBit) {
                    const uint32_t e = val[ch & ~kLeafBit];
                    a = ebox[(size_t)e * 9 + k] - pad;
                    b = ebox[(size_t)e * 9 + 3 + k] + pad;
                } else {
                    a = ((volatile float *)ibox)[(size_t)ch * 6 + k];
                    b = ((volatile float *)ibox)[(size_t)ch * 6 + 3 + k];
                }
                lo[k] = fminf(lo[k], a);
                hi[k] = fmaxf(hi[k], b);
            }
        }
        for (int k = 0; k < 3; k++) {
            ibox[(size_t)node * 6 + k] = lo[k];
            ibox[(size_t)node * 6 + 3 + k] = hi[k];
        }
        if (node == 0) return;
        node = parent_int[node];
    }
}

__device__ __forceinline__ uint32_t range_count(uint32_t code, const uint32_t *first, const uint32_t *last) {
    return (code & kLeafBit) ? 1u : last[code] - first[code] + 1u;
}

// The up to four binary nodes a wide node over binary node b holds, in range order.
__device__ __forceinline__ int wide_children(uint32_t b, const uint32_t *child, const uint32_t *first,
                                             const uint32_t *last, uint32_t out[4]) {
    int m = 0;
    for (int c = 0; c < 2; c++) {
        const uint32_t ch = child[2 * b + c];
        if (!(ch & kLeafBit) && range_count(ch, first, last) > kLeafMax) {
            out[m++] = child[2 * ch];
            out[m++] = child[2 * ch + 1];
        } else {
            out[m++] = ch;
        }
    }
    return m;
}

// Marks the binary nodes that become wide nodes (even depth, more than kLeafMax elements) and counts
// them per block. A node's depth is its climb to the root: a level-by-level collapse needs a round
// trip to the host per level (13 levels and 1.0 ms for 327,680 triangles; the climbs take 0.02 ms).
__global__ void __launch_bounds__(kT) k_wide_mark(uint32_t n_int, const uint32_t *__restrict__ first,
                                                  const uint32_t *__restrict__ last,
                                                  const uint32_t *__restrict__ parent_int, uint32_t *__restrict__ rank,
                                                  uint32_t *__restrict__ blk, Bounds *bd) {
    __shared__ uint32_t warp_count[kT / 32];
    const uint32_t i = blockIdx.x * kT + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    bool wide = false;
    uint32_t depth = 0;
    if (i < n_int && last[i] - first[i] + 1u > kLeafMax) {
        uint32_t node = i;
        while (node != 0u && depth <= 128u) {
            node = parent_int[node];
            depth++;
        }
        if (depth > 128u) atomicOr(&bd->bad, kBadTree);
        wide = (depth & 1u) == 0u;
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, wide);
    const uint32_t deepest = __reduce_max_sync(0xffffffffu, wide ? depth / 2u + 1u : 0u);
    if (lane == 0) {
        warp_count[warp] = (uint32_t)__popc(bits);
        if (deepest) atomicMax(&bd->depth, deepest);
    }
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t w = 0; w < kT / 32; w++) {
        if (w < warp) before += warp_count[w];
        all += warp_count[w];
    }
    if (i < n_int) rank[i] = wide ? before + (uint32_t)__popc(bits & ((1u << lane) - 1u)) : kNotWide;
    if (threadIdx.x == 0) blk[blockIdx.x] = all;
}

// exclusive scan of cnt values in one block; total written to *total
__global__ void __launch_bounds__(1024) k_scan(uint32_t cnt, uint32_t *v, uint32_t *total) {
    __shared__ uint32_t part[1024];
    const uint32_t tid = threadIdx.x;
    const uint32_t chunk = (cnt + 1023u) / 1024u;
    const uint32_t b = min(cnt, tid * chunk), e = min(cnt, b + chunk);
    uint32_t s = 0;
    for (uint32_t i = b; i < e; i++) s += v[i];
    part[tid] = s;
    __syncthreads();
    for (uint32_t o = 1; o < 1024u; o <<= 1) {
        const uint32_t add = tid >= o ? part[tid - o] : 0u;
        __syncthreads();
        part[tid] += add;
        __syncthreads();
    }
    if (tid == 1023u) *total = part[1023];
    uint32_t acc = part[tid] - s;
    for (uint32_t i = b; i < e; i++) {
        const uint32_t x = v[i];
        v[i] = acc;
        acc += x;
    }
}

// writes the wide node records
template <int D>
__global__ void __launch_bounds__(kT) k_wide_write(uint32_t n_int, const uint32_t *__restrict__ rank,
                                                   const uint32_t *__restrict__ blk,
                                                   const uint32_t *__restrict__ child,
                                                   const uint32_t *__restrict__ first,
                                                   const uint32_t *__restrict__ last, const uint32_t *__restrict__ val,
                                                   const float *__restrict__ ebox, const float *__restrict__ ibox,
                                                   const Bounds *__restrict__ bd, float *__restrict__ nodes) {
    const uint32_t t = blockIdx.x * kT + threadIdx.x;
    if (t >= n_int || rank[t] == kNotWide) return;
    const float pad = box_pad(*bd, D);
    constexpr int NF = D == 2 ? 24 : 32;
    float4 *r = reinterpret_cast<float4 *>(nodes + (size_t)(blk[blockIdx.x] + rank[t]) * NF);
    uint32_t ch[4];
    const int m = wide_children(t, child, first, last, ch);
    float lo[D][4], hi[D][4];
    uint32_t codes[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        codes[k] = kChildEmpty;
#pragma unroll
        for (int a = 0; a < D; a++) lo[a][k] = hi[a][k] = 0.0f;
        if (k < m) {
            const uint32_t c = ch[k];
            const uint32_t count = range_count(c, first, last);
            const uint32_t f = (c & kLeafBit) ? (c & ~kLeafBit) : first[c];
            codes[k] = count > kLeafMax ? blk[c / kT] + rank[c] : 0x80000000u | ((count - 1u) << 28) | f;
            const uint32_t e = (c & kLeafBit) ? val[c & ~kLeafBit] : 0u;
#pragma unroll
            for (int a = 0; a < D; a++) {
                if (c & kLeafBit) {
                    lo[a][k] = ebox[(size_t)e * 9 + a] - pad;
                    hi[a][k] = ebox[(size_t)e * 9 + 3 + a] + pad;
                } else {
                    lo[a][k] = ibox[(size_t)c * 6 + a];
                    hi[a][k] = ibox[(size_t)c * 6 + 3 + a];
                }
            }
        }
    }
#pragma unroll
    for (int a = 0; a < D; a++) {
        r[a] = make_float4(lo[a][0], lo[a][1], lo[a][2], lo[a][3]);
        r[D + a] = make_float4(hi[a][0], hi[a][1], hi[a][2], hi[a][3]);
    }
    r[2 * D] = make_float4(__uint_as_float(codes[0]), __uint_as_float(codes[1]), __uint_as_float(codes[2]),
                           __uint_as_float(codes[3]));
    r[2 * D + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // padding to a 32-byte multiple
}

// element records, intersection records, area and |g| weights in storage order (scene_build.cpp)
template <int D>
__global__ void k_records(uint32_t n, const uint32_t *__restrict__ val, const float *__restrict__ verts,
                          const float *__restrict__ normals, const float *__restrict__ bvals,
                          const float *__restrict__ alphas, const int32_t *__restrict__ types, float *elems,
                          float *elem_aux, float *isect, float *areas, float *bvw) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t i = val[s];
    const float *v = verts + (size_t)i * D * D;
    const float *nn = normals + (size_t)i * D;
    const float *bv = bvals + (size_t)i * D;
    float al[3] = {0, 0, 0};
    if (alphas)
        for (int k = 0; k < D; k++) al[k] = alphas[(size_t)i * D + k];
    float4 *r = reinterpret_cast<float4 *>(elems + (size_t)s * 16);
    const float type = __int_as_float(types[i]);
    if constexpr (D == 2) {
        const float dx = v[2] - v[0], dy = v[3] - v[1];
        const float area = sqrtf(dx * dx + dy * dy);
        r[0] = make_float4(v[0], v[1], v[2], v[3]);
        r[1] = make_float4(nn[0], nn[1], bv[0], bv[1]);
        r[2] = make_float4(al[0], al[1], area, type);
        r[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        areas[s] = area;
        bvw[s] = area * (fabsf(bv[0]) + fabsf(bv[1])) / 2.0f;
    } else {
        const float u0 = v[6] - v[0], u1 = v[7] - v[1], u2 = v[8] - v[2];
        const float w0 = v[3] - v[0], w1 = v[4] - v[1], w2 = v[5] - v[2];
        const float x = u1 * w2 - u2 * w1;
        const float y = u2 * w0 - u0 * w2;
        const float z = u0 * w1 - u1 * w0;
        const float area = sqrtf(x * x + y * y + z * z) / 2.0f;
        r[0] = make_float4(v[0], v[1], v[2], v[3]);
        r[1] = make_float4(v[4], v[5], v[6], v[7]);
        r[2] = make_float4(v[8], nn[0], nn[1], nn[2]);
        r[3] = make_float4(bv[0], bv[1], bv[2], type);
        reinterpret_cast<float4 *>(elem_aux)[s] = make_float4(al[0], al[1], al[2], area);
        areas[s] = area;
        bvw[s] = area * (fabsf(bv[0]) + fabsf(bv[1]) + fabsf(bv[2])) / 3.0f;
        float4 *q = reinterpret_cast<float4 *>(isect + (size_t)s * 16);
        const float e1x = v[0] - v[3], e1y = v[1] - v[4], e1z = v[2] - v[5];
        const float e2x = v[0] - v[6], e2y = v[1] - v[7], e2z = v[2] - v[8];
        q[0] = make_float4(v[0], v[1], v[2], e1x);
        q[1] = make_float4(e1y, e1z, e2x, e2y);
        q[2] = make_float4(e2z, e1y * e2z - e1z * e2y, e1z * e2x - e1x * e2z, e1x * e2y - e1y * e2x);
        q[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// New boundary data of existing records: are all offsets finite (and below 3e38)?
__global__ void k_check_offsets(uint32_t n, const float *__restrict__ delta, uint32_t *bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(fabsf(delta[i]) <= 3.0e38f)) *bad = 1u;
}
// Adds offset i to record i's vertex boundary values and recomputes its |g| weight with the host
// build's operations; nothing where a check failed.
template <int D>
__global__ void k_offset_weights(uint32_t n, const float *__restrict__ delta, const uint32_t *__restrict__ bad,
                                 float *__restrict__ elems, const float4 *__restrict__ aux, float *__restrict__ bvw) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || *bad) return;
    const float d = delta[i];
    float *r = elems + (size_t)i * 16 + (D == 2 ? 6 : 12);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < D; k++) {
        const float g = r[k] + d;
        r[k] = g;
        s = k == 0 ? fabsf(g) : s + fabsf(g);
    }
    const float area = D == 2 ? elems[(size_t)i * 16 + 10] : aux[i].w;
    bvw[i] = area * s / (float)D;
}

// The build's scratch, one allocation: take() first adds up the sizes, after allocate() it hands out
// the pointers in the same order.
struct Tmp {
    cudaStream_t stream;
    char *base = nullptr;
    size_t used = 0;
    explicit Tmp(cudaStream_t st) : stream(st) {}
    ~Tmp() { scratch_free(base, stream); }
    template <class T> void take(T **p, size_t count) {
        *p = base ? (T *)(base + used) : nullptr;
        used += (std::max<size_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
    }
    cudaError_t allocate() {
        void *q = nullptr;
        const cudaError_t e = scratch_alloc(&q, used, stream);
        if (e == cudaSuccess) base = (char *)q;
        used = 0;
        return e;
    }
};

inline uint32_t blocks(uint64_t n) { return (uint32_t)((n + kT - 1) / kT); }

template <int D>
std::string build_impl(uint32_t n, const float *verts, const float *normals, const float *bvals, const float *alphas,
                       const int32_t *types, cudaStream_t st, DeviceSceneBuild &out, cudaError_t &ce) {
    Tmp tmp(st);
#define WOB_CK(x)                            \
    do {                                     \
        if ((ce = (x)) != cudaSuccess) return "CUDA error"; \
    } while (0)
    const uint32_t n2 = sort_padded(n), n_int = n > 1 ? n - 1 : 1;
    float *box, *ibox, *areas, *bvw;
    Bounds *bd;
    uint64_t *key;
    uint32_t *val, *child, *first, *last, *pint, *pleaf, *flags, *blk;
    unsigned char *kahan;
    auto lay_out = [&]() {
        tmp.take(&key, n2);
        tmp.take(&bd, 1);
        tmp.take(&kahan, kahan_scratch_bytes(n, 2));
        tmp.take(&val, n2);
        tmp.take(&box, (size_t)n * 9);
        tmp.take(&areas, n);
        tmp.take(&bvw, n);
        tmp.take(&child, 2 * (size_t)n_int);
        for (uint32_t **p : {&first, &last, &pint, &flags}) tmp.take(p, n_int);
        tmp.take(&pleaf, n);
        tmp.take(&ibox, 6 * (size_t)n_int);
        tmp.take(&blk, n_int / kT + 1);
    };
    lay_out();  // measures; after the allocation the same calls hand out the pointers
    WOB_CK(tmp.allocate());
    lay_out();
    Bounds init;
    for (int k = 0; k < 3; k++) {
        init.lo[k] = init.clo[k] = 0xFFFFFFFFu;
        init.hi[k] = init.chi[k] = 0u;
    }
    init.mag = 0u;
    init.bad = 0u;
    init.all_dirichlet = 1u;
    init.n_nodes = init.depth = 0u;
    init.totals[0] = init.totals[1] = 0.0f;
    WOB_CK(cudaMemcpyAsync(bd, &init, sizeof(Bounds), cudaMemcpyHostToDevice, st));
    k_validate<D><<<blocks(n), kT, 0, st>>>(n, verts, normals, bvals, alphas, types, box, bd);
    WOB_CK(cudaGetLastError());

    // Morton codes and the sort
    k_morton<D><<<blocks(n2), kT, 0, st>>>(n, n2, box, bd, key, val);
    WOB_CK(cudaGetLastError());
    WOB_CK(launch_sort_keys(n2, key, val, st));

    constexpr int NF = D == 2 ? 24 : 32;
    float *nodes = nullptr;
    WOB_CK(cudaMalloc(&nodes, (size_t)n_int * NF * 4));
    out.nodes = nodes;
    out.nodes_bytes = (size_t)n_int * NF * 4;
    if (n <= kLeafMax) {
        // one wide node holding one leaf (scene_build.cpp)
        std::vector<float> root(NF, 0.0f);
        std::vector<float> hbox(9 * (size_t)n);
        Bounds hb;
        WOB_CK(cudaMemcpyAsync(hbox.data(), box, hbox.size() * 4, cudaMemcpyDeviceToHost, st));
        WOB_CK(cudaMemcpyAsync(&hb, bd, sizeof(Bounds), cudaMemcpyDeviceToHost, st));
        WOB_CK(cudaStreamSynchronize(st));
        const float pad = box_pad(hb, D);
        for (int a = 0; a < D; a++) {
            float lo = INFINITY, hi = -INFINITY;
            for (uint32_t i = 0; i < n; i++) {
                lo = std::min(lo, hbox[9 * i + a] - pad);
                hi = std::max(hi, hbox[9 * i + 3 + a] + pad);
            }
            root[4 * a] = lo;
            root[4 * (D + a)] = hi;
        }
        const uint32_t codes[4] = {make_leaf(0, n), kChildEmpty, kChildEmpty, kChildEmpty};
        for (int k = 0; k < 4; k++) std::memcpy(&root[4 * (2 * D) + k], &codes[k], 4);
        WOB_CK(cudaMemcpyAsync(nodes, root.data(), NF * 4, cudaMemcpyHostToDevice, st));
        WOB_CK(cudaStreamSynchronize(st));
    } else {
        WOB_CK(cudaMemsetAsync(flags, 0, (size_t)n_int * 4, st));
        k_radix_tree<<<blocks(n - 1), kT, 0, st>>>(n, key, child, first, last, pint, pleaf);
        k_boxes<<<blocks(n), kT, 0, st>>>(n, D, val, box, child, pint, pleaf, flags, ibox, bd);
        uint32_t *rank = flags;  // the boxes' arrival counts are done with
        k_wide_mark<<<blocks(n_int), kT, 0, st>>>(n_int, first, last, pint, rank, blk, bd);
        k_scan<<<1, 1024, 0, st>>>(blocks(n_int), blk, &bd->n_nodes);
        k_wide_write<D><<<blocks(n_int), kT, 0, st>>>(n_int, rank, blk, child, first, last, val, box, ibox, bd, nodes);
        WOB_CK(cudaGetLastError());
    }

    // records, CDFs, guides
    const int EF = 16;
    float *elems = nullptr, *elem_aux = nullptr, *isect = nullptr, *area_cdf = nullptr, *bv_cdf = nullptr;
    WOB_CK(cudaMalloc(&elems, (size_t)n * EF * 4));
    out.elems = elems;
    out.elems_bytes = (size_t)n * EF * 4;
    if (D == 3) {
        WOB_CK(cudaMalloc(&elem_aux, (size_t)n * 4 * 4));
        out.elem_aux = elem_aux;
        out.elem_aux_bytes = (size_t)n * 4 * 4;
        WOB_CK(cudaMalloc(&isect, (size_t)n * 16 * 4));
        out.isect = isect;
        out.isect_bytes = (size_t)n * 16 * 4;
    }
    WOB_CK(cudaMalloc(&area_cdf, (size_t)n * 4));
    out.area_cdf = area_cdf;
    out.area_cdf_bytes = (size_t)n * 4;
    WOB_CK(cudaMalloc(&bv_cdf, (size_t)n * 4));
    out.bv_cdf = bv_cdf;
    out.bv_cdf_bytes = (size_t)n * 4;
    k_records<D><<<blocks(n), kT, 0, st>>>(n, val, verts, normals, bvals, alphas, types, elems, elem_aux, isect, areas,
                                           bvw);
    const float *weights[2] = {areas, bvw};
    float *cdfs[2] = {area_cdf, bv_cdf};
    WOB_CK(launch_kahan_cdf(n, 2, weights, cdfs, bd->totals, kahan, st));
    Bounds hb;
    WOB_CK(cudaMemcpyAsync(&hb, bd, sizeof(Bounds), cudaMemcpyDeviceToHost, st));
    out.order.resize(n);
    WOB_CK(cudaMemcpyAsync(out.order.data(), val, (size_t)n * 4, cudaMemcpyDeviceToHost, st));
    WOB_CK(cudaStreamSynchronize(st));
    if (hb.bad & 1u) return "vertices must be finite";
    if (hb.bad & 2u) return "normals must be finite";
    if (hb.bad & 4u) return "boundary values must be finite";
    if (hb.bad & 8u) return "robin alphas must be finite";
    if (hb.bad & 16u) return "boundary_types must be 0 (Dirichlet), 1 (Neumann) or 2 (Robin)";
    if (hb.bad & 32u) return "normals must be unit vectors";
    if (hb.bad & kBadTree) return "BVH build failed: malformed radix tree";
    out.all_dirichlet = hb.all_dirichlet != 0u;
    out.n_nodes = n <= kLeafMax ? 1u : hb.n_nodes;
    out.depth = n <= kLeafMax ? 1u : hb.depth;
    if (3 * out.depth + 2 > kTraversalStack) return "BVH too deep for the traversal stack";
    out.total_area = hb.totals[0];
    out.total_bv = hb.totals[1];
    if (!(out.total_area > 0.0f) || !std::isfinite(out.total_area)) return "total boundary area must be positive and finite";
    const uint32_t G = guide_records(n);
    uint32_t *ag = nullptr, *bg = nullptr;
    WOB_CK(cudaMalloc(&ag, (size_t)G * 16));
    out.area_guide = ag;
    out.area_guide_bytes = (size_t)G * 16;
    out.area_G = G;
    WOB_CK(launch_guide(n, G, area_cdf, ag, st));
    out.bv_valid = out.total_bv > 0.0f && std::isfinite(out.total_bv);
    const uint32_t Gb = out.bv_valid ? G : 1u;
    WOB_CK(cudaMalloc(&bg, (size_t)Gb * 16));
    out.bv_guide = bg;
    out.bv_guide_bytes = (size_t)Gb * 16;
    out.bv_G = Gb;
    if (out.bv_valid) WOB_CK(launch_guide(n, G, bv_cdf, bg, st));
    else WOB_CK(cudaMemsetAsync(bg, 0, 16, st));
    WOB_CK(cudaStreamSynchronize(st));
#undef WOB_CK
    return "";
}

}  // namespace

size_t offset_scratch_bytes(uint32_t n) { return 256 + ((size_t)n * 4 + 255) / 256 * 256 + kahan_scratch_bytes(n, 1); }

cudaError_t launch_boundary_offsets(int dim, uint32_t n, const float *delta, float *elems, const float4 *aux,
                                    float *bv_cdf, uint32_t G, uint32_t *bv_guide, void *scratch, cudaStream_t st) {
    uint32_t *head = (uint32_t *)scratch;  // OffsetResult
    float *bvw = (float *)((char *)scratch + 256);
    void *kahan = (char *)scratch + 256 + ((size_t)n * 4 + 255) / 256 * 256;
    cudaError_t e = cudaMemsetAsync(head, 0, sizeof(OffsetResult), st);
    if (e != cudaSuccess) return e;
    k_check_offsets<<<blocks(n), kT, 0, st>>>(n, delta, head);
    if (dim == 2) k_offset_weights<2><<<blocks(n), kT, 0, st>>>(n, delta, head, elems, aux, bvw);
    else k_offset_weights<3><<<blocks(n), kT, 0, st>>>(n, delta, head, elems, aux, bvw);
    const float *w[1] = {bvw};
    float *cdf[1] = {bv_cdf};
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = launch_kahan_cdf(n, 1, w, cdf, (float *)(head + 1), kahan, st)) != cudaSuccess)
        return e;
    return launch_guide(n, G, bv_cdf, bv_guide, st);
}

void DeviceSceneBuild::release() {
    for (void **p : {&elems, &elem_aux, &isect, &nodes, &area_cdf, &area_guide, &bv_cdf, &bv_guide}) {
        if (*p) cudaFree(*p);
        *p = nullptr;
    }
}

std::string build_device_scene(int dim, uint32_t n, const float *verts, const float *normals, const float *bvals,
                               const float *alphas, const int32_t *types, cudaStream_t stream, DeviceSceneBuild &out,
                               cudaError_t &cuda_error) {
    cuda_error = cudaSuccess;
    if (dim != 2 && dim != 3) return "dim must be 2 or 3";
    if (n == 0) return "a scene needs at least one element";
    if (n > kMaxElements) return "too many elements";
    if (!verts || !normals || !bvals || !types) return "vertices, normals, boundary_values and boundary_types are required";
    std::string err = dim == 2 ? build_impl<2>(n, verts, normals, bvals, alphas, types, stream, out, cuda_error)
                               : build_impl<3>(n, verts, normals, bvals, alphas, types, stream, out, cuda_error);
    if (!err.empty()) out.release();
    return err;
}

}  // namespace wobgb
