// Dense triangle sums of the learned control variate for the single-layer Neumann estimators.
//
// The control variate is a density sigma~ that is constant on every stored triangle (the network
// evaluated at the triangle's centroid). Two sums over all triangles i of the scene use it:
//
//   residual data (targets: the centroids c_j of the triangles, with their normals n_j):
//     (T sigma~)(c_j) = -c / (4 pi) sum_i sigma~_i n_j . grad P_i(c_j),   c = +2 inside, -2 outside,
//     delta_j = ((T sigma~)(c_j) - sigma~_j) / c,
//   where T(x, y) = -c dG/dn_x is the kernel of the single-layer Neumann equation
//   sigma = c g + T sigma (bie_models.cuh:262-316: fredholm_equation_boundary_known / _unknown).
//   Adding delta_j to the Neumann data of triangle j turns the walk's source c g into
//   c g + T sigma~ - sigma~, whose solution is the residual sigma - sigma~;
//
//   potential (targets: evaluation points x): u~(x) = (1/4 pi) sum_i sigma~_i P_i(x) and its
//   gradient, the single-layer potential of sigma~ (solution_domain_unknown, bie_models.cuh:225-240).
//
// P_i(x) is the integral of 1/|x - y| over triangle i. Pairs farther apart than near_factor times
// the triangle's longest edge use the centroid rule A_i / |x - c_i|; nearer pairs use the closed
// form of the potential of a uniformly charged flat triangle and its gradient (Wilton et al.,
// IEEE Trans. Antennas Propag. 32(3), 1984), with coordinates taken relative to the target. A
// triangle's own term in the residual data is zero: n_j is normal to triangle j, so dG/dn_x
// vanishes on it.
//
// Far field by a treecode over consecutive stored triangles (BVH storage order keeps them
// spatially compact): clusters of 32, groups of 8 clusters (256 triangles) and groups of 8 of
// those (2048), each record with its centre z (mean centroid), radius rho, largest near radius eta
// and the moments of its centroid sources about z up to the quadrupole (M0 = sum w, M1 = sum w d,
// M2 = sum w d d^T, w = sigma~ A, d = c - z). A block takes 32 consecutive targets and the
// bounding sphere (W, omega) of their positions; a record with |W - z| > max(rho / theta,
// rho + eta) + omega is far from every target of the block and enters through its quadrupole
// expansion of sum w / |x - c| (one evaluation per target for all its triangles, error of order
// (rho / |x - z|)^3 of its share). The block starts from the largest groups and looks into the
// near ones; a near cluster is taken triangle by triangle as above. theta = 0 takes every
// triangle (the dense sum). The decisions are uniform across the block, so lanes never diverge.
//
// Work decomposition: one block per 32 targets (a lane each). Its threads decide the records, a record
// each; its 8 warps take the far records, then the near clusters, then the closed forms in turn,
// records read as broadcasts; FP32 partial sums over 32 items, FP64 across them and across the warps
// (in warp order: deterministic).
// This unit is compiled with FMA contraction (it is not part of the bit-exact walk).
#include "device_common.cuh"
#include "launch.hpp"
#include "sort_keys.hpp"

namespace wobgb {

namespace {

constexpr int kCvBlock = 256;
constexpr int kCvWarps = kCvBlock / 32;
constexpr uint32_t kNearList = 256;  // near triangles a warp lists; further ones it sums at once
constexpr double kInv4Pi = 0.07957747154594767;

struct TriVerts {
    float a[3], b[3], c[3];
};

__device__ __forceinline__ TriVerts load_tri(const SceneView<3> &s, uint32_t i) {
    const float4 *p = s.elems + 4 * i;
    const float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
    TriVerts t;
    t.a[0] = q0.x; t.a[1] = q0.y; t.a[2] = q0.z;
    t.b[0] = q0.w; t.b[1] = q1.x; t.b[2] = q1.y;
    t.c[0] = q1.z; t.c[1] = q1.w; t.c[2] = q2.x;
    return t;
}

// What the closed form needs of a triangle alone, computed once per table (TriGeom): the unit normal and
// its length before normalisation (twice the area; 0: degenerate, no contribution), and the three
// edges' unit directions and lengths.
struct TriGeom {
    float4 n, s[3];
};
__device__ __forceinline__ TriGeom triangle_geometry(const TriVerts &t) {
    const float *vs[4] = {t.a, t.b, t.c, t.a};
    TriGeom g;
    float e[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        for (int k = 0; k < 3; k++) e[i][k] = vs[i + 1][k] - vs[i][k];
        const float l = sqrtf(e[i][0] * e[i][0] + e[i][1] * e[i][1] + e[i][2] * e[i][2]);
        g.s[i] = make_float4(e[i][0] / l, e[i][1] / l, e[i][2] / l, l);
    }
    // (b - a) x (c - a), c - a = -(a - c)
    const float x = e[0][2] * e[2][1] - e[0][1] * e[2][2], y = e[0][0] * e[2][2] - e[0][2] * e[2][0],
                z = e[0][1] * e[2][0] - e[0][0] * e[2][1];
    const float nl = sqrtf(x * x + y * y + z * z);
    g.n = nl > 0.0f ? make_float4(x / nl, y / nl, z / nl, nl) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return g;
}

// P(x) = integral over the triangle of 1 / |x - y| dA and grad P(x), closed form (FP32; the
// coordinates are taken relative to x so that near pairs keep their relative precision). Per edge the
// logarithm ln((R+ + s+) / (R- + s-)), in the form without cancellation for the edge's side of the
// projection and for points near the edge's line; the three edges' arctangent terms add up to the
// triangle's solid angle, taken at once (Van Oosterom and Strackee, IEEE Trans. Biomed. Eng. 30(2),
// 1983) instead of two arctangents and two divisions per edge. Error against 64 bits, 2-norm of the
// gradient on 80, 1,280 and 5,120 triangles at points 1e-4 to 0.3 from the surface: 6.2e-7, 4.2e-7 and
// 3.0e-7 (3.7e-4, 9.1e-5 and 2.5e-5 with arctangents per edge and the cancelling logarithm; 1.2e-3,
// 1.3e-4 and 5.3e-5 with the solid angle and the cancelling logarithm); residual data 1.1e-7, 2.2e-7, 4.4e-7.
__device__ __forceinline__ void triangle_potential(const float x[3], const TriVerts &t, const TriGeom &g, float &P,
                                                   float G[3]) {
    float v[3][3];  // the vertices relative to x
#pragma unroll
    for (int k = 0; k < 3; k++) {
        v[0][k] = t.a[k] - x[k];
        v[1][k] = t.b[k] - x[k];
        v[2][k] = t.c[k] - x[k];
    }
    auto dot = [](const float *p, const float *q) { return p[0] * q[0] + p[1] * q[1] + p[2] * q[2]; };
    const float n[3] = {g.n.x, g.n.y, g.n.z};
    const float h = -dot(v[0], n), ah = fabsf(h);  // (x - a) . n with x at the origin
    const float R[3] = {sqrtf(dot(v[0], v[0])), sqrtf(dot(v[1], v[1])), sqrtf(dot(v[2], v[2]))};
    P = 0.0f;
    G[0] = G[1] = G[2] = 0.0f;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const float sv[3] = {g.s[e].x, g.s[e].y, g.s[e].z};
        const float m[3] = {sv[1] * n[2] - sv[2] * n[1], sv[2] * n[0] - sv[0] * n[2], sv[0] * n[1] - sv[1] * n[0]};
        const float sm = dot(v[e], sv), sp = sm + g.s[e].w, tt = dot(v[e], m);
        const float Rm = R[e], Rp = R[(e + 1) % 3];
        const float q = tt * tt + h * h;  // squared distance to the edge's line
        const bool ahead = sm + sp >= 0.0f;
        const float num = ahead ? Rp + sp : Rm - sm, den = ahead ? Rm + sm : Rp - sp;
        // above the edge near its line the denominator cancels: R + s = q / (R - s) for the end behind
        const bool cancels = sm < 0.0f && sp > 0.0f && den < 0.25f * num;
        const float ratio = cancels ? (Rm - sm) * (Rp + sp) / q : num / den;
        // x on the edge's line: no contribution from this edge
        const float f = q > 0.0f ? logf(ratio) : 0.0f;
        P += tt * f;
#pragma unroll
        for (int k = 0; k < 3; k++) G[k] -= m[k] * f;
    }
    const float den = R[0] * R[1] * R[2] + dot(v[0], v[1]) * R[2] + dot(v[1], v[2]) * R[0] + dot(v[2], v[0]) * R[1];
    const float omega = 2.0f * atan2f(ah * g.n.w, den);
    P -= ah * omega;
    const float sg = h > 0.0f ? omega : (h < 0.0f ? -omega : 0.0f);
#pragma unroll
    for (int k = 0; k < 3; k++) G[k] -= sg * n[k];
}

__device__ __forceinline__ void centroid_of(const TriVerts &t, float c[3]) {
    for (int k = 0; k < 3; k++) c[k] = (t.a[k] + t.b[k] + t.c[k]) / 3.0f;
}

// Per stored triangle: {centroid, sigma~ * area}, the squared near radius and the closed form's geometry.
__global__ void cv_sources_kernel(SceneView<3> s, const float *__restrict__ sigma, float near_factor,
                                  float4 *__restrict__ src, float *__restrict__ near2, float4 *__restrict__ geom) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.n_elems) return;
    const TriVerts t = load_tri(s, i);
    float c[3];
    centroid_of(t, c);
    float e1[3], e2[3];
    for (int k = 0; k < 3; k++) { e1[k] = t.b[k] - t.a[k]; e2[k] = t.c[k] - t.a[k]; }
    const float cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2],
                cz = e1[0] * e2[1] - e1[1] * e2[0];
    const float area = 0.5f * sqrtf(cx * cx + cy * cy + cz * cz);
    float h2 = 0.0f;
    const float *vs[4] = {t.a, t.b, t.c, t.a};
    for (int e = 0; e < 3; e++) {
        float l2 = 0.0f;
        for (int k = 0; k < 3; k++) l2 += (vs[e + 1][k] - vs[e][k]) * (vs[e + 1][k] - vs[e][k]);
        h2 = fmaxf(h2, l2);
    }
    src[i] = make_float4(c[0], c[1], c[2], sigma[i] * area);
    near2[i] = near_factor * near_factor * h2;
    const TriGeom g = triangle_geometry(t);
    geom[4 * (size_t)i] = g.n;
    for (int e = 0; e < 3; e++) geom[4 * (size_t)i + 1 + e] = g.s[e];
}

constexpr int kClusterSize = 32;

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Morton order of evaluation points: bounds (order-preserving integer atomics), 30-bit codes (10
// bits a coordinate), a sort of {code, index} keys padded to a power of two (k_sort.cu).
__device__ __forceinline__ uint32_t ordered_bits(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ uint32_t spread_bits10(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__global__ void bounds_init_kernel(uint32_t *bb) {
    if (threadIdx.x < 6) bb[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
}
__global__ void pts_bounds_kernel(const float *__restrict__ pts, uint32_t n, uint32_t *__restrict__ bb) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < 3; k++) {
        const uint32_t o = i < n ? ordered_bits(pts[(size_t)i * 3 + k]) : 0u;
        const uint32_t lo = __reduce_min_sync(0xffffffffu, i < n ? o : 0xffffffffu), hi = __reduce_max_sync(0xffffffffu, o);
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(bb + k, lo);
            atomicMax(bb + 3 + k, hi);
        }
    }
}
__global__ void pts_morton_kernel(const float *__restrict__ pts, uint32_t n, uint32_t n2, const uint32_t *__restrict__ bb,
                                  uint64_t *__restrict__ key) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n2) return;
    if (i >= n) {
        key[i] = ~0ull;
        return;
    }
    uint32_t code = 0;
    for (int k = 0; k < 3; k++) {
        const float lo = from_ordered_bits(bb[k]), hi = from_ordered_bits(bb[3 + k]);
        const float t = hi > lo ? (pts[(size_t)i * 3 + k] - lo) / (hi - lo) : 0.0f;
        const uint32_t q = (uint32_t)fminf(fmaxf(t * 1024.0f, 0.0f), 1023.0f);
        code |= spread_bits10(q) << k;
    }
    key[i] = ((uint64_t)code << 32) | i;
}
// One warp per cluster: the record {z, r_far}, {M0, M1}, {M2xx, M2yy, M2zz, M2xy}, {M2xz, M2yz,
// trace M2, rho + eta}; r_far = max(rho / theta, rho + eta), infinite for theta = 0.
__global__ void cv_cluster_kernel(uint32_t n, const float4 *__restrict__ src, const float *__restrict__ near2,
                                  float theta, float4 *__restrict__ cl) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_cl = (n + kClusterSize - 1) / kClusterSize;
    if (k >= n_cl) return;
    const uint32_t i = k * kClusterSize + lane;
    const bool valid = i < n;
    const float4 q = valid ? __ldg(src + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float e2 = valid ? __ldg(near2 + i) : 0.0f;
    const float cnt = (float)__popc(__ballot_sync(0xffffffffu, valid));
    const float zx = warp_sum_f(q.x) / cnt, zy = warp_sum_f(q.y) / cnt, zz = warp_sum_f(q.z) / cnt;
    const float dx = valid ? q.x - zx : 0.0f, dy = valid ? q.y - zy : 0.0f, dz = valid ? q.z - zz : 0.0f;
    const float rho = sqrtf(warp_max_f(dx * dx + dy * dy + dz * dz));
    const float eta = sqrtf(warp_max_f(e2));
    const float w = q.w;
    const float m0 = warp_sum_f(w);
    const float m1x = warp_sum_f(w * dx), m1y = warp_sum_f(w * dy), m1z = warp_sum_f(w * dz);
    const float mxx = warp_sum_f(w * dx * dx), myy = warp_sum_f(w * dy * dy), mzz = warp_sum_f(w * dz * dz);
    const float mxy = warp_sum_f(w * dx * dy), mxz = warp_sum_f(w * dx * dz), myz = warp_sum_f(w * dy * dz);
    if (lane == 0) {
        const float r_far = theta > 0.0f ? fmaxf(rho / theta, rho + eta) : __int_as_float(0x7f800000);
        cl[4 * k + 0] = make_float4(zx, zy, zz, r_far);
        cl[4 * k + 1] = make_float4(m0, m1x, m1y, m1z);
        cl[4 * k + 2] = make_float4(mxx, myy, mzz, mxy);
        cl[4 * k + 3] = make_float4(mxz, myz, mxx + myy + mzz, rho + eta);
    }
}

// Groups of kGroupFan^L clusters (L = 1, 2: 256 and 2048 consecutive stored triangles), one block
// of 256 threads each: the same record as a cluster's, from the member sources directly (centre =
// mean centroid, exact radius, largest near radius, moments about the centre).
constexpr int kGroupFan = 8;
constexpr int kGroupBlock = 256;
__device__ __forceinline__ float block_reduce(float v, bool is_max, float *red) {
    v = is_max ? warp_max_f(v) : warp_sum_f(v);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = red[0];
    for (int w = 1; w < kGroupBlock / 32; w++) t = is_max ? fmaxf(t, red[w]) : t + red[w];
    __syncthreads();
    return t;
}
template <uint32_t kSize>
__global__ void __launch_bounds__(kGroupBlock) cv_group_kernel(uint32_t n, const float4 *__restrict__ src,
                                                               const float *__restrict__ near2, float theta,
                                                               float4 *__restrict__ rec) {
    __shared__ float red[kGroupBlock / 32];
    const uint32_t g = blockIdx.x, i0 = g * kSize, i1 = min(n, i0 + kSize);
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    for (uint32_t i = i0 + threadIdx.x; i < i1; i += kGroupBlock) {
        const float4 q = __ldg(src + i);
        sx += q.x;
        sy += q.y;
        sz += q.z;
    }
    const float cnt = (float)(i1 - i0);
    const float zx = block_reduce(sx, false, red) / cnt, zy = block_reduce(sy, false, red) / cnt,
                zz = block_reduce(sz, false, red) / cnt;
    float r2 = 0.0f, e2 = 0.0f, m[10] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    for (uint32_t i = i0 + threadIdx.x; i < i1; i += kGroupBlock) {
        const float4 q = __ldg(src + i);
        const float dx = q.x - zx, dy = q.y - zy, dz = q.z - zz, w = q.w;
        r2 = fmaxf(r2, dx * dx + dy * dy + dz * dz);
        e2 = fmaxf(e2, __ldg(near2 + i));
        m[0] += w;
        m[1] += w * dx; m[2] += w * dy; m[3] += w * dz;
        m[4] += w * dx * dx; m[5] += w * dy * dy; m[6] += w * dz * dz;
        m[7] += w * dx * dy; m[8] += w * dx * dz; m[9] += w * dy * dz;
    }
    const float rho = sqrtf(block_reduce(r2, true, red)), eta = sqrtf(block_reduce(e2, true, red));
#pragma unroll
    for (int k = 0; k < 10; k++) m[k] = block_reduce(m[k], false, red);
    if (threadIdx.x == 0) {
        const float r_far = theta > 0.0f ? fmaxf(rho / theta, rho + eta) : __int_as_float(0x7f800000);
        rec[4 * g + 0] = make_float4(zx, zy, zz, r_far);
        rec[4 * g + 1] = make_float4(m[0], m[1], m[2], m[3]);
        rec[4 * g + 2] = make_float4(m[4], m[5], m[6], m[7]);
        rec[4 * g + 3] = make_float4(m[8], m[9], m[4] + m[5] + m[6], 0.0f);
    }
}

__host__ __device__ __forceinline__ uint32_t div_up(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// sum w / |x - c| over a cluster by its quadrupole expansion about z (R = x - z):
//   phi = M0 / R + (R . M1) / R^3 + (3 R.M2.R - R^2 tr M2) / (2 R^5),
// and its gradient term by term.
__device__ __forceinline__ void cluster_field(const float x[3], const float4 &q0, const float4 &q1, const float4 &q2,
                                             const float4 &q3, float &phi, float g[3]) {
    const float R[3] = {x[0] - q0.x, x[1] - q0.y, x[2] - q0.z};
    const float R2 = R[0] * R[0] + R[1] * R[1] + R[2] * R[2];
    const float ri = rsqrtf(R2);
    const float ri2 = ri * ri, ri3 = ri * ri2, ri5 = ri3 * ri2;
    const float RM1 = R[0] * q1.y + R[1] * q1.z + R[2] * q1.w;
    const float M2R[3] = {q2.x * R[0] + q2.w * R[1] + q3.x * R[2], q2.w * R[0] + q2.y * R[1] + q3.y * R[2],
                          q3.x * R[0] + q3.y * R[1] + q2.z * R[2]};
    const float RM2R = R[0] * M2R[0] + R[1] * M2R[1] + R[2] * M2R[2];
    const float Q = 3.0f * RM2R - R2 * q3.z;
    phi = q1.x * ri + RM1 * ri3 + 0.5f * Q * ri5;
    const float a = -q1.x * ri3 - 3.0f * RM1 * ri5 - q3.z * ri5 - 2.5f * Q * ri5 * ri2;
    const float m1[3] = {q1.y, q1.z, q1.w};
#pragma unroll
    for (int k = 0; k < 3; k++) g[k] = a * R[k] + m1[k] * ri3 + 3.0f * M2R[k] * ri5;
}

// kMode 0: residual data at the stored triangles' centroids; kMode 1: potential and gradient at
// points (out: [n][4] = u, du/dx, du/dy, du/dz).
constexpr uint32_t kItems = 32 * kGroupFan * kGroupFan;  // clusters of a batch: far and near records together
constexpr uint32_t kCheckNear = 0x80000000u;
static_assert(32 * kGroupFan == kCvBlock, "a thread per middle group of a batch");
template <int kMode>
__global__ void __launch_bounds__(kCvBlock, 4) cv_sum_kernel(SceneView<3> s, const float4 *__restrict__ src,
                                                          const float *__restrict__ near2,
                                                          const float4 *__restrict__ geom,
                                                          const float *__restrict__ sigma,
                                                          const float4 *__restrict__ cl, const float *__restrict__ pts,
                                                          const uint64_t *__restrict__ order, uint32_t n_targets,
                                                          float c_coef, float *__restrict__ out,
                                                          double *__restrict__ part_sums) {
    __shared__ double s_acc[kCvWarps][4][32];
    // triangles within some target's near radius, found by each warp in its order and, once all are
    // found, dealt to the warps in turn: a block's closed forms sit in the few clusters around its
    // targets, and the warps that met them kept the others waiting
    __shared__ uint32_t s_near[kCvWarps][kNearList];
    __shared__ uint32_t s_count[kCvWarps];
    __shared__ uint32_t s_items[kItems], s_open[32 * kGroupFan], s_tally[kCvWarps];
    uint32_t n_near = 0;
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
    const uint32_t slot = blockIdx.x * 32u + lane;
    const bool active = slot < n_targets;
    // points are taken in Morton order (order: sorted {code, index} keys), so that the 32 targets
    // of a block are close together; triangles are already (BVH storage order)
    const uint32_t tgt = (kMode == 1 && active) ? (uint32_t)__ldg(order + slot) : slot;
    const uint32_t act = __ballot_sync(0xffffffffu, active);
    float xd[3] = {0.0f, 0.0f, 0.0f}, nn[3] = {0.0f, 0.0f, 0.0f};
    if (active) {
        if (kMode == 0) {
            const TriVerts tv = load_tri(s, tgt);
            centroid_of(tv, xd);
            const float4 q2 = __ldg(s.elems + 4 * tgt + 2);
            nn[0] = q2.y; nn[1] = q2.z; nn[2] = q2.w;
        } else {
            for (int k = 0; k < 3; k++) xd[k] = pts[(size_t)tgt * 3 + k];
        }
    }
    // the bounding sphere of the block's targets
    const float cnt = (float)__popc(act);
    const float Wx = warp_sum_f(xd[0]) / cnt, Wy = warp_sum_f(xd[1]) / cnt, Wz = warp_sum_f(xd[2]) / cnt;
    const float ox = xd[0] - Wx, oy = xd[1] - Wy, oz = xd[2] - Wz;
    const float om = sqrtf(warp_max_f(active ? ox * ox + oy * oy + oz * oz : 0.0f));
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const uint32_t n_src = s.n_elems;
    const uint32_t n_cl = div_up(n_src, kClusterSize), n_g1 = div_up(n_cl, kGroupFan), n_g2 = div_up(n_g1, kGroupFan);
    uint32_t taken = 0;
    // far from every target of the block: |W - z| > r_far + omega
    auto is_far = [&](const float4 &q0) {
        const float Dx = Wx - q0.x, Dy = Wy - q0.y, Dz = Wz - q0.z;
        const float thr = q0.w + om;
        return Dx * Dx + Dy * Dy + Dz * Dz > thr * thr;
    };
    // a record's expansion at this lane's target; FP32 partial sums flushed to FP64 every 32 items
    auto expand = [&](const float4 *r) {
        const float4 q0 = __ldg(r), q1 = __ldg(r + 1), q2 = __ldg(r + 2), q3 = __ldg(r + 3);
        float phi, g[3];
        cluster_field(xd, q0, q1, q2, q3, phi, g);
        if (kMode == 0) {
            a[0] -= g[0] * nn[0] + g[1] * nn[1] + g[2] * nn[2];
        } else {
            a[0] += phi;
            a[1] += g[0];
            a[2] += g[1];
            a[3] += g[2];
        }
    };
    auto flush = [&]() {
        if ((++taken & 31u) == 0u) {
#pragma unroll
            for (int c = 0; c < (kMode == 0 ? 1 : 4); c++) {
                acc[c] += a[c];
                a[c] = 0.0f;
            }
        }
    };
    // triangle i's closed form at this lane's target where it is near
    auto closed_form = [&](uint32_t i, bool near) {
        if (!near || !active || (kMode == 0 && i == tgt)) return;
        const float4 *q = geom + 4 * (size_t)i;
        TriGeom g;
        g.n = __ldg(q);
        if (!(g.n.w > 0.0f)) return;
        for (int e = 0; e < 3; e++) g.s[e] = __ldg(q + 1 + e);
        float P, G[3];
        triangle_potential(xd, load_tri(s, i), g, P, G);
        const float sg = __ldg(sigma + i);
        if (kMode == 0) {
            a[0] -= sg * (G[0] * nn[0] + G[1] * nn[1] + G[2] * nn[2]);
        } else {
            a[0] += sg * P;
            a[1] += sg * G[0];
            a[2] += sg * G[1];
            a[3] += sg * G[2];
        }
    };
    // a source by the centroid rule (0 where `near`, also for a density that is not finite)
    auto centroid_rule = [&](const float4 &q, float dx, float dy, float dz, float r2, bool near) {
        const float rinv = near ? 0.0f : rsqrtf(r2), w = near ? 0.0f : q.w;
        const float r3 = rinv * rinv * rinv;
        if (kMode == 0) {
            a[0] += w * (dx * nn[0] + dy * nn[1] + dz * nn[2]) * r3;
        } else {
            a[0] += w * rinv;
            const float wr3 = w * r3;
            a[1] -= wr3 * dx;
            a[2] -= wr3 * dy;
            a[3] -= wr3 * dz;
        }
    };
    // The records are decided a thread each, in batches of 32 largest groups (at most 2048 clusters): far
    // ones are listed from the front of s_items, near clusters from its back, in a fixed order, and the
    // warps then take the two lists in turn. Deciding in every warp, all lanes alike, was a sixth of the
    // instructions, and dealing by index left the warps unevenly loaded. The largest groups are also
    // split over gridDim.y blocks of the same targets (part blockIdx.y takes k2 = part, part +
    // gridDim.y, ...), whose sums part_sums holds for cv_parts_kernel.
    uint32_t n_far = 0, n_cls = 0;  // the lists' lengths (the same in every thread)
    // appends `item` of the threads with `far` / `cls`, in thread order
    auto append = [&](bool far, bool cls, uint32_t item) {
        const uint32_t bf = __ballot_sync(0xffffffffu, far), bc = __ballot_sync(0xffffffffu, cls);
        if (lane == 0) s_tally[wid] = (uint32_t)__popc(bf) | ((uint32_t)__popc(bc) << 16);
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (uint32_t w = 0; w < kCvWarps; w++) {
            const uint32_t c = s_tally[w];
            if (w < wid) before += c;
            all += c;
        }
        const uint32_t lt = (1u << lane) - 1u;
        if (far) s_items[n_far + (before & 0xffffu) + (uint32_t)__popc(bf & lt)] = item;
        if (cls) s_items[kItems - 1u - (n_cls + (before >> 16) + (uint32_t)__popc(bc & lt))] = item;
        n_far += all & 0xffffu;
        n_cls += all >> 16;
        __syncthreads();
    };
    for (uint32_t b0 = blockIdx.y; b0 < n_g2; b0 += 32u * gridDim.y) {
        n_far = n_cls = 0;
        // the largest groups; near ones are opened (kept as the block's near list for a moment)
        const uint32_t k2 = b0 + threadIdx.x * gridDim.y;
        const bool in2 = threadIdx.x < 32u && k2 < n_g2;
        const bool far2 = in2 && is_far(__ldg(cl + 4 * (size_t)(n_cl + n_g1 + k2)));
        append(far2, in2 && !far2, far2 ? n_cl + n_g1 + k2 : k2);
        const uint32_t open2 = n_cls;
        const uint32_t slot1 = threadIdx.x / kGroupFan;
        const uint32_t k1 = slot1 < open2 ? s_items[kItems - 1u - slot1] * kGroupFan + threadIdx.x % kGroupFan : n_g1;
        const bool in1 = k1 < n_g1, far1 = in1 && is_far(__ldg(cl + 4 * (size_t)(n_cl + k1)));
        __syncthreads();
        n_cls = 0;
        append(far1, in1 && !far1, far1 ? n_cl + k1 : k1);
        const uint32_t open1 = n_cls;
        if (threadIdx.x < open1) s_open[threadIdx.x] = s_items[kItems - 1u - threadIdx.x];
        __syncthreads();
        n_cls = 0;
        for (uint32_t t0 = 0; t0 < open1 * kGroupFan; t0 += kCvBlock) {
            const uint32_t slot = (t0 + threadIdx.x) / kGroupFan;
            const uint32_t k = slot < open1 ? s_open[slot] * kGroupFan + threadIdx.x % kGroupFan : n_cl;
            bool far = false, check = false;
            if (k < n_cl) {
                const float4 q0 = __ldg(cl + 4 * (size_t)k);
                far = is_far(q0);
                // can a member lie within a near radius of a target? (rounded towards yes)
                const float Dx = Wx - q0.x, Dy = Wy - q0.y, Dz = Wz - q0.z;
                const float reach = (__ldg(cl + 4 * (size_t)k + 3).w + om) * 1.00001f;
                check = !(Dx * Dx + Dy * Dy + Dz * Dz > reach * reach);
            }
            append(far, k < n_cl && !far, k | (check && !far ? kCheckNear : 0u));
        }
        for (uint32_t e = wid; e < n_far; e += kCvWarps) {
            expand(cl + 4 * (size_t)s_items[e]);
            flush();
        }
        for (uint32_t e = wid; e < n_cls; e += kCvWarps) {
            const uint32_t item = s_items[kItems - 1u - e], k = item & ~kCheckNear;
            const uint32_t i0 = k * kClusterSize, i1 = min(n_src, i0 + kClusterSize);
            if (item & kCheckNear) {
                for (uint32_t i = i0; i < i1; i++) {
                    const float4 q = __ldg(src + i);
                    const float dx = xd[0] - q.x, dy = xd[1] - q.y, dz = xd[2] - q.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    const bool near = r2 < __ldg(near2 + i);
                    centroid_rule(q, dx, dy, dz, r2, near);
                    if (__any_sync(0xffffffffu, near && active)) {
                        if (n_near < kNearList) {
                            if (lane == 0) s_near[wid][n_near] = i;
                            n_near++;
                        } else {
                            closed_form(i, near);
                        }
                    }
                }
            } else {
#pragma unroll 4
                for (uint32_t i = i0; i < i1; i++) {
                    const float4 q = __ldg(src + i);
                    const float dx = xd[0] - q.x, dy = xd[1] - q.y, dz = xd[2] - q.z;
                    centroid_rule(q, dx, dy, dz, dx * dx + dy * dy + dz * dz, false);
                }
            }
            flush();
        }
        __syncthreads();  // the lists are rebuilt by the next batch
    }
    if (lane == 0) s_count[wid] = n_near;
    __syncthreads();
    uint32_t at = wid;  // entry of the lists laid end to end
    for (uint32_t w = 0, base = 0; w < kCvWarps; base += s_count[w], w++) {
        for (; at < base + s_count[w]; at += kCvWarps) {
            const uint32_t i = s_near[w][at - base];
            const float4 q = __ldg(src + i);
            const float dx = xd[0] - q.x, dy = xd[1] - q.y, dz = xd[2] - q.z;
            closed_form(i, dx * dx + dy * dy + dz * dz < __ldg(near2 + i));
            flush();
        }
    }
#pragma unroll
    for (int c = 0; c < 4; c++) s_acc[wid][c][lane] = acc[c] + a[c];
    __syncthreads();
    if (wid != 0 || !active) return;
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int w = 0; w < kCvWarps; w++)
#pragma unroll
        for (int c = 0; c < 4; c++) t[c] += s_acc[w][c][lane];
    if (gridDim.y > 1) {
        double *ps = part_sums + ((size_t)blockIdx.y * n_targets + slot) * 4;
        for (int k = 0; k < 4; k++) ps[k] = t[k];
    } else if (kMode == 0) {
        const double c = (double)c_coef;
        const double Tsig = c * kInv4Pi * t[0];
        out[tgt] = (float)((Tsig - (double)__ldg(sigma + tgt)) / c);
    } else {
        for (int k = 0; k < 4; k++) out[(size_t)tgt * 4 + k] = (float)(kInv4Pi * t[k]);
    }
}

// The potential from its parts, added in part order (deterministic): part_sums [parts][slot][4]
// by Morton slot, out [n][4] by point.
__global__ void cv_parts_kernel(const double *__restrict__ part_sums, uint32_t parts, const uint64_t *__restrict__ order,
                                uint32_t n, float *__restrict__ out) {
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n) return;
    const uint32_t tgt = (uint32_t)__ldg(order + slot);
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t p = 0; p < parts; p++)
#pragma unroll
        for (int k = 0; k < 4; k++) t[k] += part_sums[((size_t)p * n + slot) * 4 + k];
#pragma unroll
    for (int k = 0; k < 4; k++) out[(size_t)tgt * 4 + k] = (float)(kInv4Pi * t[k]);
}

// Blocks of the same 32 points the potential's largest groups are split over: with one block per
// 32 points there are too few blocks to fill the GPU for the slice-sized point sets.
constexpr uint32_t kPotentialParts = 8;

// The network's input at every stored element: (centroid, normal), 2D padded with zeros.
template <int D>
__global__ void element_frames_kernel(SceneView<D> s, float *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= s.n_elems) return;
    const float4 *p = s.elems + 4 * i;
    float *o = out + (size_t)i * 6;
    if constexpr (D == 2) {
        const float4 q0 = __ldg(p), q1 = __ldg(p + 1);
        o[0] = (q0.x + q0.z) / 2.0f; o[1] = (q0.y + q0.w) / 2.0f; o[2] = 0.0f;
        o[3] = q1.x; o[4] = q1.y; o[5] = 0.0f;
    } else {
        const TriVerts t = load_tri(s, i);
        float c[3];
        centroid_of(t, c);
        const float4 q2 = __ldg(p + 2);
        o[0] = c[0]; o[1] = c[1]; o[2] = c[2];
        o[3] = q2.y; o[4] = q2.z; o[5] = q2.w;
    }
}

}  // namespace

template <int D> cudaError_t launch_element_frames(const SceneView<D> &s, float *out, cudaStream_t stream) {
    element_frames_kernel<D><<<(s.n_elems + 255) / 256, 256, 0, stream>>>(s, out);
    return cudaGetLastError();
}
template cudaError_t launch_element_frames<2>(const SceneView<2> &, float *, cudaStream_t);
template cudaError_t launch_element_frames<3>(const SceneView<3> &, float *, cudaStream_t);

cudaError_t launch_cv_sources(const SceneView<3> &s, const float *sigma, float near_factor, float theta, float4 *src,
                              float *near2, float4 *geom, float4 *clusters, cudaStream_t stream) {
    cv_sources_kernel<<<(s.n_elems + 255) / 256, 256, 0, stream>>>(s, sigma, near_factor, src, near2, geom);
    const uint32_t n_cl = div_up(s.n_elems, kClusterSize), n_g1 = div_up(n_cl, kGroupFan), n_g2 = div_up(n_g1, kGroupFan);
    cv_cluster_kernel<<<(n_cl * 32 + 255) / 256, 256, 0, stream>>>(s.n_elems, src, near2, theta, clusters);
    cv_group_kernel<kClusterSize * kGroupFan><<<n_g1, kGroupBlock, 0, stream>>>(s.n_elems, src, near2, theta,
                                                                               clusters + 4 * (size_t)n_cl);
    cv_group_kernel<kClusterSize * kGroupFan * kGroupFan><<<n_g2, kGroupBlock, 0, stream>>>(
        s.n_elems, src, near2, theta, clusters + 4 * (size_t)(n_cl + n_g1));
    return cudaGetLastError();
}

uint32_t cv_cluster_records(uint32_t n_elems) {
    const uint32_t n_cl = div_up(n_elems, kClusterSize), n_g1 = div_up(n_cl, kGroupFan);
    return n_cl + n_g1 + div_up(n_g1, kGroupFan);
}

cudaError_t launch_cv_residual(const SceneView<3> &s, const float4 *src, const float *near2, const float4 *geom,
                               const float4 *clusters,
                               const float *sigma, float c_coef, float *delta, cudaStream_t stream) {
    cv_sum_kernel<0><<<(s.n_elems + 31) / 32, kCvBlock, 0, stream>>>(s, src, near2, geom, sigma, clusters, nullptr, nullptr,
                                                                     s.n_elems, c_coef, delta, nullptr);
    return cudaGetLastError();
}

uint32_t cv_point_order_words(uint32_t n_points) {
    const uint32_t n2 = sort_padded(n_points);
    // n2 keys of 8 bytes, the 6 bound words (padded to 8), the parts' FP64 sums
    return 2 * n2 + 8 + kPotentialParts * n_points * 8;
}

cudaError_t launch_cv_potential(const SceneView<3> &s, const float4 *src, const float *near2, const float4 *geom,
                                const float4 *clusters,
                                const float *sigma, const float *pts, uint32_t n_points, uint32_t *scratch,
                                float *out, cudaStream_t stream) {
    if (n_points == 0) return cudaSuccess;
    const uint32_t n2 = sort_padded(n_points);
    uint64_t *key = (uint64_t *)scratch;
    uint32_t *bb = scratch + 2 * (size_t)n2;
    bounds_init_kernel<<<1, 32, 0, stream>>>(bb);
    pts_bounds_kernel<<<(n_points + 255) / 256, 256, 0, stream>>>(pts, n_points, bb);
    pts_morton_kernel<<<(n2 + 255) / 256, 256, 0, stream>>>(pts, n_points, n2, bb, key);
    const cudaError_t e = launch_sort_keys(n2, key, nullptr, stream);
    if (e != cudaSuccess) return e;
    double *part_sums = reinterpret_cast<double *>(scratch + 2 * (size_t)n2 + 8);
    cv_sum_kernel<1><<<dim3((n_points + 31) / 32, kPotentialParts), kCvBlock, 0, stream>>>(
        s, src, near2, geom, sigma, clusters, pts, key, n_points, 0.0f, out, part_sums);
    cv_parts_kernel<<<(n_points + 255) / 256, 256, 0, stream>>>(part_sums, kPotentialParts, key, n_points, out);
    return cudaGetLastError();
}

}  // namespace wobgb
