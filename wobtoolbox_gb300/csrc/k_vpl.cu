// Virtual-point-light (VPL) variant of the walk (apps/potential_flow_with_vpl.cu:43-88):
//
// 1. paths (PathComputeFunc, :77-88): path i starts at a uniform boundary sample y_i and its walk
//    returns the unknown boundary estimate mu_i (compute_sample_unknown_boundary) -- one thread per
//    path, Philox stream kStreamVpl, point 0, path index path_offset + i;
// 2. aggregation (AggregateFunc, :43-75): every evaluation point x sums, over all VPLs,
//    mu_i * G(y_i, x) * A and mu_i * dG/dx(y_i, x) * A (the single layer's solution_domain_unknown /
//    gradient_domain_unknown, A = total boundary area) -- an N_points x N_vpl dense sum of kernel
//    evaluations, FP32-issue bound. Partial sums are FP32 per tile of 256 VPLs; tile t goes to
//    split t mod 8, each split adds its tiles in order into FP64, and the 8 split sums of a point
//    are added in split order (the oracle does the same blocking, so the sums are bit-identical).
#include "kernels.cuh"
#include "vpl.hpp"

namespace wobgb {

namespace {

constexpr uint32_t kStreamVpl = 2u;
constexpr int kVplTile = 256;

template <int D>
__global__ void __launch_bounds__(kBlock, 6) vpl_paths_kernel(SceneView<D> s, WalkParams p, uint32_t n_paths,
                                                           float *__restrict__ vpl_p, float *__restrict__ vpl_mu,
                                                           unsigned long long *__restrict__ bounces) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long b = 0;
    if (i < n_paths) {
        Walker<D, kSingleLayer, kStratSingleLayer, false> w(s, p, kStreamVpl, 0u, p.path_offset + i);
        float ip;
        const BPoint<D> y = sample_uniform<D>(s, w.rng, ip);
        const float mu = w.unknown_boundary(y);
        for (int k = 0; k < D; k++) vpl_p[(size_t)i * D + k] = y.p.v[k];
        vpl_mu[i] = mu;
        b = w.bounces;
    }
    if (bounces) {
        const unsigned long long t = warp_sum_u64(b);
        if ((threadIdx.x & 31u) == 0 && t) atomicAdd(bounces, t);
    }
}

// One block serves 32 points with 8 warps; warp w sums the tiles t = w, w + 8, ... (all lanes read
// the same VPL at a time: one shared-memory broadcast), so 8 threads share a point's pairs and the
// grid fills the GPU even for a few ten thousand points. The 8 per-warp FP64 partial sums of a
// point are then added in warp order.
//
// A pair (point x, VPL y with value mu) adds mu G(y, x) A and mu dG/dx(y, x) A = mu w (y - x), with
// r = y - x, q = |r|^2 (equation_kernel.cuh:74-79, 115-121), in this form (the oracle restates it):
//   2D: mu G A = ku log(max(q, eps^2)), ku = mu (-A / (4 pi)) -- log(max(|r|, eps)) / (2 pi)
//       written as log(max(q, eps^2)) / (4 pi); mu w = kw / q for q >= eps^2, kw / (|r| eps) for
//       0 < q < eps^2, 0 at q = 0, kw = mu A / (2 pi);
//   3D: mu G A = ku / max(|r|, eps), mu w = ku / (|r| max(q, eps)) (0 at q = 0), ku = mu A / (4 pi).
// ku and kw are computed once per VPL when its tile is staged in shared memory ({y, ku, kw} in 2D,
// {y, ku} in 3D), so a pair costs one log or one more division and no per-pair scaling.
constexpr int kVplSplit = 8;

__global__ void __launch_bounds__(32 * kVplSplit) vpl_aggregate3_kernel(const float *__restrict__ vpl_p,
                                                                        const float *__restrict__ vpl_mu, uint32_t n_vpl,
                                                                        float area, float eps,
                                                                        const float *__restrict__ pts, uint32_t n_points,
                                                                        double *__restrict__ sum) {
    __shared__ float4 tile[kVplSplit][kVplTile];
    __shared__ double red[kVplSplit][32][4];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t pt = blockIdx.x * 32u + lane;
    const bool active = pt < n_points;
    V<3> x = vzero<3>();
    if (active)
        for (int k = 0; k < 3; k++) x.v[k] = __ldg(pts + (size_t)pt * 3 + k);
    const float cu = 0x1.45f306p-4f * area;  // A/(4 pi)
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const uint32_t n_tiles = (n_vpl + kVplTile - 1) / kVplTile;
    for (uint32_t t = w; t < n_tiles; t += kVplSplit) {
        const uint32_t t0 = t * kVplTile;
        const uint32_t m = min((uint32_t)kVplTile, n_vpl - t0);
        __syncwarp();
        for (uint32_t j = lane; j < m; j += 32) {
            const float *y = vpl_p + (size_t)(t0 + j) * 3;
            tile[w][j] = make_float4(__ldg(y), __ldg(y + 1), __ldg(y + 2), __ldg(vpl_mu + t0 + j) * cu);
        }
        __syncwarp();
        float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t j = 0; j < m; j++) {
            const float4 e = tile[w][j];
            const V<3> r{{e.x - x.v[0], e.y - x.v[1], e.z - x.v[2]}};
            const float q = vsqnorm(r);
            const float n = sqrtf(q);
            part[0] = part[0] + e.w / fmax_ref(n, eps);
            const float g = q > 0.0f ? e.w / (n * fmax_ref(q, eps)) : 0.0f;
            for (int k = 0; k < 3; k++) part[1 + k] = part[1 + k] + g * r.v[k];
        }
        for (int c = 0; c < 4; c++) acc[c] += (double)part[c];
    }
    for (int c = 0; c < 4; c++) red[w][lane][c] = acc[c];
    __syncthreads();
    if (w == 0 && active) {
        for (int c = 0; c < 4; c++) {
            double total = red[0][lane][c];
            for (int k = 1; k < kVplSplit; k++) total = total + red[k][lane][c];
            sum[(size_t)pt * 4 + c] += total;
        }
    }
}

// The 2D aggregation, two tiles of a split at a time (t and t + 8): their partial sums are separate, so
// they run as the two halves of packed FP32 operations (F2), added to the FP64 sum in tile order. A
// pair's two quotients and logarithm are the scalar code's, by F2's; pairs outside the packed forms'
// range (q below eps^2 or beyond 2^60, or a weight out of the quotient's range) take the scalar
// expressions. The scalar loop was bound by issue at 95 instructions a pair, a packed instruction is issued
// for two (45 a pair): 100,000 VPLs x 39,280 points 11.7 -> 7.2 ms, the FMA pipe then at 67 % of its cycles.

// The smaller of two floats, NaN if either is (fminf returns the other one).
__device__ __forceinline__ float fmin_nan(float a, float b) {
    float m;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}

constexpr int kStage = 128;  // VPLs of each tile staged in shared memory at a time

__global__ void __launch_bounds__(32 * kVplSplit, 4) vpl_aggregate2_kernel(const float *__restrict__ vpl_p,
                                                                          const float *__restrict__ vpl_mu,
                                                                          uint32_t n_vpl, float area, float eps,
                                                                          const float *__restrict__ pts,
                                                                          uint32_t n_points, double *__restrict__ sum,
                                                                          uint64_t neg_zero) {
    const F2 z{neg_zero};
    __shared__ float4 s_pos[kVplSplit][kStage], s_wgt[kVplSplit][kStage];  // {x, x', y, y'}, {ku, ku', kw, kw'}
    __shared__ double red[kVplSplit][32][3];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t pt = blockIdx.x * 32u + lane;
    const bool active = pt < n_points;
    const size_t row = active ? pt : n_points - 1u;
    const float x0 = __ldg(pts + 2 * row), x1 = __ldg(pts + 2 * row + 1);
    const F2 nx0 = f2(-x0), nx1 = f2(-x1);
    const float cu = -0x1.45f306p-4f * area, cw = 0x1.45f306p-3f * area;  // -A/(4 pi), A/(2 pi)
    const float eps2 = eps * eps;
    const float lo = fmaxf(eps2, 0x1p-60f);
    double acc[3] = {0.0, 0.0, 0.0};
    const uint32_t n_tiles = (n_vpl + kVplTile - 1) / kVplTile;
    for (uint32_t t = w; t < n_tiles; t += 2 * kVplSplit) {
        const uint32_t a0 = t * kVplTile, b0 = (t + kVplSplit) * kVplTile;
        const uint32_t ma = min((uint32_t)kVplTile, n_vpl - a0), mb = b0 < n_vpl ? min((uint32_t)kVplTile, n_vpl - b0) : 0u;
        F2 part[3] = {f2(0.0f), f2(0.0f), f2(0.0f)};
        for (uint32_t h = 0; h < ma; h += kStage) {  // (mb <= ma)
            const uint32_t m = min((uint32_t)kStage, ma - h);
            __syncwarp();
            bool odd = false;
            for (uint32_t j = lane; j < m; j += 32) {
                const uint32_t ia = a0 + h + j, ib = h + j < mb ? b0 + h + j : ia;
                const float mua = __ldg(vpl_mu + ia), mub = h + j < mb ? __ldg(vpl_mu + ib) : 0.0f;
                const float kwa = mua * cw, kwb = mub * cw;
                s_pos[w][j] = make_float4(__ldg(vpl_p + 2 * (size_t)ia), __ldg(vpl_p + 2 * (size_t)ib),
                                          __ldg(vpl_p + 2 * (size_t)ia + 1), __ldg(vpl_p + 2 * (size_t)ib + 1));
                s_wgt[w][j] = make_float4(mua * cu, mub * cu, kwa, kwb);
                odd = odd || !(zero_or_not_tiny(kwa) && fabsf(kwa) <= 0x1p60f && zero_or_not_tiny(kwb) && fabsf(kwb) <= 0x1p60f);
            }
            const bool plain = __any_sync(0xffffffffu, odd);
            __syncwarp();
            for (uint32_t j = 0; j < m; j++) {
                const float4 e = s_pos[w][j], k = s_wgt[w][j];
                const F2 r0 = f2add(f2(e.x, e.y), nx0), r1 = f2add(f2(e.z, e.w), nx1);
                const F2 q = f2add(f2mul(r0, r0, z), f2mul(r1, r1, z));
                const float qa = f2lo(q), qb = f2hi(q);
                F2 u, g;
                if (__builtin_expect(!plain && fmin_nan(qa, qb) >= lo && fmaxf(qa, qb) <= 0x1p60f, 1)) {
                    u = f2mul(f2(k.x, k.y), f2log(q, z), z);
                    g = f2quotient(f2(k.z, k.w), q, z);
                } else {
                    auto weight = [&](float kw, float v) {
                        return v >= eps2 ? kw / v : (v > 0.0f ? kw / (sqrtf(v) * eps) : 0.0f);
                    };
                    // beyond a shorter second tile its half adds zero, also where the logarithm is infinite
                    const bool second = h + j < mb;
                    u = f2(k.x * log_own(fmax_ref(qa, eps2)), second ? k.y * log_own(fmax_ref(qb, eps2)) : 0.0f);
                    g = f2(weight(k.z, qa), second ? weight(k.w, qb) : 0.0f);
                }
                part[0] = f2add(part[0], u);
                part[1] = f2add(part[1], f2mul(g, r0, z));
                part[2] = f2add(part[2], f2mul(g, r1, z));
            }
        }
        for (int c = 0; c < 3; c++) {
            acc[c] += (double)f2lo(part[c]);
            if (mb) acc[c] += (double)f2hi(part[c]);
        }
    }
    for (int c = 0; c < 3; c++) red[w][lane][c] = acc[c];
    __syncthreads();
    if (w == 0 && active) {
        for (int c = 0; c < 3; c++) {
            double total = red[0][lane][c];
            for (int k = 1; k < kVplSplit; k++) total = total + red[k][lane][c];
            sum[(size_t)pt * 3 + c] += total;
        }
    }
}

template <int D>
cudaError_t paths_impl(const SceneView<D> &s, const WalkParams &p, uint32_t n_paths, float *vpl_p, float *vpl_mu,
                       unsigned long long *bounces, cudaStream_t st) {
    if (n_paths == 0) return cudaSuccess;
    vpl_paths_kernel<D><<<(n_paths + kBlock - 1) / kBlock, kBlock, 0, st>>>(s, p, n_paths, vpl_p, vpl_mu, bounces);
    return cudaGetLastError();
}

template <int D>
cudaError_t aggregate_impl(const float *vpl_p, const float *vpl_mu, uint32_t n_vpl, float area, float eps,
                           const float *pts, uint32_t n_points, double *sum, cudaStream_t st) {
    if (n_points == 0) return cudaSuccess;
    const uint32_t blocks = (n_points + 31) / 32;
    if constexpr (D == 2)
        vpl_aggregate2_kernel<<<blocks, 32 * kVplSplit, 0, st>>>(vpl_p, vpl_mu, n_vpl, area, eps, pts, n_points, sum,
                                                                f2_neg_zero);
    else
        vpl_aggregate3_kernel<<<blocks, 32 * kVplSplit, 0, st>>>(vpl_p, vpl_mu, n_vpl, area, eps, pts, n_points, sum);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_vpl_paths_2d(const SceneView<2> &s, const WalkParams &p, uint32_t n_paths, float *vpl_p,
                                float *vpl_mu, unsigned long long *bounces, cudaStream_t st) {
    return paths_impl<2>(s, p, n_paths, vpl_p, vpl_mu, bounces, st);
}
cudaError_t launch_vpl_paths_3d(const SceneView<3> &s, const WalkParams &p, uint32_t n_paths, float *vpl_p,
                                float *vpl_mu, unsigned long long *bounces, cudaStream_t st) {
    return paths_impl<3>(s, p, n_paths, vpl_p, vpl_mu, bounces, st);
}
cudaError_t launch_vpl_aggregate(int dim, const float *vpl_p, const float *vpl_mu, uint32_t n_vpl, float area,
                                 float eps, const float *pts, uint32_t n_points, double *sum, cudaStream_t st) {
    return dim == 2 ? aggregate_impl<2>(vpl_p, vpl_mu, n_vpl, area, eps, pts, n_points, sum, st)
                    : aggregate_impl<3>(vpl_p, vpl_mu, n_vpl, area, eps, pts, n_points, sum, st);
}

}  // namespace wobgb
