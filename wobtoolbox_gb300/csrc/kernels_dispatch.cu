// Routes a solve to the specialised kernel variant for its parameters, or to the general one.
// Variants are instantiated in k2_*.cu / k3_*.cu; every variant is compiled from the same walk
// source (walk_generic.cuh), only with some parameters fixed at compile time.
#include "launch.hpp"
#include "walk_generic.cuh"

#include <atomic>
#include <cstdio>

namespace wobgb {

// ---- autotuned variants: 0 = 3D direct uniform, 1 = 2D double-layer line intersection,
// 2 = 3D direct Neumann, 3 = 3D forward single-layer Neumann; configuration c = kernel shape
// (c % 4: for variants 0-2 the minimum resident blocks {1 (no limit), 5, 6, 8 or by the size of the
// launch}; for variant 3 the lockstep kernel at >= 5 blocks/SM or the split-phase
// wavefront k_fwd_wave.cu in its three trace shapes) and c / 4: paths-per-lane cap {launcher's choice
// (up to 8), 4, 2, 1} for the lockstep kernels, paths per wavefront chunk {2^22, 2^21, 2^20, 2^19} for
// the wavefront. Every variant starts with configuration kDefaultConfig, and what a configuration runs
// depends on nothing else, so setting the one that was read restores the state.
namespace {
// 81,920-triangle Robin slice, 512 paths: 24.4 ms at >= 8 blocks/SM, 25.0 at >= 5, 36.0 at >= 10, 37.8 without
// a register cap; direct Neumann on 81,920 triangles: 3.97 ms against 4.39, 4.01 and 4.52. 2D double layer:
// launch_dl_grid_2d. 3D forward: launch_forward_3d.
constexpr int kDefaultConfig = 3;
std::atomic<int> g_config[kNumTunable] = {{kDefaultConfig}, {kDefaultConfig}, {kDefaultConfig}, {kDefaultConfig}};
const char *kFwdNames[kTuneOccupancies] = {"lockstep walk, >=5 blocks/SM", "wavefront, trace >=8 blocks/SM",
                                           "wavefront, trace >=6 blocks/SM",
                                           "wavefront, trace >=9 blocks/SM, 64-byte compressed nodes"};
const uint32_t kWaveSlotsOf[kTunePptCaps] = {1u << 22, 1u << 21, 1u << 20, 1u << 19};
const int kMinBOf[kTuneOccupancies] = {1, 5, 6, 8};
const uint32_t kPptCapOf[kTunePptCaps] = {0u, 4u, 2u, 1u};
const char *kOccNames[kTuneOccupancies] = {"no register cap", ">=5 blocks/SM", ">=6 blocks/SM", ">=8 blocks/SM"};
const char *kPptNames[kTunePptCaps] = {"paths/lane <= 8", "paths/lane <= 4", "paths/lane <= 2", "paths/lane = 1"};
char g_names[kTuneConfigs][64];
}  // namespace

int tunable_domain_variant(int dim, const WalkParams &p) {
    if (p.n_volume != 0) return -1;
    const int st = strategy_of(p.bie, p.estimator, p.problem);
    if (dim == 3 && st == kStratUniform && p.bie == kDirect) return 0;
    if (dim == 2 && st == kStratLineIntersection) return 1;
    if (dim == 3 && st == kStratDirectNeumann) return 2;
    if (dim == 3 && st == kStratFwdSlNeumann) return 3;
    return -1;
}
int domain_config(int variant) { return (variant >= 0 && variant < kNumTunable) ? g_config[variant].load() : 0; }
void set_domain_config(int variant, int config) {
    if (variant >= 0 && variant < kNumTunable && config >= 0 && config < kTuneConfigs) g_config[variant].store(config);
}
const char *domain_config_name(int variant, int config) {
    if (config < 0 || config >= kTuneConfigs) return "";
    static char fwd_names[kTuneConfigs][80];
    if (variant == 3) {
        if (!fwd_names[config][0]) {
            if (config % kTuneOccupancies == 0)
                snprintf(fwd_names[config], sizeof fwd_names[config], "128 threads, %s, %s", kFwdNames[0],
                         kPptNames[config / kTuneOccupancies]);
            else
                snprintf(fwd_names[config], sizeof fwd_names[config], "128 threads, %s, %u paths per chunk",
                         kFwdNames[config % kTuneOccupancies], kWaveSlotsOf[config / kTuneOccupancies]);
        }
        return fwd_names[config];
    }
    if (!g_names[config][0])
        snprintf(g_names[config], sizeof g_names[config], "128 threads, %s, %s", kOccNames[config % kTuneOccupancies],
                 kPptNames[config / kTuneOccupancies]);
    return g_names[config];
}

// All warps of a launch (32 paths of a point each) are resident at `blocks` blocks per SM.
static bool resident(uint32_t n_points, uint32_t n_paths, uint32_t blocks) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (uint64_t)n_points * ((n_paths + 31u) / 32u) <= (uint64_t)sms * blocks * (kWalkBlock / 32);
}

// The 3D direct walks. By size (the last occupancy): launches that are resident without a register cap (3
// blocks per SM) take no cap, those resident at 5 blocks these, others 8. 20,480 triangles, no cap / 5 / 8: direct
// Neumann 300 points x 100 paths 0.88 / 0.88 / 0.96 ms, 600 x 128 1.65 / 1.06 / 1.10, 1000 x 128
// 2.45 / 1.95 / 1.45; mixed data 0.046 / 0.046 / 0.052, 0.085 / 0.056 / 0.062, 0.124 / 0.097 / 0.087.
template <int D, int kBie, int kStrat>
static cudaError_t launch_cfg(int config, const SceneView<D> &s, const WalkParams &p_in, const float *pts, uint32_t n,
                              double *sum, double *sumsq, unsigned long long *b, float *pp, cudaStream_t st) {
    WalkParams p = p_in;
    p.ppt_cap = kPptCapOf[config / kTuneOccupancies];
    int min_blocks = kMinBOf[config % kTuneOccupancies];
    if (config % kTuneOccupancies == 3) min_blocks = resident(n, p.n_paths, 3) ? 1 : resident(n, p.n_paths, 5) ? 5 : 8;
    switch (min_blocks) {
    case 5: return launch_domain_variant<D, kBie, kStrat, false, 5>(s, p, pts, n, sum, sumsq, b, pp, st);
    case 6: return launch_domain_variant<D, kBie, kStrat, false, 6>(s, p, pts, n, sum, sumsq, b, pp, st);
    case 8: return launch_domain_variant<D, kBie, kStrat, false, 8>(s, p, pts, n, sum, sumsq, b, pp, st);
    default: return launch_domain_variant<D, kBie, kStrat, false, 1>(s, p, pts, n, sum, sumsq, b, pp, st);
    }
}

// The double layer without a line grid. By size (0): launches that are resident at 4 blocks per SM take
// those (64 points x 64 paths on 256 segments: 0.142 ms against 0.153, 0.152 and 0.152 at >= 5, 6 and 8; 2,400
// warps on 1024: 0.336 against 0.341, 0.358 and 0.343), others 8 (2,800 warps: 0.355 against 0.571 at 4 and
// 0.359 at 5; 4,000 points x 256 paths on 8192 segments: 7.2 against 11.1, 9.4 and 8.3 at 4, 5 and 6). Without a
// limit the kernel takes 130 registers, which 3 blocks fit and 4 do not (4,000 x 256 on 1024: 5.0 ms
// against 3.9 at 4), so "no limit" is 4.
static cudaError_t launch_dl_2d(int min_blocks, const SceneView<2> &s, const WalkParams &p, const float *pts, uint32_t n,
                                double *sum, double *sumsq, unsigned long long *b, float *pp, cudaStream_t st) {
    if (min_blocks == 0) min_blocks = resident(n, p.n_paths, 4) ? 4 : 8;
    switch (min_blocks) {
    case 5: return launch_domain_variant<2, kDoubleLayer, kStratLineIntersection, false, 5>(s, p, pts, n, sum, sumsq, b, pp, st);
    case 6: return launch_domain_variant<2, kDoubleLayer, kStratLineIntersection, false, 6>(s, p, pts, n, sum, sumsq, b, pp, st);
    case 8: return launch_domain_variant<2, kDoubleLayer, kStratLineIntersection, false, 8>(s, p, pts, n, sum, sumsq, b, pp, st);
    default: return launch_domain_variant<2, kDoubleLayer, kStratLineIntersection, false, 4>(s, p, pts, n, sum, sumsq, b, pp, st);
    }
}

// Configuration 3 chooses by size: a forward walk whose warps are all resident in the lockstep kernel (5
// blocks per SM, 97,280 paths) takes that, since the wavefront's phases then have too few paths to fill
// (327,680 triangles, 4 bounces: 64,000 paths 0.85 ms lockstep, 1.07 wavefront; 128,000 paths 1.49 and
// 1.27); larger ones take the wavefront on compressed nodes, as 7, 11 and 15 do at every size.
static cudaError_t launch_forward_3d(int config, const SceneView<3> &s, const WalkParams &p, const float *pts, uint32_t n,
                                     double *sum, double *sumsq, unsigned long long *b, float *pp, cudaStream_t st) {
    WalkParams q = p;
    q.ppt_cap = kPptCapOf[config / kTuneOccupancies];
    const int shape = config % kTuneOccupancies;
    if (shape == 0 || p.no_alloc || (config == 3 && resident(n, p.n_paths, 5)))
        return launch_domain_variant<3, kSingleLayer, kStratFwdSlNeumann, false, 5>(s, q, pts, n, sum, sumsq, b, pp, st);
    return launch_fwd_wave_3d(s, p, pts, n, sum, sumsq, b, pp, shape, kWaveSlotsOf[config / kTuneOccupancies], st);
}

cudaError_t launch_domain_config(int dim, int variant, int config, const void *scene_view, const WalkParams &p,
                                 const float *pts, uint32_t n, double *sum, double *sumsq, unsigned long long *b,
                                 float *pp, cudaStream_t st) {
    if (config < 0 || config >= kTuneConfigs) config = 0;
    if (variant == 0 && dim == 3)
        return launch_cfg<3, kDirect, kStratUniform>(config, *(const SceneView<3> *)scene_view, p, pts, n, sum, sumsq, b, pp, st);
    if (variant == 1 && dim == 2) {
        // scenes with a line grid (host-built, up to 16,384 segments) take the warp-shared queries; the
        // others' BVH queries stay a lane each
        const SceneView<2> &v = *(const SceneView<2> *)scene_view;
        WalkParams q = p;
        q.ppt_cap = kPptCapOf[config / kTuneOccupancies];
        const int min_blocks = config % kTuneOccupancies == 3 ? 0 : kMinBOf[config % kTuneOccupancies];
        if (v.lg_K != 0u) return launch_dl_grid_2d(min_blocks, v, q, pts, n, sum, sumsq, b, pp, st);
        return launch_dl_2d(min_blocks, v, q, pts, n, sum, sumsq, b, pp, st);
    }
    if (variant == 2 && dim == 3)
        return launch_cfg<3, kDirect, kStratDirectNeumann>(config, *(const SceneView<3> *)scene_view, p, pts, n, sum, sumsq, b, pp, st);
    if (variant == 3 && dim == 3)
        return launch_forward_3d(config, *(const SceneView<3> *)scene_view, p, pts, n, sum, sumsq, b, pp, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_domain_2d(const SceneView<2> &s, const WalkParams &p, const float *pts, uint32_t n_points,
                             double *sum, double *sumsq, unsigned long long *bounces, float *per_path,
                             cudaStream_t stream) {
    const int v = tunable_domain_variant(2, p);
    if (v >= 0) return launch_domain_config(2, v, domain_config(v), &s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    const int st = strategy_of(p.bie, p.estimator, p.problem);
    if (p.n_volume == 0 && st == kStratDirectNeumann)
        return launch_domain_variant<2, kDirect, kStratDirectNeumann, false>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    if (p.n_volume == 0 && st == kStratSingleLayer)
        return launch_domain_variant<2, kSingleLayer, kStratSingleLayer, false, 5>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    if (p.n_volume == 0 && st == kStratFwdSlNeumann)
        return launch_domain_variant<2, kSingleLayer, kStratFwdSlNeumann, false, 5>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    return launch_domain_variant<2, -1, kStratRuntime, true>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
}

cudaError_t launch_domain_3d(const SceneView<3> &s, const WalkParams &p, const float *pts, uint32_t n_points,
                             double *sum, double *sumsq, unsigned long long *bounces, float *per_path,
                             cudaStream_t stream) {
    const int v = tunable_domain_variant(3, p);
    if (v >= 0) return launch_domain_config(3, v, domain_config(v), &s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    const int st = strategy_of(p.bie, p.estimator, p.problem);
    if (p.n_volume == 0 && st == kStratSingleLayer)
        return launch_domain_variant<3, kSingleLayer, kStratSingleLayer, false, 5>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);

    return launch_domain_variant<3, -1, kStratRuntime, true>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
}

cudaError_t launch_boundary_2d(const SceneView<2> &s, const WalkParams &p, const BoundaryInput &bin,
                               uint32_t n_points, double *sum, double *sumsq, unsigned long long *bounces,
                               float *per_path, cudaStream_t stream) {
    return launch_boundary_variant<2, -1, kStratRuntime, true>(s, p, bin, n_points, sum, sumsq, bounces, per_path, stream);
}

cudaError_t launch_boundary_3d(const SceneView<3> &s, const WalkParams &p, const BoundaryInput &bin,
                               uint32_t n_points, double *sum, double *sumsq, unsigned long long *bounces,
                               float *per_path, cudaStream_t stream) {
    const int st = strategy_of(p.bie, p.estimator, p.problem);
    if (p.n_volume == 0 && st == kStratDirectNeumann)
        return launch_boundary_variant<3, kDirect, kStratDirectNeumann, false>(s, p, bin, n_points, sum, sumsq, bounces, per_path, stream);
    return launch_boundary_variant<3, -1, kStratRuntime, true>(s, p, bin, n_points, sum, sumsq, bounces, per_path, stream);
}

cudaError_t launch_line_query_2d(const SceneView<2> &s, const float *origins, const float *dirs, uint32_t n,
                                 uint32_t *counts, uint32_t *hits, float *points, cudaStream_t stream) {
    return launch_line_query_impl<2>(s, origins, dirs, n, counts, hits, points, stream);
}
cudaError_t launch_line_query_3d(const SceneView<3> &s, const float *origins, const float *dirs, uint32_t n,
                                 uint32_t *counts, uint32_t *hits, float *points, cudaStream_t stream) {
    return launch_line_query_impl<3>(s, origins, dirs, n, counts, hits, points, stream);
}

}  // namespace wobgb
