// The 2D double-layer Dirichlet walk (line-intersection sampling, estimator.cuh:154-191, 255-262) on
// scenes with a line grid, its line queries shared by the warp.
//
// A query tests the segments its grid cell lists: 5 on average on a 1024-segment star (41 on 8192
// segments) but up to 40, so a lane per query ran at 13 of 32 lanes and 1,600 instructions a bounce
// (3.3 ms for 7,960 points x 1024 paths x 8 bounces at 12 blocks per SM; 2.46 ms for 4,000 x 256 on 8192
// segments). This kernel takes 2.8 ms and 1.23 ms, at 29 lanes and 1,130 instructions. A warp lays the
// lists of its 32 queries end to end (a scan of their lengths) and tests 32 candidates at a time, a lane each: the lane finds the query that owns its candidate from the bit mask of the
// queries that begin in the round, fetches that query's line by shuffles, and the round's ballot is
// kept in shared memory. A query's hits are then a run of ballot bits in list order, so its hit count
// and the chosen hit are bit counts. The walk's warps stay converged for it: paths that have ended
// only bring empty lists. The last bounce's query is never used by the double layer (its terms depend
// on the current point alone) and is not made.
//
// Every path makes the operations of Walker's domain() and unknown_boundary() for this strategy in
// the same order on its own stream, so path values are bit-identical to the general walk's.
#include "kernels.cuh"

namespace wobgb {

namespace {

constexpr uint32_t kFullWarp = 0xffffffffu;
constexpr uint32_t kBallots = 96;  // rounds a warp keeps: up to 3072 candidates, else each lane takes its own list

using DlWalker = Walker<2, kDoubleLayer, kStratLineIntersection, false>;

// sample_line_intersection for the lanes with `need` (all lanes of the warp call): the sample from x and
// its inv_pdf.
__device__ __forceinline__ BPoint<2> warp_line_sample(DlWalker &w, bool need, const V<2> &x, float &inv_pdf,
                                                      uint32_t *ballots, uint32_t *owners) {
    const SceneView<2> &s = w.s;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    V<2> dir = vzero<2>();
    uint32_t e0 = 0, cnt = 0;
    bool grid = true;
    if (need) {
        dir = line_sample_direction<2>(w.rng);
        grid = line_grid_cell(s, x, dir, e0, cnt);
    }
    uint32_t end = cnt;  // candidates of the warp up to and including this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFullWarp, end, o);
        if ((int)lane >= o) end += v;
    }
    const uint32_t total = __shfl_sync(kFullWarp, end, 31), start = end - cnt;
    const bool shared = total <= 32u * kBallots;
    if (shared) {
        // the lanes with candidates, in order: owners[r] is the r-th
        const uint32_t busy = __ballot_sync(kFullWarp, cnt != 0u);
        __syncwarp();
        if (cnt) owners[__popc(busy & below)] = lane;
        __syncwarp();
        const uint32_t owner_r = owners[lane];
        for (uint32_t base = 0; base < total; base += 32u) {
            const uint32_t flat = base + lane;
            const bool here = cnt != 0u && start >= base && start < base + 32u;
            const uint32_t heads = __reduce_or_sync(kFullWarp, here ? 1u << (start - base) : 0u);
            const uint32_t before = __popc(__ballot_sync(kFullWarp, cnt != 0u && start < base));
            // (at least one query has begun at or before each candidate)
            const uint32_t r = before + __popc(heads & (below | (1u << lane))) - 1u;
            const uint32_t own = __shfl_sync(kFullWarp, owner_r, r) & 31u;
            V<2> o, d;
            o.v[0] = __shfl_sync(kFullWarp, x.v[0], own);
            o.v[1] = __shfl_sync(kFullWarp, x.v[1], own);
            d.v[0] = __shfl_sync(kFullWarp, dir.v[0], own);
            d.v[1] = __shfl_sync(kFullWarp, dir.v[1], own);
            const uint32_t at = __shfl_sync(kFullWarp, e0 - start, own) + flat;
            bool hit = false;
            if (flat < total) hit = hit_seg(o, d, __ldg(s.lg_seg + __ldg(s.lg_ent + at)));
            const uint32_t bits = __ballot_sync(kFullWarp, hit);
            if (lane == 0) ballots[base >> 5] = bits;
        }
        __syncwarp();
    }
    BPoint<2> y = bp_zero<2>();
    inv_pdf = 0.0f;
    if (need) {
        uint32_t ei = 0, m = 0;
        if (grid && shared) {
            // this query's bits: [start, end) of the ballots
            const uint32_t w0 = start >> 5, w1 = (end + 31u) >> 5;
            auto word = [&](uint32_t i) {
                uint32_t b = ballots[i];
                if (i == w0) b &= 0xffffffffu << (start & 31u);
                if (i + 1u == w1 && (end & 31u)) b &= 0xffffffffu >> (32u - (end & 31u));
                return b;
            };
            if (cnt)
                for (uint32_t i = w0; i < w1; i++) m += __popc(word(i));
            m = m < kHitBuffer ? m : kHitBuffer;
            if (m) {  // line_hit_choice
                const float u = w.rng.uniform();
                uint32_t k = (uint32_t)((float)m * u);
                k = (m - 1) < k ? (m - 1) : k;
                uint32_t i = w0, b = word(w0);
                for (uint32_t c = __popc(b); k >= c; c = __popc(b)) {
                    k -= c;
                    b = word(++i);
                }
                for (; k; k--) b &= b - 1u;
                ei = __ldg(s.lg_ent + e0 + (32u * i + (uint32_t)__ffs(b) - 1u - start));
            }
        } else {
            uint32_t hits[kHitBuffer];
            m = grid ? list_hits(s, e0, cnt, x, dir, hits) : bvh_query2(s, x, dir, hits);
            ei = line_hit_choice(w.rng, hits, m);
        }
        y = line_hit_point<2>(s, ei, m, x, dir);
        inv_pdf = line_sample_inv_pdf<2>(y, x, m);
    }
    return y;
}

template <bool kPerPath, int kMinB>
__global__ void __launch_bounds__(kBlock, kMinB) dl2d_kernel(SceneView<2> s, WalkParams p, const float *__restrict__ pts,
                                                             uint32_t n_points, double *__restrict__ sum,
                                                             double *__restrict__ sumsq,
                                                             unsigned long long *__restrict__ bounces,
                                                             float *__restrict__ per_path) {
    __shared__ uint32_t s_ballots[kBlock / 32][kBallots];
    __shared__ uint32_t s_owners[kBlock / 32][32];
    __shared__ double acc[6][kBlock];  // [c]: a thread's running sum, [3 + c]: its sum of squares
    const uint32_t tid = threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t *ballots = s_ballots[threadIdx.x >> 5], *owners = s_owners[threadIdx.x >> 5];
    owners[lane] = 0u;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t n_warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t span = 32u * p.ppt;
    const uint32_t slabs = (p.n_paths + span - 1u) / span;
    const uint64_t units = (uint64_t)n_points * slabs;
    const uint32_t L = p.path_length;
    unsigned long long my_bounces = 0;
    for (uint64_t u = warp; u < units; u += n_warps) {
        const uint32_t pt = (uint32_t)(u / slabs);
        const uint32_t first = (uint32_t)(u % slabs) * span;
        V<2> x;
#pragma unroll
        for (int i = 0; i < 2; i++) x.v[i] = __ldg(pts + (size_t)pt * 2 + i);
#pragma unroll
        for (int c = 0; c < 6; c++) acc[c][tid] = 0.0;
        for (uint32_t k = 0; k < p.ppt; k++) {
            const uint32_t path = first + k * 32u + lane;
            const bool active = path < p.n_paths;
            DlWalker w(s, p, kStreamDomain, p.point_offset + pt, p.path_offset + path);
            // domain(): the first sample from x and what the path's estimate multiplies there, then
            // unknown_boundary()'s bounces, each from the sample before it
            float contrib = 0.0f, wt = 1.0f, known = 0.0f, du = 0.0f;
            V<2> gk = vzero<2>(), gu = vzero<2>();
            BPoint<2> y_prev = bp_zero<2>();
            y_prev.p = x;
            bool alive = active;
            for (uint32_t m = 0; m < L; m++) {
                if (!__any_sync(kFullWarp, alive)) break;
                float ip;
                BPoint<2> y = warp_line_sample(w, alive, y_prev.p, ip, ballots, owners);
                if (alive) {
                    if (m == 0) {
                        known = w.sdk(x, y, ip);
                        du = w.sdu(x, y, ip);
                        gk = w.gdk(x, y, ip);
                        gu = w.gdu(x, y, ip);
                    } else {
                        wt = wt * w.fbu(y_prev, y, ip, true);
                        alive = !(wt == 0.0f);
                    }
                    y_prev = y;
                    if (alive) {
                        w.bounces++;
                        if (m == L - 1) wt = 0.5f * wt;
                        contrib = contrib + wt * w.fbk(y_prev, y, 0.0f);
                    }
                }
            }
            if (active) {
                const float out[3] = {known + contrib * du, gk.v[0] + contrib * gu.v[0], gk.v[1] + contrib * gu.v[1]};
                my_bounces += w.bounces;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    if (kPerPath) per_path[((size_t)pt * p.n_paths + path) * 3 + c] = out[c];
                    const double v = (double)out[c];
                    acc[c][tid] += v;
                    acc[3 + c][tid] += v * v;
                }
            }
        }
        if (!kPerPath) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double sv = warp_sum(acc[c][tid]);
                const double qv = warp_sum(acc[3 + c][tid]);
                if (lane == 0) {
                    atomicAdd(sum + (size_t)pt * 3 + c, sv);
                    if (sumsq) atomicAdd(sumsq + (size_t)pt * 3 + c, qv);
                }
            }
        }
    }
    if (bounces) {
        const unsigned long long b = warp_sum_u64(my_bounces);
        if (lane == 0 && b) atomicAdd(bounces, b);
    }
}

template <int kMinB>
cudaError_t launch_min(const SceneView<2> &s, const WalkParams &p_in, const float *pts, uint32_t n_points, double *sum,
                       double *sumsq, unsigned long long *bounces, float *per_path, cudaStream_t stream) {
    WalkParams p = p_in;
    p.ppt = choose_ppt(p.ppt_points ? p.ppt_points : n_points, p.n_paths);
    if (p.ppt_cap && p.ppt > p.ppt_cap) p.ppt = p.ppt_cap;
    const uint64_t units = (uint64_t)n_points * ((p.n_paths + 32u * p.ppt - 1u) / (32u * p.ppt));
    if (per_path) {
        auto k = dl2d_kernel<true, kMinB>;
        k<<<persistent_grid(k, units), kBlock, 0, stream>>>(s, p, pts, n_points, sum, sumsq, bounces, per_path);
    } else {
        auto k = dl2d_kernel<false, kMinB>;
        k<<<persistent_grid(k, units), kBlock, 0, stream>>>(s, p, pts, n_points, sum, sumsq, bounces, nullptr);
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dl_grid_2d(int min_blocks, const SceneView<2> &s, const WalkParams &p, const float *pts,
                              uint32_t n_points, double *sum, double *sumsq, unsigned long long *bounces,
                              float *per_path, cudaStream_t stream) {
    if (min_blocks == 0) {
        // By size: 12 blocks per SM (1024-segment star, 7,960 points x 1024 paths: 2.87 ms against 3.88, 2.95 and
        // 2.86 at 5, 8 and 10; 8192 segments: 1.23 against 2.00, 1.45 and 1.33). With every warp of the
        // launch resident at 8 blocks, fewer registers only cost spills (64 points x 64 paths: 34 us at 8
        // blocks, 38 at 12; 1000 points x 200 paths, past the line: 76 and 64).
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        min_blocks = (uint64_t)n_points * ((p.n_paths + 31u) / 32u) <= (uint64_t)sms * 8u * (kBlock / 32) ? 8 : 12;
    }
    switch (min_blocks) {
    case 1: return launch_min<1>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    case 5: return launch_min<5>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    case 6: return launch_min<6>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    case 8: return launch_min<8>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    default: return launch_min<12>(s, p, pts, n_points, sum, sumsq, bounces, per_path, stream);
    }
}

}  // namespace wobgb
