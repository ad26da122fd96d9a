// The sampling CDFs' Kahan prefix sums (scene.cuh:274-298; kahan_cdf in scene_build.cpp) on the
// device, bit for bit the serial recurrence
//   y = w_i - c;  t = s + y;  c = (t - s) - y;  s = t.
//
// One thread running it is a chain of four dependent additions and a load per element: 33.6 ms for
// the two tables of 327,680 triangles, nearly all of a device scene build. Here it runs in parallel
// by speculation and is then verified, 0.20 ms for the same tables.
//
// While |s| >= |y| the step is exact apart from the rounding of y, so the pair (s, c) is the single
// number v = s - c (s is v rounded to float) and the recurrence is
//   v <- v + w_i, rounded to a multiple of ulp(y),
// an exact sum with a little lattice rounding at every step. Two runs over the same elements whose
// v differ by a multiple of twice the coarsest ulp(y) they meet stay apart by exactly that
// difference (y's exponent also depends on c, but only where w_i lies next to a power of two). So a
// chunk of elements maps its starting v to its final v by a function that is known everywhere once
// it is known on one period, a handful of lattice points:
//   1. kahan_prefix:   double sums of the chunks; their scan predicts each chunk's starting v. Chunks
//                      start behind the element of largest exponent in a 32-element window, so that
//                      their starting v lies on a coarse lattice.
//   2. kahan_try:      one warp per chunk runs it from 32 candidates, a lattice spacing apart (a lane
//                      each); the final v of each is tabulated (64-bit fixed point).
//   3. kahan_compose:  one warp chains the chunks' tables: v mod the period picks the candidate. The
//                      chained values replace the predictions and steps 2 and 3 repeat (kRounds in
//                      all): the later rounds' candidates sit within a few lattice spacings of the
//                      truth, which settles the elements next to powers of two.
//   4. kahan_verify:   every chunk runs from its chained state, writes its sums, and checks that it
//                      ends in exactly the (s, c) the next chunk started from. Chunk 0 starts from
//                      (0, 0), so where every check holds the sums are the serial ones.
//   5. kahan_repair:   from a failed check on, one warp continues serially from the true state until
//                      a chunk's starting state is met again. Nothing but speed depends on the
//                      predictions.
// Then the division by the total and the nondecreasing fix-up (a prefix maximum: the division is
// monotone, so the maximum is taken on the sums).
//
// Cost: kRounds + 1 passes over a chunk (about 20 ns an element, the latency of the chain) and kRounds
// compositions (about 95 ns a chunk), so the chunk length grows with sqrt(n). Up to kSerialMax
// elements the serial chain on one warp costs less than the launches of the other route.
// This unit is compiled without contraction: every step is a plain IEEE addition.
#include "kahan_scan.hpp"

#include <algorithm>
#include <cmath>

namespace wobgb {

namespace {

constexpr int kRounds = 3;
constexpr uint32_t kWindow = 32;
constexpr uint32_t kSerialMax = 2048;
constexpr int kWarps = 4;  // warps (chunks) per block of the chunk kernels
constexpr uint32_t kFullWarp = 0xffffffffu;

struct KahanArray {
    const float *w;
    float *cdf;
    double *dsum;       // [chunks] sum of the chunk; then the sum before it
    long long *start;   // [chunks + 1] predicted starting v in units of 2^E
    long long *ends;    // [chunks][32] final v of the candidates
    uint32_t *bound;    // [chunks + 1] first element of the chunk
    uint32_t *maxbits;  // [chunks] bits of the chunk's largest weight
    int *lattice;       // [chunks] log2 of the candidates' spacing | log2 of the period << 8 (units of 2^E)
    float2 *end_state;  // [chunks] (s, c) after the chunk
    float *chunk_max;   // [chunks] largest sum in the chunk; then the largest before it
    uint32_t *failed;   // [chunks] 1: the next chunk did not start from end_state
    int *E;             // exponent of the fixed point's unit
};
struct KahanArgs {
    KahanArray a[2];
    float *totals;
    uint32_t n, C, chunks;
};

__device__ __forceinline__ float kahan_step(float w, float &s, float &c) {
    const float y = w - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
    return t;
}

// Elements [b, e) from (s, c), each lane its own state: 32 weights per load, broadcast in turn.
// kKeep: all lanes run the same state; lane i keeps the sum after element i of each 32 and they are
// stored to out, and the largest is returned.
template <bool kKeep>
__device__ __forceinline__ float run_chunk(const float *__restrict__ w, uint32_t b, uint32_t e, float &s, float &c,
                                           float *out) {
    const uint32_t lane = threadIdx.x & 31u;
    float mx = -INFINITY;
    float next = b + lane < e ? w[b + lane] : 0.0f;
    for (uint32_t i0 = b; i0 < e; i0 += 32u) {
        const float mine = next;
        next = i0 + 32u + lane < e ? w[i0 + 32u + lane] : 0.0f;
        float keep = 0.0f;
        if (i0 + 32u <= e) {
#pragma unroll
            for (int k = 0; k < 32; k++) {
                const float t = kahan_step(__shfl_sync(kFullWarp, mine, k), s, c);
                if (kKeep && lane == (uint32_t)k) keep = t;
            }
        } else {
            for (uint32_t k = 0; k < e - i0; k++) {
                const float t = kahan_step(__shfl_sync(kFullWarp, mine, (int)k), s, c);
                if (kKeep && lane == k) keep = t;
            }
        }
        if (kKeep && i0 + lane < e) {
            out[i0 + lane] = keep;
            mx = fmaxf(mx, keep);
        }
    }
    if (kKeep) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFullWarp, mx, o));
    }
    return mx;
}

// v (units of 2^E) as the pair (s, c), and back.
__device__ __forceinline__ void state_of(long long v, int E, float &s, float &c) {
    const float sv = __ll2float_rn(v);
    s = (float)ldexp((double)sv, E);
    c = (float)ldexp((double)(__float2ll_rn(sv) - v), E);
}
__device__ __forceinline__ long long value_of(float s, float c, int E) {
    return __double2ll_rn(ldexp((double)s, -E)) - __double2ll_rn(ldexp((double)c, -E));
}

// log2 ulp of a positive float's bits (the smallest normal's for subnormals and zero)
__device__ __forceinline__ int log_ulp(uint32_t bits) { return max((int)((bits >> 23) & 255u), 1) - 150; }

// The chunk boundary at nominal position jC: behind the (last) element of largest exponent among the
// kWindow before it.
__device__ __forceinline__ uint32_t boundary(const float *__restrict__ w, uint32_t pos) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ex = (__float_as_uint(w[pos - kWindow + lane]) >> 23) & 255u;
    uint32_t m = ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFullWarp, m, o));
    const uint32_t at = __ballot_sync(kFullWarp, ex == m);
    return pos - kWindow + (32u - (uint32_t)__clz(at));
}

__global__ void __launch_bounds__(32 * kWarps) kahan_sums(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.y];
    const uint32_t lane = threadIdx.x & 31u, j = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (j >= g.chunks) return;
    const uint32_t b = j == 0 ? 0u : boundary(a.w, j * g.C);
    const uint32_t e = j + 1 == g.chunks ? g.n : boundary(a.w, (j + 1) * g.C);
    double sum = 0.0;
    uint32_t mb = 0;
    for (uint32_t i = b + lane; i < e; i += 32u) {
        const float w = a.w[i];
        sum += (double)w;
        mb = max(mb, __float_as_uint(w) & 0x7fffffffu);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(kFullWarp, sum, o);
        mb = max(mb, __shfl_xor_sync(kFullWarp, mb, o));
    }
    if (lane == 0) {
        a.dsum[j] = sum;
        a.maxbits[j] = mb;
        a.bound[j] = b;
        if (j + 1 == g.chunks) a.bound[g.chunks] = g.n;
    }
}

// One block per array: the scan of the chunks' sums, the fixed point's unit (total < 2^61 units) and
// the first predictions.
__global__ void __launch_bounds__(1024) kahan_prefix(KahanArgs g) {
    __shared__ double part[1024];
    const KahanArray &a = g.a[blockIdx.x];
    const uint32_t t = threadIdx.x, per = (g.chunks + 1023u) / 1024u;
    const uint32_t j0 = min(g.chunks, t * per), j1 = min(g.chunks, j0 + per);
    double mine = 0.0;
    for (uint32_t j = j0; j < j1; j++) mine += a.dsum[j];
    part[t] = mine;
    __syncthreads();
    for (uint32_t o = 1; o < 1024u; o <<= 1) {
        const double add = t >= o ? part[t - o] : 0.0;
        __syncthreads();
        part[t] += add;
        __syncthreads();
    }
    const double total = part[1023];
    int ex = 0;
    if (total > 0.0 && total < 1e300) frexp(total, &ex);
    const int E = ex - 61;
    if (t == 0) *a.E = E;
    double run = part[t] - mine;
    for (uint32_t j = j0; j < j1; j++) {
        const uint32_t b = a.bound[j];
        // the period: twice the ulp of the largest weight, and once more for a y above its weight
        const int period = min(max(log_ulp(a.maxbits[j]) + 2 - E, 0), 61);
        // the lattice the chunk starts on, but never too fine for 32 candidates to span a period
        int space = b > 0 ? log_ulp(__float_as_uint(a.w[b - 1])) - E : 0;
        space = min(max(space, max(period - 5, 0)), 61);
        if (a.maxbits[j] == 0u) space = 0;
        const long long v = __double2ll_rn(ldexp(run, -E));
        a.start[j] = j == 0 ? 0ll : ((v + ((1ll << space) >> 1)) >> space) << space;
        a.lattice[j] = space | (max(period, space) << 8);
        run += a.dsum[j];
    }
}

__global__ void __launch_bounds__(32 * kWarps) kahan_try(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.y];
    const uint32_t lane = threadIdx.x & 31u, j = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (j >= g.chunks) return;
    const int E = *a.E;
    float s = 0.0f, c = 0.0f;
    if (j > 0) state_of(a.start[j] + ((long long)lane << (a.lattice[j] & 255)), E, s, c);
    run_chunk<false>(a.w, a.bound[j], a.bound[j + 1], s, c, nullptr);
    a.ends[(size_t)j * 32u + lane] = value_of(s, c, E);
}

// One warp per array. The next kBatch chunks' tables are loaded while the current ones are chained.
__global__ void __launch_bounds__(32) kahan_compose(KahanArgs g) {
    constexpr int kBatch = 8;
    const KahanArray &a = g.a[blockIdx.x];
    const uint32_t lane = threadIdx.x;
    long long tab[kBatch], nxt[kBatch], base = 0, nbase = 0, v = 0;
    int lat = 0, nlat = 0;
    auto fetch = [&](uint32_t j0) {
#pragma unroll
        for (int k = 0; k < kBatch; k++) nxt[k] = j0 + k < g.chunks ? a.ends[(size_t)(j0 + k) * 32u + lane] : 0ll;
        const bool ok = lane < (uint32_t)kBatch && j0 + lane < g.chunks;
        nbase = ok ? a.start[j0 + lane] : 0ll;
        nlat = ok ? a.lattice[j0 + lane] : 0;
    };
    fetch(0);
    for (uint32_t j0 = 0; j0 < g.chunks; j0 += kBatch) {
#pragma unroll
        for (int k = 0; k < kBatch; k++) tab[k] = nxt[k];
        base = nbase;
        lat = nlat;
        fetch(j0 + kBatch);
        long long mine = 0;
#pragma unroll
        for (int k = 0; k < kBatch; k++) {
            if (j0 + k < g.chunks) {
                if (lane == (uint32_t)k) mine = v;
                const int l = __shfl_sync(kFullWarp, lat, k), space = l & 255, period = l >> 8;
                const long long diff = v - __shfl_sync(kFullWarp, base, k);
                const long long step = (diff + ((1ll << space) >> 1)) >> space;
                const int pick = (int)step & min(31, (1 << min(period - space, 5)) - 1);
                // the shift by whole periods; what is left below the lattice is rounded off in the chunk
                v = __shfl_sync(kFullWarp, tab[k], pick) + ((step - pick) << space);
            }
        }
        if (lane < (uint32_t)kBatch && j0 + lane < g.chunks) a.start[j0 + lane] = mine;
    }
    if (lane == 0) a.start[g.chunks] = v;
}

__global__ void __launch_bounds__(32 * kWarps) kahan_verify(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.y];
    const uint32_t lane = threadIdx.x & 31u, j = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (j >= g.chunks) return;
    const int E = *a.E;
    float s = 0.0f, c = 0.0f;
    if (j > 0) state_of(a.start[j], E, s, c);
    const float mx = run_chunk<true>(a.w, a.bound[j], a.bound[j + 1], s, c, a.cdf);
    if (lane == 0) {
        float ns, nc;
        state_of(a.start[j + 1], E, ns, nc);
        a.end_state[j] = make_float2(s, c);
        a.chunk_max[j] = mx;
        a.failed[j] = j + 1 < g.chunks && !(s == ns && c == nc) ? 1u : 0u;
    }
}

// One warp per array: repairs from failed checks on, the total, and the largest sum before each chunk.
__global__ void __launch_bounds__(32) kahan_repair(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.x];
    const uint32_t lane = threadIdx.x;
    const int E = *a.E;
    for (uint32_t j0 = 0; j0 < g.chunks;) {
        const uint32_t bad = __ballot_sync(kFullWarp, j0 + lane < g.chunks && a.failed[j0 + lane] != 0u);
        if (!bad) {
            j0 += 32u;
            continue;
        }
        uint32_t j = j0 + (uint32_t)__ffs(bad);  // the chunk after the failed check
        float s = a.end_state[j - 1].x, c = a.end_state[j - 1].y;
        for (bool met = false; j < g.chunks && !met; j++) {
            const float mx = run_chunk<true>(a.w, a.bound[j], a.bound[j + 1], s, c, a.cdf);
            float ns = 0.0f, nc = 0.0f;
            if (j + 1 < g.chunks) state_of(a.start[j + 1], E, ns, nc);
            met = s == ns && c == nc;
            if (lane == 0) {
                a.end_state[j] = make_float2(s, c);
                a.chunk_max[j] = mx;
            }
        }
        __syncwarp();
        j0 = j;  // chunks before j are the serial ones; chunk j's own check is still to be read
    }
    __syncwarp();
    if (lane == 0) g.totals[blockIdx.x] = a.end_state[g.chunks - 1].x;
    float carry = -INFINITY;
    for (uint32_t j0 = 0; j0 < g.chunks; j0 += 32u) {
        const bool ok = j0 + lane < g.chunks;
        float m = ok ? a.chunk_max[j0 + lane] : -INFINITY;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float p = __shfl_up_sync(kFullWarp, m, o);
            if ((int)lane >= o) m = fmaxf(m, p);
        }
        float before = __shfl_up_sync(kFullWarp, m, 1);
        before = lane == 0 ? carry : fmaxf(carry, before);
        carry = fmaxf(carry, __shfl_sync(kFullWarp, m, 31));
        if (ok) a.chunk_max[j0 + lane] = before;
    }
}

__global__ void __launch_bounds__(32 * kWarps) kahan_normalise(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.y];
    const uint32_t lane = threadIdx.x & 31u, j = blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (j >= g.chunks) return;
    const float total = g.totals[blockIdx.y];
    float carry = a.chunk_max[j];
    const uint32_t e = a.bound[j + 1];
    for (uint32_t i0 = a.bound[j]; i0 < e; i0 += 32u) {
        float m = i0 + lane < e ? a.cdf[i0 + lane] : -INFINITY;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float p = __shfl_up_sync(kFullWarp, m, o);
            if ((int)lane >= o) m = fmaxf(m, p);
        }
        m = fmaxf(m, carry);
        carry = __shfl_sync(kFullWarp, m, 31);
        if (i0 + lane < e) a.cdf[i0 + lane] = m / total;
    }
}

// Up to kSerialMax elements: one warp per array runs the recurrence as it stands.
__global__ void __launch_bounds__(32) kahan_serial(KahanArgs g) {
    const KahanArray &a = g.a[blockIdx.x];
    const uint32_t lane = threadIdx.x;
    float s = 0.0f, c = 0.0f;
    run_chunk<true>(a.w, 0u, g.n, s, c, a.cdf);
    __syncwarp();
    if (lane == 0) g.totals[blockIdx.x] = s;
    float carry = -INFINITY;
    for (uint32_t i0 = 0; i0 < g.n; i0 += 32u) {
        float m = i0 + lane < g.n ? a.cdf[i0 + lane] : -INFINITY;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float p = __shfl_up_sync(kFullWarp, m, o);
            if ((int)lane >= o) m = fmaxf(m, p);
        }
        m = fmaxf(m, carry);
        carry = __shfl_sync(kFullWarp, m, 31);
        if (i0 + lane < g.n) a.cdf[i0 + lane] = m / s;
    }
}

// Chunk length: a power of two from sqrt(1.25 n) up, about the least of (kRounds + 1) 20 ns C +
// kRounds 95 ns n / C.
uint32_t chunk_length(uint32_t n) {
    uint32_t C = 2 * kWindow;
    while (C < 32768u && (double)C * C < 1.25 * (double)n) C <<= 1;
    return C;
}

// Guide tables: a block's kGuideBlock records need the first indices of kGuideBlock + 2 thresholds. Two
// warps find the first and the last of them by a 32-way search (four dependent loads for a million
// elements instead of twenty), the CDF between them is staged in shared memory, and every thread
// searches there (a full search per record took 43 us for 327,680 records, about ten times this).
constexpr int kGuideBlock = 256;
constexpr uint32_t kGuideStage = 2048;
// The least float not below the host's threshold, the double nearest (j - 1/2) / G: a float is below one
// exactly when it is below the other. The numerator and denominator are integers under 2^23 + 1, so a
// float other than their quotient is at least 2^-47 of it away, and the quotient rounded up to a float
// directly is that float. (In doubles the table was bound by FP64: 67 us for 2^20 records, now 17.)
__device__ __forceinline__ float guide_threshold(uint32_t j, uint32_t G) {
    return __fdiv_ru((float)(2 * (int)j - 1), (float)(2u * G));
}
// The first i in [0, n - 1) with cdf[i] >= thr, else n - 1; all lanes of a warp take part.
__device__ __forceinline__ uint32_t warp_first(const float *__restrict__ cdf, uint32_t n, float thr) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31u) / 32u, i = lo + lane * step;
        const uint32_t below = __ballot_sync(kFullWarp, i < hi && __ldg(cdf + min(i, hi)) < thr);
        const uint32_t c = (uint32_t)__popc(below);  // the first c probes lie below the threshold
        if (c == 0) break;
        hi = min(hi, lo + c * step);
        lo = lo + (c - 1u) * step + 1u;
    }
    return lo;
}
__global__ void __launch_bounds__(kGuideBlock) k_guide(uint32_t n, uint32_t G, const float *__restrict__ cdf,
                                                       uint4 *__restrict__ rec) {
    __shared__ float stage[kGuideStage];
    __shared__ uint32_t first[kGuideBlock + 2];
    __shared__ uint32_t range[2];
    const uint32_t j0 = blockIdx.x * kGuideBlock, cnt = min((uint32_t)kGuideBlock + 2u, G - j0);
    const uint32_t warp = threadIdx.x >> 5;
    if (warp < 2u) {
        const uint32_t f = warp_first(cdf, n, guide_threshold(warp == 0u ? j0 : j0 + cnt - 1u, G));
        if ((threadIdx.x & 31u) == 0u) range[warp] = f;
    }
    __syncthreads();
    const uint32_t A = range[0], B = range[1], m = B - A + 1u;
    const bool staged = m <= kGuideStage;
    if (staged)
        for (uint32_t i = threadIdx.x; i < m; i += kGuideBlock) stage[i] = __ldg(cdf + A + i);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt; k += kGuideBlock) {
        const float thr = guide_threshold(j0 + k, G);
        uint32_t lo = A, hi = B;  // the answer lies in [A, B]: thresholds grow with j
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if ((staged ? stage[mid - A] : __ldg(cdf + mid)) < thr) lo = mid + 1;
            else hi = mid;
        }
        first[k] = lo;
    }
    __syncthreads();
    const uint32_t k = threadIdx.x, j = j0 + k;
    if (j >= G) return;
    const uint32_t lo = first[k], hi = j + 2 < G ? first[k + 2] : n - 1;
    rec[j] = make_uint4(lo, hi, __float_as_uint(__ldg(cdf + lo)), __float_as_uint(__ldg(cdf + min(lo + 1, n - 1))));
}

}  // namespace

size_t kahan_scratch_bytes(uint32_t n, int arrays) {
    const size_t ch = n / chunk_length(n) + 2;
    const size_t per = ch * (8 + 8 + 256 + 4 + 4 + 4 + 8 + 4 + 4) + 16 + 16;
    return (size_t)arrays * ((per + 255) / 256 * 256);
}

cudaError_t launch_kahan_cdf(uint32_t n, int arrays, const float *const *w, float *const *cdf, float *totals,
                             void *scratch, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    KahanArgs g{};
    g.n = n;
    g.totals = totals;
    g.C = chunk_length(n);
    g.chunks = (n + g.C - 1) / g.C;
    const size_t ch = n / g.C + 2;
    char *p = (char *)scratch;
    for (int k = 0; k < arrays; k++) {
        KahanArray &a = g.a[k];
        a.w = w[k];
        a.cdf = cdf[k];
        char *q = p + (size_t)k * (kahan_scratch_bytes(n, 1));
        auto take = [&q](size_t bytes) {
            char *r = q;
            q += bytes;
            return r;
        };
        a.ends = (long long *)take(ch * 256);
        a.dsum = (double *)take(ch * 8);
        a.start = (long long *)take(ch * 8);
        a.end_state = (float2 *)take(ch * 8);
        a.bound = (uint32_t *)take(ch * 4);
        a.maxbits = (uint32_t *)take(ch * 4);
        a.lattice = (int *)take(ch * 4);
        a.chunk_max = (float *)take(ch * 4);
        a.failed = (uint32_t *)take(ch * 4);
        a.E = (int *)take(16);
    }
    if (n <= kSerialMax) {
        kahan_serial<<<arrays, 32, 0, stream>>>(g);
        return cudaGetLastError();
    }
    const dim3 grid((g.chunks + kWarps - 1) / kWarps, arrays);
    kahan_sums<<<grid, 32 * kWarps, 0, stream>>>(g);
    kahan_prefix<<<arrays, 1024, 0, stream>>>(g);
    for (int r = 0; r < kRounds; r++) {
        kahan_try<<<grid, 32 * kWarps, 0, stream>>>(g);
        kahan_compose<<<arrays, 32, 0, stream>>>(g);
    }
    kahan_verify<<<grid, 32 * kWarps, 0, stream>>>(g);
    kahan_repair<<<arrays, 32, 0, stream>>>(g);
    kahan_normalise<<<grid, 32 * kWarps, 0, stream>>>(g);
    return cudaGetLastError();
}

cudaError_t launch_guide(uint32_t n, uint32_t G, const float *cdf, uint32_t *rec, cudaStream_t stream) {
    k_guide<<<(G + kGuideBlock - 1) / kGuideBlock, kGuideBlock, 0, stream>>>(n, G, cdf, (uint4 *)rec);
    return cudaGetLastError();
}

}  // namespace wobgb
