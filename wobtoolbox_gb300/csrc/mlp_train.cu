// Fused training step of the Fourier-feature MLP (mlp.cu's network with 4 hidden layers): one
// kernel runs the batch gather, the forward pass and the backward pass of 64 rows per block with
// every weight and activation in shared memory and writes the block's gradient; a second kernel
// sums the blocks' gradients in a fixed order (so a step is deterministic), applies Adam, writes
// the updated weights as a packed BF16 image in both operand layouts, and its first block advances
// the step counter. Both are programmatic dependent launches; wob_mlp_train captures 16 steps into a
// CUDA graph and replays it. A step is a chain of short dependent stages (14.9 us for 8,192 rows, of
// which 1.3 us are its traffic and 0.1 us its products), so what does not depend on the previous
// kernel runs before griddepcontrol.wait, under its tail: the next batch's rows and Fourier features,
// which depend on the step number alone, and in the update the schedule, the parameters and their
// moments. Within the step, SiLU' is evaluated while the next layer's forward product runs and the
// bias sums while a backward one does; gradients leave in the accumulators' order. Together these
// took a step from 21.4 us to 14.9. Each block stages the image (74 KB) into shared memory with TMA
// bulk copies (cp.async.bulk, completion on mbarriers, the waits bounded), the first layer's on its own.
//
// Network and parameter layout as in mlp.cu: phi = [sin, cos](2 pi B v) (32 frequencies of the
// 6 inputs), 4 hidden layers 64 -> 64 with SiLU, a linear 64 -> out_dim head; FP32 parameters,
// for each layer W [out][in] row-major then b [out]. The SiLU derivative is
// that of the pre-activations rounded to BF16, bias gradients are summed in FP32 from the FP32
// products. No atomics: every sum has a fixed order, so training is deterministic.
//
// Products: every 64 x 64 x 64 product C[m][n] = sum_k A[m][k] B[n][k] is four tcgen05.mma
// (kind::f16, BF16 operands from shared memory, M = 64, N = 64, K = 16 each) issued by one thread,
// the FP32 accumulator in tensor memory (TMEM), completion signalled on an mbarrier by
// tcgen05.commit. With M = 64 the accumulator's rows 16 q .. 16 q + 15 sit in TMEM lanes 32 q ..
// 32 q + 15, the lane quarter that warps w with w % 4 = q may read: warp w reads rows
// [16 (w % 4), +16) x columns [16 (w / 4), +16) with tcgen05.ld.16x256b (the mma.sync m16n8
// accumulator layout: lane l holds rows l / 4 and l / 4 + 8, columns 2 (l % 4) and + 1 of each
// 8-column tile) and runs the epilogue on them. Both operands are K-major:
//   forward  Z = A W^T:     A = activation [row][in],   B = W   [out][in]
//   weights  dW = dZ^T A:   A = dZ^T [out][row],        B = A^T [in][row]
//   inputs   dA = dZ W:     A = dZ   [row][out],        B = W^T [in][out]
// each stored in the no-swizzle core-matrix layout (cm_index): 8 x 8 BF16 core matrices of 128
// contiguous bytes, K-adjacent ones 128 bytes apart (the descriptor's leading byte offset), 8-row
// groups 1024 bytes apart (its stride byte offset). Epilogues write those layouts with stmatrix
// (.trans for the transposed copies): the 8 rows of a core matrix are one 128-byte line, so a
// phase touches 32 distinct banks.
#include "../../include/wob_capi.h"

#include "device_common.cuh"
#include "launch.hpp"
#include "mlp_train.hpp"

#include <cuda_bf16.h>

namespace wobgb {

namespace {

constexpr int kTM = 64;          // rows per block
constexpr int kW = 64;           // layer width
constexpr int kMatHalves = kW * kW;   // BF16 values per 64 x 64 operand
constexpr int kMat = kMatHalves / 2;  // 32-bit words per operand
constexpr int kHidden = 4;
constexpr int kLayers = kHidden + 1;
constexpr int kIn = 6;
// 16 warps: warp w handles rows [16 (w & 3), +16) x columns [16 (w >> 2), +16) of every product's
// accumulator
constexpr int kRowBlocks = kTM / 16;
constexpr int kColSplit = 4;
constexpr int kWarps = kRowBlocks * kColSplit;
constexpr int kThreads = kWarps * 32;
constexpr int kCols = kW / kColSplit;  // columns per warp
constexpr int kNT = kCols / 8;         // 8-column tiles per warp
static_assert(kNT == 2, "the TMEM loads and the tile stores move two 8-column tiles");
constexpr int kLayerParams = kW * kW + kW;
// TMEM: columns [0, 64) take forward and input-gradient products, [64, 128) and [128, 192) the
// weight gradients of odd and even layers (read out while the next layer's products run)
constexpr uint32_t kTmemCols = 256;

// operands: Wf (5), Wb (4), act, actT (5), dZ, dZT (2: layer l's in dZT + (l & 1) kMat, kept until its
// weight-gradient product has been read out)
constexpr size_t kSmemWords = (size_t)(kLayers + kHidden + 1 + kLayers + 3) * kMat;
constexpr size_t kSmemFloats = (kHidden - 1) * kThreads * 4 * kNT + kLayers * kW + kLayers * kRowBlocks * kW +
                               kTM * kIn + kTM * kW + kWarps;

// BF16 index of element (r, k) of a 64 x 64 K-major operand in the no-swizzle core-matrix layout.
__host__ __device__ constexpr uint32_t cm_index(uint32_t r, uint32_t k) {
    return (r >> 3) * 512u + (k >> 3) * 64u + (r & 7u) * 8u + (k & 7u);
}

// Two floats rounded to BF16 in one word, lo in the low half (one cvt.rn.bf16x2.f32).
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float lo_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_of(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- tcgen05 helpers
// Shared-memory descriptor of a no-swizzle K-major operand starting at byte address addr:
// start >> 4 (bits 0-13), leading byte offset 128 >> 4 (bits 16-29), stride byte offset
// 1024 >> 4 (bits 32-45), descriptor version 1 (bits 46-47), base offset 0, no swizzle.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(128u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) |
           (1ull << 46);
}
// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), BF16 A and B (bits 7-9,
// 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kW >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes made visible to the tensor cores' reads
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (=|+=) A B^T over K = 64: four K = 16 steps, 256 bytes apart in both operands.
__device__ __forceinline__ void issue_product(uint32_t d_tmem, const uint32_t *A, const uint32_t *B) {
    const uint32_t a = smem_u32(A), b = smem_u32(B);
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
        const uint64_t ad = operand_desc(a + kk * 256u), bd = operand_desc(b + kk * 256u);
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
            "l"(ad), "l"(bd), "r"(kIdesc), "r"(kk));
    }
}
// One lane of a converged warp, the same one each time (so a product's issue is known to be uniform).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
// Arrives on the mbarrier once every tcgen05.mma this thread issued before has completed.
__device__ __forceinline__ void commit_to(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Rows [16 q, +16) x 16 columns of a product from TMEM (taddr: lane 32 q, first column) into
// acc[j][.] in the m16n8 accumulator layout of 8-column tile j.
__device__ __forceinline__ void load_acc(float acc[kNT][4], uint32_t taddr) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < kNT; j++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[j][q] = __uint_as_float(r[4 * j + q]);
}

// A block's gradient is stored in the order the accumulators are read out ("slots"), so that its
// stores are whole 512-byte lines: for each layer, row block and column group (the head: only the row
// blocks that hold outputs) two runs of 32 lanes x 4 values, then 64 biases for each layer. (Scattered
// to the parameters' places instead, eight 4-byte stores of eight rows each took 1,000 cycles a layer.)
__host__ __device__ constexpr uint32_t weight_slots(uint32_t out_dim) {
    return (uint32_t)kHidden * kW * kW + (out_dim + 15u) / 16u * (16u * kW);
}
__host__ __device__ constexpr uint32_t gradient_slots(uint32_t out_dim) { return weight_slots(out_dim) + kLayers * kW; }
// The parameter in a slot; false for the padding of a head that is not a multiple of 16 wide.
__device__ __forceinline__ bool slot_param(uint32_t slot, uint32_t out_dim, uint32_t &i) {
    const uint32_t ws = weight_slots(out_dim);
    if (slot >= ws) {
        const uint32_t l = (slot - ws) / kW, o = (slot - ws) % kW, fo = l == kHidden ? out_dim : (uint32_t)kW;
        i = l * kLayerParams + fo * kW + o;
        return l < kLayers && o < fo;
    }
    const uint32_t l = slot >> 12, rb = (slot >> 10) & 3u, cg = (slot >> 8) & 3u, j = (slot >> 7) & 1u,
                   lane = (slot >> 2) & 31u, q = slot & 3u;
    const uint32_t row = rb * 16u + (lane >> 2) + 8u * (q >> 1), col = cg * 16u + 8u * j + 2u * (lane & 3u) + (q & 1u);
    i = l * kLayerParams + row * kW + col;
    return l < kHidden || row < out_dim;
}

// SiLU and its derivative with the fast exponential and division intrinsics (the values are rounded
// to BF16 or multiply BF16-rounded gradients, so their few-ulp error does not show). For z below
// about -88, exp(-z) overflows and __fdividef returns 0 for the huge or infinite denominator, the
// limit of both functions.
__device__ __forceinline__ float silu_f(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_d(float z) {
    const float s = __fdividef(1.0f, 1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// Stores a warp's 16 x 16 tile of packed BF16 pairs p[j][h] (accumulator layout: row m0 + gid +
// 8 h, columns n0 + 8 j + 2 tig, +1) into operand M at (row, col), or with kTrans at (col, row)
// (the transposed operand): one stmatrix.x4 of four 8 x 8 matrices, each one core matrix.
template <bool kTrans>
__device__ __forceinline__ void store_tile(uint32_t *M, const uint32_t p[kNT][2], int m0, int n0, int lane) {
    const int r = lane & 7, mi = lane >> 3;
    const int row = m0 + 8 * (mi & 1), col = n0 + 8 * (mi >> 1);
    const uint32_t idx = kTrans ? cm_index(col + r, row) : cm_index(row + r, col);
    const uint32_t addr = smem_u32(reinterpret_cast<__nv_bfloat16 *>(M) + idx);
    if (kTrans)
        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(p[0][0]),
                     "r"(p[0][1]), "r"(p[1][0]), "r"(p[1][1])
                     : "memory");
    else
        asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(p[0][0]),
                     "r"(p[0][1]), "r"(p[1][0]), "r"(p[1][1])
                     : "memory");
}

// BF16 value at (r, k) of an operand.
__device__ __forceinline__ void store_bf16(uint32_t *M, int r, int k, float v) {
    reinterpret_cast<__nv_bfloat16 *>(M)[cm_index(r, k)] = __float2bfloat16_rn(v);
}

// Column sums over the warp's 16 rows of the FP32 values in acc (accumulator layout of tile j),
// stored to the row block's row dst[n0 + 8 j + 2 tig (+1)] in shared memory (the row blocks' rows
// are added in row-block order later, so the sum does not depend on scheduling).
__device__ __forceinline__ void store_col_sums(float acc[kNT][4], float *dst, int n0, int lane, int tig) {
#pragma unroll
    for (int j = 0; j < kNT; j++) {
        float s0 = acc[j][0] + acc[j][2], s1 = acc[j][1] + acc[j][3];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        }
        if (lane < 4) {
            dst[n0 + j * 8 + 2 * tig] = s0;
            dst[n0 + j * 8 + 2 * tig + 1] = s1;
        }
    }
}

constexpr size_t kImageWords = (size_t)(kLayers + kHidden) * kMat;  // Wf then Wb, as in shared memory
constexpr uint32_t kImageBytes = (uint32_t)(kImageWords * 4);
static_assert(kImageBytes % 16 == 0, "bulk copies move multiples of 16 bytes");
// Warp that issues the weight-gradient products (warp 0 issues the others).
constexpr int kWgradWarp = 1;
// Threads that share the fetch of one batch row.
constexpr int kGatherThreads = kThreads / kTM;
// try_wait polls before a block gives up on its staging copy or a product (each poll may suspend
// the thread for a while; either normally completes within microseconds).
constexpr uint32_t kWaitPolls = 1u << 22;

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint32_t polls = kWaitPolls) {
    for (uint32_t i = 0; i < polls; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// A bulk copy into shared memory that completes `bytes` on the mbarrier.
__device__ __forceinline__ void stage_copy(uint32_t *dst, const uint32_t *src, uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Error bits of FusedTrainArgs::err.
constexpr uint32_t kErrStage = 1u;    // the weight image's bulk copy did not land within the bound
constexpr uint32_t kErrProduct = 2u;  // a product's completion did not arrive within the bound

__global__ void __launch_bounds__(kThreads, 2) mlp_train_fused_kernel(FusedTrainArgs g) {
    extern __shared__ __align__(128) uint32_t smem[];
    // mbarriers: the staging of the first layer's weights and of the rest of the image, forward /
    // input-gradient products, weight-gradient products of even and odd layers (one phase outstanding
    // at a time on each), the teardown drain
    __shared__ __align__(8) uint64_t first_bar, stage_bar, mma_bar, wgrad_bar[2], drain_bar;
    __shared__ uint32_t tmem_slot, ahead_slot;
    uint32_t *Wf = smem;                      // layer l: [out][in]
    uint32_t *Wb = Wf + kLayers * kMat;       // layer l >= 1: [in][out] at index l - 1
    uint32_t *act = Wb + kHidden * kMat;      // [row][in] of the layer being evaluated
    uint32_t *actT = act + kMat;              // layer l's input: [in][row]
    uint32_t *dZ = actT + kLayers * kMat;     // [row][out]
    uint32_t *dZT = dZ + kMat;                // two buffers [out][row]
    // silu'(Z_l) of hidden layers 0 .. 2, each thread's own values: [3][2][512] x 4
    float4 *dsil = reinterpret_cast<float4 *>(smem + kSmemWords);
    float *bias = reinterpret_cast<float *>(dsil + (kHidden - 1) * kNT * kThreads);  // [5][64]
    float *dbias = bias + kLayers * kW;                          // [5][4 row blocks][64]
    float *xin = dbias + kLayers * kRowBlocks * kW;              // [64][6]
    float *tgt = xin + kTM * kIn;                                // [64][64]
    float *red = tgt + kTM * kW;                                 // loss per warp

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    const int rb = warp & (kRowBlocks - 1), m0 = rb * 16, n0 = (warp / kRowBlocks) * kCols;
    const int out_dim = (int)g.out_dim;

    // mbarriers and TMEM columns for the accumulators first: they depend on no earlier kernel, so
    // under a programmatic dependent launch they overlap the previous update
    const uint32_t fbar = smem_u32(&first_bar), bar = smem_u32(&stage_bar), pbar = smem_u32(&mma_bar),
                   dbar = smem_u32(&drain_bar);
    const uint32_t wbar0 = smem_u32(&wgrad_bar[0]), wbar1 = smem_u32(&wgrad_bar[1]);
    if (tid == 0) {
        for (uint32_t b : {fbar, bar, pbar, wbar0, wbar1, dbar})
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(b == dbar ? 2u : 1u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // The batch of a step: its rows (Philox4x32-10 on (row, step, 0, "tran") keyed by the seed) and
    // their Fourier features (mlp.cu's fourier_kernel): phi[r][f] = sin 2 pi t, phi[r][32 + f] =
    // cos 2 pi t. Ends with a barrier after the rows; the features' stores are published later.
    auto load_batch = [&](uint32_t step) {
        for (int q = tid; q < kTM * kGatherThreads; q += kThreads) {
            const int r = q / kGatherThreads, part = q % kGatherThreads;
            const uint32_t row = blockIdx.x * kTM + r;
            const bool ok = row < g.batch;
            uint32_t idx = row;
            if (ok && g.gather) {
                const uint4 h = philox4x32_10(make_uint4(row, step, 0u, 0x7472616eu), (uint32_t)g.seed,
                                              (uint32_t)(g.seed >> 32));
                idx = (uint32_t)(((uint64_t)h.x * g.n) >> 32);
            }
            for (int k = part; k < kIn; k += kGatherThreads)
                xin[r * kIn + k] = ok ? g.inputs[(size_t)idx * kIn + k] : 0.0f;
            for (int k = part; k < out_dim; k += kGatherThreads)
                tgt[r * kW + k] = ok ? g.targets[(size_t)idx * out_dim + k] : 0.0f;
        }
        __syncthreads();
        for (int idx = tid; idx < kTM * 32; idx += kThreads) {
            const int r = idx >> 5, f = idx & 31;
            float t = 0.0f;
#pragma unroll
            for (int k = 0; k < kIn; k++) t = t + g.freqs[f * kIn + k] * xin[r * kIn + k];
            float s, c;
            sincospi_own(2.0f * t, &s, &c);
            store_bf16(act, r, f, s);
            store_bf16(act, r, 32 + f, c);
            store_bf16(actT, f, r, s);
            store_bf16(actT, 32 + f, r, c);
        }
    };
    // The batch depends on the step number alone, so a step launched during its predecessor's update
    // (g.early) prepares it meanwhile. The number is the one that update will advance the counter to,
    // noted by it in step[2] before this kernel could start; after the wait the counter itself
    // decides, and another number's batch is replaced.
    uint32_t step = 0u;
    if (g.early && tid == 0) ahead_slot = __ldcg(g.step + 2);
    for (int pass = g.early ? 0 : 1; pass < 2; pass++) {
        if (pass == 1) {
            // the previous update (weights, image, step counter) complete and visible from here (returns
            // at once without a programmatic dependency)
            asm volatile("griddepcontrol.wait;" ::: "memory");
            // loads first, one round trip for all of them
            const uint32_t now = __ldcg(g.step);
            float bv = 0.0f;
            if (tid < kLayers * kW) {
                const int l = tid / kW, o = tid % kW, fo = l == kHidden ? out_dim : kW;
                if (o < fo) bv = __ldcg(g.params + (size_t)l * kLayerParams + fo * kW + o);
            }
            // weights in both layouts: bulk copies of the packed image (rows of the head beyond out_dim
            // are zero there), the first layer's on their own barrier so that its product need not wait
            // for the rest
            if (tid == 0) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                stage_copy(Wf, g.image, kMat * 4u, fbar);
                stage_copy(Wf + kMat, g.image + kMat, kImageBytes - kMat * 4u, bar);
            }
            if (tid < kLayers * kW) bias[tid] = bv;
            if (tid < kWarps) red[tid] = 0.0f;
            // the update reads this step's number from step[1] and advances step[0] itself
            if (blockIdx.x == 0 && tid == 0) __stcg(g.step + 1, now);
            asm volatile("griddepcontrol.launch_dependents;");
            if (g.early && now == step) break;
            step = now;
        }
        __syncthreads();
        if (pass == 0) step = ahead_slot;
        load_batch(step);
    }
    fence_async_smem();  // publishes the features to the tensor cores with the next barrier
    tc_fence_before();
    bool ok = true;
    uint32_t err = 0;
    // the barriers' initialisation and the TMEM address are visible from here
    __syncthreads();
    if (!__syncthreads_and(mbar_wait_bounded(fbar, 0u))) {
        err = kErrStage;
        ok = false;
    }
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t t_lane = tmem + ((uint32_t)(32 * rb) << 16);  // this warp's lane quarter
    // parities of the next completions: mma_bar; wgrad_bar[p] in bit p of wphase
    uint32_t phase = 0, wphase = 0;
    int w_pending = -1;                      // layer whose weight gradient waits in TMEM to be read out
    if (ok) {
        // injected failure (tests): a bounded wait on drain_bar, on which nothing arrives before the
        // teardown, runs out like a product whose completion never came
        if (g.inject_wait_polls) ok = __syncthreads_and(mbar_wait_bounded(dbar, 0u, g.inject_wait_polls));

        float acc[kNT][4];
        uint32_t zp[kNT][2] = {};  // the last layer's pre-activations, BF16
        float ds[kNT][4];          // silu' of them: taken while the next layer's product runs
        auto silu_prime = [&]() {
#pragma unroll
            for (int j = 0; j < kNT; j++)
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    ds[j][2 * hh] = silu_d(lo_of(zp[j][hh]));
                    ds[j][2 * hh + 1] = silu_d(hi_of(zp[j][hh]));
                }
        };
        // ---- forward: Z_l = act W_l^T in TMEM columns [0, 64); ok is block-uniform at the top of
        // each layer (the __syncthreads_and that ends the previous one)
        for (int l = 0; l < kHidden && ok; l++) {
            if (warp == 0 && elect_one()) {
                tc_fence_after();
                issue_product(tmem, act, Wf + l * kMat);
                commit_to(pbar);
            }
            if (l > 0) {
                silu_prime();
#pragma unroll
                for (int j = 0; j < kNT; j++)
                    dsil[((l - 1) * kNT + j) * kThreads + tid] = make_float4(ds[j][0], ds[j][1], ds[j][2], ds[j][3]);
            }
            float bl[kNT][2];
#pragma unroll
            for (int j = 0; j < kNT; j++) {
                bl[j][0] = bias[l * kW + n0 + j * 8 + 2 * tig];
                bl[j][1] = bias[l * kW + n0 + j * 8 + 2 * tig + 1];
            }
            ok = mbar_wait_bounded(pbar, phase);
            phase ^= 1u;
            tc_fence_after();
            load_acc(acc, t_lane + n0);
            uint32_t hp[kNT][2];
#pragma unroll
            for (int j = 0; j < kNT; j++)
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    const float z0 = acc[j][2 * hh] + bl[j][0], z1 = acc[j][2 * hh + 1] + bl[j][1];
                    zp[j][hh] = pack2(z0, z1);
                    hp[j][hh] = pack2(silu_f(z0), silu_f(z1));
                }
            // the product has read act (its completion arrived), so act takes the layer's output
            store_tile<false>(act, hp, m0, n0, lane);
            store_tile<true>(actT + (l + 1) * kMat, hp, m0, n0, lane);
            // the rest of the image, before the second layer's product
            if (l == 0 && !mbar_wait_bounded(bar, 0u)) {
                err = kErrStage;
                ok = false;
            }
            fence_async_smem();
            tc_fence_before();
            ok = __syncthreads_and(ok);
        }
        // `run` is the block-wide verdict (a __syncthreads_and), `ok` this thread's own waits since
        bool run = ok;
        // head: y = act W^T + b; loss sum (y - t)^2 / count; acc becomes dY = 2 (y - t) / count
        if (run) {
            if (warp == 0 && elect_one()) {
                tc_fence_after();
                issue_product(tmem, act, Wf + kHidden * kMat);
                commit_to(pbar);
            }
            silu_prime();
            ok = mbar_wait_bounded(pbar, phase);
            phase ^= 1u;
            tc_fence_after();
            load_acc(acc, t_lane + n0);
            const float count = (float)g.batch * (float)out_dim;
            float ls = 0.0f;
#pragma unroll
            for (int j = 0; j < kNT; j++)
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    const int row = m0 + gid + 8 * hh, col = n0 + j * 8 + 2 * tig;
                    const bool rok = blockIdx.x * kTM + row < g.batch;
                    float d0 = 0.0f, d1 = 0.0f;
                    if (rok && col < out_dim) d0 = acc[j][2 * hh] + bias[kHidden * kW + col] - tgt[row * kW + col];
                    if (rok && col + 1 < out_dim)
                        d1 = acc[j][2 * hh + 1] + bias[kHidden * kW + col + 1] - tgt[row * kW + col + 1];
                    ls += d0 * d0 + d1 * d1;
                    // columns beyond the head are zero without dividing it (a division's slow case: 2,000
                    // cycles for a head one output wide)
                    acc[j][2 * hh] = col < out_dim ? 2.0f * d0 / count : 0.0f;
                    acc[j][2 * hh + 1] = col + 1 < out_dim ? 2.0f * d1 / count : 0.0f;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, o);
            if (lane == 0) red[warp] = ls / count;
        }
        // ---- backward: at the top of each iteration acc holds dL/dZ_l for this warp's rows and
        // columns (FP32). dA = dZ W_l goes to TMEM columns [0, 64) and is committed first (the next
        // layer waits for it); dW_l = dZ^T act_l (dZ^T from buffer l & 1) to columns 64 + 64 (l & 1),
        // committed on wgrad_bar[l & 1] and read out one iteration later, while the next layer's
        // products run. Buffer and columns l & 1 are next written by layer l - 2, after that readout
        // (and the barrier that starts layer l - 1).
        const uint32_t slots = gradient_slots(g.out_dim);
        auto drain_wgrad = [&]() {
            // weight gradient dW[o][i] of layer w_pending: warp w takes o in [m0, m0 + 16), i in
            // [n0, n0 + 16)
            const int lw = w_pending, pw = lw & 1;
            ok = mbar_wait_bounded(pw ? wbar1 : wbar0, (wphase >> pw) & 1u) && ok;
            wphase ^= 1u << pw;
            tc_fence_after();
            const int fo = lw == kHidden ? out_dim : kW;
            if (m0 < fo) {
                float wacc[kNT][4];
                load_acc(wacc, t_lane + 64u + 64u * (uint32_t)(lw & 1) + n0);
                const int run = (lw * kRowBlocks + rb) * kColSplit + n0 / kCols;
                float4 *dst = reinterpret_cast<float4 *>(g.partial + (size_t)blockIdx.x * slots + (size_t)run * 256);
#pragma unroll
                for (int j = 0; j < kNT; j++)
                    dst[j * 32 + lane] = make_float4(wacc[j][0], wacc[j][1], wacc[j][2], wacc[j][3]);
            }
            w_pending = -1;
        };
        for (int l = kHidden; l >= 0 && run; l--) {
            if (l == 0) store_col_sums(acc, dbias + rb * kW, n0, lane, tig);
            {
                uint32_t dp[kNT][2];
#pragma unroll
                for (int j = 0; j < kNT; j++)
#pragma unroll
                    for (int hh = 0; hh < 2; hh++) dp[j][hh] = pack2(acc[j][2 * hh], acc[j][2 * hh + 1]);
                store_tile<false>(dZ, dp, m0, n0, lane);
                store_tile<true>(dZT + (l & 1) * kMat, dp, m0, n0, lane);
            }
            fence_async_smem();
            tc_fence_before();
            run = __syncthreads_and(ok);
            if (!run) break;
            // the two products from two warps, so that neither waits for the other's issue
            if (warp == 0 && l > 0 && elect_one()) {
                tc_fence_after();
                issue_product(tmem, dZ, Wb + (l - 1) * kMat);
                commit_to(pbar);
            }
            if (warp == kWgradWarp && elect_one()) {
                tc_fence_after();
                issue_product(tmem + 64u + 64u * (uint32_t)(l & 1), dZT + (l & 1) * kMat, actT + l * kMat);
                commit_to((l & 1) ? wbar1 : wbar0);
            }
            // while dA's product runs: the bias sums and the previous layer's dW (in the other columns)
            if (l > 0) store_col_sums(acc, dbias + (l * kRowBlocks + rb) * kW, n0, lane, tig);
            if (w_pending >= 0) drain_wgrad();
            w_pending = l;
            if (l == 0) {
                // the block's bias gradients and loss (published by the barrier above), while the last
                // product runs
                float *dst = g.partial + (size_t)blockIdx.x * slots + weight_slots(g.out_dim);
                for (int q = tid; q < kLayers * kW; q += kThreads) {
                    const int lb = q / kW, o = q % kW, fo = lb == kHidden ? out_dim : kW;
                    if (o >= fo) continue;
                    float b = dbias[(lb * kRowBlocks) * kW + o];
                    for (int r = 1; r < kRowBlocks; r++) b += dbias[(lb * kRowBlocks + r) * kW + o];
                    dst[q] = b;
                }
                if (tid == kThreads - 1) {
                    float ls = red[0];
                    for (int q = 1; q < kWarps; q++) ls += red[q];
                    g.partial_loss[blockIdx.x] = ls;
                }
                break;
            }
            if (l < kHidden)
#pragma unroll
                for (int j = 0; j < kNT; j++) {
                    const float4 v = dsil[((l - 1) * kNT + j) * kThreads + tid];
                    ds[j][0] = v.x, ds[j][1] = v.y, ds[j][2] = v.z, ds[j][3] = v.w;
                }
            // dZ_{l-1} = dA silu'(Z_{l-1}) (dA has read dZ once mma_bar arrives, so the next iteration may
            // overwrite it)
            ok = mbar_wait_bounded(pbar, phase) && ok;
            phase ^= 1u;
            tc_fence_after();
            load_acc(acc, t_lane + n0);
#pragma unroll
            for (int j = 0; j < kNT; j++)
#pragma unroll
                for (int q = 0; q < 4; q++) acc[j][q] *= ds[j][q];
        }
        if (run && w_pending >= 0) drain_wgrad();
        if (!ok && !err) err = kErrProduct;
    }
    // teardown: on an error, one more commit of each issuing thread (on drain_bar, bounded wait) covers
    // every product this block issued, and the staging copies get one more bounded wait each so that they do not write
    // into a later block's shared memory; every TMEM load has finished; then the TMEM columns are
    // released
    tc_fence_before();
    const bool all_ok = __syncthreads_and(err == 0);
    if (!all_ok) {
        const bool staged = __syncthreads_and(err != kErrStage);
        if ((warp == 0 || warp == kWgradWarp) && elect_one()) commit_to(dbar);
        if (tid == 0) {
            mbar_wait_bounded(dbar, 0u);
            mbar_wait_bounded(fbar, 0u);
            mbar_wait_bounded(bar, 0u);
            atomicOr(g.err, staged ? kErrProduct : kErrStage);
        }
        __syncthreads();
    }
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

// Parameter i's place in the packed image: its BF16 halves in the forward operand W [out][in]
// and, for layers >= 1, in the backward operand W^T [in][out]; biases have none (returns false).
__device__ __forceinline__ bool image_slots(uint32_t i, uint32_t out_dim, uint32_t &f, uint32_t &b) {
    uint32_t l = i / kLayerParams;
    if (l > (uint32_t)kHidden) l = kHidden;
    const uint32_t r = i - l * kLayerParams;
    const uint32_t fo = l == (uint32_t)kHidden ? out_dim : (uint32_t)kW;
    if (r >= fo * kW) return false;
    const uint32_t o = r / kW, in = r % kW;
    f = l * (uint32_t)kMatHalves + cm_index(o, in);
    b = l >= 1 ? ((uint32_t)kLayers + l - 1u) * (uint32_t)kMatHalves + cm_index(in, o) : 0xFFFFFFFFu;
    return true;
}
__device__ __forceinline__ void image_store(uint32_t *image, uint32_t i, uint32_t out_dim, float v) {
    uint32_t f, b;
    if (!image_slots(i, out_dim, f, b)) return;
    __nv_bfloat16 *h = reinterpret_cast<__nv_bfloat16 *>(image);
    const __nv_bfloat16 x = __float2bfloat16_rn(v);
    h[f] = x;
    if (b != 0xFFFFFFFFu) h[b] = x;
}

__global__ void pack_weights_kernel(const float *__restrict__ p, uint32_t n_params, uint32_t out_dim,
                                    uint32_t *__restrict__ image) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_params) image_store(image, i, out_dim, p[i]);
}

// Block-ordered gradient sums: a block of 256 threads takes 32 slots, 8 threads each summing
// every 8th block gradient in order, the 8 partial sums added in order (a fixed order: the step is
// deterministic). The kernel is bound by the latency of those loads: 16 of a thread's are in flight
// at a time (all of them for batches up to 8,192 rows).
constexpr int kRedSplit = 8;
constexpr int kRedLoads = 16;
// Registers capped (as the fused kernel's, below) so that the next step's blocks fit beside these.
constexpr int kAdamMinB = 6;
__device__ __forceinline__ float ordered_gradient(const float *__restrict__ partial, uint32_t n_blocks,
                                                  uint32_t slots, uint32_t slot, bool ok, float (*red)[33]) {
    const uint32_t q = threadIdx.x & 31u, sl = threadIdx.x >> 5;
    float s = 0.0f;
    if (ok)
        for (uint32_t b0 = sl; b0 < n_blocks; b0 += kRedSplit * kRedLoads) {
            float x[kRedLoads];  // zeros beyond the last block leave the sum as it is
#pragma unroll
            for (int k = 0; k < kRedLoads; k++) {
                const uint32_t b = b0 + k * kRedSplit;
                x[k] = b < n_blocks ? __ldcg(partial + (size_t)b * slots + slot) : 0.0f;
            }
#pragma unroll
            for (int k = 0; k < kRedLoads; k++) s += x[k];
        }
    red[sl][q] = s;
    __syncthreads();
    float t = 0.0f;
    if (sl == 0)
        for (int k = 0; k < kRedSplit; k++) t += red[k][q];
    return t;
}

// The blocks' losses summed by one warp in a fixed order (lane-strided partial sums, then a
// butterfly that leaves the same value in every lane).
__device__ __forceinline__ float ordered_loss(const float *__restrict__ partial_loss, uint32_t n_blocks) {
    float l = 0.0f;
    for (uint32_t b = threadIdx.x & 31u; b < n_blocks; b += 32u) l += partial_loss[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    return l;
}

// Learning rate and Adam's two bias corrections of step s.
__device__ __noinline__ float3 schedule_of(uint32_t s, uint32_t steps, float lr0, uint32_t adam_base) {
    const float t = (float)(adam_base + s + 1u);
    return make_float3(lr0 * 0.5f * (1.0f + cospif((float)s / (float)steps)), 1.0f - powf(0.9f, t),
                       1.0f - powf(0.999f, t));
}

// Sums the blocks' gradients and applies Adam with the cosine schedule of the current step, then
// stores the new weights into the packed image; block 0 records the step's loss and advances the step
// counter, step[0]. The fused step left its number in step[1], so that no block reads the word that
// another one advances.
__global__ void __launch_bounds__(256, kAdamMinB) mlp_reduce_adam_kernel(
    float *__restrict__ p, float *__restrict__ m, float *__restrict__ v, const float *__restrict__ partial,
    const float *__restrict__ partial_loss, uint32_t n_blocks, uint32_t out_dim,
    uint32_t *__restrict__ image, uint32_t *step, uint32_t steps, float lr0, uint32_t adam_base,
    float *__restrict__ loss_hist, const uint32_t *err) {
    __shared__ float red[kRedSplit][33];
    // The step's number, the schedule and this thread's parameter and moments were settled by the
    // previous update, which the fused step waited for before it let this kernel start: read while
    // that step runs (the number is checked below). step[2] takes the number of the next step's batch:
    // the fused step's blocks have all read the last one, and the next step starts after this.
    const uint32_t s = __ldcg(step + 1);
    const uint32_t slots = gradient_slots(out_dim), slot = blockIdx.x * 32u + (threadIdx.x & 31u);
    uint32_t i;
    const bool valid = slot_param(slot, out_dim, i), mine = valid && threadIdx.x < 32;
    float3 sched = make_float3(0.0f, 1.0f, 1.0f);
    float p0 = 0.0f, m0 = 0.0f, v0 = 0.0f;
    if (mine) {
        p0 = __ldcg(p + i);
        m0 = __ldcg(m + i);
        v0 = __ldcg(v + i);
        sched = schedule_of(s, steps, lr0, adam_base);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        __stcg(step + 2, s + 1u);
        __threadfence();
    }
    // the fused step's gradients complete and visible from here; the next step may start launching
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const uint32_t failed = __ldcg(err), now = __ldcg(step + 1);  // tested after the sums' loads are out
    const float gsum = ordered_gradient(partial, n_blocks, slots, slot, valid, red);
    // a block of the fused step failed (its gradient is missing): no update, no step advance, so the
    // parameters stay those of the last complete step
    if (failed) return;
    if (mine) {
        if (now != s) sched = schedule_of(now, steps, lr0, adam_base);
        const float mi = 0.9f * m0 + 0.1f * gsum;
        const float vi = 0.999f * v0 + 0.001f * gsum * gsum;
        m[i] = mi;
        v[i] = vi;
        const float pi = p0 - sched.x * (mi / sched.y) / (sqrtf(vi / sched.z) + 1e-8f);
        p[i] = pi;
        image_store(image, i, out_dim, pi);
    }
    if (blockIdx.x == 0 && threadIdx.x >= 224) {
        const float l = loss_hist ? ordered_loss(partial_loss, n_blocks) : 0.0f;
        if (threadIdx.x == 224) {
            if (loss_hist) loss_hist[now] = l;
            step[0] = now + 1u;
        }
    }
}

__global__ void __launch_bounds__(256) mlp_reduce_grad_kernel(const float *__restrict__ partial,
                                                              const float *__restrict__ partial_loss, uint32_t n_blocks,
                                                              uint32_t out_dim, float *__restrict__ grad,
                                                              float *__restrict__ loss) {
    __shared__ float red[kRedSplit][33];
    const uint32_t slots = gradient_slots(out_dim), slot = blockIdx.x * 32u + (threadIdx.x & 31u);
    uint32_t i;
    const bool valid = slot_param(slot, out_dim, i);
    const float gsum = ordered_gradient(partial, n_blocks, slots, slot, valid, red);
    if (threadIdx.x < 32 && valid) grad[i] = gsum;
    if (loss && blockIdx.x == 0 && threadIdx.x < 32) {
        const float l = ordered_loss(partial_loss, n_blocks);
        if (threadIdx.x == 0) *loss = l;
    }
}

}  // namespace

size_t fused_train_smem_bytes() { return kSmemWords * 4 + kSmemFloats * 4; }
size_t fused_train_image_words() { return kImageWords; }
size_t fused_train_partial_words(uint32_t out_dim) { return gradient_slots(out_dim); }
uint32_t fused_train_blocks(uint32_t batch) { return (batch + kTM - 1) / kTM; }

cudaError_t launch_pack_weights(const float *params, uint32_t n_params, uint32_t out_dim, uint32_t *image,
                                cudaStream_t stream) {
    pack_weights_kernel<<<(n_params + 255) / 256, 256, 0, stream>>>(params, n_params, out_dim, image);
    return cudaGetLastError();
}

// A launch that may begin while the stream's previous kernel is still running (programmatic
// dependent launch): the kernel waits for that kernel's completion itself (griddepcontrol.wait).
template <typename... Params, typename... Args>
cudaError_t launch_after_previous(void (*kernel)(Params...), uint32_t grid, uint32_t block, size_t smem,
                                  cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t launch_fused_train_step(const FusedTrainArgs &a, float *params, float *adam_m, float *adam_v,
                                    uint32_t steps, float lr, uint32_t adam_base, float *loss_hist,
                                    cudaStream_t stream) {
    const uint32_t blocks = fused_train_blocks(a.batch);
    cudaError_t e = launch_after_previous(mlp_train_fused_kernel, blocks, kThreads, fused_train_smem_bytes(), stream, a);
    if (e != cudaSuccess) return e;
    return launch_after_previous(mlp_reduce_adam_kernel, gradient_slots(a.out_dim) / 32, 256, 0, stream, params, adam_m, adam_v,
                                 (const float *)a.partial, (const float *)a.partial_loss, blocks, a.out_dim,
                                 const_cast<uint32_t *>(a.image), a.step, steps, lr, adam_base, loss_hist,
                                 (const uint32_t *)a.err);
}

cudaError_t launch_fused_gradient(const FusedTrainArgs &a, float *grad, float *loss, cudaStream_t stream) {
    const uint32_t blocks = fused_train_blocks(a.batch);
    cudaError_t e = launch_pack_weights(a.params, a.n_params, a.out_dim, const_cast<uint32_t *>(a.image), stream);
    if (e != cudaSuccess) return e;
    mlp_train_fused_kernel<<<blocks, kThreads, fused_train_smem_bytes(), stream>>>(a);
    mlp_reduce_grad_kernel<<<gradient_slots(a.out_dim) / 32, 256, 0, stream>>>(a.partial, a.partial_loss, blocks,
                                                                               a.out_dim, grad, loss);
    return cudaGetLastError();
}

cudaError_t prepare_fused_train() {
    return cudaFuncSetAttribute(mlp_train_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)fused_train_smem_bytes());
}

}  // namespace wobgb
