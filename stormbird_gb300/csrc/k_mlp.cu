// Warm-start network kernels (sm_103a).
//
// k_mlp_gemm: C[M][N] = A[M][K] B[N][K]^T on the 5th-generation tensor cores. One CTA of
// eight warps owns a 128 x N output tile whose FP32 accumulator lives in tensor memory
// (256 columns allocated with tcgen05.alloc). The operands arrive by TMA: per 64-wide K
// step one thread issues two cp.async.bulk.tensor.2d copies (A: 64 x 128, B: 64 x N BF16)
// into a stage of shared memory in the 128-byte-swizzled K-major layout (one 128-byte row
// per matrix row, 16-byte chunks XOR-ed with the row index mod 8, 8-row atoms 1024 B
// apart), completing on the stage's `full` mbarrier. Two stages run ahead of the tensor
// cores; the same thread waits for a stage, issues four tcgen05.mma.cta_group::1.kind::f16
// (K = 16 each: the descriptor start advances 32 B inside the swizzle atom) and commits to
// the stage's `empty` mbarrier, and refills the stage of the previous step once its MMAs
// have completed, so one step of MMAs is always queued behind the running one. Two CTAs
// fit on an SM (shared memory), so one CTA's epilogue overlaps the other's MMAs. The
// epilogue reads the accumulator with tcgen05.ld (32 lanes x 32 columns per warp and
// instruction; warps w and w + 4 own tensor-memory lanes 32 (w mod 4) .. + 31 = rows and
// half of the columns each) and applies the layer's bias and GELU (forward), the GELU
// derivative (backward), or stores split-K partial sums (weight gradients). Waits are
// bounded: a wait that runs out records kDevTimeout, skips the epilogue, waits (bounded)
// for the copies and MMAs in flight and frees the tensor memory.
//
// k_mlp_forward: the whole network for inference, layers fused (see there).
//
// The rest are CUDA-core kernels: the width->1 output layer with the MSE loss, input
// packing, deterministic fixed-order reductions, Adam, weight casts, and the batch-side
// feature / candidate / target kernels of the warm start.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "sb_mlp.h"
#include "sb_ptx.cuh"

namespace sbgpu {

namespace {

constexpr int kGemmThreads = 256;  // 8 warps: warps w and w + 4 drain one lane quadrant
constexpr int kKStep = 64;       // one 128-byte swizzle row of BF16
constexpr int kStages = 2;
constexpr uint32_t kSBO = 1024;  // bytes between 8-row atoms
constexpr uint32_t kStageA = kMlpRowTile * kKStep * 2;
constexpr uint32_t kStageB = kMlpWidth * kKStep * 2;
constexpr uint32_t kStage = kStageA + kStageB;
constexpr uint32_t kTmemCols = 256;
constexpr int kTurnLd = 36;  // floats of a row of a warp's 32 x 32 turning tile
static_assert(kStageA % 1024 == 0 && kStage % 1024 == 0, "stages keep the 1024-byte swizzle alignment");

// tcgen05 shared-memory matrix descriptor of a K-major 128-byte-swizzled tile: start
// address (>> 4), leading offset 16 B (unused by this layout), SBO 1024 B (>> 4), version
// 1, layout type 2 (128-byte swizzle), base offset 0 (atoms are 1024-byte aligned).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (1ull << 16) |
           (static_cast<uint64_t>((kSBO >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}

// 2-D tiled TMA copy of the box at (x, y) (x in elements along the contiguous dimension)
// into shared memory, completing on `bar`.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// Instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major, M x N.
__device__ __forceinline__ uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
           (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// 32 consecutive FP32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// GELU with the error function, and its derivative
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__global__ void __launch_bounds__(kGemmThreads) k_mlp_gemm(const __grid_constant__ CUtensorMap map_a,
                                                           const __grid_constant__ CUtensorMap map_b, GemmArgs g) {
    extern __shared__ unsigned char dyn[];
    __shared__ __align__(8) uint64_t full[kStages];
    __shared__ __align__(8) uint64_t empty[kStages];
    __shared__ uint32_t s_tmem;
    __shared__ int s_issued, s_ok;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kMlpRowTile;
    const int split = blockIdx.y;
    // gridDim.z CTAs share a row tile's columns (two while there are no more tiles than SMs, as with the 128
    // tiles of 16,384 training rows: the epilogue takes most of the time, and two CTAs of an SM overlap the one's
    // with the other's main loop: forward 20 us at one, 18 at two)
    const int cols = g.N / gridDim.z, n0 = blockIdx.z * cols;
    const int k_begin = split * g.k_split;
    const int k_end = min(g.K, k_begin + g.k_split);
    const int nk = (k_end - k_begin) / kKStep;

    if (warp == 0) tmem_alloc(&s_tmem, kTmemCols);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        fence_mbar_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    if (tid == 0) {
        const uint32_t idesc = idesc_bf16(kMlpRowTile, cols);
        const uint32_t tx = kStageA + static_cast<uint32_t>(cols) * kKStep * 2;
        auto load = [&](int kt) {
            const int s = kt % kStages;
            unsigned char* sa = base + s * kStage;
            mbar_expect_tx(&full[s], tx);
            tma_load_2d(sa, &map_a, k_begin + kt * kKStep, m0, &full[s]);
            tma_load_2d(sa + kStageA, &map_b, k_begin + kt * kKStep, n0, &full[s]);
        };
        int loaded = 0;  // K steps whose copies were issued
        for (; loaded < min(nk, kStages); ++loaded) load(loaded);
        bool ok = true;
        int issued = 0;  // K steps whose MMAs were issued
        for (int kt = 0; kt < nk; ++kt) {
            const int s = kt % kStages;
            if (!mbar_wait_bounded(&full[s], (kt / kStages) & 1, g.err)) {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t a_addr = smem_u32(base + s * kStage), b_addr = a_addr + kStageA;
#pragma unroll
            for (int j = 0; j < kKStep / 16; ++j)
                mma_bf16(tmem, smem_desc_sw128(a_addr + j * 32), smem_desc_sw128(b_addr + j * 32), idesc,
                         (kt > 0 || j > 0) ? 1u : 0u);
            mma_commit(&empty[s]);
            issued = kt + 1;
            // refill the stage of step kt - 1 once its MMAs are done (those of step kt stay queued)
            if (kt >= 1 && loaded < nk) {
                const int p = kt - 1;
                if (!mbar_wait_bounded(&empty[p % kStages], (p / kStages) & 1, g.err)) {
                    ok = false;
                    break;
                }
                load(loaded);
                ++loaded;
            }
        }
        // copies issued but never consumed still write shared memory: wait for them
        if (!ok)
            for (int kt = issued; kt < loaded; ++kt) mbar_wait_bounded(&full[kt % kStages], (kt / kStages) & 1, g.err);
        s_issued = issued;
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    const int issued = s_issued;
    // the last commit arrives when every MMA issued before it has completed
    bool done = s_ok && issued == nk && nk > 0;
    if (issued > 0) {
        const int p = issued - 1;
        const bool w = mbar_wait_bounded(&empty[p % kStages], (p / kStages) & 1, g.err);
        done = done && w;
    }
    done = __syncthreads_and(done);
    tc_fence_after();

    if (done) {
        // a warp reads the tensor-memory lanes of its quadrant (warp mod 4); the two warps of
        // a quadrant take half of the columns each
        const int quad = warp & 3, half = warp >> 2;
        const int row = m0 + quad * 32 + lane;
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        const int c_end = n0 + (half + 1) * (cols / 2);
        // The operands are done with: their shared memory turns rows per lane into rows per warp, so that
        // a store (or load) instruction covers whole 64- or 128-byte pieces of rows (at 16,384 x 256, a lane
        // storing its own row and 2-byte columns: forward 20.7 us, backward 21.3; now 16.3 and 17.6, bound by
        // the error function's instructions). FP32: 32 x 32 values,
        // rows padded to 36; BF16: 64-byte rows of four 16-byte chunks, XOR-ed so that rows written by
        // lanes, rows read four lanes to one and columns read by ldmatrix all hit distinct banks.
        float* tf = reinterpret_cast<float*>(base) + warp * (32 * kTurnLd + 32 * 16);
        unsigned char* tb = reinterpret_cast<unsigned char*>(tf + 32 * kTurnLd);
        auto chunk = [&](int r, int c) { return tb + r * 64 + ((c ^ ((r >> 1) & 3) ^ ((r >> 3) & 3)) << 4); };
        const int r8 = lane >> 3, c8 = (lane & 7) * 4;
        for (int c0 = n0 + half * (cols / 2); c0 < c_end; c0 += 32) {
            // element (row r8 + 4 q, column c8) of the FP32 tile in memory
            const long long at = static_cast<long long>(m0 + quad * 32 + r8) * g.N + c0 + c8;
            if (g.mode == kGemmBackward) {
                float4 z[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) z[q] = *reinterpret_cast<const float4*>(g.z_in + at + 4 * q * g.N);
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q) *reinterpret_cast<float4*>(tf + (r8 + 4 * q) * kTurnLd + c8) = z[q];
                __syncwarp();
            }
            float v[32];
            tmem_ld32(lane_addr + static_cast<uint32_t>(c0 - n0), v);
            float* mine = tf + lane * kTurnLd;
            if (g.mode == kGemmBackward) {  // through the GELU of the layer below
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 z = *reinterpret_cast<const float4*>(mine + 4 * q);
                    v[4 * q] *= gelu_grad(z.x);
                    v[4 * q + 1] *= gelu_grad(z.y);
                    v[4 * q + 2] *= gelu_grad(z.z);
                    v[4 * q + 3] *= gelu_grad(z.w);
                }
            } else {
                if (g.mode == kGemmForward) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b4 = *reinterpret_cast<const float4*>(g.bias + c0 + j);
                        v[j] += b4.x;
                        v[j + 1] += b4.y;
                        v[j + 2] += b4.z;
                        v[j + 3] += b4.w;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    *reinterpret_cast<float4*>(mine + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                __syncwarp();
                float* o = g.mode == kGemmPartial ? g.part_out + static_cast<long long>(split) * g.M * g.N : g.z_out;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    *reinterpret_cast<float4*>(o + at + 4 * q * g.N) = *reinterpret_cast<const float4*>(tf + (r8 + 4 * q) * kTurnLd + c8);
                if (g.mode == kGemmPartial) continue;
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = gelu(v[j]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                __nv_bfloat162 p[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
                *reinterpret_cast<uint4*>(chunk(lane, q)) = *reinterpret_cast<uint4*>(p);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int rr = 8 * q + (lane >> 2);
                *reinterpret_cast<uint4*>(g.h_out + static_cast<long long>(m0 + quad * 32 + rr) * g.N + c0 + (lane & 3) * 8) =
                    *reinterpret_cast<const uint4*>(chunk(rr, lane & 3));
            }
            // transposed: with row 8 t + 2 m + e as row 2 t + e of matrix m, lane 4 c + t of a transposed
            // ldmatrix gets rows 8 t .. 8 t + 7 of column c, 16 bytes of a row of the transpose
            if (g.hT_out) {
                const int lr = 8 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 w;
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(smem_u32(chunk(lr, q))) : "memory");
                    *reinterpret_cast<uint4*>(g.hT_out + static_cast<long long>(c0 + 8 * q + (lane >> 2)) * g.ldt + m0 + quad * 32 +
                                              (lane & 3) * 8) = w;
                }
            }
            __syncwarp();
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------------------
// Inference: the whole network for 128-row tiles in one persistent kernel, two tiles at a time on an SM.
// The activations never leave it: a layer's epilogue writes the next layer's A operand (BF16,
// 128-byte-swizzled K-major) over the one the tensor cores have just finished with. Roles (18
// warps): one thread streams the weights by TMA in 128 x 64 half slabs through a ring of five, one
// issues the MMAs, eight warps a tile drain its accumulator (tensor memory: two tiles x 256 FP32
// columns); the two tiles take turns, so that one's MMAs and weights run under the other's epilogue.
// With no more tiles than SMs all sixteen warps drain the one.
// The epilogue is what bounds it: 1,024 GELUs a row with erff, 32 issued instructions each (98,307 rows: 85 us
// at one per cycle and SM sub-partition), against 8,192 tensor-core FMAs a cycle. Results are those of
// the layer-by-layer kernels bit for bit (the same K order in the accumulator, the same roundings,
// the output layer's sums in k_mlp_head's order).
// 98,307 rows: layer by layer (pack, four GEMMs, output layer; activations through L2 and HBM, each CTA's
// epilogue after its main loop) 290 us a call, both tiles in step 187, in turn 174 us.
constexpr int kFwdWarps = 16;
constexpr int kFwdThreads = 32 * (kFwdWarps + 2);
constexpr int kFwdRing = 5;
constexpr uint32_t kFwdSub = 128 * kKStep * 2;   // a 128 x 64 BF16 sub-tile (A quarter or half slab)
constexpr uint32_t kFwdTile = 4 * kFwdSub;       // activations of a tile
constexpr int kFwdTurnLd = 20;                   // floats of a row of a warp's 32 x 16 turning tile
constexpr int kFwdPartLd = 33;                   // row pitch of the output layer's partial sums
constexpr uint32_t kFwdSmem = 2 * kFwdTile + kFwdRing * kFwdSub + (kMlpHidden * kMlpWidth + kMlpWidth + 4) * 4 + 1024;
static_assert(128 * kFwdPartLd * 4 <= kFwdTile, "partial sums fit a tile's activations");
static_assert(kFwdWarps * 32 * kFwdTurnLd * 4 <= kFwdTile, "the turning tiles fit the second slot");

struct FwdMaps {
    CUtensorMap w[kMlpHidden];
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// TRAIN: every layer's pre-activations, activations and their transposes go out as well (FwdArgs::z, h, hT)
// and the output layer is left to k_mlp_head. One tile a CTA: the second slot's shared memory turns the
// stores, and activations go out under the next layer's MMAs. 16,384 rows: 46 us, against four GEMM launches of 13 to 16
// and the gaps between them (with activations stored before the next layer may start 53).
template <bool TRAIN>
__global__ void __launch_bounds__(kFwdThreads, 1) k_mlp_forward(const __grid_constant__ FwdMaps maps, FwdArgs g) {
    extern __shared__ unsigned char dyn[];
    unsigned char* act = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
    unsigned char* ring = act + 2 * kFwdTile;
    float* bias = reinterpret_cast<float*>(ring + kFwdRing * kFwdSub);  // [4][256]
    float* wout = bias + kMlpHidden * kMlpWidth;                        // [257]
    __shared__ __align__(8) uint64_t full[kFwdRing], empty[kFwdRing], acc_full[2], act_ready[2];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const int tiles = (g.rows + 127) / 128, G = gridDim.x;
    const bool wide = tiles <= G;  // one tile at a time
    // tile k of slot q: the first slots of all CTAs, then the second ones
    auto tile_of = [&](int k, int q) { return wide ? (q == 0 && k == 0 ? static_cast<int>(blockIdx.x) : tiles)
                                                   : (2 * k + q) * G + static_cast<int>(blockIdx.x); };
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    if (tid == 0) {
        for (int s = 0; s < kFwdRing; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(&acc_full[q], 1);
            mbar_init(&act_ready[q], wide ? kFwdWarps : kFwdWarps / 2);
        }
        fence_mbar_init();
    }
    for (int i = tid; i < kMlpHidden * kMlpWidth; i += kFwdThreads) bias[i] = g.bias[i / kMlpWidth][i % kMlpWidth];
    for (int i = tid; i <= kMlpWidth; i += kFwdThreads) wout[i] = g.w_out[i];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    // half slabs of layer l: 128 outputs x 64 inputs, the two halves of a slab after one another
    auto halves = [](int l) { return l == 0 ? 2 * (kMlpInPad / kKStep) : 2 * (kMlpWidth / kKStep); };

    if (warp == kFwdWarps) {
        if (lane == 0) {  // weights
            int n = 0;
            bool ok = true;
            for (int k = 0; tile_of(k, 0) < tiles && ok; ++k)
                for (int l = 0; l < kMlpHidden && ok; ++l)
                    for (int q = 0; q < 2 && tile_of(k, q) < tiles && ok; ++q)
                        for (int h = 0; h < halves(l); ++h, ++n) {
                            const int s = n % kFwdRing;
                            if (n >= kFwdRing && !mbar_wait_bounded(&empty[s], (n / kFwdRing - 1) & 1, g.err)) {
                                ok = false;
                                break;
                            }
                            mbar_expect_tx(&full[s], kFwdSub);
                            tma_load_2d(ring + s * kFwdSub, &maps.w[l], (h >> 1) * kKStep, (h & 1) * 128, &full[s]);
                        }
            // every copy has landed before the CTA leaves: the MMA thread waits for them as it reads them, but
            // reads no more after a wait of its own that ran out
            for (int k = n - kFwdRing > 0 ? n - kFwdRing : 0; k < n; ++k)
                mbar_wait_bounded(&full[k % kFwdRing], (k / kFwdRing) & 1, g.err);
        }
    } else if (warp == kFwdWarps + 1) {
        if (lane == 0) {  // MMAs
            const uint32_t idesc = idesc_bf16(128, 128);
            int n = 0, layer[2] = {0, 0};
            bool ok = true;
            for (int k = 0; tile_of(k, 0) < tiles && ok; ++k)
                for (int l = 0; l < kMlpHidden && ok; ++l)
                    for (int q = 0; q < 2 && tile_of(k, q) < tiles && ok; ++q) {
                        if (!mbar_wait_bounded(&act_ready[q], layer[q] & 1, g.err)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        for (int h = 0; h < halves(l); ++h, ++n) {
                            const int s = n % kFwdRing;
                            if (!mbar_wait_bounded(&full[s], (n / kFwdRing) & 1, g.err)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            const uint32_t b = smem_u32(ring + s * kFwdSub);
                            const uint32_t a = smem_u32(act + q * kFwdTile + (h >> 1) * kFwdSub);
#pragma unroll
                            for (int j = 0; j < kKStep / 16; ++j)
                                mma_bf16(tmem + q * 256 + (h & 1) * 128, smem_desc_sw128(a + j * 32), smem_desc_sw128(b + j * 32),
                                         idesc, (h > 1 || j > 0) ? 1u : 0u);
                            mma_commit(&empty[s]);
                        }
                        mma_commit(&acc_full[q]);  // after a wait that ran out: of what was issued
                        ++layer[q];
                    }
            // a commit arrives when every MMA before it is done: the last of both slots
            for (int q = 0; q < 2; ++q)
                if (layer[q] > 0) mbar_wait_bounded(&acc_full[q], (layer[q] - 1) & 1, g.err);
        }
    } else {
        const int quad = warp & 3;          // tensor-memory lanes
        const int row = quad * 32 + lane;   // of a tile
        const int q = wide ? 0 : warp >> 3;                           // slot
        const int part = wide ? warp >> 2 : (warp >> 2) & 1, parts = wide ? 4 : 2;  // of the tile's columns
        const int width = kMlpWidth / parts;
        const int meet = wide ? 32 * kFwdWarps : 16 * kFwdWarps;      // threads of the slot
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        int layer = 0;
        // a warp whose wait ran out works no more, but arrives and meets the others' barriers
        bool ok = true;
        for (int k = 0; tile_of(k, q) < tiles; ++k) {
            unsigned char* a = act + q * kFwdTile;
            const long long r = tile_of(k, q) * 128LL + row;
            // A element (row, column): 64-column sub-tiles, rows of 128 bytes, 16-byte chunks XOR-ed with row mod 8
            auto chunk = [&](int col) { return a + (col >> 6) * kFwdSub + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4); };
            {  // inputs, BF16, zeros past n_in and past the last row
                const float* x = g.x + r * g.n_in;
                for (int c = part * (kMlpInPad / parts); c < (part + 1) * (kMlpInPad / parts); c += 8) {
                    float v[8];
                    if (g.vec_x && r < g.rows && c + 8 <= g.n_in) {
                        const float4 u0 = *reinterpret_cast<const float4*>(x + c), u1 = *reinterpret_cast<const float4*>(x + c + 4);
                        v[0] = u0.x; v[1] = u0.y; v[2] = u0.z; v[3] = u0.w;
                        v[4] = u1.x; v[5] = u1.y; v[6] = u1.z; v[7] = u1.w;
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = (r < g.rows && c + j < g.n_in) ? x[c + j] : 0.f;
                    }
                    __nv_bfloat162 p[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    *reinterpret_cast<uint4*>(chunk(c)) = *reinterpret_cast<uint4*>(p);
                }
            }
            // TRAIN: what the warp has written of layer l's activations, by rows and by columns
            auto publish = [&](int l) {
                const long long row0 = static_cast<long long>(tile_of(k, q)) * 128 + quad * 32;
                auto at = [&](int rr, int col) {
                    const int w = quad * 32 + rr;
                    return a + (col >> 6) * kFwdSub + w * 128 + ((((col & 63) >> 3) ^ (w & 7)) << 4);
                };
                __syncwarp();
#pragma unroll 1
                for (int c0 = part * width; c0 < (part + 1) * width; c0 += 32) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        const int rr = i + (lane >> 2), col = c0 + (lane & 3) * 8;
                        *reinterpret_cast<uint4*>(g.h[l] + (row0 + rr) * kMlpWidth + col) = *reinterpret_cast<const uint4*>(at(rr, col));
                    }
                    if (!g.hT[l]) continue;
                    const int lr = 8 * ((lane & 7) >> 1) + 2 * (lane >> 3) + (lane & 1);  // as in k_mlp_gemm
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint4 w;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(smem_u32(at(lr, c0 + i))) : "memory");
                        *reinterpret_cast<uint4*>(g.hT[l] + static_cast<long long>(c0 + i + (lane >> 2)) * g.ldt + row0 + (lane & 3) * 8) = w;
                    }
                }
                __syncwarp();
            };
#pragma unroll 1
            for (int l = 0; l < kMlpHidden; ++l, ++layer) {
                // the operand is written (and the accumulator read): the tensor cores may start
                tc_fence_before();
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&act_ready[q]);
                if (TRAIN && l > 0) publish(l - 1);  // under this layer's MMAs
                if (ok && !mbar_wait_bounded(&acc_full[q], layer & 1, g.err)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) continue;
                tc_fence_after();
                const float* bl = bias + l * kMlpWidth;
#pragma unroll 1
                for (int c0 = part * width; c0 < (part + 1) * width; c0 += 32) {
                    float v[32];
                    tmem_ld32(lane_addr + static_cast<uint32_t>(q * 256 + c0), v);
                    const long long row0 = static_cast<long long>(tile_of(k, q)) * 128 + quad * 32;  // the warp's rows
                    if constexpr (TRAIN) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 b4 = *reinterpret_cast<const float4*>(bl + c0 + j);
                            v[j] += b4.x;
                            v[j + 1] += b4.y;
                            v[j + 2] += b4.z;
                            v[j + 3] += b4.w;
                        }
                        // sixteen columns at a time, rows of 20 floats: stores of 64 bytes a row
                        float* turn = reinterpret_cast<float*>(act + kFwdTile) + warp * (32 * kFwdTurnLd);
#pragma unroll
                        for (int j = 0; j < 32; j += 16) {
#pragma unroll
                            for (int i = 0; i < 16; i += 4)
                                *reinterpret_cast<float4*>(turn + lane * kFwdTurnLd + i) = make_float4(v[j + i], v[j + i + 1], v[j + i + 2], v[j + i + 3]);
                            __syncwarp();
#pragma unroll
                            for (int i = 0; i < 32; i += 8) {
                                const int rr = i + (lane >> 2);
                                *reinterpret_cast<float4*>(g.z[l] + (row0 + rr) * kMlpWidth + c0 + j + (lane & 3) * 4) =
                                    *reinterpret_cast<const float4*>(turn + rr * kFwdTurnLd + (lane & 3) * 4);
                            }
                            __syncwarp();
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = gelu(v[j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 b4 = *reinterpret_cast<const float4*>(bl + c0 + j);
                            v[j] = gelu(v[j] + b4.x);
                            v[j + 1] = gelu(v[j + 1] + b4.y);
                            v[j + 2] = gelu(v[j + 2] + b4.z);
                            v[j + 3] = gelu(v[j + 3] + b4.w);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        __nv_bfloat162 p[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[j + 2 * i], v[j + 2 * i + 1]);
                        if (TRAIN || l + 1 < kMlpHidden) {
                            *reinterpret_cast<uint4*>(chunk(c0 + j)) = *reinterpret_cast<uint4*>(p);
                        } else {  // output layer: the partial sum of these 8 columns
                            float s = 0.f;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const float2 f = __bfloat1622float2(p[i]);
                                s = fmaf(f.x, wout[c0 + j + 2 * i], s);
                                s = fmaf(f.y, wout[c0 + j + 2 * i + 1], s);
                            }
                            reinterpret_cast<float*>(a)[row * kFwdPartLd + ((c0 + j) >> 3)] = s;
                        }
                    }
                }
            }
            if constexpr (TRAIN) {
                publish(kMlpHidden - 1);
                break;  // the one tile
            }
            // a row's 32 partial sums in the order of a butterfly over 32 lanes
            asm volatile("bar.sync %0, %1;" ::"r"(1 + q), "r"(meet) : "memory");
            if (ok && part == 0 && r < g.rows) {
                const float* p = reinterpret_cast<const float*>(a) + row * kFwdPartLd;
                float s[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) s[i] = p[i] + p[i + 16];
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < o; ++i) s[i] += s[i + o];
                g.y[r] = s[0] + wout[kMlpWidth];
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + q), "r"(meet) : "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// A CTA takes kHeadGroups groups of kHeadRowsPerCta rows, a warp per row of a group; each group has its own
// partial sums (the sums over groups then add them in group order, k_mlp_head_sums). dz goes out
// transposed through shared memory: 64 bytes of a column's rows at a time (with 8 rows a CTA its
// 2-byte stores made the kernel 43 us at 16,384 rows).
__global__ void __launch_bounds__(32 * kHeadRowsPerCta) k_mlp_head(HeadArgs a) {
    constexpr int kRows = kHeadGroups * kHeadRowsPerCta;
    __shared__ float wacc[kHeadRowsPerCta][kMlpWidth + 2];
    __shared__ __align__(16) bf16 dzs[kRows][kMlpWidth + 8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int f0 = lane * 8;
    float w8[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w8[j] = a.w[f0 + j];
#pragma unroll 1
    for (int gr = 0; gr < kHeadGroups; ++gr) {
        const int lr = gr * kHeadRowsPerCta + warp;
        const int r = blockIdx.x * kRows + lr;  // < rows_pad
        float hv[8];
        {
            const uint4 raw = *reinterpret_cast<const uint4*>(a.h + static_cast<long long>(r) * kMlpWidth + f0);
            const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(p[j]);
                hv[2 * j] = f.x;
                hv[2 * j + 1] = f.y;
            }
        }
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(hv[j], w8[j], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float y = s + a.w[kMlpWidth];
        const float res = r < a.rows ? y - a.target[r] : 0.f;
        const float dy = 2.f * res * a.inv_n;
        const float4* zp = reinterpret_cast<const float4*>(a.z + static_cast<long long>(r) * kMlpWidth + f0);
        const float4 z0 = zp[0], z1 = zp[1];
        const float zz[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
        float dz[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) dz[j] = dy * w8[j] * gelu_grad(zz[j]);
        __nv_bfloat162 pk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) pk[j] = __floats2bfloat162_rn(dz[2 * j], dz[2 * j + 1]);
        *reinterpret_cast<uint4*>(a.dz + static_cast<long long>(r) * kMlpWidth + f0) = *reinterpret_cast<uint4*>(pk);
        *reinterpret_cast<uint4*>(&dzs[lr][f0]) = *reinterpret_cast<uint4*>(pk);
#pragma unroll
        for (int j = 0; j < 8; ++j) wacc[warp][f0 + j] = dy * hv[j];
        if (lane == 0) {
            wacc[warp][kMlpWidth] = dy;
            wacc[warp][kMlpWidth + 1] = res * res;
        }
        __syncthreads();
        for (int i = tid; i < kMlpWidth + 2; i += blockDim.x) {
            float t = 0.f;
            for (int w = 0; w < kHeadRowsPerCta; ++w) t += wacc[w][i];
            a.part[(static_cast<long long>(blockIdx.x) * kHeadGroups + gr) * (kMlpWidth + 2) + i] = t;
        }
        __syncthreads();
    }
    // column c = tid of the tile's rows, 16 bytes (8 rows) a store
    for (int c = tid; c < kMlpWidth; c += blockDim.x) {
        bf16* o = a.dzT + static_cast<long long>(c) * a.rows_pad + blockIdx.x * kRows;
#pragma unroll
        for (int k = 0; k < kRows; k += 8) {
            __align__(16) bf16 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = dzs[k + j][c];
            *reinterpret_cast<uint4*>(o + k) = *reinterpret_cast<uint4*>(v);
        }
    }
}

// Output layer's gradient and the loss: the groups' partial sums added in group order (one chain per
// column), 32 columns a CTA. Eight warps copy the next 128 groups into shared memory while the first
// adds the present ones (one thread per column with a global load per addition took 143 us at 2,048 groups).
constexpr int kSumRows = 128;
__global__ void __launch_bounds__(256) k_mlp_head_sums(const float* part, int groups, float* grad, float* loss) {
    constexpr int kCols = kMlpWidth + 2;
    __shared__ float buf[2][kSumRows][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col = blockIdx.x * 32 + lane;
    float v[kSumRows / 8];
    auto fetch = [&](int g0) {
#pragma unroll
        for (int q = 0; q < kSumRows / 8; ++q) {
            const int g = g0 + warp + 8 * q;
            v[q] = g < groups && col < kCols ? part[static_cast<long long>(g) * kCols + col] : 0.f;
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int q = 0; q < kSumRows / 8; ++q) buf[b][warp + 8 * q][lane] = v[q];
    };
    fetch(0);
    put(0);
    __syncthreads();
    float t = 0.f;
    int b = 0;
    for (int g0 = 0; g0 < groups; g0 += kSumRows, b ^= 1) {
        fetch(g0 + kSumRows);
        if (warp == 0) {
            const int n = min(kSumRows, groups - g0);
#pragma unroll 16
            for (int q = 0; q < n; ++q) t += buf[b][q][lane];
        }
        put(b ^ 1);
        __syncthreads();
    }
    if (warp == 0) {
        if (col <= kMlpWidth) grad[col] = t;
        else if (col == kMlpWidth + 1) *loss = t;
    }
}

// Inputs in BF16, zero-padded, row-major and transposed: 64 rows a CTA, turned in shared memory (a thread
// per element with 2-byte stores took 12 us at 16,384 rows).
constexpr int kPackRows = 64;
__global__ void __launch_bounds__(256) k_mlp_pack(const float* x, int rows, int n_in, int rows_pad, bf16* X, bf16* XT) {
    static_assert(256 % kMlpInPad == 0 && 256 / kMlpInPad == 4, "four rows a pass");
    __shared__ __align__(16) bf16 t[kPackRows][kMlpInPad + 8];
    const int r0 = blockIdx.x * kPackRows, tid = threadIdx.x;
    const int c0 = tid % kMlpInPad;
    float v[kPackRows / 4];
#pragma unroll
    for (int k = 0; k < kPackRows / 4; ++k) {
        const int r = r0 + tid / kMlpInPad + 4 * k;
        v[k] = r < rows && c0 < n_in ? x[static_cast<long long>(r) * n_in + c0] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kPackRows / 4; ++k) t[tid / kMlpInPad + 4 * k][c0] = __float2bfloat16_rn(v[k]);
    __syncthreads();
    for (int i = tid; i < kPackRows * kMlpInPad / 8; i += 256) {
        const int r = i / (kMlpInPad / 8), c = i % (kMlpInPad / 8) * 8;
        if (X) *reinterpret_cast<uint4*>(X + static_cast<long long>(r0 + r) * kMlpInPad + c) = *reinterpret_cast<const uint4*>(&t[r][c]);
        __align__(16) bf16 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = t[c + j][r];  // here r is a column and c a row
        *reinterpret_cast<uint4*>(XT + static_cast<long long>(r) * rows_pad + r0 + c) = *reinterpret_cast<const uint4*>(w);
    }
}

// Weight gradients from the partial products of `splits` row ranges, added in their order, and the bias
// gradients, the column sums of dZ (kMlpWidth CTAs, the last ones).
__global__ void __launch_bounds__(256) k_mlp_grads(const float* part, int splits, int n, float* gw, const bf16* dzT, int rows_pad,
                                                   float* gb) {
    __shared__ float red[256];
    const int nb = gridDim.x - kMlpWidth;
    float t = 0.f;
    if (static_cast<int>(blockIdx.x) < nb) {
        const int i = blockIdx.x * 256 + threadIdx.x;
        if (i >= n) return;
#pragma unroll 32
        for (int s = 0; s < splits; ++s) t += part[static_cast<long long>(s) * n + i];
        gw[i] = t;
        return;
    }
    const int col = blockIdx.x - nb;
    const bf16* row = dzT + static_cast<long long>(col) * rows_pad;
#pragma unroll 16
    for (int r = threadIdx.x; r < rows_pad; r += 256) t += __bfloat162float(row[r]);
    red[threadIdx.x] = t;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) gb[col] = red[0];
}

// Adam, and the updated weights' BF16 copies (row-major and transposed)
__global__ void k_mlp_adam(AdamArgs a) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= a.n) return;
    float p = a.p[i];
    if (a.g) {
        const float gi = a.g[i];
        const float mi = fmaf(1.f - a.b1, gi, a.b1 * a.m[i]);
        const float vi = fmaf((1.f - a.b2) * gi, gi, a.b2 * a.v[i]);
        a.m[i] = mi;
        a.v[i] = vi;
        p -= a.lr_t * mi / (sqrtf(vi) + a.eps);
        a.p[i] = p;
    }
    const bf16 b = __float2bfloat16_rn(p);
#pragma unroll
    for (int l = 0; l < kMlpHidden; ++l) {
        const int in = l == 0 ? kMlpInPad : kMlpWidth;
        const long long k = i - a.off_W[l];
        if (k < 0 || k >= static_cast<long long>(kMlpWidth) * in) continue;
        a.Wb[l][k] = b;
        if (a.WbT[l]) a.WbT[l][k % in * kMlpWidth + k / in] = b;
    }
}

// ---- batch side ------------------------------------------------------------------------
__device__ inline double geometric_aoa(d3 chord, d3 span_rel, d3 u) {
    const d3 v = u - project(u, span_rel);
    return len(v) > kMinPositive ? signed_angle_between(chord, v, normalize(span_rel)) : 0.0;
}

__global__ void k_batch_features(const FeatJob* jobs, int n_jobs, long long rows, float* feat, double* q_out,
                                 double* g0_out, double* tr_out) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= rows) return;
    int lo = 0, hi = n_jobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].row0 <= r) lo = mid;
        else hi = mid - 1;
    }
    const FeatJob& J = jobs[lo];
    const int i = static_cast<int>(r - J.row0);
    const int w = J.wing_of_line[i];
    const int ws = J.wing_start[w], we = J.wing_end[w];
    const d3 fs = J.fs[i];
    const double U = len(fs);
    auto qf = [&](int k) { return 0.5 * J.chord_len[k] * len(J.fs[k]); };
    auto gn = [&](int k) {
        const double qk = qf(k);
        return qk > 0.0 ? -J.gamma[k] / qk : 0.0;
    };
    const double q = 0.5 * J.chord_len[i] * U;
    const double g0 = gn(i);
    const double gl = gn(i > ws ? i - 1 : i), gr = gn(i + 1 < we ? i + 1 : i);
    double gm = 0.0;
    for (int k = ws; k < we; ++k) gm += gn(k);
    gm /= static_cast<double>(we - ws);
    const d3 fs_prev = J.hist > 0 ? J.fs_old[i] : fs;
    const double Up = len(fs_prev);
    const double gold = J.hist > 1 ? J.gamma_old[i] : J.gamma[i];
    const double trend = q > 0.0 ? -(J.gamma[i] - gold) / q : 0.0;
    const d3 span_rel = J.span_e[i] - J.span_s[i];
    const double a_t = geometric_aoa(J.chord[i], span_rel, fs);
    const double a_p = geometric_aoa(J.chord[i], span_rel, fs_prev);
    const int P = we - ws;
    const double sp = P > 1 ? static_cast<double>(i - ws) / static_cast<double>(P - 1) : 0.5;
    const double k = static_cast<double>(J.steps);
    const double Wd = static_cast<double>(J.W > 0 ? J.W : 1);
    float* f = feat + r * kMlpFeatures;
    f[0] = static_cast<float>(g0);
    f[1] = static_cast<float>(gl);
    f[2] = static_cast<float>(gr);
    f[3] = static_cast<float>(gm);
    f[4] = static_cast<float>(10.0 * trend);
    f[5] = static_cast<float>(Up > 0.0 ? 10.0 * (U / Up - 1.0) : 0.0);
    f[6] = static_cast<float>(a_t);
    f[7] = static_cast<float>(10.0 * (a_t - a_p));
    f[8] = static_cast<float>(2.0 * sp - 1.0);
    f[9] = static_cast<float>(J.chord_len[i] / 10.0);
    f[10] = static_cast<float>(J.S > 1 ? static_cast<double>(w) / (J.S - 1) : 0.0);
    f[11] = static_cast<float>(J.S / 6.0);
    f[12] = static_cast<float>(P / 96.0);
    f[13] = static_cast<float>(J.W / 400.0);
    f[14] = static_cast<float>(fmin(k, Wd) / Wd);
    f[15] = static_cast<float>(1.0 / (1.0 + k));
    q_out[r] = q;
    g0_out[r] = g0;
    tr_out[r] = trend;
    // history for the next step (only this thread touches row i of these two arrays)
    J.gamma_old[i] = J.gamma[i];
    J.fs_old[i] = fs;
}

__global__ void k_batch_candidate(const float* y, const double* q, const double* g0, const double* tr, long long rows,
                                  double* cand_ex, double* cand_net) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= rows) return;
    const double e = g0[r] + tr[r];
    cand_ex[r] = -e * q[r];
    cand_net[r] = -(e + static_cast<double>(y[r])) * q[r];
}

__global__ void k_batch_targets(const double* gamma_new, const double* q, const double* g0, const double* tr,
                                long long rows, float* t) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= rows) return;
    t[r] = q[r] > 0.0 ? static_cast<float>(-gamma_new[r] / q[r] - g0[r] - tr[r]) : 0.f;
}

unsigned blocks_for(long long n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

size_t mlp_gemm_smem_bytes() { return kStages * static_cast<size_t>(kStage) + 1024; }

cudaError_t configure_mlp_gemm() {
    for (auto kernel : {k_mlp_forward<false>, k_mlp_forward<true>}) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kFwdSmem));
        if (e != cudaSuccess) return e;
    }
    return cudaFuncSetAttribute(k_mlp_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(mlp_gemm_smem_bytes()));
}

namespace {

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to the driver
// library); null when the driver does not provide it.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// Row-major BF16 matrix [rows][cols] with leading dimension ld, copied in boxes of 64
// columns x box_rows rows into 128-byte-swizzled shared memory.
bool encode_bf16_map(CUtensorMap* map, const bf16* ptr, long long rows, long long cols, long long ld, int box_rows) {
    const auto encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * sizeof(bf16)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kKStep), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(ptr), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t launch_mlp_gemm(const GemmArgs& g, cudaStream_t s) {
    if (!mlp_gemm_args_ok(g)) return cudaErrorInvalidValue;
    CUtensorMap ma, mb;
    const int splits = (g.K + g.k_split - 1) / g.k_split, tiles = g.M / kMlpRowTile;
    const int z = g.N >= 128 && tiles * splits <= g.sms ? 2 : 1;
    if (!encode_bf16_map(&ma, g.A, g.M, g.K, g.lda, kMlpRowTile) || !encode_bf16_map(&mb, g.B, g.N, g.K, g.ldb, g.N / z))
        return cudaErrorInvalidValue;
    k_mlp_gemm<<<dim3(tiles, splits, z), kGemmThreads, mlp_gemm_smem_bytes(), s>>>(ma, mb, g);
    return cudaGetLastError();
}

cudaError_t launch_mlp_forward(const FwdArgs& args, cudaStream_t s) {
    if (args.rows <= 0) return cudaSuccess;
    FwdArgs g = args;
    g.vec_x = g.n_in % 4 == 0 && reinterpret_cast<uintptr_t>(g.x) % 16 == 0 ? 1 : 0;
    FwdMaps maps;
    for (int l = 0; l < kMlpHidden; ++l) {
        const int in = l == 0 ? kMlpInPad : kMlpWidth;
        if (!encode_bf16_map(&maps.w[l], g.w[l], kMlpWidth, in, in, 128)) return cudaErrorInvalidValue;
    }
    const int tiles = (g.rows + 127) / 128;
    if (g.z[0]) {
        if (tiles > g.sms) return cudaErrorInvalidValue;
        for (int l = 0; l < kMlpHidden; ++l)
            if (!g.z[l] || !g.h[l]) return cudaErrorInvalidValue;
        k_mlp_forward<true><<<tiles, kFwdThreads, kFwdSmem, s>>>(maps, g);
    } else {
        if (!g.y) return cudaErrorInvalidValue;
        k_mlp_forward<false><<<std::min(tiles, std::max(1, g.sms)), kFwdThreads, kFwdSmem, s>>>(maps, g);
    }
    return cudaGetLastError();
}

cudaError_t launch_mlp_head(const HeadArgs& a, cudaStream_t s) {
    constexpr int kRows = kHeadGroups * kHeadRowsPerCta;
    if (a.rows_pad % kRows) return cudaErrorInvalidValue;
    k_mlp_head<<<a.rows_pad / kRows, 32 * kHeadRowsPerCta, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_mlp_pack(const float* x, int rows, int n_in, int rows_pad, bf16* X, bf16* XT, cudaStream_t s) {
    if (rows_pad % kPackRows) return cudaErrorInvalidValue;
    k_mlp_pack<<<rows_pad / kPackRows, 256, 0, s>>>(x, rows, n_in, rows_pad, X, XT);
    return cudaGetLastError();
}

cudaError_t launch_mlp_grads(const float* part, int splits, int n, float* gw, const bf16* dzT, int rows_pad, float* gb, cudaStream_t s) {
    k_mlp_grads<<<(n + 255) / 256 + kMlpWidth, 256, 0, s>>>(part, splits, n, gw, dzT, rows_pad, gb);
    return cudaGetLastError();
}

cudaError_t launch_mlp_head_sums(const float* part, int groups, float* grad, float* loss, cudaStream_t s) {
    k_mlp_head_sums<<<(kMlpWidth + 2 + 31) / 32, 256, 0, s>>>(part, groups, grad, loss);
    return cudaGetLastError();
}

cudaError_t launch_mlp_adam(const AdamArgs& a, cudaStream_t s) {
    k_mlp_adam<<<blocks_for(a.n, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_batch_features(const FeatJob* jobs, int n_jobs, long long rows, float* feat, double* q, double* g0,
                                  double* tr, cudaStream_t s) {
    if (rows <= 0 || n_jobs <= 0) return cudaSuccess;
    k_batch_features<<<blocks_for(rows, 128), 128, 0, s>>>(jobs, n_jobs, rows, feat, q, g0, tr);
    return cudaGetLastError();
}

cudaError_t launch_batch_candidate(const float* y, const double* q, const double* g0, const double* tr, long long rows,
                                   double* cand_ex, double* cand_net, cudaStream_t s) {
    if (rows <= 0) return cudaSuccess;
    k_batch_candidate<<<blocks_for(rows, 256), 256, 0, s>>>(y, q, g0, tr, rows, cand_ex, cand_net);
    return cudaGetLastError();
}

cudaError_t launch_batch_targets(const double* gamma_new, const double* q, const double* g0, const double* tr,
                                 long long rows, float* target, cudaStream_t s) {
    if (rows <= 0) return cudaSuccess;
    k_batch_targets<<<blocks_for(rows, 256), 256, 0, s>>>(gamma_new, q, g0, tr, rows, target);
    return cudaGetLastError();
}

}  // namespace sbgpu
