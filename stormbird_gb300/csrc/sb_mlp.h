// Kernels of the warm-start network (k_mlp.cu): a multilayer perceptron with BF16
// weights and activations on the tensor cores (tcgen05, FP32 accumulation in tensor
// memory), its training kernels, and the batch-side feature and candidate kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "sb_device.cuh"

namespace sbgpu {

constexpr int kMlpWidth = 256;     // hidden width
constexpr int kMlpHidden = 4;      // hidden layers
constexpr int kMlpInPad = 64;      // input features padded to one K tile
constexpr int kMlpRowTile = 128;   // rows per GEMM tile (tcgen05 M)
constexpr int kMlpFeatures = 16;   // features per panel built by the batch

using bf16 = __nv_bfloat16;

// C[M][N] = A[M][K] * B[N][K]^T with A and B row-major BF16 (K contiguous), FP32 accumulate.
// M a multiple of 128, N in {64, 128, 256}, K a multiple of 64 (split over gridDim.y in
// chunks of k_split).
enum GemmMode : int {
    kGemmForward = 0,   // z = acc + bias; h = gelu(z) -> h_out (row-major), hT_out (transposed)
    kGemmBackward = 1,  // dz = acc * gelu'(z_in) -> h_out (row-major), hT_out (transposed)
    kGemmPartial = 2,   // part_out[split][M][N] = acc
};
struct GemmArgs {
    const bf16* A = nullptr;
    long long lda = 0;
    const bf16* B = nullptr;
    long long ldb = 0;
    int M = 0, N = 0, K = 0, k_split = 0;
    int mode = 0;
    const float* bias = nullptr;
    float* z_out = nullptr;   // [M][N] (forward)
    bf16* h_out = nullptr;    // [M][N] (forward, backward)
    bf16* hT_out = nullptr;   // [N][ldt] or nullptr (forward, backward)
    long long ldt = 0;
    const float* z_in = nullptr;  // [M][N] (backward)
    float* part_out = nullptr;    // partial
    int sms = 1;
    int* err = nullptr;
};
// Shapes the kernel takes (TMA: 16-byte aligned bases and row strides; every box lies inside its matrix) and
// every array that its mode reads or writes.
inline bool mlp_gemm_args_ok(const GemmArgs& g) {
    if (g.M <= 0 || g.M % kMlpRowTile || g.K <= 0 || g.K % 64 || g.k_split <= 0 || g.k_split % 64 ||
        (g.N != 64 && g.N != 128 && g.N != 256) || g.lda % 8 || g.ldb % 8 || g.lda < g.K || g.ldb < g.K || !g.A || !g.B ||
        reinterpret_cast<uintptr_t>(g.A) % 16 || reinterpret_cast<uintptr_t>(g.B) % 16)
        return false;
    if (g.mode == kGemmPartial) return g.part_out != nullptr;
    if (!g.h_out || (g.hT_out && g.ldt < g.M)) return false;
    return g.mode == kGemmForward ? g.bias && g.z_out : g.mode == kGemmBackward && g.z_in;
}
size_t mlp_gemm_smem_bytes();
// Raises the GEMM kernel's dynamic shared-memory limit (once, before any stream capture).
cudaError_t configure_mlp_gemm();
cudaError_t launch_mlp_gemm(const GemmArgs& g, cudaStream_t s);

// Inference: y[r] = the network at row r of x [rows][n_in] (k_mlp_forward).
struct FwdArgs {
    const float* x = nullptr;
    int rows = 0, n_in = 0, vec_x = 0;        // vec_x: set by the launch
    const bf16* w[kMlpHidden] = {nullptr};    // [256][64], then [256][256]
    const float* bias[kMlpHidden] = {nullptr};
    const float* w_out = nullptr;             // [257]
    float* y = nullptr;
    // training (z[0] not null; at most sms tiles of 128 rows): pre-activations [rows_pad][256], activations
    // [rows_pad][256] and their transposes [256][ldt] (these null: not wanted) of every layer instead of y
    float* z[kMlpHidden] = {nullptr};
    bf16* h[kMlpHidden] = {nullptr};
    bf16* hT[kMlpHidden] = {nullptr};
    long long ldt = 0;
    int sms = 1;
    int* err = nullptr;
};
cudaError_t launch_mlp_forward(const FwdArgs& g, cudaStream_t s);

// Output layer (width -> 1) of a training pass on the CUDA cores: MSE residuals, dz of the last hidden layer (row-major and
// transposed) and partials [rows_pad / kHeadRowsPerCta][width + 2] of (dw, db, sum of squared residuals).
struct HeadArgs {
    const bf16* h = nullptr;
    const float* z = nullptr;
    const float* w = nullptr;   // [width + 1]
    const float* target = nullptr;
    int rows = 0, rows_pad = 0;
    bf16* dz = nullptr;
    bf16* dzT = nullptr;
    float* part = nullptr;
    float inv_n = 0.f;
};
constexpr int kHeadRowsPerCta = 8;  // rows of a partial sum
constexpr int kHeadGroups = 4;      // partial sums a CTA makes
// The partials added up: grad [width + 1] and the sum of squared residuals.
cudaError_t launch_mlp_head_sums(const float* part, int groups, float* grad, float* loss, cudaStream_t s);
cudaError_t launch_mlp_head(const HeadArgs& a, cudaStream_t s);

// Input packing: x [rows][n_in] f32 -> X [rows_pad][64] BF16 (zero padded; null: not wanted) and its transpose XT
// [64][rows_pad].
cudaError_t launch_mlp_pack(const float* x, int rows, int n_in, int rows_pad, bf16* X, bf16* XT, cudaStream_t s);
// gw[i] = sum over s < splits of part[s * n + i] in split order; gb[o] = sum over r < rows_pad of dzT[o][r].
cudaError_t launch_mlp_grads(const float* part, int splits, int n, float* gw, const bf16* dzT, int rows_pad, float* gb, cudaStream_t s);
// Adam update of n parameters (bias-corrected step sizes precomputed on the host) and the BF16 copies of
// the weights [out][in] at off_W[l], row-major (Wb) and, when WbT is not null, transposed; g null:
// the copies alone.
struct AdamArgs {
    float* p = nullptr;
    const float* g = nullptr;
    float* m = nullptr;
    float* v = nullptr;
    long long n = 0;
    float lr_t = 0.f, b1 = 0.f, b2 = 0.f, eps = 0.f;
    long long off_W[kMlpHidden] = {0};
    bf16* Wb[kMlpHidden] = {nullptr};
    bf16* WbT[kMlpHidden] = {nullptr};
};
cudaError_t launch_mlp_adam(const AdamArgs& a, cudaStream_t s);

// ---- batch side ----------------------------------------------------------------------
// One case of a batch, for the per-panel features of the warm start.
struct FeatJob {
    const d3* fs = nullptr;          // [N] freestream at the control points, this step
    const double* gamma = nullptr;   // [N] previous solution
    double* gamma_old = nullptr;     // [N] solution of the step before (updated in place)
    d3* fs_old = nullptr;            // [N] freestream of the previous step (updated in place)
    const d3* chord = nullptr;       // [N] global chord vectors
    const d3* span_s = nullptr;
    const d3* span_e = nullptr;
    const double* chord_len = nullptr;
    const int* wing_of_line = nullptr;
    const int* wing_start = nullptr;
    const int* wing_end = nullptr;
    int N = 0, S = 0, W = 0, steps = 0;
    int hist = 0;                    // steps whose history this job's arrays hold (0, 1 or 2):
                                     // fs_old is read from 1, gamma_old from 2
    long long row0 = 0;              // first row of the case in the batch arrays
};
// Per panel, with q = chord |U| / 2 and the lift-coefficient-like variable g = -Gamma / q:
// feat [rows][kMlpFeatures], q, g0 = g of the previous solution and tr = its change over
// the previous step (zero before two solutions exist), the linear-extrapolation baseline.
cudaError_t launch_batch_features(const FeatJob* jobs, int n_jobs, long long rows, float* feat, double* q, double* g0,
                                  double* tr, cudaStream_t s);
// cand_ex = -(g0 + tr) q: extrapolation in time; cand_net = -(g0 + tr + y) q: plus the
// network's correction y
cudaError_t launch_batch_candidate(const float* y, const double* q, const double* g0, const double* tr, long long rows,
                                   double* cand_ex, double* cand_net, cudaStream_t s);
// target = -gamma_new / q - g0 - tr: the correction the network is trained to predict
cudaError_t launch_batch_targets(const double* gamma_new, const double* q, const double* g0, const double* tr,
                                 long long rows, float* target, cudaStream_t s);

}  // namespace sbgpu

// The network as the batch uses it (mlp_host.cu).
struct sb_mlp;
namespace sbhost {
int mlp_inputs(const sb_mlp* m);
// y [rows] = network(x [rows][inputs]) enqueued on s (no synchronisation).
void mlp_forward_async(sb_mlp* m, const float* x, long long rows, float* y, cudaStream_t s);
// Throws when a bounded wait in the network's kernels ran out (synchronises the device).
void mlp_check(sb_mlp* m);
}  // namespace sbhost
