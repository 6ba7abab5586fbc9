// Warm-start network: host side and the sb_mlp_* C ABI.
//
// A multilayer perceptron with kMlpHidden hidden layers of width kMlpWidth (GELU) and one
// output, trained by mean-squared error with Adam. Parameters are kept in FP32 (the master
// copy the optimizer updates) and cast to BF16 for the tensor-core GEMMs after every update
// (row-major W for the forward pass, W^T for the input gradients). Activations are BF16;
// every GEMM accumulates in FP32. The flat parameter order is
//   W1 [256][64] (input columns >= n_in stay zero), b1 [256],
//   W2 [256][256], b2, W3, b3, W4, b4, w_out [256], b_out [1].
// Every reduction (split-K weight gradients, bias sums, output-layer partials) runs in a
// fixed order, so a training step is deterministic.
#include <cmath>
#include <cstring>
#include <vector>

#include "sb_mlp.h"
#include "sim_core.hpp"

using namespace sbgpu;

struct sb_mlp {
    int device = 0;
    int n_in = 0;
    cudaStream_t stream = nullptr;
    // Beside the chain of input gradients: weight and bias gradients; the output layer's.
    cudaStream_t side[2] = {nullptr, nullptr};
    cudaEvent_t ev_dz[kMlpHidden] = {nullptr}, ev_side[2] = {nullptr, nullptr}, ev_in = nullptr;
    long long off_W[kMlpHidden] = {0}, off_b[kMlpHidden] = {0}, off_out = 0, n_params = 0;
    int in_dim[kMlpHidden] = {0};
    DevBuf<float> params, grads, adam_m, adam_v;
    DevBuf<bf16> Wb[kMlpHidden], WbT[kMlpHidden];
    int cap = 0;   // rows the training buffers hold (multiple of 128)
    int sms = 1;
    DevBuf<bf16> X0, X0T, H[kMlpHidden], HT[kMlpHidden], DZ[kMlpHidden], DZT[kMlpHidden];
    DevBuf<float> Z[kMlpHidden], part, head_part, loss;
    DevBuf<int> err;
    PinnedBuf<float> h_loss;
    PinnedBuf<int> h_err;
    int adam_step = 0;
    int splits = 1;

    ~sb_mlp() {
        for (auto& e : ev_dz) if (e) cudaEventDestroy(e);
        for (auto& e : ev_side) if (e) cudaEventDestroy(e);
        if (ev_in) cudaEventDestroy(ev_in);
        for (auto& q : side) if (q) cudaStreamDestroy(q);
        if (stream) cudaStreamDestroy(stream);
    }

    void build(int dev, int n_inputs, unsigned long long seed) {
        if (n_inputs < 1 || n_inputs > kMlpInPad) raise(SB_ERR_SIZE, "the network takes 1 to 64 inputs");
        device = dev;
        n_in = n_inputs;
        ck(cudaSetDevice(device), "cudaSetDevice");
        sms = num_sms(device);
        ck(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        for (auto& q : side) ck(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking), "cudaStreamCreate");
        for (auto& e : ev_dz) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
        for (auto& e : ev_side) ck(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
        ck(cudaEventCreateWithFlags(&ev_in, cudaEventDisableTiming), "cudaEventCreate");
        long long at = 0;
        for (int l = 0; l < kMlpHidden; ++l) {
            in_dim[l] = l == 0 ? kMlpInPad : kMlpWidth;
            off_W[l] = at;
            at += static_cast<long long>(kMlpWidth) * in_dim[l];
            off_b[l] = at;
            at += kMlpWidth;
        }
        off_out = at;
        at += kMlpWidth + 1;
        n_params = at;
        // He-uniform initialisation from a seeded splitmix64 stream, biases zero
        std::vector<float> p(static_cast<size_t>(n_params), 0.f);
        unsigned long long s = seed;
        auto next = [&]() {
            s += 0x9E3779B97F4A7C15ull;
            unsigned long long z = s;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            z ^= z >> 31;
            return static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0);
        };
        for (int l = 0; l < kMlpHidden; ++l) {
            const int fan_in = l == 0 ? n_in : kMlpWidth;
            const double a = std::sqrt(6.0 / fan_in);
            for (int o = 0; o < kMlpWidth; ++o)
                for (int i = 0; i < in_dim[l]; ++i) {
                    const double u = next();
                    if (l == 0 && i >= n_in) continue;
                    p[static_cast<size_t>(off_W[l] + static_cast<long long>(o) * in_dim[l] + i)] =
                        static_cast<float>((2.0 * u - 1.0) * a);
                }
        }
        const double ao = std::sqrt(3.0 / kMlpWidth);
        for (int i = 0; i < kMlpWidth; ++i) p[static_cast<size_t>(off_out + i)] = static_cast<float>((2.0 * next() - 1.0) * ao);
        params.upload(p);
        grads.alloc(n_params);
        adam_m.alloc(n_params);
        adam_v.alloc(n_params);
        ck(cudaMemsetAsync(grads.p, 0, n_params * sizeof(float), stream), "memset");
        ck(cudaMemsetAsync(adam_m.p, 0, n_params * sizeof(float), stream), "memset");
        ck(cudaMemsetAsync(adam_v.p, 0, n_params * sizeof(float), stream), "memset");
        for (int l = 0; l < kMlpHidden; ++l) {
            Wb[l].alloc(static_cast<size_t>(kMlpWidth) * in_dim[l]);
            if (l > 0) WbT[l].alloc(static_cast<size_t>(kMlpWidth) * in_dim[l]);
        }
        loss.alloc(1);
        err.alloc(1);
        ck(cudaMemsetAsync(err.p, 0, sizeof(int), stream), "memset");
        h_loss.alloc(1);
        h_err.alloc(1);
        ck(configure_mlp_gemm(), "GEMM shared-memory limit");
        cast_weights(stream);
        ck(cudaStreamSynchronize(stream), "mlp build");
    }

    AdamArgs adam_args() const {
        AdamArgs a;
        a.p = params.p;
        a.n = n_params;
        for (int l = 0; l < kMlpHidden; ++l) {
            a.off_W[l] = off_W[l];
            a.Wb[l] = Wb[l].p;
            a.WbT[l] = l > 0 ? WbT[l].p : nullptr;
        }
        return a;
    }
    void cast_weights(cudaStream_t s) { ck(launch_mlp_adam(adam_args(), s), "weight cast"); }

    static int pad_rows(long long rows) {
        return static_cast<int>(((rows + kMlpRowTile - 1) / kMlpRowTile) * kMlpRowTile);
    }

    // Buffers of a training step of `rows` rows (inference keeps its activations on the SMs).
    void ensure(long long rows) {
        const int need = pad_rows(std::max<long long>(rows, 1));
        if (need <= cap) return;
        cap = 0;  // until all of them are there
        const size_t w = static_cast<size_t>(need) * kMlpWidth;
        X0.alloc(static_cast<size_t>(need) * kMlpInPad);
        X0T.alloc(static_cast<size_t>(need) * kMlpInPad);
        for (int l = 0; l < kMlpHidden; ++l) {
            H[l].alloc(w);
            Z[l].alloc(w);
            HT[l].alloc(w);
            DZ[l].alloc(w);
            DZT[l].alloc(w);
        }
        head_part.alloc(static_cast<size_t>(need / kHeadRowsPerCta) * (kMlpWidth + 2));
        // split-K over the batch rows for the weight gradients: about one wave of CTAs
        splits = std::max(1, std::min(need / 64, 76));
        part.alloc(static_cast<size_t>(splits) * kMlpWidth * kMlpWidth);
        cap = need;
    }

    GemmArgs gemm(const bf16* A, long long lda, const bf16* B, long long ldb, int M, int N, int K, int mode) const {
        GemmArgs g;
        g.A = A;
        g.lda = lda;
        g.B = B;
        g.ldb = ldb;
        g.M = M;
        g.N = N;
        g.K = K;
        g.k_split = K;
        g.mode = mode;
        g.sms = sms;
        g.err = err.p;
        return g;
    }

    FwdArgs fwd_args() const {
        FwdArgs g;
        g.n_in = n_in;
        for (int l = 0; l < kMlpHidden; ++l) {
            g.w[l] = Wb[l].p;
            g.bias[l] = params.p + off_b[l];
        }
        g.w_out = params.p + off_out;
        g.sms = sms;
        g.err = err.p;
        return g;
    }

    // Inference over rows of x [rows][n_in] (device) into y [rows].
    void forward(const float* x, long long rows, float* y, cudaStream_t s) {
        FwdArgs g = fwd_args();
        constexpr long long kPass = 1 << 30;  // rows per launch (row numbers of a launch are int)
        for (long long r0 = 0; r0 < rows; r0 += kPass) {
            g.x = x + r0 * n_in;
            g.y = y + r0;
            g.rows = static_cast<int>(std::min(kPass, rows - r0));
            ck(launch_mlp_forward(g, s), "network");
        }
    }

    // Forward pass of a training step: keeps what the backward pass needs. Up to a tile of 128 rows per SM
    // the hidden layers are one launch, and the packed inputs (for the first layer's weight gradients alone) are
    // made beside it.
    void forward_train(const float* x, long long rows, const float* target, cudaStream_t s) {
        const int R = pad_rows(rows);
        if (R / kMlpRowTile <= sms) {
            ck(cudaEventRecord(ev_in, s), "event");
            ck(cudaStreamWaitEvent(side[0], ev_in, 0), "side stream");
            ck(launch_mlp_pack(x, static_cast<int>(rows), n_in, R, nullptr, X0T.p, side[0]), "pack inputs");
            FwdArgs g = fwd_args();
            g.x = x;
            g.rows = static_cast<int>(rows);
            g.ldt = R;
            for (int l = 0; l < kMlpHidden; ++l) {
                g.z[l] = Z[l].p;
                g.h[l] = H[l].p;
                g.hT[l] = l + 1 < kMlpHidden ? HT[l].p : nullptr;
            }
            ck(launch_mlp_forward(g, s), "hidden layers");
        } else {
            ck(launch_mlp_pack(x, static_cast<int>(rows), n_in, R, X0.p, X0T.p, s), "pack inputs");
            const bf16* in = X0.p;
            long long ld = kMlpInPad;
            for (int l = 0; l < kMlpHidden; ++l) {
                GemmArgs g = gemm(in, ld, Wb[l].p, in_dim[l], R, kMlpWidth, in_dim[l], kGemmForward);
                g.bias = params.p + off_b[l];
                g.z_out = Z[l].p;
                g.h_out = H[l].p;
                g.hT_out = l + 1 < kMlpHidden ? HT[l].p : nullptr;
                g.ldt = R;
                ck(launch_mlp_gemm(g, s), "forward GEMM");
                in = H[l].p;
                ld = kMlpWidth;
            }
        }
        HeadArgs h;
        h.h = H[kMlpHidden - 1].p;
        h.z = Z[kMlpHidden - 1].p;
        h.w = params.p + off_out;
        h.target = target;
        h.rows = static_cast<int>(rows);
        h.rows_pad = R;
        h.dz = DZ[kMlpHidden - 1].p;
        h.dzT = DZT[kMlpHidden - 1].p;
        h.part = head_part.p;
        h.inv_n = 1.f / static_cast<float>(std::max<long long>(rows, 1));
        ck(launch_mlp_head(h, s), "output layer");
    }

    // Gradients of the mean squared error into `grads` (after a training forward pass).
    void backward(long long rows, cudaStream_t s) {
        const int R = pad_rows(rows);
        const int nh = R / kHeadRowsPerCta;
        // Weight and bias gradients of layer l need dZ_l alone: they run on a side stream while the
        // main one goes on with dZ_{l-1}. (They share `part`, one after the other.)
        ck(cudaEventRecord(ev_dz[kMlpHidden - 1], s), "event");
        ck(cudaStreamWaitEvent(side[1], ev_dz[kMlpHidden - 1], 0), "side stream");
        // output layer: dw_out, db_out and the loss from the groups' partials
        ck(launch_mlp_head_sums(head_part.p, nh, grads.p + off_out, loss.p, side[1]), "head gradient");
        for (int l = kMlpHidden - 1; l >= 0; --l) {
            if (l > 0) {
                // dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1})
                GemmArgs b = gemm(DZ[l].p, kMlpWidth, WbT[l].p, kMlpWidth, R, kMlpWidth, kMlpWidth, kGemmBackward);
                b.z_in = Z[l - 1].p;
                b.h_out = DZ[l - 1].p;
                b.hT_out = DZT[l - 1].p;
                b.ldt = R;
                ck(launch_mlp_gemm(b, s), "input-gradient GEMM");
                ck(cudaEventRecord(ev_dz[l - 1], s), "event");
            }
            // dW_l = dZ_l^T X_{l-1}: M = 256 outputs, N = inputs, K = rows (split)
            const bf16* XT = l == 0 ? X0T.p : HT[l - 1].p;
            GemmArgs g = gemm(DZT[l].p, R, XT, R, kMlpWidth, in_dim[l], R, kGemmPartial);
            int ks = ((R / splits + 63) / 64) * 64;
            if (ks < 64) ks = 64;
            g.k_split = ks;
            g.part_out = part.p;
            ck(cudaStreamWaitEvent(side[0], ev_dz[l], 0), "side stream");
            ck(launch_mlp_gemm(g, side[0]), "weight-gradient GEMM");
            ck(launch_mlp_grads(part.p, (R + ks - 1) / ks, kMlpWidth * in_dim[l], grads.p + off_W[l], DZT[l].p, R, grads.p + off_b[l],
                                side[0]),
               "weight-gradient sums");
        }
        for (int q = 0; q < 2; ++q) {
            ck(cudaEventRecord(ev_side[q], side[q]), "event");
            ck(cudaStreamWaitEvent(s, ev_side[q], 0), "side stream");
        }
    }

    void check_err(cudaStream_t s) {
        ck(cudaMemcpyAsync(h_err.p, err.p, sizeof(int), cudaMemcpyDeviceToHost, s), "D2H status");
        ck(cudaStreamSynchronize(s), "mlp");
        if (h_err.p[0] != kDevOk) {
            ck(cudaMemsetAsync(err.p, 0, sizeof(int), s), "memset");
            raise(SB_ERR_TIMEOUT, "a bounded device-side wait ran out in the network kernels");
        }
    }

    double read_loss(cudaStream_t s) {
        ck(cudaMemcpyAsync(h_loss.p, loss.p, sizeof(float), cudaMemcpyDeviceToHost, s), "D2H loss");
        check_err(s);
        return static_cast<double>(h_loss.p[0]);
    }

    void adam(float lr, cudaStream_t s) {
        adam_step += 1;
        const double b1 = 0.9, b2 = 0.999;
        const double lr_t = lr * std::sqrt(1.0 - std::pow(b2, adam_step)) / (1.0 - std::pow(b1, adam_step));
        AdamArgs a = adam_args();
        a.g = grads.p;
        a.m = adam_m.p;
        a.v = adam_v.p;
        a.lr_t = static_cast<float>(lr_t);
        a.b1 = static_cast<float>(b1);
        a.b2 = static_cast<float>(b2);
        a.eps = 1e-8f;
        ck(launch_mlp_adam(a, s), "adam");
    }
};

namespace sbhost {
int mlp_inputs(const sb_mlp* m) { return m->n_in; }
void mlp_forward_async(sb_mlp* m, const float* x, long long rows, float* y, cudaStream_t s) {
    m->forward(x, rows, y, s);
}
void mlp_check(sb_mlp* m) {
    ck(cudaDeviceSynchronize(), "network");
    m->check_err(m->stream);
}
}  // namespace sbhost

namespace {
int null_arg() {
    report_error(SB_ERR_NULL_ARG, "null argument");
    return SB_ERR_NULL_ARG;
}
}  // namespace

extern "C" {

sb_mlp* sb_mlp_new(int device, int n_inputs, unsigned long long seed) {
    std::unique_ptr<sb_mlp> m(new sb_mlp());
    if (guard([&] { m->build(device, n_inputs, seed); }) != SB_OK) return nullptr;
    return m.release();
}

void sb_mlp_free(sb_mlp* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    delete m;
}

int sb_mlp_num_params(const sb_mlp* m, size_t* n) {
    if (!m || !n) return null_arg();
    *n = static_cast<size_t>(m->n_params);
    return SB_OK;
}

int sb_mlp_get_params(sb_mlp* m, float* p, size_t n) {
    if (!m || !p) return null_arg();
    return guard([&] {
        if (static_cast<long long>(n) != m->n_params) raise(SB_ERR_SIZE, "parameter count mismatch");
        ck(cudaMemcpyAsync(p, m->params.p, n * sizeof(float), cudaMemcpyDeviceToHost, m->stream), "D2H");
        ck(cudaStreamSynchronize(m->stream), "sync");
    });
}

int sb_mlp_set_params(sb_mlp* m, const float* p, size_t n) {
    if (!m || !p) return null_arg();
    return guard([&] {
        if (static_cast<long long>(n) != m->n_params) raise(SB_ERR_SIZE, "parameter count mismatch");
        ck(cudaMemcpyAsync(m->params.p, p, n * sizeof(float), cudaMemcpyHostToDevice, m->stream), "H2D");
        m->cast_weights(m->stream);
        ck(cudaStreamSynchronize(m->stream), "sync");
    });
}

int sb_mlp_forward(sb_mlp* m, const float* x_dev, size_t rows, float* y_dev) {
    if (!m || (rows && (!x_dev || !y_dev))) return null_arg();
    if (rows == 0) return SB_OK;
    return guard([&] {
        order_after_caller(m->stream);
        m->forward(x_dev, static_cast<long long>(rows), y_dev, m->stream);
        m->check_err(m->stream);
    });
}

int sb_mlp_gradients(sb_mlp* m, const float* x_dev, const float* target_dev, size_t rows, float* grads_host,
                     double* loss) {
    if (!m || !x_dev || !target_dev || !grads_host) return null_arg();
    if (rows == 0) {
        report_error(SB_ERR_SIZE, "no rows");
        return SB_ERR_SIZE;
    }
    return guard([&] {
        m->ensure(static_cast<long long>(rows));
        order_after_caller(m->stream);
        m->forward_train(x_dev, static_cast<long long>(rows), target_dev, m->stream);
        m->backward(static_cast<long long>(rows), m->stream);
        ck(cudaMemcpyAsync(grads_host, m->grads.p, m->n_params * sizeof(float), cudaMemcpyDeviceToHost, m->stream),
           "D2H gradients");
        const double l = m->read_loss(m->stream);
        if (loss) *loss = l / static_cast<double>(rows);
    });
}

int sb_mlp_train_step(sb_mlp* m, const float* x_dev, const float* target_dev, size_t rows, float learning_rate,
                      double* loss) {
    if (!m || !x_dev || !target_dev) return null_arg();
    if (rows == 0) {
        report_error(SB_ERR_SIZE, "no rows");
        return SB_ERR_SIZE;
    }
    return guard([&] {
        m->ensure(static_cast<long long>(rows));
        order_after_caller(m->stream);
        m->forward_train(x_dev, static_cast<long long>(rows), target_dev, m->stream);
        m->backward(static_cast<long long>(rows), m->stream);
        m->adam(learning_rate, m->stream);
        // the inputs are read by the time the call returns (the caller may reuse them)
        if (loss) *loss = m->read_loss(m->stream) / static_cast<double>(rows);
        else m->check_err(m->stream);
    });
}

}  // extern "C"
