// Linearized solver (sm_103a): Linearized::solve (stormbird/src/lifting_line/solvers/linearized.rs:
// 54-222) by an FP32 inverse and f64 refinement, on one thread-block cluster per case.
//
// The reference eliminates the N x N system in f64 (stormath/src/matrix/linalg.rs:41-103). This part's
// FP64 rate is 1/64 of its FP32 rate and a pivoted elimination takes a cluster barrier per column, so
// here:
//   1. each CTA builds its rows of the matrix in f64 (kept in global memory) and their FP32 copy in
//      shared memory (linearized.rs:61-136);
//   2. the FP32 copy is inverted in place by block Gauss-Jordan, blocks of 16 rows dealt round-robin:
//      the owner of block k inverts its diagonal block, scales its 16 rows and leaves them in
//      global memory, one cluster barrier, every CTA subtracts their multiples from its rows (a rank-16
//      update from shared memory). N / 16 barriers instead of N; the owner of block k + 1 updates those
//      rows first and publishes them before the rest of its rows, beside the others' updates;
//   3. x = x + X32 (b - A x) with the residual in f64 until the correction is rounding (two or three
//      digits short of full precision are left after the first, each further one gains as many as
//      the FP32 inverse is good for);
//   4. induced velocities, viscous correction, residual and outputs (linearized.rs:141-213), each CTA
//      its rows.
// Up to 768 lines: the whole FP32 copy has to fit the shared memory of 16 CTAs (linearized_refined_plan). Beyond,
// the elimination alone solves the case (768 lines 0.47 ms, 769 lines 114 ms).
// Steps 1 and 4 are FP64 work of N^2 entries. One large case alone has them done by all SMs before and after
// the cluster (k_lin_build, k_lin_finish; kSplitLines).
// No pivoting across blocks: the diagonal dominates (2 / (c u) plus the line's own trailing pair
// against its neighbours'), and a system where that fails shows in step 3. Where a pivot is below
// 1e-6 (the reference calls 1e-12 singular), a correction does not shrink or a value is not finite,
// scalars[5] stays 0 and the elimination kernels of k_solve.cu, launched after this one, solve the case
// as before (they return at once where scalars[5] is 1).
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "sb_device.cuh"
#include "sb_kernels.h"
#include "sb_lin_layout.h"
#include "sb_line.cuh"

namespace cg = cooperative_groups;

namespace sbgpu {

namespace {

constexpr int kThreads = 512;
constexpr int kMaxRefine = 20;

// velocity_corrections.rs:28-100 (returns freestream + induced, corrected)
__device__ __noinline__ d3 corrected_velocity(const SolveSettings& st, d3 fs, d3 ind) {
    if (st.velocity_correction == 1) {
        const double im = len(ind), mx = st.velocity_correction_ratio * len(fs);
        return fs + (im > mx ? normalize(ind) * mx : ind);
    }
    return normalize(fs + ind) * len(fs);
}

// |cl of the force - cl of the foil| (force_calculations.rs:552-607)
__device__ __forceinline__ double residual_of(const DevModel& m, int i, double gam, d3 u, double cl_pre) {
    const double area = m.chord_len[i] * m.span_len_local[i], q = len2(u);
    const double ff = 0.5 * area * m.density * q;
    const d3 s = m.output_body ? m.span_e_local[i] - m.span_s_local[i] : m.span_e[i] - m.span_s[i];
    double clg = 0.0;
    if (ff != 0.0) {
        const double force = q == 0.0 ? 0.0 : sqrt_any(len2(cross(u, s))) * fabs(gam * m.density);
        clg = -signum(gam) * (force * rcp_any(ff));
    }
    return fabs(clg - cl_pre);
}

// lin_work: scaled rows [2][16][n] floats, the f64 matrix [N][N], and for a split solve its FP32 copy [n][n], the
// right-hand side [n], the solution [n], the circulation [n] after the viscous correction, the residual terms [n]
// and a counter.
struct Work {
    float* Pg;
    double* A64;
    float* A32;
    double *rhs, *x, *g, *terms;
    unsigned* counter;
    __device__ Work(double* p, int N) {
        const size_t n = lin_padded(N);
        Pg = reinterpret_cast<float*>(p);
        A64 = p + kLinBlk * n;
        double* q = A64 + (static_cast<size_t>(N) * N + 1) / 2 * 2;
        A32 = reinterpret_cast<float*>(q);
        rhs = q + n * n / 2;
        x = rhs + n;
        g = x + n;
        terms = g + n;
        counter = reinterpret_cast<unsigned*>(terms + n);
    }
    static size_t doubles(int N) {
        const size_t n = lin_padded(N);
        return kLinBlk * n + (static_cast<size_t>(N) * N + 1) / 2 * 2 + n * n / 2 + 4 * n + 2;
    }
};

// Row i of the system (linearized.rs:61-136): dot(factors[i][c], w) + diagonal, with w = -cl slope / u_t x the
// normal of the row's in-plane velocity.
struct SystemRow {
    d3 w;
    double rhs, diag;
};
__device__ __noinline__ SystemRow system_row(const DevModel& m, const SolveBuffers& b, int i, const double* tab) {
    SystemRow r;
    const d3 sd = normalize(m.span_e[i] - m.span_s[i]);
    d3 v = m.felt_ctrl[i] + b.fixed[i];
    v = v - sd * dot(v, sd);
    const d3 un = normalize(v);
    const double iut = rcp_any(dot(v, un));
    const FoilP& f = m.foils[m.wing_of_line[i]];
    r.w = cross(un, sd) * (-f.cl_initial_slope * iut);
    r.rhs = -line_lift(f, m.chord_global[i], v, sd, tab).cl_linear;
    r.diag = 2.0 * iut * rcp_any(m.chord_len[i]);
    return r;
}
__device__ __noinline__ LineLift lift_at(const DevModel& m, int i, d3 v, const double* tab) {
    return line_lift(m.foils[m.wing_of_line[i]], m.chord_global[i], v, normalize(m.span_e[i] - m.span_s[i]), tab);
}
// The viscous correction of line i's circulation (linearized.rs:178-202)
__device__ __forceinline__ double corrected_circulation(const LineLift& o, double x) {
    return fabs(o.cl_linear) > kMinPositive ? x * (o.cl_pre / o.cl_linear) : x;
}
__device__ __forceinline__ void write_line(const SolveBuffers& b, int i, double gi, d3 v) {
    b.gamma_prev[i] = gi;
    b.vel_out[i] = v;
    if (b.wake_str_row0) b.wake_str_row0[i] = gi;
    if (b.rec32_row0) b.rec32_row0[i].v[kRec32Gamma] = static_cast<float>(gi);
    if (b.rec64_row0) b.rec64_row0[i].v[kRec64Gamma] = gi;
}
// Mean of the residual terms and the solve's flags, by one warp.
__device__ __forceinline__ void write_scalars(const SolveBuffers& b, const double* terms, int N, int lane) {
    double s = 0.0;
    for (int i = lane; i < N; i += 32) s += terms[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
        b.scalars[0] = s / static_cast<double>(N);
        b.scalars[1] = 1.0;
        b.scalars[2] = 1.0;
        b.scalars[5] = 1.0;
    }
}

// SPLIT: the system comes from k_lin_build, and the solution goes to k_lin_finish (scalars[5] = 2).
template <bool SPLIT>
__device__ void solve(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, unsigned char* dyn) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    const int N = m.N, n = lin_padded(N), R = lin_local_rows(N, C), blocks = n / kLinBlk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kWarps = kThreads / 32;
    const LinLayout L = LinLayout::make(N, C);
    float* A = reinterpret_cast<float*>(dyn + L.A);
    float* P = reinterpret_cast<float*>(dyn + L.P);
    float* M = reinterpret_cast<float*>(dyn + L.M);
    double* x = reinterpret_cast<double*>(dyn + L.x);
    double* g = reinterpret_cast<double*>(dyn + L.g);
    float* rv = reinterpret_cast<float*>(dyn + L.rv);
    float* dx = reinterpret_cast<float*>(dyn + L.dx);
    d3* vel = reinterpret_cast<d3*>(dyn + L.vel);
    d3* roww = reinterpret_cast<d3*>(dyn + L.w);
    double* rhs = reinterpret_cast<double*>(dyn + L.rhs);
    double* diag = rhs + R;
    double* tab = reinterpret_cast<double*>(dyn + L.tab);
    const Work W(b.lin_work, N);
    float* Pg = W.Pg;
    double* A64 = W.A64;
    __shared__ __align__(16) float s_inv[kLinBlk][kLinBlk];
    __shared__ float s_red[kWarps][2];
    __shared__ int s_bad;

    auto row_of = [&](int l) { return lin_row(l, rank, C); };
    const int here = lin_own_rows(N, C, rank);  // of the R local rows, those of the system
    auto barrier = [&]() {
        if (C > 1) cl.sync();
        else __syncthreads();
    };

    if (tid == 0) s_bad = 0;
    // 1. the system; rows past the end: the identity
    if constexpr (SPLIT) {
        for (int l = tid; l < R; l += kThreads) rhs[l] = row_of(l) < n ? W.rhs[row_of(l)] : 0.0;
        for (int t = tid; t < R * n / 4; t += kThreads) {
            const int l = t / (n / 4), c = t % (n / 4) * 4, i = row_of(l);
            reinterpret_cast<float4*>(A)[t] = i < n ? __ldcg(reinterpret_cast<const float4*>(W.A32 + static_cast<long long>(i) * n + c))
                                                    : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        load_f64_tables(tab, tid, kThreads);
        __syncthreads();
        for (int l = tid; l < R; l += kThreads) {
            const int i = row_of(l);
            SystemRow r = {mk(0, 0, 0), 0.0, 1.0};
            if (i < N) r = system_row(m, b, i, tab);
            roww[l] = r.w;
            rhs[l] = r.rhs;
            diag[l] = r.diag;
        }
        __syncthreads();
        for (int l = warp; l < R; l += kWarps) {
            const int i = row_of(l);
            const d3 w = roww[l];
            const double dg = diag[l];
            for (int c = lane; c < n; c += 32) {
                float a = i == c && i >= N ? 1.f : 0.f;
                if (i < N && c < N) {
                    double v = dot(b.factors[static_cast<long long>(i) * N + c], w);
                    if (i == c) v += dg;
                    A64[static_cast<long long>(i) * N + c] = v;
                    a = f64_to_f32(v);
                }
                A[static_cast<long long>(l) * n + c] = a;
            }
        }
    }
    __syncthreads();

    // 2. FP32 inverse in place
    // The diagonal block of rows lk.. (columns k 16..) inverted by warp 0 (row = lane mod 16, eight
    // columns a lane), its rows scaled into P and the global buffer: outside the block's
    // columns inverse x row, inside the inverse.
    auto publish = [&](int k, int lk) {
        float* Pk = Pg + (k & 1) * kLinBlk * n;
        if (warp == 0) {
            const int row = lane & 15, half = lane >> 4;
            float* a = A + static_cast<long long>(lk + row) * n + k * kLinBlk + 8 * half;
            float v[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = a[c];
            float least = 3e38f;
#pragma unroll
            for (int q = 0; q < kLinBlk; ++q) {
                const int holder = q & 8 ? 16 : 0;  // lanes holding column q
                const float f = __shfl_sync(0xffffffffu, v[q & 7], holder + row);  // column q of the own row
                const float p = __shfl_sync(0xffffffffu, v[q & 7], holder + q);    // the pivot
                const float ip = rcp_seed(p);
                least = fminf(least, fabsf(p));
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float t = __shfl_sync(0xffffffffu, v[c], 16 * half + q) * ip;  // scaled pivot row
                    const bool pc = 8 * half + c == q;  // the pivot's column: of the identity
                    v[c] = row == q ? (pc ? ip : t) : (pc ? -f * ip : fmaf(-f, t, v[c]));
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) s_inv[8 * half + c][row] = v[c];  // transposed
            if (lane == 0 && !(least > 1e-6f)) s_bad = 1;
        }
        __syncthreads();
        for (int t = tid; t < n / 2; t += kThreads) {
            const int j = t % (n / 4) * 4, r0 = t / (n / 4) * 8;
            float4 o[8];
            if (j / kLinBlk == k) {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    o[q] = make_float4(s_inv[j % kLinBlk][r0 + q], s_inv[j % kLinBlk + 1][r0 + q], s_inv[j % kLinBlk + 2][r0 + q],
                                       s_inv[j % kLinBlk + 3][r0 + q]);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
                for (int e = 0; e < kLinBlk; ++e) {
                    const float4 a = *reinterpret_cast<const float4*>(A + static_cast<long long>(lk + e) * n + j);
                    const float4 f0 = *reinterpret_cast<const float4*>(&s_inv[e][r0]);
                    const float4 f1 = *reinterpret_cast<const float4*>(&s_inv[e][r0 + 4]);
                    const float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        o[q].x = fmaf(f[q], a.x, o[q].x);
                        o[q].y = fmaf(f[q], a.y, o[q].y);
                        o[q].z = fmaf(f[q], a.z, o[q].z);
                        o[q].w = fmaf(f[q], a.w, o[q].w);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) __stcg(reinterpret_cast<float4*>(Pk + (r0 + q) * n + j), o[q]);
        }
    };
    // rows [l0, l1) of the CTA less their multiples of P, 8 x 4 elements a thread; rows [own, own + 16)
    // become P itself
    auto update = [&](int l0, int l1, int own) {
        const int quads = n / 4;
        for (int t = tid; t < (l1 - l0) / 8 * quads; t += kThreads) {
            const int l = l0 + t / quads * 8, j = t % quads * 4;
            float* a = A + static_cast<long long>(l) * n + j;
            float4 o[8];
            if (l >= own && l < own + kLinBlk) {
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = *reinterpret_cast<const float4*>(P + (l - own + q) * n + j);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = *reinterpret_cast<const float4*>(a + static_cast<long long>(q) * n);
#pragma unroll 2
                for (int e = 0; e < kLinBlk; ++e) {
                    const float4 p = *reinterpret_cast<const float4*>(P + e * n + j);
                    const float4 m0 = *reinterpret_cast<const float4*>(M + e * R + l);
                    const float4 m1 = *reinterpret_cast<const float4*>(M + e * R + l + 4);
                    const float f[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        o[q].x = fmaf(-f[q], p.x, o[q].x);
                        o[q].y = fmaf(-f[q], p.y, o[q].y);
                        o[q].z = fmaf(-f[q], p.z, o[q].z);
                        o[q].w = fmaf(-f[q], p.w, o[q].w);
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) *reinterpret_cast<float4*>(a + static_cast<long long>(q) * n) = o[q];
        }
    };
    if (rank == 0) publish(0, 0);
    // split cluster barrier: a CTA arrives when it has read the last block's rows (and published the
    // next block's, where it owns it) and waits after updating its own rows
    auto arrive = [&]() {
        if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        else __syncthreads();
    };
    auto wait = [&]() {
        if (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    };
    __syncthreads();
    arrive();
#pragma unroll 1
    for (int k = 0; k < blocks; ++k) {
        const float* Pk = Pg + (k & 1) * kLinBlk * n;
        const int lk = k % C == rank ? k / C * kLinBlk : -kLinBlk;  // the block's first row where it is this CTA's
        const int nx = (k + 1 < blocks && (k + 1) % C == rank) ? (k + 1) / C * kLinBlk : -1;  // the next block's
        // the rows of block k are published; the buffer of block k - 1, which the owner of block k + 1
        // writes next, has been read by every CTA
        wait();
#pragma unroll 4
        for (int t = tid; t < kLinBlk * n / 4; t += kThreads)
            reinterpret_cast<float4*>(P)[t] = __ldcg(reinterpret_cast<const float4*>(Pk) + t);
        // multipliers of the own rows; the block's columns then start from 0
        for (int t = tid; t < R * kLinBlk; t += kThreads) {
            const int l = t >> 4, e = t & (kLinBlk - 1);
            float* a = A + static_cast<long long>(l) * n + k * kLinBlk + e;
            M[e * R + l] = *a;
            *a = 0.f;
        }
        __syncthreads();
        if (nx >= 0) {
            update(nx, nx + kLinBlk, lk);
            __syncthreads();
            publish(k + 1, nx);
        }
        __syncwarp();
        if (k + 1 < blocks) arrive();
        if (nx >= 0) {
            update(0, nx, lk);
            update(nx + kLinBlk, R, lk);
        } else {
            update(0, R, lk);
        }
        __syncthreads();
    }

    // value v of row i into every CTA's array
    auto store_all = [&](auto* arr, int i, auto v) {
        if (C == 1) arr[i] = v;
        else
            for (int q = 0; q < C; ++q) cl.map_shared_rank(arr, q)[i] = v;
    };
    // 3. refinement. A bad pivot of any CTA makes its first residual NaN, so that all of them stop.
    // Only rows of the system (l < here) are stored into the other CTAs: rv and dx hold n values each, and a
    // store past rv would land in dx, which a CTA behind may still be reading (no barrier between the two).
    for (int i = tid; i < n; i += kThreads) x[i] = 0.0;
    const float poison = s_bad ? __int_as_float(0x7FC00000) : 0.f;
    barrier();
    bool ok = false;
    float last = 0.f;
#pragma unroll 1
    for (int it = 0; it < kMaxRefine; ++it) {
        // residual of the own rows, to every CTA: eight lanes a row (the FP64 pipe takes a warp
        // instruction as long for one row's tree as for four rows')
        for (int l = 4 * warp + (lane >> 3); l < here; l += 4 * kWarps) {
            const int i = row_of(l);
            double s = 0.0;
            if (it > 0 && i < N)
                for (int c = lane & 7; c < N; c += 8) s = fma(-__ldcg(A64 + static_cast<long long>(i) * N + c), x[c], s);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const float f = static_cast<float>(rhs[l] + s) + poison;
            if (C == 1) {
                if ((lane & 7) == 0) rv[i] = f;
            } else {
                for (int q = lane & 7; q < C; q += 8) cl.map_shared_rank(rv, q)[i] = f;
            }
        }
        barrier();
        // correction of the own rows, to every CTA
        for (int l = warp; l < here; l += kWarps) {
            const int i = row_of(l);
            float s = 0.f;
            for (int c = 4 * lane; c < n; c += 128) {
                const float4 a = *reinterpret_cast<const float4*>(A + static_cast<long long>(l) * n + c);
                const float4 r = *reinterpret_cast<const float4*>(rv + c);
                s = fmaf(a.x, r.x, fmaf(a.y, r.y, fmaf(a.z, r.z, fmaf(a.w, r.w, s))));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (C == 1) {
                if (lane == 0) dx[i] = s;
            } else if (lane < C) {
                cl.map_shared_rank(dx, lane)[i] = s;
            }
        }
        barrier();
        float d = 0.f, y = 0.f;  // largest |dx| and |x|; a NaN stays
        bool fin = true;
        for (int i = tid; i < N; i += kThreads) {
            x[i] += static_cast<double>(dx[i]);
            const float a = fabsf(dx[i]);
            fin = fin && a < 3e38f;
            d = fmaxf(d, a);
            y = fmaxf(y, fabsf(static_cast<float>(x[i])));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d = fmaxf(d, __shfl_xor_sync(0xffffffffu, d, o));
            y = fmaxf(y, __shfl_xor_sync(0xffffffffu, y, o));
        }
        if (lane == 0) {
            s_red[warp][0] = d;
            s_red[warp][1] = y;
        }
        fin = __syncthreads_and(fin);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            d = fmaxf(d, s_red[w][0]);
            y = fmaxf(y, s_red[w][1]);
        }
        // the same numbers, so the same decision in every CTA
        if (!fin) break;
        // what is left is at most the ratio of the last two corrections times the last
        if (d <= 0x1p-50f * y || (it > 0 && d < 0.1f * last && d * (d / last) <= 0x1p-53f * y)) {
            ok = true;
            break;
        }
        if (it > 0 && d > 0.5f * last) {
            // No longer shrinking: an inverse that is none, or the rounding of the f64 residual, by which an
            // elimination would be off as well. An inverse that leaves more than 0.32 of a correction does not bring it to
            // 1e-10 within kMaxRefine, so that there it is the latter (emulated on 109 such systems of condition
            // 1e3 to 1e7: off by 0.57 of what an f64 elimination is, median).
            ok = d <= 1e-10f * y;
            break;
        }
        last = d;
        __syncthreads();  // s_red is written again
    }
    if (!ok) {  // the elimination kernels take the case
        if (rank == 0 && tid == 0) b.scalars[5] = 0.0;
        barrier();
        return;
    }

    if constexpr (SPLIT) {
        for (int l = tid; l < R; l += kThreads)
            if (row_of(l) < N) W.x[row_of(l)] = x[row_of(l)];
        if (rank == 0 && tid == 0) b.scalars[5] = 2.0;
        barrier();
        return;
    }
    // 4. induced velocity, total velocity, viscous correction (linearized.rs:141-202)
    auto total_velocities = [&](const double* gam) {
        for (int l = 4 * warp + (lane >> 3); l < R; l += 4 * kWarps) {
            const int i = row_of(l);
            d3 s = mk(0, 0, 0);
            if (i < N)
                for (int c = lane & 7; c < N; c += 8) {
                    const d3 f = b.factors[static_cast<long long>(i) * N + c];
                    s.x = fma(f.x, gam[c], s.x);
                    s.y = fma(f.y, gam[c], s.y);
                    s.z = fma(f.z, gam[c], s.z);
                }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
                s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
                s.z += __shfl_xor_sync(0xffffffffu, s.z, o);
            }
            if ((lane & 7) == 0 && i < N) {
                const d3 ind = b.fixed[i] + s, fs = m.felt_ctrl[i];
                vel[l] = st.velocity_correction == 0 ? fs + ind : corrected_velocity(st, fs, ind);
            }
        }
        __syncthreads();
    };
    total_velocities(x);
    double* gam = x;
    if (!st.disable_viscous_corrections) {
        for (int l = tid; l < R; l += kThreads) {
            const int i = row_of(l);
            if (i >= N) break;
            store_all(g, i, corrected_circulation(lift_at(m, i, vel[l], tab), x[i]));
        }
        barrier();
        gam = g;
        if (st.full_induced_correction) total_velocities(g);
    }
    // residual terms (linearized.rs:204-213) to CTA 0 (into x, no longer needed there unless it is
    // the circulation: then into g) and the outputs
    double* terms = gam == x ? g : x;
    barrier();
    for (int l = tid; l < R; l += kThreads) {
        const int i = row_of(l);
        if (i >= N) break;
        const double gi = gam[i];
        const d3 v = vel[l];
        *(cl.map_shared_rank(terms, 0) + i) = residual_of(m, i, gi, v, lift_at(m, i, v, tab).cl_pre);
        write_line(b, i, gi, v);
    }
    barrier();
    if (rank == 0 && warp == 0) write_scalars(b, terms, N, lane);
}

// Lines from which a case alone has its system built and its results evaluated by all SMs. Solve in us, one
// kernel / split: 256 lines 121 / 131, 384 193 / 191, 570 347 / 318, 768 516 / 479 (two or three launches of
// some 20 us, of which the chain of a line's lift is 10, against N^2 / 16 entries of FP64 work a CTA).
constexpr int kSplitLines = 448;
constexpr int kRowThreads = 128;  // a warp to a row, four rows a CTA
constexpr int kRowWarps = kRowThreads / 32;

// Step 1 for four rows: one warp's lanes evaluate the rows' vectors side by side, then a warp takes each
// row's entries. FP64-bound: 4 instructions an entry.
__global__ void __launch_bounds__(kRowThreads) k_lin_build(DevModel m, SolveBuffers b) {
    __shared__ __align__(16) double tab[kF64TableDoubles + 1];
    __shared__ SystemRow rows[kRowWarps];
    const int N = m.N, n = lin_padded(N), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Work W(b.lin_work, N);
    load_f64_tables(tab, tid, kRowThreads);
    __syncthreads();
    if (tid < kRowWarps) {
        const int i = blockIdx.x * kRowWarps + tid;
        SystemRow r = {mk(0, 0, 0), 0.0, 1.0};
        if (i < N) r = system_row(m, b, i, tab);
        rows[tid] = r;
        if (i < n) W.rhs[i] = r.rhs;
        if (i == 0) *W.counter = 0;
    }
    __syncthreads();
    const int i = blockIdx.x * kRowWarps + warp;
    if (i >= n) return;
    const SystemRow r = rows[warp];
#pragma unroll 4
    for (int c = lane; c < n; c += 32) {
        float a = i == c && i >= N ? 1.f : 0.f;
        if (i < N && c < N) {
            double v = dot(b.factors[static_cast<long long>(i) * N + c], r.w);
            if (i == c) v += r.diag;
            W.A64[static_cast<long long>(i) * N + c] = v;
            a = f64_to_f32(v);
        }
        W.A32[static_cast<long long>(i) * n + c] = a;
    }
}

// Step 4 for four rows, eight lanes a row as in the one-kernel form (the same bits alone and in a batch), a
// warp to each component (a lone warp issues an FP64 instruction per 65 cycles, three of them on an SM as well).
// pass 0: the velocity from the solution and the corrected circulation; it
// is the last one unless the correction's own induced velocities are wanted (pass 1). The last CTA of the
// last pass sums the residual.
constexpr int kFinishThreads = 96;
__global__ void __launch_bounds__(kFinishThreads) k_lin_finish(DevModel m, SolveSettings st, SolveBuffers b, int pass, int last) {
    __shared__ __align__(16) double tab[kF64TableDoubles + 1];
    __shared__ double ind[kRowWarps][3];
    if (b.scalars[5] != 2.0) return;  // the elimination kernels take the case
    const int N = m.N, lane = threadIdx.x & 31, comp = threadIdx.x >> 5;
    const Work W(b.lin_work, N);
    load_f64_tables(tab, threadIdx.x, kFinishThreads);
    const double* gam = pass == 0 ? W.x : W.g;
    int i = blockIdx.x * kRowWarps + (lane >> 3);
    double s = 0.0;
    if (i < N) {
        const double* f = reinterpret_cast<const double*>(b.factors + static_cast<long long>(i) * N) + comp;
#pragma unroll 4
        for (int c = lane & 7; c < N; c += 8) s = fma(f[3 * c], gam[c], s);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((lane & 7) == 0) ind[lane >> 3][comp] = s;
    __syncthreads();
    if (comp > 0) return;
    i = blockIdx.x * kRowWarps + lane;
    if (lane < kRowWarps && i < N) {
        const d3 u = b.fixed[i] + mk(ind[lane][0], ind[lane][1], ind[lane][2]), fs = m.felt_ctrl[i];
        const d3 v = st.velocity_correction == 0 ? fs + u : corrected_velocity(st, fs, u);
        const LineLift o = lift_at(m, i, v, tab);
        double gi = gam[i];
        if (pass == 0 && !st.disable_viscous_corrections) gi = corrected_circulation(o, gi);
        if (last) {
            W.terms[i] = residual_of(m, i, gi, v, o.cl_pre);
            write_line(b, i, gi, v);
        } else {
            W.g[i] = gi;
        }
        __threadfence();
    }
    if (!last) return;
    __syncwarp();
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(W.counter, 1u);
    if (__shfl_sync(0xffffffffu, before, 0) != gridDim.x - 1) return;
    __threadfence();
    write_scalars(b, W.terms, N, lane);
}

__global__ void __launch_bounds__(kThreads, 1) k_lin_refined(DevModel m, SolveSettings st, SolveBuffers b) {
    extern __shared__ __align__(16) unsigned char refined_dyn[];
    solve<false>(m, st, b, refined_dyn);
}
__global__ void __launch_bounds__(kThreads, 1) k_lin_refined_split(DevModel m, SolveSettings st, SolveBuffers b) {
    extern __shared__ __align__(16) unsigned char refined_dyn[];
    solve<true>(m, st, b, refined_dyn);
}

// Every case of a batch whose cluster size is this launch's: cluster i solves jobs[i].
__global__ void __launch_bounds__(kThreads, 1) k_lin_refined_jobs(const SolveJob* jobs) {
    extern __shared__ __align__(16) unsigned char refined_dyn[];
    const SolveJob& j = jobs[blockIdx.x / cg::this_cluster().num_blocks()];
    solve<false>(j.m, j.st, j.b, refined_dyn);
}

void config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, int clusters, int C, size_t smem, cudaStream_t s) {
    cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * C), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(C);
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

constexpr size_t kSmemLimit = 224 * 1024;

// Raises the kernels' limits, once per device; the largest cluster the device holds at kSmemLimit.
int largest_cluster() {
    static std::mutex mu;
    static std::map<int, int> largest;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 8;
    std::lock_guard<std::mutex> lk(mu);
    auto it = largest.find(dev);
    if (it != largest.end()) return it->second;
    auto prepare = [](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit)) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    };
    int c = prepare(k_lin_refined) && prepare(k_lin_refined_split) && prepare(k_lin_refined_jobs) ? 16 : 0;
    for (; c > 8; c /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        config(cfg, attr, 1, c, kSmemLimit, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_lin_refined, &cfg) == cudaSuccess && n > 0) break;
    }
    (void)cudaGetLastError();  // a refused shape is not an error of the caller
    largest[dev] = c;
    return c;
}

}  // namespace

size_t lin_work_doubles(int N) {
    return std::max(static_cast<size_t>(N) * (N + 1), Work::doubles(N));  // the elimination's [N][N + 1], or Work
}

LinPlan linearized_refined_plan(int N, int crowding) {
    int C = largest_cluster();
    while (C > 1 && C > lin_padded(N) / kLinBlk) C /= 2;
    if (C < 1 || LinLayout::make(N, C).total > kSmemLimit) return {0, 0};
    for (; crowding > 0 && C > 1 && LinLayout::make(N, C / 2).total <= kSmemLimit; --crowding) C /= 2;
    return {C, LinLayout::make(N, C).total};
}

static int finish_passes(const SolveSettings& st) { return st.full_induced_correction && !st.disable_viscous_corrections ? 2 : 1; }

int linearized_refined_launches(int N, const SolveSettings& st) { return N < kSplitLines ? 1 : 2 + finish_passes(st); }

cudaError_t launch_solve_linearized_refined(const DevModel& m, const SolveSettings& st, const SolveBuffers& b,
                                            const LinPlan& p, cudaStream_t s) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(cfg, attr, 1, p.cluster, p.smem, s);
    if (m.N < kSplitLines) return cudaLaunchKernelEx(&cfg, k_lin_refined, m, st, b);
    k_lin_build<<<(lin_padded(m.N) + kRowWarps - 1) / kRowWarps, kRowThreads, 0, s>>>(m, b);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k_lin_refined_split, m, st, b);
    const int passes = finish_passes(st);
    for (int k = 0; k < passes && e == cudaSuccess; ++k) {
        k_lin_finish<<<(m.N + kRowWarps - 1) / kRowWarps, kFinishThreads, 0, s>>>(m, st, b, k, k + 1 == passes);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_solve_linearized_refined_jobs(const SolveJob* jobs, int n, const LinPlan& p, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (p.cluster < 1 || p.smem > kSmemLimit) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    config(cfg, attr, n, p.cluster, p.smem, s);
    return cudaLaunchKernelEx(&cfg, k_lin_refined_jobs, jobs);
}

}  // namespace sbgpu
