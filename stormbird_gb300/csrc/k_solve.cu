// Circulation solvers (sm_103a), f64.
//
// k_solve_si: the damped fixed-point solve SimpleIterative::solve
// (stormbird/src/lifting_line/solvers/simple_iterative.rs:86-212) for one case on one
// thread-block cluster. Every CTA of the cluster keeps the full circulation vector in
// shared memory; CTA r owns a contiguous block of control points. Per iteration:
//   1. induced velocity of its rows: fixed + M * Gamma (frozen_wake.rs:268-301), 8, 16 or 32
//      lanes per row, the products summed in double-float arithmetic on the FP32 pipes
//      (~2^-44 relative per product; this part's FP64 rate is 1/64 of its FP32 rate), while a
//      ninth warp sums the residual terms of the iteration before (below);
//   2. per row, in f64: total velocity (velocity_corrections.rs:28-100), span component
//      removed (line_force_model/mod.rs:235-254), angle of attack
//      (force_calculations.rs:79-107), Foil lift, circulation estimate
//      (force_calculations.rs:271-292), residual term (force_calculations.rs:552-627) and
//      the damped update; the thread's own f64 circulation stays in registers;
//   3. new Gamma (as a float pair) and residual terms are stored into every CTA's shared
//      memory through distributed shared memory, a residual term with its sign set where
//      |dGamma| reaches the strength tolerance; one cluster barrier;
//   4. every CTA's ninth warp sums the residual terms in a fixed order (the same value, hence
//      the same stopping decision, in every CTA) during the next product, which a solve that
//      stops there computes for nothing.
// All waits are hardware cluster barriers; no spin loops.
//
// k_solve_lin / k_solve_lin_jobs: Linearized::solve (solvers/linearized.rs:54-222) with
// the Gaussian elimination with partial pivoting of stormath/src/matrix/linalg.rs:41-103,
// one CTA per case: one case, or all linearized quasi-steady cases of a batch in one
// launch.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "sb_device.cuh"
#include "sb_f64.cuh"
#include "sb_kernels.h"
#include "sb_ptx.cuh"

namespace cg = cooperative_groups;

namespace sbgpu {

constexpr int kSolveThreads = 256;                    // threads of the rows
constexpr int kSolveCtaThreads = kSolveThreads + 32;  // and the warp that sums the residual
constexpr int kSolveRowsPerThread = 4;                // most rows per thread (1024 per CTA)
constexpr int kMaxCluster = 16;                       // above 8: a non-portable cluster size

// Matrix slab of a CTA (its rows of the split matrix) in shared memory. Bytes of one row:
// 2 or 3 components (SolveBuffers::split_comps) x stride floats, twice with the lo plane.
__host__ __device__ inline long long si_row_bytes(int N, int full, int comps) {
    return 4LL * comps * si_matrix_stride(N) * (full ? 2 : 1);
}
// Shared memory before the slab, in doubles: circulation pairs 2 x stride, residual terms
// 2 x N, the f64 tables, the CTA's M * Gamma pairs (3 doubles per row), the own panels' lo
// parts (2 doubles per row), rounded to 16 bytes.
__host__ __device__ inline long long si_slab_offset(int N, int cluster) {
    const long long rp = (N + cluster - 1) / cluster;
    const long long d = 2LL * si_matrix_stride(N) + 2LL * N + kF64TableDoubles + 3 * rp + 2 * rp;
    return (d + 1) & ~1LL;
}

struct RowGeom {
    d3 felt, span_dir, chord, span_rel_out;  // span_dir = normalize(span end - span start)
    double chord_len, area;
    int wing;
};

__device__ inline RowGeom row_geom(const DevModel& m, int i) {
    RowGeom g;
    g.felt = m.felt_ctrl[i];
    const d3 span_rel = m.span_e[i] - m.span_s[i];
    g.span_dir = normalize(span_rel);
    g.chord = m.chord_global[i];
    g.span_rel_out = m.output_body ? (m.span_e_local[i] - m.span_s_local[i]) : span_rel;
    g.chord_len = m.chord_len[i];
    g.area = m.chord_len[i] * m.span_len_local[i];
    g.wing = m.wing_of_line[i];
    return g;
}

// velocity_corrections.rs:28-100 (returns freestream + induced, corrected)
__device__ inline d3 total_velocity(const SolveSettings& st, d3 fs, d3 ind) {
    if (st.velocity_correction == 1) {
        double im = len(ind), fm = len(fs);
        double mx = st.velocity_correction_ratio * fm;
        d3 c = im > mx ? normalize(ind) * mx : ind;
        return fs + c;
    }
    if (st.velocity_correction == 2) return normalize(fs + ind) * len(fs);
    return fs + ind;
}

// |cl_gamma - cl_direct| of force_calculations.rs:552-607, given cl_direct = the foil's
// pre-stall lift coefficient at the line's angle of attack
__device__ inline double residual_from_cl(const DevModel& m, const RowGeom& g, double gam, d3 u, double cl_pre) {
    double ul = len(u);
    d3 force = ul == 0.0 ? mk(0, 0, 0) : (gam * cross(u, g.span_rel_out)) * m.density;
    double sign = -1.0 * signum(gam);
    double ff = 0.5 * g.area * m.density * len2(u);
    double clg = ff == 0.0 ? 0.0 : len(force) * sign / ff;
    return fabs(clg - cl_pre);
}
__device__ inline double residual_term(const DevModel& m, const RowGeom& g, const FoilP& f, double gam, d3 u, double aoa) {
    return residual_from_cl(m, g, gam, u, foil_cl_pre_stall(f, aoa));
}
// What an iteration needs of a line, fixed for the solve: the velocity without the induced
// part of the first row of panels and the chord in the line's in-plane basis (e1 along the
// chord's in-plane part, e2 = span x e1; line_basis), the foil's constants, and the stall
// sigmoid's exponent as a straight line in |angle| (units of ln 2 / 512).
struct SolveLine {
    double a0, c0;           // (felt + fixed) . e1, . e2
    double kappa, k2;        // in-plane part of the chord / |chord|; 1 - kappa^2 (0: chord in the plane)
    double half_chord;       // -chord length / 2
    double cl_gamma;         // 2 |span| / area (0 if the area or the density is 0)
    double cl0, slope, cd_angle, exp_slope, exp_pos, exp_neg;
    float fa0, fc0, fcd, fslope, fpos, fneg;  // a0, c0, cd_angle, exp_* in FP32
    bool any;                // the line takes line_flow_any: see there
    bool skew, even;         // k2 != 0; the same stall angle on both sides
};

__device__ __noinline__ void solve_line(const DevModel& m, int i, d3 fixed, SolveLine& out) {
    SolveLine L;
    const d3 e1 = m.solve_basis[2 * i], e2 = m.solve_basis[2 * i + 1];
    const d3 base = m.felt_ctrl[i] + fixed;
    L.a0 = dot(base, e1);
    L.c0 = dot(base, e2);
    const d3 span_rel = m.span_e[i] - m.span_s[i];
    const d3 chord = m.chord_global[i];
    const double cn = len(chord);
    L.kappa = cn > 0.0 ? fmax(dot(chord, e1) / cn, 0.0) : -1.0;  // -1: no chord, no angle
    const double along = cn > 0.0 ? dot(chord, normalize(span_rel)) / cn : 0.0;
    // below 1e-24 the chord's part along the span changes no angle by more than 1e-12 rad at
    // |angle| = 1e-12, far under the angle's own rounding in the lift
    L.k2 = along * along > 1e-24 ? along * along : 0.0;
    const double cl = m.chord_len[i], area = cl * m.span_len_local[i];
    L.half_chord = -0.5 * cl;
    L.cl_gamma = (area == 0.0 || m.density == 0.0) ? 0.0 : 2.0 * len(span_rel) / area;
    const FoilP& f = m.foils[m.wing_of_line[i]];
    L.cl0 = f.cl_zero_angle;
    L.slope = f.cl_initial_slope;
    L.cd_angle = f.angle_cd_min;
    constexpr double kPerLn2 = 738.6598609351491;  // 512 / ln 2
    L.exp_slope = -f.stall_slope * kPerLn2;
    L.exp_pos = f.stall_slope * fabs(f.mean_positive_stall_angle) * kPerLn2;
    L.exp_neg = f.stall_slope * fabs(f.mean_negative_stall_angle) * kPerLn2;
    L.fa0 = static_cast<float>(L.a0);
    L.fc0 = static_cast<float>(L.c0);
    L.fcd = static_cast<float>(L.cd_angle);
    L.fslope = static_cast<float>(L.exp_slope);
    L.fpos = static_cast<float>(L.exp_pos);
    L.fneg = static_cast<float>(L.exp_neg);
    // The exponent's FP32 copy, which picks its integer part and decides that it is beyond -32768, has to be
    // good to a few hundred: its terms are off by some 1e-6 of the slope (the angle in FP32) and 6e-8 of the
    // stall angles' part. A stall range of 0 has an infinite slope.
    const bool fits = fabsf(L.fslope) < 1e8f && fabsf(L.fpos) < 1e9f && fabsf(L.fneg) < 1e9f && fabsf(L.fcd) < 4.f;
    L.any = !(L.kappa > 0.0) || f.cl_high_order_power > 0.0 || !fits;
    L.skew = L.k2 != 0.0;
    L.even = L.exp_pos == L.exp_neg;
    out = L;
}

// Flow at a line with the in-plane velocity a e1 + c e2.
struct LineFlow {
    double ul, inv;  // |u|, 1 / |u| (inv = 0 where |u| is 0)
    double cl_pre;   // the foil's pre-stall lift coefficient (foil.rs:166-190)
    double cl_post;  // post-stall part (foil.rs:193-206), where asked for
};

// The same by CUDA's f64 functions, for what lies outside the ranges of line_flow's
// arithmetic: |u| = 0, infinite or beyond 2^(+-50), a chord along the span or of no length, a
// high-order lift term, a stall range so narrow that FP32 cannot tell the exponent (below 2e-3
// degrees; 0: a step), an exponent above 32000.
__device__ __noinline__ LineFlow line_flow_any(double kappa, const FoilP& f, double a, double c, bool post) {
    LineFlow o;
    o.ul = sqrt(a * a + c * c);
    o.inv = o.ul == 0.0 ? 0.0 : 1.0 / o.ul;
    double aoa = 0.0;
    if (o.ul > kMinPositive && kappa >= 0.0) {
        const double ang = acos(fmin(fmax(kappa * a / o.ul, -1.0), 1.0));
        aoa = kappa * c > 0.0 ? ang : -ang;
    }
    o.cl_pre = foil_cl_pre_stall(f, aoa);
    o.cl_post = post ? foil_cl_post_stall(f, aoa) : 0.0;
    return o;
}

// Angle of attack (signed_angle_between(chord, u, span), vector_math.rs:65-95): its cosine is
// kappa a / |u|, its sign that of kappa c, so the sine in the lift needs no angle, and the
// angle in the stall sigmoid comes from both (better conditioned than acos of the cosine
// near 0). fa, fc: a and c in FP32, from which the seeds, the table entries and the integer part of
// the exponent are picked beside the FP64 chain. 29 FP64 instructions (CUDA's sqrt, division,
// acos, sin and exp took about 150).
__device__ __forceinline__ LineFlow line_flow(const SolveLine& L, const DevModel& m, int i, double a, double c, float fa,
                                              float fc, bool post, const double* tab) {
    // FP32: 1 / |u|, the angle, the exponent of the stall sigmoid in units of ln 2 / 512
    const bool pos = f64_positive(c);
    const float fq = fmaf(fa, fa, fc * fc), fi = rsqrt_seed(fq);
    float fx = fa * fi, fy = fabsf(fc) * fi;
    if (L.skew) {
        fy = sqrtf(fmaf(static_cast<float>(L.k2) * fx, fx, fy * fy));
        fx *= static_cast<float>(L.kappa);
    }
    float fang;
    const double* e = angle_entry(fx, fy, tab, fang);
    const float fe = (pos ? fang : -fang) + L.fcd;
    const bool side = fe >= 0.f;  // which stall angle
    // below 2^-64 the exponential leaves the stall at 1 (to rounding)
    const float fw = fmaxf(fmaf(fabsf(fe), L.fslope, side ? L.fpos : L.fneg), -32768.f);
    const int n = __float2int_rn(fminf(fw, 32768.f));
    const double q = fma(a, a, c * c);
    LineFlow o;
    bool ok = !L.any && f64_seed_range(q) && fw < 32000.f;
    ok = rsqrt_step(q, fi, o.inv) && ok;
    o.ul = q * o.inv;
    double y = fabs(c) * o.inv, d, x = 0.0;
    if (L.skew) {  // a chord with a part along the span: cos = kappa a / |u|
        x = a * o.inv;
        const double y2 = fma(L.k2 * x, x, y * y);
        ok = ok && f64_seed_range(y2);
        y = y2 * rsqrt_f64(y2);
        x *= L.kappa;
        d = fma(y, e[0], -(x * e[1]));
    } else {
        d = fma(fabs(c), e[0], -(a * e[1])) * o.inv;
    }
    // |angle + angle_cd_min| = |th + sgn delta|, th the table angle with both signs in
    const double del = arcsin_f64(d), th = (pos ? e[2] : -e[2]) + L.cd_angle;
    const double ae = fabs(pos ? th + del : th - del);
    // f: what the exponent has beyond its integer part n; beyond -32768 it is left out
    double f = fma(ae, L.exp_slope, (side ? L.exp_pos : L.exp_neg) - f32_to_f64(static_cast<float>(n)));
    if (fw <= -32768.f) f = 0.0;
    const double v = 1.0 + exp2_512_f64(n, f, tab);
    double stall;  // foil_amount_of_stall
    ok = rcp_step(v, rcp_seed(1.f + exp2f(fw * (1.f / 512.f))), stall) && ok;
    // (where the two stall angles differ, an angle so small that FP32 may see the other side too)
    ok = ok && fabsf(f64_to_f32(f)) < 0.75f && (L.even || fabsf(fe) > 1e-6f);
    if (!ok) return line_flow_any(L.kappa, m.foils[m.wing_of_line[i]], a, c, post);
    const double sn = pos ? y : -y;
    const double raw = fma(L.slope, sn, L.cl0);
    o.cl_pre = fma(-raw, stall, raw);
    if (post)  // sin 2a = 2 sin a cos a, |a| <= pi
        o.cl_post = m.foils[m.wing_of_line[i]].cl_max_after_stall * (2.0 * sn * (L.skew ? x : a * o.inv)) * stall;
    else
        o.cl_post = 0.0;
    return o;
}

// Residual term of a line (force_calculations.rs:552-627): |cl of the force - cl of the foil|.
// In the global output frame the line's span vector is the one u was made perpendicular to, so
// the lift coefficient of the force -gam |u| |span| rho / (area rho |u|^2 / 2) is
// -gam cl_gamma / |u|. (Body-frame output keeps residual_from_cl: there the span vector is the
// body frame's.)
__device__ __noinline__ double residual_body(const DevModel& m, int i, double gam, double a, double c, double cl_pre) {
    return residual_from_cl(m, row_geom(m, i), gam, m.solve_basis[2 * i] * a + m.solve_basis[2 * i + 1] * c, cl_pre);
}
__device__ __forceinline__ double residual_of_line(const DevModel& m, const SolveLine& L, int i, double gam, double a,
                                                   double c, const LineFlow& o) {
    if (m.output_body) return residual_body(m, i, gam, a, c, o.cl_pre);
    return fabs(fma(-gam * L.cl_gamma, o.inv, -o.cl_pre));
}

// Double-float accumulation for the matrix-vector product: (S, C) += (xh + xl) * (gh + gl).
// The product's head xh*gh is added to S by an error-free two-sum (Knuth: exact for any
// magnitudes; a Kahan-compensated sum, two operations cheaper, is exact only while the
// running sum outweighs the new term and left the solve a residual floor near 1e-11); its
// rounding error (an exact FMA) and the cross terms xh*gl + xl*gh go into C; xl*gl (~2^-48 of
// the product) is dropped. The _rn intrinsics keep the compiler from fusing the steps.
template <bool LO>
__device__ __forceinline__ void ff_mac(float& S, float& C, float xh, float xl, float gh, float gl) {
    const float p = __fmul_rn(xh, gh);
    float t = fmaf(xh, gh, -p);
    t = fmaf(xh, gl, t);
    if (LO) t = fmaf(xl, gh, t);
    const float s = __fadd_rn(S, p);
    const float bv = __fsub_rn(s, S);
    const float err = __fadd_rn(__fsub_rn(S, __fsub_rn(s, bv)), __fsub_rn(p, bv));
    S = s;
    C = __fadd_rn(C, __fadd_rn(err, t));
}
// (S, C) += (h, l), another double-float partial sum
__device__ __forceinline__ void ff_add(float& S, float& C, float h, float l) {
    const float s = __fadd_rn(S, h);
    const float bv = __fsub_rn(s, S);
    const float err = __fadd_rn(__fsub_rn(S, __fsub_rn(s, bv)), __fsub_rn(h, bv));
    S = s;
    C = __fadd_rn(C, __fadd_rn(err, l));
}
// The same for the two in-plane components at once, as the lanes of packed FP32 operations
// (half the instructions: at two warps per SM sub-partition the product is bound by their issue and
// latency): component x in .x, y in .y, the circulation as broadcast pairs. a - b is the packed
// FMA (b * -1 + a), exact like the subtraction.
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
template <bool LO>
__device__ __forceinline__ void ff_mac2(float2& S, float2& C, float2 xh, float2 xl, float2 gh, float2 gl) {
    const float2 p = __fmul2_rn(xh, gh);
    float2 t = __ffma2_rn(xh, gh, make_float2(-p.x, -p.y));
    t = __ffma2_rn(xh, gl, t);
    if (LO) t = __ffma2_rn(xl, gh, t);
    const float2 s = __fadd2_rn(S, p);
    const float2 bv = f2_sub(s, S);
    const float2 err = __fadd2_rn(f2_sub(S, f2_sub(s, bv)), f2_sub(p, bv));
    S = s;
    C = __fadd2_rn(C, __fadd2_rn(err, t));
}
__device__ __forceinline__ void ff_add2(float2& S, float2& C, float2 h, float2 l) {
    const float2 s = __fadd2_rn(S, h);
    const float2 bv = f2_sub(s, S);
    const float2 err = __fadd2_rn(f2_sub(S, f2_sub(s, bv)), f2_sub(h, bv));
    S = s;
    C = __fadd2_rn(C, __fadd2_rn(err, l));
}
__device__ __forceinline__ float2 shfl_xor2(float2 v, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

// A row of the split matrix times the circulation Gc (pairs gh, gl), summed over the 1 << lp lanes
// of a row (every one of them gets the sum): lane gl takes four consecutive columns 4 gl + (4 << lp) t.
// out: (hi, lo) per component. Two components: pairs (x, y) per column; three: planes x, y, z of
// S floats. fl: the lo plane (LO only).
template <int NC, bool LO>
__device__ __forceinline__ void row_dot(const float* fh, const float* fl, const float2* Gc, int S, int gl, int lp,
                                        float (&out)[6]) {
    if constexpr (NC == 2) {
        float2 Sa = make_float2(0.f, 0.f), Ca = Sa, Sb = Sa, Cb = Sa;  // two chains, merged at the end
#pragma unroll 1
        for (int k = 4 * gl; k < S; k += 4 << lp) {
            const float4 g0 = *reinterpret_cast<const float4*>(Gc + k), g1 = *reinterpret_cast<const float4*>(Gc + k + 2);
            const float4 a0 = *reinterpret_cast<const float4*>(fh + 2 * k), a1 = *reinterpret_cast<const float4*>(fh + 2 * k + 4);
            float4 l0 = make_float4(0.f, 0.f, 0.f, 0.f), l1 = l0;
            if (LO) {
                l0 = *reinterpret_cast<const float4*>(fl + 2 * k);
                l1 = *reinterpret_cast<const float4*>(fl + 2 * k + 4);
            }
            ff_mac2<LO>(Sa, Ca, make_float2(a0.x, a0.y), make_float2(l0.x, l0.y), make_float2(g0.x, g0.x), make_float2(g0.y, g0.y));
            ff_mac2<LO>(Sb, Cb, make_float2(a0.z, a0.w), make_float2(l0.z, l0.w), make_float2(g0.z, g0.z), make_float2(g0.w, g0.w));
            ff_mac2<LO>(Sa, Ca, make_float2(a1.x, a1.y), make_float2(l1.x, l1.y), make_float2(g1.x, g1.x), make_float2(g1.y, g1.y));
            ff_mac2<LO>(Sb, Cb, make_float2(a1.z, a1.w), make_float2(l1.z, l1.w), make_float2(g1.z, g1.z), make_float2(g1.w, g1.w));
        }
        ff_add2(Sa, Ca, Sb, Cb);
#pragma unroll 1
        for (int o = 1 << (lp - 1); o > 0; o >>= 1) ff_add2(Sa, Ca, shfl_xor2(Sa, o), shfl_xor2(Ca, o));
        out[0] = Sa.x;
        out[1] = Ca.x;
        out[2] = Sa.y;
        out[3] = Ca.y;
    } else {
        float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
        for (int k = 4 * gl; k < S; k += 4 << lp) {
            const float4 g0 = *reinterpret_cast<const float4*>(Gc + k), g1 = *reinterpret_cast<const float4*>(Gc + k + 2);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float4 a = *reinterpret_cast<const float4*>(fh + q * S + k);
                const float4 l = LO ? *reinterpret_cast<const float4*>(fl + q * S + k) : make_float4(0.f, 0.f, 0.f, 0.f);
                ff_mac<LO>(acc[2 * q], acc[2 * q + 1], a.x, l.x, g0.x, g0.y);
                ff_mac<LO>(acc[2 * q], acc[2 * q + 1], a.y, l.y, g0.z, g0.w);
                ff_mac<LO>(acc[2 * q], acc[2 * q + 1], a.z, l.z, g1.x, g1.y);
                ff_mac<LO>(acc[2 * q], acc[2 * q + 1], a.w, l.w, g1.z, g1.w);
            }
        }
#pragma unroll 1
        for (int o = 1 << (lp - 1); o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                ff_add(acc[2 * q], acc[2 * q + 1], __shfl_xor_sync(0xffffffffu, acc[2 * q], o),
                       __shfl_xor_sync(0xffffffffu, acc[2 * q + 1], o));
#pragma unroll
        for (int q = 0; q < 6; ++q) out[q] = acc[q];
    }
}

// Sum / max over a warp in a fixed order (lane 0 gets the result): every CTA of a cluster
// reduces the same residual terms the same way and takes the same stopping decision.
__device__ __forceinline__ double warp_sum_to_lane0(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// Maxima of magnitudes on the integer pipe (this part's FP64 pipe costs a full warp
// instruction per compare): |v| as its IEEE bit pattern, which orders like an unsigned
// integer for non-negative values; a NaN maps to 0, as fmax(x, NaN) = x leaves it out.
__device__ __forceinline__ unsigned long long mag_bits(double v) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
    return b > 0x7FF0000000000000ull ? 0ull : b;
}
__device__ __forceinline__ double bits_value(unsigned long long b) { return __longlong_as_double(static_cast<long long>(b)); }
__device__ __forceinline__ unsigned long long warp_umax_to_lane0(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// SimpleIterative::solve for one case on the calling thread-block cluster (see the top of
// the file). Run by k_solve_si (one case) and k_solve_si_jobs (a cluster per case of a batch).
// RPT = rows per thread: 1 while a CTA owns at most kSolveThreads rows (registers for two
// CTAs per SM), else kSolveRowsPerThread. NC = components of a matrix entry
// (SolveBuffers::split_comps), LO: the lo plane is read (split_full). Each variant's loop is kept
// small (rare branches out of line, one copy of the product and of the row math for the guard's
// passes and the iterations alike): with every variant in one kernel the code was 325 KB, and a
// loop that does not fit the instruction cache waits for its instructions.
template <int RPT, int NC, bool LO>
__device__ void si_solve(const DevModel& m, const SolveSettings& st, const SolveBuffers& b) {
    cg::cluster_group cl = cg::this_cluster();
    const int CS = static_cast<int>(cl.num_blocks());
    const int rank = static_cast<int>(cl.block_rank());
    const int N = m.N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool sums = warp == kSolveThreads / 32;  // the warp that sums the residual and issues the copies
    extern __shared__ __align__(16) double smem[];
    // circulation of every line as (hi, lo) float pairs for the matrix-vector products, padded
    // with zeros to the matrix's row stride; the f64 circulation of the thread's own rows
    // stays in registers (gown)
    const int S = si_matrix_stride(N);
    const int rp = (N + CS - 1) / CS;
    const int r0 = min(N, rank * rp), r1 = min(N, r0 + rp);
    auto G = [&](int k) { return reinterpret_cast<float2*>(smem) + k * S; };
    auto RR = [&](int k) { return smem + 2 * S + k * N; };
    double* tab = smem + 2 * S + 2 * N;
    // M * Gamma of the CTA's rows as double-float pairs (x hi, x lo, y hi, y lo, z hi, z lo);
    // the row's owner adds them to the fixed part in f64
    float* uff = reinterpret_cast<float*>(tab + kF64TableDoubles);
    // lo parts of the own panels' entries (x, y, z), when the matrix has none elsewhere
    float* diag_lo = reinterpret_cast<float*>(tab + kF64TableDoubles + 3 * rp);
    float* slab = reinterpret_cast<float*>(smem + si_slab_offset(N, CS));
    __shared__ double s_res;
    __shared__ unsigned long long s_umax;
    __shared__ int s_conv;
    __shared__ __align__(8) uint64_t s_mbar[2];

    auto barrier = [&]() {
        if (CS > 1) cl.sync();
        else __syncthreads();
    };
    // The thread's k-th own row (offset from r0): consecutive rows on consecutive threads, so
    // that a CTA owning fewer than 256 rows fills as few warps as possible (this part's FP64
    // pipe costs the same per warp instruction however few lanes are active).
    auto own_row = [&](int k) { return tid + k * kSolveThreads; };

    const bool scale0 = fabs(st.correction_factor_initial - 1.0) > kMinPositive;
    for (int i = tid; i < N; i += kSolveCtaThreads) {
        double g = b.gamma_prev[i];
        if (scale0) g *= st.correction_factor_initial;
        G(0)[i] = split_f64(g);
    }
    for (int i = N + tid; i < S; i += kSolveCtaThreads) G(0)[i] = G(1)[i] = make_float2(0.f, 0.f);
    load_f64_tables(tab, tid, kSolveCtaThreads);
    // per-thread rows: the in-plane velocity and the circulation estimate of the last iteration
    SolveLine ln[RPT];
    double a_last[RPT], c_last[RPT], est_last[RPT], gown[RPT];
    int nrows = 0;
    for (int k = 0; k < RPT; ++k) {
        int i = r0 + own_row(k);
        if (!sums && i < r1) {
            double g = b.gamma_prev[i];
            if (scale0) g *= st.correction_factor_initial;
            gown[k] = g;
            SolveLine l;
            solve_line(m, i, b.fixed[i], l);
            ln[k] = l;
            a_last[k] = c_last[k] = est_last[k] = 0.0;
            nrows = k + 1;
        }
    }

    constexpr int C = NC;  // 2: in-plane components in the rows' bases, 3: x, y, z
    const int slab_rows = b.slab_rows;
    const int nrows_cta = r1 - r0;
    const int nch = slab_rows > 0 ? (nrows_cta + slab_rows - 1) / slab_rows : 0;
    const bool resident = slab_rows > 0 && slab_rows >= rp;      // copied once, kept
    const long long rowf = static_cast<long long>(C) * S;         // floats of a row, one plane
    const long long buf_floats = static_cast<long long>(slab_rows) * rowf * (LO ? 2 : 1);
    const long long lo_plane = static_cast<long long>(C) * N * S;
    const int lp = b.lanes_log2;  // log2 of the lanes per row of the product
    if (tid == 0) {
        mbar_init(&s_mbar[0], 1);
        mbar_init(&s_mbar[1], 1);
        fence_mbar_init();
    }
    if (!LO)
        for (int k = tid; k < nrows_cta; k += kSolveCtaThreads) {
            const long long row = r0 + k;
            const float* fl = b.factors_split + lo_plane + row * rowf;
            for (int q = 0; q < C; ++q) diag_lo[3 * k + q] = fl[C == 2 ? 2 * row + q : q * S + row];
        }

    // residual of the initial solution with zero velocity (simple_iterative.rs:180-184)
    double residual = 0.0;
    if (st.max_iterations == 0) {
        if (tid == 0) {
            double s = 0.0;
            for (int i = 0; i < N; ++i)
                s += fabs(0.0 - line_flow_any(-1.0, m.foils[m.wing_of_line[i]], 0.0, 0.0, false).cl_pre);
            s_res = s;
        }
        __syncthreads();
        residual = s_res;
    }
    barrier();

    // induced velocity of own rows for the circulation Gc: fixed + M * Gc, in double-float
    // arithmetic on the FP32 pipes (this part's FP64 rate is 1/64 of its FP32 rate). 8, 16 or 32
    // lanes take a row, four consecutive columns per step, then a butterfly over them (row_dot). The CTA's matrix rows come from its slab in
    // shared memory: one thread copies them by bulk asynchronous copies (cp.async.bulk,
    // completion on an mbarrier; bounded waits), kept for the whole solve when they fit, else
    // streamed in chunks through two buffers (the copy of chunk c + 1 runs while the warps
    // work on chunk c).
    // A slab wait that runs out records kDevTimeout (the host raises SB_ERR_TIMEOUT after the
    // launch); that thread then waits no more and the copying thread issues no more copies, and
    // the solve runs its remaining (bounded) iterations on whatever the buffers hold, through the
    // same barriers as the other CTAs of the cluster, so that none waits for it forever.
    uint32_t mph[2] = {0u, 0u};
    bool pending[2] = {false, false};  // copying thread: a copy into the buffer not yet waited for
    bool slab_loaded = false, dead = false;
    const bool copier = tid == kSolveThreads;
    auto issue = [&](int c, int bufi) {
        const long long row0 = r0 + static_cast<long long>(c) * slab_rows;
        const int nr = min(slab_rows, r1 - static_cast<int>(row0));
        const uint32_t bytes = static_cast<uint32_t>(nr * rowf * 4);
        float* dst = slab + bufi * buf_floats;
        mbar_expect_tx(&s_mbar[bufi], LO ? 2 * bytes : bytes);
        bulk_g2s(dst, b.factors_split + row0 * rowf, bytes, &s_mbar[bufi]);
        if (LO) bulk_g2s(dst + slab_rows * rowf, b.factors_split + lo_plane + row0 * rowf, bytes, &s_mbar[bufi]);
        pending[bufi] = true;
    };
    // rows [row0, row0 + nr) of the matrix at `base` (lo plane at base + lo_off) times Gc. Every
    // lane of a warp goes through the butterflies together: groups past the end repeat the last
    // row and store nothing.
    auto rows_times = [&](const float* base, long long lo_off, int row0, int nr, const float2* Gc) {
        const int group = tid >> lp, gl = tid & ((1 << lp) - 1), groups = kSolveThreads >> lp;
#pragma unroll 1
        for (int w0 = 0; w0 < nr; w0 += groups) {
            if (w0 + ((warp * 32) >> lp) >= nr) break;  // uniform in the warp
            const int w = min(w0 + group, nr - 1);
            const float* fh = base + w * rowf;
            float acc[6];
            row_dot<NC, LO>(fh, fh + lo_off, Gc, S, gl, lp, acc);
            if (gl == 0 && w0 + group < nr) {
                const int row = row0 + w;
                if (!LO) {  // the own panel's entry is f64: its lo parts times Gamma hi
                    const float g = Gc[row].x;
                    const float* dl = diag_lo + 3 * (row - r0);
#pragma unroll
                    for (int q = 0; q < NC; ++q) ff_add(acc[2 * q], acc[2 * q + 1], __fmul_rn(dl[q], g), fmaf(dl[q], g, -__fmul_rn(dl[q], g)));
                }
                float* o = uff + 6 * (row - r0);
#pragma unroll
                for (int q = 0; q < 2 * NC; ++q) o[q] = acc[q];
            }
        }
    };
    // The sum of the residual over all lines from the terms in R and whether the solve stops there
    // (the summing warp): lanes over lines lane, lane + 32, ..., then a fixed-order tree. The mean
    // is compared with its tolerance as the sum with N times it (a division is 9 FP64
    // instructions); the mean itself is the last sum over N.
    const bool want_max = st.strength_tolerance > 0.0;
    const double sum_tolerance = st.residual_tolerance * static_cast<double>(N);
    auto decide = [&](const double* R) {
        double s = 0.0;
        bool big = false;  // some |dGamma| at or above the strength tolerance (the term's sign)
#pragma unroll 1
        for (int i = lane; i < N; i += 32) {
            const double v = R[i];
            s += fabs(v);
            big = big || __double2hiint(v) < 0;
        }
        s = warp_sum_to_lane0(s);
        big = __any_sync(0xffffffffu, big) != 0;
        if (lane == 0) {
            s_res = s;
            s_conv = s < sum_tolerance || (want_max && !big);
        }
    };
    // M * Gc of the CTA's rows (none: Gc == nullptr) beside the sum of the residual terms R of the
    // iteration before (none: R == nullptr)
    auto induced_rows = [&](const float2* Gc, const double* R) {
        const bool copy = nch > 0 && !(resident && slab_loaded) && Gc;  // nch: 0 also for a CTA without rows
        if (copy && copier && !dead) {
            issue(0, 0);
            if (nch > 1) issue(1, 1);
        }
        if (sums) {
            __syncwarp();
            if (R) decide(R);
        }
        const int chunks = !Gc ? 0 : (slab_rows > 0 ? nch : (nrows_cta > 0 ? 1 : 0));
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) {
            const int bufi = c & 1;
            if (copy) {
                if (!dead) {
                    if (mbar_wait_bounded(&s_mbar[bufi], mph[bufi], b.err)) pending[bufi] = false;
                    else dead = true;
                }
                mph[bufi] ^= 1u;
            }
            const int row0 = r0 + c * slab_rows;
            const int nr = slab_rows > 0 ? min(slab_rows, r1 - row0) : nrows_cta;  // 0: rows from global memory
            const float* base = slab_rows > 0 ? slab + bufi * buf_floats : b.factors_split + static_cast<long long>(r0) * rowf;
            if (!sums) rows_times(base, slab_rows > 0 ? slab_rows * rowf : lo_plane, row0, nr, Gc);
            __syncthreads();  // every warp is done with this buffer
            if (copy && !resident && copier && !dead && c + 2 < nch) issue(c + 2, bufi);
        }
        if (chunks == 0) __syncthreads();
        else slab_loaded = true;
    };
    // In-plane velocity (a, c) of own row i: freestream + fixed + M * Gamma with the span
    // component taken out (project(u, span_rel) before the angle). With two components the
    // products are already the in-plane coordinates along the row's basis (e1, e2), and the
    // velocity correction is off (the only mode the two-component matrix is built for).
    auto row_velocity = [&](int i, const SolveLine& L, double& a, double& c, float& fa, float& fc) {
        const float* o = uff + 6 * (i - r0);
        if (C == 2) {
            fa = L.fa0 + o[0];
            fc = L.fc0 + o[2];
            // exactly: in calm air at rest the sums are 0, and so have to be the velocity and its angle
            a = L.a0 + (f32_to_f64_exact(o[0]) + f32_to_f64_exact(o[1]));
            c = L.c0 + (f32_to_f64_exact(o[2]) + f32_to_f64_exact(o[3]));
            return;
        }
        const d3 fx = b.fixed[i];
        const d3 ind = mk(fx.x + (static_cast<double>(o[0]) + static_cast<double>(o[1])),
                          fx.y + (static_cast<double>(o[2]) + static_cast<double>(o[3])),
                          fx.z + (static_cast<double>(o[4]) + static_cast<double>(o[5])));
        const d3 u = total_velocity(st, m.felt_ctrl[i], ind);
        a = dot(u, m.solve_basis[2 * i]);
        c = dot(u, m.solve_basis[2 * i + 1]);
        fa = static_cast<float>(a);
        fc = static_cast<float>(c);
    };
    // v into slot i of an array of every CTA of the cluster
    auto store_all = [&](auto* arr, int i, auto v) {
        if (CS == 1) arr[i] = v;
        else
            for (int q = 0; q < CS; ++q) cl.map_shared_rank(arr, q)[i] = v;
    };

    // Guarded warm start: residual (simple_iterative.rs:160-176) of the plain start G[0]
    // and of each candidate (staged in G[1]). A candidate replaces the current start only
    // when both its mean residual (the solver's own measure) and its largest per-line term
    // are lower: the solver stops on the mean, which a start with its error on a few lines
    // could pass while those lines are still off. The plain start wins ties. The second
    // candidate (the network's) must beat the best start so far by b.second_margin (0.5 by
    // default) on both measures: its per-line error is noise-like, and a start that is only slightly
    // better by the initial residual took more iterations than the extrapolation (566 of
    // 2,560 solves of the uneven-case batch: 108 iterations against 107 from the plain start).
    // Passes start = 0 (plain), 1, 2 (candidates) run the iteration's own product and row math;
    // 3: the iterations.
    const bool guarded = b.candidate[0] || b.candidate[1];
    int start = guarded ? 0 : 3;
    double best = 0.0, best_max = 0.0;
    int taken = guarded ? 0 : -1;
    int it = 0, cur = 0;
    bool conv = false;
#pragma unroll 1
    while (true) {
        const double* src = nullptr;
        if (start == 1 || start == 2) {
            src = b.candidate[start - 1];
            if (!src) {
                ++start;
                continue;
            }
            for (int i = tid; i < N; i += kSolveCtaThreads) G(1)[i] = split_f64(src[i]);
            __syncthreads();
        }
        const bool more = start < 3 || it < st.max_iterations;
        // 1. induced velocity of own rows; the last iteration's residual and decision
        induced_rows(more ? G(start < 3 ? start > 0 : cur) : nullptr, it > 0 ? RR((it - 1) & 1) : nullptr);
        if (it > 0) {
            residual = s_res;
            conv = s_conv != 0;
        }
        if (conv || !more) break;
        // 2. row updates
#pragma unroll 1
        for (int k = 0; k < (RPT == 1 ? min(nrows, 1) : nrows); ++k) {
            const int i = r0 + own_row(k);
            const SolveLine& L = ln[RPT == 1 ? 0 : k];
            double a, c;
            float fa, fc;
            row_velocity(i, L, a, c, fa, fc);
            const LineFlow o = line_flow(L, m, i, a, c, fa, fc, m.include_viscous_lift != 0, tab);
            const double gold = src ? src[i] : gown[RPT == 1 ? 0 : k];
            double r = residual_of_line(m, L, i, gold, a, c, o);
            if (start == 3) {
                // the pre-stall lift serves the estimate and the residual alike
                const double est = L.half_chord * o.ul * (m.include_viscous_lift ? o.cl_pre + o.cl_post : o.cl_pre);
                const double d = est - gold;
                const double gnew = fma(st.damping, d, gold);
                store_all(G(cur ^ 1), i, split_f64_int(gnew));
                // |d| >= tolerance, as integers (the FP64 pipe takes a compare like an add); not for a NaN
                const long long db = __double_as_longlong(d) & 0x7FFFFFFFFFFFFFFFll;
                if (want_max && db >= __double_as_longlong(st.strength_tolerance) && db <= 0x7FF0000000000000ll) r = -r;
                const int kk = RPT == 1 ? 0 : k;
                gown[kk] = gnew;
                a_last[kk] = a;
                c_last[kk] = c;
                est_last[kk] = est;
            }
            store_all(RR(it & 1), i, r);
        }
        if (start == 3) {
            it += 1;
            cur ^= 1;
            barrier();
            continue;
        }
        barrier();
        if (warp == 0) {
            double s = 0.0;
            unsigned long long mx = 0;
#pragma unroll 1
            for (int i = lane; i < N; i += 32) {
                s += RR(0)[i];
                const unsigned long long bi = mag_bits(RR(0)[i]);
                mx = bi > mx ? bi : mx;
            }
            s = warp_sum_to_lane0(s);
            mx = warp_umax_to_lane0(mx);
            if (lane == 0) {
                s_res = s;
                s_umax = mx;
            }
        }
        __syncthreads();
        const double rv = s_res, rmax = bits_value(s_umax), margin = start == 2 ? b.second_margin : 1.0;
        if (start == 0) {
            best = rv;
            best_max = rmax;
        } else if (isfinite(rv) && rv < margin * best && rmax < margin * best_max) {  // same decision in every CTA
            best = rv;
            best_max = rmax;
            taken = start;
            for (int i = tid; i < N; i += kSolveCtaThreads) G(0)[i] = G(1)[i];
            for (int k = 0; k < nrows; ++k) gown[k] = src[r0 + own_row(k)];
        }
        barrier();  // RR[0] and G[1] are written again by the next pass or the first iteration
        ++start;
    }

    // final circulation from the last velocities (simple_iterative.rs:200-203)
    for (int k = 0; k < nrows; ++k) {
        const int i = r0 + own_row(k);
        const double gam = est_last[k];
        b.gamma_prev[i] = gam;
        b.vel_out[i] = m.solve_basis[2 * i] * a_last[k] + m.solve_basis[2 * i + 1] * c_last[k];
        if (b.wake_str_row0) b.wake_str_row0[i] = gam;
        if (b.rec32_row0) b.rec32_row0[i].v[kRec32Gamma] = static_cast<float>(gam);
        if (b.rec64_row0) b.rec64_row0[i].v[kRec64Gamma] = gam;
    }
    if (rank == 0 && tid == 0) {
        b.scalars[0] = residual / static_cast<double>(N);
        b.scalars[1] = static_cast<double>(it);
        b.scalars[2] = conv ? 1.0 : 0.0;
        b.scalars[4] = static_cast<double>(taken);
    }
    // a copy whose wait ran out may still be in flight: wait for it (bounded) before leaving
    if (copier)
        for (int q = 0; q < 2; ++q)
            if (pending[q]) mbar_wait_bounded(&s_mbar[q], mph[q] ^ 1u, b.err);
    barrier();  // no CTA leaves while others may still write into its shared memory
}

template <int RPT, int NC, bool LO>
__global__ void __launch_bounds__(kSolveCtaThreads, 1) k_solve_si(DevModel m, SolveSettings st, SolveBuffers b) {
    si_solve<RPT, NC, LO>(m, st, b);
}

// Every case of a batch whose cluster size and variant are this launch's: cluster i solves jobs[i].
template <int RPT, int NC, bool LO>
__global__ void __launch_bounds__(kSolveCtaThreads, RPT == 1 ? 2 : 1) k_solve_si_jobs(const SolveJob* jobs) {
    cg::cluster_group cl = cg::this_cluster();
    const SolveJob& j = jobs[blockIdx.x / cl.num_blocks()];
    si_solve<RPT, NC, LO>(j.m, j.st, j.b);
}

namespace {

using SiKernel = void (*)(DevModel, SolveSettings, SolveBuffers);
using SiJobsKernel = void (*)(const SolveJob*);

// f(kernel pair) of the variant (rows per thread, components, lo plane)
template <int RPT, int NC, bool LO>
struct SiVariant {
    static SiKernel one() { return k_solve_si<RPT, NC, LO>; }
    static SiJobsKernel jobs() { return k_solve_si_jobs<RPT, NC, LO>; }
};
template <class F>
auto si_variant(int rpt, int comps, int full, F&& f) {
    if (rpt == 1) {
        if (comps == 2) return full ? f(SiVariant<1, 2, true>()) : f(SiVariant<1, 2, false>());
        return full ? f(SiVariant<1, 3, true>()) : f(SiVariant<1, 3, false>());
    }
    if (comps == 2) return full ? f(SiVariant<kSolveRowsPerThread, 2, true>()) : f(SiVariant<kSolveRowsPerThread, 2, false>());
    return full ? f(SiVariant<kSolveRowsPerThread, 3, true>()) : f(SiVariant<kSolveRowsPerThread, 3, false>());
}

void si_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, int clusters, int CS, size_t smem, cudaStream_t s) {
    cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * CS), 1, 1);
    cfg.blockDim = dim3(kSolveCtaThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(CS);
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

// Raises the kernels' shared-memory limit and allows clusters of 16, once per device; the
// largest cluster size the device can hold with kSiSmemSingle bytes per CTA.
int si_largest_cluster() {
    static std::mutex mu;
    static std::map<int, int> largest;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 8;
    std::lock_guard<std::mutex> lk(mu);
    auto it = largest.find(dev);
    if (it != largest.end()) return it->second;
    auto prepare = [](auto kernel) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSiSmemSingle)) ==
                   cudaSuccess &&
               cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    };
    bool ok = true;
    for (int rpt : {1, kSolveRowsPerThread})
        for (int comps : {2, 3})
            for (int full : {0, 1})
                ok = ok && si_variant(rpt, comps, full, [&](auto v) { return prepare(v.one()) && prepare(v.jobs()); });
    int c = ok ? kMaxCluster : 8;
    for (; c > 8; c /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        si_config(cfg, attr, 1, c, kSiSmemSingle, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_solve_si<1, 2, true>, &cfg) == cudaSuccess && n > 0) break;
    }
    (void)cudaGetLastError();  // a refused shape is not an error of the caller
    largest[dev] = c;
    return c;
}

}  // namespace

// One case alone: the cluster that ends its iterations soonest. Measured per iteration (us, the
// dynamic two-component matrix; clusters of 1, 4, 8, 16): N = 32: 4.19 / 4.47 / 4.53 / 4.75,
// 60: 4.93 / 4.65 / 4.61 / 4.81, 128: 7.49 / 5.03 / 4.83 / 5.02, 183: 18.2 / 6.22 / 5.35 / 5.19,
// 256: 25.9 / 7.07 / 5.71 / 5.37, 1024: 263 / 80.1 / 41.4 / 22.6. Each crowding level halves it, down to
// the size whose CTAs keep their matrix slab in shared memory two to an SM: with more cases than
// SMs their sum of CTA time counts (N = 128: 4 CTAs x 5.03 us against 8 x 4.83).
int solve_cluster_size(int N, int crowding) {
    const int alone = N <= 48 ? 1 : (N <= 160 ? 8 : 16), least = N <= 64 ? 1 : (N <= 256 ? 4 : 8);
    return std::min(std::max(alone >> crowding, least), si_largest_cluster());
}

SiPlan si_plan(int N, int full, int comps, int cluster, size_t smem_limit) {
    SiPlan p;
    p.cluster = cluster;
    const int rp = (N + cluster - 1) / cluster;
    p.rows_per_thread = rp <= kSolveThreads ? 1 : kSolveRowsPerThread;
    const long long off = si_slab_offset(N, cluster) * 8, rowb = si_row_bytes(N, full, comps);
    const long long budget = static_cast<long long>(smem_limit) - off;
    const long long r = budget / (2 * rowb);
    if (rp * rowb <= budget) {
        p.slab_rows = rp;
        p.smem = static_cast<size_t>(off + rp * rowb);
    } else {
        p.slab_rows = r < 4 ? 0 : static_cast<int>(std::min<long long>(r, 16));
        p.smem = static_cast<size_t>(off + 2 * p.slab_rows * rowb);
    }
    // Lanes per row: the fewest instructions of a warp over a chunk's rows, a step of four columns
    // being about 22 per component and a row's butterfly 14 per level
    const int at_once = p.slab_rows > 0 ? std::min(p.slab_rows, rp) : rp;
    long long best = 0;
    for (int l = 3; l <= 5; ++l) {
        const long long rows = kSolveThreads >> l, passes = (at_once + rows - 1) / rows;
        const long long cost = passes * ((si_matrix_stride(N) + (4 << l) - 1) / (4 << l) * 22 * comps + 14 * l + 60);
        if (l == 3 || cost < best) {
            best = cost;
            p.lanes_log2 = l;
        }
    }
    return p;
}

cudaError_t launch_solve_simple_iterative_jobs(const SolveJob* jobs, int n, int cluster, int rows_per_thread, int comps,
                                               int full, size_t smem, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (cluster < 1 || cluster > si_largest_cluster() || smem > kSiSmemSingle) return cudaErrorInvalidValue;
    if (rows_per_thread != 1 && rows_per_thread != kSolveRowsPerThread) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    si_config(cfg, attr, n, cluster, smem, s);
    return cudaLaunchKernelEx(&cfg, si_variant(rows_per_thread, comps, full, [](auto v) { return v.jobs(); }), jobs);
}

cudaError_t launch_solve_simple_iterative(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, cudaStream_t s) {
    const SiPlan p = si_plan(m.N, b.split_full, b.split_comps, solve_cluster_size(m.N, 0), kSiSmemSingle);
    if ((m.N + p.cluster - 1) / p.cluster > kSolveThreads * kSolveRowsPerThread) return cudaErrorInvalidValue;
    SolveBuffers sb = b;
    sb.slab_rows = p.slab_rows;
    sb.lanes_log2 = p.lanes_log2;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    si_config(cfg, attr, 1, p.cluster, p.smem, s);
    return cudaLaunchKernelEx(&cfg, si_variant(p.rows_per_thread, b.split_comps, b.split_full, [](auto v) { return v.one(); }),
                              m, st, sb);
}

// ---------------------------------------------------------------------------------------
// Linearized solver: one CTA per case (one case, or every case of a batch in one launch)
// ---------------------------------------------------------------------------------------
constexpr int kLinThreads = 512;
constexpr int kLinMaxCluster = 16;  // non-portable cluster size (16 SMs of one GPC)

// Per case in shared memory: control-point velocities, induced velocities and the
// circulation, then the augmented matrix [N][N+1] when it fits in what the launch gave.
__host__ __device__ inline size_t lin_vec_bytes(int N) {
    return static_cast<size_t>(N) * (2 * sizeof(d3) + sizeof(double));
}
__host__ __device__ inline size_t lin_mat_bytes(int N) { return static_cast<size_t>(N) * (N + 1) * sizeof(double); }

// Cluster of C CTAs: the vectors, the pivot row, the row permutation and its inverse, and
// the CTA's share of rows ((N + C - 1) / C rows of N + 1 values).
__host__ __device__ inline size_t lin_cluster_bytes(int N, int C) {
    const size_t W1 = static_cast<size_t>(N) + 1;
    return lin_vec_bytes(N) + W1 * sizeof(double) + 2 * static_cast<size_t>(N) * sizeof(int) +
           static_cast<size_t>((N + C - 1) / C) * W1 * sizeof(double);
}

// One row of the linearized system (linearized.rs:61-136): the velocity with the fixed part
// and the span component removed, the coefficients row[0..N-1] and the right-hand side row[N].
__device__ inline void lin_build_row(const DevModel& m, const SolveBuffers& b, int i, double* row) {
    const int N = m.N;
    RowGeom g = row_geom(m, i);
    d3 v = g.felt + b.fixed[i];
    v = v - g.span_dir * dot(v, g.span_dir);  // project(v, span_rel)
    d3 un = normalize(v);
    const d3 sd = g.span_dir;
    d3 nd = cross(un, sd);
    double aoa = len(v) > kMinPositive ? signed_angle_between(g.chord, v, g.span_dir) : 0.0;
    const FoilP f = m.foils[g.wing];
    double cll = foil_cl_linear(f, aoa);
    double ut = dot(v, un);
    double dcl = f.cl_initial_slope;
    for (int c = 0; c < N; ++c) {
        double uin = dot(b.factors[static_cast<long long>(i) * N + c], nd);
        double a = -dcl * uin / ut;
        if (i == c) a += 2.0 / (g.chord_len * ut);
        row[c] = a;
    }
    row[N] = -cll;
}

// After the solve, on one CTA: induced and total velocities, the viscous correction, the
// residual and the outputs (linearized.rs:141-213).
__device__ void lin_finish(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, d3* vel, d3* ind,
                           double* gam) {
    const int N = m.N, tid = threadIdx.x, nt = blockDim.x;
    // induced velocity and the total velocity (linearized.rs:141-156)
    auto update_induced = [&]() {
        for (int i = tid; i < N; i += nt) {
            double sx = 0.0, sy = 0.0, sz = 0.0;
            for (int c = 0; c < N; ++c) {
                d3 f = b.factors[static_cast<long long>(i) * N + c];
                sx += f.x * gam[c];
                sy += f.y * gam[c];
                sz += f.z * gam[c];
            }
            d3 fx = b.fixed[i];
            ind[i] = mk(fx.x + sx, fx.y + sy, fx.z + sz);
        }
        __syncthreads();
    };
    update_induced();
    for (int i = tid; i < N; i += nt) vel[i] = total_velocity(st, m.felt_ctrl[i], ind[i]);
    __syncthreads();
    // viscous correction (linearized.rs:158-202)
    if (!st.disable_viscous_corrections) {
        for (int i = tid; i < N; i += nt) {
            RowGeom g = row_geom(m, i);
            const FoilP f = m.foils[g.wing];
            double aoa = len(vel[i]) > kMinPositive ? signed_angle_between(g.chord, vel[i], g.span_dir) : 0.0;
            double cll = foil_cl_linear(f, aoa);
            double clf = foil_cl_pre_stall(f, aoa);
            if (fabs(cll) > kMinPositive) gam[i] *= clf / cll;
        }
        __syncthreads();
        if (st.full_induced_correction) update_induced();
        for (int i = tid; i < N; i += nt) vel[i] = total_velocity(st, m.felt_ctrl[i], ind[i]);
        __syncthreads();
    }
    // residual (linearized.rs:204-213): the terms in parallel (into the induced-velocity
    // storage, no longer needed), summed in control-point order by one thread
    double* terms = reinterpret_cast<double*>(ind);
    for (int i = tid; i < N; i += nt) {
        RowGeom g = row_geom(m, i);
        const FoilP f = m.foils[g.wing];
        double aoa = len(vel[i]) > kMinPositive ? signed_angle_between(g.chord, vel[i], g.span_dir) : 0.0;
        terms[i] = residual_term(m, g, f, gam[i], vel[i], aoa);
    }
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int i = 0; i < N; ++i) s += terms[i];
        b.scalars[0] = s / static_cast<double>(N);
        b.scalars[1] = 1.0;
        b.scalars[2] = 1.0;
    }
    for (int i = tid; i < N; i += nt) {
        b.gamma_prev[i] = gam[i];
        b.vel_out[i] = vel[i];
        if (b.wake_str_row0) b.wake_str_row0[i] = gam[i];
        if (b.rec32_row0) b.rec32_row0[i].v[kRec32Gamma] = static_cast<float>(gam[i]);
        if (b.rec64_row0) b.rec64_row0[i].v[kRec64Gamma] = gam[i];
    }
}

// Linearized::solve (linearized.rs:54-222) for one case on the calling CTA. The Gaussian
// elimination (linalg.rs:41-103) keeps the reference's arithmetic per element: the pivot is
// the first row of largest |A[i][k]| (warp 0: per-lane scan, then a butterfly on (value,
// lowest index)); row i -= (A[i][k] / pivot) * row k over columns k..N (a warp per row);
// back substitution by warp 0, one row at a time. Where the matrix lives (shared memory or
// the case's global scratch) does not change any result.
__device__ void lin_solve_case(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, unsigned char* dyn,
                               size_t dyn_bytes) {
    const int N = m.N, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int W1 = N + 1;
    d3* vel = reinterpret_cast<d3*>(dyn);                 // [N]
    d3* ind = vel + N;                                    // [N]
    double* gam = reinterpret_cast<double*>(ind + N);     // [N]
    double* A = lin_vec_bytes(N) + lin_mat_bytes(N) <= dyn_bytes ? gam + N : b.lin_work;  // [N][N+1]
    __shared__ int s_piv;
    if (b.scalars[5] != 0.0) return;  // solved by k_lin_refined

    for (int i = tid; i < N; i += nt) lin_build_row(m, b, i, A + static_cast<long long>(i) * W1);
    __syncthreads();
    // forward elimination with partial pivoting
    for (int k = 0; k < N; ++k) {
        double* Ak = A + static_cast<long long>(k) * W1;
        if (warp == 0) {
            double bv = -1.0;
            int bi = N;
            for (int i = k + lane; i < N; i += 32) {
                const double v = fabs(A[static_cast<long long>(i) * W1 + k]);
                if (v > bv) {
                    bv = v;
                    bi = i;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            if (lane == 0) s_piv = bi < N ? bi : k;
        }
        __syncthreads();
        const int mr = s_piv;
        if (mr != k) {
            double* Am = A + static_cast<long long>(mr) * W1;
            for (int j = tid; j <= N; j += nt) {
                const double t = Ak[j];
                Ak[j] = Am[j];
                Am[j] = t;
            }
        }
        __syncthreads();
        const double piv = Ak[k];
        if (fabs(piv) < 1e-12) {  // the same value in every thread: the whole CTA leaves
            if (tid == 0) {
                atomicExch(b.err, kDevSingular);
                b.scalars[3] = 1.0;
            }
            return;
        }
        for (int i = k + 1 + warp; i < N; i += nw) {
            double* Ai = A + static_cast<long long>(i) * W1;
            const double f = Ai[k] / piv;
            __syncwarp();  // every lane has read A[i][k] before lane 0 overwrites it
            for (int j = k + lane; j <= N; j += 32) Ai[j] -= f * Ak[j];
        }
        __syncthreads();
    }
    // back substitution
    if (warp == 0) {
        for (int i = N - 1; i >= 0; --i) {
            const double* Ai = A + static_cast<long long>(i) * W1;
            double part = 0.0;
            for (int j = i + 1 + lane; j < N; j += 32) part += Ai[j] * gam[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) gam[i] = (Ai[N] - part) / Ai[i];
            __syncwarp();
        }
    }
    __syncthreads();
    lin_finish(m, st, b, vel, ind, gam);
}

__global__ void __launch_bounds__(kLinThreads) k_solve_lin(DevModel m, SolveSettings st, SolveBuffers b, unsigned smem) {
    extern __shared__ __align__(16) unsigned char lin_dyn[];
    lin_solve_case(m, st, b, lin_dyn, smem);
}

// Every case of a batch in one launch: CTA i solves jobs[i].
__global__ void __launch_bounds__(kLinThreads) k_solve_lin_jobs(const SolveJob* jobs, unsigned smem) {
    extern __shared__ __align__(16) unsigned char lin_dyn[];
    const SolveJob& j = jobs[blockIdx.x];
    lin_solve_case(j.m, j.st, j.b, lin_dyn, smem);
}

// Linearized::solve for a system whose matrix does not fit one CTA's shared memory, on a
// thread-block cluster of C CTAs: physical row r lives in the shared memory of CTA r mod C
// (row r / C there). Row exchanges are kept as a permutation held by every CTA (at[k] =
// physical row at position k, pos[r] its inverse), so rows never move. Per column k, one
// cluster barrier: each CTA's warp 0 has put its candidate for column k (the rows at
// positions >= k: largest |A[r][k]|, then lowest position, i.e. the reference's first
// largest row after its swaps) into a double-buffered slot; after the barrier every CTA
// reduces the C candidates (one per lane, the same butterfly), applies the same exchange
// to its permutation,
// copies the pivot row (columns k..N; a pivot row never changes again) through distributed
// shared memory, eliminates its own rows at positions > k with lin_solve_case's per-element
// arithmetic, and posts its candidate for column k + 1. Back substitution runs on CTA 0,
// reading each pivot row from its owner as lin_solve_case reads it (warp 0, lane-strided
// sum, butterfly), while the other CTAs wait at the final barrier. CTA 0 then finishes the
// solve. The result is bit-identical to lin_solve_case; all waits are cluster barriers.
__device__ void lin_solve_cluster(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, unsigned char* dyn) {
    cg::cluster_group cl = cg::this_cluster();
    const int C = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    const int N = m.N, W1 = N + 1, R = (N + C - 1) / C;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    d3* vel = reinterpret_cast<d3*>(dyn);              // [N] (CTA 0)
    d3* ind = vel + N;                                 // [N] (CTA 0)
    double* gam = reinterpret_cast<double*>(ind + N);  // [N] (CTA 0)
    double* prow = gam + N;                            // [N + 1] pivot row of the current column
    int* at = reinterpret_cast<int*>(prow + W1);       // [N] physical row at each position
    int* pos = at + N;                                 // [N] position of each physical row
    double* A = reinterpret_cast<double*>(pos + N);    // [R][N + 1] rows rank, rank + C, ...
    __shared__ double s_cand_v[2];
    __shared__ int s_cand_p[2], s_piv;
    if (b.scalars[5] != 0.0) return;  // solved by k_lin_refined (the same value in every CTA)

    // the candidate of this CTA for column k: first largest |A[r][k]| over its rows at
    // positions >= k (lowest position among equal values), into slot k & 1
    auto post_candidate = [&](int k) {
        double bv = -1.0;
        int bp = N;
        for (int l = lane; l < R; l += 32) {
            const int r = rank + l * C;
            if (r >= N) break;
            const int p = pos[r];
            if (p < k) continue;
            const double v = fabs(A[static_cast<long long>(l) * W1 + k]);
            if (v > bv || (v == bv && p < bp)) {
                bv = v;
                bp = p;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int op = __shfl_xor_sync(0xffffffffu, bp, o);
            if (ov > bv || (ov == bv && op < bp)) {
                bv = ov;
                bp = op;
            }
        }
        if (lane == 0) {
            s_cand_v[k & 1] = bv;
            s_cand_p[k & 1] = bp;
        }
    };

    for (int i = tid; i < N; i += nt) {
        at[i] = i;
        pos[i] = i;
    }
    for (int l = tid; l < R; l += nt) {
        const int r = rank + l * C;
        if (r < N) lin_build_row(m, b, r, A + static_cast<long long>(l) * W1);
    }
    __syncthreads();
    if (warp == 0) post_candidate(0);
    for (int k = 0; k < N; ++k) {
        cl.sync();  // every CTA's candidate for column k is posted; column k of every row is final
        if (warp == 0) {  // lane q reads CTA q's candidate; the same butterfly as post_candidate
            double bv = -1.0;
            int bp = N;
            if (lane < C) {
                bv = *cl.map_shared_rank(&s_cand_v[k & 1], lane);
                bp = *cl.map_shared_rank(&s_cand_p[k & 1], lane);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int op = __shfl_xor_sync(0xffffffffu, bp, o);
                if (ov > bv || (ov == bv && op < bp)) {
                    bv = ov;
                    bp = op;
                }
            }
            if (lane == 0) {  // the cluster's first largest row: apply the exchange
                const int mr = bp < N ? bp : k;  // position of the pivot row
                const int rk = at[k], rm = at[mr];
                at[k] = rm;
                at[mr] = rk;
                pos[rm] = k;
                pos[rk] = mr;
                s_piv = rm;
            }
        }
        __syncthreads();
        const int pr = s_piv;  // physical pivot row
        {
            const double* src = cl.map_shared_rank(A, pr % C) + static_cast<long long>(pr / C) * W1;
            for (int j = k + tid; j <= N; j += nt) prow[j] = src[j];
        }
        __syncthreads();
        const double piv = prow[k];
        if (fabs(piv) < 1e-12) {  // the same value in every CTA: the whole cluster leaves
            if (rank == 0 && tid == 0) {
                atomicExch(b.err, kDevSingular);
                b.scalars[3] = 1.0;
            }
            cl.sync();  // no CTA leaves while another may still read its rows
            return;
        }
        for (int l = warp; l < R; l += nw) {
            const int r = rank + l * C;
            if (r >= N) break;
            if (pos[r] <= k) continue;
            double* Ai = A + static_cast<long long>(l) * W1;
            const double f = Ai[k] / piv;
            __syncwarp();  // every lane has read A[i][k] before lane 0 overwrites it
            for (int j = k + lane; j <= N; j += 32) Ai[j] -= f * prow[j];
        }
        __syncthreads();
        if (warp == 0 && k + 1 < N) post_candidate(k + 1);
    }
    cl.sync();  // every row is final
    if (rank == 0) {
        if (warp == 0) {
            for (int i = N - 1; i >= 0; --i) {
                const int r = at[i];
                const double* Ai = cl.map_shared_rank(A, r % C) + static_cast<long long>(r / C) * W1;
                double part = 0.0;
                for (int j = i + 1 + lane; j < N; j += 32) part += Ai[j] * gam[j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                if (lane == 0) gam[i] = (Ai[N] - part) / Ai[i];
                __syncwarp();
            }
        }
        __syncthreads();
    }
    cl.sync();  // CTA 0 has read every row it needs
    if (rank == 0) lin_finish(m, st, b, vel, ind, gam);
}

__global__ void __launch_bounds__(kLinThreads) k_solve_lin_cluster(DevModel m, SolveSettings st, SolveBuffers b) {
    extern __shared__ __align__(16) unsigned char lin_dyn[];
    lin_solve_cluster(m, st, b, lin_dyn);
}

// Every case of a batch that needs a cluster of this launch's size: cluster i solves jobs[i].
__global__ void __launch_bounds__(kLinThreads) k_solve_lin_cluster_jobs(const SolveJob* jobs) {
    extern __shared__ __align__(16) unsigned char lin_dyn[];
    cg::cluster_group cl = cg::this_cluster();
    const SolveJob& j = jobs[blockIdx.x / cl.num_blocks()];
    lin_solve_cluster(j.m, j.st, j.b, lin_dyn);
}

namespace {

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, int clusters, int C, size_t smem, cudaStream_t s) {
    cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * C), 1, 1);
    cfg.blockDim = dim3(kLinThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(C);
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
}

template <class K>
cudaError_t prepare_cluster_kernel(K kernel, int C, size_t smem) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e == cudaSuccess && C > 8) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

// Whether clusters of C CTAs with `smem` bytes of shared memory each can be resident on the
// current device (cached per device and shape).
bool cluster_fits(int C, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, size_t>, bool> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(dev, C, smem);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    bool ok = prepare_cluster_kernel(k_solve_lin_cluster, C, smem) == cudaSuccess &&
              prepare_cluster_kernel(k_solve_lin_cluster_jobs, C, smem) == cudaSuccess;
    if (ok) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        cluster_config(cfg, attr, 1, C, smem, nullptr);
        int n = 0;
        ok = cudaOccupancyMaxActiveClusters(&n, k_solve_lin_cluster, &cfg) == cudaSuccess && n > 0;
    }
    if (!ok) (void)cudaGetLastError();  // a refused shape is not an error of the caller
    cache[key] = ok;
    return ok;
}

}  // namespace

LinPlan linearized_plan(int N) {
    const size_t v = lin_vec_bytes(N), a = lin_mat_bytes(N);
    if (v + a <= kLinSmemLimit) return {1, v + a};
    for (int C = 2; C <= kLinMaxCluster; C *= 2) {
        const size_t bytes = lin_cluster_bytes(N, C);
        if (bytes <= kLinSmemLimit && cluster_fits(C, bytes)) return {C, bytes};
    }
    return {1, v};  // matrix in the case's global scratch
}

int linearized_launches(int N, const SolveSettings& st) {
    return 1 + (linearized_refined_plan(N, 0).cluster > 0 ? linearized_refined_launches(N, st) : 0);
}

cudaError_t launch_solve_linearized(const DevModel& m, const SolveSettings& st, const SolveBuffers& b, cudaStream_t s) {
    const LinPlan refined = linearized_refined_plan(m.N, 0);
    if (refined.cluster > 0) {
        const cudaError_t e = launch_solve_linearized_refined(m, st, b, refined, s);
        if (e != cudaSuccess) return e;
    }
    const LinPlan p = linearized_plan(m.N);
    if (p.cluster == 1) {
        if (p.smem > 48 * 1024) {
            cudaError_t e =
                cudaFuncSetAttribute(k_solve_lin, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(p.smem));
            if (e != cudaSuccess) return e;
        }
        k_solve_lin<<<1, kLinThreads, p.smem, s>>>(m, st, b, static_cast<unsigned>(p.smem));
        return cudaGetLastError();
    }
    cudaError_t e = prepare_cluster_kernel(k_solve_lin_cluster, p.cluster, p.smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(cfg, attr, 1, p.cluster, p.smem, s);
    return cudaLaunchKernelEx(&cfg, k_solve_lin_cluster, m, st, b);
}

cudaError_t launch_solve_linearized_jobs(const SolveJob* jobs, int n, const LinPlan& plan, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    if (plan.smem > kLinSmemLimit) return cudaErrorInvalidValue;
    if (plan.cluster == 1) {
        if (plan.smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(k_solve_lin_jobs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 static_cast<int>(plan.smem));
            if (e != cudaSuccess) return e;
        }
        k_solve_lin_jobs<<<n, kLinThreads, plan.smem, s>>>(jobs, static_cast<unsigned>(plan.smem));
        return cudaGetLastError();
    }
    cudaError_t e = prepare_cluster_kernel(k_solve_lin_cluster_jobs, plan.cluster, plan.smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    cluster_config(cfg, attr, n, plan.cluster, plan.smem, s);
    return cudaLaunchKernelEx(&cfg, k_solve_lin_cluster_jobs, jobs);
}

}  // namespace sbgpu
