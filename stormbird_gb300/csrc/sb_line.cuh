// Lift and drag of a span line at a velocity (sm_103a), f64, with the elementary functions of
// sb_f64.cuh: the angle of attack of force_calculations.rs:79-107 and the Foil section model of
// stormbird/src/section_models/foil.rs. Rare arguments (no velocity or chord, a high-order lift term,
// exponents outside the tables) go through sb_device.cuh's functions, out of line.
#pragma once

#include "sb_f64.cuh"

namespace sbgpu {

// Angle in [0, pi] from its cosine and sine (c^2 + s^2 = 1 to rounding, s >= 0)
__device__ __forceinline__ double angle_f64(double c, double s, const double* tab) {
    float a;
    const double* e = angle_entry(f64_to_f32(c), f64_to_f32(s), tab, a);
    return e[2] + arcsin_f64(fma(s, e[0], -(c * e[1])));
}

// 1 / (1 + exp(-(slope (|e| - mean)))) (foil.rs:256-270) at e = angle + angle_cd_min
static __device__ __noinline__ double stall_slow(const FoilP& f, double e) {
    const double mean = e >= 0.0 ? fabs(f.mean_positive_stall_angle) : fabs(f.mean_negative_stall_angle);
    return sigmoid_zero_to_one_slope(fabs(e), mean, f.stall_slope);
}
__device__ __forceinline__ double stall_f64(const FoilP& f, double e, const double* tab) {
    const double mean = fabs(__double2hiint(e) >= 0 ? f.mean_positive_stall_angle : f.mean_negative_stall_angle);
    const double w = (f.stall_slope * 738.6598609351493) * (mean - fabs(e));  // 512 / ln 2
    // |w| >= 32000, infinite or no number, from the high word: the FP32 copy is good only below 2^128 (a stall
    // range of 0 has an infinite slope)
    if ((static_cast<unsigned>(__double2hiint(w)) & 0x7FFFFFFFu) >= 0x40DF4000u) return w < 0.0 ? 1.0 : stall_slow(f, e);
    const float n = rintf(f64_to_f32(w));
    return rcp_f64(1.0 + exp2_512_f64(static_cast<int>(n), w - f32_to_f64(n), tab));
}

// x^p for x in [0, 1]: log2 x from 2^(j/512), j the nearest, and the series of the rest
// (|r| <= 6.8e-4, next term below 3e-17), then exp2_512_f64 (n >= -512 * 960: x >= 2^-60, p <= 16).
static __device__ __noinline__ double pow_slow(double x, double p) { return pow(x, p); }
__device__ __forceinline__ double pow_f64(double x, double p, const double* tab) {
    const int hi = __double2hiint(x), k = (hi >> 20) - 1023;
    if (!f64_normal_positive(x) || k < -60 || k > 0 || !(p >= 0.0 && p <= 16.0)) return pow_slow(x, p);
    const double m = __hiloint2double(hi - (k << 20), __double2loint(x));  // [1, 2)
    const int j = __float2int_rn(log2f(f64_to_f32(m)) * 512.f);            // 0..512
    // m 2^(-j/512): the table holds 2^(i/512) for i < 512
    const double r = j == 0 ? m - 1.0 : fma(m, 0.5 * tab[3 * 129 + 512 - j], -1.0);
    const double l = r * fma(r, fma(r, fma(r, -0.25, 1.0 / 3.0), -0.5), 1.0);
    const double w = fma(p, f32_to_f64(static_cast<float>(512 * k + j)), (p * 738.6598609351493) * l);
    const float n = rintf(f64_to_f32(w));
    return exp2_512_f64(static_cast<int>(n), w - f32_to_f64(n), tab);
}

struct LineLift {
    double aoa;         // angle of attack, [-pi, pi]
    double sn, cs;      // its sine and cosine
    double stall;       // foil_amount_of_stall
    double cl_linear, cl_pre, cl_post;
};

static __device__ __noinline__ void line_lift_slow(const FoilP& f, d3 chord, d3 v, d3 span_dir, LineLift& o) {
    o.aoa = len(v) > kMinPositive ? signed_angle_between(chord, v, span_dir) : 0.0;
    o.sn = sin(o.aoa);
    o.cs = cos(o.aoa);
    o.stall = foil_amount_of_stall(f, o.aoa);
    o.cl_linear = foil_cl_linear(f, o.aoa);
    o.cl_pre = foil_cl_pre_stall(f, o.aoa);
    o.cl_post = foil_cl_post_stall(f, o.aoa);
}

// signed_angle_between(chord, v, span_dir) (vector_math.rs:65-95) from the cosine and the sine
// (|chord x v|), and the foil's lift at it.
__device__ __forceinline__ LineLift line_lift(const FoilP& f, d3 chord, d3 v, d3 span_dir, const double* tab) {
    LineLift o;
    const double cc = len2(chord), vv = len2(v);
    if (!f64_seed_range(cc) || !f64_seed_range(vv) || f.cl_high_order_power > 0.0) {
        line_lift_slow(f, chord, v, span_dir, o);
        return o;
    }
    const double r = rsqrt_f64(cc) * rsqrt_f64(vv);
    const d3 x = cross(chord, v);
    o.cs = dot(chord, v) * r;
    const double s = sqrt_any(len2(x)) * r;
    const bool pos = f64_positive(dot(chord, cross(v, span_dir)));
    const double ang = angle_f64(o.cs, s, tab);
    o.aoa = pos ? ang : -ang;
    o.sn = pos ? s : -s;
    o.stall = stall_f64(f, o.aoa + f.angle_cd_min, tab);
    o.cl_linear = fma(f.cl_initial_slope, o.sn, f.cl_zero_angle);
    o.cl_pre = fma(-o.cl_linear, o.stall, o.cl_linear);
    o.cl_post = f.cl_max_after_stall * (2.0 * o.sn * o.cs) * o.stall;  // sin 2a, |a| <= pi
    return o;
}

// The foil's drag coefficient (foil.rs:212-243) at the lift's angle
static __device__ __noinline__ double cd_bump(double amount, double s) { return amount * ((1.0 - cos(s * kTau)) * 0.5); }
__device__ __forceinline__ double line_drag(const FoilP& f, const LineLift& o, const double* tab) {
    const double eff = fabs(o.aoa + f.angle_cd_min);
    const double pre = f.cd_min + f.cd_second_order_factor * (eff * eff);
    const double post = f.cd_max_after_stall * pow_f64(fabs(o.sn), f.cd_power_after_stall, tab);
    const double s = f.cd_stall_angle_offset == 0.0
                         ? o.stall
                         : stall_f64(f, o.aoa + f.cd_stall_angle_offset * signum(o.aoa) + f.angle_cd_min, tab);
    const double raw = pre * (1.0 - s) + s * post;
    const double cl = o.cl_post + o.cl_pre;
    return raw + f.cdi_correction_factor * (cl * cl) + (f.cd_bump_during_stall != 0.0 ? cd_bump(f.cd_bump_during_stall, s) : 0.0);
}

}  // namespace sbgpu
