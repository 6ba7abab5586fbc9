// f64 elementary functions for the per-line math (sm_103a), made for few FP64 instructions.
//
// A warp issues an FP64 instruction every 62 to 65 cycles, whatever the active lanes, independent or
// not (four independent DFMAs: 261 cycles; the SM's one pipe takes one per 19 from four or more warps), and a
// conversion between f64 and FP32 as long as a DFMA; CUDA's f64 division, square root, acos, sin and
// exp are chains of 9 to 22 of them (574 to 1,425 cycles measured, one warp). The functions here
// reach the same accuracy (an ulp or two) in 3 to 8 FP64 instructions:
//   * conversions on the integer pipe (a few 4-cycle instructions each);
//   * reciprocal and reciprocal square root: an FP32 seed (about 2^-22) and one third-order step
//     (Householder's method: with h = 1 - d y or 1 - q y^2, y (1 + h + h^2) or
//     y (1 + h/2 + 3 h^2/8)), error below h^3 = 2^-63 before rounding;
//   * an angle from its cosine and sine: the nearest table angle (picked in FP32), the rest from
//     sin(delta) = s cos(theta) - c sin(theta), |delta| <= pi/256, by the Taylor series of the
//     arcsine (next term below 2e-19);
//   * an exponential by Tang's table method (P. T. P. Tang, ACM TOMS 15 (1989) 144): the exponent in
//     units of ln 2 / 512, its integer part from a 512-entry table of 2^(j/512) and an exponent
//     shift, the rest (about ln 2 / 1024) from the Taylor series (next term below 4e-18);
//   * the parts of these series and steps whose FP32 rounding stays below 2^-60 of the result are
//     evaluated in FP32, and seeds and table entries come from an FP32 evaluation that runs beside
//     the FP64 one where the caller has it.
// Arguments outside the stated ranges are the caller's to keep on CUDA's functions.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace sbgpu {

#include "sb_f64_tables.inc"

constexpr int kF64TableDoubles = 3 * 129 + 512;

// Copies the tables into shared memory (kF64TableDoubles doubles), all threads of the CTA.
__device__ __forceinline__ void load_f64_tables(double* t, int tid, int nt) {
    for (int i = tid; i < 3 * 129; i += nt) t[i] = kAngleTable[i];
    for (int i = tid; i < 512; i += nt) t[3 * 129 + i] = kExp2Table[i];
}

// 2^-100 <= v < 2^100 (the seeds' range); false for zero, negative, infinite and NaN values.
__device__ __forceinline__ bool f64_seed_range(double v) {
    return static_cast<unsigned>(__double2hiint(v)) - 0x39B00000u < 0x0C800000u;
}
// The nearest float of v (ties away from zero) by integer arithmetic, for |v| in [2^-126, 2^128);
// all others give 0, infinities and no numbers too.
__device__ __forceinline__ float f64_to_f32(double v) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v));
    const unsigned lo = static_cast<unsigned>(__double2loint(v));
    const unsigned mag = (hi & 0x7FFFFFFFu) - 0x38000000u;  // exponent rebiased (wraps below 2^-127)
    const unsigned bits = __funnelshift_l(lo, mag, 3) + ((lo >> 28) & 1u);
    return __uint_as_float((mag - 0x00100000u < 0x0FE00000u ? bits : 0u) | (hi & 0x80000000u));
}
// The nearest float of v, ties to even (the conversion's own result), by integer arithmetic for 0 and
// |v| in [2^-126, 2^128); others through the conversion.
static __device__ __noinline__ float f64_to_f32_slow(double v) { return __double2float_rn(v); }
__device__ __forceinline__ float f64_to_f32_rn(double v) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v)), lo = static_cast<unsigned>(__double2loint(v));
    const unsigned mag = (hi & 0x7FFFFFFFu) - 0x38000000u;
    if (mag - 0x00100000u >= 0x0FE00000u) return ((hi & 0x7FFFFFFFu) | lo) == 0u ? __uint_as_float(hi) : f64_to_f32_slow(v);
    const unsigned bits = __funnelshift_l(lo, mag, 3);
    return __uint_as_float((bits + (((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (bits & 1u)) >> 29)) | (hi & 0x80000000u));
}
// v exactly, by integer arithmetic, for v finite; magnitudes below 2^-126 give a value below 2^-126, 0 too: not
// where a result of 0 counts.
__device__ __forceinline__ double f32_to_f64(float v) {
    const unsigned u = __float_as_uint(v), mag = u & 0x7FFFFFFFu;
    return __hiloint2double(static_cast<int>(((mag >> 3) + 0x38000000u) | (u & 0x80000000u)), static_cast<int>(u << 29));
}
// v exactly, whatever it is
static __device__ __noinline__ double f32_to_f64_slow(float v) { return static_cast<double>(v); }
__device__ __forceinline__ double f32_to_f64_exact(float v) {
    const unsigned u = __float_as_uint(v), mag = u & 0x7FFFFFFFu;
    if (mag - 0x00800000u >= 0x7F000000u) return mag == 0u ? __hiloint2double(static_cast<int>(u), 0) : f32_to_f64_slow(v);
    return f32_to_f64(v);
}
// f64 value as a pair of floats: hi = the nearest float, lo = the nearest float of v - hi
// (hi + lo carries about 48 significant bits)
__device__ inline float2 split_f64(double v) {
    const float h = __double2float_rn(v);
    return make_float2(h, __double2float_rn(v - static_cast<double>(h)));
}
// split_f64 with the conversions on the integer pipe where v allows
__device__ __forceinline__ float2 split_f64_int(double v) {
    const unsigned mag = static_cast<unsigned>(__double2hiint(v)) & 0x7FFFFFFFu;
    if (mag - 0x39B00000u >= 0x0C800000u) return split_f64(v);
    const float h = f64_to_f32(v);
    return make_float2(h, f64_to_f32(v - f32_to_f64(h)));
}
// FP32 seeds: the hardware approximations (within 2 ulp) of normal arguments
__device__ __forceinline__ float rcp_seed(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_seed(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// v > 0 on the integer pipe (a compare costs the FP64 pipe as much as an add)
__device__ __forceinline__ bool f64_positive(double v) { return __double_as_longlong(v) > 0; }
// Third-order step to 1 / d from a seed y within 2^-17: 3 FP64 instructions. Returns false where
// the seed was not that close (the caller then takes CUDA's division).
__device__ __forceinline__ bool rcp_step(double d, float seed, double& out) {
    const double y = f32_to_f64(seed);
    const double h = fma(-d, y, 1.0);
    const float hf = f64_to_f32(h);
    out = fma(y, h + f32_to_f64(hf * hf), y);
    return fabsf(hf) < 0x1p-17f;
}
// Third-order step to 1 / sqrt(q) from a seed y within 2^-18: 4 FP64 instructions.
__device__ __forceinline__ bool rsqrt_step(double q, float seed, double& out) {
    const double y = f32_to_f64(seed);
    const double h = fma(-(q * y), y, 1.0);
    const float hf = f64_to_f32(h);
    out = fma(y, fma(h, 0.5, f32_to_f64(0.375f * hf * hf)), y);
    return fabsf(hf) < 0x1p-17f;
}
// 1 / d and 1 / sqrt(q) for f64_seed_range arguments
__device__ __forceinline__ double rcp_f64(double d) {
    double r;
    rcp_step(d, rcp_seed(f64_to_f32(d)), r);
    return r;
}
__device__ __forceinline__ double rsqrt_f64(double q) {
    double r;
    rsqrt_step(q, rsqrt_seed(f64_to_f32(q)), r);
    return r;
}

// The same for any positive normal argument (the exponent is taken out of the seed and the step), by
// CUDA's functions for the others: out of line, so that the loops they appear in stay small.
static __device__ __noinline__ double sqrt_slow(double q) { return sqrt(q); }
static __device__ __noinline__ double rsqrt_slow(double q) { return 1.0 / sqrt(q); }
static __device__ __noinline__ double rcp_slow(double d) { return 1.0 / d; }
__device__ __forceinline__ bool f64_normal_positive(double v) {
    return static_cast<unsigned>(__double2hiint(v)) - 0x00100000u < 0x7FE00000u;
}
__device__ __forceinline__ double rsqrt_any(double q) {
    if (!f64_normal_positive(q)) return rsqrt_slow(q);
    const int hi = __double2hiint(q), e = ((hi >> 20) - 1023) >> 1;
    const double r = rsqrt_f64(__hiloint2double(hi - (e << 21), __double2loint(q)));  // [1, 4)
    return __hiloint2double(__double2hiint(r) - (e << 20), __double2loint(r));
}
__device__ __forceinline__ double sqrt_any(double q) { return f64_normal_positive(q) ? q * rsqrt_any(q) : sqrt_slow(q); }
__device__ __forceinline__ double rcp_any(double d) { return f64_seed_range(fabs(d)) ? copysign(rcp_f64(fabs(d)), d) : rcp_slow(d); }

// Entry (cos, sin, angle) of the angle table nearest to the angle of (x, y >= 0), in [0, pi].
__device__ __forceinline__ const double* angle_entry(float x, float y, const double* t, float& angle) {
    angle = atan2f(y, x);
    return t + 3 * min(max(__float2int_rn(angle * 40.743665f), 0), 128);  // 128 / pi
}
// arcsin(d) for |d| <= 0.0125: 4 FP64 instructions
__device__ __forceinline__ double arcsin_f64(double d) {
    const float df = f64_to_f32(d), d2 = df * df;
    const double p = 1.0 / 6.0 + f32_to_f64(d2 * fmaf(d2, 15.f / 336.f, 3.f / 40.f));
    return fma(d * d * d, p, d);
}

// 2^((n + f) / 512) for |f| <= 0.6 and n in [-512 * 1021, 512 * 1022] (the result a normal number: its exponent is
// shifted in place); t: the tables. 5 FP64 instructions.
__device__ __forceinline__ double exp2_512_f64(int n, double f, const double* t) {
    constexpr double kC = 0.0013538030870311431;  // ln 2 / 512
    const float ff = f64_to_f32(f);
    constexpr float c3 = static_cast<float>(kC * kC * kC / 6.0), c4 = static_cast<float>(kC * kC * kC * kC / 24.0);
    const double a = kC * kC / 2.0 + f32_to_f64(ff * fmaf(ff, c4, c3));
    const double p = fma(f * f, a, f * kC);
    const double e = t[3 * 129 + (n & 511)];
    const double v = fma(e, p, e);
    return __hiloint2double(__double2hiint(v) + ((n >> 9) << 20), __double2loint(v));
}

}  // namespace sbgpu
