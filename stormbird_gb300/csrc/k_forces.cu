// Sectional and integrated forces (sm_103a), f64: SimulationResult of one step
// (stormbird/src/line_force_model/force_calculations.rs:322-452, 669-698;
// common_utils/forces_and_moments.rs:163-245; flow_derivatives.rs:31-63).
//
// A CTA per wing: a thread per line evaluates the line's forces (about 200 FP64 instructions,
// sb_line.cuh), then a warp per force component sums the wing's forces and moments over the lines; the
// CTA that finishes last adds up the wings. Bound by the FP64 instructions of one line (a lone warp issues
// one per 65 cycles whatever the active lanes; three warps run side by side on the SM's FP64 pipe). One CTA for all wings with CUDA's f64 functions inlined (160 KB of code,
// most of it fetched once per launch) and sums by one thread per (wing, component) took 68 us at
// 21 lines, 118 at 4 x 64, 359 at 8 x 128; this takes 18, 22 and 25 us (CUDA events).
#include "sb_device.cuh"
#include "sb_kernels.h"
#include "sb_line.cuh"

namespace sbgpu {

namespace {

constexpr int kForceThreads = 256;

__device__ __noinline__ d3 body_frame(d3 v, d3 rotation) { return to_body(v, rotation); }

// force_calculations.rs:411-452 (added mass) with the line's span and chord vectors in the output frame
__device__ __noinline__ d3 added_mass(double factor, double density, double chord_len, d3 span, d3 chord, d3 acc) {
    d3 ra = acc - project(acc, normalize(span));
    ra = ra - project(ra, chord);
    const double l = len(ra);
    if (l == 0.0) return mk(0, 0, 0);
    return (factor * l) * density * (chord_len * len(span)) * normalize(ra);
}

// Sum over the warp of v[0..7]: the lane gets the sum of v[i] with i = bits 4, 3, 2 of its number
// (9 additions instead of 40: every exchange halves the values a lane goes on with).
__device__ __forceinline__ double reduce8(double (&v)[8], int lane) {
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {
        const bool upper = (lane & (4 * h)) != 0;
#pragma unroll
        for (int q = 0; q < h; ++q) {
            const double send = upper ? v[q] : v[q + h], keep = upper ? v[q + h] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
        }
    }
    double s = v[0];
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

__device__ void wing_forces(const DevModel& m, const StepParams& p, const ForceArgs& f, int wing) {
    const int N = m.N, S = m.S, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const OutLayout L = OutLayout::make(N, S);
    double* o = f.out;
    const bool body = m.output_body != 0;
    const int ws = m.wing_start[wing], we = m.wing_end[wing];
    __shared__ double tab[kF64TableDoubles];
    __shared__ int s_last;
    load_f64_tables(tab, tid, kForceThreads);
    __syncthreads();
    auto put = [&](long long at, int i, d3 v) {
        o[at + 3 * i] = v.x;
        o[at + 3 * i + 1] = v.y;
        o[at + 3 * i + 2] = v.z;
    };
#pragma unroll 1
    for (int i = ws + tid; i < we; i += kForceThreads) {
        const double g = f.gamma[i];
        const d3 v = f.vel[i], felt = m.felt_ctrl[i], ctrl = m.ctrl[i];
        const d3 sr = m.span_e[i] - m.span_s[i];
        const FoilP& fo = m.foils[wing];
        const LineLift lift = line_lift(fo, m.chord_global[i], v, normalize(sr), tab);
        const d3 h1 = f.hist1[i];
        d3 acc = mk(0, 0, 0);
        if (f.fd_count >= 2) acc = (v * 3.0 - h1 * 4.0 + f.hist0[i]) * rcp_any(2.0 * p.dt);
        f.hist0[i] = h1;
        f.hist1[i] = v;
        const d3 fv = body ? body_frame(v, p.rotation) : v;
        const d3 fa = body ? body_frame(acc, p.rotation) : acc;
        const d3 sl_local = m.span_e_local[i] - m.span_s_local[i];
        const d3 sl_out = body ? sl_local : sr;
        const double q = len2(fv), ff = 0.5 * (m.chord_len[i] * m.span_len_local[i]) * m.density * q;
        put(L.vel, i, v);
        put(L.felt, i, felt);
        put(L.fvel, i, fv);
        put(L.acc, i, fa);
        put(L.ctrl, i, ctrl);
        o[L.gamma + i] = g;
        o[L.aoa + i] = lift.aoa;
        const d3 circ = q == 0.0 ? mk(0, 0, 0) : (g * cross(fv, sl_out)) * m.density;
        d3 visc = mk(0, 0, 0);
        if (!m.include_viscous_lift) visc = normalize(cross(sl_local, fv)) * (lift.cl_post * ff);
        const d3 drag = q == 0.0 ? mk(0, 0, 0) : fv * (rsqrt_any(q) * line_drag(fo, lift, tab) * ff);  // a NaN stays
        const double none = 0.0 * (fa.x + fa.y + fa.z);  // no number where the acceleration is none
        d3 am = mk(none, none, none);
        if (fo.added_mass_factor != 0.0)
            am = added_mass(fo.added_mass_factor, m.density, m.chord_len[i], sl_out,
                            body ? m.chord_local[i] : m.chord_global[i], fa);
        const d3 gyro = mk(0, 0, 0);
        put(L.sect, i, circ);
        put(L.sect + 3LL * N, i, visc);
        put(L.sect + 6LL * N, i, drag);
        put(L.sect + 9LL * N, i, am);
        put(L.sect + 12LL * N, i, gyro);
        put(L.sect + 15LL * N, i, circ + visc + drag + am);
    }
    __syncthreads();
    // integrated force and moment of each component over the wing's lines
    if (warp < 6) {
        double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const double* sect = o + L.sect + 3LL * warp * N;
#pragma unroll 1
        for (int i = ws + lane; i < we; i += 32) {
            if (m.is_virtual[i]) continue;
            const d3 cp = body ? 0.5 * (m.span_s_local[i] + m.span_e_local[i]) : m.ctrl[i];
            const d3 sf = mk(sect[3 * i], sect[3 * i + 1], sect[3 * i + 2]), mo = cross(cp, sf);
            v[0] += sf.x;
            v[1] += sf.y;
            v[2] += sf.z;
            v[3] += mo.x;
            v[4] += mo.y;
            v[5] += mo.z;
        }
        __syncwarp();
        const double s = reduce8(v, lane);
        const int k = lane >> 2;
        if ((lane & 3) == 0 && k < 6)
            o[(k < 3 ? L.intf : L.intm) + (static_cast<long long>(wing) * 6 + warp) * 3 + k % 3] = s;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(f.counter, 1u) == static_cast<unsigned>(S - 1) ? 1 : 0;
    __syncthreads();
    if (!s_last) return;
    // the last wing to finish: the sums over the wings
    __threadfence();
    if (tid < 6) {
        const long long at = (tid < 3 ? L.intf : L.intm) + 15 + tid % 3;
        double s = 0.0;
        for (int w = 0; w < S; ++w) s += __ldcg(o + at + 18LL * w);
        o[(tid < 3 ? L.fsum : L.msum) + tid % 3] = s;
    } else if (tid < 9) {
        o[L.residual + (tid - 6)] = f.scalars[tid - 6];  // residual, iterations, converged
    } else if (tid == 32) {
        *f.counter = 0u;
    }
}

__global__ void __launch_bounds__(kForceThreads) k_forces(DevModel m, StepParams p, ForceArgs f) {
    wing_forces(m, p, f, blockIdx.x);
}

// A CTA per wing of every case of a batch; jobs ascending in their first block.
__global__ void __launch_bounds__(kForceThreads) k_forces_jobs(const ForceJob* jobs, int n) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].block_begin <= static_cast<int>(blockIdx.x)) lo = mid;
        else hi = mid - 1;
    }
    const ForceJob& j = jobs[lo];
    wing_forces(j.m, j.p, j.f, static_cast<int>(blockIdx.x) - j.block_begin);
}

}  // namespace

cudaError_t launch_forces(const DevModel& m, const StepParams& p, const ForceArgs& f, cudaStream_t s) {
    k_forces<<<m.S, kForceThreads, 0, s>>>(m, p, f);
    return cudaGetLastError();
}

cudaError_t launch_forces_jobs(const ForceJob* jobs, int n, int blocks, cudaStream_t s) {
    if (n <= 0 || blocks <= 0) return cudaSuccess;
    k_forces_jobs<<<static_cast<unsigned>(blocks), kForceThreads, 0, s>>>(jobs, n);
    return cudaGetLastError();
}

}  // namespace sbgpu
