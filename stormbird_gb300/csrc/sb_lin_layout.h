// Rows and shared memory of the refined Linearized solve (k_lin_refined.cu): host and device arithmetic.
#pragma once

#include <cstddef>

#include "sb_device.cuh"
#include "sb_f64.cuh"

namespace sbgpu {

constexpr int kLinBlk = 16;  // rows of a block

// The system's N rows padded to whole blocks, dealt round-robin to the C CTAs of a cluster (block k to
// CTA k mod C). Every CTA has room for lin_local_rows rows; the last ones lie past the system where the
// number of blocks is not a multiple of C.
__host__ __device__ inline int lin_padded(int N) { return (N + kLinBlk - 1) / kLinBlk * kLinBlk; }
__host__ __device__ inline int lin_local_rows(int N, int C) { return (lin_padded(N) / kLinBlk + C - 1) / C * kLinBlk; }
// row of the system that row l of CTA rank is
__host__ __device__ inline int lin_row(int l, int rank, int C) { return (rank + l / kLinBlk * C) * kLinBlk + l % kLinBlk; }
// rows of CTA rank that are rows of the padded system: lin_row is below lin_padded(N) for l below it
__host__ __device__ inline int lin_own_rows(int N, int C, int rank) {
    return (lin_padded(N) / kLinBlk - rank + C - 1) / C * kLinBlk;
}

// Shared memory of a CTA, in order (all multiples of 16 bytes)
struct LinLayout {
    size_t A, P, M, x, g, rv, dx, vel, w, rhs, tab, total;
    __host__ __device__ static LinLayout make(int N, int C) {
        const size_t n = lin_padded(N), R = lin_local_rows(N, C);
        LinLayout l{};
        size_t at = 0;
        l.A = at; at += R * n * 4;         // own rows, FP32
        l.P = at; at += kLinBlk * n * 4;   // scaled pivot rows
        l.M = at; at += kLinBlk * R * 4;   // multipliers, [16][R]
        l.x = at; at += n * 8;             // solution
        l.g = at; at += n * 8;             // corrected circulation, then residual terms (CTA 0)
        l.rv = at; at += n * 4;            // residual
        l.dx = at; at += n * 4;            // correction
        l.vel = at; at += R * sizeof(d3);  // velocity of the own rows
        l.w = at; at += R * sizeof(d3);    // row vectors of the matrix
        l.rhs = at; at += 2 * R * 8;       // right-hand side, diagonal term
        l.tab = at; at += (kF64TableDoubles + 1) / 2 * 16;
        l.total = at;
        return l;
    }
};

}  // namespace sbgpu
