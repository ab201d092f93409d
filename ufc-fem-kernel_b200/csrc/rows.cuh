// Shared pieces of the kernels that assemble block rows: the sign-bit numbering
// of the element nodes and the writer of finished rows.
#pragma once

#include <cuda_runtime.h>

#include "c3d8_device.cuh"
#include "ufc_internal.cuh"

namespace ufc {
namespace {

// Lane t's node (Abaqus order) has the natural-coordinate sign bits t; the map is its own inverse.
__host__ __device__ constexpr int bits_node(int t) { return t ^ ((t >> 1) & 1); }

// Upper triangle of a symmetric 6x6, row by row: entry (i, j), i <= j.
__host__ __device__ constexpr int tri6(int i, int j) {
  const int lo = i < j ? i : j, hi = i < j ? j : i;
  return lo * 6 - lo * (lo - 1) / 2 + hi - lo;
}

template <typename T>
__device__ __forceinline__ T flip_if(T v, bool neg) {
  return neg ? -v : v;
}

// Writes the accumulated block rows [half, half + ROWS) of a slice to the SELL
// values (each written once, ROWS consecutive values per warp load) and the
// Jacobi diagonal; val_r and dinv_r, when given, take the values rounded to
// FP32.  Entries in a row or a column of a Dirichlet DOF are zero, its diagonal
// 1 (symmetric elimination).  init() reads the Dirichlet flags of the first
// kAhead entries of each thread, so that their latency passes behind the
// accumulation.
template <typename T, int ROWS, int THREADS>
struct RowWriter {
  static constexpr int kAhead = 8, kStep = THREADS / ROWS;
  int r, j0, dj;       // row in the tile, first entry of this thread, entry of the diagonal (or -1)
  int64_t R, P0;       // block row, position of its entry 0
  unsigned fr, fc;     // Dirichlet flags: of the row (3 bits), of the columns of the first kAhead entries

  __device__ __forceinline__ unsigned flags(const uint8_t* __restrict__ fixed, int64_t node) const {
    return (fixed[3 * node] ? 1u : 0u) | (fixed[3 * node + 1] ? 2u : 0u) | (fixed[3 * node + 2] ? 4u : 0u);
  }

  __device__ __forceinline__ void init(int32_t N, int64_t s, int half, int64_t base, int len,
                                       const int32_t* __restrict__ scol, const int32_t* __restrict__ dpos,
                                       const uint8_t* __restrict__ fixed) {
    r = threadIdx.x & (ROWS - 1);
    j0 = threadIdx.x / ROWS;
    R = s * kSlice + half + r;
    P0 = base + half + r;
    const bool real = R < N;
    int32_t col[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) col[q] = j0 + q * kStep < len ? scol[P0 + 32 * (int64_t)(j0 + q * kStep)] : 0;
    fr = real ? flags(fixed, R) : 0u;
    dj = real ? (int)((dpos[R] - P0) >> 5) : -1;
    fc = 0;
#pragma unroll
    for (int q = 0; q < kAhead; ++q) fc |= flags(fixed, col[q]) << (3 * q);
  }

  __device__ __forceinline__ void write(int len, const int32_t* __restrict__ scol, const uint8_t* __restrict__ fixed,
                                        const T* acc, int stride, T* __restrict__ val, T* __restrict__ dinv,
                                        float* __restrict__ val_r, float* __restrict__ dinv_r) const {
    unsigned f = fc;
    int q = 0;
    for (int j = j0; j < len; j += kStep, ++q, f >>= 3) {
      const int64_t P = P0 + 32 * (int64_t)j;
      const unsigned m = q < kAhead ? f & 7u : flags(fixed, scol[P]);
      const T* a = acc + r * stride + 9 * j;
      const int64_t p = vpos(P, 0);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
          T v = (((fr >> i) | (m >> jj)) & 1u) ? T(0) : a[3 * i + jj];
          if (j == dj && i == jj && ((fr >> i) & 1u)) v = T(1);
          val[p + 32 * (3 * i + jj)] = v;
          if (val_r) val_r[p + 32 * (3 * i + jj)] = (float)v;
          if (j == dj && i == jj) {
            // Jacobi diag_inv = 1/K_ii, or 1 when |K_ii| <= 1e-30 (NM_LinSolv_Prec_Jacobi_Build,
            // ufc_core/L2_NM/Solver/LinSolv/NM_Solv_LinPrec.f90:328-353; NM_Solver_PCG uses 1e-30)
            const T di = fabs((double)v) > 1e-30 ? T(1) / v : T(1);
            dinv[3 * R + i] = di;
            if (dinv_r) dinv_r[3 * R + i] = (float)di;
          }
        }
    }
  }
};

}  // namespace
}  // namespace ufc
