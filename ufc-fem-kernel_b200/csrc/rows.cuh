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

// Where the assembled values go besides the full SELL storage and its Jacobi
// diagonal: the same rounded to FP32, and the symmetric storage (upper blocks
// only; its padding stays zero) in FP64 and rounded.  Null: not built.
template <typename T>
struct RowOutputs {
  T* val = nullptr;
  T* dinv = nullptr;
  float* val_r = nullptr;
  float* dinv_r = nullptr;
  const int64_t* uptr = nullptr;  // symmetric storage: slice starts
  T* sval = nullptr;
  float* sval_r = nullptr;
};

template <typename T, typename V>
__device__ __forceinline__ void store_sym(T* __restrict__ out, int64_t P, const V (&v)[9]) {
  T* p = out + 9 * (P & ~int64_t(31));
  const int t = (int)(P & 31);
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[t] = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
    reinterpret_cast<float4*>(p + 128)[t] = make_float4((float)v[4], (float)v[5], (float)v[6], (float)v[7]);
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) reinterpret_cast<double2*>(p + 64 * g)[t] = make_double2(v[2 * g], v[2 * g + 1]);
  }
  p[256 + t] = (T)v[8];
}

// Writes the accumulated block rows [half, half + ROWS) of a slice (each value
// once, ROWS consecutive values per warp store) and the Jacobi diagonal.
// Entries in a row or a column of a Dirichlet DOF are zero, its diagonal 1
// (symmetric elimination).  init() reads the columns and Dirichlet flags of the
// first kAhead entries of each thread, so that their latency passes behind the
// accumulation.  Writing the symmetric storage here instead of packing it from
// the full one: 2.01 -> 1.67 ms at 128x64x64 (both precisions).
template <typename T, int ROWS, int THREADS>
struct RowWriter {
  static constexpr int kAhead = 8, kStep = THREADS / ROWS;
  int r, j0, dj;       // row in the tile, first entry of this thread, entry of the diagonal (or -1)
  int64_t R, P0;       // block row, position of its entry 0
  unsigned fr, fc;     // Dirichlet flags of the row (3 bits); of the columns of the first kAhead entries (4 bits each,
                       // the fourth set for padding)

  __device__ __forceinline__ unsigned flags(const uint8_t* __restrict__ fixed, int64_t node) const {
    return (fixed[3 * node] ? 1u : 0u) | (fixed[3 * node + 1] ? 2u : 0u) | (fixed[3 * node + 2] ? 4u : 0u);
  }
  // padding points at the row itself, behind its real entries
  __device__ __forceinline__ unsigned entry(const uint8_t* __restrict__ fixed, int64_t col, int j) const {
    return flags(fixed, col) | (dj < 0 || (col == R && j != dj) ? 8u : 0u);
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
    for (int q = 0; q < kAhead; ++q) fc |= entry(fixed, col[q], j0 + q * kStep) << (4 * q);
  }

  __device__ __forceinline__ void write(int len, const int32_t* __restrict__ scol, const uint8_t* __restrict__ fixed,
                                        const T* acc, int stride, const RowOutputs<T>& o) const {
    unsigned f = fc;
    int q = 0;
    for (int j = j0; j < len; j += kStep, ++q, f >>= 4) {
      const int64_t P = P0 + 32 * (int64_t)j;
      const unsigned m = q < kAhead ? f & 15u : entry(fixed, scol[P], j);
      const T* a = acc + r * stride + 9 * j;
      const int64_t p = vpos(P, 0);
      T v[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) {
          T w = (((fr >> i) | (m >> jj)) & 1u) ? T(0) : a[3 * i + jj];
          if (j == dj && i == jj && ((fr >> i) & 1u)) w = T(1);
          v[3 * i + jj] = w;
          o.val[p + 32 * (3 * i + jj)] = w;
          if (o.val_r) o.val_r[p + 32 * (3 * i + jj)] = (float)w;
          if (j == dj && i == jj) {
            // Jacobi diag_inv = 1/K_ii, or 1 when |K_ii| <= 1e-30 (NM_LinSolv_Prec_Jacobi_Build,
            // ufc_core/L2_NM/Solver/LinSolv/NM_Solv_LinPrec.f90:328-353; NM_Solver_PCG uses 1e-30)
            const T di = fabs((double)w) > 1e-30 ? T(1) / w : T(1);
            o.dinv[3 * R + i] = di;
            if (o.dinv_r) o.dinv_r[3 * R + i] = (float)di;
          }
        }
      // the diagonal's entry is the number of lower blocks: what follows it is upper
      if (o.uptr && j >= dj && !(m & 8u)) {
        const int64_t U = o.uptr[R >> 5] + 32 * (int64_t)(j - dj) + (R & 31);
        if (o.sval) store_sym(o.sval, U, v);
        if (o.sval_r) store_sym(o.sval_r, U, v);
      }
    }
  }
};

}  // namespace
}  // namespace ufc
