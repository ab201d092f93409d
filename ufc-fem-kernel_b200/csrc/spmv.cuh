// Products with the stored stiffness: the kernels over the full SELL-32 storage,
// its coded form and the symmetric storage, each ending in an epilogue functor
// that takes the row sums (store, the CG's dot product, the multigrid
// smoother's recurrence), and their launchers.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "c3d8_device.cuh"
#include "pdl.cuh"
#include "reduce.cuh"
#include "ufc_internal.cuh"

namespace ufc {
namespace {

constexpr int kSpmvBlock = 256;

// Stored steps that a warp of a split product loads (columns and values) before
// it waits for the kernel in front: the matrix is not written inside a chain,
// so these loads pass behind that kernel's end, and what follows the wait is
// one gather.  All steps of a warp on the small meshes that take 8 warps per
// slice, where a product's time is latency.
template <typename TV, int SPLIT>
constexpr int split_ahead() {
  return SPLIT == 8 ? 4 : sizeof(TV) == 4 ? 4 : 2;
}

// Products inside an iteration chain are launched with programmatic dependence.
// Returns the grid: the number of partial sums a product with a dot leaves.
template <bool PDL, typename... K, typename... A>
int launch_product(void (*kernel)(K...), int grid, int block, cudaStream_t st, A&&... args) {
  if constexpr (PDL)
    launch_pdl(kernel, grid, block, st, std::forward<A>(args)...);
  else
    kernel<<<grid, block, 0, st>>>(std::forward<A>(args)...);
  return grid;
}

// The kernels of a CG iteration do nothing once the run has stopped or asked
// for an FP64 residual replacement: a batch of iterations launched as one graph
// then idles from the triggering iteration on, so the replacement happens at
// that iteration (before its direction update) and not at the end of the batch.
__device__ __forceinline__ bool halted(const CgScalars* s) { return (s->stop | s->want_update) != 0; }

// What a product does with a finished row sum a = (K x)_row.
//   EpiStore  y = a
//   EpiCg     q = a and the row's part of x.a, inside the CG chain
template <typename TX>
struct EpiStore {
  static constexpr bool kDot = false, kPdl = false;
  TX* y;
  __device__ __forceinline__ bool halt() const { return false; }
  __device__ __forceinline__ bool want_dot() const { return false; }
  template <typename TA>
  __device__ __forceinline__ double operator()(int64_t row, TA a0, TA a1, TA a2, const TX*) const {
    y[3 * row] = (TX)a0;
    y[3 * row + 1] = (TX)a1;
    y[3 * row + 2] = (TX)a2;
    return 0.0;
  }
};

template <typename TX>
struct EpiCg {
  static constexpr bool kDot = true, kPdl = true;
  TX* y;
  const CgScalars* scal;
  __device__ __forceinline__ bool halt() const { return halted(scal); }
  __device__ __forceinline__ bool want_dot() const { return true; }
  template <typename TA>
  __device__ __forceinline__ double operator()(int64_t row, TA a0, TA a1, TA a2, const TX* __restrict__ x) const {
    y[3 * row] = (TX)a0;
    y[3 * row + 1] = (TX)a1;
    y[3 * row + 2] = (TX)a2;
    return (double)((TA)x[3 * row] * a0 + (TA)x[3 * row + 1] * a1 + (TA)x[3 * row + 2] * a2);
  }
};

// y = K x, one thread per block row of a SELL-32 slice (a warp = a slice).
// TV: stored value type, TX: vector type, TA: accumulator type of the row sums.
// DIFF: values in difference form (diagonal slot = block row sum S_i), so the
// row is evaluated as sum_{j != i} K_ij (x_j - x_i) + S_i x_i.
template <typename TV, typename TX, typename TA, class EPI, bool DIFF>
__global__ void __launch_bounds__(kSpmvBlock)
    k_spmv(int32_t N, int64_t nrows_pad, const int64_t* __restrict__ sptr, const int32_t* __restrict__ col,
           const TV* __restrict__ val, const TX* __restrict__ x, EPI epi,
           double* __restrict__ partials) {
  pdl_enter();
  if (epi.halt()) return;
  const int64_t row = (int64_t)blockIdx.x * kSpmvBlock + threadIdx.x;
  double dot[1] = {0.0};
  if (row < nrows_pad) {
    const int64_t s = row >> 5;
    const int t = (int)(row & 31);
    const int64_t base = sptr[s];
    const int len = (int)((sptr[s + 1] - base) >> 5);
    const int32_t* cp = col + base + t;
    const TV* vp = val + 9 * base + t;
    TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
    TA xi0 = TA(0), xi1 = TA(0), xi2 = TA(0);
    if (DIFF && row < N) {
      xi0 = (TA)x[3 * row];
      xi1 = (TA)x[3 * row + 1];
      xi2 = (TA)x[3 * row + 2];
    }
#pragma unroll 2
    for (int j = 0; j < len; ++j) {
      const int64_t cj = __ldcs(cp + 32 * j);
      TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
      if (DIFF && cj != row) {
        x0 -= xi0;
        x1 -= xi1;
        x2 -= xi2;
      }
      const TV* v = vp + 288 * (int64_t)j;
      a0 += (TA)__ldcs(v) * x0 + (TA)__ldcs(v + 32) * x1 + (TA)__ldcs(v + 64) * x2;
      a1 += (TA)__ldcs(v + 96) * x0 + (TA)__ldcs(v + 128) * x1 + (TA)__ldcs(v + 160) * x2;
      a2 += (TA)__ldcs(v + 192) * x0 + (TA)__ldcs(v + 224) * x1 + (TA)__ldcs(v + 256) * x2;
    }
    if (row < N) {
      dot[0] = epi(row, a0, a1, a2, x);
    }
  }
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

// The same product with SPLIT (2, 4 or 8) warps per slice, for meshes with few
// slices per SM: the warps of a slice take the stored blocks j = part,
// part + SPLIT, ... of their 32 rows (every load stays a coalesced 32-row
// line) and their partial row sums are added in shared memory in warp order,
// so the result depends only on SPLIT, which the launcher derives from the
// problem size.
template <typename TV, typename TX, typename TA, class EPI, bool DIFF, int SPLIT>
__global__ void __launch_bounds__(kSpmvBlock)
    k_spmv_split(int32_t N, int64_t nslices, const int64_t* __restrict__ sptr, const int32_t* __restrict__ col,
                 const TV* __restrict__ val, const TX* __restrict__ x, EPI epi, double* __restrict__ partials) {
  constexpr int kWarps = kSpmvBlock / 32, kAhead = split_ahead<TV, SPLIT>();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = warp % SPLIT;
  const int64_t s = (int64_t)blockIdx.x * (kWarps / SPLIT) + warp / SPLIT;
  const int64_t row = s * kSlice + lane;
  const int64_t base = s < nslices ? sptr[s] : 0;
  const int len = s < nslices ? (int)((sptr[s + 1] - base) >> 5) : 0;
  const int32_t* cp = col + base + lane;
  const TV* vp = val + 9 * base + lane;
  int32_t ca[kAhead];
  TV va[kAhead][9];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int j = part + u * SPLIT;
    ca[u] = j < len ? __ldcs(cp + 32 * j) : 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) va[u][c] = j < len ? __ldcs(vp + 288 * (int64_t)j + 32 * c) : TV(0);
  }
  pdl_enter();
  if (epi.halt()) return;
  TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
  if (s < nslices) {
    TA xi0 = TA(0), xi1 = TA(0), xi2 = TA(0);
    if (DIFF && row < N) {
      xi0 = (TA)x[3 * row];
      xi1 = (TA)x[3 * row + 1];
      xi2 = (TA)x[3 * row + 2];
    }
    auto block = [&](int64_t cj, const TV(&v)[9]) {
      TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
      if (DIFF && cj != row) {
        x0 -= xi0;
        x1 -= xi1;
        x2 -= xi2;
      }
      a0 += (TA)v[0] * x0 + (TA)v[1] * x1 + (TA)v[2] * x2;
      a1 += (TA)v[3] * x0 + (TA)v[4] * x1 + (TA)v[5] * x2;
      a2 += (TA)v[6] * x0 + (TA)v[7] * x1 + (TA)v[8] * x2;
    };
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (part + u * SPLIT < len) block(ca[u], va[u]);
#pragma unroll 2
    for (int j = part + kAhead * SPLIT; j < len; j += SPLIT) {
      const int64_t cj = __ldcs(cp + 32 * j);
      TV v[9];
#pragma unroll
      for (int c = 0; c < 9; ++c) v[c] = __ldcs(vp + 288 * (int64_t)j + 32 * c);
      block(cj, v);
    }
  }
  {
    __shared__ TA sh[kWarps][3][32];
    sh[warp][0][lane] = a0;
    sh[warp][1][lane] = a1;
    sh[warp][2][lane] = a2;
    __syncthreads();
    if (part == 0) {
#pragma unroll
      for (int q = 1; q < SPLIT; ++q) {
        a0 += sh[warp + q][0][lane];
        a1 += sh[warp + q][1][lane];
        a2 += sh[warp + q][2][lane];
      }
    }
  }
  double dot[1] = {0.0};
  if (part == 0 && s < nslices && row < N) {
    dot[0] = epi(row, a0, a1, a2, x);
  }
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

// y = K x on the full SELL storage with coded indices (see build_full_codes):
// each row loads its 32 code bytes with two 16-byte loads when the warp
// starts, and block j's column is row + off[code j], so no column index is
// loaded inside the loop.  One warp per slice, as k_spmv, and the same order of
// sums, so the same results bit for bit.
template <typename TV, typename TX, typename TA, class EPI>
__global__ void __launch_bounds__(kSpmvBlock)
    k_spmvc(int32_t N, int64_t nslices, const int64_t* __restrict__ sptr, const uint4* __restrict__ code,
            FullOffsets tab, const TV* __restrict__ val, const TX* __restrict__ x, EPI epi,
            double* __restrict__ partials) {
  pdl_enter();
  if (epi.halt()) return;
  __shared__ int32_t soff[32];
  if (threadIdx.x < 32) soff[threadIdx.x] = tab.off[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t s = (int64_t)blockIdx.x * (kSpmvBlock / 32) + (threadIdx.x >> 5);
  const int64_t row = s * kSlice + lane;
  TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
  if (s < nslices) {
    const int64_t base = sptr[s];
    const int len = (int)((sptr[s + 1] - base) >> 5);
    const uint4 c0 = __ldcs(code + 2 * row), c1 = __ldcs(code + 2 * row + 1);
    Code256 cw{c0.x | ((uint64_t)c0.y << 32), c0.z | ((uint64_t)c0.w << 32), c1.x | ((uint64_t)c1.y << 32),
               c1.z | ((uint64_t)c1.w << 32)};
    const TV* vp = val + 9 * base + lane;
#pragma unroll 2
    for (int j = 0; j < len; ++j) {
      const unsigned cd = cw.front();
      cw.drop();
      TA x0 = TA(0), x1 = TA(0), x2 = TA(0);
      if (cd != 255u) {
        const int64_t cj = row + soff[cd];
        x0 = (TA)__ldg(x + 3 * cj);
        x1 = (TA)__ldg(x + 3 * cj + 1);
        x2 = (TA)__ldg(x + 3 * cj + 2);
      }
      const TV* v = vp + 288 * (int64_t)j;
      a0 += (TA)__ldcs(v) * x0 + (TA)__ldcs(v + 32) * x1 + (TA)__ldcs(v + 64) * x2;
      a1 += (TA)__ldcs(v + 96) * x0 + (TA)__ldcs(v + 128) * x1 + (TA)__ldcs(v + 160) * x2;
      a2 += (TA)__ldcs(v + 192) * x0 + (TA)__ldcs(v + 224) * x1 + (TA)__ldcs(v + 256) * x2;
    }
  }
  double dot[1] = {0.0};
  if (s < nslices && row < N) dot[0] = epi(row, a0, a1, a2, x);
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

// Bulk L2 prefetch (cp.async.bulk.prefetch, the TMA unit) of the first k1
// steps of one slice's stream, issued by lane 0 when the warp starts: the upper
// values and columns of the steps below ulen and the lower positions and
// columns of those below llen, four contiguous ranges that stay inside the
// slice's own part of the arrays (their starts are multiples of 128 bytes and
// their sizes of 16).  The rest of the slice is loaded on demand: prefetching
// all of it (14 steps) overfills L2 with the resident window's streams, and a
// prefetch per loop trip costs the registers of a fifth resident block.
template <typename TV>
__device__ __forceinline__ void sym_prefetch(int lane, int k1, int ulen, int llen, const TV* uv0,
                                             const int32_t* uc0, const int32_t* lp0, const int32_t* lc0) {
  if (lane != 0) return;
  const int ku = k1 < ulen ? k1 : ulen, kl = k1 < llen ? k1 : llen;
  if (ku > 0) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(uv0), "r"((unsigned)(ku * 288 * (int)sizeof(TV)))
                 : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(uc0), "r"((unsigned)(ku * 128)) : "memory");
  }
  if (kl > 0) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lp0), "r"((unsigned)(kl * 128)) : "memory");
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lc0), "r"((unsigned)(kl * 128)) : "memory");
  }
}

// The 9 values of lane t's block of one stored step of the symmetric storage
// (p: the step's 288 values), by 16-byte loads (see spos): an FP32 block takes 3
// load instructions instead of 9, an FP64 block 5, and the shifted reads of a
// lower block (the 32 lanes' blocks begin inside one step and run into the
// next row group) touch 12 cache lines instead of 18.
template <typename TV>
__device__ __forceinline__ void load_block(const TV* __restrict__ p, int t, TV (&v)[9]) {
  if constexpr (sizeof(TV) == 4) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p) + t), b = __ldg(reinterpret_cast<const float4*>(p + 128) + t);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const double2 a = __ldg(reinterpret_cast<const double2*>(p + 64 * g) + t);
      v[2 * g] = a.x;
      v[2 * g + 1] = a.y;
    }
  }
  v[8] = __ldg(p + 256 + t);
}

// y = K x from the symmetric storage: row i sums its upper blocks K_ij x_j
// (j >= i, SELL-32, coalesced) and its lower blocks as transposes K_ji^T x_j of
// the blocks stored by the earlier rows j.  Those transposed reads are from
// blocks streamed by rows at most about one node plane earlier, so they come
// from L2; the upper values are loaded with the default cache policy so that
// they stay there.
template <typename TV, typename TX, typename TA, class EPI>
__global__ void __launch_bounds__(kSpmvBlock)
    k_spmv_sym(int32_t N, int64_t nrows_pad, const int64_t* __restrict__ uptr, const int32_t* __restrict__ ucol,
               const int64_t* __restrict__ lptr, const int32_t* __restrict__ lpos, const int32_t* __restrict__ lcol,
               const TV* __restrict__ val, const TX* __restrict__ x, EPI epi,
           double* __restrict__ partials) {
  pdl_enter();
  if (epi.halt()) return;
  const int64_t row = (int64_t)blockIdx.x * kSpmvBlock + threadIdx.x;
  double dot[1] = {0.0};
  if (row < nrows_pad) {
    const int64_t s = row >> 5;
    const int t = (int)(row & 31);
    TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
    const int64_t ub = uptr[s], lb = lptr[s];
    const int ulen = (int)((uptr[s + 1] - ub) >> 5);
    const int llen = (int)((lptr[s + 1] - lb) >> 5);
    const int32_t* ucp = ucol + ub + t;
    const TV* uvp = val + 9 * ub;
    const int32_t* lpp = lpos + lb + t;
    const int32_t* lcp = lcol + lb + t;
    // step j handles upper entry j and lower entry j, whose partners are read
    // by the owning rows at about the same step; the common part has no
    // branches so that the loads of both halves are in flight together
    auto upper = [&](int j) {
      const int64_t cj = __ldcs(ucp + 32 * j);
      const TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
      TV v[9];
      load_block(uvp + 288 * (int64_t)j, t, v);
      a0 += (TA)v[0] * x0 + (TA)v[1] * x1 + (TA)v[2] * x2;
      a1 += (TA)v[3] * x0 + (TA)v[4] * x1 + (TA)v[5] * x2;
      a2 += (TA)v[6] * x0 + (TA)v[7] * x1 + (TA)v[8] * x2;
    };
    auto lower = [&](int j) {
      const int64_t P = __ldcs(lpp + 32 * j);
      const int64_t cj = __ldcs(lcp + 32 * j);
      const TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
      TV v[9];
      load_block(val + 9 * (P & ~int64_t(31)), (int)(P & 31), v);
      // transposed block: (K_ji^T x)_r = sum_c K_ji[c][r] x_c
      a0 += (TA)v[0] * x0 + (TA)v[3] * x1 + (TA)v[6] * x2;
      a1 += (TA)v[1] * x0 + (TA)v[4] * x1 + (TA)v[7] * x2;
      a2 += (TA)v[2] * x0 + (TA)v[5] * x1 + (TA)v[8] * x2;
    };
    const int mlen = ulen < llen ? ulen : llen;
    int j = 0;
    // prefetch depth in steps, measured in the CG on B200 (192x96x96): FP32
    // 8 steps (SpMV 297 -> 291 us), FP64 4 steps (516 -> 502 us)
    sym_prefetch<TV>(t, sizeof(TV) == 8 ? 4 : 8, ulen, llen, val + 9 * ub, ucol + ub, lpos + lb, lcol + lb);
    // four steps per trip for FP64 values, two for FP32 (each the faster of the
    // two on B200, measured in the CG)
    if constexpr (sizeof(TV) == 8) {
#pragma unroll 1
      for (; j + 3 < mlen; j += 4) {
        upper(j);
        lower(j);
        upper(j + 1);
        lower(j + 1);
        upper(j + 2);
        lower(j + 2);
        upper(j + 3);
        lower(j + 3);
      }
    }
#pragma unroll 1
    for (; j + 1 < mlen; j += 2) {
      upper(j);
      lower(j);
      upper(j + 1);
      lower(j + 1);
    }
    for (; j < mlen; ++j) {
      upper(j);
      lower(j);
    }
    for (int k = mlen; k < ulen; ++k) upper(k);
    for (int k = mlen; k < llen; ++k) lower(k);
    if (row < N) {
      dot[0] = epi(row, a0, a1, a2, x);
    }
  }
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

// The symmetric product with coded indices (stencil-like patterns, see
// build_sym_codes): each row loads its 16 upper and 16 lower code bytes with
// two 16-byte loads when the warp starts, so the loop loads no indices at all.
// Upper step j: column row + off[code], its x gathered at once.  Lower step j:
// column row - off[code], and the block (col, row) at position
// uptr[col / 32] + 32 rank + col % 32 of the upper storage.  The columns of a
// slice at one offset lie in two slices, so a warp takes the starts of the (at
// most 15) pairs into shared memory first: no step has a dependent global load.
// Same summation order as k_spmv_sym, so the same results bit for bit.
// Bound by the latency of the gathers (DRAM 53 %, FP32, 128x64x64).  FP32
// values: two upper and two lower steps load together, without branches, in 3
// blocks per SM (a padded upper step holds zeros itself, a padded lower step
// takes the row's own diagonal block times 0): 198 -> 181 us at 192x96x96, 97.0
// -> 94.5 us per CG iteration at 128x64x64.  FP64 values would fill the
// registers that way (336 -> 479 us) and go step by step; the starts in shared
// memory give 489 -> 476 and 160 -> 154 us per iteration.
template <typename TV, typename TX, typename TA, class EPI>
__global__ void __launch_bounds__(kSpmvBlock, sizeof(TV) + sizeof(TX) == 8 ? 3 : 0)
    k_spmv_symc(int32_t N, int64_t nrows_pad, const int64_t* __restrict__ uptr, const int64_t* __restrict__ lptr,
                const uint4* __restrict__ ucode, const uint4* __restrict__ lcode, SymOffsets tab,
                const TV* __restrict__ val, const TX* __restrict__ x, EPI epi,
           double* __restrict__ partials) {
  pdl_enter();
  if (epi.halt()) return;
  __shared__ int32_t soff[16];
  __shared__ int2 sbase[kSpmvBlock / 32][16];
  if (threadIdx.x < 16) soff[threadIdx.x] = tab.off[threadIdx.x];
  __syncthreads();
  double dot[1] = {0.0};
  int2* sb = sbase[threadIdx.x >> 5];  // (block counts stay below 2^31: their FP64 values alone would be 154 GB)
  // FP64 values: a capped grid whose warps step through the slices (measured on
  // B200, 192x96x96: 400-402 us against 453 us with one slice per warp; FP32
  // values are faster with one slice per warp, 235 against 252-275 us)
  constexpr bool kStride = sizeof(TV) == 8;
  const int64_t rstep = kStride ? (int64_t)gridDim.x * kSpmvBlock : nrows_pad;
#pragma unroll 1
  for (int64_t row = (int64_t)blockIdx.x * kSpmvBlock + threadIdx.x; row < nrows_pad; row += rstep) {
    const int64_t s = row >> 5;
    const int t = (int)(row & 31);
    TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
    const int64_t ub = uptr[s];
    const int ulen = (int)((uptr[s + 1] - ub) >> 5);
    const int llen = (int)((lptr[s + 1] - lptr[s]) >> 5);
    const uint4 uc = __ldcs(ucode + row), lc = __ldcs(lcode + row);
    uint64_t ulo = uc.x | ((uint64_t)uc.y << 32), uhi = uc.z | ((uint64_t)uc.w << 32);
    uint64_t llo = lc.x | ((uint64_t)lc.y << 32), lhi = lc.z | ((uint64_t)lc.w << 32);
    const TV* uvp = val + 9 * ub;
    __syncwarp();
    if (t < 16) {
      const int64_t sa = (32 * s - soff[t]) >> 5;
      sb[t] = make_int2((int)__ldg(uptr + (sa < 0 ? 0 : sa)), (int)__ldg(uptr + (sa + 1 < 0 ? 0 : sa + 1)));
    }
    __syncwarp();
    // first block of the slice of column row - off
    auto slice_start = [&](unsigned code, int off) {
      const int2 pb = sb[code];
      const int sh = off & 31;
      return (int64_t)(sh && t >= sh ? pb.y : pb.x);
    };
    if (t == 0) {
      const int k1 = (sizeof(TV) == 8 ? 4 : 8) < ulen ? (sizeof(TV) == 8 ? 4 : 8) : ulen;
      if (k1 > 0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(val + 9 * ub),
                     "r"((unsigned)(k1 * 288 * (int)sizeof(TV)))
                     : "memory");
    }
    auto upper = [&](int j) {
      const unsigned code = (unsigned)(ulo & 0xFF);
      ulo = (ulo >> 8) | (uhi << 56);
      uhi >>= 8;
      TA x0 = TA(0), x1 = TA(0), x2 = TA(0);
      if (code != kSymCodes) {
        const int64_t cj = row + soff[code];
        x0 = (TA)__ldg(x + 3 * cj);
        x1 = (TA)__ldg(x + 3 * cj + 1);
        x2 = (TA)__ldg(x + 3 * cj + 2);
      }
      TV v[9];
      load_block(uvp + 288 * (int64_t)j, t, v);
      a0 += (TA)v[0] * x0 + (TA)v[1] * x1 + (TA)v[2] * x2;
      a1 += (TA)v[3] * x0 + (TA)v[4] * x1 + (TA)v[5] * x2;
      a2 += (TA)v[6] * x0 + (TA)v[7] * x1 + (TA)v[8] * x2;
    };
    auto lower = [&](int) {
      const unsigned b = (unsigned)(llo & 0xFF);
      llo = (llo >> 8) | (lhi << 56);
      lhi >>= 8;
      if (b != 0xFFu) {
        const int off = soff[b >> 4];
        const int64_t cj = row - off;
        const int64_t P = slice_start(b >> 4, off) + 32 * (int64_t)(b & 15u) + (cj & 31);
        const TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
        TV v[9];
        load_block(val + 9 * (P & ~int64_t(31)), (int)(P & 31), v);
        a0 += (TA)v[0] * x0 + (TA)v[3] * x1 + (TA)v[6] * x2;
        a1 += (TA)v[1] * x0 + (TA)v[4] * x1 + (TA)v[7] * x2;
        a2 += (TA)v[2] * x0 + (TA)v[5] * x1 + (TA)v[8] * x2;
      }
    };
    const int mlen = ulen < llen ? ulen : llen;
    int j = 0;
    if constexpr (sizeof(TV) + sizeof(TX) == 8) {
      const int64_t rx = row < N ? row : 0;
#pragma unroll 1
      for (; j + 1 < mlen; j += 2) {
        TV uv[2][9], lv[2][9];
        TX ux[2][3], lx[2][3];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const unsigned code = (unsigned)(ulo & 0xFF), b = (unsigned)(llo & 0xFF);
          ulo = (ulo >> 8) | (uhi << 56);
          uhi >>= 8;
          llo = (llo >> 8) | (lhi << 56);
          lhi >>= 8;
          const bool up = code != kSymCodes, low = b != 0xFFu;
          const int off = low ? soff[b >> 4] : 0;
          const int64_t cu = rx + (up ? soff[code] : 0), cl = rx - off;
          const int64_t lstep = low ? slice_start(b >> 4, off) + 32 * (int64_t)(b & 15u) : ub;
          load_block(uvp + 288 * (int64_t)(j + h), t, uv[h]);
          load_block(val + 9 * lstep, (int)(cl & 31), lv[h]);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            ux[h][c] = __ldg(x + 3 * cu + c);
            lx[h][c] = __ldg(x + 3 * cl + c);
          }
          if (!low) {
#pragma unroll
            for (int c = 0; c < 3; ++c) lx[h][c] = TX(0);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const TV *u = uv[h], *v = lv[h];
          TA x0 = (TA)ux[h][0], x1 = (TA)ux[h][1], x2 = (TA)ux[h][2];
          a0 += (TA)u[0] * x0 + (TA)u[1] * x1 + (TA)u[2] * x2;
          a1 += (TA)u[3] * x0 + (TA)u[4] * x1 + (TA)u[5] * x2;
          a2 += (TA)u[6] * x0 + (TA)u[7] * x1 + (TA)u[8] * x2;
          x0 = (TA)lx[h][0], x1 = (TA)lx[h][1], x2 = (TA)lx[h][2];
          a0 += (TA)v[0] * x0 + (TA)v[3] * x1 + (TA)v[6] * x2;
          a1 += (TA)v[1] * x0 + (TA)v[4] * x1 + (TA)v[7] * x2;
          a2 += (TA)v[2] * x0 + (TA)v[5] * x1 + (TA)v[8] * x2;
        }
      }
    } else {
#pragma unroll 1
      for (; j + 1 < mlen; j += 2) {
        upper(j);
        lower(j);
        upper(j + 1);
        lower(j + 1);
      }
    }
    for (; j < mlen; ++j) {
      upper(j);
      lower(j);
    }
    for (int k = mlen; k < ulen; ++k) upper(k);
    for (int k = mlen; k < llen; ++k) lower(k);
    if (row < N) {
      dot[0] += epi(row, a0, a1, a2, x);
    }
  }
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

// The symmetric product with SPLIT warps per slice for meshes with too few
// slices to fill the GPU one warp each: warp `part` of a slice takes the
// upper and lower steps j = part, part + SPLIT, ..., and the row sums of the
// slice's warps are added in shared memory in warp order.
template <typename TV, typename TX, typename TA, class EPI, int SPLIT>
__global__ void __launch_bounds__(kSpmvBlock)
    k_spmv_sym_split(int32_t N, int64_t nslices, const int64_t* __restrict__ uptr, const int32_t* __restrict__ ucol,
                     const int64_t* __restrict__ lptr, const int32_t* __restrict__ lpos,
                     const int32_t* __restrict__ lcol, const TV* __restrict__ val, const TX* __restrict__ x, EPI epi,
                     double* __restrict__ partials) {
  // a warp's steps hold an upper and a lower block each: half as many ahead
  constexpr int kWarps = kSpmvBlock / 32, kAhead = split_ahead<TV, SPLIT>() / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = warp % SPLIT;
  const int64_t s = (int64_t)blockIdx.x * (kWarps / SPLIT) + warp / SPLIT;
  const int64_t row = s * kSlice + lane;
  const bool real = s < nslices;
  const int64_t ub = real ? uptr[s] : 0, lb = real ? lptr[s] : 0;
  const int ulen = real ? (int)((uptr[s + 1] - ub) >> 5) : 0;
  const int llen = real ? (int)((lptr[s + 1] - lb) >> 5) : 0;
  const int32_t* ucp = ucol + ub + lane;
  const TV* uvp = val + 9 * ub;
  const int32_t* lpp = lpos + lb + lane;
  const int32_t* lcp = lcol + lb + lane;
  auto load_lower = [&](int j, TV(&v)[9]) {
    const int64_t P = __ldcs(lpp + 32 * j);
    load_block(val + 9 * (P & ~int64_t(31)), (int)(P & 31), v);
  };
  int32_t cu[kAhead], cl[kAhead];
  TV vu[kAhead][9], vl[kAhead][9];
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    const int j = part + u * SPLIT;
    cu[u] = j < ulen ? __ldcs(ucp + 32 * j) : 0;
    cl[u] = j < llen ? __ldcs(lcp + 32 * j) : 0;
    if (j < ulen) load_block(uvp + 288 * (int64_t)j, lane, vu[u]);
    if (j < llen) load_lower(j, vl[u]);
  }
  pdl_enter();
  if (epi.halt()) return;
  TA a0 = TA(0), a1 = TA(0), a2 = TA(0);
  auto upper = [&](int64_t cj, const TV(&v)[9]) {
    const TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
    a0 += (TA)v[0] * x0 + (TA)v[1] * x1 + (TA)v[2] * x2;
    a1 += (TA)v[3] * x0 + (TA)v[4] * x1 + (TA)v[5] * x2;
    a2 += (TA)v[6] * x0 + (TA)v[7] * x1 + (TA)v[8] * x2;
  };
  // transposed block: (K_ji^T x)_r = sum_c K_ji[c][r] x_c
  auto lower = [&](int64_t cj, const TV(&v)[9]) {
    const TA x0 = (TA)__ldg(x + 3 * cj), x1 = (TA)__ldg(x + 3 * cj + 1), x2 = (TA)__ldg(x + 3 * cj + 2);
    a0 += (TA)v[0] * x0 + (TA)v[3] * x1 + (TA)v[6] * x2;
    a1 += (TA)v[1] * x0 + (TA)v[4] * x1 + (TA)v[7] * x2;
    a2 += (TA)v[2] * x0 + (TA)v[5] * x1 + (TA)v[8] * x2;
  };
#pragma unroll
  for (int u = 0; u < kAhead; ++u) {
    if (part + u * SPLIT < ulen) upper(cu[u], vu[u]);
    if (part + u * SPLIT < llen) lower(cl[u], vl[u]);
  }
  const int mlen = ulen > llen ? ulen : llen;
#pragma unroll 1
  for (int j = part + kAhead * SPLIT; j < mlen; j += SPLIT) {
    TV v[9];
    if (j < ulen) {
      const int64_t cj = __ldcs(ucp + 32 * j);
      load_block(uvp + 288 * (int64_t)j, lane, v);
      upper(cj, v);
    }
    if (j < llen) {
      const int64_t cj = __ldcs(lcp + 32 * j);
      load_lower(j, v);
      lower(cj, v);
    }
  }
  {
    __shared__ TA sh[kWarps][3][32];
    sh[warp][0][lane] = a0;
    sh[warp][1][lane] = a1;
    sh[warp][2][lane] = a2;
    __syncthreads();
    if (part == 0) {
#pragma unroll
      for (int q = 1; q < SPLIT; ++q) {
        a0 += sh[warp + q][0][lane];
        a1 += sh[warp + q][1][lane];
        a2 += sh[warp + q][2][lane];
      }
    }
  }
  double dot[1] = {0.0};
  if (part == 0 && s < nslices && row < N) {
    dot[0] = epi(row, a0, a1, a2, x);
  }
  if (EPI::kDot && epi.want_dot()) block_partial<1>(dot, partials);
}

inline int sym_grid(const Ctx* c) { return (int)((c->nslices * kSlice + kSpmvBlock - 1) / kSpmvBlock); }

int sm_count_solver() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  }
  return sms;
}

// Warps per SELL slice: the smallest power of two (<= 8) that puts at least
// 32 warps per SM in flight.
int spmv_split(const Ctx* c) {
  const int sms = sm_count_solver();
  int split = 1;
  while (split < 8 && c->nslices * split < (int64_t)sms * 32) split <<= 1;
  return split;
}

template <typename TV, typename TX, typename TA, bool DIFF, int SPLIT, class EPI>
int launch_spmv_split(const Ctx* c, cudaStream_t st, const TV* val, const TX* x, const EPI& epi) {
  // coded indices with FP32 values and one warp per slice only (measured on
  // B200: 192x96x96 FP32 product 297 against 325 us, FP64 582 against 568 us;
  // with SPLIT warps per slice each warp loads the row's 32 code bytes, more
  // than its share of 4-byte columns: J2 bar 53.7 against 51.8 us per CG
  // iteration)
  if constexpr (!DIFF && SPLIT == 1 && sizeof(TV) == 4) {
    if (c->full_coded) {
      constexpr int per_block = kSpmvBlock / 32;
      const int grid = (int)((c->nslices + per_block - 1) / per_block);
      return launch_product<EPI::kPdl>(k_spmvc<TV, TX, TA, EPI>, grid, kSpmvBlock, st, c->N, c->nslices, c->slice_ptr,
                               reinterpret_cast<const uint4*>(c->full_code), c->full_tab, val, x, epi, c->partials);
    }
  }
  if constexpr (SPLIT == 1) {
    const int grid = (int)((c->nslices * kSlice + kSpmvBlock - 1) / kSpmvBlock);
    return launch_product<EPI::kPdl>(k_spmv<TV, TX, TA, EPI, DIFF>, grid, kSpmvBlock, st, c->N, c->nslices * kSlice,
                             c->slice_ptr, c->sell_col, val, x, epi, c->partials);
  } else {
    constexpr int per_block = kSpmvBlock / 32 / SPLIT;
    const int grid = (int)((c->nslices + per_block - 1) / per_block);
    return launch_product<EPI::kPdl>(k_spmv_split<TV, TX, TA, EPI, DIFF, SPLIT>, grid, kSpmvBlock, st, c->N, c->nslices,
                             c->slice_ptr, c->sell_col, val, x, epi, c->partials);
  }
}

template <typename TV, typename TX, typename TA, bool DIFF, class EPI>
int launch_spmv_diff(const Ctx* c, cudaStream_t st, const TV* val, const TX* x, const EPI& epi) {
  switch (spmv_split(c)) {
    case 1: return launch_spmv_split<TV, TX, TA, DIFF, 1>(c, st, val, x, epi);
    case 2: return launch_spmv_split<TV, TX, TA, DIFF, 2>(c, st, val, x, epi);
    case 4: return launch_spmv_split<TV, TX, TA, DIFF, 4>(c, st, val, x, epi);
    default: return launch_spmv_split<TV, TX, TA, DIFF, 8>(c, st, val, x, epi);
  }
}

// SELL SpMV over the full (non-symmetric) storage; the FP32 difference form
// when the FP32 values were built that way.
template <typename TV, typename TX, typename TA, class EPI>
int launch_spmv(const Ctx* c, cudaStream_t st, const TV* val, const TX* x, const EPI& epi) {
  if constexpr (sizeof(TV) == 4) {
    if (c->val32_diff) return launch_spmv_diff<TV, TX, TA, true>(c, st, val, x, epi);
  }
  return launch_spmv_diff<TV, TX, TA, false>(c, st, val, x, epi);
}

template <typename TV, typename TX, typename TA, int SPLIT, class EPI>
int launch_spmv_sym_split(const Ctx* c, cudaStream_t st, const TV* val, const TX* x, const EPI& epi) {
  constexpr int per_block = kSpmvBlock / 32 / SPLIT;
  const int grid = (int)((c->nslices + per_block - 1) / per_block);
  return launch_product<EPI::kPdl>(k_spmv_sym_split<TV, TX, TA, EPI, SPLIT>, grid, kSpmvBlock, st, c->N, c->nslices, c->uptr,
                           c->ucol, c->lptr, c->lpos, c->lcol, val, x, epi, c->partials);
}

// The symmetric product: one warp per slice (grid = slices / 8 blocks), or
// SPLIT warps per slice on small meshes (the rule of spmv_split).
template <typename TV, typename TX, typename TA, class EPI>
int launch_spmv_sym(const Ctx* c, cudaStream_t st, const TV* val, const TX* x, const EPI& epi) {
  const int grid = sym_grid(c);
  switch (spmv_split(c)) {
    case 1:
      if (c->sym_coded)
        return launch_product<EPI::kPdl>(k_spmv_symc<TV, TX, TA, EPI>,
                                 sizeof(TV) == 8 ? std::min(grid, 15 * sm_count_solver()) : grid, kSpmvBlock, st, c->N,
                                 c->nslices * kSlice, c->uptr, c->lptr, reinterpret_cast<const uint4*>(c->sym_ucode),
                                 reinterpret_cast<const uint4*>(c->sym_lcode), c->sym_tab, val, x, epi, c->partials);
      return launch_product<EPI::kPdl>(k_spmv_sym<TV, TX, TA, EPI>, grid, kSpmvBlock, st, c->N, c->nslices * kSlice, c->uptr,
                               c->ucol, c->lptr, c->lpos, c->lcol, val, x, epi, c->partials);
    case 2: return launch_spmv_sym_split<TV, TX, TA, 2>(c, st, val, x, epi);
    case 4: return launch_spmv_sym_split<TV, TX, TA, 4>(c, st, val, x, epi);
    default: return launch_spmv_sym_split<TV, TX, TA, 8>(c, st, val, x, epi);
  }
}

// Sum of the nb per-block partials of the product, for grids too large to be
// summed again by every block of the update: one block, result in out[0].
__global__ void __launch_bounds__(1024)
    k_cg_sum(const double* __restrict__ partials, int nb, double* __restrict__ out, const CgScalars* __restrict__ scal) {
  pdl_enter();
  if (halted(scal)) return;
  double tot[1];
  sum_partials<1>(partials, nb, tot);
  if (threadIdx.x == 0) out[0] = tot[0];
}

// The product's partials for the update: as they are, or summed first by one
// block when every block of the update would have to read more than
// kMaxPartials of them.
constexpr int kMaxPartials = 2560;
struct Partials {
  const double* p;
  int nb;
};
Partials product_partials(Ctx* c, cudaStream_t st, int nb) {
  if (nb <= kMaxPartials) return {c->partials, nb};
  double* out = c->partials + c->partials_cap - 1;
  launch_pdl(k_cg_sum, 1, 1024, st, (const double*)c->partials, nb, out, (const CgScalars*)c->scal);
  c->launches += 1;
  return {out, 1};
}

}  // namespace
}  // namespace ufc
