// C3D8 element kernels: stiffness assembly, matrix-free FP64 operator,
// internal force with the J2 return map, Gauss-point stress, material-point
// batch update and the adjoint sensitivity.
//
// Assembly is deterministic without floating-point atomics: the stiffness is
// assembled by block rows, each value summed by one thread in ascending element
// order and written once; element vectors (forces, nodal stresses) are written
// per element node and summed by one thread per node in ascending element order.
#include <cuda_runtime.h>

#include <algorithm>

#include "c3d8_device.cuh"
#include "octet.cuh"
#include "reduce.cuh"
#include "rows.cuh"
#include "ufc_internal.cuh"

namespace ufc {

namespace {

// ---- stiffness assembly by block rows
//
// Every stored block (i, j) is the sum, over the elements that hold both nodes,
// of sum_gp w detJ B_i^T D B_j.  A CTA owns half a SELL slice (16 block rows),
// accumulates them in shared memory and writes each stored value once; nothing
// is read back and no two threads touch the same entry, so there are no
// atomics, no colour passes and no zero fill, and each entry receives its
// contributions in ascending element order (bitwise reproducible).
//
// A warp works on 4 rows at a time, 8 lanes per row.  For the row's k-th
// element, lane t first takes Gauss point t (its scaled inverse Jacobian
// adj(J)/sqrt(detJ) goes to shared memory: with that scaling on both sides the
// weight detJ needs no separate product), then takes the element's node t and
// forms the block (row node, node t) over the 8 Gauss points.  Lane t's node
// is the one whose natural coordinates have the sign bits t, and the trilinear
// factor of node t at Gauss point g equals that of node g at Gauss point t, so
// one table of 12 products per lane serves the Jacobian and the gradients.
// The linear-elastic block is formed from G = sum_gp g_a (x) g_b as
// lam G + mu G^T + mu tr(G) I (72 + 21 FP64 operations per block instead of
// about 320 when D is applied at every Gauss point); the J2 block as
// sum_gp (D B_a)^T B_b with D B_a formed once per (row, element, Gauss point).
//
// Rounding must not have one sign in every element: the response of an element
// to a rigid translation, zero but for rounding, then adds up along a slender
// box like an elastic foundation.  So (1) the Jacobian is summed over the nodes'
// coordinates instead of taken from coordinate differences, which are exact and
// the same in all elements of a regular box, and (2) the linear-elastic block of
// the row's own node is minus the sum of the row's other seven.  Displacements
// of 80x4x4 elements of one modulus against extended precision: 1e-9 with
// differences and all eight blocks summed alike, 2e-11 now; 40x8x8 with lognormal
// moduli 1.7e-12 and 2e-13.
//
// What bounds it: the shared-memory pipe (97 % busy, 400 wavefronts per element
// of 4 rows; FP64 35 %).  It serves the J2 tangents, and linear-elastic rows too
// long for the shared memory of the one-thread form below.  Recomputing an
// element's Jacobians for each of its 8 rows costs less than the
// read-modify-write of the values that an element-wise scatter needs (16.6 GB at
// 192x96x96, in 8 colour passes).
constexpr int kAsmRows = 16;                // rows per CTA
constexpr int kAsmWarps = kAsmRows / 4;
constexpr int kAsmMaxSmem = 227 * 1024;     // dynamic shared memory of one CTA

// Shared memory of one warp.
template <typename T, bool kTangent>
struct AsmWarp {
  T X[4][26];                             // element coordinates by sign bits, [row][3 bits + i], padded
  T P[4][8][kTangent ? 28 : 10];          // [row][gp]: scaled inverse Jacobian (9), then D B_a (18) for J2
};

// The stored matrix is symmetric to the last bit: the blocks (a, b) and (b, a) of
// an element come from different threads, so what both form is written as fused
// multiply-adds in a given order and not left to the compiler's contraction.
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Component i of a node's gradient from its reference derivatives.
template <typename T>
__device__ __forceinline__ T grad_at(const T* inv, int i, T d0, T d1, T d2) {
  return fma_t(inv[3 * i + 2], d2, fma_t(inv[3 * i + 1], d1, inv[3 * i] * d0));
}

// Entry (i, j) of lam G + mu G^T + mu tr(G) I.
template <typename T>
__device__ __forceinline__ T iso_entry(const T* G, T lam, T mu, T tr, int i, int j) {
  const T v = fma_t(lam, G[3 * i + j], mu * G[3 * j + i]);
  return i == j ? fma_t(mu, tr, v) : v;
}

// Entry (i, j) of the symmetric part of a 3x3 block.
template <typename T>
__device__ __forceinline__ T sym_part(const T (&v)[9], int i, int j) {
  return i == j ? v[4 * i] : T(0.5) * (v[3 * i + j] + v[3 * j + i]);
}

template <typename T, bool kTangent>
__global__ void __launch_bounds__(kAsmWarps * 32)
    k_assemble_rows(int32_t N, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nelem,
                    const double* __restrict__ coords, const int32_t* __restrict__ conn,
                    const double* __restrict__ lame, const double* __restrict__ Dt, const int32_t* __restrict__ slot,
                    const int64_t* __restrict__ sptr, const int32_t* __restrict__ scol,
                    const int32_t* __restrict__ dpos, const uint8_t* __restrict__ fixed, int stride,
                    const RowOutputs<T> to, int32_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char asm_smem[];
  using Warp = AsmWarp<T, kTangent>;
  Warp* wsm = reinterpret_cast<Warp*>(asm_smem);
  T* acc = reinterpret_cast<T*>(asm_smem + sizeof(Warp) * kAsmWarps);  // [row][stride], 9 per entry, stride odd
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, rr = lane >> 3, t = lane & 7;
  const int64_t s = blockIdx.x >> 1;
  const int half = (blockIdx.x & 1) * kAsmRows;
  const int64_t base = sptr[s];
  const int len = (int)((sptr[s + 1] - base) >> 5);
  RowWriter<T, kAsmRows, kAsmWarps * 32> out;
  out.init(N, s, half, base, len, scol, dpos, fixed);
  for (int q = threadIdx.x; q < kAsmRows * stride; q += kAsmWarps * 32) acc[q] = T(0);
  __syncthreads();

  Warp& sm = wsm[w];
  const int64_t row = s * kSlice + half + 4 * w + rr;
  T* arow = acc + (4 * w + rr) * stride;
  const int node_t = bits_node(t);
  // trilinear factors of lane t: c[d][m] = (1/8) prod over the two other
  // directions of (1 + s_t s_m g), m = the bits of those directions in order
  const T g = T(0.57735026918962576451);
  T c[3][4];
  {
    const T f0[2] = {T(1) + ((t & 1) ? -g : g), T(1) + ((t & 1) ? g : -g)};
    const T f1[2] = {T(1) + ((t & 2) ? -g : g), T(1) + ((t & 2) ? g : -g)};
    const T f2[2] = {T(1) + ((t & 4) ? -g : g), T(1) + ((t & 4) ? g : -g)};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      c[0][m] = T(0.125) * f1[m & 1] * f2[m >> 1];
      c[1][m] = T(0.125) * f0[m & 1] * f2[m >> 1];
      c[2][m] = T(0.125) * f0[m & 1] * f1[m >> 1];
    }
  }
  const int32_t kb = row < N ? nptr[row] : 0, ke = row < N ? nptr[row + 1] : 0;
  const int kmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)(ke - kb));
  bool bad = false;
  // the element of step k + 1 is fetched while step k is worked on
  int32_t el = 0, pos = 0;
  T x0 = T(0), x1 = T(0), x2 = T(0);
  auto fetch = [&](int k) {
    if (kb + k >= ke) return;
    el = nelem[kb + k];
    const int64_t e = el >> 3;
    const int64_t nd = conn[e * 8 + node_t];
    pos = slot[e * 64 + (el & 7) * 8 + node_t];
    x0 = (T)coords[nd * 3];
    x1 = (T)coords[nd * 3 + 1];
    x2 = (T)coords[nd * 3 + 2];
  };
  fetch(0);
  for (int k = 0; k < kmax; ++k) {
    const bool on = kb + k < ke;
    const int64_t e = el >> 3;
    const int ta = bits_node(el & 7);  // the row's own node in sign bits
    const int j = (int)((pos - base) >> 5);
    sm.X[rr][3 * t] = x0;
    sm.X[rr][3 * t + 1] = x1;
    sm.X[rr][3 * t + 2] = x2;
    T lam = T(0), mu = T(0), D[kTangent ? 21 : 1];
    if (on) {
      if (kTangent) {
#pragma unroll
        for (int q = 0; q < 21; ++q) D[kTangent ? q : 0] = (T)Dt[(e * 21 + q) * 8 + t];
      } else {
        lam = (T)lame[2 * e];
        mu = (T)lame[2 * e + 1];
      }
    }
    fetch(k + 1);
    __syncwarp();
    if (on) {
      // Gauss point t: J_di = dx_i / dxi_d, summed over the nodes
      const T* X = sm.X[rr];
      T J[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) J[i] = T(0);
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const T d0 = flip_if(c[0][m >> 1], !(m & 1)), d1 = flip_if(c[1][(m & 1) | ((m >> 1) & 2)], !(m & 2)),
                d2 = flip_if(c[2][m & 3], !(m & 4));
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const T x = X[3 * m + i];
          J[i] += d0 * x;
          J[3 + i] += d1 * x;
          J[6 + i] += d2 * x;
        }
      }
      const T a0 = J[4] * J[8] - J[5] * J[7], a3 = J[5] * J[6] - J[3] * J[8], a6 = J[3] * J[7] - J[4] * J[6];
      const T det = J[0] * a0 + J[1] * a3 + J[2] * a6;
      bad |= !(det > T(0));
      const T q = rsqrt(det);
      T inv[9] = {a0 * q, (J[2] * J[7] - J[1] * J[8]) * q, (J[1] * J[5] - J[2] * J[4]) * q,
                  a3 * q, (J[0] * J[8] - J[2] * J[6]) * q, (J[2] * J[3] - J[0] * J[5]) * q,
                  a6 * q, (J[1] * J[6] - J[0] * J[7]) * q, (J[0] * J[4] - J[1] * J[3]) * q};
      T* P = sm.P[rr][t];
#pragma unroll
      for (int i = 0; i < 9; ++i) P[i] = inv[i];
      if (kTangent) {
        // D B_a of the row's node at this Gauss point
        const T b0 = T(1) + ((((ta ^ t) & 1) != 0) ? -g : g), b1 = T(1) + ((((ta ^ t) & 2) != 0) ? -g : g),
                b2 = T(1) + ((((ta ^ t) & 4) != 0) ? -g : g);
        const T d0 = flip_if(T(0.125) * b1 * b2, !(ta & 1)), d1 = flip_if(T(0.125) * b0 * b2, !(ta & 2)),
                d2 = flip_if(T(0.125) * b0 * b1, !(ta & 4));
        T ga[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) ga[i] = grad_at(inv, i, d0, d1, d2);
        // B column i of a node has non-zeros at Voigt rows kIdx[i][m] with
        // gradient component kCmp[i][m] (PH_Elem_ShapeFunc.f90:225-244)
        constexpr int kIdx[3][3] = {{0, 3, 5}, {1, 3, 4}, {2, 4, 5}};
        constexpr int kCmp[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
#pragma unroll
        for (int v = 0; v < 6; ++v)
#pragma unroll
          for (int i = 0; i < 3; ++i)
            P[(kTangent ? 9 : 0) + v * 3 + i] = D[kTangent ? tri6(v, kIdx[i][0]) : 0] * ga[kCmp[i][0]] +
                                                D[kTangent ? tri6(v, kIdx[i][1]) : 0] * ga[kCmp[i][1]] +
                                                D[kTangent ? tri6(v, kIdx[i][2]) : 0] * ga[kCmp[i][2]];
      }
    }
    __syncwarp();
    T K[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) K[i] = T(0);
#pragma unroll
    for (int gp = 0; gp < 8; ++gp) {
      const T* P = sm.P[rr][gp];
      const int p0 = gp & 1, p1 = (gp >> 1) & 1, p2 = gp >> 2;
      const T d0 = flip_if(c[0][p1 + 2 * p2], !(t & 1)), d1 = flip_if(c[1][p0 + 2 * p2], !(t & 2)),
              d2 = flip_if(c[2][p0 + 2 * p1], !(t & 4));
      T gb[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) gb[i] = grad_at(P, i, d0, d1, d2);
      if (kTangent) {
        constexpr int kIdx[3][3] = {{0, 3, 5}, {1, 3, 4}, {2, 4, 5}};
        constexpr int kCmp[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
        const T* M = P + (kTangent ? 9 : 0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int jj = 0; jj < 3; ++jj)
            K[3 * i + jj] += M[kIdx[jj][0] * 3 + i] * gb[kCmp[jj][0]] + M[kIdx[jj][1] * 3 + i] * gb[kCmp[jj][1]] +
                             M[kIdx[jj][2] * 3 + i] * gb[kCmp[jj][2]];
      } else {
        T ga[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) ga[i] = __shfl_sync(0xffffffffu, gb[i], ta, 8);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) K[3 * i + jj] = fma_t(ga[i], gb[jj], K[3 * i + jj]);
      }
    }
    if (!kTangent) {
      const T tr = K[0] + K[4] + K[8];
      T v[9], own[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) v[3 * i + jj] = iso_entry(K, lam, mu, tr, i, jj);
      // the row node's own block is minus the sum of the others
#pragma unroll
      for (int i = 0; i < 9; ++i) own[i] = t == ta ? T(0) : -v[i];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int i = 0; i < 9; ++i) own[i] += __shfl_xor_sync(0xffffffffu, own[i], o, 8);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) K[3 * i + jj] = t == ta ? sym_part(own, i, jj) : v[3 * i + jj];
    } else if (t == ta) {
      const T v[9] = {K[0], K[1], K[2], K[3], K[4], K[5], K[6], K[7], K[8]};
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) K[3 * i + jj] = sym_part(v, i, jj);
    }
    if (on) {
      T* d = arow + 9 * j;
#pragma unroll
      for (int i = 0; i < 9; ++i) d[i] += K[i];
    }
    __syncwarp();  // the warp's shared memory is consumed
  }
  if (bad) atomicOr(err, (int)kDevBadJacobian);
  __syncthreads();

  out.write(len, scol, fixed, acc, stride, to);
}

// The linear-elastic assembly with one thread per (block row, element): the
// whole element is worked through in registers (72 accumulators of the row's 8
// blocks), so the lanes exchange nothing and shared memory only takes the
// element coordinates and the finished blocks.  A CTA owns one SELL slice of 32
// rows; warp q takes the elements k = q, q + 4, ... of all 32 rows, and the
// warps add their blocks in turn (named barriers pass the turn on), so each
// entry still receives its contributions in ascending element order.  The
// coordinates of a thread's next element come by cp.async while the current one
// is worked on.  The Jacobian's node sums (see above) are taken per eta and zeta
// for both faces xi = -1 and +1, so that they read the coordinates no oftener
// than differences along the edges would.  128x64x64, FP64 with FP32 copies, the
// call with its products: 1.80 ms (1.66 ms with edge differences; node sums
// formed at every Gauss point 2.26 ms; the colour-ordered element scatter before
// 6.26 ms).  The kernel is bound by latency and FP64 (8 warps per SM; the
// accumulators take the registers).
constexpr int kIsoWarps = 4;
constexpr int kIsoThreads = kIsoWarps * 32;
constexpr int kIsoXBytes = kIsoWarps * 2 * 24 * 32 * (int)sizeof(double);  // [warp][stage][coordinate][lane]

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kIsoThreads, 2)
    k_assemble_iso(int32_t N, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nelem,
                   const double* __restrict__ coords, const int32_t* __restrict__ conn,
                   const double* __restrict__ lame, const int32_t* __restrict__ slot,
                   const int64_t* __restrict__ sptr, const int32_t* __restrict__ scol,
                   const int32_t* __restrict__ dpos, const uint8_t* __restrict__ fixed, int stride,
                   const RowOutputs<T> to, int32_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char asm_smem[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* xs = reinterpret_cast<double*>(asm_smem) + w * (2 * 24 * 32) + lane;
  T* acc = reinterpret_cast<T*>(asm_smem + kIsoXBytes);  // [row][stride]
  const int64_t s = blockIdx.x;
  const int64_t base = sptr[s];
  const int len = (int)((sptr[s + 1] - base) >> 5);
  for (int i = threadIdx.x; i < kSlice * stride; i += kIsoThreads) acc[i] = T(0);
  const int64_t row = s * kSlice + lane;
  const int32_t ke = row < N ? nptr[row + 1] : 0;
  int32_t k = (row < N ? nptr[row] : 0) + w;
  const int rounds =
      ((int)__reduce_max_sync(0xffffffffu, (unsigned)(row < N ? ke - (k - w) : 0)) + kIsoWarps - 1) / kIsoWarps;
  const T g = T(0.57735026918962576451);
  const T hp = T(0.5) + T(0.5) * g, hm = T(0.5) - T(0.5) * g;  // (1 +- g) / 2
  bool bad = false;
  // an element's coordinates into this thread's column of stage r, by sign bits (xi fastest)
  auto load_x = [&](const int4& n0, const int4& n1, int r) {
    const int32_t nd[8] = {n0.x, n0.y, n0.w, n0.z, n1.x, n1.y, n1.w, n1.z};
    double* dst = xs + (r & 1) * (24 * 32);
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
      for (int i = 0; i < 3; ++i) cp_async8(dst + 32 * (3 * m + i), coords + (int64_t)nd[m] * 3 + i);
  };
  int32_t el = k < ke ? nelem[k] : 0, el_next = k + kIsoWarps < ke ? nelem[k + kIsoWarps] : 0;
  if (k < ke) {
    const int4* cn = reinterpret_cast<const int4*>(conn + (int64_t)(el >> 3) * 8);
    load_x(cn[0], cn[1], 0);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  RowWriter<T, kSlice, kIsoThreads> out;
  out.init(N, s, 0, base, len, scol, dpos, fixed);
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < rounds; ++r) {
    const bool on = k < ke, more = k + kIsoWarps < ke;
    const int64_t e = el >> 3;
    const int a = el & 7, ta = bits_node(a);
    const double* X = xs + (r & 1) * (24 * 32);
    int4 n0 = make_int4(0, 0, 0, 0), n1 = n0;
    if (more) {
      const int4* cn = reinterpret_cast<const int4*>(conn + (int64_t)(el_next >> 3) * 8);
      n0 = cn[0];
      n1 = cn[1];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    T G[8][9];
#pragma unroll
    for (int b = 0; b < 8; ++b)
#pragma unroll
      for (int i = 0; i < 9; ++i) G[b][i] = T(0);
#pragma unroll 1
    for (int iz = 0; iz < 2; ++iz) {
      const T fz = ((ta >> 2) == iz) ? hp : hm;  // factors (1 + s g) / 2 of the row's node
#pragma unroll 1
      for (int iy = 0; iy < 2; ++iy) {
        if (!on) continue;
        const T fy = (((ta >> 1) & 1) == iy) ? hp : hm;
        // products of the element nodes' factors in two directions, by the nodes' bits in them
        const T y0 = iy ? hm : hp, y1 = iy ? hp : hm, z0 = iz ? hm : hp, z1 = iz ? hp : hm;
        const T pyz[4] = {T(0.5) * (y0 * z0), T(0.5) * (y1 * z0), T(0.5) * (y0 * z1), T(0.5) * (y1 * z1)};
        // node sums for the Jacobian: d x / d xi, and the eta and zeta derivatives on the faces xi = -1 and +1
        T Jx[3], Je[2][3], Jz[2][3];
#pragma unroll
        for (int i = 0; i < 3; ++i) Jx[i] = Je[0][i] = Je[1][i] = Jz[0][i] = Jz[1][i] = T(0);
#pragma unroll
        for (int b = 0; b < 8; ++b)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const T x = (T)X[32 * (3 * b + i)];
            Jx[i] += flip_if(pyz[b >> 1], !(b & 1)) * x;
            Je[b & 1][i] += flip_if(T(0.5) * ((b & 4) ? z1 : z0), !(b & 2)) * x;
            Jz[b & 1][i] += flip_if(T(0.5) * ((b & 2) ? y1 : y0), !(b & 4)) * x;
          }
#pragma unroll 1
        for (int ix = 0; ix < 2; ++ix) {
          const T fx = ((ta & 1) == ix) ? hp : hm;
          const T x0 = ix ? hm : hp, x1 = ix ? hp : hm;
          T J[9];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            J[i] = Jx[i];
            J[3 + i] = x0 * Je[0][i] + x1 * Je[1][i];
            J[6 + i] = x0 * Jz[0][i] + x1 * Jz[1][i];
          }
          const T c0 = J[4] * J[8] - J[5] * J[7], c3 = J[5] * J[6] - J[3] * J[8], c6 = J[3] * J[7] - J[4] * J[6];
          const T det = J[0] * c0 + J[1] * c3 + J[2] * c6;
          bad |= !(det > T(0));
          const T sc = rsqrt(det);
          const T inv[9] = {c0 * sc, (J[2] * J[7] - J[1] * J[8]) * sc, (J[1] * J[5] - J[2] * J[4]) * sc,
                            c3 * sc, (J[0] * J[8] - J[2] * J[6]) * sc, (J[2] * J[3] - J[0] * J[5]) * sc,
                            c6 * sc, (J[1] * J[6] - J[0] * J[7]) * sc, (J[0] * J[4] - J[1] * J[3]) * sc};
          const T a0 = flip_if(T(0.5) * (fy * fz), !(ta & 1)), a1 = flip_if(T(0.5) * (fx * fz), !(ta & 2)),
                  a2 = flip_if(T(0.5) * (fx * fy), !(ta & 4));
          T ga[3];
#pragma unroll
          for (int i = 0; i < 3; ++i) ga[i] = grad_at(inv, i, a0, a1, a2);
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const T b0 = flip_if(pyz[b >> 1], !(b & 1)),
                    b1 = flip_if(T(0.5) * (((b & 1) ? x1 : x0) * ((b & 4) ? z1 : z0)), !(b & 2)),
                    b2 = flip_if(T(0.5) * (((b & 1) ? x1 : x0) * ((b & 2) ? y1 : y0)), !(b & 4));
            T gb[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) gb[i] = grad_at(inv, i, b0, b1, b2);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
              for (int jj = 0; jj < 3; ++jj) G[b][3 * i + jj] = fma_t(ga[i], gb[jj], G[b][3 * i + jj]);
          }
        }
      }
      if (iz == 0) {  // the next element's coordinates
        if (more) load_x(n0, n1, r + 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
    }
    k += kIsoWarps;
    el = el_next;
    el_next = k + kIsoWarps < ke ? nelem[k + kIsoWarps] : 0;
    T lam = T(0), mu = T(0);
    int4 s0 = make_int4(0, 0, 0, 0), s1 = s0;
    if (on) {
      const int4* sl = reinterpret_cast<const int4*>(slot + e * 64 + a * 8);
      s0 = sl[0];
      s1 = sl[1];
      lam = (T)lame[2 * e];
      mu = (T)lame[2 * e + 1];
    }
    // the turn of this warp: after warp w - 1 in this round (warp 3 of the round before)
    if (r > 0 || w > 0) bar_sync(1 + w, 64);
    if (on) {
      const int32_t ps[8] = {s0.x, s0.y, s0.w, s0.z, s1.x, s1.y, s1.w, s1.z};
      // the row node's own block is minus the sum of the others
      T own[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) own[i] = T(0);
      int pos = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        if (b == ta) {
          pos = ps[b];
          continue;
        }
        T* d = acc + lane * stride + 9 * (int)((ps[b] - base) >> 5);
        const T tr = G[b][0] + G[b][4] + G[b][8];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) {
            const T v = iso_entry(G[b], lam, mu, tr, i, jj);
            d[3 * i + jj] += v;
            own[3 * i + jj] -= v;
          }
      }
      T* d = acc + lane * stride + 9 * (int)((pos - base) >> 5);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jj = 0; jj < 3; ++jj) d[3 * i + jj] += sym_part(own, i, jj);
    }
    if (r + 1 < rounds || w + 1 < kIsoWarps) {
      __threadfence_block();
      bar_arrive(1 + (w + 1) % kIsoWarps, 64);
    }
  }
  if (bad) atomicOr(err, (int)kDevBadJacobian);
  __syncthreads();
  out.write(len, scol, fixed, acc, stride, to);
}

// Lower blocks from the upper ones, transposed.  The J2 block (a, b) is formed as
// (D B_a)^T B_b and (b, a) as (D B_b)^T B_a, the same but for rounding; the upper
// one stands for both, as in the symmetric storage.  A CTA per slice, its warps
// take the rows' entries in turn, so that a thread's chain (column, search in that
// column's row, block) is short and the stores of an entry's 32 rows lie together:
// bound by the latency of that chain.  Tangent assembly at 16x8x8, 32x16x16 and
// 64x32x32 without it / with it / with one thread per row: 62 / 70 / 115, 120 / 126
// / 173 and 436 / 467 / 524 us.
constexpr int kMirrorWarps = 8;

template <typename T>
__global__ void __launch_bounds__(kMirrorWarps * 32)
    k_mirror_lower(int32_t N, const int32_t* __restrict__ brow, const int32_t* __restrict__ bcol,
                   const int64_t* __restrict__ sptr, T* __restrict__ val, float* __restrict__ val_r) {
  const int64_t s = blockIdx.x, r = s * kSlice + (threadIdx.x & 31);
  if (r >= N) return;
  const int64_t P0 = sptr[s] + (threadIdx.x & 31);
  const int32_t b = brow[r], e = brow[r + 1];
  for (int32_t k = b + (int32_t)(threadIdx.x >> 5); k < e; k += kMirrorWarps) {
    const int32_t c = bcol[k];
    if (c >= r) break;
    int32_t lo = brow[c], hi = brow[c + 1] - 1;  // row c holds column r: the pattern is symmetric
    const int32_t first = lo;
    while (lo < hi) {
      const int32_t mid = (lo + hi) >> 1;
      if (bcol[mid] < r) lo = mid + 1;
      else hi = mid;
    }
    const int64_t src = sptr[c >> 5] + 32 * (int64_t)(lo - first) + (c & 31), dst = P0 + 32 * (int64_t)(k - b);
    T v[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) v[q] = val[vpos(src, q)];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        val[vpos(dst, 3 * i + j)] = v[3 * j + i];
        if (val_r) val_r[vpos(dst, 3 * i + j)] = (float)v[3 * j + i];
      }
  }
}

// Lame constants of every element, [E][2].
__global__ void k_lame(int32_t E, const double* __restrict__ props, int nprops, double* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  double lam, mu;
  lame<double>(props[e * nprops], props[e * nprops + 1], lam, mu);
  out[2 * e] = lam;
  out[2 * e + 1] = mu;
}

// Difference form: the diagonal slot of each block row holds the FP64 block
// row sum S_i = sum_j K_ij, rounded once (one thread per block row).
__global__ void k_diag_rowsum(int32_t N, const int64_t* __restrict__ sptr, const int32_t* __restrict__ dpos,
                              const double* __restrict__ v64, float* __restrict__ v32) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int64_t s = i >> 5, t = i & 31;
  const int64_t base = sptr[s], len = (sptr[s + 1] - base) >> 5;
  double S[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) S[c] = 0.0;
  for (int64_t j = 0; j < len; ++j) {
    const int64_t P = base + j * 32 + t;
#pragma unroll
    for (int c = 0; c < 9; ++c) S[c] += v64[vpos(P, c)];
  }
  const int64_t d = dpos[i];
#pragma unroll
  for (int c = 0; c < 9; ++c) v32[vpos(d, c)] = (float)S[c];
}

// ---- element vectors
//
// Internal forces and matrix-free operators run in two kernels: every element's
// nodal forces by octets (octet.cuh) into an element-ordered array, then each
// node sums those of its elements in ascending order.  One pass over the mesh
// instead of one launch per colour with read-modify-write of the result.
// 97x51x47 (232,509 elements): 8 launches of 16.5 us per operator application,
// now 50.5 + 12.8 us; 192x96x96: 801 us, now 465 + 96.  The octets are bound by
// the shuffles (108 a lane), the node sums by the 192 bytes per element between
// the two.  J2 at 64x32x32, return map and forces: 151 + 8 x 13 us, now 75 + 6.
// The array holds at most kFeElems elements (50 MB): larger meshes go through it
// in element order, each node adding to the sum of the passes before, so that
// the result is the same to the last bit and the scratch does not grow with the
// mesh (192 bytes per element would be a twentieth of a refined model).
constexpr int kOctBlock = 256;
constexpr int32_t kFeElems = 1 << 18;

// The octet's element of this thread, clamped (all lanes take part in the
// exchanges; `real` says whether to write), its node and coordinates.
struct OctElem {
  int64_t e;
  int t, a;
  int64_t node;
  bool real;
  double X[3];
  // elements [e0, e1)
  __device__ __forceinline__ OctElem(int32_t e0, int32_t e1, const double* __restrict__ coords,
                                     const int32_t* __restrict__ conn) {
    const int64_t k = e0 + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3);
    real = k < e1;
    e = real ? k : e1 - 1;
    t = threadIdx.x & 7;
    a = bits_node(t);
    node = conn[e * 8 + a];
#pragma unroll
    for (int i = 0; i < 3; ++i) X[i] = coords[3 * node + i];
  }
};

// Nodal forces of the elements [e0, e1), fe[(8 (e - e0) + a) 3 + i]:
//   kIso      B^T D B x with the linear-elastic D (masked by `fixed` when given);
//             the internal force of the material (PH_Elem_C3D8_IntForce, PH_Elem_C3D8.f90:734-757)
//   kTangent  B^T D_gp B x with the tangents of the last return map (unmasked);
//             Newton lifts a prescribed displacement increment with it
enum ForceMode { kIso, kTangent };

template <int MODE>
__global__ void __launch_bounds__(kOctBlock)
    k_oct_force(int32_t e0, int32_t e1, const double* __restrict__ coords, const int32_t* __restrict__ conn,
                const double* __restrict__ lame, const double* __restrict__ Dt, const double* __restrict__ x,
                const uint8_t* __restrict__ fixed, double* __restrict__ fe, int32_t* __restrict__ err) {
  const OctElem el(e0, e1, coords, conn);
  const Octet oct(el.t);
  double u[3], inv[9], eps[6], s[6], f[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int64_t d = 3 * el.node + i;
    u[i] = (fixed && fixed[d]) ? 0.0 : x[d];
  }
  const double det = oct.jacobian(el.X, inv);
  oct.strain(inv, u, eps);
  if (MODE == kIso) {
    if (!(det > 0.0)) atomicOr(err, (int)kDevBadJacobian);
    iso_stress<double>(lame[2 * el.e], lame[2 * el.e + 1], eps, s);
  } else {
    const double* D = Dt + el.e * 168 + el.t;  // [21][8 Gauss points]
    double d[21];
#pragma unroll
    for (int k = 0; k < 21; ++k) d[k] = D[8 * k];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      s[i] = 0.0;
#pragma unroll
      for (int j = 0; j < 6; ++j) s[i] += d[tri6(i, j)] * eps[j];
    }
  }
  oct.nodal_force(inv, det, s, f);
  if (el.real)
#pragma unroll
    for (int i = 0; i < 3; ++i) fe[((el.e - e0) * 8 + el.a) * 3 + i] = f[i];
}

// J2 return map at every Gauss point: strain increment from du = u - u_n,
// committed state (sig_n, epeq_n, epl_n) -> trial state, consistent tangent and
// the element's nodal forces of the trial stress.
__global__ void __launch_bounds__(kOctBlock)
    k_oct_j2(int32_t e0, int32_t e1, const double* __restrict__ coords, const int32_t* __restrict__ conn,
             const double* __restrict__ props, int nprops, const double* __restrict__ u,
             const double* __restrict__ u_n, const double* __restrict__ sig_n, const double* __restrict__ epeq_n,
             const double* __restrict__ epl_n, double* __restrict__ sig_t, double* __restrict__ epeq_t,
             double* __restrict__ epl_t, double* __restrict__ Dt, double* __restrict__ fe,
             int32_t* __restrict__ err) {
  const OctElem el(e0, e1, coords, conn);
  const Octet oct(el.t);
  const int64_t g = el.e * 8 + el.t;
  double du[3], inv[9], de[6], s[6], epl[6], D[36], epeq, f[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) du[i] = u[3 * el.node + i] - u_n[3 * el.node + i];
  const double det = oct.jacobian(el.X, inv);
  if (!(det > 0.0)) atomicOr(err, (int)kDevBadJacobian);
  oct.strain(inv, du, de);
  j2_update(props + el.e * nprops, de, sig_n + g * 6, epeq_n[g], epl_n + g * 6, s, &epeq, epl, D);
  bool finite = isfinite(epeq);
#pragma unroll
  for (int i = 0; i < 6; ++i) finite &= isfinite(s[i]);
  if (!finite) atomicOr(err, (int)kDevNonFinite);
  if (el.real) {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      sig_t[g * 6 + i] = s[i];
      epl_t[g * 6 + i] = epl[i];
    }
    epeq_t[g] = epeq;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j) Dt[el.e * 168 + 8 * tri6(i, j) + el.t] = D[i * 6 + j];
  }
  oct.nodal_force(inv, det, s, f);
  if (el.real)
#pragma unroll
    for (int i = 0; i < 3; ++i) fe[((el.e - e0) * 8 + el.a) * 3 + i] = f[i];
}

// y_i = sum of the element forces at DOF i, elements ascending; PART: of the
// elements [e0, e1), added to what the passes before them left (e0 = 0: none).
// With `x` the eliminated operator: y = x on fixed DOFs (identity rows).
template <bool PART>
__global__ void __launch_bounds__(256)
    k_node_sum(int64_t n, int32_t e0, int32_t e1, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nelem,
               const double* __restrict__ fe, const uint8_t* __restrict__ fixed, const double* __restrict__ x,
               double* __restrict__ y) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t node = i / 3;
  const int c = (int)(i - 3 * node);
  const int32_t k0 = nptr[node], k1 = nptr[node + 1];
  double s = 0.0;
  if constexpr (PART) {
    const int64_t lo = 8 * (int64_t)e0, hi = 8 * (int64_t)e1;
    if (e0 > 0) {
      if (k0 == k1 || nelem[k1 - 1] < lo || nelem[k0] >= hi) return;  // the node has none of these elements
      s = y[i];
    }
    for (int32_t k = k0; k < k1; ++k) {
      const int64_t el = nelem[k];
      if (el >= lo && el < hi) s += fe[3 * (el - lo) + c];
    }
  } else {
#pragma unroll 4
    for (int32_t k = k0; k < k1; ++k) s += fe[3 * (int64_t)nelem[k] + c];
  }
  y[i] = (x && fixed[i]) ? x[i] : s;
}

__device__ __forceinline__ double von_mises(const double s[6]) {
  const double p = (s[0] + s[1] + s[2]) / 3.0;
  const double j2 = 0.5 * ((s[0] - p) * (s[0] - p) + (s[1] - p) * (s[1] - p) + (s[2] - p) * (s[2] - p)) +
                    s[3] * s[3] + s[4] * s[4] + s[5] * s[5];
  return sqrt(3.0 * fmax(j2, 0.0));
}

// Elastic stress at the Gauss points: the stress and its von Mises value
// (PH_Elem_C3D8_EvalVonMises, PH_Elem_C3D8.f90:2768-2780), or, NODAL, the stress
// extrapolated to the element's nodes, fs[(8 e + a) 6 + i].  s6 non-null: the
// given Gauss-point stress instead (J2 state).
template <bool NODAL>
__global__ void __launch_bounds__(kOctBlock)
    k_oct_stress(int32_t E, const double* __restrict__ coords, const int32_t* __restrict__ conn,
                 const double* __restrict__ lame, const double* __restrict__ u, const double* __restrict__ s6,
                 double* __restrict__ sig, double* __restrict__ vm) {
  const OctElem el(0, E, coords, conn);
  const Octet oct(el.t);
  const int64_t g = el.e * 8 + el.t;
  double s[6];
  if (s6) {
#pragma unroll
    for (int i = 0; i < 6; ++i) s[i] = s6[g * 6 + i];
  } else {
    double v[3], inv[9], eps[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = u[3 * el.node + i];
    oct.jacobian(el.X, inv);
    oct.strain(inv, v, eps);
    iso_stress<double>(lame[2 * el.e], lame[2 * el.e + 1], eps, s);
  }
  if (NODAL) {
#pragma unroll
    for (int i = 0; i < 6; ++i) s[i] = oct.extrapolate(s[i]);
    if (el.real)
#pragma unroll
      for (int i = 0; i < 6; ++i) sig[(el.e * 8 + el.a) * 6 + i] = s[i];
    return;
  }
  if (!el.real) return;
  if (sig)
#pragma unroll
    for (int i = 0; i < 6; ++i) sig[g * 6 + i] = s[i];
  if (vm) vm[g] = von_mises(s);
}

// Nodal stress: the mean of the element values at the node (elements ascending) and its von Mises value.
__global__ void __launch_bounds__(256)
    k_nodal_stress(int32_t N, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nelem,
                   const double* __restrict__ fs, double* __restrict__ sig, double* __restrict__ vm) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int32_t k0 = nptr[i], k1 = nptr[i + 1];
  double s[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 2
  for (int32_t k = k0; k < k1; ++k) {
    const double* v = fs + 6 * (int64_t)nelem[k];
#pragma unroll
    for (int c = 0; c < 6; ++c) s[c] += v[c];
  }
  const double w = k1 > k0 ? 1.0 / (double)(k1 - k0) : 0.0;
#pragma unroll
  for (int c = 0; c < 6; ++c) s[c] *= w;
  if (sig)
#pragma unroll
    for (int c = 0; c < 6; ++c) sig[i * 6 + c] = s[c];
  if (vm) vm[i] = von_mises(s);
}

// Material-point batch (PH_Mat_Update_Arg rows): one thread per point.
__global__ void k_mat_batch(int32_t n, int32_t model, const double* __restrict__ props, int nprops, int per_point,
                            const double* __restrict__ stress_n, const double* __restrict__ dstrain,
                            const double* __restrict__ sdv_n, double* __restrict__ stress, double* __restrict__ sdv,
                            double* __restrict__ ddsdde, int32_t* __restrict__ yielded) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* pr = props + (per_point ? i * nprops : 0);
  double s[6], D[36], epl[6], epeq = 0.0;
  int y = 0;
  if (model == UFC_MAT_J2_ISO) {
    const double epeq_n = sdv_n ? sdv_n[i * 7] : 0.0;
    y = j2_update(pr, dstrain + i * 6, stress_n + i * 6, epeq_n, sdv_n ? sdv_n + i * 7 + 1 : nullptr, s, &epeq, epl,
                  D);
  } else {
    // PH_Mat_Elas_IP_Incr_Eval (PH_Mat_Elas_Eval.f90:41-84): sigma = sigma_n + D dstrain.
    const double big[4] = {pr[0], pr[1], 1e300, 0.0};
    j2_update(big, dstrain + i * 6, stress_n + i * 6, 0.0, nullptr, s, &epeq, epl, D);
    epeq = sdv_n ? sdv_n[i * 7] : 0.0;
    for (int k = 0; k < 6; ++k) epl[k] = sdv_n ? sdv_n[i * 7 + 1 + k] : 0.0;
  }
  for (int k = 0; k < 6; ++k) stress[i * 6 + k] = s[k];
  if (sdv) {
    sdv[i * 7] = epeq;
    for (int k = 0; k < 6; ++k) sdv[i * 7 + 1 + k] = epl[k];
  }
  if (ddsdde)
    for (int k = 0; k < 36; ++k) ddsdde[i * 36 + k] = D[k];
  if (yielded) yielded[i] = y;
}

// Adjoint sensitivity g_e = -sum_k lambda_k,e^T (Ke/E_e) u_k,e, evaluated as
// -sum_k sum_gp w detJ eps(lambda)^T (D/E_e) eps(u), by octets; no scatter (the
// output is per element).
__global__ void __launch_bounds__(kOctBlock)
    k_adjoint_sens(int32_t E, int64_t n, int nrhs, const double* __restrict__ coords,
                   const int32_t* __restrict__ conn, const double* __restrict__ props, int nprops,
                   const double* __restrict__ U, const double* __restrict__ L, double* __restrict__ g) {
  const OctElem el(0, E, coords, conn);
  const Octet oct(el.t);
  double inv[9], lam, mu;
  const double det = oct.jacobian(el.X, inv);
  lame<double>(1.0, props[el.e * nprops + 1], lam, mu);
  double acc = 0.0;
  for (int k = 0; k < nrhs; ++k) {
    double u[3], l[3], eu[6], ev[6], s[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      u[i] = U[k * n + 3 * el.node + i];
      l[i] = L[k * n + 3 * el.node + i];
    }
    oct.strain(inv, u, eu);
    oct.strain(inv, l, ev);
    iso_stress<double>(lam, mu, eu, s);
    acc += det * (ev[0] * s[0] + ev[1] * s[1] + ev[2] * s[2] + ev[3] * s[3] + ev[4] * s[4] + ev[5] * s[5]);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(kAllLanes, acc, o);
  if (el.real && el.t == 0) g[el.e] = -acc;
}

}  // namespace

int element_lame(Ctx* c) {
  UFC_TRY(dalloc(c, &c->lame, 2 * (int64_t)c->E));
  k_lame<<<grid_for(c->E, 256), 256, 0, c->stream>>>(c->E, c->props, c->nprops, c->lame);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

// The kernels' limit of dynamic shared memory is set to the most there is and not to
// what a launch takes: it belongs to the process, so another thread that assembles
// a mesh with shorter rows would lower it between this thread's setting and launch.
template <typename T, bool kTangent>
static int launch_assemble(Ctx* c, const RowOutputs<T>& to) {
  const int stride = (9 * c->max_row_blocks) | 1;  // odd: the rows of an entry lie in different banks
  if constexpr (!kTangent) {
    // while the slice's accumulators fit in shared memory
    const int bytes = kIsoXBytes + (int)sizeof(T) * kSlice * stride;
    if (bytes <= kAsmMaxSmem) {
      UFC_CUDA(c, cudaFuncSetAttribute(k_assemble_iso<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAsmMaxSmem));
      k_assemble_iso<T><<<(int)c->nslices, kIsoThreads, bytes, c->stream>>>(
          c->N, c->nptr, c->nelem, c->coords, c->conn, c->lame, c->slot, c->slice_ptr, c->sell_col, c->dpos, c->fixed,
          stride, to, c->dev_err);
      UFC_CUDA(c, cudaGetLastError());
      return UFC_STATUS_OK;
    }
  }
  const int bytes = (int)(sizeof(AsmWarp<T, kTangent>) * kAsmWarps + sizeof(T) * kAsmRows * stride);
  UFC_CUDA(c, cudaFuncSetAttribute(k_assemble_rows<T, kTangent>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   kAsmMaxSmem));
  k_assemble_rows<T, kTangent><<<(int)(2 * c->nslices), kAsmWarps * 32, bytes, c->stream>>>(
      c->N, c->nptr, c->nelem, c->coords, c->conn, c->lame, c->Dt, c->slot, c->slice_ptr, c->sell_col, c->dpos,
      c->fixed, stride, to, c->dev_err);
  if (kTangent)
    k_mirror_lower<T><<<(int)c->nslices, kMirrorWarps * 32, 0, c->stream>>>(c->N, c->brow, c->bcol, c->slice_ptr, to.val,
                                                                            to.val_r);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

int assemble(Ctx* c, int build, double* elapsed_ms) {
  if (!c->has_pattern) return fail(c, UFC_STATUS_INVALID, "ufc_elem_compute_ke: pattern not built");
  if (!c->has_material) return fail(c, UFC_STATUS_INVALID, "ufc_elem_compute_ke: material not set");
  const bool tangent = c->mat_model == UFC_MAT_J2_ISO;
  if (tangent && !c->has_trial)
    return fail(c, UFC_STATUS_INVALID,
                "ufc_elem_compute_ke: J2 tangent needs ufc_elem_compute_fint(update_state=1) first");
  mg_mark_stale(c);  // (cached CG graphs stay: they are keyed by the arrays and the SpMV form they read)
  cudaEvent_t e0, e1;
  UFC_CUDA(c, cudaEventCreate(&e0));
  UFC_CUDA(c, cudaEventCreate(&e1));
  UFC_CUDA(c, cudaEventRecord(e0, c->stream));
  UFC_CUDA(c, cudaMemsetAsync(c->dev_err, 0, sizeof(int32_t), c->stream));
  const int64_t nv = c->sell_blocks * 9;
  const bool diff = (build & UFC_BUILD_FP32_DIFF) != 0;
  const bool rounded = diff || (build & UFC_BUILD_FP32_ROUNDED) != 0;
  const bool sym = (build & UFC_BUILD_SYMMETRIC) != 0;
  const bool sym32 = sym && (build & (UFC_BUILD_FP32 | UFC_BUILD_FP32_ROUNDED | UFC_BUILD_FP32_DIFF)) != 0;
  if (rounded) build = (build | UFC_BUILD_FP64) & ~UFC_BUILD_FP32;
  if (sym) build |= UFC_BUILD_FP64;
  c->has_sval64 = c->has_sval32 = false;  // values change: symmetric copies are stale
  if (build & UFC_BUILD_FP32) c->val32_diff = false;
  if (build & UFC_BUILD_FP64) {
    if (!c->val64) UFC_TRY(dalloc(c, &c->val64, nv));
    if (!c->dinv64) UFC_TRY(dalloc(c, &c->dinv64, c->n));
  }
  if (rounded || (build & UFC_BUILD_FP32)) {
    if (!c->val32) UFC_TRY(dalloc(c, &c->val32, nv));
    if (!c->dinv32) UFC_TRY(dalloc(c, &c->dinv32, c->n));
  }
  if (build & UFC_BUILD_FP64) {
    RowOutputs<double> to;
    to.val = c->val64;
    to.dinv = c->dinv64;
    if (rounded) {  // the FP64 values rounded to nearest (Dirichlet rows included)
      to.val_r = c->val32;
      to.dinv_r = c->dinv32;
    }
    if (sym) {
      UFC_TRY(alloc_symmetric(c, sym32));
      to.uptr = c->uptr;
      to.sval = c->sval64;
      if (sym32) to.sval_r = c->sval32;
    }
    if (tangent)
      UFC_TRY((launch_assemble<double, true>(c, to)));
    else
      UFC_TRY((launch_assemble<double, false>(c, to)));
    c->has_sval64 = sym;
    c->has_sval32 = sym32;
    c->has_val64 = true;
  }
  if (build & UFC_BUILD_FP32) {
    RowOutputs<float> to;
    to.val = c->val32;
    to.dinv = c->dinv32;
    if (tangent)
      UFC_TRY((launch_assemble<float, true>(c, to)));
    else
      UFC_TRY((launch_assemble<float, false>(c, to)));
    c->has_val32 = true;
  }
  if (rounded) {
    if (diff)
      k_diag_rowsum<<<grid_for(c->N, 128), 128, 0, c->stream>>>(c->N, c->slice_ptr, c->dpos, c->val64, c->val32);
    UFC_CUDA(c, cudaGetLastError());
    c->has_val32 = true;
    c->val32_diff = diff;
  }
  UFC_CUDA(c, cudaEventRecord(e1, c->stream));
  UFC_CUDA(c, cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (elapsed_ms) *elapsed_ms = ms;
  return check_dev_err(c, "ufc_elem_compute_ke");
}

namespace {

int oct_grid(const Ctx* c) { return grid_for(8 * (int64_t)c->E, kOctBlock); }

// y = node sums of the element forces that `forces(e0, e1)` leaves in c->fe; x:
// identity rows on fixed DOFs
template <class Forces>
int sum_forces(Ctx* c, const double* x, double* y, Forces forces) {
  if (!c->fe) UFC_TRY(dalloc(c, &c->fe, 24 * (int64_t)std::min(c->E, kFeElems)));
  for (int32_t e0 = 0; e0 < c->E; e0 += kFeElems) {
    const int32_t e1 = std::min(c->E - e0, kFeElems) + e0;
    forces(e0, e1);
    UFC_CUDA(c, cudaGetLastError());
    const int grid = grid_for(c->n, 256);
    if (c->E <= kFeElems)
      k_node_sum<false><<<grid, 256, 0, c->stream>>>(c->n, e0, e1, c->nptr, c->nelem, c->fe, c->fixed, x, y);
    else
      k_node_sum<true><<<grid, 256, 0, c->stream>>>(c->n, e0, e1, c->nptr, c->nelem, c->fe, c->fixed, x, y);
    UFC_CUDA(c, cudaGetLastError());
    c->launches += 2;
  }
  return UFC_STATUS_OK;
}

int part_grid(int32_t e0, int32_t e1) { return grid_for(8 * (int64_t)(e1 - e0), kOctBlock); }

int apply_iso(Ctx* c, const double* x, const uint8_t* fixed, const double* identity, double* y) {
  return sum_forces(c, identity, y, [&](int32_t e0, int32_t e1) {
    k_oct_force<kIso><<<part_grid(e0, e1), kOctBlock, 0, c->stream>>>(e0, e1, c->coords, c->conn, c->lame, nullptr, x,
                                                                      fixed, c->fe, c->dev_err);
  });
}

}  // namespace

// y = K x matrix-free, FP64, without elimination (the linear-elastic internal force).
int apply_fp64(Ctx* c, const double* x, double* y) { return apply_iso(c, x, nullptr, nullptr, y); }

int apply_fp64_eliminated(Ctx* c, const double* x, double* y) { return apply_iso(c, x, c->fixed, x, y); }

// Newton residual R = f_ext - F_int on free DOFs (0 on fixed) and the norms
// ||R||^2, ||F_int||^2, ||F_ext||^2 into the scalars (RT_Asm_ComputeResidual,
// RT_Asm_Solv.f90:1311-1426; RT_NR_CheckConvergence, RT_Step_NR_Core.f90:231-317).
__global__ void __launch_bounds__(256)
    k_nr_resid(int64_t n, const double* __restrict__ fext, const double* __restrict__ fint,
               const uint8_t* __restrict__ fixed, double* __restrict__ R, CgScalars* __restrict__ scal,
               double* __restrict__ partials) {
  double v[3] = {0.0, 0.0, 0.0}, tot[3];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double fe = fext ? fext[i] : 0.0, fi = fint[i];
    const double r = fixed[i] ? 0.0 : fe - fi;
    R[i] = r;
    v[0] += r * r;
    v[1] += fi * fi;
    v[2] += fe * fe;
  }
  if (grid_sum<3>(v, partials, &scal->ticket[4], tot)) {
    scal->nr_rr = tot[0];
    scal->nr_ff = tot[1];
    scal->nr_ee = tot[2];
  }
}

int nr_norms(Ctx* c, const double* fext, const double* fint, double* R) {
  const int g = (int)std::min<int64_t>(grid_for(c->n, 256), 148 * 8);
  k_nr_resid<<<g, 256, 0, c->stream>>>(c->n, fext, fint, c->fixed, R, c->scal, c->partials);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

int compute_fint(Ctx* c, const double* u, double* fint, bool update_state) {
  (void)update_state;
  if (!c->has_material) return fail(c, UFC_STATUS_INVALID, "ufc_elem_compute_fint: material not set");
  if (c->ncol == 0) return fail(c, UFC_STATUS_INVALID, "ufc_elem_compute_fint: pattern not built");
  if (c->mat_model != UFC_MAT_J2_ISO) return apply_fp64(c, u, fint);
  UFC_TRY(sum_forces(c, nullptr, fint, [&](int32_t e0, int32_t e1) {
    k_oct_j2<<<part_grid(e0, e1), kOctBlock, 0, c->stream>>>(e0, e1, c->coords, c->conn, c->props, c->nprops, u,
                                                             c->u_n, c->sig_n, c->epeq_n, c->epl_n, c->sig_t, c->epeq_t,
                                                             c->epl_t, c->Dt, c->fe, c->dev_err);
  }));
  c->has_trial = true;
  return UFC_STATUS_OK;
}

int apply_tangent(Ctx* c, const double* x, double* y) {
  if (!c->has_trial) return fail(c, UFC_STATUS_INVALID, "tangent operator needs a return map first");
  return sum_forces(c, nullptr, y, [&](int32_t e0, int32_t e1) {
    k_oct_force<kTangent><<<part_grid(e0, e1), kOctBlock, 0, c->stream>>>(e0, e1, c->coords, c->conn, nullptr, c->Dt, x,
                                                                          nullptr, c->fe, c->dev_err);
  });
}

int mat_update_batch(Ctx* c, const ufc_mat_update_arg* a, const double* props, const double* stress_n,
                     const double* dstrain, const double* sdv_n, double* stress, double* sdv, double* ddsdde,
                     int32_t* yielded) {
  if (a->n_points <= 0) return UFC_STATUS_OK;
  k_mat_batch<<<grid_for(a->n_points, 128), 128, 0, c->stream>>>(a->n_points, a->mat_model_id, props, a->nprops,
                                                                 a->props_per_point, stress_n, dstrain, sdv_n, stress,
                                                                 sdv, ddsdde, yielded);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

int stress_eval(Ctx* c, const double* u, double* sig, double* vm) {
  const double* s6 = c->mat_model == UFC_MAT_J2_ISO ? c->sig_n : nullptr;
  k_oct_stress<false><<<oct_grid(c), kOctBlock, 0, c->stream>>>(c->E, c->coords, c->conn, c->lame, u, s6, sig, vm);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

// Nodal stress and its von Mises value; fs: [E][8][6] scratch.
int stress_at_nodes(Ctx* c, const double* u, double* fs, double* sig, double* vm) {
  const double* s6 = c->mat_model == UFC_MAT_J2_ISO ? c->sig_n : nullptr;
  k_oct_stress<true><<<oct_grid(c), kOctBlock, 0, c->stream>>>(c->E, c->coords, c->conn, c->lame, u, s6, fs, nullptr);
  UFC_CUDA(c, cudaGetLastError());
  k_nodal_stress<<<grid_for(c->N, 256), 256, 0, c->stream>>>(c->N, c->nptr, c->nelem, fs, sig, vm);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

int adjoint_sens(Ctx* c, int nrhs, const double* U, const double* L, double* g) {
  k_adjoint_sens<<<oct_grid(c), kOctBlock, 0, c->stream>>>(c->E, c->n, nrhs, c->coords, c->conn, c->props, c->nprops,
                                                           U, L, g);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

}  // namespace ufc
