// Geometric multigrid preconditioner for structured C3D8 boxes, in the place of
// the reference's AMG (NM_AMG_Setup, NM_AMG_V_Cycle, NM_AMG_Smooth,
// NM_AMG_Galerkin: ufc_core/L2_NM/Solver/LinSolv/NM_Solv_LinPrecAMG.f90:120-675),
// and the PCG that uses it.
//
// Hierarchy.  Level 0 is the context's own assembled FP64 matrix.  Level l+1
// is the box with half the elements in each direction; its nodes are the
// even-indexed nodes of level l.  Prolongation P is trilinear: a fine node
// takes weight 1 from the coarse node it coincides with, 1/2 from each of the
// two coarse nodes it lies between, and so on per direction.  The coarse
// operator is the Galerkin product P^T A P, formed element by element: the
// matrix of coarse element e is sum over its 8 child elements f of
// W_f^T K_f W_f, W_f the 24x24 restriction of P to the nodes of f, which for
// nested boxes adds up to exactly P^T A P.  Dirichlet DOFs stay eliminated on
// every level: P has zero rows at fixed fine DOFs and zero columns at fixed
// coarse DOFs (a coarse DOF is fixed when the fine DOF it coincides with is),
// and fixed coarse rows get a unit diagonal.
//
// Cycle.  V-cycle with a Chebyshev polynomial smoother of D^-1 A (same degree
// before and after the coarse correction, so the preconditioner is symmetric),
// on [lambda_max/ratio, 1.1 lambda_max] with lambda_max from a power iteration
// at set-up; the coarsest level is solved with its dense inverse (<= kDenseMax DOF)
// or a high-degree Chebyshev polynomial.  Restriction and prolongation are
// structured gathers, one thread per coarse or fine node, so they need no
// atomics and are deterministic; the coarse matrices are assembled by block rows
// like the fine one.
//
// Precision: the cycle runs in FP64, or (precision = UFC_PRECISION_FP32_REFINE)
// in FP32 on values rounded from the FP64 operators, half the bytes; the PCG
// around it stays FP64 (matrix, vectors, residual), so the preconditioner's
// rounding changes only the iteration count, never the answer.
//
// The PCG is NM_Solver_PCG's recurrence with z = M r from the V-cycle; all of
// an iteration's kernels (SpMV, updates, the cycle on every level) are
// captured once into a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <vector>

#include "c3d8_device.cuh"
#include "reduce.cuh"
#include "rows.cuh"
#include "spmv.cuh"
#include "ufc_internal.cuh"

namespace ufc {

template <typename T>
struct MgVecs {
  T *x = nullptr, *b = nullptr, *r = nullptr, *d = nullptr, *e = nullptr, *w = nullptr;
};

struct MgLevel {
  Ctx* c = nullptr;          // the level's context (level 0: the owner)
  ufc_ctx* own = nullptr;    // levels >= 1: a context holding the coarse box
  int32_t nx = 0, ny = 0, nz = 0;
  double* ke = nullptr;      // levels >= 1: Galerkin element matrices [E][9][64], node pairs by sign bits
  // vectors of the cycle, in its precision (FP64, level 0: x and b are the PCG's z and r)
  MgVecs<double> v64;
  MgVecs<float> v32;
  // FP32 cycle: the level's values and diagonal rounded to FP32, and the
  // symmetric storage rounded where the level holds it in FP64 only
  float *val32 = nullptr, *sval32 = nullptr, *dinv32 = nullptr;
  double* coef = nullptr;    // smoother: lambda_max, 1/theta, then c1, c2 of every further step
  double* inv = nullptr;     // coarsest level: dense inverse [ld][ld], ld = n rounded up to 32
  float* inv32 = nullptr;
  double* gj = nullptr;      // its elimination's column panel and pivot block
  double *pv = nullptr, *pw = nullptr;  // power-iteration vectors (lambda_max), kept across refreshes
};

struct Mg {
  std::vector<MgLevel> lv;
  int degree = 2;
  double ratio = 15.0;
  bool stale = false;
  bool fp32 = false;         // the cycle runs in FP32 (values, vectors); the PCG around it in FP64
  int cheb_coarse = 0;       // degree of the coarsest Chebyshev solve (0: dense inverse)
  double lmax_scale = 1.0;   // of the coefficients in place: above 1 inside a solve whose cycle was indefinite
  double* dnorm = nullptr;   // ||v||^2 of the power iteration, on the device
  int32_t* gj_flag = nullptr;  // set when the coarsest elimination met a pivot that is not positive
  // the PCG iteration as a graph, and what it baked in
  cudaGraphExec_t graph = nullptr;
  int batch = 0;
  int64_t graph_launches = 0;
  const void* key[9] = {};
};

namespace {

constexpr int kBlk = 256;
// largest coarsest level inverted densely (block Gauss-Jordan on the device at
// every set-up and refresh); larger ones get a degree-24 Chebyshev solve
constexpr int64_t kDenseMax = 1200;

int grid_n(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + kBlk - 1) / kBlk, 148 * 16)); }

__host__ __device__ inline int64_t box_node(int64_t i, int64_t j, int64_t k, int32_t nx, int32_t ny) {
  return i + (int64_t)(nx + 1) * (j + (int64_t)(ny + 1) * k);
}

// Galerkin element matrices of one coarse level: one CTA per coarse element, one
// warp per child.  A lane holds the blocks (p, q) and (p + 4, q) of the child's
// 8x8 block grid, p = lane / 8, q = lane % 8 in sign-bit numbering; FROM_KE
// reads them from the finer level's element matrices, otherwise they are formed
// from the fine element (linear-elastic D, or the J2 tangent per Gauss point)
// as in the stiffness assembly.  The restriction W of P to the child is a
// tensor product of 2x2 matrices, so W^T K W is three exchanges with the lane
// whose q differs in one bit and three for p (two by shuffles, the last between
// the lane's own two blocks); rows and columns of fixed DOFs are zeroed before
// (fine) and after (coarse).  The 8 children are added in order.
// 64x32x32, level 1 from the elements: 1298 us with one 64-thread CTA walking
// through the children and the dense W, now 153 us.
constexpr int kGalThreads = 256;

template <bool TANGENT>
struct GalWarp {
  double X[24];
  double g[8][8][3];                       // [gp][node][dir], scaled by sqrt(det J)
  double M[TANGENT ? 8 : 1][8][18];        // [node][gp]: D B_a (J2)
};

template <bool FROM_KE, bool TANGENT>
__global__ void __launch_bounds__(kGalThreads)
    k_mg_galerkin(int32_t nxc, int32_t nyc, int32_t nzc, const double* __restrict__ coords,
                  const int32_t* __restrict__ conn_f, const double* __restrict__ lame,
                  const double* __restrict__ Dt, const double* __restrict__ ke_f, const uint8_t* __restrict__ fixed_f,
                  const int32_t* __restrict__ conn_c, const uint8_t* __restrict__ fixed_c, double* __restrict__ ke_c,
                  int32_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char gal_smem[];
  double* out = reinterpret_cast<double*>(gal_smem);  // [child][9][64], over the warps' areas
  const int ch = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ec = blockIdx.x;
  const int nxf = 2 * nxc, nyf = 2 * nyc;
  const int64_t I = ec % nxc, J = (ec / nxc) % nyc, K = ec / ((int64_t)nxc * nyc);
  const int cb[3] = {ch & 1, (ch >> 1) & 1, ch >> 2};
  const int64_t ef = (2 * I + cb[0]) + (int64_t)nxf * ((2 * J + cb[1]) + (int64_t)nyf * (2 * K + cb[2]));
  const int p = lane >> 3, q = lane & 7;
  double B[2][9];
  if constexpr (FROM_KE) {
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      B[0][c] = ke_f[ef * 576 + 64 * c + lane];
      B[1][c] = ke_f[ef * 576 + 64 * c + 32 + lane];
    }
  } else {
    GalWarp<TANGENT>& sm = reinterpret_cast<GalWarp<TANGENT>*>(gal_smem)[ch];
    if (lane < 24) sm.X[lane] = coords[(int64_t)conn_f[ef * 8 + lane / 3] * 3 + lane % 3];
    __syncwarp();
    {
      // Gauss point lane / 4, gradients of the two nodes 2 (lane % 4) and the next
      const int gp = lane >> 2;
      double J9[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) J9[k] = 0.0;
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        double d0, d1, d2;
        dN_dxi<double>(gp, a, d0, d1, d2);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          J9[i] += d0 * sm.X[3 * a + i];
          J9[3 + i] += d1 * sm.X[3 * a + i];
          J9[6 + i] += d2 * sm.X[3 * a + i];
        }
      }
      const double c0 = J9[4] * J9[8] - J9[5] * J9[7], c3 = J9[5] * J9[6] - J9[3] * J9[8],
                   c6 = J9[3] * J9[7] - J9[4] * J9[6];
      const double det = J9[0] * c0 + J9[1] * c3 + J9[2] * c6;
      if (!(det > 0.0)) atomicOr(err, (int)kDevBadJacobian);
      const double sc = rsqrt(det);
      const double inv[9] = {c0 * sc, (J9[2] * J9[7] - J9[1] * J9[8]) * sc, (J9[1] * J9[5] - J9[2] * J9[4]) * sc,
                             c3 * sc, (J9[0] * J9[8] - J9[2] * J9[6]) * sc, (J9[2] * J9[3] - J9[0] * J9[5]) * sc,
                             c6 * sc, (J9[1] * J9[6] - J9[0] * J9[7]) * sc, (J9[0] * J9[4] - J9[1] * J9[3]) * sc};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = 2 * (lane & 3) + h;
        double g3[3];
        grad_x<double>(inv, gp, bits_node(t), g3);
#pragma unroll
        for (int i = 0; i < 3; ++i) sm.g[gp][t][i] = g3[i];
      }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 9; ++c) B[h][c] = 0.0;
    if constexpr (TANGENT) {
      // D B_a for node p (+ 4) at Gauss point q of this lane
      constexpr int kIdx[3][3] = {{0, 3, 5}, {1, 3, 4}, {2, 4, 5}};
      constexpr int kCmp[3][3] = {{0, 1, 2}, {1, 0, 2}, {2, 1, 0}};
      double D[21];
#pragma unroll
      for (int k = 0; k < 21; ++k) D[k] = Dt[(ef * 21 + k) * 8 + q];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double* ga = sm.g[q][p + 4 * h];
        double* M = sm.M[p + 4 * h][q];
#pragma unroll
        for (int v = 0; v < 6; ++v)
#pragma unroll
          for (int i = 0; i < 3; ++i)
            M[v * 3 + i] = D[tri6(v, kIdx[i][0])] * ga[kCmp[i][0]] + D[tri6(v, kIdx[i][1])] * ga[kCmp[i][1]] +
                           D[tri6(v, kIdx[i][2])] * ga[kCmp[i][2]];
      }
      __syncwarp();
#pragma unroll 1
      for (int gp = 0; gp < 8; ++gp) {
        const double* gb = sm.g[gp][q];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double* M = sm.M[p + 4 * h][gp];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
              B[h][3 * i + j] += M[kIdx[j][0] * 3 + i] * gb[kCmp[j][0]] + M[kIdx[j][1] * 3 + i] * gb[kCmp[j][1]] +
                                 M[kIdx[j][2] * 3 + i] * gb[kCmp[j][2]];
        }
      }
    } else {
#pragma unroll 2
      for (int gp = 0; gp < 8; ++gp) {
        const double* gb = sm.g[gp][q];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double* ga = sm.g[gp][p + 4 * h];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) B[h][3 * i + j] += ga[i] * gb[j];
        }
      }
      const double lam = lame[2 * ef], mu = lame[2 * ef + 1];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double tr = mu * (B[h][0] + B[h][4] + B[h][8]);
        double k9[9];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            k9[3 * i + j] = lam * B[h][3 * i + j] + mu * B[h][3 * j + i];
            if (i == j) k9[3 * i + j] += tr;
          }
#pragma unroll
        for (int c = 0; c < 9; ++c) B[h][c] = k9[c];
      }
    }
  }
  // zero rows and columns of P at fixed fine DOFs
  {
    const int64_t nq = conn_f[ef * 8 + bits_node(q)];
    bool fq[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) fq[j] = fixed_f[3 * nq + j] != 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t np = conn_f[ef * 8 + bits_node(p + 4 * h)];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const bool fp = fixed_f[3 * np + i] != 0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (fp || fq[j]) B[h][3 * i + j] = 0.0;
      }
    }
  }
  // W^T K W, one direction at a time: a lane's block with node bit b takes the
  // weight of its own block and of the one with the other bit (a coarse node on
  // the child's side of the box, b == cb: 1 and 1/2; across it: 1/2 and 0)
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int dir = s < 3 ? s : s - 3, bit = (lane >> s) & 1;
    const double wo = bit == cb[dir] ? 1.0 : 0.5, wx = bit == cb[dir] ? 0.5 : 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        const double other = __shfl_xor_sync(0xffffffffu, B[h][c], 1 << s);
        B[h][c] = wo * B[h][c] + wx * other;
      }
  }
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    const double lo = B[0][c], hi = B[1][c];
    B[0][c] = cb[2] == 0 ? lo + 0.5 * hi : 0.5 * lo;
    B[1][c] = cb[2] == 0 ? 0.5 * hi : hi + 0.5 * lo;
  }
  __syncthreads();  // the warps' areas are consumed
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    out[ch * 576 + 64 * c + lane] = B[0][c];
    out[ch * 576 + 64 * c + 32 + lane] = B[1][c];
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 576; k += kGalThreads) {
    const int c = k >> 6, P = (k >> 3) & 7, Q = k & 7;
    const int64_t nP = conn_c[ec * 8 + bits_node(P)], nQ = conn_c[ec * 8 + bits_node(Q)];
    double v = 0.0;
#pragma unroll
    for (int h = 0; h < 8; ++h) v += out[h * 576 + k];
    ke_c[ec * 576 + k] = (fixed_c[3 * nP + c / 3] || fixed_c[3 * nQ + c % 3]) ? 0.0 : v;
  }
}

// Block rows of a coarse level from its element matrices, 16 rows per CTA and 8
// lanes per row, each entry summed in ascending element order and written once
// (see k_assemble_rows).
constexpr int kMgRows = 16;
constexpr int kMgRowThreads = 128;

__global__ void __launch_bounds__(kMgRowThreads)
    k_mg_rows(int32_t N, const int32_t* __restrict__ nptr, const int32_t* __restrict__ nelem,
              const double* __restrict__ ke, const int32_t* __restrict__ slot, const int64_t* __restrict__ sptr,
              const int32_t* __restrict__ scol, const int32_t* __restrict__ dpos, const uint8_t* __restrict__ fixed,
              int stride, const RowOutputs<double> to) {
  extern __shared__ double mg_acc[];  // [row][stride]
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, t = lane & 7;
  const int64_t s = blockIdx.x >> 1;
  const int half = (blockIdx.x & 1) * kMgRows;
  const int64_t base = sptr[s];
  const int len = (int)((sptr[s + 1] - base) >> 5);
  RowWriter<double, kMgRows, kMgRowThreads> out;
  out.init(N, s, half, base, len, scol, dpos, fixed);
  for (int k = threadIdx.x; k < kMgRows * stride; k += kMgRowThreads) mg_acc[k] = 0.0;
  __syncthreads();
  const int r = 4 * w + (lane >> 3);
  const int64_t row = s * kSlice + half + r;
  const int32_t kb = row < N ? nptr[row] : 0, ke_end = row < N ? nptr[row + 1] : 0;
  const int kmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)(ke_end - kb));
#pragma unroll 2
  for (int k = 0; k < kmax; ++k) {
    if (kb + k < ke_end) {
      const int32_t el = nelem[kb + k];
      const int64_t e = el >> 3;
      const int a = el & 7;
      const int j = (int)((slot[e * 64 + a * 8 + bits_node(t)] - base) >> 5);
      const double* src = ke + e * 576 + bits_node(a) * 8 + t;
      double* d = mg_acc + r * stride + 9 * j;
#pragma unroll
      for (int c = 0; c < 9; ++c) d[c] += src[64 * c];
    }
    __syncwarp();  // the lanes of a row meet again at the same entries
  }
  __syncthreads();
  out.write(len, scol, fixed, mg_acc, stride, to);
}

// b = P^T r_f and d = D^-1 b / theta (the coarse smoother's first step): one
// thread per coarse node gathers the fine nodes within one fine spacing of it,
// weight prod_d (1 or 1/2).  dinv null: no smoother on the coarse level.
template <typename T>
__global__ void k_mg_restrict(int32_t nxc, int32_t nyc, int32_t nzc, const T* __restrict__ rf,
                              const uint8_t* __restrict__ fixed_f, const uint8_t* __restrict__ fixed_c,
                              const T* __restrict__ dinv, const double* __restrict__ coef, T* __restrict__ bc,
                              T* __restrict__ dc, const CgScalars* __restrict__ scal) {
  const int64_t nc = (int64_t)(nxc + 1) * (nyc + 1) * (nzc + 1);
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nxf = 2 * nxc, nyf = 2 * nyc, nzf = 2 * nzc;
  const int32_t I = (int32_t)(v % (nxc + 1)), J = (int32_t)((v / (nxc + 1)) % (nyc + 1)),
                K = (int32_t)(v / ((int64_t)(nxc + 1) * (nyc + 1)));
  // which of the 27 x 3 entries count (Dirichlet flags, box edges): read before
  // the wait for the kernel in front
  uint32_t use[3] = {0, 0, 0};
  if (v < nc) {
#pragma unroll
    for (int q = 0; q < 27; ++q) {
      const int k = 2 * K + q / 9 - 1, j = 2 * J + (q / 3) % 3 - 1, i = 2 * I + q % 3 - 1;
      if (k < 0 || k > nzf || j < 0 || j > nyf || i < 0 || i > nxf) continue;
      const int64_t f = box_node(i, j, k, nxf, nyf);
#pragma unroll
      for (int d = 0; d < 3; ++d) use[d] |= fixed_f[3 * f + d] ? 0u : 1u << q;
    }
  }
  T di[3] = {T(0), T(0), T(0)};
  bool fc[3] = {true, true, true};
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (v < nc) {
      fc[d] = fixed_c[3 * v + d] != 0;
      if (dinv) di[d] = dinv[3 * v + d];
    }
  pdl_enter();
  if (v >= nc || (scal && scal->stop)) return;
  T s[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int q = 0; q < 27; ++q) {
    const int k = q / 9 - 1, j = (q / 3) % 3 - 1, i = q % 3 - 1;
    const T w = T((i ? 0.5 : 1.0) * (j ? 0.5 : 1.0) * (k ? 0.5 : 1.0));
    const int64_t f = box_node(2 * I + i, 2 * J + j, 2 * K + k, nxf, nyf);
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] += (use[d] >> q) & 1u ? w * rf[3 * f + d] : T(0);
  }
  const T it = dinv ? (T)coef[1] : T(0);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const T b = fc[d] ? T(0) : s[d];
    bc[3 * v + d] = b;
    if (dinv) dc[3 * v + d] = di[d] * b * it;
  }
}

// v = P x_c: one thread per fine node gathers its 1, 2, 4 or 8 coarse parents.
template <typename T>
__global__ void k_mg_prolong(int32_t nxc, int32_t nyc, int32_t nzc, const T* __restrict__ xc,
                             const uint8_t* __restrict__ fixed_f, const uint8_t* __restrict__ fixed_c,
                             T* __restrict__ vf, const CgScalars* __restrict__ scal) {
  const int nxf = 2 * nxc, nyf = 2 * nyc, nzf = 2 * nzc;
  const int64_t nf = (int64_t)(nxf + 1) * (nyf + 1) * (nzf + 1);
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t i = (int32_t)(v % (nxf + 1)), j = (int32_t)((v / (nxf + 1)) % (nyf + 1)),
                k = (int32_t)(v / ((int64_t)(nxf + 1) * (nyf + 1)));
  const T w = T(((i & 1) ? 0.5 : 1.0) * ((j & 1) ? 0.5 : 1.0) * ((k & 1) ? 0.5 : 1.0));
  uint32_t use[3] = {0, 0, 0};  // as in k_mg_restrict
  bool ff[3] = {true, true, true};
  if (v < nf) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int a = q & 1, b = (q >> 1) & 1, c = q >> 2;
      if ((c && !(k & 1)) || (b && !(j & 1)) || (a && !(i & 1))) continue;
      const int64_t cn = box_node((i >> 1) + a, (j >> 1) + b, (k >> 1) + c, nxc, nyc);
#pragma unroll
      for (int d = 0; d < 3; ++d) use[d] |= fixed_c[3 * cn + d] ? 0u : 1u << q;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) ff[d] = fixed_f[3 * v + d] != 0;
  }
  pdl_enter();
  if (v >= nf || (scal && scal->stop)) return;
  T s[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int64_t cn = box_node((i >> 1) + (q & 1), (j >> 1) + ((q >> 1) & 1), (k >> 1) + (q >> 2), nxc, nyc);
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] += (use[d] >> q) & 1u ? w * xc[3 * cn + d] : T(0);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) vf[3 * v + d] = ff[d] ? T(0) : s[d];
}

// The Chebyshev smoother (three-term recurrence of Saad, Iterative Methods for
// Sparse Linear Systems, Alg. 12.1, with the Jacobi preconditioner) as the
// epilogue of the products it is made of: with w = (A v)_row for the gathered
// vector v,
//   kStep   v = d: r = rin - w, d' = c1 d + c2 D^-1 r, x = xin + d'
//   kResid  v = d: r = rin - w (the residual after the last step)
//   kStart  v = the prolonged coarse correction: r = rin - w,
//           d' = D^-1 r / theta, x = xin + v + d'
//   kPower  d' = D^-1 w and ||d'||^2 (the power iteration of set-up)
// One launch then does a product and its vector updates, and the vectors of a
// step are read once.  d' goes to another buffer than d, which other rows still
// gather.  The last step of a cycle writes z in FP64 and the row's part of r.z.
enum MgMode { kStep, kResid, kStart, kPower };

template <typename T>
struct MgEpi {
  static constexpr bool kDot = true, kPdl = true;
  int mode = kStep, step = 0;
  bool dot = false;
  const CgScalars* scal = nullptr;
  const double* coef = nullptr;
  const T *rin = nullptr, *dinv = nullptr, *xin = nullptr;
  T *rout = nullptr, *dout = nullptr, *xout = nullptr;
  double* z = nullptr;
  const double* r64 = nullptr;
  __device__ __forceinline__ bool halt() const { return scal && scal->stop; }
  __device__ __forceinline__ bool want_dot() const { return dot; }
  __device__ __forceinline__ double operator()(int64_t row, T a0, T a1, T a2, const T* __restrict__ v) const {
    const T w[3] = {a0, a1, a2};
    double part = 0.0;
    const T c1 = mode == kStep ? (T)coef[2 * step] : mode == kStart ? (T)coef[1] : T(0);
    const T c2 = mode == kStep ? (T)coef[2 * step + 1] : T(0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = 3 * row + c;
      if (mode == kPower) {
        const T dn = dinv[i] * w[c];
        dout[i] = dn;
        part += (double)dn * (double)dn;
        continue;
      }
      const T ri = rin[i] - w[c];
      if (rout) rout[i] = ri;
      if (mode == kResid) continue;
      const T vi = v[i];
      const T dn = mode == kStep ? c1 * vi + c2 * dinv[i] * ri : dinv[i] * ri * c1;
      const T xn = (mode == kStep ? xin[i] : xin[i] + vi) + dn;
      if (dout) dout[i] = dn;
      if (xout) xout[i] = xn;
      if (z) z[i] = (double)xn;
      if (dot) part += r64[i] * (double)xn;
    }
    return part;
  }
};

// x = Inv b (dense, coarsest level, leading dimension ld), one warp per row.
template <typename T>
__global__ void k_mg_dense(int64_t n, int64_t ld, const T* __restrict__ inv, const T* __restrict__ b,
                           T* __restrict__ x, const CgScalars* __restrict__ scal) {
  pdl_enter();
  if (scal && scal->stop) return;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  T s = T(0);
#pragma unroll 4
  for (int64_t j = lane; j < n; j += 32) s += inv[row * ld + j] * b[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) x[row] = s;
}

// The first smoothing step of the finest level, from the PCG's residual:
// b = r in the cycle's precision (when it is not r itself), d = D^-1 b / theta.
template <typename T>
__device__ __forceinline__ void mg_begin(int64_t i, double r, T* __restrict__ b, T* __restrict__ d,
                                         const T* __restrict__ dinv, T it) {
  const T bi = (T)r;
  if (sizeof(T) == 4) b[i] = bi;
  d[i] = dinv[i] * bi * it;
}

template <typename T>
__global__ void __launch_bounds__(kBlk)
    k_mg_begin(int64_t n, const double* __restrict__ r, T* __restrict__ b, T* __restrict__ d,
               const T* __restrict__ dinv, const double* __restrict__ coef) {
  const T it = (T)coef[1];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    mg_begin<T>(i, r[i], b, d, dinv, it);
}

// Sum of the power iteration's partials.
__global__ void __launch_bounds__(kBlk) k_mg_sum(const double* __restrict__ partials, int nb, double* __restrict__ out) {
  double tot[1];
  sum_partials<1>(partials, nb, tot);
  if (threadIdx.x == 0) *out = tot[0];
}

// The smoother's interval [1.1 lambda_max / ratio, 1.1 lambda_max] and the
// coefficients of m steps.  nb > 0: lambda_max = ||v_k|| / ||v_{k-1}|| of the
// power iteration (partials of ||v_k||^2 and *prev = ||v_{k-1}||^2), kept in
// coef[0]; nb = 0: from the kept one, times scale.
__global__ void __launch_bounds__(kBlk)
    k_mg_coef(const double* __restrict__ partials, int nb, const double* __restrict__ prev, double scale, double ratio,
              int m, double* __restrict__ coef) {
  double tot[1] = {0.0};
  if (nb > 0) sum_partials<1>(partials, nb, tot);
  if (threadIdx.x != 0) return;
  const double lambda = nb > 0 ? (*prev > 0.0 ? sqrt(tot[0] / *prev) : 0.0) : coef[0] * scale;
  if (nb > 0) coef[0] = lambda;
  const double lmax = 1.1 * lambda, lmin = lmax / ratio;
  const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
  const double sigma = theta / delta;
  coef[1] = 1.0 / theta;
  double rho = 1.0 / sigma;
  for (int k = 1; k < m; ++k) {
    const double rho_new = 1.0 / (2.0 * sigma - rho);
    coef[2 * k] = rho_new * rho;
    coef[2 * k + 1] = 2.0 * rho_new / delta;
    rho = rho_new;
  }
}

__global__ void k_mg_start_vector(int64_t n, const uint8_t* __restrict__ fixed, double* __restrict__ v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v[i] = fixed[i] ? 0.0 : 1.0 + 0.5 * (double)((i * 7919) % 13) / 13.0;
}

// ---- the PCG around the V-cycle: the Jacobi kernels' recurrence with z = M r

// alpha = r.z / p.q (from the product's partials), x += alpha p, r -= alpha q,
// the next cycle's first smoothing step, ||r||^2 and the stop tests.
template <typename T>
__global__ void __launch_bounds__(kBlk)
    k_mgcg_update(int64_t n, const double* __restrict__ p, const double* __restrict__ q, double* __restrict__ r,
                  double* __restrict__ x, T* __restrict__ b, T* __restrict__ d, const T* __restrict__ dinv,
                  const double* __restrict__ coef, CgScalars* __restrict__ scal,
                  const double* __restrict__ pq_partials, int nb, double* __restrict__ partials) {
  pdl_enter();
  if (any_in_block(scal->stop != 0)) return;  // (block 0 may set it)
  double pq[1];
  sum_partials<1>(pq_partials, nb, pq);
  if (!(fabs(pq[0]) > 1e-300) || !isfinite(pq[0])) {
    if (blockIdx.x == 0 && threadIdx.x == 0) scal->stop = 3;
    return;
  }
  const double a = scal->rz / pq[0];
  const T it0 = (T)coef[1];
  double v[1] = {0.0};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] += a * p[i];
    const double ri = r[i] - a * q[i];
    r[i] = ri;
    mg_begin<T>(i, ri, b, d, dinv, it0);
    v[0] += ri * ri;
  }
  double tot[1];
  if (grid_sum<1>(v, partials, &scal->ticket[1], tot)) {
    scal->pq = pq[0];
    scal->alpha = a;
    scal->rz_old = scal->rz;
    scal->fresh = 0;
    scal->rr = tot[0];
    const int it = scal->iter + 1;
    scal->iter = it;
    if (scal->hist && it <= scal->hist_cap) scal->hist[it - 1] = tot[0];
    if (tot[0] <= scal->tol2) scal->stop = 1;
    else if (!isfinite(tot[0])) scal->stop = 3;
    else if (it >= scal->max_iter) scal->stop = 2;
  }
}

// r.z from the cycle's partials, beta = r.z / r.z_old, p = z + beta p (beta = 0
// after a (re)start: p = z without reading p, which may hold anything).  Every
// block takes the same sum; block 0 records it.
__global__ void __launch_bounds__(kBlk)
    k_mgcg_pupdate(int64_t n, const double* __restrict__ z, double* __restrict__ p, CgScalars* __restrict__ scal,
                   const double* __restrict__ partials, int nb) {
  pdl_enter();
  if (any_in_block(scal->stop != 0)) return;  // (block 0 may set it)
  double rz[1];
  sum_partials<1>(partials, nb, rz);
  const bool fresh = scal->fresh != 0, bad = !isfinite(rz[0]) || !(rz[0] > 0.0);  // M must stay positive definite
  const double b = fresh ? 0.0 : rz[0] / scal->rz_old;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    scal->beta = b;
    scal->rz = rz[0];
    if (bad) scal->stop = 3;
  }
  if (bad) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = fresh ? z[i] : z[i] + b * p[i];
}

// ---- coarsest inverse: block Gauss-Jordan in place, blocks of 32, without
// pivoting (the matrix is symmetric positive definite); a pivot that is not
// positive sets *flag, and the host elimination with pivoting takes over.
constexpr int kGj = 32;

// The matrix of a level as a dense array, padded with the identity.
__global__ void k_gj_fill(int32_t N, int64_t n, int64_t ld, const int32_t* __restrict__ brow,
                          const int32_t* __restrict__ bcol, const int64_t* __restrict__ sptr,
                          const double* __restrict__ val, double* __restrict__ M) {
  const int64_t row = blockIdx.x;
  for (int64_t j = threadIdx.x; j < ld; j += blockDim.x) M[row * ld + j] = (row >= n && j == row) ? 1.0 : 0.0;
  __syncthreads();
  if (row >= n) return;
  const int64_t i = row / 3;
  const int r = (int)(row % 3);
  const int64_t s = i >> 5, b = brow[i], m = brow[i + 1] - b;
  for (int64_t k = threadIdx.x; k < m; k += blockDim.x) {
    const int64_t P = sptr[s] + k * kSlice + (i & 31), col = bcol[b + k];
    for (int c = 0; c < 3; ++c) M[row * ld + 3 * col + c] = val[vpos(P, 3 * r + c)];
  }
}

// Step k, first half: the inverse of the pivot block (every CTA forms it), block
// column j of the pivot row multiplied by it, and the old pivot column block of
// row j kept in C.
__global__ void __launch_bounds__(kGj* kGj)
    k_gj_panel(int64_t ld, int k, double* __restrict__ M, double* __restrict__ C, double* __restrict__ Pinv,
               int32_t* __restrict__ flag) {
  __shared__ double D[kGj][kGj + 1], A[kGj][kGj + 1];
  const int r = threadIdx.x / kGj, c = threadIdx.x % kGj, j = blockIdx.x;
  const int64_t k0 = (int64_t)k * kGj, j0 = (int64_t)j * kGj;
  D[r][c] = M[(k0 + r) * ld + k0 + c];
  A[r][c] = M[(k0 + r) * ld + j0 + c];
  C[(j0 + r) * kGj + c] = M[(j0 + r) * ld + k0 + c];
  __syncthreads();
  for (int s = 0; s < kGj; ++s) {
    const double piv = D[s][s];
    if (!(piv > 0.0) && threadIdx.x == 0) *flag = 1;
    const double ip = 1.0 / piv, row = D[s][c], col = D[r][s], own = D[r][c];
    __syncthreads();
    if (r == s)
      D[r][c] = c == s ? ip : row * ip;
    else
      D[r][c] = c == s ? -col * ip : own - col * (row * ip);
    __syncthreads();
  }
  if (j == k) {
    Pinv[r * kGj + c] = D[r][c];
    return;
  }
  double v = 0.0;
#pragma unroll
  for (int s = 0; s < kGj; ++s) v += D[r][s] * A[s][c];
  M[(k0 + r) * ld + j0 + c] = v;
}

// Second half: every block of the other rows, minus the old pivot column times
// the new pivot row; the pivot column becomes -C Pinv, the pivot block Pinv.
__global__ void __launch_bounds__(kGj* kGj)
    k_gj_update(int64_t ld, int k, double* __restrict__ M, const double* __restrict__ C,
                const double* __restrict__ Pinv) {
  __shared__ double A[kGj][kGj + 1], B[kGj][kGj + 1];
  const int r = threadIdx.x / kGj, c = threadIdx.x % kGj, i = blockIdx.y, j = blockIdx.x;
  const int64_t k0 = (int64_t)k * kGj, i0 = (int64_t)i * kGj, j0 = (int64_t)j * kGj;
  if (i == k) {
    if (j == k) M[(k0 + r) * ld + k0 + c] = Pinv[r * kGj + c];
    return;
  }
  A[r][c] = C[(i0 + r) * kGj + c];
  B[r][c] = j == k ? Pinv[r * kGj + c] : M[(k0 + r) * ld + j0 + c];
  __syncthreads();
  double v = 0.0;
#pragma unroll
  for (int s = 0; s < kGj; ++s) v += A[r][s] * B[s][c];
  const int64_t at = (i0 + r) * ld + j0 + c;
  M[at] = j == k ? -v : M[at] - v;
}

// ---------------------------------------------------------------- host side

int dinv_of(Ctx* lc) {
  if (!lc->dinv64) UFC_TRY(dalloc(lc, &lc->dinv64, lc->n));
  return UFC_STATUS_OK;
}

__global__ void k_mg_round(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

// The symmetric storage rounded to FP32, step by step (the layouts differ).
__global__ void k_mg_round_sym(int64_t nblocks, const double* __restrict__ a, float* __restrict__ b) {
  for (int64_t P = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; P < nblocks; P += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
    for (int c = 0; c < 9; ++c) b[spos<float>(P, c)] = (float)a[spos<double>(P, c)];
}

// A level's product in the cycle's precision: the symmetric storage where the
// level holds it (the finest level of a model assembled with
// UFC_BUILD_SYMMETRIC), else the full SELL storage.  Returns the number of
// partial sums.
int lv_product(const MgLevel& L, cudaStream_t st, const double* x, const MgEpi<double>& epi) {
  const Ctx* lc = L.c;
  if (lc->has_sval64) return launch_spmv_sym<double, double, double>(lc, st, lc->sval64, x, epi);
  return launch_spmv_diff<double, double, double, false>(lc, st, lc->val64, x, epi);
}
int lv_product(const MgLevel& L, cudaStream_t st, const float* x, const MgEpi<float>& epi) {
  const Ctx* lc = L.c;
  if (L.sval32) return launch_spmv_sym<float, float, float>(lc, st, L.sval32, x, epi);
  return launch_spmv_diff<float, float, float, false>(lc, st, L.val32, x, epi);
}

// Degree of the smoother (or of the Chebyshev solve) on level l.
int lv_degree(const Mg& mg, size_t l) { return l + 1 == mg.lv.size() ? mg.cheb_coarse : mg.degree; }
double lv_ratio(const Mg& mg, size_t l) { return l + 1 == mg.lv.size() ? 1000.0 : mg.ratio; }

// lambda_max of D^-1 A on level L by 15 steps of the power iteration v <- D^-1 A v
// (deterministic start, FP64), lambda = ||v_15|| / ||v_14||, and the smoother's
// coefficients from it; everything stays on the device.
int estimate_lmax(Ctx* owner, Mg& mg, size_t l) {
  constexpr int kIters = 15;
  MgLevel& L = mg.lv[l];
  Ctx* lc = L.c;
  const int64_t n = lc->n;
  const int m = lv_degree(mg, l);
  if (!L.pv) UFC_TRY(dalloc(owner, &L.pv, n));
  if (!L.pw) UFC_TRY(dalloc(owner, &L.pw, n));
  if (!L.coef) UFC_TRY(dalloc(owner, &L.coef, 2 * (int64_t)std::max(m, 1) + 2));
  if (!mg.dnorm) UFC_TRY(dalloc(owner, &mg.dnorm, 1));
  k_mg_start_vector<<<grid_n(n), kBlk, 0, owner->stream>>>(n, lc->fixed, L.pv);
  double *v = L.pv, *w = L.pw;
  int nb = 0;
  for (int it = 1; it <= kIters; ++it) {
    MgEpi<double> epi;
    epi.mode = kPower;
    epi.dinv = lc->dinv64;
    epi.dout = w;
    epi.dot = it + 1 >= kIters;
    nb = lv_product(L, owner->stream, v, epi);
    if (it + 1 == kIters) k_mg_sum<<<1, kBlk, 0, owner->stream>>>(lc->partials, nb, mg.dnorm);
    std::swap(v, w);
  }
  k_mg_coef<<<1, kBlk, 0, owner->stream>>>(lc->partials, nb, mg.dnorm, 1.0, lv_ratio(mg, l), m, L.coef);
  UFC_CUDA(owner, cudaGetLastError());
  return UFC_STATUS_OK;
}

int64_t dense_ld(int64_t n) { return (n + kGj - 1) / kGj * kGj; }

// The coarsest inverse on the device: enqueued only, *mg.gj_flag says whether it holds.
int dense_inverse_device(Ctx* owner, Mg& mg, MgLevel& L) {
  Ctx* lc = L.c;
  const int64_t n = lc->n, ld = dense_ld(n);
  const int nb = (int)(ld / kGj);
  if (!L.inv) UFC_TRY(dalloc(owner, &L.inv, ld * ld));
  if (!L.gj) UFC_TRY(dalloc(owner, &L.gj, ld * kGj + kGj * kGj));
  if (!mg.gj_flag) UFC_TRY(dalloc(owner, &mg.gj_flag, 1));
  double *C = L.gj, *Pinv = L.gj + ld * kGj;
  UFC_CUDA(owner, cudaMemsetAsync(mg.gj_flag, 0, sizeof(int32_t), owner->stream));
  k_gj_fill<<<(int)ld, 128, 0, owner->stream>>>(lc->N, n, ld, lc->brow, lc->bcol, lc->slice_ptr, lc->val64, L.inv);
  for (int k = 0; k < nb; ++k) {
    k_gj_panel<<<nb, kGj * kGj, 0, owner->stream>>>(ld, k, L.inv, C, Pinv, mg.gj_flag);
    k_gj_update<<<dim3(nb, nb), kGj * kGj, 0, owner->stream>>>(ld, k, L.inv, C, Pinv);
  }
  if (mg.fp32) {
    if (!L.inv32) UFC_TRY(dalloc(owner, &L.inv32, ld * ld));
    k_mg_round<<<grid_n(ld * ld), kBlk, 0, owner->stream>>>(ld * ld, L.inv, L.inv32);
  }
  UFC_CUDA(owner, cudaGetLastError());
  return UFC_STATUS_OK;
}

// Dense inverse of the coarsest matrix on the host (Gauss-Jordan with partial
// pivoting), for matrices whose elimination on the device met a pivot that is
// not positive.
int dense_inverse_host(Ctx* owner, MgLevel& L, bool fp32) {
  Ctx* lc = L.c;
  const int64_t n = lc->n, nnz = 9 * lc->nnzb;
  std::vector<int64_t> rp(n + 1);
  std::vector<int32_t> col(nnz);
  std::vector<double> val(nnz);
  ufc_csr_export_arg a{};
  a.index_base = 0;
  a.mem = UFC_MEM_HOST;
  a.row_ptr = rp.data();
  a.col_ind = col.data();
  a.values = val.data();
  UFC_TRY(export_csr(lc, &a));
  std::vector<double> M((size_t)n * n, 0.0), Inv((size_t)n * n, 0.0);
  for (int64_t i = 0; i < n; ++i) {
    for (int64_t k = rp[i]; k < rp[i + 1]; ++k) M[i * n + col[k]] = val[k];
    Inv[i * n + i] = 1.0;
  }
  for (int64_t c = 0; c < n; ++c) {
    int64_t piv = c;
    for (int64_t i = c + 1; i < n; ++i)
      if (std::fabs(M[i * n + c]) > std::fabs(M[piv * n + c])) piv = i;
    if (!(std::fabs(M[piv * n + c]) > 0.0))
      return fail(owner, UFC_STATUS_ERROR, "ufc_mg_setup: singular coarsest matrix (unconstrained rigid modes?)");
    if (piv != c)
      for (int64_t j = 0; j < n; ++j) {
        std::swap(M[c * n + j], M[piv * n + j]);
        std::swap(Inv[c * n + j], Inv[piv * n + j]);
      }
    const double s = 1.0 / M[c * n + c];
    for (int64_t j = 0; j < n; ++j) {
      M[c * n + j] *= s;
      Inv[c * n + j] *= s;
    }
    for (int64_t i = 0; i < n; ++i) {
      if (i == c) continue;
      const double f = M[i * n + c];
      if (f == 0.0) continue;
      for (int64_t j = 0; j < n; ++j) {
        M[i * n + j] -= f * M[c * n + j];
        Inv[i * n + j] -= f * Inv[c * n + j];
      }
    }
  }
  const int64_t ld = dense_ld(n);
  std::vector<double> out((size_t)ld * ld, 0.0);
  for (int64_t i = 0; i < n; ++i) std::copy(Inv.begin() + i * n, Inv.begin() + (i + 1) * n, out.begin() + i * ld);
  UFC_CUDA(owner, cudaMemcpyAsync(L.inv, out.data(), sizeof(double) * ld * ld, cudaMemcpyHostToDevice, owner->stream));
  if (fp32) k_mg_round<<<grid_n(ld * ld), kBlk, 0, owner->stream>>>(ld * ld, L.inv, L.inv32);
  UFC_CUDA(owner, cudaStreamSynchronize(owner->stream));
  return UFC_STATUS_OK;
}

template <typename T>
void free_vecs(MgVecs<T>& v, bool own_xb) {
  if (own_xb) {
    dfree(&v.x);
    dfree(&v.b);
  }
  dfree(&v.r);
  dfree(&v.d);
  dfree(&v.e);
  dfree(&v.w);
}

void free_level(MgLevel& L) {
  free_vecs(L.v64, L.own != nullptr);  // level 0: x and b are the caller's
  free_vecs(L.v32, true);
  dfree(&L.ke);
  dfree(&L.val32);
  dfree(&L.sval32);
  dfree(&L.dinv32);
  dfree(&L.coef);
  dfree(&L.inv);
  dfree(&L.inv32);
  dfree(&L.gj);
  dfree(&L.pv);
  dfree(&L.pw);
  if (L.own) ufc_ctx_destroy(L.own);
  L.own = nullptr;
}

// The vectors, diagonal and coarsest inverse of a level in the cycle's precision.
MgVecs<double>& vecs_of(MgLevel& L, double*) { return L.v64; }
MgVecs<float>& vecs_of(MgLevel& L, float*) { return L.v32; }
const double* dinv_of(const MgLevel& L, double*) { return L.c->dinv64; }
const float* dinv_of(const MgLevel& L, float*) { return L.dinv32; }
const double* inv_of(const MgLevel& L, double*) { return L.inv; }
const float* inv_of(const MgLevel& L, float*) { return L.inv32; }

// One V-cycle from level l, whose b and first step d = D^-1 b / theta are in
// place.  The result goes to x; on the finest level to z (FP64) with the
// partials of r.z left for the caller: returns their number.
template <typename T>
int vcycle(Ctx* owner, Mg& mg, size_t l, const CgScalars* scal, double* z, const double* r64) {
  MgLevel& L = mg.lv[l];
  Ctx* lc = L.c;
  cudaStream_t st = owner->stream;
  MgVecs<T>& V = vecs_of(L, (T*)nullptr);
  const T* dinv = dinv_of(L, (T*)nullptr);
  const bool last = l + 1 == mg.lv.size();
  if (last && !mg.cheb_coarse) {
    const int grid = (int)((lc->n * 32 + kBlk - 1) / kBlk);
    launch_pdl(k_mg_dense<T>, grid, kBlk, st, lc->n, dense_ld(lc->n), inv_of(L, (T*)nullptr), (const T*)V.b, V.x, scal);
    owner->launches += 1;
    return 0;
  }
  const int m = lv_degree(mg, l);
  MgEpi<T> e0;
  e0.scal = scal;
  e0.coef = L.coef;
  e0.dinv = dinv;
  // x = d, then m - 1 steps; `d` is gathered, the new one goes to the other buffer
  const T *rc = V.b, *xc = V.d;
  T *d = V.d, *dn = V.e;
  auto step = [&](int k, bool final_step) {
    MgEpi<T> e = e0;
    e.mode = kStep;
    e.step = k;
    e.rin = rc;
    e.xin = xc;
    e.rout = final_step ? nullptr : V.r;
    e.dout = final_step ? nullptr : dn;
    e.xout = V.x;
    if (final_step && l == 0) {
      e.xout = nullptr;
      e.z = z;
      e.r64 = r64;
      e.dot = r64 != nullptr;
    }
    const int nb = lv_product(L, st, (const T*)d, e);
    rc = V.r;
    xc = V.x;
    std::swap(d, dn);
    owner->launches += 1;
    return nb;
  };
  if (last) {  // Chebyshev solve from zero
    for (int k = 1; k < m; ++k) step(k, k + 1 == m);
    return 0;
  }
  for (int k = 1; k < m; ++k) step(k, false);
  {
    MgEpi<T> e = e0;
    e.mode = kResid;
    e.rin = rc;
    e.rout = V.r;
    lv_product(L, st, (const T*)d, e);
  }
  MgLevel& C = mg.lv[l + 1];
  MgVecs<T>& W = vecs_of(C, (T*)nullptr);
  const bool cs = l + 2 < mg.lv.size() || mg.cheb_coarse;  // the coarse level smooths
  launch_pdl(k_mg_restrict<T>, grid_for(C.c->N, 128), 128, st, C.nx, C.ny, C.nz, (const T*)V.r,
             (const uint8_t*)lc->fixed, (const uint8_t*)C.c->fixed, cs ? dinv_of(C, (T*)nullptr) : (const T*)nullptr,
             (const double*)C.coef, W.b, W.d, scal);
  vcycle<T>(owner, mg, l + 1, scal, nullptr, nullptr);
  launch_pdl(k_mg_prolong<T>, grid_for(lc->N, 128), 128, st, C.nx, C.ny, C.nz, (const T*)W.x,
             (const uint8_t*)lc->fixed, (const uint8_t*)C.c->fixed, V.w, scal);
  owner->launches += 3;
  MgEpi<T> e = e0;
  e.mode = kStart;
  e.rin = V.r;
  e.xin = xc;
  e.rout = m > 1 ? V.r : nullptr;
  e.dout = m > 1 ? dn : nullptr;
  e.xout = V.x;
  if (m == 1 && l == 0) {
    e.xout = nullptr;
    e.z = z;
    e.r64 = r64;
    e.dot = r64 != nullptr;
  }
  int nb = lv_product(L, st, (const T*)V.w, e);
  owner->launches += 1;
  std::swap(d, dn);
  rc = V.r;
  xc = V.x;
  for (int k = 1; k < m; ++k) nb = step(k, k + 1 == m);
  return nb;
}

// z = M r on the owner's stream from b and d of level 0 (mg_begin); r64, when
// given, takes part in r.z.  Returns the number of its partials.
int run_cycle(Ctx* c, Mg& mg, const double* r, double* z, const CgScalars* scal, bool dot) {
  MgLevel& L0 = mg.lv[0];
  if (mg.fp32) return vcycle<float>(c, mg, 0, scal, z, dot ? r : nullptr);
  L0.v64.b = const_cast<double*>(r);
  L0.v64.x = z;  // the smoother's running x
  return vcycle<double>(c, mg, 0, scal, z, dot ? r : nullptr);
}

// b and d of level 0 from r.
int begin_cycle(Ctx* c, Mg& mg, const double* r) {
  MgLevel& L0 = mg.lv[0];
  if (mg.fp32)
    k_mg_begin<float><<<grid_n(c->n), kBlk, 0, c->stream>>>(c->n, r, L0.v32.b, L0.v32.d, L0.dinv32, L0.coef);
  else
    k_mg_begin<double><<<grid_n(c->n), kBlk, 0, c->stream>>>(c->n, r, nullptr, L0.v64.d, c->dinv64, L0.coef);
  UFC_CUDA(c, cudaGetLastError());
  c->launches += 1;
  return UFC_STATUS_OK;
}

}  // namespace

void mg_mark_stale(Ctx* c) {
  if (c->mg) c->mg->stale = true;
}

void mg_release_graph(Ctx* c) {
  if (!c->mg || !c->mg->graph) return;
  cudaGraphExecDestroy(c->mg->graph);
  c->mg->graph = nullptr;
}

void mg_free(Ctx* c) {
  if (!c->mg) return;
  cudaStreamSynchronize(c->stream);  // the levels' own contexts free in order of their streams, not of this one
  for (auto& L : c->mg->lv) free_level(L);
  dfree(&c->mg->dnorm);
  dfree(&c->mg->gj_flag);
  if (c->mg->graph) cudaGraphExecDestroy(c->mg->graph);
  delete c->mg;
  c->mg = nullptr;
}

// The numerical part of the hierarchy, from the owner's current FP64 values
// (and J2 tangent): Galerkin element matrices, coarse matrices, diagonals,
// FP32 copies, smoother bounds and the coarsest inverse.  Run at set-up and
// again, on the same boxes and patterns, whenever the owner reassembles.
static int mg_alloc(Ctx* c, double** p, int64_t n) { return *p ? UFC_STATUS_OK : dalloc(c, p, n); }
static int mg_alloc(Ctx* c, float** p, int64_t n) { return *p ? UFC_STATUS_OK : dalloc(c, p, n); }

template <typename T>
static int alloc_vecs(Ctx* c, MgVecs<T>& v, int64_t n, bool xb) {
  if (xb) {
    UFC_TRY(mg_alloc(c, &v.x, n));
    UFC_TRY(mg_alloc(c, &v.b, n));
  }
  UFC_TRY(mg_alloc(c, &v.r, n));
  UFC_TRY(mg_alloc(c, &v.d, n));
  UFC_TRY(mg_alloc(c, &v.e, n));
  return mg_alloc(c, &v.w, n);
}

int mg_refresh(Ctx* c);

int mg_numeric(Ctx* c) {
  Mg& mg = *c->mg;
  const bool tangent = c->mat_model == UFC_MAT_J2_ISO;
  if (tangent && !c->Dt) return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: no J2 tangent");
  if (!c->dinv64) return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: no FP64 diagonal");
  for (size_t l = 1; l < mg.lv.size(); ++l) {
    MgLevel& F = mg.lv[l - 1];
    MgLevel& L = mg.lv[l];
    Ctx* lc = L.c;
    UFC_TRY(mg_alloc(c, &L.ke, (int64_t)lc->E * 576));
    constexpr int out_bytes = 8 * 576 * (int)sizeof(double);
    if (l > 1) {
      k_mg_galerkin<true, false><<<lc->E, kGalThreads, out_bytes, c->stream>>>(
          L.nx, L.ny, L.nz, nullptr, F.c->conn, nullptr, nullptr, F.ke, F.c->fixed, lc->conn, lc->fixed, L.ke,
          c->dev_err);
    } else if (tangent) {
      constexpr int bytes = std::max(out_bytes, 8 * (int)sizeof(GalWarp<true>));
      UFC_CUDA(c, cudaFuncSetAttribute(k_mg_galerkin<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
      k_mg_galerkin<false, true><<<lc->E, kGalThreads, bytes, c->stream>>>(
          L.nx, L.ny, L.nz, c->coords, c->conn, nullptr, c->Dt, nullptr, c->fixed, lc->conn, lc->fixed, L.ke,
          c->dev_err);
    } else {
      constexpr int bytes = std::max(out_bytes, 8 * (int)sizeof(GalWarp<false>));
      UFC_CUDA(c, cudaFuncSetAttribute(k_mg_galerkin<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
      k_mg_galerkin<false, false><<<lc->E, kGalThreads, bytes, c->stream>>>(
          L.nx, L.ny, L.nz, c->coords, c->conn, c->lame, nullptr, nullptr, c->fixed, lc->conn, lc->fixed, L.ke,
          c->dev_err);
    }
    UFC_CUDA(c, cudaGetLastError());
    const int64_t nv = lc->sell_blocks * 9;
    UFC_TRY(mg_alloc(c, &lc->val64, nv));
    UFC_TRY(dinv_of(lc));
    if (mg.fp32) {
      UFC_TRY(mg_alloc(c, &L.val32, nv));
      UFC_TRY(mg_alloc(c, &L.dinv32, lc->n));
    }
    const int stride = (9 * lc->max_row_blocks) | 1;
    const int bytes = (int)sizeof(double) * kMgRows * stride;  // (27 blocks a row at most: 31 KB, no limit to raise)
    RowOutputs<double> to;
    to.val = lc->val64;
    to.dinv = lc->dinv64;
    to.val_r = L.val32;
    to.dinv_r = L.dinv32;
    k_mg_rows<<<(int)(2 * lc->nslices), kMgRowThreads, bytes, c->stream>>>(
        lc->N, lc->nptr, lc->nelem, L.ke, lc->slot, lc->slice_ptr, lc->sell_col, lc->dpos, lc->fixed, stride, to);
    UFC_CUDA(c, cudaGetLastError());
    lc->has_val64 = true;
  }
  mg.lmax_scale = 1.0;
  mg.cheb_coarse = mg.lv.back().c->n <= kDenseMax ? 0 : 24;
  // level vectors in the cycle's precision (level 0: FP32 values too), smoother, coarsest solve
  for (size_t l = 0; l < mg.lv.size(); ++l) {
    MgLevel& L = mg.lv[l];
    const int64_t n = L.c->n;
    if (mg.fp32) {
      UFC_TRY(alloc_vecs(c, L.v32, n, true));
      if (l == 0) {
        UFC_TRY(mg_alloc(c, &L.dinv32, n));
        k_mg_round<<<grid_n(n), kBlk, 0, c->stream>>>(n, c->dinv64, L.dinv32);
        // the coded symmetric product reads half the bytes (128x64x64: 62 against 89 us)
        const int64_t nb = c->s_ublocks + kSlice;
        bool sym = c->has_sval64 && c->sym_coded && spmv_split(c) == 1;
        if (sym && mg_alloc(c, &L.sval32, nb * 9) != UFC_STATUS_OK) {
          // (the tangent's symmetric storage is taken where it fits; its copy need not fit too)
          if (!L.val32) return UFC_STATUS_MEM_ERROR;
          cudaGetLastError();
          c->err.clear();
          sym = false;
        }
        if (sym) {
          k_mg_round_sym<<<grid_n(nb), kBlk, 0, c->stream>>>(nb, c->sval64, L.sval32);
        } else {
          const int64_t nv = c->sell_blocks * 9;
          dfree(&L.sval32);
          UFC_TRY(mg_alloc(c, &L.val32, nv));
          k_mg_round<<<grid_n(nv), kBlk, 0, c->stream>>>(nv, c->val64, L.val32);
        }
      }
    } else {
      UFC_TRY(alloc_vecs(c, L.v64, n, l > 0));
    }
    if (l + 1 < mg.lv.size() || mg.cheb_coarse) UFC_TRY(estimate_lmax(c, mg, l));
  }
  MgLevel& Cst = mg.lv.back();
  if (!mg.cheb_coarse) UFC_TRY(dense_inverse_device(c, mg, Cst));
  UFC_TRY(check_dev_err(c, "ufc_mg_setup"));
  if (!mg.cheb_coarse) {
    int32_t flag = 0;
    UFC_CUDA(c, cudaMemcpyAsync(&flag, mg.gj_flag, sizeof(int32_t), cudaMemcpyDeviceToHost, c->stream));
    UFC_CUDA(c, cudaStreamSynchronize(c->stream));
    if (flag) UFC_TRY(dense_inverse_host(c, Cst, mg.fp32));
  }
  mg.stale = false;
  return UFC_STATUS_OK;
}

int mg_setup(Ctx* c, ufc_mg_arg* a) {
  const auto t0 = std::chrono::steady_clock::now();
  if (!c->has_pattern || !c->has_val64)
    return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: assemble the FP64 values first (UFC_BUILD_FP64)");
  const int32_t nx = a->nx, ny = a->ny, nz = a->nz;
  if (nx <= 0 || ny <= 0 || nz <= 0) return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: nx, ny, nz must be > 0");
  if ((int64_t)(nx + 1) * (ny + 1) * (nz + 1) != c->N || (int64_t)nx * ny * nz != c->E)
    return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: node or element count is not that of the nx x ny x nz box");
  const bool tangent = c->mat_model == UFC_MAT_J2_ISO;
  if (tangent && !c->has_trial)
    return fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: J2 tangent needs ufc_elem_compute_fint(update_state=1) first");
  // the connectivity must be the box numbering
  for (int64_t e = 0; e < c->E; ++e) {
    const int64_t i = e % nx, j = (e / nx) % ny, k = e / ((int64_t)nx * ny);
    for (int p = 0; p < 8; ++p) {
      const int64_t want = box_node(i + ((node_sign(p, 0) + 1) >> 1), j + ((node_sign(p, 1) + 1) >> 1),
                                    k + ((node_sign(p, 2) + 1) >> 1), nx, ny);
      if (c->h_conn[e * 8 + p] != want)
        return fail(c, UFC_STATUS_INVALID,
                    "ufc_mg_setup: element " + std::to_string(e) + " does not follow the box numbering");
    }
  }
  mg_free(c);
  release_graphs(c);
  c->mg = new Mg();
  Mg& mg = *c->mg;
  mg.degree = a->degree > 0 ? a->degree : 2;
  mg.ratio = a->ratio > 1.0 ? a->ratio : 15.0;
  const int64_t coarse_max = a->coarse_max > 0 ? a->coarse_max : 300;
  const int max_levels = a->max_levels > 0 ? a->max_levels : 32;
  auto bail = [&](int s) {
    mg_free(c);
    return s;
  };

  // level 0: the owner's matrix; its x and b are the PCG's z and r (bound at solve time)
  mg.lv.emplace_back();
  mg.lv[0].c = c;
  mg.lv[0].nx = nx;
  mg.lv[0].ny = ny;
  mg.lv[0].nz = nz;
  // the owner's FP64 Jacobi diagonal is current after every FP64 assembly
  if (!c->dinv64) return bail(fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: no FP64 diagonal"));

  // host copies of the fine coordinates and fixed mask, to derive the coarse boxes
  std::vector<double> h_coords(c->n);
  std::vector<uint8_t> h_fixed(c->n);
  if (cudaMemcpyAsync(h_coords.data(), c->coords, sizeof(double) * c->n, cudaMemcpyDeviceToHost, c->stream) !=
          cudaSuccess ||
      cudaMemcpyAsync(h_fixed.data(), c->fixed, c->n, cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
      cudaStreamSynchronize(c->stream) != cudaSuccess)
    return bail(fail(c, UFC_STATUS_ERROR, "ufc_mg_setup: copy of the mesh failed"));

  int32_t fx = nx, fy = ny, fz = nz;
  while ((int)mg.lv.size() < max_levels && fx % 2 == 0 && fy % 2 == 0 && fz % 2 == 0 &&
         3 * (int64_t)(fx + 1) * (fy + 1) * (fz + 1) > coarse_max) {
    const int32_t cx = fx / 2, cy = fy / 2, cz = fz / 2;
    const int64_t Nc = (int64_t)(cx + 1) * (cy + 1) * (cz + 1), Ec = (int64_t)cx * cy * cz;
    std::vector<double> cc(3 * Nc);
    std::vector<uint8_t> cf(3 * Nc);
    for (int64_t k = 0; k <= cz; ++k)
      for (int64_t j = 0; j <= cy; ++j)
        for (int64_t i = 0; i <= cx; ++i) {
          const int64_t vc = box_node(i, j, k, cx, cy), vf = box_node(2 * i, 2 * j, 2 * k, fx, fy);
          for (int d = 0; d < 3; ++d) {
            cc[3 * vc + d] = h_coords[3 * vf + d];
            cf[3 * vc + d] = h_fixed[3 * vf + d];
          }
        }
    std::vector<int32_t> conn(8 * Ec);
    for (int64_t e = 0; e < Ec; ++e) {
      const int64_t i = e % cx, j = (e / cx) % cy, k = e / ((int64_t)cx * cy);
      for (int p = 0; p < 8; ++p)
        conn[8 * e + p] = (int32_t)box_node(i + ((node_sign(p, 0) + 1) >> 1), j + ((node_sign(p, 1) + 1) >> 1),
                                            k + ((node_sign(p, 2) + 1) >> 1), cx, cy);
    }
    std::vector<int32_t> fixed_dofs;
    for (int64_t q = 0; q < 3 * Nc; ++q)
      if (cf[q]) fixed_dofs.push_back((int32_t)q);
    MgLevel L;
    L.nx = cx;
    L.ny = cy;
    L.nz = cz;
    int st = ufc_ctx_create(c->device, &L.own);
    if (st != UFC_STATUS_OK) return bail(fail(c, st, "ufc_mg_setup: coarse context"));
    L.c = L.own;
    mg.lv.push_back(L);
    MgLevel& M = mg.lv.back();
    ufc_mesh_desc md{(int32_t)Nc, (int32_t)Ec, cc.data(), conn.data(), 0, UFC_MEM_HOST};
    ufc_bc_desc bd{(int32_t)fixed_dofs.size(), fixed_dofs.data(), nullptr, UFC_MEM_HOST};
    ufc_pattern_info pi{};
    if ((st = ufc_mesh_set(M.own, &md)) != UFC_STATUS_OK || (st = ufc_bc_set(M.own, &bd)) != UFC_STATUS_OK ||
        (st = ufc_pattern_build(M.own, &pi)) != UFC_STATUS_OK)
      return bail(fail(c, st, "ufc_mg_setup: coarse level " + std::to_string(mg.lv.size() - 1) + ": " + M.c->err));
    h_coords.swap(cc);
    h_fixed.swap(cf);
    fx = cx;
    fy = cy;
    fz = cz;
  }
  if (mg.lv.size() < 2) return bail(fail(c, UFC_STATUS_INVALID, "ufc_mg_setup: the box cannot be coarsened"));

  mg.fp32 = a->precision == UFC_PRECISION_FP32_REFINE;
  {
    const int st = mg_numeric(c);
    if (st != UFC_STATUS_OK) return bail(st);
  }
  a->levels = (int32_t)mg.lv.size();
  a->coarse_dof = mg.lv.back().c->n;
  UFC_CUDA(c, cudaStreamSynchronize(c->stream));
  a->setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  return UFC_STATUS_OK;
}

int mg_apply(Ctx* c, const double* r, double* z) {
  if (!c->mg) return fail(c, UFC_STATUS_INVALID, "ufc_mg_apply: multigrid not set up (ufc_mg_setup)");
  if (c->mg->stale) UFC_TRY(mg_refresh(c));
  UFC_TRY(begin_cycle(c, *c->mg, r));
  run_cycle(c, *c->mg, r, z, nullptr, false);
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

int mg_level_ctx(Ctx* c, int32_t level, Ctx** out) {
  if (!c->mg) return fail(c, UFC_STATUS_INVALID, "multigrid not set up");
  if (level < 0 || level >= (int32_t)c->mg->lv.size()) return fail(c, UFC_STATUS_INVALID, "multigrid level out of range");
  *out = c->mg->lv[level].c;
  return UFC_STATUS_OK;
}

int mg_refresh(Ctx* c) {
  if (!c->has_val64) return fail(c, UFC_STATUS_INVALID, "multigrid: the FP64 values are not assembled");
  if (c->mat_model == UFC_MAT_J2_ISO && !c->has_trial)
    return fail(c, UFC_STATUS_INVALID, "multigrid: J2 tangent needs ufc_elem_compute_fint(update_state=1) first");
  return mg_numeric(c);
}

// The PCG iteration as a graph: the V-cycle from b and d of level 0 (z and the
// partials of r.z), the direction, the product, the update with the next b and
// d and the stop test.  Kept with the hierarchy (the smoothers' coefficients
// are read from memory, so a refresh keeps it); rebuilt when one of the vectors
// or values it reads has moved.  What else it bakes in (pattern, partial sums)
// is released with the CG graphs (release_graphs) when it is rebuilt.
static int pcg_mg_graph(Ctx* c, Mg& mg, int batch) {
  const void* key[9] = {c->r64, c->p64, c->q64, c->z64, c->x64, c->has_sval64 ? c->sval64 : nullptr, c->val64,
                        mg.lv[0].sval32, mg.lv[0].val32};
  if (mg.graph && mg.batch == batch && std::equal(key, key + 9, mg.key)) return UFC_STATUS_OK;
  if (mg.graph) cudaGraphExecDestroy(mg.graph);
  mg.graph = nullptr;
  MgLevel& L0 = mg.lv[0];
  const int64_t n = c->n, counted = c->launches;
  const int vg = grid_n(n);
  double* upd = c->partials + c->partials_cap / 2;  // the update's partials, behind the products'
  cudaGraph_t g;
  UFC_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  for (int b = 0; b < batch; ++b) {
    const Partials rz = product_partials(c, c->stream, run_cycle(c, mg, c->r64, c->z64, c->scal, true));
    launch_pdl(k_mgcg_pupdate, vg, kBlk, c->stream, n, (const double*)c->z64, c->p64, c->scal, rz.p, rz.nb);
    const EpiCg<double> epi{c->q64, c->scal};
    const int nb = c->has_sval64 ? launch_spmv_sym<double, double, double>(c, c->stream, c->sval64, c->p64, epi)
                                 : launch_spmv<double, double, double>(c, c->stream, c->val64, c->p64, epi);
    const Partials pq = product_partials(c, c->stream, nb);
    if (mg.fp32)
      launch_pdl(k_mgcg_update<float>, vg, kBlk, c->stream, n, (const double*)c->p64, (const double*)c->q64, c->r64,
                 c->x64, L0.v32.b, L0.v32.d, (const float*)L0.dinv32, (const double*)L0.coef, c->scal, pq.p, pq.nb,
                 upd);
    else
      launch_pdl(k_mgcg_update<double>, vg, kBlk, c->stream, n, (const double*)c->p64, (const double*)c->q64, c->r64,
                 c->x64, (double*)nullptr, L0.v64.d, (const double*)c->dinv64, (const double*)L0.coef, c->scal, pq.p,
                 pq.nb, upd);
    c->launches += 3;
  }
  cudaError_t e = cudaStreamEndCapture(c->stream, &g);
  mg.graph_launches = c->launches - counted;  // captured launches run when the graph does
  c->launches = counted;
  if (e != cudaSuccess) return cuda_fail(c, e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(&mg.graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_fail(c, e, "cudaGraphInstantiate");
  mg.batch = batch;
  std::copy(key, key + 9, mg.key);
  return UFC_STATUS_OK;
}

// The smoothers' intervals for a solve: as estimated, or widened by set().  A
// solve leaves them as it found them, so that it gives the same bits on a
// hierarchy that others have used before.
struct Widening {
  Ctx* c;
  Mg& mg;
  ~Widening() {
    if (mg.lmax_scale != 1.0) set(1.0);
  }
  void set(double scale) {
    mg.lmax_scale = scale;
    for (size_t l = 0; l < mg.lv.size(); ++l)
      if (mg.lv[l].coef && lv_degree(mg, l) > 0)
        k_mg_coef<<<1, kBlk, 0, c->stream>>>(nullptr, 0, nullptr, scale, lv_ratio(mg, l), lv_degree(mg, l),
                                             mg.lv[l].coef);
  }
};

int pcg_mg(Ctx* c, const ufc_solver_algo* algo, ufc_solver_state* st) {
  if (!c->mg) return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: multigrid not set up (ufc_mg_setup)");
  if (c->mg->stale) UFC_TRY(mg_refresh(c));
  Mg& mg = *c->mg;
  if (!c->r64 || !c->p64 || !c->q64) return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: vectors");
  if (!c->z64) UFC_TRY(dalloc(c, &c->z64, c->n));
  const int64_t n = c->n;
  const int vg = grid_n(n);
  cudaEvent_t t0, t1;
  UFC_CUDA(c, cudaEventCreate(&t0));
  UFC_CUDA(c, cudaEventCreate(&t1));
  UFC_CUDA(c, cudaEventRecord(t0, c->stream));
  c->timing = ufc_timing_info{};
  c->timing.precision = UFC_PRECISION_FP64;
  c->launches = 0;

  CgScalars h{};
  h.max_iter = algo->max_iter > 0 ? algo->max_iter : 1;
  const int32_t cap = std::min<int32_t>(h.max_iter, 1 << 20);
  if (c->hist_cap < cap) {
    UFC_TRY(dalloc(c, &c->hist, cap));
    c->hist_cap = cap;
  }
  h.hist = c->hist;
  h.hist_cap = c->hist_cap;
  UFC_CUDA(c, cudaMemcpyAsync(c->scal, &h, sizeof(CgScalars), cudaMemcpyHostToDevice, c->stream));
  // r = b - K x0 (FP64), ||b||
  UFC_TRY(true_residual_fp64(c, true));
  UFC_CUDA(c, cudaMemcpyAsync(c->h_scal, c->scal, sizeof(CgScalars), cudaMemcpyDeviceToHost, c->stream));
  UFC_CUDA(c, cudaStreamSynchronize(c->stream));
  if (!std::isfinite(c->h_scal->bb)) return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: non-finite right-hand side");
  if (!std::isfinite(c->h_scal->true_rr))
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: non-finite initial residual (initial guess or matrix)");
  const double bnorm_raw = std::sqrt(c->h_scal->bb);
  const double bnorm = bnorm_raw < 1e-30 ? 1.0 : bnorm_raw;
  const double tol = std::max(algo->tolerance * bnorm, algo->abs_tolerance);
  st->initial_residual = std::sqrt(c->h_scal->true_rr);
  double true_rr = c->h_scal->true_rr;
  bool converged = std::sqrt(true_rr) <= tol;
  int flag = 0, restarts = 0;
  const int batch = algo->check_every > 0 ? algo->check_every : 2;
  int status = UFC_STATUS_OK;
  Widening widening{c, mg};
  cudaEvent_t done[2] = {nullptr, nullptr};
  if (!converged) {
    UFC_TRY(pcg_mg_graph(c, mg, batch));
    for (auto& e : done) UFC_CUDA(c, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  }
  CgScalars* hs[2] = {c->h_scal + 1, c->h_scal + 2};
  while (!converged && status == UFC_STATUS_OK) {
    // (re)start: r = the FP64 residual, b and d of the cycle; the first iteration takes p = z = M r
    struct {
      int32_t stop, want, fresh;
    } restart{0, 0, 1};
    static_assert(offsetof(CgScalars, want_update) == offsetof(CgScalars, stop) + 4 &&
                      offsetof(CgScalars, fresh) == offsetof(CgScalars, stop) + 8,
                  "restart writes stop, want_update and fresh in one copy");
    double tol2 = tol * tol;
    UFC_CUDA(c, cudaMemcpyAsync(&c->scal->tol2, &tol2, sizeof(double), cudaMemcpyHostToDevice, c->stream));
    UFC_CUDA(c, cudaMemcpyAsync(&c->scal->stop, &restart, sizeof(restart), cudaMemcpyHostToDevice, c->stream));
    UFC_CUDA(c, cudaMemcpyAsync(c->r64, c->y64, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
    UFC_TRY(begin_cycle(c, mg, c->r64));
    // one batch stays in flight while the one before it is looked at
    int slot = 0, in_flight = 0;
    for (;;) {
      cudaError_t e = cudaGraphLaunch(mg.graph, c->stream);
      if (e != cudaSuccess) {
        status = cuda_fail(c, e, "cudaGraphLaunch");
        break;
      }
      c->launches += mg.graph_launches;
      UFC_CUDA(c, cudaMemcpyAsync(hs[slot], c->scal, sizeof(CgScalars), cudaMemcpyDeviceToHost, c->stream));
      UFC_CUDA(c, cudaEventRecord(done[slot], c->stream));
      slot ^= 1;
      if (in_flight == 0) {
        in_flight = 1;
        continue;
      }
      UFC_CUDA(c, cudaEventSynchronize(done[slot]));
      if (hs[slot]->stop) break;
    }
    if (status != UFC_STATUS_OK) break;
    const int stop = hs[slot]->stop;
    UFC_TRY(true_residual_fp64(c, false));
    UFC_CUDA(c, cudaMemcpyAsync(c->h_scal, c->scal, sizeof(CgScalars), cudaMemcpyDeviceToHost, c->stream));
    UFC_CUDA(c, cudaStreamSynchronize(c->stream));
    true_rr = c->h_scal->true_rr;
    if (std::sqrt(true_rr) <= tol) {
      converged = true;
      break;
    }
    if (stop == 2 || !std::isfinite(true_rr)) {
      flag = std::isfinite(true_rr) ? 2 : 3;
      break;
    }
    if (++restarts > 4) {
      flag = 3;
      break;
    }
    if (stop == 3) {
      // the cycle was not positive definite: lambda_max was underestimated, so
      // the smoothers' intervals are widened before the restart
      constexpr double kWiden = 1.3;
      widening.set(mg.lmax_scale * kWiden);
      UFC_CUDA(c, cudaGetLastError());
    }
  }
  for (auto& e : done)
    if (e) cudaEventDestroy(e);
  if (status != UFC_STATUS_OK) return status;
  UFC_CUDA(c, cudaEventRecord(t1, c->stream));
  UFC_CUDA(c, cudaEventSynchronize(t1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  c->hist_len = std::min(c->h_scal->iter, c->hist_cap);
  st->niter = c->h_scal->iter;
  st->n_refine = restarts;
  st->converged = converged ? 1 : 0;
  st->convergence_flag = converged ? 0 : (flag ? flag : 2);
  st->rnorm = std::sqrt(true_rr) / bnorm;
  st->solve_time = ms;
  c->timing.kernel_launches = c->launches;
  UFC_TRY(check_dev_err(c, "ufc_pcg_solve"));
  return converged ? UFC_STATUS_OK : UFC_STATUS_NOT_CONVERGED;
}

}  // namespace ufc
