// Jacobi-PCG iterations of a small FP64 system in one kernel.
//
// On the smallest meshes a CG iteration of three launches is launch and reduction
// latency (7 to 8 us whatever the size).  Here the whole loop runs in one launch:
// a CTA owns a run of SELL slices and holds their values and columns in shared
// memory as far as they fit, a thread owns a block row and keeps the row's x, r,
// p, q and D^-1 in registers across iterations, and what crosses CTAs is z and p
// (one 48-byte record per row) and two sums per iteration.  Those two sums are the
// only synchronisations between CTAs: rows gather z_j + beta p_j (the previous
// direction), so the new direction needs none of its own.  Inside a CTA a barrier
// stands before each sum's last part and before the warps' parts of a row are
// added, in the one-CTA form also between the direction and its gathers.
//
// Two forms by size:
//   one CTA       up to 4 slices: __syncthreads, the direction in shared memory;
//                 3.6 us per iteration at 99 nodes (the product's shared-memory
//                 reads are 1.3 us of it)
//   one cluster   up to 48 slices: barrier.cluster, partial sums written into each
//                 CTA's shared memory; 4.4 us at 390 nodes, 6.9 us at 1,377
// A third form over all SMs (cooperative launch, sums pushed to every CTA and
// polled there) took 10 us per iteration at 1,710 and at 3,321 nodes, 8 to 10 us
// of it in the two exchanges between CTAs; larger systems keep the graph of
// three kernels (7.9 us at 3,321 nodes).
// Sums are taken in CTA order by every CTA alike, so all take the same decisions
// and runs are reproducible.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "reduce.cuh"
#include "resident_rule.h"
#include "ufc_internal.cuh"

namespace ufc {

namespace {

namespace cg = cooperative_groups;

constexpr int kResThreads = 512;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxRows1 = (int)kOneCtaSlices * kSlice;  // rows of the one-CTA form

enum ResSync { kOneCta = 0, kCluster = 1 };

// A stored step (32 rows' blocks) in shared memory: values and columns.
constexpr int kStepBytes = 288 * (int)sizeof(double) + 32 * (int)sizeof(int32_t);
constexpr int kResSmem = 208 * 1024;       // dynamic shared memory for the steps

struct ResArgs {
  int32_t N;
  int32_t nslices;
  int32_t steps;  // stored steps of a CTA that its shared memory takes
  const int64_t* sptr;
  const int32_t* col;
  const double* val;
  const double* dinv;  // null: no preconditioner
  double *x, *r, *p;   // [n]
  double* zp;          // [N][6]: z and p of every row
  CgScalars* scal;
  int32_t chunk;    // iterations at most
};

// The next direction's entry, rounded alike in its own thread and in the rows that gather it.
__device__ __forceinline__ double next_p(double z, double beta, double p) { return __fma_rn(beta, p, z); }

template <int SYNC>
__global__ void __launch_bounds__(kResThreads, 1) k_cg_resident(const ResArgs A) {
  __shared__ double sh_row[kResWarps][3][32];
  __shared__ double sh_red[2][kResWarps][2];              // [phase][warp][value]
  __shared__ double sh_part[2][kResCluster][2];           // [phase][CTA][value] (cluster)
  __shared__ double sh_p[SYNC == kOneCta ? 3 * kResMaxRows1 : 1];
  extern __shared__ __align__(16) unsigned char res_smem[];
  double* sh_val = reinterpret_cast<double*>(res_smem);                                // [steps][288]
  int32_t* sh_col = reinterpret_cast<int32_t*>(sh_val + 288 * (int64_t)A.steps);       // [steps][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x, me = blockIdx.x;
  // slices [s0, s1) of this CTA, `split` warps per slice
  const int s0 = (int)((int64_t)A.nslices * me / G), s1 = (int)((int64_t)A.nslices * (me + 1) / G), ns = s1 - s0;
  const int split = kResWarps / ns;  // ns <= kResWarps
  const int sl = warp / split, part = warp % split;
  const bool work = sl < ns;
  const int64_t base0 = A.sptr[s0], base = work ? A.sptr[s0 + sl] : 0;
  const int len = work ? (int)((A.sptr[s0 + sl + 1] - base) >> 5) : 0;
  const int step0 = (int)((base - base0) >> 5);  // this slice's first step among the CTA's
  {
    const int have = (int)min((A.sptr[s1] - base0) >> 5, (int64_t)A.steps);
    const double2* src = reinterpret_cast<const double2*>(A.val + 9 * base0);
    double2* dst = reinterpret_cast<double2*>(sh_val);
    for (int k = threadIdx.x; k < have * 144; k += kResThreads) dst[k] = __ldcs(src + k);
    for (int k = threadIdx.x; k < have * 32; k += kResThreads) sh_col[k] = __ldcs(A.col + base0 + k);
  }
  // the row this thread owns
  const int64_t row = (int64_t)s0 * kSlice + threadIdx.x;
  const bool own = (int)threadIdx.x < ns * kSlice && row < A.N;
  double x[3] = {0, 0, 0}, r[3] = {0, 0, 0}, p[3] = {0, 0, 0}, z[3] = {0, 0, 0}, di[3] = {1, 1, 1}, q[3] = {0, 0, 0};
  if (own)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = 3 * row + c;
      x[c] = A.x[i];
      r[c] = A.r[i];
      p[c] = A.p[i];
      if (A.dinv) di[c] = A.dinv[i];
    }
  double rz = A.scal->rz, rz_old = A.scal->rz_old, rr = A.scal->rr, beta = A.scal->beta, alpha = 0.0, pq = 0.0;
  const double tol2 = A.scal->tol2;
  const int max_iter = A.scal->max_iter, hist_cap = A.scal->hist_cap;
  double* hist = A.scal->hist;
  int iter = A.scal->iter, stop = 0;

  // Sums over all CTAs of v0 (and v1 with PH = 1) held by the owning threads.
  // The second sum of an iteration also orders the CTA's z and p records before
  // the gathers that follow it in other CTAs.
  auto reduce = [&](auto phase, double v0, double v1, double& o0, double& o1) {
    constexpr int PH = decltype(phase)::value;
    if (warp < ns) {
      double v[2] = {v0, v1};
      warp_sum<2>(v);
      if (lane == 0) {
        sh_red[PH][warp][0] = v[0];
        sh_red[PH][warp][1] = v[1];
      }
    }
    __syncthreads();
    o0 = o1 = 0.0;
    if constexpr (SYNC == kOneCta) {
      for (int k = 0; k < ns; ++k) {
        o0 += sh_red[PH][k][0];
        o1 += sh_red[PH][k][1];
      }
    } else {
      cg::cluster_group cl = cg::this_cluster();
      if (warp == 0 && lane < G) {
        double a = 0.0, b = 0.0;
        for (int k = 0; k < ns; ++k) {
          a += sh_red[PH][k][0];
          b += sh_red[PH][k][1];
        }
        double* dst = cl.map_shared_rank(&sh_part[PH][me][0], lane);
        dst[0] = a;
        dst[1] = b;
      }
      cl.sync();
      for (int k = 0; k < G; ++k) {
        o0 += sh_part[PH][k][0];
        o1 += sh_part[PH][k][1];
      }
    }
  };

  bool first = true;
  int done = 0;
  // the first sum writes into the other CTAs' shared memory, which may not be
  // touched before they have started
  if constexpr (SYNC == kCluster)
    cg::this_cluster().sync();
  else
    __syncthreads();
  while (done < A.chunk) {
    // direction: given on entry, then z + beta p
    if (!first && own)
#pragma unroll
      for (int c = 0; c < 3; ++c) p[c] = next_p(z[c], beta, p[c]);
    if constexpr (SYNC == kOneCta) {
      if (own)
#pragma unroll
        for (int c = 0; c < 3; ++c) sh_p[3 * threadIdx.x + c] = p[c];
      __syncthreads();
    }
    // part of the row sums of q = K p
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
#pragma unroll 2
    for (int j = part; j < len; j += split) {
      const int k = step0 + j;
      const bool in = k < A.steps;
      const int64_t cj = in ? sh_col[32 * k + lane] : __ldg(A.col + base + 32 * (int64_t)j + lane);
      double y[3];
      if constexpr (SYNC == kOneCta) {
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = sh_p[3 * cj + c];
      } else if (first) {
#pragma unroll
        for (int c = 0; c < 3; ++c) y[c] = __ldcg(A.p + 3 * cj + c);
      } else {
        const double2* rec = reinterpret_cast<const double2*>(A.zp + 6 * cj);
        const double2 u = __ldcg(rec), v = __ldcg(rec + 1), w = __ldcg(rec + 2);
        y[0] = next_p(u.x, beta, v.y);
        y[1] = next_p(u.y, beta, w.x);
        y[2] = next_p(v.x, beta, w.y);
      }
      if (in) {
        const double* v = sh_val + 288 * k + lane;
        a0 += v[0] * y[0] + v[32] * y[1] + v[64] * y[2];
        a1 += v[96] * y[0] + v[128] * y[1] + v[160] * y[2];
        a2 += v[192] * y[0] + v[224] * y[1] + v[256] * y[2];
      } else {
        const double* v = A.val + 9 * base + 288 * (int64_t)j + lane;
        a0 += __ldg(v) * y[0] + __ldg(v + 32) * y[1] + __ldg(v + 64) * y[2];
        a1 += __ldg(v + 96) * y[0] + __ldg(v + 128) * y[1] + __ldg(v + 160) * y[2];
        a2 += __ldg(v + 192) * y[0] + __ldg(v + 224) * y[1] + __ldg(v + 256) * y[2];
      }
    }
    sh_row[warp][0][lane] = a0;
    sh_row[warp][1][lane] = a1;
    sh_row[warp][2][lane] = a2;
    __syncthreads();
    double d = 0.0;
    if (own) {
      const int w0 = (threadIdx.x >> 5) * split;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        q[c] = 0.0;
        for (int k = 0; k < split; ++k) q[c] += sh_row[w0 + k][c][lane];
        d += p[c] * q[c];
      }
    }
    double unused;
    reduce(std::integral_constant<int, 0>{}, d, 0.0, pq, unused);
    if (!(fabs(pq) > 1e-300) || !isfinite(pq)) {
      stop = 3;
      break;
    }
    alpha = rz / pq;
    double v0 = 0.0, v1 = 0.0;
    if (own) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        x[c] += alpha * p[c];
        r[c] -= alpha * q[c];
        z[c] = di[c] * r[c];
        v0 += r[c] * z[c];
        v1 += r[c] * r[c];
      }
      if constexpr (SYNC != kOneCta) {
        double2* rec = reinterpret_cast<double2*>(A.zp + 6 * row);
        __stcg(rec, make_double2(z[0], z[1]));
        __stcg(rec + 1, make_double2(z[2], p[0]));
        __stcg(rec + 2, make_double2(p[1], p[2]));
      }
    }
    rz_old = rz;
    reduce(std::integral_constant<int, 1>{}, v0, v1, rz, rr);
    beta = rz / rz_old;
    ++iter;
    ++done;
    first = false;
    if (me == 0 && threadIdx.x == 0 && hist && iter <= hist_cap) hist[iter - 1] = rr;
    if (rr <= tol2) stop = 1;
    else if (!(fabs(rz_old) > 1e-300) || !isfinite(rz)) stop = 3;
    else if (iter >= max_iter) stop = 2;
    if (stop) break;
  }
  // every CTA has left its last product by now (a sum follows it), so A.p, which
  // the first one gathers from, can be written
  if (own)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = 3 * row + c;
      A.x[i] = x[c];
      A.r[i] = r[c];
      // at the end of a run p is that of its last iteration; at the end of a
      // chunk the next direction
      A.p[i] = stop || first ? p[c] : next_p(z[c], beta, p[c]);
    }
  if (me == 0 && threadIdx.x == 0) {
    A.scal->pq = pq;
    A.scal->alpha = alpha;
    A.scal->beta = beta;
    A.scal->rz = rz;
    A.scal->rz_old = rz_old;
    A.scal->rr = rr;
    A.scal->iter = iter;
    A.scal->stop = stop;
  }
}

// The launch of the form with g CTAs.
struct ResLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  int32_t steps;
  ResLaunch(const Ctx* c, int g) {
    // no CTA has more steps than ceil(slices / CTAs) slices of the longest row
    const int64_t most = (c->nslices + g - 1) / g * c->max_row_blocks;
    steps = (int32_t)std::min<int64_t>(most, kResSmem / kStepBytes);
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(kResThreads);
    cfg.stream = c->stream;
    cfg.dynamicSmemBytes = (size_t)steps * kStepBytes;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = g;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g > 1 ? 1 : 0;
  }
};

template <int SYNC>
cudaError_t allow_resident() {
  const auto kernel = k_cg_resident<SYNC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem);
  if (e == cudaSuccess && SYNC == kCluster)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

bool cluster_placeable(const Ctx* c, int g) {
  const ResLaunch L(c, g);
  int n = 0;
  cudaError_t e = allow_resident<kCluster>();
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, k_cg_resident<kCluster>, &L.cfg);
  if (e != cudaSuccess) cudaGetLastError();  // not a failure of the solve: the chain of kernels takes over
  return e == cudaSuccess && n > 0;
}

}  // namespace

int cg_resident_plan(Ctx* c) {
  if (c->res_ctas < 0) c->res_ctas = resident_ctas(c->nslices, [c](int g) { return cluster_placeable(c, g); });
  return c->res_ctas;
}

// At most `chunk` iterations from r64, p64 and the scalars, as the kernels of a
// batch would leave them, on the g CTAs of cg_resident_plan.
int cg_resident(Ctx* c, const double* dinv, int chunk, int g) {
  ResArgs a{};
  a.N = c->N;
  a.nslices = (int32_t)c->nslices;
  a.sptr = c->slice_ptr;
  a.col = c->sell_col;
  a.val = c->val64;
  a.dinv = dinv;
  a.x = c->x64;
  a.r = c->r64;
  a.p = c->p64;
  if (!c->res_zp) UFC_TRY(dalloc(c, &c->res_zp, 6 * (int64_t)c->N));
  a.zp = c->res_zp;
  a.scal = c->scal;
  a.chunk = chunk;
  const ResLaunch L(c, g);
  a.steps = L.steps;
  if (g > 1) {
    UFC_CUDA(c, allow_resident<kCluster>());
    UFC_CUDA(c, cudaLaunchKernelEx(&L.cfg, k_cg_resident<kCluster>, a));
  } else {
    UFC_CUDA(c, allow_resident<kOneCta>());
    UFC_CUDA(c, cudaLaunchKernelEx(&L.cfg, k_cg_resident<kOneCta>, a));
  }
  c->launches += 1;
  return UFC_STATUS_OK;
}

}  // namespace ufc
