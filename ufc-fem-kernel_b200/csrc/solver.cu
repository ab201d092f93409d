// SELL-32 SpMV and the Jacobi-preconditioned CG of NM_Solver_PCG /
// iter_pcg (ufc_core/L2_NM/Solver/NM_Solv_Core.f90:363-423,
// ufc_core/L2_NM/Solver/LinSolv/NM_Solv_IterSolver.f90:713-846).
//
// One CG iteration is three kernels:
//   k_spmv<.., kCg>   q = K p, per-block partials of p.q
//   k_cg_update       alpha = r.z / p.q, x += alpha p (x in FP64), r -= alpha q,
//                     z = D^-1 r fused, per-block partials of r.z and r.r
//   k_cg_pupdate      beta, the stop test and the refinement trigger, p = D^-1 r + beta p
// A reduction ends in the kernel that follows it: every block there sums the
// partials again, in the same order (k_cg_sum first when there are thousands).
// No block waits for a fence or an election: with that wait at the end of each
// of the product's 7094 blocks the FP32 product of 192x96x96 took 230 us in the
// iteration against 186 us on its own.
// The scalars live in device memory (CgScalars) and every kernel returns at
// once when the run has stopped, so batches of iterations are launched as one
// CUDA graph and the host only looks at the scalars between batches.
//
// UFC_PRECISION_FP32_REFINE keeps the matrix and the CG vectors in FP32 and the
// solution in FP64.  Whenever the FP32 recursive residual has fallen by
// refine_delta since the last replacement, and whenever it meets the tolerance,
// the residual is recomputed in FP64 as r = b - K x with the FP64 element
// operator (matrix-free, K assembled from FP64 element stiffnesses) and
// replaces the recursive one (residual replacement).  The run ends when the
// FP64 residual meets the tolerance.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>

#include "c3d8_device.cuh"
#include "reduce.cuh"
#include "spmv.cuh"
#include "ufc_internal.cuh"

namespace ufc {

int apply_fp64_eliminated(Ctx* c, const double* x, double* y);

namespace {

constexpr int kVecBlock = 256;

// Grid of the CG vector kernels: they take 4 entries per thread (16-byte
// loads), so n / 4 threads, at most 8 blocks per SM (grid-stride beyond).
// On small meshes the kernels are bound by the launch and the grid reduction,
// which fewer blocks shorten (212k DOF: update 9.7 -> 8.8 us).
int vec_grid(int64_t n) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t need = ((n + 3) / 4 + kVecBlock - 1) / kVecBlock;
  return (int)std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)sms * 8));
}

// 4 consecutive entries through 16-byte loads and stores (allocations are
// 256-byte aligned; callers pass offsets that are multiples of 4 entries); the
// loads past L1, for those before griddepcontrol.wait.
template <typename T>
__device__ __forceinline__ void ld4_cg(const T* __restrict__ p, T (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  } else {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p + 2));
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
  }
}

template <typename T>
__device__ __forceinline__ void st4(T* __restrict__ p, const T (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  } else {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(o[2], o[3]);
  }
}

// x += alpha p, r -= alpha q with alpha = r.z / p.q (p.q from the product's nb
// partials), and the block's partials of r.z and r.r.  Block 0 moves the
// scalars on; the other blocks read only scal->rz, which this kernel leaves alone.
// A thread's first entries of p, r, x and D^-1 are read before the wait for the
// product, which writes only q and its partials (the kernels that wrote p, r and
// x were complete before the product began).
template <typename T>
__global__ void __launch_bounds__(kVecBlock)
    k_cg_update(int64_t n, const T* __restrict__ p, const T* __restrict__ q, T* __restrict__ r,
                double* __restrict__ x, const T* __restrict__ dinv, CgScalars* __restrict__ scal,
                const double* __restrict__ pq_partials, int nb, double* __restrict__ partials) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4 = n >> 2;
  T pv[4], qv[4], rv[4], dv[4];
  double xv[4];
  auto load = [&](int64_t i) {
    ld4_cg(p + i, pv);
    ld4_cg(r + i, rv);
    ld4_cg(x + i, xv);
    if (dinv) ld4_cg(dinv + i, dv);
  };
  if (gid < n4) load(gid << 2);
  pdl_enter();
  const bool seen = halted(scal);  // block 0 of this kernel may set it (breakdown)
  if (gid < n4) ld4_cg(q + (gid << 2), qv);
  if (any_in_block(seen)) return;
  double pq[1];
  sum_partials<1>(pq_partials, nb, pq);
  const bool broken = !(fabs(pq[0]) > 1e-300) || !isfinite(pq[0]);
  const double alpha = scal->rz / pq[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    scal->pq = pq[0];
    if (broken) {
      scal->stop = 3;
    } else {
      scal->alpha = alpha;
      scal->rz_old = scal->rz;
      scal->iter += 1;
    }
  }
  if (broken) return;
  const T a = (T)alpha;
  T rz = T(0), rr = T(0);
  for (int64_t k = gid; k < n4; k += stride) {
    const int64_t i = k << 2;
    if (k != gid) {
      load(i);
      ld4_cg(q + i, qv);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      xv[c] += alpha * (double)pv[c];
      rv[c] -= a * qv[c];
      const T zc = dinv ? dv[c] * rv[c] : rv[c];
      rz += rv[c] * zc;
      rr += rv[c] * rv[c];
    }
    st4(r + i, rv);
    st4(x + i, xv);
  }
  for (int64_t i = (n4 << 2) + gid; i < n; i += stride) {
    const T pi = p[i], qi = q[i];
    x[i] += alpha * (double)pi;
    const T ri = r[i] - a * qi;
    r[i] = ri;
    const T zi = dinv ? dinv[i] * ri : ri;
    rz += ri * zi;
    rr += ri * ri;
  }
  double v[2] = {(double)rz, (double)rr};
  block_partial<2>(v, partials);
}

// p = D^-1 r + beta p.  In the iteration (nb > 0) r.z and r.r come from the
// update's nb partials, every block takes the same decisions from them (stop
// test, refinement trigger: then p stays), and block 0 records them; the others
// read only scalars that this kernel leaves alone.  On its own (nb = 0) it
// takes scal->beta.
template <typename T>
__global__ void __launch_bounds__(kVecBlock)
    k_cg_pupdate(int64_t n, const T* __restrict__ r, const T* __restrict__ dinv, T* __restrict__ p,
                 CgScalars* __restrict__ scal, const double* __restrict__ partials, int nb) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4 = n >> 2;
  T rv[4], pv[4], dv[4];
  // the update in front writes r, not p and D^-1
  auto load = [&](int64_t i) {
    ld4_cg(p + i, pv);
    if (dinv) ld4_cg(dinv + i, dv);
  };
  if (gid < n4) load(gid << 2);
  pdl_enter();
  const bool seen = halted(scal);  // block 0 of this kernel may set it
  if (gid < n4) ld4_cg(r + (gid << 2), rv);
  if (any_in_block(seen)) return;
  double b;
  if (nb > 0) {
    double tot[2];
    sum_partials<2>(partials, nb, tot);
    const double rz_old = scal->rz_old;
    const int it = scal->iter;
    int stop = 0, want = 0;
    if (tot[1] <= scal->tol2) stop = 1;
    else if (!(fabs(rz_old) > 1e-300) || !isfinite(tot[0])) stop = 3;
    else if (it >= scal->max_iter) stop = 2;
    if (scal->delta2 > 0.0 && tot[1] < scal->delta2 * scal->rr_ref) want = 1;
    b = tot[0] / rz_old;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      scal->rz = tot[0];
      scal->rr = tot[1];
      scal->beta = b;
      if (scal->hist && it <= scal->hist_cap) scal->hist[it - 1] = tot[1];
      if (stop) scal->stop = stop;
      if (want) scal->want_update = 1;
    }
    if (stop | want) return;
  } else {
    b = scal->beta;
  }
  const T beta = (T)b;
  // beta = 0 (start, restart after a breakdown): p = z whatever p holds (fresh
  // memory, or the NaN of the breakdown)
  const bool fresh = b == 0.0;
  for (int64_t k = gid; k < n4; k += stride) {
    const int64_t i = k << 2;
    if (k != gid) {
      load(i);
      ld4_cg(r + i, rv);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) pv[c] = (dinv ? dv[c] * rv[c] : rv[c]) + (fresh ? T(0) : beta * pv[c]);
    st4(p + i, pv);
  }
  for (int64_t i = (n4 << 2) + gid; i < n; i += stride) {
    const T ri = r[i];
    p[i] = (dinv ? dinv[i] * ri : ri) + (fresh ? T(0) : beta * p[i]);
  }
}

// res = b - y and ||res||^2 -> scal->true_rr (and ||b||^2 -> scal->bb when asked).
__global__ void __launch_bounds__(kVecBlock)
    k_resid(int64_t n, const double* __restrict__ b, const double* y, double* res,
            CgScalars* __restrict__ scal, double* __restrict__ partials, int want_bb) {
  double rr = 0.0, bb = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double bi = b[i];
    const double ri = bi - (y ? y[i] : 0.0);
    res[i] = ri;
    rr += ri * ri;
    bb += bi * bi;
  }
  double v[2] = {rr, bb}, tot[2];
  if (grid_sum<2>(v, partials, &scal->ticket[2], tot)) {
    scal->true_rr = tot[0];
    if (want_bb) scal->bb = tot[1];
  }
}

// Residual replacement: r := res (rounded to T), z = D^-1 r, r.z and r.r.
// mode 0: mid-run (p already updated); 1: the run stopped before its p update,
// which is then done with beta = r.z / rz_old; 2: start (beta = 0, p = z).
template <typename T>
__global__ void __launch_bounds__(kVecBlock)
    k_replace(int64_t n, const double* __restrict__ res, T* __restrict__ r, const T* __restrict__ dinv,
              CgScalars* __restrict__ scal, double* __restrict__ partials, int mode) {
  T rz = T(0), rr = T(0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const T ri = (T)res[i];
    r[i] = ri;
    const T zi = dinv ? dinv[i] * ri : ri;
    rz += ri * zi;
    rr += ri * ri;
  }
  double v[2] = {(double)rz, (double)rr}, tot[2];
  if (grid_sum<2>(v, partials, &scal->ticket[3], tot)) {
    if (mode == 1) scal->beta = tot[0] / scal->rz_old;
    if (mode == 2) scal->beta = 0.0;
    scal->rz = tot[0];
    scal->rr = tot[1];
    scal->rr_ref = tot[1];
    scal->stop = 0;
    scal->want_update = 0;
  }
}

struct Run {
  Ctx* c;
  int prec;  // UFC_PRECISION_*
  int64_t n;
  int vg;    // vector-kernel grid
};

// CG vectors of type TX over stored values of type TV; sym selects the
// symmetric SpMV storage.
template <typename TV, typename TX>
struct Vecs {
  TX *r, *p, *q;
  const TV* val;
  const TX* dinv;
  bool sym;
};

template <typename TV, typename TX>
Vecs<TV, TX> vecs(Ctx* c, bool precond) {
  Vecs<TV, TX> v;
  if constexpr (sizeof(TX) == 8) {
    v.r = c->r64; v.p = c->p64; v.q = c->q64;
    v.dinv = precond ? c->dinv64 : nullptr;
  } else {
    v.r = c->r32; v.p = c->p32; v.q = c->q32;
    v.dinv = precond ? c->dinv32 : nullptr;
  }
  if constexpr (sizeof(TV) == 8) {
    v.sym = c->has_sval64;
    v.val = v.sym ? c->sval64 : c->val64;
  } else {
    v.sym = c->has_sval32;
    v.val = v.sym ? c->sval32 : c->val32;
  }
  return v;
}

template <typename TV, typename TX, typename TA>
void launch_iteration(const Run& R, const Vecs<TV, TX>& V, cudaStream_t st, cudaEvent_t ev0, cudaEvent_t ev1) {
  Ctx* c = R.c;
  if (ev0) cudaEventRecord(ev0, st);
  const EpiCg<TX> epi{V.q, c->scal};
  const int nb = V.sym ? launch_spmv_sym<TV, TX, TA>(c, st, V.val, V.p, epi)
                       : launch_spmv<TV, TX, TA>(c, st, V.val, V.p, epi);
  if (ev1) cudaEventRecord(ev1, st);
  const Partials pq = product_partials(c, st, nb);
  double* rz = c->partials + c->partials_cap / 2;  // the update's partials, behind the product's
  launch_pdl(k_cg_update<TX>, R.vg, kVecBlock, st, R.n, V.p, V.q, V.r, c->x64, V.dinv, c->scal, pq.p, pq.nb, rz);
  launch_pdl(k_cg_pupdate<TX>, R.vg, kVecBlock, st, R.n, V.r, V.dinv, V.p, c->scal, (const double*)rz, R.vg);
  c->launches += 3;
}

// FP64 residual of the current x64 into y64 / r-source, true_rr on the device.
// FP64 runs use their own matrix; refined FP32 runs use the matrix-free FP64
// element operator for the linear-elastic material and the assembled FP64
// values otherwise (the J2 tangent).
int true_residual(const Run& R, bool want_bb) {
  Ctx* c = R.c;
  if (R.prec == UFC_PRECISION_FP64 || c->mat_model != UFC_MAT_ELASTIC_ISO) {
    if (c->has_sval64)
      launch_spmv_sym<double, double, double>(c, c->stream, c->sval64, c->x64, EpiStore<double>{c->y64});
    else
      launch_spmv<double, double, double>(c, c->stream, c->val64, c->x64, EpiStore<double>{c->y64});
    UFC_CUDA(c, cudaGetLastError());
    c->launches += 1;
  } else {
    UFC_TRY(apply_fp64_eliminated(c, c->x64, c->y64));
  }
  k_resid<<<R.vg, kVecBlock, 0, c->stream>>>(R.n, c->b64, c->y64, c->y64, c->scal, c->partials, want_bb ? 1 : 0);
  UFC_CUDA(c, cudaGetLastError());
  c->launches += 1;
  return UFC_STATUS_OK;
}

template <typename TV, typename TX>
int replace(const Run& R, const Vecs<TV, TX>& V, int mode) {
  Ctx* c = R.c;
  k_replace<TX><<<R.vg, kVecBlock, 0, c->stream>>>(R.n, c->y64, V.r, V.dinv, c->scal, c->partials, mode);
  UFC_CUDA(c, cudaGetLastError());
  c->launches += 1;
  if (mode != 0) {
    k_cg_pupdate<TX><<<R.vg, kVecBlock, 0, c->stream>>>(R.n, V.r, V.dinv, V.p, c->scal, nullptr, 0);
    UFC_CUDA(c, cudaGetLastError());
    c->launches += 1;
  }
  return UFC_STATUS_OK;
}

int read_scalars(Ctx* c) {
  UFC_CUDA(c, cudaMemcpyAsync(c->h_scal, c->scal, sizeof(CgScalars), cudaMemcpyDeviceToHost, c->stream));
  UFC_CUDA(c, cudaStreamSynchronize(c->stream));
  return UFC_STATUS_OK;
}

template <typename TV, typename TX, typename TA>
int get_graph(const Run& R, const Vecs<TV, TX>& V, int batch, cudaGraphExec_t* out, int64_t* launches) {
  Ctx* c = R.c;
  // one cached graph per (value, vector, accumulator) type combination
  const int slot = sizeof(TV) == 8 ? 0 : sizeof(TX) == 8 ? 3 : sizeof(TA) == 8 ? 2 : 1;
  // graphs are rebuilt when a buffer they read, the preconditioner, the storage
  // (symmetric or full), the SpMV form (FP32 difference form, coded indices)
  // or the sizes baked into their launches (DOFs, slices) change; a reassembly
  // into the same arrays keeps them.  The vector and pattern buffers are not in
  // the key: ensure_vectors, build_sym_pattern and alloc_symmetric, which
  // reallocate them, release the graphs themselves.
  const void* key = (const void*)V.dinv;
  const void* val = (const void*)V.val;
  const int form = (V.sym ? 1 : 0) | (c->val32_diff ? 2 : 0) | (c->sym_coded ? 4 : 0) | (c->full_coded ? 8 : 0);
  if (c->cg_graph[slot] && c->cg_graph_batch[slot] == batch && c->cg_graph_key[slot] == key &&
      c->cg_graph_val[slot] == val && c->cg_graph_form[slot] == form && c->cg_graph_n[slot] == R.n &&
      c->cg_graph_slices[slot] == c->nslices) {
    *out = c->cg_graph[slot];
    *launches = c->cg_graph_launches[slot];
    return UFC_STATUS_OK;
  }
  if (c->cg_graph[slot]) cudaGraphExecDestroy(c->cg_graph[slot]);
  c->cg_graph[slot] = nullptr;
  cudaGraph_t g;
  const int64_t counted = c->launches;  // captured launches run only when the graph is launched
  UFC_CUDA(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
  for (int k = 0; k < batch; ++k) launch_iteration<TV, TX, TA>(R, V, c->stream, nullptr, nullptr);
  cudaError_t e = cudaStreamEndCapture(c->stream, &g);
  *launches = c->cg_graph_launches[slot] = c->launches - counted;
  c->launches = counted;
  if (e != cudaSuccess) return cuda_fail(c, e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(&c->cg_graph[slot], g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_fail(c, e, "cudaGraphInstantiate");
  c->cg_graph_batch[slot] = batch;
  c->cg_graph_key[slot] = key;
  c->cg_graph_val[slot] = val;
  c->cg_graph_form[slot] = form;
  c->cg_graph_n[slot] = R.n;
  c->cg_graph_slices[slot] = c->nslices;
  *out = c->cg_graph[slot];
  return UFC_STATUS_OK;
}

int ensure_vectors(Ctx* c, int prec) {
  const int64_t n = c->n;
  bool realloc = false;
  auto need = [&](auto** p) -> int {
    if (*p) return UFC_STATUS_OK;
    realloc = true;
    return dalloc(c, p, n);
  };
  UFC_TRY(need(&c->x64));
  UFC_TRY(need(&c->b64));
  UFC_TRY(need(&c->y64));
  if (prec == UFC_PRECISION_FP64 || prec == UFC_PRECISION_FP32_MATRIX) {
    UFC_TRY(need(&c->r64));
    UFC_TRY(need(&c->p64));
    UFC_TRY(need(&c->q64));
  } else {
    UFC_TRY(need(&c->r32));
    UFC_TRY(need(&c->p32));
    UFC_TRY(need(&c->q32));
  }
  if (prec != UFC_PRECISION_FP64) UFC_TRY(need(&c->xb64));
  if (realloc) release_graphs(c);
  return UFC_STATUS_OK;
}

constexpr int kResidentChunk = 1024;  // iterations of one resident launch between host checks

template <typename TV, typename TX, typename TA>
int pcg_run(Ctx* c, const ufc_solver_algo* algo, ufc_solver_state* st) {
  const int prec = algo->precision_mode;
  Run R{c, prec, c->n, vec_grid(c->n)};
  const bool precond = algo->precond_type == UFC_SOLV_PREC_JACOBI;
  Vecs<TV, TX> V = vecs<TV, TX>(c, precond);
  const int batch = algo->check_every > 0 ? algo->check_every : 32;

  cudaEvent_t t0, t1;
  UFC_CUDA(c, cudaEventCreate(&t0));
  UFC_CUDA(c, cudaEventCreate(&t1));
  UFC_CUDA(c, cudaEventRecord(t0, c->stream));
  c->timing = ufc_timing_info{};
  c->timing.precision = prec;
  c->timing.spmv_bytes = spmv_bytes(c, prec);
  c->launches = 0;

  // scalars: reset and configure
  CgScalars h{};
  h.max_iter = algo->max_iter > 0 ? algo->max_iter : 1;
  h.delta2 = 0.0;
  if (prec != UFC_PRECISION_FP64) {
    const double d = algo->refine_delta > 0.0 ? algo->refine_delta : 0.1;
    h.delta2 = d * d;
  }
  // residual history (NM_Solver_State%residual_history): one double per iteration
  const int32_t cap = std::min<int32_t>(h.max_iter, 1 << 20);
  if (c->hist_cap < cap) {
    UFC_TRY(dalloc(c, &c->hist, cap));
    c->hist_cap = cap;
  }
  h.hist = c->hist;
  h.hist_cap = c->hist_cap;
  UFC_CUDA(c, cudaMemcpyAsync(c->scal, &h, sizeof(CgScalars), cudaMemcpyHostToDevice, c->stream));
  UFC_TRY(true_residual(R, true));
  UFC_TRY(read_scalars(c));
  if (!std::isfinite(c->h_scal->bb)) return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: non-finite right-hand side");
  if (!std::isfinite(c->h_scal->true_rr))
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: non-finite initial residual (initial guess or matrix)");
  const double bnorm_raw = std::sqrt(c->h_scal->bb);
  const double bnorm = bnorm_raw < 1e-30 ? 1.0 : bnorm_raw;
  const double tol_nominal = std::max(algo->tolerance * bnorm, algo->abs_tolerance);
  const double tol = kStopMargin * tol_nominal;
  st->initial_residual = std::sqrt(c->h_scal->true_rr);
  double true_rr = c->h_scal->true_rr;
  int flag = 0;
  bool converged = std::sqrt(true_rr) <= tol;
  int n_refine = 0;

  if (!converged) {
    double tol2 = tol * tol;
    UFC_CUDA(c, cudaMemcpyAsync(&c->scal->tol2, &tol2, sizeof(double), cudaMemcpyHostToDevice, c->stream));
    UFC_TRY(replace(R, V, 2));
    cudaGraphExec_t graph = nullptr;
    int64_t graph_launches = 0;
    // small FP64 systems: all iterations in one kernel (resident.cu)
    int resident = 0;  // its CTAs
    if constexpr (sizeof(TV) == 8) resident = c->instrument ? 0 : cg_resident_plan(c);
    if (!c->instrument && !resident) UFC_TRY((get_graph<TV, TX, TA>(R, V, batch, &graph, &graph_launches)));
    std::vector<cudaEvent_t> evs;
    if (c->instrument) {
      evs.resize(2 * batch);
      for (auto& e : evs) UFC_CUDA(c, cudaEventCreate(&e));
    }
    CgScalars* hs[2] = {c->h_scal + 1, c->h_scal + 2};
    cudaEvent_t done[2];
    UFC_CUDA(c, cudaEventCreateWithFlags(&done[0], cudaEventDisableTiming));
    UFC_CUDA(c, cudaEventCreateWithFlags(&done[1], cudaEventDisableTiming));
    int slot = 0, in_flight = 0, iter_seen = 0;
    int stall = 0, restarts = 0;
    double best_rr = true_rr;
    constexpr int kMaxStall = 3;       // replacements without a 4x drop of ||b - K x||^2
    constexpr int kMaxRestarts = 4;    // restarts after a breakdown of the recurrence
    constexpr double kDiverge = 1e4;   // ||b - K x|| grew 100x above the best seen
    const bool keep_best = c->xb64 != nullptr;
    if (keep_best) cudaMemcpyAsync(c->xb64, c->x64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream);
    bool finished = false;
    int status = UFC_STATUS_OK;
    while (!finished) {
      CgScalars cur;
      if (resident) {
        if constexpr (sizeof(TV) == 8)
          status = cg_resident(c, V.dinv, algo->check_every > 0 ? algo->check_every : kResidentChunk, resident);
        if (status == UFC_STATUS_OK) status = read_scalars(c);
        if (status != UFC_STATUS_OK) break;
        cur = *c->h_scal;
      } else {
        if (graph) {
          cudaError_t e = cudaGraphLaunch(graph, c->stream);
          if (e != cudaSuccess) {
            status = cuda_fail(c, e, "cudaGraphLaunch");
            break;
          }
          c->launches += graph_launches;
        } else {
          for (int k = 0; k < batch; ++k)
            launch_iteration<TV, TX, TA>(R, V, c->stream, evs[2 * k], evs[2 * k + 1]);
        }
        cudaMemcpyAsync(hs[slot], c->scal, sizeof(CgScalars), cudaMemcpyDeviceToHost, c->stream);
        cudaEventRecord(done[slot], c->stream);
        if (c->instrument) {
          // one batch in flight at a time: the events are reused; only the
          // launches that did an iteration (not the no-op tail) are counted
          cudaEventSynchronize(done[slot]);
          const int did = std::min(batch, hs[slot]->iter - iter_seen);
          iter_seen = hs[slot]->iter;
          for (int k = 0; k < did; ++k) {
            float ms = 0.f;
            if (cudaEventElapsedTime(&ms, evs[2 * k], evs[2 * k + 1]) == cudaSuccess) {
              c->timing.spmv_ms += ms;
              c->timing.spmv_launches += 1;
            }
          }
          in_flight = 1;
          slot ^= 1;
        }
        if (in_flight == 0) {
          in_flight = 1;
          slot ^= 1;
          continue;
        }
        const int prev = slot ^ 1;
        cudaEventSynchronize(done[prev]);
        const CgScalars* s = hs[prev];
        if (!(s->stop || s->want_update)) {
          slot ^= 1;
          continue;
        }
        // act on the latest state
        cudaEventSynchronize(done[slot]);
        in_flight = 0;
        cur = *hs[c->instrument ? prev : slot];
        slot = 0;
      }
      if (cur.stop == 0 && !cur.want_update) continue;
      status = true_residual(R, false);
      if (status != UFC_STATUS_OK) break;
      status = read_scalars(c);
      if (status != UFC_STATUS_OK) break;
      true_rr = c->h_scal->true_rr;
      ++n_refine;
      if (std::sqrt(true_rr) <= tol) {
        converged = true;
        finished = true;
        break;
      }
      if (cur.stop == 2 || !std::isfinite(true_rr)) {
        flag = std::isfinite(true_rr) ? 2 : 3;
        finished = true;
        break;
      }
      // progress of the FP64 residual across replacements; the best iterate is
      // kept so that a stalled or diverging run can hand it on
      if (true_rr < best_rr) {
        if (keep_best) cudaMemcpyAsync(c->xb64, c->x64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream);
        if (true_rr < 0.25 * best_rr) stall = 0;
        else ++stall;
        best_rr = true_rr;
      } else {
        ++stall;
      }
      if (stall > kMaxStall || true_rr > kDiverge * best_rr) {
        flag = 3;
        finished = true;
        if (keep_best) {  // hand on the best iterate and its residual
          cudaMemcpyAsync(c->x64, c->xb64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream);
          true_rr = best_rr;
        }
        break;
      }
      // the iteration kernels halt right after the update that stopped the run or
      // asked for the replacement, before its direction update (mode 1)
      int mode = 1;
      if (cur.stop == 3) {
        // breakdown of the recurrence: restart CG from the FP64 residual
        if (++restarts > kMaxRestarts) {
          flag = 3;
          finished = true;
          if (keep_best) {
            cudaMemcpyAsync(c->x64, c->xb64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream);
            true_rr = best_rr;
          }
          break;
        }
        mode = 2;
      }
      if (prec != UFC_PRECISION_FP64 && algo->refine_policy == UFC_REFINE_RESTART) mode = 2;
      status = replace(R, V, mode);
      if (status != UFC_STATUS_OK) break;
    }
    for (auto& e : evs) cudaEventDestroy(e);
    cudaEventDestroy(done[0]);
    cudaEventDestroy(done[1]);
    if (status != UFC_STATUS_OK) return status;
    // stalled or out of iterations short of the margin, but within the tolerance
    if (!converged && std::isfinite(true_rr) && std::sqrt(true_rr) <= tol_nominal) {
      converged = true;
      flag = 0;
    }
  }
  UFC_TRY(read_scalars(c));
  UFC_CUDA(c, cudaEventRecord(t1, c->stream));
  UFC_CUDA(c, cudaEventSynchronize(t1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  c->timing.kernel_launches = c->launches;
  c->hist_len = std::min(c->h_scal->iter, c->hist_cap);
  st->niter = c->h_scal->iter;
  st->n_refine = n_refine;
  st->converged = converged ? 1 : 0;
  st->convergence_flag = converged ? 0 : (flag ? flag : 2);
  st->rnorm = std::sqrt(true_rr) / bnorm;
  st->solve_time = ms;
  UFC_TRY(check_dev_err(c, "ufc_pcg_solve"));
  return converged ? UFC_STATUS_OK : UFC_STATUS_NOT_CONVERGED;
}

}  // namespace

void release_graphs(Ctx* c) {
  mg_release_graph(c);
  for (int k = 0; k < kGraphSlots; ++k) {
    if (c->cg_graph[k]) cudaGraphExecDestroy(c->cg_graph[k]);
    c->cg_graph[k] = nullptr;
    c->cg_graph_batch[k] = 0;
    c->cg_graph_key[k] = nullptr;
    c->cg_graph_val[k] = nullptr;
    c->cg_graph_form[k] = 0;
    c->cg_graph_n[k] = c->cg_graph_slices[k] = 0;
  }
}

int64_t spmv_bytes(const Ctx* c, int precision) {
  // algorithmic bytes of one block-CSR SpMV: values + block column indices +
  // block row pointers + x read once + y written once (slice padding excluded)
  const int64_t sv = precision == UFC_PRECISION_FP64 ? 8 : 4;  // stored value
  const int64_t sx = precision == UFC_PRECISION_FP32_REFINE ? 4 : 8;  // vector entry
  const bool sym = precision == UFC_PRECISION_FP64 ? c->has_sval64 : c->has_sval32;
  if (sym) {
    const int64_t upper = (c->nnzb + c->N) / 2, lower = (c->nnzb - c->N) / 2;
    // coded indices (one-warp-per-slice form): upper values, 32 code bytes per
    // row, x and y; the lower values are re-read from L2
    if (c->sym_coded && spmv_split(c) == 1) return upper * 9 * sv + 32 * c->nslices * kSlice + 2 * c->n * sx;
    // symmetric storage: upper blocks (values + column), lower references
    // (position + column; their values are re-read from L2), x and y
    return upper * (9 * sv + 4) + lower * 8 + 2 * c->n * sx;
  }
  // coded indices: values, 32 code bytes per row, x and y
  if (c->full_coded && sv == 4 && !c->val32_diff && spmv_split(c) == 1)
    return c->nnzb * 9 * sv + 32 * c->nslices * kSlice + 2 * c->n * sx;
  return c->nnzb * (9 * sv + 4) + 4 * ((int64_t)c->N + 1) + 2 * c->n * sx;
}

// The products of the multigrid cycle and of its outer PCG take the symmetric
// storage of a level when it holds current values (the finest level of a model
// assembled with UFC_BUILD_SYMMETRIC: FP64 values and the same values rounded
// to FP32, as the cycle's own FP32 copy), else the full SELL storage.
void spmv64_on(const Ctx* lvl, cudaStream_t st, const double* x, double* y) {
  if (lvl->has_sval64)
    launch_spmv_sym<double, double, double>(lvl, st, lvl->sval64, x, EpiStore<double>{y});
  else
    launch_spmv<double, double, double>(lvl, st, lvl->val64, x, EpiStore<double>{y});
}

int true_residual_fp64(Ctx* c, bool want_bb) {
  spmv64_on(c, c->stream, c->x64, c->y64);
  UFC_CUDA(c, cudaGetLastError());
  k_resid<<<vec_grid(c->n), kVecBlock, 0, c->stream>>>(c->n, c->b64, c->y64, c->y64, c->scal, c->partials,
                                                       want_bb ? 1 : 0);
  UFC_CUDA(c, cudaGetLastError());
  c->launches += 2;
  return UFC_STATUS_OK;
}

int spmv(Ctx* c, int precision, const void* x, void* y) {
  if (!c->has_pattern) return fail(c, UFC_STATUS_INVALID, "ufc_spmv: pattern not built");
  if (precision == UFC_PRECISION_FP64) {
    if (!c->has_val64) return fail(c, UFC_STATUS_INVALID, "ufc_spmv: FP64 values not assembled");
    if (c->has_sval64)
      launch_spmv_sym<double, double, double>(c, c->stream, c->sval64, (const double*)x, EpiStore<double>{(double*)y});
    else
      launch_spmv<double, double, double>(c, c->stream, c->val64, (const double*)x, EpiStore<double>{(double*)y});
  } else if (precision == UFC_PRECISION_FP32_REFINE) {
    if (!c->has_val32) return fail(c, UFC_STATUS_INVALID, "ufc_spmv: FP32 values not assembled");
    if (c->has_sval32)
      launch_spmv_sym<float, float, float>(c, c->stream, c->sval32, (const float*)x, EpiStore<float>{(float*)y});
    else
      launch_spmv<float, float, float>(c, c->stream, c->val32, (const float*)x, EpiStore<float>{(float*)y});
  } else if (precision == UFC_PRECISION_FP32_MATRIX) {
    if (!c->has_val32) return fail(c, UFC_STATUS_INVALID, "ufc_spmv: FP32 values not assembled");
    if (c->has_sval32)
      launch_spmv_sym<float, double, double>(c, c->stream, c->sval32, (const double*)x, EpiStore<double>{(double*)y});
    else
      launch_spmv<float, double, double>(c, c->stream, c->val32, (const double*)x, EpiStore<double>{(double*)y});
  } else {
    return fail(c, UFC_STATUS_INVALID, "ufc_spmv: precision");
  }
  UFC_CUDA(c, cudaGetLastError());
  return UFC_STATUS_OK;
}

// True when one FP64 product of the stored matrix reads less than half the L2.
bool fp64_fits_l2(const Ctx* c) {
  int dev = 0, l2 = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess || l2 <= 0) return false;
  return spmv_bytes(c, UFC_PRECISION_FP64) < (int64_t)l2 / 2;
}

// Whether the FP64 solves of a Newton increment take the symmetric storage of the
// tangent: on a stencil-like numbering (on a random one the transposed blocks
// are scattered reads), with Jacobi where the full values exceed half the L2,
// with multigrid twice the L2.  Below, both forms come from L2 and the full one
// reads no block twice.  Second increment of a J2 bar, full against symmetric,
// ms: Jacobi 48x24x24 (59 MB) 26.9/26.5, 56x28x28 (93 MB) 40.0/37.0, 64x32x32
// 58.4/52.7, 96x48x48 (456 MB) 311/206; multigrid 56x28x28 11.0/11.5, 64x32x32
// (137 MB) 9.6/9.9, 96x48x48 25.5/19.6.  The first increment builds the
// symmetric pattern, 2 ms at 64x32x32.
// The rule looks at sizes only, so that the same increment takes the same
// products whatever else the device holds.  The storage is optional here and
// must not end a run that fits without it: it is not taken where four times the
// full values would fill the device, what the increment needs in either form is
// allocated first, and if the storage does not fit then the full form stays.
bool tangent_symmetric(Ctx* c, bool mg) {
  int dev = 0, l2 = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess || l2 <= 0) return false;
  const int64_t full = c->nnzb * 9 * 8;
  if (!c->full_coded || full < (mg ? 2 * (int64_t)l2 : (int64_t)l2 / 2)) return false;
  if (c->sval64) return true;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || (int64_t)total_b < 4 * full) return false;
  int st = UFC_STATUS_OK;
  if (!c->val64) st = dalloc(c, &c->val64, c->sell_blocks * 9);
  if (st == UFC_STATUS_OK && !c->dinv64) st = dalloc(c, &c->dinv64, c->n);
  if (st == UFC_STATUS_OK && mg && !c->z64) st = dalloc(c, &c->z64, c->n);
  if (st == UFC_STATUS_OK) st = ensure_vectors(c, UFC_PRECISION_FP64);
  if (st == UFC_STATUS_OK) st = alloc_symmetric(c, false);
  if (st == UFC_STATUS_OK) return true;
  free_symmetric(c);
  cudaGetLastError();
  c->err.clear();
  return false;
}

int pcg_solve(Ctx* c, const double* b, double* x, const ufc_solver_algo* algo, ufc_solver_state* st) {
  if (!c->has_pattern) return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: pattern not built");
  if (algo->method != UFC_SOLV_METHOD_CG) return fail(c, UFC_STATUS_UNSUPPORTED, "ufc_pcg_solve: method must be CG");
  if (algo->precond_type != UFC_SOLV_PREC_JACOBI && algo->precond_type != UFC_SOLV_PREC_NONE &&
      algo->precond_type != UFC_SOLV_PREC_MG)
    return fail(c, UFC_STATUS_UNSUPPORTED, "ufc_pcg_solve: preconditioner must be Jacobi, multigrid or none");
  const int prec = algo->precision_mode;
  if (prec == UFC_PRECISION_FP64 && !c->has_val64)
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: FP64 values not assembled (UFC_BUILD_FP64)");
  if (prec != UFC_PRECISION_FP64 && prec != UFC_PRECISION_FP32_REFINE && prec != UFC_PRECISION_FP32_MATRIX)
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: precision_mode");
  if (prec != UFC_PRECISION_FP64 && !c->has_val32)
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: FP32 values not assembled (UFC_BUILD_FP32*)");
  if (prec != UFC_PRECISION_FP64 && c->mat_model != UFC_MAT_ELASTIC_ISO && !c->has_val64)
    return fail(c, UFC_STATUS_INVALID,
                "ufc_pcg_solve: refined FP32 solves of a non-elastic tangent need its FP64 values for the residual "
                "(UFC_BUILD_FP64 | UFC_BUILD_FP32_ROUNDED)");
  if (prec == UFC_PRECISION_FP32_MATRIX && algo->precond_type == UFC_SOLV_PREC_JACOBI && !c->has_val64)
    return fail(c, UFC_STATUS_INVALID, "ufc_pcg_solve: FP32_MATRIX takes its Jacobi diagonal from the FP64 values");
  UFC_TRY(ensure_vectors(c, prec));
  UFC_CUDA(c, cudaMemcpyAsync(c->b64, b, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream));
  if (algo->use_x0)
    UFC_CUDA(c, cudaMemcpyAsync(c->x64, x, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream));
  else
    UFC_CUDA(c, cudaMemsetAsync(c->x64, 0, sizeof(double) * c->n, c->stream));
  int s;
  if (algo->precond_type == UFC_SOLV_PREC_MG) {
    if (prec != UFC_PRECISION_FP64)
      return fail(c, UFC_STATUS_UNSUPPORTED, "ufc_pcg_solve: the multigrid preconditioner runs in FP64");
    s = pcg_mg(c, algo, st);
    if (s != UFC_STATUS_OK && s != UFC_STATUS_NOT_CONVERGED) return s;
    st->fp64_iters = 0;
    UFC_CUDA(c, cudaMemcpyAsync(x, c->x64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream));
    if (s == UFC_STATUS_NOT_CONVERGED) fail(c, UFC_STATUS_NOT_CONVERGED, "[NM_Solver_PCG]: did not converge");
    return s;
  }
  if (prec == UFC_PRECISION_FP32_REFINE && algo->refine_policy != UFC_REFINE_FORCE_FP32 && c->has_val64 &&
      fp64_fits_l2(c)) {
    // a matrix this small is read from L2 in either precision: FP64 iterations
    ufc_solver_algo a64 = *algo;
    a64.precision_mode = UFC_PRECISION_FP64;
    UFC_TRY(ensure_vectors(c, UFC_PRECISION_FP64));
    s = pcg_run<double, double, double>(c, &a64, st);
    if (s != UFC_STATUS_OK && s != UFC_STATUS_NOT_CONVERGED) return s;
    st->fp64_iters = st->niter;
    UFC_CUDA(c, cudaMemcpyAsync(x, c->x64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream));
    if (s == UFC_STATUS_NOT_CONVERGED) fail(c, UFC_STATUS_NOT_CONVERGED, "[NM_Solver_PCG]: did not converge");
    return s;
  }
  if (prec == UFC_PRECISION_FP64)
    s = pcg_run<double, double, double>(c, algo, st);
  else if (prec == UFC_PRECISION_FP32_MATRIX)
    s = pcg_run<float, double, double>(c, algo, st);
  else if (algo->accumulate == UFC_ACCUMULATE_FP64)
    s = pcg_run<float, float, double>(c, algo, st);
  else
    s = pcg_run<float, float, float>(c, algo, st);
  st->fp64_iters = 0;
  if (s == UFC_STATUS_NOT_CONVERGED && prec != UFC_PRECISION_FP64 && st->convergence_flag == 3 && c->has_val64 &&
      st->niter < algo->max_iter) {
    // Stall or divergence of the refined FP32 run (the FP32 matrix is too far
    // from K for this problem): finish in FP64 from the best FP32 iterate.
    ufc_solver_algo a64 = *algo;
    a64.precision_mode = UFC_PRECISION_FP64;
    a64.max_iter = algo->max_iter - st->niter;
    ufc_solver_state s64{};
    UFC_TRY(ensure_vectors(c, UFC_PRECISION_FP64));
    s = pcg_run<double, double, double>(c, &a64, &s64);
    if (s != UFC_STATUS_OK && s != UFC_STATUS_NOT_CONVERGED) return s;
    st->fp64_iters = s64.niter;
    st->niter += s64.niter;
    st->n_refine += s64.n_refine;
    st->converged = s64.converged;
    st->convergence_flag = s64.convergence_flag;
    st->rnorm = s64.rnorm;
    st->solve_time += s64.solve_time;
  }
  if (s != UFC_STATUS_OK && s != UFC_STATUS_NOT_CONVERGED) return s;
  UFC_CUDA(c, cudaMemcpyAsync(x, c->x64, sizeof(double) * c->n, cudaMemcpyDeviceToDevice, c->stream));
  if (s == UFC_STATUS_NOT_CONVERGED)
    fail(c, UFC_STATUS_NOT_CONVERGED, "[NM_Solver_PCG]: did not converge");
  return s;
}

}  // namespace ufc
