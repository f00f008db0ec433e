// Jacobi-preconditioned conjugate gradients on the owned COO Hessian, kept on
// the device for the Newton driver's linear solve (the reference hands the
// assembled matrix to PETSc: core/petsc/scalar_problem_driver.py:154-226 and
// hyperelasticity/jax_petsc/solver.py:257-330 call ksp.setOperators,
// ksp.setTolerances(rtol, max_it), ksp.solve and ksp.getIterationNumber).
//
// One CG iteration is two kernels and no host round trip:
//   spmv        p = z + beta p_old (lazily, per gathered entry), Ap = A p and
//               the block partials of p.Ap;
//   k_cg_update x += alpha p, r -= alpha Ap, z = D^-1 r and the partials of
//               r.z and r.r.
// Every block of a kernel first sums the partials its predecessor left, in the
// same fixed order, and so knows alpha (or beta and the stop flags) without any
// block waiting for a last one to publish it (the ticket, fence and single-block
// reduction at the end of each kernel were about 3 us).  One thread per block
// reads the 96-byte state and partials come through L1: read by every warp, that
// one line was 20,000 requests to one L2 slice.  Block 0 records the
// scalars in one of two states, spmv in `after_update`, the update in
// `after_spmv`, each read only by the other kernel.  A kernel whose state says
// stopped returns at once, so a CUDA graph of iterations can run past the
// stop; a one-block kernel at its end leaves the final state for the host.
// The kernels of a graph are launched programmatically (the next kernel's
// blocks start while the last ones of the previous kernel run, load what a solve
// does not change -- columns, values, the Jacobi scaling -- and then wait for its
// completion).  z and p_old of a row lie side by side, one 16-byte gather.
// Short rows (at most 16 entries, little padding: the triangle meshes) are
// stored column-major with one thread per row, coalesced and without shuffles;
// longer rows take G lanes per row on CSR.  Creation writes CSR on the host and
// turns it around on the device.
// Reductions use a fixed launch shape and a fixed order: the result of a solve
// is reproducible bit for bit.
//
// The stopping rules are those of the scalar CG restated in oracle/krylov.py:
// stop at the first iterate with ||r|| <= rtol ||b||, at p.Ap <= 0 (the last
// iterate, or b itself when it happens at the first iteration), or after
// max_it iterations; a zero right-hand side returns x = 0 after 0 iterations.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "fne_internal.h"

namespace fne {
namespace {

constexpr int kCgThreads = 256;

// Row batches per warp iteration of the SpMV for G lanes per row.
constexpr int spmv_unroll(int G) { return G <= 8 ? 4 : 2; }

struct alignas(16) CgState {
  double rz, alpha, beta, tol2, rtol2;
  int32_t first, stop, neg_first, its, it, maxit;
  int32_t reason;  // 0 converged, 1 non-positive curvature, 2 iteration limit, 3 zero right-hand side
  int32_t chunk;   // graphs run (its low bit: the host slot)
  double rr, rr0;  // ||r||^2 now and at the start
};
static_assert(sizeof(CgState) == 96, "the state's size is named above");

struct CgVecs {
  const int32_t* crow;  // CSR; with width > 0 col and vals hold column-major rows of `width` entries at stride `stride`, column -1 = none
  const int32_t* col;
  const void* vals;
  const double* dinv;
  double* x;
  double* r;
  double* Ap;
  double* p;
  double2* zp;       // {z, p_old} of every row
  double* part_s;    // [grid_spmv]
  double* part_u;    // [2 * grid_vec]
  CgState* after_spmv;
  CgState* after_update;
  int32_t n, width, stride, grid_spmv, grid_vec;
};

// The predecessor's results are visible after this; the successor may start.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Plain cached loads of what the predecessor wrote (never the read-only path: the block may have started before).
__device__ __forceinline__ double2 ld2(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld1(const double* p) {
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block sum of up to two values (fixed order); the result is valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double (&sm)[NV][kCgThreads / 32]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    v[j] = warp_sum(v[j]);
    if (lane == 0) sm[j][w] = v[j];
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      double t = lane < kCgThreads / 32 ? sm[j][lane] : 0.0;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      v[j] = t;
    }
  }
}

// The state `src` advanced by `step(state, totals)`, totals the sums of the
// predecessor's block partials: the same in every thread of every block.
template <int NV, typename Step>
__device__ CgState next_state(const CgState* src, const double* partial, int grid, Step step) {
  __shared__ double sm[NV][kCgThreads / 32];
  __shared__ CgState state;
  double t[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    t[j] = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < grid; b += kCgThreads) t[j] += ld1(partial + j * grid + b);
  }
  CgState s;
  if (threadIdx.x == 0) {
    const double2* from = reinterpret_cast<const double2*>(src);
    double2* to = reinterpret_cast<double2*>(&s);
    static_assert(sizeof(CgState) % 16 == 0, "loaded 16 bytes at a time");
#pragma unroll
    for (int i = 0; i < (int)(sizeof(CgState) / 16); ++i) to[i] = ld2(from + i);
  }
  block_sum<NV>(t, sm);
  if (threadIdx.x == 0) {
    if (!s.stop) step(s, t);
    state = s;
  }
  __syncthreads();
  return state;
}

template <int NV>
__device__ __forceinline__ void leave_partial(double (&v)[NV], double* partial) {
  __shared__ double sm[NV][kCgThreads / 32];
  __syncthreads();
  block_sum<NV>(v, sm);
  if (threadIdx.x == 0)
#pragma unroll
    for (int j = 0; j < NV; ++j) partial[j * gridDim.x + blockIdx.x] = v[j];
}

// State after an update (or the initialisation): beta, rz and the stopping rules.
__device__ __forceinline__ CgState state_after_update(const CgVecs& a) {
  return next_state<2>(a.after_spmv, a.part_u, a.grid_vec, [](CgState& s, const double (&v)[2]) {
    if (s.first) {
      s.first = 0;
      s.rz = v[0];
      s.tol2 = s.rtol2 * v[1];
      s.beta = 0.0;
      s.rr = s.rr0 = v[1];
      if (v[1] == 0.0) {
        s.stop = 1;
        s.reason = 3;
      }
    } else {
      s.beta = v[0] / s.rz;
      s.rz = v[0];
      s.rr = v[1];
      if (v[1] <= s.tol2) {
        s.stop = 1;
        s.reason = 0;
      }
    }
    if (!s.stop && s.it >= s.maxit) {
      s.stop = 1;
      s.reason = 2;
    }
  });
}

__global__ void __launch_bounds__(kCgThreads) k_cg_init(CgVecs a, const double* __restrict__ b, double rtol,
                                                        int maxit) {
  double v[2] = {0.0, 0.0};
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += stride) {
    const double bi = b[i];
    const double zi = a.dinv[i] * bi;
    a.r[i] = bi;
    a.zp[i] = make_double2(zi, 0.0);
    a.x[i] = 0.0;
    v[0] += bi * zi;
    v[1] += bi * bi;
  }
  leave_partial<2>(v, a.part_u);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    CgState s = {};
    s.rtol2 = rtol * rtol;
    s.first = 1;
    s.maxit = maxit;
    *a.after_spmv = s;
  }
}

// The host's copy of the state: what the next spmv would find.  The update before left the state to go on
// from in after_spmv, where only the graph count moves.
__global__ void __launch_bounds__(kCgThreads) k_cg_state(CgVecs a, CgState* host) {
  grid_wait();
  const CgState s = state_after_update(a);
  if (threadIdx.x == 0) {
    host[s.chunk & 1] = s;
    a.after_spmv->chunk = s.chunk + 1;
    __threadfence_system();
  }
}

// Column-major rows, one thread per row; the first row's columns and values are
// loaded before the wait.
template <typename VT, int W>
__global__ void __launch_bounds__(kCgThreads, W <= 8 ? 4 : 2) k_cg_spmv_rows(CgVecs a) {
  grid_release();
  const VT* __restrict__ vals = static_cast<const VT*>(a.vals);
  const int stride = gridDim.x * blockDim.x;
  int row = blockIdx.x * blockDim.x + threadIdx.x;
  int c[W];
  VT w[W];
  auto fetch = [&]() {
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const bool in = k < a.width && row < a.n;
      c[k] = in ? __ldg(a.col + (size_t)k * a.stride + row) : -1;
      w[k] = in ? __ldg(vals + (size_t)k * a.stride + row) : VT(0);
    }
  };
  fetch();
  grid_wait();
  const CgState s = state_after_update(a);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.after_update = s;
  if (s.stop) return;
  const double beta = s.beta;
  double v[1] = {0.0};
  while (row < a.n) {
    const double2 own = ld2(a.zp + row);
    double sum = 0.0;
    double2 g[W];
#pragma unroll
    for (int k = 0; k < W; ++k) g[k] = c[k] >= 0 ? ld2(a.zp + c[k]) : make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < W; ++k)
      if (c[k] >= 0) sum += (double)w[k] * (g[k].x + beta * g[k].y);
    const double p = own.x + beta * own.y;
    a.p[row] = p;
    a.Ap[row] = sum;
    v[0] += p * sum;
    row += stride;
    if (row < a.n) fetch();
  }
  leave_partial<1>(v, a.part_s);
}

// CSR with G lanes per row, U row batches per warp iteration (their index,
// column and gather loads are in flight together); VT the stored value type
// (FP32 values are widened on load).
template <int G, typename VT, int U>
__global__ void __launch_bounds__(kCgThreads) k_cg_spmv(CgVecs a) {
  grid_release();
  grid_wait();
  const CgState s = state_after_update(a);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.after_update = s;
  if (s.stop) return;
  const double beta = s.beta;
  const VT* __restrict__ vals = static_cast<const VT*>(a.vals);
  // Rows are taken RPW * U at a time by each warp; the loop bound is the
  // same for all lanes of a warp, so the shuffles below see the full warp.
  constexpr int RPW = 32 / G;
  const int lane = threadIdx.x & 31, sub = lane % G, rsub = lane / G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int n_warps = gridDim.x * (kCgThreads / 32);
  double v[1] = {0.0};
  for (int base = warp * RPW * U; base < a.n; base += n_warps * RPW * U) {
    int k0[U], k1[U];
    double2 own[U];
    double sum[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int row = base + u * RPW + rsub;
      const bool valid = row < a.n;
      k0[u] = valid ? __ldg(a.crow + row) : 0;
      k1[u] = valid ? __ldg(a.crow + row + 1) : 0;
      own[u] = valid && sub == 0 ? ld2(a.zp + row) : make_double2(0.0, 0.0);
    }
    int c[U];
    double w[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0[u] + sub;
      const bool ok = k < k1[u];
      c[u] = ok ? __ldg(a.col + k) : -1;
      w[u] = ok ? (double)vals[k] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 g = c[u] >= 0 ? ld2(a.zp + c[u]) : make_double2(0.0, 0.0);
      sum[u] = c[u] >= 0 ? w[u] * (g.x + beta * g.y) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      for (int k = k0[u] + sub + G; k < k1[u]; k += G) {
        const double2 g = ld2(a.zp + __ldg(a.col + k));
        sum[u] += (double)vals[k] * (g.x + beta * g.y);
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) sum[u] += __shfl_xor_sync(0xffffffffu, sum[u], o, G);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int row = base + u * RPW + rsub;
      if (row < a.n && sub == 0) {
        const double p = own[u].x + beta * own[u].y;
        a.p[row] = p;
        a.Ap[row] = sum[u];
        v[0] += p * sum[u];
      }
    }
  }
  leave_partial<1>(v, a.part_s);
}

__device__ __forceinline__ void cg_update_one(double alpha, double& x, double p, double& r, double ap, double d,
                                              double& z, double (&v)[2]) {
  x += alpha * p;
  r -= alpha * ap;
  z = d * r;
  v[0] += r * z;
  v[1] += r * r;
}

// Vectors are padded to a multiple of 32 entries, so every vector starts on a
// 256-byte boundary and is read and written as double2 (two rows a thread); an
// odd last entry is done by thread 0.
__global__ void __launch_bounds__(kCgThreads) k_cg_update(CgVecs a) {
  grid_release();
  const int n2 = a.n >> 1;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const double2* __restrict__ dv = reinterpret_cast<const double2*>(a.dinv);
  double2 d = tid < n2 ? __ldg(dv + tid) : make_double2(0.0, 0.0);
  grid_wait();
  const CgState s = next_state<1>(a.after_update, a.part_s, a.grid_spmv, [](CgState& q, const double (&t)[1]) {
    q.it += 1;
    q.its += 1;
    const bool curv = t[0] > 0.0;
    if (q.it == 1) q.neg_first = !curv;
    q.alpha = curv ? q.rz / t[0] : 0.0;
    if (!curv) {
      q.stop = 1;
      q.reason = 1;
    }
  });
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.after_spmv = s;
  if (s.stop) return;
  const double alpha = s.alpha;
  double2* x = reinterpret_cast<double2*>(a.x);
  double2* r = reinterpret_cast<double2*>(a.r);
  const double2* p = reinterpret_cast<const double2*>(a.p);
  const double2* ap = reinterpret_cast<const double2*>(a.Ap);
  double v[2] = {0.0, 0.0};
  for (int i = tid; i < n2; i += stride) {
    double2 xa = ld2(x + i), ra = ld2(r + i), za;
    const double2 pa = ld2(p + i), aa = ld2(ap + i);
    if (i != tid) d = __ldg(dv + i);
    cg_update_one(alpha, xa.x, pa.x, ra.x, aa.x, d.x, za.x, v);
    cg_update_one(alpha, xa.y, pa.y, ra.y, aa.y, d.y, za.y, v);
    x[i] = xa;
    r[i] = ra;
    a.zp[2 * i] = make_double2(za.x, pa.x);
    a.zp[2 * i + 1] = make_double2(za.y, pa.y);
  }
  if ((a.n & 1) && tid == 0) {
    const int i = a.n - 1;
    double z;
    cg_update_one(alpha, a.x[i], a.p[i], a.r[i], a.Ap[i], a.dinv[i], z, v);
    a.zp[i] = make_double2(z, a.p[i]);
  }
  leave_partial<2>(v, a.part_u);
}

// Stored values (CSR or column-major order) from the COO values, and the Jacobi scaling
// 1 / |a_ii| (1 where the diagonal is missing, zero or not a number).
template <typename VT>
__global__ void k_cg_values(int64_t nnz, int32_t n, const int32_t* __restrict__ order,
                            const int32_t* __restrict__ diag, const VT* __restrict__ coo, VT* __restrict__ vals,
                            double* __restrict__ dinv) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += stride) {
    const int32_t o = order[k];
    vals[k] = o >= 0 ? coo[o] : VT(0);  // -1: padding of column-major rows
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t d = diag[i];
    const double v = d >= 0 ? fabs((double)coo[d]) : 1.0;
    dinv[i] = 1.0 / (v > 0.0 ? v : 1.0);
  }
}

// Column-major rows from CSR: entry k of a row at k * stride, -1 beyond its end.
__global__ void k_cg_columns(int32_t n, int32_t stride, int32_t width, const int32_t* __restrict__ crow,
                             const int32_t* __restrict__ csr, int32_t* __restrict__ out) {
  const int32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= stride) return;
  const int32_t k0 = row < n ? crow[row] : 0, len = row < n ? crow[row + 1] - k0 : 0;
  for (int32_t k = 0; k < width; ++k) out[(size_t)k * stride + row] = k < len ? csr[k0 + k] : -1;
}

int cg_status(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return FNE_OK;
}

}  // namespace
}  // namespace fne

struct fne_cg {
  int32_t n = 0;
  int64_t nv = 0;  // vector stride: n rounded up to a multiple of 32
  int64_t nnz = 0;
  int group = 8;
  int vals_fp32 = 0;
  int chunk = 16;
  int grid_spmv = 1, grid_vec = 1;
  int width = 0;        // entries per row of the column-major form, 0: CSR
  int64_t n_vals = 0;   // stored values
  int32_t* crow = nullptr;  // with diag, partial and st in one allocation
  int32_t* col = nullptr;
  int32_t* order = nullptr;
  int32_t* diag = nullptr;
  void* vals = nullptr;
  double* dinv = nullptr;
  double* work = nullptr;  // x, r, Ap, p, {z, p_old}
  double* partial = nullptr;
  fne::CgState* st = nullptr;       // [2]: after spmv, after update
  fne::CgState* st_host = nullptr;  // [2]: of the last two chunks
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaEvent_t done = nullptr;       // end of the last solve's work (the caller may go on on another stream)
  cudaStream_t cap = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool have_matrix = false;
  int64_t launches = 0;             // kernels launched by the last solve
};

namespace {

using fne::set_error;

fne::CgVecs vecs_of(const fne_cg* c) {
  fne::CgVecs a;
  const size_t nv = (size_t)c->nv;
  a.crow = c->crow;
  a.col = c->col;
  a.vals = c->vals;
  a.dinv = c->dinv;
  a.x = c->work;
  a.r = c->work + nv;
  a.Ap = c->work + 2 * nv;
  a.p = c->work + 3 * nv;
  a.zp = reinterpret_cast<double2*>(c->work + 4 * nv);
  a.part_s = c->partial;
  a.part_u = c->partial + c->grid_spmv;
  a.after_spmv = c->st;
  a.after_update = c->st + 1;
  a.n = c->n;
  a.width = c->width;
  a.stride = (int32_t)c->nv;
  a.grid_spmv = c->grid_spmv;
  a.grid_vec = c->grid_vec;
  return a;
}

// Calls f with the spmv kernel of this pattern.
template <typename F>
auto with_spmv(const fne_cg* c, F&& f) {
  using K = void (*)(fne::CgVecs);
  K k = nullptr;
  if (c->width > 8)
    k = c->vals_fp32 ? (K)fne::k_cg_spmv_rows<float, 16> : (K)fne::k_cg_spmv_rows<double, 16>;
  else if (c->width > 0)
    k = c->vals_fp32 ? (K)fne::k_cg_spmv_rows<float, 8> : (K)fne::k_cg_spmv_rows<double, 8>;
#define FNE_CG_SPMV(G)                                                               \
  else if (c->group == G) k = c->vals_fp32 ? (K)fne::k_cg_spmv<G, float, fne::spmv_unroll(G)> \
                                           : (K)fne::k_cg_spmv<G, double, fne::spmv_unroll(G)>;
  FNE_CG_SPMV(4)
  FNE_CG_SPMV(8)
  FNE_CG_SPMV(16)
  FNE_CG_SPMV(32)
#undef FNE_CG_SPMV
  return f(k);
}

// A kernel that may start before its predecessor in the stream has finished (it waits for it itself).
cudaError_t launch_after(void (*k)(fne::CgVecs), int grid, const fne::CgVecs& a, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(fne::kCgThreads);
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, a);
}

int resident_spmv(const fne_cg* c) {
  return with_spmv(c, [](void (*k)(fne::CgVecs)) {
    int r = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k, fne::kCgThreads, 0);
    return r;
  });
}

void cg_free(fne_cg* c) {
  if (!c) return;
  if (c->done) cudaEventSynchronize(c->done);  // a solve may have left a graph that reads these buffers
  if (c->exec) cudaGraphExecDestroy(c->exec);
  if (c->cap) cudaStreamDestroy(c->cap);
  cudaFree(c->crow);
  cudaFree(c->col);
  cudaFree(c->order);
  cudaFree(c->vals);
  cudaFree(c->dinv);
  cudaFree(c->work);
  if (c->st_host) cudaFreeHost(c->st_host);
  for (cudaEvent_t e : {c->ev[0], c->ev[1], c->done})
    if (e) cudaEventDestroy(e);
  delete c;
}

int build_graph(fne_cg* c) {
  cudaGraph_t graph = nullptr;
  if (cudaStreamBeginCapture(c->cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
    return fne::cg_status("fne_cg_solve: begin capture");
  const fne::CgVecs a = vecs_of(c);
  cudaError_t le = cudaSuccess;
  for (int j = 0; j < c->chunk && le == cudaSuccess; ++j) {
    le = with_spmv(c, [&](void (*k)(fne::CgVecs)) { return launch_after(k, c->grid_spmv, a, c->cap); });
    if (le == cudaSuccess) le = launch_after(fne::k_cg_update, c->grid_vec, a, c->cap);
  }
  if (le == cudaSuccess) {
    fne::k_cg_state<<<1, fne::kCgThreads, 0, c->cap>>>(a, c->st_host);
    le = cudaGetLastError();
  }
  cudaError_t e = cudaStreamEndCapture(c->cap, &graph);
  if (le != cudaSuccess) {
    if (e == cudaSuccess && graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return set_error(FNE_ECUDA, std::string("fne_cg_solve: capture: ") + cudaGetErrorString(le));
  }
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("fne_cg_solve: capture: ") + cudaGetErrorString(e));
  e = cudaGraphInstantiate(&c->exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) {
    c->exec = nullptr;
    return set_error(FNE_ECUDA, std::string("fne_cg_solve: instantiate: ") + cudaGetErrorString(e));
  }
  return FNE_OK;
}

}  // namespace

extern "C" int fne_cg_create(int32_t n, int64_t nnz, const int64_t* rows, const int64_t* cols, int32_t vals_fp32,
                             int32_t chunk, fne_cg** out) {
  if (!out || n < 0 || nnz < 0 || (nnz > 0 && (!rows || !cols)) || nnz > INT32_MAX || chunk < 1 || chunk > 4096)
    return set_error(FNE_EINVAL, "fne_cg_create: bad arguments");
  *out = nullptr;
  std::vector<int32_t> crow((size_t)n + 1, 0);
  for (int64_t k = 0; k < nnz; ++k) {
    if (rows[k] < 0 || rows[k] >= n || cols[k] < 0 || cols[k] >= n)
      return set_error(FNE_EBOUNDS, "fne_cg_create: COO entry " + std::to_string(k) + " outside the n x n block");
    ++crow[(size_t)rows[k] + 1];
  }
  for (int32_t i = 0; i < n; ++i) crow[i + 1] += crow[i];
  int32_t longest = 0;
  for (int32_t i = 0; i < n; ++i) longest = std::max(longest, crow[i + 1] - crow[i]);
  fne_cg* c = new (std::nothrow) fne_cg();
  if (!c) return set_error(FNE_EINVAL, "fne_cg_create: out of host memory");
  c->n = n;
  c->nv = ((int64_t)n + 31) / 32 * 32;
  c->nnz = nnz;
  c->vals_fp32 = vals_fp32 ? 1 : 0;
  c->chunk = chunk;
  const double avg = n > 0 ? (double)nnz / n : 0.0;
  c->group = avg <= 6.0 ? 4 : avg <= 12.0 ? 8 : avg <= 24.0 ? 16 : 32;
  // column-major rows while they are short and padding stays within a quarter
  if (longest > 0 && longest <= 16 && c->nv * longest <= nnz + nnz / 4 + 4096) c->width = longest;
  c->n_vals = c->width ? c->nv * c->width : nnz;
  // CSR on the host, written in the order of the rows; a scatter into column-major rows here would take twice as long
  // as all of this (k_cg_columns does it on the device).  The arrays need no initial values.
  std::unique_ptr<int32_t[]> col(new (std::nothrow) int32_t[(size_t)nnz]), order(new (std::nothrow) int32_t[(size_t)nnz]),
      diag(new (std::nothrow) int32_t[(size_t)n]);
  if (!col || !order || !diag) {
    cg_free(c);
    return set_error(FNE_EINVAL, "fne_cg_create: out of host memory");
  }
  std::fill_n(diag.get(), n, -1);
  std::vector<int32_t> fill(crow.begin(), crow.end() - 1);
  for (int64_t k = 0; k < nnz; ++k) {  // stable: COO order within a row
    const int32_t pos = fill[(size_t)rows[k]]++;
    order[pos] = (int32_t)k;
    col[pos] = (int32_t)cols[k];
    if (rows[k] == cols[k]) diag[rows[k]] = (int32_t)k;
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // One full wave: SMs x resident blocks of each kernel (grid-stride loops).
  const int per_sm_spmv = std::max(1, resident_spmv(c));
  int per_sm_vec = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_vec, fne::k_cg_update, fne::kCgThreads, 0);
  per_sm_vec = std::max(1, per_sm_vec);
  const int64_t want_spmv = ((int64_t)n * (c->width ? 1 : c->group) + fne::kCgThreads - 1) / fne::kCgThreads;
  const int64_t want_vec = ((int64_t)(n + 1) / 2 + fne::kCgThreads - 1) / fne::kCgThreads;
  c->grid_spmv = (int)std::max<int64_t>(1, std::min<int64_t>(want_spmv, (int64_t)sms * per_sm_spmv));
  c->grid_vec = (int)std::max<int64_t>(1, std::min<int64_t>(want_vec, (int64_t)sms * per_sm_vec));
  const size_t vsz = c->vals_fp32 ? sizeof(float) : sizeof(double);
  auto up = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
  const size_t o_diag = up(((size_t)n + 1) * sizeof(int32_t)), o_part = o_diag + up((size_t)n * sizeof(int32_t));
  const size_t o_st = o_part + up(((size_t)c->grid_spmv + 2 * (size_t)c->grid_vec) * sizeof(double));
  char* base = nullptr;
  bool ok = cudaMalloc(&base, o_st + 2 * sizeof(fne::CgState)) == cudaSuccess &&
            cudaMalloc(&c->col, std::max<size_t>(1, (size_t)c->n_vals) * sizeof(int32_t)) == cudaSuccess &&
            cudaMalloc(&c->order, std::max<size_t>(1, (size_t)c->n_vals) * sizeof(int32_t)) == cudaSuccess &&
            cudaMalloc(&c->vals, std::max<size_t>(1, (size_t)c->n_vals) * vsz) == cudaSuccess &&
            cudaMalloc(&c->dinv, std::max<size_t>(32, (size_t)c->nv) * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&c->work, std::max<size_t>(32, 6 * (size_t)c->nv) * sizeof(double)) == cudaSuccess &&
            cudaHostAlloc(&c->st_host, 2 * sizeof(fne::CgState), cudaHostAllocDefault) == cudaSuccess &&
            cudaEventCreateWithFlags(&c->ev[0], cudaEventDisableTiming) == cudaSuccess &&
            cudaEventCreateWithFlags(&c->ev[1], cudaEventDisableTiming) == cudaSuccess &&
            cudaEventCreateWithFlags(&c->done, cudaEventDisableTiming) == cudaSuccess &&
            cudaStreamCreateWithFlags(&c->cap, cudaStreamNonBlocking) == cudaSuccess;
  c->crow = reinterpret_cast<int32_t*>(base);
  if (base) {
    c->diag = reinterpret_cast<int32_t*>(base + o_diag);
    c->partial = reinterpret_cast<double*>(base + o_part);
    c->st = reinterpret_cast<fne::CgState*>(base + o_st);
  }
  auto put = [&](void* dst, const int32_t* src, size_t count) {
    ok = ok && (count == 0 || cudaMemcpy(dst, src, count * sizeof(int32_t), cudaMemcpyHostToDevice) == cudaSuccess);
  };
  put(c->crow, crow.data(), crow.size());
  put(c->diag, diag.get(), (size_t)n);
  for (auto [dst, src] : {std::pair(c->col, col.get()), std::pair(c->order, order.get())}) {
    // (the values' place, at least as long, is free until fne_cg_set_matrix)
    put(c->width ? c->vals : dst, src, (size_t)nnz);
    if (ok && c->width) {
      fne::k_cg_columns<<<(int)((c->nv + 255) / 256), 256>>>(n, (int32_t)c->nv, c->width, c->crow,
                                                           static_cast<const int32_t*>(c->vals), dst);
      ok = cudaGetLastError() == cudaSuccess;
    }
  }
  ok = ok && cudaMemset(c->st, 0, 2 * sizeof(fne::CgState)) == cudaSuccess;
  ok = ok && cudaStreamSynchronize(0) == cudaSuccess;  // (a solve may use a stream that does not wait for this one)
  if (!ok) {
    cudaGetLastError();
    cg_free(c);
    return set_error(FNE_ECUDA, "fne_cg_create: device allocation or copy failed");
  }
  *out = c;
  return FNE_OK;
}

extern "C" int fne_cg_set_matrix(fne_cg* c, const void* coo_vals, void* stream) {
  if (!c || (c->nnz > 0 && !coo_vals)) return set_error(FNE_EINVAL, "fne_cg_set_matrix: bad arguments");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // after a solve on another stream (a stream under capture keeps to its own order)
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone)
    cudaStreamWaitEvent(s, c->done, 0);
  const int64_t work = std::max<int64_t>(c->n_vals, c->n);
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((work + 255) / 256, 148 * 16));
  if (c->vals_fp32)
    fne::k_cg_values<float><<<grid, 256, 0, s>>>(c->n_vals, c->n, c->order, c->diag, static_cast<const float*>(coo_vals),
                                                 static_cast<float*>(c->vals), c->dinv);
  else
    fne::k_cg_values<double><<<grid, 256, 0, s>>>(c->n_vals, c->n, c->order, c->diag,
                                                  static_cast<const double*>(coo_vals), static_cast<double*>(c->vals),
                                                  c->dinv);
  const int rc = fne::cg_status("fne_cg_set_matrix");
  if (rc == FNE_OK) c->have_matrix = true;
  return rc;
}

namespace {

// The work of fne_cg_solve; everything it leaves in `s` is behind it there.
int cg_run(fne_cg* c, const double* b, double* x, double rtol, int32_t maxit, int32_t* its, int32_t* reason,
           cudaStream_t s) {
  const fne::CgVecs a = vecs_of(c);
  fne::k_cg_init<<<c->grid_vec, fne::kCgThreads, 0, s>>>(a, b, rtol, maxit);
  int rc = fne::cg_status("fne_cg_solve: init");
  if (rc != FNE_OK) return rc;
  c->launches = 1;
  // Graphs of `chunk` iterations run until one reports the stop.  The next is
  // put into the stream before the host has read the state of the one before
  // wherever the residual's mean rate says that it will be needed: a gap of some
  // 15 us on the device is avoided, and a solve about to stop is not followed by
  // a graph of kernels that only return.
  const fne::CgState* h = nullptr;
  auto run_chunk = [&](int i) {
    if (cudaGraphLaunch(c->exec, s) != cudaSuccess || cudaEventRecord(c->ev[i & 1], s) != cudaSuccess)
      return fne::cg_status("fne_cg_solve: graph launch");
    c->launches += 2 * c->chunk + 1;
    return (int)FNE_OK;
  };
  if ((rc = run_chunk(0))) return rc;
  int launched = 1;
  for (int i = 0;; ++i) {
    if (cudaEventSynchronize(c->ev[i & 1]) != cudaSuccess) {
      rc = fne::cg_status("fne_cg_solve: state read");
      return rc != FNE_OK ? rc : set_error(FNE_ECUDA, "fne_cg_solve: state read");
    }
    h = c->st_host + (i & 1);
    if (h->stop) break;
    if (launched == i + 1 && (rc = run_chunk(launched++))) return rc;
    // iterations still to go at the mean rate so far (rtol = 0 or no decrease yet: without end; a residual that is
    // not a finite number: none, the next iteration may stop)
    const double rate = std::log(h->rr / h->rr0) / h->it;
    const double left = rate < 0.0 ? std::log(h->tol2 / h->rr) / rate : std::isfinite(rate) ? 1e9 : 0.0;
    const bool more = left > c->chunk && h->it + c->chunk < h->maxit;
    if (more && launched == i + 2 && (rc = run_chunk(launched++))) return rc;
  }
  const double* src = h->neg_first ? b : a.x;
  if (c->n > 0 && cudaMemcpyAsync(x, src, (size_t)c->n * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return fne::cg_status("fne_cg_solve: result copy");
  if (its) *its = h->neg_first ? 1 : h->its;
  if (reason) *reason = h->reason;
  return FNE_OK;
}

}  // namespace

extern "C" int fne_cg_solve(fne_cg* c, const double* b, double* x, double rtol, int32_t maxit, int32_t* its,
                            int32_t* reason, void* stream) {
  if (!c || (c->n > 0 && (!b || !x)) || maxit < 0 || !(rtol >= 0.0))
    return set_error(FNE_EINVAL, "fne_cg_solve: bad arguments");
  if (!c->have_matrix) return set_error(FNE_EINVAL, "fne_cg_solve: fne_cg_set_matrix was not called");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) {
    cudaGetLastError();  // (nor may `done` become an event of a capture)
    return set_error(FNE_ECUDA, "fne_cg_solve: the stream is being captured, and the host drives a solve");
  }
  if (!c->exec) {
    const int rc = build_graph(c);
    if (rc != FNE_OK) return rc;
  }
  if (cudaStreamWaitEvent(s, c->done, 0) != cudaSuccess) return fne::cg_status("fne_cg_solve: stream order");
  c->launches = 0;
  const int rc = cg_run(c, b, x, rtol, maxit, its, reason, s);
  // also after a failure: graphs launched before it may still run
  if (cudaEventRecord(c->done, s) != cudaSuccess && rc == FNE_OK) return fne::cg_status("fne_cg_solve: stream order");
  return rc;
}

extern "C" int fne_cg_launches(const fne_cg* c, int64_t* launches) {
  if (!c || !launches) return set_error(FNE_EINVAL, "fne_cg_launches: bad arguments");
  *launches = c->launches;
  return FNE_OK;
}

extern "C" const char* fne_cg_kernels(const fne_cg* c) {
  return !c ? "" : c->width ? "k_cg_spmv_rows+k_cg_update" : "k_cg_spmv+k_cg_update";
}

extern "C" int fne_cg_destroy(fne_cg* c) {
  cg_free(c);
  return FNE_OK;
}
