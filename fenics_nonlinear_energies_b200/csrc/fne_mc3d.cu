// 3-D Mohr-Coulomb slope family (P1 / P2 / P4 tetrahedra, 3 DOFs per node):
// element energy, gradient and constitutive Hessian on the GPU, scattered
// into the owned gradient and COO values.
//
// Replaces the element kernels of SlopeStability3DReorderedElementAssembler
// (src/problems/slope_stability_3d/jax_petsc/reordered_element_assembler.py:
// 189-206, 377-560): the density of src/problems/slope_stability_3d/jax/
// jax_energy_3d.py:38-191, its stress, and the element Hessian
// K_e = sum_q w_q B_q^T D_q B_q of constitutive_element_hessian_3d
// (jax_energy_3d.py:262-357), where the reference differentiates through
// eigvalsh with JAX and here the hand-written spectral derivatives of
// fne_mc3d_point.cuh are used.  Inputs are the reference's per-element,
// per-quadrature-point arrays: dphix / dphiy / dphiz (E, nq, n_p),
// quad_weight and the material fields c_bar_q, sin_phi_q, shear_q, bulk_q,
// lame_q (E, nq).
//
// k_mc3d_elem (P1 / P2): a CTA of 128 threads takes a tile of 128 / nq elements.
// One thread per (element, quadrature point) forms the strain and runs the
// constitutive point function (FP64: eigen-decomposition by cyclic Jacobi,
// branch potentials, spectral tangent) and stores w sigma and the upper triangle
// of w D in shared memory.  Then one lane per node b of an element forms
// (w D) B(b) and its products with B(a) in registers, every unordered pair of
// nodes once, and its three gradient entries.  k_mc3d_elem_hi (P4) contracts one
// node at a time.  Blocks and gradients go to per-element buffers, which
// k_mc3d_gather sums by pairs of row nodes into the COO values and the gradient
// (contributions in element order, no atomics).  FP32 mode keeps the point
// function in FP64 and runs the contraction, the buffers and the Hessian output
// in FP32.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "fne_gather.cuh"
#include "fne_internal.h"
#include "fne_mc3d_point.cuh"

namespace fne {

namespace {

constexpr int kM3Warps = 4;      // warps per CTA
constexpr int kM3MaxQ = 16;      // quadrature points per element (kernel limit)
constexpr int kM3Pt = 6;         // per-point inputs: w, c_bar, sin_phi, shear, bulk, lame

struct Mc3dArgs {
  int n_el;                        // local elements
  int nq;
  const int* __restrict__ codes;   // [n_el][3 NP] gather codes
  const double* __restrict__ grad; // [n_el][3][nq][NP] physical basis gradients
  const double* __restrict__ pt;   // [n_el][nq][6] per-point inputs
  const unsigned char* __restrict__ wflag;
  const double* __restrict__ u;
  const double* __restrict__ dir;
  const double* __restrict__ rhs;  // [n_owned] or null
  int n_owned;
  long long lo;
  double tiny;
  int elastic;
  double* partials;
  unsigned* counter;
  double* energy;
};

__device__ __forceinline__ double m3_block_sum(double v, double* ws) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) ws[wid] = v;
  __syncthreads();
  v = 0.0;
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// per-CTA partial, then the last CTA to finish sums the partials in index
// order (deterministic, no spin-waits)
__device__ void m3_energy_finalize(double v, const Mc3dArgs& A) {
  __shared__ double ws[32];
  __shared__ int is_last;
  v = m3_block_sum(v, ws);
  if (threadIdx.x == 0) {
    A.partials[blockIdx.x] = v;
    __threadfence();
    is_last = atomicAdd(A.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  double s = 0.0;
  for (int j = threadIdx.x; j < (int)gridDim.x; j += blockDim.x) s += __ldcg(A.partials + j);
  s = m3_block_sum(s, ws);
  if (threadIdx.x == 0) {
    A.energy[0] = s;
    *A.counter = 0u;
  }
}

// linear elastic point: psi = lame/2 I1^2 + mu Q (the reference's elastic mode)
__device__ __forceinline__ void m3_elastic(const double e[6], double mu, double lame, double& psi, double sig[6],
                                           double D[6][6]) {
  const double I1 = e[0] + e[1] + e[2];
  psi = 0.5 * lame * I1 * I1 + mu * (e[0] * e[0] + e[1] * e[1] + e[2] * e[2] +
                                     0.5 * (e[3] * e[3] + e[4] * e[4] + e[5] * e[5]));
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) D[i][j] = 0.0;
  for (int i = 0; i < 3; ++i) {
    sig[i] = lame * I1 + 2.0 * mu * e[i];
    sig[3 + i] = mu * e[3 + i];
    for (int j = 0; j < 3; ++j) D[i][j] = lame + (i == j ? 2.0 * mu : 0.0);
    D[3 + i][3 + i] = mu;
  }
}

// strain-vector component of DOF (node a, component c): the gradient entry
// on each of the six strain rows (xx, yy, zz, xy, yz, xz)
template <typename Real>
__device__ __forceinline__ void m3_bcol(Real gx, Real gy, Real gz, int c, Real b[6]) {
  b[0] = c == 0 ? gx : Real(0);
  b[1] = c == 1 ? gy : Real(0);
  b[2] = c == 2 ? gz : Real(0);
  b[3] = c == 0 ? gy : (c == 1 ? gx : Real(0));
  b[4] = c == 1 ? gz : (c == 2 ? gy : Real(0));
  b[5] = c == 0 ? gz : (c == 2 ? gx : Real(0));
}

// One quadrature point (FP64): strain from the nodal values, the point
// function, w sigma and the upper triangle of w D to shared memory; returns
// w psi.  Not inlined, so every instantiation of the element kernel runs the
// same machine code here and the separate energy / gradient / Hessian passes
// reproduce the fused pass bit for bit.
// ``gq``: the point's row of the element's basis gradients, gx at gq[a], gy and
// gz nq * NP and 2 nq * NP behind it (shared or global memory).
template <typename Real, int NP>
__device__ __noinline__ double m3_point_update(const double* gq, const int* __restrict__ codes,
                                               const double* __restrict__ u, const double* __restrict__ dir,
                                               const double* __restrict__ pt, int el, int q, int nq, double tiny,
                                               int elastic, Real* sig_out, Real* D_out) {
  const int* cd = codes + (long long)el * 3 * NP;
  double e[6] = {0, 0, 0, 0, 0, 0};
  for (int a = 0; a < NP; ++a) {
    double uc[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int code = __ldg(cd + 3 * a + c);
      uc[c] = code >= 0 ? __ldg(u + code) : __ldg(dir + (-1 - code));
    }
    const double gx = gq[a], gy = gq[nq * NP + a], gz = gq[2 * nq * NP + a];
    e[0] += gx * uc[0];
    e[1] += gy * uc[1];
    e[2] += gz * uc[2];
    e[3] += gy * uc[0] + gx * uc[1];
    e[4] += gz * uc[1] + gy * uc[2];
    e[5] += gz * uc[0] + gx * uc[2];
  }
  const double* m = pt + ((long long)el * nq + q) * kM3Pt;
  const double w = __ldg(m);
  double psi, sig[6], D[6][6];
  if (elastic)
    m3_elastic(e, __ldg(m + 3), __ldg(m + 5), psi, sig, D);
  else
    mc3d::point(e, __ldg(m + 1), __ldg(m + 2), __ldg(m + 3), __ldg(m + 4), __ldg(m + 5), tiny, psi, sig, D);
#pragma unroll
  for (int i = 0; i < 6; ++i) sig_out[i] = (Real)(w * sig[i]);
  int t = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = i; j < 6; ++j) D_out[t++] = (Real)(w * D[i][j]);
  return w * psi;
}

// Order of the node-pair blocks of an element in kbuf, and how the block of the
// ordered pair (a, b) is read from it.
//   P1 / P2: pair {b, (b + s) mod NP} at s * NP + b, s = 0 .. NP / 2 (the last
//     distance only for b < NP / 2), holding B(b + s)^T (w D) B(b): the blocks
//     one lane per node forms, in the order the lanes write them;
//   P4: a <= b, row-major upper triangle, holding B(a)^T (w D) B(b).
template <int NP>
__host__ __device__ inline int m3_block(int a, int b, bool& transposed) {
  if constexpr (NP > 10) {
    transposed = a > b;
    const int lo = transposed ? b : a, hi = transposed ? a : b;
    return lo * NP - lo * (lo - 1) / 2 + (hi - lo);
  } else {
    const int s = a >= b ? a - b : a - b + NP;  // distance from b up to a
    transposed = 2 * s > NP || (2 * s == NP && b >= NP / 2);
    return transposed ? (s ? NP - s : 0) * NP + a : s * NP + b;
  }
}

// Tile of k_mc3d_elem in dynamic shared memory.
template <typename Real, int NP>
struct M3Tile {
  static constexpr int NT = 32 * kM3Warps, DS = 22;  // points; values of w D per point, padded to pairs
  Real D[NT][DS];                                    // w D, upper triangle row-major
  Real sig[NT][6];                                   // w sigma
  Real out[kM3Warps][32 * 9];                        // one block per lane on its way to kbuf
  // then: double g[elements of the tile][3][nq][NP], basis gradients
  static size_t bytes(int nq) { return sizeof(M3Tile) + (size_t)(NT / nq) * 3 * nq * NP * sizeof(double); }
};

// Contraction split: one lane per node b, 32 / NP elements a warp (three P2
// tets: 30 of 32 lanes, and the 11 elements of a tile in one round of the
// four warps).  Per point a lane forms T = (w D) B(b) in registers (54
// products from the 21 values every lane of the element reads alike) and adds
// B(a)^T T for the nodes a = b, b + 1, ... at distance up to NP / 2, three at
// a time, so each unordered pair is formed once.  Shared memory bounded the
// earlier split (lanes over pairs, 21 loads of T and B(a) per 27 products, and
// 72-byte blocks stored value by value: 607 us for 61,440 P2 tets, of which
// the FP64 units need 105); here a lane loads 20 values per 81 products, and
// blocks leave through shared memory in whole lines.
template <typename Real, int NP, int WANT>
__global__ void __launch_bounds__(32 * kM3Warps, 3) k_mc3d_elem(Mc3dArgs A, Real* __restrict__ kbuf,
                                                             Real* __restrict__ gbuf) {
  constexpr int N = 3 * NP, NPAIR = NP * (NP + 1) / 2, NT = 32 * kM3Warps;
  constexpr int EPW = 32 / NP, SP = 3;  // elements per warp; distances per pass
  using Tile = M3Tile<Real, NP>;
  using V2 = typename std::conditional<sizeof(Real) == 8, double2, float2>::type;
  extern __shared__ __align__(16) unsigned char m3_smem[];
  Tile& T_ = *reinterpret_cast<Tile*>(m3_smem);
  double* s_g = reinterpret_cast<double*>(m3_smem + sizeof(Tile));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = A.nq, epc = NT / nq;                // elements per tile: all their points in one pass
  const int gs = 3 * nq * NP;                        // basis gradients per element (even: NP is)
  double eacc = 0.0;
  for (int el0 = blockIdx.x * epc; el0 < A.n_el; el0 += gridDim.x * epc) {
    const int ne = min(epc, A.n_el - el0);
    {  // the tile's basis gradients, one contiguous run
      const double2* src = reinterpret_cast<const double2*>(A.grad + (long long)el0 * gs);
      double2* dst = reinterpret_cast<double2*>(s_g);
#pragma unroll 4
      for (int i = threadIdx.x; i < ne * gs / 2; i += NT) dst[i] = __ldg(src + i);
    }
    {  // the next tile's, into L2
      const int el1 = el0 + gridDim.x * epc, n1 = min(epc, A.n_el - el1);
      const char* p = reinterpret_cast<const char*>(A.grad + (long long)el1 * gs);
      for (int i = threadIdx.x * 128; i < n1 * gs * 8; i += NT * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p + i));
      const char* m = reinterpret_cast<const char*>(A.pt + (long long)el1 * nq * kM3Pt);
      for (int i = threadIdx.x * 128; i < n1 * nq * kM3Pt * 8; i += NT * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(m + i));
    }
    __syncthreads();
    // constitutive update, one thread per (element, quadrature point) of the
    // tile (FP64): strain from the nodal values, then the point function
    if ((int)threadIdx.x < ne * nq) {
      const int j = threadIdx.x / nq, q = threadIdx.x - j * nq, el = el0 + j;
      const double wpsi = m3_point_update<Real, NP>(s_g + j * gs + q * NP, A.codes, A.u, A.dir, A.pt, el, q, nq,
                                                    A.tiny, A.elastic, T_.sig[threadIdx.x], T_.D[threadIdx.x]);
      if ((WANT & 1) && __ldg(A.wflag + el)) eacc += wpsi;
    }
    __syncthreads();
    const int sub = lane / NP, b = lane - sub * NP;
    for (int j0 = warp * EPW; (WANT & 6) && j0 < ne; j0 += kM3Warps * EPW) {
      const int j = j0 + sub;
      const bool on = sub < EPW && j < ne;
      const int jj = on ? j : j0;  // idle lanes follow the first element and store nothing
      const double* gx_ = s_g + jj * gs;
      const double* gy_ = gx_ + nq * NP;
      const double* gz_ = gy_ + nq * NP;
      if (WANT & 2) {  // element gradient: node b's three components
        Real r0 = Real(0), r1 = Real(0), r2 = Real(0);
        for (int q = 0; q < nq; ++q) {
          const Real* sg = T_.sig[jj * nq + q];
          const Real gx = (Real)gx_[q * NP + b], gy = (Real)gy_[q * NP + b], gz = (Real)gz_[q * NP + b];
          r0 += gx * sg[0];
          r0 += gy * sg[3];
          r0 += gz * sg[5];
          r1 += gy * sg[1];
          r1 += gx * sg[3];
          r1 += gz * sg[4];
          r2 += gz * sg[2];
          r2 += gy * sg[4];
          r2 += gx * sg[5];
        }
        if (on) {
          Real* o = gbuf + (long long)(el0 + j) * N + 3 * b;
          o[0] = r0;
          o[1] = r1;
          o[2] = r2;
        }
      }
      if (WANT & 4) {
        for (int s0 = 0; s0 <= NP / 2; s0 += SP) {
          Real K[SP][9];
          int aa[SP];
#pragma unroll
          for (int s = 0; s < SP; ++s) {
            aa[s] = b + s0 + s < NP ? b + s0 + s : b + s0 + s - NP;
#pragma unroll
            for (int i = 0; i < 9; ++i) K[s][i] = Real(0);
          }
#pragma unroll 1
          for (int q = 0; q < nq; ++q) {
            Real d[Tile::DS];
            const V2* Dq = reinterpret_cast<const V2*>(T_.D[jj * nq + q]);
#pragma unroll
            for (int i = 0; i < 11; ++i) {
              const V2 v = Dq[i];
              d[2 * i] = v.x;
              d[2 * i + 1] = v.y;
            }
            const Real gx = (Real)gx_[q * NP + b], gy = (Real)gy_[q * NP + b], gz = (Real)gz_[q * NP + b];
            Real T[6][3];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
              Real Di[6];
#pragma unroll
              for (int k = 0; k < 6; ++k) {
                const int lo = i < k ? i : k, hi = i < k ? k : i;
                Di[k] = d[lo * 6 - lo * (lo - 1) / 2 + (hi - lo)];
              }
              T[i][0] = Di[0] * gx + Di[3] * gy + Di[5] * gz;
              T[i][1] = Di[1] * gy + Di[3] * gx + Di[4] * gz;
              T[i][2] = Di[2] * gz + Di[4] * gy + Di[5] * gx;
            }
#pragma unroll
            for (int s = 0; s < SP; ++s) {
              const Real ax = (Real)gx_[q * NP + aa[s]], ay = (Real)gy_[q * NP + aa[s]],
                         az = (Real)gz_[q * NP + aa[s]];
#pragma unroll
              for (int k = 0; k < 3; ++k) {
                K[s][k] += ax * T[0][k] + ay * T[3][k] + az * T[5][k];
                K[s][3 + k] += ay * T[1][k] + ax * T[3][k] + az * T[4][k];
                K[s][6 + k] += az * T[2][k] + ay * T[4][k] + ax * T[5][k];
              }
            }
          }
          // one distance at a time: the warp's blocks through shared memory, then per element the run of
          // blocks of that distance (NP of them, NP / 2 at the last) in whole lines
          Real* st = T_.out[warp];
#pragma unroll
          for (int s = 0; s < SP; ++s) {
            const int dist = s0 + s;
            if (2 * dist > NP) break;
            const int run = 9 * (2 * dist == NP ? NP / 2 : NP);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 9; ++i) st[lane * 9 + i] = K[s][i];
            __syncwarp();
#pragma unroll
            for (int e = 0; e < EPW; ++e)
              if (j0 + e < ne) {
                Real* o = kbuf + ((long long)(el0 + j0 + e) * NPAIR + dist * NP) * 9;
#pragma unroll
                for (int i = lane; i < 9 * NP; i += 32)
                  if (i < run) o[i] = st[e * 9 * NP + i];
              }
          }
        }
      }
    }
    __syncthreads();
  }
  if (WANT & 1) {
    if (A.rhs)  // load term -f.u of the owned DOFs
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n_owned; i += gridDim.x * blockDim.x)
        eacc -= A.rhs[i] * A.u[A.lo + i];
    m3_energy_finalize(eacc, A);
  }
}

// P4 tetrahedra (35 nodes, up to kM3MaxQHi points): the same point tiles;
// the contraction keeps one node b at a time, (w D) B(b) at every point of
// the element in shared memory, and lanes over the nodes a <= b accumulate
// B(a)^T (w D) B(b) over the points, reading the basis gradients of a from
// global memory (the 3 x nq x 35 gradient table of one element does not fit
// beside the point tiles).
constexpr int kM3MaxQHi = 32;

template <typename Real, int NP, int WANT>
__global__ void __launch_bounds__(32 * kM3Warps) k_mc3d_elem_hi(Mc3dArgs A, Real* __restrict__ kbuf,
                                                                Real* __restrict__ gbuf) {
  constexpr int N = 3 * NP, NPAIR = NP * (NP + 1) / 2, NT = 32 * kM3Warps;
  __shared__ Real s_sig[NT][6];
  __shared__ Real s_D[NT][21];
  __shared__ Real s_T[kM3Warps][kM3MaxQHi][18];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = A.nq, epc = NT / nq;
  double eacc = 0.0;
  for (int el0 = blockIdx.x * epc; el0 < A.n_el; el0 += gridDim.x * epc) {
    const int ne = min(epc, A.n_el - el0);
    if ((int)threadIdx.x < ne * nq) {
      const int j = threadIdx.x / nq, q = threadIdx.x - j * nq, el = el0 + j;
      const double wpsi = m3_point_update<Real, NP>(A.grad + (long long)el * 3 * nq * NP + q * NP, A.codes, A.u,
                                                    A.dir, A.pt, el, q, nq, A.tiny, A.elastic, s_sig[threadIdx.x],
                                                    s_D[threadIdx.x]);
      if ((WANT & 1) && __ldg(A.wflag + el)) eacc += wpsi;
    }
    __syncthreads();
    for (int j = warp; (WANT & 6) && j < ne; j += kM3Warps) {
      const int el = el0 + j;
      const Real(*sg)[6] = s_sig + j * nq;
      const Real(*sD)[21] = s_D + j * nq;
      const double* gx_ = A.grad + (long long)el * 3 * nq * NP;
      const double* gy_ = gx_ + nq * NP;
      const double* gz_ = gy_ + nq * NP;
      if (WANT & 2) {
        for (int i = lane; i < N; i += 32) {
          const int a = i / 3, c = i - 3 * a;
          Real s = Real(0);
          for (int q = 0; q < nq; ++q) {
            Real b[6];
            m3_bcol<Real>((Real)__ldg(gx_ + q * NP + a), (Real)__ldg(gy_ + q * NP + a), (Real)__ldg(gz_ + q * NP + a),
                          c, b);
#pragma unroll
            for (int k = 0; k < 6; ++k) s += b[k] * sg[q][k];
          }
          gbuf[(long long)el * N + i] = s;
        }
      }
      if (WANT & 4) {
        for (int b = 0; b < NP; ++b) {
          for (int q = lane; q < nq; q += 32) {
            const Real* Dq = sD[q];
            Real D[6][6];
            int t = 0;
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
              for (int k = i; k < 6; ++k) {
                D[i][k] = Dq[t];
                D[k][i] = Dq[t];
                ++t;
              }
            const Real gx = (Real)__ldg(gx_ + q * NP + b), gy = (Real)__ldg(gy_ + q * NP + b),
                       gz = (Real)__ldg(gz_ + q * NP + b);
            Real* T = s_T[warp][q];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
              T[i * 3 + 0] = D[i][0] * gx + D[i][3] * gy + D[i][5] * gz;
              T[i * 3 + 1] = D[i][1] * gy + D[i][3] * gx + D[i][4] * gz;
              T[i * 3 + 2] = D[i][2] * gz + D[i][4] * gy + D[i][5] * gx;
            }
          }
          __syncwarp();
          for (int a = lane; a <= b; a += 32) {
            Real K[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
              for (int d = 0; d < 3; ++d) K[c][d] = Real(0);
            for (int q = 0; q < nq; ++q) {
              const Real ax = (Real)__ldg(gx_ + q * NP + a), ay = (Real)__ldg(gy_ + q * NP + a),
                         az = (Real)__ldg(gz_ + q * NP + a);
              const Real* T = s_T[warp][q];
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                K[0][d] += ax * T[0 * 3 + d] + ay * T[3 * 3 + d] + az * T[5 * 3 + d];
                K[1][d] += ay * T[1 * 3 + d] + ax * T[3 * 3 + d] + az * T[4 * 3 + d];
                K[2][d] += az * T[2 * 3 + d] + ay * T[4 * 3 + d] + ax * T[5 * 3 + d];
              }
            }
            // pair (a, b), a <= b, in row-major upper-triangle order
            const int p = a * NP - a * (a - 1) / 2 + (b - a);
            Real* o = kbuf + ((long long)el * NPAIR + p) * 9;
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
              for (int d = 0; d < 3; ++d) o[c * 3 + d] = K[c][d];
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
  }
  if (WANT & 1) {
    if (A.rhs)  // load term -f.u of the owned DOFs
      for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < A.n_owned; i += gridDim.x * blockDim.x)
        eacc -= A.rhs[i] * A.u[A.lo + i];
    m3_energy_finalize(eacc, A);
  }
}

// One unordered pair of row nodes (A, B): the block (A, B) and, mirrored, the
// block (B, A) are the same sum over elements.
struct alignas(16) M3Pair {
  int start;      // contributions 5, 6, ... in the contribution array
  unsigned meta;  // contributions (bits 0-15), free components of B (16-18) and of A (19-21)
  unsigned off;   // column offset of B in the rows of A (bits 0-15), of A in the rows of B (16-31)
  int node_b;     // row node B whose rows get the mirrored block, -1: none (A itself, or not an owned row)
  int code[4];    // the first contributions: 2 * (block in kbuf) + transposed, element order; -1 beyond the last
};

// Sums the stored blocks into the COO values, and the element gradients into
// the owned gradient.  Nine lanes per pair of nodes: lane (c, d) adds its entry
// of every contributing element's block in element order and writes it to row
// (A, c) and, mirrored, to row (B, d); a warp takes three pairs twice.  The
// next pairs' records, with their first four contributions in them, are loaded
// while these are summed, so the blocks are the only loads waited for.  A block is read as 72 consecutive bytes by
// nine lanes, three or four lines a load instruction, and each is read once.
// (One warp per row node and one lane per block, as k_node_gather does for the
// other families, read every off-diagonal block twice, 470 MB from DRAM, with
// nine loads of 32 lines each: 234 us for 61,440 P2 tets.)  No atomics;
// bit-reproducible.
template <typename Real, typename HOut, bool WANT_G>
__global__ void __launch_bounds__(256) k_mc3d_gather(int n_pairs, const M3Pair* __restrict__ pairs,
                                                     const int* __restrict__ pair_a, NodeGatherArgs G,
                                                     const Real* __restrict__ kbuf, const Real* __restrict__ gbuf,
                                                     HOut* __restrict__ out, double* __restrict__ grad) {
  if (WANT_G)
    for (int A = blockIdx.x * blockDim.x + threadIdx.x; A < G.n_rnodes; A += gridDim.x * blockDim.x)
      rowgrad_node<Real, 3>(A, G.rn_inc, G.inc, G.rn_gpos, gbuf, G.rhs, grad);
  constexpr int U = 4;
  const int lane = threadIdx.x & 31, grp = lane / 9, ent = lane - 9 * grp;
  const int c = ent / 3, d = ent - 3 * c, ent_t = 3 * d + c;
  const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)((gridDim.x * blockDim.x) >> 5);
  if (grp == 3) return;  // no warp-wide operation below
  int4 rec[2], codes[2];
  int node_a[2];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + 3 * h + grp;
      const bool in = t >= 0 && t < n_pairs;
      rec[h] = in ? __ldg(reinterpret_cast<const int4*>(pairs + t)) : make_int4(0, 0, 0, -1);
      codes[h] = in ? __ldg(reinterpret_cast<const int4*>(pairs + t) + 1) : make_int4(-1, -1, -1, -1);
      node_a[h] = in ? __ldg(pair_a + t) : -1;
    }
  };
  // last pairs first: the blocks the element kernel wrote last are still in L2
  int t0 = (n_pairs - 1) / 6 * 6 - gw * 6;
  fetch(t0);
  for (; t0 >= 0; t0 -= nw * 6) {
    int4 pr[2];
    int row_a[2], row_b[2];
    Real v[2][4], acc[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      pr[h] = rec[h];
      const int code[4] = {codes[h].x, codes[h].y, codes[h].z, codes[h].w};
#pragma unroll
      for (int x = 0; x < 4; ++x)
        v[h][x] = code[x] >= 0 ? __ldg(kbuf + (long long)(code[x] >> 1) * 9 + ((code[x] & 1) ? ent_t : ent)) : Real(0);
      row_a[h] = node_a[h] >= 0 && (((unsigned)pr[h].y >> (16 + d)) & 1u) ? __ldg(G.rn_row + 3 * node_a[h] + c) : -1;
      row_b[h] = pr[h].w >= 0 && (((unsigned)pr[h].y >> (19 + c)) & 1u) ? __ldg(G.rn_row + 3 * pr[h].w + d) : -1;
    }
    fetch(t0 - nw * 6);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = pr[h].y & 0xFFFF;
      acc[h] = Real(0);
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (x < n) acc[h] += v[h][x];
      for (int j = 4; j < n; j += 6) {  // beyond the fourth: six at a time
        int cd[6];
        Real w[6];
#pragma unroll
        for (int x = 0; x < 6; ++x) cd[x] = j + x < n ? __ldg(G.con + pr[h].x + j + x - 4) : -1;
#pragma unroll
        for (int x = 0; x < 6; ++x)
          w[x] = cd[x] >= 0 ? __ldg(kbuf + (long long)(cd[x] >> 1) * 9 + ((cd[x] & 1) ? ent_t : ent)) : Real(0);
#pragma unroll
        for (int x = 0; x < 6; ++x)
          if (cd[x] >= 0) acc[h] += w[x];
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned meta = (unsigned)pr[h].y, off = (unsigned)pr[h].z, db = (meta >> 16) & 7u, da = (meta >> 19) & 7u;
      if (row_a[h] >= 0) out[row_a[h] + (int)(off & 0xFFFFu) + __popc(db & ((1u << d) - 1u))] = (HOut)acc[h];
      if (row_b[h] >= 0) out[row_b[h] + (int)(off >> 16) + __popc(da & ((1u << c) - 1u))] = (HOut)acc[h];
    }
  }
}

}  // namespace

struct Mc3dHandle {
  int precision = 0, hess_fp32 = 0, np = 0, nq = 0, n_local = 0, num_sms = 148;
  int64_t nnz = 0, lo = 0, hi = 0, n_free = 0, n_total = 0;
  double tiny = 1.0e-15;
  int elastic = 0;
  int *codes = nullptr;
  double *grad = nullptr, *pt = nullptr, *dir = nullptr, *rhs = nullptr, *partials = nullptr;
  unsigned char* wflag = nullptr;
  unsigned* counter = nullptr;
  void *kbuf = nullptr, *gbuf = nullptr;
  int grid_elem = 1, n_rnodes = 0;
  int *bp_rn_row = nullptr, *bp_rn_gpos = nullptr, *bp_rn_inc = nullptr, *bp_con = nullptr, *bp_inc = nullptr;
  M3Pair* pairs = nullptr;
  int *pair_a = nullptr, n_pairs = 0;
  int64_t device_bytes = 0, n_contrib = 0;
};

namespace {

template <typename T>
int m3_upload(Mc3dHandle* h, T** p, const T* src, size_t count) {
  *p = nullptr;
  if (count == 0) return FNE_OK;
  cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
  if (e != cudaSuccess) return set_error(FNE_ENOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  h->device_bytes += (int64_t)(count * sizeof(T));
  if (src) {
    e = cudaMemcpy(*p, src, count * sizeof(T), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("cudaMemcpy: ") + cudaGetErrorString(e));
  }
  return FNE_OK;
}

// Pairs of row nodes from the node-block plan: every block (A, B) with element
// contributions once, from the row node with the smaller index when both have
// owned rows.  Codes stay below 2^31: n_elem * pairs * 9 < 2^33 is checked by the
// caller.
int build_pairs(const BlockPlan& bp, int64_t n_el, int np, std::vector<M3Pair>& pairs, std::vector<int32_t>& pair_a,
                std::vector<int32_t>& con) {
  const int npair = np * (np + 1) / 2, n = bp.n_rnodes;
  // blocks with contributions by their column's row node, to find (B, A): those in column A give every row B its block
  std::vector<int32_t> col_ptr((size_t)n + 1, 0), col_blk, blk_row(bp.blk.size()), block_in_col((size_t)n, -1);
  for (int32_t k = 0; k < n; ++k)
    for (int32_t b = bp.rn_blk[k]; b < bp.rn_blk[k + 1]; ++b) {
      blk_row[b] = k;
      if (bp.blk_rn[b] >= 0 && (bp.blk[b] >> 19)) ++col_ptr[bp.blk_rn[b] + 1];
    }
  for (int32_t k = 0; k < n; ++k) col_ptr[k + 1] += col_ptr[k];
  col_blk.resize((size_t)col_ptr[n]);
  {
    std::vector<int32_t> at(col_ptr.begin(), col_ptr.end() - 1);
    for (int32_t b = 0; b < (int32_t)bp.blk.size(); ++b)
      if (bp.blk_rn[b] >= 0 && (bp.blk[b] >> 19)) col_blk[at[bp.blk_rn[b]]++] = b;
  }
  // element contributions come in both directions; a block without any (a pattern wider than the element graph,
  // which need not be symmetric) is a zero of its own
  const auto mirrored = [&](int32_t A, int32_t b) { return (bp.blk[b] >> 19) && bp.blk_rn[b] >= 0 && bp.blk_rn[b] < A; };
  // in the order of their first contributing element (pairs without one first): the blocks are then read as
  // they lie, once; in row-node order the vertices' and the edge nodes' pairs each swept the whole buffer
  std::vector<int32_t> place((size_t)n_el + 2, 0);
  const auto bucket = [&](int32_t b, int64_t first) { return (bp.blk[b] >> 19) ? bp.con[first] / (np * np) + 1 : 0; };
  for (int32_t A = 0; A < n; ++A) {
    int64_t at = bp.rn_con[A];
    for (int32_t b = bp.rn_blk[A]; b < bp.rn_blk[A + 1]; at += bp.blk[b++] >> 19)
      if (!mirrored(A, b)) ++place[bucket(b, at) + 1];
  }
  for (size_t k = 1; k < place.size(); ++k) place[k] += place[k - 1];
  pairs.resize((size_t)place.back());
  pair_a.resize((size_t)place.back());
  for (int32_t A = 0; A < n; ++A) {
    int64_t at = bp.rn_con[A];
    for (int32_t j = col_ptr[A]; j < col_ptr[A + 1]; ++j) block_in_col[blk_row[col_blk[j]]] = col_blk[j];
    for (int32_t b = bp.rn_blk[A]; b < bp.rn_blk[A + 1]; ++b) {
      const uint32_t w = bp.blk[b];
      const int32_t cnt = (int32_t)(w >> 19), B = bp.blk_rn[b];
      const int64_t c0 = at;
      at += cnt;
      if (mirrored(A, b)) continue;
      const int32_t to = place[bucket(b, c0)]++;
      pair_a[to] = A;
      M3Pair& p = pairs[to];
      for (int x = 0; x < 4; ++x) p.code[x] = -1;
      p.start = (int32_t)con.size();
      p.meta = (uint32_t)cnt | ((w >> 16) & 7u) << 16;
      p.off = w & 0xFFFFu;
      p.node_b = -1;
      if (cnt > 0 && B > A) {
        const int32_t m = block_in_col[B];  // of column A, or of an earlier one
        if (m < 0 || bp.blk_rn[m] != A || (int32_t)(bp.blk[m] >> 19) != cnt)
          return set_error(FNE_ELAYOUT, "Mohr-Coulomb 3-D: COO pattern is not symmetric over the owned rows");
        p.meta |= ((bp.blk[m] >> 16) & 7u) << 19;
        p.off |= (bp.blk[m] & 0xFFFFu) << 16;
        p.node_b = B;
      }
      for (int64_t k = c0; k < c0 + cnt; ++k) {
        const int el = bp.con[k] / (np * np), r = bp.con[k] - el * np * np, a = r / np, bb = r - a * np;
        bool tr = false;
        const int q = np == 35 ? m3_block<35>(a, bb, tr) : np == 10 ? m3_block<10>(a, bb, tr) : m3_block<4>(a, bb, tr);
        const int code = 2 * (el * npair + q) + (tr ? 1 : 0);
        if (k - c0 < 4)
          p.code[k - c0] = code;
        else
          con.push_back(code);
      }
    }
  }
  return FNE_OK;
}

// resident CTAs per SM of the fused pass (registers and shared memory); allows
// every instantiation of the P1 / P2 kernel its tile of shared memory
template <typename Real, int NP>
cudaError_t m3_prepare(int nq, int* per_sm) {
  const size_t bytes = M3Tile<Real, NP>::bytes(nq);
  cudaError_t e = cudaSuccess;
  auto allow = [&](auto* k) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  };
  allow(&k_mc3d_elem<Real, NP, 1>);
  allow(&k_mc3d_elem<Real, NP, 2>);
  allow(&k_mc3d_elem<Real, NP, 3>);
  allow(&k_mc3d_elem<Real, NP, 4>);
  allow(&k_mc3d_elem<Real, NP, 5>);
  allow(&k_mc3d_elem<Real, NP, 6>);
  allow(&k_mc3d_elem<Real, NP, 7>);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_mc3d_elem<Real, NP, 7>, 32 * kM3Warps, bytes);
  return e;
}
template <typename Real>
cudaError_t m3_ctas_per_sm(int np, int nq, int* per_sm) {
  if (np == 10) return m3_prepare<Real, 10>(nq, per_sm);
  if (np == 4) return m3_prepare<Real, 4>(nq, per_sm);
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_mc3d_elem_hi<Real, 35, 7>, 32 * kM3Warps, 0);
}

template <typename Real, typename HOut, int NP>
cudaError_t m3_launch(Mc3dHandle* h, int flags, const double* u, double* energy, double* grad, void* hess,
                      cudaStream_t st) {
  Mc3dArgs A{h->n_local, h->nq,    h->codes, h->grad,    h->pt,  h->wflag, u,
             h->dir,     h->rhs,   (int)(h->hi - h->lo), h->lo,  h->tiny,  h->elastic,
             h->partials, h->counter, energy};
  Real* kb = static_cast<Real*>(h->kbuf);
  Real* gb = static_cast<Real*>(h->gbuf);
  const dim3 grid(h->grid_elem), block(32 * kM3Warps);
#define M3_CASE(W)                                                    \
  case W:                                                             \
    if constexpr (NP > 10)                                            \
      k_mc3d_elem_hi<Real, NP, W><<<grid, block, 0, st>>>(A, kb, gb); \
    else                                                              \
      k_mc3d_elem<Real, NP, W><<<grid, block, M3Tile<Real, NP>::bytes(h->nq), st>>>(A, kb, gb); \
    break;
  switch (flags) {
    M3_CASE(1)
    M3_CASE(2)
    M3_CASE(3)
    M3_CASE(4)
    M3_CASE(5)
    M3_CASE(6)
    M3_CASE(7)
    default: return cudaErrorInvalidValue;
  }
#undef M3_CASE
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !(flags & 6) || h->n_rnodes == 0) return e;
  NodeGatherArgs G{};
  G.n_rnodes = h->n_rnodes;
  G.rn_row = h->bp_rn_row;
  G.rn_gpos = h->bp_rn_gpos;
  G.rn_inc = h->bp_rn_inc;
  G.con = h->bp_con;
  G.inc = h->bp_inc;
  G.rhs = h->rhs;
  HOut* H = static_cast<HOut*>(hess);
  if (flags & 4) {
    const int gg = std::max(1, std::min(h->num_sms * 16, (h->n_pairs + 47) / 48));
    if (flags & 2)
      k_mc3d_gather<Real, HOut, true><<<gg, 256, 0, st>>>(h->n_pairs, h->pairs, h->pair_a, G, kb, gb, H, grad);
    else
      k_mc3d_gather<Real, HOut, false><<<gg, 256, 0, st>>>(h->n_pairs, h->pairs, h->pair_a, G, kb, gb, H, grad);
  } else {
    const int gr = std::max(1, std::min(h->num_sms * 8, (h->n_rnodes + 255) / 256));
    k_rowgrad<Real, 3><<<gr, 256, 0, st>>>(h->n_rnodes, h->bp_rn_inc, h->bp_inc, h->bp_rn_gpos, gb, h->rhs, grad);
  }
  return cudaGetLastError();
}

template <typename Real, typename HOut>
cudaError_t m3_dispatch(Mc3dHandle* h, int flags, const double* u, double* energy, double* grad, void* hess,
                        cudaStream_t st) {
  if (h->np == 35) return m3_launch<Real, HOut, 35>(h, flags, u, energy, grad, hess, st);
  if (h->np == 10) return m3_launch<Real, HOut, 10>(h, flags, u, energy, grad, hess, st);
  return m3_launch<Real, HOut, 4>(h, flags, u, energy, grad, hess, st);
}

}  // namespace

void mc3d_destroy(Mc3dHandle* h) {
  if (!h) return;
  void* ptrs[] = {h->codes, h->grad, h->pt, h->dir, h->rhs, h->partials, h->wflag, h->counter, h->kbuf, h->gbuf,
                  h->bp_rn_row, h->bp_rn_gpos, h->bp_rn_inc, h->bp_con, h->bp_inc, h->pairs, h->pair_a};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  delete h;
}

int mc3d_create(const fne_desc* d, Mc3dHandle** out) {
  *out = nullptr;
  const int np = d->npe, nq = d->nq, n = 3 * np;
  if (d->block_size != 3) return set_error(FNE_EINVAL, "Mohr-Coulomb 3-D: block_size must be 3");
  if (np != 4 && np != 10 && np != 35)
    return set_error(FNE_EINVAL, "Mohr-Coulomb 3-D: P1 (4 nodes), P2 (10 nodes) or P4 (35 nodes) tetrahedra");
  if (nq < 1 || nq > (np == 35 ? kM3MaxQHi : kM3MaxQ))
    return set_error(FNE_EINVAL, "Mohr-Coulomb 3-D: 1 to 16 quadrature points (P1, P2) or 1 to 32 (P4)");
  if (d->n_elem > 0 && (!d->e0 || !d->e1 || !d->e2 || !d->e3))
    return set_error(FNE_EINVAL, "Mohr-Coulomb 3-D: missing basis gradients or per-point inputs");
  const int64_t E = d->n_elem, lo = d->lo, hi = d->hi;
  const int64_t* t2f = d->total_to_free_reord;
  const int npair = np * (np + 1) / 2;
  if (E * (int64_t)npair * 9 >= (int64_t)INT32_MAX * 4 || d->nnz >= (int64_t)INT32_MAX)
    return set_error(FNE_EBOUNDS, "Mohr-Coulomb 3-D: sizes beyond the supported indexing");
  std::vector<int32_t> codes;
  std::vector<double> grad, pt;
  std::vector<uint8_t> wflag;
  std::vector<int64_t> local;
  for (int64_t e = 0; e < E; ++e) {
    bool own = false;
    for (int i = 0; i < n; ++i) {
      const int64_t dof = d->elems[e * n + i];
      if (dof < 0 || dof >= d->n_total) return set_error(FNE_EBOUNDS, "Mohr-Coulomb 3-D: element DOF out of range");
      const int64_t r = t2f[dof];
      own |= r >= lo && r < hi;
    }
    if (!own) continue;
    local.push_back(e);
    for (int i = 0; i < n; ++i) {
      const int64_t dof = d->elems[e * n + i];
      if (dof + 1 >= (int64_t)INT32_MAX) return set_error(FNE_EBOUNDS, "Mohr-Coulomb 3-D: DOF id beyond int32");
      codes.push_back(t2f[dof] >= 0 ? (int32_t)t2f[dof] : (int32_t)(-1 - dof));
    }
    for (const double* g : {d->e0, d->e1, d->e2})
      grad.insert(grad.end(), g + e * nq * np, g + (e + 1) * nq * np);
    pt.insert(pt.end(), d->e3 + e * nq * kM3Pt, d->e3 + (e + 1) * nq * kM3Pt);
    const double w = d->energy_weights ? d->energy_weights[e] : 1.0;
    if (w != 0.0 && w != 1.0) return set_error(FNE_EINVAL, "Mohr-Coulomb 3-D: energy weights must be 0 or 1");
    wflag.push_back(w != 0.0 ? 1 : 0);
  }
  const int64_t nl = (int64_t)local.size();
  BlockPlan bp;
  {
    std::vector<int64_t> edofs((size_t)nl * n);
    for (int64_t le = 0; le < nl; ++le)
      for (int i = 0; i < n; ++i) edofs[(size_t)le * n + i] = d->elems[local[le] * n + i];
    const int rc = build_block_plan(nl, np, 3, edofs.data(), d, bp);
    if (rc) return rc;
  }
  auto* h = new (std::nothrow) Mc3dHandle();
  if (!h) return set_error(FNE_ENOMEM, "Mohr-Coulomb 3-D: out of host memory");
  h->precision = d->precision;
  h->hess_fp32 = d->precision == FNE_FP32 && d->hess_fp32;
  h->np = np;
  h->nq = nq;
  h->n_local = (int)nl;
  h->nnz = d->nnz;
  h->lo = lo;
  h->hi = hi;
  h->n_free = d->n_free;
  h->n_total = d->n_total;
  h->tiny = d->s[0] > 0.0 ? d->s[0] : 1.0e-15;
  h->elastic = d->s[5] != 0.0;
  h->n_rnodes = bp.n_rnodes;
  h->n_contrib = (int64_t)bp.con.size();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    mc3d_destroy(h);
    return set_error(FNE_ECUDA, "Mohr-Coulomb 3-D: device query");
  }
  // tiles of 128 / nq elements (all their points in one pass of the CTA);
  // one wave of resident CTAs, each striding over the tiles
  const int64_t epc = 32 * kM3Warps / nq;
  int per_sm = 0;
  const cudaError_t oe = d->precision == FNE_FP64 ? m3_ctas_per_sm<double>(h->np, nq, &per_sm)
                                                  : m3_ctas_per_sm<float>(h->np, nq, &per_sm);
  if (oe != cudaSuccess || per_sm < 1) {
    mc3d_destroy(h);
    return set_error(FNE_ECUDA, std::string("Mohr-Coulomb 3-D: occupancy: ") + cudaGetErrorString(oe));
  }
  h->grid_elem = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)h->num_sms * per_sm, (nl + epc - 1) / epc));
  const size_t rsz = d->precision == FNE_FP32 ? sizeof(float) : sizeof(double);
  int rc = FNE_OK;
#define M3_TRY(x)       \
  do {                  \
    rc = (x);           \
    if (rc) {           \
      mc3d_destroy(h);  \
      return rc;        \
    }                   \
  } while (0)
  M3_TRY(m3_upload(h, &h->codes, codes.data(), codes.size()));
  M3_TRY(m3_upload(h, &h->grad, grad.data(), grad.size()));
  M3_TRY(m3_upload(h, &h->pt, pt.data(), pt.size()));
  M3_TRY(m3_upload(h, &h->wflag, wflag.data(), wflag.size()));
  M3_TRY(m3_upload(h, &h->dir, d->dirichlet, (size_t)d->n_total));
  if (d->rhs_owned) M3_TRY(m3_upload(h, &h->rhs, d->rhs_owned, (size_t)(hi - lo)));
  M3_TRY(m3_upload(h, &h->partials, (const double*)nullptr, (size_t)h->grid_elem));
  M3_TRY(m3_upload(h, &h->counter, (const unsigned*)nullptr, 1));
  if (cudaMemset(h->counter, 0, sizeof(unsigned)) != cudaSuccess) {
    mc3d_destroy(h);
    return set_error(FNE_ECUDA, "Mohr-Coulomb 3-D: cudaMemset");
  }
  M3_TRY(m3_upload(h, &h->bp_rn_row, bp.rn_row.data(), bp.rn_row.size()));
  M3_TRY(m3_upload(h, &h->bp_rn_gpos, bp.rn_gpos.data(), bp.rn_gpos.size()));
  M3_TRY(m3_upload(h, &h->bp_rn_inc, bp.rn_inc.data(), bp.rn_inc.size()));
  std::vector<M3Pair> pairs;
  std::vector<int32_t> pair_a, con;
  M3_TRY(build_pairs(bp, nl, np, pairs, pair_a, con));
  h->n_pairs = (int)pairs.size();
  M3_TRY(m3_upload(h, &h->pairs, pairs.data(), pairs.size()));
  M3_TRY(m3_upload(h, &h->pair_a, pair_a.data(), pair_a.size()));
  M3_TRY(m3_upload(h, &h->bp_con, con.data(), con.size()));
  M3_TRY(m3_upload(h, &h->bp_inc, bp.inc.data(), bp.inc.size()));
  unsigned char* kb = nullptr;
  M3_TRY(m3_upload(h, &kb, (const unsigned char*)nullptr, std::max<size_t>(1, (size_t)nl * npair * 9 * rsz)));
  h->kbuf = kb;
  unsigned char* gb = nullptr;
  M3_TRY(m3_upload(h, &gb, (const unsigned char*)nullptr, std::max<size_t>(1, (size_t)nl * n * rsz)));
  h->gbuf = gb;
#undef M3_TRY
  *out = h;
  return FNE_OK;
}

int mc3d_eval(Mc3dHandle* h, const double* u, int flags, double* energy, double* grad, void* hess, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (h->precision == FNE_FP64)
    e = m3_dispatch<double, double>(h, flags, u, energy, grad, hess, st);
  else if (h->hess_fp32)
    e = m3_dispatch<float, float>(h, flags, u, energy, grad, hess, st);
  else
    e = m3_dispatch<float, double>(h, flags, u, energy, grad, hess, st);
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("fne_eval launch: ") + cudaGetErrorString(e));
  return FNE_OK;
}

int mc3d_set_dirichlet(Mc3dHandle* h, const double* dirichlet) {
  cudaError_t e = cudaMemcpy(h->dir, dirichlet, h->n_total * sizeof(double), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("fne_set_dirichlet: ") + cudaGetErrorString(e));
  return FNE_OK;
}

void mc3d_info(const Mc3dHandle* h, fne_info* info) {
  info->n_rows = h->hi - h->lo;
  info->nnz = h->nnz;
  info->n_elem = h->n_local;
  info->n_incidences = h->n_contrib;
  info->device_bytes = h->device_bytes;
  info->max_row_len = 0;
  info->kernel_variant = 11;
  info->row_lanes = 1;
}

const char* mc3d_kernels(const Mc3dHandle* h) {
  return h->np == 35 ? "k_mc3d_elem_hi+k_mc3d_gather" : "k_mc3d_elem+k_mc3d_gather";
}

}  // namespace fne
