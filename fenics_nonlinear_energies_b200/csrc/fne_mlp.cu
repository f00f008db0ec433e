// Kernels of the learned Newton warm start: a small MLP over nodal features
// (BF16 weights and activations, FP32 accumulation and master weights).
//
//  * k_gemm_tc: op(A)[M x K] * op(B)[K x N] on the 5th-generation tensor
//    cores (tcgen05.mma kind::f16, BF16 operands, FP32 accumulator in TMEM)
//    with the layer's elementwise work in its epilogue: bias + SiLU forward,
//    SiLU derivative + column sums backward, a plain C = A B + beta C for the
//    weight gradient and for fne_gemm_bf16.  Operands are addressed through
//    (row, col) strides, so one kernel covers the forward product H W^T, the
//    weight gradient dZ^T H and the input gradient dZ W without explicit
//    transposes.
//  * k_bias_act_fwd, k_act_bwd, k_colsum, k_adam, k_adam_set, k_cast_bf16:
//    the elementwise pieces on their own, and the optimiser.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "fne_internal.h"

namespace cg = cooperative_groups;

namespace fne {
namespace {

constexpr int kTcBM = 128;  // rows per tile of the forward and input-gradient products
constexpr long long kTcWaitLimit = 1LL << 22;

// status of the tensor-core GEMM: 1 once an MMA-completion wait gave up
__device__ int g_gemm_err = 0;

namespace tcg {

__device__ __forceinline__ uint32_t saddr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// shared-memory matrix descriptor: leading / stride byte offsets and swizzle (2, 4, 6: 128-, 64-, 32-byte lines).
// K-major: stride = 8 rows; M/N-major: leading = next block of lines, stride = 8 lines.
__device__ __forceinline__ uint64_t mat_desc(uint32_t a, uint32_t lbo, uint32_t sbo, uint32_t swizzle) {
  uint64_t d = (uint64_t)((a >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for sm_100
  d |= (uint64_t)swizzle << 61;
  return d;
}
// instruction descriptor: D f32, A / B bf16, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void arrive(uint32_t mbar) {
  asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}\n" ::"r"(mbar) : "memory");
}
// arrives once the thread's cp.async copies so far have landed
__device__ __forceinline__ void arrive_copies(uint32_t mbar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(mbar) : "memory");
}
// Polls until the phase completed; gives up after `limit` polls, or early once *stop is set (may be null).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, long long limit, const int* stop) {
  for (long long it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (stop && *reinterpret_cast<const volatile int*>(stop)) return false;
  }
  return false;
}

}  // namespace tcg

// ---------------------------------------------------------------------------
// k_gemm_tc.  A(m, k) = A[m * sam + k * sak]; B(k, n) = B[k * sbk + n * sbn].
//
// What bounds it: at the network's sizes (8192 x 256 x 256) a product is
// 1 GFLOP over 4 to 16 MB that stay in L2, so the MMAs are nearly free and the
// time is the latency of one tile: loads, a few MMA steps, epilogue.  Hence
//   * a ring of slices filled with cp.async by eight warps and multiplied by a
//     ninth (full / empty mbarriers, no block barrier in the loop), laid down
//     in the swizzled lines the MMA reads at full width: K-major for an operand
//     whose K direction is contiguous, M/N-major (transposed descriptor) for
//     one whose M/N direction is -- no operand is transposed by the threads;
//   * 128 x 64 tiles below 148 tiles of 128 x 128, so that two CTAs share an
//     SM and one's epilogue runs under the other's loads;
//   * long products with few outputs (the weight gradient: 256 x 256, K = rows
//     of the batch) take 64 x 16 tiles, 128-deep slices and an eight-stage
//     ring: 64 CTAs instead of 4, each at the rate an SM reads from L2 (20 KB a
//     slice, 43 bytes a cycle) with the MMA chain (65 cycles a step of 16) just
//     below it.  The K loop is not split: the accumulator in TMEM rounds
//     towards zero at every step, so partial sums over parts of K would change
//     the weight gradient by 1e-9 of its size per row of the batch (1e-4 at
//     60,000 rows);
//   * the epilogue goes through shared memory so that rows leave in 16-byte
//     stores.
// Measured (warm L2): 256 x 256 x 8192 with both operands M/N-contiguous 37 us
// (one 128 x 128 tile per CTA staged value by value: 2243 us); 8192 x 256 x 256
// 9.5 to 12 us (23 to 28 us).
// ---------------------------------------------------------------------------
constexpr int kTcThreads = 256;  // filling / epilogue threads; one more warp multiplies
enum { EPI_PLAIN = 0, EPI_FWD = 1, EPI_BWD = 2 };
enum { LD_K16 = 0, LD_MN16 = 1, LD_SCALAR = 2 };  // how an operand is staged

struct GemmArgs {
  int M, N, K;
  const __nv_bfloat16* A;
  long long sam, sak;
  const __nv_bfloat16* B;
  long long sbk, sbn;
  int mode_a, mode_b;
  int ra, rb;  // M / N extents that may be read (an M/N-contiguous operand's padded pitch); 0: M, N
  float* C;  // EPI_PLAIN: C = A B + beta C; EPI_FWD: the pre-activation (may be null); [M][ldc]
  long long ldc;
  float beta;
  int vec_c;  // rows of every FP32 / BF16 array of the epilogue start 16 / 8 bytes aligned
  // EPI_FWD: z = A B + bias; h32 / h16 = act ? silu(z) : z (either may be null); [M][N]
  const float* bias;
  int act;
  float* h32;
  __nv_bfloat16* h16;
  // EPI_BWD: h16 = bf16(d), d = act ? (A B) silu'(z) : A B; colpart[m tile][n] = column sums of d
  const float* z;
  double* colpart;
  // EPI_PLAIN: gb[m] = sum_j bias_part[j][m], by the CTA of n tile 0
  const double* bias_part;
  int n_parts;
  float* gb;
  long long wait_limit;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One operand's slice in shared memory, ROWS x BK values (rows r0.., depth k0..), in the swizzled layouts the
// MMA reads at full width (the unswizzled core matrices cost about four times the cycles per MMA):
//   K-major:   64-deep blocks of ROWS x 128 bytes, 16-byte chunk c of row r at chunk c ^ (r & 7);
//   M/N-major: blocks of W = min(ROWS, 64) rows, BK lines of 2 W bytes, 16-byte chunk c of line k at
//              c ^ (k & 7), (k >> 1) & 3 or (k >> 2) & 1 for lines of 128, 64 or 32 bytes.
template <int ROWS, int BK>
struct Operand {
  static constexpr int RB = ROWS < 64 ? 2 * ROWS : 128;  // bytes of an M/N-major line
  static constexpr int kChunks = ROWS * BK / 8, NC = (kChunks + kTcThreads - 1) / kTcThreads;

  static __device__ __forceinline__ uint32_t k_major(int r, int c8) {
    return (uint32_t)((c8 >> 3) * ROWS * 128 + r * 128 + (((c8 & 7) ^ (r & 7)) << 4));
  }
  static __device__ __forceinline__ uint32_t mn_major(int c, int k) {
    constexpr int per = RB / 16;
    const int sw = RB == 128 ? (k & 7) : RB == 64 ? ((k >> 1) & 3) : ((k >> 2) & 1);
    return (uint32_t)((c / per) * BK * RB + k * RB + (((c % per) ^ sw) << 4));
  }
  static __device__ __forceinline__ uint64_t desc(uint32_t addr, int mode) {
    if (mode != LD_MN16) return tcg::mat_desc(addr, 16, 1024, 2);
    return tcg::mat_desc(addr, BK * RB, 8 * RB, RB == 128 ? 2 : RB == 64 ? 4 : 6);
  }
  // address offset of the 16-deep step kk
  static __device__ __forceinline__ uint32_t step(int kk, int mode) {
    return mode == LD_MN16 ? (uint32_t)(kk * 16 * RB) : (uint32_t)((kk >> 2) * ROWS * 128 + (kk & 3) * 32);
  }

  // this thread's chunks: source of the next slice, place in the slice, depth, valid rows
  const __nv_bfloat16* p[NC];
  uint32_t d[NC];
  int kk[NC], rows[NC];
  long long adv;
  int mode;
  bool whole;

  __device__ __forceinline__ void init(const __nv_bfloat16* P, long long sr, long long sk, int md, int r0, int R) {
    mode = md;
    adv = sk * BK;
    whole = true;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int idx = threadIdx.x + i * kTcThreads;
      // consecutive threads take consecutive 16 bytes of a line: whole 128-byte requests, and no bank
      // conflicts with the swizzle
      if (md == LD_K16) {
        const int r = (idx >> 3) % ROWS, c8 = (idx & 7) + 8 * (idx / (8 * ROWS));
        p[i] = P + (long long)(r0 + r) * sr + 8 * c8;
        d[i] = k_major(r, c8);
        kk[i] = 8 * c8;
        rows[i] = r0 + r < R ? 8 : 0;
      } else {
        constexpr int per = RB / 16;
        const int g = idx % per + per * (idx / (per * BK)), k = (idx / per) % BK;
        p[i] = P + (long long)k * sk + r0 + 8 * g;
        d[i] = mn_major(g, k);
        kk[i] = k;
        rows[i] = max(0, min(8, R - r0 - 8 * g));
      }
      whole = whole && rows[i] == 8;
    }
  }
  // Issues this thread's copies of the slice at depth k0 (zero beyond (R, K)).
  __device__ __forceinline__ void copy(unsigned char* slot, int k0, int K) {
    const uint32_t dst = tcg::saddr(slot);
    if (whole && k0 + BK <= K) {  // no edge in this thread's chunks: copies back to back
#pragma unroll
      for (int i = 0; i < NC; ++i)
        if (kChunks % kTcThreads == 0 || i < NC - 1 || threadIdx.x + i * kTcThreads < kChunks)
          cp_async16(dst + d[i], p[i]);
#pragma unroll
      for (int i = 0; i < NC; ++i) p[i] += adv;
      return;
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      if (kChunks % kTcThreads && threadIdx.x + i * kTcThreads >= kChunks) break;
      const int left = K - k0 - kk[i];
      const int n = mode == LD_K16 ? min(rows[i], left) : (left > 0 ? rows[i] : 0);
      if (n == 8) {
        cp_async16(dst + d[i], p[i]);
      } else {  // edge of the operand: what is there, zeros behind it
        __nv_bfloat16 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = j < n ? p[i][j] : __float2bfloat16(0.f);
        *reinterpret_cast<uint4*>(slot + d[i]) = *reinterpret_cast<const uint4*>(v);
      }
      p[i] += adv;
    }
  }
  // Any strides and alignment (the 12 features, the 3 outputs): value by value into the K-major image, eight
  // loads in flight a thread.  Chunks without a value are zeroed when the slot is first used and in a last,
  // partial slice.
  static __device__ __forceinline__ void scalar(unsigned char* slot, const __nv_bfloat16* __restrict__ P,
                                                long long sr, long long sk, int r0, int R, int k0, int K, bool first) {
    const int rv = min(ROWS, R - r0), left = min(BK, K - k0), cv = (left + 7) >> 3;
    if (first || left < BK)
      for (int idx = threadIdx.x; idx < kChunks; idx += kTcThreads) {
        const int r = idx / (BK / 8), c8 = idx % (BK / 8);
        if (r >= rv || c8 >= cv) *reinterpret_cast<uint4*>(slot + k_major(r, c8)) = make_uint4(0u, 0u, 0u, 0u);
      }
    int lg = 3;  // depth covered by a group of threads: the power of two at or above the chunks that hold values
    while ((1 << lg) < 8 * cv) ++lg;
    const int c = threadIdx.x & ((1 << lg) - 1), step = kTcThreads >> lg;
    if (c >= 8 * cv) return;
    const bool in = c < left;
    const __nv_bfloat16* q = P + (long long)(k0 + c) * sk + (long long)r0 * sr;
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    for (int r = threadIdx.x >> lg; r < rv; r += 8 * step) {
      __nv_bfloat16 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = in && r + j * step < rv ? q[(long long)(r + j * step) * sr] : zero;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (r + j * step < rv)
          *reinterpret_cast<__nv_bfloat16*>(slot + k_major(r + j * step, c >> 3) + 2 * (c & 7)) = v[j];
    }
  }
};

// Tile shape, slice depth and ring length of one instantiation.
template <int BM_, int BN_, int BK_, int NST_>
struct GemmCfg {
  static constexpr int BM = BM_, BN = BN_, BK = BK_, NST = NST_;
  static constexpr int kA = BM * BK * 2, kB = BN * BK * 2, kStage = kA + kB;
  static constexpr int kLd = BN + 4;  // floats per row of the output tile: 16-byte rows, conflict-free quads
  static constexpr int kTile = BM * kLd * 4;
  static constexpr int kRing = NST * kStage;
  static constexpr int kBody = kRing > kTile ? kRing : kTile;
  static constexpr int kSums = 8 * 128 * 8;  // column sums: 8 warps x 128 doubles
  static constexpr int kBytes = kBody + kSums + 1024;  // + alignment of the ring
  static constexpr int kCols = BN < 32 ? 32 : BN;  // TMEM columns
};
using GemmWide = GemmCfg<128, 128, 64, 4>;
using GemmMid = GemmCfg<128, 64, 64, 4>;
using GemmNarrow = GemmCfg<128, 32, 64, 4>;
using GemmLong = GemmCfg<64, 16, 128, 8>;

template <class CF, int EPI>
__global__ void __launch_bounds__(kTcThreads + 32) k_gemm_tc(const GemmArgs a) {
  constexpr int BM = CF::BM, BN = CF::BN, BK = CF::BK, NST = CF::NST;
  extern __shared__ unsigned char smem_raw[];
  // the swizzle works on address bits: slots start on 1024-byte boundaries
  unsigned char* smem = smem_raw + ((1024u - (tcg::saddr(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) unsigned long long s_full[NST], s_empty[NST];
  __shared__ uint32_t s_tmem;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tcg::saddr(&s_tmem)),
                 "r"(CF::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) {
      tcg::mbar_init(tcg::saddr(&s_full[i]), 2 * kTcThreads);
      tcg::mbar_init(tcg::saddr(&s_empty[i]), 1);
    }
    s_fail = 0;
  }
  tcg::fence_before();
  __syncthreads();
  tcg::fence_after();
  const uint32_t tmem = s_tmem, base = tcg::saddr(smem);
  const int ns = (a.K + BK - 1) / BK;
  const uint32_t idesc = tcg::idesc_bf16(BM, BN) | (a.mode_a == LD_MN16 ? 1u << 15 : 0u) |
                         (a.mode_b == LD_MN16 ? 1u << 16 : 0u);
  using OpA = Operand<BM, BK>;
  using OpB = Operand<BN, BK>;
  // Warps 0..7 fill the ring, one thread of warp 8 multiplies.  A slice is full once every filling thread's
  // copies landed (cp.async arrival) and its plain stores are done (ordinary arrival); the multiplying thread
  // then fences the generic proxy's writes for the tensor core.  That fence has to sit in a thread without
  // copies of its own in flight: it waits for them, which held the ring to one slice per memory latency when
  // the filling threads ran it.
  int fail = 0, issued = 0;
  if (warp < 8) {
    OpA oa;
    OpB ob;
    oa.init(a.A, a.sam, a.sak, a.mode_a, m0, a.ra);
    ob.init(a.B, a.sbn, a.sbk, a.mode_b, n0, a.rb);
    for (int i = 0; i < ns; ++i) {
      if (i >= NST && !tcg::mbar_wait(tcg::saddr(&s_empty[i % NST]), ((i / NST) - 1) & 1, a.wait_limit, &s_fail)) {
        fail = 1;
        break;
      }
      unsigned char* slot = smem + (i % NST) * CF::kStage;
      const int k0 = i * BK;
      if (a.mode_a == LD_SCALAR)
        OpA::scalar(slot, a.A, a.sam, a.sak, m0, a.M, k0, a.K, i < NST);
      else
        oa.copy(slot, k0, a.K);
      if (a.mode_b == LD_SCALAR)
        OpB::scalar(slot + CF::kA, a.B, a.sbn, a.sbk, n0, a.N, k0, a.K, i < NST);
      else
        ob.copy(slot + CF::kA, k0, a.K);
      tcg::arrive_copies(tcg::saddr(&s_full[i % NST]));
      tcg::arrive(tcg::saddr(&s_full[i % NST]));
    }
  } else if (lane == 0) {
    // one thread's instruction latency is on the chain of every slice: the descriptors of stage 0 are formed
    // once, a stage or a 16-deep step only adds to their address field (14 bits of 16-byte units, no carry out)
    const uint64_t da = OpA::desc(base, a.mode_a), db = OpB::desc(base + CF::kA, a.mode_b);
    for (int i = 0; i < ns; ++i) {
      if (!tcg::mbar_wait(tcg::saddr(&s_full[i % NST]), (i / NST) & 1, a.wait_limit, &s_fail)) {
        fail = 1;
        break;
      }
      tcg::fence_proxy_async();
      const uint64_t off = (uint64_t)((i % NST) * (CF::kStage >> 4));
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk)
        tcg::mma(tmem, da + off + (OpA::step(kk, a.mode_a) >> 4), db + off + (OpB::step(kk, a.mode_b) >> 4), idesc,
                 (i > 0 || kk > 0) ? 1u : 0u);
      tcg::commit(tcg::saddr(&s_empty[i % NST]));
      issued = i + 1;
    }
    // the last commit covers every MMA before it
    if (issued > 0 && !tcg::mbar_wait(tcg::saddr(&s_empty[(issued - 1) % NST]), ((issued - 1) / NST) & 1,
                                      a.wait_limit, nullptr)) {
      fail = 1;
      // none in flight when shared memory is reused and TMEM released
      tcg::mbar_wait(tcg::saddr(&s_empty[(issued - 1) % NST]), ((issued - 1) / NST) & 1, kTcWaitLimit, nullptr);
    }
  }
  if (fail) s_fail = 1;
  cp_async_wait_all();
  fail = __syncthreads_or(fail);
  if (fail && tid == 0) atomicExch(&g_gemm_err, 1);
  // accumulator -> shared tile [BM][BN + 4] (the ring is free: all MMAs completed).  A warp reads its
  // quadrant of 32 TMEM lanes; with BM = 64 the rows sit in the first 16 lanes of each quadrant.
  float* tile = reinterpret_cast<float*>(smem);
  tcg::fence_after();
  if (!fail && warp < 8) {
    constexpr int kRowsQ = BM / 4;
    const int row = (warp & 3) * kRowsQ + lane, half = (warp >> 2) * (BN / 2);
#pragma unroll
    for (int c0 = 0; c0 < BN / 2; c0 += 8) {
      uint32_t r[8];
      const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half + c0);
      if (ns > 0) {
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(ta)
                     : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) r[q] = 0u;
      }
      if (lane < kRowsQ) {
        *reinterpret_cast<uint4*>(tile + row * CF::kLd + half + c0) = make_uint4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<uint4*>(tile + row * CF::kLd + half + c0 + 4) = make_uint4(r[4], r[5], r[6], r[7]);
      }
    }
  }
  tcg::fence_before();
  __syncthreads();
  tcg::fence_after();
  const bool ok = !fail && warp < 8;
  // epilogue: four columns a thread
  constexpr int QN = BN / 4, RPW = 32 / QN;  // quads per row; rows per warp step
  const int quad = lane % QN, sub = lane / QN, n = n0 + 4 * quad;
  double cs[4] = {0.0, 0.0, 0.0, 0.0};
  if (ok) {
    float bv[4] = {0.f, 0.f, 0.f, 0.f};
    if (EPI == EPI_FWD && a.bias)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (n + q < a.N) bv[q] = a.bias[n + q];
    const bool full = a.vec_c && n + 4 <= a.N;
#pragma unroll 4
    for (int r = warp * RPW + sub; r < BM; r += 8 * RPW) {
      const int m = m0 + r;
      if (m >= a.M || n >= a.N) continue;
      const float4 t = *reinterpret_cast<const float4*>(tile + r * CF::kLd + 4 * quad);
      float v[4] = {t.x, t.y, t.z, t.w};
      const long long at = (long long)m * a.ldc + n;
      if (EPI == EPI_PLAIN) {
        if (full) {
          if (a.beta != 0.f) {
            const float4 c = *reinterpret_cast<const float4*>(a.C + at);
            v[0] += a.beta * c.x;
            v[1] += a.beta * c.y;
            v[2] += a.beta * c.z;
            v[3] += a.beta * c.w;
          }
          *reinterpret_cast<float4*>(a.C + at) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (n + q < a.N) a.C[at + q] = v[q] + (a.beta != 0.f ? a.beta * a.C[at + q] : 0.f);
        }
      } else if (EPI == EPI_FWD) {
        float h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          v[q] += bv[q];
          h[q] = a.act ? v[q] / (1.f + expf(-v[q])) : v[q];
        }
        if (full) {
          if (a.C) *reinterpret_cast<float4*>(a.C + at) = make_float4(v[0], v[1], v[2], v[3]);
          if (a.h32) *reinterpret_cast<float4*>(a.h32 + at) = make_float4(h[0], h[1], h[2], h[3]);
          if (a.h16) {
            __nv_bfloat162 p[2] = {__floats2bfloat162_rn(h[0], h[1]), __floats2bfloat162_rn(h[2], h[3])};
            *reinterpret_cast<uint2*>(a.h16 + at) = *reinterpret_cast<uint2*>(p);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (n + q < a.N) {
              if (a.C) a.C[at + q] = v[q];
              if (a.h32) a.h32[at + q] = h[q];
              if (a.h16) a.h16[at + q] = __float2bfloat16(h[q]);
            }
        }
      } else {
        float z[4] = {0.f, 0.f, 0.f, 0.f};
        if (a.act) {
          if (full) {
            const float4 zz = *reinterpret_cast<const float4*>(a.z + at);
            z[0] = zz.x;
            z[1] = zz.y;
            z[2] = zz.z;
            z[3] = zz.w;
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (n + q < a.N) z[q] = a.z[at + q];
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float sg = 1.f / (1.f + expf(-z[q]));
            v[q] *= sg * (1.f + z[q] * (1.f - sg));
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) cs[q] += (double)v[q];
        if (full) {
          __nv_bfloat162 p[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
          *reinterpret_cast<uint2*>(a.h16 + at) = *reinterpret_cast<uint2*>(p);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (n + q < a.N) a.h16[at + q] = __float2bfloat16(v[q]);
        }
      }
    }
    if (EPI == EPI_PLAIN && a.gb && blockIdx.x == 0)
      for (int m = m0 + tid; m < min(a.M, m0 + BM); m += kTcThreads) {
        double acc = 0.0;
        for (int j = 0; j < a.n_parts; ++j) acc += a.bias_part[(long long)j * a.M + m];
        a.gb[m] = (float)acc;
      }
  }
  if (EPI == EPI_BWD) {  // column sums of this tile: warps and row lanes in a fixed order
    double* sums = reinterpret_cast<double*>(smem + CF::kBody);
    if (warp < 8)
#pragma unroll
      for (int q = 0; q < 4; ++q) sums[(warp * RPW + sub) * BN + 4 * quad + q] = cs[q];
    __syncthreads();
    if (ok && tid < BN && n0 + tid < a.N) {
      double acc = 0.0;
#pragma unroll
      for (int w = 0; w < 8 * RPW; ++w) acc += sums[w * BN + tid];
      a.colpart[(long long)blockIdx.y * a.N + n0 + tid] = acc;
    }
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CF::kCols) : "memory");
}

// How an operand with element (r, k) at P[r * sr + k * sk] is staged: 16-byte
// copies along its contiguous direction where every copy starts 16-byte
// aligned (the other stride a multiple of 8 values), else value by value.
int load_mode(const void* P, long long sr, long long sk) {
  const bool aligned = ((uintptr_t)P & 15) == 0;
  if (aligned && sk == 1 && (sr & 7) == 0) return LD_K16;
  if (aligned && sr == 1 && (sk & 7) == 0) return LD_MN16;
  return LD_SCALAR;
}

template <class CF, int EPI>
int launch_gemm(const GemmArgs& a, cudaStream_t st) {
  auto* k = &k_gemm_tc<CF, EPI>;
  const long long mt = (a.M + CF::BM - 1) / CF::BM;
  if (mt > 65535) return set_error(FNE_EBOUNDS, "fne_gemm_bf16: M too large");
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CF::kBytes);
  if (e == cudaSuccess) {
    k<<<dim3((a.N + CF::BN - 1) / CF::BN, (unsigned)mt), kTcThreads + 32, CF::kBytes, st>>>(a);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("k_gemm_tc: ") + cudaGetErrorString(e));
  return FNE_OK;
}

// Tile choice.  Width: 32 for the network's narrow outputs; 128 once that
// gives every SM a tile, else 64 (twice the CTAs, two per SM).  Plain products
// that leave most SMs without a tile of 128 x 64 and are at least 1024 deep
// take the long form (below that a tile's fixed cost outweighs the loop).
template <int EPI>
int run_gemm(GemmArgs& a, cudaStream_t st) {
  const long long mt = (a.M + kTcBM - 1) / kTcBM;
  a.mode_a = load_mode(a.A, a.sam, a.sak);
  a.mode_b = load_mode(a.B, a.sbn, a.sbk);
  if (a.ra < a.M) a.ra = a.M;
  if (a.rb < a.N) a.rb = a.N;
  if constexpr (EPI == EPI_PLAIN)
    if (a.K >= 1024 && mt * ((a.N + 63) / 64) <= 148 / 4) return launch_gemm<GemmLong, EPI>(a, st);
  if (a.N <= 32) return launch_gemm<GemmNarrow, EPI>(a, st);
  if (mt * ((a.N + 127) / 128) < 148) return launch_gemm<GemmMid, EPI>(a, st);
  return launch_gemm<GemmWide, EPI>(a, st);
}

// Z[n, m] += b[m]; H = silu(Z) (FP32 and BF16 copies); act = 0 leaves H = Z.
__global__ void k_bias_act_fwd(long long rows, int cols, float* __restrict__ Z, const float* __restrict__ b, int act,
                               float* __restrict__ H32, __nv_bfloat16* __restrict__ H16) {
  const long long n = rows * cols;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float z = Z[i] + (b ? b[i % cols] : 0.f);
    Z[i] = z;
    const float h = act ? z / (1.f + expf(-z)) : z;
    if (H32) H32[i] = h;
    if (H16) H16[i] = __float2bfloat16(h);
  }
}

// dZ = dH * silu'(Z) (act = 1) or dH (act = 0); FP32 and BF16 copies.
__global__ void k_act_bwd(long long n, const float* __restrict__ Z, const float* __restrict__ dH, int act,
                          float* __restrict__ dZ32, __nv_bfloat16* __restrict__ dZ16) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float d = dH[i];
    if (act) {
      const float z = Z[i];
      const float s = 1.f / (1.f + expf(-z));
      d *= s * (1.f + z * (1.f - s));
    }
    if (dZ32) dZ32[i] = d;
    if (dZ16) dZ16[i] = __float2bfloat16(d);
  }
}

// out[m] = sum_n X[n, m] (bias gradient) in FP64, fixed order.  A cluster of 8
// CTAs takes 32 columns: CTA r the r-th eighth of the rows, its 32 warps every
// 32nd row each (128-byte reads); the warps' sums meet in shared memory, the
// CTAs' in the distributed shared memory of rank 0.  (One thread per column
// over all rows, as before, took 567 us for 8192 x 256 on the latency of its
// serial loads.)
constexpr int kSumCtas = 8;
__global__ void __cluster_dims__(1, kSumCtas, 1) __launch_bounds__(1024)
    k_colsum(long long rows, int cols, const float* __restrict__ X, float* __restrict__ out) {
  __shared__ double s[32][33];
  __shared__ double total[32];
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.y;
  const int m = blockIdx.x * 32 + lane;
  const long long n1 = rows * (r + 1) / kSumCtas;
  double acc = 0.0;
  if (m < cols)
#pragma unroll 8
    for (long long n = rows * r / kSumCtas + w; n < n1; n += 32) acc += (double)__ldg(X + n * cols + m);
  s[w][lane] = acc;
  __syncthreads();
  if (w == 0) {
    acc = 0.0;
#pragma unroll
    for (int j = 0; j < 32; ++j) acc += s[j][lane];
    total[lane] = acc;
  }
  cluster.sync();
  if (r == 0 && w == 0) {
    acc = 0.0;
#pragma unroll
    for (int j = 0; j < kSumCtas; ++j) acc += cluster.map_shared_rank(total, j)[lane];
    if (m < cols) out[m] = (float)acc;
  }
  cluster.sync();
}

// Adam on FP32 master weights; refreshes the BF16 copy used by the GEMMs.
__global__ void k_adam(long long n, float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2,
                       __nv_bfloat16* __restrict__ p16) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    if (p16) p16[i] = __float2bfloat16(pi);
  }
}

// The same update over up to kAdamMax tensors in one launch (a step of the
// network touches eight, the largest 65,536 values: alone each launch is its
// own latency).
constexpr int kAdamMax = 32;
struct AdamSet {
  long long end[kAdamMax];  // running total of the sizes
  float* p[kAdamMax];
  const float* g[kAdamMax];
  float* m[kAdamMax];
  float* v[kAdamMax];
  __nv_bfloat16* p16[kAdamMax];
  int count;
};
__global__ void k_adam_set(const AdamSet T, float lr, float b1, float b2, float eps, float c1, float c2) {
  const long long n = T.end[T.count - 1];
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    int t = 0;
    while (k >= T.end[t]) ++t;
    const long long i = k - (t ? T.end[t - 1] : 0);
    const float gi = T.g[t][i];
    const float mi = b1 * T.m[t][i] + (1.f - b1) * gi;
    const float vi = b2 * T.v[t][i] + (1.f - b2) * gi * gi;
    T.m[t][i] = mi;
    T.v[t][i] = vi;
    const float pi = T.p[t][i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    T.p[t][i] = pi;
    if (T.p16[t]) T.p16[t][i] = __float2bfloat16(pi);
  }
}

// Rows of `cols` values (FP32 or BF16) as BF16 rows of pitch `pitch`, zeros behind them.
template <typename T>
__global__ void k_pad_rows(long long rows, int cols, const T* __restrict__ x, int pitch,
                           __nv_bfloat16* __restrict__ y) {
  const long long n = rows * pitch;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / pitch;
    const int c = (int)(i - r * pitch);
    y[i] = c < cols ? static_cast<__nv_bfloat16>(x[r * cols + c]) : __float2bfloat16(0.f);
  }
}

__global__ void k_cast_bf16(long long n, const float* __restrict__ x, __nv_bfloat16* __restrict__ y) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

int grid_for(long long n) { return (int)std::max<long long>(1, std::min<long long>(148 * 16, (n + 255) / 256)); }

int launch_status(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return FNE_OK;
}

}  // namespace
}  // namespace fne

using namespace fne;

namespace {
long long g_gemm_wait_limit = kTcWaitLimit;  // polls of the GEMM's MMA-completion waits
}  // namespace

extern "C" int fne_gemm_set_wait_limit(int64_t polls) {
  g_gemm_wait_limit = polls < 0 ? kTcWaitLimit : (long long)polls;
  return FNE_OK;
}

extern "C" int fne_gemm_check_status(void) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_gemm_err, sizeof(int));
  if (e != cudaSuccess) return set_error(FNE_ECUDA, std::string("fne_gemm_check_status: ") + cudaGetErrorString(e));
  if (v == 0) return FNE_OK;
  const int zero = 0;
  cudaMemcpyToSymbol(g_gemm_err, &zero, sizeof(int));
  return set_error(FNE_ETIMEOUT, "fne_gemm_bf16: an MMA-completion wait gave up");
}

extern "C" int fne_gemm_bf16(int M, int N, int K, const void* A, int64_t sam, int64_t sak, const void* B, int64_t sbk,
                             int64_t sbn, float* C, int64_t ldc, float beta, void* stream) {
  if (M < 0 || N < 0 || K < 0 || (M * (int64_t)N > 0 && !C) || (M * (int64_t)K > 0 && !A) ||
      (K * (int64_t)N > 0 && !B))
    return set_error(FNE_EINVAL, "fne_gemm_bf16: bad arguments");
  if (M == 0 || N == 0) return FNE_OK;
  GemmArgs a = {};
  a.M = M;
  a.N = N;
  a.K = K;
  a.A = (const __nv_bfloat16*)A;
  a.sam = sam;
  a.sak = sak;
  a.B = (const __nv_bfloat16*)B;
  a.sbk = sbk;
  a.sbn = sbn;
  a.C = C;
  a.ldc = ldc;
  a.beta = beta;
  a.vec_c = ((uintptr_t)C & 15) == 0 && (ldc & 3) == 0;
  a.wait_limit = g_gemm_wait_limit;
  return run_gemm<EPI_PLAIN>(a, (cudaStream_t)stream);
}

namespace {
bool aligned(const void* p, uintptr_t to) { return ((uintptr_t)p & (to - 1)) == 0; }
}  // namespace

extern "C" int fne_mlp_linear_fwd(int rows, int din, int dout, const void* X16, const void* W16, const float* bias,
                                  int act, float* Z, float* H32, void* H16, void* stream) {
  if (rows < 0 || din <= 0 || dout <= 0 || (rows > 0 && (!X16 || !W16)))
    return set_error(FNE_EINVAL, "fne_mlp_linear_fwd: bad arguments");
  if (rows == 0) return FNE_OK;
  GemmArgs a = {};
  a.M = rows;
  a.N = dout;
  a.K = din;
  a.A = (const __nv_bfloat16*)X16;
  a.sam = din;
  a.sak = 1;
  a.B = (const __nv_bfloat16*)W16;
  a.sbk = 1;
  a.sbn = din;
  a.C = Z;
  a.ldc = dout;
  a.bias = bias;
  a.act = act;
  a.h32 = H32;
  a.h16 = (__nv_bfloat16*)H16;
  a.vec_c = (dout & 3) == 0 && aligned(Z, 16) && aligned(H32, 16) && aligned(H16, 8);
  a.wait_limit = g_gemm_wait_limit;
  return run_gemm<EPI_FWD>(a, (cudaStream_t)stream);
}

extern "C" int fne_mlp_pad_rows(int64_t rows, int cols, const void* x, int x_fp32, int pitch, void* y, void* stream) {
  if (rows < 0 || cols <= 0 || pitch < cols || (rows > 0 && (!x || !y)))
    return set_error(FNE_EINVAL, "fne_mlp_pad_rows: bad arguments");
  if (rows == 0) return FNE_OK;
  const int grid = grid_for(rows * (long long)pitch);
  if (x_fp32)
    k_pad_rows<<<grid, 256, 0, (cudaStream_t)stream>>>(rows, cols, (const float*)x, pitch, (__nv_bfloat16*)y);
  else
    k_pad_rows<<<grid, 256, 0, (cudaStream_t)stream>>>(rows, cols, (const __nv_bfloat16*)x, pitch, (__nv_bfloat16*)y);
  return launch_status("fne_mlp_pad_rows");
}

extern "C" int fne_mlp_linear_bwd_data(int rows, int din, int dout, const void* dZ16, int ldz, const void* W16,
                                       const float* Zin, int act, void* dZin16, double* colpart, void* stream) {
  if (rows < 0 || din <= 0 || dout <= 0 || ldz < dout || (rows > 0 && (!dZ16 || !W16 || !dZin16 || !colpart || (act && !Zin))))
    return set_error(FNE_EINVAL, "fne_mlp_linear_bwd_data: bad arguments");
  if (rows == 0) return FNE_OK;
  GemmArgs a = {};
  a.M = rows;
  a.N = din;
  a.K = dout;
  a.A = (const __nv_bfloat16*)dZ16;
  a.sam = ldz;
  a.sak = 1;
  a.B = (const __nv_bfloat16*)W16;
  a.sbk = din;
  a.sbn = 1;
  a.ldc = din;
  a.act = act;
  a.z = Zin;
  a.h16 = (__nv_bfloat16*)dZin16;
  a.colpart = colpart;
  a.vec_c = (din & 3) == 0 && aligned(Zin, 16) && aligned(dZin16, 8);
  a.wait_limit = g_gemm_wait_limit;
  return run_gemm<EPI_BWD>(a, (cudaStream_t)stream);
}

extern "C" int fne_mlp_linear_bwd_weight(int rows, int din, int dout, const void* dZ16, int ldz, const void* X16,
                                         int ldx, float* gW, const double* colpart, float* gb, void* stream) {
  if (rows < 0 || din <= 0 || dout <= 0 || ldz < dout || ldx < din || !gW || (rows > 0 && (!dZ16 || !X16)) || ((gb != nullptr) != (colpart != nullptr)))
    return set_error(FNE_EINVAL, "fne_mlp_linear_bwd_weight: bad arguments");
  GemmArgs a = {};
  a.M = dout;
  a.N = din;
  a.K = rows;
  a.A = (const __nv_bfloat16*)dZ16;
  a.sam = 1;
  a.sak = ldz;
  a.ra = ldz;
  a.B = (const __nv_bfloat16*)X16;
  a.sbk = ldx;
  a.sbn = 1;
  a.rb = ldx;
  a.C = gW;
  a.ldc = din;
  a.vec_c = (din & 3) == 0 && aligned(gW, 16);
  a.bias_part = colpart;
  a.n_parts = (rows + kTcBM - 1) / kTcBM;
  a.gb = gb;
  a.wait_limit = g_gemm_wait_limit;
  return run_gemm<EPI_PLAIN>(a, (cudaStream_t)stream);
}

extern "C" int fne_mlp_bias_act(int64_t rows, int cols, float* Z, const float* bias, int act, float* H32, void* H16,
                                void* stream) {
  if (rows < 0 || cols <= 0 || !Z) return set_error(FNE_EINVAL, "fne_mlp_bias_act: bad arguments");
  const long long n = rows * (long long)cols;
  if (n == 0) return FNE_OK;
  k_bias_act_fwd<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(rows, cols, Z, bias, act, H32,
                                                                  (__nv_bfloat16*)H16);
  return launch_status("fne_mlp_bias_act");
}

extern "C" int fne_mlp_act_bwd(int64_t n, const float* Z, const float* dH, int act, float* dZ32, void* dZ16,
                               void* stream) {
  if (n < 0 || (n > 0 && (!dH || (act && !Z)))) return set_error(FNE_EINVAL, "fne_mlp_act_bwd: bad arguments");
  if (n == 0) return FNE_OK;
  k_act_bwd<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, Z, dH, act, dZ32, (__nv_bfloat16*)dZ16);
  return launch_status("fne_mlp_act_bwd");
}

extern "C" int fne_mlp_colsum(int64_t rows, int cols, const float* X, float* out, void* stream) {
  if (rows < 0 || cols <= 0 || !X || !out) return set_error(FNE_EINVAL, "fne_mlp_colsum: bad arguments");
  k_colsum<<<dim3((cols + 31) / 32, kSumCtas), 1024, 0, (cudaStream_t)stream>>>(rows, cols, X, out);
  return launch_status("fne_mlp_colsum");
}

extern "C" int fne_mlp_adam(int64_t n, float* p, const float* g, float* m, float* v, float lr, float b1, float b2,
                            float eps, int step, void* p16, void* stream) {
  if (n < 0 || step < 1 || (n > 0 && (!p || !g || !m || !v))) return set_error(FNE_EINVAL, "fne_mlp_adam: bad arguments");
  if (n == 0) return FNE_OK;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  k_adam<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2,
                                                          (__nv_bfloat16*)p16);
  return launch_status("fne_mlp_adam");
}

extern "C" int fne_mlp_adam_set(int count, const int64_t* n, float* const* p, const float* const* g, float* const* m,
                                float* const* v, void* const* p16, float lr, float b1, float b2, float eps, int step,
                                void* stream) {
  if (count < 0 || step < 1 || (count > 0 && (!n || !p || !g || !m || !v || !p16)))
    return set_error(FNE_EINVAL, "fne_mlp_adam_set: bad arguments");
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  for (int k = 0; k < count; ++k)
    if (n[k] < 0 || (n[k] > 0 && (!p[k] || !g[k] || !m[k] || !v[k])))
      return set_error(FNE_EINVAL, "fne_mlp_adam_set: bad arguments");
  for (int k0 = 0; k0 < count; k0 += kAdamMax) {
    AdamSet T = {};
    T.count = std::min(kAdamMax, count - k0);
    long long total = 0;
    for (int k = 0; k < T.count; ++k) {
      total += n[k0 + k];
      T.end[k] = total;
      T.p[k] = p[k0 + k];
      T.g[k] = g[k0 + k];
      T.m[k] = m[k0 + k];
      T.v[k] = v[k0 + k];
      T.p16[k] = (__nv_bfloat16*)p16[k0 + k];
    }
    if (total == 0) continue;
    k_adam_set<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(T, lr, b1, b2, eps, c1, c2);
    const int rc = launch_status("fne_mlp_adam_set");
    if (rc != FNE_OK) return rc;
  }
  return FNE_OK;
}

extern "C" int fne_mlp_cast_bf16(int64_t n, const float* x, void* y, void* stream) {
  if (n < 0 || (n > 0 && (!x || !y))) return set_error(FNE_EINVAL, "fne_mlp_cast_bf16: bad arguments");
  if (n == 0) return FNE_OK;
  k_cast_bf16<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, x, (__nv_bfloat16*)y);
  return launch_status("fne_mlp_cast_bf16");
}
