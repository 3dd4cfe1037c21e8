// mlp.cu -- the learned proposal filter's network: a 32 -> 256 -> 256 -> 1
// ReLU MLP on BF16 tensor cores with FP32 accumulation, with hand-written
// forward, backward and Adam kernels.  The annealing engine ranks thousands
// of candidate swaps with it every step and trains it online on the exact
// changes of ASPL the evaluator measures for the candidates it evaluates.
// No counterpart in the reference, whose annealing draws one random swap at a
// time (general/sa.c:217-369).
//
// Numerics (the CPU oracle restates them): inputs and weights are rounded to
// BF16; every product is accumulated in FP32; the first hidden layer is
// stored as BF16 after bias and ReLU; the second stays FP32 and feeds the FP32
// output dot product.  Backward: dy = 2 (y - t) / B; the gradients that enter
// a tensor-core product (dZ2, dZ1) are rounded to BF16; weight and bias
// gradients are FP32.
//
// The inference forward that ranks the proposals (4096 rows a step) is one
// kernel on the fifth-generation tensor cores, forward_tc_kernel: per 128
// rows, tcgen05.mma with both layers' FP32 accumulators in tensor memory,
// operands staged in shared memory by bulk copies, bias, ReLU and the output
// head applied between tcgen05.ld and the next product, no round trip through
// global memory.  It replaced an mma.sync kernel of the same fusion (ldmatrix
// fragments, 32 rows a CTA): 8.2 us against 10.3 us for 4096 rows.  A
// training step (at most 256 rows) is two launches of mma.sync.m16n8k16 (BF16
// in, FP32 accumulate): train_rows_kernel does all that is local to 16 rows,
// train_weights_kernel the sums over the rows and Adam.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/graphgolf_b200.h"
#include "core_internal.h"
#include "mlp_internal.h"

using ggb::core_fail;

#define MCUDA(call)                                                                                  \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess)                                                                           \
      return core_fail(GGB_ECUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                       __LINE__);                                                                    \
  } while (0)

namespace ggb {
namespace mlp {

using bf16 = __nv_bfloat16;

// D = A (16x16, row) * B (16x8, col) + D, BF16 inputs, FP32 accumulators.
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Bulk copies global -> shared (cp.async.bulk, completion on an mbarrier).
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_parity(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- the tcgen05 inference forward ---------------------------------------------------
// The same y = w3 . relu(W2 relu(W1 x + b1) + b2) + b3, on the fifth-generation
// tensor cores: one CTA per 128 rows (M of one tcgen05.mma), both layers'
// accumulators in tensor memory (TMEM), operands in shared memory.
//   * Staging: W1 and W2 sit in global memory already in the operand layout
//     (written by the cast and Adam kernels), so bulk copies bring them in:
//     W1 (16 KB) on one mbarrier, W2 (8 x 16 KB) on another, so that layer 1
//     and its epilogue run while W2 is still arriving; the CTA's rows of x are
//     stored into the same layout by plain 16-byte stores.
//   * Layer 1: two tcgen05.mma (M 128, N 256, K 16) into TMEM columns 0-255.
//   * Epilogue 1: warp w reads TMEM lanes 32 (w % 4) .. +32 (its rows) and
//     columns 128 (w / 4) .. +128 with tcgen05.ld, adds b1, applies ReLU,
//     rounds to BF16 and stores H1 in the operand layout.
//   * Layer 2: sixteen tcgen05.mma (K 16 each) into columns 256-511.
//   * Epilogue 2: bias, ReLU and the w3 dot product per thread (a thread owns
//     a row), the two column halves added in shared memory.
// One thread issues the MMAs; tcgen05.commit arrives on an mbarrier that the
// CTA waits on (bounded by %globaltimer, 2 s; a wait that runs out leaves
// NaN for the CTA's rows).  Numerics as the other forwards: BF16 operands,
// FP32 accumulation, H1 rounded to BF16.
namespace tc {
constexpr int kRows = 128;
constexpr int kThreads = 256;
constexpr uint32_t kW2Bytes = kHidden * kHidden * 2;      // 131072
constexpr uint32_t kW1Bytes = kHidden * kFeatures * 2;    // 16384
constexpr uint32_t kXBytes = kRows * kFeatures * 2;       // 8192
constexpr uint32_t kH1Bytes = kRows * kHidden * 2;        // 65536
constexpr uint32_t kSOffW1 = kW2Bytes;
constexpr uint32_t kSOffX = kSOffW1 + kW1Bytes;
constexpr uint32_t kSOffH1 = kSOffX + kXBytes;
constexpr uint32_t kSOffVec = kSOffH1 + kH1Bytes;          // b1, b2, w3 (FP32)
constexpr uint32_t kSOffPart = kSOffVec + 3 * kHidden * 4; // [kRows][2] FP32
constexpr size_t kSmem = kSOffPart + kRows * 2 * 4;
constexpr uint32_t kTmemCols = 512;                       // layer 1: 0-255, layer 2: 256-511
// Instruction descriptor of kind::f16: FP32 accumulator (bits 4-5 = 1), A and
// B BF16 (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3
// in bits 17-22, M >> 4 in bits 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kHidden >> 3) << 17) |
                            ((uint32_t)(kRows >> 4) << 24);
static_assert(kSmem + 1024 <= 227 * 1024, "the operands and the static barriers must fit one CTA's shared memory");
}  // namespace tc

// Element offset of (row r, column k) of a [rows][K] BF16 operand in the
// K-major, no-swizzle layout: 8 x 8 core matrices of 128 contiguous bytes,
// core (r / 8, k / 8) at byte (r / 8) * 16 K + (k / 8) * 128.  Descriptor:
// leading-dimension offset 128 bytes (next 8 columns), stride offset 16 K
// bytes (next 8 rows).
__host__ __device__ constexpr int umma_k_off(int r, int k, int K) {
  return (r >> 3) * (K * 8) + (k >> 3) * 64 + (r & 7) * 8 + (k & 7);
}

// Shared-memory matrix descriptor: start, leading and stride byte offsets in
// 16-byte units, descriptor version 1 (bits 46-47), no swizzle (bits 61-63 = 0).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity) {
  if (mbar_try_wait_parity(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait_parity(bar, parity))
    if (global_ns() - t0 > 2000000000ULL) return false;
  return true;
}

__global__ void __launch_bounds__(tc::kThreads, 1) forward_tc_kernel(const bf16* __restrict__ X, int rows,
                                                                   const bf16* __restrict__ W1u,
                                                                   const bf16* __restrict__ W2u,
                                                                   const float* __restrict__ params,
                                                                   float* __restrict__ y) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char s_tc[];
  __shared__ alignas(8) unsigned long long s_bars[3];   // [0] W1 staged, [1] MMA completion, [2] W2 staged
  __shared__ uint32_t s_tmem;
  __shared__ int s_ok;
  bf16* const W2s = reinterpret_cast<bf16*>(s_tc);
  bf16* const W1s = reinterpret_cast<bf16*>(s_tc + kSOffW1);
  bf16* const Xs = reinterpret_cast<bf16*>(s_tc + kSOffX);
  bf16* const H1s = reinterpret_cast<bf16*>(s_tc + kSOffH1);
  float* const b1s = reinterpret_cast<float*>(s_tc + kSOffVec);
  float* const b2s = b1s + kHidden;
  float* const w3s = b2s + kHidden;
  float* const part = reinterpret_cast<float*>(s_tc + kSOffPart);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = blockIdx.x * kRows;
  const int valid = min(kRows, rows - r0);
  const unsigned bar_st = smem_u32(&s_bars[0]), bar_mma = smem_u32(&s_bars[1]), bar_w2 = smem_u32(&s_bars[2]);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_st) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_mma) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_w2) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    // W1 first, on its own barrier: layer 1 and its epilogue run while W2 arrives
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_st), "r"(kW1Bytes) : "memory");
    bulk_copy(W1s, W1u, kW1Bytes, bar_st);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_w2), "r"(kW2Bytes) : "memory");
    for (uint32_t c = 0; c < kW2Bytes; c += 16384u)
      bulk_copy(s_tc + c, reinterpret_cast<const unsigned char*>(W2u) + c, 16384u, bar_w2);
  }
  // this CTA's rows of x (zeros past the last row) into the operand layout
  for (int i = tid; i < kRows * (kFeatures / 8); i += kThreads) {
    const int r = i / (kFeatures / 8), c = (i % (kFeatures / 8)) * 8;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < valid) v = *reinterpret_cast<const uint4*>(X + (long long)(r0 + r) * kFeatures + c);
    *reinterpret_cast<uint4*>(Xs + umma_k_off(r, c, kFeatures)) = v;
  }
  for (int i = tid; i < kHidden; i += kThreads) {
    b1s[i] = params[kOffB1 + i];
    b2s[i] = params[kOffB2 + i];
    w3s[i] = params[kOffW3 + i];
  }
  // the generic-proxy stores of x must be visible to the tensor cores' reads
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  if (tid == 0) {
    const bool staged = mbar_wait_bounded(bar_st, 0u);
    if (staged) {
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < kFeatures / 16; ++ks)
        umma_bf16(tmem, umma_desc(smem_u32(Xs) + 256u * ks, 128u, 16u * kFeatures),
                  umma_desc(smem_u32(W1s) + 256u * ks, 128u, 16u * kFeatures), kIdesc, ks > 0);
      umma_commit(bar_mma);
    }
    s_ok = staged;
  }
  __syncthreads();
  const bool ok1 = s_ok && mbar_wait_bounded(bar_mma, 0u);
  const int q = warp & 3, h = warp >> 2;
  const int row = 32 * q + lane;
  const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
  bool failed = __syncthreads_or(!ok1);
  if (!failed) {
    tc_fence_after();
    // epilogue 1: H1 = bf16(relu(acc + b1)) into the operand layout
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
      const int col0 = 128 * h + 32 * j;
      uint32_t v[32];
      tmem_ld32(lane_base + (uint32_t)col0, v);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint32_t pk[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = col0 + 8 * m + 2 * e;
          const float f0 = fmaxf(__uint_as_float(v[8 * m + 2 * e]) + b1s[c], 0.f);
          const float f1 = fmaxf(__uint_as_float(v[8 * m + 2 * e + 1]) + b1s[c + 1], 0.f);
          const __nv_bfloat162 b2v = __floats2bfloat162_rn(f0, f1);
          pk[e] = *reinterpret_cast<const uint32_t*>(&b2v);
        }
        *reinterpret_cast<uint4*>(H1s + umma_k_off(row, col0 + 8 * m, kHidden)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      }
    }
    bool w2_ok = true;
    if (tid == 0) w2_ok = mbar_wait_bounded(bar_w2, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    failed = __syncthreads_or(!w2_ok);
  }
  if (!failed) {
    if (tid == 0) {
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < kHidden / 16; ++ks)
        umma_bf16(tmem + (uint32_t)kHidden, umma_desc(smem_u32(H1s) + 256u * ks, 128u, 16u * kHidden),
                  umma_desc(smem_u32(W2s) + 256u * ks, 128u, 16u * kHidden), kIdesc, ks > 0);
      umma_commit(bar_mma);
    }
    const bool ok2 = mbar_wait_bounded(bar_mma, 1u);
    failed = __syncthreads_or(!ok2);
    if (!failed) {
      tc_fence_after();
      // epilogue 2: this thread's row, columns 128 h .. +128
      float s = 0.f;
#pragma unroll 1
      for (int j = 0; j < 4; ++j) {
        const int col0 = 128 * h + 32 * j;
        uint32_t v[32];
        tmem_ld32(lane_base + (uint32_t)(kHidden + col0), v);
#pragma unroll
        for (int e = 0; e < 32; ++e) s = fmaf(fmaxf(__uint_as_float(v[e]) + b2s[col0 + e], 0.f), w3s[col0 + e], s);
      }
      part[row * 2 + h] = s;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid < valid) y[r0 + tid] = failed ? __int_as_float(0x7fc00000) : (part[2 * tid] + part[2 * tid + 1]) + params[kOffB3];
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// ---- the training step -----------------------------------------------------------------
// Four 8 x 8 BF16 matrices, one 16-byte row address a lane (lane 8i + r: row r
// of matrix i); TRANS: each transposed.
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], unsigned saddr) {
  if constexpr (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr)
                 : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr)
                 : "memory");
}

// acc[nt] += A (16 rows, columns of A) * B^T for this warp's four column tiles
// n0 + 8 nt, over K columns in steps of 16 in ascending order.  A and W lie in
// shared memory in the operand layout (umma_k_off), whose core matrices are
// ldmatrix's 8 x 8 matrices, so every access is free of bank conflicts.
// TRANS false: B[n][k] = W[n][k], W of KW columns.  TRANS true: B[n][k] = W[k][n].
template <bool TRANS>
__device__ __forceinline__ void warp_product(float (&acc)[4][4], const bf16* A, int KA, const bf16* W, int KW, int n0,
                                             int K) {
  const int lane = threadIdx.x & 31, i = lane >> 3, r = lane & 7;
  for (int k0 = 0; k0 < K; k0 += 16) {
    // A fragment: (rows 0-7, k 0-7), (rows 8-15, k 0-7), (rows 0-7, k 8-15), (rows 8-15, k 8-15)
    uint32_t a[4];
    ldmatrix4<false>(a, smem_u32(A + umma_k_off(8 * (i & 1) + r, k0 + 8 * (i >> 1), KA)));
#pragma unroll
    for (int p = 0; p < 2; ++p) {      // two column tiles a load
      const int n = n0 + 16 * p;
      uint32_t b[4];
      if constexpr (TRANS)
        ldmatrix4<true>(b, smem_u32(W + umma_k_off(k0 + 8 * (i & 1) + r, n + 8 * (i >> 1), KW)));
      else
        ldmatrix4<false>(b, smem_u32(W + umma_k_off(n + 8 * (i >> 1) + r, k0 + 8 * (i & 1), KW)));
      mma_16816(acc[2 * p], a[0], a[1], a[2], a[3], b[0], b[1]);
      mma_16816(acc[2 * p + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
    }
  }
}

namespace tr {
constexpr int kRows = 16;                                  // rows a CTA of the row pass
constexpr int kThreads = 256;
constexpr uint32_t kSW1 = kHidden * kHidden * 2;          // behind W2
constexpr uint32_t kSX = kSW1 + kHidden * kFeatures * 2;
constexpr uint32_t kSH1 = kSX + kRows * kFeatures * 2;
constexpr uint32_t kSD2 = kSH1 + kRows * kHidden * 2;
constexpr int kPitch = kHidden + 4;                        // FP32 rows of H2, off the banks of the row before
constexpr uint32_t kSH2 = kSD2 + kRows * kHidden * 2;
constexpr uint32_t kSDy = kSH2 + kRows * kPitch * 4;
constexpr size_t kSmem = kSDy + kRows * 4;
}  // namespace tr

// Everything of a training step that is local to a row, 16 rows a CTA: both
// layers, the head, the output error, and the gradients entering both hidden
// layers.  W1 and W2 are staged once by bulk copies (W2 serves the second layer
// and, transposed by ldmatrix, its backward).  Writes H1, H2, dZ2, dZ1 and the
// errors for train_weights_kernel.  With count, CTA 0 advances the Adam step.
//
// Bound: the chain staging -> layer 1 -> layer 2 -> head -> dZ2 -> dZ1 on a few
// CTAs.  The two kernels replaced thirteen launches (products, head, the output
// layer's backward on one block, transposes, sums, Adam and its counter): eight
// steps on 64 rows, with the copies to and from the host around them, took
// 765 us and take 206.
__global__ void __launch_bounds__(tr::kThreads, 1) train_rows_kernel(const bf16* __restrict__ X,
                                                                   const int* __restrict__ idx,
                                                                   const float* __restrict__ t, int B,
                                                                   const bf16* __restrict__ W1u,
                                                                   const bf16* __restrict__ W2u,
                                                                   const float* __restrict__ params,
                                                                   bf16* __restrict__ H1, float* __restrict__ H2,
                                                                   bf16* __restrict__ dZ2, bf16* __restrict__ dZ1,
                                                                   float* __restrict__ dZ1f, float* __restrict__ err,
                                                                   int* __restrict__ step, int count) {
  using namespace tr;
  extern __shared__ __align__(1024) unsigned char s_tr[];
  __shared__ alignas(8) unsigned long long s_bars[2];      // W1 staged, W2 staged
  bf16* const W2s = reinterpret_cast<bf16*>(s_tr);
  bf16* const W1s = reinterpret_cast<bf16*>(s_tr + kSW1);
  bf16* const Xs = reinterpret_cast<bf16*>(s_tr + kSX);
  bf16* const H1s = reinterpret_cast<bf16*>(s_tr + kSH1);
  bf16* const D2s = reinterpret_cast<bf16*>(s_tr + kSD2);
  float* const H2s = reinterpret_cast<float*>(s_tr + kSH2);
  float* const dys = reinterpret_cast<float*>(s_tr + kSDy);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, q = lane & 3;                   // accumulator rows g, g + 8, columns 2q, 2q + 1
  const int r0 = blockIdx.x * kRows, n0 = 32 * warp;
  const unsigned bar1 = smem_u32(&s_bars[0]), bar2 = smem_u32(&s_bars[1]);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar2) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    constexpr uint32_t w1 = kHidden * kFeatures * 2, w2 = kHidden * kHidden * 2;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar1), "r"(w1) : "memory");
    bulk_copy(W1s, W1u, w1, bar1);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar2), "r"(w2) : "memory");
    for (uint32_t c = 0; c < w2; c += 16384u)
      bulk_copy(s_tr + c, reinterpret_cast<const unsigned char*>(W2u) + c, 16384u, bar2);
    if (count && blockIdx.x == 0) *step += 1;
  }
  if (tid < kRows * (kFeatures / 8)) {
    const int r = tid / (kFeatures / 8), c = (tid % (kFeatures / 8)) * 8;
    const int src = idx ? idx[r0 + r] : r0 + r;
    *reinterpret_cast<uint4*>(Xs + umma_k_off(r, c, kFeatures)) =
        *reinterpret_cast<const uint4*>(X + (long long)src * kFeatures + c);
  }
  float b1v[4][2], b2v[4][2];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      b1v[nt][e] = params[kOffB1 + n0 + 8 * nt + 2 * q + e];
      b2v[nt][e] = params[kOffB2 + n0 + 8 * nt + 2 * q + e];
    }
  const float w3n = params[kOffW3 + tid], b3 = params[kOffB3];
  float w3l[kHidden / 32];
#pragma unroll
  for (int i = 0; i < kHidden / 32; ++i) w3l[i] = params[kOffW3 + lane + 32 * i];
  __syncthreads();
  // layer 1
  bool ok = mbar_wait_bounded(bar1, 0u);
  float acc[4][4];
  auto clear = [&]() {
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
  };
  clear();
  warp_product<false>(acc, Xs, kFeatures, W1s, kFeatures, n0, kFeatures);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = g + 8 * h, n = n0 + 8 * nt + 2 * q;
      const float v0 = acc[nt][2 * h] + b1v[nt][0], v1 = acc[nt][2 * h + 1] + b1v[nt][1];
      __nv_bfloat162 o;
      o.x = __float2bfloat16_rn(v0 > 0.f ? v0 : 0.f);
      o.y = __float2bfloat16_rn(v1 > 0.f ? v1 : 0.f);
      *reinterpret_cast<__nv_bfloat162*>(H1s + umma_k_off(r, n, kHidden)) = o;
      *reinterpret_cast<__nv_bfloat162*>(H1 + (size_t)(r0 + r) * kHidden + n) = o;
    }
  __syncthreads();
  // layer 2
  ok = mbar_wait_bounded(bar2, 0u) && ok;
  clear();
  warp_product<false>(acc, H1s, kHidden, W2s, kHidden, n0, kHidden);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = g + 8 * h, n = n0 + 8 * nt + 2 * q;
      const float v0 = acc[nt][2 * h] + b2v[nt][0], v1 = acc[nt][2 * h + 1] + b2v[nt][1];
      const float2 o = make_float2(v0 > 0.f ? v0 : 0.f, v1 > 0.f ? v1 : 0.f);
      *reinterpret_cast<float2*>(H2s + r * kPitch + n) = o;
      *reinterpret_cast<float2*>(H2 + (size_t)(r0 + r) * kHidden + n) = o;
    }
  __syncthreads();
  // head: y = H2 . w3 + b3, one warp per row; then the output error
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = warp + 8 * h;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < kHidden / 32; ++i) s = fmaf(H2s[r * kPitch + lane + 32 * i], w3l[i], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const float y = s + b3;
      const float d = y - t[r0 + r];
      const float dy = 2.f * d / (float)B;
      dys[r] = dy;
      err[r0 + r] = ok ? dy : __int_as_float(0x7fc00000);
      err[kMaxTrainRows + r0 + r] = d;
    }
  }
  __syncthreads();
  // dZ2: thread n owns hidden unit n
#pragma unroll 4
  for (int r = 0; r < kRows; ++r) {
    const bf16 db = __float2bfloat16_rn(H2s[r * kPitch + tid] > 0.f ? dys[r] * w3n : 0.f);
    D2s[umma_k_off(r, tid, kHidden)] = db;
    dZ2[(size_t)(r0 + r) * kHidden + tid] = db;
  }
  __syncthreads();
  // dZ1 = (dZ2 W2) where H1 > 0
  clear();
  warp_product<true>(acc, D2s, kHidden, W2s, kHidden, n0, kHidden);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = g + 8 * h, n = n0 + 8 * nt + 2 * q;
      const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162*>(H1s + umma_k_off(r, n, kHidden));
      const float v0 = __bfloat162float(m.x) > 0.f ? acc[nt][2 * h] : 0.f;
      const float v1 = __bfloat162float(m.y) > 0.f ? acc[nt][2 * h + 1] : 0.f;
      __nv_bfloat162 o;
      o.x = __float2bfloat16_rn(v0);
      o.y = __float2bfloat16_rn(v1);
      const size_t at = (size_t)(r0 + r) * kHidden + n;
      *reinterpret_cast<__nv_bfloat162*>(dZ1 + at) = o;
      *reinterpret_cast<float2*>(dZ1f + at) = make_float2(v0, v1);
    }
}

// The BF16 copies of parameter i (value v) that the products read: W1 and W2
// in the operand layout.
__device__ __forceinline__ void store_bf16_copies(int i, float v, bf16* __restrict__ w1u, bf16* __restrict__ w2u) {
  if (i < kOffB1) {
    w1u[umma_k_off(i / kFeatures, i % kFeatures, kFeatures)] = __float2bfloat16_rn(v);
  } else if (i >= kOffW2 && i < kOffB2) {
    const int q = i - kOffW2;
    w2u[umma_k_off(q / kHidden, q % kHidden, kHidden)] = __float2bfloat16_rn(v);
  }
}

// What becomes of a gradient: written out, or one Adam step on the FP32 master
// parameter (the step count was advanced by the row pass) and its BF16 copies.
struct GradSink {
  float* g;                  // null: Adam
  float *p, *m1, *m2;
  const int* step;
  AdamHyper h;
  bf16 *w1u, *w2u;
};

struct AdamScale {
  float c1, c2;
  __device__ __forceinline__ explicit AdamScale(const GradSink& s) {
    const int t = s.g ? 1 : *s.step;
    c1 = 1.f / (1.f - powf(s.h.beta1, (float)t));
    c2 = 1.f / (1.f - powf(s.h.beta2, (float)t));
  }
};

__device__ __forceinline__ void sink_gradient(const GradSink& s, const AdamScale& c, int i, float gi, float m1i,
                                              float m2i, float p0) {
  if (s.g) {
    s.g[i] = gi;
    return;
  }
  const float a = s.h.beta1 * m1i + (1.f - s.h.beta1) * gi;
  const float b = s.h.beta2 * m2i + (1.f - s.h.beta2) * gi * gi;
  s.m1[i] = a;
  s.m2[i] = b;
  const float pi = p0 - s.h.lr * (a * c.c1) / (sqrtf(b * c.c2) + s.h.eps);
  s.p[i] = pi;
  store_bf16_copies(i, pi, s.w1u, s.w2u);
}

// The sums over the rows, and what becomes of them.  Blocks 0 .. 127: 16 x 32
// tiles of gW2[n][k] = sum_r dZ2[r][n] H1[r][k], a 16 x 8 tile a warp; blocks
// 128 .. 143: 16 x 32 rows of gW1[k][j] = sum_r dZ1[r][k] X[r][j]; block 144:
// the FP32 sums of w3, b2, b3 and the loss; block 145: b1.  The products run
// over r in steps of 16, the sums one row after the other.  The operands are
// staged row by row and transposed by ldmatrix, so no transposed copy exists.
constexpr int kWeightBlocks = 146;
__global__ void __launch_bounds__(128) train_weights_kernel(const bf16* __restrict__ X, const int* __restrict__ idx,
                                                            int B, const bf16* __restrict__ H1,
                                                            const float* __restrict__ H2,
                                                            const bf16* __restrict__ dZ2,
                                                            const bf16* __restrict__ dZ1,
                                                            const float* __restrict__ dZ1f,
                                                            const float* __restrict__ err, GradSink s,
                                                            float* __restrict__ loss) {
  // rows of 16 + 8 and 32 + 8 columns: ldmatrix's eight rows fall on different banks
  constexpr int kPA = 24, kPB = 40;
  __shared__ __align__(16) bf16 As[kMaxTrainRows * kPA];
  __shared__ __align__(16) bf16 Bs[kMaxTrainRows * kPB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = blockIdx.x;
  if (blk < 144) {
    const bool w2 = blk < 128;
    const int m0 = w2 ? (blk >> 3) * 16 : (blk - 128) * 16;   // rows of the gradient
    const int c0 = w2 ? (blk & 7) * 32 : 0;                   // its first column here
    const int ld = w2 ? kHidden : kFeatures, off = w2 ? kOffW2 : kOffW1;
    const bf16* const A = w2 ? dZ2 : dZ1;
    for (int i = tid; i < B * 2; i += 128)
      *reinterpret_cast<uint4*>(As + (i >> 1) * kPA + 8 * (i & 1)) =
          *reinterpret_cast<const uint4*>(A + (size_t)(i >> 1) * kHidden + m0 + 8 * (i & 1));
    for (int i = tid; i < B * 4; i += 128) {
      const int r = i >> 2;
      const bf16* row = w2 ? H1 + (size_t)r * kHidden + c0 : X + (long long)(idx ? idx[r] : r) * kFeatures;
      *reinterpret_cast<uint4*>(Bs + r * kPB + 8 * (i & 3)) = *reinterpret_cast<const uint4*>(row + 8 * (i & 3));
    }
    // the parameters this lane will update, while the rows arrive
    const int gr = lane >> 2, q = lane & 3, n0 = 8 * warp;
    int at[4];
    float m1v[4], m2v[4], pv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      at[i] = off + (m0 + gr + (i >= 2 ? 8 : 0)) * ld + c0 + n0 + 2 * q + (i & 1);
      if (!s.g) {
        m1v[i] = s.m1[at[i]];
        m2v[i] = s.m2[at[i]];
        pv[i] = s.p[at[i]];
      } else {
        m1v[i] = m2v[i] = pv[i] = 0.f;
      }
    }
    const AdamScale c(s);
    __syncthreads();
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const int i = lane >> 3, r = lane & 7;
    for (int k0 = 0; k0 < B; k0 += 16) {
      // A[m][k] = As[k][m]: (m 0-7, k 0-7), (m 8-15, k 0-7), (m 0-7, k 8-15), (m 8-15, k 8-15)
      uint32_t a[4], b[4];
      ldmatrix4<true>(a, smem_u32(As + (k0 + 8 * (i >> 1) + r) * kPA + 8 * (i & 1)));
      // B[k][n] = Bs[k][n]: (k 0-7), (k 8-15); the other two addresses repeat them
      ldmatrix4<true>(b, smem_u32(Bs + (k0 + 8 * (i & 1) + r) * kPB + n0));
      mma_16816(acc, a[0], a[1], a[2], a[3], b[0], b[1]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) sink_gradient(s, c, at[j], acc[j], m1v[j], m2v[j], pv[j]);
    return;
  }
  // FP32 sums, one row after the other; thread n owns units n and n + 128
  const AdamScale c(s);
  auto sink = [&](int i, float gi) {
    if (s.g) sink_gradient(s, c, i, gi, 0.f, 0.f, 0.f);
    else sink_gradient(s, c, i, gi, s.m1[i], s.m2[i], s.p[i]);
  };
  if (blk == 144) {
    __shared__ float s_dy[kMaxTrainRows], s_d[kMaxTrainRows];
    for (int r = tid; r < B; r += 128) {
      s_dy[r] = err[r];
      s_d[r] = err[kMaxTrainRows + r];
    }
    __syncthreads();
    const float w3a = s.p[kOffW3 + tid], w3b = s.p[kOffW3 + 128 + tid];
    float gw0 = 0.f, gw1 = 0.f, gb0 = 0.f, gb1 = 0.f;
#pragma unroll 16
    for (int r = 0; r < B; ++r) {
      const float dy = s_dy[r];
      const float h0 = H2[(size_t)r * kHidden + tid], h1 = H2[(size_t)r * kHidden + 128 + tid];
      gw0 = fmaf(dy, h0, gw0);
      gw1 = fmaf(dy, h1, gw1);
      gb0 = __fadd_rn(gb0, h0 > 0.f ? __fmul_rn(dy, w3a) : 0.f);
      gb1 = __fadd_rn(gb1, h1 > 0.f ? __fmul_rn(dy, w3b) : 0.f);
    }
    sink(kOffW3 + tid, gw0);
    sink(kOffW3 + 128 + tid, gw1);
    sink(kOffB2 + tid, gb0);
    sink(kOffB2 + 128 + tid, gb1);
    if (tid == 0) {
      float gb3 = 0.f, l = 0.f;
      for (int r = 0; r < B; ++r) {
        gb3 += s_dy[r];
        l = fmaf(s_d[r], s_d[r], l);
      }
      sink(kOffB3, gb3);
      *loss = l / (float)B;
    }
  } else {
    float g0 = 0.f, g1 = 0.f;
#pragma unroll 16
    for (int r = 0; r < B; ++r) {
      g0 += dZ1f[(size_t)r * kHidden + tid];
      g1 += dZ1f[(size_t)r * kHidden + 128 + tid];
    }
    sink(kOffB1 + tid, g0);
    sink(kOffB1 + 128 + tid, g1);
  }
}

// BF16 copies of freshly written FP32 parameters.
__global__ void cast_params_kernel(const float* __restrict__ p, bf16* __restrict__ w1u, bf16* __restrict__ w2u) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x)
    store_bf16_copies(i, p[i], w1u, w2u);
}

// FP32 features rounded to BF16 rows, four a thread.
__global__ void cast_rows_kernel(const float4* __restrict__ x, uint2* __restrict__ out, int n4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 v = x[i];
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  out[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

}  // namespace mlp

using namespace mlp;

// ---- enqueue helpers the annealing engine uses ---------------------------------

int mlp_forward(ggb_mlp* m, const bf16* X, int rows, float* y, cudaStream_t st) {
  if (rows % 16 || rows > m->max_rows) return core_fail(GGB_EINVAL, "mlp rows %d (max %d, multiple of 16)", rows, m->max_rows);
  // one fused launch on the tcgen05 tensor cores, the activations never leave the SM
  forward_tc_kernel<<<(rows + tc::kRows - 1) / tc::kRows, tc::kThreads, tc::kSmem, st>>>(X, rows, m->W1u, m->W2u, m->p,
                                                                                       y);
  core_add_launches(1);
  MCUDA(cudaGetLastError());
  return GGB_OK;
}

int mlp_step(ggb_mlp* m, const bf16* X, const int* idx, const float* t, int B, bool adam, cudaStream_t st) {
  if (B % 16 || B > kMaxTrainRows || (!idx && B > m->max_rows)) return core_fail(GGB_EINVAL, "mlp training rows %d", B);
  train_rows_kernel<<<B / tr::kRows, tr::kThreads, tr::kSmem, st>>>(X, idx, t, B, m->W1u, m->W2u, m->p, m->H1, m->H2,
                                                                   m->dZ2, m->dZ1, m->dZ1f, m->err, m->step,
                                                                   adam ? 1 : 0);
  const GradSink sink = {adam ? nullptr : m->g, m->p, m->m1, m->m2, m->step, m->hyper, m->W1u, m->W2u};
  train_weights_kernel<<<kWeightBlocks, 128, 0, st>>>(X, idx, B, m->H1, m->H2, m->dZ2, m->dZ1, m->dZ1f, m->err, sink,
                                                      m->loss);
  core_add_launches(2);
  MCUDA(cudaGetLastError());
  return GGB_OK;
}

size_t mlp_state_bytes() { return 3 * (size_t)kParams * sizeof(float) + sizeof(int); }

int mlp_save_state(ggb_mlp* m, void* host) {
  unsigned char* h = static_cast<unsigned char*>(host);
  const size_t pb = (size_t)kParams * sizeof(float);
  MCUDA(cudaDeviceSynchronize());
  MCUDA(cudaMemcpy(h, m->p, pb, cudaMemcpyDeviceToHost));
  MCUDA(cudaMemcpy(h + pb, m->m1, pb, cudaMemcpyDeviceToHost));
  MCUDA(cudaMemcpy(h + 2 * pb, m->m2, pb, cudaMemcpyDeviceToHost));
  MCUDA(cudaMemcpy(h + 3 * pb, m->step, sizeof(int), cudaMemcpyDeviceToHost));
  return GGB_OK;
}

int mlp_load_state(ggb_mlp* m, const void* host) {
  const unsigned char* h = static_cast<const unsigned char*>(host);
  const size_t pb = (size_t)kParams * sizeof(float);
  MCUDA(cudaDeviceSynchronize());
  MCUDA(cudaMemcpy(m->p, h, pb, cudaMemcpyHostToDevice));
  MCUDA(cudaMemcpy(m->m1, h + pb, pb, cudaMemcpyHostToDevice));
  MCUDA(cudaMemcpy(m->m2, h + 2 * pb, pb, cudaMemcpyHostToDevice));
  MCUDA(cudaMemcpy(m->step, h + 3 * pb, sizeof(int), cudaMemcpyHostToDevice));
  cast_params_kernel<<<64, 256>>>(m->p, m->W1u, m->W2u);
  MCUDA(cudaGetLastError());
  MCUDA(cudaDeviceSynchronize());
  return GGB_OK;
}

}  // namespace ggb

namespace {

using ggb::mlp::bf16;

template <typename T>
int mdev(T** p, size_t n) {
  if (cudaMalloc(p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return core_fail(GGB_ENOMEM, "cudaMalloc of %zu bytes failed", n * sizeof(T));
  }
  return GGB_OK;
}

// He-uniform initial weights, zero biases, from a splitmix64 stream.
void init_params(std::vector<float>& p, unsigned long long seed) {
  unsigned long long s = seed ^ 0x6a09e667f3bcc909ULL;
  auto next = [&]() {
    s += 0x9e3779b97f4a7c15ULL;
    unsigned long long z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  p.assign(ggb::mlp::kParams, 0.f);
  const double a1 = std::sqrt(6.0 / ggb::mlp::kFeatures), a2 = std::sqrt(6.0 / ggb::mlp::kHidden);
  for (int i = 0; i < ggb::mlp::kOffB1; ++i) p[i] = (float)((2.0 * next() - 1.0) * a1);
  for (int i = ggb::mlp::kOffW2; i < ggb::mlp::kOffB2; ++i) p[i] = (float)((2.0 * next() - 1.0) * a2);
  for (int i = ggb::mlp::kOffW3; i < ggb::mlp::kOffB3; ++i) p[i] = (float)((2.0 * next() - 1.0) * a2 * 0.1);
}

int create(ggb_mlp* m, int max_rows, unsigned long long seed) {
  using namespace ggb::mlp;
  m->max_rows = max_rows;
  int rc;
  MCUDA(cudaFuncSetAttribute((const void*)forward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)tc::kSmem));
  MCUDA(cudaFuncSetAttribute((const void*)train_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)tr::kSmem));
  const size_t R = (size_t)max_rows, T = (size_t)kMaxTrainRows * kHidden;
  if ((rc = mdev(&m->p, kParams)) || (rc = mdev(&m->g, kParams)) || (rc = mdev(&m->m1, kParams)) ||
      (rc = mdev(&m->m2, kParams)) || (rc = mdev(&m->step, 1)) || (rc = mdev(&m->W1u, (size_t)kOffB1)) ||
      (rc = mdev(&m->W2u, (size_t)kHidden * kHidden)) || (rc = mdev(&m->H1, T)) || (rc = mdev(&m->H2, T)) ||
      (rc = mdev(&m->dZ2, T)) || (rc = mdev(&m->dZ1, T)) || (rc = mdev(&m->dZ1f, T)) ||
      (rc = mdev(&m->err, 2 * (size_t)kMaxTrainRows)) || (rc = mdev(&m->loss, 1)) ||
      (rc = mdev(&m->X, R * kFeatures)) || (rc = mdev(&m->xf, R * kFeatures)) || (rc = mdev(&m->y, R)) ||
      (rc = mdev(&m->t, (size_t)kMaxTrainRows)))
    return rc;
  std::vector<float> p;
  init_params(p, seed);
  return ggb_mlp_set_params(m, p.data());
}

void destroy(ggb_mlp* m) {
  if (!m) return;
  for (void* q : {(void*)m->p, (void*)m->g, (void*)m->m1, (void*)m->m2, (void*)m->step, (void*)m->W1u, (void*)m->W2u,
                  (void*)m->H1, (void*)m->H2, (void*)m->dZ2, (void*)m->dZ1, (void*)m->dZ1f, (void*)m->err,
                  (void*)m->loss, (void*)m->X, (void*)m->xf, (void*)m->y, (void*)m->t})
    cudaFree(q);
  cudaGetLastError();
  delete m;
}

// Host FP32 features -> device BF16 rows of m->X (rounded on the device; on the
// host the rounding of 4096 rows took longer than the forward).
int upload_x(ggb_mlp* m, const float* x, int rows) {
  const int n4 = rows * ggb::mlp::kFeatures / 4;
  MCUDA(cudaMemcpy(m->xf, x, (size_t)rows * ggb::mlp::kFeatures * sizeof(float), cudaMemcpyHostToDevice));
  ggb::mlp::cast_rows_kernel<<<(n4 + 255) / 256, 256>>>(reinterpret_cast<const float4*>(m->xf),
                                                       reinterpret_cast<uint2*>(m->X), n4);
  ggb::core_add_launches(1);
  MCUDA(cudaGetLastError());
  return GGB_OK;
}

}  // namespace

extern "C" {

int ggb_mlp_create(int max_rows, unsigned long long seed, ggb_mlp** out) {
  if (!out || max_rows <= 0 || max_rows % 16) return core_fail(GGB_EINVAL, "max_rows must be a positive multiple of 16");
  *out = nullptr;
  ggb_mlp* m = new ggb_mlp();
  m->hyper = {1e-3f, 0.9f, 0.999f, 1e-8f};
  int rc = create(m, max_rows, seed);
  if (rc) {
    destroy(m);
    return rc;
  }
  *out = m;
  return GGB_OK;
}

void ggb_mlp_destroy(ggb_mlp* m) { destroy(m); }

int ggb_mlp_param_count(void) { return ggb::mlp::kParams; }

int ggb_mlp_set_params(ggb_mlp* m, const float* params) {
  using namespace ggb::mlp;
  if (!m || !params) return core_fail(GGB_EINVAL, "null pointer");
  MCUDA(cudaMemcpy(m->p, params, kParams * sizeof(float), cudaMemcpyHostToDevice));
  MCUDA(cudaMemset(m->m1, 0, kParams * sizeof(float)));
  MCUDA(cudaMemset(m->m2, 0, kParams * sizeof(float)));
  MCUDA(cudaMemset(m->step, 0, sizeof(int)));
  cast_params_kernel<<<64, 256>>>(m->p, m->W1u, m->W2u);
  MCUDA(cudaGetLastError());
  MCUDA(cudaDeviceSynchronize());
  return GGB_OK;
}

int ggb_mlp_get_params(ggb_mlp* m, float* params) {
  if (!m || !params) return core_fail(GGB_EINVAL, "null pointer");
  MCUDA(cudaDeviceSynchronize());
  MCUDA(cudaMemcpy(params, m->p, ggb::mlp::kParams * sizeof(float), cudaMemcpyDeviceToHost));
  return GGB_OK;
}

int ggb_mlp_set_adam(ggb_mlp* m, float lr, float beta1, float beta2, float eps) {
  if (!m || !(lr > 0.f) || !(beta1 >= 0.f && beta1 < 1.f) || !(beta2 >= 0.f && beta2 < 1.f) || !(eps > 0.f))
    return core_fail(GGB_EINVAL, "bad Adam hyper-parameters");
  m->hyper = {lr, beta1, beta2, eps};
  return GGB_OK;
}

int ggb_mlp_forward_host(ggb_mlp* m, const float* x, int rows, float* y) {
  if (!m || !x || !y) return core_fail(GGB_EINVAL, "null pointer");
  if (rows <= 0 || rows % 16 || rows > m->max_rows) return core_fail(GGB_EINVAL, "rows must be a multiple of 16 up to max_rows");
  int rc = upload_x(m, x, rows);
  if (rc) return rc;
  rc = ggb::mlp_forward(m, m->X, rows, m->y, nullptr);
  if (rc) return rc;
  MCUDA(cudaMemcpy(y, m->y, (size_t)rows * sizeof(float), cudaMemcpyDeviceToHost));
  return GGB_OK;
}

int ggb_mlp_time_forward(ggb_mlp* m, const float* x, int rows, int reps, double* ms) {
  if (!m || !x || !ms) return core_fail(GGB_EINVAL, "null pointer");
  if (rows <= 0 || rows % 16 || rows > m->max_rows || reps <= 0)
    return core_fail(GGB_EINVAL, "rows must be a multiple of 16 up to max_rows, reps positive");
  int rc = upload_x(m, x, rows);
  if (rc) return rc;
  MCUDA(cudaStreamSynchronize(nullptr));   // the timing stream below does not wait for the upload's
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  float t = 0.f;
  if (e == cudaSuccess) {
    rc = ggb::mlp_forward(m, m->X, rows, m->y, st);   // warm-up
    if (rc == GGB_OK) e = cudaEventRecord(e0, st);
    for (int i = 0; i < reps && rc == GGB_OK && e == cudaSuccess; ++i)
      rc = ggb::mlp_forward(m, m->X, rows, m->y, st);
    if (rc == GGB_OK && e == cudaSuccess) e = cudaEventRecord(e1, st);
    if (rc == GGB_OK && e == cudaSuccess) e = cudaEventSynchronize(e1);
    if (rc == GGB_OK && e == cudaSuccess) e = cudaEventElapsedTime(&t, e0, e1);
  }
  if (e1) cudaEventDestroy(e1);
  if (e0) cudaEventDestroy(e0);
  if (st) {
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
  }
  if (rc) return rc;
  if (e != cudaSuccess) return core_fail(GGB_ECUDA, "forward timing: %s", cudaGetErrorString(e));
  *ms = (double)t / reps;
  return GGB_OK;
}

int ggb_mlp_grads_host(ggb_mlp* m, const float* x, const float* t, int rows, float* loss, float* grads) {
  if (!m || !x || !t || !grads) return core_fail(GGB_EINVAL, "null pointer");
  if (rows <= 0 || rows % 16 || rows > ggb::mlp::kMaxTrainRows || rows > m->max_rows)
    return core_fail(GGB_EINVAL, "training rows must be a multiple of 16 up to %d", ggb::mlp::kMaxTrainRows);
  int rc = upload_x(m, x, rows);
  if (rc) return rc;
  MCUDA(cudaMemcpy(m->t, t, (size_t)rows * sizeof(float), cudaMemcpyHostToDevice));
  rc = ggb::mlp_step(m, m->X, nullptr, m->t, rows, false, nullptr);
  if (rc) return rc;
  MCUDA(cudaDeviceSynchronize());
  MCUDA(cudaMemcpy(grads, m->g, ggb::mlp::kParams * sizeof(float), cudaMemcpyDeviceToHost));
  if (loss) MCUDA(cudaMemcpy(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
  return GGB_OK;
}

int ggb_mlp_train_host(ggb_mlp* m, const float* x, const float* t, int rows, int steps, float* last_loss) {
  if (!m || !x || !t) return core_fail(GGB_EINVAL, "null pointer");
  if (rows <= 0 || rows % 16 || rows > ggb::mlp::kMaxTrainRows || rows > m->max_rows || steps <= 0)
    return core_fail(GGB_EINVAL, "training rows must be a multiple of 16 up to %d", ggb::mlp::kMaxTrainRows);
  int rc = upload_x(m, x, rows);
  if (rc) return rc;
  MCUDA(cudaMemcpy(m->t, t, (size_t)rows * sizeof(float), cudaMemcpyHostToDevice));
  for (int s = 0; s < steps; ++s) {
    rc = ggb::mlp_step(m, m->X, nullptr, m->t, rows, true, nullptr);
    if (rc) return rc;
  }
  MCUDA(cudaDeviceSynchronize());
  if (last_loss) MCUDA(cudaMemcpy(last_loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
  return GGB_OK;
}

}  // extern "C"
