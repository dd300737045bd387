// ci_gemm.cu -- BF16 tensor-core GEMM on sm_103a (tcgen05 + TMEM), FP32 accumulation.
//
//   C[M x N] (+)= alpha * op(A)[M x K] * op(B)[K x N]  (+ bias[N]) (then optional tanh)
//
// A, B are BF16 in global memory, row-major with leading dimensions lda/ldb; op() is a
// transpose flag per operand.  C is FP32 (row-major, ldc); an optional BF16 copy of C
// is written for the next layer.  This is the dense contraction of the surrogate (POD
// projections and the MLP's forward/backward passes); the impact step itself has none.
//
// The kernels read both operands K-major (A B^T) by TMA (cp.async.bulk.tensor, 128-byte
// swizzle): 128 x 64 and BN x 64 tiles through a shared-memory ring, one thread issuing the
// loads, one the tcgen05.mma, mbarriers handing stages back and forth (full: TMA bytes
// landed; empty: the MMAs reading a stage completed), accumulators in TMEM:
//   k_gemm_tma_pers  one CTA per SM walking the output tiles, two TMEM accumulators so the
//                    epilogue of one tile overlaps the MMAs of the next
//   k_gemm_stream    a long A past a narrow B: equal unit ranges per SM, rows off 16-byte
//                    boundaries in classes
//   k_gemm_tma       split K (few output tiles, long K): one CTA per (tile, K range)
// Operands that TMA cannot read (another transpose, rows off 16-byte boundaries) are copied
// (k_pack_bf16) or, in k_gemm_stream's A, read in place.  What the copies do not cover (see
// choose_operands) goes through k_gemm_bf16: one CTA computes a 128 x BN tile (BN = 64 or
// 128).  Per K-tile of 64:
//  1. all 128 threads stage A (128 x 64) and B (BN x 64) as K-major BF16 in shared
//     memory, in the canonical no-swizzle layout of 8-row x 16-byte core matrices
//     (core matrix (r/8, k/8) at r/8 * SBO + k/8 * LBO, LBO = 128 B, SBO = 1024 B);
//  2. fence.proxy.async makes the writes visible to the tensor core; one elected
//     thread issues 4 x tcgen05.mma.kind::f16 (K = 16 each) into the TMEM accumulator
//     and commits to an mbarrier;
//  3. every thread waits on the mbarrier (bounded spin: on timeout the kernel records
//     an error flag, frees its TMEM and returns) before the stage is overwritten.
// The epilogues read the accumulator with tcgen05.ld (each warp its 32 TMEM lanes =
// 32 rows), apply alpha, beta, bias, tanh and store.
#include <cuda.h>  // CUtensorMap and its enums; the encoder is fetched at run time
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/cppimpact_gb300.h"
#include "ci_pdl.h"

namespace ci {
int set_last_error(int code, const char* msg);
}

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr unsigned kSpinLimit = 1u << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor: start address, leading / stride byte
// offsets (all >> 4), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // version
  return d;                // base offset 0, lbo mode 0, layout 0 (no swizzle)
}

// Instruction descriptor of tcgen05.mma.kind::f16: D FP32, A and B BF16, both K-major,
// N >> 3 and M >> 4.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N) {
  return (1u << 4)      // D format F32
         | (1u << 7)    // A format BF16
         | (1u << 10)   // B format BF16
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  for (unsigned it = 0; it < kSpinLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}

// byte offset of element (r, k) of a K-major no-swizzle tile (LBO 128, SBO 1024)
__device__ __forceinline__ uint32_t kmajor_off(int r, int k) {
  return (uint32_t)((r >> 3) * 1024 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

template <int BN>
__global__ void __launch_bounds__(128) k_gemm_bf16(const __nv_bfloat16* __restrict__ A, int lda,
                                                   int transA, const __nv_bfloat16* __restrict__ B,
                                                   int ldb, int transB, float* C, int ldc,
                                                   __nv_bfloat16* Cb, int M, int N, int K,
                                                   float alpha, float beta,
                                                   const float* __restrict__ bias, int act,
                                                   int* err, int k_chunk, float* partial) {
  __shared__ __align__(1024) uint8_t sA[BM * BK * 2];
  __shared__ __align__(1024) uint8_t sB[BN * BK * 2];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  // split-K: this CTA reduces K range [kb, ke); partial results go to partial[z]
  const int kb = blockIdx.z * k_chunk;
  const int ke = min(K, kb + k_chunk);

  if (warp == 0) {
    // TMEM: BN columns (power of two >= 32) for the 128 x BN FP32 accumulator
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_base;
  const uint32_t idesc = instr_desc(BM, BN);
  bool ok = true;
  uint32_t phase = 0;
  const int ktiles = (ke - kb + BK - 1) / BK;
  for (int kt = 0; kt < ktiles && ok; kt++) {
    const int k0 = kb + kt * BK;
    // stage A: 128 rows x 64 k; consecutive threads read consecutive addresses
    for (int i = tid; i < BM * BK; i += 128) {
      const int r = transA ? i % BM : i / BK, k = transA ? i / BM : i % BK;
      const int gm = m0 + r, gk = k0 + k;
      __nv_bfloat16 v = __float2bfloat16(0.f);
      if (gm < M && gk < ke) v = transA ? A[(size_t)gk * lda + gm] : A[(size_t)gm * lda + gk];
      *reinterpret_cast<__nv_bfloat16*>(sA + kmajor_off(r, k)) = v;
    }
    // stage B as K-major rows n: B_op[k][n]
    for (int i = tid; i < BN * BK; i += 128) {
      const int n = transB ? i / BK : i % BN, k = transB ? i % BK : i / BN;
      const int gn = n0 + n, gk = k0 + k;
      __nv_bfloat16 v = __float2bfloat16(0.f);
      if (gn < N && gk < ke) v = transB ? B[(size_t)gn * ldb + gk] : B[(size_t)gk * ldb + gn];
      *reinterpret_cast<__nv_bfloat16*>(sB + kmajor_off(n, k)) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int kk = 0; kk < BK / 16; kk++) {
        // K = 16 per MMA = two core matrices along K = 2 x LBO bytes
        const uint64_t da = smem_desc(smem_u32(sA) + kk * 256, 128, 1024);
        const uint64_t db = smem_desc(smem_u32(sB) + kk * 256, 128, 1024);
        const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(da), "l"(db), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
              smem_u32(&bar))
          : "memory");
    }
    // CTA-uniform outcome: every thread leaves the loop at the same tile
    ok = __syncthreads_and(mbar_wait(smem_u32(&bar), phase)) != 0;
    phase ^= 1u;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  }
  if (!ok) {
    // give the MMAs in flight one more bounded wait before the TMEM is freed
    mbar_wait(smem_u32(&bar), phase ^ 1u);
    if (tid == 0) atomicExch(err, 1);
  } else {
    // epilogue: warp w holds TMEM lanes [32w, 32w+32) = tile rows; 8 columns per load
    const int row = m0 + warp * 32 + lane;
    for (int c = 0; c < BN; c += 8) {
      uint32_t r[8];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
            "=r"(r[7])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      if (row < M && partial) {
        float* pr = partial + ((size_t)blockIdx.z * M + row) * N;
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (n0 + c + j < N) pr[n0 + c + j] = ktiles > 0 ? __uint_as_float(r[j]) : 0.f;
      } else if (row < M) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int col = n0 + c + j;
          if (col >= N) continue;
          float v = alpha * __uint_as_float(r[j]);
          if (beta != 0.f) v += beta * C[(size_t)row * ldc + col];
          if (bias) v += bias[col];
          if (act == 1) v = tanhf(v);
          C[(size_t)row * ldc + col] = v;
          if (Cb) Cb[(size_t)row * ldc + col] = __float2bfloat16(v);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(BN)
                 : "memory");
}

constexpr int TBK = 64;      // K per stage: 64 BF16 = one 128-byte swizzle row
constexpr int TSTAGES = 4;

// Shared-memory descriptor of a K-major tile in the 128-byte swizzled layout TMA writes
// (rows of 128 bytes, 8-row groups 1024 bytes apart); LBO is unused for this layout.
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;            // LBO (ignored) = 16 B
  d |= (uint64_t)(1024 >> 4) << 32;  // SBO: 8 rows x 128 B
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)2 << 61;            // 128-byte swizzle
  return d;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

template <int BN>
__global__ void __launch_bounds__(128, 1)
    k_gemm_tma(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               float* C, int ldc, __nv_bfloat16* Cb, int M, int N, int K, float alpha, float beta,
               const float* __restrict__ bias, int act, int* err, int k_chunk, float* partial) {
  constexpr int A_BYTES = BM * TBK * 2;
  constexpr int B_BYTES = BN * TBK * 2;
  extern __shared__ uint8_t smem_raw[];
  // the swizzled tiles want 1024-byte alignment (the launch reserves the slack)
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + TSTAGES * A_BYTES;
  __shared__ __align__(8) uint64_t full[TSTAGES], empty[TSTAGES], done;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int kb = blockIdx.z * k_chunk;
  const int ke = min(K, kb + k_chunk);
  const int ktiles = (ke - kb + TBK - 1) / TBK;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < TSTAGES; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[s])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  ci::pdl_next();
  ci::pdl_wait();
  const uint32_t tmem = tmem_base;
  bool ok = true;
  int issued = 0;
  if (warp == 0 && lane == 0) {
    // producer: stage kt waits until the MMAs of stage kt - TSTAGES released its slot
    for (int kt = 0; kt < ktiles; kt++) {
      const int s = kt % TSTAGES;
      if (kt >= TSTAGES && !mbar_wait(smem_u32(&empty[s]), ((kt / TSTAGES) - 1) & 1)) {
        ok = false;
        break;
      }
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                       smem_u32(&full[s])),
                   "r"(A_BYTES + B_BYTES)
                   : "memory");
      tma_load_2d(smem_u32(sA + s * A_BYTES), &tmA, kb + kt * TBK, m0, smem_u32(&full[s]));
      tma_load_2d(smem_u32(sB + s * B_BYTES), &tmB, kb + kt * TBK, n0, smem_u32(&full[s]));
      issued = kt + 1;
    }
  } else if (warp == 1 && lane == 0) {
    // MMA issuer: 4 x (K = 16) per stage, accumulate in TMEM, release the stage
    const uint32_t idesc = instr_desc(BM, BN);
    for (int kt = 0; kt < ktiles; kt++) {
      const int s = kt % TSTAGES;
      if (!mbar_wait(smem_u32(&full[s]), (kt / TSTAGES) & 1)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
      for (int kk = 0; kk < TBK / 16; kk++) {
        const uint64_t da = desc_sw128(smem_u32(sA + s * A_BYTES) + kk * 32);
        const uint64_t db = desc_sw128(smem_u32(sB + s * B_BYTES) + kk * 32);
        const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
            "l"(da), "l"(db), "r"(idesc), "r"(acc)
            : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
              smem_u32(&empty[s]))
          : "memory");
    }
    // arrives once every MMA issued above has completed
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
            smem_u32(&done))
        : "memory");
  }
  const bool got = mbar_wait(smem_u32(&done), 0);
  ok = __syncthreads_and(ok && got) != 0;
  if (!ok) {
    // let the TMA loads still in flight land before the shared memory goes away
    if (warp == 0 && lane == 0)
      for (int kt = max(0, issued - TSTAGES); kt < issued; kt++)
        mbar_wait(smem_u32(&full[kt % TSTAGES]), (kt / TSTAGES) & 1);
    if (tid == 0) atomicExch(err, 1);
  } else {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const int row = m0 + warp * 32 + lane;
    for (int c = 0; c < BN; c += 8) {
      uint32_t r[8];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
            "=r"(r[7])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      if (row < M && partial) {
        float* pr = partial + ((size_t)blockIdx.z * M + row) * N + n0 + c;
        if (n0 + c + 8 <= N && (reinterpret_cast<uintptr_t>(pr) & 15) == 0 && ktiles > 0) {
          reinterpret_cast<float4*>(pr)[0] = make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]),
                                                         __uint_as_float(r[2]), __uint_as_float(r[3]));
          reinterpret_cast<float4*>(pr)[1] = make_float4(__uint_as_float(r[4]), __uint_as_float(r[5]),
                                                         __uint_as_float(r[6]), __uint_as_float(r[7]));
        } else {
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (n0 + c + j < N) pr[j] = ktiles > 0 ? __uint_as_float(r[j]) : 0.f;
        }
      } else if (row < M) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int col = n0 + c + j;
          v[j] = alpha * (ktiles > 0 ? __uint_as_float(r[j]) : 0.f);
          if (col < N) {
            if (beta != 0.f) v[j] += beta * C[(size_t)row * ldc + col];
            if (bias) v[j] += bias[col];
            if (act == 1) v[j] = tanhf(v[j]);
          }
        }
        float* crow = C + (size_t)row * ldc + n0 + c;
        if (n0 + c + 8 <= N && (reinterpret_cast<uintptr_t>(crow) & 15) == 0) {
          // this thread's 8 columns of its row as two 16-byte stores
          reinterpret_cast<float4*>(crow)[0] = make_float4(v[0], v[1], v[2], v[3]);
          reinterpret_cast<float4*>(crow)[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (n0 + c + j < N) crow[j] = v[j];
        }
        if (Cb)
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (n0 + c + j < N) Cb[(size_t)row * ldc + n0 + c + j] = __float2bfloat16(v[j]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(BN)
                 : "memory");
}

// ---------------------------------------------------------------------------
// Persistent form of the A B^T kernel: one CTA per SM walks the output tiles (grouped
// raster: GM consecutive 128-row tiles share every BN-column tile, so the operand
// panels in flight stay in L2).  Warps with fixed roles:
//   warp 0  TMA producer: 128 x 64 and BN x 64 tiles into a TSTAGES-deep ring;
//   warp 1  MMA issuer: tcgen05.mma into one of two TMEM accumulators (2 x BN columns),
//           tcgen05.commit releases ring stages and, after a tile's last K step,
//           hands the accumulator to the epilogue;
//   warps 2..   epilogue (EPW warps): TMEM lane quarter (warp % 4), tcgen05.ld, alpha / beta / bias /
//           tanh, stores (epi_store); then the accumulator goes back to the MMA issuer.
// The epilogue of tile i overlaps the MMAs of tile i + 1.  Every wait is bounded; a role
// that times out raises a shared abort flag so the others stop waiting, and the kernel
// reports the error through *err.
// CHAIN: an accumulator takes `chain` K steps, and the epilogue warps add the sums of a tile's
// accumulators in registers, in K order: the sums of split K without its partial tiles.
constexpr int GROUP_M = 16;

__device__ __forceinline__ bool mbar_wait_abort(uint32_t bar, uint32_t phase, volatile int* abort) {
  for (unsigned it = 0; it < kSpinLimit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
    if ((it & 255u) == 255u && *abort) return false;
  }
  *abort = 1;
  return false;
}

// The same by a whole warp, with one outcome for its lanes: a lane that gave up by itself would
// leave the others waiting for it at their next warp-wide instruction.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t phase, volatile int* abort) {
  return __all_sync(0xffffffffu, mbar_wait_abort(bar, phase, abort));
}

// Epilogue of 32 x 32 accumulators by one warp, turned through shared memory (buf, 32 rows
// of EPI_LD floats): r holds lane's row, the stores go out row by row, 128 contiguous bytes
// at a time (16-byte stores where C's rows allow it).  A lane storing its own row touches 32
// sectors per instruction.  40,960 x 6,591 x 64, bound by its 1.08 GB of output (159 us at
// the measured HBM rate): 1,356 -> 400 us, and with 6,592 columns 405 -> 231.  (Windows that
// start on a sector or a line of each row, the rest carried in the buffer, measured 422 and
// 452 us: the stores' own instructions then cost more than the parts of lines.)
constexpr int EPI_LD = 36;

__device__ __forceinline__ void epi_store(float* buf, const uint32_t (&r)[32], int row0, int M,
                                          int col0, int N, float* C, int ldc, __nv_bfloat16* Cb,
                                          float alpha, float beta, const float* __restrict__ bias,
                                          int act, int lane) {
#pragma unroll
  for (int j = 0; j < 8; j++)
    *reinterpret_cast<uint4*>(buf + lane * EPI_LD + 4 * j) =
        make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
  __syncwarp();
  const bool vec = col0 + 32 <= N && ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(Cb) & 7) == 0;
  if (vec) {
    const int col = col0 + 4 * (lane & 7);
    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (bias) b4 = make_float4(bias[col], bias[col + 1], bias[col + 2], bias[col + 3]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = 4 * i + (lane >> 3), row = row0 + k;
      const float4 t = *reinterpret_cast<const float4*>(buf + k * EPI_LD + 4 * (lane & 7));
      if (row < M) {
        const size_t at = (size_t)row * ldc + col;
        float v[4] = {alpha * t.x, alpha * t.y, alpha * t.z, alpha * t.w};
        if (beta != 0.f) {
          const float4 c = *reinterpret_cast<const float4*>(C + at);
          v[0] += beta * c.x;
          v[1] += beta * c.y;
          v[2] += beta * c.z;
          v[3] += beta * c.w;
        }
        if (bias) {
          v[0] += b4.x;
          v[1] += b4.y;
          v[2] += b4.z;
          v[3] += b4.w;
        }
        if (act == 1)
#pragma unroll
          for (int j = 0; j < 4; j++) v[j] = tanhf(v[j]);
        *reinterpret_cast<float4*>(C + at) = make_float4(v[0], v[1], v[2], v[3]);
        if (Cb) {
          __nv_bfloat162 lo, hi;
          lo.x = __float2bfloat16(v[0]);
          lo.y = __float2bfloat16(v[1]);
          hi.x = __float2bfloat16(v[2]);
          hi.y = __float2bfloat16(v[3]);
          *reinterpret_cast<uint2*>(Cb + at) =
              make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
        }
      }
    }
  } else {
    const int col = col0 + lane;
    const bool in = col < N;
    const float bc = bias && in ? bias[col] : 0.f;
    if (row0 + 32 <= M && beta == 0.f && act == 0 && !Cb) {  // whole block, C only
      float* c = C + (size_t)row0 * ldc + col;
#pragma unroll
      for (int k0 = 0; k0 < 32; k0 += 16) {
        float t[16];
#pragma unroll
        for (int k = 0; k < 16; k++) t[k] = buf[(k0 + k) * EPI_LD + lane];
        if (in) {
#pragma unroll
          for (int k = 0; k < 16; k++) {
            float v = alpha * t[k];
            if (bias) v += bc;
            *c = v;
            c += ldc;
          }
        }
      }
    } else {
#pragma unroll 8
      for (int k = 0; k < 32; k++) {
        const float t = buf[k * EPI_LD + lane];
        const int row = row0 + k;
        if (in && row < M) {
          const size_t at = (size_t)row * ldc + col;
          float v = alpha * t;
          if (beta != 0.f) v += beta * C[at];
          if (bias) v += bc;
          if (act == 1) v = tanhf(v);
          C[at] = v;
          if (Cb) Cb[at] = __float2bfloat16(v);
        }
      }
    }
  }
  __syncwarp();
}

// 32 accumulator columns of this warp's TMEM lane quarter
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// 16 of them: sums over several accumulators leave no registers for more
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& mt, int& nt) {
  const int per_group = GROUP_M * tiles_n;
  const int g = t / per_group;
  const int m_base = g * GROUP_M;
  const int gm = min(GROUP_M, tiles_m - m_base);
  const int r = t - g * per_group;
  mt = m_base + r % gm;
  nt = r / gm;
}

template <int BN, int STAGES, int EPW, bool CHAIN>
__global__ void __launch_bounds__(64 + 32 * EPW, 1)
    k_gemm_tma_pers(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    float* C, int ldc, __nv_bfloat16* Cb, int M, int N, int K, float alpha,
                    float beta, const float* __restrict__ bias, int act, int* err, int chain_steps) {
  constexpr int A_BYTES = BM * TBK * 2;
  constexpr int B_BYTES = BN * TBK * 2;
  constexpr uint32_t TCOLS = 2 * BN;  // two accumulators of BN FP32 columns
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_BYTES;
  __shared__ __align__(16) float epi_buf[EPW][32 * EPI_LD];
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int tiles = tiles_m * tiles_n;
  const int ktiles = (K + TBK - 1) / TBK;
  const int chain = CHAIN ? chain_steps : ktiles;  // K steps of an accumulator

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[s])) : "memory");
    }
    for (int b = 0; b < 2; b++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tfull[b])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&tempty[b])),
                   "r"(EPW)
                   : "memory");
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  ci::pdl_next();
  ci::pdl_wait();
  const uint32_t tmem = tmem_base;
  volatile int* abort = &abort_flag;
  bool ok = true;
  long long issued = 0;  // producer: ring steps whose loads were issued
  if (warp == 0) {
    if (lane == 0) {
      long long it = 0;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        int mt, nt;
        tile_coords(t, tiles_m, tiles_n, mt, nt);
        for (int kt = 0; kt < ktiles; kt++, it++) {
          const int s = (int)(it % STAGES);
          if (it >= STAGES &&
              !mbar_wait_abort(smem_u32(&empty[s]), (uint32_t)((it / STAGES) - 1) & 1u, abort)) {
            ok = false;
            break;
          }
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                           smem_u32(&full[s])),
                       "r"(A_BYTES + B_BYTES)
                       : "memory");
          tma_load_2d(smem_u32(sA + s * A_BYTES), &tmA, kt * TBK, mt * BM, smem_u32(&full[s]));
          tma_load_2d(smem_u32(sB + s * B_BYTES), &tmB, kt * TBK, nt * BN, smem_u32(&full[s]));
          issued = it + 1;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc(BM, BN);
      long long it = 0;
      int j = 0;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        for (int kc = 0; kc < ktiles && ok; kc += chain, j++) {
          const int b = j & 1;
          if (j >= 2 && !mbar_wait_abort(smem_u32(&tempty[b]), (uint32_t)((j >> 1) - 1) & 1u, abort)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint32_t acc_tmem = tmem + (uint32_t)(b * BN);
          const int ke = min(ktiles, kc + chain);
          for (int kt = kc; kt < ke; kt++, it++) {
            const int s = (int)(it % STAGES);
            if (!mbar_wait_abort(smem_u32(&full[s]), (uint32_t)(it / STAGES) & 1u, abort)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int kk = 0; kk < TBK / 16; kk++) {
              const uint64_t da = desc_sw128(smem_u32(sA + s * A_BYTES) + kk * 32);
              const uint64_t db = desc_sw128(smem_u32(sB + s * B_BYTES) + kk * 32);
              const uint32_t acc = (kt > kc || kk > 0) ? 1u : 0u;
              asm volatile(
                  "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc_tmem),
                  "l"(da), "l"(db), "r"(idesc), "r"(acc)
                  : "memory");
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                    smem_u32(&empty[s]))
                : "memory");
          }
          if (!ok) break;
          // the accumulator is complete once every MMA issued so far has finished
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                  smem_u32(&tfull[b]))
              : "memory");
        }
      }
    }
  } else if constexpr (CHAIN) {
    const int q = warp & 3;
    constexpr int COLS = BN * 4 / EPW;
    const int c_begin = (warp - 2) / 4 * COLS;
    int j = 0;
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      // (cleared, not set by the first chain: a choice between the two takes as many registers again)
      float sum[COLS];
#pragma unroll
      for (int n = 0; n < COLS; n++) sum[n] = 0.f;
#pragma unroll 1
      for (int kc = 0; kc < ktiles; kc += chain, j++) {
        const int b = j & 1;
        if (!mbar_wait_warp(smem_u32(&tfull[b]), (uint32_t)(j >> 1) & 1u, abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
        for (int n = 0; n < COLS; n += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + c_begin + n), r);
#pragma unroll
          for (int i = 0; i < 16; i++) sum[n + i] += __uint_as_float(r[i]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tempty[b]))
                       : "memory");
      }
      if (!ok) break;
      int mt, nt;
      tile_coords(t, tiles_m, tiles_n, mt, nt);
      const int n0 = nt * BN + c_begin;
#pragma unroll
      for (int n = 0; n < COLS; n += 32) {
        if (n0 + n >= N) break;
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 32; i++) r[i] = __float_as_uint(sum[n + i]);
        epi_store(epi_buf[warp - 2], r, mt * BM + q * 32, M, n0 + n, N, C, ldc, Cb, alpha, beta,
                  bias, act, lane);
      }
    }
  } else {
    const int q = warp & 3;  // TMEM lanes 32 q .. 32 q + 31 (a warp's accessible quarter)
    // its columns: all, or half of them where two warps share a quarter
    constexpr int COLS = BN * 4 / EPW;
    const int c_begin = (warp - 2) / 4 * COLS, c_end = c_begin + COLS;
    int j = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, j++) {
      const int b = j & 1;
      if (!mbar_wait_warp(smem_u32(&tfull[b]), (uint32_t)(j >> 1) & 1u, abort)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      int mt, nt;
      tile_coords(t, tiles_m, tiles_n, mt, nt);
      const int n0 = nt * BN;
#pragma unroll 1
      for (int c = c_begin; c < c_end && n0 + c < N; c += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + c), r);
        epi_store(epi_buf[warp - 2], r, mt * BM + q * 32, M, n0 + c, N, C, ldc, Cb, alpha, beta,
                  bias, act, lane);
      }
      // this warp's quarter of the accumulator is read: hand it back to the MMA issuer
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tempty[b]))
                     : "memory");
    }
  }
  ok = __syncthreads_and(ok) != 0;
  if (!ok) {
    // let the TMA loads still in flight land before the shared memory goes away
    if (warp == 0 && lane == 0)
      for (long long it = issued > STAGES ? issued - STAGES : 0; it < issued; it++)
        mbar_wait(smem_u32(&full[it % STAGES]), (uint32_t)(it / STAGES) & 1u);
    if (tid == 0) atomicExch(err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS)
                 : "memory");
}

// ---------------------------------------------------------------------------
// C = A B^T for products that stream a long A past a narrow B (N <= 256: the POD's sketch,
// projection and Gram products), bound by reading A once.
//
// Work split: the (tile, 64-deep K step) units of all tiles in one line, cut into one equal
// range per SM, so no SM waits for a last wave; a tile cut by a range end goes to FP32 partial
// sums that k_stream_reduce adds in K order (deterministic).  6,591 x 96 x 81,920, 1.1 GB (162 us
// at the measured HBM rate): 249-253 us with 312 CTAs of a sixth of K each on 152 SMs, 196 so.
//
// Rows that TMA cannot address (lda not a multiple of 8, or A off a 16-byte boundary): rows
// r = p i + c of one class c (p = 8 / gcd(lda, 8) classes) are a matrix whose row stride p lda
// is a multiple of 8, from the 16-byte boundary at or before row c; its rows then start delta_c
// elements into the tile.  B comes packed once per class, delta_c zeros in front, so the
// products line up; the delta_c elements in front of A's rows (the end of another row) are
// zeroed in shared memory before the first K step's MMAs, so that an infinity or a NaN there
// stays with its own row.  81,920 x 96 x 6,591: 2,711-2,760 us with element-wise staging, 238 so (163 us at the measured HBM
// rate).
//
// Accuracy: the tensor core's FP32 sums lose about 1.1e-9 of the result per product in a chain
// (measured: 7.3e-6 after 6,591, 2.9e-5 after 28,000).  A chain here is 4 or 8 K steps
// (stream_chain); the epilogue warps add the chains' sums in registers, rounded to nearest, while
// the next chain runs in the other accumulator.
constexpr int kMaxClasses = 8;

struct StreamMaps {
  CUtensorMap a[kMaxClasses];  // [c] rows of class c
  CUtensorMap b;               // [classes with a copy of B][N] rows
};

struct StreamArgs {
  float* C;
  __nv_bfloat16* Cb;
  const float* bias;
  float* partial;  // [2 gridDim.x][BN / 4][128] float4
  int* err;
  int ldc, M, N;
  float alpha, beta;
  int act;
  int p, b_copies;         // classes; 1 or p copies of B
  int delta[kMaxClasses];  // elements in front of the rows of a class
  int tm, tn, kt;          // row tiles per class, column tiles, K steps
  int chain;               // K steps of an accumulator
};

// Unit range of CTA b of g: [units b / g, units (b + 1) / g)
__host__ __device__ __forceinline__ long long stream_begin(long long units, int b, int g) {
  return units * b / g;
}

__device__ __forceinline__ void stream_tile(const StreamArgs& P, int t, int& c, int& mt, int& nt) {
  c = t / (P.tm * P.tn);
  const int r = t - c * P.tm * P.tn;
  mt = r / P.tn;
  nt = r - mt * P.tn;
}

template <int BN, int STAGES, int EPW>
__global__ void __launch_bounds__(64 + 32 * EPW, 1)
    k_gemm_stream(const __grid_constant__ StreamMaps maps, const __grid_constant__ StreamArgs P) {
  constexpr int A_BYTES = BM * TBK * 2;
  constexpr int B_BYTES = BN * TBK * 2;
  constexpr uint32_t TCOLS = 2 * BN <= 128 ? 128 : 2 * BN <= 256 ? 256 : 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_BYTES;
  __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES], tfull[2], tempty[2];
  __shared__ __align__(16) float epi_buf[EPW][32 * EPI_LD];
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chain = P.chain;
  const long long units = (long long)P.p * P.tm * P.tn * P.kt;
  const long long u0 = stream_begin(units, blockIdx.x, gridDim.x);
  const long long u1 = stream_begin(units, blockIdx.x + 1, gridDim.x);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&tmem_base)),
                 "r"(TCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&empty[s])) : "memory");
    }
    for (int b = 0; b < 2; b++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&tfull[b])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&tempty[b])),
                   "r"(EPW)
                   : "memory");
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  ci::pdl_next();
  ci::pdl_wait();
  const uint32_t tmem = tmem_base;
  volatile int* abort = &abort_flag;
  bool ok = true;
  long long issued = 0;
  if (warp == 0) {
    if (lane == 0) {
      long long it = 0;
      for (long long u = u0; u < u1 && ok;) {
        const int t = (int)(u / P.kt), k0 = (int)(u - (long long)t * P.kt);
        const int k1 = (int)min((long long)P.kt, k0 + (u1 - u));
        int c, mt, nt;
        stream_tile(P, t, c, mt, nt);
        const int brow = (P.b_copies > 1 ? c * P.N : 0) + nt * BN;
        for (int k = k0; k < k1; k++, it++) {
          const int s = (int)(it % STAGES);
          if (it >= STAGES &&
              !mbar_wait_abort(smem_u32(&empty[s]), (uint32_t)((it / STAGES) - 1) & 1u, abort)) {
            ok = false;
            break;
          }
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                           smem_u32(&full[s])),
                       "r"(A_BYTES + B_BYTES)
                       : "memory");
          tma_load_2d(smem_u32(sA + s * A_BYTES), &maps.a[c], k * TBK, mt * BM, smem_u32(&full[s]));
          tma_load_2d(smem_u32(sB + s * B_BYTES), &maps.b, k * TBK, brow, smem_u32(&full[s]));
          issued = it + 1;
        }
        u += k1 - k0;
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc(BM, BN);
    long long it = 0;
    int j = 0;
    for (long long u = u0; u < u1 && ok;) {
      const int t = (int)(u / P.kt), k0 = (int)(u - (long long)t * P.kt);
      const int k1 = (int)min((long long)P.kt, k0 + (u1 - u));
      int c, mt, nt;
      stream_tile(P, t, c, mt, nt);
      const int delta = P.delta[c];
      for (int kc = k0; kc < k1 && ok; kc += chain, j++) {
        const int b = j & 1;
        if (j >= 2 && !mbar_wait_warp(smem_u32(&tempty[b]), (uint32_t)((j >> 1) - 1) & 1u, abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t acc_tmem = tmem + (uint32_t)(b * BN);
        const int ke = min(k1, kc + chain);
        for (int k = kc; k < ke; k++, it++) {
          const int s = (int)(it % STAGES);
          // every lane waits, so that the masking below is ordered after the TMA write
          if (!mbar_wait_warp(smem_u32(&full[s]), (uint32_t)(it / STAGES) & 1u, abort)) {
            ok = false;
            break;
          }
          uint8_t* const a = sA + s * A_BYTES;
          if (k == 0 && delta > 0) {
            // elements 0 .. delta - 1 of every row: 16-byte chunk 0, at chunk (row % 8) of the
            // swizzled row
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const int row = lane + 32 * i;
              uint16_t* e = reinterpret_cast<uint16_t*>(a + row * 128 + ((row & 7) << 4));
              for (int x = 0; x < delta; x++) e[x] = 0;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
          }
          if (lane == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int kk = 0; kk < TBK / 16; kk++) {
              const uint64_t da = desc_sw128(smem_u32(a) + kk * 32);
              const uint64_t db = desc_sw128(smem_u32(sB + s * B_BYTES) + kk * 32);
              const uint32_t acc = (k > kc || kk > 0) ? 1u : 0u;
              asm volatile(
                  "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                  " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(acc_tmem),
                  "l"(da), "l"(db), "r"(idesc), "r"(acc)
                  : "memory");
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                    smem_u32(&empty[s]))
                : "memory");
          }
          __syncwarp();
        }
        if (ok && lane == 0)
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                  smem_u32(&tfull[b]))
              : "memory");
      }
      if (!ok) break;
      u += k1 - k0;
    }
  } else {
    const int q = warp & 3;
    constexpr int COLS = BN * 4 / EPW;  // this warp's columns
    const int c_begin = (warp - 2) / 4 * COLS;
    int j = 0;
    for (long long u = u0; u < u1 && ok;) {
      const int t = (int)(u / P.kt), k0 = (int)(u - (long long)t * P.kt);
      const int k1 = (int)min((long long)P.kt, k0 + (u1 - u));
      int c, mt, nt;
      stream_tile(P, t, c, mt, nt);
      float sum[COLS];  // (cleared as in k_gemm_tma_pers)
#pragma unroll
      for (int n = 0; n < COLS; n++) sum[n] = 0.f;
#pragma unroll 1
      for (int kc = k0; kc < k1; kc += chain, j++) {
        const int b = j & 1;
        if (!mbar_wait_warp(smem_u32(&tfull[b]), (uint32_t)(j >> 1) & 1u, abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
        for (int n = 0; n < COLS; n += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + c_begin + n), r);
#pragma unroll
          for (int i = 0; i < 16; i++) sum[n + i] += __uint_as_float(r[i]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&tempty[b]))
                       : "memory");
      }
      if (!ok) break;
      const int n0 = nt * BN + c_begin;
      const int rows_c = (P.M - c + P.p - 1) / P.p;  // rows of the class
      const bool whole = k0 == 0 && k1 == P.kt;
      float4* part = reinterpret_cast<float4*>(P.partial) +
                     ((size_t)(2 * blockIdx.x + (u == u0 ? 0 : 1)) * (BN / 4) + c_begin / 4) * 128 +
                     q * 32 + lane;
      if (whole) {
#pragma unroll
        for (int n = 0; n < COLS; n += 32) {
          if (n0 + n >= P.N) break;
          uint32_t r[32];
#pragma unroll
          for (int i = 0; i < 32; i++) r[i] = __float_as_uint(sum[n + i]);
          epi_store(epi_buf[warp - 2], r, mt * BM + q * 32, rows_c, n0 + n, P.N,
                          P.C + (size_t)c * P.ldc, P.p * P.ldc,
                          P.Cb ? P.Cb + (size_t)c * P.ldc : nullptr, P.alpha, P.beta, P.bias, P.act,
                          lane);
        }
      } else {
#pragma unroll
        for (int n = 0; n < COLS; n += 4)
          if (n0 + n < P.N)
            part[n / 4 * 128] = make_float4(sum[n], sum[n + 1], sum[n + 2], sum[n + 3]);
      }
      u += k1 - k0;
    }
  }
  ok = __syncthreads_and(ok) != 0;
  if (!ok) {
    // let the TMA loads still in flight land before the shared memory goes away
    if (warp == 0 && lane == 0)
      for (long long it = issued > STAGES ? issued - STAGES : 0; it < issued; it++)
        mbar_wait(smem_u32(&full[it % STAGES]), (uint32_t)(it / STAGES) & 1u);
    if (tid == 0) atomicExch(P.err, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS)
                 : "memory");
}

// The tiles that range ends cut: their partial sums in K order, then the epilogue.  Block (cut
// tile, 16 columns, 32 rows): a warp adds the parts of 4 columns, lanes along the rows, eight
// parts in flight; the sums go through shared memory, so that a row's 16 columns are written
// together.  With fewer tiles than ranges (by_tile) the blocks count tiles, else range ends, of
// which the one that begins a tile's second range stands for it: few blocks have nothing to do.
// (One block per range end, 4 columns and 32 rows whatever the tiles, 1,024 x 64 x 16,384 with
// the products 21.5 us; 13.5 so.)
__global__ void __launch_bounds__(128) k_stream_reduce(const StreamArgs P, int BN, int g, int by_tile) {
  __shared__ float4 sums[4][33];
  ci::pdl_next();
  ci::pdl_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long units = (long long)P.p * P.tm * P.tn * P.kt;
  const int t = by_tile ? blockIdx.x : (int)(stream_begin(units, blockIdx.x + 1, g) / P.kt);
  const long long ut = (long long)t * P.kt;
  // the ranges with the tile's first and last units
  const int b0 = (int)(((ut + 1) * g - 1) / units), b1 = (int)(((ut + P.kt) * g - 1) / units);
  if (b0 == b1 || (!by_tile && b0 != (int)blockIdx.x)) return;
  const size_t stride = (size_t)(BN / 4) * 128;
  const float4* part = reinterpret_cast<const float4*>(P.partial) +
                       (size_t)(4 * blockIdx.y + w) * 128 + blockIdx.z * 32 + lane;
  float4 s = part[(2 * b0 + (stream_begin(units, b0, g) == ut ? 0 : 1)) * stride];
#pragma unroll 8
  for (int b = b0 + 1; b <= b1; b++) {
    const float4 v = part[2 * b * stride];
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  sums[w][lane] = s;
  __syncthreads();
  int c, mt, nt;
  stream_tile(P, t, c, mt, nt);
  const int r = threadIdx.x >> 2, i = mt * BM + blockIdx.z * 32 + r;
  const int col = nt * BN + 16 * blockIdx.y + 4 * (threadIdx.x & 3);
  if (i >= (P.M - c + P.p - 1) / P.p || col >= P.N) return;
  s = sums[threadIdx.x & 3][r];
  const size_t at = ((size_t)i * P.p + c) * P.ldc + col;
  float v[4] = {P.alpha * s.x, P.alpha * s.y, P.alpha * s.z, P.alpha * s.w};
  const bool vec = col + 4 <= P.N && (reinterpret_cast<uintptr_t>(P.C + at) & 15) == 0;
  float old[4] = {0.f, 0.f, 0.f, 0.f};
  if (P.beta != 0.f) {
    if (vec)
      *reinterpret_cast<float4*>(old) = *reinterpret_cast<const float4*>(P.C + at);
    else
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (col + j < P.N) old[j] = P.C[at + j];
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (P.beta != 0.f) v[j] += P.beta * old[j];
    if (P.bias && col + j < P.N) v[j] += P.bias[col + j];
    if (P.act == 1) v[j] = tanhf(v[j]);
  }
  if (vec) {
    *reinterpret_cast<float4*>(P.C + at) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (col + j < P.N) P.C[at + j] = v[j];
  }
  if (P.Cb)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (col + j < P.N) P.Cb[at + j] = __float2bfloat16(v[j]);
}

// Operand copies that TMA can address: out [copies][rows][ld] with ld a multiple of 8 (the
// columns up to ld zero), copy c shifted by delta[c] zeros; the source [rows x K], or
// [K x rows] when trans.  32 x 32 tiles through shared memory, so both sides are read and
// written along their rows.  A block has 128 columns and every gridDim.y-th 32 rows (grid.y counts
// to 65,535 only).
struct PackArgs {
  const __nv_bfloat16* in;
  __nv_bfloat16* out;
  int rows, K, ld_in, trans, ld;
  int delta[kMaxClasses];
};

__global__ void __launch_bounds__(256) k_pack_bf16(const PackArgs P) {
  ci::pdl_next();
  ci::pdl_wait();
  __shared__ __nv_bfloat16 tile[32][34];
  const int d = P.delta[blockIdx.z];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  __nv_bfloat16* out = P.out + (size_t)blockIdx.z * P.rows * P.ld;
  const int x_end = min(P.ld, (int)(blockIdx.x + 1) * 128);
  for (int r0 = blockIdx.y * 32; r0 < P.rows; r0 += gridDim.y * 32) {
    for (int x0 = blockIdx.x * 128; x0 < x_end; x0 += 32) {
      if (P.trans) {
        for (int k = ty; k < 32; k += 8) {
          const int x = x0 + k - d, r = r0 + tx;
          tile[k][tx] = (x >= 0 && x < P.K && r < P.rows) ? P.in[(size_t)x * P.ld_in + r] : zero;
        }
        __syncthreads();
        for (int k = ty; k < 32; k += 8)
          if (r0 + k < P.rows && x0 + tx < P.ld) out[(size_t)(r0 + k) * P.ld + x0 + tx] = tile[tx][k];
        __syncthreads();
      } else {
        for (int k = ty; k < 32; k += 8) {
          const int x = x0 + tx - d, r = r0 + k;
          if (r < P.rows && x0 + tx < P.ld)
            out[(size_t)r * P.ld + x0 + tx] = (x >= 0 && x < P.K) ? P.in[(size_t)r * P.ld_in + x] : zero;
        }
      }
    }
  }
}

// C = alpha sum_z partial[z] (z in order) + beta C + bias, then tanh; BF16 copy.  Latency bounds
// it where many parts make a small output, so U parts are read at once: ten (20 parts of 256 x
// 256, cold under a profiler: 7.2 us four at a time, 4.5 so), or two and four where there are no
// more (8,192 x 1,024 x 2,048 in two parts, both kernels: 105.2 us with ten, 86.4 with two).
template <int U>
__global__ void k_splitk_reduce(const float* partial, int splits, float* C, int ldc,
                                __nv_bfloat16* Cb, int M, int N, float alpha, float beta,
                                const float* bias, int act) {
  ci::pdl_next();
  ci::pdl_wait();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)M * N) return;
  const int row = (int)(i / N), col = (int)(i % N);
  float acc = 0.f;
  for (int z0 = 0; z0 < splits; z0 += U) {
    float v[U];
#pragma unroll
    for (int j = 0; j < U; j++) v[j] = partial[(size_t)min(z0 + j, splits - 1) * M * N + i];
#pragma unroll
    for (int j = 0; j < U; j++)
      if (z0 + j < splits) acc += v[j];
  }
  float v = alpha * acc;
  if (beta != 0.f) v += beta * C[(size_t)row * ldc + col];
  if (bias) v += bias[col];
  if (act == 1) v = tanhf(v);
  C[(size_t)row * ldc + col] = v;
  if (Cb) Cb[(size_t)row * ldc + col] = __float2bfloat16(v);
}

// split-K workspaces, grown on demand, one per (device, stream): calls on different
// streams never share one, so they may run concurrently (the stream orders the calls
// that do share one).  At most kMaxWorkspaces are kept per device; a new stream beyond
// that frees the device's others first.  A caller holds g_ws_mu from the lookup until
// its kernels are enqueued, and cudaFree synchronises the device, so no workspace is
// freed while a call still uses it.  One that a call used while its stream was captured is
// never freed: the graph's replays use it whenever they run.
// Operand copies make workspaces of up to some 300 MB, so together a device's hold kMaxKept at
// most (beyond it, and where an allocation fails, the others are freed), and one of more than
// kKeepBytes goes back when kIdleCalls calls in a row needed less than half of it.
struct Workspace {
  float* p = nullptr;
  size_t size = 0;
  bool captured = false;
  int idle = 0;  // calls in a row that needed less than half
};
constexpr size_t kMaxWorkspaces = 32;
constexpr size_t kMaxKept = (size_t)512 << 20;
constexpr size_t kKeepBytes = (size_t)64 << 20;
constexpr int kIdleCalls = 64;
std::mutex g_ws_mu;
std::map<std::pair<int, cudaStream_t>, Workspace> g_ws;
// outgrown while their stream was captured, where nothing may be freed
std::vector<std::pair<int, void*>> g_ws_later;

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tensor_map_encoder() {
  static std::once_flag once;
  static EncodeTiledFn fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// 2-D map of a row-major BF16 matrix [rows x K] (leading dimension ld), boxes of
// box_rows x 64 with the 128-byte swizzle; out-of-range elements read as zero.
bool make_tile_map(CUtensorMap* map, const void* base, int rows, int K, long long ld, int box_rows) {
  const EncodeTiledFn enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)TBK, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box,
             es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int STAGES = TSTAGES>
constexpr int tma_smem_bytes() {
  return STAGES * (BM * TBK * 2 + BN * TBK * 2) + 1024;
}

template <int BN>
cudaError_t launch_tma(const CUtensorMap& ta, const CUtensorMap& tb, dim3 grid, cudaStream_t st,
                       float* C, int ldc, __nv_bfloat16* Cb, int M, int N, int K, float alpha,
                       float beta, const float* bias, int act, int* err, int k_chunk,
                       float* partial) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_gemm_tma<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, tma_smem_bytes<BN>());
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  return ci::launch_pdl(k_gemm_tma<BN>, grid, 128, tma_smem_bytes<BN>(), st, ta, tb, C, ldc, Cb, M, N,
                        K, alpha, beta, bias, act, err, k_chunk, partial);
}

int num_sms() {
  static int n[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 1;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev] > 0 ? n[dev] : 1;
}

// The output of a tile takes as long to write as its products to compute at K of about 650
// (128 x 256 FP32 at an SM's share of HBM against its tensor cores); up to 512 the kernel is
// a stream of stores, and eight epilogue warps (with a ring of three stages to make room for
// their buffers) keep more of them going than four.
constexpr int kShortK = 512;

template <int BN, int STAGES, int EPW, bool CHAIN = false>
cudaError_t launch_pers(const CUtensorMap& ta, const CUtensorMap& tb, cudaStream_t st, float* C,
                        int ldc, __nv_bfloat16* Cb, int M, int N, int K, float alpha, float beta,
                        const float* bias, int act, int* err, int chain = 0) {
  static bool configured[64] = {};
  constexpr int smem = tma_smem_bytes<BN, STAGES>();
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_gemm_tma_pers<BN, STAGES, EPW, CHAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int grid = std::min(tiles, num_sms());
  return ci::launch_pdl(k_gemm_tma_pers<BN, STAGES, EPW, CHAIN>, grid, 64 + 32 * EPW, smem, st, ta,
                        tb, C, ldc, Cb, M, N, K, alpha, beta, bias, act, err, chain);
}

template <int BN>
cudaError_t launch_tma_pers(const CUtensorMap& ta, const CUtensorMap& tb, cudaStream_t st, float* C,
                            int ldc, __nv_bfloat16* Cb, int M, int N, int K, float alpha,
                            float beta, const float* bias, int act, int* err) {
  return K <= kShortK ? launch_pers<BN, 3, 8>(ta, tb, st, C, ldc, Cb, M, N, K, alpha, beta, bias, act, err)
                      : launch_pers<BN, TSTAGES, 4>(ta, tb, st, C, ldc, Cb, M, N, K, alpha, beta,
                                                    bias, act, err);
}

template <int BN, int STAGES, int EPW>
cudaError_t launch_stream(const StreamMaps& maps, const StreamArgs& P, int grid, cudaStream_t st) {
  static bool configured[64] = {};
  constexpr int smem = tma_smem_bytes<BN, STAGES>();
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_gemm_stream<BN, STAGES, EPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const cudaError_t e = ci::launch_pdl(k_gemm_stream<BN, STAGES, EPW>, grid, 64 + 32 * EPW, smem, st,
                                       maps, P);
  if (e != cudaSuccess) return e;
  if (grid == 1) return cudaSuccess;
  const int cols = std::min(BN, P.N), tiles = P.p * P.tm * P.tn;
  const bool by_tile = tiles < grid - 1;
  return ci::launch_pdl(k_stream_reduce, dim3(by_tile ? tiles : grid - 1, (cols + 15) / 16, BM / 32), 128,
                        0, st, P, BN, grid, (int)by_tile);
}

inline size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

// Tiny products (the plastic-strain network's 64-wide layers) on the CUDA cores: one
// thread per output, the BF16 operands' products summed in FP32 in K order, then the
// epilogue of the tensor-core kernels (alpha, beta, bias, tanh, BF16 copy).
__global__ void __launch_bounds__(256) k_gemm_small(const __nv_bfloat16* A, int lda, int tA,
                                                    const __nv_bfloat16* B, int ldb, int tB,
                                                    float* C, int ldc, __nv_bfloat16* Cb, int M,
                                                    int N, int K, float alpha, float beta,
                                                    const float* bias, int act) {
  ci::pdl_next();
  ci::pdl_wait();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)M * N) return;
  const int row = (int)(i / N), col = (int)(i % N);
  float acc = 0.f;
  for (int k = 0; k < K; k++) {
    const float a = __bfloat162float(tA ? A[(size_t)k * lda + row] : A[(size_t)row * lda + k]);
    const float b = __bfloat162float(tB ? B[(size_t)col * ldb + k] : B[(size_t)k * ldb + col]);
    acc = fmaf(a, b, acc);
  }
  float v = alpha * acc;
  if (beta != 0.f) v += beta * C[(size_t)row * ldc + col];
  if (bias) v += bias[col];
  if (act == 1) v = tanhf(v);
  C[(size_t)row * ldc + col] = v;
  if (Cb) Cb[(size_t)row * ldc + col] = __float2bfloat16(v);
}

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;  // the legacy stream while another one is captured
}

// Empties a workspace; cudaFree synchronises the device, so no call still uses it.
void release(Workspace& w) {
  if (w.p && !w.captured) cudaFree(w.p);
  w = Workspace();
}

// The stream's workspace, grown to `need` bytes (null: no memory); takes the lock.
void* workspace(int dev, cudaStream_t st, size_t need, std::unique_lock<std::mutex>& lock) {
  lock.lock();
  const bool cap = capturing(st);
  if (!cap) {
    for (size_t i = 0; i < g_ws_later.size();)
      if (g_ws_later[i].first == dev) {
        cudaFree(g_ws_later[i].second);
        g_ws_later.erase(g_ws_later.begin() + i);
      } else {
        i++;
      }
    size_t on_dev = 0;
    for (const auto& kv : g_ws) on_dev += kv.first.first == dev;
    if (!g_ws.count({dev, st}) && on_dev >= kMaxWorkspaces)
      for (auto it = g_ws.begin(); it != g_ws.end();) {
        if (it->first.first == dev) {
          release(it->second);
          it = g_ws.erase(it);
        } else {
          ++it;
        }
      }
  }
  Workspace& w = g_ws[{dev, st}];
  w.idle = need < w.size / 2 ? w.idle + 1 : 0;
  if (!cap && w.size > kKeepBytes && w.idle >= kIdleCalls) release(w);
  if (w.size < need) {
    auto release_others = [&](size_t keep) {  // until they hold `keep` bytes
      size_t held = 0;
      for (const auto& kv : g_ws)
        if (kv.first.first == dev && &kv.second != &w) held += kv.second.size;
      for (auto& kv : g_ws)
        if (kv.first.first == dev && &kv.second != &w && !kv.second.captured && held > keep) {
          held -= kv.second.size;
          release(kv.second);
        }
    };
    if (!cap) {
      release(w);
      release_others(need < kMaxKept ? kMaxKept - need : 0);
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, need);
    if (e != cudaSuccess && !cap) {
      cudaGetLastError();
      release_others(0);
      e = cudaMalloc(&p, need);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (w.p && !w.captured) g_ws_later.push_back({dev, w.p});
    w = Workspace();
    w.p = static_cast<float*>(p);
    w.size = need;
  }
  w.captured = w.captured || cap;
  return w.p;
}

// Parts of K, multiples of a stage, where the output has too few tiles to fill the GPU and K is
// long.
struct SplitK {
  int splits, k_chunk;
};
SplitK split_k(int tiles, int K) {
  int splits = 1;
  if (tiles < 304 && K >= 8 * BK)
    splits = std::min((304 + tiles - 1) / tiles, (K + 4 * BK - 1) / (4 * BK));
  splits = std::max(1, std::min(splits, 512));
  int k_chunk = (K + splits - 1) / splits;
  k_chunk = (k_chunk + BK - 1) / BK * BK;
  return {(K + k_chunk - 1) / k_chunk, k_chunk};
}

// K steps of an accumulator of the streaming products: 256 products where K is short or split K
// would make chains of less than 512, so that none is less exact than it, else 512, which costs
// the epilogue warps half as much (40,000 x 32 x 20,480: 271 and 256 us; error against 64 bits
// 2.5e-7 and 4.7e-7, of one chain 2.2e-5).
int stream_chain(int M, int N, int K) {
  const int bn = N <= 64 ? 64 : N <= 128 ? 128 : 256;
  return K > 2048 && split_k((M + BM - 1) / BM * ((N + bn - 1) / bn), K).k_chunk >= 512 ? 8 : 4;
}

// How a product's operands reach the tensor-core kernels.
struct Operands {
  bool tma = false;     // A [M x K] and B [N x K] below can be addressed by TMA
  bool stream = false;  // k_gemm_stream
  const void* A = nullptr;
  const void* B = nullptr;
  long long lda = 0, ldb = 0;
  int p = 1, b_copies = 1, b_cols = 0, max_delta = 0;
  int delta[kMaxClasses] = {};
  // copies to make: 0, 1 or 2 of them
  PackArgs pack_a{}, pack_b{};
  bool do_a = false, do_b = false;
  size_t pack_bytes = 0;
};

// Copies are made for products that the CUDA cores do not take (more than 2^20 multiply-adds)
// and whose copies stay below this; beyond it, and while the stream is captured into a graph
// (whose replays would outlive the workspace), the staging kernel k_gemm_bf16 reads the
// operands as they are.
constexpr size_t kMaxPackBytes = (size_t)256 << 20;

// Operands as they are where TMA can read them (A B^T, 16-byte rows).  Otherwise: a tall A
// before a narrow B (the streaming products) stays in place, in row classes; any other
// operand is copied to aligned rows, transposed if need be, which costs a pass over it
// (81,920 x 96 x 96, A B: 97.2 us staged element by element, 22.7 with B copied; 96 x 96 x
// 327,680, A^T B: 466 and 204 with both).
int choose_operands(const void* A, int lda, int transA, const void* B, int ldb, int transB, int M,
                    int N, int K, bool tma_shape, bool plain, cudaStream_t st, Operands* op) {
  const bool a_ok = !transA && lda >= K && lda % 8 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
  const bool b_ok = transB && ldb >= K && ldb % 8 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0;
  op->A = A;
  op->B = B;
  op->lda = lda;
  op->ldb = ldb;
  op->b_cols = K;
  if (!tensor_map_encoder()) return CI_OK;  // everything through the staging kernel
  if (plain) {  // no workspace for copies or ranges
    op->tma = tma_shape;
    return CI_OK;
  }
  // A of 8 MB or more read once past a B of at most 256 rows, K long enough to cut
  const bool streams = N <= 256 && (long long)M * K >= (1 << 22) && K >= 1024;
  if ((!tma_shape || streams) && capturing(st)) {
    op->tma = tma_shape;
    return CI_OK;
  }
  if (!tma_shape) {
    if ((transA ? lda < M : lda < K) || (transB ? ldb < K : ldb < N)) return CI_OK;
    const int kp8 = (K + 7) / 8 * 8;
    if (!a_ok && !transA && streams && M >= 4096) {
      const int g = lda % 8 == 0 ? 8 : lda % 4 == 0 ? 4 : lda % 2 == 0 ? 2 : 1;
      op->p = kMaxClasses / g;
      for (int c = 0; c < op->p; c++) {
        op->delta[c] = (int)((reinterpret_cast<uintptr_t>(A) / 2 + (size_t)c * lda) & 7);
        op->max_delta = std::max(op->max_delta, op->delta[c]);
      }
      op->b_copies = op->p;
    } else if (!a_ok) {
      op->do_a = true;
      op->pack_a = {static_cast<const __nv_bfloat16*>(A), nullptr, M, K, lda, transA, kp8, {}};
      op->pack_bytes += align256(sizeof(__nv_bfloat16) * (size_t)M * kp8);
    }
    if (!b_ok || op->max_delta > 0 || op->p > 1) {
      op->do_b = true;
      op->b_cols = op->max_delta ? (K + op->max_delta + 7) / 8 * 8 : K;
      const int ld = (op->b_cols + 7) / 8 * 8;
      op->pack_b = {static_cast<const __nv_bfloat16*>(B), nullptr, N, K, ldb, !transB, ld, {}};
      for (int c = 0; c < op->p; c++) op->pack_b.delta[c] = op->delta[c];
      op->pack_bytes += align256(sizeof(__nv_bfloat16) * (size_t)op->b_copies * N * ld);
    }
    if (op->pack_bytes > kMaxPackBytes) {
      *op = Operands();
      op->A = A;
      op->B = B;
      op->lda = lda;
      op->ldb = ldb;
      return CI_OK;
    }
  }
  op->tma = true;
  op->stream = streams;
  return CI_OK;
}

// Enqueues the copies into `at` and points the operands to them.
bool pack_operands(Operands* op, char* at, cudaStream_t st) {
  auto run = [&](PackArgs& a, int copies) {
    a.out = reinterpret_cast<__nv_bfloat16*>(at);
    at += align256(sizeof(__nv_bfloat16) * (size_t)copies * a.rows * a.ld);
    const dim3 grid((a.ld + 127) / 128, std::min((a.rows + 31) / 32, 65535), copies);
    return ci::launch_pdl(k_pack_bf16, grid, 256, 0, st, a) == cudaSuccess;
  };
  if (op->do_a) {
    if (!run(op->pack_a, 1)) return false;
    op->A = op->pack_a.out;
    op->lda = op->pack_a.ld;
  }
  if (op->do_b) {
    if (!run(op->pack_b, op->b_copies)) return false;
    op->B = op->pack_b.out;
    op->ldb = op->pack_b.ld;
  }
  return true;
}

// plain: without the streaming kernel and without copies (after an allocation for them failed)
int gemm_bf16(const void* A, int lda, int transA, const void* B, int ldb, int transB, float* C,
              int ldc, void* C_bf16, int M, int N, int K, float alpha, float beta,
              const float* bias, int activation, int* d_error, void* stream, bool plain) {
  if (!A || !B || !C || !d_error || M <= 0 || N <= 0 || K <= 0)
    return ci::set_last_error(CI_ERR_INVALID, "ci_gemm_bf16: null pointer or empty shape");
  if (activation != 0 && activation != 1)
    return ci::set_last_error(CI_ERR_INVALID, "ci_gemm_bf16: activation must be 0 or 1");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // A B^T with both operands K-major and TMA-compatible rows: the pipelined kernel
  const bool tma_shape = !transA && transB && M >= BM && N >= 16 && K >= TBK && lda >= K &&
                         ldb >= K && lda % 8 == 0 && ldb % 8 == 0 &&
                         reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(B) % 16 == 0;
  // other shapes of at most 2^20 multiply-adds (a 64-wide layer, a single output column):
  // CUDA cores, where a 128-row tile pipeline would cost more than the product
  if (!tma_shape && (long long)M * N * K <= (1LL << 20)) {
    const long long outs = (long long)M * N;
    return ci::launch_pdl(k_gemm_small, (unsigned)((outs + 255) / 256), 256, 0, st,
                          static_cast<const __nv_bfloat16*>(A), lda, transA,
                          static_cast<const __nv_bfloat16*>(B), ldb, transB, C, ldc,
                          static_cast<__nv_bfloat16*>(C_bf16), M, N, K, alpha, beta, bias,
                          activation) == cudaSuccess
               ? CI_OK
               : ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: small-product launch failed");
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess)
    return ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: no current device");
  __nv_bfloat16* cb = static_cast<__nv_bfloat16*>(C_bf16);
  std::unique_lock<std::mutex> ws_lock(g_ws_mu, std::defer_lock);  // held until enqueued
  Operands op;
  {
    const int rc = choose_operands(A, lda, transA, B, ldb, transB, M, N, K, tma_shape, plain, st, &op);
    if (rc) return rc;
  }
  int chain = 0;  // K steps of an accumulator of the persistent kernel (0: all)
  // A streamed product of many tiles goes to the persistent kernel, in the same chains of K, where
  // the SMs' idle time in its last round (0.37 us a K step: 16 KB of A at an SM's share of HBM)
  // is below what cut tiles cost (a launch, and partial sums of BN columns).  65,536 x 256 x 1,024
  // 65.4 us cut, 52.7 so; 65,536 x 64 x 1,024 36.7 and 31.6.
  if (op.stream && op.p == 1 && op.max_delta == 0) {
    const int w = N <= 64 ? 64 : N <= 128 ? 128 : 256, sms = num_sms();
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + w - 1) / w);
    const double idle = (double)(((tiles + sms - 1) / sms) * sms - tiles) / sms * ((K + TBK - 1) / TBK);
    if (tiles >= 2 * sms && 0.37 * idle <= 5.0 + 0.04 * N) {
      op.stream = false;
      chain = stream_chain(M, N, K);
    }
  }
  if (op.stream) {
    const int bn = N <= 64 ? 64 : N <= 96 ? 96 : N <= 128 ? 128 : 256;
    StreamArgs P{};
    P.C = C;
    P.Cb = cb;
    P.bias = bias;
    P.err = d_error;
    P.ldc = ldc;
    P.M = M;
    P.N = N;
    P.alpha = alpha;
    P.beta = beta;
    P.act = activation;
    P.p = op.p;
    P.b_copies = op.b_copies;
    for (int c = 0; c < kMaxClasses; c++) P.delta[c] = op.delta[c];
    P.tm = ((M + op.p - 1) / op.p + BM - 1) / BM;
    P.tn = (N + bn - 1) / bn;
    P.kt = (K + op.max_delta + TBK - 1) / TBK;
    P.chain = stream_chain(M, N, K);
    const long long units = (long long)P.p * P.tm * P.tn * P.kt;
    const int grid = (int)std::min<long long>(num_sms(), units);
    const size_t part = align256(sizeof(float) * 2 * (size_t)grid * BM * bn);
    char* ws = static_cast<char*>(workspace(dev, st, part + op.pack_bytes, ws_lock));
    if (!ws) {
      ws_lock.unlock();
      return gemm_bf16(A, lda, transA, B, ldb, transB, C, ldc, C_bf16, M, N, K, alpha, beta, bias,
                       activation, d_error, stream, true);
    }
    P.partial = reinterpret_cast<float*>(ws);
    if (!pack_operands(&op, ws + part, st))
      return ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: packing launch failed");
    StreamMaps maps;
    bool ok = make_tile_map(&maps.b, op.B, N * op.b_copies, op.b_cols, op.ldb, bn);
    for (int c = 0; c < op.p && ok; c++) {
      const uintptr_t row = reinterpret_cast<uintptr_t>(op.A) + 2 * (size_t)c * op.lda;
      ok = make_tile_map(&maps.a[c], reinterpret_cast<const void*>(row & ~(uintptr_t)15),
                         (M - c + op.p - 1) / op.p, K + op.delta[c], (long long)op.p * op.lda, BM);
    }
    if (!ok) return ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: tensor map");
    const cudaError_t e = bn == 64   ? launch_stream<64, 8, 4>(maps, P, grid, st)
                          : bn == 96  ? launch_stream<96, 7, 4>(maps, P, grid, st)
                          : bn == 128 ? launch_stream<128, 5, 8>(maps, P, grid, st)
                                      : launch_stream<256, 3, 8>(maps, P, grid, st);
    return e == cudaSuccess ? CI_OK : ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(e));
  }
  bool tma = op.tma;
  const int bn_tma = N <= 64 ? 64 : N <= 128 ? 128 : 256;
  int bn = tma ? bn_tma : (N <= 64 ? 64 : 128);
  const int tiles = ((M + BM - 1) / BM) * ((N + bn - 1) / bn);
  SplitK cut = split_k(tiles, K);
  if (chain) cut = {1, K};
  // With more than half a tile per SM and a short K the partial tiles cost more than the CTAs give
  // (4,096 x 1,024 x 512 39.2 us, 8,192 x 512 x 896 49.6), but one chain of products over all of K
  // would lose accuracy
  // (8,192 x 512 x 896: 8.6e-7, in chains of 320 products 2.7e-7): the same chains, one after
  // the other in the persistent kernel (12.2 and 15.6 us; as one chain 11.4 and 14.9).
  if (tma && cut.splits > 1 && 2 * tiles > num_sms() && K <= 896) {
    chain = cut.k_chunk / BK;
    cut = {1, K};
    bn = std::min(bn, 128);  // (8,192 x 1,024 x 512 18.5 us, with 256 columns 19.6)
  }
  const int splits = cut.splits, k_chunk = cut.k_chunk;
  // Narrower tiles while they leave the GPU half empty: 256 x 256 x 256, two tiles of 256
  // columns, 13.5 us, eight of 64 7.3 (cold, under a profiler).  The sums of an output do not
  // depend on its tile.
  if (tma)
    while (bn > 64 && 2LL * ((M + BM - 1) / BM) * ((N + bn - 1) / bn) * splits <= num_sms()) bn /= 2;
  float* partial = nullptr;
  const size_t part = splits > 1 ? align256(sizeof(float) * (size_t)splits * M * N) : 0;
  if (part + op.pack_bytes) {
    char* ws = static_cast<char*>(workspace(dev, st, part + op.pack_bytes, ws_lock));
    if (!ws && op.pack_bytes) {
      ws_lock.unlock();
      return gemm_bf16(A, lda, transA, B, ldb, transB, C, ldc, C_bf16, M, N, K, alpha, beta, bias,
                       activation, d_error, stream, true);
    }
    if (!ws) return ci::set_last_error(CI_ERR_NOMEM, "ci_gemm_bf16: workspace");
    if (splits > 1) partial = reinterpret_cast<float*>(ws);
    if (!pack_operands(&op, ws + part, st))
      return ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: packing launch failed");
  }
  CUtensorMap ta, tb;
  if (tma && !(make_tile_map(&ta, op.A, M, K, op.lda, BM) &&
               make_tile_map(&tb, op.B, N, K, op.ldb, bn)))
    return ci::set_last_error(CI_ERR_CUDA, "ci_gemm_bf16: tensor map");
  dim3 grid((M + BM - 1) / BM, (N + bn - 1) / bn, splits);
  cudaError_t le = cudaSuccess;
  if (tma && chain) {
    if (bn == 64)
      le = launch_pers<64, TSTAGES, 8, true>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias,
                                             activation, d_error, chain);
    else if (bn == 128)
      le = launch_pers<128, TSTAGES, 8, true>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias,
                                              activation, d_error, chain);
    else
      le = launch_pers<256, 3, 8, true>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation,
                                        d_error, chain);
    if (le != cudaSuccess) return ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(le));
  } else if (tma && splits == 1) {
    if (bn == 64)
      le = launch_tma_pers<64>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation, d_error);
    else if (bn == 128)
      le = launch_tma_pers<128>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation, d_error);
    else
      le = launch_tma_pers<256>(ta, tb, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation, d_error);
    if (le != cudaSuccess) return ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(le));
  } else if (tma) {
    if (bn == 64)
      le = launch_tma<64>(ta, tb, grid, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation,
                          d_error, k_chunk, partial);
    else if (bn == 128)
      le = launch_tma<128>(ta, tb, grid, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation,
                           d_error, k_chunk, partial);
    else
      le = launch_tma<256>(ta, tb, grid, st, C, ldc, cb, M, N, K, alpha, beta, bias, activation,
                           d_error, k_chunk, partial);
    if (le != cudaSuccess) return ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(le));
  } else if (bn == 64) {
    k_gemm_bf16<64><<<grid, 128, 0, st>>>(
        static_cast<const __nv_bfloat16*>(A), lda, transA, static_cast<const __nv_bfloat16*>(B),
        ldb, transB, C, ldc, cb, M, N, K, alpha, beta, bias, activation, d_error, k_chunk, partial);
  } else {
    k_gemm_bf16<128><<<grid, 128, 0, st>>>(
        static_cast<const __nv_bfloat16*>(A), lda, transA, static_cast<const __nv_bfloat16*>(B),
        ldb, transB, C, ldc, cb, M, N, K, alpha, beta, bias, activation, d_error, k_chunk, partial);
  }
  if (splits > 1) {
    const long long mn = (long long)M * N;
    le = ci::launch_pdl(splits == 2  ? k_splitk_reduce<2>
                        : splits <= 4 ? k_splitk_reduce<4>
                                      : k_splitk_reduce<10>,
                        (unsigned)((mn + 255) / 256), 256, 0, st, partial, splits, C, ldc, cb, M, N,
                        alpha, beta, bias, activation);
    if (le != cudaSuccess) return ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(le));
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ci::set_last_error(CI_ERR_CUDA, cudaGetErrorString(e));
  return CI_OK;
}

}  // namespace

extern "C" int ci_gemm_bf16(const void* A, int lda, int transA, const void* B, int ldb, int transB,
                            float* C, int ldc, void* C_bf16, int M, int N, int K, float alpha,
                            float beta, const float* bias, int activation, int* d_error,
                            void* stream) {
  return gemm_bf16(A, lda, transA, B, ldb, transB, C, ldc, C_bf16, M, N, K, alpha, beta, bias,
                   activation, d_error, stream, false);
}
