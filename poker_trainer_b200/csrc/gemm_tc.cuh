// BF16 x BF16 -> FP32 GEMM on the 5th-generation tensor cores (tcgen05) for
// the leaf-value network (mlp.cu):
//
//   C[M][N] = epilogue( sum_k A[M][K] * B[N][K] )
//
// A and B are row-major with K contiguous (both operands "K-major"). One CTA
// computes a 128 x BN tile of C:
//   * warp 0, one thread: TMA loads of 128 x 64 tiles of A and BN x 64 tiles of
//     B, DEPTH of each a step, into a ring of STAGES steps in shared memory
//     (128-byte swizzle, the canonical K-major layout the tensor core reads);
//   * warp 1, one thread: tcgen05.mma (M=128, N=BN, K=16 per instruction,
//     FP32 accumulator in tensor memory), a tcgen05.commit per stage frees
//     the stage, a last commit marks the accumulator complete;
//   * all eight warps: the epilogue reads the accumulator with tcgen05.ld
//     (warp w owns rows 32 (w % 4) on, and half the columns) and writes C
//     through the epilogue.
// The tile and the ring depend on how many CTAs a product gives (gemm_shape):
// the network's products at a few hundred rows are a few dozen 128 x 128
// tiles, bound by the ring's latency (a TMA round trip is about 1 us, a
// 64-deep step of the tile a tenth of that) and, with GELU, by the epilogue.
// Narrower tiles put more SMs to work on both, and a CTA that has an SM to
// itself takes a ring twice as deep. us a launch, against 128 x 128 tiles with
// 3 stages and 4 warps throughout: 896 x 1024 x 2816 with GELU 44.8 to 18.7,
// 896 x 1024 x 1024 37.1 to 10.9, 256 x 1024 x 2816 41.3 to 17.4, 256 x 1024 x
// 1024 33.0 to 9.4, 896 x 2688 x 1024 with bias 18.2 to 12.4; 8192 x 1024 x 2816
// with GELU 105.7 to 60.0, plain 4096 x 1024 x 2816 28.4 to 27.6.
// In one CTA alone on an SM a step of the ring costs about 0.14 us of barriers,
// commit and polling, whatever the tile, and 0.14 us for each 64 of K: steps of
// 128 or 192 there, and one warp that polls instead of eight. us a launch at
// steps of 64 and now: 256 x 1024 x 2816 with GELU 17.4 to 12.2, 256 x 1024 x 1024
// 9.6 to 7.2, 896 x 1024 x 2816 19.1 to 15.1, 896 x 1024 x 1024 10.9 to 9.9, 896 x
// 2688 x 1024 15.6 to 14.7. Two CTAs on an SM hide each other's steps (256 x 2688 x
// 1024: 10.1, one CTA with long steps 13.3; 4096 x 1024 x 2816: one polling warp
// 28.4 against 27.9).
// Every wait on an mbarrier is bounded; a wait that gives up records an error
// code and the CTA skips the rest of its work, frees its tensor memory and
// returns.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"

namespace dcfr {

constexpr int GEMM_BM = 128, GEMM_BK = 64, GEMM_THREADS = 256;
constexpr uint32_t GEMM_A_BYTES = GEMM_BM * GEMM_BK * 2;  // one 128 x 64 bf16 tile
constexpr size_t gemm_smem(int bn, int stages, int depth) {
  return 1024 + (size_t)stages * depth * (GEMM_A_BYTES + (size_t)bn * GEMM_BK * 2) + 256;
}
constexpr long long GEMM_WAIT_LIMIT = 1ll << 22;  // polls before a wait gives up (well over a second)

// Epilogues.
enum GemmEpi : int {
  EPI_F32 = 0,            // C (f32) = acc
  EPI_BIAS_F32 = 1,       // C (f32) = acc + bias[n]
  EPI_BIAS_GELU = 2,      // Z (bf16) = acc + bias[n]; C (bf16) = gelu(acc + bias[n])
  EPI_GELU_GRAD = 3,      // C (bf16) = acc * gelu'(Z[m][n])
};

struct GemmArgs {
  void* c;               // f32 or bf16 output [M][ldc]
  __nv_bfloat16* z;      // EPI_BIAS_GELU: pre-activation out; EPI_GELU_GRAD: pre-activation in
  const float* bias;     // [N]
  int ldc;
  int epi;
  int M, N, K;
  int wide;              // bf16 outputs: c, z and ldc allow 16-byte accesses
  int* error;            // set to a nonzero code when a bounded wait gives up
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: false if the barrier did not complete the phase in time.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (long long i = 0; i < GEMM_WAIT_LIMIT; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// Shared-memory matrix descriptor (tcgen05): K-major, 128-byte swizzle,
// 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t sw128_desc(const void* p) {
  const uint64_t addr = smem_u32(p);
  uint64_t d = 0;
  d |= (addr & 0x3FFFF) >> 4;       // start address [0,14)
  d |= (uint64_t)1 << 16;           // leading byte offset (unused for swizzled K-major), [16,30)
  d |= (uint64_t)(1024 >> 4) << 32; // stride byte offset [32,46)
  d |= (uint64_t)1 << 46;           // descriptor version [46,48)
  d |= (uint64_t)2 << 61;           // layout: 128-byte swizzle [61,64)
  return d;
}

// Instruction descriptor: kind::f16, BF16 A and B, FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int m, int n) {
  return (1u << 4)                     // D format F32
         | (1u << 7)                   // A format BF16
         | (1u << 10)                  // B format BF16
         | ((uint32_t)(n >> 3) << 17)  // N >> 3
         | ((uint32_t)(m >> 4) << 24); // M >> 4
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * expf(-0.5f * x * x);
}

template <int BN, int STAGES, int CTAS, int DEPTH>
__global__ void __launch_bounds__(GEMM_THREADS, CTAS)
    gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                        GemmArgs G) {
  extern __shared__ __align__(1024) unsigned char gemm_smem_raw[];
  constexpr uint32_t B_BYTES = BN * GEMM_BK * 2;
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)gemm_smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sa = smem;
  unsigned char* sb = smem + STAGES * DEPTH * GEMM_A_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(sb + STAGES * DEPTH * B_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* accf = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accf + 1);
  __shared__ int failed;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * GEMM_BM, n0 = blockIdx.x * BN;
  const int nb = G.K / GEMM_BK, nk = (nb + DEPTH - 1) / DEPTH;  // 64-wide blocks of K, steps

  if (tid == 0) {
    failed = 0;
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accf, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();
  pdl_wait();

  if (warp == 0 && lane == 0) {
    // Producer.
    for (int kb = 0; kb < nk; kb++) {
      const int s = kb % STAGES;
      if (kb >= STAGES && !mbar_wait(&empty[s], ((kb / STAGES) - 1) & 1)) {
        failed = 1;
        break;
      }
      const int d1 = min(DEPTH, nb - kb * DEPTH);
      mbar_expect_tx(&full[s], d1 * (GEMM_A_BYTES + B_BYTES));
#pragma unroll
      for (int d = 0; d < DEPTH; d++) {
        if (d >= d1) break;
        const int at = s * DEPTH + d, x = (kb * DEPTH + d) * GEMM_BK;
        tma_load_2d(sa + at * GEMM_A_BYTES, &map_a, &full[s], x, m0);
        tma_load_2d(sb + at * B_BYTES, &map_b, &full[s], x, n0);
      }
    }
  } else if (warp == 1 && lane == 0) {
    // Tensor-core issue.
    const uint32_t idesc = idesc_bf16_f32(GEMM_BM, BN);
    for (int kb = 0; kb < nk; kb++) {
      const int s = kb % STAGES;
      if (!mbar_wait(&full[s], (kb / STAGES) & 1)) {
        failed = 2;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int d1 = min(DEPTH, nb - kb * DEPTH);
#pragma unroll
      for (int d = 0; d < DEPTH; d++) {
        if (d >= d1) break;
        const int at = s * DEPTH + d;
        const uint64_t da = sw128_desc(sa + at * GEMM_A_BYTES), db = sw128_desc(sb + at * B_BYTES);
#pragma unroll
        for (int k = 0; k < GEMM_BK / 16; k++)  // K = 16 per instruction: 32 bytes along the swizzled row
          umma_bf16(tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kb > 0 || d > 0 || k > 0) ? 1u : 0u);
      }
      umma_commit(&empty[s]);
    }
    umma_commit(accf);
  }
  __syncwarp();
  // Epilogue: every thread owns half a row of the tile.
  bool go;  // the same for a warp at least: tcgen05.ld is warp-collective
  if constexpr (CTAS == 1) {
    // One warp polls, the others wait at the barrier.
    if (warp == 0 && !mbar_wait(accf, 0) && lane == 0) atomicExch(&failed, 3);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    go = *(volatile int*)&failed == 0;
  } else {
    const bool ok = mbar_wait(accf, 0);
    if (!ok && lane == 0) atomicExch(&failed, 3);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    go = __all_sync(0xffffffffu, ok && *(volatile int*)&failed == 0);
  }
  if (go) {
    constexpr int HALF = BN / 2, STEP = HALF < 32 ? HALF : 32;
    const int quarter = warp & 3;
    const int m = m0 + quarter * 32 + lane;
    const uint32_t row_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const int cbeg = (warp >> 2) * HALF;
#pragma unroll 1
    for (int c0 = cbeg; c0 < cbeg + HALF; c0 += STEP) {
      uint32_t v[STEP];
      if constexpr (STEP == 32) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
            "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16 % STEP]), "=r"(v[17 % STEP]), "=r"(v[18 % STEP]), "=r"(v[19 % STEP]), "=r"(v[20 % STEP]),
              "=r"(v[21 % STEP]), "=r"(v[22 % STEP]), "=r"(v[23 % STEP]), "=r"(v[24 % STEP]), "=r"(v[25 % STEP]),
              "=r"(v[26 % STEP]), "=r"(v[27 % STEP]), "=r"(v[28 % STEP]), "=r"(v[29 % STEP]), "=r"(v[30 % STEP]),
              "=r"(v[31 % STEP])
            : "r"(row_addr + (uint32_t)c0));
      } else {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(row_addr + (uint32_t)c0));
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (m < G.M) {
        const int nb = n0 + c0;
        if (G.epi == EPI_F32 || G.epi == EPI_BIAS_F32) {
          float* out = reinterpret_cast<float*>(G.c) + (size_t)m * G.ldc + nb;
#pragma unroll
          for (int j = 0; j < STEP; j += 4) {
            float4 o;
            o.x = __uint_as_float(v[j]) + (G.epi == EPI_BIAS_F32 ? G.bias[nb + j] : 0.0f);
            o.y = __uint_as_float(v[j + 1]) + (G.epi == EPI_BIAS_F32 ? G.bias[nb + j + 1] : 0.0f);
            o.z = __uint_as_float(v[j + 2]) + (G.epi == EPI_BIAS_F32 ? G.bias[nb + j + 2] : 0.0f);
            o.w = __uint_as_float(v[j + 3]) + (G.epi == EPI_BIAS_F32 ? G.bias[nb + j + 3] : 0.0f);
            *reinterpret_cast<float4*>(out + j) = o;
          }
        } else {
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(G.c) + (size_t)m * G.ldc + nb;
          __nv_bfloat16* zz = G.z + (size_t)m * G.ldc + nb;
#pragma unroll
          for (int j = 0; j < STEP; j += 8) {
            union {
              uint4 u;
              __nv_bfloat162 h[4];
            } z4, r4;
            if (G.epi == EPI_GELU_GRAD) {
              if (G.wide) z4.u = *reinterpret_cast<const uint4*>(zz + j);
              else
                for (int i = 0; i < 4; i++) z4.h[i] = *reinterpret_cast<const __nv_bfloat162*>(zz + j + 2 * i);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
              float a = __uint_as_float(v[j + 2 * i]), b = __uint_as_float(v[j + 2 * i + 1]);
              if (G.epi == EPI_BIAS_GELU) {
                a += G.bias[nb + j + 2 * i];
                b += G.bias[nb + j + 2 * i + 1];
                z4.h[i] = __floats2bfloat162_rn(a, b);
                r4.h[i] = __floats2bfloat162_rn(gelu(a), gelu(b));
              } else {
                r4.h[i] = __floats2bfloat162_rn(a * gelu_grad(__bfloat162float(z4.h[i].x)),
                                                b * gelu_grad(__bfloat162float(z4.h[i].y)));
              }
            }
            if (G.wide) {
              if (G.epi == EPI_BIAS_GELU) *reinterpret_cast<uint4*>(zz + j) = z4.u;
              *reinterpret_cast<uint4*>(out + j) = r4.u;
            } else {
              for (int i = 0; i < 4; i++) {
                if (G.epi == EPI_BIAS_GELU) *reinterpret_cast<__nv_bfloat162*>(zz + j + 2 * i) = z4.h[i];
                *reinterpret_cast<__nv_bfloat162*>(out + j + 2 * i) = r4.h[i];
              }
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (failed && tid == 0 && G.error) atomicExch(G.error, failed);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
  }
}

}  // namespace dcfr
