// The leaf-value network: an MLP trained and evaluated on the GPU with the
// project's own BF16 tcgen05 GEMM (gemm_tc.cuh), FP32 accumulation and FP32
// master weights. No counterpart in the reference solver.
//
// Shapes: input in_dim -> `layers` hidden layers of width `hidden` with GELU
// -> linear output out_dim. Every dimension is padded to a multiple of 128
// (the GEMM tile); padded inputs, weights and outputs are zero and carry no
// gradient. Weights live in FP32 (Adam master copy, layout W_t[out][in]) and
// in two BF16 copies: W_t[out][in] (B operand of the forward GEMM) and
// W[in][out] (B operand of the input-gradient GEMM).
//
// Forward: X_{l+1} = gelu(X_l W_l + b_l) (pre-activation Z_l kept in BF16),
// Y = X_L W_L + b_L in FP32.
// Loss: sum over valid outputs of mask * (Y - T)^2 / sum(mask).
// Backward: dW_t[l] = dY_l^T X_l and db_l = column sums of dY_l (FP32);
// dY_{l-1} = (dY_l W_l) * gelu'(Z_{l-1}) fused in the GEMM epilogue.
// Adam updates the FP32 weights and writes both BF16 copies.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "../../include/dcfr.h"
#include "engine.hpp"
#include "gemm_tc.cuh"

namespace dcfr {
void set_last_error(const std::string& msg);
}

namespace {

using namespace dcfr;
using bf16 = __nv_bfloat16;

int fail(int code, const std::string& msg) {
  set_last_error(msg);
  return code;
}

#define MK(call)                                                                       \
  do {                                                                                 \
    cudaError_t _e = (call);                                                           \
    if (_e != cudaSuccess) return fail(DCFR_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
  } while (0)

inline int pad128(int x) { return (x + 127) / 128 * 128; }

// cuTensorMapEncodeTiled through the runtime's driver entry point.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// Tensor map of a row-major bf16 matrix [rows][cols] (cols contiguous), read
// in boxes of box_rows x 64 with the 128-byte swizzle.
int make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  auto enc = tensor_map_encoder();
  if (!enc) return fail(DCFR_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  if (((uintptr_t)base & 15) || (cols * 2) % 16) return fail(DCFR_ERR_INVALID_ARG, "GEMM operand is not 16-byte aligned");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {GEMM_BK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DCFR_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return DCFR_OK;
}

using GemmKernel = void (*)(CUtensorMap, CUtensorMap, GemmArgs);
struct GemmShape {
  GemmKernel kernel;
  int bn;
  size_t smem;
};
template <int BN, int STAGES, int CTAS, int DEPTH = 1>
GemmShape gemm_variant() {
  return GemmShape{(GemmKernel)gemm_bf16_tc_kernel<BN, STAGES, CTAS, DEPTH>, BN, gemm_smem(BN, STAGES, DEPTH)};
}

// The tile of an [M][N] output. 128 x 128, two to an SM with 3-stage rings, once
// that gives more CTAs than SMs (one's epilogue runs under the other's MMAs). With
// fewer, one to an SM with long steps, of the narrowest tile whose CTAs still
// run at once: 64 wide where those are 90 or more and no more than the SMs
// (M = 896, N = 1024), 128 where they are more (us a launch, 64 wide in two waves
// against 128 in one: 512 x 2688 x 1024 14.7 and 10.9, 2688 x 512 x 512 10.4 and 6.9,
// 1280 x 1024 x 2816 with GELU 27.7 and 20.3, 1408 x 1024 x 1024 18.2 and 14.1; 144 CTAs
// of 64, 512 x 2304 x 1024, 8.0 and 10.9). Below, 32 wide (M = 256), two to an SM only
// where there are more CTAs than SMs.
constexpr int SMS = 148;
GemmShape gemm_shape(int M, int N) {
  const int rows = M / GEMM_BM;
  if (rows * (N / 128) > SMS) return gemm_variant<128, 3, 2>();
  if (rows * (N / 64) > SMS) return gemm_variant<128, 3, 1, 2>();
  if (rows * (N / 64) >= 90) return gemm_variant<64, 3, 1, 3>();
  if (rows * (N / 32) > SMS) return gemm_variant<32, 5, 2>();
  return gemm_variant<32, 3, 1, 3>();
}

// Before a context's first gemm().
int gemm_setup() {
  for (const GemmShape& v : {gemm_variant<128, 3, 2>(), gemm_variant<128, 3, 1, 2>(), gemm_variant<64, 3, 1, 3>(),
                             gemm_variant<32, 5, 2>(), gemm_variant<32, 3, 1, 3>()})
    MK(cudaFuncSetAttribute((const void*)v.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v.smem));
  return DCFR_OK;
}

// C = epi(A[M][K] x B[N][K]^T); M, N multiples of 128, K of 64.
int gemm(const bf16* A, const bf16* B, int M, int N, int K, int epi, void* C, int ldc, bf16* z, const float* bias,
         int* err, cudaStream_t s) {
  if (M % GEMM_BM || N % 128 || K % GEMM_BK || M <= 0 || N <= 0 || K <= 0)
    return fail(DCFR_ERR_INVALID_ARG, "GEMM: M and N must be multiples of 128 and K of 64");
  const GemmShape v = gemm_shape(M, N);
  CUtensorMap ma, mb;
  int rc = make_map(&ma, A, (uint64_t)M, (uint64_t)K, GEMM_BM);
  if (rc) return rc;
  if ((rc = make_map(&mb, B, (uint64_t)N, (uint64_t)K, (uint32_t)v.bn))) return rc;
  const int wide = (((uintptr_t)C | (uintptr_t)z) & 15) == 0 && ldc % 8 == 0;
  GemmArgs G{C, z, bias, ldc, epi, M, N, K, wide, err};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(N / v.bn), (unsigned)(M / GEMM_BM));
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = v.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MK(cudaLaunchKernelEx(&cfg, v.kernel, ma, mb, G));
  return DCFR_OK;
}

// out[c][r] = in[r][c] (bf16, rows and cols multiples of 64) for up to 8
// matrices in one launch, tiles of 64 x 64 through shared memory with 16-byte
// accesses on both sides. The first `sums` blocks add up 64 columns each of
// the first matrix, 8 runs of rows a block, into db: a launch of its own for
// them took 7 us for 256 x 1024, as one for each matrix took 3 to 5 us.
constexpr int TRANSPOSE_MOST = 8;
struct TransposeSet {
  const bf16* in[TRANSPOSE_MOST];
  bf16* out[TRANSPOSE_MOST];
  int rows[TRANSPOSE_MOST], cols[TRANSPOSE_MOST];
  int n, sums;
  float* db;
};
// A tile of 64 x 64 at (r0, c0), transposed into out (whose rows are `rows` long).
__device__ __forceinline__ void store_transposed(const uint16_t (*t)[66], bf16* to, int rows, int r0, int c0) {
  uint16_t* out = reinterpret_cast<uint16_t*>(to);
  for (int i = threadIdx.x; i < 512; i += 256) {
    // Neighbouring threads take neighbouring columns of t: no bank conflicts.
    const int c = (i & 7) + ((i >> 6) << 3), r = ((i >> 3) & 7) * 8;
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = (uint32_t)t[r + 2 * k][c] | (uint32_t)t[r + 2 * k + 1][c] << 16;
    *reinterpret_cast<uint4*>(out + (size_t)(c0 + c) * rows + r0 + r) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
__device__ __forceinline__ void column_sums(const bf16* __restrict__ in0, int rows, int cols, float* __restrict__ db) {
  __shared__ float2 part[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const __nv_bfloat162* in = reinterpret_cast<const __nv_bfloat162*>(in0 + blockIdx.x * 64) + x;
  float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll 8
  for (int r = y; r < rows; r += 8) {
    const float2 v = __bfloat1622float2(in[(size_t)r * (cols / 2)]);
    acc.x += v.x;
    acc.y += v.y;
  }
  part[y][x] = acc;
  __syncthreads();
  if (y == 0) {
    for (int k = 1; k < 8; k++) {
      acc.x += part[k][x].x;
      acc.y += part[k][x].y;
    }
    reinterpret_cast<float2*>(db + blockIdx.x * 64)[x] = acc;
  }
}
__global__ void __launch_bounds__(256) transpose_bf16(const __grid_constant__ TransposeSet S) {
  if ((int)blockIdx.x < S.sums) return column_sums(S.in[0], S.rows[0], S.cols[0], S.db);
  __shared__ uint16_t t[64][66];
  int b = (int)blockIdx.x - S.sums, k = 0;
  while (b >= (S.rows[k] / 64) * (S.cols[k] / 64)) {
    b -= (S.rows[k] / 64) * (S.cols[k] / 64);
    k++;
  }
  const int rows = S.rows[k], cols = S.cols[k], r0 = b / (cols / 64) * 64, c0 = b % (cols / 64) * 64;
  const uint16_t* in = reinterpret_cast<const uint16_t*>(S.in[k]);
  for (int i = threadIdx.x; i < 512; i += 256) {
    const int r = i >> 3, c = (i & 7) * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(in + (size_t)(r0 + r) * cols + c0 + c);
    uint32_t* d = reinterpret_cast<uint32_t*>(&t[r][c]);
    d[0] = v.x;
    d[1] = v.y;
    d[2] = v.z;
    d[3] = v.w;
  }
  __syncthreads();
  store_transposed(t, S.out[k], rows, r0, c0);
}

// A set of transposes being put together.
struct Transposes : TransposeSet {
  int blocks = 0;
  Transposes() : TransposeSet{} {}
  void add(const bf16* from, bf16* to, int nrows, int ncols) {
    in[n] = from;
    out[n] = to;
    rows[n] = nrows;
    cols[n] = ncols;
    blocks += (nrows / 64) * (ncols / 64);
    n++;
  }
  // The column sums of the first matrix.
  void add_sums(float* to) {
    sums = cols[0] / 64;
    db = to;
    blocks += sums;
  }
  void launch(cudaStream_t s) const { transpose_bf16<<<blocks, 256, 0, s>>>(*this); }
};

// Row-major f32 [rows][cols] into a zero-padded bf16 [prow][pcol].
__global__ void pack_bf16(const float* __restrict__ in, int rows, int cols, bf16* __restrict__ out, int prow, int pcol) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)prow * pcol) return;
  const int r = (int)(i / pcol), c = (int)(i % pcol);
  out[i] = __float2bfloat16(r < rows && c < cols ? in[(size_t)r * cols + c] : 0.0f);
}

// f32 -> bf16, same layout.
__global__ void f32_to_bf16(const float* __restrict__ in, bf16* __restrict__ out, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16(in[i]);
}

// Sum over the block (256 threads), added to *to by its first thread: one
// atomic per block.
__device__ __forceinline__ void block_add(float v, float* to) {
  __shared__ float red[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < 8; w++) t += red[w];
    if (t != 0.0f) atomicAdd(to, t);
  }
}
// Blocks of the reductions: one atomic each on one address (an atomic per
// warp of a thread per element cost 34 us a reduction of 0.7 M elements).
constexpr int REDUCE_BLOCKS = 296;

// count[0] = number of valid outputs (sum of the mask, or rows * cols).
__global__ void __launch_bounds__(256) mask_count(const float* __restrict__ mask, size_t n, float* __restrict__ count) {
  float c = 0.0f;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    c += mask ? mask[i] : 1.0f;
  block_add(c, count);
}

// dY = 2 * mask * (Y - T) / count (bf16) and loss += mask * (Y - T)^2 / count,
// over the padded [prow][pcol] output; T and mask are [rows][cols] f32.
__global__ void __launch_bounds__(256) loss_grad(const float* __restrict__ Y, const float* __restrict__ T,
                                                 const float* __restrict__ mask, int rows, int cols, int prow, int pcol,
                                                 const float* __restrict__ count, bf16* __restrict__ dY,
                                                 float* __restrict__ loss) {
  const float inv_count = *count > 0.0f ? 1.0f / *count : 0.0f;
  float l = 0.0f;
  for (int r = blockIdx.x; r < prow; r += gridDim.x)
#pragma unroll 4
    for (int c = threadIdx.x; c < pcol; c += blockDim.x) {
      float g = 0.0f;
      if (r < rows && c < cols) {
        const size_t j = (size_t)r * cols + c;
        const float m = mask ? mask[j] : 1.0f;
        const float d = Y[(size_t)r * pcol + c] - T[j];
        g = 2.0f * m * d * inv_count;
        l += m * d * d * inv_count;
      }
      dY[(size_t)r * pcol + c] = __float2bfloat16(g);
    }
  block_add(l, loss);
}

// Adam on the f32 master copy: a block takes 64 x 64 weights of a layer and
// also writes their two bf16 copies, the second transposed through shared
// memory; the blocks after the tiles take 1024 biases each. Gradients of padded
// entries are zero by construction (pmask marks the real entries). Bound by
// memory: 33 bytes a weight (17 read, 16 written). As two launches (Adam with the first copy, then
// transposes that read it back) a step of 8.8 M parameters took 3 us longer.
struct AdamSet {
  bf16* wt[TRANSPOSE_MOST];
  size_t first[TRANSPOSE_MOST];
  int rows[TRANSPOSE_MOST], cols[TRANSPOSE_MOST];
  int n;
  size_t bias, biases;  // none: 0 biases
};
struct AdamArgs {
  float4* w;
  const float4* g;
  float4 *m, *v;
  const uchar4* pmask;
  bf16* w16;
  float lr, b1, b2, eps, c1, c2, gscale;
};
// The update of entries 4 i to 4 i + 3 for U values of i, all loads first.
template <int U>
__device__ __forceinline__ void adam4(const AdamArgs& A, const size_t (&at)[U], float4 (&wi)[U]) {
  uchar4 on[U];
  float4 mi[U], vi[U], gi[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    on[u] = A.pmask[at[u]];
    wi[u] = A.w[at[u]];
    gi[u] = A.g[at[u]];
    mi[u] = A.m[at[u]];
    vi[u] = A.v[at[u]];
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (!(&on[u].x)[k]) continue;
      const float gk = (&gi[u].x)[k] * A.gscale;
      const float mk = A.b1 * (&mi[u].x)[k] + (1.0f - A.b1) * gk;
      const float vk = A.b2 * (&vi[u].x)[k] + (1.0f - A.b2) * gk * gk;
      (&mi[u].x)[k] = mk;
      (&vi[u].x)[k] = vk;
      (&wi[u].x)[k] -= A.lr * (mk / A.c1) / (sqrtf(vk / A.c2) + A.eps);
    }
    A.w[at[u]] = wi[u];
    A.m[at[u]] = mi[u];
    A.v[at[u]] = vi[u];
  }
}
__global__ void __launch_bounds__(256) adam(const __grid_constant__ AdamSet S, const __grid_constant__ AdamArgs A) {
  __shared__ uint16_t t[64][66];
  int b = (int)blockIdx.x, k = 0;
  while (k < S.n && b >= (S.rows[k] / 64) * (S.cols[k] / 64)) {
    b -= (S.rows[k] / 64) * (S.cols[k] / 64);
    k++;
  }
  if (k == S.n) {
    const size_t i = (size_t)b * 256 + threadIdx.x, at[1] = {S.bias / 4 + i};
    float4 w[1];
    if (i < S.biases / 4) adam4<1>(A, at, w);
    return;
  }
  const int rows = S.rows[k], cols = S.cols[k], r0 = b / (cols / 64) * 64, c0 = b % (cols / 64) * 64;
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
#pragma unroll
  for (int half = 0; half < 64; half += 32) {
    size_t at[2];
    float4 w[2];
#pragma unroll
    for (int u = 0; u < 2; u++) at[u] = (S.first[k] + (size_t)(r0 + half + 16 * u + r) * cols + c0 + c) / 4;
    adam4<2>(A, at, w);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      union {
        uint2 u2;
        __nv_bfloat162 h[2];
      } o;
      o.h[0] = __floats2bfloat162_rn(w[u].x, w[u].y);
      o.h[1] = __floats2bfloat162_rn(w[u].z, w[u].w);
      reinterpret_cast<uint2*>(A.w16)[at[u]] = o.u2;
      uint32_t* d = reinterpret_cast<uint32_t*>(&t[half + 16 * u + r][c]);
      d[0] = o.u2.x;
      d[1] = o.u2.y;
    }
  }
  __syncthreads();
  store_transposed(t, S.wt[k], rows, r0, c0);
}

__global__ void copy_rows_f32(const float* __restrict__ in, int pcol, int rows, int cols, float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (size_t)rows * cols) out[i] = in[(i / cols) * pcol + (i % cols)];
}

inline unsigned blocks_for(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

struct dcfr_mlp {
  int in_dim, out_dim, hidden, layers;  // `layers` hidden layers + 1 output layer
  int max_batch;
  std::vector<int> kin, nout;           // padded dims per layer (L + 1 layers)
  std::vector<size_t> woff, boff;       // offsets of W_t and b in the flat parameter arrays
  size_t nparams = 0, nw = 0;
  float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // flat: all W_t then all b
  uint8_t* pmask = nullptr;
  bf16* w16 = nullptr;                  // all W_t in bf16, laid out as w
  std::vector<bf16*> wt_bf, w_bf;       // per layer: [N][K] (in w16) and [K][N]
  std::vector<bf16*> X, Z;              // activations [Mp][kin[l]] (X_0 = input) and pre-activations
  std::vector<bf16*> dY;                // [Mp][nout[l]]
  bf16 *tA = nullptr, *tB = nullptr;    // transposes for the weight-gradient GEMM
  float* Y = nullptr;                   // [Mp][nout[L]]
  float* loss = nullptr;                // [0] the loss, [1] the valid outputs, [2] err
  int* err = nullptr;                   // set by a GEMM whose wait gave up
  float* result = nullptr;              // page-locked copy of loss[0..2]
  int step = 0;
  cudaStream_t stream = nullptr, side = nullptr;      // side: the weights' gradients
  cudaEvent_t handed = nullptr;                       // work handed from one to the other
  ~dcfr_mlp() {
    if (side) cudaStreamSynchronize(side);
    for (void* p : std::vector<void*>{w, g, m, v, pmask, w16, tA, tB, Y, loss}) cudaFree(p);
    if (result) cudaFreeHost(result);
    for (auto* p : w_bf) cudaFree(p);
    for (auto* p : X) cudaFree(p);
    for (auto* p : Z) cudaFree(p);
    for (auto* p : dY) cudaFree(p);
    if (handed) cudaEventDestroy(handed);
    if (side) cudaStreamDestroy(side);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

// The transposed weights, from the bf16 copy.
int refresh_transposed(dcfr_mlp* n) {
  for (int l = 0; l <= n->layers;) {
    Transposes T;
    for (; l <= n->layers && T.n < TRANSPOSE_MOST; l++) T.add(n->wt_bf[l], n->w_bf[l], n->nout[l], n->kin[l]);
    T.launch(n->stream);
  }
  MK(cudaGetLastError());
  return DCFR_OK;
}

int refresh_bf16(dcfr_mlp* n) {
  f32_to_bf16<<<blocks_for(n->nw, 256), 256, 0, n->stream>>>(n->w, n->w16, n->nw);
  return refresh_transposed(n);
}

// The layers on Mp packed input rows.
int forward_packed(dcfr_mlp* n, int Mp, cudaStream_t s) {
  int rc;
  for (int l = 0; l < n->layers; l++)
    if ((rc = gemm(n->X[l], n->wt_bf[l], Mp, n->nout[l], n->kin[l], EPI_BIAS_GELU, n->X[l + 1], n->nout[l], n->Z[l],
                   n->w + n->boff[l], n->err, s)))
      return rc;
  const int L = n->layers;
  return gemm(n->X[L], n->wt_bf[L], Mp, n->nout[L], n->kin[L], EPI_BIAS_F32, n->Y, n->nout[L], nullptr,
              n->w + n->boff[L], n->err, s);
}

int forward(dcfr_mlp* n, const float* x, int M, int Mp) {
  pack_bf16<<<blocks_for((size_t)Mp * n->kin[0], 256), 256, 0, n->stream>>>(x, M, n->in_dim, n->X[0], Mp, n->kin[0]);
  return forward_packed(n, Mp, n->stream);
}

// Lets `to` wait for what `from` holds now.
int after(cudaStream_t to, cudaStream_t from, cudaEvent_t e) {
  MK(cudaEventRecord(e, from));
  MK(cudaStreamWaitEvent(to, e, 0));
  return DCFR_OK;
}

// Forward pass, then the gradients of the loss into n->g (and the loss into
// n->loss). The chain dY_L .. dY_0 is what takes the time (a GEMM of 256 rows
// uses less than half the SMs), so the weights' gradients, which only need
// each dY, run beside it on a second stream, and so does the count of valid
// outputs, beside the forward pass: a step of 256 rows, 1024 wide, 362 us
// before, 280 now.
int gradients(dcfr_mlp* n, const float* x, const float* target, const float* mask, int M) {
  const int L = n->layers, Mp = pad128(M);
  int rc;
  // loss[0]: the loss; loss[1]: the number of valid outputs (the normaliser).
  if ((rc = after(n->side, n->stream, n->handed))) return rc;
  MK(cudaMemsetAsync(n->loss, 0, 8, n->side));
  mask_count<<<REDUCE_BLOCKS, 256, 0, n->side>>>(mask, (size_t)M * n->out_dim, n->loss + 1);
  if ((rc = forward(n, x, M, Mp))) return rc;
  if ((rc = after(n->stream, n->side, n->handed))) return rc;
  loss_grad<<<std::min(Mp, REDUCE_BLOCKS), 256, 0, n->stream>>>(
      n->Y, target, mask, M, n->out_dim, Mp, n->nout[L], n->loss + 1, n->dY[L], n->loss);
  for (int l = L; l >= 0; l--) {
    const int K = n->kin[l], N = n->nout[l];
    if ((rc = after(n->side, n->stream, n->handed))) return rc;
    if (l > 0) {
      // dY_{l-1} = (dY_l W_l) * gelu'(Z_{l-1}): B operand W_l as [K][N].
      if ((rc = gemm(n->dY[l], n->w_bf[l], Mp, K, N, EPI_GELU_GRAD, n->dY[l - 1], K, n->Z[l - 1], nullptr, n->err,
                     n->stream)))
        return rc;
    }
    // dW_t[l] [N][K] = dY_l^T X_l: operands dY_l^T [N][Mp] and X_l^T [K][Mp].
    Transposes T;
    T.add(n->dY[l], n->tA, Mp, N);
    T.add(n->X[l], n->tB, Mp, K);
    T.add_sums(n->g + n->boff[l]);
    T.launch(n->side);
    if ((rc = gemm(n->tA, n->tB, N, K, Mp, EPI_F32, n->g + n->woff[l], K, nullptr, nullptr, n->err, n->side)))
      return rc;
  }
  if ((rc = after(n->stream, n->side, n->handed))) return rc;
  MK(cudaGetLastError());
  return DCFR_OK;
}

// Waits for the stream; the loss and the GEMMs' error flag come back in one
// copy.
int check_err(dcfr_mlp* n, float* loss = nullptr) {
  MK(cudaMemcpyAsync(n->result, n->loss, 12, cudaMemcpyDeviceToHost, n->stream));
  MK(cudaStreamSynchronize(n->stream));
  int e = 0;
  std::memcpy(&e, n->result + 2, 4);
  if (e) return fail(DCFR_ERR_DEVICE_TIMEOUT, "tensor-core GEMM: a bounded wait gave up (code " + std::to_string(e) + ")");
  if (loss) *loss = n->result[0];
  return DCFR_OK;
}

int batch_ok(dcfr_mlp* n, int M) {
  if (M <= 0 || M > n->max_batch) return fail(DCFR_ERR_INVALID_ARG, "batch size out of range");
  return DCFR_OK;
}

}  // namespace

namespace dcfr {

int mlp_shape(const dcfr_mlp* n, int* in_dim, int* out_dim, int* max_batch) {
  if (!n) return fail(DCFR_ERR_INVALID_ARG, "NULL network");
  *in_dim = n->in_dim;
  *out_dim = n->out_dim;
  *max_batch = n->max_batch;
  return DCFR_OK;
}

// The rows that a forward pass reads: a solver writes its inputs there.
bf16* mlp_input(dcfr_mlp* n, int* ldx) {
  *ldx = n->kin[0];
  return n->X[0];
}

// The network's forward pass on the first m packed input rows on stream s,
// nothing synchronised: a solver enqueues it between its kernels (and captures
// it in its graphs). y is the network's own padded output buffer, valid until
// its next forward pass.
int mlp_enqueue_forward(dcfr_mlp* n, int m, cudaStream_t s, const float** y, int* ldy) {
  int rc = batch_ok(n, m);
  if (rc) return rc;
  if ((rc = forward_packed(n, pad128(m), s))) return rc;
  *y = n->Y;
  *ldy = n->nout[n->layers];
  return DCFR_OK;
}

}  // namespace dcfr

extern "C" {

int dcfr_gemm_bf16(const void* a, const void* b, void* c, int32_t m, int32_t n, int32_t k, int32_t epi,
                   const float* bias, void* z, int32_t ldc, void* stream) {
  int* err = nullptr;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  MK(cudaMalloc(&err, 4));
  MK(cudaMemsetAsync(err, 0, 4, s));
  int rc = gemm_setup();
  if (!rc)
    rc = gemm(static_cast<const bf16*>(a), static_cast<const bf16*>(b), m, n, k, epi, c, ldc, static_cast<bf16*>(z),
              bias, err, s);
  int e = 0;
  if (!rc) {
    MK(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, s));
    MK(cudaStreamSynchronize(s));
  }
  cudaFree(err);
  if (rc) return rc;
  if (e) return fail(DCFR_ERR_DEVICE_TIMEOUT, "tensor-core GEMM: a bounded wait gave up");
  set_last_error("");
  return DCFR_OK;
}

int dcfr_gemm_bf16_timed(const void* a, const void* b, void* c, int32_t m, int32_t n, int32_t k, int32_t epi,
                         const float* bias, void* z, int32_t ldc, int32_t reps, void* stream, float* ms_per_launch) {
  if (reps <= 0 || !ms_per_launch) return fail(DCFR_ERR_INVALID_ARG, "reps must be positive; ms_per_launch not NULL");
  int* err = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  MK(cudaMalloc(&err, 4));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  MK(cudaMemsetAsync(err, 0, 4, s));
  MK(cudaEventCreate(&e0));
  MK(cudaEventCreate(&e1));
  int rc = gemm_setup(), e = 0;
  MK(cudaEventRecord(e0, s));
  for (int r = 0; r < reps && !rc; r++)
    rc = gemm(static_cast<const bf16*>(a), static_cast<const bf16*>(b), m, n, k, epi, c, ldc, static_cast<bf16*>(z),
              bias, err, s);
  MK(cudaEventRecord(e1, s));
  if (!rc) {
    MK(cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, s));
    MK(cudaStreamSynchronize(s));
    float ms = 0.0f;
    MK(cudaEventElapsedTime(&ms, e0, e1));
    *ms_per_launch = ms / (float)reps;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(err);
  if (rc) return rc;
  if (e) return fail(DCFR_ERR_DEVICE_TIMEOUT, "tensor-core GEMM: a bounded wait gave up");
  set_last_error("");
  return DCFR_OK;
}

int dcfr_mlp_create(int32_t in_dim, int32_t hidden, int32_t layers, int32_t out_dim, int32_t max_batch,
                    uint64_t seed, dcfr_mlp** out) {
  if (!out || in_dim <= 0 || out_dim <= 0 || hidden <= 0 || hidden % 128 || layers < 1 || max_batch <= 0)
    return fail(DCFR_ERR_INVALID_ARG, "MLP shape: positive dims, hidden a multiple of 128, at least one layer");
  std::unique_ptr<dcfr_mlp> n(new dcfr_mlp());
  n->in_dim = in_dim;
  n->out_dim = out_dim;
  n->hidden = hidden;
  n->layers = layers;
  n->max_batch = max_batch;
  const int L = layers + 1;
  for (int l = 0; l < L; l++) {
    n->kin.push_back(l == 0 ? pad128(in_dim) : hidden);
    n->nout.push_back(l == layers ? pad128(out_dim) : hidden);
  }
  for (int l = 0; l < L; l++) {
    n->woff.push_back(n->nw);
    n->nw += (size_t)n->nout[l] * n->kin[l];
  }
  n->nparams = n->nw;
  for (int l = 0; l < L; l++) {
    n->boff.push_back(n->nparams);
    n->nparams += n->nout[l];
  }
  MK(cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking));
  MK(cudaStreamCreateWithFlags(&n->side, cudaStreamNonBlocking));
  if (int set = gemm_setup()) return set;
  MK(cudaEventCreateWithFlags(&n->handed, cudaEventDisableTiming));
  // He-style init of the real entries, zeros in the padding; biases zero.
  std::vector<float> hw(n->nparams, 0.0f);
  std::vector<uint8_t> hm(n->nparams, 0);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < L; l++) {
    const int kr = l == 0 ? in_dim : hidden, nr = l == layers ? out_dim : hidden;
    std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)kr) * (l == layers ? 0.5f : 1.0f));
    for (int r = 0; r < nr; r++)
      for (int c = 0; c < kr; c++) {
        const size_t i = n->woff[l] + (size_t)r * n->kin[l] + c;
        hw[i] = nd(rng);
        hm[i] = 1;
      }
    for (int r = 0; r < nr; r++) hm[n->boff[l] + r] = 1;
  }
  const int Mp = pad128(max_batch);
  MK(cudaMalloc(&n->w, n->nparams * 4));
  MK(cudaMalloc(&n->g, n->nparams * 4));
  MK(cudaMalloc(&n->m, n->nparams * 4));
  MK(cudaMalloc(&n->v, n->nparams * 4));
  MK(cudaMalloc(&n->pmask, n->nparams));
  MK(cudaMemcpy(n->w, hw.data(), n->nparams * 4, cudaMemcpyHostToDevice));
  MK(cudaMemcpy(n->pmask, hm.data(), n->nparams, cudaMemcpyHostToDevice));
  MK(cudaMemset(n->m, 0, n->nparams * 4));
  MK(cudaMemset(n->v, 0, n->nparams * 4));
  MK(cudaMalloc(&n->w16, n->nw * 2));
  size_t tmax = 0;
  for (int l = 0; l < L; l++) {
    bf16* b = nullptr;
    MK(cudaMalloc(&b, (size_t)n->nout[l] * n->kin[l] * 2));
    n->wt_bf.push_back(n->w16 + n->woff[l]);
    n->w_bf.push_back(b);
    tmax = std::max(tmax, (size_t)std::max(n->kin[l], n->nout[l]));
  }
  for (int l = 0; l < L; l++) {
    bf16* x = nullptr;
    MK(cudaMalloc(&x, (size_t)Mp * n->kin[l] * 2));
    MK(cudaMemset(x, 0, (size_t)Mp * n->kin[l] * 2));
    n->X.push_back(x);
  }
  for (int l = 0; l < L; l++) {
    bf16 *z = nullptr, *d = nullptr;
    MK(cudaMalloc(&z, (size_t)Mp * n->nout[l] * 2));
    MK(cudaMalloc(&d, (size_t)Mp * n->nout[l] * 2));
    n->Z.push_back(z);
    n->dY.push_back(d);
  }
  MK(cudaMalloc(&n->tA, (size_t)Mp * tmax * 2));
  MK(cudaMalloc(&n->tB, (size_t)Mp * tmax * 2));
  MK(cudaMalloc(&n->Y, (size_t)Mp * n->nout[layers] * 4));
  MK(cudaMalloc(&n->loss, 12));
  MK(cudaMemset(n->loss, 0, 12));
  n->err = reinterpret_cast<int*>(n->loss + 2);
  MK(cudaMallocHost(&n->result, 12));
  MK(cudaStreamSynchronize(cudaStreamLegacy));  // the copies and memsets above
  int rc = refresh_bf16(n.get());
  if (rc) return rc;
  MK(cudaStreamSynchronize(n->stream));
  *out = n.release();
  set_last_error("");
  return DCFR_OK;
}

void dcfr_mlp_destroy(dcfr_mlp* n) { delete n; }

int dcfr_mlp_num_params(const dcfr_mlp* n, uint64_t* out) {
  if (!n || !out) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  *out = n->nparams;
  return DCFR_OK;
}

// Parameters in the padded flat layout (all W_t[l][out][in], then all b[l]).
int dcfr_mlp_get_params(const dcfr_mlp* n, float* host) {
  if (!n || !host) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  MK(cudaMemcpy(host, n->w, n->nparams * 4, cudaMemcpyDeviceToHost));
  return DCFR_OK;
}

int dcfr_mlp_set_params(dcfr_mlp* n, const float* host) {
  if (!n || !host) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  // On the stream that reads them next: a copy from pageable memory may still
  // be on its way to the device when cudaMemcpy returns.
  MK(cudaMemcpyAsync(n->w, host, n->nparams * 4, cudaMemcpyHostToDevice, n->stream));
  int rc = refresh_bf16(n);
  if (rc) return rc;
  MK(cudaStreamSynchronize(n->stream));
  return DCFR_OK;
}

int dcfr_mlp_forward(dcfr_mlp* n, const float* x, int32_t M, float* y) {
  if (!n || !x || !y) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  int rc = batch_ok(n, M);
  if (rc) return rc;
  const int Mp = pad128(M);
  if ((rc = forward(n, x, M, Mp))) return rc;
  const int L = n->layers;
  copy_rows_f32<<<blocks_for((size_t)M * n->out_dim, 256), 256, 0, n->stream>>>(n->Y, n->nout[L], M, n->out_dim, y);
  MK(cudaGetLastError());
  return check_err(n);
}

// Loss and gradients (flat padded layout, host) without updating.
int dcfr_mlp_gradients(dcfr_mlp* n, const float* x, const float* target, const float* mask, int32_t M, float* loss,
                       float* grads_host) {
  if (!n || !x || !target) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  int rc = batch_ok(n, M);
  if (rc) return rc;
  if ((rc = gradients(n, x, target, mask, M))) return rc;
  if ((rc = check_err(n, loss))) return rc;
  if (grads_host) MK(cudaMemcpy(grads_host, n->g, n->nparams * 4, cudaMemcpyDeviceToHost));
  return DCFR_OK;
}

// One Adam step (beta1 0.9, beta2 0.999, eps 1e-8, bias-corrected) on the
// device gradients times gscale, then the bf16 weight copies.
static int adam_step(dcfr_mlp* n, float lr, float gscale) {
  n->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - std::pow(b1, (float)n->step), c2 = 1.0f - std::pow(b2, (float)n->step);
  const AdamArgs A{reinterpret_cast<float4*>(n->w), reinterpret_cast<const float4*>(n->g),
                   reinterpret_cast<float4*>(n->m), reinterpret_cast<float4*>(n->v),
                   reinterpret_cast<const uchar4*>(n->pmask), n->w16, lr, b1, b2, 1e-8f, c1, c2, gscale};
  for (int l = 0; l <= n->layers;) {
    AdamSet S{};
    unsigned blocks = 0;
    for (; l <= n->layers && S.n < TRANSPOSE_MOST; l++, S.n++) {
      S.wt[S.n] = n->w_bf[l];
      S.first[S.n] = n->woff[l];
      S.rows[S.n] = n->nout[l];
      S.cols[S.n] = n->kin[l];
      blocks += (unsigned)((n->nout[l] / 64) * (n->kin[l] / 64));
    }
    if (l > n->layers) {
      S.bias = n->nw;
      S.biases = n->nparams - n->nw;
      blocks += blocks_for(S.biases / 4, 256);
    }
    adam<<<blocks, 256, 0, n->stream>>>(S, A);
  }
  MK(cudaGetLastError());
  return DCFR_OK;
}

int dcfr_mlp_train_step(dcfr_mlp* n, const float* x, const float* target, const float* mask, int32_t M, float lr,
                        float* loss) {
  if (!n || !x || !target) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  int rc = batch_ok(n, M);
  if (rc) return rc;
  if ((rc = gradients(n, x, target, mask, M))) return rc;
  if ((rc = adam_step(n, lr, 1.0f))) return rc;
  if ((rc = check_err(n, loss))) return rc;
  return DCFR_OK;
}

// Data-parallel training: the loss and gradients of this rank's batch stay
// on the device (the stream is synchronised on return), the caller sums them
// across ranks in place (an all-reduce on dcfr_mlp_gradients_device's
// buffer), then dcfr_mlp_adam_step applies Adam to the sum times gscale.
int dcfr_mlp_backward(dcfr_mlp* n, const float* x, const float* target, const float* mask, int32_t M, float* loss) {
  if (!n || !x || !target) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  int rc = batch_ok(n, M);
  if (rc) return rc;
  if ((rc = gradients(n, x, target, mask, M))) return rc;
  return check_err(n, loss);
}

int dcfr_mlp_gradients_device(dcfr_mlp* n, float** grads, uint64_t* count) {
  if (!n || !grads || !count) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  *grads = n->g;
  *count = n->nparams;
  return DCFR_OK;
}

int dcfr_mlp_adam_step(dcfr_mlp* n, float lr, float gscale) {
  if (!n) return fail(DCFR_ERR_INVALID_ARG, "NULL argument");
  int rc = adam_step(n, lr, gscale);
  if (rc) return rc;
  return check_err(n);
}

}  // extern "C"
