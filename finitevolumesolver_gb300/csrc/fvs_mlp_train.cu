// fvs_mlp_train.cu -- the learned Newton start value: tcgen05 GEMM, training
// (forward, backward, Adam) and batched inference of the 5 -> 64 -> 64 -> 1
// GELU perceptron, all hand-written for sm_103a.
//
// A training step is two kernels.  FusedStepKernel: a CTA takes tiles of 128
// batch rows through the whole forward and backward pass, every operand of
// the five products staged in shared memory and every accumulator in tensor
// memory (bf16 operands, fp32 accumulation):
//   X   [128][16] bf16   sampled rows, standardised, columns 5..15 zero
//   Z1  = X W1^T + b1,   H1 = GELU(Z1) (bf16)
//   Z2  = H1 W2^T + b2,  y = GELU(Z2) . w3 + b3 (CUDA cores)
//   dZ2 = (dy w3) * GELU'(Z2) (bf16), dH1 = dZ2 W2, dZ1 = dH1 * GELU'(Z1) (bf16)
//   [dZ2 | dZ1]^T [H1 | X]: one 128 x 80 product whose diagonal blocks are dW2
//   and dW1, accumulated in tensor memory over the CTA's tiles
// with the loss the mean squared error against y* = log(p* / max(pL, pR)).
// It writes the CTA's sums of the gradient; UpdateKernel adds them over the
// CTAs in a fixed order, applies Adam and publishes the bf16 weights.
//
// The step is latency: 0.2 GFLOP at batch 8192.  As twelve kernels (gather,
// one GEMM kernel per product, activations, reductions by atomics, Adam) with
// their operands in global memory it took 121 us on the GB300; fused it takes
// 20 us.
#include "../../include/fvs_gpu.h"
#include "fvs_internal.h"
#include "fvs_mlp.cuh"
#include "fvs_tcgen05.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace fvs {
namespace mlpk {

constexpr int kH = mlp::kHidden;  // 64
constexpr int kXin = 16;          // padded input width

// ---------------------------------------------------------------------------
// tcgen05 GEMM: C[M x N] (+)= A[M x K] . B[N x K]^T

struct GemmArgs {
  const __nv_bfloat16* A;
  int lda;
  const __nv_bfloat16* B;
  int ldb;
  float* C;
  int ldc;
  int M, K;
  int k_per_cta;  // multiple of 16; blockIdx.y selects the K range
  int atomic;     // 1: atomicAdd into C (split K), 0: store
  int* error;
};

// Operands arrive by TMA: for every 8-element K slice of a chunk, one 2-D
// tensor-map box of 16 bytes x rows lands as `rows` consecutive 16-byte rows,
// i.e. a column of 8 x 16-byte core matrices.  In the canonical K-major
// no-swizzle layout that is SBO = 128 bytes (next 8-row group) and LBO =
// rows * 16 bytes (next K slice).  Rows beyond the tensor are zero-filled.
template <int N>
__global__ void __launch_bounds__(tc::kThreads)
    TcGemmKernel(GemmArgs a, const __grid_constant__ CUtensorMap tmA,
                 const __grid_constant__ CUtensorMap tmB) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar, mma_bar;
  __shared__ uint32_t tmem_base;
  const uint32_t raw = tc::SmemAddr(smem_raw);
  uint8_t* sA = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  uint8_t* sB = sA + tc::kTileM * tc::kChunkK * 2;
  constexpr uint32_t kCols = N < 32 ? 32 : N;
  constexpr uint32_t kSbo = 128;
  constexpr uint32_t kLboA = tc::kTileM * 16;
  constexpr uint32_t kLboB = N * 16;
  constexpr uint32_t kIdesc = tc::InstrDescBf16(tc::kTileM, N);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * tc::kTileM;
  const int k_begin = blockIdx.y * a.k_per_cta;
  const int k_end = min(a.K, k_begin + a.k_per_cta);
  if (warp == 0) tc::TmemAlloc(&tmem_base, kCols);
  if (tid == 0) {
    tc::MbarInit(&full_bar, 1);
    tc::MbarInit(&mma_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::FenceBeforeSync();
  __syncthreads();
  tc::FenceAfterSync();
  const uint32_t tmem = tmem_base;
  uint32_t phase = 0;
  bool ok = true;       // CTA-uniform: decided with __syncthreads_or
  bool pending = false;  // copies or MMAs issued but not seen complete
  bool first = true;
  for (int kc = k_begin; kc < k_end && ok; kc += tc::kChunkK) {
    const int slices = min(tc::kChunkK, k_end - kc) / 8;
    if (tid == 0) {
      tc::MbarArriveExpectTx(&full_bar, uint32_t(slices) * (kLboA + kLboB));
      for (int sl = 0; sl < slices; ++sl) {
        tc::TmaLoad2D(sA + sl * kLboA, &tmA, kc + 8 * sl, m0, &full_bar);
        tc::TmaLoad2D(sB + sl * kLboB, &tmB, kc + 8 * sl, 0, &full_bar);
      }
    }
    pending = true;
    const bool landed = tc::MbarWait(&full_bar, phase, 1u << 22);
    ok = !__syncthreads_or(landed ? 0 : 1);
    if (!ok) break;
    if (tid == 0) {
      tc::FenceAfterSync();
      const uint32_t abase = tc::SmemAddr(sA), bbase = tc::SmemAddr(sB);
      for (int ks = 0; ks < slices / 2; ++ks) {
        const uint64_t ad = tc::SmemDesc(abase + 2 * ks * kLboA, kLboA, kSbo);
        const uint64_t bd = tc::SmemDesc(bbase + 2 * ks * kLboB, kLboB, kSbo);
        tc::Mma(tmem, ad, bd, kIdesc, (first && ks == 0) ? 0u : 1u);
      }
      tc::Commit(&mma_bar);
    }
    first = false;
    const bool done = tc::MbarWait(&mma_bar, phase, 1u << 22);
    tc::FenceAfterSync();
    ok = !__syncthreads_or(done ? 0 : 1);
    if (ok) {
      phase ^= 1u;
      pending = false;
    }
  }
  if (!ok && pending) {
    // A copy or the tensor core did not signal in time: record it and give
    // the copies and MMAs of this chunk a second bounded chance to drain
    // before shared and tensor memory are released.
    if (tid == 0 && a.error) atomicOr(a.error, 1);
    tc::MbarWait(&full_bar, phase, 1u << 22);
    tc::MbarWait(&mma_bar, phase, 1u << 22);
  }
  if (ok && !first) {
    const int row = m0 + warp * 32 + lane;
#pragma unroll
    for (int c0 = 0; c0 < N; c0 += 16) {
      float v[16];
      tc::TmemLoad16(tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), v);
      if (row < a.M) {
        float* crow = a.C + int64_t(row) * a.ldc + c0;
        if (a.atomic) {
#pragma unroll
          for (int i = 0; i < 16; ++i) atomicAdd(crow + i, v[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) crow[i] = v[i];
        }
      }
    }
  }
  tc::FenceBeforeSync();
  __syncthreads();
  if (warp == 0) tc::TmemDealloc(tmem, kCols);
}

using tma::EncodeTiled;
using tma::EncodeTiledFn;

// Tensor map of a row-major bf16 matrix [rows][inner] with row pitch `ld`
// elements; boxes of 8 elements x box_rows rows.
cudaError_t MakeOperandMap(CUtensorMap* m, const __nv_bfloat16* base, int inner, int rows, int ld,
                           int box_rows) {
  EncodeTiledFn fn = EncodeTiled();
  if (!fn) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {cuuint64_t(inner), cuuint64_t(rows)};
  const cuuint64_t strides[1] = {cuuint64_t(ld) * 2};
  const cuuint32_t box[2] = {8u, cuuint32_t(box_rows)};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                        const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int N>
cudaError_t LaunchGemm(const GemmArgs& a, int splits, cudaStream_t s) {
  // the operands' rows must start on 16-byte boundaries (TMA global strides)
  if ((a.lda % 8) != 0 || (a.ldb % 8) != 0 || (reinterpret_cast<uintptr_t>(a.A) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(a.B) & 15) != 0 || (a.K % 16) != 0 || (a.k_per_cta % 16) != 0)
    return cudaErrorInvalidValue;
  alignas(64) CUtensorMap tmA, tmB;
  cudaError_t e = MakeOperandMap(&tmA, a.A, a.K, a.M, a.lda, tc::kTileM);
  if (e == cudaSuccess) e = MakeOperandMap(&tmB, a.B, a.K, N, a.ldb, N);
  if (e != cudaSuccess) return e;
  const size_t smem = 1024 + size_t(tc::kTileM) * tc::kChunkK * 2 + size_t(N) * tc::kChunkK * 2;
  static bool attr_set = false;
  if (!attr_set) {
    e = cudaFuncSetAttribute(TcGemmKernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(smem));
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  dim3 grid(unsigned((a.M + tc::kTileM - 1) / tc::kTileM), unsigned(splits));
  TcGemmKernel<N><<<grid, tc::kThreads, smem, s>>>(a, tmA, tmB);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The network

// GELU and its derivative from one tanh.
__device__ __forceinline__ float GeluBoth(float x, float* grad) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float t = tanhf(k0 * fmaf(k1 * x * x, x, x));
  *grad = 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * k0 * fmaf(3.0f * k1, x * x, 1.0f);
  return 0.5f * x * (1.0f + t);
}

// Features and labels of Riemann problems given by primitive states.
__global__ void FeaturesKernel(int64_t n, const double* rhoL, const double* uL, const double* pL,
                               const double* rhoR, const double* uR, const double* pR,
                               const double* pstar, double gamma, float* feat, float* label) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double aL = sqrt(gamma * pL[i] / rhoL[i]);
  const double aR = sqrt(gamma * pR[i] / rhoR[i]);
  float x[mlp::kIn];
  mlp::Features(x, rhoL[i], uL[i], pL[i], aL, rhoR[i], uR[i], pR[i], aR);
#pragma unroll
  for (int k = 0; k < mlp::kIn; ++k) feat[i * mlp::kIn + k] = x[k];
  if (label && pstar) {
    const double pref = pL[i] > pR[i] ? pL[i] : pR[i];
    label[i] = static_cast<float>(log(pstar[i] / pref));
  }
}

// Mean and standard deviation of the raw features (double accumulation).
__global__ void MomentsKernel(int64_t n, const float* feat, double* acc) {
  double s[mlp::kIn] = {0}, q[mlp::kIn] = {0};
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
#pragma unroll
    for (int k = 0; k < mlp::kIn; ++k) {
      const double v = feat[i * mlp::kIn + k];
      s[k] += v;
      q[k] += v * v;
    }
  }
#pragma unroll
  for (int k = 0; k < mlp::kIn; ++k) {
    atomicAdd(acc + k, s[k]);
    atomicAdd(acc + mlp::kIn + k, q[k]);
  }
}

struct Net {
  // fp32 master parameters in the inference blob layout (mlp::kParams floats)
  float* master;
  // Adam moments, same layout
  float* m1;
  float* m2;
  float* grad;
  // inference blob: bf16-rounded weights widened to fp32
  float* blob;
  __nv_bfloat16* W1;   // [64][16]
  __nv_bfloat16* W2;   // [64][64]
  __nv_bfloat16* W2t;  // [64][64] transposed
};

// Parameter i's bf16 copies (weights) and its entry of the inference blob.
__device__ __forceinline__ void PublishOne(const Net& net, int i, float w) {
  float out = w;
  if (i >= mlp::kOffW1 && i < mlp::kOffB1) {
    const int o = (i - mlp::kOffW1) / mlp::kIn, k = (i - mlp::kOffW1) % mlp::kIn;
    const __nv_bfloat16 b = __float2bfloat16_rn(w);
    net.W1[o * kXin + k] = b;
    out = __bfloat162float(b);
  } else if (i >= mlp::kOffW2 && i < mlp::kOffB2) {
    const int o = (i - mlp::kOffW2) / kH, k = (i - mlp::kOffW2) % kH;
    const __nv_bfloat16 b = __float2bfloat16_rn(w);
    net.W2[o * kH + k] = b;
    net.W2t[k * kH + o] = b;
    out = __bfloat162float(b);
  }
  net.blob[i] = out;
}

__global__ void PublishKernel(Net net) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < mlp::kParams) PublishOne(net, i, net.master[i]);
}

__device__ __forceinline__ uint64_t Mix(uint64_t x) {
  // SplitMix64 finaliser
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// 512 threads: thread t works on row 32 (warp % 4) + lane of the tile (the
// TMEM lanes its warp can read) and on the 16 hidden units 16 (warp / 4) ...
constexpr int kFusedThreads = 512;
constexpr int kTile = tc::kTileM;  // 128 rows
// shared-memory operands (canonical K-major layout, element (r, k) at
// (k / 8) * LBO + 16 r + 2 (k % 8)); the transposed operands' slices are
// padded by 16 bytes so that a warp's 2-byte stores to them (consecutive k of
// one r) fall into different banks
constexpr uint32_t kLboRow = kTile * 16;     // X, H1, dZ2: 128 rows
constexpr uint32_t kLboW = kH * 16;          // W1, W2, W2^T: 64 rows
constexpr uint32_t kLboG = kTile * 16 + 16;  // [dZ2 | dZ1]^T: 128 rows
constexpr int kNG = kH + kXin;               // columns of [H1 | X]
constexpr uint32_t kLboN = kNG * 16 + 16;    // [H1 | X]^T: 80 rows
constexpr uint32_t kOffSX = 0;
constexpr uint32_t kOffSW1 = kOffSX + 2 * kLboRow;
constexpr uint32_t kOffSW2 = kOffSW1 + 2 * kLboW;
constexpr uint32_t kOffSH1 = kOffSW2 + 8 * kLboW;
// GELU(Z2) of the tile, [128][65] fp32: the output layer's sum runs over a
// row's units in order, so that its rounding does not depend on the tiling
constexpr int kActPitch = kH + 1;
constexpr uint32_t kOffAct = kOffSH1 + 8 * kLboRow;
constexpr uint32_t kForwardSmem = kOffAct + kTile * kActPitch * 4;
constexpr uint32_t kOffSW2t = kForwardSmem;
constexpr uint32_t kOffSD2 = kOffSW2t + 8 * kLboW;
constexpr uint32_t kOffSG = kOffSD2 + 8 * kLboRow;
constexpr uint32_t kOffSN = kOffSG + 16 * kLboG;
constexpr uint32_t kFusedSmem = kOffSN + 16 * kLboN;
// tensor-memory columns: Z1, Z2, dH1 (64 each), the weight gradients (80)
constexpr uint32_t kColZ1 = 0, kColZ2 = 64, kColDh = 128, kColDw = 192;
constexpr uint32_t kFusedCols = 512, kInferCols = 128;
constexpr int kPartial = mlp::kParams + 1;  // a CTA's gradient sums and its loss
constexpr int kMaxCtas = 152;
constexpr uint32_t kPolls = 1u << 22;

// One product into tensor-memory columns `col`: A (128 rows) and B of `slices`
// 8-element K slices.  Issued by one thread.
__device__ __forceinline__ void IssueMma(uint32_t tmem, uint32_t col, uint32_t a, uint32_t lbo_a,
                                         uint32_t b, uint32_t lbo_b, int n, int slices,
                                         bool accumulate, uint64_t* bar) {
  tc::FenceAfterSync();
  const uint32_t idesc = tc::InstrDescBf16(tc::kTileM, n);
  for (int ks = 0; ks < slices / 2; ++ks)
    tc::Mma(tmem + col, tc::SmemDesc(a + 2 * ks * lbo_a, lbo_a, 128),
            tc::SmemDesc(b + 2 * ks * lbo_b, lbo_b, 128), idesc, (accumulate || ks > 0) ? 1u : 0u);
  tc::Commit(bar);
}

// The CTA's MMAs and their completion barrier.  Every wait is bounded: after
// a timeout `ok` is false (in every thread alike), the error flag is set and
// no further product is issued.
struct MmaPhases {
  uint64_t* bar;
  int* error;
  uint32_t phase = 0;
  bool ok = true;
  // operands in shared memory are written, thread 0 issues `f`, all wait
  template <class F> __device__ __forceinline__ void Run(F f) {
    tc::FenceProxyAsync();
    tc::FenceBeforeSync();
    __syncthreads();
    if (ok) {
      if (threadIdx.x == 0) f();
      const bool landed = tc::MbarWait(bar, phase, kPolls);
      ok = !__syncthreads_or(landed ? 0 : 1);
      if (!ok) {
        if (threadIdx.x == 0 && error) atomicOr(error, 1);
        tc::MbarWait(bar, phase, kPolls);  // a second bounded chance to drain
      }
      phase ^= 1u;
    }
    tc::FenceAfterSync();
  }
};

__device__ __forceinline__ uint32_t Pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// 16 units of a row as two 16-byte K slices of a row-major operand.
__device__ __forceinline__ void StoreUnits(uint8_t* op, int row, int group, const float* v) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint4 w;
    w.x = Pack2(v[8 * h], v[8 * h + 1]);
    w.y = Pack2(v[8 * h + 2], v[8 * h + 3]);
    w.z = Pack2(v[8 * h + 4], v[8 * h + 5]);
    w.w = Pack2(v[8 * h + 6], v[8 * h + 7]);
    *reinterpret_cast<uint4*>(op + (2 * group + h) * kLboRow + row * 16) = w;
  }
}

// 16 units of a row into the transposed operand (rows unit0.., K = row).
__device__ __forceinline__ void StoreTransposed(uint8_t* op, uint32_t lbo, int unit0, int row,
                                                const float* v) {
#pragma unroll
  for (int i = 0; i < 16; ++i)
    *reinterpret_cast<__nv_bfloat16*>(op + (row >> 3) * lbo + (unit0 + i) * 16 + (row & 7) * 2) =
        __float2bfloat16_rn(v[i]);
}

// bf16 weights [64][width] (row-major) as K slices of 64 rows.
__device__ __forceinline__ void LoadWeights(uint8_t* op, const __nv_bfloat16* w, int width) {
  for (int c = threadIdx.x; c < kH * width / 8; c += blockDim.x) {
    const int r = c / (width / 8), sl = c % (width / 8);
    *reinterpret_cast<uint4*>(op + sl * kLboW + r * 16) =
        *reinterpret_cast<const uint4*>(w + r * width + sl * 8);
  }
}

// Standardised features of a row as its X operand (columns 5..15 zero).
__device__ __forceinline__ void StoreFeatures(uint8_t* op, int row, const float* f,
                                              const float* stats, float* x) {
#pragma unroll
  for (int k = 0; k < mlp::kIn; ++k)
    x[k] = (f[k] - stats[mlp::kOffMean + k]) * stats[mlp::kOffInvStd + k];
  uint4 w;
  w.x = Pack2(x[0], x[1]);
  w.y = Pack2(x[2], x[3]);
  w.z = Pack2(x[4], 0.0f);
  w.w = 0u;
  *reinterpret_cast<uint4*>(op + row * 16) = w;
  *reinterpret_cast<uint4*>(op + kLboRow + row * 16) = make_uint4(0u, 0u, 0u, 0u);
}

// Sums over the warp's 32 lanes of 16 values each: lane l (even) ends with the
// sum of value *index (16 shuffles instead of 80).
__device__ __forceinline__ float SumUnits(float* v, int lane, int* index) {
  int at = 0;
#pragma unroll
  for (int m = 16, n = 8; m >= 2; m >>= 1, n >>= 1) {
    const bool up = (lane & m) != 0;
    at += up ? n : 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n];
      const float keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
  }
  *index = at;
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The output layer of a row.
__device__ __forceinline__ float OutputSum(const float* act, const float* w3, float b3) {
  float y = b3;
#pragma unroll 16
  for (int o = 0; o < kH; ++o) y = fmaf(w3[o], act[o], y);
  return y;
}

struct FusedArgs {
  const float* feat;   // raw features [n][5]
  const float* label;  // [n]
  int64_t n;
  uint64_t seed;
  int batch;
  int given_rows;      // 1: rows 0..batch-1 of feat (gradient check)
  int count;           // 1: a training step (the step counter advances)
  // step[0]: steps the sampling has seen (UpdateKernel advances it);
  // step[1]: Adam's step number (this kernel advances it, UpdateKernel takes
  // that back for a failed step).  Neither kernel reads the counter it writes.
  unsigned long long* step;
  const float* blob;   // statistics, biases, output weights
  const __nv_bfloat16* W1;
  const __nv_bfloat16* W2;
  const __nv_bfloat16* W2t;
  float* partial;      // [gridDim.x][kPartial]
  int* error;
};

__global__ void __launch_bounds__(kFusedThreads) FusedStepKernel(FusedArgs a) {
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ float vec[mlp::kParams - mlp::kOffB2];  // b2, w3, b3
  __shared__ float b1[kH], stats[2 * mlp::kIn];
  __shared__ float residual[kTile], target[kTile];
  // per row-warp sums over the tiles: db1, db2, dw3 and (db3, loss)
  __shared__ float sums[4][3 * kH + 2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rw = warp & 3, group = warp >> 2, row = rw * 32 + lane, u0 = group * 16;
  if (warp == 0) tc::TmemAlloc(&tmem_base, kFusedCols);
  if (tid == 0) {
    tc::MbarInit(&bar, 1);
    tma::FenceMbarInit();
  }
  // (nothing here waits for memory ahead of the weights' loads)
  if (tid == 32 && a.count && blockIdx.x == 0) atomicAdd(a.step + 1, 1ull);
  LoadWeights(sm + kOffSW1, a.W1, kXin);
  LoadWeights(sm + kOffSW2, a.W2, kH);
  LoadWeights(sm + kOffSW2t, a.W2t, kH);
  for (int i = tid; i < mlp::kParams - mlp::kOffB2; i += blockDim.x) vec[i] = a.blob[mlp::kOffB2 + i];
  if (tid < kH) b1[tid] = a.blob[mlp::kOffB1 + tid];
  if (tid < 2 * mlp::kIn) stats[tid] = a.blob[mlp::kOffMean + tid];
  for (int i = tid; i < 4 * (3 * kH + 2); i += blockDim.x) (&sums[0][0])[i] = 0.0f;
  tc::FenceBeforeSync();
  __syncthreads();
  tc::FenceAfterSync();
  const uint32_t tmem = tmem_base;
  const uint32_t lanes = tmem + (uint32_t(rw * 32) << 16);
  const uint32_t base = tc::SmemAddr(sm);
  const float* w3 = vec + (mlp::kOffW3 - mlp::kOffB2);
  const float b3 = vec[mlp::kOffB3 - mlp::kOffB2];
  float* act = reinterpret_cast<float*>(sm + kOffAct);
  const unsigned long long step = a.step[0];
  MmaPhases mma{&bar, a.error};
  const int tiles = a.batch / kTile;
  bool first = true;
  for (int tile = blockIdx.x; tile < tiles && mma.ok; tile += gridDim.x) {
    if (group == 0) {
      const int r = tile * kTile + row;
      int64_t src = r;
      if (!a.given_rows) {
        const uint64_t h = Mix(a.seed ^ Mix(step * 0x100000001ull + uint64_t(r)));
        src = int64_t(h % uint64_t(a.n));
      }
      float f[mlp::kIn], x[mlp::kIn];
#pragma unroll
      for (int k = 0; k < mlp::kIn; ++k) f[k] = a.feat[src * mlp::kIn + k];
      target[row] = a.label[src];
      StoreFeatures(sm + kOffSX, row, f, stats, x);
#pragma unroll
      for (int k = 0; k < kXin; ++k)
        *reinterpret_cast<__nv_bfloat16*>(sm + kOffSN + (row >> 3) * kLboN + (kH + k) * 16 +
                                          (row & 7) * 2) =
            __float2bfloat16_rn(k < mlp::kIn ? x[k < mlp::kIn ? k : 0] : 0.0f);
    }
    float v[16], g1[16], d[16], gw[16];
    mma.Run([&] {
      IssueMma(tmem, kColZ1, base + kOffSX, kLboRow, base + kOffSW1, kLboW, kH, 2, false, &bar);
    });
    tc::TmemLoad16(lanes + kColZ1 + u0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = GeluBoth(v[i] + b1[u0 + i], &g1[i]);
    StoreUnits(sm + kOffSH1, row, group, v);
    StoreTransposed(sm + kOffSN, kLboN, u0, row, v);
    mma.Run([&] {
      IssueMma(tmem, kColZ2, base + kOffSH1, kLboRow, base + kOffSW2, kLboW, kH, 8, false, &bar);
    });
    tc::TmemLoad16(lanes + kColZ2 + u0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      gw[i] = GeluBoth(v[i] + vec[u0 + i], &d[i]);
      act[row * kActPitch + u0 + i] = gw[i];
    }
    __syncthreads();
    if (group == 0) residual[row] = OutputSum(act + row * kActPitch, w3, b3) - target[row];
    __syncthreads();
    const float e = residual[row];
    const float dy = 2.0f * e / float(a.batch);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      gw[i] = dy * gw[i];
      d[i] = dy * w3[u0 + i] * d[i];
    }
    StoreUnits(sm + kOffSD2, row, group, d);
    StoreTransposed(sm + kOffSG, kLboG, u0, row, d);
    int at;
    const float sd = SumUnits(d, lane, &at), sw = SumUnits(gw, lane, &at);
    if (!(lane & 1)) {
      sums[rw][kH + u0 + at] += sd;
      sums[rw][2 * kH + u0 + at] += sw;
    }
    if (group == 0) {
      float g3 = dy, e2 = e * e;
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        g3 += __shfl_xor_sync(0xffffffffu, g3, m);
        e2 += __shfl_xor_sync(0xffffffffu, e2, m);
      }
      if (lane == 0) {
        sums[rw][3 * kH] += g3;
        sums[rw][3 * kH + 1] += e2;
      }
    }
    mma.Run([&] {
      IssueMma(tmem, kColDh, base + kOffSD2, kLboRow, base + kOffSW2t, kLboW, kH, 8, false, &bar);
    });
    tc::TmemLoad16(lanes + kColDh + u0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= g1[i];
    StoreTransposed(sm + kOffSG, kLboG, kH + u0, row, v);
    const float s1 = SumUnits(v, lane, &at);
    if (!(lane & 1)) sums[rw][u0 + at] += s1;
    mma.Run([&] {
      IssueMma(tmem, kColDw, base + kOffSG, kLboG, base + kOffSN, kLboN, kNG, 16, !first, &bar);
    });
    first = false;
  }
  __syncthreads();
  float* out = a.partial + int64_t(blockIdx.x) * kPartial;
  if (mma.ok && !first) {
    // rows 0..63: dW2 [out][in]; rows 64..127, columns 64..68: dW1
    if (rw < 2) {
      float v[16];
      tc::TmemLoad16(lanes + kColDw + u0, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) out[mlp::kOffW2 + row * kH + u0 + i] = v[i];
    } else if (group == 0) {
      float v[16];
      tc::TmemLoad16(lanes + kColDw + kH, v);
#pragma unroll
      for (int k = 0; k < mlp::kIn; ++k) out[mlp::kOffW1 + (row - kH) * mlp::kIn + k] = v[k];
    }
  }
  if (tid < 3 * kH + 2) {
    const float t = ((sums[0][tid] + sums[1][tid]) + sums[2][tid]) + sums[3][tid];
    const int k = tid % kH;
    const int at = tid < kH ? mlp::kOffB1 + k
                 : tid < 2 * kH ? mlp::kOffB2 + k
                 : tid < 3 * kH ? mlp::kOffW3 + k
                 : tid == 3 * kH ? mlp::kOffB3
                                 : mlp::kParams;
    out[at] = t;
  }
  if (tid < mlp::kOffW1) out[tid] = 0.0f;
  tc::FenceBeforeSync();
  __syncthreads();
  if (warp == 0) tc::TmemDealloc(tmem, kFusedCols);
}

// The gradient (the CTAs' partial sums added in a fixed order), and with
// `update` Adam (lr, beta1 0.9, beta2 0.999, eps 1e-8) and the published
// weights.  Blocks of 32 parameters x 8 parts of the CTAs.  Once a wait for the
// tensor cores has run out (*error), the sums are not a gradient: the weights,
// the moments and the counters stay as they were before the step.
__global__ void __launch_bounds__(256)
    UpdateKernel(Net net, const float* partial, int ctas, int update, float lr,
                 unsigned long long* step, float* loss, const int* error) {
  __shared__ float part[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + x;
  const bool failed = *error != 0;
  float s = 0.0f;
  if (i < kPartial)
    for (int c = y; c < ctas; c += 8) s += partial[int64_t(c) * kPartial + i];
  part[y][x] = s;
  __syncthreads();
  if (y != 0 || i >= kPartial) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) s += part[k][x];
  if (i == mlp::kParams) {
    if (failed) {
      if (update) step[1] -= 1;
      return;
    }
    *loss += s;
    if (update) step[0] += 1;
    return;
  }
  if (failed) return;
  net.grad[i] = s;
  if (!update || i < mlp::kOffW1) return;
  const unsigned long long t = step[1];
  const float m = 0.9f * net.m1[i] + 0.1f * s;
  const float v = 0.999f * net.m2[i] + 0.001f * s * s;
  net.m1[i] = m;
  net.m2[i] = v;
  const float mh = m / (1.0f - powf(0.9f, float(t)));
  const float vh = v / (1.0f - powf(0.999f, float(t)));
  const float w = net.master[i] - lr * mh / (sqrtf(vh) + 1e-8f);
  net.master[i] = w;
  PublishOne(net, i, w);
}

// Inference: the forward half of FusedStepKernel over tiles of 128 rows.
__global__ void __launch_bounds__(kFusedThreads)
    InferKernel(int64_t n, const float* feat, const float* blob, const __nv_bfloat16* W1,
                const __nv_bfloat16* W2, float* y_out, int* error) {
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ float vec[mlp::kParams - mlp::kOffB2];
  __shared__ float b1[kH], stats[2 * mlp::kIn];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rw = warp & 3, group = warp >> 2, row = rw * 32 + lane, u0 = group * 16;
  if (warp == 0) tc::TmemAlloc(&tmem_base, kInferCols);
  if (tid == 0) {
    tc::MbarInit(&bar, 1);
    tma::FenceMbarInit();
  }
  LoadWeights(sm + kOffSW1, W1, kXin);
  LoadWeights(sm + kOffSW2, W2, kH);
  for (int i = tid; i < mlp::kParams - mlp::kOffB2; i += blockDim.x) vec[i] = blob[mlp::kOffB2 + i];
  if (tid < kH) b1[tid] = blob[mlp::kOffB1 + tid];
  if (tid < 2 * mlp::kIn) stats[tid] = blob[mlp::kOffMean + tid];
  tc::FenceBeforeSync();
  __syncthreads();
  tc::FenceAfterSync();
  const uint32_t tmem = tmem_base;
  const uint32_t lanes = tmem + (uint32_t(rw * 32) << 16);
  const uint32_t base = tc::SmemAddr(sm);
  const float* w3 = vec + (mlp::kOffW3 - mlp::kOffB2);
  float* act = reinterpret_cast<float*>(sm + kOffAct);
  MmaPhases mma{&bar, error};
  const int64_t tiles = (n + kTile - 1) / kTile;
  for (int64_t tile = blockIdx.x; tile < tiles && mma.ok; tile += gridDim.x) {
    const int64_t r = tile * kTile + row;
    if (group == 0) {
      const int64_t src = r < n ? r : n - 1;
      float f[mlp::kIn], x[mlp::kIn];
#pragma unroll
      for (int k = 0; k < mlp::kIn; ++k) f[k] = feat[src * mlp::kIn + k];
      StoreFeatures(sm + kOffSX, row, f, stats, x);
    }
    float v[16], unused;
    mma.Run([&] {
      IssueMma(tmem, kColZ1, base + kOffSX, kLboRow, base + kOffSW1, kLboW, kH, 2, false, &bar);
    });
    tc::TmemLoad16(lanes + kColZ1 + u0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = GeluBoth(v[i] + b1[u0 + i], &unused);
    StoreUnits(sm + kOffSH1, row, group, v);
    mma.Run([&] {
      IssueMma(tmem, kColZ2, base + kOffSH1, kLboRow, base + kOffSW2, kLboW, kH, 8, false, &bar);
    });
    tc::TmemLoad16(lanes + kColZ2 + u0, v);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      act[row * kActPitch + u0 + i] = GeluBoth(v[i] + vec[u0 + i], &unused);
    __syncthreads();
    if (group == 0 && r < n && mma.ok)
      y_out[r] = OutputSum(act + row * kActPitch, w3, vec[mlp::kOffB3 - mlp::kOffB2]);
  }
  tc::FenceBeforeSync();
  __syncthreads();
  if (warp == 0) tc::TmemDealloc(tmem, kInferCols);
}

}  // namespace mlpk
}  // namespace fvs

// ---------------------------------------------------------------------------
// C ABI

using namespace fvs::mlpk;

struct fvs_mlp {
  Net net{};
  float* buf = nullptr;  // master, m1, m2, grad, blob
  __nv_bfloat16* wbuf = nullptr;
  int* error = nullptr;
  unsigned long long* step = nullptr;  // [2], see FusedArgs::step
  cudaStream_t stream = nullptr;
  float* partial = nullptr;  // [kMaxCtas][kPartial]
  float* loss = nullptr;     // sum of squared errors of the steps since its reset
  int ctas = 1;              // CTAs of the fused kernels (one per SM)
  ~fvs_mlp() {
    if (partial) cudaFree(partial);
    if (loss) cudaFree(loss);
    if (buf) cudaFree(buf);
    if (wbuf) cudaFree(wbuf);
    if (error) cudaFree(error);
    if (step) cudaFree(step);
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

int MlpFail(int code, const std::string& msg) {
  fvs::SetLastError(msg);
  return code;
}

int MlpCuda(cudaError_t e, const char* what) {
  fvs::SetLastError(std::string(what) + ": " + cudaGetErrorString(e));
  return FVS_ERR_CUDA;
}

#define MLP_CUDA(call)                                  \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return MlpCuda(e_, #call);   \
  } while (0)

// The fused kernels' dynamic shared memory, set once per handle.
cudaError_t SetSmem() {
  cudaError_t e = cudaFuncSetAttribute(
      FusedStepKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFusedSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(InferKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             int(kForwardSmem));
  return e;
}

// One training step (update) or one gradient of the given rows on the stream.
cudaError_t EnqueueStep(fvs_mlp* m, FusedArgs a, bool update, float lr) {
  a.step = m->step;
  a.blob = m->net.blob;
  a.W1 = m->net.W1;
  a.W2 = m->net.W2;
  a.W2t = m->net.W2t;
  a.partial = m->partial;
  a.error = m->error;
  a.count = update ? 1 : 0;
  const int grid = std::min(a.batch / kTile, m->ctas);
  FusedStepKernel<<<grid, kFusedThreads, kFusedSmem, m->stream>>>(a);
  UpdateKernel<<<(kPartial + 31) / 32, 256, 0, m->stream>>>(m->net, m->partial, grid,
                                                            update ? 1 : 0, lr, m->step, m->loss,
                                                            m->error);
  return cudaGetLastError();
}

uint64_t HostMix(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

}  // namespace

extern "C" {

int fvs_mlp_param_count(void) { return fvs::mlp::kParams; }

int fvs_tc_gemm_bf16(const void* A_dev, int lda, const void* B_dev, int ldb, float* C_dev, int ldc,
                     int M, int N, int K, int splits, int accumulate, void* stream) {
  if (!A_dev || !B_dev || !C_dev || M < 1 || K < 16 || K % 16 != 0 || splits < 1)
    return MlpFail(FVS_ERR_INVALID, "need M >= 1, K a positive multiple of 16, splits >= 1");
  if (N != 16 && N != 32 && N != 64)
    return MlpFail(FVS_ERR_UNSUPPORTED, "N must be 16, 32 or 64");
  if (lda < K || ldb < K || ldc < N || lda % 8 != 0 || ldb % 8 != 0 ||
      (reinterpret_cast<uintptr_t>(A_dev) & 15) != 0 || (reinterpret_cast<uintptr_t>(B_dev) & 15) != 0)
    return MlpFail(FVS_ERR_INVALID, "operands must be 16-byte aligned with lda, ldb >= K (multiples of 8)");
  if (splits > 1 && !accumulate)
    return MlpFail(FVS_ERR_INVALID, "split K needs accumulate = 1");
  const int per = (K / splits + 15) / 16 * 16;
  const int used = (K + per - 1) / per;
  static int* err = nullptr;
  if (!err) {
    MLP_CUDA(cudaMalloc(&err, sizeof(int)));
    MLP_CUDA(cudaMemset(err, 0, sizeof(int)));
  }
  GemmArgs g{};
  g.A = static_cast<const __nv_bfloat16*>(A_dev);
  g.lda = lda;
  g.B = static_cast<const __nv_bfloat16*>(B_dev);
  g.ldb = ldb;
  g.C = C_dev;
  g.ldc = ldc;
  g.M = M;
  g.K = K;
  g.k_per_cta = per;
  g.atomic = accumulate;
  g.error = err;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = N == 16 ? LaunchGemm<16>(g, used, s)
                : N == 32 ? LaunchGemm<32>(g, used, s)
                          : LaunchGemm<64>(g, used, s);
  MLP_CUDA(e);
  int h = 0;
  MLP_CUDA(cudaMemcpyAsync(&h, err, sizeof h, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(cudaStreamSynchronize(s));
  if (h) return MlpFail(FVS_ERR_CUDA, "tensor-core wait timed out");
  return FVS_OK;
}

int fvs_mlp_create(uint64_t seed, fvs_mlp** out) {
  if (!out) return MlpFail(FVS_ERR_INVALID, "NULL argument");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return MlpFail(FVS_ERR_NO_DEVICE, "no CUDA device available");
  }
  fvs_mlp* m = new fvs_mlp();
  const int P = fvs::mlp::kParams;
  cudaError_t e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&m->buf, sizeof(float) * P * 5);
  if (e == cudaSuccess) e = cudaMalloc(&m->wbuf, sizeof(__nv_bfloat16) * (64 * 16 + 2 * 64 * 64));
  if (e == cudaSuccess) e = cudaMalloc(&m->error, sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&m->step, 2 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&m->partial, sizeof(float) * kMaxCtas * kPartial);
  if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(float));
  if (e == cudaSuccess) e = SetSmem();
  int dev = 0, sms = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  m->ctas = std::max(1, std::min(sms, kMaxCtas));
  if (e == cudaSuccess) e = cudaMemset(m->buf, 0, sizeof(float) * P * 5);
  if (e == cudaSuccess) e = cudaMemset(m->wbuf, 0, sizeof(__nv_bfloat16) * (64 * 16 + 2 * 64 * 64));
  if (e == cudaSuccess) e = cudaMemset(m->error, 0, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(m->step, 0, 2 * sizeof(unsigned long long));
  if (e != cudaSuccess) {
    delete m;
    return MlpCuda(e, "fvs_mlp_create");
  }
  m->net.master = m->buf;
  m->net.m1 = m->buf + P;
  m->net.m2 = m->buf + 2 * P;
  m->net.grad = m->buf + 3 * P;
  m->net.blob = m->buf + 4 * P;
  m->net.W1 = m->wbuf;
  m->net.W2 = m->wbuf + 64 * 16;
  m->net.W2t = m->wbuf + 64 * 16 + 64 * 64;
  // He-style uniform initialisation on the host (deterministic from seed)
  std::vector<float> h(P, 0.0f);
  for (int k = 0; k < fvs::mlp::kIn; ++k) h[fvs::mlp::kOffInvStd + k] = 1.0f;
  uint64_t st = seed;
  auto uni = [&]() {
    st = HostMix(st);
    return float((st >> 11) * (1.0 / 9007199254740992.0)) * 2.0f - 1.0f;
  };
  const float s1 = std::sqrt(6.0f / fvs::mlp::kIn), s2 = std::sqrt(6.0f / kH);
  for (int i = 0; i < kH * fvs::mlp::kIn; ++i) h[fvs::mlp::kOffW1 + i] = s1 * uni();
  for (int i = 0; i < kH * kH; ++i) h[fvs::mlp::kOffW2 + i] = s2 * uni();
  for (int i = 0; i < kH; ++i) h[fvs::mlp::kOffW3 + i] = 0.5f * s2 * uni();
  e = cudaMemcpy(m->net.master, h.data(), sizeof(float) * P, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    delete m;
    return MlpCuda(e, "fvs_mlp_create upload");
  }
  PublishKernel<<<(P + 255) / 256, 256, 0, m->stream>>>(m->net);
  e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) {
    delete m;
    return MlpCuda(e, "fvs_mlp_create publish");
  }
  *out = m;
  return FVS_OK;
}

int fvs_mlp_destroy(fvs_mlp* m) {
  if (m) {
    cudaStreamSynchronize(m->stream);
    delete m;
  }
  return FVS_OK;
}

int fvs_riemann_features(int64_t n, double gamma, const double* rhoL_dev, const double* uL_dev,
                         const double* pL_dev, const double* rhoR_dev, const double* uR_dev,
                         const double* pR_dev, const double* pstar_dev, float* features_dev,
                         float* labels_dev, void* stream) {
  if (n < 0 || !features_dev) return MlpFail(FVS_ERR_INVALID, "bad arguments");
  if (n == 0) return FVS_OK;
  FeaturesKernel<<<unsigned((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      n, rhoL_dev, uL_dev, pL_dev, rhoR_dev, uR_dev, pR_dev, pstar_dev, gamma, features_dev,
      labels_dev);
  MLP_CUDA(cudaGetLastError());
  return FVS_OK;
}

int fvs_mlp_set_normalization(fvs_mlp* m, const float* features_dev, int64_t n) {
  if (!m || !features_dev || n < 2) return MlpFail(FVS_ERR_INVALID, "bad arguments");
  double* acc = nullptr;
  MLP_CUDA(cudaMallocAsync(&acc, sizeof(double) * 2 * fvs::mlp::kIn, m->stream));
  MLP_CUDA(cudaMemsetAsync(acc, 0, sizeof(double) * 2 * fvs::mlp::kIn, m->stream));
  MomentsKernel<<<152 * 4, 256, 0, m->stream>>>(n, features_dev, acc);
  double h[2 * fvs::mlp::kIn];
  MLP_CUDA(cudaMemcpyAsync(h, acc, sizeof h, cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(cudaFreeAsync(acc, m->stream));
  MLP_CUDA(cudaStreamSynchronize(m->stream));
  float st[2 * fvs::mlp::kIn];
  for (int k = 0; k < fvs::mlp::kIn; ++k) {
    const double mean = h[k] / double(n);
    const double var = h[fvs::mlp::kIn + k] / double(n) - mean * mean;
    st[k] = float(mean);
    st[fvs::mlp::kIn + k] = float(1.0 / std::sqrt(var > 1e-12 ? var : 1e-12));
  }
  MLP_CUDA(cudaMemcpyAsync(m->net.master + fvs::mlp::kOffMean, st, sizeof st,
                           cudaMemcpyHostToDevice, m->stream));
  PublishKernel<<<(fvs::mlp::kParams + 255) / 256, 256, 0, m->stream>>>(m->net);
  MLP_CUDA(cudaStreamSynchronize(m->stream));
  return FVS_OK;
}

int fvs_mlp_train(fvs_mlp* m, const float* features_dev, const float* labels_dev, int64_t n,
                  int steps, int batch, float lr, uint64_t seed, float* mean_loss) {
  if (!m || !features_dev || !labels_dev || n < 1 || steps < 0)
    return MlpFail(FVS_ERR_INVALID, "bad arguments");
  if (batch < 128 || batch % 256 != 0 || batch > (1 << 20))
    return MlpFail(FVS_ERR_INVALID, "batch must be a multiple of 256 in [256, 2^20]");
  FusedArgs a{};
  a.feat = features_dev;
  a.label = labels_dev;
  a.n = n;
  a.seed = seed;
  a.batch = batch;
  MLP_CUDA(cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
  for (int i = 0; i < steps; ++i) MLP_CUDA(EnqueueStep(m, a, true, lr));
  float loss = 0.f;
  int err = 0;
  MLP_CUDA(cudaMemcpyAsync(&loss, m->loss, sizeof loss, cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(cudaMemcpyAsync(&err, m->error, sizeof err, cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(cudaStreamSynchronize(m->stream));
  if (err) return MlpFail(FVS_ERR_CUDA, "tensor-core wait timed out");
  if (mean_loss) *mean_loss = steps > 0 ? loss / float(int64_t(steps) * batch) : 0.f;
  return FVS_OK;
}

int fvs_mlp_gradients(fvs_mlp* m, const float* features_dev, const float* labels_dev, int batch,
                      float* grads_host, float* loss_host) {
  if (!m || !features_dev || !labels_dev || !grads_host)
    return MlpFail(FVS_ERR_INVALID, "bad arguments");
  if (batch < 128 || batch % 256 != 0) return MlpFail(FVS_ERR_INVALID, "batch multiple of 256");
  FusedArgs a{};
  a.feat = features_dev;
  a.label = labels_dev;
  a.n = batch;
  a.batch = batch;
  a.given_rows = 1;
  MLP_CUDA(cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream));
  MLP_CUDA(EnqueueStep(m, a, false, 0.f));
  int err = 0;
  MLP_CUDA(cudaMemcpyAsync(grads_host, m->net.grad, sizeof(float) * fvs::mlp::kParams,
                           cudaMemcpyDeviceToHost, m->stream));
  float loss = 0.f;
  MLP_CUDA(cudaMemcpyAsync(&loss, m->loss, sizeof loss, cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(cudaMemcpyAsync(&err, m->error, sizeof err, cudaMemcpyDeviceToHost, m->stream));
  MLP_CUDA(cudaStreamSynchronize(m->stream));
  if (err) return MlpFail(FVS_ERR_CUDA, "tensor-core wait timed out");
  if (loss_host) *loss_host = loss / float(batch);
  return FVS_OK;
}

int fvs_mlp_predict(fvs_mlp* m, const float* features_dev, int64_t n, float* y_dev) {
  if (!m || !features_dev || !y_dev || n < 0) return MlpFail(FVS_ERR_INVALID, "bad arguments");
  if (n == 0) return FVS_OK;
  cudaStream_t s = m->stream;
  // three CTAs fit an SM's shared and tensor memory; their phases overlap
  const int64_t grid = std::min<int64_t>((n + kTile - 1) / kTile, int64_t(m->ctas) * 3);
  InferKernel<<<unsigned(grid), kFusedThreads, kForwardSmem, s>>>(
      n, features_dev, m->net.blob, m->net.W1, m->net.W2, y_dev, m->error);
  MLP_CUDA(cudaGetLastError());
  int err = 0;
  MLP_CUDA(cudaMemcpyAsync(&err, m->error, sizeof err, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(cudaStreamSynchronize(s));
  if (err) return MlpFail(FVS_ERR_CUDA, "tensor-core wait timed out");
  return FVS_OK;
}

int fvs_mlp_params(fvs_mlp* m, const float** params_dev) {
  if (!m || !params_dev) return MlpFail(FVS_ERR_INVALID, "NULL argument");
  *params_dev = m->net.blob;
  return FVS_OK;
}

int fvs_mlp_get_master(fvs_mlp* m, float* host) {
  if (!m || !host) return MlpFail(FVS_ERR_INVALID, "NULL argument");
  MLP_CUDA(cudaMemcpy(host, m->net.master, sizeof(float) * fvs::mlp::kParams,
                      cudaMemcpyDeviceToHost));
  return FVS_OK;
}

int fvs_mlp_set_master(fvs_mlp* m, const float* host) {
  if (!m || !host) return MlpFail(FVS_ERR_INVALID, "NULL argument");
  MLP_CUDA(cudaMemcpy(m->net.master, host, sizeof(float) * fvs::mlp::kParams,
                      cudaMemcpyHostToDevice));
  PublishKernel<<<(fvs::mlp::kParams + 255) / 256, 256, 0, m->stream>>>(m->net);
  MLP_CUDA(cudaStreamSynchronize(m->stream));
  return FVS_OK;
}

}  // extern "C"
