// lp_train.cu - the proposal network layer by layer: forward, input gradient
// and weight gradient of one layer, on the tcgen05 tensor cores.
//
// Every layer is a GEMM over many rows (up to 64 per macroblock) with at most
// 128 columns on either side, so each kernel is bound by the rows it reads and
// writes, not by the tensor cores: a 1080p picture's second layer reads 33 MB of
// activations. Rows are contiguous in memory and a 16-byte unit (8 BF16) is also
// the unit of the operand layouts, so operands go from memory to shared memory
// by 16-byte asynchronous copies, a tile ahead of the MMAs, with no register
// work: K-major units for the forward and input-gradient GEMMs (K runs along a
// row), MN-major ones for the weight gradient (K runs over the rows). What
// followed a GEMM as a pass of its own is in its epilogue: bias and ReLU, the
// ReLU mask of the backward pass and its BF16 rounding; the bias gradient sums
// come from the weight gradient's staged rows. One gradient of a 1080p picture
// (8,160 macroblocks, 522,240 rows in the first layer): 66 us forward, 128 us
// backward; the general GEMM (tc_gemm.cu, element-wise staging of strided
// operands, one chunk in flight) with mask and bias passes of its own took
// 2,640 us.
#include <cuda_bf16.h>

#include <algorithm>

#include "b200enc_internal.h"
#include "proposal.cuh"
#include "umma.cuh"

namespace b200enc {

namespace {

constexpr uint64_t kWaitNs = 2000000000ull;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// Copy i of a tile of R rows of U 16-byte units: eight lanes write one unit of
// eight rows (128 consecutive bytes of shared memory, no bank conflict), and a
// warp reads four neighbouring units of each row.
template <int U, int R>
__device__ __forceinline__ int unit_row(int i) {
  return U >= 4 ? (i & 7) | ((i >> 5) % (R / 8)) << 3 : i % R;
}
template <int U, int R>
__device__ __forceinline__ int unit_col(int i) {
  return U >= 4 ? ((i >> 3) & 3) | (i / (4 * R)) << 2 : i / R;
}

enum : int { kRowRelu = 0, kRowLogits = 1, kRowGrad = 2 };

// C[m][n] = sum_k A[m][k] B(n, k) for 128-row tiles of A (row pitch lda, K
// contiguous), N columns. EPI kRowRelu: max(. + bias, 0) as BF16 (pitch ldc);
// kRowLogits: . + bias as FP32; kRowGrad: B(n, k) = W[k][n], and where
// mask[m][n] > 0 the sum, else 0, as BF16 (the gradient behind a ReLU).
template <int K, int N, int EPI>
struct RowShared {
  static constexpr int KP = K < 16 ? 16 : K;  // the MMA's K step is 16
  alignas(128) uint8_t a[2][KP / 8 * 128 * 16];
  alignas(128) uint16_t b[KP * (N < 32 ? 32 : N)];
  uint64_t bar;
  uint32_t tmem;
};

template <int K, int N, int EPI>
__global__ void __launch_bounds__(128) lp_row_gemm(int M, const __nv_bfloat16* __restrict__ A, int lda,
                                                   const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias,
                                                   const __nv_bfloat16* __restrict__ mask, int ldm,
                                                   void* __restrict__ C, int ldc, uint32_t* __restrict__ err) {
  pdl_wait();
  using S = RowShared<K, N, EPI>;
  constexpr int KP = S::KP, NB = N < 32 ? 32 : N, KU = K / 8;  // KU: 16-byte units of a row
  constexpr uint32_t kCols = NB <= 32 ? 32 : (NB <= 64 ? 64 : 128);
  extern __shared__ __align__(128) uint8_t smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = (M + 127) / 128;

  auto load = [&](int tile, int buf) {
    // unit u of row r at (u * 16 + r / 8) * 128 + (r % 8) * 16
    for (int i = tid; i < 128 * KU; i += 128) {
      const int r = unit_row<KU, 128>(i), u = unit_col<KU, 128>(i);
      const long long row = (long long)tile * 128 + r;
      const bool in = row < M;
      cp_async16(smem_u32(s.a[buf]) + (u * 128 + r) * 16, A + (in ? row : 0) * lda + u * 8, in);
    }
    cp_async_commit();
  };

  int tile = blockIdx.x;
  if (tile < tiles) load(tile, 0);
  if (warp == 0) tmem_alloc(&s.tmem, kCols);
  if (tid == 0) {
    mbar_init(&s.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < KP * NB; i += 128) {
    const int k = EPI == kRowGrad ? i / NB : i % KP, n = EPI == kRowGrad ? i % NB : i / KP;
    uint16_t v = 0;
    if (k < K && n < N) v = __bfloat16_as_ushort(EPI == kRowGrad ? W[(long long)k * ldc + n] : W[n * K + k]);
    s.b[canon_off(n, k, NB)] = v;
  }
  if (K < 16)  // the unused second half of the K step
    for (int i = tid; i < 2 * 128; i += 128) *reinterpret_cast<uint4*>(&s.a[i >> 7][(128 + (i & 127)) * 16]) = make_uint4(0u, 0u, 0u, 0u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem;
  constexpr uint32_t idesc = umma_idesc_bf16(128, NB);
  uint32_t phase = 0;
  int buf = 0;
  bool failed = false;
  for (; tile < tiles; tile += gridDim.x, buf ^= 1) {
    const int next = tile + gridDim.x;
    if (next < tiles) {
      load(next, buf ^ 1);  // the MMAs that read that buffer have been waited for
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t ab = smem_u32(s.a[buf]), bb = smem_u32(s.b);
#pragma unroll
      for (int k = 0; k < KP; k += 16) umma_bf16(tmem, canon_desc(ab, 128, k), canon_desc(bb, NB, k), idesc, k > 0);
      umma_commit(&s.bar);
    }
    const long long row = (long long)tile * 128 + warp * 32 + lane;
    const bool in = row < M;
    if (!mbar_wait(&s.bar, phase, kWaitNs)) failed = true;
    phase ^= 1;
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < N; c += 16) {
      uint4 m0 = make_uint4(0u, 0u, 0u, 0u), m1 = m0;
      if (EPI == kRowGrad && in) {
        const uint4* mp = reinterpret_cast<const uint4*>(mask + row * ldm + c);
        m0 = __ldg(mp);
        m1 = __ldg(mp + 1);
      }
      uint32_t v[16];
      tmem_row16(tmem, warp, c, v);
      if (!in) continue;
      float x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        x[j] = __uint_as_float(v[j]);
        if (EPI != kRowGrad) x[j] += __ldg(bias + c + j);
        if (EPI == kRowRelu) x[j] = x[j] < 0.f ? 0.f : x[j];
      }
      if (EPI == kRowLogits) {
        float4* dst = reinterpret_cast<float4*>(static_cast<float*>(C) + row * ldc + c);
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
      } else {
        if (EPI == kRowGrad) {
          const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float y = __uint_as_float((j & 1) ? mw[j >> 1] & 0xffff0000u : mw[j >> 1] << 16);
            x[j] = y > 0.f ? x[j] : 0.f;
          }
        }
        uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(C) + row * (EPI == kRowGrad ? N : ldc) + c);
        dst[0] = make_uint4(bf16x2(x[0], x[1]), bf16x2(x[2], x[3]), bf16x2(x[4], x[5]), bf16x2(x[6], x[7]));
        dst[1] = make_uint4(bf16x2(x[8], x[9]), bf16x2(x[10], x[11]), bf16x2(x[12], x[13]), bf16x2(x[14], x[15]));
      }
    }
    tc_fence_before();
    if (__syncthreads_or(failed)) {  // TMEM read by every warp before the next tile's MMAs
      if (tid == 0 && err) atomicExch(err, 1u);
      break;
    }
    tc_fence_after();
  }
  cp_async_wait<0>();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kCols);
}

// ---- weight gradient -------------------------------------------------------------
// dW[out][in] += sum over rows of G[row][out] A[row][in], db[out] += sum of
// G[row][out]. D (TMEM lane = input channel, column = output channel) collects
// a CTA's share of the 64-row chunks; FP32 atomics add the shares. Operands
// MN-major: 16-byte units of eight channels, the eight rows of a group 16 B
// apart (a core matrix), row groups 128 B apart (leading byte offset), channel
// units 1024 B apart (stride byte offset).
constexpr int kWgRows = 64, kWgStages = 4;

template <int IN, int OUT>
struct WgShared {
  alignas(128) uint8_t a[kWgStages][16 * kWgRows * 16];  // 128 input channels (IN of them loaded)
  alignas(128) uint8_t b[kWgStages][(OUT < 32 ? 32 : OUT) / 8 * kWgRows * 16];
  uint64_t done[kWgStages];  // the MMAs that read a stage
  float sum[OUT];
  uint32_t tmem;
};

template <int IN, int OUT>
__global__ void __launch_bounds__(128) lp_wgrad(int rows, const __nv_bfloat16* __restrict__ G,
                                                const __nv_bfloat16* __restrict__ A, int lda, float* __restrict__ gW,
                                                float* __restrict__ gb, uint32_t* __restrict__ err) {
  pdl_wait();
  using S = WgShared<IN, OUT>;
  constexpr int NB = OUT < 32 ? 32 : OUT, AU = IN / 8, BU = OUT / 8, kSumT = 128 / BU;
  constexpr uint32_t kCols = NB <= 32 ? 32 : 64;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  S& s = *reinterpret_cast<S*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks = (rows + kWgRows - 1) / kWgRows;

  // unit u of row r at u * 1024 + r * 16
  auto load = [&](int chunk, int st) {
    const long long row0 = (long long)chunk * kWgRows;
    for (int i = tid; i < kWgRows * AU; i += 128) {
      const int r = unit_row<AU, kWgRows>(i), u = unit_col<AU, kWgRows>(i);
      const bool in = row0 + r < rows;
      cp_async16(smem_u32(s.a[st]) + u * 1024 + r * 16, A + (in ? row0 + r : 0) * lda + u * 8, in);
    }
    for (int i = tid; i < kWgRows * BU; i += 128) {
      const int r = unit_row<BU, kWgRows>(i), u = unit_col<BU, kWgRows>(i);
      const bool in = row0 + r < rows;
      cp_async16(smem_u32(s.b[st]) + u * 1024 + r * 16, G + (in ? row0 + r : 0) * OUT + u * 8, in);
    }
  };

  if (warp == 0) tmem_alloc(&s.tmem, kCols);
  if (tid == 0) {
    for (int i = 0; i < kWgStages; ++i) mbar_init(&s.done[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < OUT) s.sum[tid] = 0.f;
  // channels the MMA reads and no row has: zeros
  for (int st = 0; st < kWgStages; ++st) {
    for (int i = tid; i < (16 - AU) * kWgRows; i += 128) *reinterpret_cast<uint4*>(s.a[st] + AU * 1024 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < (NB / 8 - BU) * kWgRows; i += 128) *reinterpret_cast<uint4*>(s.b[st] + BU * 1024 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  }
  for (int i = 0; i < kWgStages - 1; ++i) {
    const int c = blockIdx.x + i * gridDim.x;
    if (c < chunks) load(c, i);
    cp_async_commit();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem;
  // both operands MN-major (bits 15 and 16)
  constexpr uint32_t idesc = umma_idesc_bf16(128, NB) | (1u << 15) | (1u << 16);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // of output channels 8 (tid / kSumT) ..
  int n = 0;
  bool failed = false;
  for (int c = blockIdx.x; c < chunks; c += gridDim.x, ++n) {
    const int st = n % kWgStages;
    cp_async_wait<kWgStages - 2>();  // one group per chunk: this chunk's is complete
    fence_async_smem();
    if (__syncthreads_or(failed)) {
      failed = true;
      break;
    }
    if (tid == 0) {
      tc_fence_after();
      const uint32_t ab = smem_u32(s.a[st]), bb = smem_u32(s.b[st]);
#pragma unroll
      for (int k = 0; k < kWgRows; k += 16)  // two row groups per MMA
        umma_bf16(tmem, umma_desc(ab + (k / 8) * 128, 128, 1024), umma_desc(bb + (k / 8) * 128, 128, 1024), idesc,
                  n > 0 || k > 0);
      umma_commit(&s.done[st]);
    }
    // The stage of the chunk before this one takes the chunk three ahead: its
    // MMAs are waited for here, its bias sums ended before the barrier above.
    const long long ahead = c + (long long)(kWgStages - 1) * gridDim.x;
    const int sa = (n + kWgStages - 1) % kWgStages;
    if (n > 0 && !mbar_wait(&s.done[sa], ((n - 1) / kWgStages) & 1, kWaitNs)) failed = true;
    if (ahead < chunks) load((int)ahead, sa);
    cp_async_commit();
    // bias gradient: this thread's unit of the staged rows of G
#pragma unroll
    for (int r = tid % kSumT; r < kWgRows; r += kSumT) {
      const uint4 v = *reinterpret_cast<const uint4*>(s.b[st] + (tid / kSumT) * 1024 + r * 16);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += __uint_as_float((j & 1) ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
    }
  }
  cp_async_wait<0>();
  if (n > 0 && !failed && !mbar_wait(&s.done[(n - 1) % kWgStages], ((n - 1) / kWgStages) & 1, kWaitNs)) failed = true;
  if (__syncthreads_or(failed)) {
    if (tid == 0 && err) atomicExch(err, 1u);
  } else if (n > 0) {
    tc_fence_after();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int o = (kSumT < 32 ? kSumT : 32) / 2; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
      if (lane % kSumT == 0) atomicAdd(&s.sum[8 * (tid / kSumT) + j], acc[j]);
    }
    const int ch = warp * 32 + lane;  // input channel
#pragma unroll
    for (int c = 0; c < OUT; c += 16) {
      uint32_t v[16];
      tmem_row16(tmem, warp, c, v);
      if (ch < IN) {
#pragma unroll
        for (int j = 0; j < 16; ++j) atomicAdd(gW + (c + j) * IN + ch, __uint_as_float(v[j]));
      }
    }
    __syncthreads();
    if (tid < OUT) atomicAdd(gb + tid, s.sum[tid]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kCols);
}

int sm_count() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// As many CTAs per SM as shared memory (and TMEM: 512 columns) allows; tiles
// beyond them are walked in strides.
template <int K, int N, int EPI>
int row_gemm(long long M, const __nv_bfloat16* A, int lda, const __nv_bfloat16* W, const float* bias,
             const __nv_bfloat16* mask, int ldm, void* C, int ldc, uint32_t* err, cudaStream_t st) {
  auto k = lp_row_gemm<K, N, EPI>;
  const int smem = (int)sizeof(RowShared<K, N, EPI>) + 128;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1;
  const int per_sm = std::max(1, std::min(N > 64 ? 4 : 6, 220 * 1024 / (smem + 1024)));
  const long long tiles = (M + 127) / 128;
  launch_early(k, (unsigned)std::min<long long>(tiles, (long long)per_sm * sm_count()), 128, smem, st, (int)M, A, lda, W, bias,
               mask, ldm, C, ldc, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <int IN, int OUT>
int wgrad(long long rows, const __nv_bfloat16* G, const __nv_bfloat16* A, int lda, float* gW, float* gb, uint32_t* err,
          cudaStream_t st) {
  auto k = lp_wgrad<IN, OUT>;
  const int smem = (int)sizeof(WgShared<IN, OUT>) + 128;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1;
  const long long chunks = (rows + kWgRows - 1) / kWgRows;
  // two CTAs per SM; a CTA's share at least four chunks (its FP32 atomics cost as much as loading them)
  const long long ctas = std::max<long long>(1, std::min<long long>(2ll * sm_count(), chunks / 4));
  launch_early(k, (unsigned)ctas, 128, smem, st, (int)rows, G, A, lda, gW, gb, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

// Forward pass of B macroblocks: conv1..conv4 (2x2 stride 2, a GEMM over rows
// of the previous output), fc1, fc2.
int lp_forward_layers(const LpBuf& b, const __nv_bfloat16* wb, const float* params, long long B, uint32_t* err,
                      cudaStream_t st) {
  auto W = [&](int l) { return wb + layer_woff(l); };
  auto bias = [&](int l) { return params + layer_boff(l); };
  int rc = 0;
  rc |= row_gemm<8, 32, kRowRelu>(B * 64, b.x0, 8, W(0), bias(0), nullptr, 0, b.y1, 32, err, st);
  rc |= row_gemm<128, 32, kRowRelu>(B * 16, b.y1, 128, W(1), bias(1), nullptr, 0, b.y2, 32, err, st);
  rc |= row_gemm<128, 32, kRowRelu>(B * 4, b.y2, 128, W(2), bias(2), nullptr, 0, b.y3, 32, err, st);
  rc |= row_gemm<128, 32, kRowRelu>(B, b.y3, 128, W(3), bias(3), nullptr, 0, b.f, kFIn, err, st);
  rc |= row_gemm<kFIn, 64, kRowRelu>(B, b.f, kFIn, W(4), bias(4), nullptr, 0, b.h, 64, err, st);
  rc |= row_gemm<64, kOut, kRowLogits>(B, b.h, 64, W(5), bias(5), nullptr, 0, b.logits, kOut, err, st);
  return rc ? -1 : 0;
}

// Backward pass from the BF16 logit gradient g[5] ([B][16]): weight and bias
// gradients added into grads, each layer's masked BF16 input gradient in g[4]
// .. g[0] ([B][64], [B][32], [4B][32], [16B][32], [64B][32]).
int lp_backward_layers(const LpBuf& b, const __nv_bfloat16* wb, float* grads, __nv_bfloat16* const g[6], long long B,
                       uint32_t* err, cudaStream_t st) {
  auto W = [&](int l) { return wb + layer_woff(l); };
  auto gW = [&](int l) { return grads + layer_woff(l); };
  auto gb = [&](int l) { return grads + layer_boff(l); };
  int rc = 0;
  rc |= wgrad<64, kOut>(B, g[5], b.h, 64, gW(5), gb(5), err, st);
  rc |= row_gemm<kOut, 64, kRowGrad>(B, g[5], kOut, W(5), nullptr, b.h, 64, g[4], 64, err, st);
  rc |= wgrad<kFIn, 64>(B, g[4], b.f, kFIn, gW(4), gb(4), err, st);
  // only the conv features' 32 of fc1's 96 inputs are layers' outputs
  rc |= row_gemm<64, 32, kRowGrad>(B, g[4], 64, W(4), nullptr, b.f, kFIn, g[3], kFIn, err, st);
  rc |= wgrad<128, 32>(B, g[3], b.y3, 128, gW(3), gb(3), err, st);
  rc |= row_gemm<32, 128, kRowGrad>(B, g[3], 32, W(3), nullptr, b.y3, 128, g[2], 128, err, st);
  rc |= wgrad<128, 32>(B * 4, g[2], b.y2, 128, gW(2), gb(2), err, st);
  rc |= row_gemm<32, 128, kRowGrad>(B * 4, g[2], 32, W(2), nullptr, b.y2, 128, g[1], 128, err, st);
  rc |= wgrad<128, 32>(B * 16, g[1], b.y1, 128, gW(1), gb(1), err, st);
  rc |= row_gemm<32, 128, kRowGrad>(B * 16, g[1], 32, W(1), nullptr, b.y1, 128, g[0], 128, err, st);
  rc |= wgrad<8, 32>(B * 64, g[0], b.x0, 8, gW(0), gb(0), err, st);
  return rc ? -1 : 0;
}

}  // namespace b200enc
