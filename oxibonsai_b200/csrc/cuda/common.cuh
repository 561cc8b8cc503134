// Shared device helpers and the packed weight layout used by every kernel in this library.
//
// Device weight layout ("planar SM"): a quantised matrix of N output rows by K inputs is stored as
//   codes  : uint32 [N][K/16]  - one word per 16 consecutive inputs k0..k0+15
//   scales : f16    [N][K/128] - one scale per 128-input group (the GGUF block scale)
// Inside a word, nibble i (bits 4i..4i+3) = { S(k0+i), S(k0+8+i), M(k0+i), M(k0+8+i) } from bit 3
// down to bit 0, where M = 1 for a non-zero weight and S = 1 for a negative one.  Two masks turn a
// word into sixteen e2m1 (fp4) values for the tensor cores:  (w & 0xAAAAAAAA) holds inputs
// k0..k0+7 and ((w & 0x55555555) << 1) holds k0+8..k0+15, each nibble being S0M0 = +-1.0 or 0.
// The same two bits, moved to bits 31 and 29 of a word, are the float +-2^-63 (or 0), which is
// how the CUDA-core kernels multiply without any integer-to-float conversion.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define BONSAI_CUDA_OK 0
#define BONSAI_CUDA_BAD_ARG (-13)
#define BONSAI_CUDA_LAUNCH_FAILED (-18)

namespace bonsai {

constexpr float kPow2_63 = 9223372036854775808.0f;  // 2^63

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the whole block (blockDim.x <= 1024, multiple of 32); every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* smem32) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) smem32[wid] = v;
  __syncthreads();
  float t = (lane < nw) ? smem32[lane] : 0.0f;
  t = warp_sum(t);
  return t;
}

// position of logical input k inside its 128-input group in the hmma-K order
__host__ __device__ inline int hmma_k_pos(int k) {
  const int r = k & 127, wq = r >> 4, e = r & 15;
  const int c = wq >> 1, j = wq & 1, plane = e >> 3, p = e & 3, h = (e >> 2) & 1;
  return (k & ~127) | ((j * 4 + p) * 16 + plane * 8 + 2 * c + h);
}

// One row: y = rmsnorm(x) * w (a plain copy when w is null) as f16 in the K order that the consumer reads.
// A thread takes eight neighbouring inputs, so that every order stores whole words: in natural and paired-K order (inputs k and k + 4
// of every eight side by side) they are one 16-byte word, in hmma-K order four pairs (k, k + 4).  The row is read once and kept in
// registers between the sum of squares and the scaling (up to 32 * blockDim.x elements; longer rows are read twice).  Needs 16-byte
// aligned rows and K % 8 == 0.
//
// The squares are added up as by 2 * blockDim.x threads with four neighbouring inputs each: a thread keeps the two sums apart, its half-warp
// is a warp of that order, and warps are added last.  The order is part of the result: f16 rounds the rows, every product carries a
// flipped bit on, and a short prompt over INT4 pages would move by 3 % with another one.  norm_threads gives the block size.
enum KOrder { K_NATURAL = 0, K_PAIRED = 1, K_HMMA = 2 };
__host__ __device__ inline int norm_threads(int K, bool wide) { return wide && K >= 4096 ? 512 : (wide && K >= 2048 ? 256 : 128); }
__device__ __forceinline__ float norm_square4(float4 v) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.x, v.x, __fmul_rn(v.y, v.y)))); }
template <int ORDER>
__device__ __forceinline__ void norm_row_to_f16(const float* __restrict__ xr, const float* __restrict__ w, float eps, int K,
                                                __half* __restrict__ orow, float* s32) {
  constexpr int kKeep = 4;
  const int nch = K >> 3;
  const float4* x4 = reinterpret_cast<const float4*>(xr);
  float4 v[kKeep][2];
  float ss[2] = {0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[i][h] = c < nch ? x4[2 * c + h] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      ss[h] = __fadd_rn(ss[h], norm_square4(v[i][h]));
    }
  }
  for (int c = threadIdx.x + kKeep * blockDim.x; c < nch; c += blockDim.x)
    for (int h = 0; h < 2; ++h) ss[h] = __fadd_rn(ss[h], norm_square4(x4[2 * c + h]));
  float inv = 1.0f;
  if (w != nullptr) {
    const int lane = threadIdx.x & 31, parts = blockDim.x >> 4;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int h = 0; h < 2; ++h) ss[h] = __fadd_rn(ss[h], __shfl_xor_sync(0xffffffffu, ss[h], o));
    if ((lane & 15) == 0) s32[threadIdx.x >> 4] = __fadd_rn(ss[0], ss[1]);
    __syncthreads();
    const float sum = warp_sum(lane < parts ? s32[lane] : 0.0f);
    inv = 1.0f / sqrtf(sum / (float)K + eps);
  }
  auto emit = [&](int c, float4 a, float4 b) {
    if (w != nullptr) {
      const float4 wa = reinterpret_cast<const float4*>(w)[2 * c], wb = reinterpret_cast<const float4*>(w)[2 * c + 1];
      a.x *= wa.x * inv; a.y *= wa.y * inv; a.z *= wa.z * inv; a.w *= wa.w * inv;
      b.x *= wb.x * inv; b.y *= wb.y * inv; b.z *= wb.z * inv; b.w *= wb.w * inv;
    }
    __align__(16) __half2 h[4];
    if (ORDER == K_NATURAL) {
      h[0] = __floats2half2_rn(a.x, a.y); h[1] = __floats2half2_rn(a.z, a.w); h[2] = __floats2half2_rn(b.x, b.y); h[3] = __floats2half2_rn(b.z, b.w);
    } else {
      h[0] = __floats2half2_rn(a.x, b.x); h[1] = __floats2half2_rn(a.y, b.y); h[2] = __floats2half2_rn(a.z, b.z); h[3] = __floats2half2_rn(a.w, b.w);
    }
    if (ORDER == K_HMMA) {
      const int pos = hmma_k_pos(8 * c);
#pragma unroll
      for (int p = 0; p < 4; ++p) *reinterpret_cast<__half2*>(orow + pos + p * 16) = h[p];
    } else {
      *reinterpret_cast<uint4*>(orow + 8 * c) = *reinterpret_cast<const uint4*>(h);
    }
  };
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < nch) emit(c, v[i][0], v[i][1]);
  }
  for (int c = threadIdx.x + kKeep * blockDim.x; c < nch; c += blockDim.x) emit(c, x4[2 * c], x4[2 * c + 1]);
}

// Dot of one packed word (16 ternary weights, scaled by 2^-63) with 16 floats.
__device__ __forceinline__ float dot_word16(uint32_t w, const float* x) {
  float acc = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float wa = __uint_as_float((w << (28 - 4 * i)) & 0xA0000000u);
    float wb = __uint_as_float((w << (29 - 4 * i)) & 0xA0000000u);
    acc = fmaf(wa, x[i], acc);
    acc = fmaf(wb, x[8 + i], acc);
  }
  return acc;
}

// Launch with programmatic dependent launch enabled: the kernel may start while its predecessor in
// the stream is still running and must execute griddepcontrol.wait before touching anything the
// predecessor writes (or writing anything it reads).
template <typename Kern, typename... Args>
static inline cudaError_t launch_pdl(Kern kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

}  // namespace bonsai
