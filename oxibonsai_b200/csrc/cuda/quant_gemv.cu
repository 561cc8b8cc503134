// Decode GEMV straight from GGUF blocks for the formats that have no planar repack: Q4_0, Q8_0,
// FP8 E4M3 / E5M2 blocks, the K-quants Q2_K .. Q8_K, the 256-wide TQ2_0, F16, BF16 and F32 rows.
//
// Replaces the reference's per-format single-GEMV wrappers cuda_gemv_q4_0 / q8_0, cuda_gemv_q{2..8}k
// and cuda_gemv_fp8_* (crates/oxibonsai-kernels/src/gpu_backend/cuda_q_std_kernels.rs:200-,
// cuda_k_quant_kernels.rs:640-, cuda_fp8_kernels.rs:300-) with kernels templated on the block decoder.
// Products and sums are f32 (exact integers inside a block in one kernel), with optional fused RMSNorm of the input and residual add.
// quant_stream_imma_kernel serves Q4_0, Q8_0 and Q4_K of whole 256-input units, its sums of 32 products exact integers; quant_stream_kernel the other
// matrices whose rows can be copied in 16-byte units; quant_gemv_kernel and its
// batched form take the rest: one warp owns a row, for 32-element blocks every lane decodes a whole block per step
// (32 blocks = 1024 inputs per warp step), for 256-element super-blocks the 32 lanes share a block, eight elements each.
// Block layouts are the ones documented in csrc/core/blocks.hpp and csrc/core/kquants.hpp.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace bonsai {

__device__ __forceinline__ float ld_f16(const uint8_t* p) { return __half2float(__ushort_as_half((unsigned short)(p[0] | (p[1] << 8)))); }
__device__ __forceinline__ float fp8_to_f32(uint8_t q, bool e5m2) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)q, e5m2 ? __NV_E5M2 : __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

// Decoders: value of element i (0 <= i < kElems) of the block at p.
struct DecQ4_0 { static constexpr int kElems = 32, kBytes = 18;
  static __device__ float at(const uint8_t* p, int i) { const int q = (p[2 + (i >> 1)] >> ((i & 1) * 4)) & 15; return ld_f16(p) * (float)(q - 8); } };
struct DecQ8_0 { static constexpr int kElems = 32, kBytes = 34;
  static __device__ float at(const uint8_t* p, int i) { return ld_f16(p) * (float)(int8_t)p[2 + i]; } };
template <bool E5M2> struct DecFp8 { static constexpr int kElems = 32, kBytes = 34;
  static __device__ float at(const uint8_t* p, int i) { return ld_f16(p + 32) * fp8_to_f32(p[i], E5M2); } };
struct DecTq2_256 { static constexpr int kElems = 256, kBytes = 66;
  static __device__ float at(const uint8_t* p, int i) { const int c = (p[i >> 2] >> (2 * (i & 3))) & 3; return ld_f16(p + 64) * (c == 0 ? -1.0f : (c == 2 ? 1.0f : 0.0f)); } };
struct DecQ2K { static constexpr int kElems = 256, kBytes = 84;
  static __device__ float at(const uint8_t* p, int i) {
    const int q = (p[16 + (i >> 2)] >> ((i & 3) * 2)) & 3;
    return ld_f16(p + 80) * (float)(p[i >> 4] & 15) * (float)q - ld_f16(p + 82) * (float)(p[i >> 4] >> 4); } };
struct DecQ3K { static constexpr int kElems = 256, kBytes = 110;
  static __device__ float at(const uint8_t* p, int i) {
    const int q = ((p[32 + (i >> 2)] >> ((i & 3) * 2)) & 3) | (((p[i >> 3] >> (i & 7)) & 1) << 2);
    const int sub = i >> 4, sc = ((p[96 + (sub >> 1)] >> (4 * (sub & 1))) & 15) - 8;
    return ld_f16(p + 108) * (float)sc * (float)(q - 4); } };
__device__ __forceinline__ void k6_at(const uint8_t* s, int j, int& sc, int& mn) {
  sc = ((s[j >> 1] >> (4 * (j & 1))) & 15) | (((s[8 + (j >> 2)] >> (2 * (j & 3))) & 3) << 4);
  mn = ((s[4 + (j >> 1)] >> (4 * (j & 1))) & 15) | (((s[10 + (j >> 2)] >> (2 * (j & 3))) & 3) << 4);
}
struct DecQ4K { static constexpr int kElems = 256, kBytes = 144;
  static __device__ float at(const uint8_t* p, int i) {
    int sc, mn; k6_at(p + 4, i >> 5, sc, mn);
    const int q = (p[16 + (i >> 1)] >> ((i & 1) * 4)) & 15;
    return ld_f16(p) * (float)sc * (float)q - ld_f16(p + 2) * (float)mn; } };
struct DecQ5K { static constexpr int kElems = 256, kBytes = 176;
  static __device__ float at(const uint8_t* p, int i) {
    int sc, mn; k6_at(p + 4, i >> 5, sc, mn);
    const int q = ((p[48 + (i >> 1)] >> ((i & 1) * 4)) & 15) | (((p[16 + (i >> 3)] >> (i & 7)) & 1) << 4);
    return ld_f16(p) * (float)sc * (float)q - ld_f16(p + 2) * (float)mn; } };
struct DecQ6K { static constexpr int kElems = 256, kBytes = 210;
  static __device__ float at(const uint8_t* p, int i) {
    const int q = ((p[i >> 1] >> ((i & 1) * 4)) & 15) | (((p[128 + (i >> 2)] >> (2 * (i & 3))) & 3) << 4);
    return ld_f16(p + 208) * (float)(int8_t)p[192 + (i >> 4)] * (float)(q - 32); } };
struct DecQ8K { static constexpr int kElems = 256, kBytes = 292;
  static __device__ float at(const uint8_t* p, int i) { float d; memcpy(&d, p, 4); return d * (float)(int8_t)p[4 + i]; } };
struct DecF16 { static constexpr int kElems = 32, kBytes = 64;
  static __device__ float at(const uint8_t* p, int i) { return ld_f16(p + 2 * i); } };
struct DecBF16 { static constexpr int kElems = 32, kBytes = 64;
  static __device__ float at(const uint8_t* p, int i) { return __uint_as_float((uint32_t)(p[2 * i] | (p[2 * i + 1] << 8)) << 16); } };
struct DecF32 { static constexpr int kElems = 32, kBytes = 128;
  static __device__ float at(const uint8_t* p, int i) { float v; memcpy(&v, p + 4 * i, 4); return v; } };

// ---- streamed rows ------------------------------------------------------------------------------------------------------
// One or two tokens over a matrix of blocks.  The rows of a matrix are one contiguous byte string, so a CTA owns a range of
// rows and a producer lane streams it through a shared-memory ring with bulk copies (the first stages before it waits for the
// kernel ahead: weights depend on nothing).  Blocks of 18, 34, 110 or 210 bytes are no friends of wide global loads; out of
// shared memory the aligned words around a block cost at most two wavefronts each.
// A lane decodes 32 consecutive weights of a row per step, a warp 1024: it keeps its 32 inputs (times the norm weights) of
// every token in registers for the whole range of rows, so an input is loaded once per CTA.  A group's codes are multiplied as
// exact integers and the scale is applied once per group; a minimum is multiplied into the group's sum of inputs, made once.
// K is spread over KW warps; their partial sums stay in shared memory until the end, where they are added in K order.
// What bounds it: instructions.  24576 x 4096 in Q4_0 takes 19.6 M warp instructions (some six per weight with addresses, shuffles and
// the hand-over of stages), half of the issue slots; more rows side by side do not help.  24576 x 4096, one token: Q4_0 27.8 us, Q8_0
// 25.9 (4.1 TB/s), Q4_K 27.9, Q6_K 40.8, F16 40.7 (4.9 TB/s).  Before (a warp per row, one byte load per weight) the matrices of a
// quarter-depth 8B model in Q4_K took 113 us on average, 20 here; a token of it 4370 us, 815 here (555 with the integer form further down, which
// takes Q4_0, Q8_0 and Q4_K of whole 256-input units).
constexpr int kQsMaxWarps = 16;
constexpr int kQsMaxStages = 8;
constexpr int kQsRing = 112 * 1024;
constexpr int kQsRows = 256;        // rows of a CTA whose partial sums are kept

__device__ __forceinline__ uint64_t qs_pack(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t qs_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t qs_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float qs_sum2(uint64_t a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}

// Integers become floats without a conversion: a field of a word that lies at bit `at` of a float with exponent 2^(23 - at) counts in
// ones above the base 2^(23 - at), which is then taken off exactly, two values at a time.
__device__ __forceinline__ float qs_int(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.0f; }   // v < 2^23
template <int AT>
__device__ __forceinline__ float qs_raw(uint32_t w, uint32_t mask) { return __uint_as_float((w & (mask << AT)) | ((150u - AT) << 23)); }
template <int A0, int A1>
__device__ __forceinline__ uint64_t qs_take(float a, float b, float less) {
  return qs_add2(qs_pack(a, b), qs_pack(-(float)(1 << (23 - A0)) - less, -(float)(1 << (23 - A1)) - less));
}
// nibbles n, n + 1 (n even) of w, minus `less`: five nibbles of a word lie inside a mantissa, the other three after one shift
__device__ __forceinline__ uint64_t qs_nibbles(uint32_t w, int n, float less) {
  const uint32_t u = w >> 20;
  if (n == 0) return qs_take<0, 4>(qs_raw<0>(w, 15u), qs_raw<4>(w, 15u), less);
  if (n == 2) return qs_take<8, 12>(qs_raw<8>(w, 15u), qs_raw<12>(w, 15u), less);
  if (n == 4) return qs_take<16, 0>(qs_raw<16>(w, 15u), qs_raw<0>(u, 15u), less);
  return qs_take<4, 8>(qs_raw<4>(u, 15u), qs_raw<8>(u, 15u), less);
}
// signed bytes b, b + 1 of w, w with its sign bits flipped
__device__ __forceinline__ uint64_t qs_bytes(uint32_t w, int b) {
  const float x = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u + (uint32_t)b)), y = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7651u + (uint32_t)b));
  return qs_add2(qs_pack(x, y), qs_pack(-8388736.0f, -8388736.0f));
}
// two integers below 2^23, minus `less`
__device__ __forceinline__ uint64_t qs_ints(uint32_t a, uint32_t b, float less) {
  return qs_take<0, 0>(__uint_as_float(0x4B000000u | a), __uint_as_float(0x4B000000u | b), less);
}

// NW words at p: aligned to A bytes (2, 4 or 16)
template <int NW, int A>
__device__ __forceinline__ void qs_words(const uint8_t* p, uint32_t* out) {
  if (A == 16 && NW % 4 == 0) {
#pragma unroll
    for (int i = 0; i < NW / 4; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(p)[i];
      out[4 * i] = v.x; out[4 * i + 1] = v.y; out[4 * i + 2] = v.z; out[4 * i + 3] = v.w;
    }
  } else if (A >= 4) {
#pragma unroll
    for (int i = 0; i < NW; ++i) out[i] = reinterpret_cast<const uint32_t*>(p)[i];
  } else {
    const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 2u);
    const uint32_t* a = reinterpret_cast<const uint32_t*>(p - odd);
    uint32_t w[NW + 1];
#pragma unroll
    for (int i = 0; i <= NW; ++i) w[i] = a[i];       // the word behind the last block lies in the ring's slack
#pragma unroll
    for (int i = 0; i < NW; ++i) out[i] = __funnelshift_r(w[i], w[i + 1], odd * 8);
  }
}
__device__ __forceinline__ uint32_t qs_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }
__device__ __forceinline__ float qs_f16(const uint8_t* p) { return __half2float(__ushort_as_half((unsigned short)qs_u16(p))); }

// 32 weights: block number b (of 32) of the row at `row`.  Weights j, j + 1 (j even) are s[j / (32 / kScales)] * q2(j) - m[...].
#define QS_HEAD(scales, mins) static constexpr int kScales = scales; static constexpr bool kMin = mins; float s[scales], m[mins ? scales : 1];
struct QsQ4_0 { QS_HEAD(1, false) uint32_t w[4];
  __device__ void load(const uint8_t* row, int b) { const uint8_t* p = row + b * 18; s[0] = qs_f16(p); qs_words<4, 2>(p + 2, w); }
  __device__ uint64_t q2(int j) const { return qs_nibbles(w[j >> 3], j & 7, 8.0f); } };
struct QsQ8_0 { QS_HEAD(1, false) uint32_t w[8];
  __device__ void load(const uint8_t* row, int b) { const uint8_t* p = row + b * 34; s[0] = qs_f16(p); qs_words<8, 2>(p + 2, w);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] ^= 0x80808080u; }
  __device__ uint64_t q2(int j) const { return qs_bytes(w[j >> 2], j & 3); } };
template <bool E5M2> struct QsFp8 { QS_HEAD(1, false) uint32_t w[8];
  __device__ void load(const uint8_t* row, int b) { const uint8_t* p = row + b * 34; s[0] = qs_f16(p + 32); qs_words<8, 2>(p, w); }
  __device__ uint64_t q2(int j) const {
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w[j >> 2] >> (8 * (j & 3))), E5M2 ? __NV_E5M2 : __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return qs_pack(f.x, f.y); } };
struct QsTq2_256 { QS_HEAD(1, false) uint32_t w[2];
  __device__ void load(const uint8_t* row, int b) { const uint8_t* p = row + (b >> 3) * 66; s[0] = qs_f16(p + 64); qs_words<2, 2>(p + 8 * (b & 7), w); }
  __device__ float q(int j) const { const uint32_t c = (w[j >> 4] >> (2 * (j & 15))) & 3u; return c == 0 ? -1.0f : (c == 2 ? 1.0f : 0.0f); }
  __device__ uint64_t q2(int j) const { return qs_pack(q(j), q(j + 1)); } };
struct QsQ2K { QS_HEAD(2, true) uint32_t w[2];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 84;
    const int j = b & 7;
    const float d = qs_f16(p + 80), dm = qs_f16(p + 82);
    const uint32_t sc = qs_u16(p + 2 * j);
    s[0] = d * qs_int(sc & 15u); m[0] = dm * qs_int((sc >> 4) & 15u); s[1] = d * qs_int((sc >> 8) & 15u); m[1] = dm * qs_int(sc >> 12);
    qs_words<2, 4>(p + 16 + 8 * j, w); }
  __device__ uint64_t q2(int j) const { const uint32_t v = w[j >> 4] >> (2 * (j & 15)); return qs_take<0, 2>(qs_raw<0>(v, 3u), qs_raw<2>(v, 3u), 0.0f); } };
struct QsQ3K { QS_HEAD(2, false) uint32_t w[2], h[1];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 110;
    const int j = b & 7;
    const float d = qs_f16(p + 108);
    const uint32_t sc = p[96 + j];
    s[0] = d * (qs_int(sc & 15u) - 8.0f); s[1] = d * (qs_int(sc >> 4) - 8.0f);
    qs_words<2, 2>(p + 32 + 8 * j, w); qs_words<1, 2>(p + 4 * j, h); }
  __device__ uint32_t q(int j) const { return ((w[j >> 4] >> (2 * (j & 15))) & 3u) | (((h[0] >> j) & 1u) << 2); }
  __device__ uint64_t q2(int j) const { return qs_ints(q(j), q(j + 1), 4.0f); } };
__device__ __forceinline__ void qs_k6(const uint32_t* t, int j, float d, float dm, float& s, float& m) {   // t: the 12 scale bytes
  s = d * qs_int(((t[0] >> (4 * j)) & 15u) | (((t[2] >> (2 * j)) & 3u) << 4));
  m = dm * qs_int(((t[1] >> (4 * j)) & 15u) | (((t[2] >> (16 + 2 * j)) & 3u) << 4));
}
struct QsQ4K { QS_HEAD(1, true) uint32_t w[4];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 144;
    uint32_t t[4];
    qs_words<4, 16>(p, t);
    const __half2 dd = *reinterpret_cast<const __half2*>(t);
    qs_k6(t + 1, b & 7, __low2float(dd), __high2float(dd), s[0], m[0]);
    qs_words<4, 16>(p + 16 + 16 * (b & 7), w); }
  __device__ uint64_t q2(int j) const { return qs_nibbles(w[j >> 3], j & 7, 0.0f); } };
struct QsQ5K { QS_HEAD(1, true) uint32_t w[4], h[1];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 176;
    uint32_t t[4];
    qs_words<4, 16>(p, t);
    const __half2 dd = *reinterpret_cast<const __half2*>(t);
    qs_k6(t + 1, b & 7, __low2float(dd), __high2float(dd), s[0], m[0]);
    qs_words<4, 16>(p + 48 + 16 * (b & 7), w); qs_words<1, 4>(p + 16 + 4 * (b & 7), h); }
  __device__ uint32_t q(int j) const { return ((w[j >> 3] >> (4 * (j & 7))) & 15u) | (((h[0] >> j) & 1u) << 4); }
  __device__ uint64_t q2(int j) const { return qs_ints(q(j), q(j + 1), 0.0f); } };
struct QsQ6K { QS_HEAD(2, false) uint32_t w[4], h[2];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 210;
    const int j = b & 7;
    const float d = qs_f16(p + 208);
    const uint32_t sc = qs_u16(p + 192 + 2 * j);
    s[0] = d * (float)(int8_t)(sc & 255u); s[1] = d * (float)(int8_t)(sc >> 8);
    qs_words<4, 2>(p + 16 * j, w); qs_words<2, 2>(p + 128 + 8 * j, h); }
  __device__ uint32_t q(int j) const { return ((w[j >> 3] >> (4 * (j & 7))) & 15u) | (((h[j >> 4] >> (2 * (j & 15))) & 3u) << 4); }
  __device__ uint64_t q2(int j) const { return qs_ints(q(j), q(j + 1), 32.0f); } };
struct QsQ8K { QS_HEAD(1, false) uint32_t w[8];
  __device__ void load(const uint8_t* row, int b) {
    const uint8_t* p = row + (b >> 3) * 292;
    s[0] = *reinterpret_cast<const float*>(p);
    qs_words<8, 4>(p + 4 + 32 * (b & 7), w);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] ^= 0x80808080u; }
  __device__ uint64_t q2(int j) const { return qs_bytes(w[j >> 2], j & 3); } };
struct QsF16 { QS_HEAD(1, false) uint32_t w[16];
  __device__ void load(const uint8_t* row, int b) { s[0] = 1.0f; qs_words<16, 16>(row + b * 64, w); }
  __device__ uint64_t q2(int j) const { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j >> 1])); return qs_pack(f.x, f.y); } };
struct QsBF16 { QS_HEAD(1, false) uint32_t w[16];
  __device__ void load(const uint8_t* row, int b) { s[0] = 1.0f; qs_words<16, 16>(row + b * 64, w); }
  __device__ uint64_t q2(int j) const { return qs_pack(__uint_as_float(w[j >> 1] << 16), __uint_as_float(w[j >> 1] & 0xFFFF0000u)); } };
struct QsF32 { QS_HEAD(1, false) uint32_t w[32];
  __device__ void load(const uint8_t* row, int b) { s[0] = 1.0f; qs_words<32, 16>(row + b * 128, w); }
  __device__ uint64_t q2(int j) const { return qs_pack(__uint_as_float(w[j]), __uint_as_float(w[j + 1])); } };
#undef QS_HEAD

struct QsParams {
  const uint8_t* w;
  const float* x;          // [NB][x_ld]
  const float* norm_w;
  float* out;              // [NB][out_ld]
  const float* residual;   // [NB][out_ld]
  int* status;             // may be null; 5 after a copy that never arrived
  float eps;
  int x_ld, out_ld, N, K, R, KW, RW, stages;
  long long row_bytes;
};

template <typename D, int NB>
__global__ void __launch_bounds__(kQsMaxWarps * 32 + 32, 1) quant_stream_kernel(QsParams p) {
  constexpr int U = NB == 1 && sizeof(D) < 64 ? 2 : 1;      // where the registers hold two rows; F16 gains nothing (40.6 us with one and with two)
  extern __shared__ __align__(128) uint8_t qs_smem[];     // ring, 16 bytes of slack, one token's inputs, partial sums [rows][NB][KW]
  __shared__ uint64_t full[kQsMaxStages], empty[kQsMaxStages];
  __shared__ float s_sq[NB][kQsMaxWarps];
  __shared__ int s_failed;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = p.KW * p.RW;
  const int nchunks = (p.N + p.R - 1) / p.R;
  const int c0 = (int)(((long long)blockIdx.x * nchunks) / gridDim.x), c1 = (int)(((long long)(blockIdx.x + 1) * nchunks) / gridDim.x);
  const int stage_bytes = (int)(p.R * p.row_bytes);
  float* xbuf = reinterpret_cast<float*>(qs_smem + (((size_t)p.stages * stage_bytes + 16 + 127) & ~(size_t)127));   // [K / 32][36]
  float* part = xbuf + (p.K >> 5) * 36;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (t == 0) {
    for (int i = 0; i < p.stages; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], nwarps);
    }
    tc::mbar_fence_init();
    s_failed = 0;
  }
  __syncthreads();
  bool failed = false;
  if (warp == nwarps) {
    if (lane == 0) {
      int issued = 0;
      for (int c = c0; c < c1 && !failed; ++c, ++issued) {
        const int i = c - c0, st = i % p.stages;
        if (!tc::mbar_wait_sleep<40>(&empty[st], ((i / p.stages) & 1) ^ 1)) { failed = true; break; }
        const uint32_t bytes = (uint32_t)(min(p.R, p.N - c * p.R) * p.row_bytes);      // a multiple of 16: the caller checked
        tc::mbar_arrive_expect_tx(&full[st], bytes);
        tc::bulk_g2s(qs_smem + (size_t)st * stage_bytes, p.w + (size_t)c * p.R * p.row_bytes, bytes, &full[st]);
      }
      tc::mbar_drain(full, issued, p.stages);
    }
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int kw = warp % p.KW, rw = warp / p.KW;
    const int b = kw * 32 + lane;                 // this lane's block of 32 inputs
    const bool live = b * 32 < p.K;
    uint64_t x2[NB][16];
    float xs[NB][D::kScales];
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      // coalesced loads into padded shared memory, from there 32 neighbours per lane (strided global loads took 4 us)
      const float4* xp = reinterpret_cast<const float4*>(p.x + (size_t)n * p.x_ld);
      const float4* np = reinterpret_cast<const float4*>(p.norm_w);
      float sq = 0.0f;
      for (int i = t; i < (p.K >> 2); i += nwarps * 32) {
        float4 v = xp[i];
        if (p.norm_w != nullptr) {
          const float4 g = __ldg(np + i);
          sq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
          v.x *= g.x; v.y *= g.y; v.z *= g.z; v.w *= g.w;
        }
        *reinterpret_cast<float4*>(xbuf + (i >> 3) * 36 + (i & 7) * 4) = v;
      }
      sq = warp_sum(sq);
      if (lane == 0) s_sq[n][warp] = sq;
      asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32) : "memory");
      float xv[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 v = live ? *reinterpret_cast<const float4*>(xbuf + b * 36 + i * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        xv[4 * i] = v.x; xv[4 * i + 1] = v.y; xv[4 * i + 2] = v.z; xv[4 * i + 3] = v.w;
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) x2[n][i] = qs_pack(xv[2 * i], xv[2 * i + 1]);
      constexpr int G = 32 / D::kScales;
#pragma unroll
      for (int g = 0; g < D::kScales; ++g) {
        xs[n][g] = 0.0f;
#pragma unroll
        for (int i = 0; i < G; ++i) xs[n][g] += xv[g * G + i];
      }
      if (n + 1 < NB) asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32) : "memory");
    }
    for (int c = c0; c < c1 && !failed; ++c) {
      const int i = c - c0, st = i % p.stages, rows = min(p.R, p.N - c * p.R);
      if (!tc::mbar_wait(&full[st], (i / p.stages) & 1)) { failed = true; break; }
      const uint8_t* chunk = qs_smem + (size_t)st * stage_bytes;
      // U rows side by side: their loads, sums and shuffles overlap
      for (int r = rw; r < rows; r += U * p.RW) {
        float acc[U][NB];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int n = 0; n < NB; ++n) acc[u][n] = 0.0f;
        if (live) {
          D d[U];
#pragma unroll
          for (int u = 0; u < U; ++u) d[u].load(chunk + (size_t)min(r + u * p.RW, rows - 1) * p.row_bytes, b);
          constexpr int G2 = 16 / D::kScales;
#pragma unroll
          for (int g = 0; g < D::kScales; ++g) {
            uint64_t a[U][NB];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int n = 0; n < NB; ++n) a[u][n] = 0ull;
#pragma unroll
            for (int k = 0; k < G2; ++k)
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const uint64_t q = d[u].q2((g * G2 + k) * 2);
#pragma unroll
                for (int n = 0; n < NB; ++n) a[u][n] = qs_fma2(q, x2[n][g * G2 + k], a[u][n]);
              }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
              for (int n = 0; n < NB; ++n) {
                acc[u][n] = fmaf(d[u].s[g], qs_sum2(a[u][n]), acc[u][n]);
                if (D::kMin) acc[u][n] = fmaf(-d[u].m[g], xs[n][g], acc[u][n]);
              }
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int n = 0; n < NB; ++n) acc[u][n] += __shfl_xor_sync(0xffffffffu, acc[u][n], o);
        if (lane == 0) {
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int n = 0; n < NB; ++n)
              if (r + u * p.RW < rows) part[((size_t)(i * p.R + r + u * p.RW) * NB + n) * p.KW + kw] = acc[u][n];
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[st]);
    }
  }
  if (failed) {                  // a copy that never arrived: its rows come out as NaN instead of numbers made of old data
    s_failed = 1;
    if (lane == 0 && p.status != nullptr) atomicExch(p.status, 5);
  }
  __syncthreads();
  if (warp >= nwarps) return;
  float inv[NB];
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    float ss = 0.0f;
    for (int k = 0; k < nwarps; ++k) ss += s_sq[n][k];
    inv[n] = p.norm_w != nullptr ? 1.0f / sqrtf(ss / (float)p.K + p.eps) : 1.0f;
  }
  const int row0 = c0 * p.R, rows = min(c1 * p.R, p.N) - row0;
  for (int i = t; i < rows; i += nwarps * 32) {
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      float v = 0.0f;
      for (int k = 0; k < p.KW; ++k) v += part[((size_t)i * NB + n) * p.KW + k];
      const size_t o = (size_t)n * p.out_ld + row0 + i;
      p.out[o] = s_failed ? __int_as_float(0x7FFFFFFF) : (p.residual ? p.residual[o] : 0.0f) + v * inv[n];
    }
  }
}

// Whether a matrix can be streamed, and how: chunks of R rows that start and end on 16-byte boundaries (a last chunk of fewer rows
// must end on one too), two stages at least, inputs in 16-byte loads, at most sixteen warps over K.
template <typename D>
static bool qs_plan(QsParams& p, int& grid, size_t& smem, int nb) {
  constexpr int unroll = sizeof(D) < 64 ? 2 : 1;
  if (p.K % 32 != 0 || p.K > kQsMaxWarps * 1024 || p.x_ld % 4 != 0) return false;
  if (((reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.norm_w)) & 15) != 0) return false;
  if (((long long)p.N * p.row_bytes) % 16 != 0) return false;
  int R = 1;
  while ((R * p.row_bytes) % 16 != 0) R *= 2;                    // 1 to 8: a row has an even number of bytes
  p.KW = (p.K + 1023) / 1024;
  p.RW = 1;
  while (p.RW * 2 * p.KW <= kQsMaxWarps && p.RW < 8) p.RW *= 2;
  while (R < p.RW) R *= 2;
  if (unroll == 2 && R == p.RW && 2 * R * p.row_bytes <= kQsRing / 3) R *= 2;      // two rows for every warp over rows, three copies ahead
  if (R * p.row_bytes > kQsRing / 2) return false;
  p.R = R;
  const long long stage = R * p.row_bytes;
  p.stages = (int)(kQsRing / stage < kQsMaxStages ? kQsRing / stage : kQsMaxStages);
  if (p.stages < 2) return false;
  const int nchunks = (p.N + R - 1) / R;
  grid = nchunks < 148 ? nchunks : 148;
  const int most = kQsRows / R;                                   // chunks of a CTA
  if ((nchunks + grid - 1) / grid > most) grid = (nchunks + most - 1) / most;
  const int per = (nchunks + grid - 1) / grid;
  if (p.stages > per) p.stages = per < 2 ? 2 : per;
  smem = (((size_t)p.stages * stage + 16 + 127) & ~(size_t)127) + (size_t)(p.K / 32) * 36 * sizeof(float) + (size_t)per * R * nb * p.KW * sizeof(float);
  return smem <= 220 * 1024;
}

template <typename D>
static QsParams qs_params(const void* w, const float* x, int x_ld, const float* norm_w, float eps, float* out, const float* residual, int out_ld,
                          int N, int K, int* status) {
  QsParams p{};
  p.status = status;
  p.w = (const uint8_t*)w; p.x = x; p.norm_w = norm_w; p.out = out; p.residual = residual; p.eps = eps;
  p.x_ld = x_ld; p.out_ld = out_ld; p.N = N; p.K = K;
  p.row_bytes = (long long)(K / D::kElems) * D::kBytes;
  return p;
}

// Rows of x that one launch takes: two where the matrix is streamed, else up to eight.
template <typename D, typename Q>
static int qs_rows(const void* w, int N, int K) {
  QsParams p = qs_params<D>(w, nullptr, K, nullptr, 0.0f, nullptr, nullptr, N, N, K, nullptr);
  int grid;
  size_t smem;
  return qs_plan<Q>(p, grid, smem, 2) ? 2 : 8;
}

template <typename D, int NB>
static int qs_launch(const QsParams& p, int grid, size_t smem, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BONSAI_CUDA_LAUNCH_FAILED;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(quant_stream_kernel<D, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) != cudaSuccess) return BONSAI_CUDA_LAUNCH_FAILED;
    configured[dev] = true;
  }
  const cudaError_t e = launch_pdl(quant_stream_kernel<D, NB>, dim3(grid), dim3((p.KW * p.RW + 1) * 32), smem, st, p);
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

// ---- one or two tokens on the integer tensor cores ----------------------------------------------------------------------------------
// Q4_0, Q8_0 and Q4_K rows: a block of 32 codes times 32 inputs is one K extent of mma.sync.m16n8k32, for sixteen rows at once.  The inputs of a
// block are eight int8 terms of seven bits, x = s (q1 + q2 / 2^7 + ... + q8 / 2^49) with s a power of two that brings the block's largest input to
// [2^5, 2^6), every step of the split exact: an input of at least 2^-31 of the largest is held to its last bit (four terms, 28 bits of the largest,
// lost what stood beside an outlier whose code is zero: 3e-5 of the result for outliers of 10^4).  A block with a smaller one, an infinity or a NaN
// is multiplied in f32 instead.  The terms are the eight columns, so that a token has an accumulator per block.  Products and their sums are exact
// integers; scales, minima (times the sum of the block's inputs) and the sums over blocks are f32.
// A CTA owns tiles of sixteen rows and goes through them a segment of K at a time.  A producer warp copies a tile's piece row by row into a ring whose
// pitch keeps the rows' words apart; a consumer warp has 256 inputs of the segment, which it alone splits, and adds to its sums of the tile; the warps'
// sums meet in warp order at the end.  The warps and the order of additions follow from the matrix alone, whatever tokens there are.
// Bound by the codes' way from shared memory to operands and the blocks' scales, some two instructions per weight where the kernel above takes six.
// One token, us above -> here: Q4_K 6144 x 4096 10.9 -> 7.5, 24576 x 4096 30.6 -> 18.8 (8.8 at the copy rate; 17.1 with four terms), 4096 x 12288 20.0 -> 14.3;
// Q4_0 24576 x 4096 30.7 -> 17.4; Q8_0 24576 x 4096 30.5 -> 23.4 (16.6).  Two tokens: Q4_K 24576 x 4096 37.4 -> 27.1, Q8_0 38.7 -> 29.1.  Relative error
// against 64 bits, with an input of twenty times the others in every third block: Q4_K 2.0e-7 -> 1.4e-7, Q4_0 1.1e-7 -> 8.0e-8, Q8_0 1.1e-7 -> 8.0e-8; with
// inputs of 30 to 10^14 under zero codes in every block 0.4 to 4.1e-7 -> 0.3 to 2.3e-7.
struct QiParams {
  const uint8_t* w;
  const float *x, *norm_w, *residual;
  float* out;
  int* status;
  float eps;
  int N, K, nseg, warps, stages, pitch;      // segments of K; consumer warps = 256-input units of a segment
  int x_ld, out_ld;
};
constexpr int kQiMaxWarps = 20, kQiMaxTiles = 12, kQiMaxStages = 4, kQiTerms = 8;
constexpr int kQiSmem = 226 * 1024;
constexpr int kQiUnitBytes = kQiTerms * 256 + 8 * 8;      // of shared memory for a token's unit of inputs: terms and {scale, sum} of its blocks

// d = kQiZero + a b as floats: the sums start at the bits of 1.5 * 2^23, so that an integer below 2^22 comes out in that float's last places
constexpr float kQiZero = 12582912.0f;
template <bool SIGNED>
__device__ __forceinline__ void qi_mma(float* d, const uint32_t* a, uint2 b) {
  int r[4];
  const int z = __float_as_int(kQiZero);
  if (SIGNED)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "r"(z));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "r"(z));
#pragma unroll
  for (int i = 0; i < 4; ++i) d[i] = __int_as_float(r[i]);
}
__device__ __forceinline__ uint32_t qi_word(const uint8_t* p) { return *reinterpret_cast<const uint32_t*>(p); }      // 4-byte aligned
// word number i of bytes that lie two behind a 4-byte boundary
__device__ __forceinline__ uint32_t qi_word2(const uint8_t* p, int i) {
  const uint32_t* a = reinterpret_cast<const uint32_t*>(p - 2) + i;
  return __funnelshift_r(a[0], a[1], 16);
}

// A unit of a row: 256 weights, kUnit bytes at `p` (16-byte aligned).  codes: the lane's share (t of four) of block j as the first operand's two words.
// A Head has what the scales of a row's unit are made of; scale and (kSums) minimum of block j, the latter for the sum of its inputs.
struct QiQ4_0 { static constexpr int kUnit = 144; static constexpr bool kSigned = true, kNibbles = true, kSums = false;
  struct Head { const uint8_t* p; };
  static __device__ Head head(const uint8_t* p) { return Head{p}; }
  static __device__ void codes(const uint8_t* p, int j, int t, uint32_t& lo, uint32_t& hi) {
    const uint8_t* b = p + 18 * j + 2;                        // two bytes off a boundary for even j
    const uint32_t w = (j & 1) ? qi_word(b + 4 * t) : qi_word2(b, t);
    lo = ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u; hi = (w & 0xF0F0F0F0u) ^ 0x80808080u; }      // 16 (q - 8)
  static __device__ float scale(const Head& h, int j) { return qs_f16(h.p + 18 * j) * 0.0625f; }
  static __device__ float minimum(const Head&, int) { return 0.0f; } };
struct QiQ8_0 { static constexpr int kUnit = 272; static constexpr bool kSigned = true, kNibbles = false, kSums = false;
  struct Head { const uint8_t* p; };
  static __device__ Head head(const uint8_t* p) { return Head{p}; }
  static __device__ void codes(const uint8_t* p, int j, int t, uint32_t& lo, uint32_t& hi) {
    const uint8_t* b = p + 34 * j + 2;
    if (j & 1) { lo = qi_word(b + 4 * t); hi = qi_word(b + 16 + 4 * t); }
    else { lo = qi_word2(b, t); hi = qi_word2(b, t + 4); } }
  static __device__ float scale(const Head& h, int j) { return qs_f16(h.p + 34 * j); }
  static __device__ float minimum(const Head&, int) { return 0.0f; } };
struct QiQ4K { static constexpr int kUnit = 144; static constexpr bool kSigned = false, kNibbles = true, kSums = true;
  struct Head { uint4 v; };  // d and dmin, twelve bytes of scales
  static __device__ Head head(const uint8_t* p) { return Head{*reinterpret_cast<const uint4*>(p)}; }
  static __device__ void codes(const uint8_t* p, int j, int t, uint32_t& lo, uint32_t& hi) {
    const uint32_t w = qi_word(p + 16 + 16 * j + 4 * t);
    lo = w & 0x0F0F0F0Fu; hi = (w >> 4) & 0x0F0F0F0Fu; }
  static __device__ float six(uint32_t low, uint32_t high, int j) { return qs_int(((low >> (4 * j)) & 15u) | (((high >> (2 * j)) & 3u) << 4)); }
  static __device__ float scale(const Head& h, int j) { return __low2float(*reinterpret_cast<const __half2*>(&h.v.x)) * six(h.v.y, h.v.w, j); }
  static __device__ float minimum(const Head& h, int j) { return -__high2float(*reinterpret_cast<const __half2*>(&h.v.x)) * six(h.v.z, h.v.w >> 16, j); } };

template <typename D, int NB>
__global__ void __launch_bounds__((kQiMaxWarps + 1) * 32, 1) quant_stream_imma_kernel(const __grid_constant__ QiParams p) {
  extern __shared__ __align__(128) uint8_t qi_smem[];      // ring, [warps][NB] units of inputs, [tiles][warps][NB][16] sums
  __shared__ uint64_t full[kQiMaxStages], empty[kQiMaxStages];
  __shared__ float s_sq[NB][kQiMaxWarps];
  __shared__ int s_failed;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = p.warps * 32;
  const int stage_bytes = 16 * p.pitch;
  float* part = reinterpret_cast<float*>(qi_smem + p.stages * stage_bytes + p.warps * NB * kQiUnitBytes);
  const unsigned ntiles = (unsigned)(p.N + 15) >> 4, per = ntiles / gridDim.x, over = ntiles - per * gridDim.x;
  const int tile_lo = (int)(per * blockIdx.x + over * blockIdx.x / gridDim.x), tile_hi = (int)(per * (blockIdx.x + 1) + over * (blockIdx.x + 1) / gridDim.x);
  const int units = p.K >> 8, steps = (tile_hi - tile_lo) * p.nseg;
  const long long row_bytes = (long long)units * D::kUnit;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid < kQiMaxStages) {
    tc::mbar_init(&full[tid], 1);
    tc::mbar_init(&empty[tid], p.warps);
    tc::mbar_fence_init();
  }
  if (tid == 0) s_failed = 0;
  __syncthreads();
  bool failed = false;

  if (warp == p.warps) {
    // ---- producer: lanes 0-15 copy a row's piece each; weights depend on no earlier kernel --------------------------------------------------
    int s = 0, seg = 0, tile = tile_lo, issued = 0;
    uint32_t phase = 1;
    for (; issued < steps; ++issued) {
      if (!__all_sync(0xffffffffu, tc::mbar_wait_sleep<40>(&empty[s], phase))) { failed = true; break; }
      const int first = seg * p.warps, nu = min(p.warps, units - first);
      const uint32_t bytes = (uint32_t)nu * D::kUnit;
      if (lane == 0) tc::mbar_arrive_expect_tx(&full[s], 16 * bytes);
      __syncwarp();
      if (lane < 16)
        tc::bulk_g2s(qi_smem + s * stage_bytes + lane * p.pitch, p.w + (long long)min(tile * 16 + lane, p.N - 1) * row_bytes + (long long)first * D::kUnit, bytes, &full[s]);
      if (++s == p.stages) { s = 0; phase ^= 1; }
      if (++tile == tile_hi) { tile = tile_lo; ++seg; }
    }
    if (lane == 0) tc::mbar_drain(full, issued, p.stages);
    __syncwarp();
  } else if (warp < p.warps) {
    // A lane has terms 2t + 1 and 2t + 2 of rows g and g + 8; of a pair of blocks it comes to add up block t / 2 of row g + 8 (t & 1).
    const int g = lane >> 2, t = lane & 3;
    const bool second = t >> 1, lower = t & 1;
    const float u0 = __uint_as_float((127u - 14u * t) << 23), u1 = u0 * (1.0f / 128.0f), zero = -kQiZero * (u0 + u1);
    // the warp's inputs: block j of term k at 32 (j ^ k) of its 256 bytes, so that the eight terms' words meet no bank twice
    int8_t* const xq = reinterpret_cast<int8_t*>(qi_smem + p.stages * stage_bytes + warp * NB * kQiUnitBytes);
    float2* const blocks = reinterpret_cast<float2*>(xq + NB * kQiTerms * 256);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float sq[NB] = {};
    uint32_t apart[NB] = {};       // bit j: block j of the unit is multiplied in f32
    float4 x[2 * NB], nw[2];       // the unit's inputs and norm weights, first and second half, requested a segment ahead
    auto request = [&](int unit) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = unit * 64 + h * 32 + lane;
        nw[h] = p.norm_w != nullptr ? __ldg(reinterpret_cast<const float4*>(p.norm_w) + c) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
#pragma unroll
        for (int n = 0; n < NB; ++n) x[2 * n + h] = reinterpret_cast<const float4*>(p.x + (size_t)n * p.x_ld)[c];
      }
    };
    request(warp);
    int s = 0;
    uint32_t phase = 0;
    for (int seg = 0; seg < p.nseg && !failed; ++seg) {
      const int unit = seg * p.warps + warp;
      if (unit < units) {
        // ---- inputs: a lane has four neighbours, eight lanes a block of 32 ---------------------------------------------------------------------------
#pragma unroll
        for (int n = 0; n < NB; ++n) {
          apart[n] = 0;
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            const int i = lane & 7, j = half * 4 + (lane >> 3);
            float4 v = half ? x[2 * n + 1] : x[2 * n];
            const float4 ww = half ? nw[1] : nw[0];
            sq[n] += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
            v.x *= ww.x; v.y *= ww.y; v.z *= ww.z; v.w *= ww.w;
            float top = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))), sum = (v.x + v.y) + (v.z + v.w);
            bool odd = !(sum - sum == 0.0f);           // an infinity or a NaN, or close to it
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
              top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
              if (D::kSums) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            }
            // the largest input comes to [2^5, 2^6)
            float scale = __uint_as_float(__float_as_uint(fminf(fmaxf(top, 7.9e-31f), 3.0e38f)) & 0x7F800000u) * 0.03125f;
            const float back = __uint_as_float(0x7F000000u - __float_as_uint(scale));
            float f[4] = {v.x, v.y, v.z, v.w};
            if (D::kNibbles) {     // of eight neighbours the even ones to the even lane, the odd ones to the odd lane, as their codes lie in the words
              const float a = __shfl_xor_sync(0xffffffffu, i & 1 ? f[0] : f[1], 1), b = __shfl_xor_sync(0xffffffffu, i & 1 ? f[2] : f[3], 1);
              const float own0 = i & 1 ? f[1] : f[0], own1 = i & 1 ? f[3] : f[2];
              f[0] = i & 1 ? a : own0; f[1] = i & 1 ? b : own1;
              f[2] = i & 1 ? own0 : a; f[3] = i & 1 ? own1 : b;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool some = f[e] != 0.0f;
              f[e] *= back;
              odd |= some && fabsf(f[e]) < 0x1p-26f;   // its last places lie below those of the eighth term
            }
            const uint32_t lanes = __ballot_sync(0xffffffffu, odd);
            if (lanes != 0) {
#pragma unroll
              for (int b = 0; b < 4; ++b) apart[n] |= ((lanes >> (8 * b)) & 255u) != 0 ? 1u << (half * 4 + b) : 0u;
              if ((apart[n] >> j) & 1) {
#pragma unroll
                for (int e = 0; e < 4; ++e) f[e] = 0.0f;
                scale = 0.0f;
              }
            }
            // (f + 1.5 * 2^23) holds rint(f) in its low byte, and with 2^-7 of it the next term; what is left, at most a half, is up to 64 of the next
            // term's units.  A lane's codes of a block are those of inputs 8t .. 8t + 7, even before odd (nibbles), or 4t .. 4t + 3 and 16 + 4t .. (bytes).
            int8_t* dst = xq + n * kQiTerms * 256 + (D::kNibbles ? (i >> 1) * 8 + (i & 1) * 4 : (i & 3) * 8 + (i >> 2) * 4);
#pragma unroll
            for (int k = 0; k < kQiTerms; ++k) {
              constexpr float kUnits[kQiTerms] = {1.0f, 0x1p-7f, 0x1p-14f, 0x1p-21f, 0x1p-28f, 0x1p-35f, 0x1p-42f, 0x1p-49f};
              const float z = kQiZero * kUnits[k];
              uint32_t q[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float m = f[e] + z;
                q[e] = __float_as_uint(m);
                f[e] -= m - z;
              }
              *reinterpret_cast<uint32_t*>(dst + k * 256 + 32 * (j ^ k)) = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
            }
            if (i == 0) blocks[n * 8 + j] = make_float2(scale, sum);
          }
        }
        if (unit + p.warps < units) request(unit + p.warps);
        __syncwarp();
      }
      // ---- rows -----------------------------------------------------------------------------------------------------------------------------------
      for (int tl = 0; tl < tile_hi - tile_lo; ++tl) {
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&full[s], phase))) { failed = true; break; }
        if (unit < units) {
          const uint8_t *r0 = qi_smem + s * stage_bytes + g * p.pitch + warp * D::kUnit, *r1 = r0 + 8 * p.pitch;
          const auto head = D::head(lower ? r1 : r0);
          float tot[NB] = {};
#pragma unroll
          for (int pr = 0; pr < 4; ++pr) {
            uint32_t a[4], b[4];
            D::codes(r0, 2 * pr, t, a[0], a[2]);
            D::codes(r1, 2 * pr, t, a[1], a[3]);
            D::codes(r0, 2 * pr + 1, t, b[0], b[2]);
            D::codes(r1, 2 * pr + 1, t, b[1], b[3]);
            const int j = 2 * pr + second;
            const float scale = D::scale(head, j), minimum = D::minimum(head, j);
#pragma unroll
            for (int n = 0; n < NB; ++n) {
              const int8_t* xu = xq + (n * kQiTerms + g) * 256 + t * 8;
              const float2 bl = blocks[n * 8 + j];
              float da[4], db[4];
              qi_mma<D::kSigned>(da, a, *reinterpret_cast<const uint2*>(xu + 32 * ((2 * pr) ^ g)));
              qi_mma<D::kSigned>(db, b, *reinterpret_cast<const uint2*>(xu + 32 * ((2 * pr + 1) ^ g)));
              // two terms of a sum: the inner step is exact (integers below 2^19 in units of u0)
              const float a0 = fmaf(da[1], u1, fmaf(da[0], u0, zero)), a1 = fmaf(da[3], u1, fmaf(da[2], u0, zero));
              const float b0 = fmaf(db[1], u1, fmaf(db[0], u0, zero)), b1 = fmaf(db[3], u1, fmaf(db[2], u0, zero));
              const float v0 = (second ? b0 : a0) + __shfl_xor_sync(0xffffffffu, second ? a0 : b0, 2);
              const float v1 = (second ? b1 : a1) + __shfl_xor_sync(0xffffffffu, second ? a1 : b1, 2);
              const float v = (lower ? v1 : v0) + __shfl_xor_sync(0xffffffffu, lower ? v0 : v1, 1);
              tot[n] = fmaf(scale * bl.x, v, tot[n]);
              if (D::kSums) tot[n] = fmaf(minimum, bl.y, tot[n]);
            }
          }
#pragma unroll
          for (int n = 0; n < NB; ++n) {
#pragma unroll 1
            for (uint32_t left = apart[n]; left != 0; left &= left - 1) {
              const int j = __ffs(left) - 1;
              uint32_t w[2][2];
              D::codes(r0, j, t, w[0][0], w[0][1]);
              D::codes(r1, j, t, w[1][0], w[1][1]);
              float v[2] = {0.0f, 0.0f};
#pragma unroll 1
              for (int e = 0; e < 8; ++e) {
                const int k = unit * 256 + j * 32 + (D::kNibbles ? 8 * t + 2 * (e & 3) + (e >> 2) : 16 * (e >> 2) + 4 * t + (e & 3));
                const float in = p.x[(size_t)n * p.x_ld + k] * (p.norm_w != nullptr ? __ldg(p.norm_w + k) : 1.0f);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  const uint32_t q = (e < 4 ? w[r][0] : w[r][1]) >> (8 * (e & 3));
                  v[r] = fmaf(D::kSigned ? (float)(int8_t)q : (float)(q & 255u), in, v[r]);
                }
              }
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                v[r] += __shfl_xor_sync(0xffffffffu, v[r], 1);
                v[r] += __shfl_xor_sync(0xffffffffu, v[r], 2);
              }
              if (!second) tot[n] += D::scale(head, j) * (lower ? v[1] : v[0]);
            }
            const float v = tot[n] + __shfl_xor_sync(0xffffffffu, tot[n], 2);
            if (!second) {
              float* sum = part + ((tl * p.warps + warp) * NB + n) * 16 + g + 8 * lower;
              *sum = seg == 0 ? v : *sum + v;
            }
          }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[s]);
        if (++s == p.stages) { s = 0; phase ^= 1; }
      }
    }
#pragma unroll
    for (int n = 0; n < NB; ++n) {
      sq[n] = warp_sum(sq[n]);
      if (lane == 0) s_sq[n][warp] = sq[n];
    }
  }
  if (failed) {                  // a copy that never arrived: its rows come out as NaN instead of numbers made of old data
    s_failed = 1;
    if (lane == 0 && p.status != nullptr) atomicExch(p.status, 5);
  }
  __syncthreads();
  if (warp >= p.warps) return;
  const int row0 = tile_lo * 16, rows = min(tile_hi * 16, p.N) - row0;
#pragma unroll
  for (int n = 0; n < NB; ++n) {
    float inv = 1.0f;
    if (p.norm_w != nullptr) {
      float ss = 0.0f;
      for (int k = 0; k < p.warps; ++k) ss += s_sq[n][k];
      inv = 1.0f / sqrtf(ss / (float)p.K + p.eps);
    }
    for (int i = tid; i < rows; i += nthr) {
      float a[4] = {};           // four short sums: one of them long would round more than the rest together
      for (int k = 0; k < p.warps; k += 4) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (k + e < p.warps) a[e] += part[(((i >> 4) * p.warps + k + e) * NB + n) * 16 + (i & 15)];
      }
      const float v = (a[0] + a[1]) + (a[2] + a[3]);
      const size_t o = (size_t)n * p.out_ld + row0 + i;
      p.out[o] = s_failed ? __int_as_float(0x7FFFFFFF) : (p.residual ? p.residual[o] : 0.0f) + v * inv;
    }
  }
}

// Of the matrices that can be streamed: whole units of 256 inputs, a tile of rows at least, and what makes the split of the inputs by every CTA worth
// its time whether there is a second token or not.  Rows of more than 12288 gain with one token and lose with two (2560 x 14336 in Q4_K: 16.4 us above
// and 15.5 here, two tokens 20.9 and 24.9), small matrices with two (2048 x 2048 in Q4_K: 4.0 and 4.0, two tokens 5.4 and 6.7; 2560 x 2560: 6.0 and 5.0,
// 8.0 and 7.6).  The rule looks at the matrix alone, and warps and segments leave room for two tokens: a token's sums are the same with and without a
// second one.
template <typename D, int NB>
static bool qi_launch(const QsParams& q, cudaStream_t st, int& rc) {
  const int N = q.N, K = q.K;
  if (K % 256 != 0 || K > 12288 || N < 16 || (long long)N * K < 6000000) return false;
  QiParams p{q.w, q.x, q.norm_w, q.residual, q.out, q.status, q.eps, N, K, 0, 0, 0, 0, q.x_ld, q.out_ld};
  const int units = K / 256, tiles = (N + 15) / 16;
  int grid = tiles < 148 ? tiles : 148;
  if ((tiles + grid - 1) / grid > kQiMaxTiles) grid = (tiles + kQiMaxTiles - 1) / kQiMaxTiles;
  const int per = (tiles + grid - 1) / grid;
  int token, stage;
  p.nseg = (units + kQiMaxWarps - 1) / kQiMaxWarps - 1;
  do {                           // (with one warp it is far less)
    ++p.nseg;
    p.warps = (units + p.nseg - 1) / p.nseg;
    p.pitch = p.warps * D::kUnit;
    if ((p.pitch / 16) % 2 == 0) p.pitch += 16;
    token = p.warps * (kQiUnitBytes + per * 16 * 4);
    stage = 16 * p.pitch;
  } while (2 * (token + stage) > kQiSmem);
  p.stages = (kQiSmem - NB * token) / stage;
  if (p.stages > kQiMaxStages) p.stages = kQiMaxStages;
  const size_t smem = (size_t)NB * token + (size_t)p.stages * stage;
  static std::atomic<bool> configured[64];
  int dev = 0;
  rc = BONSAI_CUDA_LAUNCH_FAILED;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(quant_stream_imma_kernel<D, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kQiSmem) != cudaSuccess) return true;
    configured[dev].store(true, std::memory_order_release);
  }
  if (launch_pdl(quant_stream_imma_kernel<D, NB>, dim3(grid), dim3((p.warps + 1) * 32), smem, st, p) == cudaSuccess) rc = BONSAI_CUDA_OK;
  return true;
}
template <typename D, int NB>
static bool qi_try(const QsParams& p, cudaStream_t st, int& rc) {
  if constexpr (std::is_same_v<D, DecQ4_0>) return qi_launch<QiQ4_0, NB>(p, st, rc);
  else if constexpr (std::is_same_v<D, DecQ8_0>) return qi_launch<QiQ8_0, NB>(p, st, rc);
  else if constexpr (std::is_same_v<D, DecQ4K>) return qi_launch<QiQ4K, NB>(p, st, rc);
  else return false;
}

template <typename D>
__global__ void __launch_bounds__(256) quant_gemv_kernel(const uint8_t* __restrict__ w, const float* __restrict__ x,
                                                        const float* __restrict__ norm_w, float eps, float* __restrict__ out,
                                                        const float* __restrict__ residual, int N, int K) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblk = K / D::kElems;
  const size_t row_bytes = (size_t)nblk * D::kBytes;
  float inv = 1.0f;
  if (norm_w != nullptr) {
    float ss = 0.0f;
    for (int k = lane; k < K; k += 32) ss += x[k] * x[k];
    inv = 1.0f / sqrtf(warp_sum(ss) / (float)K + eps);
  }
  for (int row = blockIdx.x * 8 + warp; row < N; row += gridDim.x * 8) {
    const uint8_t* rp = w + (size_t)row * row_bytes;
    float acc = 0.0f;
    if (D::kElems == 32) {
      for (int b = lane; b < nblk; b += 32) {
        const uint8_t* p = rp + (size_t)b * D::kBytes;
        const float* xp = x + b * 32;
        const float* nw = norm_w ? norm_w + b * 32 : nullptr;
#pragma unroll 8
        for (int i = 0; i < 32; ++i) acc = fmaf(D::at(p, i), nw ? xp[i] * nw[i] : xp[i], acc);
      }
    } else {
      for (int b = 0; b < nblk; ++b) {
        const uint8_t* p = rp + (size_t)b * D::kBytes;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = lane * 8 + j, k = b * 256 + i;
          acc = fmaf(D::at(p, i), norm_w ? x[k] * norm_w[k] : x[k], acc);
        }
      }
    }
    acc = warp_sum(acc) * inv;
    if (lane == 0) out[row] = (residual ? residual[row] : 0.0f) + acc;
  }
}

template <typename D, typename Q>
static int launch_quant_gemv(const void* w, const float* x, const float* norm_w, float eps, float* out, const float* residual, int N, int K,
                             int* status, cudaStream_t st) {
  if (K % D::kElems != 0) return BONSAI_CUDA_BAD_ARG;
  QsParams p = qs_params<D>(w, x, K, norm_w, eps, out, residual, N, N, K, status);
  int sgrid;
  size_t smem;
  if (qs_plan<Q>(p, sgrid, smem, 1)) {
    int rc;
    return qi_try<D, 1>(p, st, rc) ? rc : qs_launch<Q, 1>(p, sgrid, smem, st);
  }
  int grid = (N + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  quant_gemv_kernel<D><<<grid, 256, 0, st>>>((const uint8_t*)w, x, norm_w, eps, out, residual, N, K);
  return launch_status();
}

// The same product for NB activation rows at once (a decode batch): every weight element is decoded once and multiplied into
// NB accumulators.  x: [B][x_ld], out / residual: [B][out_ld]; rows b >= B of the NB-wide template are computed on row B - 1's
// input and not stored.
template <typename D, int NB>
__global__ void __launch_bounds__(256) quant_gemv_batched_kernel(const uint8_t* __restrict__ w, const float* __restrict__ x, int x_ld,
                                                                const float* __restrict__ norm_w, float eps, float* __restrict__ out,
                                                                const float* __restrict__ residual, int out_ld, int N, int K, int B) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblk = K / D::kElems;
  const size_t row_bytes = (size_t)nblk * D::kBytes;
  const float* xs[NB];
  float inv[NB];
#pragma unroll
  for (int t = 0; t < NB; ++t) {
    xs[t] = x + (size_t)(t < B ? t : B - 1) * x_ld;
    inv[t] = 1.0f;
    if (norm_w != nullptr) {
      float ss = 0.0f;
      for (int k = lane; k < K; k += 32) ss += xs[t][k] * xs[t][k];
      inv[t] = 1.0f / sqrtf(warp_sum(ss) / (float)K + eps);
    }
  }
  for (int row = blockIdx.x * 8 + warp; row < N; row += gridDim.x * 8) {
    const uint8_t* rp = w + (size_t)row * row_bytes;
    float acc[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) acc[t] = 0.0f;
    if (D::kElems == 32) {
      for (int b = lane; b < nblk; b += 32) {
        const uint8_t* p = rp + (size_t)b * D::kBytes;
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
          const int k = b * 32 + i;
          const float wv = D::at(p, i) * (norm_w ? norm_w[k] : 1.0f);
#pragma unroll
          for (int t = 0; t < NB; ++t) acc[t] = fmaf(wv, xs[t][k], acc[t]);
        }
      }
    } else {
      for (int b = 0; b < nblk; ++b) {
        const uint8_t* p = rp + (size_t)b * D::kBytes;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = lane * 8 + j, k = b * 256 + i;
          const float wv = D::at(p, i) * (norm_w ? norm_w[k] : 1.0f);
#pragma unroll
          for (int t = 0; t < NB; ++t) acc[t] = fmaf(wv, xs[t][k], acc[t]);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const float v = warp_sum(acc[t]) * inv[t];
      if (lane == 0 && t < B) out[(size_t)t * out_ld + row] = (residual ? residual[(size_t)t * out_ld + row] : 0.0f) + v;
    }
  }
}

template <typename D, typename Q>
static int launch_quant_gemv_batched(const void* w, const float* x, int x_ld, const float* norm_w, float eps, float* out, const float* residual,
                                     int out_ld, int N, int K, int B, int* status, cudaStream_t st) {
  if (K % D::kElems != 0) return BONSAI_CUDA_BAD_ARG;
  int grid = (N + 7) / 8;
  if (grid > 148 * 8) grid = 148 * 8;
  const uint8_t* wp = (const uint8_t*)w;
  {
    QsParams p = qs_params<D>(w, x, x_ld, norm_w, eps, out, residual, out_ld, N, K, status);
    int sgrid, rc = BONSAI_CUDA_OK;
    size_t smem;
    if (qs_plan<Q>(p, sgrid, smem, 2)) {
      for (int b = 0; b < B && rc == BONSAI_CUDA_OK; b += 2) {       // the second pair's weights come from L2 when the matrix fits there
        p.x = x + (size_t)b * x_ld;
        p.out = out + (size_t)b * out_ld;
        p.residual = residual ? residual + (size_t)b * out_ld : nullptr;
        const bool two = b + 1 < B;
        if (two ? qi_try<D, 2>(p, st, rc) : qi_try<D, 1>(p, st, rc)) continue;
        rc = two ? qs_launch<Q, 2>(p, sgrid, smem, st) : qs_launch<Q, 1>(p, sgrid, smem, st);
      }
      return rc;
    }
  }
  // groups of up to eight rows: the weights of a later group come from L2 when the matrix fits there
  for (int b0 = 0; b0 < B; b0 += 8) {
    const int nb = B - b0 < 8 ? B - b0 : 8;
    const float* xb = x + (size_t)b0 * x_ld;
    float* ob = out + (size_t)b0 * out_ld;
    const float* rb = residual ? residual + (size_t)b0 * out_ld : nullptr;
    if (nb == 1) quant_gemv_kernel<D><<<grid, 256, 0, st>>>(wp, xb, norm_w, eps, ob, rb, N, K);
    else if (nb == 2) quant_gemv_batched_kernel<D, 2><<<grid, 256, 0, st>>>(wp, xb, x_ld, norm_w, eps, ob, rb, out_ld, N, K, nb);
    else if (nb <= 4) quant_gemv_batched_kernel<D, 4><<<grid, 256, 0, st>>>(wp, xb, x_ld, norm_w, eps, ob, rb, out_ld, N, K, nb);
    else quant_gemv_batched_kernel<D, 8><<<grid, 256, 0, st>>>(wp, xb, x_ld, norm_w, eps, ob, rb, out_ld, N, K, nb);
  }
  return launch_status();
}

// Decodes an [N][K] matrix of blocks into row-major f16 for the dense tensor-core GEMM of the prompt path.  One thread
// owns eight consecutive inputs and stores them as one 16-byte word.  With `paired` the eight values are written in the
// K order of the GEMM's activation operand (inside every 16 inputs: position (j & 8) | ((j & 3) * 2 + ((j >> 2) & 1))
// for input j), so the prompt path's normalisation and attention kernels can feed the GEMM without a transpose.
template <typename D>
__global__ void __launch_bounds__(256) quant_to_f16_kernel(const uint8_t* __restrict__ w, __half* __restrict__ out, int N, int K, int paired) {
  const int nblk = K / D::kElems, per_row = K / 8;
  const size_t row_bytes = (size_t)nblk * D::kBytes;
  const size_t total = (size_t)N * per_row;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(idx / per_row), k0 = (int)(idx % per_row) * 8;
    const uint8_t* bp = w + (size_t)row * row_bytes + (size_t)(k0 / D::kElems) * D::kBytes;
    const int i0 = k0 % D::kElems;
    __align__(16) __half v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int dst = paired ? ((j & 3) * 2 + ((j >> 2) & 1)) : j;
      v[dst] = __float2half_rn(D::at(bp, i0 + j));
    }
    *reinterpret_cast<uint4*>(out + (size_t)row * K + k0) = *reinterpret_cast<const uint4*>(v);
  }
}

// The same with 32 weights per thread, decoded from whole words: a warp turns 32 neighbouring blocks of 32 into 2 KB of rows, which go through
// shared memory so that its stores are whole lines.  Row r of the matrix becomes row r * mul + add of out.  The last block, behind whose words
// nothing needs to be readable, is decoded value by value.  2560 x 9728 in Q8_0: 18.5 us with eight byte loads per thread, 13.5 here.
template <typename D, typename Q>
__global__ void __launch_bounds__(256) quant_rows_kernel(const uint8_t* __restrict__ w, uint4* __restrict__ out, int N, int K, int paired, int mul, int add) {
  __shared__ uint4 stage[8][128];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");      // the product ahead reads the scratch matrix
  const int per_row = K >> 5, total = N * per_row, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row_bytes = (long long)(K / D::kElems) * D::kBytes;
  for (int first = (blockIdx.x * 8 + warp) * 32; first < total; first += gridDim.x * 256) {
    const int i = first + lane, row = min(i, total - 1) / per_row, b = min(i, total - 1) - row * per_row;
    uint32_t o[16];
    auto put = [&](int g, const float* v) {               // eight neighbours
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const __half2 h = paired ? __floats2half2_rn(v[k], v[k + 4]) : __floats2half2_rn(v[2 * k], v[2 * k + 1]);
        o[4 * g + k] = *reinterpret_cast<const uint32_t*>(&h);
      }
    };
    if (i < total - 1) {
      Q d;
      d.load(w + row * row_bytes, b);
      constexpr int G = 32 / Q::kScales;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          const uint64_t q = d.q2(g * 8 + j);
          float x, y;
          asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(q));
          const float sc = d.s[(g * 8 + j) / G];
          const float m = Q::kMin ? d.m[(g * 8 + j) / G] : 0.0f;
          v[j] = Q::kMin ? fmaf(sc, x, -m) : sc * x;
          v[j + 1] = Q::kMin ? fmaf(sc, y, -m) : sc * y;
        }
        put(g, v);
      }
    } else {
      const uint8_t* p = w + row * row_bytes + (size_t)(b * 32 / D::kElems) * D::kBytes;
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = D::at(p, b * 32 % D::kElems + g * 8 + j);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (g == k) put(k, v);
      }
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) stage[warp][lane * 4 + (g ^ ((lane >> 1) & 3))] = make_uint4(o[4 * g], o[4 * g + 1], o[4 * g + 2], o[4 * g + 3]);
    const long long base = ((long long)(row * mul + add) * per_row + b) * 4;
    __syncwarp();
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int src = 8 * g + (lane >> 2);                // the lane whose block this is
      const long long at = __shfl_sync(0xffffffffu, base, src);
      if (first + src < total) out[at + (lane & 3)] = stage[warp][src * 4 + ((lane & 3) ^ ((src >> 1) & 3))];
    }
    __syncwarp();
  }
}

template <typename D, typename Q>
static int launch_quant_to_f16(const void* w, void* out, int N, int K, int paired, int mul, int add, cudaStream_t st) {
  if (K % D::kElems != 0 || K % 16 != 0) return BONSAI_CUDA_BAD_ARG;
  if (K % 32 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (long long)N * K < (1ll << 36)) {
    const long long groups = ((long long)N * (K >> 5) + 255) / 256;
    const int grid = (int)(groups < 148 * 8 ? groups : 148 * 8);
    return launch_pdl(quant_rows_kernel<D, Q>, dim3(grid), dim3(256), 0, st, (const uint8_t*)w, (uint4*)out, N, K, paired, mul, add) == cudaSuccess
               ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
  }
  if (mul != 1 || add != 0) return BONSAI_CUDA_BAD_ARG;
  const size_t total = (size_t)N * (K / 8);
  int grid = (int)((total + 255) / 256 < (size_t)(148 * 16) ? (total + 255) / 256 : (size_t)(148 * 16));
  quant_to_f16_kernel<D><<<grid, 256, 0, st>>>((const uint8_t*)w, (__half*)out, N, K, paired);
  return launch_status();
}

static int quant_to_f16(int type, const void* w, void* out, int N, int K, int paired, int mul, int add, cudaStream_t st) {
  switch (type) {
    case 0: return launch_quant_to_f16<DecF32, QsF32>(w, out, N, K, paired, mul, add, st);
    case 1: return launch_quant_to_f16<DecF16, QsF16>(w, out, N, K, paired, mul, add, st);
    case 30: return launch_quant_to_f16<DecBF16, QsBF16>(w, out, N, K, paired, mul, add, st);
    case 2: return launch_quant_to_f16<DecQ4_0, QsQ4_0>(w, out, N, K, paired, mul, add, st);
    case 8: return launch_quant_to_f16<DecQ8_0, QsQ8_0>(w, out, N, K, paired, mul, add, st);
    case 10: return launch_quant_to_f16<DecQ2K, QsQ2K>(w, out, N, K, paired, mul, add, st);
    case 11: return launch_quant_to_f16<DecQ3K, QsQ3K>(w, out, N, K, paired, mul, add, st);
    case 12: return launch_quant_to_f16<DecQ4K, QsQ4K>(w, out, N, K, paired, mul, add, st);
    case 13: return launch_quant_to_f16<DecQ5K, QsQ5K>(w, out, N, K, paired, mul, add, st);
    case 14: return launch_quant_to_f16<DecQ6K, QsQ6K>(w, out, N, K, paired, mul, add, st);
    case 15: return launch_quant_to_f16<DecQ8K, QsQ8K>(w, out, N, K, paired, mul, add, st);
    case 35: return launch_quant_to_f16<DecTq2_256, QsTq2_256>(w, out, N, K, paired, mul, add, st);
    case 43: return launch_quant_to_f16<DecFp8<false>, QsFp8<false>>(w, out, N, K, paired, mul, add, st);
    case 44: return launch_quant_to_f16<DecFp8<true>, QsFp8<true>>(w, out, N, K, paired, mul, add, st);
    default: return BONSAI_CUDA_BAD_ARG;
  }
}

int quant_rows_to_f16(int type, const void* w, int rows, int K, void* out, int mul, int add, cudaStream_t st) {
  return quant_to_f16(type, w, out, rows, K, 1, mul, add, st);
}
long long quant_row_bytes(int type, int K) {
  switch (type) {
    case 0: return (long long)K * 4;
    case 1: case 30: return (long long)K * 2;
    case 2: return (long long)K / 32 * DecQ4_0::kBytes;
    case 8: return (long long)K / 32 * DecQ8_0::kBytes;
    case 10: return (long long)K / 256 * DecQ2K::kBytes;
    case 11: return (long long)K / 256 * DecQ3K::kBytes;
    case 12: return (long long)K / 256 * DecQ4K::kBytes;
    case 13: return (long long)K / 256 * DecQ5K::kBytes;
    case 14: return (long long)K / 256 * DecQ6K::kBytes;
    case 15: return (long long)K / 256 * DecQ8K::kBytes;
    case 35: return (long long)K / 256 * DecTq2_256::kBytes;
    case 43: case 44: return (long long)K / 32 * DecFp8<false>::kBytes;
    default: return -1;
  }
}

// out[t][i] = silu(gu[t][i]) * gu[t][inter + i]: the activation after a fused gate || up projection of T rows
__global__ void swiglu_rows_kernel(const float* __restrict__ gu, int gu_ld, float* __restrict__ out, int out_ld, int inter, int T) {
  const size_t total = (size_t)T * inter;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(idx / inter), i = (int)(idx % inter);
    const float g = gu[(size_t)t * gu_ld + i];
    out[(size_t)t * out_ld + i] = g / (1.0f + __expf(-g)) * gu[(size_t)t * gu_ld + inter + i];
  }
}

__global__ void swiglu_kernel(const float* __restrict__ gate, const float* __restrict__ up, float* __restrict__ out, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float g = gate[i];
    out[i] = g / (1.0f + __expf(-g)) * up[i];
  }
}

}  // namespace bonsai

extern "C" {

// out[N] = (residual or 0) + W (rmsnorm(x) or x) for a row-major matrix of GGUF blocks of `type`
// (GGUF type ids: 0 F32, 1 F16, 30 BF16, 2 Q4_0, 8 Q8_0, 10-15 Q2_K..Q8_K, 35 TQ2_0, 43 / 44 FP8 E4M3 / E5M2).
// status (may be null): a word that takes code 5 when a wait for a copy of the matrix expired; its rows are then NaN.
int bonsai_quant_gemv_status(int type, const void* w, const float* x, const float* norm_w, float eps, float* out, const float* residual,
                             int N, int K, int* status, cudaStream_t stream) {
  using namespace bonsai;
  if (N <= 0 || K <= 0) return BONSAI_CUDA_BAD_ARG;
  switch (type) {
    case 0: return launch_quant_gemv<DecF32, QsF32>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 1: return launch_quant_gemv<DecF16, QsF16>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 30: return launch_quant_gemv<DecBF16, QsBF16>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 2: return launch_quant_gemv<DecQ4_0, QsQ4_0>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 8: return launch_quant_gemv<DecQ8_0, QsQ8_0>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 10: return launch_quant_gemv<DecQ2K, QsQ2K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 11: return launch_quant_gemv<DecQ3K, QsQ3K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 12: return launch_quant_gemv<DecQ4K, QsQ4K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 13: return launch_quant_gemv<DecQ5K, QsQ5K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 14: return launch_quant_gemv<DecQ6K, QsQ6K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 15: return launch_quant_gemv<DecQ8K, QsQ8K>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 35: return launch_quant_gemv<DecTq2_256, QsTq2_256>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 43: return launch_quant_gemv<DecFp8<false>, QsFp8<false>>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    case 44: return launch_quant_gemv<DecFp8<true>, QsFp8<true>>(w, x, norm_w, eps, out, residual, N, K, status, stream);
    default: return BONSAI_CUDA_BAD_ARG;
  }
}

// The same for B activation rows (a decode batch): x [B][x_ld], out and residual [B][out_ld].
int bonsai_quant_gemv_batched_status(int type, const void* w, const float* x, int x_ld, const float* norm_w, float eps, float* out,
                                     const float* residual, int out_ld, int N, int K, int B, int* status, cudaStream_t stream) {
  using namespace bonsai;
  if (N <= 0 || K <= 0 || B <= 0 || x_ld < K || out_ld < N) return BONSAI_CUDA_BAD_ARG;
#define BONSAI_QGB(...) return launch_quant_gemv_batched<__VA_ARGS__>(w, x, x_ld, norm_w, eps, out, residual, out_ld, N, K, B, status, stream)
  switch (type) {
    case 0: BONSAI_QGB(DecF32, QsF32);
    case 1: BONSAI_QGB(DecF16, QsF16);
    case 30: BONSAI_QGB(DecBF16, QsBF16);
    case 2: BONSAI_QGB(DecQ4_0, QsQ4_0);
    case 8: BONSAI_QGB(DecQ8_0, QsQ8_0);
    case 10: BONSAI_QGB(DecQ2K, QsQ2K);
    case 11: BONSAI_QGB(DecQ3K, QsQ3K);
    case 12: BONSAI_QGB(DecQ4K, QsQ4K);
    case 13: BONSAI_QGB(DecQ5K, QsQ5K);
    case 14: BONSAI_QGB(DecQ6K, QsQ6K);
    case 15: BONSAI_QGB(DecQ8K, QsQ8K);
    case 35: BONSAI_QGB(DecTq2_256, QsTq2_256);
    case 43: BONSAI_QGB(DecFp8<false>, QsFp8<false>);
    case 44: BONSAI_QGB(DecFp8<true>, QsFp8<true>);
    default: return BONSAI_CUDA_BAD_ARG;
  }
#undef BONSAI_QGB
}

int bonsai_quant_gemv(int type, const void* w, const float* x, const float* norm_w, float eps, float* out, const float* residual,
                      int N, int K, cudaStream_t stream) {
  return bonsai_quant_gemv_status(type, w, x, norm_w, eps, out, residual, N, K, nullptr, stream);
}

int bonsai_quant_gemv_batched(int type, const void* w, const float* x, int x_ld, const float* norm_w, float eps, float* out,
                              const float* residual, int out_ld, int N, int K, int B, cudaStream_t stream) {
  return bonsai_quant_gemv_batched_status(type, w, x, x_ld, norm_w, eps, out, residual, out_ld, N, K, B, nullptr, stream);
}

// Rows of x that a launch of bonsai_quant_gemv_batched takes for this matrix (inputs in rows of 16-byte multiples); 0 for a type it does not know.
int bonsai_quant_gemv_rows(int type, const void* w, int N, int K) {
  using namespace bonsai;
  if (N <= 0 || K <= 0) return 0;
  switch (type) {
    case 0: return qs_rows<DecF32, QsF32>(w, N, K);
    case 1: return qs_rows<DecF16, QsF16>(w, N, K);
    case 30: return qs_rows<DecBF16, QsBF16>(w, N, K);
    case 2: return qs_rows<DecQ4_0, QsQ4_0>(w, N, K);
    case 8: return qs_rows<DecQ8_0, QsQ8_0>(w, N, K);
    case 10: return qs_rows<DecQ2K, QsQ2K>(w, N, K);
    case 11: return qs_rows<DecQ3K, QsQ3K>(w, N, K);
    case 12: return qs_rows<DecQ4K, QsQ4K>(w, N, K);
    case 13: return qs_rows<DecQ5K, QsQ5K>(w, N, K);
    case 14: return qs_rows<DecQ6K, QsQ6K>(w, N, K);
    case 15: return qs_rows<DecQ8K, QsQ8K>(w, N, K);
    case 35: return qs_rows<DecTq2_256, QsTq2_256>(w, N, K);
    case 43: return qs_rows<DecFp8<false>, QsFp8<false>>(w, N, K);
    case 44: return qs_rows<DecFp8<true>, QsFp8<true>>(w, N, K);
    default: return 0;
  }
}

int bonsai_swiglu_rows(const float* gu, int gu_ld, float* out, int out_ld, int inter, int T, cudaStream_t stream) {
  if (inter <= 0 || T <= 0 || gu_ld < 2 * inter || out_ld < inter) return BONSAI_CUDA_BAD_ARG;
  const size_t total = (size_t)T * inter;
  int grid = (int)((total + 255) / 256 < (size_t)(148 * 8) ? (total + 255) / 256 : (size_t)(148 * 8));
  bonsai::swiglu_rows_kernel<<<grid, 256, 0, stream>>>(gu, gu_ld, out, out_ld, inter, T);
  return bonsai::launch_status();
}

// out f16 [N][K] = the decoded matrix (same type ids as bonsai_quant_gemv); `paired` selects the activation K order of
// the tcgen05 GEMM instead of the natural one.  `out` must be 16-byte aligned.
int bonsai_quant_to_f16(int type, const void* w, void* out, int N, int K, int paired, cudaStream_t stream) {
  using namespace bonsai;
  if (N <= 0 || K <= 0 || (reinterpret_cast<uintptr_t>(out) & 15) != 0) return BONSAI_CUDA_BAD_ARG;
  return quant_to_f16(type, w, out, N, K, paired, 1, 0, stream);
}

int bonsai_swiglu(const float* gate, const float* up, float* out, int n, cudaStream_t stream) {
  if (n <= 0) return BONSAI_CUDA_BAD_ARG;
  int grid = (n + 255) / 256;
  if (grid > 148 * 4) grid = 148 * 4;
  bonsai::swiglu_kernel<<<grid, 256, 0, stream>>>(gate, up, out, n);
  return bonsai::launch_status();
}

}  // extern "C"
