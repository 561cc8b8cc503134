// Causal GQA attention of a prompt chunk on tcgen05, head size 128.
//
// attention_prefill.cu computes 64 queries x 64 keys per step on mma.sync: one ldmatrix per two MMAs, 130 TFLOP/s over a 4096-token
// prompt.  Here a CTA owns two tiles of 128 query rows of one kv head (128 / G neighbouring tokens x the G heads of the group, so
// that they share keys and values) and walks the keys 128 at a time:
//   warp 8      copies K and V tiles (TMA, 64-key boxes; a page of the cache is a box, quantised caches are decoded to f16 first)
//   warp 9      S = Q K^T and O += P V for the two tiles in turn: while the tensor core works for one tile, the other's scores
//               are in its softmax
//   warps 0-3, 4-7   softmax of a tile: a thread owns a query row, reads its 128 scores from TMEM, and leaves P as f16 in their
//               place, from where the second product takes it as its first operand; no shuffles, no shared memory
// The sums are rescaled only when a row's maximum has grown by more than 2^8 since its scale was set (P stays below 2^8 then, well
// inside f16, and keeps its relative precision); a tile that needs it rescales O in TMEM.  That, and two query tiles taking turns on the
// tensor core, are published ideas (FlashAttention-4).
// Scores are base-2 (scale and log2 e are folded into the f16 queries), sums and maxima f32, P f16, as in the other kernel.
// Both products of a 128 x 128 tile take 1024 cycles of the tensor core, its 16 K exponentials as many of the MUFU: what is left is
// their overlap.  Figures at attn_prefill_tc below.
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace bonsai {

constexpr int kAtThreads = 320;
constexpr int kAtStalled = 6;                          // status of an expired wait
constexpr int kAtTile = 128 * 128 * 2;                 // bytes of a [128][128] f16 tile: two halves of 64 columns, 128-byte swizzle
constexpr int kAtSmem = 1024 + 6 * kAtTile;            // Q of two tiles, two stages of K and V

struct AtParams {
  const float* q;
  const int* bt;
  __half* out;
  int* status;             // may be null
  int T, pos0, nq, nkv, page, paged, n_pad, out_ld;
  float scale;
};

__device__ __forceinline__ void at_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map),
               "r"(x), "r"(y), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void at_mma_tmem(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void at_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void at_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float at_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// V as the second operand with its columns contiguous: 64-column blocks 16 KB apart, groups of eight keys 1 KB apart
__device__ __forceinline__ uint64_t at_desc_v(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)(16384 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// grid (kv heads, query blocks); G: query heads of a kv head
template <int G>
__global__ void __launch_bounds__(kAtThreads, 1) attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                                                                       AtParams p) {
  constexpr int TOK = 128 / G;                         // tokens of a tile
  extern __shared__ uint8_t at_smem[];
  uint8_t* base = (uint8_t*)(((uintptr_t)at_smem + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = base;                                  // two tiles
  uint8_t* sK = base + 2 * kAtTile;                    // two stages
  uint8_t* sV = base + 4 * kAtTile;
  __shared__ uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_full[2];
  __shared__ uint32_t tmem_slot;
  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
  const int kvh = blockIdx.x, tok_first = (gridDim.y - 1 - blockIdx.y) * 2 * TOK;      // the longest blocks go first
  const int total = p.pos0 + p.T;                      // keys of the sequence
  // key tiles of the two query tiles; the second one may have no tokens at all
  const int n0 = (min(p.pos0 + tok_first + TOK, total) + 127) >> 7, n1 = (min(p.pos0 + tok_first + 2 * TOK, total) + 127) >> 7;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == 9) {
    tc::tmem_alloc(&tmem_slot, 512);
    tc::tmem_relinquish();
  }
  if (t == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&k_full[i], 1);
      tc::mbar_init(&k_empty[i], 1);
      tc::mbar_init(&v_full[i], 1);
      tc::mbar_init(&v_empty[i], 1);
      tc::mbar_init(&s_full[i], 1);
      tc::mbar_init(&p_ready[i], 4);
      tc::mbar_init(&o_full[i], 1);
    }
    tc::mbar_fence_init();
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp < 8) {
    // queries as f16, scaled: a row per warp and step, four columns per lane
    const int tile = warp >> 2;
    for (int r = warp & 3; r < 128; r += 4) {
      const int tok = tok_first + tile * TOK + r / G, head = kvh * G + r % G;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (tok < p.T) v = __ldg(reinterpret_cast<const float4*>(p.q + ((size_t)tok * p.nq + head) * 128) + lane);
      const __half2 a = __floats2half2_rn(v.x * p.scale, v.y * p.scale), b = __floats2half2_rn(v.z * p.scale, v.w * p.scale);
      uint2 w;
      w.x = *reinterpret_cast<const uint32_t*>(&a);
      w.y = *reinterpret_cast<const uint32_t*>(&b);
      *reinterpret_cast<uint2*>(sQ + tile * kAtTile + (lane >> 4) * 16384 + tc::sw128_offset(r, (lane & 15) >> 1) + (lane & 1) * 8) = w;
    }
    tc::fence_proxy_async();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t taddr = tmem_slot;
  bool failed = false;

  if (warp == 8) {
    if (tc::elect_one()) {
      int issued[2] = {0, 0};
      for (int j = 0; j < n1 && !failed; ++j) {
        const int st = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        int row[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int key = min(j * 128 + h * 64, ((total - 1) >> 6) << 6);      // a box behind the last key: any box that exists
          row[h] = p.paged ? (p.bt[key / p.page] * p.nkv + kvh) * p.page + key % p.page : kvh * p.n_pad + key;
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint64_t* full = m ? &v_full[st] : &k_full[st];
          const uint32_t dst = tc::smem_u32((m ? sV : sK) + st * kAtTile);
          if (!tc::mbar_wait(m ? &v_empty[st] : &k_empty[st], ph)) { failed = true; break; }
          tc::mbar_arrive_expect_tx(full, kAtTile);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int x = 0; x < 2; ++x) at_load(dst + x * 16384 + h * 8192, m ? &vmap : &kmap, x * 64, row[h], full);
          ++issued[m];
        }
      }
      tc::mbar_drain(k_full, issued[0], 2);
      tc::mbar_drain(v_full, issued[1], 2);
      if (failed && p.status != nullptr) atomicExch(p.status, kAtStalled);
    }
  } else if (warp == 9) {
    const uint32_t ids = tc::idesc_f32acc(tc::FMT_F16, tc::FMT_F16, 128, 128), idv = ids | (1u << 16);
    for (int j = 0; j <= n1 && !failed; ++j) {
      if (j < n1 && !__all_sync(0xffffffffu, tc::mbar_wait(&k_full[j & 1], (j >> 1) & 1))) { failed = true; break; }
      if (j > 0) {
        const int i = j - 1;
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&v_full[i & 1], (i >> 1) & 1))) { failed = true; break; }
        if (i * 128 + 128 > total) {      // rows behind the last key may hold anything; 0 x anything has to be 0
          uint8_t* v = sV + (i & 1) * kAtTile;
          for (int r = (total & 127) * 16 + lane; r < 128 * 16; r += 32)
            *reinterpret_cast<uint4*>(v + ((r & 8) << 11) + (r >> 4) * 128 + (r & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          tc::fence_proxy_async();
          __syncwarp();
        }
      }
      for (int u = 0; u < 2; ++u) {
        const int n = u ? n1 : n0;
        if (j > 0 && j <= n) {
          if (!__all_sync(0xffffffffu, tc::mbar_wait(&p_ready[u], (j - 1) & 1))) { failed = true; break; }
          tc::tc_fence_after();
          if (tc::elect_one()) {
            const uint64_t dv = at_desc_v(tc::smem_u32(sV + ((j - 1) & 1) * kAtTile));
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) at_mma_tmem(taddr + 256 + u * 128, taddr + u * 128 + k * 8, dv + k * (2048 >> 4), idv, j > 1 || k > 0);
            if (j == n) tc::mma_commit(&o_full[u]);
          }
          __syncwarp();
        }
        if (u == 1 && j > 0 && j < n1 && tc::elect_one()) tc::mma_commit(&v_empty[(j - 1) & 1]);
        __syncwarp();
        if (j < n) {
          tc::tc_fence_after();
          if (tc::elect_one()) {
            const uint64_t dq = tc::smem_desc_sw128(tc::smem_u32(sQ + u * kAtTile)), dk = tc::smem_desc_sw128(tc::smem_u32(sK + (j & 1) * kAtTile));
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
              tc::mma_f16(taddr + u * 128, dq + (k >> 2) * (16384 >> 4) + (k & 3) * 2, dk + (k >> 2) * (16384 >> 4) + (k & 3) * 2, ids, k > 0);
            tc::mma_commit(&s_full[u]);
          }
          __syncwarp();
        }
      }
      if (j < n1 && tc::elect_one()) tc::mma_commit(&k_empty[j & 1]);
      __syncwarp();
    }
    if (failed && lane == 0 && p.status != nullptr) atomicExch(p.status, kAtStalled);
  } else {
    const int u = warp >> 2, n = u ? n1 : n0, r = t & 127;
    const int tok = tok_first + u * TOK + r / G, head = kvh * G + r % G, last = p.pos0 + tok;      // last key that this row sees
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, tS = taddr + lanes + u * 128, tO = taddr + lanes + 256 + u * 128;
    const int first_masked = (p.pos0 + tok_first + u * TOK + 1) >> 7;       // tiles from here on hold keys that some row does not see
    float m = 0.0f, l = 0.0f;
    for (int j = 0; j < n; ++j) {
      if (!__all_sync(0xffffffffu, tc::mbar_wait(&s_full[u], j & 1))) { failed = true; break; }
      tc::tc_fence_after();
      float s[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tc::tmem_ld32(tS + c * 32, reinterpret_cast<uint32_t*>(s) + c * 32);
      tc::tmem_wait_ld();
      if (j >= first_masked) {
        const int seen = last - j * 128;
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (c > seen) s[c] = -INFINITY;
      }
      float x[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int c = 4; c < 128; c += 4)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = fmaxf(x[e], s[c + e]);
      const float top = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
      if (j == 0) {
        m = top == -INFINITY ? 0.0f : top;
      } else if (__any_sync(0xffffffffu, top > m + 8.0f)) {
        const float to = fmaxf(m, top), f = at_ex2(m - to);
        m = to;
        l *= f;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tc::tmem_ld32(tO + c * 32, o);
          tc::tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
          at_st32(tO + c * 32, o);
        }
      }
      float ls[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t w[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float a = at_ex2(s[c * 64 + 2 * e] - m), b = at_ex2(s[c * 64 + 2 * e + 1] - m);
          ls[(2 * e) & 3] += a;
          ls[(2 * e + 1) & 3] += b;
          const __half2 h = __floats2half2_rn(a, b);
          w[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        at_st32(tS + c * 32, w);
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      at_wait_st();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&p_ready[u]);
    }
    if (!failed && n > 0 && !tc::mbar_wait_warp<0>(&o_full[u], 0, lane)) failed = true;
    if (failed && lane == 0 && p.status != nullptr) atomicExch(p.status, kAtStalled);
    tc::tc_fence_after();
    if (tok_first + u * TOK < p.T) {
      const float inv = failed ? __int_as_float(0x7FFFFFFF) : (l > 0.0f ? 1.0f / l : 0.0f);      // an expired wait: NaN, not numbers
      __half* dst = p.out + (size_t)tok * p.out_ld + head * 128;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        float o[32];
        tc::tmem_ld32(tO + c * 32, reinterpret_cast<uint32_t*>(o));
        tc::tmem_wait_ld();
        if (tok < p.T) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {      // paired-K order: inputs k and k + 4 of every eight side by side
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __half2 h = __floats2half2_rn(o[e + i] * inv, o[e + i + 4] * inv);
              w[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(dst + c * 32 + e) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (warp == 9) tc::tmem_dealloc(taddr, 512);
}

// INT8 / INT4 rows of one sequence and layer as f16 [kv head][n_pad][128], keys then values; rows from n on are zero.  A thread makes eight values.
__global__ void __launch_bounds__(256) kv_to_f16_kernel(const uint8_t* __restrict__ kpool, const uint8_t* __restrict__ vpool, const float* __restrict__ ks,
                                                        const float* __restrict__ vs, const int* __restrict__ bt, int n, int n_pad, int nkv, int page,
                                                        int int4_rows, uint4* __restrict__ out) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const size_t half = (size_t)nkv * n_pad * 16;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < 2 * half; i += (size_t)gridDim.x * blockDim.x) {
    const bool v = i >= half;
    const size_t j = v ? i - half : i;
    const int c = (int)(j & 15), key = (int)((j >> 4) % n_pad), kvh = (int)((j >> 4) / n_pad);
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (key < n) {
      const size_t row = ((size_t)bt[key / page] * nkv + kvh) * page + key % page;
      const float s = (v ? vs : ks)[row];
      const uint8_t* pool = v ? vpool : kpool;
      float x[8];
      if (int4_rows) {
        const uint32_t q = *reinterpret_cast<const uint32_t*>(pool + row * 64 + c * 4);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = s * (float)((int)((q >> (4 * e)) & 15u) - 8);
      } else {
        const uint2 q = *reinterpret_cast<const uint2*>(pool + row * 128 + c * 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = s * (float)(int8_t)((e < 4 ? q.x : q.y) >> (8 * (e & 3)));
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __half2 h = __floats2half2_rn(x[2 * e], x[2 * e + 1]);
        w[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    out[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

static bool at_map(CUtensorMap* map, const void* base, uint64_t rows) {
  cuuint64_t dims[2] = {128, (cuuint64_t)rows}, strides[1] = {256};
  cuuint32_t box[2] = {64, 64}, estr[2] = {1, 1};
  return cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int G>
static int at_launch(const CUtensorMap& kmap, const CUtensorMap& vmap, const AtParams& p, cudaStream_t st) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BONSAI_CUDA_LAUNCH_FAILED;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(attn_prefill_tc_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAtSmem) != cudaSuccess) return BONSAI_CUDA_LAUNCH_FAILED;
    configured[dev] = true;
  }
  const int per = 2 * 128 / G;
  const cudaError_t e = launch_pdl(attn_prefill_tc_kernel<G>, dim3(p.nkv, (p.T + per - 1) / per), dim3(kAtThreads), kAtSmem, st, kmap, vmap, p);
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

// Measured, 32 / 8 heads (before, on mma.sync): a prompt of 4096 147 us, 937 TFLOP/s (1034); of 777 19.9 us (78.9), INT8 pages 22.9 with
// their decoding (107.6); 512 tokens behind 8000 127 us (744); 333 behind 1000 28.3 us (121); 64 10.4 us (10.0).  Error against 64 bits
// 3.2e-4 in both kernels.
//
// Arguments as bonsai_attn_prefill_order (k_order 0).  f16 pages of a multiple of 64 tokens are read in place; INT8 / INT4 pages are
// decoded into scratch (f16 elements, 16-byte aligned), 2 * nkv * 128 per key.  Anything else: BAD_ARG, the caller has another kernel.
int attn_prefill_tc(const float* q, int T, int pos0, const int* bt, int nq, int nkv, int hd, int kvt, int page, const void* kpool, const void* vpool,
                    const float* kscale, const float* vscale, void* out, int out_ld, void* scratch, size_t scratch_elems, int* status, cudaStream_t st) {
  const int G = nkv > 0 && nq % nkv == 0 ? nq / nkv : 0, n = pos0 + T, n_pad = (n + 127) / 128 * 128;
  if (hd != 128 || (G != 1 && G != 2 && G != 4 && G != 8) || out_ld % 8 != 0) return BONSAI_CUDA_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(kpool) | reinterpret_cast<uintptr_t>(vpool)) & 15) != 0)
    return BONSAI_CUDA_BAD_ARG;
  AtParams p{q, bt, (__half*)out, status, T, pos0, nq, nkv, page, kvt == 1 ? 1 : 0, n_pad, out_ld, 1.4426950408889634f / sqrtf((float)hd)};
  CUtensorMap kmap, vmap;
  if (kvt == 1) {
    if (page % 64 != 0 || !at_map(&kmap, kpool, 0x7FFFFFFFu) || !at_map(&vmap, vpool, 0x7FFFFFFFu)) return BONSAI_CUDA_BAD_ARG;
  } else if (kvt == 2 || kvt == 3) {
    const size_t need = (size_t)nkv * n_pad * 128;
    if (scratch == nullptr || (reinterpret_cast<uintptr_t>(scratch) & 15) != 0 || scratch_elems < 2 * need) return BONSAI_CUDA_BAD_ARG;
    if (!at_map(&kmap, scratch, (uint64_t)nkv * n_pad) || !at_map(&vmap, static_cast<__half*>(scratch) + need, (uint64_t)nkv * n_pad)) return BONSAI_CUDA_BAD_ARG;
    const size_t blocks = (need / 4 + 255) / 256;
    const cudaError_t e = launch_pdl(kv_to_f16_kernel, dim3((unsigned)(blocks < 148 * 16 ? blocks : 148 * 16)), dim3(256), 0, st, (const uint8_t*)kpool,
                                     (const uint8_t*)vpool, kscale, vscale, bt, n, n_pad, nkv, page, kvt == 3 ? 1 : 0, (uint4*)scratch);
    if (e != cudaSuccess) return BONSAI_CUDA_LAUNCH_FAILED;
  } else {
    return BONSAI_CUDA_BAD_ARG;
  }
  if (G == 1) return at_launch<1>(kmap, vmap, p, st);
  if (G == 2) return at_launch<2>(kmap, vmap, p, st);
  if (G == 4) return at_launch<4>(kmap, vmap, p, st);
  return at_launch<8>(kmap, vmap, p, st);
}

}  // namespace bonsai
