// Split-KV decode attention for head_dim 128 over INT8 and INT4 pages on the warp-level tensor cores, queries and probabilities as two f16
// terms each (22 bits).
//
// The CUDA-core kernel (attention_decode.cu) spends some 190 warp instructions per token and kv head on products, shuffles and the
// softmax bookkeeping; at 64 sequences of about 1100 tokens it took 145 us where the rows are 147 MB.  Here a warp handles 16 tokens:
//   * codes are exact in f16; a pair of them comes out of a packed word with a byte or nibble shuffle under an exponent and one exact HADD2;
//   * a query and a probability are two f16 terms, x = hi + lo (22 bits): the group's heads are rows 0..G-1 of the first operand as hi
//     and rows 8..8+G-1 as lo, rows that the instruction computes anyway, and the two sums meet in one lane;
//   * a head's queries are scaled by a power of two to [2^7, 2^8), its probabilities times their rows' scales, tile by tile, to [2^14, 2^15):
//     neither leaves the range in which the two terms hold 22 bits;
//   * the dimensions and tokens of a tile may come in any order as long as both operands agree, so that every lane loads whole 16-byte
//     words of the rows straight into registers, a tile ahead.
// Scores, maxima, sums and accumulators are f32.  The error against 64 bits is no larger than that of the CUDA-core kernel's f32 products for
// unit-normal queries and rows (one to 64 sequences of 16 to 20001 tokens: INT8 1.66e-7 and 1.78e-7, INT4 1.52e-7 and 1.71e-7); over INT8
// rows and queries twice as large 2.9e-7 and 2.7e-7.  32 / 8 heads, before and now: 64 sequences of 128 to 2048 tokens 111 -> 46 us (3.2 TB/s),
// one of 20001 40 -> 22 us, 24 of 100 to 1500 in INT4 38 -> 24 us, one of 300 8.1 -> 9.2 us (its step: launch and merge).  Bound by instructions,
// some 20 per token and kv head, and for few sequences by the chain of one tile.  Work decomposition, workspace and the last CTA's merge
// are those of the other kernels.
#include <cuda_fp16.h>

#include "common.cuh"

namespace bonsai {

struct QaParams {
  const float* q;            // [batch][nq][128]
  const int* positions;
  const int* block_table;    // [batch][max_pages]
  const uint8_t* k;          // codes: rows of 128 bytes (INT8) or 64 (INT4)
  const uint8_t* v;
  const float* k_scale;
  const float* v_scale;
  float* ws_acc;             // [batch][nq][nsplit][128]
  float* ws_ml;              // [batch][nq][nsplit][2]
  int* counters;             // [batch][nkv], zero between launches
  float* out;                // [batch][nq][128]
  int max_pages, nq, nkv, page_size, extra_len;
  float sm_scale;
};

__device__ __forceinline__ void qa_mma(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t qa_sub(uint32_t h, uint32_t less) {      // h - less in halves, exact here
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&h), *reinterpret_cast<const __half2*>(&less));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// x, y as two f16 terms each: hi = {x, y} rounded, lo = what that leaves
__device__ __forceinline__ void qa_split(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// 2^e with e from the exponent of x (x > 0): x / qa_pow2(x) lies in [1, 2)
__device__ __forceinline__ float qa_pow2(float x) { return __uint_as_float(__float_as_uint(x) & 0x7F800000u); }

// KVT 2: INT8, a lane's words of a key row: 16-byte chunks c and c + 4;  KVT 3: INT4, chunk c.
template <int KVT, int G, int NW>
__global__ void __launch_bounds__(NW * 32, NW == 8 ? 1 : 2) attn_decode_quant_kernel(QaParams p) {
  constexpr int hd = 128, RB = KVT == 2 ? 128 : 64, KW = KVT == 2 ? 2 : 1;
  extern __shared__ float qa_sh[];          // [warp][G][hd + 2]
  __shared__ int s_last;
  const int kvh = blockIdx.x, split = blockIdx.y, nsplit = gridDim.y, b = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = lane >> 2, c = lane & 3;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int len = p.positions[b] + 1 + p.extra_len;
  int chunk = (len + nsplit - 1) / nsplit;
  // Tiles of 16 never straddle a split or (page_size is a multiple of 16) a page, and a split has a tile for each of its warps at least;
  // splits that are left without tokens leave (the first one stays: rows over no tokens are zero), and a single part needs no merge.
  chunk = max((chunk + 15) & ~15, NW * 16);
  if (split > 0 && split * chunk >= len) return;
  const int t0 = split * chunk, t1 = min(len, t0 + chunk), ntiles = t1 > t0 ? (t1 - t0 + 15) >> 4 : 0;
  const int* bt = p.block_table + (size_t)b * p.max_pages;
  const int pshift = 31 - __clz(p.page_size), pmask = p.page_size - 1;

  struct Tile {
    uint4 k[2][KW];      // keys: token 8 n + row, chunk c (and c + 4)
    uint4 v[4];          // values: tokens 2c, 2c + 1, 8 + 2c, 9 + 2c, dimensions 16 row .. (INT4: 8 bytes each)
    float s;             // lanes 0-15: key scale of token `lane`, 16-31: value scale
  };
  auto load = [&](Tile& x, int j) {
    const int tb = t0 + j * 16;
    const size_t base = ((size_t)bt[tb >> pshift] * p.nkv + kvh) * p.page_size + (tb & pmask);
    const int left = t1 - tb;                // tokens of the tile; the others' rows are not read
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < KW; ++h)
        x.k[n][h] = 8 * n + row < left ? __ldcg(reinterpret_cast<const uint4*>(p.k + (base + 8 * n + row) * RB) + c + 4 * h) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tok = (i >> 1) * 8 + 2 * c + (i & 1);
      if (KVT == 2) {
        x.v[i] = tok < left ? __ldcg(reinterpret_cast<const uint4*>(p.v + (base + tok) * RB) + row) : make_uint4(0u, 0u, 0u, 0u);
      } else {
        const uint2 w = tok < left ? __ldcg(reinterpret_cast<const uint2*>(p.v + (base + tok) * RB) + row) : make_uint2(0u, 0u);
        x.v[i] = make_uint4(w.x, w.y, 0u, 0u);
      }
    }
    x.s = (lane & 15) < left ? __ldcg((lane < 16 ? p.k_scale : p.v_scale) + base + (lane & 15)) : 0.0f;
  };
  Tile cur;
  if (warp < ntiles) load(cur, warp);

  // ---- queries: MMA i takes, for every c, four dimensions: the codes 4i .. 4i + 3 of a lane's chunk (INT8), nibbles of word i / 2 (INT4) --------
  uint32_t qa[8][4];
  float q_back;                              // takes the power of two off the scores again
  {
    const float* qp = p.q + ((size_t)b * p.nq + kvh * G + (row < G ? row : 0)) * hd;
    float x[8][4], top = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      // eight dimensions: INT8 codes 4i .. 4i + 7 of the chunk; INT4 word i / 2, whose half2 number e holds nibbles e and e + 4
      const int d = KVT == 2 ? (i >> 2) * 64 + 16 * c + 4 * (i & 3) : 32 * c + 4 * i;
      const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float4 lo = row < G ? *reinterpret_cast<const float4*>(qp + d) : z, hi = row < G ? *reinterpret_cast<const float4*>(qp + d + 4) : z;
      const float t[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float y = t[KVT == 2 ? e : (e >> 1) + 4 * (e & 1)] * p.sm_scale;
        x[i + (e >> 2)][e & 3] = y;
        top = fmaxf(top, fabsf(y));
      }
    }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    const float unit = top > 1e-30f && top < INFINITY ? qa_pow2(top) * 0.0078125f : 1.0f;
    const float up = 1.0f / unit;            // a power of two: exact
    q_back = unit;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      qa_split(x[i][0] * up, x[i][1] * up, qa[i][0], qa[i][1]);
      qa_split(x[i][2] * up, x[i][3] * up, qa[i][2], qa[i][3]);
    }
  }
  float o[16][2];          // dimensions 32 c + i and 32 c + 16 + i of head `row`
#pragma unroll
  for (int i = 0; i < 16; ++i) o[i][0] = o[i][1] = 0.0f;
  float m = -INFINITY, l = 0.0f;

  for (int j = warp; j < ntiles; j += NW) {
    Tile nxt;
    if (j + NW < ntiles) load(nxt, j + NW);
    // ---- S = Q K^T -----------------------------------------------------------------------------------------------------------------
    float s[2][2];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      // INT4: two chains, whose sums of 11-bit times 4-bit products hardly round.  INT8: every product in a sum of its own, added up in f32: the
      // tensor core cuts a running sum off where f32 rounds it (1.80 -> 1.66e-7 over unit queries, f32 1.78e-7; 64 sequences 62.6 -> 64.2 us).
      constexpr int CH = KVT == 2 ? 8 : 2;
      float acc[CH][4] = {};
#pragma unroll
      for (int h = 0; h < KW; ++h) {
        const uint32_t w[4] = {cur.k[n][h].x, cur.k[n][h].y, cur.k[n][h].z, cur.k[n][h].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (KVT == 2) {
            const uint32_t x = w[i] ^ 0x80808080u;      // 1024 + code + 128 in a half
            qa_mma(acc[h * 4 + i], qa[h * 4 + i], qa_sub(__byte_perm(x, 0x64646464u, 0x4140), 0x64806480u), qa_sub(__byte_perm(x, 0x64646464u, 0x4342), 0x64806480u));
          } else {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const uint32_t x = w[i] >> (8 * u);       // 1024 + nibble
              qa_mma(acc[u], qa[i * 2 + u], qa_sub((x & 0x000F000Fu) | 0x64006400u, 0x64086408u),
                     qa_sub(((x >> 4) & 0x000F000Fu) | 0x64006400u, 0x64086408u));
            }
          }
        }
      }
#pragma unroll
      for (int step = 1; step < CH; step *= 2)
#pragma unroll
        for (int i = 0; i < CH; i += 2 * step)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][e] += acc[i + step][e];
      s[n][0] = acc[0][0] + acc[0][2];
      s[n][1] = acc[0][1] + acc[0][3];
    }
    // ---- softmax; the scales of tokens 8 n + 2c + e ----------------------------------------------------------------------------------------
    const int tb = t0 + j * 16;
    float pr[2][2], mx = m;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tok = 8 * n + 2 * c + e;
        const float ks = __shfl_sync(0xffffffffu, cur.s, tok);
        pr[n][e] = tb + tok < t1 ? s[n][e] * (ks * q_back) : -INFINITY;
        mx = fmaxf(mx, pr[n][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float down = mx == -INFINITY ? 1.0f : expf(m - mx);
    float ps = 0.0f, x[2][2], top = 0.0f;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float vs = __shfl_sync(0xffffffffu, cur.s, 16 + 8 * n + 2 * c + e);
        const float pe = mx == -INFINITY ? 0.0f : expf(pr[n][e] - mx);
        ps += pe;
        x[n][e] = pe * vs;
        top = fmaxf(top, x[n][e]);
      }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    // the head's largest weight of the tile comes to [2^14, 2^15); weights below 2^-110 lose digits
    const float unit = top < INFINITY ? qa_pow2(fmaxf(top, 7.8e-34f)) * (1.0f / 16384.0f) : 1.0f, up = 1.0f / unit;
    uint32_t pa[4];
#pragma unroll
    for (int n = 0; n < 2; ++n) qa_split(x[n][0] * up, x[n][1] * up, pa[2 * n], pa[2 * n + 1]);
    l = l * down + ps;
    m = mx;
    // a tile's product starts from zero (the tensor core would truncate a long running sum); its hi and lo rows are in one lane
    auto add = [&](int i, uint32_t b0, uint32_t b1) {
      float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      qa_mma(t, pa, b0, b1);
      o[i][0] = fmaf(t[0] + t[2], unit, o[i][0] * down);
      o[i][1] = fmaf(t[1] + t[3], unit, o[i][1] * down);
    };
    // ---- O += P V: MMA i has, in column `row`, dimension 16 row + i -------------------------------------------------------------------------------
    {
#pragma unroll
      for (int wd = 0; wd < (KVT == 2 ? 4 : 2); ++wd) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = wd == 0 ? cur.v[i].x : (wd == 1 ? cur.v[i].y : (wd == 2 ? cur.v[i].z : cur.v[i].w));
        if (KVT == 2) {
#pragma unroll
          for (int i = 0; i < 4; ++i) w[i] ^= 0x80808080u;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            // bytes 2u, 2u + 1 of two tokens: {t, t', t, t'}
            const uint32_t x = __byte_perm(w[0], w[1], u ? 0x7362 : 0x5140), y = __byte_perm(w[2], w[3], u ? 0x7362 : 0x5140);
            add(4 * wd + 2 * u, qa_sub(__byte_perm(x, 0x64646464u, 0x4140), 0x64806480u), qa_sub(__byte_perm(y, 0x64646464u, 0x4140), 0x64806480u));
            add(4 * wd + 2 * u + 1, qa_sub(__byte_perm(x, 0x64646464u, 0x4342), 0x64806480u), qa_sub(__byte_perm(y, 0x64646464u, 0x4342), 0x64806480u));
          }
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t sel = (uint32_t)(u | (u << 4) | ((4 + u) << 8) | ((4 + u) << 12));      // byte u of both tokens
            const uint32_t x = __byte_perm(w[0], w[1], sel), y = __byte_perm(w[2], w[3], sel);
            add(8 * wd + 2 * u, qa_sub((x & 0x000F000Fu) | 0x64006400u, 0x64086408u), qa_sub((y & 0x000F000Fu) | 0x64006400u, 0x64086408u));
            add(8 * wd + 2 * u + 1, qa_sub(((x >> 4) & 0x000F000Fu) | 0x64006400u, 0x64086408u),
                   qa_sub(((y >> 4) & 0x000F000Fu) | 0x64006400u, 0x64086408u));
          }
        }
      }
    }
    cur = nxt;
  }
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  const int parts = max(1, (len + chunk - 1) / chunk);

  // ---- the CTA's warps, then the splits: as in attention_decode.cu ------------------------------------------------------------------------------
  constexpr int stride = hd + 2;
  if (row < G) {
    float* dst = qa_sh + ((size_t)warp * G + row) * stride;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      dst[32 * c + i] = o[i][0];
      dst[32 * c + 16 + i] = o[i][1];
    }
    if (c == 0) {
      dst[hd] = m;
      dst[hd + 1] = l;
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * hd; idx += NW * 32) {
    const int g = idx / hd, d = idx - g * hd;
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; ++w) M = fmaxf(M, qa_sh[((size_t)w * G + g) * stride + hd]);
    float a = 0.0f, L = 0.0f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float* src = qa_sh + ((size_t)w * G + g) * stride;
      const float f = src[hd] == -INFINITY ? 0.0f : expf(src[hd] - M);
      a += f * src[d];
      L += f * src[hd + 1];
    }
    const size_t head = (size_t)b * p.nq + kvh * G + g;
    if (parts == 1) {
      p.out[head * hd + d] = L > 0.0f ? a / L : 0.0f;
    } else {
      p.ws_acc[(head * nsplit + split) * hd + d] = a;
      if (d == 0) *reinterpret_cast<float2*>(p.ws_ml + (head * nsplit + split) * 2) = make_float2(M, L);
    }
  }
  if (parts == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int* ctr = p.counters + (size_t)b * p.nkv + kvh;
    s_last = atomicAdd(ctr, 1) == parts - 1;
    if (s_last) *ctr = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int idx = threadIdx.x; idx < G * hd; idx += NW * 32) {
    const int g = idx / hd, d = idx - g * hd;
    const size_t head = (size_t)b * p.nq + kvh * G + g;
    const float2* ml = reinterpret_cast<const float2*>(p.ws_ml) + head * nsplit;
    const float* ac = p.ws_acc + head * nsplit * hd + d;
    // eight splits per step, all of a step's loads before the first use
    float M = -INFINITY;
    for (int s0 = 0; s0 < parts; s0 += 8) {
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = s0 + i < parts ? __ldcg(ml + s0 + i).x : -INFINITY;
#pragma unroll
      for (int i = 0; i < 8; ++i) M = fmaxf(M, x[i]);
    }
    float a = 0.0f, L = 0.0f;
    for (int s0 = 0; s0 < parts; s0 += 8) {
      float2 x[8];
      float y[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool ok = s0 + i < parts;
        x[i] = ok ? __ldcg(ml + s0 + i) : make_float2(-INFINITY, 0.0f);
        y[i] = ok ? __ldcg(ac + (size_t)(s0 + i) * hd) : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float f = x[i].x == -INFINITY ? 0.0f : expf(x[i].x - M);
        a += f * y[i];
        L += f * x[i].y;
      }
    }
    p.out[head * hd + d] = L > 0.0f ? a / L : 0.0f;
  }
}

template <int KVT, int G>
static int qa_launch(const QaParams& p, int batch, int nsplit, cudaStream_t st) {
  const dim3 grid(p.nkv, nsplit, batch);
  const bool wide = (long long)p.nkv * nsplit * batch <= 148;      // one CTA per SM or fewer: eight warps
  const size_t smem = (size_t)(wide ? 8 : 4) * G * 130 * sizeof(float);
  const cudaError_t e = wide ? launch_pdl(attn_decode_quant_kernel<KVT, G, 8>, grid, dim3(256), smem, st, p)
                             : launch_pdl(attn_decode_quant_kernel<KVT, G, 4>, grid, dim3(128), smem, st, p);
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

// Head size 128, INT8 or INT4 rows: the group sizes, pages and alignments of this kernel.
bool attn_decode_quant_takes(const float* q, int nq, int nkv, int page_size, const void* kpool, const void* vpool) {
  const int G = nq / nkv;
  return (G == 1 || G == 2 || G == 4 || G == 8) && page_size >= 16 && (page_size & (page_size - 1)) == 0 &&
         ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kpool) | reinterpret_cast<uintptr_t>(vpool)) & 15) == 0;
}

// kvt 2 (INT8) or 3 (INT4); BAD_ARG for what the caller's other kernels take.
int attn_decode_quant(const float* q, const int* positions, const int* block_table, int max_pages, int batch, int nq, int nkv, int kvt, int page_size,
                      const void* kpool, const void* vpool, const float* kscale, const float* vscale, int nsplit, float* ws_acc, float* ws_ml, int* counters,
                      float* out, int extra_len, float sm_scale, cudaStream_t st) {
  if (!attn_decode_quant_takes(q, nq, nkv, page_size, kpool, vpool)) return BONSAI_CUDA_BAD_ARG;
  QaParams p{q, positions, block_table, (const uint8_t*)kpool, (const uint8_t*)vpool, kscale, vscale, ws_acc, ws_ml, counters, out,
             max_pages, nq, nkv, page_size, extra_len, sm_scale};
#define BONSAI_QA(g) (kvt == 2 ? qa_launch<2, g>(p, batch, nsplit, st) : qa_launch<3, g>(p, batch, nsplit, st))
  switch (nq / nkv) {
    case 1: return BONSAI_QA(1);
    case 2: return BONSAI_QA(2);
    case 4: return BONSAI_QA(4);
    case 8: return BONSAI_QA(8);
    default: return BONSAI_CUDA_BAD_ARG;
  }
#undef BONSAI_QA
}

}  // namespace bonsai
