// Split-KV decode attention for head_dim 128 over INT8 and INT4 pages on the warp-level tensor cores, queries and probabilities as two f16
// terms each (22 bits).
//
// A warp handles 16 tokens of one kv head at a time:
//   * codes are exact in f16; a pair of them comes out of a packed word with a byte or nibble shuffle under an exponent and one exact HADD2;
//   * a query and a probability are two f16 terms, x = hi + lo (22 bits): the group's heads are rows 0..G-1 of the first operand as hi
//     and rows 8..8+G-1 as lo, rows that the instruction computes anyway, and the two sums meet in one lane;
//   * a head's queries are scaled by a power of two to [2^7, 2^8), its probabilities times their rows' scales, tile by tile, to [2^14, 2^15):
//     neither leaves the range in which the two terms hold 22 bits;
//   * the dimensions and tokens of a tile may come in any order as long as both operands agree, so that every lane reads whole 16-byte
//     words of the rows.
// Scores, maxima, sums and accumulators are f32.  The error against 64 bits is no larger than that of the CUDA-core kernel's f32 products for
// unit-normal queries and rows (one to 64 sequences of 16 to 20001 tokens: INT8 1.66e-7 and 1.78e-7, INT4 1.52e-7 and 1.71e-7); over INT8
// rows and queries twice as large 2.9e-7 and 2.7e-7.
//
// Work: the tiles of all (sequence, kv head) pairs stand in one line, which is cut into equal pieces, one per CTA, whatever the
// lengths are.  A pair that lies in one piece is finished there; of any other each CTA leaves a partial sum (a CTA has two at most, of
// its first and of its last pair), and the last one to do so merges them.  The lengths are read on the device, so that a
// captured launch serves every step.  The cuts follow from the lengths of all sequences of the launch: the last bits of a sequence's result depend on
// its neighbours' lengths, as they do on their number (the CUDA-core kernel's splits: on the number alone).  Rows come through a ring of three tiles per warp in shared memory (cp.async), two ahead and across the
// pairs, which leaves registers for three warps per scheduler.
// What bounds it: not the rows (a warp waits 20 cycles for its next tile) but its instructions, some 400 per tile of 16 tokens in 2100 cycles with
// three warps in turn; turning to another pair 3000 to 4000 cycles, and merging parts 5 to 7 us at the end, a chain of launch-cold code and L2 trips.
// 32 / 8 heads, us (one CTA per split, sequence and kv head, tiles in registers / now): 64 sequences of 128 to 2048 tokens, INT8 67 / 42 (3.5 TB/s), 24 of 100 to
// 1500, INT4 31 / 22, one of 20001 22.4 / 20.7, one of 300 9.2 / 6.2.
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"

namespace bonsai {

constexpr int kQaStages = 3, kQaSmWarps = 12;
constexpr int qa_ctas(int warps) { return 148 * kQaSmWarps / warps; }      // that the device holds, by warps of a CTA

// mode: see attn_decode_quant (words of their own made the parameters larger, and the compiler spilled: 20001 tokens 472 -> 482 us a step)
enum { kQaOlder = 1, kQaAlone = 2, kQaClose = 4 };
struct QaParams {
  const float* q;            // [batch][nq][128]
  const int* positions;
  const int* block_table;    // [batch][max_pages]
  const uint8_t* k;          // codes: rows of 128 bytes (INT8) or 64 (INT4)
  const uint8_t* v;
  const float* k_scale;
  const float* v_scale;
  float* ws_acc;             // [CTA][2][G][128]: partial sums of a CTA's first and last pair; close: [CTA + pair][G][128]
  float* ws_ml;              // [..][G][2]
  int* counters;             // [batch][nkv], zero between launches
  float* out;                // [batch][nq][128]
  int batch, max_pages, nq, nkv, page_size, extra_len, ctas, mode;
  float sm_scale;
};

// d = a b, from zero
__device__ __forceinline__ void qa_mma(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void qa_mma_add(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two f32 in one instruction, each rounded as alone
__device__ __forceinline__ float2 qa_add2(float2 x, float2 y) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
  return r;
}
__device__ __forceinline__ float2 qa_fma2(float2 x, float2 y, float2 z) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y));
  return r;
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
__device__ __forceinline__ float qa_inverse(float pow2) { return __uint_as_float(0x7F000000u - __float_as_uint(pow2)); }      // of 2^-126 .. 2^126
__device__ __forceinline__ float qa_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kQaNone = -3.0e38f;      // below every score: the maximum over no tokens, from which differences stay defined

__device__ __forceinline__ void qa_copy16(uint32_t dst, const void* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void qa_copy4(uint32_t dst, const void* src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(real ? 4 : 0) : "memory");
}

// TIGHT: a workspace with less room than two partial sums a CTA (the two cases cost the others up to 3 % in spilled registers)
template <int KVT, int G, int NW, bool TIGHT>
__global__ void __launch_bounds__(NW * 32, kQaSmWarps / NW) attn_decode_quant_kernel(QaParams p) {
  constexpr int hd = 128, RB = KVT == 2 ? 128 : 64, KW = KVT == 2 ? 2 : 1;
  constexpr int kTile = 32 * RB + 128, kChunks = RB / 16;       // a tile: 16 rows of keys, 16 of values, 32 scales
  constexpr int stride = hd + 2;
  constexpr int kAhead = NW + NW / 2;                           // tiles' time that turning to a pair costs: it stands in the line before the pair's tiles
  extern __shared__ __align__(128) uint8_t qa_smem[];
  float* qa_sh = reinterpret_cast<float*>(qa_smem + NW * kQaStages * kTile);      // [warp][G][hd + 2]
  int* ends = reinterpret_cast<int*>(qa_sh + NW * G * stride);                    // tiles of the sequences before b and of b, of one kv head
  int* lens = ends + p.batch;
  __shared__ int s_last[2], s_first;
  const int cta = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, row = lane >> 2, c = lane & 3;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (cta >= p.ctas) return;
  // Where positions and page lists are older than the kernel ahead (a model's step: it appends rows and queries), the line is laid out before that
  // has ended.  A sequence without keys has one empty tile, which writes its zeros.
  if (!(p.mode & kQaOlder)) asm volatile("griddepcontrol.wait;" ::: "memory");
  if (warp == 0) {
    int sum = 0, most = 0;
    for (int b0 = 0; b0 < p.batch; b0 += 32) {
      const int b = b0 + lane, len = b < p.batch ? p.positions[b] + 1 + p.extra_len : 0;
      int n = b < p.batch ? max(1, (len + 15) >> 4) : 0;
      most = max(most, n);
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const int x = __shfl_up_sync(0xffffffffu, n, o);
        if (lane >= o) n += x;
      }
      if (b < p.batch) {
        ends[b] = sum + n;
        lens[b] = len;
      }
      sum += __shfl_sync(0xffffffffu, n, 31);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0) s_first = most;
  }
  __syncthreads();
  const int total = (ends[p.batch - 1] + kAhead * p.batch) * p.nkv;
  // Places of the line that a CTA takes: at least a pair's start and a tile, and so many that no pair has more than 65 parts for each warp of the CTA
  // that adds them up, one after the other (one kv head, 149 sequences of 60 tokens and one of 9000, in CTAs of two warps: 33.4 us over INT8 rows
  // in 94 parts, 40.8 in 141).  Where no pair has more than four tiles for each warp of a CTA and every pair has its CTA, each gets a whole one:
  // merging parts takes as long as four tiles (one sequence of 300 tokens 11.3 us cut, 6.6 whole).
  constexpr int kParts = 65 * NW;
  const bool whole = (TIGHT && (p.mode & kQaAlone)) || (s_first <= 4 * NW && p.batch * p.nkv <= p.ctas);
  const int per = whole ? 1 << 30 : (max((total + p.ctas - 1) / p.ctas, max(kAhead + 1, (s_first + kParts - 3) / (kParts - 2))) + NW - 1) / NW * NW;
  const int begin = whole ? 0 : cta * per;
  int end = min(total, begin + per);
  if (whole ? cta >= p.batch * p.nkv : begin >= end) return;
  __syncthreads();
  auto start_of = [&](int b) { return ((b == 0 ? 0 : ends[b - 1]) + kAhead * b) * p.nkv; };
  for (int b = t; b < p.batch; b += NW * 32)
    if (begin >= start_of(b) && (b + 1 == p.batch || begin < start_of(b + 1))) s_first = b;
  __syncthreads();
  const int pshift = 31 - __clz(p.page_size), pmask = p.page_size - 1;

  // a run of tiles of one pair: j0 .. j1 - 1 of sequence b, kv head h; the pair's first tile has place `at` of the line
  struct Run { int b, h, n, at, j0, j1; };
  auto first_run = [&] {
    Run r;
    if (whole) {
      r.b = cta / p.nkv;
      r.h = cta - r.b * p.nkv;
      r.n = ends[r.b] - (r.b == 0 ? 0 : ends[r.b - 1]);
      r.at = start_of(r.b) + r.h * (r.n + kAhead) + kAhead;
      r.j0 = 0;
      r.j1 = r.n;
      return r;
    }
    r.b = s_first;
    r.n = ends[r.b] - (r.b == 0 ? 0 : ends[r.b - 1]);
    const int off = begin - start_of(r.b);
    r.h = off / (r.n + kAhead);
    r.at = start_of(r.b) + r.h * (r.n + kAhead) + kAhead;
    r.j0 = max(0, begin - r.at);
    r.j1 = min(r.n, end - r.at);
    return r;
  };
  auto next_run = [&](Run& r) {             // false: the CTA's piece ends here
    r.at += r.n + kAhead;
    if (r.at >= end) return false;
    if (++r.h == p.nkv) {
      r.h = 0;
      ++r.b;
      r.n = ends[r.b] - ends[r.b - 1];
    }
    r.j0 = 0;
    r.j1 = min(r.n, end - r.at);
    return true;
  };

  // ---- copies: the warp's tiles in the order in which they are used ------------------------------------------------------------------------------
  // The sixteen rows of a tile are one range of memory; a lane copies every 32nd 16-byte chunk.  Chunks change places within their row so that
  // the reads below meet no bank twice: keys chunk ^ 4 in odd rows (INT8), values chunk ^ (token & 6) (INT8) or ^ (token / 2 & 3) (INT4).
  constexpr int kCopies = 16 * kChunks / 32;
  const int ctok = lane / kChunks, cch = lane % kChunks;
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(qa_smem + warp * kQaStages * kTile);
  const uint32_t kdst = ring_at + ctok * RB + (KVT == 2 ? cch ^ ((ctok & 1) << 2) : cch) * 16;
  const uint32_t vdst = ring_at + (16 + ctok) * RB + (KVT == 2 ? cch ^ (ctok & 2) : cch ^ ((ctok >> 1) & 3)) * 16;      // INT8: rows 4 .. 7 of eight one bit further
  Run cr = first_run();
  if (whole) end = cr.at + cr.n;
  int cj = cr.j0 + warp, cstage = 0, window = -1, pages = 0;      // lane i: page `window + i` of the sequence
  bool more = true;
  auto settle = [&] {                       // moves on to the warp's next tile, and asks for its page
    while (more && cj >= cr.j1) {
      more = next_run(cr);
      cj = cr.j0 + warp;
      window = -1;
    }
    if (!more) return;
    const int page = (cj * 16) >> pshift;
    if (window < 0 || page >= window + 32) {
      window = page;
      const int last = (max(lens[cr.b], 1) - 1) >> pshift;
      pages = lens[cr.b] > 0 ? __ldg(p.block_table + (size_t)cr.b * p.max_pages + min(window + lane, last)) : 0;
    }
  };
  auto copy = [&] {
    if (more) {
      const int tb = cj * 16, left = lens[cr.b] - tb;      // rows behind the last token are not read
      const int page = __shfl_sync(0xffffffffu, pages, (tb >> pshift) - window);
      const size_t base = ((size_t)page * p.nkv + cr.h) * p.page_size + (tb & pmask);
      const uint8_t *ks = p.k + base * RB + lane * 16, *vs = p.v + base * RB + lane * 16;
      const uint32_t at = cstage * kTile;
      const float* sc = lane < 16 ? p.k_scale : p.v_scale;
      const uint32_t kd = kdst + at, vd = vdst + at, vd2 = KVT == 2 ? vd ^ 64 : vd;
      if (left >= 16) {
#pragma unroll
        for (int i = 0; i < kCopies; ++i) {
          qa_copy16(kd + i * 512, ks + i * 512, true);
          qa_copy16((i & 1 ? vd2 : vd) + i * 512, vs + i * 512, true);
        }
        qa_copy4(ring_at + at + 32 * RB + lane * 4, sc + base + (lane & 15), true);
      } else {
#pragma unroll
        for (int i = 0; i < kCopies; ++i) {
          const bool real = ctok + i * (32 / kChunks) < left;
          qa_copy16(kd + i * 512, real ? ks + i * 512 : p.k, real);
          qa_copy16((i & 1 ? vd2 : vd) + i * 512, real ? vs + i * 512 : p.v, real);
        }
        const bool real = (lane & 15) < left;
        qa_copy4(ring_at + at + 32 * RB + lane * 4, real ? sc + base + (lane & 15) : sc, real);
      }
      cj += NW;
      settle();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++cstage == kQaStages) cstage = 0;
  };
  settle();
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // the queries of a pair, as they are: four dimensions for every MMA and c
  float qx[8][4];
  auto load_queries = [&](const Run& r) {
    const float* qp = p.q + ((size_t)r.b * p.nq + r.h * G + (row < G ? row : 0)) * hd;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      // eight dimensions: INT8 codes 4i .. 4i + 7 of the chunk; INT4 word i / 2, whose half2 number e holds nibbles e and e + 4
      const int d = KVT == 2 ? (i >> 2) * 64 + 16 * c + 4 * (i & 3) : 32 * c + 4 * i;
      const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float4 lo = row < G ? __ldcg(reinterpret_cast<const float4*>(qp + d)) : z, hi = row < G ? __ldcg(reinterpret_cast<const float4*>(qp + d + 4)) : z;
      const float t[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) qx[i + (e >> 2)][e & 3] = t[KVT == 2 ? e : (e >> 1) + 4 * (e & 1)];
    }
  };
  Run run = first_run();
  __shared__ Run s_open[2];                  // the pairs of which this CTA has left a partial sum, its first and its last
  if (t < 2) s_open[t].b = -1;
  load_queries(run);
  copy();
  copy();

  int stage = 0, turn = 0;
  bool merging = false;                      // a pair's parts are added up instead of its tiles
  for (;;) {
    const int cta0 = run.at / per, parts = (run.at + run.n - 1) / per - cta0 + 1;
    // a CTA's first pair has its first partial sum, any other pair that it does not finish is its last
    // (close: along the line a part has a later CTA or a later pair than the one before it)
    auto slot = [&](int i) { return (TIGHT && (p.mode & kQaClose) ? i + run.b * p.nkv + run.h : 2 * i + (run.at - kAhead > i * per ? 1 : 0)) * G; };
    float2 o[16];            // dimensions 32 c + i and 32 c + 16 + i of head `row`
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i] = make_float2(0.0f, 0.0f);
    float m = kQaNone, l = 0.0f;

    if (!merging) {
      const int len = lens[run.b];
      // ---- queries: MMA i takes, for every c, four dimensions: the codes 4i .. 4i + 3 of a lane's chunk (INT8), nibbles of word i / 2 (INT4) --------
      uint32_t qa[8][4];
      float q_back;                              // takes the power of two off the scores again
      {
        float top = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            qx[i][e] *= p.sm_scale;              // times log2 e: scores are exponents of two
            top = fmaxf(top, fabsf(qx[i][e]));
          }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        q_back = top > 1e-30f && top < INFINITY ? qa_pow2(top) * 0.0078125f : 1.0f;
        const float up = qa_inverse(q_back);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          qa_split(qx[i][0] * up, qx[i][1] * up, qa[i][0], qa[i][1]);
          qa_split(qx[i][2] * up, qx[i][3] * up, qa[i][2], qa[i][3]);
        }
      }
      for (int j = run.j0 + warp; j < run.j1; j += NW) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        copy();
        const uint8_t* tile = qa_smem + (warp * kQaStages + stage) * kTile;
        const int left = len - j * 16;
        if (++stage == kQaStages) stage = 0;
        // ---- S = Q K^T -----------------------------------------------------------------------------------------------------------------
        float s[2][2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          // INT4: two chains, whose sums of 11-bit times 4-bit products hardly round.  INT8: every product in a sum of its own, added up in f32: the
          // tensor core cuts a running sum off where f32 rounds it (1.80 -> 1.66e-7 over unit queries, f32 1.78e-7; 64 sequences 62.6 -> 64.2 us).
          constexpr int CH = KVT == 2 ? 8 : 2;
          float acc[CH][4];
#pragma unroll
          for (int h = 0; h < KW; ++h) {
            // INT8: chunks c and c + 4 of the row, at places that odd rows swap;  INT4: chunk c
            const uint4 kw = *reinterpret_cast<const uint4*>(tile + (8 * n + row) * RB + (KVT == 2 ? ((c + 4 * h) ^ ((row & 1) << 2)) : c) * 16);
            const uint32_t w[4] = {kw.x, kw.y, kw.z, kw.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (KVT == 2) {
                const uint32_t x = w[i] ^ 0x80808080u;      // 1024 + code + 128 in a half
                qa_mma(acc[h * 4 + i], qa[h * 4 + i], qa_sub(__byte_perm(x, 0x64646464u, 0x4140), 0x64806480u), qa_sub(__byte_perm(x, 0x64646464u, 0x4342), 0x64806480u));
              } else {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const uint32_t x = w[i] >> (8 * u);       // 1024 + nibble
  const uint32_t b0 = qa_sub((x & 0x000F000Fu) | 0x64006400u, 0x64086408u), b1 = qa_sub(((x >> 4) & 0x000F000Fu) | 0x64006400u, 0x64086408u);
                  if (i == 0) qa_mma(acc[u], qa[i * 2 + u], b0, b1);
                  else qa_mma_add(acc[u], qa[i * 2 + u], b0, b1);
                }
              }
            }
          }
          float2 sum[CH][2];
#pragma unroll
          for (int i = 0; i < CH; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) sum[i][e] = make_float2(acc[i][2 * e], acc[i][2 * e + 1]);
#pragma unroll
          for (int step = 1; step < CH; step *= 2)
#pragma unroll
            for (int i = 0; i < CH; i += 2 * step)
#pragma unroll
              for (int e = 0; e < 2; ++e) sum[i][e] = qa_add2(sum[i][e], sum[i + step][e]);
          const float2 hl = qa_add2(sum[0][0], sum[0][1]);
          s[n][0] = hl.x;
          s[n][1] = hl.y;
        }
        // ---- softmax; the scales of tokens 8 n + 2c + e ----------------------------------------------------------------------------------------
        const float* tile_scale = reinterpret_cast<const float*>(tile + 32 * RB) + 2 * c;      // 16 of the keys, 16 of the values
        const float2 ks2[2] = {*reinterpret_cast<const float2*>(tile_scale), *reinterpret_cast<const float2*>(tile_scale + 8)};
        const float2 vs2[2] = {*reinterpret_cast<const float2*>(tile_scale + 16), *reinterpret_cast<const float2*>(tile_scale + 24)};
        float pr[2][2], mx = m;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            pr[n][e] = 8 * n + 2 * c + e < left ? s[n][e] * ((e ? ks2[n].y : ks2[n].x) * q_back) : -INFINITY;
            mx = fmaxf(mx, pr[n][e]);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float down = qa_exp2(m - mx);
        float ps = 0.0f, x[2][2], top = 0.0f;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float pe = qa_exp2(pr[n][e] - mx);
            ps += pe;
            x[n][e] = pe * (e ? vs2[n].y : vs2[n].x);
            top = fmaxf(top, x[n][e]);
          }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        // the head's largest weight of the tile comes to [2^14, 2^15); weights below 2^-110 lose digits
        const float unit = top < INFINITY ? qa_pow2(fmaxf(top, 7.8e-34f)) * (1.0f / 16384.0f) : 1.0f, up = qa_inverse(unit);
        uint32_t pa[4];
#pragma unroll
        for (int n = 0; n < 2; ++n) qa_split(x[n][0] * up, x[n][1] * up, pa[2 * n], pa[2 * n + 1]);
        l = l * down + ps;
        m = mx;
        if (__any_sync(0xffffffffu, down != 1.0f)) {       // a new maximum: rare behind the first tiles
          const float2 d2 = make_float2(down, down);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            o[i].x *= d2.x;
            o[i].y *= d2.y;
          }
        }
        // a tile's product starts from zero (the tensor core would truncate a long running sum); its hi and lo rows are in one lane
        const float2 unit2 = make_float2(unit, unit);
        auto add = [&](int i, uint32_t b0, uint32_t b1) {
          float t[4];
          qa_mma(t, pa, b0, b1);
          o[i] = qa_fma2(qa_add2(make_float2(t[0], t[1]), make_float2(t[2], t[3])), unit2, o[i]);
        };
        // ---- O += P V: MMA i has, in column `row`, dimension 16 row + i -------------------------------------------------------------------------------
        {
          uint4 vw[4];           // tokens 2c, 2c + 1, 8 + 2c, 9 + 2c, dimensions 16 row ..
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int tok = (i >> 1) * 8 + 2 * c + (i & 1);
            const uint8_t* vr = tile + (16 + tok) * RB;
            if (KVT == 2) {
              vw[i] = *reinterpret_cast<const uint4*>(vr + ((row ^ (2 * c)) << 4));
            } else {
              const uint2 w2 = *reinterpret_cast<const uint2*>(vr + (((row >> 1) ^ c) << 4) + (row & 1) * 8);
              vw[i] = make_uint4(w2.x, w2.y, 0u, 0u);
            }
          }
#pragma unroll
          for (int wd = 0; wd < (KVT == 2 ? 4 : 2); ++wd) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = wd == 0 ? vw[i].x : (wd == 1 ? vw[i].y : (wd == 2 ? vw[i].z : vw[i].w));
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
        __syncwarp();
      }
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
    } else if (row < G) {
#pragma unroll 1
      for (int i = warp; i < parts; i += NW) {
        const size_t from = slot(cta0 + i) + row;
        const float4* src = reinterpret_cast<const float4*>(p.ws_acc + from * hd + 32 * c);
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.ws_ml) + from);
        float4 x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = __ldcg(src + k);
        const float mx = fmaxf(m, ml.x), down = qa_exp2(m - mx), f = qa_exp2(ml.x - mx);
        m = mx;
        l = l * down + f * ml.y;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float* lo = reinterpret_cast<const float*>(&x[k >> 2]), *hi = reinterpret_cast<const float*>(&x[4 + (k >> 2)]);
          o[k] = make_float2(fmaf(f, lo[k & 3], o[k].x * down), fmaf(f, hi[k & 3], o[k].y * down));
        }
      }
    }

    // ---- the CTA's warps, then the pieces ----------------------------------------------------------------------------------------------------------
    if (row < G) {
      float* dst = qa_sh + ((size_t)warp * G + row) * stride;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        dst[32 * c + i] = o[i].x;
        dst[32 * c + 16 + i] = o[i].y;
      }
      if (c == 0) {
        dst[hd] = m;
        dst[hd + 1] = l;
      }
    }
    __syncthreads();
    const size_t head0 = (size_t)run.b * p.nq + run.h * G;
    constexpr int kQuads = G * hd / 4;
    for (int idx = t; idx < kQuads; idx += NW * 32) {
      const int g = idx / (hd / 4), d = idx % (hd / 4) * 4;
      const float* src = qa_sh + g * stride;
      float M = src[hd];
#pragma unroll
      for (int w = 1; w < NW; ++w) M = fmaxf(M, src[w * G * stride + hd]);
      float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float L = 0.0f;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float2 x0 = *reinterpret_cast<const float2*>(src + w * G * stride + d), x1 = *reinterpret_cast<const float2*>(src + w * G * stride + d + 2);
        const float2 ml = *reinterpret_cast<const float2*>(src + w * G * stride + hd);
        const float f = qa_exp2(ml.x - M);
        a.x += f * x0.x; a.y += f * x0.y; a.z += f * x1.x; a.w += f * x1.y;
        L += f * ml.y;
      }
      if (merging || parts == 1) {
        *reinterpret_cast<float4*>(p.out + (head0 + g) * hd + d) =
            L > 0.0f ? make_float4(a.x / L, a.y / L, a.z / L, a.w / L) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      } else {
        __stcg(reinterpret_cast<float4*>(p.ws_acc + (size_t)(slot(cta) + g) * hd + d), a);
        if (d == 0) __stcg(reinterpret_cast<float2*>(p.ws_ml) + slot(cta) + g, make_float2(M, L));
      }
    }
    if (!merging) {
      if (parts > 1 && t == 0) s_open[run.at - kAhead > cta * per ? 1 : 0] = run;
      if (next_run(run)) {
        load_queries(run);
        __syncthreads();         // the sums have been read
        continue;
      }
      // Pairs in several pieces: whoever leaves the last part adds up all, the warps taking turns in the order of the line, and goes the way of any run.
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (s_open[0].b < 0 && s_open[1].b < 0) break;
      if (t < 2) {
        const Run at = s_open[t];
        int is_last = 0;
        if (at.b >= 0) {
          int* ctr = p.counters + (size_t)at.b * p.nkv + at.h;
          int before;
          asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(before) : "l"(ctr) : "memory");
          is_last = before == (at.at + at.n - 1) / per - at.at / per;
          if (is_last) *ctr = 0;
        }
        s_last[t] = is_last;
      }
      merging = true;
    }
    __syncthreads();
    while (turn < 2 && !s_last[turn]) ++turn;
    if (turn == 2) break;
    run = s_open[turn++];
  }
}

template <int KVT, int G, int NW, bool TIGHT = false>
static int qa_launch(const QaParams& p, dim3 grid, cudaStream_t st) {
  static std::atomic<bool> configured[64];
  const size_t smem = (size_t)NW * kQaStages * (32 * (KVT == 2 ? 128 : 64) + 128) + (size_t)NW * G * 130 * sizeof(float) + (size_t)p.batch * 2 * sizeof(int);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BONSAI_CUDA_LAUNCH_FAILED;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attn_decode_quant_kernel<KVT, G, NW, TIGHT>, cudaFuncAttributeMaxDynamicSharedMemorySize, NW == 12 ? 226 * 1024 : 113 * 1024) != cudaSuccess) return BONSAI_CUDA_LAUNCH_FAILED;
    configured[dev].store(true, std::memory_order_release);
  }
  return launch_pdl(attn_decode_quant_kernel<KVT, G, NW, TIGHT>, grid, dim3(NW * 32), smem, st, p) == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

// Head size 128, INT8 or INT4 rows: the group sizes, pages and alignments of this kernel.
bool attn_decode_quant_takes(const float* q, int nq, int nkv, int page_size, const void* kpool, const void* vpool) {
  const int G = nq / nkv;
  return (G == 1 || G == 2 || G == 4 || G == 8) && page_size >= 16 && (page_size & (page_size - 1)) == 0 &&
         ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kpool) | reinterpret_cast<uintptr_t>(vpool)) & 15) == 0;
}

// The more warps in a CTA, the more sums meet in shared memory and the fewer parts of a long context are left to merge; the fewer, the less they wait
// for one another at the end of a run.  A CTA has an SM up to four sequences of eight heads, a sixth of one from a pair per SM on.  us over INT8 rows with
// twelve / six / two warps, 32 / 8 heads: one sequence of 300 tokens 6.5 / 8.4 / 8.9, four of up to 530 8.3 / 10.9 / 12.0 (whole pairs), four of 4000
// 19.5 / 18.1 / 26.4, five of 100 to 1377 13.1 / 12.2 / 15.6, one of 20001 22.0 / 22.1 / 44.0; 18 of 100 to 1496 17.9 / 16.6 / 19.2, 24 22.2 / 19.8 / 21.6, 32
// 26.8 / 25.1 / 25.3, 64 44.5 / 37.9 / 37.6: between 19 and 32 sequences six warps would be up to a tenth faster, from there on it is even.
static int qa_warps(int pairs) { return pairs >= 148 ? 2 : (pairs > 36 ? 6 : 12); }
// Splits (grid rows per pair) that give every SM its CTAs: whole ones, a further one where these would leave more than a quarter of the places empty.
int attn_decode_quant_splits(int pairs) {
  const int ctas = qa_ctas(qa_warps(pairs));
  int n = ctas / pairs;
  if (n * pairs * 4 < ctas * 3) ++n;
  return n < 1 ? 1 : n;
}

// kvt 2 (INT8) or 3 (INT4); BAD_ARG for what the caller's other kernels take.  ws_rows: rows of 128 floats in ws_acc (of 2 in ws_ml).  A CTA may leave
// two partial sums of G rows, but n CTAs and m pairs no more than n + m - 1 together: where two places each would leave a third of the CTAs idle they are
// CTAs of twelve warps whose sums stand close, and where these are fewer than the pairs (one split) each pair has its own, whatever the lengths are.
// Fewer CTAs, with two places each, took 61 / 26 / 18 / 15 us for one sequence of 4000 tokens over INT8 rows and 1 / 4 / 8 / 16 splits where it now takes
// 33 / 21 / 16 / 15, 29 / 15 us for four of 1000 and 1 / 4 splits where it takes 12 / 14, 34 for sixteen of 1000 and one split where it takes 14.
// older: positions and block_table were not written by the kernel directly ahead in the stream.
int attn_decode_quant(const float* q, const int* positions, const int* block_table, int max_pages, int batch, int nq, int nkv, int kvt, int page_size,
                      const void* kpool, const void* vpool, const float* kscale, const float* vscale, int nsplit, float* ws_acc, float* ws_ml, long long ws_rows,
                      int* counters, float* out, int extra_len, int older, float sm_scale, cudaStream_t st) {
  if (!attn_decode_quant_takes(q, nq, nkv, page_size, kpool, vpool)) return BONSAI_CUDA_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(ws_acc)) & 15) != 0 || (reinterpret_cast<uintptr_t>(ws_ml) & 7) != 0) return BONSAI_CUDA_BAD_ARG;
  const int G = nq / nkv;
  constexpr int kMost = 1024;              // sequences of a launch: their lengths stand in shared memory
  for (int b0 = 0; b0 < batch; b0 += kMost) {
    const int n = batch - b0 < kMost ? batch - b0 : kMost;
    const long long pairs = (long long)nkv * n, room = ws_rows / G;
    int warps = qa_warps(nkv * n);
    long long most = std::min(pairs * nsplit, (long long)qa_ctas(warps)), ctas = std::min(most, room / 2);
    bool alone = false, close = false;
    if (3 * ctas < 2 * most) {
      warps = 12;
      most = std::min(pairs * nsplit, (long long)qa_ctas(warps));
      ctas = std::min(most, std::max(room / 2, room - pairs + 1));
      alone = ctas < pairs && pairs <= most;
      close = !alone && ctas > room / 2;
      if (alone) ctas = pairs;
    }
    QaParams p{q + (size_t)b0 * nq * 128, positions + b0, block_table + (size_t)b0 * max_pages, (const uint8_t*)kpool, (const uint8_t*)vpool, kscale, vscale,
               ws_acc, ws_ml, counters + (size_t)b0 * nkv, out + (size_t)b0 * nq * 128, n, max_pages, nq, nkv, page_size, extra_len,
               ctas < 1 ? 1 : (int)ctas, (older ? kQaOlder : 0) | (alone ? kQaAlone : 0) | (close ? kQaClose : 0), sm_scale * 1.4426950408889634f};
    const dim3 grid(nkv, nsplit, n);
    int rc;
#define BONSAI_QA_12(k, g) (alone || close ? qa_launch<k, g, 12, true>(p, grid, st) : qa_launch<k, g, 12>(p, grid, st))
#define BONSAI_QA_W(k, g) (warps == 2 ? qa_launch<k, g, 2>(p, grid, st) : (warps == 6 ? qa_launch<k, g, 6>(p, grid, st) : BONSAI_QA_12(k, g)))
#define BONSAI_QA(g) (kvt == 2 ? BONSAI_QA_W(2, g) : BONSAI_QA_W(3, g))
    switch (G) {
      case 1: rc = BONSAI_QA(1); break;
      case 2: rc = BONSAI_QA(2); break;
      case 4: rc = BONSAI_QA(4); break;
      default: rc = BONSAI_QA(8);
    }
#undef BONSAI_QA
#undef BONSAI_QA_W
#undef BONSAI_QA_12
    if (rc != BONSAI_CUDA_OK) return rc;
  }
  return BONSAI_CUDA_OK;
}

}  // namespace bonsai
