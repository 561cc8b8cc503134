// Prompts of models whose layer weights stay in GGUF blocks (Q4_0, Q8_0, K-quants, FP8, dense rows): every launch of a chunk of more than 64 tokens
// from one call, and every launch of one token, which is how a prompt's last token makes its logits.
//
// Per layer: norm -> QKV -> rotation and append -> causal attention -> O + residual -> norm -> gate / up with SwiGLU in the epilogue -> down +
// residual.  A matrix is decoded to f16 into a scratch matrix that stays in L2 and multiplied densely (gemm_pair.cu).  Gate and up rows are interleaved while they are decoded, so that the product's epilogue makes the
// activation; they pass in slabs where the scratch does not hold both.  Matrices that share their input and stand one behind the other are one
// product.  500 tokens of a quarter-depth 4B model in Q8_0: 300 us and 22 launches a layer from Python, 213 us and 14 from here, the same bits.
#include "common.cuh"

extern "C" {
int bonsai_embed_rows_f16(const void*, const int*, float*, int, int, int, cudaStream_t);
int bonsai_norm_to_f16_paired(const float*, int, const float*, float, int, int, void*, int, int, cudaStream_t);
int bonsai_qknorm_rope_kvstore(const float*, int, const float*, const float*, float, const float*, const float*, const int*, const int*, int, float*, int, int,
                               int, int, int, int, void*, void*, float*, float*, cudaStream_t);
int bonsai_attn_prefill_ws(const float*, int, int, const int*, int, int, int, int, int, const void*, const void*, const float*, const float*, void*, int, int,
                           void*, size_t, int*, cudaStream_t);
int bonsai_quant_gemv_batched_status(int, const void*, const float*, int, const float*, float, float*, const float*, int, int, int, int, int*, cudaStream_t);
int bonsai_attn_decode_route(const float*, const int*, const int*, int, int, int, int, int, int, int, const void*, const void*, const float*, const float*, int,
                             float*, float*, long long, int*, float*, int, int, int, cudaStream_t);
int bonsai_swiglu_rows(const float*, int, float*, int, int, int, cudaStream_t);
int bonsai_f16gemv(const void*, const float*, const float*, float, float*, int, int, cudaStream_t);
int bonsai_bitgemm_prefill_ws(const void*, const void*, const void*, int, float*, const float*, void*, int*, int, int, int, int, int, int, const void*, void*,
                              size_t, int, cudaStream_t);
}

namespace bonsai {

// rows of K weights in blocks of `type` as f16 in paired-K order: out row r * mul + add
int quant_rows_to_f16(int type, const void* w, int rows, int K, void* out, int mul, int add, cudaStream_t st);
long long quant_row_bytes(int type, int K);      // -1: not a block type

// one matrix of a layer: block type, rows, bytes
struct BlockMatrix { long long type, rows; const uint8_t* data; };
enum { BM_Q, BM_K, BM_V, BM_O, BM_GATE, BM_UP, BM_DOWN, BM_COUNT };      // rows 0: in the matrix before, behind its own
struct BlockLayer {
  BlockMatrix m[BM_COUNT];
  const float *attn_norm, *ffn_norm, *q_norm, *k_norm;
  void *kpool, *vpool;
  float *kscale, *vscale;
};
struct BlockPrompt {
  const void* embd;
  const float *rope_cos, *rope_sin;
  const int *tokens, *positions, *block_table;      // one page list
  float *h, *qkv, *q;                               // [T][hidden], [T][qkv], [T][heads][head size]
  void *xn, *attn, *act;                            // f16 [T][hidden], [T][heads * head size], [T][inter]
  void* scratch;
  long long scratch_elems;
  void* gemm_ws;
  long long gemm_ws_bytes;
  int* status;
  long long hidden, inter, layers, heads, kv_heads, head_dim, vocab, kvt, page_size;
};

// the buffers of one sequence's step
struct BlockRow {
  const void *embd, *lm_head;
  const float *out_norm, *rope_cos, *rope_sin;
  const int *token, *position, *block_table;
  float *h, *qkv, *q, *attn, *gu, *act, *logits, *ws_acc, *ws_ml;
  int *counters, *status;
  long long ws_rows, hidden, inter, layers, heads, kv_heads, head_dim, vocab, lm_rows, kvt, page_size, nsplit;
};

#define RC(expr) do { int _rc = (expr); if (_rc != 0) return _rc; } while (0)

static int chunk(const BlockPrompt& p, const BlockLayer* layers, float eps, int T, int pos0, cudaStream_t st) {
  const int hidden = (int)p.hidden, inter = (int)p.inter, hd = (int)p.head_dim, nq = (int)p.heads, nkv = (int)p.kv_heads, qd = nq * hd, qkv_n = qd + 2 * nkv * hd;
  const int kvt = (int)p.kvt, page = (int)p.page_size;
  auto dense = [&](const void* x, int rows, int K, float* out, const float* residual, void* out16, int epi, int out_ld) {
    return bonsai_bitgemm_prefill_ws(nullptr, nullptr, x, K, out, residual, out16, p.status, rows, K, T, epi, out_ld, 148, p.scratch, p.gemm_ws,
                                     (size_t)p.gemm_ws_bytes, 1, st);
  };
  auto product = [&](const BlockMatrix& m, const void* x, int K, float* out, const float* residual, int out_ld) -> int {
    const long long row_bytes = quant_row_bytes((int)m.type, K), most = p.scratch_elems / K;
    if (row_bytes < 0 || (m.rows > most && most < 256)) return BONSAI_CUDA_BAD_ARG;
    const int step = (int)(m.rows <= most ? m.rows : most / 256 * 256);
    for (int r0 = 0; r0 < m.rows; r0 += step) {
      const int rows = (int)(m.rows - r0 < step ? m.rows - r0 : step);
      RC(quant_rows_to_f16((int)m.type, m.data + r0 * row_bytes, rows, K, p.scratch, 1, 0, st));
      RC(dense(x, rows, K, out + r0, residual ? residual + r0 : nullptr, nullptr, residual ? 1 : 0, out_ld));
    }
    return 0;
  };
  RC(bonsai_embed_rows_f16(p.embd, p.tokens, p.h, T, hidden, (int)p.vocab, st));
  for (int l = 0; l < p.layers; ++l) {
    const BlockLayer& w = layers[l];
    RC(bonsai_norm_to_f16_paired(p.h, hidden, w.attn_norm, eps, T, hidden, p.xn, hidden, 0, st));
    for (int i = BM_Q, c0 = 0; i <= BM_V; c0 += (int)w.m[i++].rows)
      if (w.m[i].rows > 0) RC(product(w.m[i], p.xn, hidden, p.qkv + c0, nullptr, qkv_n));
    RC(bonsai_qknorm_rope_kvstore(p.qkv, qkv_n, w.q_norm, w.k_norm, eps, p.rope_cos, p.rope_sin, p.positions, p.block_table, 0, p.q, T, nq, nkv, hd, kvt, page,
                                  w.kpool, w.vpool, w.kscale, w.vscale, st));
    // INT4 pages keep the attention kernel that they have always had: another order of sums moves keys and values to other codes (model_runner.cu)
    const bool settled = kvt == 3;
    RC(bonsai_attn_prefill_ws(p.q, T, pos0, p.block_table, nq, nkv, hd, kvt, page, w.kpool, w.vpool, w.kscale, w.vscale, p.attn, qd, 0,
                              settled ? nullptr : p.scratch, settled ? 0 : (size_t)p.scratch_elems, p.status, st));
    RC(product(w.m[BM_O], p.attn, qd, p.h, p.h, hidden));
    RC(bonsai_norm_to_f16_paired(p.h, hidden, w.ffn_norm, eps, T, hidden, p.xn, hidden, 0, st));
    {
      const BlockMatrix& g = w.m[BM_GATE];
      BlockMatrix u = w.m[BM_UP];
      if (u.rows == 0) u = {g.type, inter, g.data + inter * quant_row_bytes((int)g.type, hidden)};
      const long long gb = quant_row_bytes((int)g.type, hidden), ub = quant_row_bytes((int)u.type, hidden), most = p.scratch_elems / hidden / 2;      // pairs of rows
      if (gb < 0 || ub < 0 || (inter > most && most < 128)) return BONSAI_CUDA_BAD_ARG;
      const int slabs = (int)((inter + most - 1) / most), per = ((inter + slabs - 1) / slabs + 127) / 128 * 128, step = slabs == 1 ? inter : (per <= most ? per : (int)(most / 128 * 128));
      for (int r0 = 0; r0 < inter; r0 += step) {
        const int rows = inter - r0 < step ? inter - r0 : step;
        RC(quant_rows_to_f16((int)g.type, g.data + r0 * gb, rows, hidden, p.scratch, 2, 0, st));
        RC(quant_rows_to_f16((int)u.type, u.data + r0 * ub, rows, hidden, p.scratch, 2, 1, st));
        RC(dense(p.xn, 2 * rows, hidden, nullptr, nullptr, static_cast<char*>(p.act) + (size_t)r0 * 2, 2, inter));
      }
    }
    RC(product(w.m[BM_DOWN], p.act, inter, p.h, p.h, hidden));
  }
  return 0;
}

static int forward_row(const BlockRow& p, const BlockLayer* layers, float eps, cudaStream_t st) {
  const int hidden = (int)p.hidden, inter = (int)p.inter, hd = (int)p.head_dim, nq = (int)p.heads, nkv = (int)p.kv_heads, qd = nq * hd, qkv_n = qd + 2 * nkv * hd;
  const int kvt = (int)p.kvt, page = (int)p.page_size;
  auto product = [&](const BlockMatrix& m, const float* x, int K, const float* norm, float* out, const float* residual, int out_ld) {
    return m.rows == 0 ? 0 : bonsai_quant_gemv_batched_status((int)m.type, m.data, x, K, norm, eps, out, residual, out_ld, (int)m.rows, K, 1, p.status, st);
  };
  RC(bonsai_embed_rows_f16(p.embd, p.token, p.h, 1, hidden, (int)p.vocab, st));
  for (int l = 0; l < p.layers; ++l) {
    const BlockLayer& w = layers[l];
    for (int i = BM_Q, c0 = 0; i <= BM_V; c0 += (int)w.m[i++].rows) RC(product(w.m[i], p.h, hidden, w.attn_norm, p.qkv + c0, nullptr, qkv_n));
    RC(bonsai_qknorm_rope_kvstore(p.qkv, qkv_n, w.q_norm, w.k_norm, eps, p.rope_cos, p.rope_sin, p.position, p.block_table, 0, p.q, 1, nq, nkv, hd, kvt, page,
                                  w.kpool, w.vpool, w.kscale, w.vscale, st));
    RC(bonsai_attn_decode_route(p.q, p.position, p.block_table, 0, 1, nq, nkv, hd, kvt, page, w.kpool, w.vpool, w.kscale, w.vscale, (int)p.nsplit, p.ws_acc,
                                p.ws_ml, p.ws_rows, p.counters, p.attn, 0, 0, 1, st));
    RC(product(w.m[BM_O], p.attn, qd, nullptr, p.h, p.h, hidden));
    for (int i = BM_GATE, c0 = 0; i <= BM_UP; c0 += (int)w.m[i++].rows) RC(product(w.m[i], p.h, hidden, w.ffn_norm, p.gu + c0, nullptr, 2 * inter));
    RC(bonsai_swiglu_rows(p.gu, 2 * inter, p.act, inter, inter, 1, st));
    RC(product(w.m[BM_DOWN], p.act, inter, nullptr, p.h, p.h, hidden));
  }
  return bonsai_f16gemv(p.lm_head, p.h, p.out_norm, eps, p.logits, (int)p.lm_rows, hidden, st);
}

}  // namespace bonsai

extern "C" {

int bonsai_blocks_forward_row(const void* row, const void* layers, float eps, cudaStream_t stream) {
  return bonsai::forward_row(*static_cast<const bonsai::BlockRow*>(row), static_cast<const bonsai::BlockLayer*>(layers), eps, stream);
}
int bonsai_blocks_row_words() { return (int)(sizeof(bonsai::BlockRow) / 8); }
int bonsai_blocks_prompt_chunk(const void* prompt, const void* layers, float eps, int T, int pos0, cudaStream_t stream) {
  if (T < 1 || pos0 < 0) return BONSAI_CUDA_BAD_ARG;
  return bonsai::chunk(*static_cast<const bonsai::BlockPrompt*>(prompt), static_cast<const bonsai::BlockLayer*>(layers), eps, T, pos0, stream);
}
int bonsai_blocks_prompt_words() { return (int)(sizeof(bonsai::BlockPrompt) / 8); }
int bonsai_blocks_layer_words() { return (int)(sizeof(bonsai::BlockLayer) / 8); }

}  // extern "C"
