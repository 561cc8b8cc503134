// Dense f16 GEMM for prompts on pairs of SMs, and the expansion of packed weights into its operand.
//
//   out[t][n] = sum_k X[t][k] * W[n][k]        t < T tokens, n < N rows
//
// A cluster of two CTAs works on a tile of 256 weight rows x up to 256 tokens with tcgen05.mma cta_group::2: each CTA stages its own
// 128 weight rows and half of the tokens per 64-input block, so a block costs 32 KB of copies per SM where the single-SM tile of
// 128 x 256 (bitgemm_prefill.cu) costs 48 KB, and six blocks fit instead of four.  Copies and tensor core together are what bounds
// the single-SM kernel: its operands come and go at the shared-memory rate.
//   warp 8      copies (TMA) of this CTA's halves; they all report to the leader's barrier
//   warp 9      of the leader: one thread issues the MMAs of both SMs and commits to the barriers of both
//   warps 0-7   epilogue: a warp has a quarter of the CTA's rows and half of the tile's tokens; two accumulators in TMEM
// Tiles go round robin to the clusters, those that share weight rows one after another (they are read from L2 then).
//
// The tokens per tile (a multiple of 16) are chosen per call: pair_tile_tokens below.
//
// Packed weights (planar layout, common.cuh) are expanded to f16 once per prompt chunk, slab by slab into one scratch matrix that
// stays in L2, in the paired-K order that the activations have.  Expanding inside the GEMM instead repeats the work for every 256
// tokens and holds the tensor core to half its rate.  4096 x 4096, dense, 4096 tokens: 124 us with the single-SM tile, 104 here
// (1.32 PFLOP/s); 6144 x 4096 packed, 192 tokens: 44 us in place, 25 expanded first.  Issued by elected threads: 53 us instead of 17 for 64
// blocks behind `lane == 0`.
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace bonsai {

constexpr int kGpStages = 6;
constexpr int kGpBlock = 64;                         // inputs per stage
constexpr int kGpABytes = 128 * kGpBlock * 2;        // 16 KB: this CTA's 128 weight rows
constexpr int kGpBBytes = 128 * kGpBlock * 2;        // 16 KB: half of up to 256 tokens
constexpr int kGpEpiWarps = 8;
constexpr int kGpThreads = (kGpEpiWarps + 2) * 32;
constexpr int kGpCols = 256;                         // TMEM columns of one accumulator, two of them

struct GpParams {
  float* out_f32;          // epi 0, 1: [T][out_ld]
  const float* residual;   // epi 1
  __half* out_f16;         // epi 2 (SwiGLU over interleaved gate / up rows, paired-K order), 3
  int* status;
  int n_rows, K, T, epi, out_ld, tile_tok;
};

__device__ __forceinline__ uint32_t gp_map(uint32_t addr, uint32_t rank) {      // the same shared-memory place in CTA `rank` of the cluster
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void gp_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this place in both CTAs once the MMAs issued so far are done
__device__ __forceinline__ void gp_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(tc::smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void gp_arrive_at(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__host__ __device__ inline int gp_paired_k(int k) { return (k & ~7) | (((k & 3) << 1) | ((k >> 2) & 1)); }

__global__ void __launch_bounds__(kGpThreads, 1) __cluster_dims__(2, 1, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                                           const __grid_constant__ CUtensorMap wmap, GpParams p) {
  extern __shared__ uint8_t gp_smem[];
  uint8_t* base = (uint8_t*)(((uintptr_t)gp_smem + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = base;
  uint8_t* sB = base + kGpStages * kGpABytes;
  __shared__ uint64_t full[kGpStages], empty[kGpStages], accf[2], acce[2];
  __shared__ uint32_t tmem_slot;
  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
  const uint32_t rank = blockIdx.x & 1;
  const int cid = blockIdx.x >> 1, nclusters = gridDim.x >> 1;
  const int nblk = p.K / kGpBlock, tn = p.tile_tok;
  const int tok_tiles = (p.T + tn - 1) / tn, ntiles = ((p.n_rows + 255) >> 8) * tok_tiles;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == kGpEpiWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_slot)), "r"(2 * kGpCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    for (int i = 0; i < kGpStages; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&accf[i], 1);
      tc::mbar_init(&acce[i], 2 * kGpEpiWarps);
    }
    tc::mbar_fence_init();
  }
  tc::tc_fence_before();
  __syncthreads();
  gp_cluster_sync();                 // both CTAs' barriers exist and both have their TMEM
  tc::tc_fence_after();
  const uint32_t taddr = tmem_slot;
  bool failed = false;

  if (warp == kGpEpiWarps) {
    if (tc::elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      const uint32_t bytes = 2u * (kGpABytes + (uint32_t)tn * kGpBlock);      // both CTAs' weight rows and halves of the tokens
      int s = 0, issued = 0;
      uint32_t phase = 1;
      for (int tile = cid; tile < ntiles && !failed; tile += nclusters) {
        const int row0 = (tile / tok_tiles) * 256 + (int)rank * 128, tok0 = (tile % tok_tiles) * tn + (int)rank * (tn >> 1);
        for (int kb = 0; kb < nblk; ++kb, ++issued) {
          if (!tc::mbar_wait(&empty[s], phase)) { failed = true; break; }
          const uint32_t bar = gp_map(tc::smem_u32(&full[s]), 0);
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], bytes);
          gp_load(tc::smem_u32(sA + s * kGpABytes), &wmap, kb * kGpBlock, row0, bar);
          gp_load(tc::smem_u32(sB + s * kGpBBytes), &xmap, kb * kGpBlock, tok0, bar);
          if (++s == kGpStages) { s = 0; phase ^= 1; }
        }
      }
      if (failed) atomicExch(p.status, 1);
      if (rank == 0) tc::mbar_drain(full, issued, kGpStages);      // both CTAs' copies; the other one waits at the barrier below
    }
  } else if (warp == kGpEpiWarps + 1) {
    if (rank == 0 && tc::elect_one()) {
      const uint32_t idesc = tc::idesc_f32acc(tc::FMT_F16, tc::FMT_F16, 256, (uint32_t)tn);
      int s = 0, seg = 0;
      uint32_t phase = 0;
      for (int tile = cid; tile < ntiles && !failed; tile += nclusters, ++seg) {
        const int ab = seg & 1;
        if (!tc::mbar_wait(&acce[ab], ((seg >> 1) & 1) ^ 1)) { failed = true; break; }
        tc::tc_fence_after();
        for (int kb = 0; kb < nblk; ++kb) {
          if (!tc::mbar_wait(&full[s], phase)) { failed = true; break; }
          tc::tc_fence_after();
          const uint64_t da = tc::smem_desc_sw128(tc::smem_u32(sA + s * kGpABytes)), db = tc::smem_desc_sw128(tc::smem_u32(sB + s * kGpBBytes));
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) gp_mma(taddr + ab * kGpCols, da + 2 * k, db + 2 * k, idesc, kb > 0 || k > 0);
          gp_commit(&empty[s]);
          if (++s == kGpStages) { s = 0; phase ^= 1; }
        }
        gp_commit(&accf[ab]);
      }
      if (failed) atomicExch(p.status, 1);
    }
    __syncwarp();
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int CB = 16;
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t drained[2] = {gp_map(tc::smem_u32(&acce[0]), 0), gp_map(tc::smem_u32(&acce[1]), 0)};
    int seg = 0;
    for (int tile = cid; tile < ntiles; tile += nclusters, ++seg) {
      const int ab = seg & 1;
      const int row = (tile / tok_tiles) * 256 + (int)rank * 128 + quarter * 32 + lane, tok0 = (tile % tok_tiles) * tn;
      const bool row_ok = row < p.n_rows;
      const int end = min(tn, p.T - tok0);
      if (!tc::mbar_wait_warp<64>(&accf[ab], (seg >> 1) & 1, lane)) { failed = true; break; }
      tc::tc_fence_after();
#pragma unroll 1
      for (int c0 = half * CB; c0 < end; c0 += 2 * CB) {
        uint32_t r[CB];
        tc::tmem_ld16(taddr + lane_base + ab * kGpCols + c0, r);
        const int tok = tok0 + c0;
        float res[CB];
        if (p.epi == 1) {      // residuals as a block before the stores: output and residual usually alias
#pragma unroll
          for (int j = 0; j < CB; ++j) res[j] = row_ok && c0 + j < end ? p.residual[(size_t)(tok + j) * p.out_ld + row] : 0.0f;
        }
        tc::tmem_wait_ld();
        if (p.epi == 2) {
          // gate (even) and up (odd) rows are neighbouring lanes: the even lane finishes the even tokens, the odd lane the odd ones
          const bool odd = lane & 1;
          __half* dst = p.out_f16 + gp_paired_k(row >> 1);
#pragma unroll
          for (int j = 0; j < CB / 2; ++j) {
            const float keep = __uint_as_float(odd ? r[2 * j + 1] : r[2 * j]);
            const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[2 * j] : r[2 * j + 1]), 1);
            const float g = odd ? other : keep, u = odd ? keep : other;
            const int c = 2 * j + (odd ? 1 : 0);
            if (row_ok && c0 + c < end) dst[(size_t)(tok + c) * p.out_ld] = __float2half_rn(g / (1.0f + __expf(-g)) * u);
          }
        } else if (p.epi == 3) {
#pragma unroll
          for (int j = 0; j < CB; ++j)
            if (row_ok && c0 + j < end) p.out_f16[(size_t)(tok + j) * p.out_ld + row] = __float2half_rn(__uint_as_float(r[j]));
        } else {
#pragma unroll
          for (int j = 0; j < CB; ++j)
            if (row_ok && c0 + j < end) p.out_f32[(size_t)(tok + j) * p.out_ld + row] = p.epi == 1 ? res[j] + __uint_as_float(r[j]) : __uint_as_float(r[j]);
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) gp_arrive_at(drained[ab]);
    }
  }
  if (warp < kGpEpiWarps && failed && lane == 0) atomicExch(p.status, 1);
  tc::tc_fence_before();
  __syncwarp();
  gp_cluster_sync();                 // nobody leaves while the other CTA may still read its shared memory or TMEM, or signal it
  tc::tc_fence_after();
  if (warp == kGpEpiWarps + 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(2 * kGpCols) : "memory");
}

// Rows row0 .. row0 + rows - 1 of a planar matrix as f16 [rows][K] in paired-K order: a thread writes eight weights, one 16-byte word.
// Two lanes share a code word (its a pairs and its b pairs).  Bound by the stores.
__global__ void __launch_bounds__(256) expand_rows_kernel(const uint32_t* __restrict__ codes, const __half* __restrict__ scales, int rows, int K,
                                                          uint4* __restrict__ out) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");      // the GEMM ahead reads the scratch matrix
  const size_t total = (size_t)rows * (K >> 3), stride = (size_t)gridDim.x * blockDim.x;
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int U = 4;
  for (; i < total; i += U * stride) {
    uint32_t w[U];
    __half sc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t j = i + u * stride;
      w[u] = j < total ? __ldg(codes + (j >> 1)) : 0u;
      sc[u] = j < total ? __ldg(scales + (j >> 4)) : __float2half(0.0f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t j = i + u * stride;
      const __half2 d2 = __half2half2(sc[u]), up = __half2half2(__float2half(128.0f));
      const uint32_t v = (j & 1) ? w[u] << 1 : w[u];
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t m = (v << (12 - 4 * k)) & 0xA000A000u;       // +-2^-7 or 0, two weights four inputs apart
        const __half2 h = __hmul2(__hmul2(*reinterpret_cast<const __half2*>(&m), up), d2);      // in this order any f16 scale stays in range
        o[k] = *reinterpret_cast<const uint32_t*>(&h);
      }
      if (j < total) out[j] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

static bool gp_map_f16(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_rows) {
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {kGpBlock, box_rows}, estr[2] = {1, 1};
  return cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tokens per tile: the fewest rounds of tiles times the cycles that a 64-input block takes, which is 2 per token on the tensor core,
// or the copies of 128 weight rows and half of the tokens at some 70 bytes a cycle, whichever is longer.
static int pair_tile_tokens(int n_rows, int T, int clusters) {
  const long long row_tiles = (n_rows + 255) / 256;
  int best = 256;
  long long best_cost = -1;
  for (int tn = 256; tn >= 32; tn -= 16) {
    const long long tiles = row_tiles * ((T + tn - 1) / tn), rounds = (tiles + clusters - 1) / clusters;
    const long long tensor = 2 * tn, copies = (kGpABytes + 64 * tn) / 70;
    const long long cost = rounds * ((tensor > copies ? tensor : copies) + 16);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = tn;
    }
  }
  return best;
}

static int launch_pair(const void* w, const void* x, int x_ld, GpParams p, int sms, cudaStream_t st) {
  const int clusters_max = sms / 2 < 1 ? 1 : sms / 2;
  if (p.tile_tok == 0) p.tile_tok = pair_tile_tokens(p.n_rows, p.T, clusters_max);
  CUtensorMap xmap, wmap;
  if (!gp_map_f16(&xmap, x, p.K, p.T, x_ld, p.tile_tok / 2) || !gp_map_f16(&wmap, w, p.K, p.n_rows, p.K, 128)) return BONSAI_CUDA_BAD_ARG;
  const long long tiles = (long long)((p.n_rows + 255) / 256) * ((p.T + p.tile_tok - 1) / p.tile_tok);
  const int clusters = (int)(tiles < clusters_max ? tiles : clusters_max);
  const size_t smem = 1024 + (size_t)kGpStages * (kGpABytes + kGpBBytes);
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BONSAI_CUDA_LAUNCH_FAILED;
  if (!configured[dev]) {
    if (cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return BONSAI_CUDA_LAUNCH_FAILED;
    configured[dev] = true;
  }
  const cudaError_t e = launch_pdl(gemm_pair_kernel, dim3(2 * clusters), dim3(kGpThreads), smem, st, xmap, wmap, p);
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

}  // namespace bonsai

extern "C" {

// x_f16 [T][x_ld], w_f16 [n_rows][K] in one K order, 16-byte aligned, K a multiple of 64, x_ld of 8.  epi 0: out_f32 = W x; 1: out_f32 =
// residual + W x; 2: out_f16 = SwiGLU over interleaved gate / up rows (paired-K order, out_ld at least n_rows / 2 rounded up to 8); 3: out_f16 =
// W x.  tile_tok: tokens per tile (a multiple of 16 up to 256), 0 = chosen here.
int bonsai_gemm_pair(const void* w_f16, const void* x_f16, int x_ld, float* out_f32, const float* residual, void* out_f16, int* status, int n_rows,
                     int K, int T, int epi, int out_ld, int sms, int tile_tok, cudaStream_t stream) {
  using namespace bonsai;
  if (K < 64 || K % 64 != 0 || n_rows < 1 || T < 1 || epi < 0 || epi > 3 || x_ld < K || x_ld % 8 != 0 || status == nullptr) return BONSAI_CUDA_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(w_f16) | reinterpret_cast<uintptr_t>(x_f16)) & 15) != 0) return BONSAI_CUDA_BAD_ARG;
  if (tile_tok < 0 || tile_tok > 256 || tile_tok % 16 != 0) return BONSAI_CUDA_BAD_ARG;
  if ((epi <= 1 && out_f32 == nullptr) || (epi == 1 && residual == nullptr) || (epi >= 2 && out_f16 == nullptr) ||
      (epi == 2 && (n_rows % 2 != 0 || out_ld < (n_rows / 2 + 7) / 8 * 8)))
    return BONSAI_CUDA_BAD_ARG;
  return launch_pair(w_f16, x_f16, x_ld, GpParams{out_f32, residual, (__half*)out_f16, status, n_rows, K, T, epi, out_ld, tile_tok}, sms, stream);
}

int bonsai_expand_rows(const void* codes, const void* scales, int row0, int rows, int K, void* out, cudaStream_t stream) {
  using namespace bonsai;
  if (rows < 1 || row0 < 0 || K < 128 || K % 128 != 0) return BONSAI_CUDA_BAD_ARG;
  const size_t total = (size_t)rows * (K >> 3);
  const int grid = (int)((total + 1023) / 1024 < 148 * 8 ? (total + 1023) / 1024 : 148 * 8);
  const cudaError_t e = launch_pdl(expand_rows_kernel, dim3(grid), dim3(256), 0, stream, (const uint32_t*)codes + (size_t)row0 * (K >> 4),
                                   (const __half*)scales + (size_t)row0 * (K >> 7), rows, K, (uint4*)out);
  return e == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

}  // extern "C"
