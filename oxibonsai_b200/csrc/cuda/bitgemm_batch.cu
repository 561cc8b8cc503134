// Packed GEMM for up to 64 tokens (decode batches, verification, short prompts): expanded weights go through tensor memory.
//
//   out[t][n] = sum_k X[t][k] * W[n][k]        t < T <= 64 tokens, n < N rows
//
// With few tokens the work is turning two-bit codes into f16 operands.  bitgemm_prefill.cu puts them into shared memory, 16 KB per
// 128 rows x 64 inputs that are written, fenced, and read back by the tensor core; bitgemm_hmma.cu keeps them in registers, at the
// legacy MMA rate, behind a barrier per 128 inputs.  Here a thread owns a weight row, makes 64 f16 weights in 32 registers and stores them to its
// lane of tensor memory (tcgen05.st), where tcgen05.mma takes its first operand from; the shared memory only sees the packed codes
// and the activations:
//   warps 0-11   expanders in three groups of four; group e fills the operand slots e and e + 3 of six, 128 inputs each
//   warps 12-15  epilogue
//   warps 16-17  MMA issuers, every other block each, with an accumulator of its own;  warp 18: codes (TMA tiles of 128 rows x 512 inputs,
//                before the kernel ahead has ended);  warp 19: activations
// Waits, MMAs and commits hold their thread for some 100 cycles each whatever they move, so a block is as deep as the slots allow and
// two threads issue: blocks of 64 inputs with one issuer took 0.33 us each, 24576 x 4096 and 16 tokens 33 us (with two 22, with three 24).
// The K range of a 128-row tile is cut over the S CTAs of a cluster, so that projections with few rows fill the GPU too; each CTA
// then adds up, in CTA order, the partial sums of its share of the tokens, which the others wrote into its shared memory.  A cluster
// takes tile after tile; the accumulators and the exchange are double-buffered.
// What bounds it: the expanders' chain of wait, expansion and store, 0.27 us per 16 K weights and SM (a slope over K; 0.28 at 64 tokens; 1.5
// instructions per weight for shift, mask and scale would allow 0.12), and 5 to 7 us per launch.  us at 8 / 32 / 64 tokens (before: the better of
// bitgemm_hmma and bitgemm_prefill): 6144 x 4096 10.2 / 12.1 / 15.7 (16.0 / 20.7 / 24.0), 4096 x 4096 9.5 / 11.0 / 13.8 (8.4 / 13.3 / 22.1),
// 24576 x 4096 19.4 / 24.6 / 36.3 (24.5 / 38.3 / 44.7), 4096 x 12288 13.2 / 14.4 / 17.0 (21.4 / 31.5 / 41.1).
#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

namespace bonsai {

constexpr int kGbSlots = 6;                            // operand slots in TMEM, one 128-input block (64 columns) each
constexpr int kGbGroups = 3, kGbIssuers = 2;
constexpr int kGbMaxCodes = 5, kGbMaxActs = 12;        // stages of codes (512 inputs) and of activations (128 inputs)
constexpr int kGbCodeBytes = 128 * 128;                // 128 rows x 512 inputs
constexpr int kGbEpiWarp = 4 * kGbGroups, kGbMmaWarp = kGbEpiWarp + 4, kGbCodeWarp = kGbMmaWarp + kGbIssuers, kGbActWarp = kGbCodeWarp + 1;
constexpr int kGbThreads = (kGbActWarp + 1) * 32;
constexpr int kGbMaxSplit = 8;
// Accumulators behind the operand slots, 128 columns: one per issuer, two sets up to 32 tokens.  A slot and a stage of activations always
// meet the same issuer (a wait must not be more than a phase behind its barrier): their numbers are multiples of the issuers.
constexpr int kGbAccCol = kGbSlots * 64;
// What shared memory holds beside the exchange.
__host__ __device__ inline int gb_code_stages(int tok) { return tok == 64 ? 3 : 5; }
__host__ __device__ inline int gb_act_stages(int tok) { return tok == 64 ? 6 : (tok == 32 ? 10 : 12); }

struct GbParams {
  const __half* scales;
  float* out_f32;          // epi 0, 1
  const float* residual;   // epi 1
  __half* out_f16;         // epi 2: SwiGLU over interleaved gate / up rows, paired-K order
  int* status;
  int n_rows, K, T, epi, out_ld, split, tok;           // tok: T rounded up to 16, 32 or 64
};

__device__ __forceinline__ void gb_load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(tc::smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void gb_load3(void* dst, const CUtensorMap* map, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3}], [%4];" ::"r"(tc::smem_u32(dst)),
               "l"(map), "r"(0), "r"(z), "r"(tc::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void gb_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void gb_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
      "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ uint32_t gb_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void gb_st_remote(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void gb_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// bounded wait that also acquires what other CTAs of the cluster wrote before they arrived; every lane polls
__device__ __forceinline__ bool gb_wait_cluster(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < tc::kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(tc::smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

__global__ void __launch_bounds__(kGbThreads, 1) bitgemm_batch_kernel(const __grid_constant__ CUtensorMap cmap, const __grid_constant__ CUtensorMap xmap,
                                                                     GbParams p) {
  extern __shared__ uint8_t gb_smem[];
  uint8_t* base = (uint8_t*)(((uintptr_t)gb_smem + 1023) & ~(uintptr_t)1023);
  uint8_t* sC = base;                                                       // codes
  const int nC = gb_code_stages(p.tok), nA = gb_act_stages(p.tok), act_bytes = p.tok * 256;
  uint8_t* sB = base + nC * kGbCodeBytes;                                    // activations
  float* sR = reinterpret_cast<float*>(sB + nA * act_bytes);                 // partial sums [2][split][share of the tokens][128 rows]
  __shared__ uint64_t c_full[kGbMaxCodes], c_empty[kGbMaxCodes], a_full[kGbMaxActs], a_empty[kGbMaxActs], full[kGbSlots], empty[kGbSlots], accf[2], acce[2], red[2];
  __shared__ uint32_t tmem_slot;
  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
  const int S = p.split, rank = blockIdx.x % S, cid = blockIdx.x / S, nclusters = gridDim.x / S;
  const int groups = p.K >> 7, row_tiles = (p.n_rows + 127) >> 7;
  const int g0 = rank * groups / S, nb = (rank + 1) * groups / S - g0;      // this CTA's 128-input blocks of every tile
  const int share = (p.tok + S - 1) / S;                                   // tokens that a CTA of the cluster finishes
  const int sets = p.tok <= 32 ? 2 : 1;                                    // of accumulators
  // Blocks are numbered through over the CTA's tiles: block `it` goes through group it % 3, slot it % 6, issuer it % 2.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp == kGbMmaWarp) {
    tc::tmem_alloc(&tmem_slot, 512);
    tc::tmem_relinquish();
  }
  if (t == 0) {
    for (int i = 0; i < nC; ++i) {
      tc::mbar_init(&c_full[i], 1);
      tc::mbar_init(&c_empty[i], 4 * kGbGroups);
    }
    for (int i = 0; i < nA; ++i) {
      tc::mbar_init(&a_full[i], 1);
      tc::mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < kGbSlots; ++i) {
      tc::mbar_init(&full[i], 4);              // the expander warps of the group
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&accf[i], kGbIssuers);
      tc::mbar_init(&acce[i], 4);
      tc::mbar_init(&red[i], 4 * S);
    }
    tc::mbar_fence_init();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc::tc_fence_after();
  const uint32_t taddr = tmem_slot;
  bool failed = false;

  if (warp == kGbCodeWarp) {
    if (tc::elect_one()) {
      int s = 0, issued = 0;
      uint32_t phase = 1;
      for (int tile = cid; tile < row_tiles && !failed; tile += nclusters)
        for (int kb = 0; kb < nb; kb += 4, ++issued) {
          if (!tc::mbar_wait_sleep<100>(&c_empty[s], phase)) { failed = true; break; }
          tc::mbar_arrive_expect_tx(&c_full[s], kGbCodeBytes);
          gb_load(sC + s * kGbCodeBytes, &cmap, (g0 + kb) * 8, tile * 128, &c_full[s]);
          if (++s == nC) { s = 0; phase ^= 1; }
        }
      if (failed) atomicExch(p.status, 1);
      tc::mbar_drain(c_full, issued, nC);
    }
    __syncwarp();
  } else if (warp == kGbActWarp) {
    if (tc::elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      int s = 0, issued = 0;
      uint32_t phase = 1;
      for (int tile = cid; tile < row_tiles && !failed; tile += nclusters)
        for (int kb = 0; kb < nb; ++kb, ++issued) {
          if (!tc::mbar_wait_sleep<100>(&a_empty[s], phase)) { failed = true; break; }
          tc::mbar_arrive_expect_tx(&a_full[s], act_bytes);
          gb_load3(sB + s * act_bytes, &xmap, (g0 + kb) * 2, &a_full[s]);
          if (++s == nA) { s = 0; phase ^= 1; }
        }
      if (failed) atomicExch(p.status, 1);
      tc::mbar_drain(a_full, issued, nA);
    }
    __syncwarp();
  } else if (warp >= kGbMmaWarp) {
    if (tc::elect_one()) {
      const uint32_t idesc = tc::idesc_f32acc(tc::FMT_F16, tc::FMT_F16, 128, (uint32_t)p.tok);
      const int me = warp - kGbMmaWarp;
      int it0 = 0, seg = 0;
      for (int tile = cid; tile < row_tiles && !failed; tile += nclusters, ++seg, it0 += nb) {
        const int ab = sets == 2 ? seg & 1 : 0, use = sets == 2 ? seg >> 1 : seg;
        if (!tc::mbar_wait(&acce[ab], (use & 1) ^ 1)) { failed = true; break; }
        tc::tc_fence_after();
        const uint32_t acc = taddr + kGbAccCol + (ab * kGbIssuers + me) * p.tok;
        bool fresh = true;
        for (int kb = (it0 + me) & 1; kb < nb; kb += 2) {
          const int it = it0 + kb, s = it % kGbSlots, as = it % nA;
          if (!tc::mbar_wait(&a_full[as], (it / nA) & 1) || !tc::mbar_wait(&full[s], (it / kGbSlots) & 1)) { failed = true; break; }
          tc::tc_fence_after();
          const uint64_t db = tc::smem_desc_sw128(tc::smem_u32(sB + as * act_bytes));
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)
            gb_mma(acc, taddr + s * 64 + k * 8, db + (k >> 2) * (uint32_t)(p.tok * 128 >> 4) + (k & 3) * 2, idesc, !(fresh && k == 0));
          fresh = false;
          tc::mma_commit(&empty[s]);
          tc::mma_commit(&a_empty[as]);
        }
        tc::mma_commit(&accf[ab]);
      }
      if (failed) atomicExch(p.status, 1);
    }
    __syncwarp();
  } else if (warp < kGbEpiWarp) {
    // thread = weight row of the tile; all lanes poll (one that passes the outcome on is a shuffle later: 24576 x 4096, 8 tokens 22.3 against 19.6 us)
    const int group = warp >> 2, r = t & 127;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    auto scale_of = [&](int tile, int kb) {
      while (kb >= nb) { kb -= nb; tile += nclusters; }
      return tile < row_tiles ? __ldg(p.scales + (size_t)min(tile * 128 + r, p.n_rows - 1) * groups + g0 + kb) : __float2half(0.0f);
    };
    int it0 = 0, cs = 0;
    uint32_t cphase = 0;
    __half next = scale_of(cid, group);         // scale of this group's next block, requested a block ahead
    for (int tile = cid; tile < row_tiles && !failed; tile += nclusters, it0 += nb) {
      for (int kb0 = 0; kb0 < nb && !failed; kb0 += 4) {
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&c_full[cs], cphase))) { failed = true; break; }
        const int end = min(kb0 + 4, nb);
        for (int kb = kb0 + (group + 3 - (it0 + kb0) % 3) % 3; kb < end; kb += 3) {
          const int it = it0 + kb, s = it % kGbSlots;
          // A masked code is +-2^-7 or 0 and the scale is taken times 128; a row of the warp with a scale of 512 or more (none in earnest) takes the
          // other order, which leaves every f16 scale in range.
          const __half d = next;
          next = scale_of(tile, kb + 3);
          auto block = [&](auto large) {
            const __half2 up = __half2half2(__float2half(128.0f)), d2 = large ? __half2half2(d) : __hmul2(__half2half2(d), up);
            auto weights = [&](uint32_t m) {
              const __half2 c = *reinterpret_cast<const __half2*>(&m), w = large ? __hmul2(__hmul2(c, up), d2) : __hmul2(c, d2);
              return *reinterpret_cast<const uint32_t*>(&w);
            };
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint4 code = *reinterpret_cast<const uint4*>(sC + cs * kGbCodeBytes + tc::sw128_offset(r, 2 * (kb - kb0) + h));
              const uint32_t w4[4] = {code.x, code.y, code.z, code.w};
              uint32_t o[32];
#pragma unroll
              for (int wd = 0; wd < 4; ++wd)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  o[wd * 8 + i] = weights((w4[wd] << (12 - 4 * i)) & 0xA000A000u);
                  o[wd * 8 + 4 + i] = weights((w4[wd] << (13 - 4 * i)) & 0xA000A000u);
                }
              if (h == 0) {
                if (!__all_sync(0xffffffffu, tc::mbar_wait(&empty[s], ((it / kGbSlots) & 1) ^ 1))) return false;
                tc::tc_fence_after();
              }
              gb_st32(taddr + lanes + s * 64 + h * 32, o);
            }
            return true;
          };
          if (__any_sync(0xffffffffu, __hge(__habs(d), __float2half(512.0f)))) failed = !block(std::true_type{});
          else failed = !block(std::false_type{});
          if (failed) break;
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&full[s]);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&c_empty[cs]);
        if (++cs == nC) { cs = 0; cphase ^= 1; }
      }
    }
    if (failed && lane == 0) atomicExch(p.status, 1);
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int CB = 16;
    const int a = t - kGbEpiWarp * 32, quarter = warp & 3;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const int tok_lo = rank * share, tok_hi = min(p.T, tok_lo + share);
    const uint32_t share_inv = (65536u + share - 1) / share;      // c / share for c < 64
    int seg = 0, it0 = 0;
    for (int tile = cid; tile < row_tiles; tile += nclusters, ++seg, it0 += nb) {
      const int rb = seg & 1, ab = sets == 2 ? rb : 0, use = sets == 2 ? seg >> 1 : seg, row = tile * 128 + a;
      const bool row_ok = row < p.n_rows;
      if (!tc::mbar_wait_warp<64>(&accf[ab], use & 1, lane)) { failed = true; break; }
      tc::tc_fence_after();
      float* mine = sR + (size_t)rb * S * share * 128;
      const uint32_t mine_at = tc::smem_u32(mine + a);
      const uint32_t acc = taddr + lanes + kGbAccCol + ab * kGbIssuers * p.tok;
      const int one = nb == 1 ? it0 & 1 : 0;        // a tile of one block was in one issuer's accumulator only
      for (int c0 = 0; c0 < p.T; c0 += CB) {
        uint32_t v[CB], w[CB];
        tc::tmem_ld16(acc + one * p.tok + c0, v);
        if (nb > 1) tc::tmem_ld16(acc + p.tok + c0, w);
        tc::tmem_wait_ld();
        if (nb > 1) {
#pragma unroll
          for (int j = 0; j < CB; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        }
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          const int c = c0 + j, to = (int)((uint32_t)c * share_inv >> 16);
          const uint32_t at = mine_at + (uint32_t)(rank * share + c - to * share) * 512;
          if (c < p.T) gb_st_remote(S > 1 ? gb_map(at, (uint32_t)to) : at, __uint_as_float(v[j]));
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[ab]);
      if (lane < S) gb_arrive_remote(gb_map(tc::smem_u32(&red[rb]), (uint32_t)lane));
      if (!gb_wait_cluster(&red[rb], (seg >> 1) & 1)) { failed = true; break; }
      __syncwarp();
      // this CTA's tokens, eight at a time: partial sums in CTA order, the residuals as a block before the stores (they usually alias)
      for (int c0 = tok_lo; c0 < tok_hi; c0 += 8) {
        float v[8], res[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) res[j] = p.epi == 1 && row_ok && c0 + j < tok_hi ? p.residual[(size_t)(c0 + j) * p.out_ld + row] : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = 0.0f;
          if (c0 + j < tok_hi)
            for (int i = 0; i < S; ++i) v[j] += mine[((size_t)i * share + (c0 + j - tok_lo)) * 128 + a];
        }
        if (p.epi == 2) {
          const bool odd = lane & 1;      // gate (even) and up (odd) rows are neighbouring lanes; each finishes every other token
          const int o = row >> 1;
          __half* dst = p.out_f16 + ((o & ~7) | ((o & 3) << 1) | ((o >> 2) & 1));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float keep = odd ? v[2 * j + 1] : v[2 * j], other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * j] : v[2 * j + 1], 1);
            const float g = odd ? other : keep, u = odd ? keep : other;
            const int c = c0 + 2 * j + (odd ? 1 : 0);
            if (row_ok && c < tok_hi) dst[(size_t)c * p.out_ld] = __float2half_rn(g / (1.0f + __expf(-g)) * u);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (row_ok && c0 + j < tok_hi) p.out_f32[(size_t)(c0 + j) * p.out_ld + row] = p.epi == 1 ? res[j] + v[j] : v[j];
        }
      }
      __syncwarp();
    }
    if (failed && lane == 0) atomicExch(p.status, 1);
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (warp == kGbMmaWarp) tc::tmem_dealloc(taddr, 512);
  // nobody leaves while another CTA of the cluster may still write to it (after an expired wait it would)
  if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static bool gb_maps(CUtensorMap* cmap, CUtensorMap* xmap, const void* codes, int n_rows, int K, const void* x, int x_ld, int T, int tok) {
  cuuint64_t cd[2] = {(cuuint64_t)K / 16, (cuuint64_t)n_rows}, cst[1] = {(cuuint64_t)K / 4};
  cuuint64_t xd[3] = {64, (cuuint64_t)T, (cuuint64_t)K / 64}, xst[2] = {(cuuint64_t)x_ld * 2, 128};      // [K / 64][T][64]
  cuuint32_t cbox[2] = {32, 128}, xbox[3] = {64, (cuuint32_t)tok, 2}, estr[3] = {1, 1, 1};
  return cuTensorMapEncodeTiled(cmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(codes), cd, cst, cbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
         cuTensorMapEncodeTiled(xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), xd, xst, xbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static size_t gb_smem_bytes(int tok, int split) {
  const int share = (tok + split - 1) / split;
  return 1024 + (size_t)gb_code_stages(tok) * kGbCodeBytes + (size_t)gb_act_stages(tok) * tok * 256 + (size_t)2 * split * share * 128 * sizeof(float);
}

static cudaLaunchConfig_t gb_config(cudaLaunchAttribute* attr, int clusters, int split, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * split);
  cfg.blockDim = dim3(kGbThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = split;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

// How many clusters of each size the device holds at once (the CTA's shared memory allows one per SM whatever the tokens are); null when the
// device does not say.  The table is published behind its flag: threads that come first together ask one after another.
static const int* gb_clusters() {
  static int held[64][kGbMaxSplit + 1];
  static std::atomic<bool> known[64];
  static std::mutex asking;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  if (known[dev].load(std::memory_order_acquire)) return held[dev];
  std::lock_guard<std::mutex> lock(asking);
  if (!known[dev].load(std::memory_order_relaxed)) {
    if (cudaFuncSetAttribute(bitgemm_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) return nullptr;
    for (int s = 1; s <= kGbMaxSplit; ++s) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t cfg = gb_config(attr, 1, s, gb_smem_bytes(64, s), nullptr);
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, bitgemm_batch_kernel, &cfg) != cudaSuccess || n < 1) n = 0;
      held[dev][s] = n;
    }
    (void)cudaGetLastError();
    known[dev].store(true, std::memory_order_release);
  }
  return held[dev];
}

}  // namespace bonsai

extern "C" {

// codes / scales: planar layout (common.cuh), x_f16 [T][x_ld] in paired-K order, T <= 64, K a multiple of 128.  epi 0: out_f32 = W x; 1: out_f32 =
// residual + W x; 2: out_f16 = SwiGLU over interleaved gate / up rows (paired-K order, out_ld at least n_rows / 2 rounded up to 8).  split: CTAs that share a tile's K range (1 to 8),
// 0 = chosen by size.
int bonsai_bitgemm_batch(const void* codes, const void* scales, const void* x_f16, int x_ld, float* out_f32, const float* residual, void* out_f16,
                         int* status, int n_rows, int K, int T, int epi, int out_ld, int split, cudaStream_t stream) {
  using namespace bonsai;
  if (K < 128 || K % 128 != 0 || n_rows < 1 || T < 1 || T > 64 || epi < 0 || epi > 2 || x_ld < K || x_ld % 8 != 0 || status == nullptr) return BONSAI_CUDA_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(codes) | reinterpret_cast<uintptr_t>(x_f16)) & 15) != 0 || split < 0 || split > kGbMaxSplit) return BONSAI_CUDA_BAD_ARG;
  if ((epi <= 1 && out_f32 == nullptr) || (epi == 1 && residual == nullptr) || (epi == 2 && (out_f16 == nullptr || n_rows % 2 != 0))) return BONSAI_CUDA_BAD_ARG;
  const int* held = gb_clusters();
  if (held == nullptr) return BONSAI_CUDA_LAUNCH_FAILED;
  const int groups = K / 128, tiles = (n_rows + 127) / 128;
  const int most = groups < kGbMaxSplit ? groups : kGbMaxSplit;
  if (split > most) split = most;
  if (split == 0 || held[split] < 1) {
    // rounds of tiles times the 128-input blocks that a CTA goes through, plus what a tile costs whatever its depth (accumulator drain and
    // exchange, six blocks' time) and a cluster for its size.  16 tokens, us by split 1 / 2 / 3 / 4 / 6: 6144 x 4096 15.8 / 11.3 / 11.8 / 11.4 / 12.9;
    // 24576 x 4096 27.0 / 22.7 / 25.3 / 27.1 / 35.4; 4096 x 12288 38.4 / 20.3 / 17.0 / 15.4 / 15.7; 2560 x 4096 15.6 / 9.2 / 7.8 / 7.9 / 8.7.
    long long best = -1;
    for (int s = 1; s <= most; ++s) {
      if (held[s] < 1) continue;
      const long long rounds = (tiles + held[s] - 1) / held[s], cost = rounds * ((groups + s - 1) / s + 6) + 3 * s;
      if (best < 0 || cost < best) {
        best = cost;
        split = s;
      }
    }
    if (best < 0) return BONSAI_CUDA_LAUNCH_FAILED;
  }
  const int tok = T <= 16 ? 16 : (T <= 32 ? 32 : 64);
  CUtensorMap cmap, xmap;
  if (!gb_maps(&cmap, &xmap, codes, n_rows, K, x_f16, x_ld, T, tok)) return BONSAI_CUDA_BAD_ARG;
  GbParams p{(const __half*)scales, out_f32, residual, (__half*)out_f16, status, n_rows, K, T, epi, out_ld, split, tok};
  cudaLaunchAttribute attr[2];
  const int clusters = tiles < held[split] ? tiles : held[split];
  // the request is that of 64 tokens, so that one CTA has an SM whatever the batch is
  cudaLaunchConfig_t cfg = gb_config(attr, clusters, split, gb_smem_bytes(64, split), stream);
  return cudaLaunchKernelEx(&cfg, bitgemm_batch_kernel, cmap, xmap, p) == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

}  // extern "C"
