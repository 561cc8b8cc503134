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
//   warps 16-17  MMA issuers, every other block each, with an accumulator of its own;  warp 18: asks L2 for the weights of the CTA's share;
//                warp 19: activations
// The K range of a 128-row tile is cut over the S CTAs of a cluster, so that projections with few rows fill the GPU too; each CTA
// then adds up, in CTA order, the partial sums of its share of the tokens, which the others wrote into its shared memory.  A cluster
// takes tile after tile; the accumulators and the exchange are double-buffered.
// What bounds it: chains.  A block of 16 K weights takes 390 cycles of an SM: the expanders' integer pipe (a mask per pair of weights), and behind it
// their chain of load, expansion, store and barriers (300 with the expansion taken out, whatever the MMAs and the tokens are; 256 is the
// tensor pipe at 64 tokens).  Around the blocks stand set-up 2600, the first activations 1900, drain and exchange 2000, sums and stores 600 to 1700 cycles.
// Two issuers, since waits, MMAs and commits hold their thread for some 100 cycles each whatever they move (one 33 us, three 24 us where two took 22).
// Codes come by plain loads, 32 bytes of its row per thread: through a ring of TMA copies the barriers cost 484 cycles a block, and copies small
// enough for one group each kept their thread busy for 420.
// us at 8 / 24 / 64 tokens behind its norm, weights from memory: 6144 x 4096 9.7 / 10.0 / 10.6 (with codes by TMA, four warps and a store per value in the
// epilogue 11.0 / 13.3 / 17.4), 4096 x 4096 7.4 / 7.9 / 10.5 (10.0 / 12.3 / 15.8), 24576 x 4096 18.6 / 19.4 / 25.1 (20.5 / 28.3 / 42.2), 4096 x 12288 12.7 / 13.9 / 16.3
// (13.5 / 16.2 / 21.1).
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
constexpr int kGbMaxActs = 12;                         // stages of activations (128 inputs)
constexpr int kGbEpiWarp = 4 * kGbGroups, kGbMmaWarp = kGbEpiWarp + 4, kGbCodeWarp = kGbMmaWarp + kGbIssuers, kGbActWarp = kGbCodeWarp + 1;
constexpr int kGbThreads = (kGbActWarp + 1) * 32;
constexpr int kGbMaxSplit = 8;
// Accumulators behind the operand slots, 128 columns: one per issuer, two sets up to 32 tokens.  A slot and a stage of activations always
// meet the same issuer (a wait must not be more than a phase behind its barrier): their numbers are multiples of the issuers.
constexpr int kGbAccCol = kGbSlots * 64;
// What shared memory holds beside the exchange.
__host__ __device__ inline int gb_act_stages(int tok) { return tok == 64 ? 8 : 12; }
// Tokens that a CTA of a cluster finishes: whole groups of four, which travel as one 16-byte store.
__host__ __device__ inline int gb_share(int T, int split) { return ((T + split - 1) / split + 3) & ~3; }

struct GbParams {
  const uint4* codes;      // planar rows of K / 4 bytes
  const __half* scales;
  float* out_f32;          // epi 0, 1
  const float* residual;   // epi 1
  __half* out_f16;         // epi 2: SwiGLU over interleaved gate / up rows, paired-K order
  int* status;
  int n_rows, K, T, epi, out_ld, split, tok;           // tok: T rounded up to 16, 32 or 64
  int first[kGbMaxSplit + 1];                          // CTA i of a cluster takes the 128-input blocks first[i] .. first[i + 1] - 1
  uint32_t up[8];                                      // powers of two: see the expansion
};

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
__device__ __forceinline__ void gb_st_remote4(uint32_t addr, const uint32_t* v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void gb_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool gb_test(uint64_t* bar, uint32_t parity) {      // asks and does not wait
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(tc::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void gb_prefetch(const CUtensorMap* map, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
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
                                                                     const __grid_constant__ GbParams p) {
  extern __shared__ uint8_t gb_smem[];
  uint8_t* sB = (uint8_t*)(((uintptr_t)gb_smem + 1023) & ~(uintptr_t)1023);  // activations
  const int nA = gb_act_stages(p.tok), act_bytes = p.tok * 256;
  float* sR = reinterpret_cast<float*>(sB + nA * act_bytes);                 // partial sums [2][split][share of the tokens / 4][128 rows][4]
  __shared__ uint64_t a_full[kGbMaxActs], a_empty[kGbMaxActs], full[kGbSlots], empty[kGbSlots], accf[2], acce[2], red[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_failed;
  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0), lane = t & 31;
  const int S = p.split, rank = blockIdx.x, cid = blockIdx.y, nclusters = gridDim.y;
  const int groups = p.K >> 7, row_tiles = (p.n_rows + 127) >> 7;
  const int g0 = p.first[rank], nb = p.first[rank + 1] - g0;                // this CTA's 128-input blocks of every tile
  const int share = gb_share(p.T, S);                                      // tokens that a CTA of the cluster finishes
  const int sets = p.tok <= 32 ? 2 : 1;                                    // of accumulators
  // Blocks are numbered through over the CTA's tiles: block `it` goes through group it % 3, slot it % 6, issuer it % 2.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // Expanders: thread = weight row of the tile.  Codes and scales come straight to the thread that expands them, the next block's while this one is
  // expanded, and the first before anything is set up; warp 18 brings all of the CTA's share into L2.
  int tile = cid, kb = warp >> 2;             // the group's next block
  const uint4* code_at = p.codes;
  const __half* scale_at = p.scales;
  auto settle = [&] {                         // (tile, kb) and the addresses, kb counted from the tile's first block
    while (kb >= nb) { kb -= nb; tile += nclusters; }
    if (tile < row_tiles) {
      const size_t row = min(tile * 128 + (t & 127), p.n_rows - 1);
      code_at = p.codes + row * (size_t)(2 * groups) + 2 * (g0 + kb);
      scale_at = p.scales + row * groups + g0 + kb;
    }
  };
  uint4 code0 = make_uint4(0u, 0u, 0u, 0u), code1 = code0;
  __half scale = __float2half(0.0f);
  auto request = [&] {
    code0 = __ldg(code_at);
    code1 = __ldg(code_at + 1);
    scale = __ldg(scale_at);
  };
  if (warp < kGbEpiWarp) {
    settle();
    if (tile < row_tiles) request();
  }
  if (warp == kGbMmaWarp) {
    tc::tmem_alloc(&tmem_slot, 512);
    tc::tmem_relinquish();
  }
  if (t == 0) s_failed = 0;
  if (t < kGbMaxActs) {
    tc::mbar_init(&a_full[t], 1);
    tc::mbar_init(&a_empty[t], 1);
    if (t < kGbSlots) {
      tc::mbar_init(&full[t], 4);              // the expander warps of the group
      tc::mbar_init(&empty[t], 1);
    }
    if (t < 2) {
      tc::mbar_init(&accf[t], kGbIssuers);
      tc::mbar_init(&acce[t], 4);
      tc::mbar_init(&red[t], 4 * S);
    }
    tc::mbar_fence_init();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // met before the first exchange
  tc::tc_fence_after();
  const uint32_t taddr = tmem_slot;
  bool failed = false;

  if (warp == kGbCodeWarp) {
    if (tc::elect_one()) {
      for (int tl = cid; tl < row_tiles; tl += nclusters)
        for (int k = 0; k < nb; k += 4) gb_prefetch(&cmap, (g0 + k) * 8, tl * 128);
    }
    __syncwarp();
  } else if (warp == kGbActWarp) {
    if (tc::elect_one()) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
      asm volatile("griddepcontrol.wait;" ::: "memory");
      int s = 0, issued = 0;
      uint32_t phase = 1;
      for (int tl = cid; tl < row_tiles && !failed; tl += nclusters)
        for (int k = 0; k < nb; ++k, ++issued) {
          if (!tc::mbar_wait_sleep<100>(&a_empty[s], phase)) { failed = true; break; }
          tc::mbar_arrive_expect_tx(&a_full[s], act_bytes);
          gb_load3(sB + s * act_bytes, &xmap, (g0 + k) * 2, &a_full[s]);
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
      int s = me, as = me, seg = 0, k = me;              // slot, stage and block, two further each time
      uint32_t sphase = 0, aphase = 0;
      for (int tl = cid; tl < row_tiles && !failed; tl += nclusters, ++seg, k -= nb) {
        const int ab = sets == 2 ? seg & 1 : 0, use = sets == 2 ? seg >> 1 : seg;
        if (!tc::mbar_wait(&acce[ab], (use & 1) ^ 1)) { failed = true; break; }
        tc::tc_fence_after();
        const uint32_t acc = taddr + kGbAccCol + (ab * kGbIssuers + me) * p.tok;
        bool fresh = true;
        for (; k < nb; k += kGbIssuers) {
          // both barriers are asked before either answer is needed
          const bool there = gb_test(&a_full[as], aphase), filled = gb_test(&full[s], sphase);
          if ((!there && !tc::mbar_wait(&a_full[as], aphase)) || (!filled && !tc::mbar_wait(&full[s], sphase))) { failed = true; break; }
          tc::tc_fence_after();
          const uint64_t db = tc::smem_desc_sw128(tc::smem_u32(sB + as * act_bytes));
#pragma unroll
          for (uint32_t i = 0; i < 8; ++i)
            gb_mma(acc, taddr + s * 64 + i * 8, db + (i >> 2) * (uint32_t)(p.tok * 128 >> 4) + (i & 3) * 2, idesc, !(fresh && i == 0));
          fresh = false;
          tc::mma_commit(&empty[s]);
          tc::mma_commit(&a_empty[as]);
          if ((s += kGbIssuers) >= kGbSlots) { s -= kGbSlots; sphase ^= 1; }
          if ((as += kGbIssuers) >= nA) { as -= nA; aphase ^= 1; }
        }
        tc::mma_commit(&accf[ab]);
      }
      if (failed) atomicExch(p.status, 1);
    }
    __syncwarp();
  } else if (warp < kGbEpiWarp) {
    // What is not expansion costs as much as the expansion here - an instruction of a warp is some five cycles behind the one before it, a barrier
    // asked a hundred - so counters run along instead of being computed from the block's number, and barriers are asked before the answer is needed.
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    int s = warp >> 2;                          // operand slot: group and group + 3 in turn
    uint32_t sphase = 1;
    while (tile < row_tiles) {
      // A masked code is +-2^-7 or 0 and the scale is taken times 128; a row of the warp with a scale of 512 or more (none in earnest) takes the
      // other order, which leaves every f16 scale in range.  The shifts (by 12 - 4 i and 13 - 4 i) are products: the masks and counters already fill the
      // pipe that shifts run on (432 -> 390 cycles a block).
      const __half d = scale;
      const uint4 codes[2] = {code0, code1};
      const bool vacant = gb_test(&empty[s], sphase);
      kb += kGbGroups;
      code_at += 2 * kGbGroups;
      scale_at += kGbGroups;
      if (kb >= nb) settle();
      if (tile < row_tiles) request();
      auto block = [&](auto large) {
        const __half2 up = __half2half2(__float2half(128.0f)), d2 = large ? __half2half2(d) : __hmul2(__half2half2(d), up);
        auto weights = [&](uint32_t m) {
          const __half2 c = *reinterpret_cast<const __half2*>(&m), w = large ? __hmul2(__hmul2(c, up), d2) : __hmul2(c, d2);
          return *reinterpret_cast<const uint32_t*>(&w);
        };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t w4[4] = {codes[h].x, codes[h].y, codes[h].z, codes[h].w};
          uint32_t o[32];
#pragma unroll
          for (int wd = 0; wd < 4; ++wd)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              o[wd * 8 + i] = weights((w4[wd] * p.up[2 * i]) & 0xA000A000u);
              o[wd * 8 + 4 + i] = weights((w4[wd] * p.up[2 * i + 1]) & 0xA000A000u);
            }
          if (h == 0) {
            if (!__all_sync(0xffffffffu, vacant) && !__all_sync(0xffffffffu, tc::mbar_wait(&empty[s], sphase))) return false;
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
      if (s >= kGbGroups) { s -= kGbGroups; sphase ^= 1; }
      else s += kGbGroups;
    }
  }
  if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp < kGbMmaWarp) {
    // A tile's end is a chain (drain, exchange, sum, store): few, wide accesses and short loops.  Warps 12-15 take it beside the expansion of the next
    // tile; the last tile has the expanders' warps too, every group a quarter of the tokens.  us of 64 / 24 / 5 tokens with four warps for every tile, a
    // 4-byte store per value and loops unrolled over tokens: 6144 x 4096 16.2 / 12.3 / 10.0, 24576 x 4096 40.2 / 26.6 / 19.5.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int CB = 16;
    const int a = t & 127, part = warp >= kGbEpiWarp ? 0 : 1 + (warp >> 2);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const int tok_lo = rank * share, tok_hi = min(p.T, tok_lo + share), quads = share >> 2;
    const uint32_t share_inv = (65536u + share - 1) / share;      // c / share for c < 64
    const int last = (row_tiles - 1 - cid) / nclusters;            // the CTA's last tile, counted from 0
    for (int seg = part == 0 ? 0 : last; seg <= last; ++seg) {
      const int rb = seg & 1, ab = sets == 2 ? rb : 0, use = sets == 2 ? seg >> 1 : seg, row = (cid + seg * nclusters) * 128 + a;
      const int parts = seg == last ? 1 + kGbGroups : 1;
      const bool row_ok = row < p.n_rows;
      // the residuals of a group of four tokens are requested a group ahead, the first group's before the sums are there (they usually alias the outputs)
      float res[4];
      auto residuals = [&](int c) {
#pragma unroll
        for (int j = 0; j < 4; ++j) res[j] = row_ok && c + j < tok_hi ? p.residual[(size_t)(c + j) * p.out_ld + row] : 0.0f;
      };
      if (p.epi == 1) residuals(tok_lo + 4 * part);
      const float4* mine = reinterpret_cast<const float4*>(sR) + (size_t)rb * S * quads * 128 + a;
      if (part == 0 && !failed) failed = !tc::mbar_wait_warp<20>(&accf[ab], use & 1, lane);
      // The expanders have not followed the tiles before: their accumulator barrier may be phases ahead of what they could wait for.
      if (parts > 1) {                                               // all sixteen warps come here, whatever failed
        tc::tc_fence_before();
        asm volatile("bar.sync 2, %0;" ::"n"(kGbMmaWarp * 32) : "memory");
      }
      if (!failed) {
        tc::tc_fence_after();
        const uint32_t mine_at = tc::smem_u32(mine) + (uint32_t)(rank * quads) * 2048;
        const uint32_t acc = taddr + lanes + kGbAccCol + ab * kGbIssuers * p.tok;
        const int one = nb == 1 ? seg & 1 : 0;        // a tile of one block was in one issuer's accumulator only
#pragma unroll 1
        for (int c0 = CB * part; c0 < p.T; c0 += CB * parts) {
          uint32_t v[CB], w[CB];
          tc::tmem_ld16(acc + one * p.tok + c0, v);
          if (nb > 1) tc::tmem_ld16(acc + p.tok + c0, w);
          tc::tmem_wait_ld();
          if (nb > 1) {
#pragma unroll
            for (int j = 0; j < CB; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
          }
#pragma unroll
          for (int j = 0; j < CB; j += 4) {
            const int c = c0 + j, to = (int)((uint32_t)c * share_inv >> 16);
            const uint32_t at = mine_at + (uint32_t)((c - to * share) >> 2) * 2048;
            if (c < p.T) gb_st_remote4(gb_map(at, (uint32_t)to), v + j);
          }
        }
        tc::tc_fence_before();
        __syncwarp();
      }
      if (parts > 1) asm volatile("bar.sync 1, %0;" ::"n"(kGbMmaWarp * 32) : "memory");
      if (failed) continue;
      if (part == 0) {
        if (lane == 0) tc::mbar_arrive(&acce[ab]);
        if (lane < S) gb_arrive_remote(gb_map(tc::smem_u32(&red[rb]), (uint32_t)lane));
      }
      if (!__all_sync(0xffffffffu, gb_wait_cluster(&red[rb], (seg >> 1) & 1))) { failed = true; continue; }
      // this CTA's tokens, four at a time: partial sums in CTA order
#pragma unroll 1
      for (int c = tok_lo + 4 * part; c < tok_hi; c += 4 * parts) {
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const float4* src = mine + (size_t)((c - tok_lo) >> 2) * 128;
#pragma unroll 2
        for (int i = 0; i < S; ++i, src += quads * 128) {
          const float4 x = *src;
          v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
        if (p.epi == 2) {
          const bool odd = lane & 1;      // gate (even) and up (odd) rows are neighbouring lanes; each finishes every other token
          const int o = row >> 1;
          __half* dst = p.out_f16 + ((o & ~7) | ((o & 3) << 1) | ((o >> 2) & 1)) + (size_t)(c + odd) * p.out_ld;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float keep = odd ? v[2 * j + 1] : v[2 * j], other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * j] : v[2 * j + 1], 1);
            const float g = odd ? other : keep, u = odd ? keep : other;
            if (row_ok && c + 2 * j + odd < tok_hi) dst[(size_t)(2 * j) * p.out_ld] = __float2half_rn(g / (1.0f + __expf(-g)) * u);
          }
        } else {
          if (p.epi == 1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] += res[j];
            residuals(c + 4 * parts);
          }
          float* dst = p.out_f32 + (size_t)c * p.out_ld + row;
          if (row_ok) {
#pragma unroll
            for (int j = 0; j < 4; ++j, dst += p.out_ld)
              if (c + j < tok_hi) *dst = v[j];
          }
        }
      }
      __syncwarp();
    }
    if (failed && lane == 0) atomicExch(p.status, 1);
  }
  if (failed) s_failed = 1;
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (warp == kGbMmaWarp) tc::tmem_dealloc(taddr, 512);
  // Whoever has its last sums is written to no more and leaves; after an expired wait it stays until the others have left or wait here too.
  if (S > 1 && s_failed) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

static bool gb_maps(CUtensorMap* cmap, CUtensorMap* xmap, const void* codes, int n_rows, int K, const void* x, int x_ld, int T, int tok) {
  cuuint64_t cd[2] = {(cuuint64_t)K / 16, (cuuint64_t)n_rows}, cst[1] = {(cuuint64_t)K / 4};
  cuuint64_t xd[3] = {64, (cuuint64_t)T, (cuuint64_t)K / 64}, xst[2] = {(cuuint64_t)x_ld * 2, 128};      // [K / 64][T][64]
  cuuint32_t cbox[2] = {32, 128}, xbox[3] = {64, (cuuint32_t)tok, 2}, estr[3] = {1, 1, 1};
  return cuTensorMapEncodeTiled(cmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(codes), cd, cst, cbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
         cuTensorMapEncodeTiled(xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), xd, xst, xbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static size_t gb_smem_bytes(int tok, int split) {
  const int share = gb_share(tok, split);
  return 1024 + (size_t)gb_act_stages(tok) * tok * 256 + (size_t)2 * split * share * 128 * sizeof(float);
}

static cudaLaunchConfig_t gb_config(cudaLaunchAttribute* attr, int clusters, int split, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split, clusters);
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
    // Rounds of tiles times the 128-input blocks that a CTA goes through, plus what a tile costs whatever its depth (accumulator drain and
    // exchange, six blocks' time), and for the cluster's size what waiting for one more CTA costs: 1.5 blocks' time, 2.8 with the 33 to 64 tokens' sums to
    // exchange, where more than four CTAs never paid.  us by split 1 / 2 / 3 / 4 / 6 behind the norm at 8 tokens: 6144 x 4096 13.0 / 9.7 / 13.1 / 9.4 / 10.2;
    // 24576 x 4096 22.0 / 18.6 / 20.3 / 20.6 / 26.4; 4096 x 12288 28.6 / 17.9 / 16.2 / 12.7 / 16.0; 2560 x 4096 13.0 / 9.2 / 8.0 / 6.9 / 7.0; 2560 x 9728 23.7 / 15.1 / 12.5 /
    // 10.9 / 10.1; at 64 tokens 2560 x 4096 14.3 / 10.3 / 9.4 / 8.5 / 10.3, 2560 x 9728 25.6 / 16.4 / 14.9 / 11.8 / 14.2.  A tensor-core sum is cut off where
    // f32 would round it, so that more CTAs have less error (4096 x 12288, normal inputs: 5.9 / 2.8 / 1.8 / 1.4 / 0.9e-6 of the result by split 1 / 2 / 3 / 4 / 6).
    long long best = -1;
    for (int s = 1; s <= (T > 32 && most > 4 ? 4 : most); ++s) {
      if (held[s] < 1) continue;
      const long long rounds = (tiles + held[s] - 1) / held[s], cost = 10 * rounds * ((groups + s - 1) / s + 6) + (T > 32 ? 28 : 15) * s;
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
  GbParams p{(const uint4*)codes, (const __half*)scales, out_f32, residual, (__half*)out_f16, status, n_rows, K, T, epi, out_ld, split, tok, {}, {1u << 12, 1u << 13, 1u << 8, 1u << 9, 1u << 4, 1u << 5, 1u, 2u}};
  for (int i = 0; i <= split; ++i) p.first[i] = i * groups / split;
  cudaLaunchAttribute attr[2];
  const int clusters = tiles < held[split] ? tiles : held[split];
  // the request is that of 64 tokens, so that one CTA has an SM whatever the batch is
  cudaLaunchConfig_t cfg = gb_config(attr, clusters, split, gb_smem_bytes(64, split), stream);
  return cudaLaunchKernelEx(&cfg, bitgemm_batch_kernel, cmap, xmap, p) == cudaSuccess ? BONSAI_CUDA_OK : BONSAI_CUDA_LAUNCH_FAILED;
}

}  // extern "C"
