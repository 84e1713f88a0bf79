// Gate / up projections of prefill-sized batches on SM pairs (tcgen05, cta_group::2):  Out[token, n] = silu(X Wg^T) * (X Wu^T).
//
// Why pairs.  A gate / up tile of one SM has two accumulators, which leave TMEM for 128 tokens with double buffering: per 64 k-columns its MMAs read 64 KB of
// operands from shared memory and TMA writes 48 KB there, 900 cycles of shared memory for 512 of the tensor core (912 TFLOP/s measured).  Here two CTAs of
// a cluster work on a tile of 256 features and up to 256 tokens: each holds the weights of 128 features (gate and up rows: two MMAs) and HALF of the token rows,
// and the pair's MMA reads both halves, so a token row is staged once for 256 features: 900 cycles of shared memory for 1024 of the tensor core.  The
// accumulators fill TMEM; eight epilogue warps take everything out of it before they store, so that the next tile starts early.  12288 features, k = 4096:
// 8300 tokens 1765 -> 1205 us (1386 TFLOP/s), 3000 tokens 675 -> 492 us, 768 tokens 168 -> 120 us, 129 tokens 84 -> 64 us (pair_pays: where it is the faster form).
// (Products with one accumulator stay on the kernel of gemm_tc.cu, whose 256-token tile is not bound by shared memory: 8300 tokens by 6144 features 311 us there,
// 328 us in this form, which starts 4 us later, behind the cluster's barriers.)
//
// Roles of a CTA (320 threads): warp 0 producer (TMA; both CTAs' loads report to the leader's barrier), warp 1 MMA issuer (leader CTA only; its commits
// arrive in both CTAs), warps 2-9 epilogue (lane quarter warp % 4, token half (warp - 2) / 4 of the CTA's own accumulators).  All waits are bounded.
//
// Tile order: eight token tiles (X of 8 tn tokens, at most 2048, which stay in L2) are walked for one block of features before the next block, so that the weights
// stream from memory once per 8 tn tokens.
#pragma once
#include "sm100.cuh"
#include "host_common.h"

namespace gb {

constexpr int kPairThreads = 320;
constexpr int kPairTN = 256;              // most tokens of a tile
constexpr int kPairStages = 4;
constexpr int kPairGroup = 8;             // token tiles walked per block of features

struct PairArgs {
  int n_blocks, tok_tiles, tn, m_tok, num_kb;
  int up_row_offset;                      // first "up" row
  __nv_bfloat16* out; int ldo; size_t out_bytes;
  int w_tiled;
  KernelStatus* status;
};

__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" :: "r"(bar) : "memory");
}
// Into this CTA's shared memory; the bytes count on a barrier of the pair (shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               :: "r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void mma_f16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               :: "r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrive on the barrier at this offset in both CTAs once the MMAs issued so far have finished.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               :: "r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const PairArgs args) {
  constexpr int TILE_BYTES = 128 * 128;                 // 128 rows x 64 bf16
  constexpr int STAGE_BYTES = 3 * TILE_BYTES;           // gate rows, up rows, tokens
  constexpr int S = kPairStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + S * STAGE_BYTES);   // [S] of the leader: one arrival + the bytes of both CTAs
  uint64_t* empty_bar = full_bar + S;                          // [S] per CTA: commit
  uint64_t* accf_bar = empty_bar + S;                          // per CTA: commit
  uint64_t* acce_bar = accf_bar + 1;                           // of the leader: 8 warps of both CTAs
  uint32_t* tmem_slot = (uint32_t*)(acce_bar + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int n_tiles = args.n_blocks * args.tok_tiles;
  const int pair0 = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(accf_bar, 1); mbar_init(acce_bar, 16);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  pair_sync();                                         // both CTAs' barriers and TMEM exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  struct PTile { int nb, x_row0, valid, width; };      // width: token columns of the MMA (valid, in steps of 32)
  auto tile_at = [&](int t) {
    const int per = kPairGroup * args.n_blocks, g = t / per;
    const int gt = min(kPairGroup, args.tok_tiles - g * kPairGroup), r = t - g * per;
    PTile o;
    o.nb = r / gt;
    o.x_row0 = (g * kPairGroup + r % gt) * args.tn;
    o.valid = min(args.tn, args.m_tok - o.x_row0);
    o.width = (o.valid + 31) & ~31;
    return o;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one lane of either CTA)
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      bool ok = true;
      for (int ti = pair0; ok && ti < n_tiles; ti += n_pairs) {
        const PTile t = tile_at(ti);
        const int w0 = t.nb * 256 + (int)rank * 128, w1 = args.up_row_offset + w0;
        const int y0 = ((w0 >> 7) * args.num_kb) << 7, y1 = ((w1 >> 7) * args.num_kb) << 7;       // tiled weights: rows of 16 KB blocks
        const int xr = t.x_row0 + (int)rank * (t.width >> 1);
        for (int kb = 0; kb < args.num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, args.status, 1400, s)) { ok = false; break; }
          uint8_t* st = smem + s * STAGE_BYTES;
          const uint32_t bar = map_to_cta(smem_u32(&full_bar[s]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
          if (args.w_tiled) {
            tma_load_2d_pair(st, &tmW, bar, 0, y0 + (kb << 7));
            tma_load_2d_pair(st + TILE_BYTES, &tmW, bar, 0, y1 + (kb << 7));
          } else {
            tma_load_2d_pair(st, &tmW, bar, kb * 64, w0);
            tma_load_2d_pair(st + TILE_BYTES, &tmW, bar, kb * 64, w1);
          }
          tma_load_2d_pair(st + 2 * TILE_BYTES, &tmX, bar, kb * 64, xr);
          if (++s == S) { s = 0; ph ^= 1; }
        }
      }
      // the last commits arrive in both CTAs: neither may leave before they have
      for (int i = 0; ok && i < S; ++i) {
        if (!mbar_wait(&empty_bar[s], ph ^ 1, abort_flag, args.status, 1401, s)) ok = false;
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (one lane of the leader)
    if (lane == 0 && rank == 0) {
      int s = 0; uint32_t ph = 0, acc_ph = 0;
      bool ok = true;
      for (int ti = pair0; ok && ti < n_tiles; ti += n_pairs) {
        const PTile t = tile_at(ti);
        const uint32_t idesc = make_idesc(256, t.width, 1, 1);
        if (!mbar_wait(acce_bar, acc_ph ^ 1, abort_flag, args.status, 1410)) { ok = false; break; }
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
        tc_fence_after();
        for (int kb = 0; kb < args.num_kb; ++kb) {
          if (!mbar_wait(&full_bar[s], ph, abort_flag, args.status, 1411, s)) { ok = false; break; }
          tc_fence_after();
          const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t a0 = make_sdesc_sw128(st), b = make_sdesc_sw128(st + 2 * TILE_BYTES);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            mma_f16_pair(tmem_base, sdesc_at(a0, j * 32), sdesc_at(b, j * 32), idesc, (kb > 0 || j > 0) ? 1u : 0u);
            mma_f16_pair(tmem_base + kPairTN, sdesc_at(a0, TILE_BYTES + j * 32), sdesc_at(b, j * 32), idesc, (kb > 0 || j > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty_bar[s]);
          if (++s == S) { s = 0; ph ^= 1; }
        }
        if (!ok) break;
        tc_commit_pair(accf_bar);
        acc_ph ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (8 warps)
    const int q = warp & 3, c0 = ((warp - 2) >> 2) * 128;
    uint32_t acc_ph = 0;
    for (int ti = pair0; ti < n_tiles; ti += n_pairs) {
      const PTile t = tile_at(ti);
      if (!__all_sync(0xffffffffu, mbar_wait(accf_bar, acc_ph, abort_flag, args.status, 1420))) break;
      tc_fence_after();
      const uint32_t tacc = tmem_base + c0 + ((uint32_t)(q * 32) << 16);
      const int n = t.nb * 256 + (int)rank * 128 + q * 32 + lane;
      const int live = min(128, t.valid - c0);              // token columns of this warp (may be <= 0)
      uint32_t pk[64];                                      // two tokens each
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        if (c < live) {                                     // uniform over the warp
          uint32_t g[32], u[32];
          tmem_ld_x32(tacc + c, g);
          tmem_ld_x32(tacc + kPairTN + c, u);
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float g0 = __uint_as_float(g[2 * j]), g1 = __uint_as_float(g[2 * j + 1]);
            pk[c / 2 + j] = pack_bf16x2(g0 / (1.0f + __expf(-g0)) * __uint_as_float(u[2 * j]), g1 / (1.0f + __expf(-g1)) * __uint_as_float(u[2 * j + 1]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(acce_bar), 0));
      acc_ph ^= 1;
      const size_t off0 = ((size_t)t.x_row0 + c0) * args.ldo + n;
      if (live > 0 && (off0 + (size_t)(live - 1) * args.ldo + 1) * 2 > args.out_bytes) {
        report_status(args.status, ST_BAD_ARG, 1430, t.x_row0 + c0, n, ti);
        continue;
      }
      unsigned short* o = (unsigned short*)args.out + off0;
#pragma unroll
      for (int i = 0; i < 64; ++i) {
        if (2 * i < live) o[(size_t)(2 * i) * args.ldo] = (unsigned short)(pk[i] & 0xffffu);
        if (2 * i + 1 < live) o[(size_t)(2 * i + 1) * args.ldo] = (unsigned short)(pk[i] >> 16);
      }
    }
  }

  if (*abort_flag) {                                        // copies may still be landing: bounded grace period
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  pair_sync();                                              // no MMA or arrival of the pair is under way any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" :: "r"(tmem_base) : "memory");
  }
}

// Tokens of a tile: the even cut whose rounds of tiles cost least.  A step of 64 k-columns takes four cycles of the tensor core per token, or 512 + 1.5 per
// token of shared memory, which is more below 205 tokens (320 tokens by 12288 features: two tiles of 160, not one of 256 and one of 64, 112 -> 102 us).
inline int pair_tile_tokens(int m_tok, int n_blocks, int pairs) {
  int best = kPairTN;
  long best_cost = -1;
  for (int tiles = (m_tok + kPairTN - 1) / kPairTN; tiles <= (m_tok + 95) / 96; ++tiles) {
    const int tn = ((m_tok + tiles - 1) / tiles + 31) & ~31;
    const long n = (long)n_blocks * ((m_tok + tn - 1) / tn);
    const long cost = (n + pairs - 1) / pairs * (4 * tn > 512 + 3 * tn / 2 ? 4 * tn : 512 + 3 * tn / 2);
    if (best_cost < 0 || cost < best_cost) { best = tn; best_cost = cost; }
  }
  return best;
}

// Whether the pair form is the faster one of a gate / up projection (`n_out` features of `k`), against one SM per 128 features and 128 tokens.
// Both forms timed in turn, in streams of launches that find their weights in memory: 512 to 25600 features, k 512 to 8192, 65 to 3000 tokens (us, one SM / pairs).
//  * Up to 96 tokens: one SM (3072 x 1024, 65 tokens: 20.6 / 23.8; 12288 x 4096, 80 tokens: 54.9 / 58.9).
//  * One round of tiles in either form: pairs, which end earlier, in the readout (3072 x 1024, 256 tokens: 23.6 / 21.3).  Not for long k, where their longer steps
//    outweigh that (2048 x 8192, 384 tokens: 80.4 / 81.0), nor where single tiles fill the SMs (6144 x 2048, 320 tokens: 33.3 / 34.0) or up to 128 tokens stay one tile
//    (10240 x 2560, 112 tokens: 41.1 / 45.1).
//  * More rounds: a round of pairs costs 1.17 (160 tokens) to 1.30 (256) of a round of single tiles (12288 x 4096: 320 tokens, two rounds each, 90 / 101; 512 tokens,
//    three and two, 127 / 104; 25600 x 5120, 256 tokens, three and two, 185 / 143).
// Over those 502 sizes the choice takes 0.1 % longer than the better form of each, at worst 6 %.
inline bool pair_pays(int n_out, int k, int m_tok, int sms) {
  if (m_tok <= 96) return false;
  const int pairs = sms / 2, n_blocks = n_out / 256, tn = pair_tile_tokens(m_tok, n_blocks, pairs);
  const long single = 2l * n_blocks * ((m_tok + 127) / 128), single_rounds = (single + sms - 1) / sms;
  const long rounds = ((long)n_blocks * ((m_tok + tn - 1) / tn) + pairs - 1) / pairs;
  if (single_rounds == 1 && rounds == 1) return k <= 4096 && single <= 128 && (m_tok > 128 || tn <= 64);
  return rounds * (95000 + 137 * tn) < 100000 * single_rounds;
}

// n_out a multiple of 256; tmW as gemm_tc.cu builds it, tmX with a box of 128 rows.
static int launch_gemm_pair(const CUtensorMap& tmW, const CUtensorMap& tmX, int n_out, PairArgs a, cudaStream_t stream) {
  const int smem = kPairStages * 3 * 16384 + 1024 + 256;
  static bool attr_set = false;
  if (!attr_set) {
    GB_CUDA_OK(cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set = true;
  }
  const int sm_pairs = sm_count() / 2;
  a.n_blocks = n_out / 256;
  a.tn = pair_tile_tokens(a.m_tok, a.n_blocks, sm_pairs);
  a.tok_tiles = (a.m_tok + a.tn - 1) / a.tn;
  const int tiles = a.n_blocks * a.tok_tiles;
  const int pairs = tiles < sm_pairs ? tiles : sm_pairs;
  GB_CUDA_OK(launch_k_cluster(gemm_pair_kernel, dim3(2 * pairs), dim3(kPairThreads), smem, stream, 2u, tmW, tmX, a));
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace gb
