// Fused dequant-GEMM for ggml-quantised weights (Q4_K, Q8_0) that stay quantised in HBM:
//   out[token, n] = sum_k W[n, k] * x[token, k],  five tokens and more (prefill, batched decode).
//
// The quantised blocks never become a bf16 matrix in memory.  Per 128-row x 256-column tile of W (one contiguous piece of the
// tiled layout of ops/ggml_torch.py) a bulk copy brings the raw blocks into shared memory; sixteen warps unpack them in registers
// (nibbles -> bf16 pairs with byte permutes, d * sc and dmin * m applied per 32-wide sub-block in packed bf16 arithmetic; int8 ->
// fp32 -> bf16 for Q8_0) and write the result straight into the 128-byte-swizzled K-major operand tile that tcgen05.mma reads;
// the tokens come in by TMA; the accumulator lives in TMEM.  Orientation as in the dense GEMM: W is the MMA A operand (128 rows
// = 128 TMEM lanes), the tokens are N (16 .. 128 per tile).
//
// Warp roles of a CTA (704 threads): warp 0 producer (bulk copies of raw tiles, TMA loads of token tiles), warp 1 MMA issuer,
// warps 2-5 epilogue (TMEM -> registers -> global), warps 6-21 unpack (a thread per 32-value sub-block and row).  Rings: raw tiles (2-4, what shared memory leaves), bf16 operand tiles of 128 x 128
// (2), token tiles (2-3), accumulators (2); all waits are bounded and report into the status word.
//
// A raw Q4_K tile is 18 KB for 64 KB of bf16 operand: at decode sizes the kernel is bound by the HBM stream of the quantised
// bytes, not by the four times larger operand it feeds to the tensor core.
//
// Replaces in the reference: mmq_q4_K_grouped and the other mma.sync MMQ kernels (cuda/llm/cuda_llm_runner.c:5295-7329,
// mmq/mmq_q4_K_test.cu:17-24 describes the scale handling), the dequant_*_to_f16 + cuBLAS pairs (:999-5447, :15488-17418) and
// batch_matvec_q4_K / q8_0 (:4433-4854); CPU oracle gemm_*_tokmajor of common/ggml_dequant.h:298-349.
#include "sm100.cuh"
#include "host_common.h"
#include <cuda_bf16.h>

namespace gb {

constexpr int kQgThreads = 704;
constexpr int kQgUnpackWarp0 = 6;          // first unpack warp
constexpr int kQgUnpackThreads = 512;   // 16 warps: a thread unpacks one 32-value sub-block of one row
constexpr int kQgA = 128 * 256;            // bytes of one bf16 operand stage: 2 atoms of [128 rows][64 k]

struct QGemmArgs {
  const uint8_t* w;                 // tiled weights [row_tiles][num_kb][tile bytes]
  void* out; int ldo; int out_f32;
  const float* bias;
  int n_out, m_tok, num_kb, row_tiles, tok_tiles;
  int splits, kb_per;            // K splits per output tile (>= 1) and 256-column blocks per split
  long partial_stride;           // splits > 1: split ks stores its fp32 partial at out + ks * partial_stride (elements)
  int b_stages, raw_stages;
  KernelStatus* status;
};

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { return __byte_perm(a, b, sel); }

// One 32-value sub-block of a Q4_K chunk: the low (nib = 0) or high (nib = 1) nibbles of the 32 bytes `q0 q1`, scale a = d * sc
// and offset b = dmin * m  ->  four 16-byte chunks of bf16 (values 32 * nib + 8c .. + 7, c < 4) in the swizzled operand row.
__device__ __forceinline__ void unpack_q4k_sub(const uint4 q0, const uint4 q1, int nib, float a, float b, uint8_t* dst_row, int row) {
  const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
  const __nv_bfloat162 sixteen = __float2bfloat162_rn(16.0f);
  const __nv_bfloat162 a2 = __float2bfloat162_rn(a), b2 = __float2bfloat162_rn(-b);
  const int sh = nib ? 1 : 0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 o;
    uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      // bf16(16 + q) = 0x4180 | (q << 3): exact for q < 16; the low byte carries 0x80 | q << 3, the high byte is 0x41
      const uint32_t x = w[2 * c + u];
      const uint32_t n3 = ((sh ? (x >> 1) : (x << 3)) & 0x78787878u) | 0x80808080u;
      uint32_t p0 = prmt(n3, 0x41414141u, 0x4140), p1 = prmt(n3, 0x41414141u, 0x4342);
      __nv_bfloat162 x0 = *reinterpret_cast<__nv_bfloat162*>(&p0), x1 = *reinterpret_cast<__nv_bfloat162*>(&p1);
      x0 = __hfma2(__hsub2(x0, sixteen), a2, b2);            // q * a - b, one rounding
      x1 = __hfma2(__hsub2(x1, sixteen), a2, b2);
      po[2 * u] = *reinterpret_cast<uint32_t*>(&x0); po[2 * u + 1] = *reinterpret_cast<uint32_t*>(&x1);
    }
    *reinterpret_cast<uint4*>(dst_row + (((4 * nib + c) ^ (row & 7)) << 4)) = o;
  }
}

// One Q8_0 block (32 int8 in two 16-byte vectors, scale d) -> four swizzled 16-byte chunks of bf16 (chunk index 4 * nib + c).
__device__ __forceinline__ void unpack_q80_sub(const uint4 qa, const uint4 qb, int nib, float d, uint8_t* dst_row, int row) {
  const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 o;
    uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t x = w[2 * c + u];
      const float f0 = (float)(int)(int8_t)(x & 0xff), f1 = (float)(int)(int8_t)((x >> 8) & 0xff);
      const float f2 = (float)(int)(int8_t)((x >> 16) & 0xff), f3 = (float)(int)(int8_t)(x >> 24);
      po[2 * u] = pack_bf16x2(f0 * d, f1 * d); po[2 * u + 1] = pack_bf16x2(f2 * d, f3 * d);
    }
    *reinterpret_cast<uint4*>(dst_row + (((4 * nib + c) ^ (row & 7)) << 4)) = o;
  }
}

// TYPE: 0 = Q4_K, 1 = Q8_0.  TN: token tile.
template <int TYPE, int TN>
__global__ void __launch_bounds__(kQgThreads, 1)
qgemm_kernel(const __grid_constant__ CUtensorMap tmX, const QGemmArgs args) {
  constexpr int RAW = TYPE == 0 ? 128 * 144 : 128 * 272;                 // bytes of a raw tile (Q8_0 row: 256 values + 8 f16 scales)
  constexpr int RAW_PAD = (RAW + 1023) & ~1023;
  constexpr int B_BYTES = TN * 256;                                      // token stage: 2 atoms of [TN rows][64 k]
  constexpr int TMEM_COLS = 2 * TN < 32 ? 32 : 2 * TN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int BS = args.b_stages, RS = args.raw_stages;
  uint8_t* rawb = smem;                                  // [RS][RAW_PAD]
  uint8_t* Ab = rawb + (size_t)RS * RAW_PAD;             // [2][kQgA]
  uint8_t* Bb = Ab + 2 * kQgA;                           // [BS][B_BYTES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(Bb + (size_t)BS * B_BYTES);
  uint64_t* raw_full = bars;            // [4]
  uint64_t* raw_empty = bars + 4;       // [4]  8 arrivals (unpack warps)
  uint64_t* a_full = bars + 8;          // [2]  8 arrivals
  uint64_t* a_empty = bars + 10;        // [2]  1 (tcgen05.commit)
  uint64_t* b_full = bars + 12;         // [4]
  uint64_t* b_empty = bars + 16;        // [4]  1 (commit)
  uint64_t* accf = bars + 20;           // [2]
  uint64_t* acce = bars + 22;           // [2]  4 arrivals (epilogue warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 24);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = args.row_tiles * args.tok_tiles * args.splits;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&a_full[i], kQgUnpackThreads / 32); mbar_init(&a_empty[i], 1); mbar_init(&accf[i], 1); mbar_init(&acce[i], 4); }
    for (int i = 0; i < 4; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kQgUnpackThreads / 32); mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      int rs = 0; uint32_t rph = 0; int bs = 0; uint32_t bph = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        const int ksp = t % args.splits, tt = t / args.splits;
        const int rt = tt % args.row_tiles, tb = tt / args.row_tiles;
        const uint8_t* wt = args.w + (size_t)rt * args.num_kb * RAW;
        const int kb0 = ksp * args.kb_per, kb1 = min(args.num_kb, kb0 + args.kb_per);
        for (int kb = kb0; ok && kb < kb1; ++kb) {
          if (!mbar_wait(&raw_empty[rs], rph ^ 1, abort_flag, args.status, 1200, rs)) { ok = false; break; }
          mbar_expect_tx(&raw_full[rs], RAW);
          bulk_load(rawb + (size_t)rs * RAW_PAD, wt + (size_t)kb * RAW, RAW, &raw_full[rs]);
          if (++rs == RS) { rs = 0; rph ^= 1; }
          for (int h = 0; h < 2; ++h) {
            if (!mbar_wait(&b_empty[bs], bph ^ 1, abort_flag, args.status, 1201, bs)) { ok = false; break; }
            mbar_expect_tx(&b_full[bs], B_BYTES);
            uint8_t* dst = Bb + (size_t)bs * B_BYTES;
            const int kx = kb * 256 + h * 128;
            tma_load_2d(dst, &tmX, &b_full[bs], kx, tb * TN);
            tma_load_2d(dst + TN * 128, &tmX, &b_full[bs], kx + 64, tb * TN);
            if (++bs == BS) { bs = 0; bph ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int as = 0; uint32_t aph = 0; int bs = 0; uint32_t bph = 0; int acc = 0; uint32_t acc_ph = 0;
      bool ok = true;
      constexpr uint32_t idesc = make_idesc(128, TN, 1, 1);
      for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        if (!mbar_wait(&acce[acc], acc_ph ^ 1, abort_flag, args.status, 1210, acc)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d0 = tmem_base + acc * TN;
        const int kb0 = (t % args.splits) * args.kb_per, nkb = min(args.num_kb, kb0 + args.kb_per) - kb0;
        for (int ks = 0; ok && ks < 2 * nkb; ++ks) {
          if (!mbar_wait(&a_full[as], aph, abort_flag, args.status, 1211, as)) { ok = false; break; }
          if (!mbar_wait(&b_full[bs], bph, abort_flag, args.status, 1212, bs)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a0 = smem_u32(Ab + (size_t)as * kQgA), b0 = smem_u32(Bb + (size_t)bs * B_BYTES);
#pragma unroll
          for (int at = 0; at < 2; ++at)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              mma_f16_ss(d0, make_sdesc_sw128(a0 + at * (128 * 128) + j * 32), make_sdesc_sw128(b0 + at * (TN * 128) + j * 32), idesc,
                         (ks > 0 || at > 0 || j > 0) ? 1u : 0u);
          tc_commit(&a_empty[as]);
          tc_commit(&b_empty[bs]);
          if (++as == 2) { as = 0; aph ^= 1; }
          if (++bs == BS) { bs = 0; bph ^= 1; }
        }
        if (!ok) break;
        tc_commit(&accf[acc]);
        if (++acc == 2) { acc = 0; acc_ph ^= 1; }
      }
    }
  } else if (warp < kQgUnpackWarp0) {
    // ------------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;
    const int row = q * 32 + lane;
    int acc = 0; uint32_t acc_ph = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
      const int ksp = t % args.splits, tt = t / args.splits;
      const int rt = tt % args.row_tiles, tb = tt / args.row_tiles;
      if (!mbar_wait(&accf[acc], acc_ph, abort_flag, args.status, 1220, acc)) { ok = false; break; }
      tc_fence_after();
      const uint32_t tacc = tmem_base + acc * TN + ((uint32_t)(q * 32) << 16);
      const int n = rt * 128 + row;
      const bool n_ok = n < args.n_out;
      const float bias = (args.bias != nullptr && n_ok && ksp == 0) ? args.bias[n] : 0.f;
      const int tok0 = tb * TN, valid = min(TN, args.m_tok - tok0);
      const size_t part = (size_t)ksp * (size_t)args.partial_stride;
#pragma unroll 1
      for (int c = 0; c < TN; c += 16) {
        uint32_t r[16];
        __syncwarp();                                      // rows past n_out left the round before early
        tmem_ld_x16(tacc + c, r);
        tc_wait_ld();
        if (c >= valid || !n_ok) continue;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j >= valid) break;
          const float v = __uint_as_float(r[j]) + bias;
          const size_t off = part + (size_t)(tok0 + c + j) * args.ldo + n;
          if (args.out_f32) reinterpret_cast<float*>(args.out)[off] = v;
          else reinterpret_cast<__nv_bfloat16*>(args.out)[off] = __float2bfloat16(v);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acce[acc]);
      if (++acc == 2) { acc = 0; acc_ph ^= 1; }
    }
  } else {
    // ------------------------------------------------------------------ unpack (warps 6..21): raw blocks -> swizzled bf16 operand
    const int ut = threadIdx.x - kQgUnpackWarp0 * 32;     // 0..511
    const int row = ut >> 2, cpar = (ut >> 1) & 1, nib = ut & 1;       // item: sub-block (2j + nib) of row `row`, atom cpar of every stage
    int rs = 0; uint32_t rph = 0; int as = 0; uint32_t aph = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
      const int kb0 = (t % args.splits) * args.kb_per, kb1 = min(args.num_kb, kb0 + args.kb_per);
      for (int kb = kb0; ok && kb < kb1; ++kb) {
        if (!mbar_wait(&raw_full[rs], rph, abort_flag, args.status, 1230, rs)) { ok = false; break; }
        const uint8_t* rb = rawb + (size_t)rs * RAW_PAD;
        for (int h = 0; h < 2; ++h) {
          if (!mbar_wait(&a_empty[as], aph ^ 1, abort_flag, args.status, 1231, as)) { ok = false; break; }
          const int j = 2 * h + cpar;                      // 64-value chunk of the 256-column tile
          uint8_t* dst_row = Ab + (size_t)as * kQgA + cpar * (128 * 128) + row * 128;
          if (TYPE == 0) {
            const uint8_t* b = rb + row * 144;
            const uint4 hd = *reinterpret_cast<const uint4*>(b);
            const uint4 q0 = *reinterpret_cast<const uint4*>(b + 16 + 32 * j), q1 = *reinterpret_cast<const uint4*>(b + 32 + 32 * j);
            const __half2 dd = *reinterpret_cast<const __half2*>(&hd.x);
            const float d = __low2float(dd), dmin = __high2float(dd);
            const int bsh = 16 * cpar + 8 * nib;           // byte (2 * cpar + nib) of the scale words
            uint32_t sc, mn;
            if (h == 0) {                                  // sub-blocks 0..3: 6 bits straight from bytes 0..3 / 4..7
              sc = (hd.y >> bsh) & 63u; mn = (hd.z >> bsh) & 63u;
            } else {                                       // sub-blocks 4..7: low 4 bits in bytes 8..11, high 2 bits in the top of bytes 0..7
              const uint32_t x = (hd.w >> bsh) & 0xffu, y = (hd.y >> bsh) & 0xffu, z = (hd.z >> bsh) & 0xffu;
              sc = (x & 15u) | ((y >> 6) << 4); mn = (x >> 4) | ((z >> 6) << 4);
            }
            unpack_q4k_sub(q0, q1, nib, d * (float)sc, dmin * (float)mn, dst_row, row);
          } else {
            const uint4* qp = reinterpret_cast<const uint4*>(rb + row * 272 + 64 * j + 32 * nib);
            const __half dh = *reinterpret_cast<const __half*>(rb + row * 272 + 256 + (2 * j + nib) * 2);
            unpack_q80_sub(qp[0], qp[1], nib, __half2float(dh), dst_row, row);
          }
          fence_proxy_async_smem();                        // this thread's operand bytes -> visible to the tensor core
          __syncwarp();
          if (lane == 0) mbar_arrive(&a_full[as]);
          if (++as == 2) { as = 0; aph ^= 1; }
        }
        if (!ok) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[rs]);
        if (++rs == RS) { rs = 0; rph ^= 1; }
      }
    }
  }

  if (*abort_flag) {                                       // copies may still be landing: bounded grace period
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// ------------------------------------------------------------------------------------------------------------------------------------------
// More than 128 tokens.  The kernel above unpacks W anew for every 128 tokens, and writes it to shared memory for the MMAs to read back.  Here the unpacked operand
// never meets shared memory: sixteen warps (a thread per weight row and 64-value chunk) write it straight into TMEM (tcgen05.st) and the MMA takes its A operand
// from there; what shared memory keeps free holds token tiles of up to 256, so W is unpacked once per 256 tokens.  Same operands, same order of sums as above.
// 512 tokens by 51200 rows of 5120: 379 -> 247 us, by 5120 rows of 25600: 334 -> 188 us.
//
// TMEM: columns 0-255 the accumulator (token tiles are wider than 128: two would not fit), 256-511 four operand stages of 128 rows x 128 bf16 (64 columns each).
// Roles (864 threads): warp 0 producer of token tiles, warp 26 of raw tiles, warp 1 MMA issuer, warps 2-9 epilogue (token half (warp - 2) / 4), warps 10-25
// unpack: two groups of eight take the raw tiles in turn (one group alone: 5 to 10 % more), and each fills its own two operand stages.
constexpr int kQwThreads = 864;
constexpr int kQwA = 4;                    // operand stages in TMEM
// Stages of 64 token columns (32 KB each) and raw tiles (18 KB Q4_K, 34 KB Q8_0) in flight: what shared memory holds, the tokens' bytes first.
__host__ __device__ constexpr int qw_b_stages(int type) { return type == 0 ? 4 : 3; }
__host__ __device__ constexpr int qw_raw_stages(int type) { return type == 0 ? 4 : 3; }

struct QWideArgs {
  QGemmArgs g;
  int tn;                                  // tokens of a tile: a multiple of 16, from 144 to 256
};

template <int TYPE>
__global__ void __launch_bounds__(kQwThreads, 1)
qgemm_wide_kernel(const __grid_constant__ CUtensorMap tmX, const QWideArgs wargs) {
  constexpr int RAW = TYPE == 0 ? 128 * 144 : 128 * 272;
  constexpr int RAW_PAD = (RAW + 1023) & ~1023;
  constexpr int RS = qw_raw_stages(TYPE), BS = qw_b_stages(TYPE);
  const QGemmArgs& args = wargs.g;
  const int TN = wargs.tn, b_bytes = TN * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* Bb = smem;                                    // [BS][256 rows][128 B]
  uint8_t* rawb = smem + BS * 32768;                     // [RS][RAW_PAD]
  uint64_t* bars = reinterpret_cast<uint64_t*>(rawb + RS * RAW_PAD);
  uint64_t* raw_full = bars;            // [RS]
  uint64_t* raw_empty = raw_full + RS;  // [RS]  8 arrivals (unpack warps)
  uint64_t* a_full = raw_empty + RS;    // [kQwA]  8 arrivals
  uint64_t* a_empty = a_full + kQwA;    // [kQwA]  1 (commit)
  uint64_t* b_full = a_empty + kQwA;    // [BS]
  uint64_t* b_empty = b_full + BS;      // [BS]  1 (commit)
  uint64_t* accf = b_empty + BS;        // commit
  uint64_t* acce = accf + 1;            // 8 arrivals (epilogue warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acce + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = args.row_tiles * args.tok_tiles * args.splits;
  // token tiles vary fastest: the CTAs that run together share a tile of W
  auto tile_at = [&](int t, int& rt, int& tb, int& kb0, int& kb1) {
    const int ksp = t % args.splits, tt = t / args.splits;
    tb = tt % args.tok_tiles; rt = tt / args.tok_tiles;
    kb0 = ksp * args.kb_per; kb1 = min(args.num_kb, kb0 + args.kb_per);
    return ksp;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < RS; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 8); }
    for (int i = 0; i < kQwA; ++i) { mbar_init(&a_full[i], 8); mbar_init(&a_empty[i], 1); }
    for (int i = 0; i < BS; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
    mbar_init(accf, 1); mbar_init(acce, 8);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + 256;
  pdl_wait();
  pdl_trigger();

  if (warp == 0) {
    // ------------------------------------------------------------------ producer of token tiles
    if (lane == 0) {
      int bs = 0; uint32_t bph = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        int rt, tb, kb0, kb1;
        tile_at(t, rt, tb, kb0, kb1);
        for (int h = 4 * kb0; h < 4 * kb1; ++h) {
          if (!mbar_wait(&b_empty[bs], bph ^ 1, abort_flag, args.status, 1241, bs)) { ok = false; break; }
          mbar_expect_tx(&b_full[bs], b_bytes);
          tma_load_2d(Bb + bs * 32768, &tmX, &b_full[bs], h * 64, tb * TN);
          if (++bs == BS) { bs = 0; bph ^= 1; }
        }
      }
    }
  } else if (warp == 26) {
    // ------------------------------------------------------------------ producer of raw tiles
    if (lane == 0) {
      int rs = 0; uint32_t rph = 0;
      bool ok = true;
      for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        int rt, tb, kb0, kb1;
        tile_at(t, rt, tb, kb0, kb1);
        const uint8_t* wt = args.w + (size_t)rt * args.num_kb * RAW;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&raw_empty[rs], rph ^ 1, abort_flag, args.status, 1240, rs)) { ok = false; break; }
          mbar_expect_tx(&raw_full[rs], RAW);
          bulk_load(rawb + rs * RAW_PAD, wt + (size_t)kb * RAW, RAW, &raw_full[rs]);
          if (++rs == RS) { rs = 0; rph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      int as = 0; uint32_t aph = 0; int bs = 0; uint32_t bph = 0; uint32_t acc_ph = 0;
      bool ok = true;
      const uint32_t idesc = make_idesc(128, TN, 1, 1);
      for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
        int rt, tb, kb0, kb1;
        tile_at(t, rt, tb, kb0, kb1);
        if (!mbar_wait(acce, acc_ph ^ 1, abort_flag, args.status, 1250)) { ok = false; break; }
        tc_fence_after();
        for (int ks = 0; ok && ks < 2 * (kb1 - kb0); ++ks) {
          if (!mbar_wait(&a_full[as], aph, abort_flag, args.status, 1251, as)) { ok = false; break; }
          for (int half = 0; half < 2; ++half) {
            if (!mbar_wait(&b_full[bs], bph, abort_flag, args.status, 1252, bs)) { ok = false; break; }
            tc_fence_after();
            const uint64_t b = make_sdesc_sw128(smem_u32(Bb + bs * 32768));
#pragma unroll
            for (int j = 0; j < 4; ++j)
              mma_f16_ts(tmem_base, tmem_a + as * 64 + half * 32 + j * 8, sdesc_at(b, j * 32), idesc, (ks > 0 || half > 0 || j > 0) ? 1u : 0u);
            tc_commit(&b_empty[bs]);
            if (++bs == BS) { bs = 0; bph ^= 1; }
          }
          if (!ok) break;
          tc_commit(&a_empty[as]);
          if (++as == kQwA) { as = 0; aph ^= 1; }
        }
        if (!ok) break;
        tc_commit(accf);
        acc_ph ^= 1;
      }
    }
  } else if (warp < 10) {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    const int q = warp & 3, c0 = ((warp - 2) >> 2) * 128;
    uint32_t acc_ph = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
      int rt, tb, kb0, kb1;
      const int ksp = tile_at(t, rt, tb, kb0, kb1);
      if (!__all_sync(0xffffffffu, mbar_wait(accf, acc_ph, abort_flag, args.status, 1260))) break;
      tc_fence_after();
      const uint32_t tacc = tmem_base + c0 + ((uint32_t)(q * 32) << 16);
      const int n = rt * 128 + q * 32 + lane;
      const bool n_ok = n < args.n_out;
      const float bias = (args.bias != nullptr && n_ok && ksp == 0) ? args.bias[n] : 0.f;
      const int tok0 = tb * TN + c0, live = min(min(128, TN - c0), args.m_tok - tok0);        // this warp's tokens (may be <= 0)
      const size_t off0 = (size_t)ksp * (size_t)args.partial_stride + (size_t)tok0 * args.ldo + n;
#pragma unroll 1
      for (int c = 0; c < live; c += 16) {
        uint32_t r[16];
        __syncwarp();                                      // rows past n_out left the round before early
        tmem_ld_x16(tacc + c, r);
        tc_wait_ld();
        if (!n_ok) continue;
        const size_t off = off0 + (size_t)c * args.ldo;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j >= live) break;
          const float v = __uint_as_float(r[j]) + bias;
          if (args.out_f32) reinterpret_cast<float*>(args.out)[off + (size_t)j * args.ldo] = v;
          else reinterpret_cast<__nv_bfloat16*>(args.out)[off + (size_t)j * args.ldo] = __float2bfloat16(v);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acce);
      acc_ph ^= 1;
    }
  } else {
    // ------------------------------------------------------------------ unpack (warps 10..25): raw blocks -> operand in TMEM
    const int q = warp & 3, part = ((warp - 10) >> 2) & 1, grp = (warp - 10) >> 3, row = q * 32 + lane;
    const uint32_t ta = tmem_a + grp * 128 + part * 32 + ((uint32_t)(q * 32) << 16);
    int rs = 0; uint32_t rph = 0, aph = 0; int turn = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && t < n_tiles; t += gridDim.x) {
      int rt, tb, kb0, kb1;
      tile_at(t, rt, tb, kb0, kb1);
      for (int kb = kb0; ok && kb < kb1; ++kb, turn ^= 1) {
        const int slot = rs;
        const uint32_t slot_ph = rph;
        if (++rs == RS) { rs = 0; rph ^= 1; }
        if (turn != grp) continue;
        // warp-uniform, as are all steps below (stores to TMEM are a warp's)
        if (!__all_sync(0xffffffffu, mbar_wait(&raw_full[slot], slot_ph, abort_flag, args.status, 1270, slot))) { ok = false; break; }
        const uint8_t* rb = rawb + slot * RAW_PAD;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int j = 2 * h + part;                      // 64-value chunk of the 256-column tile
          uint32_t o[32];                                  // two values each, in k order
          if (TYPE == 0) {
            const uint8_t* b = rb + row * 144;
            const uint4 hd = *reinterpret_cast<const uint4*>(b);
            const uint4 q0 = *reinterpret_cast<const uint4*>(b + 16 + 32 * j), q1 = *reinterpret_cast<const uint4*>(b + 32 + 32 * j);
            const __half2 dd = *reinterpret_cast<const __half2*>(&hd.x);
            const float d = __low2float(dd), dmin = __high2float(dd);
            const int bsh = 16 * part;
            uint32_t sc, mn;                               // two bytes: sub-blocks 2 j (low nibbles) and 2 j + 1 (high)
            if (h == 0) { sc = (hd.y >> bsh) & 0x3f3fu; mn = (hd.z >> bsh) & 0x3f3fu; }
            else {
              const uint32_t x = hd.w >> bsh, y = hd.y >> bsh, z = hd.z >> bsh;
              sc = (x & 0x0f0fu) | ((y >> 2) & 0x3030u); mn = ((x >> 4) & 0x0f0fu) | ((z >> 2) & 0x3030u);
            }
            const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            const __nv_bfloat162 sixteen = __float2bfloat162_rn(16.0f);
#pragma unroll
            for (int nib = 0; nib < 2; ++nib) {
              const __nv_bfloat162 a2 = __float2bfloat162_rn(d * (float)((sc >> (8 * nib)) & 0xffu));
              const __nv_bfloat162 b2 = __float2bfloat162_rn(-(dmin * (float)((mn >> (8 * nib)) & 0xffu)));
#pragma unroll
              for (int i = 0; i < 8; ++i) {                // as unpack_q4k_sub: bf16(16 + q) = 0x4180 | (q << 3)
                const uint32_t n3 = ((nib ? (w[i] >> 1) : (w[i] << 3)) & 0x78787878u) | 0x80808080u;
                const uint32_t p0 = prmt(n3, 0x41414141u, 0x4140), p1 = prmt(n3, 0x41414141u, 0x4342);
                const __nv_bfloat162 x0 = __hfma2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&p0), sixteen), a2, b2);
                const __nv_bfloat162 x1 = __hfma2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&p1), sixteen), a2, b2);
                o[16 * nib + 2 * i] = *reinterpret_cast<const uint32_t*>(&x0); o[16 * nib + 2 * i + 1] = *reinterpret_cast<const uint32_t*>(&x1);
              }
            }
          } else {
            const uint4* qp = reinterpret_cast<const uint4*>(rb + row * 272 + 64 * j);
            const uint32_t scw = *reinterpret_cast<const uint32_t*>(rb + row * 272 + 256 + 4 * j);
            const __half2 dd = *reinterpret_cast<const __half2*>(&scw);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const float d = v < 2 ? __low2float(dd) : __high2float(dd);
              const uint4 x4 = qp[v];
              const uint32_t w[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t x = w[i];
                const float f0 = (float)(int)(int8_t)(x & 0xff), f1 = (float)(int)(int8_t)((x >> 8) & 0xff);
                const float f2 = (float)(int)(int8_t)((x >> 16) & 0xff), f3 = (float)(int)(int8_t)(x >> 24);
                o[8 * v + 2 * i] = pack_bf16x2(f0 * d, f1 * d); o[8 * v + 2 * i + 1] = pack_bf16x2(f2 * d, f3 * d);
              }
            }
          }
          const int as = 2 * grp + h;
          if (!__all_sync(0xffffffffu, mbar_wait(&a_empty[as], aph ^ 1, abort_flag, args.status, 1271, as))) { ok = false; break; }
          tc_fence_after();
          tmem_st_x32(ta + h * 64, o);
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&a_full[as]);
            if (h == 1) mbar_arrive(&raw_empty[slot]);     // the words stored above were formed from the tile's bytes: all reads of it have returned
          }
        }
        aph ^= 1;
      }
    }
  }

  if (*abort_flag) {                                       // copies may still be landing: bounded grace period
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// Tokens of a tile of the wide kernel: the even cut of the tokens whose rounds of CTAs cost least, a step of 128 k-columns being a fixed part (the unpacking) and one per
// token (51200 rows of 5120: 160 tokens 122 us in three rounds, 512 tokens 247 us in six; 512 tokens over 40 row tiles: three tiles of 176 tokens in one round).
// At most 128: the narrow kernel's tiles do, see gb_qgemm.
static int qgemm_wide_tn(int m, int row_tiles, int splits, int sms) {
  int best = 256;
  long best_cost = -1;
  for (int tiles = (m + 255) / 256; tiles <= (m + 63) / 64; ++tiles) {
    const int tn = ((m + tiles - 1) / tiles + 15) & ~15;
    const long ctas = (long)row_tiles * ((m + tn - 1) / tn) * splits;
    const long cost = (ctas + sms - 1) / sms * (600 + 2 * tn);
    if (best_cost < 0 || cost < best_cost) { best = tn; best_cost = cost; }
  }
  return best;
}

template <int TYPE>
static int launch_qgemm_wide(const CUtensorMap& tmX, const QWideArgs& a, cudaStream_t stream) {
  constexpr int RAW = TYPE == 0 ? 128 * 144 : 128 * 272;
  const int smem = 1024 + qw_b_stages(TYPE) * 32768 + qw_raw_stages(TYPE) * ((RAW + 1023) & ~1023) + 512;
  auto kern = qgemm_wide_kernel<TYPE>;
  static bool attr_set = false;
  if (!attr_set) { GB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); attr_set = true; }
  int grid = sm_count();
  const int tiles = a.g.row_tiles * a.g.tok_tiles * a.g.splits;
  if (tiles < grid) grid = tiles;
  launch_k(kern, grid, kQwThreads, smem, stream, tmX, a);
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int TYPE, int TN>
static int launch_qgemm(const CUtensorMap& tmX, QGemmArgs a, cudaStream_t stream) {
  constexpr int RAW = TYPE == 0 ? 128 * 144 : 128 * 272;
  constexpr int RAW_PAD = (RAW + 1023) & ~1023;
  constexpr int B_BYTES = TN * 256;
  // token ring first, the rest of shared memory buys depth for the raw-tile ring:
  // the quantised bytes in flight are what a decode-sized launch is bound by
  const int budget = 220 * 1024 - 2048 - 2 * kQgA;
  const int bs = TN < 128 ? 4 : TYPE == 0 ? 3 : 2;
  int rs = (budget - bs * B_BYTES) / RAW_PAD;
  if (rs > 4) rs = 4;
  if (rs < 2) return fail("qgemm: token tile does not fit shared memory%s");
  a.b_stages = bs; a.raw_stages = rs;
  const int smem = 1024 + rs * RAW_PAD + 2 * kQgA + bs * B_BYTES + 512;
  auto kern = qgemm_kernel<TYPE, TN>;
  static bool attr_set = false;
  if (!attr_set) { GB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024)); attr_set = true; }
  int grid = sm_count();
  const int tiles = a.row_tiles * a.tok_tiles * a.splits;
  if (tiles < grid) grid = tiles;
  launch_k(kern, grid, kQgThreads, smem, stream, tmX, a);
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace gb

using namespace gb;

// w: tiled Q4_K (ggml type 12) or Q8_0 (8) weights, ceil(n_out / 128) row tiles x k / 256 K tiles.  x bf16 [m, ldx].
// out bf16 (or f32) [m, ldo].  tn: token tile 16, 32, 64, or 128 for more than 64 tokens (which may then be cut into tiles of up to 256).  splits > 1 cuts K: `out` is then f32 [splits][m, ldo] (slabs
// m * ldo apart), one partial sum per split for the consumer to add; no split may be empty.
GB_API int gb_qgemm(const void* w, int ggml_type, const void* x, int ldx, void* out, int ldo, int out_f32, const float* bias, int n_out,
                    int k, int m, int tn, int splits, void* status, cudaStream_t stream) {
  if (ggml_type != 12 && ggml_type != 8) return fail("qgemm: only Q4_K and Q8_0 have a fused tensor-core path%s");
  if (k <= 0 || k % 256 || n_out <= 0) return fail("qgemm: k must be a positive multiple of 256%s");
  if (m <= 0) return 0;
  if (ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return fail("qgemm: operands must be 16-byte aligned%s");
  if (tn != 16 && tn != 32 && tn != 64 && tn != 128) return fail("qgemm: token tile must be 16, 32, 64 or 128%s");
  // A step of 128 k-columns takes the wide kernel longer than the narrow one its 128 tokens (160 tokens 1.14 times, 256 tokens 1.22 times): it is taken where its
  // tiles, which are fewer, save a round of CTAs; by these figures that pays at every size (51200 rows of 5120: 128 tokens 107 us narrow, 117 wide; 160 tokens 204
  // and 122; 512 tokens 371 and 247; 5120 rows of 8192: 384 tokens 61 and 65, 512 tokens 114 and 65).  Tiles of at most 128 tokens cannot save one.
  bool wide = false;
  if (tn == 128) {
    const int row_tiles = (n_out + 127) / 128, sp = splits > 1 ? splits : 1, sms = sm_count(), wtn = qgemm_wide_tn(m, row_tiles, sp, sms);
    auto rounds = [&](int t) { return ((long)row_tiles * ((m + t - 1) / t) * sp + sms - 1) / sms; };
    wide = rounds(wtn) < rounds(128);
    if (wide) tn = wtn;
  }
  CUtensorMap tmX;
  if (make_tmap_2d(&tmX, x, TM_BF16, (uint64_t)k, (uint64_t)m, (uint64_t)ldx * 2, 64, (uint32_t)tn, TM_SW_128)) return -1;
  QGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.w = (const uint8_t*)w; a.out = out; a.ldo = ldo; a.out_f32 = out_f32; a.bias = bias; a.n_out = n_out; a.m_tok = m; a.num_kb = k / 256;
  a.row_tiles = (n_out + 127) / 128; a.tok_tiles = (m + tn - 1) / tn; a.status = (KernelStatus*)status;
  a.splits = splits > 1 ? splits : 1;
  a.kb_per = (a.num_kb + a.splits - 1) / a.splits;
  if (a.splits > 1) {
    if (!out_f32) return fail("qgemm: K-split partials need an fp32 output%s");
    if ((a.num_kb + a.kb_per - 1) / a.kb_per != a.splits) return fail("qgemm: a K split would be empty%s");
    a.partial_stride = (long)m * ldo;
  }
  const int t = ggml_type == 12 ? 0 : 1;
  if (wide) {
    const QWideArgs wa = {a, tn};
    return t == 0 ? launch_qgemm_wide<0>(tmX, wa, stream) : launch_qgemm_wide<1>(tmX, wa, stream);
  }
#define GB_QG(TNV)                                                             \
  if (tn == TNV) return t == 0 ? launch_qgemm<0, TNV>(tmX, a, stream) : launch_qgemm<1, TNV>(tmX, a, stream);
  GB_QG(16) GB_QG(32) GB_QG(64) GB_QG(128)
#undef GB_QG
  return fail("qgemm: unsupported token tile%s");
}
