// Linear layers of one or two tokens on bf16 weights (a decode step of one or two sequences), without tensor cores:
//   out[m, n] = sum_k W[n, k] * x[m, k]   (+ bias), f32;   or the gate / up form  act[m, n] = silu(Wg x) * (Wu x), bf16.
//
// Such a step is a chain of small kernels, each bound by its own start: a GEMM tile has barriers, TMEM, a TMA round trip, the MMA and the way back through TMEM
// behind its dependency wait, and its K splits need a kernel that adds them.  Here a warp owns whole weight rows: the first 16 KB to 64 KB of them per CTA
// are requested into registers BEFORE the dependency wait (weights do not depend on the step), so behind the wait there are the activations (a few KB from L2), the
// products and one warp reduction.  No K split, no partial sums, and the RMSNorm in front of a projection (residual += delta; rows of the next residual
// written by the first CTA) is formed by every CTA for itself, in the order of rmsnorm_kernel, so that its launch disappears.  Qwen3-0.6B, one token: GEMM,
// partial sums and norms 9 launches and 48 us a layer, 6 launches and 27 us in this form (1358 -> 811 us a step).
#include "sm100.cuh"
#include "host_common.h"

namespace gb {

constexpr int kGvThreads = 256;

struct GemvArgs {
  const __nv_bfloat16* w; int ldw; int tiled;      // [rows, k], row-major or [rows / 128][k / 64][128][64]
  int n, k, up_off;                                // up_off > 0: rows n + up_off are the "up" rows of a gate / up pair
  const __nv_bfloat16* x; int ldx;                 // activations [m, k], or (x null) the normalised sum of
  const __nv_bfloat16* res_in; __nv_bfloat16* res_out;     // residual rows [m, k] in and out (different buffers)
  const float* delta; int n_delta; long delta_stride;      // f32 [n_delta][m, k], what joins the residual; n_delta = 0: nothing
  const __nv_bfloat16* norm_w; float eps;
  float* out; __nv_bfloat16* act; int ldo;         // act: gate / up form
  const float* bias;
};

__device__ __forceinline__ void gv_spread(const uint4& r, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}

// M tokens; RW rows per warp (gate / up: RW / 2 pairs); S steps of 256 columns in flight; NORM: the input is a sum and its RMSNorm.
template <int M, int RW, int S, bool PAIR, bool NORM>
__global__ void __launch_bounds__(kGvThreads)
gemv_kernel(const GemvArgs a) {
  extern __shared__ uint4 gv_x[];                  // NORM: [M][k / 8] normalised rows, bf16
  __shared__ float red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kv = a.k >> 3, num_kb = (a.k + 63) >> 6;
  constexpr int RP = PAIR ? RW / 2 : RW;           // output features per warp
  const int n0 = (blockIdx.x * (kGvThreads / 32) + warp) * RP;
  const __nv_bfloat16* wp[RW];                     // row starts; rows past the end repeat the last one
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const int row = min(n0 + (PAIR ? r >> 1 : r), a.n - 1) + (PAIR && (r & 1) ? a.up_off : 0);
    wp[r] = a.tiled ? a.w + ((size_t)(row >> 7) * num_kb << 13) + ((row & 127) << 6) : a.w + (size_t)row * a.ldw;
  }
  uint4 wv[S][RW];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int v = lane + 32 * (i0 + s);
      const size_t off = a.tiled ? ((size_t)(v >> 3) << 13) + ((v & 7) << 3) : (size_t)v << 3;
#pragma unroll
      for (int r = 0; r < RW; ++r) wv[s][r] = v < kv ? __ldcs(reinterpret_cast<const uint4*>(wp[r] + off)) : make_uint4(0, 0, 0, 0);
    }
  };
  fetch(0);
  pdl_wait();
  pdl_trigger();

  if constexpr (NORM) {
    // as rmsnorm_kernel: vectors threadIdx.x + 256 i of a row, the same order of sums and the same roundings
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
      float ss = 0.f;
      for (int v = threadIdx.x; v < kv; v += kGvThreads) {
        float r[8];
        gv_spread(*reinterpret_cast<const uint4*>(a.res_in + (size_t)m * a.k + v * 8), r);
        uint4 keep;
        uint32_t* pk = reinterpret_cast<uint32_t*>(&keep);
        if (a.n_delta > 0) {
          float d[8] = {};
          const float* src = a.delta + (size_t)m * a.k + v * 8;
          for (int p = 0; p < a.n_delta; ++p, src += a.delta_stride) {
            const float4 u0 = *reinterpret_cast<const float4*>(src), u1 = *reinterpret_cast<const float4*>(src + 4);
            d[0] += u0.x; d[1] += u0.y; d[2] += u0.z; d[3] += u0.w; d[4] += u1.x; d[5] += u1.y; d[6] += u1.z; d[7] += u1.w;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) r[j] = __bfloat162float(__float2bfloat16(r[j] + d[j]));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) pk[j] = pack_bf16x2(r[2 * j], r[2 * j + 1]);
        gv_x[m * kv + v] = keep;
        if (blockIdx.x == 0 && a.res_out != nullptr) *reinterpret_cast<uint4*>(a.res_out + (size_t)m * a.k + v * 8) = keep;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += r[j] * r[j];
      }
      ss = warp_sum(ss);
      if (m > 0) __syncthreads();                  // the sums of the row before have been read
      if (lane == 0) red[warp] = ss;
      __syncthreads();
      float tot = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) tot += red[i];
      const float scale = rsqrtf(tot / (float)a.k + a.eps);
      for (int v = threadIdx.x; v < kv; v += kGvThreads) {       // a thread's own vectors
        float r[8], g[8];
        gv_spread(gv_x[m * kv + v], r);
        gv_spread(*reinterpret_cast<const uint4*>(a.norm_w + v * 8), g);
        uint4 y;
        uint32_t* pk = reinterpret_cast<uint32_t*>(&y);
#pragma unroll
        for (int j = 0; j < 4; ++j) pk[j] = pack_bf16x2(r[2 * j] * scale * g[2 * j], r[2 * j + 1] * scale * g[2 * j + 1]);
        gv_x[m * kv + v] = y;
      }
    }
    __syncthreads();
  }

  float acc[RW][M];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
  const int steps = (kv + 31) >> 5;
  for (int i0 = 0; i0 < steps; i0 += S) {
    uint4 xr[S][M];
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int v = lane + 32 * (i0 + s);
        if (v >= kv) xr[s][m] = make_uint4(0, 0, 0, 0);
        else if constexpr (NORM) xr[s][m] = gv_x[m * kv + v];
        else xr[s][m] = *reinterpret_cast<const uint4*>(a.x + (size_t)m * a.ldx + v * 8);
      }
    if (i0 > 0) fetch(i0);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      float xf[M][8];
#pragma unroll
      for (int m = 0; m < M; ++m) gv_spread(xr[s][m], xf[m]);
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        float wf[8];
        gv_spread(wv[s][r], wf);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[r][m] = fmaf(wf[j], xf[m][j], acc[r][m]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = warp_sum(acc[r][m]);
  if (lane < RP && n0 + lane < a.n) {
#pragma unroll
    for (int r = 0; r < RP; ++r) {
      if (r != lane) continue;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        if constexpr (PAIR) {
          const float g = acc[2 * r][m];
          a.act[(size_t)m * a.ldo + n0 + r] = __float2bfloat16(g / (1.0f + __expf(-g)) * acc[2 * r + 1][m]);
        } else {
          a.out[(size_t)m * a.ldo + n0 + r] = acc[r][m] + (a.bias != nullptr ? a.bias[n0 + r] : 0.f);
        }
      }
    }
  }
}

template <int M, int RW, int S, bool PAIR, bool NORM>
static int launch_gemv(const GemvArgs& a, cudaStream_t stream) {
  constexpr int per = kGvThreads / 32 * (PAIR ? RW / 2 : RW);
  const size_t smem = NORM ? (size_t)M * a.k * 2 : 0;
  launch_k(gemv_kernel<M, RW, S, PAIR, NORM>, (unsigned)((a.n + per - 1) / per), kGvThreads, smem, stream, a);
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int M, bool PAIR, bool NORM>
static int pick_gemv(const GemvArgs& a, cudaStream_t stream) {
  // rows per warp: enough for the loads in flight (8 to 16 vectors a lane), few enough that every SM has warps
  const long rows = (long)a.n * (PAIR ? 2 : 1);
  if (rows >= 8L * 4 * 2 * sm_count()) return launch_gemv<M, 4, 4, PAIR, NORM>(a, stream);
  if (PAIR || rows >= 8L * 2 * sm_count()) return launch_gemv<M, 2, 4, PAIR, NORM>(a, stream);
  if constexpr (!PAIR) return launch_gemv<M, 1, 8, false, NORM>(a, stream);
  return 0;
}

}  // namespace gb

using namespace gb;

// m = 1 or 2 tokens.  up_off > 0: gate / up form into `act` (bf16), else f32 into `out`.  x == null: the input is rmsnorm(res_in + sum of delta's slabs) * norm_w,
// and the new residual goes to res_out (optional, another buffer than res_in).
GB_API int gb_gemv(const void* w, int ldw, int tiled, int n, int k, int up_off, int m, const void* x, int ldx, const void* res_in, void* res_out,
                   const float* delta, int n_delta, long delta_stride, const void* norm_w, float eps, float* out, void* act, int ldo, const float* bias,
                   cudaStream_t stream) {
  if (m < 1 || m > 2 || n <= 0 || k <= 0 || k % 8) return fail("gemv: one or two tokens, k a multiple of 8%s");
  if (tiled && k % 64) return fail("gemv: tiled weights need k %% 64 == 0%s");
  const bool norm = x == nullptr, pair = up_off > 0;
  const uintptr_t al = (uintptr_t)w | (uintptr_t)x | (uintptr_t)res_in | (uintptr_t)res_out | (uintptr_t)delta | (uintptr_t)norm_w;
  if (al % 16 || ldw % 8 || ldx % 8 || delta_stride % 4) return fail("gemv: operands must be 16-byte aligned%s");
  if (norm && (res_in == nullptr || norm_w == nullptr || res_in == res_out || k > 8192)) return fail("gemv: bad normalised input%s");
  if ((pair ? act : (void*)out) == nullptr || (pair && bias != nullptr)) return fail("gemv: bad output%s");
  GemvArgs a;
  memset(&a, 0, sizeof(a));
  a.w = (const __nv_bfloat16*)w; a.ldw = ldw; a.tiled = tiled; a.n = n; a.k = k; a.up_off = up_off; a.x = (const __nv_bfloat16*)x; a.ldx = ldx;
  a.res_in = (const __nv_bfloat16*)res_in; a.res_out = (__nv_bfloat16*)res_out; a.delta = delta; a.n_delta = n_delta; a.delta_stride = delta_stride;
  a.norm_w = (const __nv_bfloat16*)norm_w; a.eps = eps; a.out = out; a.act = (__nv_bfloat16*)act; a.ldo = ldo; a.bias = bias;
  if (m == 1) return pair ? (norm ? pick_gemv<1, true, true>(a, stream) : pick_gemv<1, true, false>(a, stream))
                          : (norm ? pick_gemv<1, false, true>(a, stream) : pick_gemv<1, false, false>(a, stream));
  return pair ? (norm ? pick_gemv<2, true, true>(a, stream) : pick_gemv<2, true, false>(a, stream))
              : (norm ? pick_gemv<2, false, true>(a, stream) : pick_gemv<2, false, false>(a, stream));
}
