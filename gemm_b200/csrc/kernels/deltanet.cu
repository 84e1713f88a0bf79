// Gated Delta-Net layers of the Qwen3.5 hybrid models (linear attention with a per-head matrix state) and the sigmoid output
// gate of their full-attention layers.
//
//   gb_ssm_conv_silu     causal depthwise conv1d (kernel conv_k, history carried per sequence) + SiLU over packed tokens
//   gb_deltanet          per (sequence, value head): L2-normalised q, k; S *= exp(alpha); delta = (v - S k) * beta;
//                        S += delta k^T; o = S q; gated RMSNorm: o * rsqrt(mean(o^2) + eps) * w * SiLU(z)
//   gb_sigmoid_gate_mul  a[t, c] *= sigmoid(gate[t, c])
//
// The recurrence keeps one row of the d_state x d_state state per thread in registers and walks the tokens of its sequence
// in order, so one launch serves decode (one token) and prefill chunks alike; the state is read once and written once per
// launch.  Prefill launches take the chunked scan of deltanet_chunk.cu instead.
//
// Math and tensor conventions follow common/transformer.h:2861-3113 (tf_ssm_deltanet_forward) and :2829-2851 (the scalar
// recurrence): qkv channels are ordered [Q (n_group heads) | K (n_group heads) | V (dt_rank heads)], value head h uses the
// q/k group h % n_group, alpha = softplus(alpha_raw + dt_bias) * a, beta = sigmoid(beta_raw), q is scaled by
// 1/sqrt(d_state) after the L2 normalisation (x / sqrt(sum x^2 + eps)).  The reference keeps the conv history in a ring
// buffer (transformer.h:2927-2998); here it is a plain oldest-to-newest window, rewritten at the end of every launch.
#include "sm100.cuh"
#include "host_common.h"

namespace gb {

constexpr int kMaxConvK = 8;

constexpr int kConvTile = 32;        // tokens per tile: at least kMaxConvK - 1, so that only a sequence's first tile meets the history

// Bound by memory: every row is read and written once.  A CTA takes one tile of up to 32 tokens of one sequence and 256 threads' channels, VEC
// neighbouring ones per thread (one 8-byte access per token), with eight tokens' loads in flight.  One thread per channel that walked its whole sequence
// left 48 CTAs with one 2-byte load in flight each: 1621 us for 3001 tokens of 12288 channels, 77 us in this form (1.9 TB/s; the rest is the sigmoid's
// arithmetic).  One token for each of 16 sequences takes 4.9 us in both.
// K: taps (0: conv_k of them, at most kMaxConvK).  The thread of a sequence's first tile reads its channels' history and writes the new one (which
// follows from the last rows of the sequence): nobody else touches that state, so the order of the tiles does not matter.
template <int K, int VEC>
__global__ void __launch_bounds__(256)
ssm_conv_silu_kernel(const __nv_bfloat16* __restrict__ x, int ld_x, const float* __restrict__ w, float* __restrict__ state,
                     const int* __restrict__ cu_q, const int* __restrict__ seq_slots, __nv_bfloat16* __restrict__ out, int ld_out,
                     int channels, int conv_k, int n_seqs) {
  constexpr int MK = K ? K : kMaxConvK;
  const int nh = K ? K - 1 : conv_k - 1;
  const int c = (blockIdx.y * 256 + threadIdx.x) * VEC;
  pdl_wait();
  pdl_trigger();
  float wk[MK][VEC];
#pragma unroll
  for (int u = 0; u < VEC; ++u) {
    if constexpr (K == 4 && VEC == 4) {
      const float4 r = c < channels ? *reinterpret_cast<const float4*>(w + (size_t)(c + u) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      wk[0][u] = r.x; wk[1][u] = r.y; wk[2][u] = r.z; wk[3][u] = r.w;
    } else {
#pragma unroll
      for (int f = 0; f < MK; ++f) wk[f][u] = (f <= nh && c < channels) ? w[(size_t)(c + u) * (nh + 1) + f] : 0.f;
    }
  }
  // tile -> sequence: running sum of the sequences' tile counts, 32 sequences at a time
  const int lane = threadIdx.x & 31;
  int tile = blockIdx.x, seq = -1, s_t0 = 0, s_t1 = 0;
  for (int s0 = 0; s0 < n_seqs; s0 += 32) {
    const int s = min(s0 + lane, n_seqs - 1);
    const int q0 = cu_q[s], q1 = cu_q[s + 1];
    const int n = s0 + lane < n_seqs ? max(0, q1 - q0 + kConvTile - 1) / kConvTile : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    const uint32_t hit = __ballot_sync(0xffffffffu, tile < incl);
    if (hit) {
      const int l = __ffs(hit) - 1;
      tile -= __shfl_sync(0xffffffffu, incl - n, l);
      seq = s0 + l;
      s_t0 = __shfl_sync(0xffffffffu, q0, l); s_t1 = __shfl_sync(0xffffffffu, q1, l);
      break;
    }
    tile -= __shfl_sync(0xffffffffu, incl, 31);
  }
  if (seq < 0 || c >= channels) return;
  const int b = s_t0 + tile * kConvTile, e = min(b + kConvTile, s_t1);

  auto load = [&](int t, float* v) {
    const __nv_bfloat16* p = x + (size_t)t * ld_x + c;
    if constexpr (VEC == 4) {
      const uint2 r = *reinterpret_cast<const uint2*>(p);
      const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
      v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
    } else v[0] = __bfloat162float(*p);
  };
  float win[MK - 1][VEC];                               // window: oldest row first
  auto push = [&](float (*q)[VEC], const float* v) {    // the window one token on
#pragma unroll
    for (int f = 0; f < MK - 1; ++f)
#pragma unroll
      for (int u = 0; u < VEC; ++u)
        if (f < nh) q[f][u] = (f + 1 < nh) ? q[f + 1 < MK - 1 ? f + 1 : f][u] : v[u];
  };
  if (tile == 0) {
    float* st = state + (size_t)seq_slots[seq] * nh * channels + c;
    float next[MK - 1][VEC];
#pragma unroll
    for (int f = 0; f < MK - 1; ++f)
#pragma unroll
      for (int u = 0; u < VEC; ++u) next[f][u] = win[f][u] = (f < nh) ? st[(size_t)f * channels + u] : 0.f;
    for (int t = max(s_t0, s_t1 - nh); t < s_t1; ++t) { float v[VEC]; load(t, v); push(next, v); }
#pragma unroll
    for (int f = 0; f < MK - 1; ++f)
#pragma unroll
      for (int u = 0; u < VEC; ++u) if (f < nh) st[(size_t)f * channels + u] = next[f][u];
  } else {
#pragma unroll
    for (int f = 0; f < MK - 1; ++f) if (f < nh) load(b - nh + f, win[f]);
  }
  constexpr int G = 8;
  for (int t0 = b; t0 < e; t0 += G) {
    float v[G][VEC];
#pragma unroll
    for (int g = 0; g < G; ++g) if (t0 + g < e) load(t0 + g, v[g]);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if (t0 + g >= e) break;
      float y[VEC];
#pragma unroll
      for (int u = 0; u < VEC; ++u) {
        float acc = 0.f;
#pragma unroll
        for (int f = 0; f < MK - 1; ++f) if (f < nh) acc += wk[f][u] * win[f][u];
#pragma unroll
        for (int f = 0; f < MK; ++f) if (f == nh) acc += wk[f][u] * v[g][u];
        y[u] = acc / (1.0f + __expf(-acc));
      }
      __nv_bfloat16* o = out + (size_t)(t0 + g) * ld_out + c;
      if constexpr (VEC == 4) *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]));
      else *o = __float2bfloat16(y[0]);
      push(win, v[g]);
    }
  }
}

struct DeltaNetArgs {
  const __nv_bfloat16* qkv;   // [T, ld_qkv] after conv + SiLU: Q | K | V
  int ld_qkv;
  const __nv_bfloat16* z;     // [T, ld_z] gate input (d_inner columns)
  int ld_z;
  const float* ab;            // [T, 2 * dt_rank]: alpha_raw | beta_raw
  const float* a;             // [dt_rank]
  const float* dt_bias;       // [dt_rank]
  const float* norm_w;        // [d_state]
  float* state;               // [slots, dt_rank, d_state, d_state]
  const int* cu_q;
  const int* seq_slots;
  __nv_bfloat16* out;         // [T, dt_rank * d_state]
  int n_group, dt_rank;
  float eps;
};

template <int DS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) red[w] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < DS / 32; ++i) t += red[i];
  __syncthreads();
  return t;
}

// grid (dt_rank, sequences), DS threads: thread r owns row r of the state (the value index), columns are the key index.
template <int DS>
__global__ void __launch_bounds__(DS)
deltanet_kernel(const DeltaNetArgs a) {
  pdl_wait();
  pdl_trigger();
  const int h = blockIdx.x, s = blockIdx.y, r = threadIdx.x;
  const int t0 = a.cu_q[s], t1 = a.cu_q[s + 1];
  if (t1 <= t0) return;
  __shared__ float sq[DS], sk[DS], red[DS / 32];
  const int g = h % a.n_group;
  const int q_off = g * DS, k_off = a.n_group * DS + g * DS, v_off = 2 * a.n_group * DS + h * DS;
  float* st = a.state + (((size_t)a.seq_slots[s] * a.dt_rank + h) * DS + r) * DS;
  float S[DS];
#pragma unroll
  for (int c = 0; c < DS; c += 4) {
    const float4 v4 = *reinterpret_cast<const float4*>(st + c);
    S[c] = v4.x; S[c + 1] = v4.y; S[c + 2] = v4.z; S[c + 3] = v4.w;
  }
  const float a_h = a.a[h], bias_h = a.dt_bias[h], nw = a.norm_w[r];
  const float q_scale = rsqrtf((float)DS);
  for (int t = t0; t < t1; ++t) {
    const __nv_bfloat16* row = a.qkv + (size_t)t * a.ld_qkv;
    const float qv = __bfloat162float(row[q_off + r]), kv = __bfloat162float(row[k_off + r]), vv = __bfloat162float(row[v_off + r]);
    const float qn = block_sum<DS>(qv * qv, red), kn = block_sum<DS>(kv * kv, red);
    sq[r] = qv * rsqrtf(qn + a.eps) * q_scale;
    sk[r] = kv * rsqrtf(kn + a.eps);
    const float ar = a.ab[(size_t)t * 2 * a.dt_rank + h] + bias_h;
    const float sp = ar > 20.0f ? ar : log1pf(__expf(ar));
    const float decay = __expf(sp * a_h);
    const float beta = 1.0f / (1.0f + __expf(-a.ab[(size_t)t * 2 * a.dt_rank + a.dt_rank + h]));
    __syncthreads();
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < DS; ++c) { S[c] *= decay; dot += S[c] * sk[c]; }
    const float delta = (vv - dot) * beta;
    float o = 0.f;
#pragma unroll
    for (int c = 0; c < DS; ++c) { S[c] += delta * sk[c]; o += S[c] * sq[c]; }
    const float ss = block_sum<DS>(o * o, red);          // also the barrier that lets the next token overwrite sq / sk
    const float zv = __bfloat162float(a.z[(size_t)t * a.ld_z + h * DS + r]);
    const float y = o * rsqrtf(ss / (float)DS + a.eps) * nw * (zv / (1.0f + __expf(-zv)));
    a.out[((size_t)t * a.dt_rank + h) * DS + r] = __float2bfloat16(y);
  }
#pragma unroll
  for (int c = 0; c < DS; c += 4) *reinterpret_cast<float4*>(st + c) = make_float4(S[c], S[c + 1], S[c + 2], S[c + 3]);
}

__global__ void sigmoid_gate_mul_kernel(__nv_bfloat16* __restrict__ x, int ld_x, const __nv_bfloat16* __restrict__ gate, int ld_g, long rows,
                                        int cols) {
  pdl_wait();
  pdl_trigger();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int vpr = cols >> 3;
  if (idx >= rows * vpr) return;
  const long rr = idx / vpr;
  const int c = (int)(idx % vpr) * 8;
  const uint4 xr = *reinterpret_cast<const uint4*>(x + rr * ld_x + c), gr = *reinterpret_cast<const uint4*>(gate + rr * ld_g + c);
  const __nv_bfloat162* xh = reinterpret_cast<const __nv_bfloat162*>(&xr);
  const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gr);
  uint4 o;
  uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 xf = __bfloat1622float2(xh[i]), gf = __bfloat1622float2(gh[i]);
    ow[i] = pack_bf16x2(xf.x / (1.0f + __expf(-gf.x)), xf.y / (1.0f + __expf(-gf.y)));
  }
  *reinterpret_cast<uint4*>(x + rr * ld_x + c) = o;
}

}  // namespace gb

using namespace gb;

// `total_tokens`: rows of x in all sequences (the grid's bound on their tiles).
GB_API int gb_ssm_conv_silu(const void* x, int ld_x, const float* w, float* state, const int* cu_q, const int* seq_slots, void* out, int ld_out,
                            int channels, int conv_k, int n_seqs, long total_tokens, cudaStream_t stream) {
  if (conv_k < 2 || conv_k > kMaxConvK) return fail("ssm_conv: conv_k must be in [2, 8]%s");
  if (n_seqs <= 0 || total_tokens <= 0 || channels <= 0) return 0;
  // 8-byte rows where every row starts on 8 bytes; else a channel per thread
  const bool vec = channels % 4 == 0 && ld_x % 4 == 0 && ld_out % 4 == 0 && ((uintptr_t)x | (uintptr_t)out) % 8 == 0 && (uintptr_t)w % 16 == 0;
  const int per_cta = 256 * (vec ? 4 : 1);
  const dim3 grid((unsigned)(total_tokens / kConvTile + n_seqs), (unsigned)((channels + per_cta - 1) / per_cta));
#define GB_CONV(KV, VV) launch_k(ssm_conv_silu_kernel<KV, VV>, grid, 256, 0, stream, (const __nv_bfloat16*)x, ld_x, w, state, cu_q, seq_slots, \
                                 (__nv_bfloat16*)out, ld_out, channels, conv_k, n_seqs)
  if (conv_k == 4) { if (vec) GB_CONV(4, 4); else GB_CONV(4, 1); }
  else { if (vec) GB_CONV(0, 4); else GB_CONV(0, 1); }
#undef GB_CONV
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

GB_API int gb_deltanet(const void* qkv, int ld_qkv, const void* z, int ld_z, const float* ab, const float* a, const float* dt_bias,
                       const float* norm_w, float* state, const int* cu_q, const int* seq_slots, void* out, int n_group, int dt_rank,
                       int d_state, float eps, int n_seqs, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (n_group <= 0 || dt_rank % n_group) return fail("deltanet: dt_rank must be a multiple of n_group%s");
  DeltaNetArgs g;
  g.qkv = (const __nv_bfloat16*)qkv; g.ld_qkv = ld_qkv; g.z = (const __nv_bfloat16*)z; g.ld_z = ld_z; g.ab = ab; g.a = a; g.dt_bias = dt_bias;
  g.norm_w = norm_w; g.state = state; g.cu_q = cu_q; g.seq_slots = seq_slots; g.out = (__nv_bfloat16*)out; g.n_group = n_group;
  g.dt_rank = dt_rank; g.eps = eps;
  if (d_state == 128) launch_k(deltanet_kernel<128>, dim3(dt_rank, n_seqs), 128, 0, stream, g);
  else if (d_state == 64) launch_k(deltanet_kernel<64>, dim3(dt_rank, n_seqs), 64, 0, stream, g);
  else return fail("deltanet: d_state must be 64 or 128%s");
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}

GB_API int gb_sigmoid_gate_mul(void* x, int ld_x, const void* gate, int ld_g, long rows, int cols, cudaStream_t stream) {
  if (cols % 8 || ld_x % 8 || ld_g % 8) return fail("sigmoid_gate_mul: columns and strides must be multiples of 8%s");
  const long n = rows * (cols / 8);
  if (n <= 0) return 0;
  launch_k(sigmoid_gate_mul_kernel, (unsigned)((n + 255) / 256), 256, 0, stream, (__nv_bfloat16*)x, ld_x, (const __nv_bfloat16*)gate, ld_g, rows, cols);
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}
