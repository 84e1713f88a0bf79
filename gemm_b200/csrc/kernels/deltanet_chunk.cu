// Chunked scan of the gated Delta-Net recurrence for prefill (the per-token form and the math conventions are in deltanet.cu).
//
// Per value head the recurrence is  S_t = g_t S_{t-1} + u_t k_t^T,  u_t = beta_t (v_t - g_t S_{t-1} k_t),  o_t = S_t q_t
// with the scalar decay g_t = exp(a_t).  Over a chunk of C = 64 tokens, with c_i the running sum of a_t inside the chunk and S0 the
// state in front of it, the u_t solve a unit lower-triangular system, and everything else is matrix products:
//
//   L_ij   = beta_i exp(c_i - c_j) (k_i . k_j)   (j < i)          T = (I + L)^-1 diag(beta)
//   U      = T V - (T diag(exp c) K) S0^T                          (rows u_i)
//   O      = diag(exp c) Q S0^T + M U,   M_ij = exp(c_i - c_j) (q_i . k_j)  (j <= i)
//   S_end  = exp(c_last) S0 + U^T diag(exp(c_last - c_j)) K
//
// Two kernels.  dn_chunk_prep_kernel (one CTA per chunk and value head, all chunks of all sequences in parallel) computes what
// does not depend on the state: the normalised q / k, T (forward substitution, one thread per column), T V, -T diag(exp c) K, M,
// diag(exp c) Q and the decayed keys, all as bf16 tiles in a workspace.  dn_chunk_scan_kernel (one or two CTAs per sequence and
// value head) walks the chunks in order: three products per chunk (U, O, the state update), the gated RMSNorm of O, and the output.  The products
// are 64 x 128 x 128 at most and sit on a serial chain.  Written with the value index as the rows of every product (U^T, O^T, S), each
// one's accumulator IS the next one's left operand, register for register, so a warp carries 16 values through all three without
// meeting another warp or shared memory; only the right operands come from there (ldmatrix), the next chunk's copied while this one
// is worked on.  Warp-level mma (bf16 in, fp32 out) rather than tcgen05: a TMEM round trip per link of the chain would cost more than
// the tiles themselves.  3001 tokens, 32 heads: 929 us with every link staged through shared memory, 359 us in this form on one SM per
// head, bound by the rate of the warp-level mma (1792 of them per chunk, two warps on each tensor core), 322 us with a head's values
// over a cluster of two CTAs; the preparation 246 -> 150 us.
//
// The reference's counterpart is the chunked scan of cuda/llm/cuda_llm_runner.c:8128 (batch_deltanet_scan_f32) and its test
// cuda/llm/scan/deltanet_chunk_test.c; the per-token recurrence is common/transformer.h:2829-2851.

#include <mma.h>

#include "sm100.cuh"
#include "host_common.h"

namespace gb {

using namespace nvcuda;

constexpr int kDnC = 64;            // tokens per chunk
constexpr int kDnD = 128;           // d_state
constexpr int kDnLd = kDnD + 8;     // bf16 row stride of a 128-wide tile in shared memory (the pad spreads the rows over the banks)
constexpr int kDnLc = kDnC + 8;     // bf16 row stride of a 64-wide tile
constexpr int kDnLf = kDnD + 4;     // fp32 row stride of the 64 x 128 staging tile
constexpr int kDnLo = kDnC;         // L transposed (64 x 64, fp32) lives in the columns 64 .. 127 of the staging tile while T is solved
constexpr int kDnThreads = 256;

struct DnChunkArgs {
  const __nv_bfloat16* qkv; int ld_qkv;
  const __nv_bfloat16* z; int ld_z;
  const float* ab; const float* a; const float* dt_bias; const float* norm_w;
  float* state; const int* cu_q; const int* seq_slots; __nv_bfloat16* out;
  int n_group, dt_rank, n_seqs; float eps;
  // workspace: entry (chunk, head) at index chunk * dt_rank + head
  __nv_bfloat16* gq;     // [64][128]  exp(c_i) q_i
  __nv_bfloat16* nw;     // [64][128]  -(T diag(exp c) K)
  __nv_bfloat16* uv;     // [128][64]  T V, transposed
  __nv_bfloat16* kdt;    // [128][64]  exp(c_last - c_j) k_j, transposed
  __nv_bfloat16* mqk;    // [64][64]   M
  float* glast;          // exp(c_last)
};

// chunk `cb` (numbered through the sequences in order) -> its sequence and token range
__device__ __forceinline__ bool dn_find_chunk(const int* __restrict__ cu_q, int n_seqs, int cb, int& t0, int& t1) {
  int acc = 0;
  for (int s = 0; s < n_seqs; ++s) {
    const int b = cu_q[s], e = cu_q[s + 1];
    const int n = (e - b + kDnC - 1) / kDnC;
    if (cb < acc + n) {
      t0 = b + (cb - acc) * kDnC;
      t1 = min(t0 + kDnC, e);
      return true;
    }
    acc += n;
  }
  return false;
}

__device__ __forceinline__ float dn_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

using FragA = wmma::fragment<wmma::matrix_a, 16, 16, 16, __nv_bfloat16, wmma::row_major>;
using FragB = wmma::fragment<wmma::matrix_b, 16, 16, 16, __nv_bfloat16, wmma::col_major>;     // B given as [n][k] rows
using FragC = wmma::fragment<wmma::accumulator, 16, 16, 16, float>;

// 112.5 KB: two CTAs per SM
constexpr int kPrepSmem = (2 * kDnC * kDnLd + 2 * kDnD * kDnLc + kDnC * kDnLc) * 2 + (kDnC * kDnLf + 2 * kDnC) * 4;

__global__ void __launch_bounds__(kDnThreads)
dn_chunk_prep_kernel(const DnChunkArgs a) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(128) uint8_t dn_smem[];
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(dn_smem);          // [64][kDnLd] normalised, scaled q
  __nv_bfloat16* sK = sQ + kDnC * kDnLd;                                   // [64][kDnLd] normalised k
  __nv_bfloat16* sVT = sK + kDnC * kDnLd;                                  // [128][kDnLc] v transposed
  __nv_bfloat16* sGKT = sVT + kDnD * kDnLc;                                // [128][kDnLc] exp(c_j) k_j transposed
  __nv_bfloat16* sT = sGKT + kDnD * kDnLc;                                 // [64][kDnLc]
  float* sF = reinterpret_cast<float*>(sT + kDnC * kDnLc);                 // [64][kDnLf]
  float* sL = sF + kDnLo;                                                  // [64][.. kDnLf], the right half of sF
  float* sc = sF + kDnC * kDnLf;                                           // [64] running log decay
  float* sb = sc + kDnC;                                                   // [64] beta

  const int cb = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int t0 = 0, t1 = 0;
  if (!dn_find_chunk(a.cu_q, a.n_seqs, cb, t0, t1)) return;
  const int g = h % a.n_group;
  const int q_off = g * kDnD, k_off = (a.n_group + g) * kDnD, v_off = 2 * a.n_group * kDnD + h * kDnD;
  const size_t ws = (size_t)cb * a.dt_rank + h;

  // rows of the chunk: L2-normalised q (scaled by 1 / sqrt(d)) and k, v transposed; tokens past the end are zero rows
  // (warp w: rows 8 w .. 8 w + 7, all requested before the first is used; v leaves as eight tokens of a channel at a time)
  {
    uint2 qr[8], kr[8], vr[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int t = t0 + 8 * warp + r;
      qr[r] = kr[r] = vr[r] = make_uint2(0u, 0u);
      if (t < t1) {
        const __nv_bfloat16* row = a.qkv + (size_t)t * a.ld_qkv;
        qr[r] = *reinterpret_cast<const uint2*>(row + q_off + 4 * lane);
        kr[r] = *reinterpret_cast<const uint2*>(row + k_off + 4 * lane);
        vr[r] = *reinterpret_cast<const uint2*>(row + v_off + 4 * lane);
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = 8 * warp + r;
      const __nv_bfloat16* qb = reinterpret_cast<const __nv_bfloat16*>(&qr[r]);
      const __nv_bfloat16* kb = reinterpret_cast<const __nv_bfloat16*>(&kr[r]);
      float q4[4], k4[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) { q4[e] = __bfloat162float(qb[e]); k4[e] = __bfloat162float(kb[e]); }
      const float qs = dn_warp_sum(q4[0] * q4[0] + q4[1] * q4[1] + q4[2] * q4[2] + q4[3] * q4[3]);
      const float ks = dn_warp_sum(k4[0] * k4[0] + k4[1] * k4[1] + k4[2] * k4[2] + k4[3] * k4[3]);
      const float qsc = rsqrtf(qs + a.eps) * rsqrtf((float)kDnD), ksc = rsqrtf(ks + a.eps);
      *reinterpret_cast<uint2*>(sQ + i * kDnLd + 4 * lane) = make_uint2(pack_bf16x2(q4[0] * qsc, q4[1] * qsc), pack_bf16x2(q4[2] * qsc, q4[3] * qsc));
      *reinterpret_cast<uint2*>(sK + i * kDnLd + 4 * lane) = make_uint2(pack_bf16x2(k4[0] * ksc, k4[1] * ksc), pack_bf16x2(k4[2] * ksc, k4[3] * ksc));
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint4 o;
      uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t lo = e < 2 ? vr[2 * u].x : vr[2 * u].y, hi = e < 2 ? vr[2 * u + 1].x : vr[2 * u + 1].y;
        po[u] = __byte_perm(lo, hi, e & 1 ? 0x7632 : 0x5410);
      }
      *reinterpret_cast<uint4*>(sVT + (4 * lane + e) * kDnLc + 8 * warp) = o;
    }
  }
  if (tid < kDnC) {
    const int t = t0 + tid;
    float al = 0.f, beta = 0.f;
    if (t < t1) {
      const float ar = a.ab[(size_t)t * 2 * a.dt_rank + h] + a.dt_bias[h];
      const float sp = ar > 20.0f ? ar : log1pf(__expf(ar));
      al = sp * a.a[h];
      beta = 1.0f / (1.0f + __expf(-a.ab[(size_t)t * 2 * a.dt_rank + a.dt_rank + h]));
    }
    sc[tid] = al;
    sb[tid] = beta;
  }
  __syncthreads();
  if (tid == 0) {
    float acc = 0.f;
    for (int i0 = 0; i0 < kDnC; i0 += 16) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(sc + i0 + 4 * u);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        v[u].x = acc += v[u].x; v[u].y = acc += v[u].y; v[u].z = acc += v[u].z; v[u].w = acc += v[u].w;
        *reinterpret_cast<float4*>(sc + i0 + 4 * u) = v[u];
      }
    }
  }
  __syncthreads();
  const float c_last = sc[kDnC - 1];
  // K K^T and Q K^T (64 x 64 x 128): warp w computes the tiles (m = w & 3, n = 2 (w >> 2) and the next)
  const int tm = warp & 3, tn0 = (warp >> 2) * 2;
  for (int pass = 0; pass < 2; ++pass) {
    const __nv_bfloat16* sA = pass == 0 ? sK : sQ;
    FragC acc[2];
    wmma::fill_fragment(acc[0], 0.f);
    wmma::fill_fragment(acc[1], 0.f);
    for (int kk = 0; kk < kDnD / 16; ++kk) {
      FragA fa;
      wmma::load_matrix_sync(fa, sA + (16 * tm) * kDnLd + 16 * kk, kDnLd);
#pragma unroll
      for (int n2 = 0; n2 < 2; ++n2) {
        FragB fb;
        wmma::load_matrix_sync(fb, sK + (16 * (tn0 + n2)) * kDnLd + 16 * kk, kDnLd);
        wmma::mma_sync(acc[n2], fa, fb, acc[n2]);
      }
    }
    wmma::store_matrix_sync(sF + (16 * tm) * kDnLf + 16 * tn0, acc[0], kDnLf, wmma::mem_row_major);
    wmma::store_matrix_sync(sF + (16 * tm) * kDnLf + 16 * (tn0 + 1), acc[1], kDnLf, wmma::mem_row_major);
    __syncthreads();
    for (int idx = tid; idx < kDnC * kDnC; idx += kDnThreads) {
      const int i = idx / kDnC, j = idx % kDnC;
      if (pass == 0) {                  // row i of L^T: L_ji (K K^T is symmetric)
        sL[i * kDnLf + j] = (i < j) ? sb[j] * __expf(sc[j] - sc[i]) * sF[i * kDnLf + j] : 0.f;
      } else {
        const float m = (j <= i) ? __expf(sc[i] - sc[j]) * sF[i * kDnLf + j] : 0.f;
        a.mqk[(ws * kDnC + i) * kDnC + j] = __float2bfloat16(m);
      }
    }
    __syncthreads();
  }

  // T = (I + L)^-1 diag(beta) by forward substitution: two warps, a thread per column, 16 rows at a time in registers (the rows above them come back
  // from shared memory, a row of L^T serves 16 unknowns with four broadcast loads).  A thread's 2016 products are independent but for the 64 steps of
  // the diagonal blocks; one column over four lanes with a shuffle pair per row had a chain of 64 x (16 products + 2 shuffles).  The other warps
  // meanwhile form the operands that only need q, k and the decays.
  if (warp < 2) {
    const int col = tid;
    const float bcol = sb[col];
    for (int i0 = 0; i0 < kDnC; i0 += 16) {
      float xr[16], part[16][4];                         // a row's products in four sums, by j & 3: short chains
#pragma unroll
      for (int i = 0; i < 16; ++i) part[i][0] = part[i][1] = part[i][2] = part[i][3] = 0.f;
      for (int j0 = 0; j0 < i0; j0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float xj = sF[(j0 + u) * kDnLf + col];
          const float4* l4 = reinterpret_cast<const float4*>(sL + (j0 + u) * kDnLf + i0);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const float4 l = l4[v];
            part[4 * v][u] += l.x * xj; part[4 * v + 1][u] += l.y * xj; part[4 * v + 2][u] += l.z * xj; part[4 * v + 3][u] += l.w * xj;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float xj = xr[j] = ((i0 + j == col) ? bcol : 0.f) - ((part[j][0] + part[j][1]) + (part[j][2] + part[j][3]));
        const float4* l4 = reinterpret_cast<const float4*>(sL + (i0 + j) * kDnLf + i0);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if (4 * v + 3 <= j) continue;
          const float4 l = l4[v];
          if (4 * v > j) part[4 * v][j & 3] += l.x * xj;
          if (4 * v + 1 > j) part[4 * v + 1][j & 3] += l.y * xj;
          if (4 * v + 2 > j) part[4 * v + 2][j & 3] += l.z * xj;
          if (4 * v + 3 > j) part[4 * v + 3][j & 3] += l.w * xj;
        }
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        sF[(i0 + i) * kDnLf + col] = xr[i];
        sT[(i0 + i) * kDnLc + col] = __float2bfloat16(xr[i]);
      }
    }
  } else {
    const int t2 = tid - 64;
    for (int idx = t2; idx < kDnC * kDnD / 8; idx += kDnThreads - 64) {             // exp(c_i) q_i, 16 bytes at a time
      const int i = idx / (kDnD / 8), c = 8 * (idx % (kDnD / 8));
      const float e = __expf(sc[i]);
      const uint4 r = *reinterpret_cast<const uint4*>(sQ + i * kDnLd + c);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&r);
      uint4 o;
      uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int u = 0; u < 4; ++u) { const float2 f = __bfloat1622float2(h2[u]); po[u] = pack_bf16x2(e * f.x, e * f.y); }
      *reinterpret_cast<uint4*>(a.gq + ws * kDnC * kDnD + (size_t)i * kDnD + c) = o;
    }
    for (int idx = t2; idx < kDnD * kDnC / 8; idx += kDnThreads - 64) {             // keys transposed: eight tokens of one key column
      const int c = idx % kDnD, j = 8 * (idx / kDnD);
      float kv[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) kv[u] = __bfloat162float(sK[(j + u) * kDnLd + c]);
      uint4 og, od;
      uint32_t* pg = reinterpret_cast<uint32_t*>(&og);
      uint32_t* pd = reinterpret_cast<uint32_t*>(&od);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        pg[u] = pack_bf16x2(__expf(sc[j + 2 * u]) * kv[2 * u], __expf(sc[j + 2 * u + 1]) * kv[2 * u + 1]);
        pd[u] = pack_bf16x2(__expf(c_last - sc[j + 2 * u]) * kv[2 * u], __expf(c_last - sc[j + 2 * u + 1]) * kv[2 * u + 1]);
      }
      *reinterpret_cast<uint4*>(sGKT + c * kDnLc + j) = og;
      *reinterpret_cast<uint4*>(a.kdt + ws * kDnD * kDnC + (size_t)c * kDnC + j) = od;
    }
  }
  __syncthreads();

  // T V and -(T diag(exp c) K) (64 x 128 x 64): warp w computes the 16 output columns 16 w ..
  for (int pass = 0; pass < 2; ++pass) {
    const __nv_bfloat16* sB = pass == 0 ? sVT : sGKT;
    FragC acc[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) wmma::fill_fragment(acc[m], 0.f);
    for (int kk = 0; kk < kDnC / 16; ++kk) {
      FragB fb;
      wmma::load_matrix_sync(fb, sB + (16 * warp) * kDnLc + 16 * kk, kDnLc);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        FragA fa;
        wmma::load_matrix_sync(fa, sT + (16 * m) * kDnLc + 16 * kk, kDnLc);
        wmma::mma_sync(acc[m], fa, fb, acc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) wmma::store_matrix_sync(sF + (16 * m) * kDnLf + 16 * warp, acc[m], kDnLf, wmma::mem_row_major);
    __syncthreads();
    if (pass == 0) {                    // transposed: 16 values x 2 groups of eight tokens per warp step (whole 32-byte sectors)
      __nv_bfloat16* dst = a.uv + ws * kDnC * kDnD;
      for (int idx = tid; idx < kDnD * kDnC / 8; idx += kDnThreads) {
        const int j = 8 * ((idx & 1) + 2 * (idx / (2 * kDnD))), v = (idx >> 1) % kDnD;
        uint4 o;
        uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int u = 0; u < 4; ++u) po[u] = pack_bf16x2(sF[(j + 2 * u) * kDnLf + v], sF[(j + 2 * u + 1) * kDnLf + v]);
        *reinterpret_cast<uint4*>(dst + (size_t)v * kDnC + j) = o;
      }
    } else {
      __nv_bfloat16* dst = a.nw + ws * kDnC * kDnD;
      for (int idx = tid; idx < kDnC * kDnD / 4; idx += kDnThreads) {
        const float4 f = *reinterpret_cast<const float4*>(sF + (idx / (kDnD / 4)) * kDnLf + 4 * (idx % (kDnD / 4)));
        *reinterpret_cast<uint2*>(dst + 4 * idx) = make_uint2(pack_bf16x2(-f.x, -f.y), pack_bf16x2(-f.z, -f.w));
      }
    }
    __syncthreads();
  }
  if (tid == 0) a.glast[ws] = __expf(c_last);
}

// One stage of the scan's operands in shared memory (bf16): exp(c) Q and -(T diag(exp c) K) [token][key], decayed keys [key][token], M, T V [value][token]
constexpr int kScanNw = kDnC * kDnLd, kScanKd = 2 * kDnC * kDnLd, kScanM = kScanKd + kDnD * kDnLc, kScanUv = kScanM + kDnC * kDnLc;
// NS CTAs share a head: each has 128 / NS values, and finishes (norm, gate) 64 / NS tokens of a chunk, in one or (NS > 1) two buffers of output rows.
__host__ __device__ constexpr int scan_stage(int ns) { return kScanUv + kDnD / ns * kDnLc; }
__host__ __device__ constexpr int scan_smem(int ns) { return 2 * scan_stage(ns) * 2 + (ns > 1 ? 2 : 1) * kDnC / ns * kDnLf * 4; }

__device__ __forceinline__ void dn_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The right operands of two neighbouring 8-column tiles for 16 k: rows n .. n + 15 of a tile stored [n][k]; `addr` is this lane's row address
// (row (lane >> 4) * 8 + (lane & 7), k offset ((lane >> 3) & 1) * 8).
__device__ __forceinline__ void dn_ldm(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dn_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_u32(dst)), "l"(src) : "memory");
}
// accumulators of the column tiles 2j and 2j + 1 -> the left operand for k = 16 j .. 16 j + 15
__device__ __forceinline__ void dn_to_a(uint32_t* a, const float* c0, const float* c1) {
  a[0] = pack_bf16x2(c0[0], c0[1]); a[1] = pack_bf16x2(c0[2], c0[3]); a[2] = pack_bf16x2(c1[0], c1[1]); a[3] = pack_bf16x2(c1[2], c1[3]);
}

// c[0 .. 7] (16 x 64) += a (16 x 16 K) times 64 rows of a tile stored [n][k] with LD elements per row; the next k step's operands are requested before this
// one's products.
template <int K, int LD>
__device__ __forceinline__ void dn_product(float (*c)[4], const uint32_t (*a)[4], uint32_t addr) {
  uint32_t b[2][4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p) dn_ldm(b[0][p], addr + (uint32_t)(16 * p * LD) * 2);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k + 1 < K)
#pragma unroll
      for (int p = 0; p < 4; ++p) dn_ldm(b[(k + 1) & 1][p], addr + (uint32_t)(16 * p * LD + 16 * (k + 1)) * 2);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      dn_mma(c[2 * p], a[k], b[k & 1][p][0], b[k & 1][p][1]);
      dn_mma(c[2 * p + 1], a[k], b[k & 1][p][2], b[k & 1][p][3]);
    }
  }
}

template <int NS>
__global__ void __launch_bounds__(kDnThreads / NS, 1)
dn_chunk_scan_kernel(const DnChunkArgs a) {
  constexpr int THREADS = kDnThreads / NS, STAGE = scan_stage(NS), TOK = kDnC / NS;
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(128) uint8_t dn_smem[];
  __nv_bfloat16* ring = reinterpret_cast<__nv_bfloat16*>(dn_smem);        // [2][STAGE]
  float* sO = reinterpret_cast<float*>(ring + 2 * STAGE);                  // [1 or 2][TOK tokens][kDnLf]

  const int h = blockIdx.x / NS, rank = blockIdx.x % NS, s = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
  const int lwarp = tid >> 5, warp = rank * (THREADS / 32) + lwarp;        // warp of the head: values 16 warp .., tokens 8 warp .. of a chunk
  const int seq_t0 = a.cu_q[s], seq_t1 = a.cu_q[s + 1];
  if (seq_t1 <= seq_t0) return;
  int cb = 0;
  for (int i = 0; i < s; ++i) cb += (a.cu_q[i + 1] - a.cu_q[i] + kDnC - 1) / kDnC;
  const int n_chunks = (seq_t1 - seq_t0 + kDnC - 1) / kDnC;

  auto fetch = [&](int ci) {                                               // chunk ci -> its stage, 16 bytes per copy
    const size_t ws = (size_t)(cb + ci) * a.dt_rank + h;
    __nv_bfloat16* st = ring + (ci & 1) * STAGE;
    const __nv_bfloat16* gq = a.gq + ws * kDnC * kDnD;
    const __nv_bfloat16* nw = a.nw + ws * kDnC * kDnD;
    const __nv_bfloat16* kd = a.kdt + ws * kDnC * kDnD;
    const __nv_bfloat16* uv = a.uv + ws * kDnC * kDnD + rank * (kDnD / NS) * kDnC;
    const __nv_bfloat16* mq = a.mqk + ws * kDnC * kDnC;
#pragma unroll
    for (int i = 0; i < kDnC * kDnD / 8 / THREADS; ++i) {
      const int idx = tid + i * THREADS;
      const int r = idx / (kDnD / 8) * kDnLd + 8 * (idx % (kDnD / 8)), q = idx / (kDnC / 8) * kDnLc + 8 * (idx % (kDnC / 8));
      dn_copy16(st + r, gq + 8 * idx);
      dn_copy16(st + kScanNw + r, nw + 8 * idx);
      dn_copy16(st + kScanKd + q, kd + 8 * idx);
      if (i < kDnC * kDnD / NS / 8 / THREADS) dn_copy16(st + kScanUv + q, uv + 8 * idx);
      if (i < kDnC * kDnC / 8 / THREADS) dn_copy16(st + kScanM + q, mq + 8 * idx);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0);

  // state rows 16 warp .. of this head as accumulators: value rows g and g + 8, keys 8 f + 2 q and the next
  const int g = lane >> 2, q = lane & 3;
  float* st = a.state + ((size_t)a.seq_slots[s] * a.dt_rank + h) * kDnD * kDnD + (size_t)(16 * warp + g) * kDnD + 2 * q;
  float S[16][4];
#pragma unroll
  for (int f = 0; f < 16; ++f) {
    const float2 lo = *reinterpret_cast<const float2*>(st + 8 * f), hi = *reinterpret_cast<const float2*>(st + 8 * kDnD + 8 * f);
    S[f][0] = lo.x; S[f][1] = lo.y; S[f][2] = hi.x; S[f][3] = hi.y;
  }
  const int lrow = (lane >> 4) * 8 + (lane & 7), lk = ((lane >> 3) & 1) * 8;
  const uint32_t ring_u = smem_u32(ring);
  const uint32_t off_d = (uint32_t)(lrow * kDnLd + lk) * 2, off_c = (uint32_t)(lrow * kDnLc + lk) * 2;
  const float4 nwt = *reinterpret_cast<const float4*>(a.norm_w + 4 * lane);

  if constexpr (NS > 1) {     // the other CTA runs: its shared memory may be written to
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  for (int ci = 0; ci < n_chunks; ++ci) {
    const int t0 = seq_t0 + ci * kDnC, t1 = min(t0 + kDnC, seq_t1);
    const float g_last = a.glast[(size_t)(cb + ci) * a.dt_rank + h];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();          // this chunk's tiles have landed; everyone is done with the other stage and with sO
    if (ci + 1 < n_chunks) fetch(ci + 1);
    const __nv_bfloat16* stg = ring + (ci & 1) * STAGE;
    const uint32_t su = ring_u + (uint32_t)(ci & 1) * (STAGE * 2);
    float* out_rows = sO + (NS > 1 ? (ci & 1) * TOK * kDnLf : 0);

    uint32_t aS[8][4];                                                     // the state in front of the chunk as a bf16 operand
#pragma unroll
    for (int k = 0; k < 8; ++k) dn_to_a(aS[k], S[2 * k], S[2 * k + 1]);

    // U^T = (T V)^T - S0 (T diag(exp c) K)^T
    uint32_t aU[4][4];
    {
      float U[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const __nv_bfloat16* p = stg + kScanUv + (16 * lwarp + g) * kDnLc + 8 * n + 2 * q;
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + 8 * kDnLc));
        U[n][0] = lo.x; U[n][1] = lo.y; U[n][2] = hi.x; U[n][3] = hi.y;
      }
      dn_product<8, kDnLd>(U, aS, su + kScanNw * 2 + off_d);
#pragma unroll
      for (int k = 0; k < 4; ++k) dn_to_a(aU[k], U[2 * k], U[2 * k + 1]);
    }

    // O^T = S0 (diag(exp c) Q)^T + U^T M^T
    {
      float O[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) O[n][e] = 0.f;
      dn_product<8, kDnLd>(O, aS, su + off_d);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int p = k; p < 4; ++p) {                                      // M is lower triangular
          uint32_t b[4];
          dn_ldm(b, su + kScanM * 2 + off_c + (uint32_t)(16 * p * kDnLc + 16 * k) * 2);
          dn_mma(O[2 * p], aU[k], b[0], b[1]);
          dn_mma(O[2 * p + 1], aU[k], b[2], b[3]);
        }
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const int t = 8 * n + 2 * q;                                       // tokens t and t + 1 go to the CTA that finishes them
        float* o = out_rows + (t % TOK) * kDnLf + 16 * warp + g;
        if constexpr (NS == 1) {
          o[0] = O[n][0]; o[kDnLf] = O[n][1]; o[8] = O[n][2]; o[kDnLf + 8] = O[n][3];
        } else {
          uint32_t r;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(o)), "r"(8 * n / TOK));
#pragma unroll
          for (int e = 0; e < 4; ++e)
            asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(r + (uint32_t)((e & 1) * kDnLf + (e >> 1) * 8) * 4), "f"(O[n][e]) : "memory");
        }
      }
    }
    uint2 zr[8];                                                           // gates of the tokens this warp will finish
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = t0 + 8 * warp + i;
      zr[i] = t < t1 ? *reinterpret_cast<const uint2*>(a.z + (size_t)t * a.ld_z + h * kDnD + 4 * lane) : make_uint2(0u, 0u);
    }
    // the output rows are complete.  (NS > 1: a CTA writes this buffer again two chunks on, behind a barrier at which the others arrive with this one read)
    if constexpr (NS == 1) __syncthreads();
    else {
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    // S = exp(c_last) S + U^T diag(exp(c_last - c_j)) K
#pragma unroll
    for (int f = 0; f < 16; ++f)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[f][e] *= g_last;
    dn_product<4, kDnLc>(S, aU, su + kScanKd * 2 + off_c);
    dn_product<4, kDnLc>(S + 8, aU, su + (kScanKd + 64 * kDnLc) * 2 + off_c);

    // gated RMSNorm of the output rows: warp w takes the tokens 8 w .. 8 w + 7, a lane four features
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = t0 + 8 * warp + i;
      if (t >= t1) break;
      const float4 o = *reinterpret_cast<const float4*>(out_rows + (8 * lwarp + i) * kDnLf + 4 * lane);
      const float ss = dn_warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w);
      const float sc = rsqrtf(ss / (float)kDnD + a.eps);
      const __nv_bfloat16* zb = reinterpret_cast<const __nv_bfloat16*>(&zr[i]);
      const float ov[4] = {o.x, o.y, o.z, o.w}, nv[4] = {nwt.x, nwt.y, nwt.z, nwt.w};
      __nv_bfloat16 y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float zv = __bfloat162float(zb[e]);
        y[e] = __float2bfloat16(ov[e] * sc * nv[e] * (zv / (1.0f + __expf(-zv))));
      }
      *reinterpret_cast<uint2*>(a.out + ((size_t)t * a.dt_rank + h) * kDnD + 4 * lane) = *reinterpret_cast<const uint2*>(y);
    }
  }
#pragma unroll
  for (int f = 0; f < 16; ++f) {
    *reinterpret_cast<float2*>(st + 8 * f) = make_float2(S[f][0], S[f][1]);
    *reinterpret_cast<float2*>(st + 8 * kDnD + 8 * f) = make_float2(S[f][2], S[f][3]);
  }
}

// bytes of one workspace entry (chunk, head): three 64 x 128 tiles, one 128 x 64, one 64 x 64 (bf16) and the chunk's total decay
constexpr size_t kDnEntryBf16 = 3 * (size_t)kDnC * kDnD + (size_t)kDnD * kDnC + (size_t)kDnC * kDnC;

}  // namespace gb

using namespace gb;

// Upper bound of the chunks of `total_tokens` tokens in `n_seqs` sequences (each sequence may end in a partial chunk), and the
// workspace the chunked scan needs for it.
GB_API long gb_deltanet_chunk_workspace(long total_tokens, int n_seqs, int dt_rank) {
  const long chunks = total_tokens / kDnC + n_seqs;
  return chunks * dt_rank * (long)(kDnEntryBf16 * 2 + 4) + 1024;
}

GB_API int gb_deltanet_chunked(const void* qkv, int ld_qkv, const void* z, int ld_z, const float* ab, const float* a, const float* dt_bias,
                               const float* norm_w, float* state, const int* cu_q, const int* seq_slots, void* out, int n_group, int dt_rank,
                               int d_state, float eps, int n_seqs, long total_tokens, void* workspace, long workspace_bytes,
                               cudaStream_t stream) {
  if (n_seqs <= 0 || total_tokens <= 0) return 0;
  if (d_state != kDnD) return fail("deltanet_chunked: d_state must be 128%s");
  if (n_group <= 0 || dt_rank % n_group) return fail("deltanet_chunked: dt_rank must be a multiple of n_group%s");
  if ((ld_qkv % 4) || (ld_z % 4) || ((uintptr_t)qkv % 8) || ((uintptr_t)z % 8) || ((uintptr_t)out % 8) || ((uintptr_t)norm_w % 16) ||
      ((uintptr_t)state % 32))
    return fail("deltanet_chunked: rows must be 8-byte aligned (state 32, norm weights 16)%s");
  if (workspace == nullptr || workspace_bytes < gb_deltanet_chunk_workspace(total_tokens, n_seqs, dt_rank) || ((uintptr_t)workspace % 256))
    return fail("deltanet_chunked: workspace too small or not 256-byte aligned%s");
  const long chunks = total_tokens / kDnC + n_seqs;
  const size_t entries = (size_t)chunks * dt_rank;
  DnChunkArgs g;
  g.qkv = (const __nv_bfloat16*)qkv; g.ld_qkv = ld_qkv; g.z = (const __nv_bfloat16*)z; g.ld_z = ld_z; g.ab = ab; g.a = a; g.dt_bias = dt_bias;
  g.norm_w = norm_w; g.state = state; g.cu_q = cu_q; g.seq_slots = seq_slots; g.out = (__nv_bfloat16*)out; g.n_group = n_group;
  g.dt_rank = dt_rank; g.n_seqs = n_seqs; g.eps = eps;
  __nv_bfloat16* w = (__nv_bfloat16*)workspace;
  g.gq = w; w += entries * kDnC * kDnD;
  g.nw = w; w += entries * kDnC * kDnD;
  g.uv = w; w += entries * kDnC * kDnD;
  g.kdt = w; w += entries * kDnD * kDnC;
  g.mqk = w; w += entries * kDnC * kDnC;
  g.glast = (float*)w;
  static bool attr_set = false;
  if (!attr_set) {
    GB_CUDA_OK(cudaFuncSetAttribute(dn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrepSmem));
    GB_CUDA_OK(cudaFuncSetAttribute(dn_chunk_scan_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, scan_smem(1)));
    GB_CUDA_OK(cudaFuncSetAttribute(dn_chunk_scan_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, scan_smem(2)));
    attr_set = true;
  }
  launch_k(dn_chunk_prep_kernel, dim3((unsigned)chunks, dt_rank), kDnThreads, kPrepSmem, stream, g);
  GB_CUDA_OK(cudaGetLastError());
  // two CTAs per head where they all fit the GPU at once; else a second round would cost more than the shared tensor cores
  if (2L * dt_rank * n_seqs <= sm_count())
    GB_CUDA_OK(launch_k_cluster(dn_chunk_scan_kernel<2>, dim3(2 * dt_rank, n_seqs), dim3(kDnThreads / 2), (size_t)scan_smem(2), stream, 2u, g));
  else
    launch_k(dn_chunk_scan_kernel<1>, dim3(dt_rank, n_seqs), kDnThreads, scan_smem(1), stream, g);
  GB_CUDA_OK(cudaGetLastError());
  return 0;
}
