// Gated-delta-rule recurrence of a linear-attention (gated delta net) layer over packed sequences: the LinearAttention contrib op
// with update_rule "gated_delta" that the reference's builder emits for Qwen3-Next / Qwen3.5 style hybrids
// (src/python/py/models/builders/base.py:3419-3452, qwen.py:1842-1860; state handling src/models/recurrent_state.h:12-66).
//
// Two kernels over the same state pool (fp32, [slots][value heads][dk][dv] with a slot stride), for bf16 and fp32 activations and any
// dk / dv (rows and columns past the sizes are zeros):
//   gated_delta_kernel        decode-shaped steps and portions of a few tokens.  One CTA = (request, value head, 32 columns of the head's state S [dk, dv]); a thread
//                             keeps 16 to 64 rows of one column, the lanes of a warp are neighbouring columns (the state streams in
//                             full lines), the row splits of a column meet in shared memory.
//   gated_delta_chunk_kernel  prompts.  Tokens four at a time; the row splits of a column are lanes of one warp, so that dot products are
//                             finished by shuffles and the loop over blocks has no barrier; the keys and queries of a chunk of tokens
//                             are normalised into shared memory; lengths, gates and the products within a block come from gdn_prepare_kernel.
// Per token, with k_t, q_t of the head:
//     S[:, j] *= exp(g);   mem = sum_i S[i, j] k[i];   delta = (v[j] - mem) * beta;   S[i, j] += k[i] * delta;   o[j] = sum_i S[i, j] q[i]
// Tokens of a request are walked in order inside the kernel (a decode step is one token, a prompt chunk many); the state is read
// from / written to the request's slot once per launch.  A request whose past length is 0 starts from zero.
// This file is built without fast-math: the recurrence and all that feeds it is plain fp32.
#include "common.cuh"
#include "kernels.h"

namespace ogb {

template <typename T> __device__ __forceinline__ float act_f32(T v);
template <> __device__ __forceinline__ float act_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float act_f32<__nv_bfloat16>(__nv_bfloat16 v) { return bf2f(v); }
template <typename T> __device__ __forceinline__ T act_from(float v);
template <> __device__ __forceinline__ float act_from<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 act_from<__nv_bfloat16>(float v) { return f2bf(v); }

template <typename T>
struct GdnParams {
  const T *q, *k, *v;                 // rows of token t at q + t * tok_stride (+ head offsets): separate tensors or slices of one projection
  long long tok_stride_qk, tok_stride_v;
  const float *g, *beta;              // [T, Hv] log-decay and write strength ...
  const T *b_raw, *a_raw;             // ... or (g == null) their raw projections [T, Hv] with a row stride: beta = sigmoid(b),
  long long ba_stride;                //     g = neg_exp_a[h] * softplus(a + dt_bias[h])
  const float *neg_exp_a, *dt_bias;
  int l2norm;                         // q and k are L2-normalised per head here (q then scaled by q_scale)
  float q_scale;
  float l2_eps;                       // > 0: unit vectors are x / sqrt(sum(x^2) + l2_eps); 0: x / max(sqrt(sum(x^2)), 1e-6)
  float* state;
  long long slot_stride;              // floats between the states of consecutive slots
  const int32_t *slots, *cu_seqlens, *past_lens;
  T* out;
  int Hk, Hv, dv, dk;
};

__device__ __forceinline__ float inv_length(float sumsq, float l2_eps) {
  return l2_eps > 0.f ? 1.f / sqrtf(sumsq + l2_eps) : 1.f / fmaxf(sqrtf(sumsq), 1e-6f);
}

// decay exp(g) and write strength beta of token t, value head h
template <typename T>
__device__ __forceinline__ void gdn_gates(const GdnParams<T>& p, int t, int h, float& decay, float& beta) {
  if (p.g) {
    decay = expf(p.g[size_t(t) * p.Hv + h]);
    beta = p.beta[size_t(t) * p.Hv + h];
  } else {
    const float ar = act_f32(p.a_raw[size_t(t) * p.ba_stride + h]) + p.dt_bias[h];
    const float soft = ar > 20.f ? ar : log1pf(expf(ar));
    decay = expf(p.neg_exp_a[h] * soft);
    beta = 1.f / (1.f + expf(-act_f32(p.b_raw[size_t(t) * p.ba_stride + h])));
  }
}

constexpr int GDN_MAX_DK = 1024, GDN_MAX_SPLITS = 16;

// FULL: dk is a multiple of NPT, no row is past the size.
template <typename T, int NPT, bool FULL>
__global__ void __launch_bounds__(512) gated_delta_kernel(GdnParams<T> p) {
  // thread (j, sp): column j of the state, rows [sp * NPT, (sp + 1) * NPT); the two dot products of a token (with k, then with q)
  // are summed over the splits through shared memory
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y;
  const int Hk = p.Hk, Hv = p.Hv, dv = p.dv, dk = p.dk;
  const int splits = blockDim.x / 32;                         // 32 columns per CTA (blockIdx.z walks the column tiles)
  const int jj = threadIdx.x % 32, j = blockIdx.z * 32 + jj, sp = threadIdx.x / 32, n0 = sp * NPT;
  const int hk = h / (Hv / Hk);
  const int t0 = p.cu_seqlens[b], t1 = p.cu_seqlens[b + 1];
  if (t0 >= t1) return;
  __shared__ float sk[GDN_MAX_DK], sq[GDN_MAX_DK];
  __shared__ float sM[GDN_MAX_SPLITS][32], sO[GDN_MAX_SPLITS][32];
  __shared__ float sNorm[2][16];
  float* S = p.state + size_t(p.slots[b]) * p.slot_stride + (size_t(h) * dk + n0) * dv;
  float col[NPT];
  const bool live = j < dv;
  const bool fresh = p.past_lens[b] == 0;
#pragma unroll
  for (int i = 0; i < NPT; ++i) col[i] = (live && !fresh && (FULL || n0 + i < dk)) ? S[size_t(i) * dv + j] : 0.f;
  if (!FULL) for (int i = dk + threadIdx.x; i < splits * NPT; i += blockDim.x) { sk[i] = 0.f; sq[i] = 0.f; }
  for (int t = t0; t < t1; ++t) {
    __syncthreads();
    float ssk = 0.f, ssq = 0.f;
    for (int i = threadIdx.x; i < dk; i += blockDim.x) {
      const float kv_ = act_f32(p.k[size_t(t) * p.tok_stride_qk + size_t(hk) * dk + i]);
      const float qv_ = act_f32(p.q[size_t(t) * p.tok_stride_qk + size_t(hk) * dk + i]);
      sk[i] = kv_; sq[i] = qv_;
      ssk += kv_ * kv_; ssq += qv_ * qv_;
    }
    float rk = 1.f, rq = 1.f;
    if (p.l2norm) {
      ssk = warp_sum(ssk); ssq = warp_sum(ssq);
      if ((threadIdx.x & 31) == 0) { sNorm[0][threadIdx.x >> 5] = ssk; sNorm[1][threadIdx.x >> 5] = ssq; }
    }
    __syncthreads();
    if (p.l2norm) {
      float tk = 0.f, tq = 0.f;
      for (int w = 0; w < splits; ++w) { tk += sNorm[0][w]; tq += sNorm[1][w]; }
      rk = inv_length(tk, p.l2_eps);
      rq = p.q_scale * inv_length(tq, p.l2_eps);
    }
    float decay, bt;
    gdn_gates(p, t, h, decay, bt);
    float part[4] = {0.f, 0.f, 0.f, 0.f};                  // (four short chains: half the rounding error of one long one, and less latency)
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      col[i] *= decay;
      part[i & 3] = fmaf(col[i], sk[n0 + i], part[i & 3]);
    }
    float mem = (part[0] + part[1]) + (part[2] + part[3]);
    if (splits > 1) {
      sM[sp][jj] = mem;
      __syncthreads();
      mem = 0.f;
      for (int s2 = 0; s2 < splits; ++s2) mem += sM[s2][jj];
    }
    const float vj = live ? act_f32(p.v[size_t(t) * p.tok_stride_v + size_t(h) * dv + j]) : 0.f;
    const float delta = (vj - mem * rk) * bt * rk;       // the normalised key is rk * sk: once in the read, once in the write
    part[0] = part[1] = part[2] = part[3] = 0.f;
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      col[i] = fmaf(sk[n0 + i], delta, col[i]);
      part[i & 3] = fmaf(col[i], sq[n0 + i], part[i & 3]);
    }
    float o = (part[0] + part[1]) + (part[2] + part[3]);
    if (splits > 1) {
      sO[sp][jj] = o;
      __syncthreads();
      if (sp == 0)
        for (int s2 = 1; s2 < splits; ++s2) o += sO[s2][jj];
    }
    if (live && sp == 0) p.out[(size_t(t) * Hv + h) * dv + j] = act_from<T>(o * rq);
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < NPT; ++i) if (FULL || n0 + i < dk) S[size_t(i) * dv + j] = col[i];
  }
}

// What the chunk kernel needs of a block of four tokens beside their rows, per value head: E_st (k_s . k_t) for (s, t) = (0,1) (0,2) (1,2) (0,3) (1,3)
// (2,3) at 0 .. 5; E_st (k_s . q_t) at 8 + 4 t + s, s <= t; D_t at 24; E_t3 at 28; beta_t at 32 (names below).  Tokens past a request's end:
// keys, values and beta zero, decay one.  Blocks of request r are numbered from cu_seqlens[r] / 4 + r on.
constexpr int GDN_BLOCK = 4, GDN_COEF = 40;
__host__ __device__ inline long long gdn_blocks(long long T, long long B) { return T / GDN_BLOCK + B; }

// One warp per block and value head: lengths of the block's keys and queries (`lengths` [T, Hk]: the factors that make them unit vectors)
// and its coefficients.
template <typename T>
__global__ void __launch_bounds__(256) gdn_prepare_kernel(GdnParams<T> p, int B, float2* __restrict__ lengths, float* __restrict__ coef) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, h = blockIdx.y * 8 + (threadIdx.x >> 5), id = blockIdx.x;
  if (h >= p.Hv) return;
  int lo = 0, hi = B - 1;                                  // the request: last r with its first block <= id
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.cu_seqlens[mid] / GDN_BLOCK + mid <= id) lo = mid; else hi = mid - 1;
  }
  const int t0 = p.cu_seqlens[lo] + (id - p.cu_seqlens[lo] / GDN_BLOCK - lo) * GDN_BLOCK, n = min(GDN_BLOCK, p.cu_seqlens[lo + 1] - t0);
  if (n <= 0) return;
  const int dk = p.dk, rep = p.Hv / p.Hk, hk = h / rep;
  float val[16], len[8];
#pragma unroll
  for (int i = 0; i < 16; ++i) val[i] = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) len[i] = 0.f;
  for (int i = lane; i < dk; i += 32) {
    float k[4], q[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const size_t at = size_t(t0 + t) * p.tok_stride_qk + size_t(hk) * dk + i;
      k[t] = t < n ? act_f32(p.k[at]) : 0.f;
      q[t] = t < n ? act_f32(p.q[at]) : 0.f;
      len[t] = fmaf(k[t], k[t], len[t]);
      len[4 + t] = fmaf(q[t], q[t], len[4 + t]);
    }
    int j = 0;
#pragma unroll
    for (int t = 1; t < 4; ++t)
#pragma unroll
      for (int s = 0; s < t; ++s, ++j) val[j] = fmaf(k[s], k[t], val[j]);
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int s = 0; s <= t; ++s, ++j) val[j] = fmaf(k[s], q[t], val[j]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    len[i] = p.l2norm ? inv_length(warp_sum(len[i]), p.l2_eps) : 1.f;
    if (p.l2norm && i >= 4) len[i] *= p.q_scale;
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? val[i] : val[i + o], keep = up ? val[i + o] : val[i];
      val[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  const float dot = val[0] + __shfl_xor_sync(0xffffffffu, val[0], 16);       // sum number lane % 16
  float decay = 1.f, beta = 0.f;
  if (lane < n) gdn_gates(p, t0 + lane, h, decay, beta);
  float g[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) g[u] = __shfl_sync(0xffffffffu, decay, u);
  beta = __shfl_sync(0xffffffffu, beta, lane & 3);
  const int pr = lane & 15;
  const bool kq = pr >= 6;
  int t = kq ? 0 : 1, s = kq ? pr - 6 : pr;
  while (s >= t + (kq ? 1 : 0)) { s -= t + (kq ? 1 : 0); ++t; }
  auto pick = [&](int base, int i) { return i == 0 ? len[base] : i == 1 ? len[base + 1] : i == 2 ? len[base + 2] : len[base + 3]; };
  auto span = [&](int from, int to) {                      // decays of tokens from .. to
    float e = 1.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) e *= u >= from && u <= to ? g[u] : 1.f;
    return e;
  };
  float* c = coef + (size_t(id) * p.Hv + h) * GDN_COEF;
  if (lane < 16) c[kq ? 8 + 4 * t + s : pr] = dot * pick(0, s) * (kq ? pick(4, t) : pick(0, t)) * span(s + 1, t);
  else if (lane < 20) c[24 + (lane & 3)] = span(0, lane & 3);
  else if (lane < 24) c[28 + (lane & 3)] = span((lane & 3) + 1, 3);
  else if (lane < 28) c[32 + (lane & 3)] = beta;
  if (h == hk * rep && lane < n) lengths[size_t(t0 + lane) * p.Hk + hk] = make_float2(pick(0, lane), pick(4, lane));
}

// A read that the compiler does not merge with an earlier one of the same place: the value is not to be kept in registers in between.
__device__ __forceinline__ float4 ld_shared_again(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}

// A thread owns two columns and NPT rows of each, 16 * NPT >= dk; the lanes of a warp are 2 column pairs x 16 row splits.  Row of split sp,
// register i: (i / 4) * 64 + sp * 4 + i % 4, so that a thread's rows come as groups of four and the splits of a warp read two
// 128-byte lines of a key together.  CH tokens per chunk, walked in blocks of four.
// With one token at a time the kernel is a chain of latencies (dot products, shuffles, the update: 980 cycles a token).  The tokens of a block
// therefore meet the state S before the block, m_t = S^T k_t and r_t = S^T q_t, eight dot products at once, and the block's own part is put right
// with the dot products of its keys and queries, which do not depend on the state (gdn_prepare_kernel).  With the decays g_t,
// D_t = g_0 .. g_t and E_st = g_(s+1) .. g_t:
//     delta_t = beta_t (v_t - D_t m_t - sum_(s<t) E_st (k_s . k_t) delta_s)
//     o_t = D_t r_t + sum_(s<=t) E_st (k_s . q_t) delta_s            S <- D_3 S + sum_s E_s3 k_s delta_s^T
// The sixteen sums of a column pair are reduced over its lanes by halving (8 + 4 + 2 + 1 shuffles, lane j ends with sum j).
// 3001 tokens, 16 heads of 128 x 128: 1535 us with one token at a time, 1202 with all of this inside the kernel, 766 + 19 (prepare).
// vec: rows of keys and queries start on 16 bytes and dk is a multiple of 8.
// WARPS: 4 columns each; CTAS: wanted per SM (0: no bound on registers); KEEP: a block's keys stay in registers for the update, else they are read again.
// A launch that fits the GPU at once is latency bound and takes four warps with all the registers they want; one of several waves takes eight warps,
// which stage a chunk once for 32 columns, and fewer registers (us, four / eight warps: 16 requests of 400 tokens, 32 heads of 128 x 128 1690 / 1162,
// 8 of 40 111 / 81; one of 3001, 16 heads 810 / 1067).
template <typename T, int NPT, int CH, int WARPS, int CTAS, bool KEEP>
__global__ void __launch_bounds__(32 * WARPS, CTAS) gated_delta_chunk_kernel(GdnParams<T> p, const float2* __restrict__ lengths, const float* __restrict__ coef,
                                                                             int vec) {
  constexpr int DKP = NPT * 16, G4 = NPT / 4, LD = DKP + 4, BLK = GDN_BLOCK, NB = CH / BLK, COLS = 4 * WARPS, THREADS = 32 * WARPS;
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y;
  const int Hv = p.Hv, dv = p.dv, dk = p.dk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sp = lane & 15;
  const int jj = warp * 4 + (lane >> 4) * 2, j = blockIdx.z * COLS + jj;      // columns j, j + 1
  const int hk = h / (Hv / p.Hk);
  const int t0 = p.cu_seqlens[b], t1 = p.cu_seqlens[b + 1];
  if (t0 >= t1) return;
  __shared__ __align__(16) float sk[CH][LD];
  __shared__ __align__(16) float sq[CH][LD];
  __shared__ __align__(8) float sv[CH][COLS];
  __shared__ __align__(16) float scoef[NB][GDN_COEF];
  const bool live0 = j < dv, live1 = j + 1 < dv, fresh = p.past_lens[b] == 0;
  float* S = p.state + size_t(p.slots[b]) * p.slot_stride + size_t(h) * dk * dv;
  auto row_of = [&](int i) { return (i >> 2) * 64 + sp * 4 + (i & 3); };
  float c0[NPT], c1[NPT];
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    const bool ok = !fresh && row_of(i) < dk;
    c0[i] = ok && live0 ? S[size_t(row_of(i)) * dv + j] : 0.f;
    c1[i] = ok && live1 ? S[size_t(row_of(i)) * dv + j + 1] : 0.f;
  }

  // a chunk's raw keys / queries / values on their way from global memory: held in registers while the previous chunk is computed
  constexpr int VEC = DKP / 8, U = CH * VEC / THREADS;         // groups of eight columns of a row; groups of keys (and of queries) per thread
  static_assert(U * THREADS == CH * VEC && NB * (GDN_COEF / 4) <= THREADS && CH % 8 == 0, "whole passes");
  const T zero = act_from<T>(0.f);
  const int first_block = t0 / BLK + b;
  struct alignas(16) Eight { T v[8]; };
  Eight raw[2 * U];
  float2 len[U];
  T rv[CH / 8];
  float4 rc;
  auto fetch = [&](int f0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = threadIdx.x + THREADS * u, t = f0 + idx / VEC, c = (idx % VEC) * 8;
      const bool in = t < t1;
      len[u] = in ? lengths[size_t(t) * p.Hk + hk] : make_float2(0.f, 0.f);
      const size_t at = size_t(in ? t : t0) * p.tok_stride_qk + size_t(hk) * dk + c;
      if (vec && in && c < dk) {
        raw[u] = *reinterpret_cast<const Eight*>(p.k + at);
        raw[U + u] = *reinterpret_cast<const Eight*>(p.q + at);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const bool ok = in && c + e < dk;
          raw[u].v[e] = ok ? p.k[at + e] : zero;
          raw[U + u].v[e] = ok ? p.q[at + e] : zero;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < CH / 8; ++u) {
      const int idx = threadIdx.x + THREADS * u, t = f0 + idx / COLS, c = blockIdx.z * COLS + idx % COLS;
      rv[u] = t < t1 && c < dv ? p.v[size_t(t) * p.tok_stride_v + size_t(h) * dv + c] : zero;
    }
    const int blk = threadIdx.x / (GDN_COEF / 4);
    if (blk < NB && f0 + blk * BLK < t1)
      rc = reinterpret_cast<const float4*>(coef + (size_t(first_block + (f0 - t0) / BLK + blk) * Hv + h) * GDN_COEF)[threadIdx.x % (GDN_COEF / 4)];
  };
  fetch(t0);
  for (int f0 = t0; f0 < t1; f0 += CH) {
    __syncthreads();                                       // the previous chunk is no longer read
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = threadIdx.x + THREADS * u, tt = idx / VEC, c = (idx % VEC) * 8;
      float4* dk4 = reinterpret_cast<float4*>(&sk[tt][c]);
      float4* dq4 = reinterpret_cast<float4*>(&sq[tt][c]);
      const T* k = raw[u].v;
      const T* q = raw[U + u].v;
      const float nk = len[u].x, nq = len[u].y;
      dk4[0] = make_float4(act_f32(k[0]) * nk, act_f32(k[1]) * nk, act_f32(k[2]) * nk, act_f32(k[3]) * nk);
      dk4[1] = make_float4(act_f32(k[4]) * nk, act_f32(k[5]) * nk, act_f32(k[6]) * nk, act_f32(k[7]) * nk);
      dq4[0] = make_float4(act_f32(q[0]) * nq, act_f32(q[1]) * nq, act_f32(q[2]) * nq, act_f32(q[3]) * nq);
      dq4[1] = make_float4(act_f32(q[4]) * nq, act_f32(q[5]) * nq, act_f32(q[6]) * nq, act_f32(q[7]) * nq);
    }
#pragma unroll
    for (int u = 0; u < CH / 8; ++u) {
      const int idx = threadIdx.x + THREADS * u;
      sv[idx / COLS][idx % COLS] = act_f32(rv[u]);
    }
    if (threadIdx.x < NB * (GDN_COEF / 4)) reinterpret_cast<float4*>(&scoef[0][0])[threadIdx.x] = rc;
    __syncthreads();
    if (f0 + CH < t1) fetch(f0 + CH);
    const int n = min(CH, t1 - f0);
    for (int blk = 0; blk * BLK < n; ++blk) {
      const int tt = blk * BLK;
      float kk[KEEP ? BLK : 1][KEEP ? NPT : 1], val[16];
#pragma unroll
      for (int t = 0; t < BLK; ++t) {
        const float4* k4 = reinterpret_cast<const float4*>(sk[tt + t]) + sp;
        const float4* q4 = reinterpret_cast<const float4*>(sq[tt + t]) + sp;
        float m0 = 0.f, m1 = 0.f, r0 = 0.f, r1 = 0.f;
#pragma unroll
        for (int i = 0; i < G4; ++i) {
          const float4 kv = k4[i * 16], qv = q4[i * 16];
          if constexpr (KEEP) { kk[t][4 * i] = kv.x; kk[t][4 * i + 1] = kv.y; kk[t][4 * i + 2] = kv.z; kk[t][4 * i + 3] = kv.w; }
          m0 = fmaf(c0[4 * i], kv.x, m0); m1 = fmaf(c1[4 * i], kv.x, m1); r0 = fmaf(c0[4 * i], qv.x, r0); r1 = fmaf(c1[4 * i], qv.x, r1);
          m0 = fmaf(c0[4 * i + 1], kv.y, m0); m1 = fmaf(c1[4 * i + 1], kv.y, m1); r0 = fmaf(c0[4 * i + 1], qv.y, r0); r1 = fmaf(c1[4 * i + 1], qv.y, r1);
          m0 = fmaf(c0[4 * i + 2], kv.z, m0); m1 = fmaf(c1[4 * i + 2], kv.z, m1); r0 = fmaf(c0[4 * i + 2], qv.z, r0); r1 = fmaf(c1[4 * i + 2], qv.z, r1);
          m0 = fmaf(c0[4 * i + 3], kv.w, m0); m1 = fmaf(c1[4 * i + 3], kv.w, m1); r0 = fmaf(c0[4 * i + 3], qv.w, r0); r1 = fmaf(c1[4 * i + 3], qv.w, r1);
        }
        val[2 * t] = m0; val[2 * t + 1] = m1; val[8 + 2 * t] = r0; val[8 + 2 * t + 1] = r1;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        const bool up = (sp & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float send = up ? val[i] : val[i + o], keep = up ? val[i + o] : val[i];
          val[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      const float mine = val[0];                           // sum number sp: m_t of column c at 2 t + c, r_t at 8 + 2 t + c
      const float* co = scoef[blk];
      const float4 dec = *reinterpret_cast<const float4*>(co + 24), to_end = *reinterpret_cast<const float4*>(co + 28);
      const float4 beta = *reinterpret_cast<const float4*>(co + 32), kk0 = *reinterpret_cast<const float4*>(co);
      const float2 kk1 = *reinterpret_cast<const float2*>(co + 4);
      float d[BLK][2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float v0 = sv[tt][jj + c], v1 = sv[tt + 1][jj + c], v2 = sv[tt + 2][jj + c], v3 = sv[tt + 3][jj + c];
        const float m0 = __shfl_sync(0xffffffffu, mine, c, 16), m1 = __shfl_sync(0xffffffffu, mine, 2 + c, 16);
        const float m2 = __shfl_sync(0xffffffffu, mine, 4 + c, 16), m3 = __shfl_sync(0xffffffffu, mine, 6 + c, 16);
        d[0][c] = (v0 - dec.x * m0) * beta.x;
        d[1][c] = (v1 - dec.y * m1 - kk0.x * d[0][c]) * beta.y;
        d[2][c] = (v2 - dec.z * m2 - kk0.y * d[0][c] - kk0.z * d[1][c]) * beta.z;
        d[3][c] = (v3 - dec.w * m3 - kk0.w * d[0][c] - kk1.x * d[1][c] - kk1.y * d[2][c]) * beta.w;
      }
      if (sp >= 8) {
        const int t = (sp - 8) >> 1, c = sp & 1;
        const float4 w = *reinterpret_cast<const float4*>(co + 8 + 4 * t);
        float o = co[24 + t] * mine;
        o = fmaf(w.x, c ? d[0][1] : d[0][0], o);
        if (t > 0) o = fmaf(w.y, c ? d[1][1] : d[1][0], o);      // (a later token's values stay out, whatever they are)
        if (t > 1) o = fmaf(w.z, c ? d[2][1] : d[2][0], o);
        if (t > 2) o = fmaf(w.w, c ? d[3][1] : d[3][0], o);
        if (tt + t < n && (c ? live1 : live0)) p.out[(size_t(f0 + tt + t) * Hv + h) * dv + j + c] = act_from<T>(o);
      }
      const float e[BLK] = {to_end.x, to_end.y, to_end.z, to_end.w};
#pragma unroll
      for (int i = 0; i < NPT; ++i) { c0[i] *= dec.w; c1[i] *= dec.w; }
#pragma unroll
      for (int t = 0; t < BLK; ++t) {
        const float e0 = e[t] * d[t][0], e1 = e[t] * d[t][1];
        if constexpr (KEEP) {
#pragma unroll
          for (int i = 0; i < NPT; ++i) { c0[i] = fmaf(kk[t][i], e0, c0[i]); c1[i] = fmaf(kk[t][i], e1, c1[i]); }
        } else {
          const uint32_t row = smem_u32(sk[tt + t]) + sp * 16;
#pragma unroll
          for (int i = 0; i < G4; ++i) {
            const float4 kv = ld_shared_again(row + i * 256);
            c0[4 * i] = fmaf(kv.x, e0, c0[4 * i]); c1[4 * i] = fmaf(kv.x, e1, c1[4 * i]);
            c0[4 * i + 1] = fmaf(kv.y, e0, c0[4 * i + 1]); c1[4 * i + 1] = fmaf(kv.y, e1, c1[4 * i + 1]);
            c0[4 * i + 2] = fmaf(kv.z, e0, c0[4 * i + 2]); c1[4 * i + 2] = fmaf(kv.z, e1, c1[4 * i + 2]);
            c0[4 * i + 3] = fmaf(kv.w, e0, c0[4 * i + 3]); c1[4 * i + 3] = fmaf(kv.w, e1, c1[4 * i + 3]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NPT; ++i) {
    if (row_of(i) >= dk) continue;
    if (live0) S[size_t(row_of(i)) * dv + j] = c0[i];
    if (live1) S[size_t(row_of(i)) * dv + j + 1] = c1[i];
  }
}

// Output gate of a gated-delta-net layer: per value head, RMS norm of the recurrence output times its weight, times silu of the gate
// projection z (a column slice of the layer's input projection).  One warp per (token, head); out rows have a stride of their own.
template <typename T>
__global__ void gdn_gate_norm_kernel(const T* __restrict__ o, const T* __restrict__ z, long long z_stride, const float* __restrict__ w, float eps,
                                     T* __restrict__ out, long long out_stride, int rows, int Hv, int dv) {
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int t = row / Hv, h = row % Hv;
  const T* src = o + size_t(row) * dv;
  float ss = 0.f;
  for (int e = lane; e < dv; e += 32) { const float x = act_f32(src[e]); ss += x * x; }
  ss = warp_sum(ss);
  const float inv = 1.f / sqrtf(ss / dv + eps);
  T* dst = out + size_t(t) * out_stride + size_t(h) * dv;
  for (int e = lane; e < dv; e += 32) {
    const float zz = act_f32(z[size_t(t) * z_stride + size_t(h) * dv + e]);
    dst[e] = act_from<T>(act_f32(src[e]) * inv * w[e] * (zz / (1.f + expf(-zz))));
  }
}

}  // namespace ogb

using namespace ogb;

template <typename T, int NPT>
static bool LaunchGdnDecode(const GdnParams<T>& p, int B, int splits, cudaStream_t s) {
  const dim3 grid(B, p.Hv, (p.dv + 31) / 32), block(32 * splits);
  return p.dk % NPT == 0 ? launch_pdl(gated_delta_kernel<T, NPT, true>, grid, block, 0, s, p)
                         : launch_pdl(gated_delta_kernel<T, NPT, false>, grid, block, 0, s, p);
}
template <typename T, int NPT, int CH, int WARPS, int CTAS, bool KEEP>
static bool LaunchGdnChunk(const GdnParams<T>& p, int B, int tokens, void* scratch, cudaStream_t s) {
  float* coef = static_cast<float*>(scratch);
  float2* lengths = reinterpret_cast<float2*>(coef + gdn_blocks(tokens, B) * p.Hv * GDN_COEF);
  const int vec = p.dk % 8 == 0 && ((reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) | size_t(p.tok_stride_qk) * sizeof(T)) & 15) == 0;
  return launch_pdl(gdn_prepare_kernel<T>, dim3(unsigned(gdn_blocks(tokens, B)), (p.Hv + 7) / 8), dim3(256), 0, s, p, B, lengths, coef) &&
         launch_pdl(gated_delta_chunk_kernel<T, NPT, CH, WARPS, CTAS, KEEP>, dim3(B, p.Hv, (p.dv + 4 * WARPS - 1) / (4 * WARPS)), dim3(32 * WARPS), 0, s, p,
                    static_cast<const float2*>(lengths), static_cast<const float*>(coef), vec);
}

// CTAs of a launch of the chunk kernel with four warps
static long long GdnTiles(int B, int Hv, int dv) { return (long long)B * Hv * ((dv + 15) / 16); }
// Whether portions of up to max_q_len tokens (0: unknown) run in blocks.  A few tokens are walked by the decode kernel, which has no second launch and
// stages nothing (us, blocks / walked, 32 heads of 128 x 128: one request of 2 / 5 tokens 14.3 / 8.0, 15.3 / 13.1; 32 of 2 / 8 tokens 162 / 36,
// 182 / 100; 8 heads of 64 x 64: one of 4 / 5 10.1 / 10.2, 10.6 / 11.9; 32 of 5 / 8 23 / 14, 22 / 19; 16 heads of 128, 8 of 8 / 12 33 / 24, 38 / 33).
// Both are 32-bit sums: 1.0e-7 to 1.3e-7 of the result's norm from 64 bits with 32-bit activations.
static bool GdnInBlocks(int B, int Hv, int dk, int dv, int max_q_len) {
  if (dk > 256) return false;
  return max_q_len == 0 || max_q_len > (GdnTiles(B, Hv, dv) >= 1024 ? 8 : dk > 64 ? 5 : 4);
}

// Bytes of scratch that a launch over `tokens` tokens of `requests` requests needs (16-byte aligned); 0: none.
OGB_API long long ogb_gated_delta_scratch_bytes(int tokens, int requests, int Hk, int Hv, int dk, int dv, int max_q_len) {
  return GdnInBlocks(requests, Hv, dk, dv, max_q_len) ? (gdn_blocks(tokens, requests) * Hv * GDN_COEF + 2ll * tokens * Hk) * 4 : 0;
}

// max_q_len: the most tokens a request of the launch feeds (1: the decode kernel; 0: unknown, treated as a prompt)
// scratch: ogb_gated_delta_scratch_bytes(tokens, B, Hk, Hv, dk, dv, max_q_len) bytes, or null: the decode kernel walks the tokens
template <typename T>
static int LaunchGatedDelta(const GdnParams<T>& p, int B, int tokens, int max_q_len, void* scratch, void* stream) {
  if (B <= 0) return 0;
  const int dk = p.dk, dv = p.dv;
  if (p.Hk <= 0 || p.Hv % p.Hk || dv <= 0 || dk <= 0) return -1;
  if (dk > GDN_MAX_DK) return -5;
  auto s = static_cast<cudaStream_t>(stream);
  bool ok;
  if (scratch && GdnInBlocks(B, p.Hv, dk, dv, max_q_len)) {
    if (reinterpret_cast<uintptr_t>(scratch) & 15) return -1;
    const bool many = GdnTiles(B, p.Hv, dv) > 2 * 148;       // more than the two per SM that are resident at once
    if (dk <= 64) ok = many ? LaunchGdnChunk<T, 4, 32, 8, 2, true>(p, B, tokens, scratch, s) : LaunchGdnChunk<T, 4, 32, 4, 1, true>(p, B, tokens, scratch, s);
    else if (dk <= 128) ok = many ? LaunchGdnChunk<T, 8, 16, 8, 2, false>(p, B, tokens, scratch, s) : LaunchGdnChunk<T, 8, 32, 4, 0, true>(p, B, tokens, scratch, s);
    else ok = many ? LaunchGdnChunk<T, 16, 16, 8, 1, true>(p, B, tokens, scratch, s) : LaunchGdnChunk<T, 16, 16, 4, 0, true>(p, B, tokens, scratch, s);
    return ok ? 0 : -4;
  }
  // measured at Qwen3.5 shapes: 32 rows per thread 51 us, 16 rows 63 us, 64 rows 54 us (64 requests)
  if (dk <= 16) ok = LaunchGdnDecode<T, 16>(p, B, 1, s);
  else if (dk <= 32 * GDN_MAX_SPLITS) ok = LaunchGdnDecode<T, 32>(p, B, (dk + 31) / 32, s);
  else ok = LaunchGdnDecode<T, 64>(p, B, (dk + 63) / 64, s);
  return ok ? 0 : -4;
}

OGB_API int ogb_gated_delta(const void* q, const void* k, const void* v, const float* g, const float* beta, float* state, const int32_t* slots,
                            const int32_t* cu_seqlens, const int32_t* past_lens, void* out, int B, int Hk, int Hv, int dk, int dv, int tokens,
                            int max_q_len, void* scratch, void* stream) {
  using T = __nv_bfloat16;
  GdnParams<T> p{};
  p.q = static_cast<const T*>(q); p.k = static_cast<const T*>(k); p.v = static_cast<const T*>(v);
  p.tok_stride_qk = static_cast<long long>(Hk) * dk; p.tok_stride_v = static_cast<long long>(Hv) * dv;
  p.g = g; p.beta = beta; p.l2norm = 0; p.q_scale = 1.f;
  p.state = state; p.slot_stride = static_cast<long long>(Hv) * dk * dv;
  p.slots = slots; p.cu_seqlens = cu_seqlens; p.past_lens = past_lens; p.out = static_cast<T*>(out);
  p.Hk = Hk; p.Hv = Hv; p.dv = dv; p.dk = dk;
  return LaunchGatedDelta(p, B, tokens, max_q_len, scratch, stream);
}

template <typename T>
static int GatedDeltaFused(const void* conv, long long conv_stride, long long q_off, long long k_off, long long v_off, const void* ba,
                           long long ba_stride, long long b_off, long long a_off, const float* neg_exp_a, const float* dt_bias, float q_scale,
                           float l2_eps, float* state, long long slot_stride, const int32_t* slots, const int32_t* cu_seqlens,
                           const int32_t* past_lens, void* out, int B, int Hk, int Hv, int dk, int dv, int tokens, int max_q_len, void* scratch, void* stream) {
  GdnParams<T> p{};
  auto c = static_cast<const T*>(conv);
  auto r = static_cast<const T*>(ba);
  p.q = c + q_off; p.k = c + k_off; p.v = c + v_off; p.tok_stride_qk = conv_stride; p.tok_stride_v = conv_stride;
  p.g = nullptr; p.beta = nullptr; p.b_raw = r + b_off; p.a_raw = r + a_off; p.ba_stride = ba_stride;
  p.neg_exp_a = neg_exp_a; p.dt_bias = dt_bias; p.l2norm = 1; p.q_scale = q_scale; p.l2_eps = l2_eps;
  p.state = state; p.slot_stride = slot_stride > 0 ? slot_stride : static_cast<long long>(Hv) * dk * dv;
  p.slots = slots; p.cu_seqlens = cu_seqlens; p.past_lens = past_lens; p.out = static_cast<T*>(out);
  p.Hk = Hk; p.Hv = Hv; p.dv = dv; p.dk = dk;
  return LaunchGatedDelta(p, B, tokens, max_q_len, scratch, stream);
}

// The recurrence fed straight from the layer's tensors: q / k / v are column ranges of the convolved projection `conv` [T, row
// stride] (q at q_off, k at k_off, v at v_off), normalised here; the decay and the write strength come from the raw b / a
// projections (column ranges of `ba`, row stride ba_stride) with the layer's -exp(A_log) and dt_bias.  l2_eps, slot_stride and
// max_q_len as in GdnParams / LaunchGatedDelta (slot_stride 0: dense); fp32: element type of conv, ba and out (else bf16).
OGB_API int ogb_gated_delta_fused(const void* conv, long long conv_stride, long long q_off, long long k_off, long long v_off, const void* ba,
                                  long long ba_stride, long long b_off, long long a_off, const float* neg_exp_a, const float* dt_bias,
                                  float q_scale, float l2_eps, float* state, long long slot_stride, const int32_t* slots,
                                  const int32_t* cu_seqlens, const int32_t* past_lens, void* out, int B, int Hk, int Hv, int dk, int dv,
                                  int tokens, int max_q_len, int fp32, void* scratch, void* stream) {
  return fp32 ? GatedDeltaFused<float>(conv, conv_stride, q_off, k_off, v_off, ba, ba_stride, b_off, a_off, neg_exp_a, dt_bias, q_scale, l2_eps,
                                       state, slot_stride, slots, cu_seqlens, past_lens, out, B, Hk, Hv, dk, dv, tokens, max_q_len, scratch, stream)
              : GatedDeltaFused<__nv_bfloat16>(conv, conv_stride, q_off, k_off, v_off, ba, ba_stride, b_off, a_off, neg_exp_a, dt_bias, q_scale,
                                               l2_eps, state, slot_stride, slots, cu_seqlens, past_lens, out, B, Hk, Hv, dk, dv, tokens, max_q_len, scratch, stream);
}

OGB_API int ogb_gdn_gate_norm(const void* o, const void* z, long long z_stride, const float* w, float eps, void* out, long long out_stride, int T,
                              int Hv, int dv, int fp32, void* stream) {
  if (T <= 0) return 0;
  if (dv <= 0) return -1;
  const int rows = T * Hv;
  const dim3 grid((rows + 7) / 8), block(256);
  auto s = static_cast<cudaStream_t>(stream);
  using H = __nv_bfloat16;
  return (fp32 ? launch_pdl(gdn_gate_norm_kernel<float>, grid, block, 0, s, static_cast<const float*>(o), static_cast<const float*>(z), z_stride, w, eps,
                            static_cast<float*>(out), out_stride, rows, Hv, dv)
               : launch_pdl(gdn_gate_norm_kernel<H>, grid, block, 0, s, static_cast<const H*>(o), static_cast<const H*>(z), z_stride, w, eps,
                            static_cast<H*>(out), out_stride, rows, Hv, dv)) ? 0 : -4;
}

// ---------------------------------------------------------------------------------------------- Mamba-2 selective scan
// The state-space recurrence of a Mamba-2 layer over packed sequences (GraniteMoeHybrid; reference: the Mamba2 branch of
// src/models/recurrent_state.cpp keeps its conv / ssm states, the layer itself is an opaque graph there).  Per head h with
// group gr = h / (heads / groups), per token t, with dt already softplus'ed:
//     S *= exp(dt[t, h] * A[h]);   S[n][p] += dt[t, h] * x[t, h, p] * B[t, gr, n];   y[t, h, p] = sum_n S[n][p] * C[t, gr, n] + D[h] * x[t, h, p]
// state [slots][heads][N][P] fp32, updated in place for the request slots (a request whose past length is 0 starts from a
// zero state).  One CTA per (request, head); a thread keeps 16 to 64 rows of one state column in registers (the rows of a column
// are split over up to 8 threads whose partial sums meet in shared memory), the token's B and C rows sit in
// shared memory; the tokens of a chunk are walked in order.
namespace ogb {
template <int NPT>
__global__ void __launch_bounds__(512) mamba2_scan_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ dt, const float* __restrict__ neg_a, const __nv_bfloat16* __restrict__ Bm,
    const __nv_bfloat16* __restrict__ Cm, const float* __restrict__ Dv, float* __restrict__ state, const int32_t* __restrict__ slots,
    const int32_t* __restrict__ cu_seqlens, const int32_t* __restrict__ past_lens, __nv_bfloat16* __restrict__ out, int heads, int groups, int P,
    int N, long long x_stride, long long bc_stride, const __nv_bfloat16* __restrict__ dt_raw, long long dt_stride,
    const float* __restrict__ dt_bias) {
  // x_stride / bc_stride: elements between the rows of consecutive tokens in x and in Bm / Cm (tensors of their own, or column
  // ranges of one convolved projection);
  // dt_raw (dt == null): the raw step projection [T, heads] with a row stride, step = softplus(dt_raw + dt_bias[h]) computed here
  // thread (j, sp): column j of the state, rows [sp * NPT, (sp + 1) * NPT); the partial dot products of the splits meet in shared memory
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y;
  const int splits = N / NPT, Pp = blockDim.x / splits;
  const int j = threadIdx.x % Pp, sp = threadIdx.x / Pp, n0 = sp * NPT;
  const int gr = h / (heads / groups);
  const int t0 = cu_seqlens[b], t1 = cu_seqlens[b + 1];
  if (t0 >= t1) return;
  __shared__ float sB[256], sC[256];
  __shared__ float sY[8][128];
  float* S = state + ((size_t(slots[b]) * heads + h) * N + n0) * P;
  float col[NPT];
  const bool live = j < P;
  const bool fresh = past_lens[b] == 0;
#pragma unroll
  for (int i = 0; i < NPT; ++i) col[i] = (live && !fresh) ? S[size_t(i) * P + j] : 0.f;
  const float a = neg_a[h], d = Dv[h];
  for (int t = t0; t < t1; ++t) {
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      sB[i] = bf2f(Bm[size_t(t) * bc_stride + size_t(gr) * N + i]);
      sC[i] = bf2f(Cm[size_t(t) * bc_stride + size_t(gr) * N + i]);
    }
    __syncthreads();
    float step;
    if (dt) step = dt[size_t(t) * heads + h];
    else {
      const float r = bf2f(dt_raw[size_t(t) * dt_stride + h]) + dt_bias[h];
      step = r > 20.f ? r : log1pf(__expf(r));
    }
    const float decay = __expf(step * a);
    const float xj = live ? bf2f(x[size_t(t) * x_stride + size_t(h) * P + j]) : 0.f;
    const float dx = step * xj;
    float y = 0.f;
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      col[i] = fmaf(col[i], decay, dx * sB[n0 + i]);
      y = fmaf(col[i], sC[n0 + i], y);
    }
    if (splits > 1) {
      sY[sp][j] = y;
      __syncthreads();
      if (sp == 0)
        for (int q = 1; q < splits; ++q) y += sY[q][j];
    }
    if (live && sp == 0) out[(size_t(t) * heads + h) * P + j] = f2bf(y + d * xj);
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < NPT; ++i) S[size_t(i) * P + j] = col[i];
  }
}
}  // namespace ogb

static int LaunchMamba2(const void* x, const float* dt, const float* neg_a, const void* Bm, const void* Cm, const float* Dv, float* state,
                        const int32_t* slots, const int32_t* cu_seqlens, const int32_t* past_lens, void* out, int B, int heads, int groups, int P,
                        int N, long long x_stride, long long bc_stride, const void* dt_raw, long long dt_stride, const float* dt_bias, void* stream) {
  if (B <= 0) return 0;
  if (heads <= 0 || groups <= 0 || heads % groups || P <= 0 || P > 128) return -1;
  if (N < 16 || N > 256 || (N & (N - 1))) return -5;
  const int Pp = (P + 31) / 32 * 32;
  int npt = N < 32 ? N : 32;
  if (Pp * (N / npt) > 512) npt = 64;
  const int splits = N / npt;
  if (splits > 8 || Pp * splits > 512) return -5;
  dim3 grid(B, heads), block(Pp * splits);
  auto s = static_cast<cudaStream_t>(stream);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto Bp = static_cast<const __nv_bfloat16*>(Bm);
  auto Cp = static_cast<const __nv_bfloat16*>(Cm);
  auto O = static_cast<__nv_bfloat16*>(out);
  auto R = static_cast<const __nv_bfloat16*>(dt_raw);
  bool ok;
  switch (npt) {
    case 16: ok = ogb::launch_pdl(ogb::mamba2_scan_kernel<16>, grid, block, 0, s, X, dt, neg_a, Bp, Cp, Dv, state, slots, cu_seqlens, past_lens, O, heads, groups, P, N, x_stride, bc_stride, R, dt_stride, dt_bias); break;
    case 32: ok = ogb::launch_pdl(ogb::mamba2_scan_kernel<32>, grid, block, 0, s, X, dt, neg_a, Bp, Cp, Dv, state, slots, cu_seqlens, past_lens, O, heads, groups, P, N, x_stride, bc_stride, R, dt_stride, dt_bias); break;
    case 64: ok = ogb::launch_pdl(ogb::mamba2_scan_kernel<64>, grid, block, 0, s, X, dt, neg_a, Bp, Cp, Dv, state, slots, cu_seqlens, past_lens, O, heads, groups, P, N, x_stride, bc_stride, R, dt_stride, dt_bias); break;
    default: return -5;
  }
  return ok ? 0 : -4;
}

OGB_API int ogb_mamba2_scan(const void* x, const float* dt, const float* neg_a, const void* Bm, const void* Cm, const float* Dv, float* state,
                            const int32_t* slots, const int32_t* cu_seqlens, const int32_t* past_lens, void* out, int B, int heads, int groups,
                            int P, int N, void* stream) {
  return LaunchMamba2(x, dt, neg_a, Bm, Cm, Dv, state, slots, cu_seqlens, past_lens, out, B, heads, groups, P, N,
                      static_cast<long long>(heads) * P, static_cast<long long>(groups) * N, nullptr, 0, nullptr, stream);
}

// The scan fed straight from the layer's tensors: x / B / C are column ranges of the convolved projection `conv` (row stride
// conv_stride; x at 0, B at heads * P, C after B), the step comes from the raw dt projection (a column range of `proj`) with dt_bias.
OGB_API int ogb_mamba2_scan_fused(const void* conv, long long conv_stride, const void* dt_raw, long long dt_stride, const float* dt_bias,
                                  const float* neg_a, const float* Dv, float* state, const int32_t* slots, const int32_t* cu_seqlens,
                                  const int32_t* past_lens, void* out, int B, int heads, int groups, int P, int N, void* stream) {
  auto c = static_cast<const __nv_bfloat16*>(conv);
  const long long I = static_cast<long long>(heads) * P, GN = static_cast<long long>(groups) * N;
  return LaunchMamba2(c, nullptr, neg_a, c + I, c + I + GN, Dv, state, slots, cu_seqlens, past_lens, out, B, heads, groups, P, N, conv_stride,
                      conv_stride, dt_raw, dt_stride, dt_bias, stream);
}

// Output gate of a Mamba-2 layer: y * silu(z) (z a column range of the input projection), then an RMS norm over the whole width with
// the layer's weight.  One CTA per token.
namespace ogb {
__global__ void __launch_bounds__(256) mamba_gate_norm_kernel(const __nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ z,
                                                             long long z_stride, const float* __restrict__ w, float eps,
                                                             __nv_bfloat16* __restrict__ out, int I) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  __shared__ float part[8];
  float v[16];
  float ss = 0.f;
  int n = 0;
  for (int e = threadIdx.x; e < I; e += blockDim.x, ++n) {
    const float zz = bf2f(z[size_t(t) * z_stride + e]);
    v[n] = bf2f(y[size_t(t) * I + e]) * (zz / (1.f + __expf(-zz)));
    ss += v[n] * v[n];
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int i = 0; i < int(blockDim.x >> 5); ++i) tot += part[i];
  const float inv = rsqrtf(tot / I + eps);
  n = 0;
  for (int e = threadIdx.x; e < I; e += blockDim.x, ++n) out[size_t(t) * I + e] = f2bf(v[n] * inv * w[e]);
}
}  // namespace ogb

OGB_API int ogb_mamba_gate_norm(const void* y, const void* z, long long z_stride, const float* w, float eps, void* out, int T, int I, void* stream) {
  if (T <= 0) return 0;
  if (I <= 0 || I > 16 * 256) return -1;
  return ogb::launch_pdl(ogb::mamba_gate_norm_kernel, dim3(T), dim3(256), 0, static_cast<cudaStream_t>(stream),
                         static_cast<const __nv_bfloat16*>(y), static_cast<const __nv_bfloat16*>(z), z_stride, w, eps,
                         static_cast<__nv_bfloat16*>(out), I) ? 0 : -4;
}

// ---------------------------------------------------------------------------------------------- state snapshots
// Copies the recurrent states of `count` slots between two pools of the same shape [layers][slots][slot_elems] (or inside
// one): dst[l][dst_slots[i]] = src[l][src_slots[i]].  Speculative decoding saves a request's state before the verification
// pass feeds draft tokens into it and puts it back when some of them are rejected (reference: CopyStateSlotsKernel,
// src/cuda/model_kernels.cu:488-520, used by src/models/recurrent_state.cpp for its snapshot slots).  16 bytes per thread.
namespace ogb {
__global__ void copy_state_slots_kernel(const float4* __restrict__ src, float4* __restrict__ dst, long long layer_vecs, long long slot_vecs,
                                        const int* __restrict__ src_slots, const int* __restrict__ dst_slots, int count) {
  const int pair = blockIdx.y % count, layer = blockIdx.y / count;
  const float4* s = src + size_t(layer) * layer_vecs + size_t(src_slots[pair]) * slot_vecs;
  float4* d = dst + size_t(layer) * layer_vecs + size_t(dst_slots[pair]) * slot_vecs;
  for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < slot_vecs; i += (long long)gridDim.x * blockDim.x) d[i] = s[i];
}
}  // namespace ogb

OGB_API int ogb_copy_state_slots(const float* src, float* dst, int layers, int slots, long long slot_elems, const int32_t* src_slots,
                                 const int32_t* dst_slots, int count, void* stream) {
  if (count <= 0 || layers <= 0) return 0;
  if (slot_elems <= 0 || (slot_elems % 4) || slots <= 0) return -1;
  if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) return -1;
  if (static_cast<long long>(layers) * count > 65535) return -1;
  const long long slot_vecs = slot_elems / 4;
  const int threads = 256;
  int bx = int((slot_vecs + threads - 1) / threads);
  if (bx > 128) bx = 128;
  ogb::copy_state_slots_kernel<<<dim3(bx, layers * count), threads, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), static_cast<long long>(slots) * slot_vecs, slot_vecs, src_slots, dst_slots, count);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
