// Attention over a cached latent (sm_100a), float32 and bfloat16.
//
// A token's cache row is [c | k_rot]: R = kv_rank elements of the normed latent and Dr rotated key elements that all
// heads share; pages are [n_pages, 1, 64, R + Dr].  The keys and values of the heads are never formed: a query is
// taken into the latent's space, attention weights are applied to c itself, and the value matrix of a head is applied
// to the weighted latent.  Queries in the latent's space, scores, softmax and the weighted latents are 32-bit.
//
//   latent_prepare_kernel  one block a token, from the stacked input projection proj [T, row]:
//                          cq = rmsnorm(proj[0:Rq]) * gq  -> cq_out [T, Rq]  (compute dtype)
//                          c  = rmsnorm(proj[col:col+R]) * gkv, k_rot = rotate(proj[col+R : col+R+Dr])  -> the page row
//                          (col < 0 or no pages: the layer reads another layer's cache and writes nothing)
//   latent_query_kernel    one block a (tile of 8 tokens, head): q' = [Wuk_h^T q_h | rotate(q_rot_h)], float32
//                          [T, H, R + Dr]; Wuk is [H * D, R], so q'[r] = sum_d q_h[d] Wuk[h D + d, r]
//   latent_attn_kernel     (float32, and sizes latent_attn_mma_kernel does not take) one block a (token, group of 8 heads), a warp a head: key rows of the window staged in shared
//                          memory 32 at a time for all heads of the block; a lane scores one key, the softmax runs
//                          over the warp, and the weighted sum of c has a lane own the elements r = lane, lane + 32, ...
//                          -> float32 [T, H, splits, R] without the division, and each part's maximum and sum
//   latent_output_kernel   one block a (tile of 8 tokens, head): the parts merged and divided, then
//                          y[h Dv + j] = sigmoid(gate) * sum_r Wuv[h Dv + j, r] o'[h, r], the gate one number a head or one
//                          an output element; a sink per head (a term exp(sink) of the denominator without a key) joins
//                          once, where the parts are merged
// Rotation: dims elements, pair i at angle position * inv_freq[i]; pairs = 1: elements (2i, 2i + 1), pairs = 0:
// elements (i, i + dims / 2); elements from dims on pass unchanged.  `mag` multiplies cos and sin (1 for a plain rotation;
// a stretched rotation scales both).
#include "common.cuh"
#include <math.h>

#define LT_THREADS 256
#define LT_QTHREADS 128       // threads of a block of the query kernel
#define LT_TOKENS 8          // tokens a block of the query / output kernels
#define LT_HEADS 8           // heads (warps) a block of the attention kernel
#define LT_KEYS 32           // keys staged at a time

__device__ __forceinline__ void rot_pair_index(int i, int dims, int pairs, int& a, int& b) {
  if (pairs) { a = 2 * i; b = 2 * i + 1; } else { a = i; b = i + dims / 2; }
}

template <typename T>
__global__ void __launch_bounds__(LT_THREADS) latent_prepare_kernel(
    const T* __restrict__ proj, int row, int Rq, int col, int R, int Dr, const float* __restrict__ gq,
    const float* __restrict__ gkv, float eps, const float* __restrict__ inv_freq, int dims, int pairs, float mag,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp,
    T* __restrict__ k_pages, T* __restrict__ cq_out) {
  __shared__ float red[33];
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, tid = threadIdx.x;
  const T* pr = proj + (size_t)t * row;
  float ss = 0.f, inv;
  if (Rq > 0) {                  // a layer whose queries come straight from the projection has no query latent
    for (int i = tid; i < Rq; i += LT_THREADS) { const float v = to_f32(pr[i]); ss += v * v; }
    ss = block_sum(ss, red);
    inv = rsqrtf(ss / (float)Rq + eps);
    for (int i = tid; i < Rq; i += LT_THREADS) cq_out[(size_t)t * Rq + i] = from_f32<T>(to_f32(pr[i]) * inv * gq[i]);
  }
  if (col < 0 || k_pages == nullptr) return;
  const int pos = positions[t];
  const int page = block_table[(size_t)seq_of_token[t] * maxp + (pos >> 6)];
  T* kr = k_pages + ((size_t)page * SX_PAGE + (pos & 63)) * (R + Dr);
  ss = 0.f;
  for (int i = tid; i < R; i += LT_THREADS) { const float v = to_f32(pr[col + i]); ss += v * v; }
  ss = block_sum(ss, red);
  inv = rsqrtf(ss / (float)R + eps);
  for (int i = tid; i < R; i += LT_THREADS) kr[i] = from_f32<T>(to_f32(pr[col + i]) * inv * gkv[i]);
  const T* rr = pr + col + R;
  for (int i = tid; i < dims / 2; i += LT_THREADS) {
    int ia, ib;
    rot_pair_index(i, dims, pairs, ia, ib);
    float sn, cs;
    sincosf((float)pos * inv_freq[i], &sn, &cs);
    sn *= mag;
    cs *= mag;
    const float u = to_f32(rr[ia]), v = to_f32(rr[ib]);
    kr[R + ia] = from_f32<T>(u * cs - v * sn);
    kr[R + ib] = from_f32<T>(v * cs + u * sn);
  }
  for (int i = dims + tid; i < Dr; i += LT_THREADS) kr[R + i] = rr[i];
}

extern "C" int sx_latent_prepare(const void* proj, int row, int Rq, int col, int R, int Dr, const float* gq, const float* gkv,
                                 float eps, const float* inv_freq, int dims, int pairs, float mag, const int* positions,
                                 const int* seq_of_token, const int* block_table, int maxp, void* k_pages, void* cq_out,
                                 int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (Rq < 0 || (Rq > 0 && (gq == nullptr || cq_out == nullptr)) || dims < 0 || dims > Dr || (dims & 1) || (dims > 0 && inv_freq == nullptr)) return SX_ERR_SIZE;
  if (dt == SX_F32)
    return sx_launch(latent_prepare_kernel<float>, dim3(T), dim3(LT_THREADS), 0, stream, (const float*)proj, row, Rq, col, R, Dr,
                     gq, gkv, eps, inv_freq, dims, pairs, mag, positions, seq_of_token, block_table, maxp, (float*)k_pages, (float*)cq_out);
  if (dt == SX_BF16)
    return sx_launch(latent_prepare_kernel<bf16>, dim3(T), dim3(LT_THREADS), 0, stream, (const bf16*)proj, row, Rq, col, R, Dr,
                     gq, gkv, eps, inv_freq, dims, pairs, mag, positions, seq_of_token, block_table, maxp, (bf16*)k_pages, (bf16*)cq_out);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------------------------------
// the rotated part of a head's queries and what follows it
template <typename T>
__device__ __forceinline__ void latent_query_rest(const T* q, int QW, int h, int H, int D, int Dr, int R, const float* inv_freq, int dims,
                                                  int pairs, float mag, const int* positions, float* qa, int t0, int nt, int tid, int threads) {
  for (int i = tid; i < nt * (dims / 2); i += threads) {
    const int tt = i / (dims / 2), p = i % (dims / 2);
    int ia, ib;
    rot_pair_index(p, dims, pairs, ia, ib);
    const T* qr = q + (size_t)(t0 + tt) * QW + h * (D + Dr) + D;
    float sn, cs;
    sincosf((float)positions[t0 + tt] * inv_freq[p], &sn, &cs);
    sn *= mag;
    cs *= mag;
    const float u = to_f32(qr[ia]), v = to_f32(qr[ib]);
    float* o = qa + ((size_t)(t0 + tt) * H + h) * (R + Dr) + R;
    o[ia] = u * cs - v * sn;
    o[ib] = v * cs + u * sn;
  }
  const int rest = Dr - dims;
  for (int i = tid; i < nt * rest; i += threads) {
    const int tt = i / rest, j = dims + i % rest;
    qa[((size_t)(t0 + tt) * H + h) * (R + Dr) + R + j] = to_f32(q[(size_t)(t0 + tt) * QW + h * (D + Dr) + D + j]);
  }
}

template <typename T>
__global__ void __launch_bounds__(LT_QTHREADS) latent_query_kernel(
    const T* __restrict__ q, int QW, const T* __restrict__ wuk, int H, int D, int Dr, int R, const float* __restrict__ inv_freq,
    int dims, int pairs, float mag, const int* __restrict__ positions, float* __restrict__ qa, int n_tokens) {
  extern __shared__ float qs[];          // LT_TOKENS * D; QW: elements between two tokens' queries (>= H (D + Dr))
  pdl_wait();
  pdl_trigger();
  const int t0 = blockIdx.x * LT_TOKENS, h = blockIdx.y, tid = threadIdx.x;
  const int nt = min(LT_TOKENS, n_tokens - t0);
  for (int i = tid; i < LT_TOKENS * D; i += LT_QTHREADS) {
    const int tt = i / D, d = i % D;
    qs[i] = tt < nt ? to_f32(q[(size_t)(t0 + tt) * QW + h * (D + Dr) + d]) : 0.f;
  }
  __syncthreads();
  // the grid's z axis shares the latent's elements: LT_QTHREADS a block
  for (int r = blockIdx.z * LT_QTHREADS + tid; r < min(R, (int)(blockIdx.z + 1) * LT_QTHREADS); r += LT_QTHREADS) {
    float acc[LT_TOKENS];
#pragma unroll
    for (int tt = 0; tt < LT_TOKENS; ++tt) acc[tt] = 0.f;
#pragma unroll 16
    for (int d = 0; d < D; ++d) {
      const float w = to_f32(wuk[((size_t)h * D + d) * R + r]);
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) acc[tt] = fmaf(qs[tt * D + d], w, acc[tt]);
    }
#pragma unroll
    for (int tt = 0; tt < LT_TOKENS; ++tt)
      if (tt < nt) qa[((size_t)(t0 + tt) * H + h) * (R + Dr) + r] = acc[tt];
  }
  if (blockIdx.z == 0) latent_query_rest(q, QW, h, H, D, Dr, R, inv_freq, dims, pairs, mag, positions, qa, t0, nt, tid, LT_QTHREADS);
}

// The same for even R and aligned rows: a thread forms two neighbouring elements of the latent over a quarter of the head's D
// elements (16 loads of two weights, all on their way at once, where the kernel above has a chain of 64 in batches of 16), and
// the quarters are added up in shared memory.  The weights are asked for before the wait.  Latency-bound (1.3 MB of Wuk): 23 us in
// a decode step of 8 tokens with the kernel above, 12 with this one.
#define LT_Q2_R 128           // elements of the latent a block forms
#define LT_Q2_D 16            // elements of the head whose weights a thread asks for ahead
template <typename T> struct lt_pair;
template <> struct lt_pair<bf16> { static __device__ __forceinline__ float2 get(const bf16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); } };
template <> struct lt_pair<float> { static __device__ __forceinline__ float2 get(const float* p) { return *reinterpret_cast<const float2*>(p); } };

template <typename T>
__global__ void __launch_bounds__(256) latent_query2_kernel(
    const T* __restrict__ q, int QW, const T* __restrict__ wuk, int H, int D, int Dr, int R, const float* __restrict__ inv_freq,
    int dims, int pairs, float mag, const int* __restrict__ positions, float* __restrict__ qa, int n_tokens) {
  extern __shared__ __align__(16) float sm[];
  float* part = sm;                                     // [4][LT_TOKENS][LT_Q2_R]
  float* qs = sm + 4 * LT_TOKENS * LT_Q2_R;             // [LT_TOKENS][D]
  const int t0 = blockIdx.x * LT_TOKENS, h = blockIdx.y, tid = threadIdx.x;
  const int nt = min(LT_TOKENS, n_tokens - t0);
  const int dg = tid >> 6, r = blockIdx.z * LT_Q2_R + (tid & 63) * 2;
  const int per = (D + 3) / 4, d0 = dg * per, d1 = min(D, d0 + per);
  const T* w0 = wuk + (size_t)h * D * R + r;
  float2 w[LT_Q2_D];
#pragma unroll
  for (int i = 0; i < LT_Q2_D; ++i) w[i] = r < R && d0 + i < d1 ? lt_pair<T>::get(w0 + (size_t)(d0 + i) * R) : make_float2(0.f, 0.f);
  pdl_wait();
  pdl_trigger();
  for (int i = tid; i < LT_TOKENS * D; i += 256) {
    const int tt = i / D, d = i % D;
    qs[i] = tt < nt ? to_f32(q[(size_t)(t0 + tt) * QW + h * (D + Dr) + d]) : 0.f;
  }
  __syncthreads();
  float2 acc[LT_TOKENS];
#pragma unroll
  for (int tt = 0; tt < LT_TOKENS; ++tt) acc[tt] = make_float2(0.f, 0.f);
  for (int d = d0; d < d1; d += LT_Q2_D) {
    if (d != d0) {
#pragma unroll
      for (int i = 0; i < LT_Q2_D; ++i) w[i] = r < R && d + i < d1 ? lt_pair<T>::get(w0 + (size_t)(d + i) * R) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < LT_Q2_D; ++i) {
      const int dd = min(d + i, D - 1);                 // (beyond the share the weights are zeros)
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) {
        const float x = d + i < d1 ? qs[tt * D + dd] : 0.f;
        acc[tt].x = fmaf(x, w[i].x, acc[tt].x);
        acc[tt].y = fmaf(x, w[i].y, acc[tt].y);
      }
    }
  }
#pragma unroll
  for (int tt = 0; tt < LT_TOKENS; ++tt)
    *reinterpret_cast<float2*>(part + (dg * LT_TOKENS + tt) * LT_Q2_R + (tid & 63) * 2) = acc[tt];
  __syncthreads();
  for (int i = tid; i < nt * LT_Q2_R; i += 256) {
    const int tt = i / LT_Q2_R, rr = i % LT_Q2_R, ro = blockIdx.z * LT_Q2_R + rr;
    if (ro >= R) continue;
    float v = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) v += part[(g * LT_TOKENS + tt) * LT_Q2_R + rr];
    qa[((size_t)(t0 + tt) * H + h) * (R + Dr) + ro] = v;
  }
  if (blockIdx.z == 0) latent_query_rest(q, QW, h, H, D, Dr, R, inv_freq, dims, pairs, mag, positions, qa, t0, nt, tid, 256);
}

extern "C" int sx_latent_query(const void* q, int q_ld, const void* wuk, int H, int D, int Dr, int R, const float* inv_freq, int dims,
                               int pairs, float mag, const int* positions, float* qa, int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (q_ld < H * (D + Dr)) return SX_ERR_SIZE;
  if (H <= 0 || H > 65535 || D < 0 || R <= 0 || dims < 0 || dims > Dr || (dims & 1)) return SX_ERR_SIZE;
  const size_t smem = (size_t)LT_TOKENS * (D > 0 ? D : 1) * sizeof(float);
  if (smem > 48 * 1024) return SX_ERR_SIZE;
  const size_t smem2 = (size_t)LT_TOKENS * (4 * LT_Q2_R + D) * sizeof(float);
  if ((R & 1) == 0 && D > 0 && smem2 <= 48 * 1024 && ((uintptr_t)wuk & 7) == 0) {
    dim3 grid2((T + LT_TOKENS - 1) / LT_TOKENS, H, (R + LT_Q2_R - 1) / LT_Q2_R);
    if (dt == SX_F32)
      return sx_launch(latent_query2_kernel<float>, grid2, dim3(256), smem2, stream, (const float*)q, q_ld, (const float*)wuk, H, D, Dr,
                       R, inv_freq, dims, pairs, mag, positions, qa, T);
    if (dt == SX_BF16)
      return sx_launch(latent_query2_kernel<bf16>, grid2, dim3(256), smem2, stream, (const bf16*)q, q_ld, (const bf16*)wuk, H, D, Dr,
                       R, inv_freq, dims, pairs, mag, positions, qa, T);
    return SX_ERR_DTYPE;
  }
  dim3 grid((T + LT_TOKENS - 1) / LT_TOKENS, H, (R + LT_QTHREADS - 1) / LT_QTHREADS);
  if (dt == SX_F32)
    return sx_launch(latent_query_kernel<float>, grid, dim3(LT_QTHREADS), smem, stream, (const float*)q, q_ld, (const float*)wuk, H, D, Dr,
                     R, inv_freq, dims, pairs, mag, positions, qa, T);
  if (dt == SX_BF16)
    return sx_launch(latent_query_kernel<bf16>, grid, dim3(LT_QTHREADS), smem, stream, (const bf16*)q, q_ld, (const bf16*)wuk, H, D, Dr,
                     R, inv_freq, dims, pairs, mag, positions, qa, T);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------------------------------
// RI: elements of the weighted latent a lane owns (R <= 32 * RI; with V4, R <= 128 * RI / 4).  The grid's z axis splits the
// window's key tiles among blocks (single-token steps of few sequences would otherwise fill a fraction of the SMs); every
// block writes its weighted sum without the division, out [T, H, splits, R], and its maximum and sum of weights,
// ml [T, H, splits, 2]; the output kernel merges them.
// V4 (R and Dr multiples of 4): staged rows are padded by four floats, so that rows stay 16-byte aligned and the lanes'
// 16-byte loads of different rows fall on different banks; scores take four elements of q and of the key a load, and a
// lane owns the latent's elements 4 lane .. 4 lane + 3 (+ 128, ...), which it reads and writes 16 bytes at a time.
template <typename T, int RI, bool V4>
__global__ void __launch_bounds__(LT_HEADS * 32) latent_attn_kernel(
    const float* __restrict__ qa, const T* __restrict__ k_pages, const int* __restrict__ positions,
    const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp, int H, int R, int Dr, float scale,
    int window, float* __restrict__ out, float* __restrict__ ml) {
  extern __shared__ __align__(16) float sm[];
  const int E = R + Dr, ES = V4 ? E + 4 : E + 1;   // lanes read different rows: the padding spreads them over the banks
  float* ks = sm;                          // LT_KEYS * ES
  float* qs = ks + LT_KEYS * ES;           // LT_HEADS * E
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y * LT_HEADS + warp;
  const int split = blockIdx.z, splits = gridDim.z;
  const bool live = h < H;
  const int pos = positions[t];
  const int* bt = block_table + (size_t)seq_of_token[t] * maxp;
  if (live)
    for (int i = lane; i < E; i += 32) qs[warp * E + i] = qa[((size_t)t * H + h) * E + i];
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int tiles = (pos - lo) / LT_KEYS + 1;
  const int per = (tiles + splits - 1) / splits;
  const int j_begin = lo + split * per * LT_KEYS;
  const int j_end = min(pos, lo + (split + 1) * per * LT_KEYS - 1);      // last key of this block
  float m = -INFINITY, l = 0.f;
  float acc[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) acc[i] = 0.f;
  const float* qh = qs + warp * E;
  for (int j0 = j_begin; j0 <= j_end; j0 += LT_KEYS) {
    const int nk = min(LT_KEYS, j_end - j0 + 1);
    __syncthreads();                        // the tile before is read out (and qs is written)
    constexpr int VEC = 16 / (int)sizeof(T);
    if (E % VEC == 0) {
      // a warp takes whole rows: the page is looked up once a row and the lanes copy 16 bytes each
      for (int jj = warp; jj < nk; jj += LT_HEADS) {
        const int j = j0 + jj;
        const uint4* src = reinterpret_cast<const uint4*>(k_pages + ((size_t)bt[j >> 6] * SX_PAGE + (j & 63)) * E);
        float* dst = ks + jj * ES;
        for (int c = lane; c < E / VEC; c += 32) {
          const uint4 v = src[c];
          const T* x = reinterpret_cast<const T*>(&v);
          if (V4) {
#pragma unroll
            for (int i = 0; i < VEC; i += 4)
              *reinterpret_cast<float4*>(dst + c * VEC + i) = make_float4(to_f32(x[i]), to_f32(x[i + 1]), to_f32(x[i + 2]), to_f32(x[i + 3]));
          } else {
#pragma unroll
            for (int i = 0; i < VEC; ++i) dst[c * VEC + i] = to_f32(x[i]);
          }
        }
      }
    } else {
      for (int i = tid; i < nk * E; i += LT_HEADS * 32) {
        const int jj = i / E, e = i % E;
        const int j = j0 + jj;
        ks[jj * ES + e] = to_f32(k_pages[((size_t)bt[j >> 6] * SX_PAGE + (j & 63)) * E + e]);
      }
    }
    __syncthreads();
    if (!live) continue;
    float s = -INFINITY;
    if (lane < nk) {
      const float* kr = ks + lane * ES;
      float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;      // four sums side by side: the chain of one would wait on itself
      if (V4) {
#pragma unroll 4
        for (int e = 0; e < E; e += 4) {
          const float4 q4 = *reinterpret_cast<const float4*>(qh + e), k4 = *reinterpret_cast<const float4*>(kr + e);
          d0 = fmaf(q4.x, k4.x, d0); d1 = fmaf(q4.y, k4.y, d1); d2 = fmaf(q4.z, k4.z, d2); d3 = fmaf(q4.w, k4.w, d3);
        }
      } else {
        int e = 0;
        for (; e + 3 < E; e += 4) {
          d0 = fmaf(qh[e], kr[e], d0);
          d1 = fmaf(qh[e + 1], kr[e + 1], d1);
          d2 = fmaf(qh[e + 2], kr[e + 2], d2);
          d3 = fmaf(qh[e + 3], kr[e + 3], d3);
        }
        for (; e < E; ++e) d0 = fmaf(qh[e], kr[e], d0);
      }
      s = ((d0 + d1) + (d2 + d3)) * scale;
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float p = lane < nk ? expf(s - m_new) : 0.f;
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    l = l * corr + warp_sum(p);
    m = m_new;
#pragma unroll
    for (int i = 0; i < RI; ++i) acc[i] *= corr;
    for (int jj = 0; jj < nk; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const float* kr = ks + jj * ES;
      if (V4) {
#pragma unroll
        for (int i = 0; i < RI / 4; ++i) {
          const int r = lane * 4 + 128 * i;
          if (r < R) {
            const float4 c4 = *reinterpret_cast<const float4*>(kr + r);
            acc[4 * i] = fmaf(pj, c4.x, acc[4 * i]); acc[4 * i + 1] = fmaf(pj, c4.y, acc[4 * i + 1]);
            acc[4 * i + 2] = fmaf(pj, c4.z, acc[4 * i + 2]); acc[4 * i + 3] = fmaf(pj, c4.w, acc[4 * i + 3]);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const int r = lane + 32 * i;
          if (r < R) acc[i] = fmaf(pj, kr[r], acc[i]);
        }
      }
    }
  }
  if (live) {
    float* o = out + (((size_t)t * H + h) * splits + split) * R;
    if (V4) {
#pragma unroll
      for (int i = 0; i < RI / 4; ++i) {
        const int r = lane * 4 + 128 * i;
        if (r < R) *reinterpret_cast<float4*>(o + r) = make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        const int r = lane + 32 * i;
        if (r < R) o[r] = acc[i];
      }
    }
    if (lane == 0) {
      ml[(((size_t)t * H + h) * splits + split) * 2] = m;
      ml[(((size_t)t * H + h) * splits + split) * 2 + 1] = l;
    }
  }
}

template <typename T, int RI, bool V4>
static int latent_attn_launch(const float* qa, const void* k_pages, const int* positions, const int* seq_of_token,
                              const int* block_table, int maxp, int H, int R, int Dr, float scale, int window, float* out,
                              float* ml, int splits, int T_, cudaStream_t stream) {
  const size_t smem = (size_t)(LT_KEYS * (R + Dr + (V4 ? 4 : 1)) + LT_HEADS * (R + Dr)) * sizeof(float);
  if (smem > 200 * 1024) return SX_ERR_SIZE;
  if (smem > 48 * 1024) cudaFuncSetAttribute(latent_attn_kernel<T, RI, V4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  dim3 grid(T_, (H + LT_HEADS - 1) / LT_HEADS, splits);
  return sx_launch(latent_attn_kernel<T, RI, V4>, grid, dim3(LT_HEADS * 32), smem, stream, qa, (const T*)k_pages, positions,
                   seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml);
}

template <typename T>
static int latent_attn_any(const float* qa, const void* k_pages, const int* positions, const int* seq_of_token,
                           const int* block_table, int maxp, int H, int R, int Dr, float scale, int window, float* out, float* ml,
                           int splits, int T_, cudaStream_t stream) {
#define LT_CASE(RI, V4) return latent_attn_launch<T, RI, V4>(qa, k_pages, positions, seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, splits, T_, stream)
  if (R % 4 == 0 && Dr % 4 == 0 && (((uintptr_t)qa | (uintptr_t)out) & 15) == 0) {      // a lane owns groups of four elements
    if (R <= 128) LT_CASE(4, true);
    if (R <= 256) LT_CASE(8, true);
    if (R <= 384) LT_CASE(12, true);
    if (R <= 512) LT_CASE(16, true);
    if (R <= 1024) LT_CASE(32, true);
    return SX_ERR_SIZE;
  }
  if (R <= 32 * 2) LT_CASE(2, false);
  if (R <= 32 * 4) LT_CASE(4, false);
  if (R <= 32 * 8) LT_CASE(8, false);
  if (R <= 32 * 12) LT_CASE(12, false);
  if (R <= 32 * 16) LT_CASE(16, false);
  if (R <= 32 * 32) LT_CASE(32, false);
#undef LT_CASE
  return SX_ERR_SIZE;
}

// ---------------------------------------------------------------------------------------------------------------
// The attention above for bfloat16 cache rows on the tensor cores (mma.sync m16n8k16), 16 heads a block as the rows of the
// fragments.  What is 32-bit stays 32-bit: a query in the latent's space, and a weight, is split into three bfloat16 pieces that
// add up to it (24 bits), each piece times a cache element is exact, and sums are 32-bit; three instructions stand for one.
//   scores   the eight warps share the E elements of a row (KSW slices of 16 a warp, whose query pieces stay in registers for
//            all keys) and add their partial scores up in shared memory, in warp order
//   softmax  16 threads a head, two keys each; the weights' pieces go to shared memory
//   sum      the warps share the R elements of the latent (NTW tiles of eight a warp)
// Keys come 32 at a time (half a page) by cp.async, double-buffered.  A token's window is shared by `shares` blocks: the
// `cluster` blocks of a cluster merge through one another's shared memory, what is left (parts) is merged by the output kernel.
// Latency-bound in steps of few sequences.  Batch 8, 32 heads, rows of 320 + 64, windows of 1,000, inside a decode step beside
// the experts' stream: 61 us with the FFMA kernel above, 18 with this one.
// ---------------------------------------------------------------------------------------------------------------
#define LM_KEYS 32
#define LM_SP (LM_KEYS + 4)        // floats between two heads' partial scores
#define LM_PP (LM_KEYS + 8)        // elements between two heads' weights

// ANY: a value above the largest bfloat16 is cut to it and not rounded to infinity (finite float32 values all have three pieces).
// (Cutting all pieces would do, too, but smaller pieces of either sign leave less to round off: 3.7e-7 against 4.0e-7 from 64-bit
// sums with 32 heads and windows of 1,000.)
template <bool ANY>
__device__ __forceinline__ void lm_split3(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    uint32_t v = *reinterpret_cast<const uint32_t*>(&b);
    if (ANY && i == 0) {
      const uint32_t bx = __float_as_uint(x), by = __float_as_uint(y);
      if ((bx & 0x7fffffffu) > 0x7f7f0000u) v = __byte_perm(v, bx, 0x3276);
      if ((by & 0x7fffffffu) > 0x7f7f0000u) v = __byte_perm(v, by, 0x7610);
    }
    p[i] = v;
    x -= __uint_as_float(v << 16);
    y -= __uint_as_float(v & 0xffff0000u);
  }
}
__device__ __forceinline__ void lm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool TRANS>
__device__ __forceinline__ void lm_ldsm4(uint32_t (&r)[4], const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (TRANS) asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
  else asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}

__host__ __device__ inline size_t lm_smem_bytes(int E) {
  return (size_t)2 * LM_KEYS * (E + 8) * sizeof(bf16) + (size_t)8 * 16 * LM_SP * sizeof(float) + (size_t)3 * 16 * LM_PP * sizeof(bf16) +
         (size_t)16 * (1 + 2 + 8) * sizeof(float);
}

template <int KSW, int NTW>
__global__ void __launch_bounds__(256) latent_attn_mma_kernel(
    const float* __restrict__ qa, const bf16* __restrict__ k_pages, const int* __restrict__ positions,
    const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp, int H, int R, int Dr, float scale,
    int window, float* __restrict__ out, float* __restrict__ ml, int parts, int cluster) {
  extern __shared__ __align__(16) unsigned char lm_smem[];
  const int E = R + Dr, LD = E + 8;
  bf16* ks = reinterpret_cast<bf16*>(lm_smem);                       // [2][LM_KEYS][LD]; at the end the weighted latents [16][R + 4]
  float* sp = reinterpret_cast<float*>(ks + 2 * LM_KEYS * LD);       // [8][16][LM_SP]
  bf16* pp = reinterpret_cast<bf16*>(sp + 8 * 16 * LM_SP);           // [3][16][LM_PP]
  float* corr_s = reinterpret_cast<float*>(pp + 3 * 16 * LM_PP);     // [16]
  float* ml_s = corr_s + 16;                                         // [16][2]
  float* w_s = ml_s + 32;                                            // [16][8]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int t = blockIdx.z, h0 = blockIdx.y * 16;
  const int part = blockIdx.x / cluster, rank = blockIdx.x % cluster, shares = parts * cluster;
  pdl_wait();
  pdl_trigger();
  const int pos = positions[t];
  const int* bt = block_table + (size_t)seq_of_token[t] * maxp;
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  const int tile0 = lo / LM_KEYS, tiles = pos / LM_KEYS - tile0 + 1, share = part * cluster + rank;
  const int begin = tile0 + (int)((long long)tiles * share / shares), end = tile0 + (int)((long long)tiles * (share + 1) / shares);
  auto load = [&](int tile, int buf) {
    const bf16* page = k_pages + (size_t)bt[tile >> 1] * SX_PAGE * E;
#pragma unroll
    for (int i = 0; i < LM_KEYS / 8; ++i) {
      const int r = warp + 8 * i, j = tile * LM_KEYS + r;
      const bool live = j >= lo && j <= pos;                         // (other rows may hold anything: zeros stand for them)
      const bf16* src = page + (size_t)(j & 63) * E;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(ks + ((size_t)buf * LM_KEYS + r) * LD);
      for (int c = lane; c < E / 8; c += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + c * 16), "l"(src + c * 8), "r"(live ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  if (begin < end) load(begin, 0);
  // this warp's slices of the queries, in pieces
  uint32_t qf[KSW][3][4];
#pragma unroll
  for (int s = 0; s < KSW; ++s) {
    const int k = (warp * KSW + s) * 16 + t4 * 2;
#pragma unroll
    for (int i = 0; i < 4; ++i) {                                    // (rows g, g + 8) x (elements k, k + 8)
      const int h = h0 + g + (i & 1) * 8, kk = k + (i >> 1) * 8;
      float2 v = make_float2(0.f, 0.f);
      if (h < H && kk < E) v = *reinterpret_cast<const float2*>(qa + ((size_t)t * H + h) * E + kk);
      uint32_t p[3];
      lm_split3<true>(v.x, v.y, p);
      qf[s][0][i] = p[0]; qf[s][1][i] = p[1]; qf[s][2][i] = p[2];
    }
  }
  float acc[NTW][4];
#pragma unroll
  for (int i = 0; i < NTW; ++i)
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[i][x] = 0.f;
  const int row = tid >> 4, kq = tid & 15;                           // softmax: a head and two of the keys
  float m = -INFINITY, l = 0.f;
  for (int tile = begin; tile < end; ++tile) {
    const int buf = (tile - begin) & 1;
    if (tile + 1 < end) load(tile + 1, buf ^ 1);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const bf16* kt = ks + (size_t)buf * LM_KEYS * LD;
    float sacc[LM_KEYS / 8][4];
#pragma unroll
    for (int n = 0; n < LM_KEYS / 8; ++n)
#pragma unroll
      for (int x = 0; x < 4; ++x) sacc[n][x] = 0.f;
#pragma unroll
    for (int s = 0; s < KSW; ++s) {
      const int k = (warp * KSW + s) * 16;
      if (k < E) {
#pragma unroll
        for (int n = 0; n < LM_KEYS / 8; n += 2) {
          uint32_t b[4];
          lm_ldsm4<false>(b, kt + (size_t)(n * 8 + (lane >> 4) * 8 + (lane & 7)) * LD + k + ((lane >> 3) & 1) * 8);
#pragma unroll
          for (int i = 2; i >= 0; --i) {
            lm_mma(sacc[n], qf[s][i], b[0], b[1]);
            lm_mma(sacc[n + 1], qf[s][i], b[2], b[3]);
          }
        }
      }
    }
#pragma unroll
    for (int n = 0; n < LM_KEYS / 8; ++n) {
      *reinterpret_cast<float2*>(sp + (warp * 16 + g) * LM_SP + n * 8 + t4 * 2) = make_float2(sacc[n][0], sacc[n][1]);
      *reinterpret_cast<float2*>(sp + (warp * 16 + g + 8) * LM_SP + n * 8 + t4 * 2) = make_float2(sacc[n][2], sacc[n][3]);
    }
    __syncthreads();
    {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float2 v = *reinterpret_cast<const float2*>(sp + (w * 16 + row) * LM_SP + kq * 2);
        s0 += v.x; s1 += v.y;
      }
      const int j = tile * LM_KEYS + kq * 2;
      const bool ok0 = j >= lo && j <= pos, ok1 = j + 1 >= lo && j + 1 <= pos;
      // An infinite cache element times a piece that is zero is no number, and one piece's products may overflow to the other sign
      // before the largest piece's are added: a score that is not finite is formed again as one sum of whole products.
      if (!(fabsf(s0) < INFINITY && fabsf(s1) < INFINITY) && h0 + row < H) {
        const float* qr = qa + ((size_t)t * H + h0 + row) * E;
        const bf16* kr = kt + kq * 2 * LD;
        s0 = s1 = 0.f;
#pragma unroll 1
        for (int e = 0; e < E; ++e) {
          s0 = fmaf(qr[e], __bfloat162float(kr[e]), s0);
          s1 = fmaf(qr[e], __bfloat162float(kr[LD + e]), s1);
        }
      }
      s0 = ok0 ? s0 * scale : -INFINITY;
      s1 = ok1 ? s1 * scale : -INFINITY;
      float mx = fmaxf(s0, s1);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m, mx);
      // (a score of minus infinity has no weight, also where there has been no other yet)
      const float p0 = s0 == -INFINITY ? 0.f : expf(s0 - m_new), p1 = s1 == -INFINITY ? 0.f : expf(s1 - m_new);
      const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
      float sum = p0 + p1;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l = l * corr + sum;
      m = m_new;
      uint32_t p[3];
      lm_split3<false>(p0, p1, p);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(pp + (i * 16 + row) * LM_PP + kq * 2) = p[i];
      if (kq == 0) corr_s[row] = corr;
    }
    __syncthreads();
    const float c0 = corr_s[g], c1 = corr_s[g + 8];
#pragma unroll
    for (int i = 0; i < NTW; ++i) { acc[i][0] *= c0; acc[i][1] *= c0; acc[i][2] *= c1; acc[i][3] *= c1; }
#pragma unroll
    for (int kk = 0; kk < LM_KEYS / 16; ++kk) {
      uint32_t a[3][4];
#pragma unroll
      for (int i = 0; i < 3; ++i) lm_ldsm4<false>(a[i], pp + (i * 16 + (lane & 15)) * LM_PP + kk * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int n = 0; n < NTW; n += 2) {
        const int r = (warp * NTW + n) * 8;
        if (r < R) {
          uint32_t b[4];
          lm_ldsm4<true>(b, kt + (size_t)(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)) * LD + r + (lane >> 4) * 8);
#pragma unroll
          for (int i = 2; i >= 0; --i) {
            lm_mma(acc[n], a[i], b[0], b[1]);
            lm_mma(acc[n + 1], a[i], b[2], b[3]);
          }
        }
      }
    }
    __syncthreads();                                                 // the tile, the partial scores and the weights are read out
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  float* os = reinterpret_cast<float*>(lm_smem);
  const int OL = R + 4;
#pragma unroll
  for (int n = 0; n < NTW; ++n) {
    const int r = (warp * NTW + n) * 8 + t4 * 2;
    if (r < R) {
      *reinterpret_cast<float2*>(os + g * OL + r) = make_float2(acc[n][0], acc[n][1]);
      *reinterpret_cast<float2*>(os + (g + 8) * OL + r) = make_float2(acc[n][2], acc[n][3]);
    }
  }
  if (kq == 0) { ml_s[row * 2] = m; ml_s[row * 2 + 1] = l; }
  const int r4 = R / 4;
  if (cluster == 1) {
    __syncthreads();
    for (int i = tid; i < 16 * r4; i += 256) {
      const int hh = i / r4, c = i % r4;
      if (h0 + hh < H) *reinterpret_cast<float4*>(out + (((size_t)t * H + h0 + hh) * parts + part) * R + c * 4) = *reinterpret_cast<const float4*>(os + hh * OL + c * 4);
    }
    if (tid < 32 && h0 + tid / 2 < H) ml[(((size_t)t * H + h0 + tid / 2) * parts + part) * 2 + (tid & 1)] = ml_s[tid];
    return;
  }
  cluster_sync_all();
  // the heads' maxima and sums over the cluster; a block's weight is exp(its maximum - the common one)
  if (tid < 16) {
    float mb[8], lb[8], M = -INFINITY, L = 0.f;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      mb[b] = cluster_load_f32(ml_s + tid * 2, (uint32_t)min(b, cluster - 1));
      lb[b] = cluster_load_f32(ml_s + tid * 2 + 1, (uint32_t)min(b, cluster - 1));
    }
#pragma unroll
    for (int b = 0; b < 8; ++b) M = fmaxf(M, mb[b]);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const float f = b >= cluster || mb[b] == -INFINITY ? 0.f : expf(mb[b] - M);
      w_s[tid * 8 + b] = f;
      L = fmaf(f, lb[b], L);
    }
    if (rank == 0 && h0 + tid < H) {
      ml[(((size_t)t * H + h0 + tid) * parts + part) * 2] = M;
      ml[(((size_t)t * H + h0 + tid) * parts + part) * 2 + 1] = L;
    }
  }
  __syncthreads();
  const uint32_t os_a = (uint32_t)__cvta_generic_to_shared(os);
  for (int i = tid + rank * 256; i < 16 * r4; i += 256 * cluster) {
    const int hh = i / r4, c = i % r4;
    float4 v[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      uint32_t from;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(from) : "r"(os_a + (uint32_t)(hh * OL + c * 4) * 4), "r"((uint32_t)min(b, cluster - 1)));
      asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v[b].x), "=f"(v[b].y), "=f"(v[b].z), "=f"(v[b].w) : "r"(from) : "memory");
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const float f = w_s[hh * 8 + b];
      o.x = fmaf(f, v[b].x, o.x); o.y = fmaf(f, v[b].y, o.y); o.z = fmaf(f, v[b].z, o.z); o.w = fmaf(f, v[b].w, o.w);
    }
    if (h0 + hh < H) *reinterpret_cast<float4*>(out + (((size_t)t * H + h0 + hh) * parts + part) * R + c * 4) = o;
  }
  cluster_sync_all();                                                // nobody's shared memory goes away while it is read
}

// which sizes the kernel above takes
static bool latent_mma_fits(int R, int Dr, int T) {
  return R % 16 == 0 && Dr % 16 == 0 && R > 0 && R <= 512 && R + Dr <= 640 && T <= 65535;
}
extern "C" int sx_latent_mma_fits(int R, int Dr, int T) { return latent_mma_fits(R, Dr, T) ? 1 : 0; }

template <int KSW, int NTW>
static int latent_attn_mma_launch(const float* qa, const void* k_pages, const int* positions, const int* seq_of_token,
                                  const int* block_table, int maxp, int H, int R, int Dr, float scale, int window, float* out,
                                  float* ml, int parts, int cluster, int T, cudaStream_t stream) {
  const size_t smem = lm_smem_bytes(R + Dr);
  cudaError_t e = cudaFuncSetAttribute(latent_attn_mma_kernel<KSW, NTW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  dim3 grid(parts * cluster, (H + 15) / 16, T);
  if (cluster == 1)
    return sx_launch(latent_attn_mma_kernel<KSW, NTW>, grid, dim3(256), smem, stream, qa, (const bf16*)k_pages, positions, seq_of_token,
                     block_table, maxp, H, R, Dr, scale, window, out, ml, parts, 1);
  return sx_launch_cluster(latent_attn_mma_kernel<KSW, NTW>, grid, dim3(256), smem, stream, cluster, qa, (const bf16*)k_pages, positions,
                           seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, parts, cluster);
}

static int latent_attn_mma(const float* qa, const void* k_pages, const int* positions, const int* seq_of_token, const int* block_table,
                           int maxp, int H, int R, int Dr, float scale, int window, float* out, float* ml, int parts, int cluster,
                           int T, cudaStream_t stream) {
  const int ksw = ((R + Dr) / 16 + 7) / 8;                           // slices of a row a warp takes
  const int ntw = ((R / 16 + 7) / 8) * 2;                            // tiles of the latent a warp takes, in pairs
#define LM_CASE(K_, N_) if (ksw <= K_ && ntw <= N_) return latent_attn_mma_launch<K_, N_>(qa, k_pages, positions, seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, parts, cluster, T, stream)
  LM_CASE(1, 2); LM_CASE(2, 2); LM_CASE(2, 4); LM_CASE(3, 4); LM_CASE(3, 6); LM_CASE(4, 6); LM_CASE(5, 8);
#undef LM_CASE
  return SX_ERR_SIZE;
}

extern "C" int sx_latent_attention(const float* qa, const void* k_pages, const int* positions, const int* seq_of_token,
                                   const int* block_table, int maxp, int H, int R, int Dr, float scale, int window, float* out,
                                   float* ml, int splits, int cluster, int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H <= 0 || R <= 0 || Dr < 0 || (H + LT_HEADS - 1) / LT_HEADS > 65535 || splits < 1 || splits > 64) return SX_ERR_SIZE;
  // cluster: blocks that share each of the `splits` parts' keys and merge among themselves (0: the kernel for every size)
  if (cluster > 0) {
    if (dt != SX_BF16 || !latent_mma_fits(R, Dr, T) || cluster > 8 || (((uintptr_t)qa | (uintptr_t)out | (uintptr_t)k_pages) & 15)) return SX_ERR_SIZE;
    return latent_attn_mma(qa, k_pages, positions, seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, splits, cluster, T, stream);
  }
  if (dt == SX_F32) return latent_attn_any<float>(qa, k_pages, positions, seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, splits, T, stream);
  if (dt == SX_BF16) return latent_attn_any<bf16>(qa, k_pages, positions, seq_of_token, block_table, maxp, H, R, Dr, scale, window, out, ml, splits, T, stream);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------------------------------
#define LT_OUTS 4            // outputs a warp of the output kernel computes side by side

template <typename T>
__global__ void __launch_bounds__(LT_THREADS) latent_output_kernel(
    const float* __restrict__ ol, const float* __restrict__ ml, int splits, const T* __restrict__ wuv, int H, int Dv, int R,
    const T* __restrict__ proj, int row, int col_g, int g_elem, const float* __restrict__ sinks, T* __restrict__ y, int n_tokens) {
  extern __shared__ float os[];          // LT_TOKENS * R
  __shared__ float wsp[LT_TOKENS][64];   // each split's weight exp(m_s - M) / L
  pdl_wait();
  pdl_trigger();
  const int t0 = blockIdx.x * LT_TOKENS, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = min(LT_TOKENS, n_tokens - t0);
  if (tid < LT_TOKENS) {
    const int tt = tid;
    if (tt < nt) {
      const float* p = ml + ((size_t)(t0 + tt) * H + h) * splits * 2;
      float M = sinks ? sinks[h] : -INFINITY;
      for (int s = 0; s < splits; ++s) M = fmaxf(M, p[2 * s]);
      float L = sinks ? expf(sinks[h] - M) : 0.f;
      for (int s = 0; s < splits; ++s) L += p[2 * s + 1] * (p[2 * s] == -INFINITY ? 0.f : expf(p[2 * s] - M));
      for (int s = 0; s < splits; ++s) wsp[tt][s] = (p[2 * s] == -INFINITY ? 0.f : expf(p[2 * s] - M)) / L;
    }
  }
  __syncthreads();
#pragma unroll 4                 // the loads of several elements on the way together: they are all the kernel waits for
  for (int i = tid; i < LT_TOKENS * R; i += LT_THREADS) {
    const int tt = i / R, r = i % R;
    float v = 0.f;
    if (tt < nt) {
      const float* p = ol + ((size_t)(t0 + tt) * H + h) * splits * R + r;
#pragma unroll 8
      for (int s = 0; s < splits; ++s) v = fmaf(wsp[tt][s], p[(size_t)s * R], v);
    }
    os[i] = v;
  }
  __syncthreads();
  // the grid's z axis shares the head's outputs: 32 a block
  const int j_hi = min(Dv, (int)(blockIdx.z + 1) * (LT_THREADS / 32) * LT_OUTS);
  for (int j0 = blockIdx.z * (LT_THREADS / 32) * LT_OUTS + warp * LT_OUTS; j0 < j_hi; j0 += (LT_THREADS / 32) * LT_OUTS) {
    float acc[LT_OUTS][LT_TOKENS];
#pragma unroll
    for (int a = 0; a < LT_OUTS; ++a)
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) acc[a][tt] = 0.f;
#pragma unroll 4
    for (int r = lane; r < R; r += 32) {
      float w[LT_OUTS];
#pragma unroll
      for (int a = 0; a < LT_OUTS; ++a) w[a] = j0 + a < Dv ? to_f32(wuv[((size_t)h * Dv + j0 + a) * R + r]) : 0.f;
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) {
        const float x = os[tt * R + r];
#pragma unroll
        for (int a = 0; a < LT_OUTS; ++a) acc[a][tt] = fmaf(x, w[a], acc[a][tt]);
      }
    }
#pragma unroll
    for (int a = 0; a < LT_OUTS; ++a)
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) {
        const float s = warp_sum(acc[a][tt]);
        if (lane == 0 && tt < nt && j0 + a < Dv) {
          float g = 1.f;
          if (col_g >= 0) g = 1.f / (1.f + expf(-to_f32(proj[(size_t)(t0 + tt) * row + col_g + (g_elem ? h * Dv + j0 + a : h)])));
          y[(size_t)(t0 + tt) * H * Dv + h * Dv + j0 + a] = from_f32<T>(s * g);
        }
      }
  }
}

// The same for R % 4 == 0, R <= 512 and aligned rows: a lane takes four elements a load, a warp's weights are asked for before the
// wait, and the 32 sums of a warp (4 outputs x 8 tokens) fold over its lanes in 31 shuffles that leave one in each lane, where
// the kernel above takes 5 shuffles a sum and finishes them all in lane 0.  8 tokens, 32 heads of 128, latents of 320, in a decode
// step: 79 us with the kernel above (behind 9 parts), 19 with this one (behind one).
template <typename T> struct lt_quad;
template <> struct lt_quad<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <> struct lt_quad<bf16> {
  uint2 v;
  __device__ __forceinline__ void load(const bf16* p) { v = __ldg(reinterpret_cast<const uint2*>(p)); }
  __device__ __forceinline__ void zero() { v = make_uint2(0u, 0u); }
  __device__ __forceinline__ float4 get() const {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    return make_float4(a.x, a.y, b.x, b.y);
  }
};

template <typename T>
__global__ void __launch_bounds__(LT_THREADS) latent_output4_kernel(
    const float* __restrict__ ol, const float* __restrict__ ml, int splits, const T* __restrict__ wuv, int H, int Dv, int R,
    const T* __restrict__ proj, int row, int col_g, int g_elem, const float* __restrict__ sinks, T* __restrict__ y, int n_tokens) {
  constexpr int IT = 4;                  // pieces of 128 elements of the latent
  extern __shared__ __align__(16) float os[];          // LT_TOKENS * R
  __shared__ float wsp[LT_TOKENS][64];   // each part's weight exp(m_s - M) / L
  const int t0 = blockIdx.x * LT_TOKENS, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = min(LT_TOKENS, n_tokens - t0);
  const int j0 = (blockIdx.z * (LT_THREADS / 32) + warp) * LT_OUTS;
  lt_quad<T> w[IT][LT_OUTS];
#pragma unroll
  for (int i = 0; i < IT; ++i)
#pragma unroll
    for (int a = 0; a < LT_OUTS; ++a) {
      const int r = i * 128 + lane * 4;
      if (r < R && j0 + a < Dv) w[i][a].load(wuv + ((size_t)h * Dv + j0 + a) * R + r);
      else w[i][a].zero();
    }
  pdl_wait();
  pdl_trigger();
  // a warp a token: a lane a part (two from 33 parts on)
  if (warp < nt) {
    const float* p = ml + ((size_t)(t0 + warp) * H + h) * splits * 2;
    const float m0 = lane < splits ? p[2 * lane] : -INFINITY, m1 = lane + 32 < splits ? p[2 * lane + 64] : -INFINITY;
    const float M = fmaxf(sinks ? sinks[h] : -INFINITY, warp_max(fmaxf(m0, m1)));
    const float e0 = m0 == -INFINITY ? 0.f : expf(m0 - M), e1 = m1 == -INFINITY ? 0.f : expf(m1 - M);
    const float L = (sinks ? expf(sinks[h] - M) : 0.f) +
                    warp_sum((lane < splits ? p[2 * lane + 1] * e0 : 0.f) + (lane + 32 < splits ? p[2 * lane + 65] * e1 : 0.f));
    if (lane < splits) wsp[warp][lane] = e0 / L;
    if (lane + 32 < splits) wsp[warp][lane + 32] = e1 / L;
  }
  __syncthreads();
  const int r4 = R / 4;
  for (int i = tid; i < LT_TOKENS * r4; i += LT_THREADS) {
    const int tt = i / r4, c = i % r4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tt < nt) {
      const float4* p = reinterpret_cast<const float4*>(ol + ((size_t)(t0 + tt) * H + h) * splits * R) + c;
#pragma unroll 8
      for (int s = 0; s < splits; ++s) {
        const float4 x = p[(size_t)s * r4];
        const float f = wsp[tt][s];
        v.x = fmaf(f, x.x, v.x); v.y = fmaf(f, x.y, v.y); v.z = fmaf(f, x.z, v.z); v.w = fmaf(f, x.w, v.w);
      }
    }
    reinterpret_cast<float4*>(os)[i] = v;
  }
  __syncthreads();
  float acc[LT_OUTS * LT_TOKENS];
#pragma unroll
  for (int i = 0; i < LT_OUTS * LT_TOKENS; ++i) acc[i] = 0.f;
#pragma unroll
  for (int i = 0; i < IT; ++i) {
    const int r = i * 128 + lane * 4;
    if (r < R) {
      float4 wf[LT_OUTS];
#pragma unroll
      for (int a = 0; a < LT_OUTS; ++a) wf[a] = w[i][a].get();
#pragma unroll
      for (int tt = 0; tt < LT_TOKENS; ++tt) {
        const float4 x = *reinterpret_cast<const float4*>(os + tt * R + r);
#pragma unroll
        for (int a = 0; a < LT_OUTS; ++a)
          acc[a * LT_TOKENS + tt] = fmaf(x.w, wf[a].w, fmaf(x.z, wf[a].z, fmaf(x.y, wf[a].y, fmaf(x.x, wf[a].x, acc[a * LT_TOKENS + tt]))));
      }
    }
  }
  const float s = warp_fold<LT_OUTS * LT_TOKENS>(acc, lane);
  const int tt = lane % LT_TOKENS, j = j0 + lane / LT_TOKENS;
  if (tt < nt && j < Dv) {
    float g = 1.f;
    if (col_g >= 0) g = 1.f / (1.f + expf(-to_f32(proj[(size_t)(t0 + tt) * row + col_g + (g_elem ? h * Dv + j : h)])));
    y[(size_t)(t0 + tt) * H * Dv + h * Dv + j] = from_f32<T>(s * g);
  }
}

extern "C" int sx_latent_output(const float* ol, const float* ml, int splits, const void* wuv, int H, int Dv, int R,
                                const void* proj, int row, int col_g, int g_elem, const float* sinks, void* y, int T, int dt,
                                cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H <= 0 || H > 65535 || Dv <= 0 || R <= 0 || splits < 1 || splits > 64) return SX_ERR_SIZE;
  const size_t smem = (size_t)LT_TOKENS * R * sizeof(float);
  if (smem > 48 * 1024) return SX_ERR_SIZE;
  dim3 grid((T + LT_TOKENS - 1) / LT_TOKENS, H, (Dv + (LT_THREADS / 32) * LT_OUTS - 1) / ((LT_THREADS / 32) * LT_OUTS));
  if (R % 4 == 0 && R <= 512 && (((uintptr_t)ol | (uintptr_t)wuv) & 15) == 0) {
    if (dt == SX_F32)
      return sx_launch(latent_output4_kernel<float>, grid, dim3(LT_THREADS), smem, stream, ol, ml, splits, (const float*)wuv, H, Dv, R,
                       (const float*)proj, row, col_g, g_elem, sinks, (float*)y, T);
    if (dt == SX_BF16)
      return sx_launch(latent_output4_kernel<bf16>, grid, dim3(LT_THREADS), smem, stream, ol, ml, splits, (const bf16*)wuv, H, Dv, R,
                       (const bf16*)proj, row, col_g, g_elem, sinks, (bf16*)y, T);
    return SX_ERR_DTYPE;
  }
  if (dt == SX_F32)
    return sx_launch(latent_output_kernel<float>, grid, dim3(LT_THREADS), smem, stream, ol, ml, splits, (const float*)wuv, H, Dv, R,
                     (const float*)proj, row, col_g, g_elem, sinks, (float*)y, T);
  if (dt == SX_BF16)
    return sx_launch(latent_output_kernel<bf16>, grid, dim3(LT_THREADS), smem, stream, ol, ml, splits, (const bf16*)wuv, H, Dv, R,
                     (const bf16*)proj, row, col_g, g_elem, sinks, (bf16*)y, T);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------------------------------
// Whole prompts with per-head keys and values (the form that a tensor-core attention kernel over paged keys and values
// takes): the step's latents are gathered from the cache, one product makes every head's unrotated keys and values
// from them, and these kernels lay them out.
//   latent_gather_kernel   c [T, R] and k_rot [T, Dr] of the step's tokens out of their cache rows
//   latent_expand_kernel   kv [T, H * D + H * Dv] (the product's result) and k_rot -> key pages [P, H, 64, D + Dr] =
//                          [k_h | k_rot] and value pages [P, H, 64, Dv], token t of sequence s in page
//                          table[s, pos / 64] at row pos % 64
//   latent_rotate_q_kernel the rotated part of every query head rotated in place ([T, H, D + Dr])
//   head_gate_kernel       y[t, h, :] *= sigmoid(proj[t, col + h])
// ---------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void latent_gather_kernel(const T* __restrict__ k_pages, const int* __restrict__ positions,
                                     const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp,
                                     int R, int Dr, T* __restrict__ c, T* __restrict__ kr) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, pos = positions[t];
  const int page = block_table[(size_t)seq_of_token[t] * maxp + (pos >> 6)];
  const T* row = k_pages + ((size_t)page * SX_PAGE + (pos & 63)) * (R + Dr);
  for (int i = threadIdx.x; i < R; i += blockDim.x) c[(size_t)t * R + i] = row[i];
  for (int i = threadIdx.x; i < Dr; i += blockDim.x) kr[(size_t)t * Dr + i] = row[R + i];
}

template <typename T>
__global__ void latent_expand_kernel(const T* __restrict__ kv, const T* __restrict__ kr, const int* __restrict__ positions,
                                     const int* __restrict__ seq_of_token, const int* __restrict__ table, int maxp, int H, int D,
                                     int Dr, int Dv, T* __restrict__ kp, T* __restrict__ vp) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, pos = positions[t];
  const int page = table[(size_t)seq_of_token[t] * maxp + (pos >> 6)];
  const int E = D + Dr, row = pos & 63;
  const T* src = kv + (size_t)t * (H * D + H * Dv);
  constexpr int VEC = 16 / (int)sizeof(T);
  if (D % VEC == 0 && Dr % VEC == 0 && Dv % VEC == 0 && (((uintptr_t)kv | (uintptr_t)kr | (uintptr_t)kp | (uintptr_t)vp) & 15) == 0) {
    const int e4 = E / VEC, d4 = D / VEC, v4 = Dv / VEC;               // 16-byte pieces
    for (int i = threadIdx.x; i < H * e4; i += blockDim.x) {
      const int h = i / e4, e = i % e4;
      const uint4 v = e < d4 ? reinterpret_cast<const uint4*>(src + h * D)[e]
                             : reinterpret_cast<const uint4*>(kr + (size_t)t * Dr)[e - d4];
      reinterpret_cast<uint4*>(kp + (((size_t)page * H + h) * SX_PAGE + row) * E)[e] = v;
    }
    for (int i = threadIdx.x; i < H * v4; i += blockDim.x) {
      const int h = i / v4, e = i % v4;
      reinterpret_cast<uint4*>(vp + (((size_t)page * H + h) * SX_PAGE + row) * Dv)[e] = reinterpret_cast<const uint4*>(src + H * D + h * Dv)[e];
    }
    return;
  }
  for (int i = threadIdx.x; i < H * E; i += blockDim.x) {
    const int h = i / E, e = i % E;
    kp[(((size_t)page * H + h) * SX_PAGE + row) * E + e] = e < D ? src[h * D + e] : kr[(size_t)t * Dr + (e - D)];
  }
  for (int i = threadIdx.x; i < H * Dv; i += blockDim.x) {
    const int h = i / Dv, e = i % Dv;
    vp[(((size_t)page * H + h) * SX_PAGE + row) * Dv + e] = src[H * D + i];
  }
}

template <typename T>
__global__ void latent_rotate_q_kernel(const T* q, int q_ld, T* out, const int* __restrict__ positions,
                                       const float* __restrict__ inv_freq, int dims, int pairs, float mag, int H, int D, int Dr) {
  // out [T, H (D + Dr)] takes the queries with their rotated parts rotated; `q` (rows q_ld apart) may be `out` itself:
  // a thread reads both elements of a pair before it writes them, and copies touch one element each
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  const float pos = (float)positions[t];
  const int half = dims / 2, HD = D + Dr;
  const T* qi = q + (size_t)t * q_ld;
  T* qo = out + (size_t)t * H * HD;
  if (qi != qo)
    for (int i = threadIdx.x; i < H * HD; i += blockDim.x) {
      const int d = i % HD;
      if (d < D || d >= D + dims) qo[i] = qi[i];
    }
  for (int i = threadIdx.x; i < H * half; i += blockDim.x) {
    const int h = i / half, p = i % half;
    int ia, ib;
    rot_pair_index(p, dims, pairs, ia, ib);
    const T* qr = qi + h * HD + D;
    float sn, cs;
    sincosf(pos * inv_freq[p], &sn, &cs);
    sn *= mag;
    cs *= mag;
    const float u = to_f32(qr[ia]), v = to_f32(qr[ib]);
    qo[h * HD + D + ia] = from_f32<T>(u * cs - v * sn);
    qo[h * HD + D + ib] = from_f32<T>(v * cs + u * sn);
  }
}

template <typename T>
__global__ void head_gate_kernel(T* __restrict__ y, const T* __restrict__ proj, int row, int col, int H, int Dv) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  constexpr int VEC = 16 / (int)sizeof(T);
  if (Dv % VEC == 0 && ((uintptr_t)y & 15) == 0) {
    const int v4 = Dv / VEC;
    for (int i = threadIdx.x; i < H * v4; i += blockDim.x) {
      const float g = 1.f / (1.f + expf(-to_f32(proj[(size_t)t * row + col + i / v4])));
      uint4* p = reinterpret_cast<uint4*>(y + (size_t)t * H * Dv) + i;
      uint4 v = *p;
      T* x = reinterpret_cast<T*>(&v);
#pragma unroll
      for (int k = 0; k < VEC; ++k) x[k] = from_f32<T>(to_f32(x[k]) * g);
      *p = v;
    }
    return;
  }
  for (int i = threadIdx.x; i < H * Dv; i += blockDim.x) {
    const float g = 1.f / (1.f + expf(-to_f32(proj[(size_t)t * row + col + i / Dv])));
    y[(size_t)t * H * Dv + i] = from_f32<T>(to_f32(y[(size_t)t * H * Dv + i]) * g);
  }
}

extern "C" int sx_latent_gather(const void* k_pages, const int* positions, const int* seq_of_token, const int* block_table,
                                int maxp, int R, int Dr, void* c, void* kr, int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (dt == SX_F32) return sx_launch(latent_gather_kernel<float>, dim3(T), dim3(256), 0, stream, (const float*)k_pages, positions, seq_of_token, block_table, maxp, R, Dr, (float*)c, (float*)kr);
  if (dt == SX_BF16) return sx_launch(latent_gather_kernel<bf16>, dim3(T), dim3(256), 0, stream, (const bf16*)k_pages, positions, seq_of_token, block_table, maxp, R, Dr, (bf16*)c, (bf16*)kr);
  return SX_ERR_DTYPE;
}

extern "C" int sx_latent_expand(const void* kv, const void* kr, const int* positions, const int* seq_of_token, const int* table,
                                int maxp, int H, int D, int Dr, int Dv, void* kp, void* vp, int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (dt == SX_F32) return sx_launch(latent_expand_kernel<float>, dim3(T), dim3(256), 0, stream, (const float*)kv, (const float*)kr, positions, seq_of_token, table, maxp, H, D, Dr, Dv, (float*)kp, (float*)vp);
  if (dt == SX_BF16) return sx_launch(latent_expand_kernel<bf16>, dim3(T), dim3(256), 0, stream, (const bf16*)kv, (const bf16*)kr, positions, seq_of_token, table, maxp, H, D, Dr, Dv, (bf16*)kp, (bf16*)vp);
  return SX_ERR_DTYPE;
}

extern "C" int sx_latent_rotate_q(const void* q, int q_ld, void* out, const int* positions, const float* inv_freq, int dims, int pairs,
                                  float mag, int H, int D, int Dr, int T, int dt, cudaStream_t stream) {
  if (T <= 0 || (dims <= 0 && q == out)) return 0;
  if (dims > Dr || (dims & 1) || dims < 0 || q_ld < H * (D + Dr)) return SX_ERR_SIZE;
  if (dt == SX_F32) return sx_launch(latent_rotate_q_kernel<float>, dim3(T), dim3(256), 0, stream, (const float*)q, q_ld, (float*)out, positions, inv_freq, dims, pairs, mag, H, D, Dr);
  if (dt == SX_BF16) return sx_launch(latent_rotate_q_kernel<bf16>, dim3(T), dim3(256), 0, stream, (const bf16*)q, q_ld, (bf16*)out, positions, inv_freq, dims, pairs, mag, H, D, Dr);
  return SX_ERR_DTYPE;
}

extern "C" int sx_head_gate(void* y, const void* proj, int row, int col, int H, int Dv, int T, int dt, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (dt == SX_F32) return sx_launch(head_gate_kernel<float>, dim3(T), dim3(256), 0, stream, (float*)y, (const float*)proj, row, col, H, Dv);
  if (dt == SX_BF16) return sx_launch(head_gate_kernel<bf16>, dim3(T), dim3(256), 0, stream, (bf16*)y, (const bf16*)proj, row, col, H, Dv);
  return SX_ERR_DTYPE;
}
