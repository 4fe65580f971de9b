// Plain kernels for every operation of a decoder step, for float32 and bfloat16 storage,
// all numbers and sums in 32-bit (no TF32; float32 products of more than 16 rows and attention of prompt portions run on the tensor
// cores, with operands in pieces that keep all 24 bits; everything else is FFMA).  They take every size;
// they are the whole of the float32 path, and the fallback of the bfloat16 path for sizes
// that the fast kernels refuse.
//
// What they compute follows the reference's formulas:
//   embedding   crates/synaptix-kernels-cuda/src/cu/embed/embed.cu:18-46
//   RMSNorm     crates/synaptix-kernels-cuda/src/cu/reduction/rms_norm.cu:26-98 (plain gain w)
//   residual    crates/synaptix-kernels-cuda/src/cu/fused/norm/rmsnorm_residual.cu:97-159
//   rotary      crates/synaptix-kernels-cuda/src/cu/elementwise/rope.cu:27-118 (rotate-half)
//   KV append   crates/synaptix-kernels-cuda/src/cu/elementwise/kv_append.cu:53-78
//   attention   crates/synaptix-kernels-cuda/src/cu/fused/attention/flash_decode.cu:92-205
//   SiLU*mul    crates/synaptix-kernels-cuda/src/cu/fused/mlp/silu_and_mul.cu:11-52
//   f32 GEMM    crates/synaptix-kernels-cuda/src/best_cu/gemm/gemm_f32.cu:1-69
// but not how: the residual stream is kept in 32-bit, the cache is paged, tokens of
// sequences with unequal lengths are packed into one stream.
#include "common.cuh"

// ---------------------------------------------------------------------------------------
// embedding gather: out[t, :] = float(table[ids[t], :]) * scale [+ float(pos_table[positions[t], :])]; an id outside its
// table gives zeros for that part, a position beyond the last row reads the last row (the engine refuses such steps)
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void embed_gather_kernel(const T* __restrict__ table, const int* __restrict__ ids,
                                    float* __restrict__ out, int H, int V, float scale, const T* __restrict__ pos_table,
                                    const int* __restrict__ positions, int P) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  const int id = ids[t];
  const bool ok = id >= 0 && id < V;
  const T* row = table + (size_t)(ok ? id : 0) * H;
  float* o = out + (size_t)t * H;
  if (pos_table) {
    const T* pr = pos_table + (size_t)min(max(positions[t], 0), P - 1) * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) o[i] = fmaf(ok ? to_f32(row[i]) : 0.f, scale, to_f32(pr[i]));
    return;
  }
  for (int i = threadIdx.x; i < H; i += blockDim.x) o[i] = ok ? to_f32(row[i]) * scale : 0.f;
}

// pos_table null: no positions
extern "C" int sx_embed_gather(const void* table, int dt, const int* ids, float* out, int n_tokens, int H, int V, float scale,
                               const void* pos_table, const int* positions, int P, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (pos_table != nullptr && (positions == nullptr || P <= 0)) return SX_ERR_SIZE;
  if (dt == SX_F32)
    return sx_launch(embed_gather_kernel<float>, dim3(n_tokens), dim3(256), 0, stream, (const float*)table, ids, out, H, V, scale,
                     (const float*)pos_table, positions, P);
  if (dt == SX_BF16)
    return sx_launch(embed_gather_kernel<bf16>, dim3(n_tokens), dim3(256), 0, stream, (const bf16*)table, ids, out, H, V, scale,
                     (const bf16*)pos_table, positions, P);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------
// residual add + RMSNorm.
//   v = h[t] (+ delta[t]);  if write_h: h[t] = v;  y[r] = v * rsqrt(mean(v^2) + eps) * w
// Rows: r = 0..R-1, t = rows ? rows[r] : r.  h and the sum of squares are 32-bit.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void add_rmsnorm_kernel(float* __restrict__ h, const T* __restrict__ delta,
                                   const float* __restrict__ w, float eps, T* __restrict__ y,
                                   const int* __restrict__ rows, int H, int write_h) {
  __shared__ float red[33];
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x;
  const int t = rows ? rows[r] : r;
  float* hr = h + (size_t)t * H;
  const T* dr = delta ? delta + (size_t)t * H : nullptr;
  T* yr = y + (size_t)r * H;
  float ss = 0.f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float v = hr[i];
    if (dr) {
      v += to_f32(dr[i]);
      if (write_h) hr[i] = v;
    }
    ss += v * v;
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)H + eps);
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float v = hr[i];
    if (dr && !write_h) v += to_f32(dr[i]);
    yr[i] = from_f32<T>(v * inv * w[i]);
  }
}

// the same with the whole row held in registers (one pass over memory, one reduction):
// rows of up to 256 * 4 * VEC4 elements, H a multiple of 4, 16-byte aligned rows
template <typename T, int VEC4>
__global__ void __launch_bounds__(256) add_rmsnorm_reg_kernel(float* __restrict__ h, const T* __restrict__ delta,
                                                              const float* __restrict__ w, float eps, T* __restrict__ y,
                                                              const int* __restrict__ rows, int H, int write_h) {
  __shared__ float red[33];
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x;
  const int t = rows ? rows[r] : r;
  float4* hr = reinterpret_cast<float4*>(h + (size_t)t * H);
  const T* dr = delta ? delta + (size_t)t * H : nullptr;
  const int n4 = H >> 2;
  float4 v[VEC4];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VEC4; ++k) {
    const int i = threadIdx.x + k * 256;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n4) {
      v[k] = hr[i];
      if (dr) {
        v[k].x += to_f32(dr[4 * i]); v[k].y += to_f32(dr[4 * i + 1]);
        v[k].z += to_f32(dr[4 * i + 2]); v[k].w += to_f32(dr[4 * i + 3]);
        if (write_h) hr[i] = v[k];
      }
      ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    }
  }
  ss = block_sum(ss, red);
  const float inv = rsqrtf(ss / (float)H + eps);
  T* yr = y + (size_t)r * H;
#pragma unroll
  for (int k = 0; k < VEC4; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < n4) {
      const float4 g = reinterpret_cast<const float4*>(w)[i];
      yr[4 * i] = from_f32<T>(v[k].x * inv * g.x);
      yr[4 * i + 1] = from_f32<T>(v[k].y * inv * g.y);
      yr[4 * i + 2] = from_f32<T>(v[k].z * inv * g.z);
      yr[4 * i + 3] = from_f32<T>(v[k].w * inv * g.w);
    }
  }
}

template <typename T>
static int add_rmsnorm_launch(float* h, const void* delta, const float* w, float eps, void* y, const int* rows, int R,
                              int H, int write_h, cudaStream_t stream) {
  const bool aligned = (H % 4 == 0) && (((uintptr_t)h | (uintptr_t)w) % 16 == 0);
  if (aligned && H <= 256 * 4 * 4)
    return sx_launch(add_rmsnorm_reg_kernel<T, 4>, dim3(R), dim3(256), 0, stream, h, (const T*)delta, w, eps, (T*)y, rows, H, write_h);
  if (aligned && H <= 256 * 4 * 8)
    return sx_launch(add_rmsnorm_reg_kernel<T, 8>, dim3(R), dim3(256), 0, stream, h, (const T*)delta, w, eps, (T*)y, rows, H, write_h);
  return sx_launch(add_rmsnorm_kernel<T>, dim3(R), dim3(256), 0, stream, h, (const T*)delta, w, eps, (T*)y, rows, H, write_h);
}

extern "C" int sx_add_rmsnorm(float* h, const void* delta, const float* w, float eps, void* y,
                              const int* rows, int R, int H, int dt, int write_h,
                              cudaStream_t stream) {
  if (R <= 0) return 0;
  if (dt == SX_F32) return add_rmsnorm_launch<float>(h, delta, w, eps, y, rows, R, H, write_h, stream);
  if (dt == SX_BF16) return add_rmsnorm_launch<bf16>(h, delta, w, eps, y, rows, R, H, write_h, stream);
  return SX_ERR_DTYPE;
}

// h[t] += delta[t] (32-bit residual sum), for the places where no norm follows
template <typename T>
__global__ void residual_add_kernel(float* __restrict__ h, const T* __restrict__ delta, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) h[i] += to_f32(delta[i]);
}
extern "C" int sx_residual_add(float* h, const void* delta, long long n, int dt, cudaStream_t stream) {
  if (n <= 0) return 0;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (dt == SX_F32) residual_add_kernel<float><<<grid, 256, 0, stream>>>(h, (const float*)delta, (size_t)n);
  else if (dt == SX_BF16) residual_add_kernel<bf16><<<grid, 256, 0, stream>>>(h, (const bf16*)delta, (size_t)n);
  else return SX_ERR_DTYPE;
  return sx_launch_status();
}

// ---------------------------------------------------------------------------------------
// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]), then soft_limit(., cap), 32-bit accumulation in k order.  Two kernels:
//   gemm_tile: 64x64x16 tiles, 4x4 outputs per thread (any M);
//   gemm_rows: one warp per output column, up to 8 rows of A at a time (M <= 16).
// ---------------------------------------------------------------------------------------
template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256) gemm_tile_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                        TC* __restrict__ C, int M, int N, int K,
                                                        const float* __restrict__ bias, float cap) {
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int r = idx >> 4, c = idx & 15;
      const int k = k0 + c;
      const int m = m0 + r, n = n0 + r;
      As[c][r] = (m < M && k < K) ? to_f32(A[(size_t)m * K + k]) : 0.f;
      Ws[c][r] = (n < N && k < K) ? to_f32(W[(size_t)n * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * N + n] = from_f32<TC>(soft_limit(bias ? acc[i][j] + bias[n] : acc[i][j], cap));
    }
  }
}

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(128) gemm_rows_kernel(const TA* __restrict__ A, const TW* __restrict__ W,
                                                        TC* __restrict__ C, int M, int N, int K,
                                                        const float* __restrict__ bias, float cap) {
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (n >= N) return;
  const TW* wr = W + (size_t)n * K;
  for (int m0 = 0; m0 < M; m0 += 8) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
    for (int k = lane; k < K; k += 32) {
      const float w = to_f32(wr[k]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (m0 + i < M) acc[i] = fmaf(to_f32(A[(size_t)(m0 + i) * K + k]), w, acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = warp_sum(acc[i]);
      if (lane == 0 && m0 + i < M) C[(size_t)(m0 + i) * N + n] = from_f32<TC>(soft_limit(bias ? s + bias[n] : s, cap));
    }
  }
}

// ---------------------------------------------------------------------------------------
// The float32 product, rows of whole 16-byte pieces (K % 4 == 0, aligned operands): every sum in 32-bit, in an order fixed by the
// sizes; FFMA up to 16 rows, the tensor cores on pieces beyond.
//
// Up to 16 rows: gemm_rows_f32_kernel streams W once.  A warp owns four rows of W and every KS-th 128-wide slice of K (the KS
// warps of a group cover a row, so a narrow matrix still puts some 16 warps on every SM and a row's bytes are all on their way
// at once); A comes through L1; the 4 x MR sums of a warp fold over its lanes in V - 1 shuffles (each step halves the values a
// lane keeps) and over the warps in order.  Bound by HBM: N x K x 4 bytes.  Two rows, weights from HBM: 4,096 x 1,024 4.6 us (3.6
// TB/s), 1,024 x 3,072 4.3 us, 151,936 x 1,024 98 us (6.3 TB/s); a warp per row of W with 4-byte loads, one in flight, took 45 us
// over a step's products on average where this takes 8.
//
// What stands around a product of a few rows is done by the product (kernels of 3 to 4 us each, that did nothing but wait and copy;
// two rows, 28 layers of a 0.6B model and its head 1.24 -> 1.13 ms a step): with NORM, A is the residual stream and the rows' RMS
// norm is formed as they are read (the sum of squares beside the products, gain on the way, the factor on the results, but for a
// power of two of it that keeps small rows above the least number);
// F32_ROWS_SILU reads a stacked [gate; up] and stores silu(gate) * up; F32_ROWS_ADD adds into C, the residual stream.
// Each is a kernel of its own: told apart at run time they cost the plain product of 9 to 16 rows 10 % (4,096 x 1,024 11.0 -> 12.5 us,
// 151,936 x 1,024 319 -> 357).  G rows of A are asked for together: four where K is short and the rows' latency counts (12 rows, 1,024 x
// 252 6.6 -> 4.1 us), one where W streams (151,936 x 1,024 with 9 to 16 rows 318 us, 341 with four) and with a norm.
enum { F32_ROWS_STORE = 0, F32_ROWS_SILU = 1, F32_ROWS_ADD = 2 };
struct F32RowsEnd {
  const float* bias;     // [N] or null
  float cap;             // F32_ROWS_STORE: soft_limit of the results
  int epi;
  const float* gain;     // [K] (NORM)
  float eps;
  float up;              // a power of two at most as large as the rows' largest factor: see the kernel
};
// (1 / sqrt(eps) is what rows of next to nothing are multiplied by; without it ahead of the sums they would fall below the least number)
static float f32_rows_up(float eps) {
  float up = 1.f;
  while (up < 0x1p20f && 4.f * up * up * eps <= 1.f) up *= 2.f;
  return up;
}
template <int MR, int KS, bool NORM, int EPI>
__global__ void __launch_bounds__(256, MR <= 2 ? 4 : (MR == 4 ? 3 : 2)) gemm_rows_f32_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                            float* __restrict__ C, int M, int N, int K, const F32RowsEnd end) {
  constexpr bool SILU = EPI == F32_ROWS_SILU;
  constexpr int R = 4, G = KS == 8 || MR < 4 || NORM ? 1 : 4, GROUPS = 8 / KS, V = MR * R, FV = V < 32 ? V : 32;
  __shared__ float part[8][V];
  __shared__ float squares[8][MR];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp / KS, ks = warp % KS;
  const int n_out = SILU ? N / 2 : N, cols = SILU ? R / 2 : R;           // outputs in all, and of a warp's four rows
  const int n0 = (blockIdx.x * GROUPS + group) * cols;
  const float* wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = SILU ? min(n0 + (r & 1), n_out - 1) + (r >> 1) * n_out : min(n0 + r, N - 1);      // (two gate rows, two up rows)
    wr[r] = W + (size_t)row * K;
  }
  float acc[MR][R], sq[MR];
#pragma unroll
  for (int i = 0; i < MR; ++i) {
    sq[i] = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) acc[i][r] = 0.f;
  }
  // the first slice of W is on its way into L2 before the kernel ahead has ended (a hint: whatever it brings is read below;
  // two prompts and eight steps of a 0.6B model in 32 bits: 21.75 -> 21.5 ms, with the activation launched early as well)
  if ((lane & 7) == 0 && (ks * 32 + lane) * 4 < K) {
#pragma unroll
    for (int r = 0; r < R; ++r) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(wr[r] + (ks * 32 + lane) * 4));
  }
  pdl_wait();
  pdl_trigger();
#pragma unroll (MR <= 2 ? 2 : 1)
  for (int k = (ks * 32 + lane) * 4; k < K; k += KS * 128) {
    float4 w[R], gn;
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = __ldg(reinterpret_cast<const float4*>(wr[r] + k));
    if (NORM) {
      gn = __ldg(reinterpret_cast<const float4*>(end.gain + k));
      gn.x *= end.up; gn.y *= end.up; gn.z *= end.up; gn.w *= end.up;
    }
#pragma unroll
    for (int i0 = 0; i0 < MR; i0 += G) {
      float4 a[G];
#pragma unroll
      for (int i = 0; i < G; ++i) a[i] = *reinterpret_cast<const float4*>(A + (size_t)min(i0 + i, M - 1) * K + k);
#pragma unroll
      for (int i = 0; i < G; ++i) {
        if (NORM) {
          sq[i0 + i] = fmaf(a[i].w, a[i].w, fmaf(a[i].z, a[i].z, fmaf(a[i].y, a[i].y, fmaf(a[i].x, a[i].x, sq[i0 + i]))));
          a[i].x *= gn.x; a[i].y *= gn.y; a[i].z *= gn.z; a[i].w *= gn.w;
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
          acc[i0 + i][r] = fmaf(a[i].w, w[r].w, fmaf(a[i].z, w[r].z, fmaf(a[i].y, w[r].y, fmaf(a[i].x, w[r].x, acc[i0 + i][r]))));
      }
    }
  }
#pragma unroll
  for (int b = 0; b < V / FV; ++b) {
    float v[FV];
#pragma unroll
    for (int i = 0; i < FV; ++i) v[i] = acc[(b * FV + i) / R][i % R];
    const float s = warp_fold<FV>(v, lane);
    constexpr int REP = 32 / FV;               // lanes that hold the same sum
    if (lane % REP == 0) part[warp][b * FV + lane / REP] = s;
  }
  if (NORM) {
    const float s = warp_fold<MR>(sq, lane);
    constexpr int REP = 32 / MR;
    if (lane % REP == 0) squares[warp][lane / REP] = s;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < GROUPS * V; i += 256) {
    const int g = i / V, m = (i % V) / R, r = i % R, n = (blockIdx.x * GROUPS + g) * cols + r;
    if (m >= M || n >= n_out || r >= cols) continue;
    float s = 0.f, u = 0.f, f = 1.f;
#pragma unroll
    for (int w = 0; w < KS; ++w) s += part[g * KS + w][i % V];
    if (SILU)
#pragma unroll
      for (int w = 0; w < KS; ++w) u += part[g * KS + w][i % V + 2];
    if (NORM) {
      float q = 0.f;
#pragma unroll
      for (int w = 0; w < KS; ++w) q += squares[g * KS + w][m];
      f = rsqrtf(q / (float)K + end.eps) / end.up;
      if (f == 0.f) {                             // squares beyond the largest number: the rows are their elements times nothing
        bool finite = true;
        for (int k = 0; k < K; ++k) finite &= isfinite(A[(size_t)m * K + k]);
        s = u = finite ? 0.f : NAN;
        f = 1.f;
      }
    }
    float* c = C + (size_t)m * n_out + n;
    s = s * f + (end.bias ? end.bias[n] : 0.f);
    if (SILU) {
      u = u * f + (end.bias ? end.bias[n_out + n] : 0.f);
      *c = s / (1.f + expf(-s)) * u;
    } else if (EPI == F32_ROWS_ADD) {
      *c += s;
    } else {
      *c = soft_limit(s, end.cap);
    }
  }
}

// More rows: gemm_tile_f32_kernel, tiles of BM x 128 by four warps, slices of 16 of K through a ring of four stages (cp.async).
// Bound by the FP32 pipe a product of 32-bit numbers ran at 35 TFLOP/s of 74; here it runs on the tensor cores with all 24 bits: an
// operand is cut into three bfloat16 pieces (8 bits each, rounded, what is left goes to the next), and of the nine products of pieces
// the six that reach 2^-24 of the whole are taken, the smallest first.  The six of a slice are summed on their own from zero and
// the slice's sum is added in 32 bits, rounded to nearest, so nothing depends on how the tensor cores round a long sum: one such
// addition for 16 products, where a chain of multiply-adds had eight.  263 rows of 4,096 x 1,024 98 -> 49 us, 1,024 of 6,144 x 1,024
// 353 -> 258 (50 TFLOP/s, 300 in bfloat16 instructions, which is what bounds it), 2,048 of 2,560 x 9,728 2.73 -> 2.00 ms; error
// against 64 bits (2-norm, N(0, 1) operands) 4.1e-7 -> 1.5e-7 at K = 1,024, 1.3e-6 -> 4.5e-7 at 9,728.
// The pieces are those of 2^16 times a number, so that none of its bits lies below the least bfloat16, and sums are
// taken back by 2^-32 at the end.  Where one is not finite (a piece of an infinity is no number; operands from 2^112 on and sums from
// 2^96 on are too large) its block forms the tile again in multiply-adds of whole numbers and takes those of it
// (2,048 of 2,560 x 9,728 2.00 ms, with a row of NaN 2.01, all of them NaN 4.8).
// A thread's four values of a row are neighbours (16 bytes; their order within the instruction's 16 does not matter), so rows need no
// padding: eight lanes read two rows of 64 bytes.  Where tiles are few, K is shared by the blocks of a cluster (grid x =
// column tile * cluster), which lay their partial tiles into shared memory and add them up in block order, each a share of the rows.
#define F32_BK 16
#define F32_STAGES 4
__device__ __forceinline__ void f32_cp16(uint32_t dst, const void* src, bool live) {
  const int bytes = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// the first of a sum: from zero
__device__ __forceinline__ void f32_mma0(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void f32_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// What is cut into pieces is 2^16 times a number: every 32-bit number is a multiple of 2^-149, so 2^16 of it one of 2^-133, the least
// bfloat16, and its three pieces are all of it whatever its size.  (From 2^112 on the first piece is infinite, and so no sum with it
// is finite.)
#define F32_UP 0x1p16f
#define F32_DOWN 0x1p-32f             // a product of two such
// (Two numbers an instruction.  Against pieces of the numbers themselves, which lose bits below 2^-109: products 0 to 2 %, 300 rows of
// 4,096 x 1,024 75.0 -> 75.6 us; attention of 2,048 tokens, 16 heads of 128, 530 -> 549, of 64 322 -> 316.  One at a time 2 to 3.5 and 5.5 %.)
__device__ __forceinline__ float4 f32_up(float4 v) {
  asm("{\n .reg .b64 a, b, u;\n mov.b64 u, {%4, %4};\n mov.b64 a, {%0, %1};\n mov.b64 b, {%2, %3};\n mul.rn.f32x2 a, a, u;\n mul.rn.f32x2 b, b, u;\n"
      " mov.b64 {%0, %1}, a;\n mov.b64 {%2, %3}, b;\n}\n" : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "f"(F32_UP));
  return v;
}
// two numbers in three pieces each: p[i] holds piece i of x (low half) and of y
__device__ __forceinline__ void f32_split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  uint32_t p[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    p[i] = *reinterpret_cast<const uint32_t*>(&b);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
  p0 = p[0]; p1 = p[1]; p2 = p[2];
}
// slices of 16 of N products, in two sums: of the leading pieces (their products have 16 bits, so little is rounded), and of the
// other five products of pieces, 2^-8 of the whole
template <int N>
__device__ __forceinline__ void f32_products(float (&c)[N][4], float (&d)[N][4], const uint32_t (&a)[3][4], const uint32_t (&b)[N][3][2]) {
  constexpr int PA[5] = {2, 0, 1, 1, 0}, PB[5] = {0, 2, 1, 0, 1};
#pragma unroll
  for (int n = 0; n < N; ++n) f32_mma0(c[n], a[0], b[n][0]);
#pragma unroll
  for (int p = 0; p < 5; ++p)
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (p == 0) f32_mma0(d[n], a[PA[p]], b[n][PB[p]]);
      else f32_mma(d[n], a[PA[p]], b[n][PB[p]]);
    }
}
template <int BM>
__global__ void __launch_bounds__(128, BM == 32 ? 4 : 3) gemm_tile_f32_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                            float* __restrict__ C, int M, int N, int K,
                                                            const float* __restrict__ bias, float cap, int cluster) {
  constexpr int BN = 128, ROWS = BM + BN, STAGE = ROWS * F32_BK, WM = BM / 32, WN = 4 / WM, NT = BN / WN / 8;   // a warp: 32 rows x NT tiles of 8 columns
  extern __shared__ __align__(16) float f32_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int wm = (warp % WM) * 32, wn = (warp / WM) * NT * 8;
  const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / cluster) * BN, z = blockIdx.x % cluster;
  const int nkb_all = (K + F32_BK - 1) / F32_BK, kper = (nkb_all + cluster - 1) / cluster;
  const int kb0 = z * kper, nkb = max(0, min(nkb_all, kb0 + kper) - kb0);
  // a thread brings the 16 bytes `lc` of every 32nd row from `lr` on
  const int lr = tid >> 2, lc = tid & 3;
  const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(f32_smem) + (uint32_t)(lr * F32_BK + lc * 4) * 4;
  const float *a0 = A + (size_t)(m0 + lr) * K + kb0 * F32_BK + lc * 4, *w0 = W + (size_t)(n0 + lr) * K + kb0 * F32_BK + lc * 4;
  const size_t rows32 = (size_t)32 * K;
  auto load = [&](int kb, int s) {
    const bool in = (kb0 + kb) * F32_BK + lc * 4 < K;
    const uint32_t dst = dst0 + (uint32_t)s * (STAGE * 4);
#pragma unroll
    for (int i = 0; i < BM / 32; ++i) {
      const bool live = in && m0 + lr + i * 32 < M;
      f32_cp16(dst + i * 32 * F32_BK * 4, live ? a0 + i * rows32 + kb * F32_BK : A, live);
    }
#pragma unroll
    for (int i = 0; i < BN / 32; ++i) {
      const bool live = in && n0 + lr + i * 32 < N;
      f32_cp16(dst + (BM + i * 32) * F32_BK * 4, live ? w0 + i * rows32 + kb * F32_BK : W, live);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  pdl_wait();
  pdl_trigger();
#pragma unroll
  for (int s = 0; s < F32_STAGES - 1; ++s) {
    if (s < nkb) load(s, s);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int kb = 0; kb < nkb; ++kb) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(F32_STAGES - 2) : "memory");
    __syncthreads();
    if (kb + F32_STAGES - 1 < nkb) load(kb + F32_STAGES - 1, (kb + F32_STAGES - 1) % F32_STAGES);
    else asm volatile("cp.async.commit_group;\n" ::: "memory");
    const float* as = f32_smem + (kb % F32_STAGES) * STAGE + (wm + g) * F32_BK + t * 4;
    const float* ws = f32_smem + (kb % F32_STAGES) * STAGE + (BM + wn + g) * F32_BK + t * 4;
    uint32_t a[2][3][4];                          // [tile of 16 rows][piece][register]
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {               // rows g and g + 8
        const float4 v = f32_up(*reinterpret_cast<const float4*>(as + (i * 16 + h * 8) * F32_BK));
        f32_split3(v.x, v.y, a[i][0][h], a[i][1][h], a[i][2][h]);
        f32_split3(v.z, v.w, a[i][0][h + 2], a[i][1][h + 2], a[i][2][h + 2]);
      }
#pragma unroll
    for (int j0 = 0; j0 < NT; j0 += 4) {
      uint32_t b[4][3][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 v = f32_up(*reinterpret_cast<const float4*>(ws + (j0 + j) * 8 * F32_BK));
        f32_split3(v.x, v.y, b[j][0][0], b[j][1][0], b[j][2][0]);
        f32_split3(v.z, v.w, b[j][0][1], b[j][1][1], b[j][2][1]);
      }
      float c[2][4][4];
      constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
      for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (p == 0) f32_mma0(c[i][j], a[i][PA[p]], b[j][PB[p]]);
            else f32_mma(c[i][j], a[i][PA[p]], b[j][PB[p]]);
          }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[i][j0 + j][x] += c[i][j][x];
    }
  }
  float* part = f32_smem + F32_STAGES * STAGE;    // (a cluster's: the block's partial tile)
  auto store = [&](int m, int n, float v) { C[(size_t)m * N + n] = soft_limit(bias ? v + bias[n] : v, cap); };
  auto put = [&](int i, int j, int x, float v) {
    const int r = wm + i * 16 + g + (x >> 1) * 8, c = wn + j * 8 + 2 * t + (x & 1);
    if (cluster > 1) part[r * BN + c] = v;
    else if (m0 + r < M && n0 + c < N) store(m0 + r, n0 + c, v);
  };
  uint32_t odd[2] = {0u, 0u};                     // of a thread's sums, those that are not finite
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float v = acc[i][j][x] * F32_DOWN;
        odd[i] |= isfinite(v) ? 0u : 1u << (j * 4 + x);
        put(i, j, x, v);
      }
  // (every copy has landed and been read: the groups behind the last slice are empty)
  if (__syncthreads_or(odd[0] | odd[1])) {        // the tile once more, in whole numbers, for those sums
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
#pragma unroll 1
    for (int s = 0; s < F32_STAGES - 1; ++s) {
      if (s < nkb) load(s, s);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
#pragma unroll 1
    for (int kb = 0; kb < nkb; ++kb) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(F32_STAGES - 2) : "memory");
      __syncthreads();
      if (kb + F32_STAGES - 1 < nkb) load(kb + F32_STAGES - 1, (kb + F32_STAGES - 1) % F32_STAGES);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
      const float* as = f32_smem + (kb % F32_STAGES) * STAGE + (wm + g) * F32_BK;
      const float* ws = f32_smem + (kb % F32_STAGES) * STAGE + (BM + wn + 2 * t) * F32_BK;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const int k = ((q + t) & 3) * 4;          // (lanes with other columns at other places of a row: other banks)
        float4 v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] = *reinterpret_cast<const float4*>(as + r * 8 * F32_BK + k);
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float4 w = *reinterpret_cast<const float4*>(ws + (j * 8 + e) * F32_BK + k);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              float& c = acc[r >> 1][j][(r & 1) * 2 + e];
              c = fmaf(v[r].w, w.w, fmaf(v[r].z, w.z, fmaf(v[r].y, w.y, fmaf(v[r].x, w.x, c))));
            }
          }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (odd[i] >> (j * 4 + x) & 1u) put(i, j, x, acc[i][j][x]);
  }
  if (cluster == 1) return;
  cluster_sync_all();
  const int per = (BM + cluster - 1) / cluster, r1 = min(BM, (z + 1) * per);
  for (int r = z * per; r < r1; ++r) {
    const int m = m0 + r, n = n0 + tid;
    if (m >= M) break;
    float s = 0.f;
    for (int c = 0; c < cluster; ++c) s += cluster_load_f32(part + r * BN + tid, (uint32_t)c);
    if (n < N) store(m, n, s);
  }
  cluster_sync_all();                             // nobody's shared memory goes away while it is read
}

template <int MR, bool NORM, int EPI>
static int gemm_rows_f32_launch(const float* A, const float* W, float* C, int M, int N, int K, const F32RowsEnd& end, cudaStream_t stream) {
  const int n_out = EPI == F32_ROWS_SILU ? N / 2 : N, cols = EPI == F32_ROWS_SILU ? 2 : 4, tiles = (n_out + cols - 1) / cols;
  if (K >= 1024) return sx_launch(gemm_rows_f32_kernel<MR, 8, NORM, EPI>, dim3(tiles), dim3(256), 0, stream, A, W, C, M, N, K, end);
  if (K >= 256) return sx_launch(gemm_rows_f32_kernel<MR, 2, NORM, EPI>, dim3((tiles + 3) / 4), dim3(256), 0, stream, A, W, C, M, N, K, end);
  return sx_launch(gemm_rows_f32_kernel<MR, 1, NORM, EPI>, dim3((tiles + 7) / 8), dim3(256), 0, stream, A, W, C, M, N, K, end);
}
template <bool NORM, int EPI>
static int gemm_rows_f32_of(const float* A, const float* W, float* C, int M, int N, int K, const F32RowsEnd& end, cudaStream_t stream) {
  if (M <= 1) return gemm_rows_f32_launch<1, NORM, EPI>(A, W, C, M, N, K, end, stream);
  if (M <= 2) return gemm_rows_f32_launch<2, NORM, EPI>(A, W, C, M, N, K, end, stream);
  if (M <= 4) return gemm_rows_f32_launch<4, NORM, EPI>(A, W, C, M, N, K, end, stream);
  if (M <= 8) return gemm_rows_f32_launch<8, NORM, EPI>(A, W, C, M, N, K, end, stream);
  return gemm_rows_f32_launch<16, NORM, EPI>(A, W, C, M, N, K, end, stream);
}
template <bool NORM>
static int gemm_rows_f32(const float* A, const float* W, float* C, int M, int N, int K, const F32RowsEnd& end, cudaStream_t stream) {
  if (end.epi == F32_ROWS_SILU) return gemm_rows_f32_of<NORM, F32_ROWS_SILU>(A, W, C, M, N, K, end, stream);
  if (end.epi == F32_ROWS_ADD) return gemm_rows_f32_of<NORM, F32_ROWS_ADD>(A, W, C, M, N, K, end, stream);
  return gemm_rows_f32_of<NORM, F32_ROWS_STORE>(A, W, C, M, N, K, end, stream);
}

// The tiles of more rows: rows of a tile, and blocks that share a tile's K.
// Tiles of 64 rows only where they come to two a SM (us, tiles of 32 and of 64: 263 x 4,096 x 1,024 49 and 95, 300 x 6,144 x 1,024 98
// and 95, 512 x 6,144 143 and 135, 1,024 x 6,144 257 and 259).  About a block an SM is mostly enough (tiles of 32 by one, two, four and eight
// blocks on 148 SMs: 200 x 1,024 x 2,048 67, 41, 30, 31; 263 x 1,024 x 3,072 99, 57, 62, 52; 263 x 4,096 x 1,024 49, 59, 64, 64; not so 600 x
// 1,024 x 3,072, 140, 120, 98, 89); every block of a cluster keeps at least 128 of K.
struct F32Plan { int rows, cluster; };
static F32Plan gemm_f32_plan(int M, int N, int K, int sms) {
  const long long tiles_n = (N + 127LL) / 128;
  F32Plan p;
  p.rows = (M + 63) / 64 * tiles_n < 2LL * sms ? 32 : 64;
  const long long tiles = (M + p.rows - 1) / p.rows * tiles_n;
  p.cluster = 1;
  while (p.cluster < 8 && tiles * p.cluster < sms - sms / 18 && K >= 256 * p.cluster) p.cluster *= 2;
  return p;
}
extern "C" void sx_gemm_f32_plan(int M, int N, int K, int sms, int* out2) {
  const F32Plan p = gemm_f32_plan(M, N, K, sms);
  out2[0] = p.rows; out2[1] = p.cluster;
}

template <int BM>
static int gemm_tile_f32_launch(const float* A, const float* W, float* C, int M, int N, int K, const float* bias, float cap,
                                int cluster, cudaStream_t stream) {
  constexpr int BN = 128;
  const long long tiles_n = (N + BN - 1) / BN, tiles_m = (M + BM - 1) / BM;
  const size_t ring = ((size_t)F32_STAGES * (BM + BN) * F32_BK + (cluster > 1 ? BM * BN : 0)) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(gemm_tile_f32_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ring);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid((unsigned)(tiles_n * cluster), (unsigned)tiles_m);
  // Not launched early: blocks that may start while the kernel before still runs crowd the SMs that are free first, and few blocks
  // an SM then finish late (a 263-row step of a 0.6B model 10.6 ms, like this 8.7).
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = ring;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, gemm_tile_f32_kernel<BM>, A, W, C, M, N, K, bias, cap, cluster);
}

static int gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, const float* bias, float cap, cudaStream_t stream) {
  if (M <= 16) {
    F32RowsEnd end = {};
    end.bias = bias; end.cap = cap;
    return gemm_rows_f32<false>(A, W, C, M, N, K, end, stream);
  }
  const F32Plan p = gemm_f32_plan(M, N, K, sx_sm_count());
  return p.rows == 32 ? gemm_tile_f32_launch<32>(A, W, C, M, N, K, bias, cap, p.cluster, stream)
                      : gemm_tile_f32_launch<64>(A, W, C, M, N, K, bias, cap, p.cluster, stream);
}

template <typename TA, typename TW, typename TC>
static int gemm_generic_launch(const void* A, const void* W, void* C, int M, int N, int K, const float* bias, float cap,
                               cudaStream_t stream) {
  if (M <= 16) {
    gemm_rows_kernel<TA, TW, TC><<<(N + 3) / 4, 128, 0, stream>>>((const TA*)A, (const TW*)W, (TC*)C, M, N, K, bias, cap);
  } else {
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    gemm_tile_kernel<TA, TW, TC><<<grid, 256, 0, stream>>>((const TA*)A, (const TW*)W, (TC*)C, M, N, K, bias, cap);
  }
  return sx_launch_status();
}

extern "C" int sx_gemm_generic(const void* A, int a_dt, const void* W, int w_dt, void* C, int c_dt,
                               int M, int N, int K, const float* bias, float cap, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return SX_ERR_SIZE;
  if ((size_t)((M + 63) / 64) > 65535) return SX_ERR_SIZE;
  // (whole, aligned 16-byte pieces of every row, or the kernels that take every size)
  if (a_dt == SX_F32 && w_dt == SX_F32 && c_dt == SX_F32 && (K & 3) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0)
    return gemm_f32((const float*)A, (const float*)W, (float*)C, M, N, K, bias, cap, stream);
  if (a_dt == SX_F32 && w_dt == SX_F32 && c_dt == SX_F32)
    return gemm_generic_launch<float, float, float>(A, W, C, M, N, K, bias, cap, stream);
  if (a_dt == SX_BF16 && w_dt == SX_BF16 && c_dt == SX_BF16)
    return gemm_generic_launch<bf16, bf16, bf16>(A, W, C, M, N, K, bias, cap, stream);
  if (a_dt == SX_BF16 && w_dt == SX_BF16 && c_dt == SX_F32)
    return gemm_generic_launch<bf16, bf16, float>(A, W, C, M, N, K, bias, cap, stream);
  if (a_dt == SX_F32 && w_dt == SX_BF16 && c_dt == SX_F32)
    return gemm_generic_launch<float, bf16, float>(A, W, C, M, N, K, bias, cap, stream);
  return SX_ERR_DTYPE;
}

// Up to 16 float32 rows of whole, aligned 16-byte pieces.  gain (or null): A is normed on the way, rows of A * rsqrt(mean(A^2) + eps) * gain.
// epi 0: C [M, N] = the product (+ bias); 1: W = [gate; up] stacked, C [M, N/2] = silu(gate) * up; 2: C [M, N] += the product (+ bias).
extern "C" int sx_gemm_rows_f32(const float* A, const float* W, float* C, int M, int N, int K, const float* bias, int epi,
                                const float* gain, float eps, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 16 || K <= 0 || (K & 3) || epi < 0 || epi > 2 || (epi == F32_ROWS_SILU && (N & 1))) return SX_ERR_SIZE;
  if (((uintptr_t)A | (uintptr_t)W | (uintptr_t)gain) & 15) return SX_ERR_ALIGN;
  F32RowsEnd end = {bias, 0.f, epi, gain, eps, f32_rows_up(eps)};
  return gain ? gemm_rows_f32<true>(A, W, C, M, N, K, end, stream) : gemm_rows_f32<false>(A, W, C, M, N, K, end, stream);
}

// ---------------------------------------------------------------------------------------
// head preparation and cache write, one block per (token, head of the fused projection):
//   q heads: optional RMSNorm over the head (gain wq), optional rotate-half rotation of the
//            first rotary_dim elements by angle pos * inv_freq[i], written to q_out[t, head, :];
//   k heads: the same with wk, written into the sequence's page at the token's position;
//   v heads: copied into the page.
// qkv is [T, (nh + 2 nkv) * hd]: q heads, then k heads, then v heads.
// ---------------------------------------------------------------------------------------
// One block per token, one warp per head at a time.  A lane owns the rotation pairs
// (p, p + rotary_dim/2) for p = lane, lane + 32, ...; their angles, sines and cosines are computed
// once per token and reused for every q and k head.
#define QP_WARPS 8
#define QP_MAXP 8            // pairs per lane: head sizes up to 512
// PP: rotation pairs a lane owns (rotary_dim / 2 <= 32 * PP); angles, sines, cosines and the norm
// gains of its pairs stay in registers for all heads of the token
template <typename T, int PP>
__global__ void __launch_bounds__(QP_WARPS * 32) qkv_prepare_kernel(
    const T* __restrict__ qkv, T* __restrict__ q_out, T* __restrict__ k_pages, T* __restrict__ v_pages,
    const float* __restrict__ wq, const float* __restrict__ wk, const float* __restrict__ inv_freq,
    int rotary_dim, float eps, const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ block_table, int maxp, int nh, int nkv, int hd, int n_pages, int row, int vd) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = positions[t];
  const T* src_tok = qkv + (size_t)t * row;
  const int half = inv_freq ? rotary_dim / 2 : 0;

  float cs[PP], sn[PP], gq1[PP], gq2[PP], gk1[PP], gk2[PP];
#pragma unroll
  for (int k = 0; k < PP; ++k) {
    const int p = lane + 32 * k;
    cs[k] = 1.f; sn[k] = 0.f;
    gq1[k] = gq2[k] = gk1[k] = gk2[k] = 1.f;
    if (p < half) {
      sincosf((float)pos * inv_freq[p], &sn[k], &cs[k]);
      if (wq) { gq1[k] = wq[p]; gq2[k] = wq[p + half]; }
      if (wk) { gk1[k] = wk[p]; gk2[k] = wk[p + half]; }
    }
  }
  // where this token's keys and values go
  const int s = seq_of_token[t];
  const int page = block_table[(size_t)s * maxp + (pos >> 6)];
  const bool page_ok = page >= 0 && page < n_pages;     // the host guarantees a page; never write outside
  const bool vec_copy = (vd % 8 == 0) && (row % 8 == 0) && ((nh + nkv) * hd % 8 == 0) && sizeof(T) == 2 &&
                        (((uintptr_t)qkv | (uintptr_t)v_pages) & 15) == 0;

  for (int head = blockIdx.y * QP_WARPS + warp; head < nh + 2 * nkv; head += gridDim.y * QP_WARPS) {
    const bool is_q = head < nh, is_k = !is_q && head < nh + nkv;
    const int kvh = is_q ? 0 : (is_k ? head - nh : head - nh - nkv);
    // value heads have a size of their own (vd) and follow the nh + nkv heads of size hd
    const T* src = (is_q || is_k) ? src_tok + (size_t)head * hd : src_tok + (size_t)(nh + nkv) * hd + (size_t)kvh * vd;
    T* dst;
    if (is_q) {
      dst = q_out + ((size_t)t * nh + head) * hd;
    } else {
      T* base = is_k ? k_pages : v_pages;
      if (!base || !page_ok) continue;                   // a layer that reads another layer's cache writes nothing
      dst = base + (((size_t)page * nkv + kvh) * SX_PAGE + (pos & 63)) * (is_k ? hd : vd);
    }
    if (!is_q && !is_k) {                                // v: copy
      if (vec_copy) {
        for (int i = lane; i < vd / 8; i += 32) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
      } else {
        for (int i = lane; i < vd; i += 32) dst[i] = src[i];
      }
      continue;
    }
    const float* w = is_q ? wq : wk;
    float x1[PP], x2[PP];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < PP; ++k) {
      const int p = lane + 32 * k;
      x1[k] = x2[k] = 0.f;
      if (p < half) {
        x1[k] = to_f32(src[p]);
        x2[k] = to_f32(src[p + half]);
        ss += x1[k] * x1[k] + x2[k] * x2[k];
      }
    }
    for (int i = 2 * half + lane; i < hd; i += 32) {     // elements that are not rotated
      const float v = to_f32(src[i]);
      ss += v * v;
    }
    float inv = 1.f;
    if (w) inv = rsqrtf(warp_sum(ss) / (float)hd + eps);
#pragma unroll
    for (int k = 0; k < PP; ++k) {
      const int p = lane + 32 * k;
      if (p < half) {
        const float a = x1[k] * inv * (is_q ? gq1[k] : gk1[k]);
        const float b = x2[k] * inv * (is_q ? gq2[k] : gk2[k]);
        dst[p] = from_f32<T>(a * cs[k] - b * sn[k]);
        dst[p + half] = from_f32<T>(a * sn[k] + b * cs[k]);
      }
    }
    for (int i = 2 * half + lane; i < hd; i += 32) {
      const float v = to_f32(src[i]);
      dst[i] = from_f32<T>(w ? v * inv * w[i] : v);
    }
  }
}

// The common case (the whole head is rotated, head size a multiple of 4) with two adjacent pairs per
// lane and iteration, so that every access is 4 bytes (bfloat16) or 8 bytes (float) wide:
// a lane owns pairs p = 64 k + 2 lane + {0, 1}.
template <typename T> struct qp_vec2;
template <> struct qp_vec2<bf16> {
  static __device__ __forceinline__ float2 load(const bf16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }
  static __device__ __forceinline__ void store(bf16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }
};
template <> struct qp_vec2<float> {
  static __device__ __forceinline__ float2 load(const float* p) { return *reinterpret_cast<const float2*>(p); }
  static __device__ __forceinline__ void store(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
};

template <typename T, int PQ>
__global__ void __launch_bounds__(QP_WARPS * 32) qkv_prepare_vec_kernel(
    const T* __restrict__ qkv, T* __restrict__ q_out, T* __restrict__ k_pages, T* __restrict__ v_pages,
    const float* __restrict__ wq, const float* __restrict__ wk, const float* __restrict__ inv_freq, float eps,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table,
    int maxp, int nh, int nkv, int hd, int n_pages) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = positions[t];
  const int row = (nh + 2 * nkv) * hd;
  const T* src_tok = qkv + (size_t)t * row;
  const int half = hd / 2;

  float cs[PQ][2], sn[PQ][2], gq1[PQ][2], gq2[PQ][2], gk1[PQ][2], gk2[PQ][2];
#pragma unroll
  for (int k = 0; k < PQ; ++k)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int p = 64 * k + 2 * lane + j;
      cs[k][j] = 1.f; sn[k][j] = 0.f;
      gq1[k][j] = gq2[k][j] = gk1[k][j] = gk2[k][j] = 1.f;
      if (p < half) {
        if (inv_freq) sincosf((float)pos * inv_freq[p], &sn[k][j], &cs[k][j]);
        if (wq) { gq1[k][j] = wq[p]; gq2[k][j] = wq[p + half]; }
        if (wk) { gk1[k][j] = wk[p]; gk2[k][j] = wk[p + half]; }
      }
    }
  const int s = seq_of_token[t];
  const int page = block_table[(size_t)s * maxp + (pos >> 6)];
  const bool page_ok = page >= 0 && page < n_pages;

  for (int head = blockIdx.y * QP_WARPS + warp; head < nh + 2 * nkv; head += gridDim.y * QP_WARPS) {
    const bool is_q = head < nh, is_k = !is_q && head < nh + nkv;
    const int kvh = is_q ? 0 : (is_k ? head - nh : head - nh - nkv);
    const T* src = src_tok + (size_t)head * hd;
    T* dst;
    if (is_q) {
      dst = q_out + ((size_t)t * nh + head) * hd;
    } else {
      T* base = is_k ? k_pages : v_pages;
      if (!base || !page_ok) continue;
      dst = base + (((size_t)page * nkv + kvh) * SX_PAGE + (pos & 63)) * hd;
    }
    if (!is_q && !is_k) {                                // v: copy, 4 elements a lane and round
      for (int i = lane * 4; i < hd; i += 128) {
        const float2 a = qp_vec2<T>::load(src + i), b = qp_vec2<T>::load(src + i + 2);
        qp_vec2<T>::store(dst + i, a.x, a.y);
        qp_vec2<T>::store(dst + i + 2, b.x, b.y);
      }
      continue;
    }
    const bool normed = (is_q ? wq : wk) != nullptr;
    float2 x1[PQ], x2[PQ];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < PQ; ++k) {
      const int p = 64 * k + 2 * lane;
      x1[k] = x2[k] = make_float2(0.f, 0.f);
      if (p < half) {
        x1[k] = qp_vec2<T>::load(src + p);
        x2[k] = qp_vec2<T>::load(src + p + half);
        ss += x1[k].x * x1[k].x + x1[k].y * x1[k].y + x2[k].x * x2[k].x + x2[k].y * x2[k].y;
      }
    }
    float inv = 1.f;
    if (normed) inv = rsqrtf(warp_sum(ss) / (float)hd + eps);
#pragma unroll
    for (int k = 0; k < PQ; ++k) {
      const int p = 64 * k + 2 * lane;
      if (p < half) {
        const float a0 = x1[k].x * inv * (is_q ? gq1[k][0] : gk1[k][0]), a1 = x1[k].y * inv * (is_q ? gq1[k][1] : gk1[k][1]);
        const float b0 = x2[k].x * inv * (is_q ? gq2[k][0] : gk2[k][0]), b1 = x2[k].y * inv * (is_q ? gq2[k][1] : gk2[k][1]);
        qp_vec2<T>::store(dst + p, a0 * cs[k][0] - b0 * sn[k][0], a1 * cs[k][1] - b1 * sn[k][1]);
        qp_vec2<T>::store(dst + p + half, a0 * sn[k][0] + b0 * cs[k][0], a1 * sn[k][1] + b1 * cs[k][1]);
      }
    }
  }
}

// bfloat16, the whole head rotated (or nothing), head size 64 or 128, many tokens: 16 values a lane (8 from
// each half of the head, two 16-byte loads), so HD/16 lanes share a head and a warp works on 32/(HD/16) heads
// at once; sines, cosines and gains are computed once per block into shared memory.  The kernel above spends
// ~25 instructions per value (4 values a lane, every warp recomputing the token's sines): measured 24 us for
// 2,048 tokens x 48 heads, bound by instruction issue, where memory alone would need 8.
template <int HD>
__global__ void __launch_bounds__(QP_WARPS * 32) qkv_prepare_wide_kernel(
    const bf16* __restrict__ qkv, bf16* __restrict__ q_out, bf16* __restrict__ k_pages, bf16* __restrict__ v_pages,
    const float* __restrict__ wq, const float* __restrict__ wk, const float* __restrict__ inv_freq, float eps,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table,
    int maxp, int nh, int nkv, int n_pages, int row) {
  constexpr int HALF = HD / 2, LPH = HD / 16, HPW = 32 / LPH;      // lanes a head, heads a warp
  __shared__ float s_cs[HALF], s_sn[HALF], s_gq[HD], s_gk[HD];
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = positions[t];
  for (int i = threadIdx.x; i < HALF; i += QP_WARPS * 32) {
    float sn = 0.f, cs = 1.f;
    if (inv_freq) sincosf((float)pos * inv_freq[i], &sn, &cs);
    s_cs[i] = cs;
    s_sn[i] = sn;
  }
  for (int i = threadIdx.x; i < HD; i += QP_WARPS * 32) {
    s_gq[i] = wq ? wq[i] : 1.f;
    s_gk[i] = wk ? wk[i] : 1.f;
  }
  const int s = seq_of_token[t];
  const int page = block_table[(size_t)s * maxp + (pos >> 6)];
  const bool page_ok = page >= 0 && page < n_pages;
  __syncthreads();

  const int n_heads = nh + 2 * nkv;
  const bf16* src_tok = qkv + (size_t)t * row;                      // a row may hold other columns behind the heads
  const int sub = lane / LPH, e0 = (lane % LPH) * 8;               // which head of the warp's group; first value
  for (int hg = (blockIdx.y * QP_WARPS + warp) * HPW; hg < n_heads; hg += gridDim.y * QP_WARPS * HPW) {
    const int head = hg + sub;
    const bool live = head < n_heads;
    const bool is_q = head < nh, is_k = !is_q && head < nh + nkv;
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    if (live) {
      const bf16* src = src_tok + (size_t)head * HD + e0;
      a = *reinterpret_cast<const uint4*>(src);
      b = *reinterpret_cast<const uint4*>(src + HALF);
    }
    bf16* dst = nullptr;
    if (live) {
      if (is_q) {
        dst = q_out + ((size_t)t * nh + head) * HD + e0;
      } else {
        bf16* base = is_k ? k_pages : v_pages;
        const int kvh = is_k ? head - nh : head - nh - nkv;
        if (base && page_ok) dst = base + (((size_t)page * nkv + kvh) * SX_PAGE + (pos & 63)) * HD + e0;
      }
    }
    float x1[8], x2[8];
    const uint32_t* au = reinterpret_cast<const uint32_t*>(&a);
    const uint32_t* bu = reinterpret_cast<const uint32_t*>(&b);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 fa = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&au[i]));
      const float2 fb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bu[i]));
      x1[2 * i] = fa.x; x1[2 * i + 1] = fa.y; x2[2 * i] = fb.x; x2[2 * i + 1] = fb.y;
      ss += fa.x * fa.x + fa.y * fa.y + fb.x * fb.x + fb.y * fb.y;
    }
    // the head's sum of squares over its LPH lanes (every lane takes part; v heads carry theirs along unused)
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (!dst) continue;
    if (is_q || is_k) {
      const float* gn = is_q ? s_gq : s_gk;
      const bool normed = (is_q ? wq : wk) != nullptr;
      const float inv = normed ? rsqrtf(ss / (float)HD + eps) : 1.f;
      uint32_t* ao = reinterpret_cast<uint32_t*>(&a);
      uint32_t* bo = reinterpret_cast<uint32_t*>(&b);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float lo[2], hi[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int e = e0 + 2 * i + j;
          const float u = x1[2 * i + j] * inv * gn[e], w = x2[2 * i + j] * inv * gn[e + HALF];
          lo[j] = u * s_cs[e] - w * s_sn[e];
          hi[j] = u * s_sn[e] + w * s_cs[e];
        }
        __nv_bfloat162 plo = __floats2bfloat162_rn(lo[0], lo[1]), phi = __floats2bfloat162_rn(hi[0], hi[1]);
        ao[i] = *reinterpret_cast<uint32_t*>(&plo);
        bo[i] = *reinterpret_cast<uint32_t*>(&phi);
      }
    }
    *reinterpret_cast<uint4*>(dst) = a;
    *reinterpret_cast<uint4*>(dst + HALF) = b;
  }
}

template <typename T>
static int qkv_prepare_launch(dim3 grid, cudaStream_t stream, const void* qkv, void* q_out, void* k_pages, void* v_pages,
                              const float* wq, const float* wk, const float* inv_freq, int rotary_dim, float eps,
                              const int* positions, const int* seq_of_token, const int* block_table, int maxp, int nh,
                              int nkv, int hd, int n_pages, int row, int vd) {
  const int pairs = inv_freq ? rotary_dim / 2 : 0;
  const bool packed = row == (nh + 2 * nkv) * hd && vd == hd;      // the layout the two faster kernels assume
  const bool aligned = (((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_pages | (uintptr_t)v_pages) & 7) == 0;
  if (vd == hd && row % 8 == 0 && sizeof(T) == 2 && (hd == 128 || hd == 64) && (!inv_freq || rotary_dim == hd) && grid.y == 1 &&
      (((uintptr_t)qkv | (uintptr_t)q_out | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0) {
#define QP_WGO(HD)                                                                                                       \
  return sx_launch(qkv_prepare_wide_kernel<HD>, grid, dim3(QP_WARPS * 32), 0, stream, (const bf16*)qkv, (bf16*)q_out,      \
                   (bf16*)k_pages, (bf16*)v_pages, wq, wk, inv_freq, eps, positions, seq_of_token, block_table, maxp, nh,  \
                   nkv, n_pages, row)
    if (hd == 128) QP_WGO(128);
    QP_WGO(64);
#undef QP_WGO
  }
  if (packed && hd % 4 == 0 && hd <= 512 && aligned && (!inv_freq || rotary_dim == hd)) {
#define QP_VGO(PQ)                                                                                                     \
  return sx_launch(qkv_prepare_vec_kernel<T, PQ>, grid, dim3(QP_WARPS * 32), 0, stream, (const T*)qkv, (T*)q_out, (T*)k_pages, \
                   (T*)v_pages, wq, wk, inv_freq, eps, positions, seq_of_token, block_table, maxp, nh, nkv, hd, n_pages)
    if (hd <= 128) QP_VGO(1);
    else if (hd <= 256) QP_VGO(2);
    else QP_VGO(4);
#undef QP_VGO
  }
#define QP_GO(PP)                                                                                                   \
  return sx_launch(qkv_prepare_kernel<T, PP>, grid, dim3(QP_WARPS * 32), 0, stream, (const T*)qkv, (T*)q_out, (T*)k_pages, \
                   (T*)v_pages, wq, wk, inv_freq, rotary_dim, eps, positions, seq_of_token, block_table, maxp, nh, nkv, hd, n_pages, row, vd)
  if (pairs <= 32) QP_GO(1);
  else if (pairs <= 64) QP_GO(2);
  else if (pairs <= 128) QP_GO(4);
  else QP_GO(8);
#undef QP_GO
}

static int qkv_prepare_any(const void* qkv, void* q_out, void* k_pages, void* v_pages,
                              const float* wq, const float* wk, const float* inv_freq, int rotary_dim,
                              float eps, const int* positions, const int* seq_of_token,
                              const int* block_table, int maxp, int n_tokens, int nh, int nkv, int hd,
                              int n_pages, int dt, int row, int vd, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (hd <= 0 || (rotary_dim & 1) || rotary_dim > hd || rotary_dim / 2 > 32 * QP_MAXP) return SX_ERR_SIZE;
  if (vd <= 0 || row < (nh + nkv) * hd + nkv * vd) return SX_ERR_SIZE;
  // few tokens: spread the heads over blocks too, so that the step is one round of work
  const int heads = nh + 2 * nkv;
  dim3 grid(n_tokens, n_tokens <= 64 ? (heads + QP_WARPS - 1) / QP_WARPS : 1);
  if (dt == SX_F32)
    return qkv_prepare_launch<float>(grid, stream, qkv, q_out, k_pages, v_pages, wq, wk, inv_freq, rotary_dim, eps, positions,
                                     seq_of_token, block_table, maxp, nh, nkv, hd, n_pages, row, vd);
  if (dt == SX_BF16)
    return qkv_prepare_launch<bf16>(grid, stream, qkv, q_out, k_pages, v_pages, wq, wk, inv_freq, rotary_dim, eps, positions,
                                    seq_of_token, block_table, maxp, nh, nkv, hd, n_pages, row, vd);
  return SX_ERR_DTYPE;
}

extern "C" int sx_qkv_prepare(const void* qkv, void* q_out, void* k_pages, void* v_pages,
                              const float* wq, const float* wk, const float* inv_freq, int rotary_dim,
                              float eps, const int* positions, const int* seq_of_token,
                              const int* block_table, int maxp, int n_tokens, int nh, int nkv, int hd,
                              int n_pages, int dt, cudaStream_t stream) {
  return qkv_prepare_any(qkv, q_out, k_pages, v_pages, wq, wk, inv_freq, rotary_dim, eps, positions, seq_of_token, block_table,
                         maxp, n_tokens, nh, nkv, hd, n_pages, dt, (nh + 2 * nkv) * hd, hd, stream);
}

// The same for a projection whose rows are `row` elements long (q heads, k heads and v heads first, other columns
// behind them) and whose value heads have `vd` elements.
extern "C" int sx_qkv_prepare_strided(const void* qkv, void* q_out, void* k_pages, void* v_pages,
                                      const float* wq, const float* wk, const float* inv_freq, int rotary_dim,
                                      float eps, const int* positions, const int* seq_of_token,
                                      const int* block_table, int maxp, int n_tokens, int nh, int nkv, int hd,
                                      int n_pages, int dt, int row, int vd, cudaStream_t stream) {
  return qkv_prepare_any(qkv, q_out, k_pages, v_pages, wq, wk, inv_freq, rotary_dim, eps, positions, seq_of_token, block_table,
                         maxp, n_tokens, nh, nkv, hd, n_pages, dt, row, vd, stream);
}

// ---------------------------------------------------------------------------------------
// cosines and sines of position * inv_freq[i] for every token of a step, [n_tokens, pairs] each: what the head
// preparation computes per token, made once for a product whose epilogue prepares the heads
// ---------------------------------------------------------------------------------------
__global__ void rope_table_kernel(const int* __restrict__ positions, const float* __restrict__ inv_freq, int pairs,
                                  float* __restrict__ cs, float* __restrict__ sn, size_t n) {
  pdl_wait();
  pdl_trigger();
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const size_t t = idx / pairs;
  const int i = (int)(idx - t * pairs);
  float s, c;
  sincosf((float)positions[t] * inv_freq[i], &s, &c);
  cs[idx] = c;
  sn[idx] = s;
}
extern "C" int sx_rope_table(const int* positions, const float* inv_freq, int pairs, int n_tokens, float* cs, float* sn,
                             cudaStream_t stream) {
  if (n_tokens <= 0 || pairs <= 0) return 0;
  const size_t n = (size_t)n_tokens * pairs;
  return sx_launch(rope_table_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, positions, inv_freq, pairs, cs, sn, n);
}

// ---------------------------------------------------------------------------------------
// attention over the paged cache, one block per (token, query head): scores of the keys
// lo..pos in tiles of 128, running maximum and sum (online softmax), all in 32-bit.
//   lo = window > 0 ? max(0, pos - window + 1) : 0, and with chunk > 0 at least (pos / chunk) * chunk: a query then
//   sees only keys of its own chunk of positions;  query head h reads kv head h / (nh/nkv).
//   softcap > 0: score <- softcap * tanh(score / softcap) after the scale.
//   sinks: one number per query head that stands in the softmax's denominator as exp(sink) beside the keys' terms
//   (no key, no value, neither scaled nor capped): the running maximum starts at the sink and the running sum at 1.
//   Keys have hd elements, values vd; the result goes to out[t * out_stride + h * vd + d], times out_scale.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) attn_generic_kernel(
    const T* __restrict__ q, const T* __restrict__ k_pages, const T* __restrict__ v_pages,
    T* __restrict__ out, const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ block_table, int maxp, int nh, int nkv, int hd, float scale, int window,
    int vd, float softcap, const float* __restrict__ sinks, int chunk, int out_stride, float out_scale) {
  extern __shared__ float smem[];
  float* qs = smem;            // hd
  float* ps = smem + hd;       // 128
  __shared__ float red[33];
  const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int pos = positions[t];
  const int* bt = block_table + (size_t)seq_of_token[t] * maxp;
  const int kvh = h / (nh / nkv);
  const T* qr = q + ((size_t)t * nh + h) * hd;
  for (int i = tid; i < hd; i += 128) qs[i] = to_f32(qr[i]);
  __syncthreads();

  int lo = window > 0 ? max(0, pos - window + 1) : 0;
  if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
  float m = sinks ? sinks[h] : -INFINITY, l = sinks ? 1.f : 0.f;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};     // vd <= 512

  for (int j0 = lo; j0 <= pos; j0 += 128) {
    const int j = j0 + tid;
    float s = -INFINITY;
    if (j <= pos) {
      const int page = bt[j >> 6];
      const T* kr = k_pages + (((size_t)page * nkv + kvh) * SX_PAGE + (j & 63)) * hd;
      float d = 0.f;
      for (int i = 0; i < hd; ++i) d = fmaf(qs[i], to_f32(kr[i]), d);
      s = d * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    }
    const float tmax = block_max(s, red);
    const float m_new = fmaxf(m, tmax);
    const float p = (j <= pos) ? expf(s - m_new) : 0.f;
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    ps[tid] = p;
    const float psum = block_sum(p, red);   // also orders the writes to ps before the reads below
    l = l * corr + psum;
    const int ntile = min(128, pos - j0 + 1);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int d = tid + a * 128;
      if (d < vd) {
        float v = acc[a] * corr;
        for (int jj = 0; jj < ntile; ++jj) {
          const int jk = j0 + jj;
          const int page = bt[jk >> 6];
          v = fmaf(ps[jj], to_f32(v_pages[(((size_t)page * nkv + kvh) * SX_PAGE + (jk & 63)) * vd + d]), v);
        }
        acc[a] = v;
      }
    }
    m = m_new;
    __syncthreads();
  }
  T* o = out + (size_t)t * out_stride + (size_t)h * vd;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int d = tid + a * 128;
    if (d < vd) o[d] = from_f32<T>(acc[a] / l * out_scale);
  }
}

// ---------------------------------------------------------------------------------------
// The float32 form of the kernel above for heads of 64 and 128 (keys and values alike): eight lanes share a key, so that a
// key's or value's row is read in whole 128-byte lines, and the R query rows of a block (the heads that share a kv head; with
// fewer heads than R also neighbouring tokens of the same sequence) read it once.  Every group of eight lanes is an online
// softmax of its own over every 32nd (times the cluster's blocks) key; the groups, warps and blocks are merged at the end,
// in order.  A few tokens: the keys are shared by the blocks of a cluster too.  Bound by the latency of a few dependent loads in
// single-token steps: 14 us where the plain kernel, in which a thread walks a whole key alone, 4 bytes a load and each lane on
// lines of its own, took 55 (steps of 2 and of 263 tokens, 16 heads, up to 158 keys).
// ---------------------------------------------------------------------------------------
// Whether the sequence whose neighbouring tokens [from, to) these are brings fewer than `few` (up to 33) in all, going by the tokens
// beside them (a whole warp asks).
__device__ __forceinline__ bool attn_f32_few(const int* __restrict__ seq_of_token, int n_tokens, int from, int to, int seq, int few) {
  if (to - from >= few) return false;
  const int lane = threadIdx.x & 31, a = from - 1 - lane, b = to + lane;
  const unsigned ahead = __ballot_sync(0xffffffffu, a >= 0 && seq_of_token[a] == seq);
  const unsigned behind = __ballot_sync(0xffffffffu, b < n_tokens && seq_of_token[b] == seq);
  const int n = (ahead == 0xffffffffu ? 32 : __ffs(~ahead) - 1) + (behind == 0xffffffffu ? 32 : __ffs(~behind) - 1);
  return to - from + n < few;
}

// (tokens `begin` .. `n_tokens` - 1; few > 0: only those of sequences that bring fewer)
template <int HD, int R>
__global__ void __launch_bounds__(256) attn_f32_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages, float* __restrict__ out,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp,
    int n_tokens, int nh, int nkv, float scale, int window, float softcap, const float* __restrict__ sinks, int chunk,
    int out_stride, float out_scale, int tpb, int cluster, int begin, int few) {
  constexpr int C4 = HD / 32;                     // 16-byte pieces a lane holds of a head
  __shared__ float s_acc[8][R][HD];
  __shared__ float s_ml[8][R][2], s_blk[R][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, grp = lane >> 3;
  const int G = nh / nkv, hg = (G + R - 1) / R;   // blocks that share a kv head's query heads (1 when tpb > 1)
  const int kvh = blockIdx.y / hg, h0 = (blockIdx.y % hg) * R;
  const int t0 = begin + blockIdx.z * tpb, rank = blockIdx.x;
  const int stream0 = (rank * 8 + warp) * 4 + grp, streams = cluster * 32;
  pdl_wait();
  pdl_trigger();
  int first = 0;                                  // tokens of one sequence at a time
  const int n_here = min(tpb, n_tokens - t0);
  while (first < n_here) {
    const int seq = seq_of_token[t0 + first];
    int end = first + 1;
    while (end < n_here && seq_of_token[t0 + end] == seq) ++end;
    if (few > 0 && !attn_f32_few(seq_of_token, n_tokens, t0 + first, t0 + end, seq, few)) {      // (all blocks of a cluster alike)
      first = end;
      continue;
    }
    const int* bt = block_table + (size_t)seq * maxp;
    int pos[R], lo[R];
    float4 qv[R][C4], acc[R][C4];
    float m[R], l[R];
    int jlo = 0x7fffffff, jhi = -1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int tok = tpb > 1 ? r / G : 0, head = tpb > 1 ? r % G : h0 + r;
      const bool live = tok >= first && tok < end && head < G;
      pos[r] = live ? positions[t0 + tok] : -1;
      lo[r] = window > 0 ? max(0, pos[r] - window + 1) : 0;
      if (chunk > 0 && live) lo[r] = max(lo[r], (pos[r] / chunk) * chunk);
      if (live) { jlo = min(jlo, lo[r]); jhi = max(jhi, pos[r]); }
      m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
      for (int c = 0; c < C4; ++c) {
        acc[r][c] = qv[r][c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) qv[r][c] = *reinterpret_cast<const float4*>(q + ((size_t)(t0 + tok) * nh + kvh * G + head) * HD + (c * 8 + sub) * 4);
      }
    }
    auto row_of = [&](int j) { return (((size_t)bt[j >> 6] * nkv + kvh) * SX_PAGE + (j & 63)) * HD + sub * 4; };
    float4 kc[C4], vc[C4];
    auto fetch = [&](int j) {
      if (j <= jhi) {
        const size_t at = row_of(j);
#pragma unroll
        for (int c = 0; c < C4; ++c) kc[c] = *reinterpret_cast<const float4*>(k_pages + at + c * 32);
#pragma unroll
        for (int c = 0; c < C4; ++c) vc[c] = *reinterpret_cast<const float4*>(v_pages + at + c * 32);
      } else {
#pragma unroll
        for (int c = 0; c < C4; ++c) kc[c] = vc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    // (the warp's groups walk together: the sums over eight lanes are whole-warp shuffles)
    const int j_warp = jlo + (rank * 8 + warp) * 4;
    fetch(jlo + stream0);
    for (int jw = j_warp; jw <= jhi; jw += streams) {
      const int j = jw + grp;
      float s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float d = 0.f;
#pragma unroll
        for (int c = 0; c < C4; ++c)
          d = fmaf(qv[r][c].w, kc[c].w, fmaf(qv[r][c].z, kc[c].z, fmaf(qv[r][c].y, kc[c].y, fmaf(qv[r][c].x, kc[c].x, d))));
        s[r] = d;
      }
      float4 v[C4];
#pragma unroll
      for (int c = 0; c < C4; ++c) v[c] = vc[c];
      fetch(j + streams);                         // the next key is on its way behind the softmax
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
        s[r] *= scale;
        if (softcap > 0.f) s[r] = softcap * tanhf(s[r] / softcap);
        if (j > pos[r] || j < lo[r]) continue;
        const float m_new = fmaxf(m[r], s[r]);
        // (a score of minus infinity has no weight, also where a group has seen no other yet)
        const float corr = m[r] == -INFINITY ? 0.f : expf(m[r] - m_new), p = s[r] == -INFINITY ? 0.f : expf(s[r] - m_new);
        m[r] = m_new;
        l[r] = fmaf(l[r], corr, p);
#pragma unroll
        for (int c = 0; c < C4; ++c) {
          acc[r][c].x = fmaf(p, v[c].x, acc[r][c].x * corr); acc[r][c].y = fmaf(p, v[c].y, acc[r][c].y * corr);
          acc[r][c].z = fmaf(p, v[c].z, acc[r][c].z * corr); acc[r][c].w = fmaf(p, v[c].w, acc[r][c].w * corr);
        }
      }
    }
    // the four groups of the warp, then its result to shared memory
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 8; o < 32; o <<= 1) {
        const float mo = __shfl_xor_sync(0xffffffffu, m[r], o), lo_ = __shfl_xor_sync(0xffffffffu, l[r], o);
        const float mx = fmaxf(m[r], mo);
        const float a = m[r] == -INFINITY ? 0.f : expf(m[r] - mx), b = mo == -INFINITY ? 0.f : expf(mo - mx);
        l[r] = l[r] * a + lo_ * b;
        m[r] = mx;
#pragma unroll
        for (int c = 0; c < C4; ++c) {
          acc[r][c].x = acc[r][c].x * a + __shfl_xor_sync(0xffffffffu, acc[r][c].x, o) * b;
          acc[r][c].y = acc[r][c].y * a + __shfl_xor_sync(0xffffffffu, acc[r][c].y, o) * b;
          acc[r][c].z = acc[r][c].z * a + __shfl_xor_sync(0xffffffffu, acc[r][c].z, o) * b;
          acc[r][c].w = acc[r][c].w * a + __shfl_xor_sync(0xffffffffu, acc[r][c].w, o) * b;
        }
      }
      if (grp == 0) {
#pragma unroll
        for (int c = 0; c < C4; ++c) *reinterpret_cast<float4*>(&s_acc[warp][r][(c * 8 + sub) * 4]) = acc[r][c];
        if (sub == 0) { s_ml[warp][r][0] = m[r]; s_ml[warp][r][1] = l[r]; }
      }
    }
    __syncthreads();
    // the block's warps; with a cluster the result stays in shared memory (in the place of warp 0's, which only this thread reads)
    for (int i = threadIdx.x; i < R * HD; i += 256) {
      const int r = i / HD, d = i % HD;
      const int tok = tpb > 1 ? r / G : 0, head = tpb > 1 ? r % G : h0 + r;
      const bool live = tok >= first && tok < end && head < G;
      const int h = kvh * G + head;
      float mx = cluster == 1 && sinks && live ? sinks[h] : -INFINITY;
#pragma unroll
      for (int w = 0; w < 8; ++w) mx = fmaxf(mx, s_ml[w][r][0]);
      float sum = cluster == 1 && sinks && live ? expf(sinks[h] - mx) : 0.f, o = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float f = s_ml[w][r][0] == -INFINITY ? 0.f : expf(s_ml[w][r][0] - mx);
        sum = fmaf(s_ml[w][r][1], f, sum);
        o = fmaf(s_acc[w][r][d], f, o);
      }
      if (cluster == 1) {
        if (live) out[(size_t)(t0 + tok) * out_stride + (size_t)h * HD + d] = o / sum * out_scale;
      } else {
        s_acc[0][r][d] = o;
        if (d == 0) { s_blk[r][0] = mx; s_blk[r][1] = sum; }
      }
    }
    if (cluster > 1) {
      cluster_sync_all();
      // block `rank` finishes every cluster-th piece of 256 elements
      for (int i = threadIdx.x + rank * 256; i < R * HD; i += 256 * cluster) {
        const int r = i / HD, d = i % HD, head = h0 + r;
        if (head >= G) continue;
        const int h = kvh * G + head;
        float mb[8], lb[8], ob[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const uint32_t from = (uint32_t)min(b, cluster - 1);
          mb[b] = cluster_load_f32(&s_blk[r][0], from);
          lb[b] = cluster_load_f32(&s_blk[r][1], from);
          ob[b] = cluster_load_f32(&s_acc[0][r][d], from);
        }
        float mx = sinks ? sinks[h] : -INFINITY;
#pragma unroll
        for (int b = 0; b < 8; ++b) mx = fmaxf(mx, mb[b]);
        float sum = sinks ? expf(sinks[h] - mx) : 0.f, o = 0.f;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const float f = b < cluster && mb[b] != -INFINITY ? expf(mb[b] - mx) : 0.f;
          sum = fmaf(lb[b], f, sum);
          o = fmaf(ob[b], f, o);
        }
        out[(size_t)t0 * out_stride + (size_t)h * HD + d] = o / sum * out_scale;
      }
      cluster_sync_all();                         // nobody's shared memory goes away while it is read
    } else {
      __syncthreads();
    }
    first = end;
  }
}

// ---------------------------------------------------------------------------------------
// Prompt portions: 32 query rows of a head a block on the tensor cores, with operands in three bfloat16 pieces as in
// gemm_tile_f32_kernel (six products of pieces, each slice of 16 summed from zero and added in 32 bits; here the leading product on
// its own, f32_products, which keeps the error below that of the kernel above: 1.2e-7 against 1.3e-7 with 300 keys, 1.9e-7 against 2.0e-7
// with 1,000).  Eight warps: 16 rows and every fourth 16 of a page's 64 keys each; the four parts of the keys are added up at the end.
// A row's query pieces lie in shared memory as the instructions take them; keys and values come through two stages (cp.async), rows
// padded so that 16-byte reads meet no bank twice.  Within an instruction the order of the 16 elements of a head (scores) and of
// the 32 columns of four instructions (values) is the one in which a thread's numbers are neighbours in memory.  A row with a
// score or result that is not finite is done again in 32 bits by a warp (attn_f32_row; two prompts of 150 tokens, all rows so, 32 -> 76 us,
// 2,048 tokens 0.55 -> 3.07 ms, where the kernel above takes 2.5).  Two prompts of 150 tokens, 16 heads of 128: 70 -> 30 us, what is left is the latency of a page
// (3.5 to 4.4 us: 192 products of pieces and 1,000 other instructions a warp); with four warps and 32 keys a turn 37 us (2,048 tokens of
// 32 heads 930, where this took 1,059 and now takes 1,095), with the results scaled and divided by the threads that hold them, 64 divisions
// one after the other, 44.
// ---------------------------------------------------------------------------------------
// one query row by one warp, 16 keys at a time: their keys and values are on the way together
template <int HD>
__device__ __noinline__ void attn_f32_row(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                                          float* __restrict__ out, const int* __restrict__ bt, int nkv, int kvh, int lo, int pos,
                                          float scale, float softcap, const float* sink, float out_scale, int lane) {
  constexpr int C = HD / 32, B = 16;
  float qv[C], acc[C], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int c = 0; c < C; ++c) { qv[c] = q[c * 32 + lane]; acc[c] = 0.f; }
#pragma unroll 1
  for (int j0 = lo & ~(B - 1); j0 <= pos; j0 += B) {
    const size_t at = (((size_t)bt[j0 >> 6] * nkv + kvh) * SX_PAGE + (j0 & 63)) * HD + lane;
    float d[B], v[B][C];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const bool seen = j0 + b >= lo && j0 + b <= pos;           // (what lies beside them may be anything)
      d[b] = 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        d[b] = fmaf(qv[c], seen ? k_pages[at + b * HD + c * 32] : 0.f, d[b]);
        v[b][c] = seen ? v_pages[at + b * HD + c * 32] : 0.f;
      }
    }
    float s = warp_fold<B>(d, lane) * scale;                     // of key lane / 2
    if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    const int j = j0 + lane / 2;
    if (j < lo || j > pos) s = -INFINITY;
    const float m_new = fmaxf(m, warp_max(s));
    const float corr = m == -INFINITY ? 0.f : expf(m - m_new), p = s == -INFINITY ? 0.f : expf(s - m_new);
    m = m_new;
    l = fmaf(l, corr, warp_sum(lane & 1 ? 0.f : p));
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] *= corr;
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const float pb = __shfl_sync(0xffffffffu, p, 2 * b);
#pragma unroll
      for (int c = 0; c < C; ++c) acc[c] = fmaf(pb, v[b][c], acc[c]);
    }
  }
  const float mx = sink ? fmaxf(m, *sink) : m, f = m == -INFINITY ? 0.f : expf(m - mx);
  const float sum = l * f + (sink ? expf(*sink - mx) : 0.f);
#pragma unroll
  for (int c = 0; c < C; ++c) out[c * 32 + lane] = acc[c] * f / sum * out_scale;
}

__device__ __noinline__ float f32_capped(float s, float cap) { return cap * tanhf(s / cap); }

template <int HD, int KW>
__global__ void __launch_bounds__(64 * KW, 4 / KW) attn_f32_tile_kernel(
    const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages, float* __restrict__ out,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int maxp,
    int n_tokens, int nh, int nkv, float scale, int window, float softcap, const float* __restrict__ sinks, int chunk,
    int out_stride, float out_scale, int few) {
  constexpr int KS = HD / 16, NB = HD / 32, SK = HD + 16, SV = HD + 4, KEYS = 16 * KW, THREADS = 64 * KW, STAGE = KEYS * (SK + SV);
  extern __shared__ __align__(16) float f32_smem[];
  uint4* s_q = reinterpret_cast<uint4*>(f32_smem + 2 * STAGE);             // [row warp][slice][piece][lane]
  __shared__ float s_m[KW][32], s_l[KW][32];
  __shared__ int s_bad[KW][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, wr = warp & 1, wk = warp >> 1;
  const int h = blockIdx.x, kvh = h / (nh / nkv), t0 = (gridDim.y - 1 - blockIdx.y) * 32;      // (rows with many keys first)
  const int n_here = min(32, n_tokens - t0);
  const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(f32_smem);
  pdl_wait();
  pdl_trigger();
  int first = 0;                                  // tokens of one sequence at a time
  while (first < n_here) {
    const int seq = seq_of_token[t0 + first];
    int end = first + 1;
    while (end < n_here && seq_of_token[t0 + end] == seq) ++end;
    if (few > 0 && attn_f32_few(seq_of_token, n_tokens, t0 + first, t0 + end, seq, few)) {
      first = end;
      continue;
    }
    const int* bt = block_table + (size_t)seq * maxp;
    auto low = [&](int p) {
      const int a = window > 0 ? max(0, p - window + 1) : 0;
      return chunk > 0 ? max(a, p / chunk * chunk) : a;
    };
    const bool mine = lane >= first && lane < end;
    const int p_lane = mine ? positions[t0 + lane] : -1;
    const int jhi = __reduce_max_sync(0xffffffffu, p_lane), jlo = __reduce_min_sync(0xffffffffu, mine ? low(p_lane) : 0x7fffffff);
    // (keys outside jlo .. jhi are zeros: their pages may hold anything)
    auto load = [&](int jb, int s) {
      const size_t at = (((size_t)bt[jb >> 6] * nkv + kvh) * SX_PAGE + (jb & 63)) * HD;
#pragma unroll 4
      for (int i = 0; i < KEYS * HD / 4 / THREADS; ++i) {
        const int idx = tid + i * THREADS, r = idx / (HD / 4), c = idx % (HD / 4) * 4;
        const bool live = jb + r >= jlo && jb + r <= jhi;
        const uint32_t dst = smem0 + (uint32_t)(s * STAGE + r * SK + c) * 4, dst_v = smem0 + (uint32_t)(s * STAGE + KEYS * SK + r * SV + c) * 4;
        f32_cp16(dst, live ? k_pages + at + r * HD + c : k_pages, live);
        f32_cp16(dst_v, live ? v_pages + at + r * HD + c : v_pages, live);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int jb0 = jlo & ~(KEYS - 1);
    load(jb0, 0);
    int pos[2], lo[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = wr * 16 + g + i * 8;
      const bool live = row >= first && row < end;
      pos[i] = live ? positions[t0 + row] : -1;
      lo[i] = live ? low(pos[i]) : 0;
    }
    for (int ks = wk; ks < KS; ks += KW) {         // the row's pieces, as the instructions take them
      uint32_t a[3][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float4 v = f32_up(pos[i] >= 0 ? *reinterpret_cast<const float4*>(q + ((size_t)(t0 + wr * 16 + g + i * 8) * nh + h) * HD + ks * 16 + t * 4)
                                            : make_float4(0.f, 0.f, 0.f, 0.f));
        f32_split3(v.x, v.y, a[0][i], a[1][i], a[2][i]);
        f32_split3(v.z, v.w, a[0][i + 2], a[1][i + 2], a[2][i + 2]);
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) s_q[((wr * KS + ks) * 3 + p) * 32 + lane] = make_uint4(a[p][0], a[p][1], a[p][2], a[p][3]);
    }
    float acc[NB][4][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    bool bad[2] = {false, false};
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[b][j][0] = acc[b][j][1] = acc[b][j][2] = acc[b][j][3] = 0.f;
    int stage = 0;
    for (int jb = jb0; jb <= jhi; jb += KEYS, stage ^= 1) {
      if (jb + KEYS <= jhi) load(jb + KEYS, stage ^ 1);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      __syncthreads();
      const float* ks_ = f32_smem + stage * STAGE + (wk * 16 + g) * SK + t * 4;
      const float* vs_ = f32_smem + stage * STAGE + KEYS * SK + (wk * 16 + 2 * t) * SV + g * 4;
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 2
      for (int ks = 0; ks < KS; ++ks) {
        uint32_t a[3][4], b[2][3][2];
        float c[2][4], d[2][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          const uint4 v = s_q[((wr * KS + ks) * 3 + p) * 32 + lane];
          a[p][0] = v.x; a[p][1] = v.y; a[p][2] = v.z; a[p][3] = v.w;
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float4 v = f32_up(*reinterpret_cast<const float4*>(ks_ + n * 8 * SK + ks * 16));
          f32_split3(v.x, v.y, b[n][0][0], b[n][1][0], b[n][2][0]);
          f32_split3(v.z, v.w, b[n][0][1], b[n][1][1], b[n][2][1]);
        }
        f32_products<2>(c, d, a, b);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int x = 0; x < 4; ++x) s[n][x] += c[n][x] + d[n][x];
      }
      float corr[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float mx = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = jb + wk * 16 + n * 8 + 2 * t + e;
            float v = s[n][i * 2 + e] * F32_DOWN * scale;
            const bool valid = j <= pos[i] && j >= lo[i];
            if (valid && !isfinite(v)) bad[i] = true;
            if (softcap > 0.f) v = f32_capped(v, softcap);
            v = valid && isfinite(v) ? v : -INFINITY;
            s[n][i * 2 + e] = v;
            mx = fmaxf(mx, v);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float m_new = fmaxf(m[i], mx);
        corr[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
        m[i] = m_new;
        l[i] *= corr[i];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float v = s[n][i * 2 + e], p = v == -INFINITY ? 0.f : expf(v - m_new);
            s[n][i * 2 + e] = p;
            l[i] += p;
          }
      }
      uint32_t pa[3][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) f32_split3(s[n][i * 2] * F32_UP, s[n][i * 2 + 1] * F32_UP, pa[0][n * 2 + i], pa[1][n * 2 + i], pa[2][n * 2 + i]);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float4 v[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) v[r] = f32_up(*reinterpret_cast<const float4*>(vs_ + ((r & 1) + (r >> 1) * 8) * SV + b * 32));
        uint32_t w[4][3][2];
        float c[4][4], d[4][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float4 x = v[2 * r], y = v[2 * r + 1];
          f32_split3(x.x, y.x, w[0][0][r], w[0][1][r], w[0][2][r]);
          f32_split3(x.y, y.y, w[1][0][r], w[1][1][r], w[1][2][r]);
          f32_split3(x.z, y.z, w[2][0][r], w[2][1][r], w[2][2][r]);
          f32_split3(x.w, y.w, w[3][0][r], w[3][1][r], w[3][2][r]);
        }
        f32_products<4>(c, d, pa, w);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[b][j][x] = fmaf(acc[b][j][x], corr[x >> 1], c[j][x] + d[j][x]);
      }
      __syncthreads();                            // the stage has been read
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");      // (a run of rows that see no key has one on its way)
    __syncthreads();
    // the parts of the keys: every warp's results to shared memory, then all threads add them up
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = wr * 16 + g + i * 8;
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
      l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
      const unsigned any = __ballot_sync(0xffffffffu, bad[i]);
      if (t == 0) { s_m[wk][row] = m[i]; s_l[wk][row] = l[i]; s_bad[wk][row] = (any >> (g * 4)) & 15u; }
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<float4*>(f32_smem + (wk * 32 + row) * SV + b * 32 + t * 8 + e * 4) =
              make_float4(acc[b][0][i * 2 + e], acc[b][1][i * 2 + e], acc[b][2][i * 2 + e], acc[b][3][i * 2 + e]);
    }
    __syncthreads();
    const float* sink = sinks ? sinks + h : nullptr;
    if (tid < 32) {                               // what each part counts
      float mx = sink ? *sink : -INFINITY, f[KW], sum = 0.f;
#pragma unroll
      for (int w = 0; w < KW; ++w) mx = fmaxf(mx, s_m[w][tid]);
#pragma unroll
      for (int w = 0; w < KW; ++w) {
        f[w] = s_m[w][tid] == -INFINITY ? 0.f : expf(s_m[w][tid] - mx);
        sum = fmaf(s_l[w][tid], f[w], sum);
        if (w > 0) s_bad[0][tid] |= s_bad[w][tid];
      }
      if (sink) sum += expf(*sink - mx);
#pragma unroll
      for (int w = 0; w < KW; ++w) s_m[w][tid] = f[w];
      s_l[0][tid] = sum;
    }
    __syncthreads();
    constexpr int RT = HD / 4;                    // threads a row
    for (int idx = tid; idx < 32 * RT; idx += THREADS) {
      const int r = idx / RT, c = idx % RT * 4;
      const float* src = f32_smem + r * SV + c;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < KW; ++w) {
        const float4 x = *reinterpret_cast<const float4*>(src + w * 32 * SV);
        const float f = s_m[w][r];
        v.x = fmaf(x.x, f, v.x); v.y = fmaf(x.y, f, v.y); v.z = fmaf(x.z, f, v.z); v.w = fmaf(x.w, f, v.w);
      }
      const float sum = s_l[0][r];
      v.x = v.x / sum * F32_DOWN; v.y = v.y / sum * F32_DOWN; v.z = v.z / sum * F32_DOWN; v.w = v.w / sum * F32_DOWN;
      if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w))) s_bad[0][r] = 1;
      if (r >= first && r < end) {
        float* o = out + (size_t)(t0 + r) * out_stride + (size_t)h * HD + c;
        o[0] = v.x * out_scale; o[1] = v.y * out_scale; o[2] = v.z * out_scale; o[3] = v.w * out_scale;
      }
    }
    __syncthreads();
    for (int r = warp; r < 32; r += THREADS / 32)
      if (r >= first && r < end && s_bad[0][r]) {
        const int p_r = positions[t0 + r];
        attn_f32_row<HD>(q + ((size_t)(t0 + r) * nh + h) * HD, k_pages, v_pages, out + (size_t)(t0 + r) * out_stride + (size_t)h * HD, bt, nkv, kvh,
                         low(p_r), p_r, scale, softcap, sink, out_scale, lane);
      }
    __syncthreads();                              // the parts have been read, before the next sequence's keys
    first = end;
  }
}

// How many neighbouring tokens a block takes, and how many blocks share the keys.  Few tokens: one a block, and the keys shared by up
// to eight blocks.  Tokens enough for every SM: as many neighbours a block as fit its rows (a cluster's blocks finish ONE token).
struct AttnF32Plan { int tpb, cluster; };
static AttnF32Plan attn_f32_plan(int R, int n_tokens, int nh, int nkv, int maxp, int sms) {
  const int G = nh / nkv, hg = (G + R - 1) / R;
  AttnF32Plan p = {1, 1};
  const long long blocks = (long long)nkv * hg * n_tokens;
  while (p.cluster < 8 && blocks * p.cluster < sms && maxp >= 2 * p.cluster) p.cluster *= 2;
  if (p.cluster == 1 && G < R && R % G == 0 && blocks >= (long long)sms * (R / G)) p.tpb = R / G;
  return p;
}
// (rows a block: two query heads a kv head or fewer, two; else four)
static int attn_f32_rows(int nh, int nkv) { return nh / nkv <= 2 ? 2 : 4; }
extern "C" void sx_attn_f32_plan(int n_tokens, int nh, int nkv, int maxp, int sms, int* out2) {
  const AttnF32Plan p = attn_f32_plan(attn_f32_rows(nh, nkv), n_tokens, nh, nkv, maxp, sms);
  out2[0] = p.tpb; out2[1] = p.cluster;
}

// Tiles of 32 rows where a sequence brings 16 tokens and more on average and there are tiles for a third of the SMs, more where a tile
// has several sequences, which it walks through one after the other (us, the kernel of eight lanes a key first; 16 heads of 128: 33
// tokens 7.6 and 11.4, 65 14.9 and 14.5, 129 30.5 and 18.5, 300 95 and 29, 4 x 16 12.4 and 20.3, 16 x 16 41 and 21; 16 of 64: 65 8.5
// and 9.1, 96 12.7 and 10.7; 32 of 64: 4 x 16 behind 500 47 and 54; 32 of 128: 64 23 and 12, 8 x 16 34 and 21, 2,048 4,246 and 1,095).
static bool attn_f32_tiles(int n_tokens, int n_seqs, int nh, int sms) {
  const long long per_seq = n_seqs > 0 ? n_tokens / n_seqs : 0, blocks = (n_tokens + 31LL) / 32 * nh;
  return per_seq >= 16 && blocks * (per_seq < 32 ? per_seq : 32) >= 32LL * sms / 3;
}

// How a step of several sequences is dealt out.  A tile costs a sequence's pages, for one row as for 32, so sequences of fewer than
// `few` tokens go to the kernel of eight lanes a key, whatever the others bring; `from` .. `to`: the tokens among which they are.
// Where the sequences' lengths are known (`cu`: first tokens and the number of all, `past`: keys held before; host memory, or null),
// `few` is the one of 6, 17 and 33 that is the fastest by what the kernels take, us: a tile 3 + 4.4 a page of each of its sequences, a
// block an SM; a block of R rows of the other kernel 1.6 + 0.0098 R a key, by all SMs; 4 for the second launch.  Else it is 6.  Measured
// (16 heads of 128 over 8, us; kernel of eight lanes for all, tiles for all, this): 500 tokens and 20 of one behind 1,000 262, 898, 111;
// 500 and 8 behind 8,000 373, 589, 151; 300 and 8 x 8 behind 4,000 430, 1,353, 374; 512 and 32 x 8 behind 500 408, 185, 189.  A
// call that does not know the lengths pays the second launch where it has several sequences: 4 x 64 tokens 48, 12, 24.
struct AttnF32Mix { int tiles, few, from, to; };
static AttnF32Mix attn_f32_mix(const int* cu, const int* past, int n_tokens, int n_seqs, int nh, int nkv, int R, int sms) {
  AttnF32Mix best = {attn_f32_tiles(n_tokens, n_seqs, nh, sms), n_seqs > 1 ? 6 : 0, 0, n_seqs > 1 ? n_tokens : 0};
  if (n_seqs <= 1 || !cu || !past || cu[0] != 0 || cu[n_seqs] != n_tokens) return best;
  for (int i = 0; i < n_seqs; ++i)
    if (cu[i + 1] < cu[i]) return best;
  const double row_blocks = (double)nkv * ((nh / nkv + R - 1) / R);
  const int choices[3] = {6, 17, 33};
  double best_us = -1.0;
  for (int few : choices) {
    AttnF32Mix m = {0, few, 0, 0};
    int tokens = n_tokens, seqs = n_seqs, tile = -1;
    double here = 0.0, longest = 0.0, all = 0.0, row = 0.0, rows = 0.0;
    for (int i = 0; i < n_seqs; ++i) {
      const int n = cu[i + 1] - cu[i];
      if (n < few) {
        if (m.to == 0) m.from = cu[i];
        m.to = cu[i + 1];
        tokens -= n;
        --seqs;
        const double us = 1.6 + 0.0098 * R * (past[i] + n);
        row = us > row ? us : row;
        rows += n * row_blocks * us;
        continue;
      }
      for (int at = cu[i]; at < cu[i + 1]; at = (at / 32 + 1) * 32) {
        const int end = cu[i + 1] < (at / 32 + 1) * 32 ? cu[i + 1] : (at / 32 + 1) * 32;
        const double us = 3.0 + 4.4 * ((past[i] + end - cu[i] + 63) / 64);
        here = at / 32 == tile ? here + us : us;
        tile = at / 32;
        longest = here > longest ? here : longest;
        all += us * nh;
      }
    }
    m.tiles = attn_f32_tiles(tokens, seqs, nh, sms);
    if (!m.tiles) continue;                        // (then the one kernel takes all, or fewer go to it)
    double us = all / sms > longest ? all / sms : longest;
    if (m.to > m.from) us += 4.0 + (rows / sms > row ? rows / sms : row);
    else m.few = 0;
    if (best_us < 0.0 || us < best_us) { best = m; best_us = us; }
  }
  if (best_us < 0.0) best.tiles = 0;
  return best;
}
extern "C" void sx_attn_f32_mix(const int* cu, const int* past, int n_tokens, int n_seqs, int nh, int nkv, int sms, int* out4) {
  const AttnF32Mix m = attn_f32_mix(cu, past, n_tokens, n_seqs, nh, nkv, attn_f32_rows(nh, nkv), sms);
  out4[0] = m.tiles; out4[1] = m.few; out4[2] = m.from; out4[3] = m.to;
}

template <int HD>
static int attn_f32_tile_launch(const float* q, const float* k, const float* v, float* out, const int* positions, const int* seq_of_token,
                                const int* block_table, int maxp, int n_tokens, int nh, int nkv, float scale, int window, float softcap,
                                const float* sinks, int chunk, int out_stride, float out_scale, int few, cudaStream_t stream) {
  constexpr int KW = 4;
  const size_t smem = (size_t)2 * 16 * KW * (2 * HD + 20) * 4 + (size_t)2 * (HD / 16) * 3 * 32 * 16;
  cudaError_t e = cudaFuncSetAttribute(attn_f32_tile_kernel<HD, KW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return sx_launch(attn_f32_tile_kernel<HD, KW>, dim3((unsigned)nh, (unsigned)((n_tokens + 31) / 32)), dim3(64 * KW), smem, stream, q, k, v, out, positions,
                   seq_of_token, block_table, maxp, n_tokens, nh, nkv, scale, window, softcap, sinks, chunk, out_stride, out_scale, few);
}

template <int HD, int R>
static int attn_f32_launch(const float* q, const float* k, const float* v, float* out, const int* positions, const int* seq_of_token,
                           const int* block_table, int maxp, int begin, int end, int few, int nh, int nkv, float scale, int window, float softcap,
                           const float* sinks, int chunk, int out_stride, float out_scale, cudaStream_t stream) {
  const int G = nh / nkv, hg = (G + R - 1) / R;
  const AttnF32Plan plan = attn_f32_plan(R, end - begin, nh, nkv, maxp, sx_sm_count());
  const int tpb = plan.tpb, cluster = plan.cluster;
  const dim3 grid((unsigned)cluster, (unsigned)(nkv * hg), (unsigned)((end - begin + tpb - 1) / tpb));
  if (cluster > 1)
    return sx_launch_cluster(attn_f32_kernel<HD, R>, grid, dim3(256), 0, stream, cluster, q, k, v, out, positions, seq_of_token, block_table,
                             maxp, end, nh, nkv, scale, window, softcap, sinks, chunk, out_stride, out_scale, tpb, cluster, begin, few);
  return sx_launch(attn_f32_kernel<HD, R>, grid, dim3(256), 0, stream, q, k, v, out, positions, seq_of_token, block_table, maxp,
                   end, nh, nkv, scale, window, softcap, sinks, chunk, out_stride, out_scale, tpb, 1, begin, few);
}

static int attn_generic_any(const void* q, const void* k_pages, const void* v_pages, void* out,
                            const int* positions, const int* seq_of_token, const int* block_table,
                            int maxp, int n_tokens, int nh, int nkv, int hd, float scale, int window,
                            int dt, int vd, float softcap, const float* sinks, int chunk, int out_stride, float out_scale,
                            int n_seqs, const int* cu, const int* past, int* launched, cudaStream_t stream) {
  *launched = 1;
  if (n_tokens <= 0) return 0;
  if (hd <= 0 || hd > 512 || vd <= 0 || vd > 512 || nkv <= 0 || nh % nkv != 0 || nh > 65535 || out_stride < nh * vd)
    return SX_ERR_SIZE;
  if (dt == SX_F32 && hd == vd && (hd == 64 || hd == 128) && n_tokens <= 65535 && nkv <= 8191 &&
      (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0) {
    const AttnF32Mix mix = attn_f32_mix(cu, past, n_tokens, n_seqs, nh, nkv, attn_f32_rows(nh, nkv), sx_sm_count());
    int begin = 0, end = n_tokens;
    if (mix.tiles) {
#define ATTN_F32_TILES(HD) attn_f32_tile_launch<HD>((const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, positions, \
                                                    seq_of_token, block_table, maxp, n_tokens, nh, nkv, scale, window, softcap, sinks,  \
                                                    chunk, out_stride, out_scale, mix.few, stream)
      const int rc = hd == 64 ? ATTN_F32_TILES(64) : ATTN_F32_TILES(128);
#undef ATTN_F32_TILES
      if (rc || mix.to <= mix.from) return rc;
      begin = mix.from;
      end = mix.to;
      *launched = 2;
    }
#define ATTN_F32(HD, R) attn_f32_launch<HD, R>((const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, positions, \
                                               seq_of_token, block_table, maxp, begin, end, mix.tiles ? mix.few : 0, nh, nkv, scale, window, softcap, \
                                               sinks, chunk, out_stride, out_scale, stream)
    if (attn_f32_rows(nh, nkv) == 2) return hd == 64 ? ATTN_F32(64, 2) : ATTN_F32(128, 2);
    return hd == 64 ? ATTN_F32(64, 4) : ATTN_F32(128, 4);
#undef ATTN_F32
  }
  dim3 grid(n_tokens, nh);
  const size_t smem = (size_t)(hd + 128) * sizeof(float);
  if (dt == SX_F32)
    attn_generic_kernel<float><<<grid, 128, smem, stream>>>(
        (const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, positions, seq_of_token,
        block_table, maxp, nh, nkv, hd, scale, window, vd, softcap, sinks, chunk, out_stride, out_scale);
  else if (dt == SX_BF16)
    attn_generic_kernel<bf16><<<grid, 128, smem, stream>>>(
        (const bf16*)q, (const bf16*)k_pages, (const bf16*)v_pages, (bf16*)out, positions, seq_of_token,
        block_table, maxp, nh, nkv, hd, scale, window, vd, softcap, sinks, chunk, out_stride, out_scale);
  else
    return SX_ERR_DTYPE;
  return sx_launch_status();
}

extern "C" int sx_attn_generic(const void* q, const void* k_pages, const void* v_pages, void* out,
                               const int* positions, const int* seq_of_token, const int* block_table,
                               int maxp, int n_tokens, int nh, int nkv, int hd, float scale, int window,
                               int dt, cudaStream_t stream) {
  int launched;
  return attn_generic_any(q, k_pages, v_pages, out, positions, seq_of_token, block_table, maxp, n_tokens, nh, nkv, hd, scale,
                          window, dt, hd, 0.f, nullptr, 0, nh * hd, 1.f, n_tokens, nullptr, nullptr, &launched, stream);
}

// with the options the plain entry point leaves out (see the kernel's comment), how many sequences the tokens are of (at most: rows of
// the block table), and in host memory, or null, the first token of each and the number of all, and the keys each had before; launched: how
// many kernels it was
extern "C" int sx_attn_generic_ex(const void* q, const void* k_pages, const void* v_pages, void* out,
                                  const int* positions, const int* seq_of_token, const int* block_table,
                                  int maxp, int n_tokens, int nh, int nkv, int hd, float scale, int window,
                                  int dt, int vd, float softcap, const float* sinks, int chunk, int out_stride,
                                  float out_scale, int n_seqs, const int* cu, const int* past, int* launched, cudaStream_t stream) {
  return attn_generic_any(q, k_pages, v_pages, out, positions, seq_of_token, block_table, maxp, n_tokens, nh, nkv, hd, scale,
                          window, dt, vd, softcap, sinks, chunk, out_stride, out_scale, n_seqs, cu, past, launched, stream);
}

// ---------------------------------------------------------------------------------------
// out[t, i] = silu(gu[t, i]) * gu[t, I + i],  silu(x) = x / (1 + exp(-x)), in 32-bit
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void silu_mul_kernel(const T* __restrict__ gu, T* __restrict__ out, int I, size_t n) {
  pdl_wait();
  pdl_trigger();
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const size_t t = idx / I;
  const int i = (int)(idx - t * I);
  const float g = to_f32(gu[t * 2 * I + i]);
  const float u = to_f32(gu[t * 2 * I + I + i]);
  out[idx] = from_f32<T>(g / (1.f + expf(-g)) * u);
}

extern "C" int sx_silu_mul(const void* gu, void* out, int n_tokens, int I, int dt, cudaStream_t stream) {
  const size_t n = (size_t)n_tokens * I;
  if (n == 0) return 0;
  const unsigned grid = (unsigned)((n + 255) / 256);
  if (dt == SX_F32) return sx_launch(silu_mul_kernel<float>, dim3(grid), dim3(256), 0, stream, (const float*)gu, (float*)out, I, n);
  if (dt == SX_BF16) return sx_launch(silu_mul_kernel<bf16>, dim3(grid), dim3(256), 0, stream, (const bf16*)gu, (bf16*)out, I, n);
  return SX_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------
// Decoding that stays on the device.  Before a step: a row whose control word is not negative
// runs that token instead of the one sampled for it in the step before (and its history of
// tokens, if kept for the penalties, ends with that token).  After a step: every live row
// (advance_by = 1) takes its sampled token as the next input, appends it to its history, and
// moves one position and one word of its random stream on; rows that pad the batch stay put.
// ---------------------------------------------------------------------------------------
__global__ void decode_begin_kernel(int* __restrict__ token_ids, const int* __restrict__ control,
                                    int* __restrict__ history, const int* __restrict__ hist_len, int hist_cap, int S) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S) return;
  const int t = control[i];
  if (t < 0) return;
  token_ids[i] = t;
  if (history != nullptr) {
    const int n = hist_len[i];
    if (n > 0 && n <= hist_cap) history[(size_t)i * hist_cap + n - 1] = t;
  }
}
extern "C" int sx_decode_begin(int* token_ids, const int* control, int* history, const int* hist_len, int hist_cap,
                               int S, cudaStream_t stream) {
  if (S <= 0) return 0;
  return sx_launch(decode_begin_kernel, dim3((S + 127) / 128), dim3(128), 0, stream, token_ids, control, history,
                   hist_len, hist_cap, S);
}

__global__ void decode_advance_kernel(int* __restrict__ token_ids, const int* __restrict__ sampled,
                                      int* __restrict__ positions, int* __restrict__ seq_past,
                                      int* __restrict__ seq_lens, int* __restrict__ rng_step,
                                      const int* __restrict__ advance_by, int* __restrict__ history,
                                      int* __restrict__ hist_len, int hist_cap, int S) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S) return;
  const int by = advance_by != nullptr ? advance_by[i] : 1;
  if (by == 0) return;
  const int t = sampled[i];
  token_ids[i] = t;
  positions[i] += 1;
  seq_past[i] += 1;
  seq_lens[i] += 1;
  if (rng_step != nullptr) rng_step[i] += 1;
  if (history != nullptr) {
    const int n = hist_len[i];
    if (n < hist_cap) {
      history[(size_t)i * hist_cap + n] = t;
      hist_len[i] = n + 1;
    }
  }
}
extern "C" int sx_decode_advance(int* token_ids, const int* sampled, int* positions, int* seq_past, int* seq_lens,
                                 int* rng_step, const int* advance_by, int* history, int* hist_len, int hist_cap,
                                 int S, cudaStream_t stream) {
  if (S <= 0) return 0;
  return sx_launch(decode_advance_kernel, dim3((S + 127) / 128), dim3(128), 0, stream, token_ids, sampled, positions,
                   seq_past, seq_lens, rng_step, advance_by, history, hist_len, hist_cap, S);
}
