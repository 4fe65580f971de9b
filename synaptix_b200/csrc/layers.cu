// All layers of a dense decoder in ONE kernel, for single-token steps of one or two rows in bfloat16.
//
// A layer is  h += Wo attention(norm1(h) Wqkv);  h += Wdown(silu(g) * u),  [g; u] = norm2(h) Wgu,  with per-head RMSNorm of q and k,
// rotate-half rotation and a paged cache: products of a few rows, bound by reading the weights once.  As kernels of their
// own they stream at 3.4 to 5.4 TB/s and pay 1.5 to 3 us at each of their five boundaries, because nothing is on its way
// from HBM while one kernel ends and the next begins.  Here
//   * one block an SM (a cooperative launch) stays for all layers.  Two producer warps walk the SM's share of ALL matrices and of
//     the cached keys and values in the order of their use and keep a ring of some 33 KB stages filled, whatever the other warps
//     wait for: while a layer's parts exchange their results, the next 130 to 165 KB an SM arrive;
//   * rows of a matrix are dealt out evenly in pairs (16 or 18 of 2,560 an SM), in groups of up to 16 that are the M side of
//     mma.sync.m16n8k16; the 8 compute warps share K (chunks of 1,024: 128 a warp).  Four other warps add their parts up, so that the
//     compute warps go on with the next group;
//   * what one product hands to the next goes through L2 as 8-byte words of two bfloat16 values (or one float) and a tag that
//     is new in every layer and launch.  A word is valid when its tag is; the reader polls the words it needs.  No barrier
//     over the grid, no fence, no flag behind the data: one store and one load latency an exchange.  A word is
//     overwritten a layer later, by a block that has read what its readers made of it.  Words that every block reads exist in 4
//     copies, so that fewer blocks poll one line;
//   * the residual stream never leaves the SM that owns its columns (shared memory, float32): o and down own the same columns.
//     The norms are split as elsewhere: x = bf16(h * gain) and a partial sum of squares go out, the reader multiplies its
//     results by the rows' factors;
//   * attention: a block per (sequence, kv head, share of the pages); a warp takes 16 keys at a time, K and V come
//     through the same ring (TMA, 128-byte swizzle); shares are merged by their blocks through the same tagged words.
// Measured (ms a step with head and sampling, five kernels a layer -> this; one row): 0.6B, 28 layers, 200 keys 0.65 -> 0.56, 1,500
// keys 0.67 -> 0.59; 1.7B 1.00 -> 0.83, 1.01 -> 0.85; 4B, 36 layers 1.90 -> 1.64, 1.94 -> 1.72 (7.5 GB in 1.58, 4.75 TB/s); 8B 3.18 ->
// 2.60, 3.19 -> 2.69.  Two rows: 0.69 -> 0.59, 1.11 -> 0.90, 1.96 -> 1.76, 2.98 -> 2.74 at 200 keys; 7,000 keys 0.94 -> 0.82, 1.34 -> 1.16,
// 2.26 -> 2.09, 3.30 -> 3.07.  Models of two or four layers 1 to 10 % shorter.  What is left: 11 to 12 us a layer beyond its bytes, at 0.6B
// as at 4B: the parts' exchanges (1 us from the last store to the last reader, six times) and attention's few blocks, beyond what the ring holds.
// What the warps of a block run is kept small (loops not unrolled, every part of the code in one place): a layer walks through all
// of it once, and code that does not fit the instruction cache (32 KB) is fetched again in every layer:
// the first form, 104 KB of code, took 0.78 ms a step where 52 KB took 0.64 (0.6B, 30 keys).  And warps wait suspended (mbarrier.try_wait, named barriers) where they can:
// another polling warp beside the others cost 5 to 20 %.
//
// Every wait is bounded: a wait that runs out sets the library's status word and lets all later waits of the block pass, so
// that the block walks to its end (its barriers included) without waiting, its copies in flight being waited for first.
//
// The reference replays a graph of separate kernels here (crates/synaptix-models/llm/common/src/model.rs:1489-1549).
#include "tcgen05.cuh"

#define LY_WARPS 8                        // compute warps
#define LY_EPI 4                          // warps that add up the compute warps' results and hand them on
#define LY_PRODUCERS 2
#define LY_THREADS ((LY_WARPS + LY_EPI + LY_PRODUCERS) * 32)
#define LY_KC 1024                        // values of a row a chunk: 128 for each compute warp
#define LY_ROW (LY_KC * 2 + 64)           // a row's place in a stage: 64 bytes on, so that 8 lanes' 16-byte loads (2 rows x 4) meet no bank twice
#define LY_STAGE (16 * LY_ROW)            // a multiple of 1,024: the swizzle's period (keys and values)
#define LY_MAX_STAGES 6
#define LY_MIN_STAGES 3
#define LY_MAX_T 2                        // rows (tokens) of a step
#define LY_COPIES 4                       // copies of the words that every block reads: what the lanes of columns without a token can write beside the words themselves
#define LY_MAX_LAYERS 64
#define LY_MAX_G 4                        // query heads a kv head
#define LY_HD 128
#define LY_MAX_COLS 64                    // columns of the residual stream an SM owns at most
#define LY_MAX_SPLITS 32
#define LY_SPIN (1u << 21)                // looks at words of another block (half a microsecond each), at a barrier of this one
#define LY_SPIN_BAR (1u << 20)             // (a look at a barrier suspends the warp for up to LY_NAP ns: spinning warps slow the others down)
#define LY_NAP 2000
#define SX_ERR_NO_ROOM 10006

struct LyLayer {
  const bf16* w[4];                       // q/k/v, o, gate and up, down
  const float* gain[2];                   // norm1, norm2
  const float* qn;                        // gains of the heads' norms, or null
  const float* kn;
  long long kv_row0;                      // the layer's first row in the cache seen as rows of 128 values
};

// Product p of a layer: 0 q/k/v, 1 o, 2 gate and up, 3 down.  in[p]: the exchange it reads, `in_row` words a token, `in_copy` words
// between copies; out[p]: the one it writes.
struct LyArgs {
  const LyLayer* layers;
  int n_layers, T, W, nh, nkv, G, ff, K[4];
  float eps, qk_eps, scale_log2;
  const float* h_in;
  float* h_out;
  const int* seq_lens;
  const int* block_table;
  int maxp, n_pages, max_splits;
  const float* inv_freq;
  bf16* kc;
  bf16* vc;
  unsigned long long* words;              // [0]: the launch's number; then the exchanges
  int in[4], in_copy[4], out[4], out_copy[4], out_row[4], sums[2];
  int part, part_words, s_copy;          // shares of attention
  int stages, xs_bytes, pass;             // the ring's depth; room for activations; how many values of a row fit it (a multiple of LY_KC)
  int* status;
};

struct LyProduct { int row0, rows; };
// a block's share of attention: pages `first` .. of a sequence, in `stages` stages; own: the token's place in a layer's cache rows (-1: in another share)
struct LyItem { int has, seq, kvh, split, splits, len, first, stages, merge0, merge1, log_w, words; long long own; };

struct LyShared {                         // behind the ring, the activations and the 8 KB of partial sums
  LyLayer layers[LY_MAX_LAYERS];
  LyProduct prod[4];
  LyItem item;
  alignas(16) bf16 q[LY_MAX_G * LY_HD];          // (read 16 bytes at a time)
  alignas(16) bf16 kv[2 * LY_HD];
  float cs[LY_HD / 2], sn[LY_HD / 2];
  float h[LY_MAX_COLS][LY_MAX_T];
  float carry[LY_MAX_COLS][LY_MAX_T];
  alignas(16) float top[LY_MAX_G][LY_WARPS];      // the warps' maxima and sums of a head
  float sum[LY_MAX_G][LY_WARPS];
  float ssq[(LY_MAX_COLS / 16) * 4][LY_MAX_T];
  float factor[2][LY_MAX_T];
  uint64_t full[LY_MAX_STAGES], empty[LY_MAX_STAGES];
  int dead;
};
#define LY_RED (2 * LY_WARPS * 128 * 4)
#define LY_FIXED (LY_RED + (int)sizeof(LyShared))
#define LY_SMEM_MAX (227 * 1024)

// ---- words ----------------------------------------------------------------------------------------------------------
typedef unsigned long long ly_word;
__device__ __forceinline__ ly_word ly_ld(const ly_word* p) {
  ly_word v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// two words; each is whole by itself
__device__ __forceinline__ void ly_ld2(const ly_word* p, ly_word& a, ly_word& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ ly_word ly_make(uint32_t value, uint32_t tag) { return ((ly_word)tag << 32) | value; }
__device__ __forceinline__ void ly_st(ly_word* p, uint32_t value, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;\n" ::"l"(p), "l"(ly_make(value, tag)) : "memory");
}
__device__ __forceinline__ void ly_st2(ly_word* p, float a, float b, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};\n"
               ::"l"(p), "l"(ly_make(__float_as_uint(a), tag)), "l"(ly_make(__float_as_uint(b), tag)) : "memory");
}
__device__ __forceinline__ bool ly_is(ly_word v, uint32_t tag) { return (uint32_t)(v >> 32) == tag; }
__device__ __forceinline__ float ly_f(ly_word v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ uint32_t ly_pack(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Poll until `once` is true for the whole warp.  `dead` (shared): a wait of this block ran out, nothing is waited for any more.
template <class F>
__device__ __forceinline__ void ly_poll(F once, volatile int* dead, int* status, int code, uint32_t limit = LY_SPIN) {
  uint32_t i = 0;
  while (!__all_sync(0xffffffffu, once())) {
    if (__any_sync(0xffffffffu, *dead != 0)) break;
    if (++i == limit) {
      *dead = 1;
      *(volatile int*)status = code;
    }
  }
}
__device__ __forceinline__ bool ly_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok) : "r"(bar), "r"(parity), "r"(LY_NAP) : "memory");
  return ok;
}
__device__ __forceinline__ void ly_bar_wait(uint32_t bar, uint32_t parity, volatile int* dead, int* status, int code) {
  ly_poll([&] { return ly_test(bar, parity); }, dead, status, code, LY_SPIN_BAR);
}
__device__ __forceinline__ void ly_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ly_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(LY_WARPS * 32) : "memory"); }      // the compute warps
// Partial sums go from the compute warps to the epilogue warps through two buffers in turn: barriers 2 and 3 say that one is
// full, 4 and 5 that it is free.  All of these warps walk the same groups in the same order, whatever their waits come to.
#define LY_BOTH ((LY_WARPS + LY_EPI) * 32)
__device__ __forceinline__ void ly_meet(int id) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "n"(LY_BOTH) : "memory"); }
__device__ __forceinline__ void ly_tell(int id) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "n"(LY_BOTH) : "memory"); }
// 7: the block's own part of an exchange has been handed on (the others' will not be there much sooner), 6: among the epilogue warps
__device__ __forceinline__ void ly_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void ly_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ly_lds(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ly_lds_or_0(uint32_t a, bool on) {       // (lanes that do not load cost shared memory nothing)
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n @p ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n}\n"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w) : "r"(a), "r"((uint32_t)on) : "memory");
  return v;
}
__device__ __forceinline__ void ly_ldsm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ly_ldsm_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ float ly_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// ---- who does what --------------------------------------------------------------------------------------------------
// the share of block `i` of `n` (even) columns, in pairs
__device__ __forceinline__ int ly_lo(int n, int i, int blocks) { return 2 * (int)((unsigned)(n >> 1) * (unsigned)i / (unsigned)blocks); }

// A product as one block sees it: `rows` rows of the matrix from `row0` on (gate and up: `rows / 2` columns of either from column
// `row0` on, a gate row and an up row in turn).  They go in groups of up to 16 rows; of small groups a stage holds several chunks.
__device__ __forceinline__ int ly_chunks(int R) { return R > 8 ? 1 : R > 4 ? 2 : R > 2 ? 4 : 8; }

// Up to 4 pages of keys are one block's (256 keys: two rounds of the 8 warps); more are dealt out among the blocks there are for a
// (sequence, kv head).
__device__ __forceinline__ void ly_item(const LyArgs& A, LyItem& t, int i) {
  const int pair = i / A.max_splits;
  t.split = i - pair * A.max_splits;
  t.seq = pair / A.nkv;
  t.kvh = pair - t.seq * A.nkv;
  t.has = t.seq < A.T;
  if (!t.has) return;
  t.len = max(A.seq_lens[t.seq], 1);
  const int all = min((t.len + 63) >> 6, A.maxp);
  t.splits = all <= 4 ? 1 : min(A.max_splits, all);
  const int per = (all + t.splits - 1) / t.splits;
  t.splits = (all + per - 1) / per;
  t.first = t.split * per;
  t.stages = min(per, all - t.first);
  t.has = t.split < t.splits;
  // its part of the pair's outputs (pairs of values) when the shares are merged, a lane a share
  const int total = A.G * (LY_HD / 2), each = (total + t.splits - 1) / t.splits;
  t.merge0 = min(total, t.split * each);
  t.merge1 = min(total, t.merge0 + each);
  t.log_w = 1;
  while ((1 << t.log_w) < t.splits) ++t.log_w;
  t.words = (t.seq * A.nh + t.kvh * A.G) * (LY_HD / 2);        // its heads' place among a step's
  t.own = -1;
  if (t.has && t.first + t.stages == all) {
    const int pos = t.len - 1, page = A.block_table[(size_t)t.seq * A.maxp + (all - 1)];
    if (page >= 0 && page < A.n_pages) t.own = ((long long)page * A.nkv + t.kvh) * SX_PAGE + (pos & 63);
  }
}

// ---- producers ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ly_produce(const LyArgs& A, const CUtensorMap* mk, const CUtensorMap* mv, LyShared* sh, uint32_t ring) {
  const int lane = threadIdx.x & 31, who = (threadIdx.x >> 5) - LY_WARPS - LY_EPI;
  const bool leader = tc_elect_one();
  const uint32_t bars = tc_smem(sh->full);
  volatile int* dead = &sh->dead;
  const int* bt = A.block_table + (size_t)(sh->item.has ? sh->item.seq : 0) * A.maxp;
  const int kv = sh->item.has ? sh->item.stages : 0;
  int st = 0, use = 0, turn = 0;                        // the stage, how often it was used before, whose turn it is to fill it
  int pages = 0, page0 = -1;                            // lane i: the page page0 + i of the item's
  bool ok = true;
  auto next = [&](uint32_t bytes) {                     // this warp's turn: a free stage, which will receive `bytes`
    if (use > 0) ly_bar_wait(bars + (LY_MAX_STAGES + st) * 8, (use - 1) & 1, dead, A.status, 1);
    ok = !__any_sync(0xffffffffu, *dead != 0);
    if (ok && leader) tc_mbar_expect_tx(bars + st * 8, bytes);
    __syncwarp();
  };
  auto advance = [&] {
    if (++st == A.stages) { st = 0; ++use; }
    turn ^= 1;
  };
#pragma unroll 1
  for (int step = 0; ok && step < 4 * A.n_layers; ++step) {
    const int p = step & 3;
    const LyLayer* L = &sh->layers[step >> 2];
#pragma unroll 1
    for (int t = 0; ok && p == 1 && t < kv; ++t, advance()) {
      if (turn != who) continue;
      const int pg = sh->item.first + t;
      if ((pg & ~31) != page0) {
        page0 = pg & ~31;
        pages = page0 + lane < A.maxp ? bt[page0 + lane] : 0;
      }
      const int page = min(max(__shfl_sync(0xffffffffu, pages, pg & 31), 0), A.n_pages - 1);
      next(4 * 8192);
      if (ok && leader) {
        const uint32_t dst = ring + st * LY_STAGE, bar = bars + st * 8;
        const int row = (int)(L->kv_row0 + ((long long)page * A.nkv + sh->item.kvh) * SX_PAGE);
        tc_tma_load_2d(dst, mk, 0, row, bar);
        tc_tma_load_2d(dst + 8192, mk, 64, row, bar);
        tc_tma_load_2d(dst + 16384, mv, 0, row, bar);
        tc_tma_load_2d(dst + 24576, mv, 64, row, bar);
      }
      __syncwarp();
    }
    const LyProduct x = sh->prod[p];
    const int K = A.K[p];
    const size_t odd = p == 2 ? (size_t)A.ff * K : (size_t)K, pair = p == 2 ? (size_t)K : 2 * (size_t)K;      // to a pair's second row, to the next pair
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += A.pass) {
      const int k1 = min(K, k0 + A.pass);
      const bf16* group = L->w[p] + (size_t)x.row0 * K;
#pragma unroll 1
      for (int g0 = 0; g0 < x.rows; g0 += 16, group += 8 * pair) {
        const int R = min(16, x.rows - g0), span = ly_chunks(R) * LY_KC;
#pragma unroll 1
        for (int k = k0; ok && k < k1; k += span, advance()) {
          if (turn != who) continue;
          const int until = min(k + span, k1);
          next((uint32_t)(R * (until - k) * 2));
          if (!ok) break;
          uint32_t dst = ring + st * LY_STAGE;
          const uint32_t bar = bars + st * 8;
#pragma unroll 1
          for (int c = k; c < until; c += LY_KC) {
            const uint32_t bytes = (uint32_t)(min(LY_KC, until - c) * 2);
            const bf16* src = group + c;
#pragma unroll 1
            for (int r = 0; r < R; r += 2, dst += 2 * LY_ROW, src += pair)
              if (leader) {
                ly_copy(dst, src, bytes, bar);
                ly_copy(dst + LY_ROW, src + odd, bytes, bar);
              }
          }
          __syncwarp();
        }
      }
    }
  }
  if (!ok)            // a wait ran out: what is in flight lands before the block ends
    for (int s = 0; s < A.stages; ++s) {
      const int n = use + (s < st ? 1 : 0);           // times stage s was filled, by either warp
      for (uint32_t i = 0; n > 0 && i < LY_SPIN_BAR && !__all_sync(0xffffffffu, ly_test(bars + s * 8, (n - 1) & 1)); ++i) {}
    }
}

// ---- compute warps ----------------------------------------------------------------------------------------------------
// the stage that is used next: its address, its `full` barrier's (`empty` lies LY_MAX_STAGES further on) and that one's parity
struct LyRing { uint32_t stage, bar, parity; };
__device__ __forceinline__ void ly_done(LyRing& at, uint32_t ring, uint32_t bars, int stages) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) ly_arrive(at.bar + LY_MAX_STAGES * 8);
  at.stage += LY_STAGE;
  at.bar += 8;
  if (at.bar == bars + stages * 8) { at.stage = ring; at.bar = bars; at.parity ^= 1; }
}

// 16 keys of a stage (from key `key` of its page on) for one warp, as an online softmax over the warp's keys.  The products are
// taken with the keys (then the values' columns) as the M side: S^T = K Q^T has 16 keys x 8 heads, O^T = V^T P^T 16 values x 8
// heads, so that the few heads of a group fill N and not half of an M of 16.  A thread holds heads 2t and 2t + 1: m, l and
// the factors are two numbers.  (`left` keys of the 16 are visible; the cache may hold anything behind them.)
__device__ __forceinline__ void ly_attend(const uint32_t (&qf)[8][2], uint32_t stage, int key, int left, float scale_log2,
                                          float (&m)[2], float (&l)[2], float (&o)[8][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, lrow = lane & 7, lmat = lane >> 3;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
  // a lane's 16 bytes of values 16 d .. 16 d + 15 lie at place (2 (d & 3) + its half) XOR row of the row's 8: all but the first is one lane value
  const uint32_t k0 = stage + (key + (lmat & 1) * 8 + lrow) * 128 + (((lmat >> 1) ^ lrow) << 4);
#pragma unroll
  for (int d = 0; d < 8; d += 2) {
    uint32_t a[4], b[4];
    ly_ldsm(a, (k0 ^ ((d & 3) << 5)) + (d >> 2) * 8192);
    ly_ldsm(b, (k0 ^ (((d & 3) + 1) << 5)) + (d >> 2) * 8192);
    ly_mma(s, a[0], a[1], a[2], a[3], qf[d][0], qf[d][1]);
    ly_mma(u, b[0], b[1], b[2], b[3], qf[d + 1][0], qf[d + 1][1]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = (i < 2 ? g : 8 + g) < left ? s[i] + u[i] : -INFINITY;
  float corr[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float mx = fmaxf(m[h], fmaxf(s[h], s[h + 2]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    const bool none = mx == -INFINITY;                   // nothing visible yet: 2^(-inf - 0) = 0
    const float ms = none ? 0.f : mx * scale_log2;
    corr[h] = none ? 1.f : ly_ex2((m[h] - mx) * scale_log2);
    m[h] = mx;
    s[h] = ly_ex2(fmaf(s[h], scale_log2, -ms));
    s[h + 2] = ly_ex2(fmaf(s[h + 2], scale_log2, -ms));
    l[h] = l[h] * corr[h] + (s[h] + s[h + 2]);
  }
  // P^T as the second operand: its 8 x 8 blocks turned round
  uint32_t p0 = ly_pack(s[0], s[1]), p1 = ly_pack(s[2], s[3]);
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %0;\n" : "+r"(p0));
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %0;\n" : "+r"(p1));
  const uint32_t keep0 = (2 * t < left ? 0xffffu : 0u) | (2 * t + 1 < left ? 0xffff0000u : 0u);
  const uint32_t keep1 = (8 + 2 * t < left ? 0xffffu : 0u) | (9 + 2 * t < left ? 0xffff0000u : 0u);
  const uint32_t v0 = stage + 16384 + (key + (lmat >> 1) * 8 + lrow) * 128 + (((lmat & 1) ^ lrow) << 4);
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    uint32_t a[4];
    ly_ldsm_t(a, (v0 ^ ((n & 3) << 5)) + (n >> 2) * 8192);
    o[n][0] *= corr[0]; o[n][1] *= corr[1];
    o[n][2] *= corr[0]; o[n][3] *= corr[1];
    ly_mma(o[n], a[0] & keep0, a[1] & keep0, a[2] & keep1, a[3] & keep1, p0, p1);
  }
}

// `part`: [warps][heads of the group][128] floats (the activations' room, which is free between q/k/v and o)
__device__ __forceinline__ void ly_attention(const LyArgs& A, LyShared* sh, float* part, unsigned char* smem, LyRing& at, int l, uint32_t tag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, G = A.G;
  const uint32_t ring = tc_smem(smem), bars = tc_smem(sh->full);
  volatile int* dead = &sh->dead;
  const LyLayer& L = sh->layers[l];
  const LyItem& item = sh->item;
  const bool own = item.own >= 0;
  // heads: norm and rotation in float32, one head a warp; the new key and value also into the cache
  if (warp < G + (own ? 2 : 0)) {
    const int kind = max(0, warp - G + 1);                // 0 a query, 1 the key, 2 the value
    const int head = kind == 0 ? item.kvh * G + warp : A.nh + (kind - 1) * A.nkv + item.kvh;
    const float* gp = kind == 0 ? L.qn : kind == 1 ? L.kn : nullptr;
    float2 g1 = make_float2(1.f, 1.f), g2 = g1;
    if (gp) {
      g1 = *reinterpret_cast<const float2*>(gp + 2 * lane);
      g2 = *reinterpret_cast<const float2*>(gp + 64 + 2 * lane);
    }
    const ly_word* src = A.words + A.out[0] + item.seq * A.out_row[0] + head * (LY_HD / 2) + lane;
    ly_word a = 0, b = 0;
    ly_poll([&] { a = ly_ld(src); b = ly_ld(src + 32); return ly_is(a, tag) && ly_is(b, tag); }, dead, A.status, 2);
    uint32_t ua = (uint32_t)a, ub = (uint32_t)b;
    if (kind < 2) {
      const float2 x1 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&ua));
      const float2 x2 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&ub));
      const float2 cs = *reinterpret_cast<const float2*>(sh->cs + 2 * lane), sn = *reinterpret_cast<const float2*>(sh->sn + 2 * lane);
      float inv = 1.f;
      if (gp) inv = rsqrtf(warp_sum(x1.x * x1.x + x1.y * x1.y + x2.x * x2.x + x2.y * x2.y) * (1.f / LY_HD) + A.qk_eps);
      const float a0 = x1.x * inv * g1.x, a1 = x1.y * inv * g1.y, b0 = x2.x * inv * g2.x, b1 = x2.y * inv * g2.y;
      ua = ly_pack(a0 * cs.x - b0 * sn.x, a1 * cs.y - b1 * sn.y);
      ub = ly_pack(a0 * sn.x + b0 * cs.x, a1 * sn.y + b1 * cs.y);
    }
    uint32_t* dst = reinterpret_cast<uint32_t*>(kind == 0 ? sh->q + warp * LY_HD : sh->kv + (kind - 1) * LY_HD);
    dst[lane] = ua;
    dst[32 + lane] = ub;
    if (kind > 0) {
      uint32_t* row = reinterpret_cast<uint32_t*>((kind == 1 ? A.kc : A.vc) + (size_t)(L.kv_row0 + item.own) * LY_HD);
      row[lane] = ua;
      row[32 + lane] = ub;
    }
  }
  ly_sync();
  uint32_t qf[8][2];
  const bf16* qg = sh->q + (g < G ? g : 0) * LY_HD + 2 * t;       // (heads beyond the group: results unused)
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    qf[k][0] = *reinterpret_cast<const uint32_t*>(qg + k * 16);
    qf[k][1] = *reinterpret_cast<const uint32_t*>(qg + k * 16 + 8);
  }
  float m[2] = {-INFINITY, -INFINITY}, ls[2] = {0.f, 0.f}, o[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  // a page's 64 keys are four warps' work; every warp passes every stage, so that a stage's barrier counts all of them
  const int key = (warp & 3) * 16;
  int left = item.len - item.first * 64 - key;                     // visible keys from the warp's first on
#pragma unroll 1
  for (int s = 0; s < item.stages; ++s, left -= 64) {
    ly_bar_wait(at.bar, at.parity, dead, A.status, 3);
    if ((s & 1) == warp >> 2 && left > 0) {
      const bool patch = left <= 16 && own;
      if (patch) {                                          // the token's own key and value are not in the cache yet
        const int row = key + left - 1, c16 = lane & 15;
        *reinterpret_cast<uint4*>(smem + (at.stage - ring) + (lane >> 4) * 16384 + (c16 >> 3) * 8192 + row * 128 + (((c16 & 7) ^ (row & 7)) << 4)) =
            reinterpret_cast<const uint4*>(sh->kv)[lane];
        __syncwarp();
      }
      ly_attend(qf, at.stage, key, left, A.scale_log2, m, ls, o);
      if (patch) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // (the write comes before the copy that refills the stage)
    }
    ly_done(at, ring, bars, A.stages);
  }
  // the warps' results.  A thread's 16 values of a head lie together: value d = 16 n + 8 j + g at place 16 g + 2 n + j.
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    ls[h] += __shfl_xor_sync(0xffffffffu, ls[h], 4);
    ls[h] += __shfl_xor_sync(0xffffffffu, ls[h], 8);
    ls[h] += __shfl_xor_sync(0xffffffffu, ls[h], 16);
    if (2 * t + h < G) {
      if (g == 0) { sh->top[2 * t + h][warp] = m[h] * A.scale_log2; sh->sum[2 * t + h][warp] = ls[h]; }     // (-inf and 0 of a warp without keys)
      float4* r = reinterpret_cast<float4*>(part + (warp * G + 2 * t + h) * LY_HD + g * 16);
#pragma unroll
      for (int n = 0; n < 4; ++n) r[n] = make_float4(o[2 * n][h], o[2 * n][h + 2], o[2 * n + 1][h], o[2 * n + 1][h + 2]);
    }
  }
  ly_sync();
  ly_word* att = A.words + A.in[1] + item.words;
  ly_word* parts = A.words + A.part + (item.seq * A.nkv + item.kvh) * A.max_splits * A.part_words;
  const int copy_step = A.in_copy[1];
  if (threadIdx.x < G * (LY_HD / 2)) {                   // two neighbouring values a thread
    const int r = threadIdx.x >> 6, rem = threadIdx.x & 63, gp = rem >> 4, idx = rem & 15;
    const int word = r * (LY_HD / 2) + (idx >> 1) * 8 + (idx & 1) * 4 + gp;
    float M = -INFINITY, Ls = 0.f, O0 = 0.f, O1 = 0.f;
    const float* x = part + r * LY_HD + gp * 32 + idx;
#pragma unroll
    for (int w = 0; w < LY_WARPS; ++w) M = fmaxf(M, sh->top[r][w]);
#pragma unroll 2
    for (int w = 0; w < LY_WARPS; ++w, x += G * LY_HD) {
      const float m1 = sh->top[r][w], f1 = m1 == -INFINITY ? 0.f : ly_ex2(m1 - M), x0 = x[0], x1 = x[16];
      Ls += sh->sum[r][w] * f1;
      O0 += f1 != 0.f ? x0 * f1 : 0.f;
      O1 += f1 != 0.f ? x1 * f1 : 0.f;
    }
    if (item.splits == 1) {
      const uint32_t v = Ls > 0.f ? ly_pack(__fdividef(O0, Ls), __fdividef(O1, Ls)) : 0u;
#pragma unroll 1
      for (int c = 0; c < LY_COPIES; ++c) ly_st(att + c * copy_step + word, v, tag);
    } else {
      ly_word* mine = parts + item.split * A.part_words;
      ly_st2(mine + 2 * word, O0, O1, tag);
      if (rem == 0) ly_st2(mine + G * LY_HD + 2 * r, M, Ls, tag);
    }
  }
  ly_sync();                                             // `part` is free again
  if (item.splits > 1) {
    const int width = 1 << item.log_w, sl = lane & (width - 1), tasks = 32 >> item.log_w;
#pragma unroll 1
    for (int base = item.merge0 + warp * tasks; base < item.merge1; base += LY_WARPS * tasks) {
      const int q = base + (lane >> item.log_w);
      const bool have = q < item.merge1 && sl < item.splits;
      const ly_word* src = parts + sl * A.part_words;
      ly_word o0 = 0, o1 = 0, mw = 0, lw = 0;
      ly_poll([&] {
        if (have) {
          ly_ld2(src + 2 * q, o0, o1);
          ly_ld2(src + G * LY_HD + 2 * (q >> 6), mw, lw);
        }
        return !have || (ly_is(o0, tag) && ly_is(o1, tag) && ly_is(mw, tag) && ly_is(lw, tag));
      }, dead, A.status, 4);
      const float ms = have ? ly_f(mw) : -INFINITY;
      float M = ms;
#pragma unroll 1
      for (int w = 1; w < width; w <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, w));
      const float f = ms == -INFINITY ? 0.f : ly_ex2(ms - M);
      float L1 = f != 0.f ? ly_f(lw) * f : 0.f, a = f != 0.f ? ly_f(o0) * f : 0.f, b = f != 0.f ? ly_f(o1) * f : 0.f;
#pragma unroll 1
      for (int w = 1; w < width; w <<= 1) {
        L1 += __shfl_xor_sync(0xffffffffu, L1, w);
        a += __shfl_xor_sync(0xffffffffu, a, w);
        b += __shfl_xor_sync(0xffffffffu, b, w);
      }
      if (have) {
        const uint32_t v = L1 > 0.f ? ly_pack(__fdividef(a, L1), __fdividef(b, L1)) : 0u;
#pragma unroll 1
        for (int c = sl; c < LY_COPIES; c += item.splits) ly_st(att + c * copy_step + q, v, tag);
      }
    }
  }
}

// A warp's values of an exchange (128 of every chunk of 1,024, `mine` chunks) into shared memory: a lane takes two words, that is
// four values, at a time, and the lanes are shared out over 1 << LOG rows.  `src` and `dst` are the lane's first places.
template <int LOG>
__device__ __forceinline__ void ly_fetch(const ly_word* src, int mine, unsigned char* dst, uint32_t tag, volatile int* dead, int* status) {
  constexpr int STEP = 128 >> LOG, B = 10, CHUNKS = B * STEP / 128;      // values a row and load; loads on the way; chunks they cover
#pragma unroll 1
  for (; mine > 0; mine -= CHUNKS, src += CHUNKS * (LY_KC / 2), dst += CHUNKS * LY_KC * 2) {
    ly_word v[B][2];
    ly_poll([&] {
      uint32_t off = 0;
#pragma unroll
      for (int j = 0; j < B; ++j)
        if ((j * STEP >> 7) < mine) ly_ld2(src + (j * STEP >> 7) * (LY_KC / 2) + (j * STEP & 127) / 2, v[j][0], v[j][1]);
#pragma unroll
      for (int j = 0; j < B; ++j)
        if ((j * STEP >> 7) < mine) off |= ((uint32_t)(v[j][0] >> 32) ^ tag) | ((uint32_t)(v[j][1] >> 32) ^ tag);
      return off == 0;
    }, dead, status, 5);
#pragma unroll
    for (int j = 0; j < B; ++j)
      if ((j * STEP >> 7) < mine)
        *reinterpret_cast<uint2*>(dst + (j * STEP >> 7) * (LY_KC * 2) + (j * STEP & 127) * 2) = make_uint2((uint32_t)v[j][0], (uint32_t)v[j][1]);
  }
  __syncwarp();
}

// a step of 1 << LOG_T rows
template <int LOG_T>
__global__ void __launch_bounds__(LY_THREADS, 1) decode_layers_kernel(const __grid_constant__ CUtensorMap mk,
                                                                      const __grid_constant__ CUtensorMap mv, const __grid_constant__ LyArgs A) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* xs = smem + A.stages * LY_STAGE;
  float* red = reinterpret_cast<float*>(xs + A.xs_bytes);
  LyShared* sh = reinterpret_cast<LyShared*>(xs + A.xs_bytes + LY_RED);
  const uint32_t ring = tc_smem(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blocks = gridDim.x, me = blockIdx.x;
  volatile int* dead = &sh->dead;
  if (tid == 0) {
    for (int s = 0; s < A.stages; ++s) {
      tc_mbar_init(tc_smem(&sh->full[s]), 1);
      tc_mbar_init(tc_smem(&sh->empty[s]), LY_WARPS);
    }
    sh->dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (tid == 32) ly_item(A, sh->item, me);
  if (tid >= 64 && tid < 68) {
    const int p = tid & 3, N = p == 0 ? (A.nh + 2 * A.nkv) * LY_HD : p == 2 ? A.ff : A.W;
    sh->prod[p].row0 = ly_lo(N, me, blocks);
    sh->prod[p].rows = (ly_lo(N, me + 1, blocks) - sh->prod[p].row0) * (p == 2 ? 2 : 1);
  }
#pragma unroll 1
  for (int i = tid; i < A.n_layers * (int)(sizeof(LyLayer) / 8); i += LY_THREADS)
    reinterpret_cast<ly_word*>(sh->layers)[i] = reinterpret_cast<const ly_word*>(A.layers)[i];
  const uint32_t launch = (uint32_t)ly_ld(A.words);
  __syncthreads();
  if (tid < LY_HD / 2 && A.inv_freq && sh->item.has)
    sincosf((float)(sh->item.len - 1) * A.inv_freq[tid], &sh->sn[tid], &sh->cs[tid]);
  else if (tid < LY_HD / 2) { sh->cs[tid] = 1.f; sh->sn[tid] = 0.f; }
  __syncthreads();
  const uint32_t tag0 = launch * LY_MAX_LAYERS + 1;        // of layer 0; one more a layer
  const int copy = me & (LY_COPIES - 1);
  constexpr int T = 1 << LOG_T;

  if (warp < LY_WARPS) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t bars = tc_smem(sh->full);
    LyRing at = {ring, bars, 0u};
    const int stride = A.pass * 2 + 64;                 // bytes between two rows' activations: as a stage's rows, 64 off
    // the lane's activations: token g (mod 1 << LOG_T), and the chunk of those taken together that its column stands for
    const uint32_t xa = tc_smem(xs) + (g & ((1 << LOG_T) - 1)) * stride + (g >> LOG_T) * (LY_KC * 2) + warp * 256 + t * 16;
    // fetching: the lane's row, and its first place there
    const int fn = lane >> (5 - LOG_T), f0 = (lane & ((32 >> LOG_T) - 1)) * 4;
    unsigned char* fdst = xs + fn * stride + warp * 256 + f0 * 2;
    int turn = 0;                                       // groups so far: which buffer of partial sums
#pragma unroll 1
    for (int step = 0; step < 4 * A.n_layers; ++step) {
      const int p = step & 3;
      const uint32_t tag = tag0 + (step >> 2);
      ly_meet(7);
      if (p == 1 && sh->item.has) ly_attention(A, sh, reinterpret_cast<float*>(xs), smem, at, step >> 2, tag);
      const int rows = sh->prod[p].rows, K = A.K[p];
      const ly_word* src = A.words + A.in[p] + copy * A.in_copy[p] + fn * (K >> 1) + warp * 64 + f0 / 2;
#pragma unroll 1
      for (int k0 = 0; k0 < K; k0 += A.pass) {
        const int width = min(K - k0, A.pass), nch = (width + LY_KC - 1) / LY_KC;
        const int mine = max(0, (width - warp * 128 + LY_KC - 1) / LY_KC);     // chunks that this warp has a part of
        ly_fetch<LOG_T>(src + (k0 >> 1), mine, fdst, tag, dead, A.status);
#pragma unroll 1
        for (int g0 = 0; g0 < rows; g0 += 16, ++turn) {
          const int R = min(16, rows - g0), cps = ly_chunks(R), subs = min(cps, 8 >> LOG_T);
          float acc[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 1
          for (int c = 0; c < nch;) {
            ly_bar_wait(at.bar, at.parity, dead, A.status, 7);
            uint32_t a = at.stage + warp * 256 + t * 16;
            const int until = min(c + cps, nch);
            // `subs` chunks of a few rows at a time are the M side's 16 rows; a chunk's activations are the N side's columns of their
            // own, and the sums of chunk and column i are the ones that count
#pragma unroll 1
            for (; c < until; c += subs, a += subs * R * LY_ROW) {
              const int have = min(min(until, mine) - c, subs);    // chunks here that this warp has a part of
              if (have > 0) {
                const uint32_t off0 = a + min(g, have * R - 1) * LY_ROW, off1 = a + min(g + 8, have * R - 1) * LY_ROW, xk = xa + c * (LY_KC * 2);
                const bool on = have > g >> LOG_T;
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                  const uint4 w0 = ly_lds(off0 + j * 64), w1 = ly_lds(off1 + j * 64), v = ly_lds_or_0(xk + j * 64, on);
                  const uint4 y0 = ly_lds(off0 + j * 64 + 64), y1 = ly_lds(off1 + j * 64 + 64), z = ly_lds_or_0(xk + j * 64 + 64, on);
                  ly_mma(acc[0], w0.x, w1.x, w0.y, w1.y, v.x, v.y);
                  ly_mma(acc[1], w0.z, w1.z, w0.w, w1.w, v.z, v.w);
                  ly_mma(acc[2], y0.x, y1.x, y0.y, y1.y, z.x, z.y);
                  ly_mma(acc[3], y0.z, y1.z, y0.w, y1.w, z.z, z.w);
                }
              }
            }
            ly_done(at, ring, bars, A.stages);
          }
          // the warp's part of the sums, [warp][row][token]
          if (turn > 1) ly_meet(4 + (turn & 1));
          float* buf = red + (turn & 1) * (LY_WARPS * 128) + warp * 128 + g * 8 + 2 * t;
          *reinterpret_cast<float2*>(buf) = make_float2((acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]), (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]));
          *reinterpret_cast<float2*>(buf + 64) = make_float2((acc[0][2] + acc[1][2]) + (acc[2][2] + acc[3][2]), (acc[0][3] + acc[1][3]) + (acc[2][3] + acc[3][3]));
          ly_tell(2 + (turn & 1));
        }
      }
    }
    if (turn > 1) ly_meet(4 + (turn & 1));              // (the epilogue warps' last two words)
    if (turn > 0) ly_meet(4 + ((turn + 1) & 1));
  } else if (warp < LY_WARPS + LY_EPI) {
    // ---- epilogue warps: the compute warps' parts added up in warp order, and what comes behind the product.  A thread has row r
    // of a group and token n; lanes of tokens beyond the step's hand on copies of a row's words.
    const int ew = warp - LY_WARPS, e = ew * 32 + lane, r = e >> 3, n = e & 7, tn = lane & ((1 << LOG_T) - 1);
    int turn = 0;
#pragma unroll 1
    for (int g0 = 0; g0 < sh->prod[1].rows; g0 += 16)
      if (g0 + r < sh->prod[1].rows && n < T) sh->h[g0 + r][n] = A.h_in[(size_t)n * A.W + sh->prod[1].row0 + g0 + r];
    // (the step before the first: the stream as it came in, handed to the first layer's norm as `down` hands it on)
#pragma unroll 1
    for (int step = -1; step < 4 * A.n_layers; ++step) {
      const int p = step & 3, l = step >> 2;
      const bool more = l + 1 < A.n_layers, stream = p & 1;
      const uint32_t tag = tag0 + l + (p == 3 ? 1 : 0);
      const LyProduct x = sh->prod[p];
      const int K = step < 0 ? 1 : A.K[p], sh_word = p == 2 ? 2 : 1;
      const float* gains = !stream || !(more || p == 1) ? nullptr : p == 1 ? sh->layers[l].gain[1] : sh->layers[l + 1].gain[0];
      ly_word* out = A.words + A.out[p] + tn * A.out_row[p] + (x.row0 >> 1);
      const int c = n >> LOG_T;                         // which copy the lane writes
      const bool writes = c < (p == 0 ? 1 : LY_COPIES) && !(r & (p == 2 ? 3 : 1)) && (p != 3 || more);
      out += c * A.out_copy[p];
#pragma unroll 1
      for (int k0 = 0; k0 < K; k0 += A.pass) {
#pragma unroll 1
        for (int g0 = 0; g0 < x.rows; g0 += 16) {
          const int R = min(16, x.rows - g0), row = g0 + r;        // of the block's share
          const bool ok = r < R && n < T;
          const float gain = gains && ok ? gains[x.row0 + row] : 1.f;     // (on its way before the sums are there)
          float v = 0.f;
          if (step >= 0) {
            // (where chunks went side by side, column n's sums of chunk n >> LOG_T)
            const int subs = min(ly_chunks(R), 8 >> LOG_T), sub = n >> LOG_T;
            const float* buf = red + (turn & 1) * (LY_WARPS * 128) + (subs > 1 ? (min(sub, subs - 1) * R + min(r, R - 1)) * 8 + n : e);
            ly_meet(2 + (turn & 1));
#pragma unroll
            for (int w = 0; w < LY_WARPS; ++w) v += buf[w * 128];
            ly_tell(4 + (turn & 1));
            if (subs > 1) {
              if (sub >= subs) v = 0.f;
#pragma unroll
              for (int o = 4; o >= 1 << LOG_T; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            ++turn;
            if (k0 > 0 && ok) v += sh->carry[row][n];
            if (k0 + A.pass < K) {                      // (o and down only: more of K is to come)
              if (ok) sh->carry[row][n] = v;
              continue;
            }
          }
          if (!stream) {
            if (g0 == 0) asm volatile("bar.sync 6, %0;\n" ::"n"(LY_EPI * 32) : "memory");      // (the factors, see below)
            v *= sh->factor[p >> 1][tn];                // (columns without a token: results that nothing reads)
          } else if (ok) {
            v += sh->h[row][n];
            sh->h[row][n] = v;
            if (!more && p == 3) A.h_out[(size_t)n * A.W + x.row0 + row] = v;
          }
          float y = v * gain, y1 = __shfl_xor_sync(0xffffffffu, y, 8);
          if (p == 2) {
            const GateAct silu = {0.f, 0.f, SX_GATE_SIGMOID};
            y = gate_mul(y, y1, silu);
            y1 = __shfl_xor_sync(0xffffffffu, y, 16);
          }
          const uint32_t word = __shfl_sync(0xffffffffu, ly_pack(y, y1), (p == 2 ? 0 : lane & 16) | tn);
          if (writes && r < R) ly_st(out + (row >> sh_word), word, tag);
          if (g0 + 16 >= x.rows && (p != 3 || more)) ly_tell(7);
          if (!stream || (p == 3 && !more)) continue;
          float s = ok ? v * v : 0.f;
          s += __shfl_xor_sync(0xffffffffu, s, 8);
          s += __shfl_xor_sync(0xffffffffu, s, 16);
          if (lane < LY_MAX_T) sh->ssq[(g0 >> 4) * 4 + ew][lane] = s;
          if (g0 + 16 >= x.rows) {
            asm volatile("bar.sync 6, %0;\n" ::"n"(LY_EPI * 32) : "memory");
            if ((e >> LOG_T) < LY_COPIES) {
              float q = 0.f;
#pragma unroll 1
              for (int i = 0; i < (g0 >> 4) * 4 + 4; ++i) q += sh->ssq[i][tn];
              ly_st(A.words + A.sums[p == 1 ? 1 : 0] + (e >> LOG_T) * A.s_copy + me * 16 + tn, __float_as_uint(q), tag);
            }
            // the rows' factors 1 / rms for the next product: all blocks' sums of squares added up in block order, a row a warp
#pragma unroll 1
            for (int m = ew; m < T; m += LY_EPI) {
              const ly_word* src = A.words + A.sums[p == 1 ? 1 : 0] + copy * A.s_copy + lane * 16 + m;
              float f = 0.f;
#pragma unroll 1
              for (int i0 = 0; i0 < blocks; i0 += 160) {
                ly_word u[5];
                ly_poll([&] {
                  uint32_t off = 0;
#pragma unroll
                  for (int j = 0; j < 5; ++j) {
                    u[j] = ly_make(0u, tag);
                    if (i0 + j * 32 + lane < blocks) u[j] = ly_ld(src + (i0 + j * 32) * 16);
                  }
#pragma unroll
                  for (int j = 0; j < 5; ++j) off |= (uint32_t)(u[j] >> 32) ^ tag;
                  return off == 0;
                }, dead, A.status, 6);
#pragma unroll
                for (int j = 0; j < 5; ++j) f += ly_f(u[j]);
              }
              f = warp_sum(f);
              if (lane == 0) sh->factor[p == 1 ? 1 : 0][m] = rsqrtf(__fdividef(f, (float)A.W) + A.eps);
            }
          }
        }
      }
    }
  } else {
    ly_produce(A, &mk, &mv, sh, ring);
  }
  __syncthreads();
  // every block has begun by now (this one has read what each of them made), so the number may move on
  if (me == 0 && tid == 0) *reinterpret_cast<volatile ly_word*>(A.words) = (ly_word)((launch + 1) & 0x01ffffffu);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
static int* ly_status_word() {
  static int* p = nullptr;
  if (!p) p = sx_status_word_alloc();
  return p;
}

// the cache as rows of 128 values: boxes of a page's 64 rows of one kv head x 64 values
static int ly_map(CUtensorMap* map, const void* base, long long rows) {
  tc_encode_fn enc = tc_get_encode();
  if (!enc) return SX_ERR_SIZE;
  cuuint64_t dims[2] = {LY_HD, (cuuint64_t)rows};
  cuuint64_t strides[1] = {LY_HD * 2};
  cuuint32_t box[2] = {64, SX_PAGE};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : 20000 + (int)r;
}

typedef void (*LyKernel)(const CUtensorMap, const CUtensorMap, const LyArgs);
static LyKernel ly_kernel(int T) { return T > 1 ? decode_layers_kernel<1> : decode_layers_kernel<0>; }

// The sizes' part of the arguments: places in the workspace, room in shared memory; the workspace's words, or 0.
static long long ly_plan(LyArgs* a, int T, int W, int nh, int nkv, int hd, int ff, int n_layers, int blocks) {
  if (T < 1 || T > LY_MAX_T || hd != LY_HD || nkv < 1 || nh < nkv || nh % nkv || nh / nkv > LY_MAX_G || n_layers < 1 || n_layers > LY_MAX_LAYERS)
    return 0;
  if (W < 128 || W % 128 || ff % 128 || ff < 128 || W > 16384 || ff > 65536 || nh > 512 || T * nkv > blocks) return 0;
  if (W / 2 < blocks || ff / 2 < blocks || (nh + 2 * nkv) * (hd / 2) < blocks) return 0;      // every block has columns of everything
  if (2 * ((W / 2 + blocks - 1) / blocks) > LY_MAX_COLS) return 0;
  a->n_layers = n_layers; a->T = T; a->W = W; a->nh = nh; a->nkv = nkv; a->G = nh / nkv; a->ff = ff;
  a->K[0] = a->K[2] = W; a->K[1] = nh * hd; a->K[3] = ff;
  const int aux = LY_WARPS * a->G * LY_HD * 4, need = T * ((W + LY_KC - 1) / LY_KC * LY_KC * 2 + 64);    // q/k/v, gate and up: their rows at once
  const int most = nh * hd > ff ? nh * hd : ff, whole = T * ((most + LY_KC - 1) / LY_KC * LY_KC * 2 + 64);
  a->xs_bytes = need > aux ? need : aux;
  if (whole <= 24576 && whole > a->xs_bytes) a->xs_bytes = whole;      // (one row: o and down in one go, too)
  a->xs_bytes = (a->xs_bytes + 127) / 128 * 128;
  a->pass = (a->xs_bytes / T - 64) / 2 / LY_KC * LY_KC;
  a->stages = (LY_SMEM_MAX - LY_FIXED - a->xs_bytes) / LY_STAGE;
  if (a->stages > LY_MAX_STAGES) a->stages = LY_MAX_STAGES;
  if (a->stages < LY_MIN_STAGES) return 0;
  a->max_splits = blocks / (T * nkv);
  if (a->max_splits > LY_MAX_SPLITS) a->max_splits = LY_MAX_SPLITS;
  a->part_words = (a->G * (LY_HD + 2) + 15) / 16 * 16;
  long long at = 16;
  auto take = [&](long long n) { const long long here = at; at += (n + 15) / 16 * 16; return (int)here; };
  auto round16 = [](int n) { return (n + 15) / 16 * 16; };
  const int widths[4] = {(nh + 2 * nkv) * hd, W, ff, W};
  for (int p = 0; p < 4; ++p) {
    a->out_row[p] = widths[p] / 2;
    a->out_copy[p] = round16(T * a->out_row[p]);
    a->out[p] = take((long long)(p == 0 ? 1 : LY_COPIES) * a->out_copy[p]);
  }
  a->in[0] = a->out[3]; a->in_copy[0] = a->out_copy[3];
  a->in[2] = a->out[1]; a->in_copy[2] = a->out_copy[1];
  a->in[3] = a->out[2]; a->in_copy[3] = a->out_copy[2];
  a->in_copy[1] = round16(T * nh * (hd / 2));
  a->in[1] = take((long long)LY_COPIES * a->in_copy[1]);
  a->s_copy = 16 * blocks;
  a->sums[0] = take((long long)LY_COPIES * a->s_copy);
  a->sums[1] = take((long long)LY_COPIES * a->s_copy);
  a->part = take((long long)T * nkv * a->max_splits * a->part_words);
  return at < (1 << 28) ? at : 0;
}

// Whether these sizes run here, and the workspace they need (8-byte words, zeroed once by the caller; launches that share one are
// ordered among themselves): a word count > 0, or 0.
extern "C" int sx_decode_layers_plan(int T, int W, int nh, int nkv, int hd, int ff, int n_layers) {
  LyArgs a = {};
  const long long words = ly_plan(&a, T, W, nh, nkv, hd, ff, n_layers, sx_sm_count());
  if (!words) return 0;
  static int coops[64][LY_MAX_T] = {{0}};         // 1: a block an SM can be launched together on all of them; -1: not
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int& coop = coops[dev][T - 1];
  if (!coop) {
    int can = 0, n = 0;
    const bool ok = cudaDeviceGetAttribute(&can, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && can &&
                    cudaFuncSetAttribute(ly_kernel(T), cudaFuncAttributeMaxDynamicSharedMemorySize, LY_SMEM_MAX) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ly_kernel(T), LY_THREADS, LY_SMEM_MAX) == cudaSuccess && n >= 1;
    (void)cudaGetLastError();
    coop = ok ? 1 : -1;
  }
  return coop > 0 ? (int)words : 0;
}

// layers: n_layers records on the device, 9 x 8 bytes each (`LyLayer`); h_in, h_out float32 [T, W] (one tensor may be both); the
// cache's keys and values as rows of 128 values from k_base / v_base on, `kv_rows` of them; words: see sx_decode_layers_plan.
// SX_ERR_NO_ROOM: the stream has a part of the device's SMs only, so that the blocks cannot run at once; nothing was launched.
extern "C" int sx_decode_layers(const void* layers, int n_layers, void* words, const float* h_in, float* h_out, const int* seq_lens,
                                const int* block_table, int maxp, int n_pages, void* k_base, void* v_base, long long kv_rows,
                                const float* inv_freq, int T, int W, int nh, int nkv, int hd, int ff, float scale, float eps, float qk_eps,
                                cudaStream_t stream) {
  if (sx_decode_layers_plan(T, W, nh, nkv, hd, ff, n_layers) <= 0 || maxp < 1 || n_pages < 1 || kv_rows < SX_PAGE || kv_rows > 0x7fffffffLL) return SX_ERR_SIZE;
  if (((uintptr_t)layers & 7) || ((uintptr_t)words & 127) || ((uintptr_t)k_base & 15) || ((uintptr_t)v_base & 15) ||
      ((uintptr_t)h_in & 3) || ((uintptr_t)h_out & 3)) return SX_ERR_ALIGN;
  int* status = ly_status_word();
  if (!status) return (int)cudaErrorMemoryAllocation;
  CUtensorMap mk, mv;
  int rc = ly_map(&mk, k_base, kv_rows);
  if (rc || (rc = ly_map(&mv, v_base, kv_rows))) return rc;
  const int blocks = sx_sm_count();
  LyArgs a = {};
  if (!ly_plan(&a, T, W, nh, nkv, hd, ff, n_layers, blocks)) return SX_ERR_SIZE;
  a.layers = (const LyLayer*)layers;
  a.eps = eps; a.qk_eps = qk_eps; a.scale_log2 = scale * 1.4426950408889634f;
  a.h_in = h_in; a.h_out = h_out; a.seq_lens = seq_lens; a.block_table = block_table;
  a.maxp = maxp; a.n_pages = n_pages; a.inv_freq = inv_freq;
  a.kc = (bf16*)k_base; a.vc = (bf16*)v_base; a.words = (ly_word*)words; a.status = status;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(LY_THREADS);
  cfg.dynamicSmemBytes = a.stages * LY_STAGE + a.xs_bytes + LY_FIXED;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;         // the blocks wait for one another: all of them run at once, or none
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, ly_kernel(T), mk, mv, (const LyArgs)a);
  if (e != cudaErrorCooperativeLaunchTooLarge) return (int)e;
  (void)cudaGetLastError();                             // (nothing was launched, and nothing else is told of it)
  return SX_ERR_NO_ROOM;
}

// as the other libraries' status words: which bounded wait ran out (0: none)
extern "C" int sx_decode_layers_status(int* host_value, int reset) {
  int* p = ly_status_word();
  if (!p) return (int)cudaErrorMemoryAllocation;
  *host_value = *(volatile int*)p;
  if (reset) *(volatile int*)p = 0;
  return 0;
}
