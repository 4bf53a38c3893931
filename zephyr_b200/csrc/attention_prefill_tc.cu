// Paged causal attention for prompt portions on the fifth-generation tensor cores: tcgen05.mma with
// the queries, keys and values in shared memory and the scores, probabilities and results in tensor
// memory (TMEM).  bfloat16; head size 128, or rows of 160 values that are keys and (their first 128)
// values at once, as latent attention keeps them.
//
// One CTA = 128 consecutive new tokens of one request and two SLOTS that share the tensor core by turns:
// while one slot's softmax runs, the other slot's products do.  Two forms of a CTA:
//   * a pair of heads that share a key/value head, a slot each: a tile of keys and values is fetched
//     once for both (what bounds larger launches is the fetch: 64 KB a tile and slot would be twice the
//     bytes a cycle that L2 delivers to all SMs);
//   * one head whose tiles of keys the slots take by turns, even and odd, and merge at the end: half as
//     long a chain, for the tiles that would otherwise end last (and for heads without a partner).
// Roles:
//   * loader warps copy a tile's rows from the cache pages (TMA tiled copies per page; at an edge of the context the values'
//     rows beyond it are set to zero once their page has landed; 16-byte asynchronous copies for a cache of
//     more rows than a tensor map counts).  A cache row's 16-byte chunks are stored permuted with the position (common.cuh: kv_swizzle); for
//     rows of 256 bytes that permutation IS the 128-byte swizzle of the tensor core's canonical
//     shared-memory layout over blocks of 64 values, for rows of 320 bytes the 64-byte swizzle over
//     blocks of 32, so a row is copied as it lies, block by block;
//   * one thread issues the products: S = Q K^T (M 128 queries, N 128 keys, steps of K = 16; both
//     operands K-major in shared memory) into a slot's 128 columns of TMEM, and O += P V (A = the
//     probabilities, which the softmax leaves where their S lay; B = the values as they lie, MN-major)
//     into the slot's other 128; completion is reported to mbarriers by tcgen05.commit;
//   * eight softmax warps, four a slot, a thread a row (TMEM lane = row): they read S with tcgen05.ld,
//     keep the running sum in float32 in base 2, store the probabilities as bfloat16 pairs with
//     tcgen05.st, and rescale O in TMEM when the row's maximum has grown by more than 2^8 since the
//     value the row last rescaled to (the softmax does not care which shift it is given as long as it
//     is given everywhere; the bound keeps exp2 far from overflow).
// What bounds it: the turn of a slot, S -> softmax -> P -> O += P V -> next S (some 2350 + 1450 cycles a tile of 128 x 128), of
// which the other slot hides half; of 3900 cycles for both slots' tiles the products take 2048 and the exponentials 2048.  (One
// slot a CTA, as it was, took 5000 for two tiles.)  Measured there and here: 2048 tokens, 16/8 heads 38 -> 33 us; rows of 1531, 500
// and 17 tokens, 32/8 heads 62 -> 41 us; 3000 tokens in a window of 1024 with 64 kept 73 -> 46 us; 8192 tokens, 32/8 heads
// 703 -> 530 us (1040 TFLOP/s); 2048 tokens of 16 heads over rows of 160 values, on the mma.sync kernel before, 119 -> 39 us.
// Taken back: a pass that takes the row's maximum and the probabilities under the old shift at once, and repeats where the shift has
// to move (registers; 3 to 15 % slower), two threads a row (5 % slower), loads of S further ahead (7 % faster at
// 8192 tokens, 4 to 8 % slower below 1000: spills).
// A window may keep the first tokens of a sequence, and a chunk may bound what a query sees: masks of the same loop.
// Math and masking as in attention_prefill.cu and attention_simt.cu (causal, lower-right aligned on
// the cached context, optional window, whose first tokens may be kept, and optional chunk; probabilities rounded to
// bfloat16 for the second product;
// reference: src/layer/paged_attention.cpp:118-296, deps/ttl/src/kernels/attention/attention.cu:58-170).
// Every wait is bounded and reports instead of hanging; TMEM is given back on every path.
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace zb {

constexpr int TC_BM = 128;                 // query rows per slot
constexpr int TC_BN = 128;                 // positions per key/value tile
constexpr int TC_VD = 128;                 // values per row of the result
constexpr int TC_SOFTMAX_WARPS = 8;        // warps 0..3: slot 0, warps 4..7: slot 1; TMEM lanes 32 (w % 4) .. + 31
constexpr int TC_MMA_WARP = 8;
constexpr int TC_LOADER_WARPS = 3;         // warps 9..11: one for the keys and one for the values, or all for rows that are both
constexpr int TC_THREADS = (TC_SOFTMAX_WARPS + 1 + TC_LOADER_WARPS) * 32;      // 12 warps: 168 registers a thread (with 13 it is 128, and the softmax spills)
constexpr int TC_WAIT_LIMIT = 1 << 18;
constexpr int TC_TMEM_COLUMNS = 512;        // S of slot 0, S of slot 1, O of slot 0, O of slot 1
constexpr int TC_O_COLUMN = 2 * TC_BN;
constexpr float TC_RESCALE_THRESHOLD = 8.0f;

// How rows of HD values lie in shared memory: blocks of BLOCK values, [HD / BLOCK][128 rows][BLOCK], swizzled over 2 BLOCK bytes.
// SHARED: a row is key and value at once, so a tile is one item of the ring, not two.
template <int HD, bool SHARED>
struct TcShape {
  static constexpr int BLOCK = HD % 64 == 0 ? 64 : 32;
  static constexpr int BLOCKS = HD / BLOCK;
  static constexpr int BLOCK_BYTES = TC_BN * BLOCK * 2;
  static constexpr int ITEM_BYTES = BLOCKS * BLOCK_BYTES;          // 32 KB (128), 40 KB (160)
  static constexpr int Q_BYTES = TC_BM * HD * 2;
  static constexpr int STAGES = SHARED ? 3 : 5;
  static constexpr int KIND_WARPS = SHARED ? TC_LOADER_WARPS : 1;
  static constexpr int SMEM = 2 * Q_BYTES + STAGES * ITEM_BYTES;
  static_assert(SMEM <= 225 * 1024, "the queries and the ring fit an SM's shared memory");
};

struct PrefillTcArgs {
  CUtensorMap cache_map;         // the cache as [rows of all pages, keys and values, heads][hd]; box: a block's values x one page's rows (at most 128)
  int n_tiles, n_split;          // tiles; the last n_split of the list run a head a CTA, the others two heads a CTA
  int tiled;                     // 0: no map (every tile goes through 16-byte copies)
  const __nv_bfloat16* q;        // [T, nh*hd]
  __nv_bfloat16* out;            // [T, nh*hd]
  const __nv_bfloat16* kv_cache; // [num_pages][2][nkv][page_size][hd]
  const int* block_table;        // [R, max_blocks]
  const int* tile_row;           // [n_tiles]
  const int* tile_q0;            // [n_tiles]
  const int* row_q_start;        // [R]
  const int* row_q_len;          // [R]
  const int* row_ctx;            // [R]
  int max_blocks, page_shift, num_pages, num_rows;
  int nh, nkv, window;
  int chunk;                     // > 0: a query at position p sees only keys j with j / chunk == p / chunk
  int keep_first;                // with a window: keys below this position stay visible to every later query
  float scale_log2;
  float softcap_log2;            // > 0: scores are softcap * tanh(scale * s / softcap); this is softcap * log2(e)
  float scale_over_cap;          // scale / softcap
  int keys_only;                 // a page holds keys alone, [nkv][page_size][hd], and they are the values too
  const float* sinks;            // null, or [nh]: exp(sinks[h]) joins the softmax's denominator of head h
  const float* bias_r1;          // null, or [nh] each: r1_h ln(1 + r2_h d) is taken off head h's scaled score of the
  const float* bias_r2;          // key d positions back
  int* status;
  int* trace;                    // null, or 4 ints per tile of the first CTA's slot 0 (the longest work of the launch): the global
                                 // timer (ns, low 32 bits) when S of the tile was issued, when its softmax began (S
                                 // complete), when its probabilities were written, when O += P V of it was issued
};

__device__ __forceinline__ int tc_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return static_cast<int>(t);
}

// Descriptors of the operands (tcgen05.cuh: desc_k_major has the fields) in blocks of BLOCK values with the swizzle of that
// width.  K-major (queries, keys): groups of 8 rows are 16 BLOCK bytes apart (the stride offset).
template <int BLOCK>
__device__ __forceinline__ unsigned long long tc_desc_k(unsigned smem_address) {
  return static_cast<unsigned long long>((smem_address >> 4) & 0x3FFFu) | (1ull << 16) |
         (static_cast<unsigned long long>(BLOCK) << 32) | (1ull << 46) | ((BLOCK == 64 ? 2ull : 4ull) << 61);
}
// MN-major (values): a row is one position's values of a block; the stride offset steps over groups of 8 positions (K), the
// leading offset over the blocks (N).
template <int BLOCK>
__device__ __forceinline__ unsigned long long tc_desc_mn(unsigned smem_address) {
  return static_cast<unsigned long long>((smem_address >> 4) & 0x3FFFu) |
         (static_cast<unsigned long long>(TC_BN * BLOCK * 2 >> 4) << 16) | (static_cast<unsigned long long>(BLOCK) << 32) | (1ull << 46) |
         ((BLOCK == 64 ? 2ull : 4ull) << 61);
}
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float log2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// tanh from the special-function unit's exp2 and reciprocal, 1 - 2 / (e^(2x) + 1): absolute error about 1e-7 over
// the whole line (the unit's own tanh is good to 2^-11 only, which would move a score capped at 30 by 0.02).
__device__ __forceinline__ float tanh_from_exp2(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(exp2_approx(x * 2.8853900817779268f) + 1.0f));
  return fmaf(-2.0f, r, 1.0f);
}

// Two float32 side by side (one instruction each): a b + c, a + b.
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The largest score of a row of S (this thread's TMEM lane), as it lies there.  MASKED: column i counts only if
// first <= i <= last (positions relative to the tile's first key).
// BIASED: the scores become raw * scale - r1 log2(1 + r2 d), d = at - i being how far the key of column i lies behind the
// query, and are written back as that.
template <bool MASKED, bool BIASED>
__device__ __forceinline__ float tc_row_max(unsigned tmem_row, int last, int first, float scale, int at, float r1, float r2) {
  // Several running maxima (and in the other pass sums) side by side: a single chain of 128 dependent operations would
  // cost its full latency 128 times.  A piece of 32 columns is on its way while the one before is worked on.
  float max4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  unsigned v[2][32];
  tmem_ld32(tmem_row, v[0]);
#pragma unroll
  for (int c = 0; c < TC_BN / 32; ++c) {
    unsigned (&now)[32] = v[c & 1];
    tmem_wait_ld32(now);
    if (c + 1 < TC_BN / 32) tmem_ld32(tmem_row + (c + 1) * 32, v[(c + 1) & 1]);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float raw[2] = {__uint_as_float(now[i]), __uint_as_float(now[i + 1])};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int column = c * 32 + i + e;
        if (BIASED) {
          raw[e] = fmaf(raw[e], scale, -r1 * log2_approx(fmaf(r2, static_cast<float>(at - column), 1.0f)));
          now[i + e] = __float_as_uint(raw[e]);
        }
        if (MASKED && (column > last || column < first)) raw[e] = -INFINITY;
      }
      asm("max.f32 %0, %1, %2, %3;\n" : "=f"(max4[(i >> 1) & 3]) : "f"(max4[(i >> 1) & 3]), "f"(raw[0]), "f"(raw[1]));
    }
    if (BIASED) tmem_st32(tmem_row + c * 32, now);
  }
  if (BIASED) tc_wait_st();
  return fmaxf(fmaxf(max4[0], max4[1]), fmaxf(max4[2], max4[3]));
}

// 64 columns (from `column0` on) of a row of S -> probabilities exp2(s * scale + neg_shift) as 32 words of two bfloat16 each,
// and their sums on top of `sums`.  CAPPED: the exponent is cap_log2 * tanh(s * scale) + neg_shift, `scale` then being
// scale / softcap.
template <bool MASKED, bool CAPPED>
__device__ __forceinline__ void tc_exponentials(unsigned tmem_row, int column0, unsigned (&words)[32], unsigned long long (&sums)[4],
                                                float scale, float neg_shift, int last, int first, float cap_log2) {
  const unsigned long long scale2 = pack_f32x2(scale, scale), shift2 = pack_f32x2(neg_shift, neg_shift);
  unsigned v[2][32];
  tmem_ld32(tmem_row + column0, v[0]);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    tmem_wait_ld32(v[c]);
    if (c == 0) tmem_ld32(tmem_row + column0 + 32, v[1]);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float raw[2] = {__uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1])};
      float x[2], p[2];
      if (CAPPED) {
#pragma unroll
        for (int e = 0; e < 2; ++e) x[e] = fmaf(cap_log2, tanh_from_exp2(raw[e] * scale), neg_shift);
      } else {
        unpack_f32x2(fma_f32x2(pack_f32x2(raw[0], raw[1]), scale2, shift2), x[0], x[1]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int column = column0 + c * 32 + i + e;
        p[e] = !MASKED || (column <= last && column >= first) ? exp2_approx(x[e]) : 0.0f;
      }
      sums[(i >> 1) & 3] = add_f32x2(sums[(i >> 1) & 3], pack_f32x2(p[0], p[1]));
      words[16 * c + (i >> 1)] = pack_bf16(p[0], p[1]);
    }
  }
}

// FORM: which of the masks and biases beside causality and a window the kernel knows (forms of their own, so that the plain one
// keeps its registers: with the chunk in it, seven prompts of 300 tokens took 58.8 us, 57.2 without).
enum { TC_FORM_PLAIN, TC_FORM_BIASED, TC_FORM_CHUNKED, TC_FORM_KEPT };      // KEPT: first tokens kept, and a chunk
template <int FORM, int HD, bool SHARED>
__global__ void __launch_bounds__(TC_THREADS, 1)
paged_prefill_tc_kernel(const __grid_constant__ PrefillTcArgs a) {
  constexpr bool BIASED_SCORES = FORM == TC_FORM_BIASED, KEPT = FORM == TC_FORM_KEPT, CHUNKED = KEPT || FORM == TC_FORM_CHUNKED;
  using Shape = TcShape<HD, SHARED>;
  constexpr int STAGES = Shape::STAGES, BLOCK = Shape::BLOCK, BLOCK_BYTES = Shape::BLOCK_BYTES, ITEM_BYTES = Shape::ITEM_BYTES;
  constexpr int CHUNKS = HD / 8, BLOCK_CHUNKS = BLOCK / 8;      // 16-byte pieces of a row, and of a block's row
  // Shared memory: the slots' queries, then the ring of key and value tiles (a stage holds either; keys_j, values_j,
  // keys_j+1 ... in turn), all on 1024-byte boundaries as the swizzles want them.
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* const ring = smem + 2 * Shape::Q_BYTES;
  __shared__ unsigned long long bars[2 * STAGES + 9];
  unsigned long long* kv_full = bars;                   // [stages] the rows have landed (the loader warps of the kind)
  unsigned long long* kv_empty = bars + STAGES;         // [stages] the products that read them are complete
  unsigned long long* s_full = bars + 2 * STAGES;       // [2 slots] S of the slot's next tile is complete, and with it all products before it
  unsigned long long* p_full = s_full + 2;              // [2 slots][2 halves] P is written, O has been rescaled (the slot's warps)
  unsigned long long* o_done = s_full + 6;              // [2 slots] the slot's last O += P V is complete
  unsigned long long* q_full = s_full + 8;              // the queries are in shared memory (the softmax warps)
  __shared__ float note[2][TC_BM][2];                   // a head a CTA: each slot's shift and sum of every row
  __shared__ unsigned long long edge_full;              // the pages of a tile at an edge have landed
  __shared__ unsigned tmem_base_s;
  __shared__ volatile int abort_flag;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int b = 0; b < STAGES; ++b) {
      mbar_init(&kv_full[b], Shape::KIND_WARPS);
      mbar_init(&kv_empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[2 * b], TC_SOFTMAX_WARPS / 2);
      mbar_init(&p_full[2 * b + 1], TC_SOFTMAX_WARPS / 2);
      mbar_init(&o_done[b], 1);
    }
    mbar_init(q_full, TC_SOFTMAX_WARPS);
    mbar_init(&edge_full, 1);
    fence_barrier_init();
  }
  wait_for_prior_grids();          // tiles, queries, keys and values: all of it earlier kernels' work
  let_dependents_launch();

  // The host lists the tiles by the number of keys they see, fewest first: take the list back to
  // front, and all heads of a tile before the next tile, so that the longest work of the whole
  // launch starts first and the short tiles fill the gaps at the end.
  const bool split = static_cast<long long>(blockIdx.x) < static_cast<long long>(a.n_split) * a.nh;
  int tile, head0;
  if (split) {
    tile = a.n_tiles - 1 - blockIdx.x / a.nh;
    head0 = blockIdx.x % a.nh;
  } else {
    const int rest = blockIdx.x - a.n_split * a.nh, pairs = a.nh / 2;
    tile = a.n_tiles - 1 - a.n_split - rest / pairs;
    head0 = rest % pairs * 2;
  }
  const int row = a.tile_row[tile], q0 = a.tile_q0[tile];
  if (row < 0 || row >= a.num_rows) {
    if (threadIdx.x == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, row, tile);
    return;
  }
  if ((smem_u32(smem) & 1023u) != 0) {          // the tiles must lie on 1024-byte boundaries
    if (threadIdx.x == 0) report(a.status, STATUS_INTERNAL_CHECK, static_cast<int>(smem_u32(smem) & 1023u), tile);
    return;
  }
  const int kvh = head0 / (a.nh / a.nkv);
  const int q_len = a.row_q_len[row], ctx = a.row_ctx[row], tok0 = a.row_q_start[row] + q0;
  const int n_tok = min(TC_BM, q_len - q0);
  if (n_tok <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int page_size = 1 << a.page_shift;
  int* const trace = a.trace != nullptr && blockIdx.x == 0 ? a.trace : nullptr;

  // Keys any query of this tile may see: [lo, hi).
  const int hi = ctx + q0 + n_tok;
  int lo = a.window > 0 ? max(0, ctx + q0 - a.window + 1) : 0;
  if (CHUNKED && a.chunk > 0) lo = max(lo, (ctx + q0) / a.chunk * a.chunk);
  // First tokens that a window keeps, [0, kept), are tiles of their own in front as soon as some row has left a key
  // behind; what follows them is the window's (and the chunk's) alone.
  int kept = 0;
  if (KEPT && max(hi - a.window, a.chunk > 0 ? (hi - 1) / a.chunk * a.chunk : 0) > 0) kept = min(a.keep_first, hi);
  lo = max(lo, kept);
  const int first_tile = lo / TC_BN * TC_BN;
  const int kept_tiles = KEPT ? (kept + TC_BN - 1) / TC_BN : 0;
  const int n_tiles = kept_tiles + (lo < hi ? (hi - first_tile + TC_BN - 1) / TC_BN : 0);
  auto tile_start = [&](int j) { return KEPT && j < kept_tiles ? j * TC_BN : first_tile + (j - kept_tiles) * TC_BN; };
  auto run_lo = [&](int j) { return KEPT && j < kept_tiles ? 0 : lo; };                // the positions a tile's rows are taken from
  auto run_hi = [&](int j) { return KEPT && j < kept_tiles ? kept : hi; };
  // A slot's tiles: all of them, or every other one.
  auto slot_tiles = [&](int slot) { return split ? (n_tiles + 1 - slot) >> 1 : n_tiles; };
  auto slot_tile = [&](int slot, int i) { return split ? 2 * i + slot : i; };

  if (warp == TC_MMA_WARP) {
    tmem_alloc(&tmem_base_s, TC_TMEM_COLUMNS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const unsigned tmem_base = tmem_base_s;

  auto wait = [&](unsigned long long* bar, unsigned parity) -> bool {
    if (mbar_try_wait(bar, parity)) return true;
    for (int i = 0; i < TC_WAIT_LIMIT; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if ((i & 63) == 63 && abort_flag) return false;
    }
    return false;
  };
  auto give_up = [&](int where) {
    if (!abort_flag) report(a.status, STATUS_COPY_TIMEOUT, where, tile);
    abort_flag = 1;
  };

  if (warp > TC_MMA_WARP) {
    // ------------------------------------------------------------------------- the loaders
    // One warp fetches the keys and one the values, each at its own pace; rows that are both have all three.
    constexpr int KIND_THREADS = Shape::KIND_WARPS * 32;
    const int lk = threadIdx.x - (TC_MMA_WARP + 1) * 32;          // 0..95
    const int kv = lk / KIND_THREADS, lt = lk % KIND_THREADS;     // 0: keys, 1: values (2: nothing to do)
    const int* table = a.block_table + static_cast<size_t>(row) * a.max_blocks;
    const int planes = a.keys_only ? 1 : 2;                       // a page's halves: keys and values, or keys that are both
    // Tiles come by TMA: one tiled copy per page and block of values (copied as they lie: the cache's own chunk
    // permutation is already the canonical swizzle), a copy a thread, the bytes counted on the stage's barrier.
    const int rows_per_copy = min(page_size, TC_BN), copies_per_block = TC_BN / rows_per_copy;
    const int piece = lt % copies_per_block;
    const bool issues = lt / copies_per_block < Shape::BLOCKS;
    // The page id of the next tile is asked for as soon as this tile's copy is out, so that the table's
    // latency is not in front of it.
    int ahead_tile = -1, ahead_page = 0;
    auto look_up = [&](int j) {
      const int block = (tile_start(j) + piece * rows_per_copy) >> a.page_shift;
      return issues && block < a.max_blocks ? table[block] : -1;
    };
    auto copy_piece = [&](int j, int id, int pg, unsigned char* dst, unsigned long long* bar) {
      const int my_block = id / copies_per_block, piece = id % copies_per_block;
      if (pg <= 0 || pg >= a.num_pages) {
        report(a.status, STATUS_PAGE_OUT_OF_RANGE, pg, tok0);
        pg = 0;                       // the bytes must arrive all the same
      }
      const int pos = tile_start(j) + piece * rows_per_copy;
      const int cache_row = ((pg * planes + (a.keys_only ? 0 : kv)) * a.nkv + kvh) * page_size + (pos & (page_size - 1));
      tiled_copy_2d_g2s(dst + my_block * BLOCK_BYTES + piece * rows_per_copy * BLOCK * 2, &a.cache_map, my_block * BLOCK, cache_row, bar);
    };
    auto issue_tiled = [&](int j, unsigned char* dst, unsigned long long* bar) {
      const int pg = ahead_tile == j ? ahead_page : look_up(j);
      if (lt == 0) mbar_arrive_expect_tx(bar, ITEM_BYTES);
      else if (lane == 0) tc_mbar_arrive(bar);
      if (issues) copy_piece(j, lt, pg, dst, bar);
      if (j + 1 < n_tiles) {
        ahead_page = look_up(j + 1);
        ahead_tile = j + 1;
      }
    };
    // A tile at an edge of [lo, hi): the pages that hold some of its rows come the same way, by the kind's first warp.  What
    // lies in the other rows does not matter where they are only keys (their scores are masked); values there are set to
    // zero once the pages have landed (a zero probability times a zero value stays zero).
    int edges = 0;
    auto issue_edge = [&](int j, unsigned char* dst, unsigned long long* bar) {
      if (lt >= 32) {
        if (lane == 0) tc_mbar_arrive(bar);
        return;
      }
      const int k0 = tile_start(j), from = max(run_lo(j) - k0, 0), until = min(run_hi(j) - k0, TC_BN);      // the rows that count
      const int first_piece = from / rows_per_copy, pieces = (until - 1) / rows_per_copy + 1 - first_piece;
      const bool zeros = SHARED || kv == 1;
      unsigned long long* landed = zeros ? &edge_full : bar;
      if (lane == 0) mbar_arrive_expect_tx(landed, pieces * Shape::BLOCKS * rows_per_copy * BLOCK * 2);
      __syncwarp();
      for (int id = lane; id < pieces * Shape::BLOCKS; id += 32) {
        const int piece = first_piece + id % pieces, block = (k0 + piece * rows_per_copy) >> a.page_shift;
        copy_piece(j, id / pieces * copies_per_block + piece, block < a.max_blocks ? table[block] : -1, dst, landed);
      }
      if (!zeros) return;
      if (!__all_sync(0xffffffffu, wait(&edge_full, edges & 1))) { give_up(-2); return; }
      ++edges;
      for (int e = lane; e < TC_BN * CHUNKS; e += 32) {
        const int r = e % TC_BN, c = e / TC_BN;
        if (r < from || r >= until)
          *reinterpret_cast<uint4*>(dst + (c / BLOCK_CHUNKS) * BLOCK_BYTES + r * (BLOCK * 2) + (c % BLOCK_CHUNKS) * 16) = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async();           // the tensor core reads these zeros through the asynchronous proxy
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(bar);
    };
    // Without a tensor map (a cache of more rows than a coordinate counts): 16-byte copies, zeros where a row does not count.
    auto issue_plain = [&](int j, unsigned char* dst, unsigned long long* bar) {
      const int k0 = tile_start(j), rows_lo = run_lo(j), rows_hi = run_hi(j);
      const long long v_offset = a.keys_only || kv == 0 ? 0LL : static_cast<long long>(a.nkv) * page_size * HD;
      // 32 rows at a time: a lane looks up a row's page each, then the warp copies two rows at a time, 16 lanes a row.
#pragma unroll 1
      for (int r0 = lt & ~31; r0 < TC_BN; r0 += KIND_THREADS) {
        const int own_pos = k0 + r0 + lane;
        int page = 0;
        if (own_pos >= rows_lo && own_pos < rows_hi) {
          const int block = own_pos >> a.page_shift;
          page = block < a.max_blocks ? table[block] : -1;
          if (page <= 0 || page >= a.num_pages) {
            report(a.status, STATUS_PAGE_OUT_OF_RANGE, page, tok0);
            page = 0;
          }
        }
        const int half = lane >> 4;
#pragma unroll 4
        for (int i = 0; i < 16; ++i) {
          const int from = 2 * i + half, r = r0 + from, pos = k0 + r;
          const int pg = __shfl_sync(0xffffffffu, page, from);
          const __nv_bfloat16* src = a.kv_cache;
          if (pg > 0) src += ((static_cast<long long>(pg) * planes * a.nkv + kvh) * page_size + (pos & (page_size - 1))) * HD + v_offset;
#pragma unroll
          for (int c = lane & 15; c < CHUNKS; c += 16)
            cp_async_16(dst + (c / BLOCK_CHUNKS) * BLOCK_BYTES + r * (BLOCK * 2) + (c % BLOCK_CHUNKS) * 16, src + (pg > 0 ? c * 8 : 0), pg > 0);
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async();           // the tensor core reads what the copies wrote through the asynchronous proxy
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(bar);
    };
    for (int j = 0; j < n_tiles && kv < 2; ++j) {
      const int item = SHARED ? j : 2 * j + kv, stage = item % STAGES;
      if (!__all_sync(0xffffffffu, wait(&kv_empty[stage], ((item / STAGES) & 1) ^ 1))) {
        give_up(-1);
        break;
      }
      const int k0 = tile_start(j);
      if (trace && lt == 0 && j < 64) trace[256 + 4 * j + kv] = tc_timer_ns();
      unsigned char* dst = ring + stage * ITEM_BYTES;
      if (!a.tiled) issue_plain(j, dst, &kv_full[stage]);
      else if (k0 >= run_lo(j) && k0 + TC_BN <= run_hi(j)) issue_tiled(j, dst, &kv_full[stage]);
      else issue_edge(j, dst, &kv_full[stage]);
    }
  } else if (warp == TC_MMA_WARP) {
    // ------------------------------------------------------------- the warp that issues products
    // The whole warp takes every turn and wait, one elected thread issues: operands of the products are then the same in
    // all lanes.
    {
      constexpr unsigned IDESC_QK = tc_idesc(false), IDESC_PV = tc_idesc(true);
      constexpr int KSTEP = BLOCK * 2 * 16;        // bytes between 16 positions' values
      const bool leader = elect_one();
      const int count0 = slot_tiles(0), count1 = slot_tiles(1);
      auto key_item = [&](int t) { return SHARED ? t : 2 * t; };
      auto value_item = [&](int t) { return SHARED ? t : 2 * t + 1; };
      auto arrived = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, wait(bar, parity)); };
      auto landed = [&](int item) { return arrived(&kv_full[item % STAGES], (item / STAGES) & 1); };
      auto issue_scores = [&](int slot, int i) -> bool {
        const int t = slot_tile(slot, i), item = key_item(t);
        if (!landed(item)) return false;
        tc_fence_after_sync();
        const unsigned long long k_desc = tc_desc_k<BLOCK>(smem_u32(ring + item % STAGES * ITEM_BYTES));
        const unsigned long long q_desc = tc_desc_k<BLOCK>(smem_u32(smem + (split ? 0 : slot) * Shape::Q_BYTES));
        const unsigned tmem_s = tmem_base + slot * TC_BN;
        if (leader) {
#pragma unroll
          for (int k = 0; k < HD / 16; ++k) {
            const unsigned long long step = ((k / (BLOCK / 16)) * BLOCK_BYTES + (k % (BLOCK / 16)) * 32) >> 4;
            tc_mma(tmem_s, q_desc + step, k_desc + step, IDESC_QK, k > 0 ? 1u : 0u);
          }
          tc_commit(&s_full[slot]);
          // A stage of keys alone is free as soon as the last slot's products that read it are complete.
          if (!SHARED && (split || slot == 1)) tc_commit(&kv_empty[item % STAGES]);
          if (trace && slot == 0 && i < 64) trace[4 * i] = tc_timer_ns();
        }
        return true;
      };
      bool ok = arrived(q_full, 0);
      if (ok && count0 > 0) ok = issue_scores(0, 0);
      if (ok && count1 > 0) ok = issue_scores(1, 0);
      for (int i = 0; i < count0 && ok; ++i) {
#pragma unroll
        for (int slot = 0; slot < 2; ++slot) {
          const int count = slot == 0 ? count0 : count1;
          if (!ok || i >= count) continue;
          const int item = value_item(slot_tile(slot, i));
          ok = landed(item);
          const unsigned tmem_o = tmem_base + TC_O_COLUMN + slot * TC_VD, tmem_p = tmem_base + slot * TC_BN;
          const unsigned long long v_desc = tc_desc_mn<BLOCK>(smem_u32(ring + item % STAGES * ITEM_BYTES));
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            ok = ok && arrived(&p_full[2 * slot + half], i & 1);
            if (!ok) continue;
            tc_fence_after_sync();
            if (leader) {
#pragma unroll
              for (int k = 4 * half; k < 4 * half + 4; ++k)
                tc_mma_ts_if(tmem_o, tmem_p + k * 8, v_desc + ((k * KSTEP) >> 4), IDESC_PV, k > 0 || i > 0 ? 1u : 0u);
            }
          }
          if (!ok) continue;
          if (leader) {
            if (split || slot == 1) tc_commit(&kv_empty[item % STAGES]);
            if (i + 1 >= count) tc_commit(&o_done[slot]);
            if (trace && slot == 0 && i < 64) trace[4 * i + 3] = tc_timer_ns();
          }
          // S of the slot's next tile overwrites these probabilities: the tensor core takes its work in the order of issue.
          if (i + 1 < count) ok = issue_scores(slot, i + 1);
        }
      }
      if (!ok) give_up(-3);
    }
  } else {
    // --------------------------------------------------------------------------- the softmax
    const int slot = warp >> 2, r = threadIdx.x & (TC_BM - 1);
    const int head = split ? head0 : head0 + slot;
    // The queries, rows past the tile's tokens zero: a slot's head each, or half of the one head's values each.
    {
      const uint4* src = reinterpret_cast<const uint4*>(a.q + (static_cast<size_t>(tok0 + (r < n_tok ? r : 0)) * a.nh + head) * HD);
      unsigned char* dst = smem + (split ? 0 : slot) * Shape::Q_BYTES;
      constexpr int HALF = CHUNKS / 2;
      const int from = split && slot == 1 ? HALF : 0, until = split && slot == 0 ? HALF : CHUNKS;
      const int turn = kv_swizzle(r, CHUNKS);
#pragma unroll
      for (int c0 = 0; c0 < CHUNKS; c0 += HALF) {
        if (c0 < from || c0 >= until) continue;
        uint4 v[HALF];
#pragma unroll
        for (int c = 0; c < HALF; ++c) v[c] = r < n_tok ? src[c0 + c] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int c = 0; c < HALF; ++c) {
          const int stored = (c0 + c) ^ turn;
          *reinterpret_cast<uint4*>(dst + (stored / BLOCK_CHUNKS) * BLOCK_BYTES + r * (BLOCK * 2) + (stored % BLOCK_CHUNKS) * 16) = v[c];
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(q_full);
    }
    const unsigned lane_base = static_cast<unsigned>((warp & 3) * 32) << 16;
    const unsigned tmem_s = tmem_base + lane_base + slot * TC_BN, tmem_o = tmem_base + lane_base + TC_O_COLUMN + slot * TC_VD;
    const int qp = ctx + q0 + r;
    float m_used = -INFINITY, l_run = 0.0f;
    const bool capped = !BIASED_SCORES && a.softcap_log2 > 0.0f;
    const float r1 = BIASED_SCORES ? a.bias_r1[head] : 0.0f, r2 = BIASED_SCORES ? a.bias_r2[head] : 0.0f;
    bool failed = false;
    // With a chunk: the last position that this row's window and chunk leave out, and the first key that all rows of the CTA see.
    int passed = -1, open_from = 0;
    if (CHUNKED) {
      if (a.window > 0) {
        passed = qp - a.window;
        open_from = ctx + q0 + TC_BM - a.window;
      }
      if (a.chunk > 0) {
        passed = max(passed, qp / a.chunk * a.chunk - 1);
        open_from = max(open_from, (ctx + q0 + TC_BM - 1) / a.chunk * a.chunk);
      }
    }
    const int count = slot_tiles(slot);
    for (int i = 0; i < count; ++i) {
      const int j = slot_tile(slot, i), k0 = tile_start(j);
      const bool in_kept = KEPT && j < kept_tiles;
      // Whether to go on is decided by the warp as one: the tensor-memory instructions below are
      // for all of its lanes together.
      if (!__all_sync(0xffffffffu, wait(&s_full[slot], i & 1))) { give_up(-4); failed = true; break; }
      tc_fence_after_sync();
      if (trace && threadIdx.x == 0 && i < 64) trace[4 * i + 1] = tc_timer_ns();
      // Most tiles lie wholly in every row's past (and inside its window): no mask to evaluate.
      const bool all_see = CHUNKED ? k0 >= open_from : a.window == 0 || k0 > ctx + q0 + TC_BM - 1 - a.window;
      const bool open_tile = k0 + TC_BN - 1 <= ctx + q0 && (in_kept ? k0 + TC_BN <= kept : k0 >= lo && all_see);
      const int at = qp - k0;
      const int after = in_kept ? -1 : CHUNKED ? passed - k0 : a.window > 0 ? qp - a.window - k0 : -(1 << 30);
      const int last = min(qp, run_hi(j) - 1) - k0, first = max(run_lo(j) - k0, after + 1);
      const float raw_max = open_tile ? tc_row_max<false, BIASED_SCORES>(tmem_s, last, first, a.scale_log2, at, r1, r2)
                                      : tc_row_max<true, BIASED_SCORES>(tmem_s, last, first, a.scale_log2, at, r1, r2);
      // The scale is positive and the bound grows with its argument: the largest raw score gives the largest exponent.
      const float row_max = capped ? a.softcap_log2 * tanh_from_exp2(raw_max * a.scale_over_cap) : BIASED_SCORES ? raw_max : raw_max * a.scale_log2;
      const bool grow = raw_max > -INFINITY && (row_max > m_used + TC_RESCALE_THRESHOLD || m_used == -INFINITY);
      if (__any_sync(0xffffffffu, grow)) {
        // Some row of the warp moves its shift: every lane takes part in the tensor-memory
        // instructions, rows that stay multiply by one.
        const float factor = grow ? exp2f(m_used - row_max) : 1.0f;       // 0 for a row's first keys
        if (grow) m_used = row_max;
        l_run *= factor;
        if (i > 0) {
          // O holds the tiles before this one: their products were issued before this tile's S, which is complete, and this
          // tile's product waits for this warp's arrival below.
#pragma unroll 1
          for (int c4 = 0; c4 < TC_VD / 32; ++c4) {
            unsigned v[32];
            tmem_ld32(tmem_o + c4 * 32, v);
            tmem_wait_ld32(v);
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * factor);
            tmem_st32(tmem_o + c4 * 32, v);
          }
          tc_wait_st();
        }
      }
      const float neg_shift = m_used == -INFINITY ? 0.0f : -m_used;
      // Two probabilities a column, as the second product reads its A operand from tensor memory, over columns of S
      // that have been read; the product of the first 64 positions runs while the others are worked on.
      unsigned long long sums[4] = {0, 0, 0, 0};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        unsigned words[32];
        if (capped) {
          tc_exponentials<true, true>(tmem_s, 64 * half, words, sums, a.scale_over_cap, neg_shift, last, first, a.softcap_log2);
        } else if (open_tile) {
          tc_exponentials<false, false>(tmem_s, 64 * half, words, sums, BIASED_SCORES ? 1.0f : a.scale_log2, neg_shift, last, first, 0.0f);
        } else {
          tc_exponentials<true, false>(tmem_s, 64 * half, words, sums, BIASED_SCORES ? 1.0f : a.scale_log2, neg_shift, last, first, 0.0f);
        }
        tmem_st32(tmem_s + 32 * half, words);
        tc_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&p_full[2 * slot + half]);
      }
      float sum_lo, sum_hi;
      unpack_f32x2(add_f32x2(add_f32x2(sums[0], sums[1]), add_f32x2(sums[2], sums[3])), sum_lo, sum_hi);
      l_run += sum_lo + sum_hi;
      if (trace && threadIdx.x == 0 && i < 64) trace[4 * i + 2] = tc_timer_ns();
    }
    if (!failed && count > 0 && !__all_sync(0xffffffffu, wait(&o_done[slot], 0))) { give_up(-6); failed = true; }
    tc_fence_after_sync();
    // One more exponential: the sink, relative to the shift the row's sums were formed with (both in powers of two).
    auto with_sink = [&](float sum, float shift) {
      return a.sinks != nullptr && shift > -INFINITY ? sum + exp2f(a.sinks[head] * 1.4426950408889634f - shift) : sum;
    };
    // Each warp puts 32 rows x 64 columns into shared memory, 16-byte pieces permuted by the row so that neither the writes
    // (a thread a row) nor the reads (eight threads a row) meet in a bank, and then writes whole 128-byte row pieces, four rows
    // an instruction.  (A thread storing its own row's pieces touches 32 rows with every instruction, which cost 1.4 us a CTA.)
    auto store_half = [&](unsigned char* stage_out, int half, auto value) {
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        unsigned v[32];
        tmem_ld32(tmem_o + half * 64 + cc * 32, v);
        tmem_wait_ld32(v);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = value(__uint_as_float(v[8 * q4 + e]), cc * 32 + 8 * q4 + e);
          uint4 o4;
          o4.x = pack_bf16(f[0], f[1]);
          o4.y = pack_bf16(f[2], f[3]);
          o4.z = pack_bf16(f[4], f[5]);
          o4.w = pack_bf16(f[6], f[7]);
          *reinterpret_cast<uint4*>(stage_out + lane * 128 + (((cc * 4 + q4) ^ (lane & 7)) << 4)) = o4;
        }
      }
      __syncwarp();
      const int row_base = (warp & 3) * 32, piece = lane & 7;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int rr = 4 * i + (lane >> 3);
        if (row_base + rr < n_tok) {
          const uint4 o4 = *reinterpret_cast<const uint4*>(stage_out + rr * 128 + ((piece ^ (rr & 7)) << 4));
          *reinterpret_cast<uint4*>(a.out + (static_cast<size_t>(tok0 + row_base + rr) * a.nh + head) * HD + half * 64 + piece * 8) = o4;
        }
      }
      __syncwarp();
    };
    if (!split) {
      // The slot's own queries are no longer read: its S are complete.
      if (!failed) {
        const float l_row = with_sink(l_run, m_used), inv = l_row > 0.0f ? 1.0f / l_row : 0.0f;
        unsigned char* stage_out = smem + slot * Shape::Q_BYTES + (warp & 3) * 4096;
#pragma unroll 1
        for (int half = 0; half < 2; ++half) store_half(stage_out, half, [&](float o, int) { return count > 0 ? o * inv : 0.0f; });
      }
    } else {
      // The slots' results meet: each hands the other the half of its columns that the other writes out.
      auto slots_meet = [] { asm volatile("bar.sync 1, 256;\n" ::: "memory"); };
      note[slot][r][0] = m_used;
      note[slot][r][1] = l_run;
      slots_meet();                   // every product of both slots is complete (or the launch has failed): all of shared memory is free
      const float m_other = note[slot ^ 1][r][0], m = fmaxf(m_used, m_other);
      const float mine = m_used > -INFINITY ? exp2f(m_used - m) : 0.0f, others = m_other > -INFINITY ? exp2f(m_other - m) : 0.0f;
      float4* const give = reinterpret_cast<float4*>(smem + slot * 32768), * const take = reinterpret_cast<float4*>(smem + (slot ^ 1) * 32768);
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        unsigned v[32];
        tmem_ld32(tmem_o + (slot ^ 1) * 64 + cc * 32, v);
        tmem_wait_ld32(v);
#pragma unroll
        for (int q4 = 0; q4 < 8; ++q4)
          give[(cc * 8 + q4) * TC_BM + r] = make_float4(__uint_as_float(v[4 * q4]), __uint_as_float(v[4 * q4 + 1]),
                                                        __uint_as_float(v[4 * q4 + 2]), __uint_as_float(v[4 * q4 + 3]));
      }
      slots_meet();
      const float l_row = with_sink(l_run * mine + note[slot ^ 1][r][1] * others, m), inv = l_row > 0.0f ? 1.0f / l_row : 0.0f;
      const float f_mine = mine * inv, f_others = others * inv;
      if (!abort_flag && !failed)
        store_half(smem + 65536 + warp * 4096, slot, [&](float o, int column) {
          const float other = reinterpret_cast<const float*>(&take[(column >> 2) * TC_BM + r])[column & 3];
          return (count > 0 ? o * f_mine : 0.0f) + (slot_tiles(slot ^ 1) > 0 ? other * f_others : 0.0f);
        });
    }
  }

  // Everybody meets here on every path, and the warp that took the tensor memory gives it back.
  tc_fence_before_sync();
  __syncthreads();
  if (abort_flag) let_copies_land();
  if (warp == TC_MMA_WARP) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TC_TMEM_COLUMNS);
  }
}

// The cache [pages][2][nkv][page_size][hd] as rows of hd bfloat16; a box is one block of values (TcShape) by one
// page's rows (at most a tile's 128).  Maps are kept: the same caches come back every step.
bool cache_tensor_map(const __nv_bfloat16* cache, long long rows, int hd, int block, int box_rows, CUtensorMap* out) {
  static std::mutex mutex;
  static std::map<std::tuple<const void*, long long, int, int>, CUtensorMap> kept;
  std::lock_guard<std::mutex> lock(mutex);
  const auto key = std::make_tuple(static_cast<const void*>(cache), rows, hd, box_rows);
  const auto found = kept.find(key);
  if (found != kept.end()) {
    *out = found->second;
    return true;
  }
  const EncodeTiled encode = tensor_map_encoder();
  if (encode == nullptr) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(hd), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(hd) * 2};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(block), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t element_strides[2] = {1, 1};
  if (encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(cache), dims, strides, box, element_strides,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (kept.size() > 4096) kept.clear();
  kept.emplace(key, *out);
  return true;
}

// How many tiles, from the longest on, run a head a CTA (see the top): all where even so every CTA gets an SM at once, or where
// pairs of heads would not fill the SMs and rows are long, so that the longest chain is the launch's time; else none.  `tile_rows`:
// the rows that these tiles come from (a step's decoding rows do not count: 2048 tokens beside four of them took 43 us in pairs).  (us, heads
// singly / in pairs: one row of 300 tokens, 16/8 heads 11.3 / 13.9; one of 2048 33 / 43; 552 tokens behind 2048 beside a row
// of 1496 39 / 51; but 16 rows of 128 35 / 23, 3000 tokens in a window of 1024 54 / 46, rows of 1531, 500 and 17 tokens, 32/8
// heads, 53 / 41.  Halfway between, 25 to 75 % of the tiles, was never the best.)
int tc_split_tiles(int nh, int nkv, int n_tiles, int tile_rows, int sms) {
  if (nh / nkv % 2 != 0) return n_tiles;
  const long long single = static_cast<long long>(nh) * n_tiles;
  return single <= sms || (single / 2 <= sms && n_tiles >= 4LL * tile_rows) ? n_tiles : 0;
}

template <int FORM, int HD, bool SHARED>
int prefill_tc_launch(PrefillTcArgs& a, long long cache_rows, int page_size, cudaStream_t stream) {
  using Shape = TcShape<HD, SHARED>;
  a.tiled = cache_rows < (1LL << 31) &&
            cache_tensor_map(a.kv_cache, cache_rows, HD, Shape::BLOCK, page_size < TC_BN ? page_size : TC_BN, &a.cache_map) ? 1 : 0;
  auto kernel = paged_prefill_tc_kernel<FORM, HD, SHARED>;
  if (cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM))) return ERR_CUDA;
  const long long ctas = static_cast<long long>(a.n_split) * a.nh + static_cast<long long>(a.n_tiles - a.n_split) * (a.nh / 2);
  if (ctas >= (1LL << 31)) return ERR_UNSUPPORTED;
  return launch_dependent(kernel, dim3(static_cast<unsigned>(ctas)), dim3(TC_THREADS), Shape::SMEM, stream, false, a);
}

}  // namespace zb

using namespace zb;

namespace zb {
inline int*& prefill_tc_trace() {
  static int* buffer = nullptr;
  return buffer;
}
}  // namespace zb

// Timelines for later launches of zb_paged_prefill_tc: null (off) or 512 ints on the device (see
// PrefillTcArgs::trace; the second half: per tile, when the first loader thread began the issue of its keys
// and of its values).
ZB_API int zb_paged_prefill_tc_set_trace(int* buffer) {
  prefill_tc_trace() = buffer;
  return OK;
}

// 1 if zb_paged_prefill_tc takes this shape.  Rows of 160 values are keys and values at once, of which the result holds
// the first 128 (`keys_only` with a `value_dim` of 128), without chunk, kept tokens or a distance bias.
ZB_API int zb_paged_prefill_tc_supported(int nh, int nkv, int hd, int value_dim, int keys_only, int dtype, int page_size) {
  if (dtype != DTYPE_BF16 || nkv <= 0 || nh <= 0 || nh % nkv != 0 || nh > 65535) return 0;
  if (page_size < 8 || (page_size & (page_size - 1)) != 0) return 0;
  return hd == 128 || (hd == 160 && value_dim == TC_VD && keys_only) ? 1 : 0;
}

// Attention of the tiles' tokens (tiles of 128 new tokens of one request) over their requests'
// pages; writes those tokens' rows of `out`.  Arguments as zb_paged_prefill_masked:
// `tile_rows`: how many of the `num_rows` rows have tiles in the list;
// `softcap` > 0 bounds the scaled scores by softcap * tanh(. / softcap); `keys_only`: a page holds keys alone
// and they are the values too; `value_dim`: how many values of a row of `out` are wanted (the others may stay as they are);
// `sinks` (null, or one float32 per query head) join the softmax's denominator;
// `bias_r1`, `bias_r2` (null, or one float32 per query head each; not with a softcap, a chunk or kept tokens) bias the distances;
// `keep_first` (with a window): keys below this position stay visible.
ZB_API int zb_paged_prefill_tc_masked(void* out, const void* q, const void* kv_cache, const int* block_table,
                                      int max_blocks, int page_size, int num_pages, int num_rows, const int* tile_row,
                                      const int* tile_q0, int n_tiles, int tile_rows, const int* row_q_start, const int* row_q_len,
                                      const int* row_ctx, int nh, int nkv, int hd, int window, int value_dim, int chunk, int keep_first,
                                      float scale, float softcap, int keys_only, const float* sinks, const float* bias_r1,
                                      const float* bias_r2, int* status, void* stream) {
  if ((bias_r1 == nullptr) != (bias_r2 == nullptr) || (bias_r1 != nullptr && softcap > 0.0f) || n_tiles < 0 || page_size <= 0 || window < 0 || softcap < 0.0f ||
      chunk < 0 || keep_first < 0 || (keep_first > 0 && window <= 0) || (bias_r1 != nullptr && (keep_first > 0 || chunk > 0)))
    return ERR_BAD_ARGUMENT;
  if (!zb_paged_prefill_tc_supported(nh, nkv, hd, value_dim, keys_only, DTYPE_BF16, page_size)) return ERR_UNSUPPORTED;
  const bool rows_are_both = hd != 128;
  if (rows_are_both && (bias_r1 != nullptr || chunk > 0 || keep_first > 0)) return ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(q) % 16 != 0 || reinterpret_cast<uintptr_t>(out) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(kv_cache) % 16 != 0)
    return ERR_BAD_ARGUMENT;
  if (n_tiles == 0) return OK;
  if (tile_rows <= 0) return ERR_BAD_ARGUMENT;
  if (n_tiles > 65535) return ERR_UNSUPPORTED;
  int device = 0, sms = 0;
  if (cuda_failed(cudaGetDevice(&device)) || cuda_failed(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device))) return ERR_CUDA;
  PrefillTcArgs a;
  a.n_tiles = n_tiles;
  a.n_split = tc_split_tiles(nh, nkv, n_tiles, tile_rows, sms);
  a.q = static_cast<const __nv_bfloat16*>(q);
  a.out = static_cast<__nv_bfloat16*>(out);
  a.kv_cache = static_cast<const __nv_bfloat16*>(kv_cache);
  a.block_table = block_table; a.tile_row = tile_row; a.tile_q0 = tile_q0;
  a.row_q_start = row_q_start; a.row_q_len = row_q_len; a.row_ctx = row_ctx;
  a.max_blocks = max_blocks; a.num_pages = num_pages; a.num_rows = num_rows;
  a.page_shift = 0;
  while ((1 << a.page_shift) < page_size) ++a.page_shift;
  a.nh = nh; a.nkv = nkv; a.window = window; a.chunk = chunk; a.keep_first = keep_first;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.softcap_log2 = softcap * 1.4426950408889634f;
  a.scale_over_cap = softcap > 0.0f ? scale / softcap : 0.0f;
  a.keys_only = keys_only;
  a.sinks = sinks;
  a.bias_r1 = bias_r1; a.bias_r2 = bias_r2;
  a.status = status;
  a.trace = prefill_tc_trace();
  const long long cache_rows = static_cast<long long>(num_pages) * (keys_only ? 1 : 2) * nkv * page_size;
  const auto s = static_cast<cudaStream_t>(stream);
  if (rows_are_both) return prefill_tc_launch<TC_FORM_PLAIN, 160, true>(a, cache_rows, page_size, s);
  if (bias_r1 != nullptr) return prefill_tc_launch<TC_FORM_BIASED, 128, false>(a, cache_rows, page_size, s);
  if (keep_first > 0) return prefill_tc_launch<TC_FORM_KEPT, 128, false>(a, cache_rows, page_size, s);
  if (chunk > 0) return prefill_tc_launch<TC_FORM_CHUNKED, 128, false>(a, cache_rows, page_size, s);
  return prefill_tc_launch<TC_FORM_PLAIN, 128, false>(a, cache_rows, page_size, s);
}

ZB_API int zb_paged_prefill_tc(void* out, const void* q, const void* kv_cache, const int* block_table, int max_blocks,
                               int page_size, int num_pages, int num_rows, const int* tile_row, const int* tile_q0,
                               int n_tiles, const int* row_q_start, const int* row_q_len, const int* row_ctx, int nh,
                               int nkv, int hd, int window, float scale, int* status, void* stream) {
  return zb_paged_prefill_tc_masked(out, q, kv_cache, block_table, max_blocks, page_size, num_pages, num_rows, tile_row,
                                    tile_q0, n_tiles, num_rows, row_q_start, row_q_len, row_ctx, nh, nkv, hd, window, hd, 0, 0, scale, 0.0f, 0,
                                    nullptr, nullptr, nullptr, status, stream);
}
