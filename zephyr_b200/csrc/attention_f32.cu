// Paged causal attention of the true 32-bit path for rows that bring several tokens, on the fifth-generation tensor cores: every
// product of two float32 values and their float32 sum, no TF32.
//
// A float32 value is three bfloat16 values, hi + mid + lo, to its last bit; both products, scores Q K^T and weights times values, are
// formed from six products of parts (gemm_tc_f32.cu has the why): hi hi in a sum of its own, 8 steps of the tensor core long for a
// score and 4 for the values, which is added to the row's total in registers with float32's rounding; the five small ones in another.
// Error against 64 bits, 700 tokens of 16 heads over 8 of 128: 2.1e-7 (3.6e-7 by multiply-adds), two tokens behind 600 2.9e-7 (6.0e-7).
//
// One CTA = 128 (token, head) pairs of neighbouring tokens and one key/value head, the tensor core's rows, against F_KEYS keys at a
// time.  Eight warps: a thread owns a row and, of a step, half of the keys' scores and half of the output's columns.  A step:
//   wait for the scores; their maximum (both halves meet in shared memory) and the weights; the next step's keys, split, to shared
//   memory, upon which one thread of a ninth warp issues the next step's scores; the weighted values of the step before, added to the
//   totals; this step's values, split, to shared memory and the weights' parts to tensor memory, where the scores lay, upon which
//   the weighted values of this step are issued.
// Keys and values of the next step are on their way in registers meanwhile.  What does not lie in [lo, hi) comes as zeros.
// All are split times 2^39 (gemm_tc_f32.cu), which the scores' scale and the totals take back.  Scores that are not finite then are formed
// again by multiply-adds; a value beyond 2^40, or not finite, is left out of the product and added by hand to the rows whose weight
// for it is not zero, so that it stays with those that see it.
// Bound by the eight warps' part of a step, some 6500 cycles, of which the tensor cores' 72 products take 3900: scores' reads 400, maximum
// and weights 1800, both splits 1600, values' sums 450, fetches 800.  (With the maximum taken under a branch per score, and every thread
// looking its keys' pages up by divisions, 12000; registers spilled to an L1 of the 28 KB that the CTA's shared memory leaves,
// 7500.)
// 700 tokens, 16 heads over 8 of 128: 54 us (multiply-adds on CUDA cores, 64 pairs a CTA, 122); 4000 tokens 428 (1680); two tokens
// behind a context of 600 44 (97), two tokens of a new prompt 12.4 (17.5), eight rows of sixteen 12.8 (24); 700 tokens of width 64 40 (72).
// (Splitting without the factor, which loses the last bits of values below 2^-110: 52.6 and 419.)
// Every row with several tokens runs here, so that its result hangs on that row alone.
//
// Masks: causal, a window, a chunk (key and query in the same run of `chunk` positions); `sinks` join the softmax's
// denominators; `softcap` > 0 bounds the scaled scores.  Keys and values have one width, a multiple of 4 up to 128.
// Every wait is bounded and reports instead of hanging; tensor memory is given back on every path.
#include <initializer_list>

#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

namespace zb {

constexpr int F_ROWS = 128;     // (token, head) pairs of a CTA
constexpr int F_GROUP = 64;     // query heads a key/value head may have
constexpr int F_KEYS = 64;      // keys of a step
constexpr int F_WARPS = 8;       // and four more, of which one issues the products and one looks the keys' places up
constexpr int F_PLACES = 4;     // steps whose keys' places are kept
constexpr int F_THREADS = (F_WARPS + 4) * 32;
constexpr int F_WAIT_LIMIT = 1 << 18;
constexpr int F_WORKER_REGISTERS = 216, F_OTHER_REGISTERS = 72;       // of 168 at launch: 256 x 216 + 128 x 72 = 384 x 168

struct AttentionF32Args {
  const float* q;           // [T, nh * d]
  float* out;               // [T, nh * d]
  const float* kv_cache;    // pages {[nkv][page_size][d] keys, the same of values}
  const int* block_table;   // [R, max_blocks]
  const int* tile_row;      // [n_tiles], by the number of keys a tile sees, fewest first
  const int* tile_q0;
  const int* row_q_start;
  const int* row_q_len;
  const int* row_ctx;
  int max_blocks, page_size, num_pages, num_rows, n_tiles;
  int nh, nkv, d, window, chunk, tile_tokens, cta_tokens, subs;
  float scale, softcap;
  const float* sinks;       // null, or [nh]
  int* status;
};

// D: the padded width, 64 or 128.  Rows lie as blocks of 64 values, [part][D / 64][rows][64] bfloat16, 128-byte swizzle; a block's 16-byte
// piece c holds its values 4 c .. 4 c + 3 and 32 + 4 c .. 35 + 4 c (queries, keys and values alike).
template <int D>
struct AttentionF32Shape {
  static constexpr int BLOCKS = D / 64;
  static constexpr int Q_PART = BLOCKS * F_ROWS * 128, K_PART = BLOCKS * F_KEYS * 128;
  static constexpr int K_BYTES = 3 * K_PART > F_KEYS * F_ROWS * 4 ? 3 * K_PART : F_KEYS * F_ROWS * 4;      // or all weights of a step
  static constexpr int SMEM = 3 * (Q_PART + K_PART) + K_BYTES + 1024;
  static constexpr int O_COLUMN = 256;      // tensor memory: two steps of 64 scores and 64 small sums (then the weights' parts), the values' two sums
  static_assert(SMEM <= 227 * 1024 - 2048, "fits an SM's shared memory");
};

// The values of a CTA's columns as MN-major operand: rows of keys, groups of 8 of them 1024 bytes apart, blocks of 64 values F_KEYS * 128.
__device__ __forceinline__ unsigned long long f32_values_desc(unsigned smem_address) {
  return static_cast<unsigned long long>((smem_address >> 4) & 0x3FFFu) | (static_cast<unsigned long long>(F_KEYS * 128 >> 4) << 16) |
         (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// A barrier of the eight warps; true if `any` holds for one of their threads.
__device__ __forceinline__ bool f32_workers_any(bool any) {
  unsigned r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.pred q, 1, 256, p;\nselp.u32 %0, 1, 0, q;\n}\n"
               : "=r"(r) : "r"(static_cast<unsigned>(any)) : "memory");
  return r != 0;
}

// Eight values (two runs of four) as 16-byte pieces of their three parts, times 2^39.
__device__ __forceinline__ void f32_store_parts(float4 p, float4 q, unsigned char* to, int part) {
  unsigned hi[4], mid[4], lo[4];
  const float x[4] = {p.x, p.z, q.x, q.z}, y[4] = {p.y, p.w, q.y, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) three_parts_scaled(x[i], y[i], hi[i], mid[i], lo[i]);
  *reinterpret_cast<uint4*>(to) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  *reinterpret_cast<uint4*>(to + part) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
  *reinterpret_cast<uint4*>(to + 2 * part) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

constexpr float F_LARGEST = 1.0995116e12f;      // 2^40: 64 of them times weights of one stay below float32's end, both times 2^39
__device__ __forceinline__ float zero_if_wild(float x) { return fabsf(x) <= F_LARGEST ? x : 0.0f; }

template <int D>
__global__ void __launch_bounds__(F_THREADS, 1) paged_attention_f32_kernel(const AttentionF32Args a) {
  using Shape = AttentionF32Shape<D>;
  constexpr int Q_PART = Shape::Q_PART, K_PART = Shape::K_PART, COLUMNS = D / 2, PER = F_KEYS * Shape::BLOCKS / 32;
  extern __shared__ unsigned char f_smem_raw[];
  __shared__ unsigned long long k_full, s_done, pv_full, o_done, place_full[F_PLACES], place_empty[F_PLACES];
  __shared__ long long place_s[F_PLACES][F_KEYS];        // where a step's keys begin in the cache, or -1
  __shared__ float half_of_row[2][F_ROWS];
  __shared__ unsigned tmem_base_s;
  __shared__ volatile int failed;
  unsigned char* const q_s = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(f_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  unsigned char* const k_s = q_s + 3 * Q_PART;
  unsigned char* const v_s = k_s + Shape::K_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(&k_full, F_WARPS);
    mbar_init(&s_done, 1);
    mbar_init(&pv_full, F_WARPS);
    mbar_init(&o_done, 1);
    for (int i = 0; i < F_PLACES; ++i) {
      mbar_init(&place_full[i], 1);
      mbar_init(&place_empty[i], F_WARPS);
    }
    failed = 0;
    fence_barrier_init();
  }
  if (warp == F_WARPS) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const unsigned tmem_base = tmem_base_s;
  wait_for_prior_grids();
  let_dependents_launch();

  // The last tiles of the list see the most keys and run first.
  const int kvh = blockIdx.x % a.nkv, place = blockIdx.x / a.nkv;
  const int tile = a.n_tiles - 1 - place / a.subs, sub = a.subs - 1 - place % a.subs;
  const int row = a.tile_row[tile], q0 = a.tile_q0[tile] + sub * a.cta_tokens;
  const int g = a.nh / a.nkv, d = a.d, chunks = d / 4;      // chunks: 16-byte pieces of a row
  int n_tok = 0;
  if (row < 0 || row >= a.num_rows) {
    if (tid == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, row, tile);
  } else {
    n_tok = min(min(a.cta_tokens, a.tile_tokens - sub * a.cta_tokens), a.row_q_len[row] - q0);
  }
  // Keys any row of this CTA may see: [lo, hi).
  const int ctx = n_tok > 0 ? a.row_ctx[row] : 0, tok0 = n_tok > 0 ? a.row_q_start[row] + q0 : 0, rows = n_tok * g;
  const int hi = ctx + q0 + n_tok;
  int lo = a.window > 0 ? max(0, ctx + q0 - a.window + 1) : 0;
  if (a.chunk > 0) lo = max(lo, (ctx + q0) / a.chunk * a.chunk);
  const int begin = lo / F_KEYS * F_KEYS, steps = n_tok > 0 ? (hi - begin + F_KEYS - 1) / F_KEYS : 0;

  auto arrived = [&](unsigned long long* bar, unsigned parity, int where) -> bool {
    bool ok = false;
    for (int i = 0; i < F_WAIT_LIMIT && !ok; ++i) {
      ok = mbar_try_wait(bar, parity);
      if (!ok && (i & 255) == 255 && failed) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0 && !failed) report(a.status, STATUS_BARRIER_TIMEOUT, where, tile);
      failed = 1;
    }
    return ok;
  };

  const size_t page_elems = static_cast<size_t>(2) * a.nkv * a.page_size * d;
  const size_t value_part = static_cast<size_t>(a.nkv) * a.page_size * d;
  const int* const table = a.block_table + static_cast<size_t>(n_tok > 0 ? row : 0) * a.max_blocks;
  // Where position `pos` of this head begins in the cache; -1 outside [lo, hi) (its rows are zeros) or if its page
  // is none (reported).
  auto locate = [&](int pos) -> long long {
    if (pos < lo || pos >= hi) return -1;
    const int block = pos / a.page_size;
    const int page = block < a.max_blocks ? table[block] : -1;
    if (page <= 0 || page >= a.num_pages) {
      report(a.status, STATUS_PAGE_OUT_OF_RANGE, page, tok0);
      return -1;
    }
    return page * page_elems + (static_cast<size_t>(kvh) * a.page_size + pos % a.page_size) * d;
  };

  if (warp >= F_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(F_OTHER_REGISTERS));
    if (warp == F_WARPS) {
      constexpr unsigned IDESC_S = tc_idesc(false, F_KEYS), IDESC_O = tc_idesc(true, D);
      // The products of parts (of the first operand, of the second) behind hi hi, smallest first.
      constexpr int FIRST[5] = {2, 1, 0, 1, 0}, SECOND[5] = {0, 1, 2, 0, 1};
      const bool leader = elect_one();
      const unsigned long long q_desc = desc_k_major(smem_u32(q_s)), k_desc = desc_k_major(smem_u32(k_s)), v_desc = f32_values_desc(smem_u32(v_s));
      auto scores = [&](int i) -> bool {
        if (!arrived(&k_full, i & 1, i)) return false;
        tc_fence_after_sync();
        const unsigned s = tmem_base + (i & 1) * 128;
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < D / 16; ++k) {
            const unsigned long long q_k = q_desc + ((k / 4 * (F_ROWS * 128) + k % 4 * 32) >> 4), k_k = k_desc + ((k / 4 * (F_KEYS * 128) + k % 4 * 32) >> 4);
#pragma unroll
            for (int e = 0; e < 5; ++e)
              tc_mma(s + 64, q_k + (FIRST[e] * Q_PART >> 4), k_k + (SECOND[e] * K_PART >> 4), IDESC_S, (k | e) != 0 ? 1u : 0u);
            tc_mma(s, q_k, k_k, IDESC_S, k != 0 ? 1u : 0u);
          }
          tc_commit(&s_done);
        }
        return true;
      };
      bool ok = steps > 0 && scores(0);
      for (int i = 0; i < steps && ok; ++i) {
        if (i + 1 < steps) ok = scores(i + 1);
        ok = ok && arrived(&pv_full, i & 1, 1000000 + i);
        if (!ok) break;
        tc_fence_after_sync();
        const unsigned p = tmem_base + (i & 1) * 128, o = tmem_base + Shape::O_COLUMN;
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < F_KEYS / 16; ++k) {
            const unsigned p_k = p + 8 * k;
            const unsigned long long v_k = v_desc + (k * 2048 >> 4);
#pragma unroll
            for (int e = 0; e < 5; ++e)
              tc_mma_ts_if(o + D, p_k + 32 * FIRST[e], v_k + (SECOND[e] * K_PART >> 4), IDESC_O, (k | e) != 0 ? 1u : 0u);
            tc_mma_ts_if(o, p_k, v_k, IDESC_O, k != 0 ? 1u : 0u);
          }
          tc_commit(&o_done);
        }
      }
    } else if (warp == F_WARPS + 1) {
      for (int i = 0; i < steps; ++i) {
        if (!arrived(&place_empty[i % F_PLACES], (i / F_PLACES & 1) ^ 1, 5000000 + i)) break;
#pragma unroll
        for (int w = 0; w < 2; ++w) place_s[i % F_PLACES][lane + 32 * w] = locate(begin + i * F_KEYS + lane + 32 * w);
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&place_full[i % F_PLACES]);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(F_WORKER_REGISTERS));
    // Eight lanes bring a block of a row: lane c its pieces c and 8 + c of four values.  A thread has the keys r0 and r0 + 32 of a step.
    const int c = tid & 7, r0 = tid >> 3;
    const float* const pieces = a.kv_cache + 4 * (c ^ kv_swizzle(r0, chunks));      // (steps begin at multiples of 64)
    float4 keys[PER][2], values[PER][2];
    auto fetch = [&](float4 (&to)[PER][2], int step, size_t part) {
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const long long place = place_s[step % F_PLACES][r0 + 32 * w];
#pragma unroll
        for (int block = 0; block < Shape::BLOCKS; ++block)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int piece = 16 * block + 8 * half;
            to[2 * block + w][half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (place >= 0 && piece + c < chunks) to[2 * block + w][half] = *reinterpret_cast<const float4*>(pieces + place + part + 4 * piece);
          }
      }
    };
    bool ok = true;
    auto fetch_keys = [&](int step) {
      if (step >= steps) return;
      ok = arrived(&place_full[step % F_PLACES], step / F_PLACES & 1, 6000000 + step) && ok;
      fetch(keys, step, 0);
    };
    auto fetch_values = [&](int step) {          // (behind the same step's keys)
      if (step >= steps) return;
      fetch(values, step, value_part);
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&place_empty[step % F_PLACES]);
    };
    auto store = [&](const float4 (&from)[PER][2], unsigned char* to) {
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int key = r0 + 32 * (u & 1);
        f32_store_parts(from[u][0], from[u][1], to + (u >> 1) * (F_KEYS * 128) + key * 128 + ((c ^ (key & 7)) << 4), K_PART);
      }
    };
    // The queries; rows past the tile's tokens are zeros.
    fetch_keys(0);
#pragma unroll 4
    for (int e = r0; e < F_ROWS * Shape::BLOCKS; e += 32) {
      const int r = e % F_ROWS, block = e / F_ROWS;
      float4 x[2];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int piece = 16 * block + 8 * half + c;
        x[half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r < rows && piece < chunks)
          x[half] = *reinterpret_cast<const float4*>(a.q + (static_cast<size_t>(tok0 + r / g) * a.nh + kvh * g + r % g) * d + 4 * piece);
      }
      f32_store_parts(x[0], x[1], q_s + block * (F_ROWS * 128) + r * 128 + ((c ^ (r & 7)) << 4), Q_PART);
    }
    store(keys, k_s);
    fence_proxy_async();                // the tensor core reads the parts through the asynchronous proxy
    __syncwarp();
    if (lane == 0) tc_mbar_arrive(&k_full);
    fetch_values(0);
    fetch_keys(1);

    // This thread's row, and of it the keys 32 half .. + 31 of a step and the output's columns half * COLUMNS .. .
    const int half = warp >> 2, r = (warp & 3) * 32 + lane;
    const unsigned lane_base = static_cast<unsigned>((warp & 3) * 32) << 16;
    const int qpos = r < rows ? ctx + q0 + r / g : -1;
    int first = a.window > 0 ? max(0, qpos - a.window + 1) : 0;
    if (a.chunk > 0) first = max(first, qpos / a.chunk * a.chunk);
    float m = -INFINITY, l = 0.0f, acc[COLUMNS];
#pragma unroll
    for (int i = 0; i < COLUMNS; ++i) acc[i] = 0.0f;
    // acc = (acc + the weighted values of the last step) * by
    auto take_values = [&](float by) {
#pragma unroll
      for (int i0 = 0; i0 < COLUMNS; i0 += 16) {
        unsigned x[16], y[16];
        tmem_ld16(tmem_base + lane_base + Shape::O_COLUMN + half * COLUMNS + i0, x);
        tmem_ld16(tmem_base + lane_base + Shape::O_COLUMN + D + half * COLUMNS + i0, y);
        tmem_wait_ld16(x);
        tmem_wait_ld16(y);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i0 + i] = fmaf(__uint_as_float(x[i]) + __uint_as_float(y[i]), PARTS_UNSCALE, acc[i0 + i]) * by;
      }
    };
    // Column i of the thread's output is this value of the row.
    auto value_of = [&](int i) {
      const int n = half * COLUMNS + i;
      return n / 64 * 64 + n % 64 / 8 * 4 + (n & 3) + (n & 4) * 8;
    };
    for (int i = 0; i < steps; ++i) {
      const int k0 = begin + i * F_KEYS;
      ok = arrived(&s_done, i & 1, 2000000 + i) && ok;
      tc_fence_after_sync();
      const unsigned tmem_s = tmem_base + lane_base + (i & 1) * 128;
      const float score_scale = a.scale * PARTS_UNSCALE;
      float s[32];
      {
        float check = 0.0f;
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 16) {
          unsigned x[16], y[16];
          tmem_ld16(tmem_s + 32 * half + j0, x);
          tmem_ld16(tmem_s + 64 + 32 * half + j0, y);
          tmem_wait_ld16(x);
          tmem_wait_ld16(y);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            s[j0 + j] = (__uint_as_float(x[j]) + __uint_as_float(y[j])) * score_scale;
            check = fmaf(0.0f, s[j0 + j], check);
          }
        }
        if (check != 0.0f && r < rows) {        // some score is not finite
          const float* q = a.q + (static_cast<size_t>(tok0 + r / g) * a.nh + kvh * g + r % g) * d;
#pragma unroll 1
          for (int j = 0; j < 32; ++j) {
            const int pos = k0 + 32 * half + j;
            const long long place = pos >= first && pos <= qpos ? locate(pos) : -1;
            const float* k = a.kv_cache + place;
            float sum = 0.0f;
            for (int e = 0; place >= 0 && e < d; ++e) sum = fmaf(q[e], k[kv_element_index(e, pos, d, 4)], sum);
#pragma unroll
            for (int w = 0; w < 32; ++w)
              if (w == j && !(fabsf(s[w]) <= 3.4e38f)) s[w] = sum * a.scale;
          }
        }
      }
      if (a.softcap > 0.0f) {
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = a.softcap * tanhf(s[j] / a.softcap);
      }
      const int last_seen = qpos - k0 - 32 * half, first_seen = first - k0 - 32 * half;
      if (!__all_sync(0xffffffffu, last_seen >= 31 && first_seen <= 0)) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j > last_seen || j < first_seen) s[j] = -INFINITY;
      }
      float top4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 32; ++j) top4[j & 3] = fmaxf(top4[j & 3], s[j]);
      const float top = fmaxf(fmaxf(top4[0], top4[1]), fmaxf(top4[2], top4[3]));
      half_of_row[half][r] = top;
      unsigned largest = 0;             // twice the bits of the step's value that is the farthest from zero (a NaN is beyond infinity)
#pragma unroll
      for (int u = 0; u < PER; ++u)
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
          for (int e = 0; e < 4; ++e) largest = max(largest, __float_as_uint(reinterpret_cast<const float*>(&values[u][w])[e]) << 1);
      tc_fence_before_sync();           // (the halves' weights go where the other half's scores lay)
      const bool rare = f32_workers_any(!ok || largest > __float_as_uint(F_LARGEST) << 1);
      tc_fence_after_sync();
      const float new_m = fmaxf(m, fmaxf(top, half_of_row[half ^ 1][r]));
      // (a row that has seen no key yet keeps zeros: its weights are exp(-inf) of a finite difference)
      const float from = new_m == -INFINITY ? 0.0f : new_m, corr = expf(m - from);
      float sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        s[j] = expf(s[j] - from);
        sums[j & 3] += s[j];
      }
      l = fmaf(l, corr, (sums[0] + sums[1]) + (sums[2] + sums[3]));
      m = new_m;
      // The totals on the new maximum's scale, with the weighted values of the step before.
      auto rescale = [&] {
        if (i == 0) return;               // (zeros)
        ok = arrived(&o_done, (i - 1) & 1, 3000000 + i) && ok;
        tc_fence_after_sync();
        take_values(corr);
      };
      if (rare) {
        if (f32_workers_any(!ok)) break;
        rescale();                      // (what is added by hand is on that scale)
        // The keys' place is free (their scores are complete): the weights of all rows, [key][row].
        float* weights = reinterpret_cast<float*>(k_s);
#pragma unroll
        for (int j = 0; j < 32; ++j) weights[(32 * half + j) * F_ROWS + r] = s[j];
        f32_workers_any(false);
#pragma unroll 1
        for (int j = 0; j < F_KEYS; ++j) {
          const int pos = k0 + j;
          const float p = weights[j * F_ROWS + r];
          const long long place = p != 0.0f ? locate(pos) : -1;
          if (place < 0) continue;
          const float* v = a.kv_cache + place;
#pragma unroll
          for (int e = 0; e < COLUMNS; ++e) {
            const int at = value_of(e);
            const float x = at < d ? v[value_part + kv_element_index(at, pos, d, 4)] : 0.0f;
            if (zero_if_wild(x) != x) acc[e] = fmaf(p, x, acc[e]);
          }
        }
#pragma unroll
        for (int u = 0; u < PER; ++u)
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            float4& v = values[u][w];
            v = make_float4(zero_if_wild(v.x), zero_if_wild(v.y), zero_if_wild(v.z), zero_if_wild(v.w));
          }
        f32_workers_any(false);
      }
      if (i + 1 < steps) {
        store(keys, k_s);               // (free: this step's scores are complete)
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc_mbar_arrive(&k_full);
        fetch_keys(i + 2);
      }
      if (!rare) rescale();
      store(values, v_s);               // (free: the step before's products are complete)
      fence_proxy_async();
      {
        unsigned part[3][16];
#pragma unroll
        for (int j = 0; j < 16; ++j) three_parts_scaled(s[2 * j], s[2 * j + 1], part[0][j], part[1][j], part[2][j]);
#pragma unroll
        for (int e = 0; e < 3; ++e) tmem_st16(tmem_s + 32 * e + 16 * half, part[e]);
        tc_wait_st();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&pv_full);
      fetch_values(i + 1);
    }
    if (steps > 0) {
      ok = ok && arrived(&o_done, (steps - 1) & 1, 4000000);
      tc_fence_after_sync();
      take_values(1.0f);
      half_of_row[half][r] = l;
      ok = !f32_workers_any(!ok);
      if (ok && r < rows) {
        const int head = kvh * g + r % g;
        float denominator = half_of_row[0][r] + half_of_row[1][r], keep = 1.0f;
        if (a.sinks != nullptr) {
          // The sink joins the sum as one more exponential: rescale to the larger of the two maxima.
          const float sink = a.sinks[head], top = fmaxf(m, sink);
          keep = expf(m - top);
          denominator = denominator * keep + expf(sink - top);
        }
        const float inv = denominator > 0.0f ? keep / denominator : 0.0f;
        float* to = a.out + (static_cast<size_t>(tok0 + r / g) * a.nh + head) * d;
#pragma unroll
        for (int e = 0; e < COLUMNS; e += 4)
          if (value_of(e) < d)
            *reinterpret_cast<float4*>(to + value_of(e)) = make_float4(acc[e] * inv, acc[e + 1] * inv, acc[e + 2] * inv, acc[e + 3] * inv);
      }
    }
  }

  // Everybody meets here on every path, and the warp that took the tensor memory gives it back.
  tc_fence_before_sync();
  __syncthreads();
  if (failed) let_copies_land();        // (the products in flight)
  if (warp == F_WARPS) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int D>
static int attention_f32_launch(const AttentionF32Args& a, cudaStream_t s) {
  constexpr int smem = AttentionF32Shape<D>::SMEM;
  auto kernel = paged_attention_f32_kernel<D>;
  if (cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) return ERR_CUDA;
  return launch_dependent(kernel, dim3(a.n_tiles * a.subs * a.nkv), dim3(F_THREADS), smem, s, false, a);
}

}  // namespace zb

using namespace zb;

// 1 if the kernel takes heads of this width and this many query heads per key/value head.
ZB_API int zb_paged_attention_f32_supported(int nh, int nkv, int d) {
  return nh > 0 && nkv > 0 && nh % nkv == 0 && nh / nkv <= F_GROUP && d > 0 && d % 4 == 0 && d <= 128;
}

// Tiles of `tile_tokens` tokens, each cut among CTAs of F_ROWS (token, head) pairs.  q, out and the cache start on
// 16-byte boundaries.
ZB_API int zb_paged_attention_f32(float* out, const float* q, const float* kv_cache, const int* block_table, int max_blocks,
                                  int page_size, int num_pages, int num_rows, const int* tile_row, const int* tile_q0, int n_tiles,
                                  int tile_tokens, const int* row_q_start, const int* row_q_len, const int* row_ctx, int nh, int nkv,
                                  int d, int window, int chunk, float scale, float softcap, const float* sinks, int* status,
                                  void* stream) {
  if (page_size <= 0 || max_blocks <= 0 || n_tiles < 0 || tile_tokens <= 0 || window < 0 || chunk < 0 || softcap < 0.0f)
    return ERR_BAD_ARGUMENT;
  for (const void* p : {static_cast<const void*>(out), static_cast<const void*>(q), static_cast<const void*>(kv_cache)})
    if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return ERR_BAD_ARGUMENT;
  if (!zb_paged_attention_f32_supported(nh, nkv, d)) return ERR_UNSUPPORTED;
  if (n_tiles == 0) return OK;
  AttentionF32Args a;
  a.q = q; a.out = out; a.kv_cache = kv_cache; a.block_table = block_table; a.tile_row = tile_row; a.tile_q0 = tile_q0;
  a.row_q_start = row_q_start; a.row_q_len = row_q_len; a.row_ctx = row_ctx; a.max_blocks = max_blocks; a.page_size = page_size;
  a.num_pages = num_pages; a.num_rows = num_rows; a.n_tiles = n_tiles; a.nh = nh; a.nkv = nkv; a.d = d; a.window = window;
  a.chunk = chunk; a.tile_tokens = tile_tokens; a.cta_tokens = F_ROWS / (nh / nkv);
  a.subs = (tile_tokens + a.cta_tokens - 1) / a.cta_tokens;
  a.scale = scale; a.softcap = softcap; a.sinks = sinks; a.status = status;
  if (static_cast<long long>(n_tiles) * a.subs * nkv > 0x7fffffffLL) return ERR_UNSUPPORTED;
  auto s = static_cast<cudaStream_t>(stream);
  return d <= 64 ? attention_f32_launch<64>(a, s) : attention_f32_launch<128>(a, s);
}
