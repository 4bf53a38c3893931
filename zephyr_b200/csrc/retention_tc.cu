// Retention over runs of tokens on the fifth-generation tensor cores: per head, with one decay a per token,
//
//   S_t = a S_{t-1} + k_t v_t^T,   o_t = S_t^T q_t      (S [D key channels x V value channels], float32; q, k, v float32)
//
// A CTA owns a request, a head and 64 value columns and walks the request's tokens in pieces of 128 with the state in registers.  With S the
// state at a piece's start and n its tokens (counted from 0):
//
//   o_i   = a^(i+1) S^T q_i + sum_{j <= i} a^(i-j) (q_i . k_j) v_j
//   S    <- a^n S + sum_j a^(n-1-j) k_j v_j^T
//
// so a piece is four products on tcgen05 with 128 rows: scores Q K^T (128 columns), S^T q, K^T (a^(n-1-j) v) and the weights times V (64
// columns each); the weights go from the scores' place in tensor memory, through the registers of sixteen warps (a thread a row and a
// quarter of the columns), to tensor memory as the first operand of their product.  One thread of a seventeenth issues the products.
// Every operand is two bfloat16 values, hi hi + hi lo + lo hi (and lo lo), float32 sums, as in the walk in pieces of 64 (state_walk.cu: a
// relative error of about 2^-16 an operand); the state itself is only ever touched by float32 multiply-adds.
// q and k, which may still have to be turned by the tokens' positions, are split by retention_split_kernel for all pieces side by side, as
// the walk's bulk copies bring them to shared memory.
// In shared memory a row is 64 values side by side (128-byte swizzle), a head's 128 channels two such blocks; of a block's 16-byte piece
// c the values are 4 c .. 4 c + 3 and 32 + 4 c .. 35 + 4 c, for q, k and the state's rows alike.
// A value that is not finite is left out of the weights' product and added by hand to the outputs of the tokens from its own on, so that
// it stays with those; the state behind it is not finite either.
// Bound by shared memory: a piece is some 600 KB of the tensor cores' operand reads (products with 64 columns read their 128 rows again for
// each) and 300 KB of copies and stores, of the 128 bytes a cycle that there are; 8200 cycles a piece.  lo lo is added where the products wait for
// the warps anyway: error against 64 bits 5.7e-6 of the outputs and 3.5e-6 of the state, 6.3e-6 and 4.5e-6 in pieces of 64.
// 1500 and 548 tokens, 32 heads of 128 x 128, turned: 27 + 68 us, and 100 for both together, where the walk in pieces of 64 took 45 + 116
// (163 together); with eight warps and the first operands split by them 131.
// Every wait is bounded and reports instead of hanging; tensor memory is given back on every path.
#include <initializer_list>

#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

namespace zb {

constexpr int RT_TOKENS = 128;              // of a piece
constexpr int RT_D = 128;                   // key channels, those beyond a head's zeros
constexpr int RT_COLS = 64;                 // value columns of a CTA
constexpr int RT_WARPS = 16;                // that bring operands and take results; one of the four behind them issues the products
constexpr int RT_THREADS = (RT_WARPS + 4) * 32;
constexpr int RT_WORKER_REGISTERS = 104, RT_OTHER_REGISTERS = 64;       // of 96 at launch: 512 x 104 + 128 x 64 = 640 x 96
constexpr int RT_QUARTER = RT_COLS / 4;     // value columns of a thread
constexpr int RT_POWERS = 208;              // floats of a copy of the powers: half of the banks on from the copy before, zeros for 46 keys behind a row and more
constexpr int RT_WAIT_LIMIT = 1 << 18;
constexpr int RT_BLOCK = RT_TOKENS * 128;   // bytes of 128 rows of 64 values
constexpr int RT_ROWS_PART = 2 * RT_BLOCK;  // a part of q or k
constexpr int RT_Q = 0, RT_K = RT_Q + 2 * RT_ROWS_PART, RT_V = RT_K + 2 * RT_ROWS_PART, RT_WV = RT_V + 2 * RT_BLOCK, RT_S = RT_WV + 2 * RT_BLOCK;
constexpr int RT_SMEM = RT_S + 2 * RT_BLOCK;
constexpr int RT_TMEM_S1 = 0, RT_TMEM_P = 128, RT_TMEM_INTER = 256, RT_TMEM_INTRA = 320, RT_TMEM_DS = 384;      // columns
constexpr float RT_LARGEST = 3.3e38f;       // beyond it a value rounds to infinity in bfloat16

struct RetentionTcArgs {
  float* out;                               // [tokens, H * V]
  const float* q; long long q_stride;       // [tokens, .]: head h at column h * D
  const float* k; long long k_stride;
  const float* v; long long v_stride;       // head h at column h * V
  const float* decay;                       // [H]
  float* state; long long slot_stride;      // slot s at state + s * slot_stride: [H][D][V]
  const int* slots; const int* row_q_start; const int* row_q_len;
  int H, D, V, num_slots, write_state;
  unsigned char* ws;                        // [pieces][H]{q, k}[part][block of 64 channels][token of the piece][64] bfloat16
  const float* freqs; const int* positions; // null, or q and k are still to be turned
  float k_scale;                            // of k, where it is turned
  int rows, heads_each;                     // heads_each: heads that a CTA of retention_split_kernel takes one after the other
  int* status;
};
constexpr int RT_PIECE_BYTES = 4 * RT_ROWS_PART;                 // of a head: q and k in two parts

// An operand whose rows are the contraction's (64 of its other side's values each): groups of 8 rows 1024 bytes apart, blocks of 64 values RT_BLOCK.
__device__ __forceinline__ unsigned long long rt_desc_mn(unsigned smem_address) {
  return static_cast<unsigned long long>((smem_address >> 4) & 0x3FFFu) | (static_cast<unsigned long long>(RT_BLOCK >> 4) << 16) | (64ull << 32) |
         (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void two_parts(float x, float y, unsigned& hi, unsigned& lo) {
  hi = pack_bf16(x, y);
  lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}
// Eight values as 16-byte pieces of their two parts.
__device__ __forceinline__ void rt_store_parts(const float4& p, const float4& q, unsigned char* to, int part) {
  uint4 hi, lo;
  two_parts(p.x, p.y, hi.x, lo.x);
  two_parts(p.z, p.w, hi.y, lo.y);
  two_parts(q.x, q.y, hi.z, lo.z);
  two_parts(q.z, q.w, hi.w, lo.w);
  *reinterpret_cast<uint4*>(to) = hi;
  *reinterpret_cast<uint4*>(to + part) = lo;
}

// q and k of a piece and some of the heads, turned and in parts, as retention_tc_kernel's copies bring them to shared memory.  Eight lanes a
// token's row, lane c its pieces of eight values.  ROT: dimensions that turn: 0, 64 or 128.
template <int ROT>
__global__ void __launch_bounds__(256) retention_split_kernel(const RetentionTcArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  const int c = threadIdx.x & 7, r0 = threadIdx.x >> 3, piece = blockIdx.x;
  int own;
  const int row = row_of_piece<RT_TOKENS>(a.row_q_len, a.rows, 1, piece, own);
  if (row < 0) return;
  const int n = a.row_q_len[row] - own * RT_TOKENS, h0 = blockIdx.y * a.heads_each, h1 = min(h0 + a.heads_each, a.H);
  const long long t0 = a.row_q_start[row] + own * RT_TOKENS;
  auto turned = [](float4& y, float4& z, const float (&cs)[4], const float (&sn)[4], float scale) {
    const float4 u = y, w = z;
    y = make_float4((u.x * cs[0] - w.x * sn[0]) * scale, (u.y * cs[1] - w.y * sn[1]) * scale, (u.z * cs[2] - w.z * sn[2]) * scale, (u.w * cs[3] - w.w * sn[3]) * scale);
    z = make_float4((w.x * cs[0] + u.x * sn[0]) * scale, (w.y * cs[1] + u.y * sn[1]) * scale, (w.z * cs[2] + u.z * sn[2]) * scale, (w.w * cs[3] + u.w * sn[3]) * scale);
  };
#pragma unroll 1
  for (int u = 0; u < 4; ++u) {
    const int r = r0 + 32 * u;
    const bool here = r < n;
    float cs[2][4], sn[2][4];        // [channels 4 c .., 32 + 4 c ..]
    if (ROT != 0) {
      const float position = here ? static_cast<float>(a.positions[t0 + r]) : 0.0f;
#pragma unroll
      for (int half = 0; half < ROT / 64; ++half)
#pragma unroll
        for (int e = 0; e < 4; ++e) sincosf(position * a.freqs[32 * half + 4 * c + e], &sn[half][e], &cs[half][e]);
    }
#pragma unroll 2
    for (int h = h0; h < h1; ++h) {
      float4 x[2][2][2];             // [q, k][block][half of it]
#pragma unroll
      for (int block = 0; block < 2; ++block)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int d = 64 * block + 32 * half + 4 * c;
          x[0][block][half] = x[1][block][half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (here && d < a.D) {
            x[0][block][half] = *reinterpret_cast<const float4*>(a.q + (t0 + r) * a.q_stride + h * a.D + d);
            x[1][block][half] = *reinterpret_cast<const float4*>(a.k + (t0 + r) * a.k_stride + h * a.D + d);
          }
        }
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const float scale = w ? a.k_scale : 1.0f;
        if (ROT == 128) {
          turned(x[w][0][0], x[w][1][0], cs[0], sn[0], scale);
          turned(x[w][0][1], x[w][1][1], cs[1], sn[1], scale);
        } else if (ROT == 64) {
          turned(x[w][0][0], x[w][0][1], cs[0], sn[0], scale);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            float4& y = x[w][1][half];
            y = make_float4(y.x * scale, y.y * scale, y.z * scale, y.w * scale);
          }
        }
        unsigned char* to = a.ws + (static_cast<long long>(piece) * a.H + h) * RT_PIECE_BYTES + w * 2 * RT_ROWS_PART + r * 128 + ((c ^ (r & 7)) << 4);
        rt_store_parts(x[w][0][0], x[w][0][1], to, RT_ROWS_PART);
        rt_store_parts(x[w][1][0], x[w][1][1], to + RT_BLOCK, RT_ROWS_PART);
      }
    }
  }
}

__global__ void __launch_bounds__(RT_THREADS, 1) retention_tc_kernel(const RetentionTcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ unsigned long long q_full, k_full, q_free, s_full, v_full, p_full, s1_done, ds_done, o_done;
  __shared__ float power[RT_TOKENS + 1];    // a^i
  // A row's weights along the keys, a^(i - j): copy s holds a^(127 - x) at x + s, zeros from 128 on, so that two neighbours of any row begin on 8
  // bytes in one of them, and sixteen lanes' rows in sixteen different pairs of banks.
  __shared__ __align__(8) float falling[2 * RT_POWERS];
  __shared__ unsigned tmem_base_s;
  __shared__ volatile int failed, wild[2];  // wild: the last even and odd piece with a value that is left out of the product
  __shared__ volatile unsigned char wild_token[2][RT_TOKENS];      // and whose values
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int v0 = blockIdx.x * RT_COLS, h = blockIdx.y, row = blockIdx.z;
  if (tid == 0) {
    for (unsigned long long* bar : {&s_full, &v_full, &p_full}) mbar_init(bar, RT_WARPS);
    for (unsigned long long* bar : {&q_full, &k_full, &q_free, &s1_done, &ds_done, &o_done}) mbar_init(bar, 1);
    failed = 0;
    wild[0] = wild[1] = -1;
    fence_barrier_init();
  }
  if (warp == RT_WARPS) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  if (tid <= RT_TOKENS) {
    // (a decay below 2^-1000 is zero either way; the bound keeps the products finite)
    const double bits = fmin(-log2(static_cast<double>(a.decay[h])), 1000.0);
    const float x = exp2f(static_cast<float>(-bits * tid));
    power[tid] = x;
    if (tid < RT_TOKENS) {
#pragma unroll
      for (int copy = 0; copy < 2; ++copy) falling[copy * RT_POWERS + RT_TOKENS - 1 - tid + copy] = x;
    }
  }
  for (int e = tid; e < 2 * (RT_POWERS - RT_TOKENS); e += RT_THREADS) {
    const int copy = e / (RT_POWERS - RT_TOKENS), x = RT_TOKENS + e % (RT_POWERS - RT_TOKENS);
    if (x + copy < RT_POWERS) falling[copy * RT_POWERS + x + copy] = 0.0f;
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const unsigned tmem_base = tmem_base_s;
  wait_for_prior_grids();
  let_dependents_launch();

  const int slot = a.slots[row], n = a.row_q_len[row];
  const bool ours = slot >= 0 && slot < a.num_slots;
  if (!ours && tid == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
  const bool aligned = (smem_u32(smem) & 1023u) == 0;            // the operands must lie on 1024-byte boundaries
  if (!aligned && tid == 0) report(a.status, STATUS_INTERNAL_CHECK, static_cast<int>(smem_u32(smem) & 1023u), row);
  const int pieces = aligned && ours && n > 0 ? (n + RT_TOKENS - 1) / RT_TOKENS : 0;
  const long long t0 = a.row_q_start[row];

  auto arrived = [&](unsigned long long* bar, unsigned parity, int where) -> bool {
    bool ok = false;
    for (int i = 0; i < RT_WAIT_LIMIT && !ok; ++i) {
      ok = mbar_try_wait(bar, parity);
      if (!ok && (i & 255) == 255 && failed) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0 && !failed) report(a.status, STATUS_BARRIER_TIMEOUT, where, row);
      failed = 1;
    }
    return ok;
  };

  if (warp >= RT_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(RT_OTHER_REGISTERS));
    if (warp == RT_WARPS) {
      constexpr unsigned SCORES = tc_idesc(false, RT_TOKENS), VALUES = tc_idesc(true, RT_COLS), WRITE = VALUES | (1u << 15);      // (bit 15: rows of the first operand likewise)
      constexpr int FIRST[4] = {1, 0, 0, 1}, SECOND[4] = {0, 1, 0, 1};      // parts; hi hi behind the small ones; lo lo where it costs nothing
      const bool leader = elect_one();
      const unsigned at = smem_u32(smem);
      const unsigned long long q_desc = desc_k_major(at + RT_Q), k_desc = desc_k_major(at + RT_K), kt_desc = rt_desc_mn(at + RT_K);
      const unsigned long long v_desc = rt_desc_mn(at + RT_V), wv_desc = rt_desc_mn(at + RT_WV), s_desc = rt_desc_mn(at + RT_S);
      for (int p = 0; p < pieces; ++p) {
        if (!arrived(&q_full, p & 1, p) || !arrived(&k_full, p & 1, p)) break;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < RT_D / 16; ++k) {
            const unsigned step = (k / 4 * RT_BLOCK + k % 4 * 32) >> 4;
#pragma unroll
            for (int e = 0; e < 3; ++e)
              tc_mma(tmem_base + RT_TMEM_S1, q_desc + step + (FIRST[e] * RT_ROWS_PART >> 4), k_desc + step + (SECOND[e] * RT_ROWS_PART >> 4), SCORES, (k | e) != 0 ? 1u : 0u);
          }
          tc_commit(&s1_done);
        }
        if (!arrived(&s_full, p & 1, 1000000 + p)) break;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < RT_D / 16; ++k) {
            const unsigned step = (k / 4 * RT_BLOCK + k % 4 * 32) >> 4;
#pragma unroll
            for (int e = 0; e < 3; ++e)
              tc_mma(tmem_base + RT_TMEM_INTER, q_desc + step + (FIRST[e] * RT_ROWS_PART >> 4), s_desc + (k * 2048 >> 4) + (SECOND[e] * RT_BLOCK >> 4), VALUES, (k | e) != 0 ? 1u : 0u);
          }
          tc_commit(&q_free);
        }
        if (!arrived(&v_full, p & 1, 2000000 + p)) break;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < RT_TOKENS / 16; ++k)
#pragma unroll
            for (int e = 3, o = 0; o < 4; e = o++)
              tc_mma(tmem_base + RT_TMEM_DS, kt_desc + (k * 2048 >> 4) + (FIRST[e] * RT_ROWS_PART >> 4), wv_desc + (k * 2048 >> 4) + (SECOND[e] * RT_BLOCK >> 4), WRITE, (k | o) != 0 ? 1u : 0u);
          tc_commit(&ds_done);
        }
        if (!arrived(&p_full, p & 1, 3000000 + p)) break;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll 1
          for (int k = 0; k < RT_TOKENS / 16; ++k)
#pragma unroll
            for (int e = 3, o = 0; o < 4; e = o++)
              tc_mma_ts_if(tmem_base + RT_TMEM_INTRA, tmem_base + RT_TMEM_P + FIRST[e] * 64 + 8 * k, v_desc + (k * 2048 >> 4) + (SECOND[e] * RT_BLOCK >> 4), VALUES, (k | o) != 0 ? 1u : 0u);
          tc_commit(&o_done);
        }
      }
    } else if (warp == RT_WARPS + 1) {
      // q and k of the next piece as soon as the products that read this one's are complete.
      const unsigned char* from = a.ws + (static_cast<long long>(first_piece_of_row<RT_TOKENS>(a.row_q_len, row, 1)) * a.H + h) * RT_PIECE_BYTES;
      for (int p = 0; p < pieces; ++p, from += static_cast<long long>(a.H) * RT_PIECE_BYTES) {
        if (p > 0 && !arrived(&q_free, (p - 1) & 1, 7000000 + p)) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&q_full, 2 * RT_ROWS_PART);
          bulk_copy_g2s(smem + RT_Q, from, 2 * RT_ROWS_PART, &q_full);
        }
        if (p > 0 && !arrived(&ds_done, (p - 1) & 1, 8000000 + p)) break;
        if (lane == 0) {
          mbar_arrive_expect_tx(&k_full, 2 * RT_ROWS_PART);
          bulk_copy_g2s(smem + RT_K, from + 2 * RT_ROWS_PART, 2 * RT_ROWS_PART, &k_full);
        }
        __syncwarp();
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(RT_WORKER_REGISTERS));
    // Values: eight lanes a token's row, lane c eight of them; the thread's rows are r0 + 64 u of a piece.
    const int c = tid & 7, r0 = tid >> 3;
    const float* const v = a.v + t0 * a.v_stride + h * a.V + v0 + 8 * c;
    float4 values[2][2];
    auto fetch_values = [&](int p) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = p * RT_TOKENS + r0 + 64 * u;
          values[u][i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (t < n && v0 + 8 * c + 4 * i < a.V) values[u][i] = *reinterpret_cast<const float4*>(v + t * a.v_stride + 4 * i);
        }
    };
    // Results: the thread's row of tensor memory and a quarter of the columns.
    const int quarter = warp >> 2, r = (warp & 3) * 32 + lane;
    const unsigned mine = tmem_base + (static_cast<unsigned>((warp & 3) * 32) << 16);
    const int behind_all = RT_TOKENS - 1 - r, copy = behind_all & 1;
    const float* const falling_row = falling + copy * RT_POWERS + behind_all + copy;      // a^(r - j) at j
    // The state: row r of the products is channel `channel`.
    const int channel = r / 64 * 64 + r % 64 / 8 * 4 + (r & 3) + (r & 4) * 8;
    float* const state = a.state + static_cast<long long>(ours ? slot : 0) * a.slot_stride + (static_cast<long long>(h) * a.D + channel) * a.V + v0 + RT_QUARTER * quarter;
    float S[RT_QUARTER];
#pragma unroll
    for (int i = 0; i < RT_QUARTER; i += 4) {
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (pieces > 0 && channel < a.D && v0 + RT_QUARTER * quarter + i < a.V) x = *reinterpret_cast<const float4*>(state + i);
      S[i] = x.x; S[i + 1] = x.y; S[i + 2] = x.z; S[i + 3] = x.w;
    }
    auto signal = [&](unsigned long long* bar) {
      fence_proxy_async();            // the tensor core reads what was stored through the asynchronous proxy
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(bar);
    };
    auto store_state = [&] {
#pragma unroll
      for (int i = 0; i < RT_QUARTER / 8; ++i)
        rt_store_parts(make_float4(S[8 * i], S[8 * i + 1], S[8 * i + 2], S[8 * i + 3]), make_float4(S[8 * i + 4], S[8 * i + 5], S[8 * i + 6], S[8 * i + 7]),
                       smem + RT_S + r * 128 + (((RT_QUARTER / 8 * quarter + i) ^ (r & 7)) << 4), RT_BLOCK);
      signal(&s_full);
    };
    if (pieces > 0) {
      fetch_values(0);
      store_state();
    }
    bool ok = true;
    for (int p = 0; p < pieces; ++p) {
      const int count = min(RT_TOKENS, n - p * RT_TOKENS);
      // (the products of the piece before are complete: its values' place is free)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = r0 + 64 * u, to = i * 128 + ((c ^ (i & 7)) << 4);
        const float weight = i < count ? power[count - 1 - i] : 0.0f;
        float4 x[2] = {values[u][0], values[u][1]};
        rt_store_parts(make_float4(x[0].x * weight, x[0].y * weight, x[0].z * weight, x[0].w * weight),
                       make_float4(x[1].x * weight, x[1].y * weight, x[1].z * weight, x[1].w * weight), smem + RT_WV + to, RT_BLOCK);
        bool odd = false;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float& y = reinterpret_cast<float*>(x)[e];
          if (!(fabsf(y) <= RT_LARGEST)) { y = 0.0f; odd = true; }
        }
        const unsigned any = __ballot_sync(0xffffffffu, odd) >> (lane & 24) & 0xffu;      // of the eight lanes of the row
        if (c == 0) wild_token[p & 1][i] = any != 0 ? 1 : 0;
        if (odd) wild[p & 1] = p;
        rt_store_parts(x[0], x[1], smem + RT_V + to, RT_BLOCK);
      }
      signal(&v_full);
      if (p + 1 < pieces) fetch_values(p + 1);
      // Scores to weights: row r, keys 32 quarter .. + 31.
      ok = arrived(&s1_done, p & 1, 4000000 + p);
      // (Behind a piece with such a value the weights' place is read until its outputs are there, by four warps a row.  Each of them has
      // then given the state of this piece.)
      if (ok && p > 0 && wild[(p - 1) & 1] == p - 1) ok = arrived(&s_full, p & 1, 9000000 + p);
      if (!ok) break;
      tc_fence_after_sync();
#pragma unroll
      for (int i = 0; i < 32; i += 16) {
        const int j0 = 32 * quarter + i;
        const bool seen = j0 + 15 <= r - lane;            // by every row of the warp
        unsigned x[16], hi[8] = {}, lo[8] = {};
        tmem_ld16(mine + RT_TMEM_S1 + j0, x);
        tmem_wait_ld16(x);
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          if (j0 > r - lane + 31) continue;               // (by none of them)
          const float2 w = *reinterpret_cast<const float2*>(falling_row + j0 + e), z = *reinterpret_cast<const float2*>(falling_row + j0 + e + 2);
          float y[4] = {__uint_as_float(x[e]) * w.x, __uint_as_float(x[e + 1]) * w.y, __uint_as_float(x[e + 2]) * z.x, __uint_as_float(x[e + 3]) * z.y};
          if (!seen) {
#pragma unroll
            for (int f = 0; f < 4; ++f)
              if (j0 + e + f > r) y[f] = 0.0f;            // (a later token's score may be anything)
          }
          two_parts(y[0], y[1], hi[e / 2], lo[e / 2]);
          two_parts(y[2], y[3], hi[e / 2 + 1], lo[e / 2 + 1]);
        }
        tmem_st8(mine + RT_TMEM_P + j0 / 2, hi);
        tmem_st8(mine + RT_TMEM_P + 64 + j0 / 2, lo);
      }
      tc_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(&p_full);
      // The state.
      ok = arrived(&ds_done, p & 1, 5000000 + p);
      if (!ok) break;
      tc_fence_after_sync();
      const float whole = power[count];
#pragma unroll
      for (int i = 0; i < RT_QUARTER; i += 16) {
        unsigned x[16];
        tmem_ld16(mine + RT_TMEM_DS + RT_QUARTER * quarter + i, x);
        tmem_wait_ld16(x);
#pragma unroll
        for (int e = 0; e < 16; ++e) S[i + e] = fmaf(whole, S[i + e], __uint_as_float(x[e]));
      }
      ok = arrived(&o_done, p & 1, 6000000 + p);
      if (!ok) break;
      tc_fence_after_sync();
      // The outputs, eight rows at a time: by the warp's own rows of the weighted values' place, whose product is complete.
      const float lead = power[min(r + 1, RT_TOKENS)];
      auto staged = [&](int i, int piece) {       // 16 bytes of row i of the warp's 32: 64 bytes each in its 8 rows of the two parts
        const int line = i >> 1, own = 4 * warp + (line >> 1 & 3) + 64 * (line >> 3);
        return reinterpret_cast<float4*>(smem + RT_WV + (line & 1) * RT_BLOCK + own * 128 + (((i & 1) * 4 + (piece ^ (line & 3))) << 4));
      };
#pragma unroll
      for (int i = 0; i < RT_QUARTER; i += 16) {
        unsigned x[16], y[16];
        float o[16];
        tmem_ld16(mine + RT_TMEM_INTER + RT_QUARTER * quarter + i, x);
        tmem_ld16(mine + RT_TMEM_INTRA + RT_QUARTER * quarter + i, y);
        tmem_wait_ld16(x);
        tmem_wait_ld16(y);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = fmaf(lead, __uint_as_float(x[e]), __uint_as_float(y[e]));
        if (wild[p & 1] == p) {
#pragma unroll 1
          for (int j = 0; j < RT_TOKENS; ++j) {
            if (!wild_token[p & 1][j]) continue;               // (the same for the whole CTA)
            unsigned hi[16], lo[16];                    // 32 tokens' weights
            tmem_ld16(mine + RT_TMEM_P + j / 32 * 16, hi);
            tmem_ld16(mine + RT_TMEM_P + 64 + j / 32 * 16, lo);
            tmem_wait_ld16(hi);
            tmem_wait_ld16(lo);
            float weight = 0.0f;
#pragma unroll
            for (int e = 0; e < 16; ++e)
              if (e == j % 32 / 2)
                weight = j & 1 ? __uint_as_float(hi[e] & 0xffff0000u) + __uint_as_float(lo[e] & 0xffff0000u)
                               : __uint_as_float(hi[e] << 16) + __uint_as_float(lo[e] << 16);
            const float* from = a.v + (t0 + p * RT_TOKENS + j) * a.v_stride + h * a.V + v0 + RT_QUARTER * quarter + i;
            for (int e = 0; e < 16; ++e) {
              const float value = v0 + RT_QUARTER * quarter + i + e < a.V ? from[e] : 0.0f;
              if (j > r || fabsf(value) <= RT_LARGEST) continue;
#pragma unroll
              for (int f = 0; f < 16; ++f)
                if (f == e) o[f] = fmaf(weight, value, o[f]);
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 16; e += 4) *staged(lane, (i + e) / 4) = make_float4(o[e], o[e + 1], o[e + 2], o[e + 3]);
      }
      tc_fence_before_sync();
      if (p + 1 < pieces) store_state();
      else __syncwarp();
      {
        const int piece = lane & 3, column = v0 + RT_QUARTER * quarter + 4 * piece;
        float* const out = a.out + (t0 + p * RT_TOKENS) * a.H * a.V + static_cast<long long>(h) * a.V + column;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int own = 8 * i + (lane >> 2), token = (warp & 3) * 32 + own;
          if (token < count && column < a.V) *reinterpret_cast<float4*>(out + static_cast<long long>(token) * a.H * a.V) = *staged(own, piece);
        }
      }
      __syncwarp();
    }
    if (ok && pieces > 0 && a.write_state && channel < a.D) {
#pragma unroll
      for (int i = 0; i < RT_QUARTER; i += 4)
        if (v0 + RT_QUARTER * quarter + i < a.V) *reinterpret_cast<float4*>(state + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    }
  }

  // Everybody meets here on every path, and the warp that took the tensor memory gives it back.
  tc_fence_before_sync();
  __syncthreads();
  if (failed) let_copies_land();        // (the products in flight)
  if (warp == RT_WARPS) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace zb

using namespace zb;

// 1 if zb_retention_tc takes these sizes: heads of more than 64 and up to 128 key channels, rows of four values on 16-byte boundaries.
ZB_API int zb_retention_tc_supported(int D, int V, int rot_dims) {
  return D > 64 && D <= RT_D && D % 4 == 0 && V > 0 && V % 4 == 0 && (rot_dims == 0 || rot_dims == 64 || (rot_dims == 128 && D == 128)) ? 1 : 0;
}

ZB_API int zb_retention_tc_piece_tokens() { return RT_TOKENS; }
// Floats of workspace a piece needs.
ZB_API int zb_retention_tc_piece_floats(int H) { return H * (RT_PIECE_BYTES / 4); }

// Retention as zb_state_walk's fixed decays, all rows; q, k, v and the state on 16-byte boundaries, as their rows.  With `freqs` (rot_dims / 2 of
// them) q and k are turned by the tokens' positions first, k times k_scale.  ws: (tokens / piece tokens + rows) * zb_retention_tc_piece_floats
// floats, 16-byte aligned, contents irrelevant.  The rows' tokens may lie in the stream in any order.
ZB_API int zb_retention_tc(float* out, const float* q, long long q_stride, const float* k, long long k_stride, const float* v, long long v_stride,
                           const float* decay, float* state, long long slot_stride, const int* slots, const int* row_q_start, const int* row_q_len,
                           int rows, int tokens, int H, int D, int V, int num_slots, int write_state, const float* freqs, int rot_dims, float k_scale,
                           const int* positions, float* ws, int* status, void* stream) {
  const int rot = freqs != nullptr ? rot_dims : 0;
  if (rows < 0 || tokens < 0 || H <= 0 || num_slots <= 0 || decay == nullptr || ws == nullptr || (freqs != nullptr && positions == nullptr))
    return ERR_BAD_ARGUMENT;
  if (!zb_retention_tc_supported(D, V, rot) || H > 65535 || rows > 65535) return ERR_UNSUPPORTED;
  for (const void* p : {static_cast<const void*>(out), static_cast<const void*>(q), static_cast<const void*>(k), static_cast<const void*>(v),
                        static_cast<const void*>(state), static_cast<const void*>(ws)})
    if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return ERR_BAD_ARGUMENT;
  if (q_stride % 4 != 0 || k_stride % 4 != 0 || v_stride % 4 != 0 || slot_stride % 4 != 0) return ERR_BAD_ARGUMENT;
  if (rows == 0 || tokens == 0) return OK;
  RetentionTcArgs a;
  a.out = out; a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride; a.decay = decay;
  a.state = state; a.slot_stride = slot_stride; a.slots = slots; a.row_q_start = row_q_start; a.row_q_len = row_q_len;
  a.H = H; a.D = D; a.V = V; a.num_slots = num_slots; a.write_state = write_state; a.rows = rows;
  a.ws = reinterpret_cast<unsigned char*>(ws);
  a.freqs = freqs; a.positions = positions; a.k_scale = k_scale; a.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  // A CTA of the first kernel shares a token's cosines and sines among up to four heads while that leaves two CTAs an SM.
  const int pieces = tokens / RT_TOKENS + rows;
  a.heads_each = static_cast<long long>(pieces) * H >= 4 * 2 * 148 ? 4 : static_cast<long long>(pieces) * H >= 2 * 2 * 148 ? 2 : 1;
  auto split = rot == 128 ? retention_split_kernel<128> : rot == 64 ? retention_split_kernel<64> : retention_split_kernel<0>;
  const int launched = launch_dependent(split, dim3(pieces, (H + a.heads_each - 1) / a.heads_each), dim3(256), 0, s, false, a);
  if (launched != OK) return launched;
  if (cuda_failed(cudaFuncSetAttribute(retention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RT_SMEM))) return ERR_CUDA;
  return launch_dependent(retention_tc_kernel, dim3((V + RT_COLS - 1) / RT_COLS, H, rows), dim3(RT_THREADS), RT_SMEM, s, false, a);
}
