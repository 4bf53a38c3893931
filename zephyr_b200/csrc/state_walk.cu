// Linear attention with one decay per head and token over runs of tokens: per head
//
//   S_t = a_t S_{t-1} + s_t k_t v_t^T,   o_t = S_t^T q_t (+ skip v_t)      (S [D key channels x V value channels], float32)
//
// in two settings: WALK_SPACE, the state-space form of Mamba-2 (a_t = exp(-exp(A_log) dt_t), s_t = dt_t, dt = softplus(. +
// dt_bias); q, k, v bfloat16, q and k shared by the heads of a group), and WALK_FIXED, retention (a_t = a, s_t = 1; q, k, v
// float32).  A request's new tokens of a step are cut into pieces of W tokens.  With S_in the state at a piece's start, n its
// tokens and c_i the sum of the logarithms of its decays up to token i,
//
//   o_i   = e^(c_i) S_in^T q_i + sum_{j <= i} e^(c_i - c_j) s_j (q_i . k_j) v_j
//   S_out = e^(c_n) S_in + sum_j e^(c_n - c_j) s_j k_j v_j^T
//
//   walk_prepare   for all pieces side by side: the scores q . k, and what else a piece needs (sums of logarithms; the
//                  float32 q and k as pairs of bfloat16 values)
//   state_walk     a CTA owns a request, a head and some value columns and walks the pieces with the state in registers
//
// so the state never leaves the SM, where passes over all pieces at once write and read every piece's state (2048
// tokens, 32 heads of 128 x 64: 33 MB four times), and a piece is two barriers.
//
// Products run on the tensor cores, float32 sums.  A bfloat16 operand is exact; beside it a float32 operand is the sum
// of three bfloat16 values (all its 24 bits); two float32 operands (WALK_FIXED) are two bfloat16 values each, hi hi + hi lo +
// lo hi, a relative error of about 2^-16 an operand.  The state itself is only ever touched by float32 multiply-adds.
// Sums of logarithms are kept as two float32 values, so that a difference of two is good to a rounding of itself.
//
// Piece p of row r has the number row_q_start[r] / W + r + p: distinct for all pieces of a step, and below
// tokens / W + rows.
#include "common.cuh"
#include "mma.cuh"

namespace zb {

constexpr int W = 64;                    // tokens of a piece
constexpr int W_THREADS = 256;
constexpr int W_GST = W + 8;             // a row of the scores
constexpr int W_STEP = 3 * W;            // WALK_SPACE, a head of a piece: sums of logarithms (base 2), two values each, and s

enum { WALK_SPACE = 0, WALK_FIXED = 1 };

struct WalkArgs {
  const void* q; long long q_stride;     // [tokens, .]: head h (or its group) at column h * D
  const void* k; long long k_stride;
  const void* v; long long v_stride;     // head h at column h * V
  const void* dt; long long dt_stride;   // WALK_SPACE: [tokens, H], bfloat16
  const float* dt_bias; const float* a_log; const float* skip;        // WALK_SPACE: [H] each
  const float* decay;                    // WALK_FIXED: [H]
  float* scores;                         // [pieces][qk heads][W][W_GST]
  float* steps;                          // WALK_SPACE: [pieces][H][W_STEP]
  __nv_bfloat16* parts;                  // WALK_FIXED: [pieces][H][q hi, q lo, k hi, k lo][W][DP + 8]
  float* out;                            // [tokens, H * V]
  float* state; long long slot_stride;   // slot s at state + s * slot_stride: [H][D][V]
  const int* slots; const int* row_q_start; const int* row_q_len;
  int rows, H, D, V, heads_per_group, num_slots, write_state;
  int* status;
};

__device__ __forceinline__ float walk_softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

// x and y as PARTS pairs of bfloat16 values whose sums they are, the largest first.
template <int PARTS>
__device__ __forceinline__ void split_parts(float x, float y, unsigned (&part)[PARTS]) {
#pragma unroll
  for (int i = 0; i < PARTS; ++i) {
    part[i] = pack_bf16(x, y);
    x -= __uint_as_float(part[i] << 16);
    y -= __uint_as_float(part[i] & 0xffff0000u);
  }
}

// Which products of parts count: all of one exact operand's with the other's, or of two pairs all but lo lo.
template <int PA, int PB>
__device__ __forceinline__ constexpr bool counts(int a, int b) { return a + b < (PA > PB ? PA : PB); }

// acc[N tiles of 8 columns] += A B over 16 of k: A's fragments in parts; B in parts, [k][st] tiles `part_stride` elements
// apart, from this lane's ldmatrix address inside the first 16 x 16 block on.
template <int N, int PA, int PB>
__device__ __forceinline__ void walk_product(float (&acc)[N][4], const unsigned (&af)[PA][4], const __nv_bfloat16* b, int part_stride) {
#pragma unroll
  for (int n = 0; n < N; n += 2) {
#pragma unroll
    for (int pb = PB - 1; pb >= 0; --pb) {                   // the small products first
      unsigned bf[4];
      ldmatrix_x4_trans(bf, b + pb * part_stride + n * 8);
#pragma unroll
      for (int pa = PA - 1; pa >= 0; --pa)
        if (counts<PA, PB>(pa, pb)) {
          mma_bf16_16816(acc[n], af[pa], bf[0], bf[1]);
          mma_bf16_16816(acc[n + 1], af[pa], bf[2], bf[3]);
        }
    }
  }
}

__device__ __forceinline__ int walk_first_piece(const WalkArgs& a, int row) { return a.row_q_start[row] / W + row; }

// The scores of a piece for one q/k head, and its sums of logarithms (WALK_SPACE, the heads of the group) or its operands in
// parts (WALK_FIXED).  DP: the channels padded with zeros.
template <int MODE, int DP>
__global__ void __launch_bounds__(W_THREADS) walk_prepare_kernel(const WalkArgs a) {
  extern __shared__ __align__(16) unsigned char w_smem[];
  constexpr int ST = DP + 8, PA = MODE == WALK_SPACE ? 1 : 2;
  __shared__ int found;
  const int piece = blockIdx.x, qk_head = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) found = -1;
  __syncthreads();
  for (int r = tid; r < a.rows; r += W_THREADS) {
    const int p = piece - walk_first_piece(a, r);
    if (p >= 0 && p * W < a.row_q_len[r]) found = r;         // at most one row
  }
  __syncthreads();
  const int row = found;
  if (row < 0) return;
  const int begin = (piece - walk_first_piece(a, row)) * W, n = min(W, a.row_q_len[row] - begin);
  const long long t0 = a.row_q_start[row] + begin;
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(w_smem);        // [PA][W][ST]
  __nv_bfloat16* k_s = q_s + PA * W * ST;                               // [PA][W][ST]
  if (MODE == WALK_SPACE) {
    const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a.q) + t0 * a.q_stride + qk_head * a.D;
    const __nv_bfloat16* k = static_cast<const __nv_bfloat16*>(a.k) + t0 * a.k_stride + qk_head * a.D;
    for (int e = tid; e < W * (DP / 8); e += W_THREADS) {
      const int i = e / (DP / 8), c = e % (DP / 8) * 8;
      const bool ok = i < n && c < a.D;
      cp_async_16(q_s + i * ST + c, ok ? q + i * a.q_stride + c : q, ok);
      cp_async_16(k_s + i * ST + c, ok ? k + i * a.k_stride + c : k, ok);
    }
    cp_async_commit();
    // Meanwhile the heads' steps and decays: a warp a head, two tokens a lane, their sum scanned in 64 bits.
    for (int j = warp; j < a.heads_per_group; j += W_THREADS / 32) {
      const int h = qk_head * a.heads_per_group + j;
      const __nv_bfloat16* dt = static_cast<const __nv_bfloat16*>(a.dt) + t0 * a.dt_stride + h;
      const float rate = expf(a.a_log[h]), bias = a.dt_bias[h];
      float step[2];
      double sum[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = 2 * lane + u;
        step[u] = i < n ? walk_softplus(__bfloat162float(dt[i * a.dt_stride]) + bias) : 0.0f;
        // (a decay below e^-1000 is zero either way; the bound keeps the sums finite)
        sum[u] = -fmin(static_cast<double>(rate) * static_cast<double>(step[u]), 1000.0) * 1.4426950408889634;
      }
      sum[1] += sum[0];
      double before = sum[1];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += other;
      }
      before -= sum[1];
      float* to = a.steps + (static_cast<long long>(piece) * a.H + h) * W_STEP + 2 * lane;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double c = before + sum[u];
        const float hi = static_cast<float>(c);
        to[u] = hi;
        to[W + u] = static_cast<float>(c - hi);
        to[2 * W + u] = step[u];
      }
    }
    cp_async_wait<0>();
  } else {
    const float* q = static_cast<const float*>(a.q) + t0 * a.q_stride + qk_head * a.D;
    const float* k = static_cast<const float*>(a.k) + t0 * a.k_stride + qk_head * a.D;
    const bool vectors = a.D % 4 == 0 && a.q_stride % 4 == 0 && a.k_stride % 4 == 0 && reinterpret_cast<uintptr_t>(a.q) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(a.k) % 16 == 0;
#pragma unroll 4
    for (int e = tid; e < 2 * W * (DP / 4); e += W_THREADS) {
      const int which = e / (W * (DP / 4)), r = e % (W * (DP / 4)), i = r / (DP / 4), c = r % (DP / 4) * 4;
      const float* from = which ? k + i * a.k_stride + c : q + i * a.q_stride + c;
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (i < n && c < a.D) {
        if (vectors) {
          x = *reinterpret_cast<const float4*>(from);
        } else {
          x.x = from[0];
          if (c + 1 < a.D) x.y = from[1];
          if (c + 2 < a.D) x.z = from[2];
          if (c + 3 < a.D) x.w = from[3];
        }
      }
      unsigned lo[2], hi[2];
      split_parts<2>(x.x, x.y, lo);
      split_parts<2>(x.z, x.w, hi);
      __nv_bfloat16* to = (which ? k_s : q_s) + i * ST + c;
#pragma unroll
      for (int p = 0; p < 2; ++p) *reinterpret_cast<uint2*>(to + p * W * ST) = make_uint2(lo[p], hi[p]);
    }
  }
  __syncthreads();
  if (MODE == WALK_FIXED) {
    uint4* to = reinterpret_cast<uint4*>(a.parts + (static_cast<long long>(piece) * a.H + qk_head) * 4 * W * ST);
    const uint4* from = reinterpret_cast<const uint4*>(q_s);
    for (int e = tid; e < 4 * W * ST / 8; e += W_THREADS) to[e] = from[e];
  }
  // A warp owns 16 rows of the scores and 32 columns.
  const int g = lane >> 2, t = lane & 3, row0 = (warp & 3) * 16, col0 = (warp >> 2) * 32;
  const int qk_heads = a.H / a.heads_per_group;
  float* scores = a.scores + (static_cast<long long>(piece) * qk_heads + qk_head) * W * W_GST;
  const int q_off = (row0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ST + (lane >> 4) * 8;
  const int k_off = ((lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int c0 = col0 + u * 16;
    float s[2][4] = {};
    if (c0 <= row0 + 15) {                                   // (later keys: never read)
#pragma unroll
      for (int ks = 0; ks < DP / 16; ++ks) {
        unsigned af[PA][4], bf[PA][4];
#pragma unroll
        for (int p = 0; p < PA; ++p) {
          ldmatrix_x4(af[p], q_s + p * W * ST + q_off + ks * 16);
          ldmatrix_x4(bf[p], k_s + p * W * ST + c0 * ST + k_off + ks * 16);
        }
#pragma unroll
        for (int pa = PA - 1; pa >= 0; --pa)
#pragma unroll
          for (int pb = PA - 1; pb >= 0; --pb)
            if (counts<PA, PA>(pa, pb)) {
              mma_bf16_16816(s[0], af[pa], bf[pb][0], bf[pb][1]);
              mma_bf16_16816(s[1], af[pa], bf[pb][2], bf[pb][3]);
            }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float* to = scores + (row0 + g) * W_GST + c0 + 8 * i + 2 * t;
      *reinterpret_cast<float2*>(to) = make_float2(s[i][0], s[i][1]);
      *reinterpret_cast<float2*>(to + 8 * W_GST) = make_float2(s[i][2], s[i][3]);
    }
  }
}

template <int MODE, int DP, int NT>
struct WalkShape {
  static constexpr int PA = MODE == WALK_SPACE ? 1 : 2;      // parts of q, k and v
  static constexpr int PB = MODE == WALK_SPACE ? 3 : 2;      // parts of the state, the weights and the weighted values
  static constexpr int ST = DP + 8, COLS = 8 * NT, CST = COLS + 8, OST = COLS + 4;
  static constexpr int STAGES = MODE == WALK_SPACE ? 3 : 2;
  static constexpr int qk_bytes = 2 * PA * W * ST * 2;
  static constexpr int stage_bytes = qk_bytes + W * W_GST * 4 + (MODE == WALK_SPACE ? W_STEP * 4 : 0);
  static constexpr int smem = STAGES * stage_bytes + PB * DP * CST * 2 + (PA + PB) * W * CST * 2 + W * OST * 4;
};

// NT: tiles of 8 value columns of a CTA.  Warp w owns the state's channels 16 w .. (C fragments); for the outputs it owns
// tokens 16 (w % 4) .. and takes half the channels (S^T q) and every other 16 keys (the scores).  A piece:
//   barrier; both terms of the outputs and the state's sums from shared memory; one half of the outputs' sums to shared memory;
//   barrier; the other half adds it and writes; the state and the next piece's values go to shared memory in parts.
// The next pieces' operands are copied meanwhile.
template <int MODE, int DP, int NT>
__global__ void __launch_bounds__(W_THREADS) state_walk_kernel(const WalkArgs a) {
  using Shape = WalkShape<MODE, DP, NT>;
  constexpr int PA = Shape::PA, PB = Shape::PB, ST = Shape::ST, COLS = Shape::COLS, CST = Shape::CST, OST = Shape::OST;
  constexpr int STAGES = Shape::STAGES, PER = W * COLS / W_THREADS / 2;      // pairs of values a thread brings of a piece
  extern __shared__ __align__(16) unsigned char w_smem[];
  __nv_bfloat16* s_s = reinterpret_cast<__nv_bfloat16*>(w_smem + STAGES * Shape::stage_bytes);    // [PB][DP][CST]
  __nv_bfloat16* v_s = s_s + PB * DP * CST;                  // [PA][W][CST]
  __nv_bfloat16* wv_s = v_s + PA * W * CST;                  // [PB][W][CST]: e^(c_n - c_j) s_j v_j
  float* o_s = reinterpret_cast<float*>(wv_s + PB * W * CST);            // [W][OST]
  __shared__ float power_s[W + 1];                           // WALK_FIXED: a^0 .. a^W
  const int row = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) {
    if (tid == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
    return;
  }
  const int n_all = a.row_q_len[row], pieces = (n_all + W - 1) / W;
  const long long t0 = a.row_q_start[row];
  const int first = walk_first_piece(a, row), qk_head = h / a.heads_per_group, qk_heads = a.H / a.heads_per_group;
  if (MODE == WALK_FIXED && tid <= W) power_s[tid] = powf(a.decay[h], static_cast<float>(tid));
  if (MODE == WALK_SPACE && a.D < DP)                        // the channels beyond D: zeros in every stage
    for (int e = tid; e < STAGES * 2 * W * (DP / 8); e += W_THREADS) {
      const int c = e % (DP / 8) * 8, r = e / (DP / 8);
      if (c >= a.D)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(w_smem + r / (2 * W) * Shape::stage_bytes) + r % (2 * W) * ST + c) =
            make_uint4(0, 0, 0, 0);
    }

  auto copy_piece = [&](int p) {
    unsigned char* stage = w_smem + p % STAGES * Shape::stage_bytes;
    if (MODE == WALK_SPACE) {
      __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(stage);
      const int n = min(W, n_all - p * W), chunks = a.D / 8;
      const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a.q) + (t0 + p * W) * a.q_stride + qk_head * a.D;
      const __nv_bfloat16* k = static_cast<const __nv_bfloat16*>(a.k) + (t0 + p * W) * a.k_stride + qk_head * a.D;
#pragma unroll
      for (int u = 0; u < W * (DP / 8) / W_THREADS; ++u) {
        const int e = tid + u * W_THREADS, i = e / (DP / 8), c = e % (DP / 8);
        if (c >= chunks) continue;
        cp_async_16(q_s + i * ST + 8 * c, i < n ? q + i * a.q_stride + 8 * c : q, i < n);
        cp_async_16(q_s + (W + i) * ST + 8 * c, i < n ? k + i * a.k_stride + 8 * c : k, i < n);
      }
      const float* steps = a.steps + (static_cast<long long>(first + p) * a.H + h) * W_STEP;
      if (tid < W_STEP / 4) cp_async_16(stage + Shape::qk_bytes + W * W_GST * 4 + tid * 16, steps + tid * 4, true);
    } else {
      const __nv_bfloat16* parts = a.parts + (static_cast<long long>(first + p) * a.H + h) * 4 * W * ST;
      for (int e = tid; e < Shape::qk_bytes / 16; e += W_THREADS) cp_async_16(stage + e * 16, parts + e * 8, true);
    }
    const float* scores = a.scores + (static_cast<long long>(first + p) * qk_heads + qk_head) * W * W_GST;
    for (int e = tid; e < W * W_GST / 4; e += W_THREADS) cp_async_16(stage + Shape::qk_bytes + e * 16, scores + e * 4, true);
  };
  // This thread's values of a piece: pairs of columns (my_c, my_c + 1) of tokens my_i, my_i + W / PER, ...; with their weights.
  constexpr int TOKENS = W / PER;
  const int my_c = tid % (COLS / 2) * 2, my_i = tid / (COLS / 2);
  float value[PER][2], weight[PER];
  auto fetch_values = [&](int p) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = my_i + u * TOKENS, at = p * W + i, n = min(W, n_all - p * W);
      value[u][0] = value[u][1] = weight[u] = 0.0f;
      if (p >= pieces || i >= n) continue;
      if (MODE == WALK_SPACE) {
        const __nv_bfloat16* v = static_cast<const __nv_bfloat16*>(a.v) + (t0 + at) * a.v_stride + h * a.V + v0 + my_c;
        if (v0 + my_c < a.V) value[u][0] = __bfloat162float(v[0]);
        if (v0 + my_c + 1 < a.V) value[u][1] = __bfloat162float(v[1]);
        const float* c = a.steps + (static_cast<long long>(first + p) * a.H + h) * W_STEP;
        weight[u] = exp2f((c[W - 1] - c[i]) + (c[2 * W - 1] - c[W + i])) * c[2 * W + i];
      } else {
        const float* v = static_cast<const float*>(a.v) + (t0 + at) * a.v_stride + h * a.V + v0 + my_c;
        if (v0 + my_c < a.V) value[u][0] = v[0];
        if (v0 + my_c + 1 < a.V) value[u][1] = v[1];
        weight[u] = power_s[n - 1 - i];
      }
    }
  };
  auto store_values = [&]() {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int at = (my_i + u * TOKENS) * CST + my_c;
      unsigned vp[PA], wp[PB];
      split_parts<PA>(value[u][0], value[u][1], vp);
      split_parts<PB>(value[u][0] * weight[u], value[u][1] * weight[u], wp);
#pragma unroll
      for (int p = 0; p < PA; ++p) *reinterpret_cast<unsigned*>(v_s + p * W * CST + at) = vp[p];
#pragma unroll
      for (int p = 0; p < PB; ++p) *reinterpret_cast<unsigned*>(wv_s + p * W * CST + at) = wp[p];
    }
  };
  // This thread's part of the state: channels d0 and d0 + 8, columns 8 i + 2 t and the next.
  const int d0 = warp * 16 + g;
  const bool holds = warp * 16 < DP;
  float S[NT][4];
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride + static_cast<long long>(h) * a.D * a.V + v0;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      S[i][e] = holds && d < a.D && v0 + c < a.V ? state[static_cast<long long>(d) * a.V + c] : 0.0f;
    }
  auto store_state = [&]() {
    if (!holds) return;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        unsigned sp[PB];
        split_parts<PB>(S[i][2 * half], S[i][2 * half + 1], sp);
#pragma unroll
        for (int p = 0; p < PB; ++p) *reinterpret_cast<unsigned*>(s_s + (p * DP + d0 + 8 * half) * CST + 8 * i + 2 * t) = sp[p];
      }
  };
  if (MODE == WALK_FIXED) __syncthreads();                   // the powers
  store_state();
  fetch_values(0);
  store_values();
#pragma unroll
  for (int p = 0; p < STAGES - 1; ++p) {
    if (p < pieces) copy_piece(p);
    cp_async_commit();
  }
  const float skip = MODE == WALK_SPACE ? a.skip[h] : 0.0f;
  // ldmatrix addresses: A rows as they lie, A transposed, B as [k][n].
  const int a_off = ((lane & 7) + ((lane >> 3) & 1) * 8) * ST + (lane >> 4) * 8;
  const int at_off = ((lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8;
  const int b_off = ((lane & 7) + ((lane >> 3) & 1) * 8) * CST + (lane >> 4) * 8;
  const int row0 = (warp & 3) * 16, half = warp >> 2;
  for (int p = 0; p < pieces; ++p) {
    const unsigned char* stage = w_smem + p % STAGES * Shape::stage_bytes;
    const __nv_bfloat16* q_s = reinterpret_cast<const __nv_bfloat16*>(stage);              // [PA][W][ST]
    const __nv_bfloat16* k_s = q_s + PA * W * ST;
    const float* scores = reinterpret_cast<const float*>(stage + Shape::qk_bytes);
    const float* c_s = scores + W * W_GST;
    const int n = min(W, n_all - p * W);
    cp_async_wait<STAGES - 2>();
    __syncthreads();               // the piece, the state and the values are there; the buffer of the piece before is free
    if (p + STAGES - 1 < pieces) copy_piece(p + STAGES - 1);
    cp_async_commit();
    fetch_values(p + 1);
    const int i0 = row0 + g, i1 = i0 + 8;
    float c_hi[2] = {}, c_lo[2] = {}, lead[2];
    if (MODE == WALK_SPACE) {
      c_hi[0] = c_s[i0]; c_hi[1] = c_s[i1];
      c_lo[0] = c_s[W + i0]; c_lo[1] = c_s[W + i1];
      lead[0] = exp2f(c_hi[0] + c_lo[0]); lead[1] = exp2f(c_hi[1] + c_lo[1]);
    } else {
      lead[0] = power_s[i0 + 1]; lead[1] = power_s[i1 + 1];
    }
    float o[NT][4] = {};
    if (row0 < n) {
#pragma unroll
      for (int ks = 0; ks < DP / 32; ++ks) {
        const int d = half * (DP / 2) + ks * 16;
        unsigned af[PA][4];
#pragma unroll
        for (int x = 0; x < PA; ++x) ldmatrix_x4(af[x], q_s + (x * W + row0) * ST + a_off + d);
        walk_product<NT, PA, PB>(o, af, s_s + d * CST + b_off, DP * CST);
      }
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        o[i][0] *= lead[0]; o[i][1] *= lead[0];
        o[i][2] *= lead[1]; o[i][3] *= lead[1];
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j0 = (half + 2 * u) * 16;
        if (j0 > row0) continue;
        unsigned pf[PB][4];                                  // the decayed scores, in parts
#pragma unroll
        for (int e = 0; e < 4; ++e) {                        // rows (e & 1), columns 2 t + 8 (e >> 1) and the next
          const int i = e & 1 ? i1 : i0, j = j0 + 2 * t + 8 * (e >> 1);
          const float2 s = *reinterpret_cast<const float2*>(scores + i * W_GST + j);
          float x, y;
          if (MODE == WALK_SPACE) {
            x = j <= i ? s.x * (exp2f((c_hi[e & 1] - c_s[j]) + (c_lo[e & 1] - c_s[W + j])) * c_s[2 * W + j]) : 0.0f;
            y = j + 1 <= i ? s.y * (exp2f((c_hi[e & 1] - c_s[j + 1]) + (c_lo[e & 1] - c_s[W + j + 1])) * c_s[2 * W + j + 1]) : 0.0f;
          } else {
            x = j <= i ? s.x * power_s[i - j] : 0.0f;
            y = j + 1 <= i ? s.y * power_s[i - j - 1] : 0.0f;
          }
          unsigned xy[PB];
          split_parts<PB>(x, y, xy);
#pragma unroll
          for (int q = 0; q < PB; ++q) pf[q][e] = xy[q];
        }
        walk_product<NT, PB, PA>(o, pf, v_s + j0 * CST + b_off, W * CST);
      }
      if (half == 1) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int tok = i0 + 8 * r, c = 8 * i + 2 * t;
            float2 y = make_float2(o[i][2 * r], o[i][2 * r + 1]);
            if (MODE == WALK_SPACE) {
              const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(v_s + tok * CST + c));
              y.x = fmaf(skip, v.x, y.x);
              y.y = fmaf(skip, v.y, y.y);
            }
            *reinterpret_cast<float2*>(o_s + tok * OST + c) = y;
          }
      }
    }
    if (holds) {
      float sum[NT][4] = {};
#pragma unroll
      for (int ks = 0; ks < W / 16; ++ks) {
        if (ks * 16 >= n) continue;
        unsigned af[PA][4];
#pragma unroll
        for (int x = 0; x < PA; ++x) ldmatrix_x4_trans(af[x], k_s + (x * W + ks * 16) * ST + at_off + warp * 16);
        walk_product<NT, PA, PB>(sum, af, wv_s + ks * 16 * CST + b_off, W * CST);
      }
      const float whole = MODE == WALK_SPACE ? exp2f(c_s[W - 1] + c_s[2 * W - 1]) : power_s[n];
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[i][e] = fmaf(whole, S[i][e], sum[i][e]);
    }
    __syncthreads();               // the state's, the values' and the other half's reads are done
    store_state();
    store_values();
    if (half == 0 && row0 < n) {
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int tok = i0 + 8 * r, c = 8 * i + 2 * t;
          if (tok >= n) continue;
          float* to = a.out + (t0 + p * W + tok) * a.H * a.V + static_cast<long long>(h) * a.V + v0 + c;
          const float2 y = *reinterpret_cast<const float2*>(o_s + tok * OST + c);
          if (a.V % 2 == 0 && v0 + c < a.V) {
            *reinterpret_cast<float2*>(to) = make_float2(o[i][2 * r] + y.x, o[i][2 * r + 1] + y.y);
          } else {
            if (v0 + c < a.V) to[0] = o[i][2 * r] + y.x;
            if (v0 + c + 1 < a.V) to[1] = o[i][2 * r + 1] + y.y;
          }
        }
    }
  }
  cp_async_wait<0>();
  if (!a.write_state || !holds) return;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      if (d < a.D && v0 + c < a.V) state[static_cast<long long>(d) * a.V + c] = S[i][e];
    }
}

template <int MODE, int DP, int NT>
static int walk_launch(const WalkArgs& a, int pieces, cudaStream_t s) {
  using Shape = WalkShape<MODE, DP, NT>;
  static_assert(Shape::smem + 1024 <= 227 * 1024, "what a CTA keeps fits in shared memory");
  const int prepare_smem = Shape::qk_bytes;
  auto prepare = walk_prepare_kernel<MODE, DP>;
  auto walk = state_walk_kernel<MODE, DP, NT>;
  if (cuda_failed(cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, prepare_smem)) ||
      cuda_failed(cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::smem)))
    return ERR_CUDA;
  prepare<<<dim3(pieces, a.H / a.heads_per_group), W_THREADS, prepare_smem, s>>>(a);
  walk<<<dim3(a.rows, a.H, (a.V + Shape::COLS - 1) / Shape::COLS), W_THREADS, Shape::smem, s>>>(a);
  return launch_result();
}

template <int MODE>
static int walk_dispatch(const WalkArgs& a, int pieces, cudaStream_t s) {
  // 16 value columns a CTA, 32 where that would be more CTAs than SMs: a CTA takes a whole SM's shared memory, and the
  // second half of them would walk alone.
  const bool wide = static_cast<long long>(a.rows) * a.H * ((a.V + 15) / 16) > 148;
  if (a.D <= 64) return wide ? walk_launch<MODE, 64, 4>(a, pieces, s) : walk_launch<MODE, 64, 2>(a, pieces, s);
  return wide ? walk_launch<MODE, 128, 4>(a, pieces, s) : walk_launch<MODE, 128, 2>(a, pieces, s);
}

}  // namespace zb

using namespace zb;

ZB_API int zb_walk_max_channels() { return 128; }
ZB_API int zb_walk_piece_tokens() { return W; }
// Floats of workspace a piece needs.
ZB_API int zb_walk_piece_floats(int mode, int H, int heads_per_group, int D) {
  const int dp = D <= 64 ? 64 : 128;
  return mode == WALK_SPACE ? H / heads_per_group * W * W_GST + H * W_STEP : H * (W * W_GST + 2 * W * (dp + 8));
}

// mode 0 (state space): q, k, v, dt bfloat16; q, k and their rows on 16-byte boundaries, D a multiple of 8.  mode 1 (fixed
// decays): q, k, v float32.  Constants float32.  ws: (tokens / piece tokens + rows) * zb_walk_piece_floats floats, 16-byte
// aligned, contents irrelevant.  The rows' tokens lie behind one another in the stream, row_q_start ascending.
ZB_API int zb_state_walk(int mode, float* out, const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                         long long v_stride, const void* dt, long long dt_stride, const float* dt_bias, const float* a_log,
                         const float* skip, const float* decay, float* state, long long slot_stride, const int* slots,
                         const int* row_q_start, const int* row_q_len, int rows, int tokens, int H, int D, int V,
                         int heads_per_group, int num_slots, int write_state, float* ws, int* status, void* stream) {
  if (rows < 0 || tokens < 0 || H <= 0 || D <= 0 || V <= 0 || heads_per_group <= 0 || H % heads_per_group != 0 || num_slots <= 0 ||
      (mode != WALK_SPACE && mode != WALK_FIXED) || (mode == WALK_FIXED && (decay == nullptr || heads_per_group != 1)) ||
      (mode == WALK_SPACE && (dt == nullptr || dt_bias == nullptr || a_log == nullptr || skip == nullptr)))
    return ERR_BAD_ARGUMENT;
  if (D > zb_walk_max_channels() || H > 65535 || (V + 15) / 16 > 65535) return ERR_UNSUPPORTED;
  if (rows == 0 || tokens == 0) return OK;
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (ws == nullptr || !aligned(ws) ||
      (mode == WALK_SPACE && (D % 8 != 0 || q_stride % 8 != 0 || k_stride % 8 != 0 || !aligned(q) || !aligned(k))))
    return ERR_BAD_ARGUMENT;
  const int pieces = tokens / W + rows, qk_heads = H / heads_per_group;
  if (qk_heads > 65535) return ERR_UNSUPPORTED;
  WalkArgs a;
  a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride; a.dt = dt; a.dt_stride = dt_stride;
  a.dt_bias = dt_bias; a.a_log = a_log; a.skip = skip; a.decay = decay;
  a.scores = ws;
  a.steps = ws + static_cast<long long>(pieces) * qk_heads * W * W_GST;
  a.parts = reinterpret_cast<__nv_bfloat16*>(a.steps);
  a.out = out; a.state = state; a.slot_stride = slot_stride; a.slots = slots; a.row_q_start = row_q_start; a.row_q_len = row_q_len;
  a.rows = rows; a.H = H; a.D = D; a.V = V; a.heads_per_group = heads_per_group; a.num_slots = num_slots; a.write_state = write_state;
  a.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  return mode == WALK_SPACE ? walk_dispatch<WALK_SPACE>(a, pieces, s) : walk_dispatch<WALK_FIXED>(a, pieces, s);
}
