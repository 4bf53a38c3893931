// Linear attention with one decay per head and token over runs of tokens: per head
//
//   S_t = a_t S_{t-1} + s_t k_t v_t^T,   o_t = S_t^T q_t (+ skip v_t)      (S [D key channels x V value channels], float32)
//
// in two settings: WALK_SPACE, the state-space form of Mamba-2 (a_t = exp(-exp(A_log) dt_t), s_t = dt_t, dt = softplus(. +
// dt_bias); q, k, v bfloat16, q and k shared by the heads of a group), and WALK_FIXED, retention (a_t = a, s_t = 1; q, k, v
// float32).  A request's new tokens of a step are cut into pieces of W tokens.  With S_in the state at a piece's start, n its
// tokens and c_i the sum of the logarithms of its decays up to token i,
//
//   o_i   = e^(c_i) S_in^T q_i + sum_{j <= i} P_ij v_j,   P_ij = e^(c_i - c_j) s_j (q_i . k_j)
//   S_out = e^(c_n) S_in + sum_j w_j k_j v_j^T,           w_j = e^(c_n - c_j) s_j
//
//   walk_prepare   for all pieces side by side: P, e^(c) and w, and q and k as the walk reads them
//   state_walk     a CTA owns a request, a head and some value columns and walks the pieces with the state in registers
//
// so the state never leaves the SM, where passes over all pieces at once write and read every piece's state (2048
// tokens, 32 heads of 128 x 64: 33 MB four times), and a piece is one or two barriers.  Measured: the state-space form, 2048 and 77 tokens,
// 32 heads of 128 x 64: 19 + 61 us, 290 as a scan in segments.  Retention's heads of more than 64 channels take pieces of 128 tokens on
// tcgen05 (retention_tc.cu) but for a few heads' long rows (8 heads of 128 x 128, one row of 2048 tokens 62 us).
//
// Products run on the tensor cores, float32 sums.  A bfloat16 operand is exact; beside it a float32 operand is the sum of three
// bfloat16 values (all its 24 bits).  The tensor cores cut a sum at every step, so there the products of the small parts have
// a sum of their own, and scores two (error against 64 bits over 2048 and 77 tokens: 1.32e-7, 1.82e-7 with one sum each,
// 1.29e-7 token by token).  Two float32 operands (WALK_FIXED) are two bfloat16 values each, hi hi + hi lo + lo hi, a relative
// error of about 2^-16 an operand.  The state itself is only ever touched by float32 multiply-adds.
//
// A value that is not finite must not reach the tokens before it through the zeros above P's diagonal: it is left out of the
// product and added by hand to the outputs of the tokens from its own on.  What is behind it is not finite either, an
// infinity or a NaN.
//
// Sums of logarithms are formed in 64 bits and kept as two float32 values, so that a difference of two is good to a
// rounding of itself.
//
// Pieces are numbered row by row (first_piece_of_row).
#include <type_traits>

#include "common.cuh"
#include "mma.cuh"

namespace zb {

constexpr int W = 64;                    // tokens of a piece
constexpr int W_THREADS = 256;           // of a role: eight warps
constexpr int W_PST = W + 8;             // a row of P
constexpr int W_STEP = 2 * W + 4;        // a head of a piece: e^(c), w, e^(c_n)
constexpr int W_WAIT_LIMIT = 1 << 20;

enum { WALK_SPACE = 0, WALK_FIXED = 1 };

struct WalkArgs {
  const void* q; long long q_stride;     // [tokens, .]: head h (or its group) at column h * D
  const void* k; long long k_stride;
  const void* v; long long v_stride;     // head h at column h * V
  const void* dt; long long dt_stride;   // WALK_SPACE: [tokens, H], bfloat16
  const float* dt_bias; const float* a_log; const float* skip;        // WALK_SPACE: [H] each
  const float* decay;                    // WALK_FIXED: [H]
  unsigned char* qk;                     // [pieces][qk heads][q, k][parts][W][DP + 8] bfloat16
  unsigned char* heads;                  // [pieces][H]{P [parts][W][W_PST] bfloat16, W_STEP floats}
  float* out;                            // [tokens, H * V]
  float* state; long long slot_stride;   // slot s at state + s * slot_stride: [H][D][V]
  const int* slots; const int* row_q_start; const int* row_q_len;
  int rows, from, H, D, V, heads_per_group, num_slots, write_state;      // rows of `from` tokens and more
  const float* freqs; const int* positions;      // WALK_FIXED: null, or q and k are still to be turned (as rotate_qk does)
  int rot_dims;
  float k_scale;
  int vectors, pairs;                    // rows of q and k move as 16-byte pieces; neighbouring values of v move together
  int* status;
};

template <int MODE, int DP>
struct WalkParts {
  using Value = typename std::conditional<MODE == WALK_SPACE, __nv_bfloat16, float>::type;
  static constexpr int PA = MODE == WALK_SPACE ? 1 : 2;      // parts of q, k and v
  static constexpr int PB = MODE == WALK_SPACE ? 3 : 2;      // parts of P, the state and the weighted values
  static constexpr int ST = DP + 8;
  static constexpr int qk_bytes = 2 * PA * W * ST * 2;
  static constexpr int p_bytes = PB * W * W_PST * 2;
  static constexpr int head_bytes = p_bytes + W_STEP * 4;
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

// B over 16 of k and N tiles of 8 columns: parts of [k][st] tiles `part_stride` elements apart, from this lane's ldmatrix
// address inside the first 16 x 16 block on.
template <int N, int PB>
struct WalkB {
  unsigned f[PB][N / 2][4];
  __device__ __forceinline__ void load(const __nv_bfloat16* b, int part_stride) {
#pragma unroll
    for (int pb = 0; pb < PB; ++pb)
#pragma unroll
      for (int n = 0; n < N / 2; ++n) ldmatrix_x4_trans(f[pb][n], b + pb * part_stride + n * 16);
  }
};
// acc + low += A B, the products of large parts in acc, all others in low (which may be acc).  The tiles take turns, so that no
// product waits for the one before it.
template <int N, int PA, int PB>
__device__ __forceinline__ void walk_product(float (&acc)[N][4], float (&low)[N][4], const unsigned (&af)[PA][4], const WalkB<N, PB>& b) {
#pragma unroll
  for (int pb = PB - 1; pb >= 0; --pb)                       // the small products first
#pragma unroll
    for (int pa = PA - 1; pa >= 0; --pa)
      if (counts<PA, PB>(pa, pb)) {
#pragma unroll
        for (int n = 0; n < N; ++n) mma_bf16_16816(pa + pb > 0 ? low[n] : acc[n], af[pa], b.f[pb][n / 2][n % 2 * 2], b.f[pb][n / 2][n % 2 * 2 + 1]);
      }
}

// A piece of one q/k head and up to W_HEADS of the heads that share it (their scores are the same).  DP: the channels padded
// with zeros.
constexpr int W_HEADS = 4;
template <int MODE, int DP>
__global__ void __launch_bounds__(W_THREADS) walk_prepare_kernel(const WalkArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  using Parts = WalkParts<MODE, DP>;
  constexpr int ST = Parts::ST, PA = Parts::PA, PB = Parts::PB, HEADS = MODE == WALK_SPACE ? W_HEADS : 1;
  extern __shared__ __align__(16) unsigned char w_smem[];
  __shared__ float c_hi[HEADS][W], c_lo[HEADS][W], s_s[HEADS][W];
  const int piece = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int runs = (a.heads_per_group + HEADS - 1) / HEADS;              // runs of heads in a group
  const int qk_head = blockIdx.y / runs, first_head = blockIdx.y % runs * HEADS, qk_heads = a.H / a.heads_per_group;
  const int heads = min(HEADS, a.heads_per_group - first_head), h0 = qk_head * a.heads_per_group + first_head;
  int own;
  const int row = row_of_piece<W>(a.row_q_len, a.rows, a.from, piece, own);
  if (row < 0) return;
  const int begin = own * W, n = min(W, a.row_q_len[row] - begin);
  const long long t0 = a.row_q_start[row] + begin;
  __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(w_smem);        // [PA][W][ST]
  __nv_bfloat16* k_s = q_s + PA * W * ST;                               // [PA][W][ST]
  if (MODE == WALK_SPACE) {
    const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(a.q) + t0 * a.q_stride + qk_head * a.D;
    const __nv_bfloat16* k = static_cast<const __nv_bfloat16*>(a.k) + t0 * a.k_stride + qk_head * a.D;
#pragma unroll
    for (int u = 0; u < W * (DP / 8) / W_THREADS; ++u) {
      const int e = tid + u * W_THREADS, i = e / (DP / 8), c = e % (DP / 8) * 8;
      const bool ok = i < n && c < a.D;
      cp_async_16(q_s + i * ST + c, ok ? q + i * a.q_stride + c : q, ok);
      cp_async_16(k_s + i * ST + c, ok ? k + i * a.k_stride + c : k, ok);
    }
    cp_async_commit();
  } else {
    const float* q = static_cast<const float*>(a.q) + t0 * a.q_stride + qk_head * a.D;
    const float* k = static_cast<const float*>(a.k) + t0 * a.k_stride + qk_head * a.D;
    const int half = a.freqs != nullptr ? a.rot_dims / 2 : 0;
    // Values that turn: four pairs of q and four of k a thread and step, on one set of angles.
    for (int e = tid; e < W * (half / 4); e += W_THREADS) {
      const int i = e / (half / 4), c = e % (half / 4) * 4;
      float4 x[2][2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          x[u][w] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (i < n) x[u][w] = *reinterpret_cast<const float4*>((u ? k + i * a.k_stride : q + i * a.q_stride) + c + w * half);
        }
      const float pos = i < n ? static_cast<float>(a.positions[t0 + i]) : 0.0f;
      float sn[4], cs[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) sincosf(pos * a.freqs[c + w], &sn[w], &cs[w]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float scale = u ? a.k_scale : 1.0f;
        const float4 y = x[u][0], z = x[u][1];
        const float4 out[2] = {make_float4((y.x * cs[0] - z.x * sn[0]) * scale, (y.y * cs[1] - z.y * sn[1]) * scale,
                                           (y.z * cs[2] - z.z * sn[2]) * scale, (y.w * cs[3] - z.w * sn[3]) * scale),
                               make_float4((z.x * cs[0] + y.x * sn[0]) * scale, (z.y * cs[1] + y.y * sn[1]) * scale,
                                           (z.z * cs[2] + y.z * sn[2]) * scale, (z.w * cs[3] + y.w * sn[3]) * scale)};
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          unsigned lo[2], hi[2];
          split_parts<2>(out[w].x, out[w].y, lo);
          split_parts<2>(out[w].z, out[w].w, hi);
          __nv_bfloat16* to = (u ? k_s : q_s) + i * ST + c + w * half;
#pragma unroll
          for (int p = 0; p < 2; ++p) *reinterpret_cast<uint2*>(to + p * W * ST) = make_uint2(lo[p], hi[p]);
        }
      }
    }
    const float passing = a.freqs != nullptr ? a.k_scale : 1.0f;         // what does not turn, k times its multiplier
    const int from_c = 2 * half, quads = (DP - from_c) / 4;
    constexpr int AHEAD = 8;             // loads on their way before the first of them is waited for
    for (int e0 = tid; e0 < 2 * W * quads; e0 += W_THREADS * AHEAD) {
      float4 x[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int e = e0 + u * W_THREADS, r = e % (W * quads), i = r / quads, c = from_c + r % quads * 4;
        const float* from = e >= W * quads ? k + i * a.k_stride + c : q + i * a.q_stride + c;
        x[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (e < 2 * W * quads && i < n && c < a.D) {
          if (a.vectors) {
            x[u] = *reinterpret_cast<const float4*>(from);
          } else {
            x[u].x = from[0];
            if (c + 1 < a.D) x[u].y = from[1];
            if (c + 2 < a.D) x[u].z = from[2];
            if (c + 3 < a.D) x[u].w = from[3];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int e = e0 + u * W_THREADS, r = e % (W * quads), i = r / quads, c = from_c + r % quads * 4;
        if (e >= 2 * W * quads) break;
        const float scale = e >= W * quads ? passing : 1.0f;
        unsigned lo[2], hi[2];
        split_parts<2>(x[u].x * scale, x[u].y * scale, lo);
        split_parts<2>(x[u].z * scale, x[u].w * scale, hi);
        __nv_bfloat16* to = (e >= W * quads ? k_s : q_s) + i * ST + c;
#pragma unroll
        for (int p = 0; p < 2; ++p) *reinterpret_cast<uint2*>(to + p * W * ST) = make_uint2(lo[p], hi[p]);
      }
    }
  }
  unsigned char* head0 = a.heads + (static_cast<long long>(piece) * a.H + h0) * Parts::head_bytes;
  if (warp < heads) {
    const int h = h0 + warp;
    // Steps and decays: two tokens a lane, the sum scanned in 64 bits (in powers of two).
    float step[2];
    double sum[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = 2 * lane + u;
      if (MODE == WALK_SPACE) {
        const __nv_bfloat16* dt = static_cast<const __nv_bfloat16*>(a.dt) + t0 * a.dt_stride + h;
        step[u] = i < n ? walk_softplus(__bfloat162float(dt[i * a.dt_stride]) + a.dt_bias[h]) : 0.0f;
        sum[u] = static_cast<double>(expf(a.a_log[h])) * static_cast<double>(step[u]) * 1.4426950408889634;
      } else {
        step[u] = i < n ? 1.0f : 0.0f;
        sum[u] = i < n ? -log2(static_cast<double>(a.decay[h])) : 0.0;
      }
      // (a decay below 2^-1000 is zero either way; the bound keeps the sums finite)
      sum[u] = -fmin(sum[u], 1000.0);
    }
    sum[1] += sum[0];
    double before = sum[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double other = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += other;
    }
    const double all = __shfl_sync(0xffffffffu, before, 31);
    before -= sum[1];
    float* steps = reinterpret_cast<float*>(head0 + warp * Parts::head_bytes + Parts::p_bytes);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = 2 * lane + u;
      const double c = before + sum[u];
      c_hi[warp][i] = static_cast<float>(c);
      c_lo[warp][i] = static_cast<float>(c - static_cast<float>(c));
      s_s[warp][i] = step[u];
      steps[i] = exp2f(static_cast<float>(c));
      steps[W + i] = exp2f(static_cast<float>(all - c)) * step[u];
    }
    if (lane == 0) steps[2 * W] = exp2f(static_cast<float>(all));
  }
  if (MODE == WALK_SPACE) cp_async_wait<0>();
  __syncthreads();
  if (first_head == 0) {
    uint4* to = reinterpret_cast<uint4*>(a.qk + (static_cast<long long>(piece) * qk_heads + qk_head) * Parts::qk_bytes);
    const uint4* from = reinterpret_cast<const uint4*>(q_s);
    for (int e = tid; e < Parts::qk_bytes / 16; e += W_THREADS) to[e] = from[e];
  }
  // A warp owns 16 rows of P and 32 columns; what lies behind the diagonal tile is never read.
  const int g = lane >> 2, t = lane & 3, row0 = (warp & 3) * 16, col0 = (warp >> 2) * 32;
  const int q_off = (row0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ST + (lane >> 4) * 8;
  const int k_off = ((lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int c0 = col0 + u * 16;
    if (c0 > row0) continue;
    float s2[2][2][4] = {}, s[2][4];
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
            mma_bf16_16816(s2[ks & 1][0], af[pa], bf[pb][0], bf[pb][1]);
            mma_bf16_16816(s2[ks & 1][1], af[pa], bf[pb][2], bf[pb][3]);
          }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[i][e] = s2[0][i][e] + s2[1][i][e];
    for (int w = 0; w < heads; ++w) {
      unsigned char* head = head0 + w * Parts::head_bytes;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int at = row0 + g + 8 * r, j = c0 + 8 * i + 2 * t;
          float x[2];
#pragma unroll
          for (int e = 0; e < 2; ++e)
            x[e] = j + e <= at
                       ? s[i][2 * r + e] * (exp2f((c_hi[w][at] - c_hi[w][j + e]) + (c_lo[w][at] - c_lo[w][j + e])) * s_s[w][j + e])
                       : 0.0f;
          unsigned part[PB];
          split_parts<PB>(x[0], x[1], part);
#pragma unroll
          for (int p = 0; p < PB; ++p) *reinterpret_cast<unsigned*>(head + ((p * W + at) * W_PST + j) * 2) = part[p];
        }
    }
  }
}

template <int MODE, int DP, bool ROLES>
struct WalkShape : WalkParts<MODE, DP> {
  using Parts = WalkParts<MODE, DP>;
  static constexpr int NT = ROLES ? 2 : 4; // tiles of 8 value columns of a CTA
  static constexpr int BUFFERS = ROLES ? 2 : 1, THREADS = ROLES ? 2 * W_THREADS : W_THREADS;
  static constexpr int COLS = 8 * NT, CST = COLS + 8, OST = COLS + 4, STAGES = 2;
  static constexpr int stage_bytes = Parts::qk_bytes + Parts::head_bytes;
  static constexpr int state_elems = Parts::PB * DP * CST, value_elems = (Parts::PA + Parts::PB) * W * CST;       // of a buffer each
  static constexpr int smem = STAGES * stage_bytes + BUFFERS * (state_elems + value_elems) * 2 + W * OST * 4;
};

// The values of a piece that are not finite, added to the outputs of tokens i0 and i0 + 8, columns c0 and c0 + 1 of each of `tiles`
// tiles of 8; `v` and `out` begin at the piece's first token and the CTA's first of `cols` columns.  (A call of its own, with plain
// arguments: inlined, its registers cost every piece 10 % of the walk.)
template <typename T, int PB>
__device__ __noinline__ void add_wild(float* out, long long out_stride, const T* v, long long v_stride, int n, int cols, int tiles, int i0,
                                      int c0, float skip, const __nv_bfloat16* p_s) {
  for (int e = 0; e < 4 * tiles; ++e) {
    const int tok = i0 + (e & 2) * 4, c = e / 4 * 8 + c0 + (e & 1);
    if (tok >= n || c >= cols) continue;
    for (int j = 0; j <= tok; ++j) {
      const float x = to_float(v[j * v_stride + c]);
      if (isfinite(x)) continue;
      float weight = j == tok ? skip : 0.0f;
      for (int q = 0; q < PB; ++q) weight += __bfloat162float(p_s[(q * W + tok) * W_PST + j]);
      out[tok * out_stride + c] = fmaf(weight, x, out[tok * out_stride + c]);
    }
  }
}

// Zeros in the place of values that are not finite.
__device__ __noinline__ void drop_wild(__nv_bfloat16* v_s, int count) {
  for (int e = threadIdx.x; e < count; e += W_THREADS)
    if (!isfinite(__bfloat162float(v_s[e]))) v_s[e] = __float2bfloat16_rn(0.0f);
}

// For the outputs, warp w owns tokens 16 (w % 4) .. and takes half the channels (S^T q) and every other 16 keys (P); the halves meet in
// shared memory, each writing out half of the columns.  Of the state, warp w owns the channels 16 w .. (C fragments).  The next
// piece comes meanwhile, in two bulk copies.  Two forms:
//   * ROLES: sixteen warps and 16 value columns; eight warps make the outputs, eight carry the state on, and a piece is one barrier of all
//     of them, behind which both work from the state's and the values' parts in one of two buffers while the state's warps
//     fill the other: 2900 cycles a piece of the state-space form, where eight warps that did both one after the other took 3150;
//   * else eight warps and 32 value columns: outputs and state one after the other, a barrier, the next piece's parts.
// Bound by shared memory, ROLES at four fifths of it: 40 ldmatrix a warp of 16 columns, the parts' stores and the copies of 63 KB a piece.
template <int MODE, int DP, bool ROLES>
__global__ void __launch_bounds__(ROLES ? 2 * W_THREADS : W_THREADS, 1) state_walk_kernel(const WalkArgs a) {
  using Shape = WalkShape<MODE, DP, ROLES>;
  constexpr int NT = Shape::NT;
  constexpr bool SPLIT_SUMS = MODE == WALK_SPACE;
  constexpr int PA = Shape::PA, PB = Shape::PB, ST = Shape::ST, COLS = Shape::COLS, CST = Shape::CST, OST = Shape::OST;
  constexpr int STAGES = Shape::STAGES, PER = W * COLS / W_THREADS / 2;      // pairs of values a thread brings of a piece
  extern __shared__ __align__(16) unsigned char w_smem[];
  __nv_bfloat16* const state_s = reinterpret_cast<__nv_bfloat16*>(w_smem + STAGES * Shape::stage_bytes);     // [buffers][PB][DP][CST]
  __nv_bfloat16* const values_s = state_s + Shape::BUFFERS * Shape::state_elems;      // [buffers]{v [PA][W][CST], w_j v_j [PB][W][CST]}
  float* o_s = reinterpret_cast<float*>(values_s + Shape::BUFFERS * Shape::value_elems);        // [W][OST]
  __shared__ unsigned long long landed[STAGES];
  __shared__ int wild[2];                                    // the last even and odd piece with a value that is not finite
  const int row = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * COLS;
  const bool states = !ROLES || threadIdx.x >= W_THREADS;    // the warp's role
  const int tid = threadIdx.x % W_THREADS, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;      // within it
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) {
    if (threadIdx.x == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
    return;
  }
  const int n_all = a.row_q_len[row], pieces = (n_all + W - 1) / W;
  if (n_all < a.from) return;
  const long long t0 = a.row_q_start[row];
  const int first = first_piece_of_row<W>(a.row_q_len, row, a.from), qk_head = h / a.heads_per_group, qk_heads = a.H / a.heads_per_group;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < STAGES; ++i) mbar_init(&landed[i], 1);
    fence_barrier_init();
    wild[0] = wild[1] = -1;
  }
  __syncthreads();

  auto copy_piece = [&](int p) {                             // one thread
    unsigned char* stage = w_smem + p % STAGES * Shape::stage_bytes;
    unsigned long long* bar = &landed[p % STAGES];
    mbar_arrive_expect_tx(bar, Shape::stage_bytes);
    bulk_copy_g2s(stage, a.qk + (static_cast<long long>(first + p) * qk_heads + qk_head) * Shape::qk_bytes, Shape::qk_bytes, bar);
    bulk_copy_g2s(stage + Shape::qk_bytes, a.heads + (static_cast<long long>(first + p) * a.H + h) * Shape::head_bytes,
                  Shape::head_bytes, bar);
  };
  // This thread's values of a piece: columns my_c and my_c + 1 of tokens my_i, my_i + TOKENS, ..., and their weights.
  constexpr int TOKENS = W / PER;
  const int my_c = tid % (COLS / 2) * 2, my_i = tid / (COLS / 2);
  float value[PER][2], weight[PER];
  unsigned raw[PER];
  const bool col0 = v0 + my_c < a.V, col1 = v0 + my_c + 1 < a.V;
  auto fetch_values = [&](int p) {                           // (nothing here waits for what it loads)
    const float* w = reinterpret_cast<const float*>(a.heads + (static_cast<long long>(first + p) * a.H + h) * Shape::head_bytes +
                                                    Shape::p_bytes) + W;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = my_i + u * TOKENS, at = p * W + i, n = min(W, n_all - p * W);
      value[u][0] = value[u][1] = weight[u] = 0.0f;
      raw[u] = 0;
      if (p >= pieces || i >= n) continue;
      weight[u] = w[i];
      if (MODE == WALK_SPACE) {
        const unsigned short* v = static_cast<const unsigned short*>(a.v) + (t0 + at) * a.v_stride + h * a.V + v0 + my_c;
        if (a.pairs && col1) raw[u] = *reinterpret_cast<const unsigned*>(v);
        else if (col0) raw[u] = v[0] | (col1 ? static_cast<unsigned>(v[1]) << 16 : 0u);
      } else {
        const float* v = static_cast<const float*>(a.v) + (t0 + at) * a.v_stride + h * a.V + v0 + my_c;
        if (a.pairs && col1) {
          const float2 x = *reinterpret_cast<const float2*>(v);
          value[u][0] = x.x;
          value[u][1] = x.y;
        } else {
          if (col0) value[u][0] = v[0];
          if (col1) value[u][1] = v[1];
        }
      }
    }
  };
  auto store_values = [&](int p) {
    __nv_bfloat16* const v_s = values_s + p % Shape::BUFFERS * Shape::value_elems, * const wv_s = v_s + PA * W * CST;
    float top = 0.0f;                                        // NaN if one of the values is not finite
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int at = (my_i + u * TOKENS) * CST + my_c;
      unsigned vp[PA], wp[PB];
      if (MODE == WALK_SPACE) {
        vp[0] = raw[u];
        value[u][0] = __uint_as_float(raw[u] << 16);
        value[u][1] = __uint_as_float(raw[u] & 0xffff0000u);
      } else {
        split_parts<PA>(value[u][0], value[u][1], vp);
      }
      top = fmaf(0.0f, value[u][0], fmaf(0.0f, value[u][1], top));
      split_parts<PB>(value[u][0] * weight[u], value[u][1] * weight[u], wp);
#pragma unroll
      for (int i = 0; i < PA; ++i) *reinterpret_cast<unsigned*>(v_s + i * W * CST + at) = vp[i];
#pragma unroll
      for (int i = 0; i < PB; ++i) *reinterpret_cast<unsigned*>(wv_s + i * W * CST + at) = wp[i];
    }
    if (top != 0.0f) wild[p & 1] = p;
  };
  // This thread's part of the state: channels d0 and d0 + 8, columns 8 i + 2 t and the next.
  const int d0 = warp * 16 + g;
  const bool holds = states && warp * 16 < DP;
  float S[NT][4];
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride + static_cast<long long>(h) * a.D * a.V + v0;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      S[i][e] = holds && d < a.D && v0 + c < a.V ? state[static_cast<long long>(d) * a.V + c] : 0.0f;
    }
  auto store_state = [&](int p) {                            // as piece p finds it
    if (!holds) return;
    __nv_bfloat16* const s_s = state_s + p % Shape::BUFFERS * Shape::state_elems;
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
  if (threadIdx.x == 0 && pieces > 0) copy_piece(0);
  if (states) {
    store_state(0);
    fetch_values(0);
    store_values(0);
  }
  const float skip = MODE == WALK_SPACE ? a.skip[h] : 0.0f;
  // ldmatrix addresses: A rows as they lie, P's likewise, A transposed, B as [k][n].
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;
  const int a_off = lrow * ST + lcol, p_off = lrow * W_PST + lcol, b_off = lrow * CST + lcol;
  const int at_off = ((lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8;
  constexpr int MINE = NT / 2;                               // tiles of value columns whose outputs a warp writes
  const int row0 = (warp & 3) * 16, half = warp >> 2, first_c = half * MINE * 8;
  for (int p = 0; p < pieces; ++p) {
    const unsigned char* stage = w_smem + p % STAGES * Shape::stage_bytes;
    const __nv_bfloat16* q_s = reinterpret_cast<const __nv_bfloat16*>(stage);              // [PA][W][ST]
    const __nv_bfloat16* k_s = q_s + PA * W * ST;
    const __nv_bfloat16* p_s = reinterpret_cast<const __nv_bfloat16*>(stage + Shape::qk_bytes);        // [PB][W][W_PST]
    const float* steps = reinterpret_cast<const float*>(stage + Shape::qk_bytes + Shape::p_bytes);
    const __nv_bfloat16* s_s = state_s + p % Shape::BUFFERS * Shape::state_elems;
    __nv_bfloat16* v_s = values_s + p % Shape::BUFFERS * Shape::value_elems;
    const __nv_bfloat16* wv_s = v_s + PA * W * CST;
    const int n = min(W, n_all - p * W);
    const bool here = mbar_wait(&landed[p % STAGES], (p / STAGES) & 1, W_WAIT_LIMIT);
    // The piece, the state and the values are there; the buffers of the piece before are free.
    if (!__syncthreads_and(here)) {
      if (threadIdx.x == 0) report(a.status, STATUS_COPY_TIMEOUT, p, row);
      let_copies_land();
      return;
    }
    if (states) {
      if (tid == W_THREADS - 32 && p + 1 < pieces) copy_piece(p + 1);
      fetch_values(p + 1);
    }
    auto carry_on = [&] {
      if (!holds) return;
      float sum[NT][4] = {}, sum_low[NT][4] = {};
#pragma unroll
      for (int ks = 0; ks < W / 16; ++ks) {
        unsigned af[PA][4];
        WalkB<NT, PB> b;
#pragma unroll
        for (int x = 0; x < PA; ++x) ldmatrix_x4_trans(af[x], k_s + (x * W + ks * 16) * ST + at_off + warp * 16);
        b.load(wv_s + ks * 16 * CST + b_off, W * CST);
        walk_product<NT, PA, PB>(sum, SPLIT_SUMS ? sum_low : sum, af, b);
      }
      const float whole = steps[2 * W];
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[i][e] = fmaf(whole, S[i][e], SPLIT_SUMS ? sum[i][e] + sum_low[i][e] : sum[i][e]);
    };
    if (ROLES && states) {
      carry_on();
      store_state(p + 1);
      store_values(p + 1);
      continue;
    }
    const int i0 = row0 + g, i1 = i0 + 8;
    const bool tame = wild[p & 1] != p;
    auto outputs_meet = [] { asm volatile("bar.sync 1, 256;\n" ::: "memory"); };
    if (!tame) {
      drop_wild(v_s, PA * W * CST);
      outputs_meet();
    }
    float o[NT][4] = {}, own_low[NT][4] = {};
    float (&low)[NT][4] = SPLIT_SUMS ? own_low : o;
    if (row0 < n) {
#pragma unroll
      for (int ks = 0; ks < DP / 32; ++ks) {
        const int d = half * (DP / 2) + ks * 16;
        unsigned af[PA][4];
        WalkB<NT, PB> b;
#pragma unroll
        for (int x = 0; x < PA; ++x) ldmatrix_x4(af[x], q_s + (x * W + row0) * ST + a_off + d);
        b.load(s_s + d * CST + b_off, DP * CST);
        walk_product<NT, PA, PB>(o, low, af, b);
      }
      const float lead0 = steps[i0], lead1 = steps[i1];
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        o[i][0] *= lead0; o[i][1] *= lead0;
        o[i][2] *= lead1; o[i][3] *= lead1;
        if (SPLIT_SUMS) {
          low[i][0] *= lead0; low[i][1] *= lead0;
          low[i][2] *= lead1; low[i][3] *= lead1;
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j0 = (half + 2 * u) * 16;
        if (j0 > row0) continue;
        unsigned pf[PB][4];
        WalkB<NT, PA> b;
#pragma unroll
        for (int x = 0; x < PB; ++x) ldmatrix_x4(pf[x], p_s + (x * W + row0) * W_PST + p_off + j0);
        b.load(v_s + j0 * CST + b_off, W * CST);
        walk_product<NT, PB, PA>(o, low, pf, b);
      }
      if (SPLIT_SUMS) {
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[i][e] += low[i][e];
      }
      // The other half of the tokens' warps gets what this one has of the tiles that it writes out.
      {
#pragma unroll
        for (int i = 0; i < MINE; ++i)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int tok = i0 + 8 * r, c = 8 * (half == 0 ? MINE + i : i) + 2 * t;
            float2 y = half == 0 ? make_float2(o[MINE + i][2 * r], o[MINE + i][2 * r + 1]) : make_float2(o[i][2 * r], o[i][2 * r + 1]);
            if (MODE == WALK_SPACE) {
              const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(v_s + tok * CST + c));
              y.x = fmaf(skip, v.x, y.x);
              y.y = fmaf(skip, v.y, y.y);
            }
            *reinterpret_cast<float2*>(o_s + tok * OST + c) = y;
          }
      }
    }
    if (ROLES) {
      outputs_meet();
    } else {
      carry_on();
      __syncthreads();             // the state's, the values' and the piece's reads are done
      store_state(p + 1);
      store_values(p + 1);
    }
    if (row0 < n) {
#pragma unroll
      for (int i = 0; i < MINE; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int tok = i0 + 8 * r, c = first_c + 8 * i + 2 * t;
          if (tok >= n) continue;
          float* to = a.out + (t0 + p * W + tok) * a.H * a.V + static_cast<long long>(h) * a.V + v0 + c;
          const float2 y = *reinterpret_cast<const float2*>(o_s + tok * OST + c);
          const float2 x = half == 0 ? make_float2(o[i][2 * r], o[i][2 * r + 1]) : make_float2(o[MINE + i][2 * r], o[MINE + i][2 * r + 1]);
          if (a.V % 2 == 0 && v0 + c < a.V) {
            *reinterpret_cast<float2*>(to) = make_float2(x.x + y.x, x.y + y.y);
          } else {
            if (v0 + c < a.V) to[0] = x.x + y.x;
            if (v0 + c + 1 < a.V) to[1] = x.y + y.y;
          }
        }
      // (the outputs that this thread has just written; the piece's buffer is filled again behind the next barrier of all warps)
      if (!tame) {
        using T = typename Shape::Value;
        const long long at = t0 + p * W;
        add_wild<T, PB>(a.out + at * a.H * a.V + static_cast<long long>(h) * a.V + v0 + first_c, static_cast<long long>(a.H) * a.V,
                        static_cast<const T*>(a.v) + at * a.v_stride + h * a.V + v0 + first_c, a.v_stride, n, a.V - v0 - first_c, MINE, i0, 2 * t,
                        skip, p_s);
      }
    }
  }
  if (!a.write_state || !holds) return;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      if (d < a.D && v0 + c < a.V) state[static_cast<long long>(d) * a.V + c] = S[i][e];
    }
}

template <int MODE, int DP, bool ROLES>
static int walk_launch(const WalkArgs& a, int pieces, cudaStream_t s) {
  using Shape = WalkShape<MODE, DP, ROLES>;
  static_assert(Shape::smem + 256 <= 227 * 1024, "what a CTA keeps fits in shared memory");
  static_assert(Shape::qk_bytes % 16 == 0 && Shape::head_bytes % 16 == 0, "bulk copies move 16-byte pieces");
  auto prepare = walk_prepare_kernel<MODE, DP>;
  auto walk = state_walk_kernel<MODE, DP, ROLES>;
  if (cuda_failed(cudaFuncSetAttribute(prepare, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::qk_bytes)) ||
      cuda_failed(cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::smem)))
    return ERR_CUDA;
  const int heads = MODE == WALK_SPACE ? W_HEADS : 1;
  launch_dependent(prepare, dim3(pieces, a.H / a.heads_per_group * ((a.heads_per_group + heads - 1) / heads)),
      dim3(W_THREADS), Shape::qk_bytes, s, false, a);
  // (Not as a dependent, which would fill the SMs that are free first instead of all of them.)
  walk<<<dim3(a.rows, a.H, (a.V + Shape::COLS - 1) / Shape::COLS), Shape::THREADS, Shape::smem, s>>>(a);
  return launch_result();
}

template <int MODE>
static int walk_dispatch(const WalkArgs& a, int pieces, cudaStream_t s) {
  // 16 value columns a CTA and a role a warp, or 32 and all of it: a CTA takes an SM.  Up to two of the narrow ones an SM they are ahead, far so where one
  // row is much the longest (us, narrow / wide, state-space form, 32 heads of 128 x 64: 2048 and 77 tokens 74 / 90, one row of 2048 65; but twelve of
  // 150 87 / 83, thirty of 64 121 / 97, four of 500 72 / 68; fixed decays, 32 heads of 64 x 128, three rows of 700 125 / 107).
  const bool wide = static_cast<long long>(a.rows) * a.H * ((a.V + 15) / 16) > 2 * 148;
  if (a.D <= 64) return wide ? walk_launch<MODE, 64, false>(a, pieces, s) : walk_launch<MODE, 64, true>(a, pieces, s);
  return wide ? walk_launch<MODE, 128, false>(a, pieces, s) : walk_launch<MODE, 128, true>(a, pieces, s);
}


}  // namespace zb

using namespace zb;

ZB_API int zb_walk_max_channels() { return 128; }
ZB_API int zb_walk_piece_tokens() { return W; }
// Floats of workspace a piece needs.
ZB_API int zb_walk_piece_floats(int mode, int H, int heads_per_group, int D) {
  if (mode == WALK_SPACE) {
    const int qk = D <= 64 ? WalkParts<WALK_SPACE, 64>::qk_bytes : WalkParts<WALK_SPACE, 128>::qk_bytes;
    return (H / heads_per_group * qk + H * WalkParts<WALK_SPACE, 64>::head_bytes) / 4;
  }
  const int qk = D <= 64 ? WalkParts<WALK_FIXED, 64>::qk_bytes : WalkParts<WALK_FIXED, 128>::qk_bytes;
  return H * (qk + WalkParts<WALK_FIXED, 64>::head_bytes) / 4;
}

// mode 0 (state space): q, k, v, dt bfloat16; q, k and their rows on 16-byte boundaries, D a multiple of 8.  mode 1 (fixed
// decays): q, k, v float32; with `freqs` (rot_dims / 2 of them) q and k are turned by the tokens' positions first, as
// zb_rotate_qk does, k times k_scale (rot_dims a multiple of 8, D of 4, rows on 16-byte boundaries).  Constants float32.
// ws: (tokens / piece tokens + rows) * zb_walk_piece_floats floats, 16-byte aligned, contents irrelevant.  Rows of fewer than
// `from` tokens are left alone; the rows' tokens may lie in the stream in any order.
ZB_API int zb_state_walk(int mode, float* out, const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                         long long v_stride, const void* dt, long long dt_stride, const float* dt_bias, const float* a_log,
                         const float* skip, const float* decay, float* state, long long slot_stride, const int* slots,
                         const int* row_q_start, const int* row_q_len, int rows, int tokens, int from, int H, int D, int V,
                         int heads_per_group, int num_slots, int write_state, const float* freqs, int rot_dims, float k_scale,
                         const int* positions, float* ws, int* status, void* stream) {
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
  WalkArgs a;
  a.freqs = freqs; a.positions = positions; a.rot_dims = freqs != nullptr ? rot_dims : 0; a.k_scale = k_scale;
  a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride; a.dt = dt; a.dt_stride = dt_stride;
  a.dt_bias = dt_bias; a.a_log = a_log; a.skip = skip; a.decay = decay;
  a.qk = reinterpret_cast<unsigned char*>(ws);
  const int qk_bytes = mode == WALK_SPACE ? (D <= 64 ? WalkParts<WALK_SPACE, 64>::qk_bytes : WalkParts<WALK_SPACE, 128>::qk_bytes)
                                          : (D <= 64 ? WalkParts<WALK_FIXED, 64>::qk_bytes : WalkParts<WALK_FIXED, 128>::qk_bytes);
  a.heads = a.qk + static_cast<long long>(pieces) * qk_heads * qk_bytes;
  a.vectors = mode == WALK_SPACE || (D % 4 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && aligned(q) && aligned(k));
  if (freqs != nullptr && (mode != WALK_FIXED || !a.vectors || positions == nullptr || rot_dims < 0 || rot_dims > D || rot_dims % 8 != 0))
    return ERR_BAD_ARGUMENT;
  a.out = out; a.state = state; a.slot_stride = slot_stride; a.slots = slots; a.row_q_start = row_q_start; a.row_q_len = row_q_len;
  a.pairs = V % 2 == 0 && v_stride % 2 == 0 && reinterpret_cast<uintptr_t>(v) % (mode == WALK_SPACE ? 4 : 8) == 0;
  a.rows = rows; a.from = from; a.H = H; a.D = D; a.V = V; a.heads_per_group = heads_per_group; a.num_slots = num_slots; a.write_state = write_state;
  a.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  return mode == WALK_SPACE ? walk_dispatch<WALK_SPACE>(a, pieces, s) : walk_dispatch<WALK_FIXED>(a, pieces, s);
}
