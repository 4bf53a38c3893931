// The gated delta rule: per head a state S [D key channels x V value channels], float32, and per token
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//
// with one decay g and one step beta per head and token.  Token by token, in two kernels:
//
//   delta_gates   per token: q and k heads (the model's type, as a convolution left them) made unit
//                 vectors, x / sqrt(sum(x^2) + unit_eps), q also times `q_scale`, both written as
//                 float32; beta = sigmoid(b); g = exp(-exp(A_log) softplus(a + dt_bias)), from float32
//                 projections b and a.
//   delta_scan    a CTA owns a request, a head and a run of value columns; a column is shared by L
//                 lanes that hold D / L key channels of it each.  With r_k = S^T k and r_q = S^T q of
//                 the state BEFORE the token, u = beta (v - g r_k) and o = g r_q + u (k . q): both
//                 reductions run side by side on the old state, and the write S <- g S + k u^T
//                 follows.  A request's tokens run in their order, 16 at a time staged in shared memory;
//                 the state is read from the request's slot at the start of the step's portion and
//                 written back at its end, so a prompt may be cut anywhere.  In the slot a head's state
//                 lies [V][D] (a column's channels together).
//
// Rows that bring runs of tokens go to two other kernels (delta_blocks, delta_block_scan below): the same rule, block by
// block of 16 tokens.
//
// Everything here is float32 multiply-adds in either form; the values v are read in the model's type.
#include "common.cuh"
#include "mma.cuh"

namespace zb {

__device__ __forceinline__ float softplus_d(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

struct DeltaGatesArgs {
  float* q_out;            // [T, qk_heads * D]
  float* k_out;            // [T, qk_heads * D]
  float* beta;             // [T, heads]
  float* decay;            // [T, heads]
  const void* q;           // [T, q_stride] the model's type
  const void* k;
  long long q_stride, k_stride;
  const float* b;          // [T, ba_stride]
  const float* a;
  long long ba_stride;
  const float* a_log;      // [heads]
  const float* dt_bias;    // [heads]
  int qk_heads, heads, D;
  float q_scale, unit_eps;
  const int* row_q_start;  // below > 0: only the tokens of rows with fewer than `below` tokens
  const int* row_q_len;
  int rows, below;
};

template <typename T>
__global__ void __launch_bounds__(128) delta_gates_kernel(const DeltaGatesArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  const long long t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (a.below > 0) {
    bool wanted = false;
    for (int r = threadIdx.x; r < a.rows; r += blockDim.x) {
      const int n = a.row_q_len[r];
      wanted |= n < a.below && t >= a.row_q_start[r] && t < a.row_q_start[r] + n;
    }
    if (!__syncthreads_or(wanted)) return;
  }
  for (int h = warp; h < 2 * a.qk_heads; h += 4) {
    const bool is_q = h < a.qk_heads;
    const int own = is_q ? h : h - a.qk_heads;
    const T* src = is_q ? static_cast<const T*>(a.q) + t * a.q_stride + own * a.D
                        : static_cast<const T*>(a.k) + t * a.k_stride + own * a.D;
    float ss = 0.0f;
    for (int i = lane; i < a.D; i += 32) {
      const float x = to_float(src[i]);
      ss = fmaf(x, x, ss);
    }
    const float inv = (is_q ? a.q_scale : 1.0f) / sqrtf(warp_sum(ss) + a.unit_eps);
    float* dst = (is_q ? a.q_out : a.k_out) + (t * a.qk_heads + own) * a.D;
    for (int i = lane; i < a.D; i += 32) dst[i] = to_float(src[i]) * inv;
  }
  for (int h = threadIdx.x; h < a.heads; h += blockDim.x) {
    a.beta[t * a.heads + h] = 1.0f / (1.0f + expf(-a.b[t * a.ba_stride + h]));
    a.decay[t * a.heads + h] = expf(-expf(a.a_log[h]) * softplus_d(a.a[t * a.ba_stride + h] + a.dt_bias[h]));
  }
}

// ------------------------------------------------------------------------------------------------
constexpr int DS_THREADS = 128;
constexpr int DS_TOKENS = 16;       // tokens staged at a time

struct DeltaScanArgs {
  float* out;              // [T, heads * V]
  const float* q;          // [T, qk_heads * D]
  const float* k;
  const void* v;           // [T, v_stride], head h at column h * V, the model's type
  long long v_stride;
  const float* beta;       // [T, heads]
  const float* decay;
  float* state;            // slot s at state + s * slot_stride: [heads][V][D]
  long long slot_stride;
  const int* slots;
  const int* row_q_start;
  const int* row_q_len;
  int heads, heads_per_group, D, V, num_slots, write_state;
  int below;               // SHORT: only rows with fewer than this many tokens
  int* status;
};

// KPL: key channels a lane holds (a multiple of 4); L: lanes of a column (a power of two, L * KPL >= D);
// lane l holds the channels l * KPL .. l * KPL + KPL - 1.  Both are compile-time, so every address inside the
// token loop is a base plus a constant.  Tokens are staged 16 at a time into one of two buffers: while a
// portion's 16 tokens are worked on, the next 16 are on their way (q and k by 16-byte asynchronous copies
// where D is a multiple of 4, else by plain loads; v, beta and the decays through registers).  In shared
// memory a token's q (and k) is L runs of KPL + 4 floats (the 4 keep the lanes' 16-byte loads on separate
// banks); what lies beyond D is zero, so the token loop needs no bounds.  Inside the 16 tokens a lane holds
// the NEXT token's k and q in registers while the chain S -> S^T k -> u -> S of the present token runs, and
// sums its products in four separate sums, so the chain a token adds is the reduction over the L lanes, one
// multiply-add and the write, not the loads.  k . q is summed over the same lanes beside the two read-outs.
// CPT: value columns a thread holds (its group's column and the one `groups` further on): two columns are two
// chains whose waits overlap; a step of single tokens keeps one, so that its CTAs stay many.
// SHORT: only rows with fewer than `below` tokens (a form of its own, so that the other's loads do not wait for a row's length).
template <typename T, int KPL, int L, int CPT, bool ASYNC, bool SHORT>
__global__ void __launch_bounds__(DS_THREADS) delta_scan_kernel(const DeltaScanArgs a) {
  extern __shared__ __align__(16) float ds_smem[];
  constexpr int RUN = KPL + 4, DP = L * RUN;      // a lane's run and a token's row in shared memory
  constexpr int groups = DS_THREADS / L;          // groups of L lanes
  constexpr int cols = groups * CPT;              // value columns of this CTA: CPT a group (column group + c * groups)
  constexpr int stage_floats = 2 * DS_TOKENS * DP + DS_TOKENS * cols + 2 * DS_TOKENS;
  // one stage: q [DS_TOKENS][DP], k [DS_TOKENS][DP], v [DS_TOKENS][cols], beta [DS_TOKENS], decay [DS_TOKENS]
  const int D = a.D, V = a.V;

  const int row = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * cols;
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) {
    if (threadIdx.x == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
    return;
  }
  const int t0 = a.row_q_start[row], n = a.row_q_len[row];
  if (SHORT && n >= a.below) return;
  const int l = threadIdx.x % L, my_group = threadIdx.x / L;
  const int group = head / a.heads_per_group, qk_heads = a.heads / a.heads_per_group;
  // A thread's CPT columns are separate chains: one column's exchanges and writes run under the other's sums.
  bool live[CPT];
  float* mine[CPT];
  float S[CPT][KPL];
  const bool state_vectors = ASYNC && D % 4 == 0;
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    const int col = col0 + my_group + c * groups;
    live[c] = col < V;
    mine[c] = a.state + static_cast<long long>(slot) * a.slot_stride +
              (static_cast<long long>(head) * V + (live[c] ? col : 0)) * D + l * KPL;
    if (state_vectors) {
#pragma unroll
      for (int i = 0; i < KPL; i += 4) {
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (live[c] && l * KPL + i < D) x = *reinterpret_cast<const float4*>(mine[c] + i);
        S[c][i] = x.x; S[c][i + 1] = x.y; S[c][i + 2] = x.z; S[c][i + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < KPL; ++i) S[c][i] = (live[c] && l * KPL + i < D) ? mine[c][i] : 0.0f;
    }
  }
  for (int e = threadIdx.x; e < 2 * stage_floats; e += DS_THREADS) ds_smem[e] = 0.0f;
  __syncthreads();
  const T* v = static_cast<const T*>(a.v);
  const int chunks = (n + DS_TOKENS - 1) / DS_TOKENS;
  const int vec = D / 4;                         // 16-byte pieces of a row of q or k (ASYNC: D % 4 == 0)

  auto fetch_v = [&](int base, int nt, int e) -> float {
    const int j = e / cols, c = e - j * cols;
    return (j < nt && col0 + c < V)
               ? to_float(v[static_cast<long long>(t0 + base + j) * a.v_stride + head * V + col0 + c]) : 0.0f;
  };
  auto issue_qk = [&](int base, int nt, float* stage) {
    float* q_s = stage;
    float* k_s = stage + DS_TOKENS * DP;
    if (ASYNC) {
      for (int e = threadIdx.x; e < nt * vec; e += DS_THREADS) {
        const int j = e / vec, c = (e - j * vec) * 4;
        const long long at = (static_cast<long long>(t0 + base + j) * qk_heads + group) * D + c;
        const int to = j * DP + (c / KPL) * RUN + c % KPL;
        cp_async_16(q_s + to, a.q + at, true);
        cp_async_16(k_s + to, a.k + at, true);
      }
    } else {
      for (int e = threadIdx.x; e < nt * D; e += DS_THREADS) {
        const int j = e / D, d = e - j * D;
        const long long at = (static_cast<long long>(t0 + base + j) * qk_heads + group) * D + d;
        const int to = j * DP + (d / KPL) * RUN + d % KPL;
        q_s[to] = a.q[at];
        k_s[to] = a.k[at];
      }
    }
    cp_async_commit();
  };
  constexpr int V_PER = (DS_TOKENS * cols + DS_THREADS - 1) / DS_THREADS;
  float v_next[V_PER], beta_next = 0.0f, decay_next = 0.0f;
  auto fetch_rest = [&](int base, int nt) {
#pragma unroll
    for (int r = 0; r < V_PER; ++r) {
      const int e = threadIdx.x + r * DS_THREADS;
      v_next[r] = e < DS_TOKENS * cols ? fetch_v(base, nt, e) : 0.0f;
    }
    if (threadIdx.x < nt) {
      beta_next = a.beta[static_cast<long long>(t0 + base + threadIdx.x) * a.heads + head];
      decay_next = a.decay[static_cast<long long>(t0 + base + threadIdx.x) * a.heads + head];
    }
  };
  auto store_rest = [&](float* stage) {
    float* v_s = stage + 2 * DS_TOKENS * DP;
#pragma unroll
    for (int r = 0; r < V_PER; ++r) {
      const int e = threadIdx.x + r * DS_THREADS;
      if (e < DS_TOKENS * cols) v_s[e] = v_next[r];
    }
    if (threadIdx.x < DS_TOKENS) {
      v_s[DS_TOKENS * cols + threadIdx.x] = beta_next;
      v_s[DS_TOKENS * cols + DS_TOKENS + threadIdx.x] = decay_next;
    }
  };
  auto load_run = [&](float (&x)[KPL], const float* from) {
#pragma unroll
    for (int i = 0; i < KPL; i += 4) {
      const float4 r = *reinterpret_cast<const float4*>(from + i);
      x[i] = r.x; x[i + 1] = r.y; x[i + 2] = r.z; x[i + 3] = r.w;
    }
  };
  float* out = a.out + static_cast<long long>(t0) * a.heads * V + head * V + col0 + my_group;
  const long long out_stride = static_cast<long long>(a.heads) * V;
  // One token: the read-outs of the old state, the write, the output, for each of the thread's columns.
  auto token = [&](const float (&kr)[KPL], const float (&qr)[KPL], float g, float beta, const float* vj, long long at) {
    float kq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < KPL; ++i) kq[i & 3] = fmaf(kr[i], qr[i], kq[i & 3]);
    float skq = (kq[0] + kq[1]) + (kq[2] + kq[3]);
    float sk[CPT], sq[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      float rk[4] = {0.0f, 0.0f, 0.0f, 0.0f}, rq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int i = 0; i < KPL; ++i) {
        rk[i & 3] = fmaf(S[c][i], kr[i], rk[i & 3]);
        rq[i & 3] = fmaf(S[c][i], qr[i], rq[i & 3]);
      }
      sk[c] = (rk[0] + rk[1]) + (rk[2] + rk[3]);
      sq[c] = (rq[0] + rq[1]) + (rq[2] + rq[3]);
    }
#pragma unroll
    for (int o = L >> 1; o > 0; o >>= 1) {
      skq += __shfl_xor_sync(0xffffffffu, skq, o);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        sk[c] += __shfl_xor_sync(0xffffffffu, sk[c], o);
        sq[c] += __shfl_xor_sync(0xffffffffu, sq[c], o);
      }
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const float u = beta * (vj[c * groups] - g * sk[c]);
#pragma unroll
      for (int i = 0; i < KPL; ++i) S[c][i] = fmaf(kr[i], u, g * S[c][i]);
      if (l == 0 && live[c]) out[at * out_stride + c * groups] = fmaf(u, skq, g * sq[c]);
    }
  };

  if (chunks > 0) {
    issue_qk(0, min(DS_TOKENS, n), ds_smem);
    fetch_rest(0, min(DS_TOKENS, n));
    store_rest(ds_smem);
  }
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int base = chunk * DS_TOKENS, nt = min(DS_TOKENS, n - base);
    float* stage = ds_smem + (chunk & 1) * stage_floats;
    float* other = ds_smem + ((chunk + 1) & 1) * stage_floats;
    cp_async_wait<0>();
    __syncthreads();             // this portion has landed, and the other buffer is no longer read
    const bool more = chunk + 1 < chunks;
    if (more) {
      issue_qk(base + DS_TOKENS, min(DS_TOKENS, n - base - DS_TOKENS), other);
      fetch_rest(base + DS_TOKENS, min(DS_TOKENS, n - base - DS_TOKENS));
    }
    const float* q_s = stage + l * RUN;
    const float* k_s = stage + DS_TOKENS * DP + l * RUN;
    const float* v_s = stage + 2 * DS_TOKENS * DP + my_group;
    const float* beta_s = stage + 2 * DS_TOKENS * DP + DS_TOKENS * cols;
    const float* decay_s = beta_s + DS_TOKENS;
    // Tokens in pairs: while one token's chain runs on one set of registers, the next token's k and q are
    // fetched into the other set.
    float k0[KPL], q0[KPL], k1[KPL], q1[KPL];
    load_run(k0, k_s);
    load_run(q0, q_s);
    for (int j = 0; j < nt; j += 2) {
      const int j1 = j + 1 < DS_TOKENS ? j + 1 : j, j2 = j + 2 < DS_TOKENS ? j + 2 : j;
      load_run(k1, k_s + j1 * DP);
      load_run(q1, q_s + j1 * DP);
      token(k0, q0, decay_s[j], beta_s[j], v_s + j * cols, base + j);
      if (j + 1 >= nt) break;
      load_run(k0, k_s + j2 * DP);
      load_run(q0, q_s + j2 * DP);
      token(k1, q1, decay_s[j + 1], beta_s[j + 1], v_s + (j + 1) * cols, base + j + 1);
    }
    if (more) store_rest(other);
  }
  cp_async_wait<0>();
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    if (!a.write_state || !live[c]) continue;
    if (state_vectors) {
#pragma unroll
      for (int i = 0; i < KPL; i += 4)
        if (l * KPL + i < D)
          *reinterpret_cast<float4*>(mine[c] + i) = make_float4(S[c][i], S[c][i + 1], S[c][i + 2], S[c][i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < KPL; ++i)
        if (l * KPL + i < D) mine[c][i] = S[c][i];
    }
  }
}

// ------------------------------------------------------------------------------------------------ blocks of tokens
// Token by token the recurrence is a chain: the state's read-out with k, u, the write, 0.26 us a token whatever the SMs
// could do besides.  Over a block of B tokens, with S the state at its start, c_t the sum of the logarithms of the
// decays up to token t, R_k = S^T k_t and R_q = S^T q_t,
//
//   v'_t = v_t - e^(c_t) R_k(t)
//   u    = (I + A)^-1 diag(beta) v',   A_tj = beta_t e^(c_t - c_j) (k_t . k_j) for j < t
//   o_t  = e^(c_t) R_q(t) + sum_{j <= t} e^(c_t - c_j) (q_t . k_j) u_j
//   S   <- e^(c_B) S + sum_j e^(c_B - c_j) k_j u_j^T
//
// so the chain is one read-out and one write a block, both plain products.  All but the products with S and v' depends
// on the block alone: delta_blocks makes, for all blocks side by side, the unit vectors (a block's k and q with their
// tokens side by side, the layout that the products read) and per head
//
//   Tu = diag(e^(c_B - c_t)) (I + A)^-1 diag(beta)       (what the write takes is Tu v')
//   M  = P (I + A)^-1 diag(beta),  P_tj = e^(c_t - c_j) (q_t . k_j)   (o = e^(c) R_q + M v')
//
// and delta_block_scan walks a request's blocks.  Exponents are differences of sums within a block, never positive; the sums
// are formed in 64 bits and kept as two float32 values, so that a difference is good to a rounding of itself, also behind a
// token that forgets everything.
// Tokens behind a portion's end have beta 0 and decay 1.  Blocks are numbered row by row (first_piece_of_row).
constexpr int DB = 16;                     // tokens of a block
constexpr int DB_THREADS = 256;
constexpr int DB_COLS = 16;                // value columns of a CTA
constexpr int DB_COEF = 2 * DB * DB + 2 * DB;      // Tu and M, both [j][t], e^(c_t), e^(c_B) and padding

struct DeltaBlocksArgs {
  float* qk;               // [blocks][qk_heads][DP][2 DB]: k of the block's tokens, then q
  float* coef;             // [blocks][heads][DB_COEF]
  const void* q; long long q_stride;
  const void* k; long long k_stride;
  const float* b; const float* a; long long ba_stride;
  const float* a_log; const float* dt_bias;
  const int* row_q_start; const int* row_q_len;
  int rows, from, qk_heads, heads, D;      // rows of `from` tokens and more
  float q_scale, unit_eps;
};

// DP: the channels padded with zeros.
template <typename T, int DP>
__global__ void __launch_bounds__(DB_THREADS) delta_blocks_kernel(const DeltaBlocksArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  extern __shared__ __align__(16) float db_smem[];
  constexpr int ST = DP + 4;
  float* x_s = db_smem;                    // [2 DB][ST]: k, q
  float* kk_s = x_s + 2 * DB * ST;         // [DB][DB]
  float* qk_s = kk_s + DB * DB;
  float* a_s = qk_s + DB * DB;             // [DB][DB]: A
  float* p_s = a_s + DB * DB;              // [DB][DB]: P
  float* t_s = p_s + DB * DB;              // [DB][DB]: (I + A)^-1 diag(beta)
  float* c_hi = t_s + DB * DB;             // [DB]: the sums of logarithms c_t = c_hi + c_lo
  float* c_lo = c_hi + DB;
  float* lead_s = c_lo + DB;               // [DB]: e^(c_t)
  float* tail_s = lead_s + DB;             // [DB]: e^(c_B - c_t)
  float* beta_s = tail_s + DB;
  const int block = blockIdx.x, group = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int own;
  const int row = row_of_piece<DB>(a.row_q_len, a.rows, a.from, block, own);
  if (row < 0) return;
  const int begin = own * DB, n = min(DB, a.row_q_len[row] - begin);
  const long long t0 = a.row_q_start[row] + begin;
#pragma unroll
  for (int u = 0; u < 2 * DB / (DB_THREADS / 32); ++u) {
    const int i = warp + u * (DB_THREADS / 32);
    const bool is_q = i >= DB;
    const int t = i % DB;
    const T* src = is_q ? static_cast<const T*>(a.q) + (t0 + t) * a.q_stride + group * a.D
                        : static_cast<const T*>(a.k) + (t0 + t) * a.k_stride + group * a.D;
    float x[DP / 32], ss = 0.0f;
#pragma unroll
    for (int j = 0; j < DP / 32; ++j) {
      const int d = lane + 32 * j;
      x[j] = t < n && d < a.D ? to_float(src[d]) : 0.0f;
      ss = fmaf(x[j], x[j], ss);
    }
    const float inv = (is_q ? a.q_scale : 1.0f) / sqrtf(warp_sum(ss) + a.unit_eps);
#pragma unroll
    for (int j = 0; j < DP / 32; ++j) x_s[i * ST + lane + 32 * j] = t < n ? x[j] * inv : 0.0f;
  }
  __syncthreads();
  float4* to = reinterpret_cast<float4*>(a.qk + (static_cast<long long>(block) * a.qk_heads + group) * DP * 2 * DB);
  for (int e = tid; e < DP * 2 * DB / 4; e += DB_THREADS) {
    const int d = e / (2 * DB / 4), i = e % (2 * DB / 4) * 4;
    to[e] = make_float4(x_s[i * ST + d], x_s[(i + 1) * ST + d], x_s[(i + 2) * ST + d], x_s[(i + 3) * ST + d]);
  }
  {
    // k . k and q . k: a thread takes two tokens by two over a quarter of the channels (every fourth run of four).
    const int part = tid & 3, j0 = tid >> 2 & 7, i0 = tid >> 5;        // tokens i0, i0 + 8 against j0, j0 + 8
    float kk[2][2] = {}, qk[2][2] = {};
#pragma unroll
    for (int d = 4 * part; d < DP; d += 16) {
      float4 kj[2], ki[2], qi[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        kj[u] = *reinterpret_cast<const float4*>(x_s + (j0 + 8 * u) * ST + d);
        ki[u] = *reinterpret_cast<const float4*>(x_s + (i0 + 8 * u) * ST + d);
        qi[u] = *reinterpret_cast<const float4*>(x_s + (DB + i0 + 8 * u) * ST + d);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          kk[u][w] = fmaf(ki[u].x, kj[w].x, fmaf(ki[u].y, kj[w].y, fmaf(ki[u].z, kj[w].z, fmaf(ki[u].w, kj[w].w, kk[u][w]))));
          qk[u][w] = fmaf(qi[u].x, kj[w].x, fmaf(qi[u].y, kj[w].y, fmaf(qi[u].z, kj[w].z, fmaf(qi[u].w, kj[w].w, qk[u][w]))));
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          kk[u][w] += __shfl_xor_sync(0xffffffffu, kk[u][w], o);
          qk[u][w] += __shfl_xor_sync(0xffffffffu, qk[u][w], o);
        }
        if (part == 0) {
          kk_s[(i0 + 8 * u) * DB + j0 + 8 * w] = kk[u][w];
          qk_s[(i0 + 8 * u) * DB + j0 + 8 * w] = qk[u][w];
        }
      }
  }
  const int t = tid / DB, j = tid % DB;
  const int per = a.heads / a.qk_heads;
  for (int h = group * per; h < (group + 1) * per; ++h) {
    __syncthreads();                       // the products are there, and the head before is done
    if (tid < 32) {
      double c = 0.0;
      float beta = 0.0f;
      if (lane < n) {
        const long long at = (t0 + lane) * a.ba_stride + h;
        beta = 1.0f / (1.0f + expf(-a.b[at]));
        c = -static_cast<double>(expf(a.a_log[h])) * static_cast<double>(softplus_d(a.a[at] + a.dt_bias[h]));
        if (c < -1000.0) c = -1000.0;      // zero either way; the bound keeps the sums finite (a NaN passes)
      }
#pragma unroll
      for (int o = 1; o < DB; o <<= 1) {
        const double before = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += before;
      }
      const double all = __shfl_sync(0xffffffffu, c, DB - 1);
      if (lane < DB) {
        const float hi = static_cast<float>(c), lo = static_cast<float>(c - hi), lead = expf(hi);
        c_hi[lane] = hi;
        c_lo[lane] = lo;
        lead_s[lane] = fmaf(lead, lo, lead);
        tail_s[lane] = expf(static_cast<float>(all - c));
        beta_s[lane] = beta;
      }
    }
    __syncthreads();
    const float decay = j <= t ? expf((c_hi[t] - c_hi[j]) + (c_lo[t] - c_lo[j])) : 0.0f;
    a_s[tid] = j < t ? beta_s[t] * decay * kk_s[tid] : 0.0f;
    p_s[tid] = decay * qk_s[tid];
    __syncthreads();
    float* coef = a.coef + (static_cast<long long>(block) * a.heads + h) * DB_COEF;
    if (tid < DB) {
      // A column of the inverse by forward substitution, times beta of the column.
      float x[DB];
#pragma unroll
      for (int i = 0; i < DB; ++i) {
        float sum = i == tid ? 1.0f : 0.0f;
#pragma unroll
        for (int m = 0; m < i; ++m) sum = fmaf(-a_s[i * DB + m], x[m], sum);
        x[i] = sum;
      }
#pragma unroll
      for (int i = 0; i < DB; ++i) t_s[i * DB + tid] = x[i] * beta_s[tid];
    }
    __syncthreads();
    // (threads run over the rows of the transposed matrices: t fastest)
    const int tt = tid % DB, jj = tid / DB;
    coef[jj * DB + tt] = tail_s[tt] * t_s[tt * DB + jj];
    float m = 0.0f;
    for (int i = jj; i <= tt; ++i) m = fmaf(p_s[tt * DB + i], t_s[i * DB + jj], m);
    coef[(DB + jj) * DB + tt] = m;
    if (tid < DB) coef[2 * DB * DB + tid] = lead_s[tid];
    if (tid == 0) coef[2 * DB * DB + DB] = lead_s[DB - 1];
  }
}

struct DeltaBlockScanArgs {
  float* out;              // [T, heads * V]
  const float* qk;
  const float* coef;
  const void* v; long long v_stride;
  float* state; long long slot_stride;     // slot s at state + s * slot_stride: [heads][V][D]
  const int* slots; const int* row_q_start; const int* row_q_len;
  int from, heads, qk_heads, D, V, num_slots, write_state;
  int* status;
};

// A CTA owns a request, a head and DB_COLS value columns; its state lies in registers (two channels by four columns a
// thread) and, for the read-outs, in shared memory.  A block: every warp forms the read-outs of all 32 rows (k and q)
// over its share of the channels, 4 x 4 a thread; the warps' sums are added and v' made; u and o from the block's
// matrices; the state.  The next block's operands are copied meanwhile.  Bound by the reads of shared memory beside the
// multiply-adds and by the chain of a block, four barriers with eight warps between them (2048 tokens, 16 heads of 128 x 128: 240 us
// with the matrices, 522 token by token).  Products on the tensor cores with operands of two TF32 values each took 30 us less,
// at 1.5 to 1.9 times the token-by-token form's error against 64 bits; this form has 0.5 to 0.9 of it.
template <typename T, int DP>
__global__ void __launch_bounds__(DB_THREADS, 2) delta_block_scan_kernel(const DeltaBlockScanArgs a) {
  extern __shared__ __align__(16) float db_smem[];
  constexpr int QK_ST = 2 * DB + 4, S_ST = DB_COLS + 4, RED_ST = 2 * DB + 4;
  constexpr int stage_floats = DP * QK_ST + DB_COEF;
  float* stages = db_smem;                                   // two of [DP][QK_ST] and the coefficients
  float* s_s = stages + 2 * stage_floats;                    // [DP][S_ST]
  float* red_s = s_s + DP * S_ST;                            // [warps][DB_COLS][RED_ST]
  float* vp_s = red_s + DB_THREADS / 32 * DB_COLS * RED_ST;  // [DB_COLS][DB]: v'
  float* u_s = vp_s + DB_COLS * DB;                          // [DB][S_ST]: what the write takes
  float* o_s = u_s + DB * S_ST;                              // [DB][S_ST]
  __shared__ int wild;                                       // the last block with a v' that is not finite
  const int row = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * DB_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) wild = -1;
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) {
    if (tid == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
    return;
  }
  const int n = a.row_q_len[row], blocks = (n + DB - 1) / DB;
  if (n < a.from) return;
  const long long t0 = a.row_q_start[row];
  const int first = first_piece_of_row<DB>(a.row_q_len, row, a.from);
  const int group = head / (a.heads / a.qk_heads);

  auto copy_block = [&](int p, float* stage) {
    const float* qk = a.qk + (static_cast<long long>(first + p) * a.qk_heads + group) * DP * 2 * DB;
    for (int e = tid; e < DP * 2 * DB / 4; e += DB_THREADS) {
      const int d = e / (2 * DB / 4), i = e % (2 * DB / 4) * 4;
      cp_async_16(stage + d * QK_ST + i, qk + e * 4, true);
    }
    const float* coef = a.coef + (static_cast<long long>(first + p) * a.heads + head) * DB_COEF;
    for (int e = tid; e < DB_COEF / 4; e += DB_THREADS) cp_async_16(stage + DP * QK_ST + e * 4, coef + e * 4, true);
    cp_async_commit();
  };
  // This thread's token and column in the small products.
  const int my_t = tid % DB, my_c = tid / DB;
  const T* v = static_cast<const T*>(a.v) + t0 * a.v_stride + head * a.V + col0 + my_c;
  auto fetch_v = [&](int p) {
    const int t = p * DB + my_t;
    return t < n && col0 + my_c < a.V ? to_float(v[t * a.v_stride]) : 0.0f;
  };
  // This thread's part of the state: channels d0 and d0 + 1, columns c0 .. c0 + 3.
  const int d0 = tid / 4 * 2, c0 = tid % 4 * 4;
  const bool holds = d0 < DP;
  float S[2][4];
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride + (static_cast<long long>(head) * a.V + col0) * a.D;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      S[i][c] = holds && d0 + i < a.D && col0 + c0 + c < a.V ? state[static_cast<long long>(c0 + c) * a.D + d0 + i] : 0.0f;
  auto store_state = [&]() {
    if (holds) {
#pragma unroll
      for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(s_s + (d0 + i) * S_ST + c0) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    }
  };
  store_state();
  float v_now = 0.0f;
  if (blocks > 0) {
    copy_block(0, stages);
    v_now = fetch_v(0);
  }
  for (int p = 0; p < blocks; ++p) {
    const float* stage = stages + (p & 1) * stage_floats;
    const float* coef = stage + DP * QK_ST;
    cp_async_wait<0>();
    __syncthreads();             // the block and the state are there; the other buffer is no longer read
    float v_next = 0.0f;
    if (p + 1 < blocks) {
      copy_block(p + 1, stages + ((p + 1) & 1) * stage_floats);
      v_next = fetch_v(p + 1);
    }
    {
      const int i0 = (lane & 7) * 4, rc = (lane >> 3) * 4;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
#pragma unroll
      for (int u = 0; u < DP / 8; ++u) {
        const int d = warp * (DP / 8) + u;
        float x[4], y[4];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(stage + d * QK_ST + i0);
        *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(s_s + d * S_ST + rc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[c][i] = fmaf(x[i], y[c], acc[c][i]);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
        *reinterpret_cast<float4*>(red_s + (warp * DB_COLS + rc + c) * RED_ST + i0) = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
    }
    __syncthreads();
    float rk = 0.0f, rq = 0.0f;
#pragma unroll
    for (int w = 0; w < DB_THREADS / 32; ++w) {
      rk += red_s[(w * DB_COLS + my_c) * RED_ST + my_t];
      rq += red_s[(w * DB_COLS + my_c) * RED_ST + DB + my_t];
    }
    const float lead = coef[2 * DB * DB + my_t], whole = coef[2 * DB * DB + DB];
    const float vp = v_now - lead * rk;
    vp_s[my_c * DB + my_t] = vp;
    if (!isfinite(vp)) wild = p;
    __syncthreads();
    {
      float u = 0.0f, o = 0.0f;
      if (wild != p) {
#pragma unroll
        for (int j = 0; j < DB; j += 4) {
          float x[4];
          *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(vp_s + my_c * DB + j);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            u = fmaf(coef[(j + i) * DB + my_t], x[i], u);
            o = fmaf(coef[DB * DB + (j + i) * DB + my_t], x[i], o);
          }
        }
      } else {
        // The same sums, without a zero times a later token's value.
        for (int j = 0; j <= my_t; ++j) {
          u = fmaf(coef[j * DB + my_t], vp_s[my_c * DB + j], u);
          o = fmaf(coef[(DB + j) * DB + my_t], vp_s[my_c * DB + j], o);
        }
      }
      u_s[my_t * S_ST + my_c] = u;
      o_s[my_t * S_ST + my_c] = fmaf(lead, rq, o);
    }
    __syncthreads();
    {
      const int t = p * DB + tid / DB_COLS, c = tid % DB_COLS;
      if (t < n && col0 + c < a.V)
        a.out[(t0 + t) * a.heads * a.V + static_cast<long long>(head) * a.V + col0 + c] = o_s[tid / DB_COLS * S_ST + c];
    }
    if (holds) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) S[i][c] *= whole;
#pragma unroll
      for (int j = 0; j < DB; j += 4) {
        float k0[4], k1[4];
        *reinterpret_cast<float4*>(k0) = *reinterpret_cast<const float4*>(stage + d0 * QK_ST + j);
        *reinterpret_cast<float4*>(k1) = *reinterpret_cast<const float4*>(stage + (d0 + 1) * QK_ST + j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float u[4];
          *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(u_s + (j + i) * S_ST + c0);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            S[0][c] = fmaf(k0[i], u[c], S[0][c]);
            S[1][c] = fmaf(k1[i], u[c], S[1][c]);
          }
        }
      }
    }
    store_state();               // (nobody reads the state's tile between the barriers above and the next one)
    v_now = v_next;
  }
  if (!a.write_state || !holds) return;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (d0 + i < a.D && col0 + c0 + c < a.V) state[static_cast<long long>(c0 + c) * a.D + d0 + i] = S[i][c];
}

template <int DP>
constexpr size_t delta_blocks_smem() { return sizeof(float) * (2 * DB * (DP + 4) + 5 * DB * DB + 5 * DB); }
template <int DP>
constexpr size_t delta_block_scan_smem() {
  return sizeof(float) * (2 * (DP * (2 * DB + 4) + DB_COEF) + DP * (DB_COLS + 4) + DB_THREADS / 32 * DB_COLS * (2 * DB + 4) +
                          DB_COLS * DB + 2 * DB * (DB_COLS + 4));
}

}  // namespace zb

using namespace zb;

ZB_API int zb_delta_max_channels() { return 512; }

// `below` > 0: only the tokens of rows with fewer than `below` tokens (here and in zb_delta_scan; zb_delta_block_scan takes the
// others).
ZB_API int zb_delta_gates(float* q_out, float* k_out, float* beta, float* decay, const void* q, long long q_stride,
                          const void* k, long long k_stride, const float* b, const float* a, long long ba_stride,
                          const float* a_log, const float* dt_bias, int tokens, int qk_heads, int heads, int D,
                          float q_scale, float unit_eps, const int* row_q_start, const int* row_q_len, int rows, int below, int dtype,
                          void* stream) {
  if (rows < 0 || tokens < 0 || qk_heads <= 0 || heads <= 0 || D <= 0) return ERR_BAD_ARGUMENT;
  if (tokens == 0) return OK;
  DeltaGatesArgs g;
  g.q_out = q_out; g.k_out = k_out; g.beta = beta; g.decay = decay; g.q = q; g.k = k; g.q_stride = q_stride;
  g.k_stride = k_stride; g.b = b; g.a = a; g.ba_stride = ba_stride; g.a_log = a_log; g.dt_bias = dt_bias;
  g.qk_heads = qk_heads; g.heads = heads; g.D = D; g.q_scale = q_scale; g.unit_eps = unit_eps;
  g.row_q_start = row_q_start; g.row_q_len = row_q_len; g.rows = rows; g.below = below;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == DTYPE_F32) launch_dependent(delta_gates_kernel<float>, dim3(tokens), dim3(128), 0, s, false, g);
  else launch_dependent(delta_gates_kernel<__nv_bfloat16>, dim3(tokens), dim3(128), 0, s, false, g);
  return launch_result();
}

template <typename T, int KPL, int L, int CPT, bool SHORT>
static int delta_scan_launch(const DeltaScanArgs& a, int rows, cudaStream_t s) {
  constexpr int cols = DS_THREADS / L * CPT;
  const size_t smem = 2 * sizeof(float) * (2 * DS_TOKENS * L * (KPL + 4) + DS_TOKENS * cols + 2 * DS_TOKENS);
  const bool async = a.D % 4 == 0 && reinterpret_cast<uintptr_t>(a.q) % 16 == 0 && reinterpret_cast<uintptr_t>(a.k) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(a.state) % 16 == 0 && a.slot_stride % 4 == 0;
  auto kernel = async ? delta_scan_kernel<T, KPL, L, CPT, true, SHORT> : delta_scan_kernel<T, KPL, L, CPT, false, SHORT>;
  if (smem > 48 * 1024 &&
      cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem))))
    return ERR_CUDA;
  kernel<<<dim3(rows, a.heads, (a.V + cols - 1) / cols), DS_THREADS, smem, s>>>(a);
  return launch_result();
}

template <typename T, int KPL, int L>
static int delta_scan_columns(const DeltaScanArgs& a, int rows, int tokens, cudaStream_t s) {
  // Two columns a thread where requests bring runs of tokens (the chains hide each other's waits) and a head has
  // columns enough; one where a step is single tokens, whose time is the state's bytes.
  const bool runs = tokens >= 4 * rows && a.V >= 2 * (DS_THREADS / L);
  if (a.below > 0) return delta_scan_launch<T, KPL, L, 1, true>(a, rows, s);
  return runs ? delta_scan_launch<T, KPL, L, 2, false>(a, rows, s) : delta_scan_launch<T, KPL, L, 1, false>(a, rows, s);
}

template <typename T>
static int delta_scan_dispatch(const DeltaScanArgs& a, int rows, int tokens, cudaStream_t s) {
  // Channels a lane holds and lanes a column: a column spreads over 4 lanes up to 64 channels (two rounds of
  // exchanges a token), over 8 up to 128, 16 up to 256, a whole warp beyond.
  const int D = a.D;
  if (D <= 16) return delta_scan_columns<T, 4, 4>(a, rows, tokens, s);
  if (D <= 32) return delta_scan_columns<T, 8, 4>(a, rows, tokens, s);
  if (D <= 64) return delta_scan_columns<T, 16, 4>(a, rows, tokens, s);
  if (D <= 128) return delta_scan_columns<T, 16, 8>(a, rows, tokens, s);
  if (D <= 256) return delta_scan_columns<T, 16, 16>(a, rows, tokens, s);
  return delta_scan_columns<T, 16, 32>(a, rows, tokens, s);
}

ZB_API int zb_delta_scan(float* out, const float* q, const float* k, const void* v, long long v_stride,
                         const float* beta, const float* decay, float* state, long long slot_stride, const int* slots,
                         const int* row_q_start, const int* row_q_len, int rows, int tokens, int heads,
                         int heads_per_group, int D, int V, int num_slots, int write_state, int below, int dtype, int* status,
                         void* stream) {
  if (rows < 0 || heads <= 0 || heads_per_group <= 0 || heads % heads_per_group != 0 || D <= 0 || V <= 0)
    return ERR_BAD_ARGUMENT;
  if (D > zb_delta_max_channels()) return ERR_UNSUPPORTED;
  if (rows == 0) return OK;
  DeltaScanArgs a;
  a.out = out; a.q = q; a.k = k; a.v = v; a.v_stride = v_stride; a.beta = beta; a.decay = decay; a.state = state;
  a.slot_stride = slot_stride; a.slots = slots; a.row_q_start = row_q_start; a.row_q_len = row_q_len;
  a.heads = heads; a.heads_per_group = heads_per_group; a.D = D; a.V = V; a.num_slots = num_slots;
  a.write_state = write_state; a.below = below; a.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  return dtype == DTYPE_F32 ? delta_scan_dispatch<float>(a, rows, tokens, s)
                            : delta_scan_dispatch<__nv_bfloat16>(a, rows, tokens, s);
}

// The blocks' form takes up to this many key channels per head.
ZB_API int zb_delta_block_max_channels() { return 128; }
ZB_API int zb_delta_block_tokens() { return DB; }
// Floats of workspace a block needs: its unit vectors and its matrices.
ZB_API int zb_delta_block_floats(int qk_heads, int heads, int D) { return qk_heads * (D <= 64 ? 64 : 128) * 2 * DB + heads * DB_COEF; }

template <typename T, int DP>
static int delta_block_launch(const DeltaBlocksArgs& b, const DeltaBlockScanArgs& a, int rows, int blocks, cudaStream_t s) {
  constexpr int first = static_cast<int>(delta_blocks_smem<DP>()), second = static_cast<int>(delta_block_scan_smem<DP>());
  if (cuda_failed(cudaFuncSetAttribute(delta_block_scan_kernel<T, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, second)))
    return ERR_CUDA;
  launch_dependent(delta_blocks_kernel<T, DP>, dim3(blocks, b.qk_heads), dim3(DB_THREADS), first, s, false, b);
  // (Not as a dependent: its CTAs would take the SMs that the kernel before it leaves first, two a SM, while others stay empty:
  // the layer over 2048 tokens, 16 heads 347 -> 500 us.)
  delta_block_scan_kernel<T, DP><<<dim3(rows, a.heads, (a.V + DB_COLS - 1) / DB_COLS), DB_THREADS, second, s>>>(a);
  return launch_result();
}

// The rule over rows of `from` tokens and more, block by block.  `ws`: (tokens / block tokens + rows) * zb_delta_block_floats floats,
// 16-byte aligned, contents irrelevant.  The rows' tokens may lie in the stream in any order.
ZB_API int zb_delta_block_scan(float* out, const void* q, long long q_stride, const void* k, long long k_stride, const void* v,
                               long long v_stride, const float* b, const float* a, long long ba_stride, const float* a_log,
                               const float* dt_bias, float* state, long long slot_stride, const int* slots, const int* row_q_start,
                               const int* row_q_len, int rows, int tokens, int from, int qk_heads, int heads, int D, int V,
                               int num_slots, int write_state, float q_scale, float unit_eps, float* ws, int dtype, int* status, void* stream) {
  if (rows < 0 || tokens < 0 || qk_heads <= 0 || heads <= 0 || heads % qk_heads != 0 || D <= 0 || V <= 0 || num_slots <= 0)
    return ERR_BAD_ARGUMENT;
  if (D > zb_delta_block_max_channels() || heads > 65535 || (V + DB_COLS - 1) / DB_COLS > 65535) return ERR_UNSUPPORTED;
  if (rows == 0 || tokens == 0) return OK;
  if (ws == nullptr || reinterpret_cast<uintptr_t>(ws) % 16 != 0) return ERR_BAD_ARGUMENT;
  const int blocks = tokens / DB + rows, dp = D <= 64 ? 64 : 128;
  DeltaBlocksArgs g;
  g.qk = ws; g.coef = ws + static_cast<long long>(blocks) * qk_heads * dp * 2 * DB; g.q = q; g.q_stride = q_stride; g.k = k;
  g.k_stride = k_stride; g.b = b; g.a = a; g.ba_stride = ba_stride; g.a_log = a_log; g.dt_bias = dt_bias;
  g.row_q_start = row_q_start; g.row_q_len = row_q_len; g.rows = rows; g.from = from; g.qk_heads = qk_heads; g.heads = heads; g.D = D;
  g.q_scale = q_scale; g.unit_eps = unit_eps;
  DeltaBlockScanArgs c;
  c.out = out; c.qk = g.qk; c.coef = g.coef; c.v = v; c.v_stride = v_stride; c.state = state; c.slot_stride = slot_stride;
  c.slots = slots; c.row_q_start = row_q_start; c.row_q_len = row_q_len; c.heads = heads; c.qk_heads = qk_heads; c.D = D; c.V = V;
  c.num_slots = num_slots; c.write_state = write_state; c.from = from; c.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == DTYPE_F32) return dp == 64 ? delta_block_launch<float, 64>(g, c, rows, blocks, s) : delta_block_launch<float, 128>(g, c, rows, blocks, s);
  return dp == 64 ? delta_block_launch<__nv_bfloat16, 64>(g, c, rows, blocks, s) : delta_block_launch<__nv_bfloat16, 128>(g, c, rows, blocks, s);
}
