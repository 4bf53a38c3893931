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
// block of 32 tokens.
//
// Token by token everything is float32 multiply-adds; in blocks products are formed on the tensor cores from three bfloat16 parts a value, all
// 24 bits of it, with float32 sums.  The values v are read in the model's type.
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
constexpr int DB = 32;                     // tokens of a block
constexpr int DB_THREADS = 256;
constexpr int DB_COLS = 16;                // value columns of a CTA
constexpr int DB_HEADS = 2;                // heads whose matrices a CTA of delta_blocks makes side by side
constexpr int DB_MST = DB + 8;             // a row of Tu or M in bfloat16
constexpr int DB_FST = DB + 1;             // a row of a float32 matrix
constexpr int DB_COEF_PARTS = 3 * 2 * DB * DB_MST * 2;
constexpr int DB_COEF_BYTES = DB_COEF_PARTS + (DB + 4) * 4;       // Tu over M, [part][t][j], then e^(c_t), e^(c_B) and padding
constexpr float DB_LARGEST = 3.3e38f;      // beyond it a value rounds to infinity in bfloat16
constexpr int DB_WAIT_LIMIT = 1 << 20;

// DP: the channels padded with zeros.
template <int DP>
struct DeltaShape {
  static constexpr int ST = DP + 8;                               // a row of k or q in bfloat16
  static constexpr int QK_BYTES = 3 * 2 * DB * ST * 2;            // [part][k of the block's tokens, then q][ST]
  static constexpr int STAGE_BYTES = QK_BYTES + DB_COEF_BYTES;
  static constexpr int CST = DB_COLS + 8, FST = DB_COLS + 4;      // rows of value columns: bfloat16, float32
  static constexpr int S_BYTES = 3 * DP * CST * 2, V_BYTES = 3 * DB * CST * 2, F_BYTES = DB * FST * 4, RED_BYTES = DP / 16 * 2 * DB * DB_COLS * 4;
  static constexpr int BLOCKS_SMEM = QK_BYTES + (2 + 3 * DB_HEADS) * DB * DB_FST * 4 + DB_HEADS * 5 * DB * 4;
  static constexpr int SCAN_SMEM = 2 * STAGE_BYTES + S_BYTES + 2 * V_BYTES + 2 * F_BYTES + RED_BYTES;
  static_assert(QK_BYTES % 16 == 0 && DB_COEF_BYTES % 16 == 0, "bulk copies move 16-byte pieces");
  static_assert(SCAN_SMEM <= 226 * 1024, "fits an SM's shared memory");
};

struct DeltaBlocksArgs {
  unsigned char* qk;       // [blocks][qk_heads][QK_BYTES]
  unsigned char* coef;     // [blocks][heads][DB_COEF_BYTES]
  const void* q; long long q_stride;
  const void* k; long long k_stride;
  const float* b; const float* a; long long ba_stride;
  const float* a_log; const float* dt_bias;
  const int* row_q_start; const int* row_q_len;
  int rows, from, qk_heads, heads, D;      // rows of `from` tokens and more
  float q_scale, unit_eps;
};

// M products of 16 rows by NT tiles of 8 columns, operands in three parts: low += the products of parts behind hi hi, smallest first; high +=
// hi hi.  (The tensor cores cut a sum's last bits at every step: what is cut off the small products' sum is 2^-8 of that.)  The
// tiles take turns, so that no product waits for the one before it.
template <int M, int NT>
__device__ __forceinline__ void delta_products(float (&high)[M][NT][4], float (&low)[M][NT][4], const unsigned (&a)[M][3][4],
                                               const unsigned (&b)[M][3][2 * NT]) {
  constexpr int FIRST[6] = {2, 1, 0, 1, 0, 0}, SECOND[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
  for (int e = 0; e < 6; ++e)
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
        mma_bf16_16816(e < 5 ? low[m][n] : high[m][n], a[m][FIRST[e]], b[m][SECOND[e]][2 * n], b[m][SECOND[e]][2 * n + 1]);
}

template <typename T, int DP>
__global__ void __launch_bounds__(DB_THREADS) delta_blocks_kernel(const DeltaBlocksArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  using Shape = DeltaShape<DP>;
  constexpr int ST = Shape::ST, MATRIX = DB * DB_FST;
  extern __shared__ __align__(16) unsigned char db_smem[];
  __nv_bfloat16* x_s = reinterpret_cast<__nv_bfloat16*>(db_smem);              // [part][k, q][ST]
  float* kk_s = reinterpret_cast<float*>(db_smem + Shape::QK_BYTES);           // [DB][DB_FST] each
  float* qk_s = kk_s + MATRIX;
  float* a_s = qk_s + MATRIX;              // [head]: A
  float* p_s = a_s + DB_HEADS * MATRIX;    // [head]: P
  float* t_s = p_s + DB_HEADS * MATRIX;    // [head]: (I + A)^-1
  float* c_hi = t_s + DB_HEADS * MATRIX;   // [head][DB]: the sums of logarithms c_t = c_hi + c_lo
  float* c_lo = c_hi + DB_HEADS * DB;
  float* lead_s = c_lo + DB_HEADS * DB;    // [head][DB]: e^(c_t)
  float* tail_s = lead_s + DB_HEADS * DB;  // [head][DB]: e^(c_B - c_t)
  float* beta_s = tail_s + DB_HEADS * DB;
  const int block = blockIdx.x, group = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int own;
  const int row = row_of_piece<DB>(a.row_q_len, a.rows, a.from, block, own);
  if (row < 0) return;
  const int begin = own * DB, n = min(DB, a.row_q_len[row] - begin);
  const long long t0 = a.row_q_start[row] + begin;
#pragma unroll
  for (int u = 0; u < 2 * DB / (DB_THREADS / 32); ++u) {
    const int i = warp + u * (DB_THREADS / 32), t = i % DB;
    const bool is_q = i >= DB;
    const T* src = is_q ? static_cast<const T*>(a.q) + (t0 + t) * a.q_stride + group * a.D
                        : static_cast<const T*>(a.k) + (t0 + t) * a.k_stride + group * a.D;
    float x[DP / 64][2], ss = 0.0f;
#pragma unroll
    for (int j = 0; j < DP / 64; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int d = 64 * j + 2 * lane + e;
        x[j][e] = t < n && d < a.D ? to_float(src[d]) : 0.0f;
        ss = fmaf(x[j][e], x[j][e], ss);
      }
    const float inv = t < n ? (is_q ? a.q_scale : 1.0f) / sqrtf(warp_sum(ss) + a.unit_eps) : 0.0f;
#pragma unroll
    for (int j = 0; j < DP / 64; ++j) {
      unsigned part[3];
      three_parts(x[j][0] * inv, x[j][1] * inv, part[0], part[1], part[2]);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<unsigned*>(x_s + (e * 2 * DB + i) * ST + 64 * j + 2 * lane) = part[e];
    }
  }
  __syncthreads();
  uint4* to = reinterpret_cast<uint4*>(a.qk + (static_cast<long long>(block) * a.qk_heads + group) * Shape::QK_BYTES);
  for (int e = tid; e < Shape::QK_BYTES / 16; e += DB_THREADS) to[e] = reinterpret_cast<const uint4*>(x_s)[e];
  {
    // k . k and q . k: a warp takes 16 rows of k or q against 16 of k; what lies above the diagonal tiles is not read.
    const int row0 = warp / 2 * 16, col0 = warp % 2 * 16, g = lane >> 2, t = lane & 3;
    if (row0 % DB >= col0) {
      const __nv_bfloat16* rows = x_s + (row0 + (lane & 7) + ((lane >> 3) & 1) * 8) * ST + (lane >> 4) * 8;
      const __nv_bfloat16* columns = x_s + (col0 + (lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8;
      float high[2][2][4] = {}, low[2][2][4] = {};
#pragma unroll
      for (int ks = 0; ks < DP / 16; ks += 2) {
        unsigned af[2][3][4], bf[2][3][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            ldmatrix_x4(af[u][e], rows + e * 2 * DB * ST + (ks + u) * 16);
            ldmatrix_x4(bf[u][e], columns + e * 2 * DB * ST + (ks + u) * 16);
          }
        delta_products<2, 2>(high, low, af, bf);
      }
      float* out = row0 < DB ? kk_s : qk_s;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          out[(row0 % DB + g + (e >> 1) * 8) * DB_FST + col0 + 8 * i + 2 * t + (e & 1)] = (high[0][i][e] + high[1][i][e]) + (low[0][i][e] + low[1][i][e]);
    }
  }
  const int per = a.heads / a.qk_heads;
  for (int h0 = group * per; h0 < (group + 1) * per; h0 += DB_HEADS) {
    const int count = min(DB_HEADS, (group + 1) * per - h0);
    __syncthreads();                       // the products are there, and the heads before are done
    if (warp < count) {
      const int h = h0 + warp;
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
      const float hi = static_cast<float>(c), lo = static_cast<float>(c - hi), lead = expf(hi);
      const int at = warp * DB + lane;
      c_hi[at] = hi;
      c_lo[at] = lo;
      lead_s[at] = fmaf(lead, lo, lead);
      tail_s[at] = expf(static_cast<float>(all - c));
      beta_s[at] = beta;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < DB_HEADS * DB * DB / DB_THREADS; ++u) {
      const int e = tid + u * DB_THREADS, w = e / (DB * DB), t = e / DB % DB, j = e % DB;
      if (w >= count) break;
      const float* hi = c_hi + w * DB, * lo = c_lo + w * DB;
      const float decay = j <= t ? expf((hi[t] - hi[j]) + (lo[t] - lo[j])) : 0.0f;
      a_s[w * MATRIX + t * DB_FST + j] = j < t ? beta_s[w * DB + t] * decay * kk_s[t * DB_FST + j] : 0.0f;
      p_s[w * MATRIX + t * DB_FST + j] = j <= t ? decay * qk_s[t * DB_FST + j] : 0.0f;
    }
    __syncthreads();
    // (I + A)^-1 = [T1 0; -T2 A21 T1, T2]: a column of T1 or T2 a lane, by forward substitution.
    if (warp < count) {
      const int half = lane / 16, column = lane % 16;
      const float* from = a_s + warp * MATRIX + 16 * half * (DB_FST + 1);
      float* result = t_s + warp * MATRIX + 16 * half * (DB_FST + 1);
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float sum = i == column ? 1.0f : 0.0f;
#pragma unroll
        for (int m = 0; m < i; ++m) sum = fmaf(-from[i * DB_FST + m], x[m], sum);
        x[i] = sum;
        result[i * DB_FST + column] = sum;
      }
    }
    __syncthreads();
    // A21 T1, into the quarter of A that is zero.
    const int ti = tid / 16, tj = tid % 16;
#pragma unroll
    for (int w = 0; w < DB_HEADS; ++w) {
      if (w >= count) break;
      const float* from = a_s + w * MATRIX + (16 + ti) * DB_FST, * t1 = t_s + w * MATRIX + tj;
      float sum = 0.0f;
#pragma unroll
      for (int m = 0; m < 16; ++m) sum = fmaf(from[m], t1[m * DB_FST], sum);
      a_s[w * MATRIX + ti * DB_FST + 16 + tj] = sum;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < DB_HEADS; ++w) {
      if (w >= count) break;
      const float* t2 = t_s + w * MATRIX + (16 + ti) * DB_FST + 16, * from = a_s + w * MATRIX + 16 + tj;
      float sum = 0.0f;
#pragma unroll
      for (int m = 0; m < 16; ++m) sum = fmaf(-t2[m], m <= ti ? from[m * DB_FST] : 0.0f, sum);      // (a later token's row may hold anything)
      t_s[w * MATRIX + (16 + ti) * DB_FST + tj] = sum;
      t_s[w * MATRIX + ti * DB_FST + 16 + tj] = 0.0f;
    }
    __syncthreads();
    // A thread makes columns j and j + 1 of rows t, t + 8, t + 16 and t + 24 of a head's matrices.
    static_assert(DB_HEADS * DB * DB / 8 == DB_THREADS, "eight values a thread");
    const int w = tid / (DB_THREADS / DB_HEADS), t = tid / 16 % 8, j = tid % 16 * 2;
    if (w < count) {
      unsigned char* coef = a.coef + (static_cast<long long>(block) * a.heads + h0 + w) * DB_COEF_BYTES;
      const float* inverse = t_s + w * MATRIX + j, * p = p_s + w * MATRIX + t * DB_FST;
      float m[4][2] = {};
#pragma unroll
      for (int i0 = 0; i0 < DB; i0 += 8)
#pragma unroll
        for (int i = i0; i < i0 + 8; ++i) {
          const float x = inverse[i * DB_FST], y = inverse[i * DB_FST + 1];
#pragma unroll
          for (int r = i0 / 8; r < 4; ++r) {
            const bool seen = 8 * r > i || i - 8 * r <= t;                // (a later token's row may hold anything)
            const float weight = p[8 * r * DB_FST + i];
            m[r][0] = fmaf(weight, seen ? x : 0.0f, m[r][0]);
            m[r][1] = fmaf(weight, seen ? y : 0.0f, m[r][1]);
          }
        }
      const float beta0 = beta_s[w * DB + j], beta1 = beta_s[w * DB + j + 1];
      float* steps = reinterpret_cast<float*>(coef + DB_COEF_PARTS);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row_t = t + 8 * r;
        const float tail = tail_s[w * DB + row_t];
        unsigned up[3], mp[3];
        three_parts(tail * (inverse[row_t * DB_FST] * beta0), tail * (inverse[row_t * DB_FST + 1] * beta1), up[0], up[1], up[2]);
        three_parts(m[r][0] * beta0, m[r][1] * beta1, mp[0], mp[1], mp[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          *reinterpret_cast<unsigned*>(coef + ((i * 2 * DB + row_t) * DB_MST + j) * 2) = up[i];
          *reinterpret_cast<unsigned*>(coef + ((i * 2 * DB + DB + row_t) * DB_MST + j) * 2) = mp[i];
        }
        if (j == 0) steps[row_t] = lead_s[w * DB + row_t];
      }
      if (t == 0 && j == 0) steps[DB] = lead_s[w * DB + DB - 1];
    }
  }
}

struct DeltaBlockScanArgs {
  float* out;              // [T, heads * V]
  const unsigned char* qk;
  const unsigned char* coef;
  const void* v; long long v_stride;
  float* state; long long slot_stride;     // slot s at state + s * slot_stride: [heads][V][D]
  const int* slots; const int* row_q_start; const int* row_q_len;
  int from, heads, qk_heads, D, V, num_slots, write_state;
  int* status;
};

// What the values v' that are not finite (or that bfloat16 parts do not hold), left out of the product, add to row `row` of Tu over M, token t.
// (A call of its own, so that its registers cost the other blocks nothing.)
__device__ __noinline__ float delta_wild(const __nv_bfloat16* coef, int row, int t, const float* values, int stride) {
  float sum = 0.0f;
  for (int j = 0; j <= t; ++j) {
    const float x = values[j * stride];
    if (fabsf(x) <= DB_LARGEST) continue;
    float weight = 0.0f;
    for (int e = 2; e >= 0; --e) weight += __bfloat162float(coef[(e * 2 * DB + row) * DB_MST + j]);
    sum = fmaf(weight, x, sum);
  }
  return sum;
}

// A CTA owns a request, a head and DB_COLS value columns; its state lies in registers (a warp 16 channels) and, for the read-outs, in
// shared memory in three parts.  A block: every warp forms the read-outs of all 64 rows (k and q) over its 16 channels;
// the warps' sums are added and v' made; a warp a tile of u or o from the block's matrices; the state.  The next block comes meanwhile, in two
// bulk copies.  Every product is one of float32 values in three bfloat16 parts each, all 24 bits, with sums of 16 or 32 products on the
// tensor cores; sums across channels and blocks are float32 additions.
// Bound by the 84 products a warp and block (of 3650 cycles a block the tensor cores take 2000, 12 a product and scheduler) between four
// barriers; bringing operands to registers in front of the barriers made it slower (4100).  2048 tokens, 16 heads of 128 x 128: 30 us
// for the matrices and 132 for the walk; in blocks of 16 with multiply-adds, bound by the reads of shared memory beside them, 31 and 210;
// token by token 522.  Error against 64 bits 0.8 of the token-by-token form's, as before (4 heads of 128 x 128, 777 tokens: 1.6e-7 and 1.2e-7 of
// the outputs and the state; blocks of 16 with multiply-adds 1.75e-7 and 1.35e-7, token by token 2.0e-7 and 1.9e-7).
template <typename T, int DP>
__global__ void __launch_bounds__(DB_THREADS, 1) delta_block_scan_kernel(const DeltaBlockScanArgs a) {
  using Shape = DeltaShape<DP>;
  constexpr int ST = Shape::ST, CST = Shape::CST, FST = Shape::FST, WARPS = DP / 16;      // WARPS: that hold channels
  extern __shared__ __align__(16) unsigned char db_smem[];
  unsigned char* at = db_smem + 2 * Shape::STAGE_BYTES;
  __nv_bfloat16* s_s = reinterpret_cast<__nv_bfloat16*>(at);                   // [part][DP][CST]
  __nv_bfloat16* vp_s = reinterpret_cast<__nv_bfloat16*>(at += Shape::S_BYTES);        // [part][DB][CST]: v'
  __nv_bfloat16* u_s = reinterpret_cast<__nv_bfloat16*>(at += Shape::V_BYTES);         // [part][DB][CST]: what the write takes
  float* vf_s = reinterpret_cast<float*>(at += Shape::V_BYTES);                // [DB][FST]: v'
  float* o_s = reinterpret_cast<float*>(at += Shape::F_BYTES);                 // [DB][FST]
  float* red_s = reinterpret_cast<float*>(at += Shape::F_BYTES);               // [warps][2 DB][DB_COLS], every other pair of rows turned by 8 columns
  __shared__ unsigned long long landed[2];
  __shared__ int wild;                                       // the last block with a v' that is left out of the product
  const int row = blockIdx.x, head = blockIdx.y, col0 = blockIdx.z * DB_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
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
  if (tid == 0) {
    mbar_init(&landed[0], 1);
    mbar_init(&landed[1], 1);
    fence_barrier_init();
    wild = -1;
  }
  __syncthreads();

  auto copy_block = [&](int p) {                             // one thread
    unsigned char* stage = db_smem + (p & 1) * Shape::STAGE_BYTES;
    mbar_arrive_expect_tx(&landed[p & 1], Shape::STAGE_BYTES);
    bulk_copy_g2s(stage, a.qk + (static_cast<long long>(first + p) * a.qk_heads + group) * Shape::QK_BYTES, Shape::QK_BYTES, &landed[p & 1]);
    bulk_copy_g2s(stage + Shape::QK_BYTES, a.coef + (static_cast<long long>(first + p) * a.heads + head) * DB_COEF_BYTES, DB_COEF_BYTES,
                  &landed[p & 1]);
  };
  // This thread's token and pair of columns where v' is made.
  const int my_t = tid / (DB_COLS / 2), my_c = tid % (DB_COLS / 2) * 2;
  const bool live0 = col0 + my_c < a.V, live1 = col0 + my_c + 1 < a.V;
  const T* v = static_cast<const T*>(a.v) + t0 * a.v_stride + head * a.V + col0 + my_c;
  auto fetch_v = [&](int p) {
    const int at_t = p * DB + my_t;
    return make_float2(at_t < n && live0 ? to_float(v[at_t * a.v_stride]) : 0.0f, at_t < n && live1 ? to_float(v[at_t * a.v_stride + 1]) : 0.0f);
  };
  // This thread's part of the state: channels d0 and d0 + 8, columns 8 i + 2 t and the next.
  const int d0 = warp * 16 + g;
  const bool holds = warp < WARPS;
  float S[2][4];
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride + (static_cast<long long>(head) * a.V + col0) * a.D;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      S[i][e] = holds && d < a.D && col0 + c < a.V ? state[static_cast<long long>(c) * a.D + d] : 0.0f;
    }
  auto store_state = [&]() {
    if (!holds) return;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        unsigned part[3];
        three_parts(S[i][2 * half], S[i][2 * half + 1], part[0], part[1], part[2]);
#pragma unroll
        for (int e = 0; e < 3; ++e) *reinterpret_cast<unsigned*>(s_s + (e * DP + d0 + 8 * half) * CST + 8 * i + 2 * t) = part[e];
      }
  };
  if (tid == 0 && blocks > 0) copy_block(0);
  store_state();
  float2 v_now = fetch_v(0);
  // ldmatrix addresses: rows as they lie, keys transposed, value columns as [k][n].
  const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lcol = (lane >> 4) * 8;
  const int a_off = lrow * ST + lcol, at_off = ((lane & 7) + (lane >> 4) * 8) * ST + ((lane >> 3) & 1) * 8, m_off = lrow * DB_MST + lcol;
  const int b_off = lrow * CST + lcol;
  constexpr int TILES = 2 * DB / 16, STEPS = DB / 16;
  for (int p = 0; p < blocks; ++p) {
    const unsigned char* stage = db_smem + (p & 1) * Shape::STAGE_BYTES;
    const __nv_bfloat16* qk_s = reinterpret_cast<const __nv_bfloat16*>(stage);                      // [part][k, q][ST]
    const __nv_bfloat16* coef_s = reinterpret_cast<const __nv_bfloat16*>(stage + Shape::QK_BYTES);  // [part][Tu, M][DB_MST]
    const float* steps = reinterpret_cast<const float*>(stage + Shape::QK_BYTES + DB_COEF_PARTS);
    const bool here = mbar_wait(&landed[p & 1], p >> 1 & 1, DB_WAIT_LIMIT);
    // The block and the state are there; the other buffer is no longer read.
    if (!__syncthreads_and(here)) {
      if (tid == 0) report(a.status, STATUS_COPY_TIMEOUT, p, row);
      let_copies_land();
      return;
    }
    if (tid == 0 && p + 1 < blocks) copy_block(p + 1);
    const float2 v_next = fetch_v(p + 1);
    if (holds) {
      unsigned af[TILES][3][4], bf[TILES][3][4];
      float high[TILES][2][4] = {}, low[TILES][2][4] = {};
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        ldmatrix_x4_trans(bf[0][e], s_s + (e * DP + warp * 16) * CST + b_off);
#pragma unroll
        for (int mt = 0; mt < TILES; ++mt) ldmatrix_x4(af[mt][e], qk_s + (e * 2 * DB + mt * 16) * ST + a_off + warp * 16);
#pragma unroll
        for (int mt = 1; mt < TILES; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) bf[mt][e][i] = bf[0][e][i];
      }
      delta_products<TILES, 2>(high, low, af, bf);
#pragma unroll
      for (int mt = 0; mt < TILES; ++mt)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int r = mt * 16 + g + 8 * half;
            *reinterpret_cast<float2*>(red_s + (warp * 2 * DB + r) * DB_COLS + ((8 * i + 2 * t + (r >> 1 & 1) * 8) & 15)) =
                make_float2(high[mt][i][2 * half] + low[mt][i][2 * half], high[mt][i][2 * half + 1] + low[mt][i][2 * half + 1]);
          }
    }
    __syncthreads();
    {
      float2 rk = make_float2(0.0f, 0.0f), rq = rk;
      const float* from = red_s + my_t * DB_COLS + ((my_c + (my_t >> 1 & 1) * 8) & 15);
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float2 x = *reinterpret_cast<const float2*>(from + w * 2 * DB * DB_COLS);
        const float2 y = *reinterpret_cast<const float2*>(from + (w * 2 * DB + DB) * DB_COLS);
        rk.x += x.x; rk.y += x.y; rq.x += y.x; rq.y += y.y;
      }
      const float lead = steps[my_t];
      float x = v_now.x - lead * rk.x, y = v_now.y - lead * rk.y;
      *reinterpret_cast<float2*>(vf_s + my_t * FST + my_c) = make_float2(x, y);
      *reinterpret_cast<float2*>(o_s + my_t * FST + my_c) = make_float2(lead * rq.x, lead * rq.y);
      if (!(fabsf(x) <= DB_LARGEST)) { x = 0.0f; wild = p; }
      if (!(fabsf(y) <= DB_LARGEST)) { y = 0.0f; wild = p; }
      unsigned part[3];
      three_parts(x, y, part[0], part[1], part[2]);
#pragma unroll
      for (int e = 0; e < 3; ++e) *reinterpret_cast<unsigned*>(vp_s + (e * DB + my_t) * CST + my_c) = part[e];
    }
    __syncthreads();
    {
      // Rows 16 mt .. + 15 of Tu over M, columns 8 nt .. + 7.  (What lies above the diagonal is zeros.)
      const int mt = warp >> 1, nt = warp & 1;
      unsigned af[STEPS][3][4], bf[STEPS][3][2];
      float high[STEPS][1][4] = {}, low[STEPS][1][4] = {};
      const int b_tile = (lane & 7) + ((lane >> 3) & 1) * 8;      // (the other lanes' addresses are not used)
#pragma unroll
      for (int ks = 0; ks < STEPS; ++ks)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          ldmatrix_x4(af[ks][e], coef_s + (e * 2 * DB + mt * 16) * DB_MST + m_off + ks * 16);
          ldmatrix_x2_trans(bf[ks][e], vp_s + (e * DB + ks * 16 + b_tile) * CST + nt * 8);
        }
      delta_products<STEPS, 1>(high, low, af, bf);
      const bool tame = wild != p;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = mt * 16 + g + 8 * half, tok = r % DB, c = 8 * nt + 2 * t;
        float x = (high[0][0][2 * half] + high[1][0][2 * half]) + (low[0][0][2 * half] + low[1][0][2 * half]);
        float y = (high[0][0][2 * half + 1] + high[1][0][2 * half + 1]) + (low[0][0][2 * half + 1] + low[1][0][2 * half + 1]);
        if (!tame) {
          x += delta_wild(coef_s, r, tok, vf_s + c, FST);
          y += delta_wild(coef_s, r, tok, vf_s + c + 1, FST);
        }
        if (r < DB) {
          unsigned part[3];
          three_parts(x, y, part[0], part[1], part[2]);
#pragma unroll
          for (int e = 0; e < 3; ++e) *reinterpret_cast<unsigned*>(u_s + (e * DB + tok) * CST + c) = part[e];
        } else if (p * DB + tok < n) {
          float* to = a.out + (t0 + p * DB + tok) * a.heads * a.V + static_cast<long long>(head) * a.V + col0 + c;
          const float2 o = *reinterpret_cast<const float2*>(o_s + tok * FST + c);
          if (a.V % 2 == 0 && col0 + c < a.V) {
            *reinterpret_cast<float2*>(to) = make_float2(x + o.x, y + o.y);
          } else {
            if (col0 + c < a.V) to[0] = x + o.x;
            if (col0 + c + 1 < a.V) to[1] = y + o.y;
          }
        }
      }
    }
    __syncthreads();
    if (holds) {
      unsigned af[STEPS][3][4], bf[STEPS][3][4];
      float high[STEPS][2][4] = {}, low[STEPS][2][4] = {};
#pragma unroll
      for (int ks = 0; ks < STEPS; ++ks)
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          ldmatrix_x4_trans(af[ks][e], qk_s + (e * 2 * DB + ks * 16) * ST + at_off + warp * 16);
          ldmatrix_x4_trans(bf[ks][e], u_s + (e * DB + ks * 16) * CST + b_off);
        }
      delta_products<STEPS, 2>(high, low, af, bf);
      const float whole = steps[DB];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[i][e] = fmaf(whole, S[i][e], (high[0][i][e] + high[1][i][e]) + (low[0][i][e] + low[1][i][e]));
    }
    store_state();               // (nobody reads the state's tile between the first barrier above and the next one)
    v_now = v_next;
  }
  if (!a.write_state || !holds) return;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = d0 + (e >> 1) * 8, c = 8 * i + 2 * t + (e & 1);
      if (d < a.D && col0 + c < a.V) state[static_cast<long long>(c) * a.D + d] = S[i][e];
    }
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
ZB_API int zb_delta_block_floats(int qk_heads, int heads, int D) {
  return (qk_heads * (D <= 64 ? DeltaShape<64>::QK_BYTES : DeltaShape<128>::QK_BYTES) + heads * DB_COEF_BYTES) / 4;
}

template <typename T, int DP>
static int delta_block_launch(DeltaBlocksArgs b, DeltaBlockScanArgs a, float* ws, int rows, int blocks, cudaStream_t s) {
  using Shape = DeltaShape<DP>;
  b.qk = reinterpret_cast<unsigned char*>(ws);
  b.coef = b.qk + static_cast<long long>(blocks) * b.qk_heads * Shape::QK_BYTES;
  a.qk = b.qk; a.coef = b.coef;
  if (cuda_failed(cudaFuncSetAttribute(delta_blocks_kernel<T, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::BLOCKS_SMEM)) ||
      cuda_failed(cudaFuncSetAttribute(delta_block_scan_kernel<T, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SCAN_SMEM)))
    return ERR_CUDA;
  launch_dependent(delta_blocks_kernel<T, DP>, dim3(blocks, b.qk_heads), dim3(DB_THREADS), Shape::BLOCKS_SMEM, s, false, b);
  // (Not as a dependent: its CTAs would take the SMs that the kernel before it leaves first, while others stay empty.)
  delta_block_scan_kernel<T, DP><<<dim3(rows, a.heads, (a.V + DB_COLS - 1) / DB_COLS), DB_THREADS, Shape::SCAN_SMEM, s>>>(a);
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
  const int blocks = tokens / DB + rows;
  DeltaBlocksArgs g;
  g.q = q; g.q_stride = q_stride; g.k = k;
  g.k_stride = k_stride; g.b = b; g.a = a; g.ba_stride = ba_stride; g.a_log = a_log; g.dt_bias = dt_bias;
  g.row_q_start = row_q_start; g.row_q_len = row_q_len; g.rows = rows; g.from = from; g.qk_heads = qk_heads; g.heads = heads; g.D = D;
  g.q_scale = q_scale; g.unit_eps = unit_eps;
  DeltaBlockScanArgs c;
  c.out = out; c.v = v; c.v_stride = v_stride; c.state = state; c.slot_stride = slot_stride;
  c.slots = slots; c.row_q_start = row_q_start; c.row_q_len = row_q_len; c.heads = heads; c.qk_heads = qk_heads; c.D = D; c.V = V;
  c.num_slots = num_slots; c.write_state = write_state; c.from = from; c.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == DTYPE_F32)
    return D <= 64 ? delta_block_launch<float, 64>(g, c, ws, rows, blocks, s) : delta_block_launch<float, 128>(g, c, ws, rows, blocks, s);
  return D <= 64 ? delta_block_launch<__nv_bfloat16, 64>(g, c, ws, rows, blocks, s)
                 : delta_block_launch<__nv_bfloat16, 128>(g, c, ws, rows, blocks, s);
}
