// Layers that carry a state of fixed size from token to token, and the norms around them.
//
//   * layer norm with scale and shift, alone and fused with the residual sum: the residual stream is
//     float32; r += m * LN_post(delta), then y = LN_pre(r), in one pass over the row;
//   * a table lookup that writes float32 rows (the start of a float32 residual stream);
//   * the causal convolution over a few taps per channel with its SiLU, whose last taps - 1 inputs
//     live in the request's state slot;
//   * the decayed outer-product recurrence  S_t = diag(a_t) S_{t-1} + k_t v_t^T,  o_t = S_t^T q_t
//     per head, S [D, V] float32 in the request's state slot, in three settings: a decay per key channel
//     a = sigmoid(z)^(1/tau) (gated linear attention), and one decay per head a = exp(-exp(A) dt)
//     with k = dt B, q = C and a skip term D x (the state-space form of Mamba-2), and a constant decay per
//     head (retention); long portions with one decay per head run on tensor cores, state_walk.cu and
//     retention.cu;
//   * the rotation of halves on the q and k heads of a fused projection, k with a multiplier;
//   * the RMS norm over equal groups of a row with a SiLU gate before or behind it.
//
// Everything that enters the recurrence is float32: decays, their logarithms, softplus, step sizes,
// the state, the sums.  A row's tokens are run in their order, so a result does not depend on how a
// prompt was cut into steps or on what else a step carries.
#include <algorithm>
#include <initializer_list>

#include "common.cuh"

namespace zb {

// z / (1 + e^-z).  The quotient is the reciprocal's estimate times z, corrected once by its remainder (fused, so exact to
// rounding, after Markstein: of all 2^32 inputs none differs from the divide operator's result): that operator's guarded form
// kept a thread's values one behind the other.  Where the correction has no
// meaning (an infinite z or e^-z), the uncorrected product is the quotient.
__device__ __forceinline__ float silu_f(float z) {
  const float d = 1.0f + expf(-z);
  float r;
  asm("rcp.approx.f32 %0, %1;\n" : "=f"(r) : "f"(d));
  const float q = z * r, better = fmaf(fmaf(-d, q, z), r, q);
  return better == better ? better : q;
}
__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.0f) - log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

// ------------------------------------------------------------------------------------------------
// Layer norm.  One CTA per row; the row sits in shared memory as float32, mean and variance are
// two passes over it (the variance is the mean of the squared deviations).
// A norm without a shift passes a null pointer for it.
__device__ __forceinline__ float load_shift(const void* b, int w_dtype, int i) {
  return b != nullptr ? load_scale(b, w_dtype, i) : 0.0f;
}

__device__ __forceinline__ void layer_norm_stats(const float* row, int H, float eps, float* scratch, float& mean,
                                                 float& rstd, bool rms = false) {
  if (rms) {          // an RMS norm: no mean is taken off, the statistic is the mean square
    float v = 0.0f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) v = fmaf(row[i], row[i], v);
    mean = 0.0f;
    rstd = 1.0f / sqrtf(block_sum(v, scratch) / static_cast<float>(H) + eps);
    return;
  }
  float s = 0.0f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) s += row[i];
  mean = block_sum(s, scratch) / static_cast<float>(H);
  float v = 0.0f;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float d = row[i] - mean;
    v = fmaf(d, d, v);
  }
  rstd = 1.0f / sqrtf(block_sum(v, scratch) / static_cast<float>(H) + eps);
}

template <typename X, typename T>
__global__ void layer_norm_kernel(T* out, const X* x, const void* w, const void* b, int w_dtype, float eps, int H) {
  extern __shared__ __align__(16) float ln_row[];
  __shared__ float scratch[33];
  const size_t base = static_cast<size_t>(blockIdx.x) * H;
  for (int i = threadIdx.x; i < H; i += blockDim.x) ln_row[i] = to_float(x[base + i]);
  __syncthreads();
  float mean, rstd;
  layer_norm_stats(ln_row, H, eps, scratch, mean, rstd);
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    out[base + i] = from_float<T>(fmaf((ln_row[i] - mean) * rstd, load_scale(w, w_dtype, i), load_shift(b, w_dtype, i)));
}

// residual += mult * LN(delta; w1, b1); then, if `out`, out = LN(residual; w2, b2), or with a null w2
// the sum itself in T (what a part that reads the stream unnormed takes).  RMS: both norms are RMS norms
// (x / sqrt(mean(x^2) + eps) * w, no mean taken off, no shift).
template <typename T, bool RMS>
__global__ void residual_layer_norm_kernel(float* residual, const T* delta, const void* w1, const void* b1, float mult,
                                           T* out, const void* w2, const void* b2, int w_dtype, float eps1, float eps2,
                                           int H) {
  extern __shared__ __align__(16) float ln_row[];
  __shared__ float scratch[33];
  const size_t base = static_cast<size_t>(blockIdx.x) * H;
  for (int i = threadIdx.x; i < H; i += blockDim.x) ln_row[i] = to_float(delta[base + i]);
  __syncthreads();
  float mean, rstd;
  layer_norm_stats(ln_row, H, eps1, scratch, mean, rstd, RMS);
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float y = fmaf((ln_row[i] - mean) * rstd, load_scale(w1, w_dtype, i), load_shift(b1, w_dtype, i));
    const float r = fmaf(mult, y, residual[base + i]);
    residual[base + i] = r;
    ln_row[i] = r;              // each thread rewrites only the elements it read
    if (out != nullptr && w2 == nullptr) out[base + i] = from_float<T>(r);     // no second norm: the sum, rounded
  }
  if (out == nullptr || w2 == nullptr) return;
  __syncthreads();
  layer_norm_stats(ln_row, H, eps2, scratch, mean, rstd, RMS);
  for (int i = threadIdx.x; i < H; i += blockDim.x)
    out[base + i] = from_float<T>(fmaf((ln_row[i] - mean) * rstd, load_scale(w2, w_dtype, i), load_shift(b2, w_dtype, i)));
}

// The same two kernels for rows of up to LN_VEC_MAX elements whose length is a multiple of four: a thread
// keeps its share of the row in registers as vectors of four, loads and stores move 8 or 16 bytes, and
// nothing passes through shared memory but the two sums.  All that a row of up to 2048 elements needs is asked for before the
// first sum (the row it is added to was read behind it, the scales behind that): a decode step's few rows wait for one latency,
// not three, 12 rows of 2048 into the residual stream 6.1 -> 3.6 us.  A longer row's thread would hold 64 values that way, and
// half as many CTAs share an SM (2048 rows of 4096: 27 us, 21 read where they are used).
constexpr int LN_VEC_THREADS = 256;
constexpr int LN_VEC_ITEMS = 8;
constexpr int LN_VEC_MAX = LN_VEC_THREADS * LN_VEC_ITEMS * 4;

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  uint2 raw;
  *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(v.x, v.y);
  *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = raw;
}

template <int ITEMS>
__device__ __forceinline__ void vec_stats(const float4 (&r)[ITEMS], int nv, int H, float eps, float* scratch,
                                          float& mean, float& rstd, bool rms = false) {
  if (rms) {
    float v = 0.0f;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (static_cast<int>(threadIdx.x) + j * LN_VEC_THREADS < nv)
        v += (r[j].x * r[j].x + r[j].y * r[j].y) + (r[j].z * r[j].z + r[j].w * r[j].w);
    mean = 0.0f;
    rstd = 1.0f / sqrtf(block_sum(v, scratch) / static_cast<float>(H) + eps);
    return;
  }
  float s = 0.0f;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (static_cast<int>(threadIdx.x) + j * LN_VEC_THREADS < nv) s += (r[j].x + r[j].y) + (r[j].z + r[j].w);
  mean = block_sum(s, scratch) / static_cast<float>(H);
  float v = 0.0f;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j)
    if (static_cast<int>(threadIdx.x) + j * LN_VEC_THREADS < nv) {
      const float a = r[j].x - mean, b = r[j].y - mean, c = r[j].z - mean, d = r[j].w - mean;
      v += (a * a + b * b) + (c * c + d * d);
    }
  rstd = 1.0f / sqrtf(block_sum(v, scratch) / static_cast<float>(H) + eps);
}

__device__ __forceinline__ float4 vec_affine(float4 x, float mean, float rstd, float4 wv, float4 bv) {
  return make_float4(fmaf((x.x - mean) * rstd, wv.x, bv.x), fmaf((x.y - mean) * rstd, wv.y, bv.y),
                     fmaf((x.z - mean) * rstd, wv.z, bv.z), fmaf((x.w - mean) * rstd, wv.w, bv.w));
}

// A thread's scales and shifts: a short row's are asked for before its first sum, a long row's where they are used.
template <int ITEMS> struct VecAffine {
  static constexpr bool KEPT = ITEMS <= 2;
  const float* w;
  const float* b;
  float4 wv[KEPT ? ITEMS : 1], bv[KEPT ? ITEMS : 1];
  __device__ __forceinline__ VecAffine(const float* w_, const float* b_, int nv) : w(w_), b(b_) {
    if (!KEPT || w == nullptr) return;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int i = threadIdx.x + j * LN_VEC_THREADS;
      if (i < nv) {
        wv[j] = load4(w + 4 * i);
        bv[j] = b != nullptr ? load4(b + 4 * i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
  }
  __device__ __forceinline__ float4 operator()(float4 x, float mean, float rstd, int j) const {
    if (KEPT) return vec_affine(x, mean, rstd, wv[j], bv[j]);
    const int at = 4 * (threadIdx.x + j * LN_VEC_THREADS);
    return vec_affine(x, mean, rstd, load4(w + at), b != nullptr ? load4(b + at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f));
  }
};

template <typename X, typename T, int ITEMS>
__global__ void __launch_bounds__(LN_VEC_THREADS)
layer_norm_vec_kernel(T* out, const X* x, const float* w, const float* b, float eps, int H) {
  wait_for_prior_grids();
  let_dependents_launch();
  __shared__ float scratch[33];
  const size_t base = static_cast<size_t>(blockIdx.x) * H;
  const int nv = H / 4;
  float4 r[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x + j * LN_VEC_THREADS;
    if (i < nv) r[j] = load4(x + base + 4 * i);
  }
  const VecAffine<ITEMS> affine(w, b, nv);
  float mean, rstd;
  vec_stats(r, nv, H, eps, scratch, mean, rstd);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x + j * LN_VEC_THREADS;
    if (i < nv) store4(out + base + 4 * i, affine(r[j], mean, rstd, j));
  }
}

template <typename T, bool RMS, int ITEMS>
__global__ void __launch_bounds__(LN_VEC_THREADS)
residual_layer_norm_vec_kernel(float* residual, const T* delta, const float* w1, const float* b1, float mult, T* out,
                               const float* w2, const float* b2, float eps1, float eps2, int H) {
  wait_for_prior_grids();
  let_dependents_launch();
  __shared__ float scratch[33];
  const size_t base = static_cast<size_t>(blockIdx.x) * H;
  const int nv = H / 4;
  constexpr bool AHEAD = VecAffine<ITEMS>::KEPT;
  float4 r[ITEMS], old[AHEAD ? ITEMS : 1];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x + j * LN_VEC_THREADS;
    if (i < nv) {
      r[j] = load4(delta + base + 4 * i);
      if (AHEAD) old[AHEAD ? j : 0] = load4(residual + base + 4 * i);
    }
  }
  const VecAffine<ITEMS> first(w1, b1, nv), second(out != nullptr ? w2 : nullptr, b2, nv);
  float mean, rstd;
  vec_stats(r, nv, H, eps1, scratch, mean, rstd, RMS);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x + j * LN_VEC_THREADS;
    if (i < nv) {
      const float4 y = first(r[j], mean, rstd, j), was = AHEAD ? old[AHEAD ? j : 0] : load4(residual + base + 4 * i);
      r[j] = make_float4(fmaf(mult, y.x, was.x), fmaf(mult, y.y, was.y), fmaf(mult, y.z, was.z), fmaf(mult, y.w, was.w));
      store4(residual + base + 4 * i, r[j]);
      if (out != nullptr && w2 == nullptr) store4(out + base + 4 * i, r[j]);   // no second norm: the sum, rounded
    }
  }
  if (out == nullptr || w2 == nullptr) return;
  vec_stats(r, nv, H, eps2, scratch, mean, rstd, RMS);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x + j * LN_VEC_THREADS;
    if (i < nv) store4(out + base + 4 * i, second(r[j], mean, rstd, j));
  }
}

// True if rows of H elements and these pointers take the vector kernels (float32 scales).
inline bool ln_vectors(int H, int w_dtype, std::initializer_list<const void*> pointers) {
  if (H % 4 != 0 || H > LN_VEC_MAX || w_dtype != DTYPE_F32) return false;
  for (const void* p : pointers)
    if (p != nullptr && reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
  return true;
}

// out = scale * table[id] as float32; `rounded` (may be null) gets the same rows in the table's type.
template <typename T>
__global__ void embedding_f32_kernel(float* out, T* rounded, const T* table, const int* ids, float scale, int H, int V,
                                     int* status) {
  const int t = blockIdx.x, id = ids[t];
  const bool ok = id >= 0 && id < V;
  if (!ok && threadIdx.x == 0) report(status, STATUS_TOKEN_OUT_OF_RANGE, id, t);
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    const float v = ok ? scale * to_float(table[static_cast<size_t>(id) * H + i]) : 0.0f;
    out[static_cast<size_t>(t) * H + i] = v;
    if (rounded != nullptr) rounded[static_cast<size_t>(t) * H + i] = from_float<T>(v);
  }
}

// The same four values a thread and a CTA for every 512 columns, where rows are whole aligned pieces of four: a few tokens'
// rows are one load each instead of a loop of single values that waits for every store (12 rows of 2048: 10.8 us, now below 2.9).
template <typename T>
__global__ void __launch_bounds__(128) embedding_f32_vec_kernel(float* out, T* rounded, const T* table, const int* ids, float scale,
                                                                int H, int V, int* status) {
  wait_for_prior_grids();
  let_dependents_launch();
  const int t = blockIdx.x, id = ids[t], i = 4 * (blockIdx.y * 128 + threadIdx.x);
  const bool ok = id >= 0 && id < V;
  if (!ok && threadIdx.x == 0 && blockIdx.y == 0) report(status, STATUS_TOKEN_OUT_OF_RANGE, id, t);
  if (i >= H) return;
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (ok) {
    v = load4(table + static_cast<size_t>(id) * H + i);
    v = make_float4(scale * v.x, scale * v.y, scale * v.z, scale * v.w);
  }
  store4(out + static_cast<size_t>(t) * H + i, v);
  if (rounded != nullptr) store4(rounded + static_cast<size_t>(t) * H + i, v);
}

template <typename T>
void embedding_f32(float* out, T* rounded, const T* table, const int* ids, float scale, int tokens, int H, int V, int* status,
                   cudaStream_t s) {
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (H % 4 == 0 && H <= 512 * 65535 && aligned(out) && aligned(rounded) && aligned(table))
    launch_dependent(embedding_f32_vec_kernel<T>, dim3(tokens, (H + 511) / 512), dim3(128), 0, s, false, out, rounded,
        table, ids, scale, H, V, status);
  else
    embedding_f32_kernel<T><<<tokens, 128, 0, s>>>(out, rounded, table, ids, scale, H, V, status);
}

// ------------------------------------------------------------------------------------------------
// Causal convolution per channel with SiLU, over all new tokens of the step at once; the inputs before
// a request's first new token come from its state (zeros for a new request), and a second small
// kernel then puts the request's last taps - 1 inputs there.
constexpr int CONV_MAX_TAPS = 8;

struct ConvArgs {
  void* out;                 // [tokens, C]
  const void* x;             // [tokens, x_stride], channel c at column c
  long long x_stride;
  float* state;              // slot s at state + s * slot_stride: [taps - 1][C], oldest input first
  long long slot_stride;
  const int* slots;
  const int* row_q_start;
  const int* row_q_len;
  const void* w;             // [C, taps], the last column weighs the current token
  const void* bias;          // [C]
  int w_dtype, C, taps, num_slots, write_state;
  int* status;
};

// The convolution proper: a thread owns a channel of one token (CONV_TOKENS consecutive ones) of the
// step's stream.  Input i of a request's new tokens is row t0 + i of x for i >= 0 and entry taps - 1 + i of
// the request's state for i < 0; nothing is written to the state here.
constexpr int CONV_TOKENS = 1;

template <typename T>
__global__ void causal_conv_silu_kernel(const ConvArgs a, const int* token_row, int tokens) {
  wait_for_prior_grids();
  let_dependents_launch();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= a.C) return;
  float w[CONV_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) w[j] = j < a.taps ? load_scale(a.w, a.w_dtype, c * a.taps + j) : 0.0f;
  const float bias = load_scale(a.bias, a.w_dtype, c);
  const T* x = static_cast<const T*>(a.x);
  T* out = static_cast<T*>(a.out);
  const int first = blockIdx.x * CONV_TOKENS;
  for (int t = first; t < min(first + CONV_TOKENS, tokens); ++t) {
    const int row = token_row[t];
    const int slot = a.slots[row];
    if (slot < 0 || slot >= a.num_slots) {
      report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
      continue;
    }
    const int i = t - a.row_q_start[row];
    const float* state = a.state + static_cast<long long>(slot) * a.slot_stride;
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {          // oldest input first, as the weights lie
      if (j < a.taps) {
        const int back = a.taps - 1 - j;
        const float in = i - back >= 0 ? to_float(x[static_cast<long long>(t - back) * a.x_stride + c])
                                       : state[static_cast<long long>(a.taps - 1 + i - back) * a.C + c];
        acc = fmaf(w[j], in, acc);
      }
    }
    out[static_cast<long long>(t) * a.C + c] = from_float<T>(silu_f(acc + bias));
  }
}

// The form for runs of tokens (rows that start on a vector's boundary): a CTA takes CONV_RUN consecutive tokens of the
// stream, a thread VEC neighbouring channels of them.  Bound by latency where a thread walks its tokens one load
// behind the other, so it asks for all its inputs, the TAPS - 1 before the first token among them, before it uses any
// (they come again from the cache for the next CTA); inputs before a request's first new token come from its state.
// 2125 tokens of 2560 bfloat16 channels 13.5 us (15.3 with a divide in the activation, 21.7 walked 32 tokens a thread), 2048
// tokens of 4096 float32 channels 17.6 us (20.3; 69.6 with a thread a channel and token).  Six CTAs an SM: at five, which the
// registers of its own choice allow, 14.2 and 17.0 us; at seven and eight registers spill, 14.5 and 17.9, 15.5 and 19.3 us.
// TAPS: the taps of the kernel, `taps` of them in use (the others, at the old end, are skipped).
constexpr int CONV_RUN = 8;

template <typename T, int VEC>
__device__ __forceinline__ void conv_load(float (&x)[VEC], const T* p) {
  if constexpr (VEC == 4) {
    const float4 v = load4(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else if constexpr (sizeof(T) == 4) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x[0] = v.x; x[1] = v.y;
  } else {
    const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
    x[0] = v.x; x[1] = v.y;
  }
}
template <typename T, int VEC>
__device__ __forceinline__ void conv_store(T* p, const float (&y)[VEC]) {
  if constexpr (VEC == 4) store4(p, make_float4(y[0], y[1], y[2], y[3]));
  else if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(p) = make_float2(y[0], y[1]);
  else *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(y[0], y[1]);
}

template <typename T, int VEC, int TAPS>
__global__ void __launch_bounds__(128, VEC == 4 && TAPS == 4 ? 6 : 1) causal_conv_silu_run_kernel(const ConvArgs a, const int* token_row, int tokens) {
  wait_for_prior_grids();
  let_dependents_launch();
  __shared__ int first_s[CONV_RUN], slot_s[CONV_RUN];         // per token: index within its request's new tokens, slot
  const int t0 = blockIdx.x * CONV_RUN, nt = min(CONV_RUN, tokens - t0);
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * VEC;
  const bool works = c < a.C;
  const int skipped = TAPS - a.taps;
  const T* x = static_cast<const T*>(a.x);
  float in[TAPS - 1 + CONV_RUN][VEC];
#pragma unroll
  for (int i = 0; i < TAPS - 1 + CONV_RUN; ++i) {
    const int t = t0 - (TAPS - 1) + i;
#pragma unroll
    for (int v = 0; v < VEC; ++v) in[i][v] = 0.0f;
    if (works && i >= skipped && t >= 0 && t < tokens) conv_load<T, VEC>(in[i], x + t * a.x_stride + c);
  }
  if (threadIdx.x < nt) {
    const int row = token_row[t0 + threadIdx.x];
    const int slot = a.slots[row];
    first_s[threadIdx.x] = t0 + threadIdx.x - a.row_q_start[row];
    slot_s[threadIdx.x] = slot;
    if (slot < 0 || slot >= a.num_slots) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
  }
  const float* wp = static_cast<const float*>(a.w);
  float w[TAPS][VEC], bias[VEC];
  const bool quads = a.taps == 4 && reinterpret_cast<uintptr_t>(wp) % 16 == 0;      // a channel's weights in one read
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    bias[v] = works ? static_cast<const float*>(a.bias)[c + v] : 0.0f;
    if (TAPS == 4 && quads) {
      const float4 four = works ? load4(wp + (c + v) * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      w[0][v] = four.x; w[1][v] = four.y; w[2][v] = four.z; w[3][v] = four.w;
      continue;
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j) w[j][v] = works && j >= skipped ? wp[(c + v) * a.taps + (j - skipped)] : 0.0f;
  }
  __syncthreads();
  if (!works) return;
  T* out = static_cast<T*>(a.out);
#pragma unroll
  for (int k = 0; k < CONV_RUN; ++k) {
    if (k >= nt) break;
    const int i = first_s[k], slot = slot_s[k];
    if (slot < 0 || slot >= a.num_slots) continue;
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.0f;
    if (i >= TAPS - 1) {
#pragma unroll
      for (int j = 0; j < TAPS; ++j)
        if (j >= skipped) {
#pragma unroll
          for (int v = 0; v < VEC; ++v) acc[v] = fmaf(w[j][v], in[k + j][v], acc[v]);
        }
    } else {
      const float* state = a.state + static_cast<long long>(slot) * a.slot_stride;
#pragma unroll
      for (int j = 0; j < TAPS; ++j)
        if (j >= skipped) {
          const int back = TAPS - 1 - j;
#pragma unroll
          for (int v = 0; v < VEC; ++v)
            acc[v] = fmaf(w[j][v], i >= back ? in[k + j][v] : state[static_cast<long long>(a.taps - 1 + i - back) * a.C + c + v], acc[v]);
        }
    }
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = silu_f(acc[v] + bias[v]);
    conv_store<T, VEC>(out + static_cast<long long>(t0 + k) * a.C + c, acc);
  }
}

template <typename T>
static void conv_run_launch(const ConvArgs& a, const int* token_row, int tokens, bool four, cudaStream_t s) {
  const int vectors = a.C / (four ? 4 : 2);
  const dim3 grid((tokens + CONV_RUN - 1) / CONV_RUN, (vectors + 127) / 128);
  if (a.taps <= 4) {
    if (four) launch_dependent(causal_conv_silu_run_kernel<T, 4, 4>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
    else launch_dependent(causal_conv_silu_run_kernel<T, 2, 4>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
  } else {
    if (four) launch_dependent(causal_conv_silu_run_kernel<T, 4, 8>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
    else launch_dependent(causal_conv_silu_run_kernel<T, 2, 8>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
  }
}

// After it: every request's last taps - 1 inputs go to its state.  A thread owns a channel of one request.
template <typename T>
__global__ void conv_state_update_kernel(const ConvArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  const int c = blockIdx.x * blockDim.x + threadIdx.x, row = blockIdx.y;
  if (c >= a.C) return;
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) return;       // reported by the convolution
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride;
  const T* x = static_cast<const T*>(a.x);
  const int t0 = a.row_q_start[row], n = a.row_q_len[row], keep = a.taps - 1;
  float last[CONV_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j) {
    if (j < keep) {
      const int i = n - keep + j;                     // the input that becomes entry j
      last[j] = i >= 0 ? to_float(x[static_cast<long long>(t0 + i) * a.x_stride + c])
                       : state[static_cast<long long>(keep + i) * a.C + c];
    }
  }
#pragma unroll
  for (int j = 0; j < CONV_MAX_TAPS; ++j)
    if (j < keep) state[static_cast<long long>(j) * a.C + c] = last[j];
}

// ------------------------------------------------------------------------------------------------
// The recurrence.  A CTA owns one request, one head and 64 value columns; warp w owns the key
// channels 16 w .. 16 w + 15 of those columns, each lane two columns (32 apart) with their 2 x 16 state
// values in registers, so that a decay, key and query fetched from shared memory serve two columns (two warps per scheduler and more: one warp's shared-memory loads hide behind another's
// multiply-adds).  The tokens of the request are taken SCAN_CHUNK at a time: decays, keys, queries and
// values of the chunk lie in shared memory (all float32), every warp runs the chunk's tokens in
// order, and the warps' partial outputs are added in warp order.  While a chunk runs, the next one's
// inputs are already on their way into registers.  The gated form's decays are made beforehand, in
// place of their logits, by a kernel of their own (every CTA of a head would otherwise repeat them).
constexpr int SCAN_CHUNK = 16;
constexpr int SCAN_ROWS = 16;        // key channels per warp
constexpr int SCAN_COLS = 64;        // value columns per CTA: two a lane, 32 apart
constexpr int SCAN_V_REGS = SCAN_CHUNK * SCAN_COLS / 64;   // values a thread fetches ahead, at most (a CTA has two warps or more)

constexpr int SCAN_GATED = 0;        // a[d] given per key channel (made from the logits by gated_decay_kernel), q scaled
constexpr int SCAN_STATE_SPACE = 1;  // a = exp(-exp(A_log[h]) dt), k = dt B, q = C, o += skip[h] v, dt = softplus(. + dt_bias[h])
constexpr int SCAN_FIXED = 2;        // a = decay[h], the same for every token

struct ScanArgs {
  const void* q; long long q_stride;   // [tokens, .]: head h (or its group) at column h * D
  const void* k; long long k_stride;
  const void* v; long long v_stride;   // [tokens, .]: head h at column h * V
  const float* z; long long z_stride;  // gated: decays [tokens, H * D], float32
  const void* dt; long long dt_stride; // state space: [tokens, H]
  const void* dt_bias; const void* a_log; const void* skip;   // state space: [H] each
  const float* decay;                  // fixed: [H]
  int w_dtype;
  float* state; long long slot_stride; // slot s at state + s * slot_stride: [H][D][V]
  float* out;                          // [tokens, H * V] float32
  const int* slots; const int* row_q_start; const int* row_q_len;
  int H, D, V, heads_per_group, num_slots, write_state;
  int below;                           // SCAN_PASS_SHORT: only requests with fewer than this many new tokens
  float q_scale;
  // Long requests in segments that run side by side (seg_len 0: every request is one piece).  Segment g of
  // a request covers its new tokens g seg_len .. (g + 1) seg_len - 1.  A first pass runs every segment
  // but a request's last from a zero state and leaves the state it ends with and the product of its
  // decays per key channel in ws_state / ws_decay; scan_carry_kernel turns those into the true state at
  // the start of every segment; the second pass runs every segment from there and writes the outputs.
  int seg_len, segs;                   // segs: segments per request in the grid (an upper bound)
  float* ws_state;                     // [rows * segs][H][D][V]
  float* ws_decay;                     // [rows * segs][H][D]
  int* status;
};

constexpr int SCAN_PASS_OUTPUT = 0;  // from the request's state (or a segment's start state), with outputs
constexpr int SCAN_PASS_LOCAL = 1;   // from zero, without outputs: what a segment adds, and its decays' product
// As SCAN_PASS_OUTPUT, for requests of fewer than `below` new tokens.  A form of its own: a request's length looked at in front of
// the loop, wherever it stood, cost 30 rows of 20 tokens 87 -> 113 us.
constexpr int SCAN_PASS_SHORT = 2;

// ws_state[g] <- the state at the start of segment g + 1: decay(g) * (state at the start of g) + ws_state[g].
__global__ void scan_carry_kernel(float* ws_state, const float* ws_decay, const float* state, long long slot_stride,
                                  const int* slots, const int* row_q_len, int segs, int seg_len, int H, int D, int V,
                                  int num_slots) {
  const long long per = static_cast<long long>(H) * D * V;
  const long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int row = blockIdx.y;
  if (e >= per) return;
  const int slot = slots[row];
  if (slot < 0 || slot >= num_slots) return;
  const int used = (row_q_len[row] + seg_len - 1) / seg_len;
  const long long channel = e / V;                       // h * D + d
  float prev = state[static_cast<long long>(slot) * slot_stride + e];
  for (int g = 0; g + 1 < used; ++g) {
    const long long at = static_cast<long long>(row) * segs + g;
    prev = fmaf(ws_decay[at * H * D + channel], prev, ws_state[at * per + e]);
    ws_state[at * per + e] = prev;
  }
}

// z <- sigmoid(z + bias)^(1/tau), through the logarithm: exp(log_sigmoid(z + bias) / tau).
__global__ void gated_decay_kernel(float* z, long long z_stride, const void* bias, int w_dtype, int width, float inv_tau,
                                   long long count) {
  wait_for_prior_grids();
  let_dependents_launch();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const long long t = i / width;
  const int c = static_cast<int>(i - t * width);
  float* at = z + t * z_stride + c;
  *at = expf(log_sigmoid_f(*at + load_scale(bias, w_dtype, c)) * inv_tau);
}

template <typename T, int MODE, int PASS>
__global__ void __launch_bounds__(512) decayed_state_scan_kernel(const ScanArgs a) {
  wait_for_prior_grids();
  let_dependents_launch();
  extern __shared__ __align__(16) float scan_smem[];
  const int D = a.D, V = a.V, nwarps = blockDim.x >> 5, Dp = nwarps * SCAN_ROWS;     // blockDim.x == 2 Dp
  float* a_s = scan_smem;                                   // [SCAN_CHUNK][Dp]
  float* k_s = a_s + SCAN_CHUNK * Dp;                       // [SCAN_CHUNK][Dp]
  float* q_s = k_s + SCAN_CHUNK * Dp;                       // [SCAN_CHUNK][Dp]
  float* v_s = q_s + SCAN_CHUNK * Dp;                       // [SCAN_CHUNK][SCAN_COLS]
  float* o_s = v_s + SCAN_CHUNK * SCAN_COLS;                // [SCAN_CHUNK][nwarps][SCAN_COLS]
  float* step_s = o_s + SCAN_CHUNK * nwarps * SCAN_COLS;    // [2][SCAN_CHUNK]: state space: step sizes, decays
  const int v0 = blockIdx.x * SCAN_COLS, h = blockIdx.y;
  const int row = blockIdx.z / a.segs, seg = blockIdx.z - row * a.segs;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slot = a.slots[row];
  if (slot < 0 || slot >= a.num_slots) {
    if (tid == 0 && seg == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, slot, row);
    return;
  }
  int t0 = a.row_q_start[row], n = a.row_q_len[row];
  if (PASS == SCAN_PASS_SHORT && n >= a.below) return;
  bool last = true;
  if (a.seg_len > 0) {
    const int begin = seg * a.seg_len;
    last = begin + a.seg_len >= n;
    n = min(n, begin + a.seg_len) - begin;
    t0 += begin;
    if (n <= 0 || (PASS == SCAN_PASS_LOCAL && last)) return;      // nothing here, or nobody needs what it adds
  }
  const int col = v0 + lane, col2 = col + 32, d0 = warp * SCAN_ROWS;
  float* state = a.state + static_cast<long long>(slot) * a.slot_stride + static_cast<long long>(h) * D * V;
  const long long piece = static_cast<long long>(row) * a.segs + seg;
  // Where this piece starts from: zero, the state the carry left for it, or the request's slot.
  const float* from = PASS == SCAN_PASS_LOCAL ? nullptr
                      : (a.seg_len > 0 && seg > 0) ? a.ws_state + ((piece - 1) * a.H + h) * D * V : state;
  float S[SCAN_ROWS], S2[SCAN_ROWS], decay_product[PASS == SCAN_PASS_LOCAL ? SCAN_ROWS : 1];
#pragma unroll
  for (int d = 0; d < SCAN_ROWS; ++d) {
    S[d] = (from != nullptr && d0 + d < D && col < V) ? from[static_cast<long long>(d0 + d) * V + col] : 0.0f;
    S2[d] = (from != nullptr && d0 + d < D && col2 < V) ? from[static_cast<long long>(d0 + d) * V + col2] : 0.0f;
    if (PASS == SCAN_PASS_LOCAL) decay_product[d] = 1.0f;
  }

  const T* qp = static_cast<const T*>(a.q);
  const T* kp = static_cast<const T*>(a.k);
  const T* vp = static_cast<const T*>(a.v);
  const int qk_col = (MODE == SCAN_STATE_SPACE ? h / a.heads_per_group : h) * D;
  float head_decay = 0.0f, head_dt_bias = 0.0f, head_skip = 0.0f;
  if (MODE == SCAN_FIXED) head_decay = a.decay[h];
  if (MODE == SCAN_STATE_SPACE) {
    head_decay = -expf(load_scale(a.a_log, a.w_dtype, h));
    head_dt_bias = load_scale(a.dt_bias, a.w_dtype, h);
    head_skip = load_scale(a.skip, a.w_dtype, h);
  }

  // What this thread fetches ahead: one key channel of every second token of the chunk (the threads'
  // two halves take the even and the odd tokens), a share of the values, and (state space, the first
  // SCAN_CHUNK threads) a token's raw step size.
  constexpr int PER = SCAN_CHUNK / 2;
  const int my_d = tid < Dp ? tid : tid - Dp, my_t = tid < Dp ? 0 : 1;
  // Keys, queries, values and step sizes stay in their own type until they are stored to shared memory:
  // a conversion at the load would make the thread wait for the load there and then.
  float pa[PER];
  T pk[PER], pq[PER], pv[SCAN_V_REGS], pdt = from_float<T>(0.0f);
  auto fetch = [&](int c0) {
    const int nc = min(SCAN_CHUNK, n - c0);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int t = 2 * j + my_t;
      pa[j] = 0.0f;
      pk[j] = pq[j] = from_float<T>(0.0f);
      if (t < nc && my_d < D) {
        const long long tok = t0 + c0 + t;
        pk[j] = kp[tok * a.k_stride + qk_col + my_d];
        pq[j] = qp[tok * a.q_stride + qk_col + my_d];
        if (MODE == SCAN_GATED) pa[j] = a.z[tok * a.z_stride + h * D + my_d];
      }
    }
#pragma unroll
    for (int j = 0; j < SCAN_V_REGS; ++j) {
      const int e = tid + j * static_cast<int>(blockDim.x);
      pv[j] = from_float<T>(0.0f);
      if (e < SCAN_CHUNK * SCAN_COLS) {
        const int t = e / SCAN_COLS, c = v0 + (e - t * SCAN_COLS);
        if (t < nc && c < V) pv[j] = vp[static_cast<long long>(t0 + c0 + t) * a.v_stride + h * V + c];
      }
    }
    if (MODE == SCAN_STATE_SPACE && tid < nc)
      pdt = static_cast<const T*>(a.dt)[static_cast<long long>(t0 + c0 + tid) * a.dt_stride + h];
  };

  if (n > 0) fetch(0);
  for (int c0 = 0; c0 < n; c0 += SCAN_CHUNK) {
    const int nc = min(SCAN_CHUNK, n - c0);
    __syncthreads();                      // the chunk before is no longer read
    if (MODE == SCAN_STATE_SPACE) {
      if (tid < nc) {
        const float dt = softplus_f(to_float(pdt) + head_dt_bias);
        step_s[tid] = dt;
        step_s[SCAN_CHUNK + tid] = expf(head_decay * dt);
      }
      __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int t = 2 * j + my_t, e = t * Dp + my_d;
      if (MODE == SCAN_GATED) {
        a_s[e] = pa[j];
        k_s[e] = to_float(pk[j]);
        q_s[e] = to_float(pq[j]) * a.q_scale;
      } else if (MODE == SCAN_FIXED) {
        k_s[e] = to_float(pk[j]);
        q_s[e] = to_float(pq[j]) * a.q_scale;
      } else {
        a_s[e] = t < nc ? step_s[SCAN_CHUNK + t] : 0.0f;
        k_s[e] = t < nc ? to_float(pk[j]) * step_s[t] : 0.0f;
        q_s[e] = to_float(pq[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < SCAN_V_REGS; ++j) {
      const int e = tid + j * static_cast<int>(blockDim.x);
      if (e < SCAN_CHUNK * SCAN_COLS) v_s[e] = to_float(pv[j]);
    }
    __syncthreads();
    if (c0 + SCAN_CHUNK < n) fetch(c0 + SCAN_CHUNK);      // lands while this chunk runs
    for (int t = 0; t < nc; ++t) {
      const float vt = v_s[t * SCAN_COLS + lane], vt2 = v_s[t * SCAN_COLS + 32 + lane];
      const float4* at = reinterpret_cast<const float4*>(a_s + t * Dp + d0);
      const float4* kt = reinterpret_cast<const float4*>(k_s + t * Dp + d0);
      const float4* qt = reinterpret_cast<const float4*>(q_s + t * Dp + d0);
      float o0 = 0.0f, o1 = 0.0f, o2 = 0.0f, o3 = 0.0f, p0 = 0.0f, p1 = 0.0f, p2 = 0.0f, p3 = 0.0f;
#pragma unroll
      for (int d4 = 0; d4 < SCAN_ROWS / 4; ++d4) {
        const float4 av = MODE == SCAN_FIXED ? make_float4(head_decay, head_decay, head_decay, head_decay) : at[d4];
        const float4 kv = kt[d4], qv = qt[d4];
        const int d = 4 * d4;
        S[d] = fmaf(av.x, S[d], kv.x * vt);
        S[d + 1] = fmaf(av.y, S[d + 1], kv.y * vt);
        S[d + 2] = fmaf(av.z, S[d + 2], kv.z * vt);
        S[d + 3] = fmaf(av.w, S[d + 3], kv.w * vt);
        S2[d] = fmaf(av.x, S2[d], kv.x * vt2);
        S2[d + 1] = fmaf(av.y, S2[d + 1], kv.y * vt2);
        S2[d + 2] = fmaf(av.z, S2[d + 2], kv.z * vt2);
        S2[d + 3] = fmaf(av.w, S2[d + 3], kv.w * vt2);
        if (PASS == SCAN_PASS_LOCAL) {
          decay_product[d] *= av.x;
          decay_product[d + 1] *= av.y;
          decay_product[d + 2] *= av.z;
          decay_product[d + 3] *= av.w;
        } else {
          o0 = fmaf(S[d], qv.x, o0);
          o1 = fmaf(S[d + 1], qv.y, o1);
          o2 = fmaf(S[d + 2], qv.z, o2);
          o3 = fmaf(S[d + 3], qv.w, o3);
          p0 = fmaf(S2[d], qv.x, p0);
          p1 = fmaf(S2[d + 1], qv.y, p1);
          p2 = fmaf(S2[d + 2], qv.z, p2);
          p3 = fmaf(S2[d + 3], qv.w, p3);
        }
      }
      if (PASS != SCAN_PASS_LOCAL) {
        o_s[(t * nwarps + warp) * SCAN_COLS + lane] = (o0 + o1) + (o2 + o3);
        o_s[(t * nwarps + warp) * SCAN_COLS + 32 + lane] = (p0 + p1) + (p2 + p3);
      }
    }
    if (PASS == SCAN_PASS_LOCAL) continue;
    __syncthreads();
    for (int e = tid; e < nc * SCAN_COLS; e += blockDim.x) {
      const int t = e / SCAN_COLS, l = e - t * SCAN_COLS, c = v0 + l;
      if (c >= V) continue;
      float o = 0.0f;
      for (int w = 0; w < nwarps; ++w) o += o_s[(t * nwarps + w) * SCAN_COLS + l];
      if (MODE == SCAN_STATE_SPACE) o = fmaf(head_skip, v_s[t * SCAN_COLS + l], o);
      a.out[static_cast<long long>(t0 + c0 + t) * a.H * V + h * V + c] = o;
    }
  }
  if (PASS == SCAN_PASS_LOCAL) {
    float* to = a.ws_state + (piece * a.H + h) * D * V;
#pragma unroll
    for (int d = 0; d < SCAN_ROWS; ++d) {
      if (d0 + d < D && col < V) to[static_cast<long long>(d0 + d) * V + col] = S[d];
      if (d0 + d < D && col2 < V) to[static_cast<long long>(d0 + d) * V + col2] = S2[d];
      if (d0 + d < D && blockIdx.x == 0 && lane == 0) a.ws_decay[(piece * a.H + h) * D + d0 + d] = decay_product[d];
    }
  } else if (a.write_state && last) {
#pragma unroll
    for (int d = 0; d < SCAN_ROWS; ++d) {
      if (d0 + d < D && col < V) state[static_cast<long long>(d0 + d) * V + col] = S[d];
      if (d0 + d < D && col2 < V) state[static_cast<long long>(d0 + d) * V + col2] = S2[d];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// From a fused projection (float32 rows: q heads, then k heads) to rotated queries and keys: value i of the first
// `rot_dims` values of a head turns with value i + rot_dims / 2 by position * freqs[i] (float32 products); k times
// `k_scale` behind the rotation.  One CTA a token, which works its angles out once for all heads.
__global__ void __launch_bounds__(256) rotate_qk_kernel(float* out, const float* x, long long stride, const float* freqs, int rot_dims,
                                                        float k_scale, const int* positions, int heads, int dim, int vectors) {
  extern __shared__ float2 turn_s[];                        // [rot_dims / 2]: cosine, sine
  const long long t = blockIdx.x;
  const int half = rot_dims / 2, cols = heads * dim;
  const float pos = static_cast<float>(positions[t]);
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float s, c;
    sincosf(pos * freqs[i], &s, &c);
    turn_s[i] = make_float2(c, s);
  }
  __syncthreads();
  const float* src = x + t * stride;
  float* dst = out + t * 2 * cols;
  if (vectors) {                       // four pairs, or four values that pass, a thread and step
    const int turned = half / 4, units = turned + (dim - rot_dims) / 4;
    for (int e = threadIdx.x; e < 2 * heads * units; e += blockDim.x) {
      const int h = e / units, j = e - h * units;
      const float scale = h < heads ? 1.0f : k_scale;
      const float* from = src + h * dim;
      float* to = dst + h * dim;
      if (j < turned) {
        const float4 u = load4(from + 4 * j), v = load4(from + half + 4 * j);
        const float2 a = turn_s[4 * j], b = turn_s[4 * j + 1], c = turn_s[4 * j + 2], d = turn_s[4 * j + 3];
        store4(to + 4 * j, make_float4((u.x * a.x - v.x * a.y) * scale, (u.y * b.x - v.y * b.y) * scale,
                                       (u.z * c.x - v.z * c.y) * scale, (u.w * d.x - v.w * d.y) * scale));
        store4(to + half + 4 * j, make_float4((v.x * a.x + u.x * a.y) * scale, (v.y * b.x + u.y * b.y) * scale,
                                              (v.z * c.x + u.z * c.y) * scale, (v.w * d.x + u.w * d.y) * scale));
      } else {
        const int i = rot_dims + 4 * (j - turned);
        const float4 u = load4(from + i);
        store4(to + i, make_float4(u.x * scale, u.y * scale, u.z * scale, u.w * scale));
      }
    }
    return;
  }
  for (int e = threadIdx.x; e < 2 * cols; e += blockDim.x) {
    const int i = e % dim;
    float y = src[e];
    if (i < rot_dims) {
      const float2 cs = turn_s[i < half ? i : i - half];
      y = i < half ? y * cs.x - src[e + half] * cs.y : y * cs.x + src[e - half] * cs.y;
    }
    dst[e] = e < cols ? y : y * k_scale;
  }
}

// ------------------------------------------------------------------------------------------------
// RMS norm over equal groups of a float32 row with a SiLU gate: y = unit_rms(o * silu(g)) * w when the
// gate comes first, y = unit_rms(o) * w * silu(g) otherwise.  w has `w_len` entries and is used
// periodically (a scale per column, or one scale vector shared by all groups).  One warp per group.
template <typename T, typename G>
__global__ void gated_group_rms_norm_kernel(T* out, const float* o, const G* gate, long long gate_stride, const void* w,
                                            int w_dtype, int w_len, int width, int group, float eps, int gate_first,
                                            int tokens) {
  const int groups = width / group;
  const long long item = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= static_cast<long long>(tokens) * groups) return;
  const int lane = threadIdx.x & 31;
  const long long t = item / groups;
  const int c0 = static_cast<int>(item - t * groups) * group;
  float ss = 0.0f;
  for (int i = lane; i < group; i += 32) {
    float val = o[t * width + c0 + i];
    if (gate_first) val *= silu_f(to_float(gate[t * gate_stride + c0 + i]));
    ss = fmaf(val, val, ss);
  }
  const float r = 1.0f / sqrtf(warp_sum(ss) / static_cast<float>(group) + eps);
  for (int i = lane; i < group; i += 32) {
    const float g = silu_f(to_float(gate[t * gate_stride + c0 + i]));
    float val = o[t * width + c0 + i];
    if (gate_first) val *= g;
    val = val * r * load_scale(w, w_dtype, (c0 + i) % w_len);
    if (!gate_first) val *= g;
    out[t * width + c0 + i] = from_float<T>(val);
  }
}

// The same for groups of up to GN_VEC_MAX columns that are a multiple of four, with aligned rows: o and the gate are
// read once, all loads before the first use, and stay in registers.  A group is LANES lanes' of a warp, eight values each and
// more, up to 512 columns, and a CTA's of four warps beyond: what a group costs besides its values (where it lies, the sum
// over its lanes, the root) is issued once for all the groups of a warp.  Bound by the instructions of the activation (a
// warp a group: 79 % of all issue slots).  2048 tokens of 32 groups of 128 in bfloat16 12.8 us as a warp a group, now 10.7
// (its bytes: 9 us); 2048 tokens of 32 groups of 64 24.6 us (with a float32 out) and 10.1; 2125 tokens of two groups of 1024
// 11.4 and 11.3 us.
constexpr int GN_WARPS = 4;
constexpr int GN_VEC_ITEMS = 4;
constexpr int GN_VEC_MAX = GN_WARPS * 32 * GN_VEC_ITEMS * 4;

template <typename T, typename G, int LANES, int ITEMS>      // LANES: of a group
__global__ void __launch_bounds__(32 * GN_WARPS) gated_group_rms_norm_vec_kernel(T* out, const float* o, const G* gate, long long gate_stride,
                                                const float* w, int w_len, int width, int group, float eps,
                                                int gate_first, unsigned items) {
  wait_for_prior_grids();
  let_dependents_launch();
  __shared__ float part[GN_WARPS];
  constexpr int PER_CTA = 32 * GN_WARPS / LANES;
  const unsigned groups = width / group, item = blockIdx.x * static_cast<unsigned>(PER_CTA) + threadIdx.x / LANES;
  const int lane = threadIdx.x % LANES, nv = item < items ? group / 4 : 0;
  const unsigned t = item / groups;
  const int c0 = static_cast<int>(item - t * groups) * group;
  const float* o_row = o + static_cast<long long>(t) * width + c0;
  const G* gate_row = gate + t * gate_stride + c0;
  float4 val[ITEMS], g[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = lane + LANES * j;
    val[j] = g[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < nv) {
      val[j] = load4(o_row + 4 * i);
      g[j] = load4(gate_row + 4 * i);
    }
  }
  float ss = 0.0f;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    g[j] = make_float4(silu_f(g[j].x), silu_f(g[j].y), silu_f(g[j].z), silu_f(g[j].w));
    if (gate_first) val[j] = make_float4(val[j].x * g[j].x, val[j].y * g[j].y, val[j].z * g[j].z, val[j].w * g[j].w);
    ss += (val[j].x * val[j].x + val[j].y * val[j].y) + (val[j].z * val[j].z + val[j].w * val[j].w);
  }
#pragma unroll
  for (int d = (LANES < 32 ? LANES : 32) / 2; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  if (LANES > 32) {
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = (part[0] + part[1]) + (part[2] + part[3]);
  }
  const float r = 1.0f / sqrtf(ss / static_cast<float>(group) + eps);
  const int w0 = c0 < w_len ? c0 : c0 % w_len;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = lane + LANES * j;
    if (i < nv) {
      const int at = w0 + 4 * i;
      const float4 wv = load4(w + (at < w_len ? at : at % w_len));
      float4 y = make_float4(val[j].x * r * wv.x, val[j].y * r * wv.y, val[j].z * r * wv.z, val[j].w * r * wv.w);
      if (!gate_first) y = make_float4(y.x * g[j].x, y.y * g[j].y, y.z * g[j].z, y.w * g[j].w);
      store4(out + static_cast<long long>(t) * width + c0 + 4 * i, y);
    }
  }
}

template <typename T, typename G>
void gated_group_rms_norm_vec(T* out, const float* o, const G* gate, long long gate_stride, const float* w, int w_len, int width,
                              int group, float eps, int gate_first, unsigned items, cudaStream_t s) {
#define ZB_GN(LANES, ITEMS)                                                                                                  \
  launch_dependent(gated_group_rms_norm_vec_kernel<T, G, LANES, ITEMS>,                                                       \
      dim3((items - 1) / (32 * GN_WARPS / LANES) + 1), dim3(32 * GN_WARPS), 0, s, false, out, o, gate, gate_stride, w, w_len,    \
      width, group, eps, gate_first, items)
  // Few groups, which leave SMs idle, are a warp each: 12 tokens of 32 groups of 128 take 2.3 us, two a warp 2.7.
  if (group <= 128 && items < 4 * 148 * GN_WARPS) ZB_GN(32, 1);
  else if (group <= 64) ZB_GN(8, 2);
  else if (group <= 128) ZB_GN(16, 2);
  else if (group <= 256) ZB_GN(32, 2);
  else if (group <= 512) ZB_GN(32, 4);
  else if (group <= 1024) ZB_GN(128, 2);
  else ZB_GN(128, GN_VEC_ITEMS);
#undef ZB_GN
}

// out = sa * (a + bias) + sb * b, float32 arithmetic, one rounding behind that of a + bias; a and b may be float32 whatever out
// is; bias [width], or null.
template <typename IN, typename T>
__global__ void scaled_sum_kernel(T* out, const IN* a, const IN* b, const float* bias, int width, float sa, float sb, long long n) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float x = to_float(a[i]);
  if (bias != nullptr) x += bias[i % width];
  out[i] = from_float<T>(fmaf(sa, x, sb * to_float(b[i])));
}

// The same eight values a thread, all four loads before the first use, where the three rows are whole aligned pieces of
// four values: 35 MB read and 9 MB written (2125 x 2048) in 6.2 us instead of 15.0, which one value a thread took.  A bias of
// the first summand, added here, saves the pass over that summand which a kernel of its own takes
// (the two one behind the other 11.4 us, now 7.5).
template <typename IN, typename T>
__global__ void __launch_bounds__(256) scaled_sum_vec_kernel(T* out, const IN* a, const IN* b, const float* bias, int width, float sa,
                                                             float sb, long long pieces) {
  wait_for_prior_grids();
  let_dependents_launch();
  const long long i = static_cast<long long>(blockIdx.x) * 512 + threadIdx.x;
  float4 x[2], y[2], c[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (i + 256 * j < pieces) {
      x[j] = load4(a + 4 * (i + 256 * j));
      y[j] = load4(b + 4 * (i + 256 * j));
      if (bias != nullptr) c[j] = load4(bias + 4 * ((i + 256 * j) % (width / 4)));
    }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (i + 256 * j < pieces) {
      if (bias != nullptr) x[j] = make_float4(x[j].x + c[j].x, x[j].y + c[j].y, x[j].z + c[j].z, x[j].w + c[j].w);
      store4(out + 4 * (i + 256 * j), make_float4(fmaf(sa, x[j].x, sb * y[j].x), fmaf(sa, x[j].y, sb * y[j].y),
                                                  fmaf(sa, x[j].z, sb * y[j].z), fmaf(sa, x[j].w, sb * y[j].w)));
    }
}

template <typename IN, typename T>
void scaled_sum(T* out, const IN* a, const IN* b, const float* bias, int width, float sa, float sb, long long n, cudaStream_t s) {
  auto aligned = [](const void* p, size_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
  if (n % 4 == 0 && (bias == nullptr || (width % 4 == 0 && aligned(bias, 16))) && aligned(out, 4 * sizeof(T)) &&
      aligned(a, 4 * sizeof(IN)) && aligned(b, 4 * sizeof(IN)))
    launch_dependent(scaled_sum_vec_kernel<IN, T>, dim3(static_cast<unsigned>((n / 4 + 511) / 512)), dim3(256), 0, s, false,
        out, a, b, bias, width, sa, sb, n / 4);
  else
    scaled_sum_kernel<IN, T><<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(out, a, b, bias, width, sa, sb, n);
}

inline int norm_threads(int H) { return H >= 2048 ? 512 : (H >= 512 ? 256 : 128); }

template <typename K>
inline int allow_shared(K kernel, size_t bytes) {
  if (bytes > 227 * 1024) return ERR_UNSUPPORTED;
  if (bytes > 48 * 1024 &&
      cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes))))
    return ERR_CUDA;
  return OK;
}

}  // namespace zb

using namespace zb;

// out [rows, H] (out_dtype) = LN(x [rows, H] (x_dtype)); scale and shift in w_dtype.
ZB_API int zb_layer_norm(void* out, const void* x, const void* w, const void* b, int w_dtype, float eps, int rows,
                         int H, int x_dtype, int out_dtype, void* stream) {
  if (rows < 0 || H <= 0) return ERR_BAD_ARGUMENT;
  if (rows == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if (ln_vectors(H, w_dtype, {out, x, w, b})) {
    const float* wf = static_cast<const float*>(w);
    const float* bf = static_cast<const float*>(b);
    using bf16 = __nv_bfloat16;
#define ZB_LNV(X, T)                                                                                                      \
  {                                                                                                                       \
    if (H <= 2 * LN_VEC_THREADS * 4)                                                                                      \
      launch_dependent(layer_norm_vec_kernel<X, T, 2>, dim3(rows), dim3(LN_VEC_THREADS), 0, s, false, static_cast<T*>(out),   \
          static_cast<const X*>(x), wf, bf, eps, H);                                                                          \
    else                                                                                                                  \
      launch_dependent(layer_norm_vec_kernel<X, T, LN_VEC_ITEMS>, dim3(rows), dim3(LN_VEC_THREADS), 0, s, false,              \
          static_cast<T*>(out), static_cast<const X*>(x), wf, bf, eps, H);                                                    \
  }
    if (x_dtype == DTYPE_F32 && out_dtype == DTYPE_F32) ZB_LNV(float, float)
    else if (x_dtype == DTYPE_F32) ZB_LNV(float, bf16)
    else if (out_dtype == DTYPE_F32) ZB_LNV(bf16, float)
    else ZB_LNV(bf16, bf16)
#undef ZB_LNV
    return launch_result();
  }
  const size_t smem = static_cast<size_t>(H) * sizeof(float);
  const int threads = norm_threads(H);
#define ZB_LN(X, T)                                                                                    \
  {                                                                                                    \
    auto kernel = layer_norm_kernel<X, T>;                                                             \
    if (int rc = allow_shared(kernel, smem)) return rc;                                                \
    kernel<<<rows, threads, smem, s>>>(static_cast<T*>(out), static_cast<const X*>(x), w, b, w_dtype, eps, H); \
  }
  if (x_dtype == DTYPE_F32 && out_dtype == DTYPE_F32) ZB_LN(float, float)
  else if (x_dtype == DTYPE_F32) ZB_LN(float, __nv_bfloat16)
  else if (out_dtype == DTYPE_F32) ZB_LN(__nv_bfloat16, float)
  else ZB_LN(__nv_bfloat16, __nv_bfloat16)
#undef ZB_LN
  return launch_result();
}

template <bool RMS>
static int residual_norm_launch(float* residual, const void* delta, const void* w1, const void* b1, float mult,
                                  void* out, const void* w2, const void* b2, int w_dtype, float eps1, float eps2,
                                  int rows, int H, int dtype, void* stream) {
  if (rows < 0 || H <= 0) return ERR_BAD_ARGUMENT;
  if (rows == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if (ln_vectors(H, w_dtype, {residual, delta, out, w1, b1, w2, b2})) {
    const float* f1 = static_cast<const float*>(w1);
    const float* g1 = static_cast<const float*>(b1);
    const float* f2 = static_cast<const float*>(w2);
    const float* g2 = static_cast<const float*>(b2);
#define ZB_RN(T, ITEMS)                                                                                       \
  launch_dependent(residual_layer_norm_vec_kernel<T, RMS, ITEMS>, dim3(rows), dim3(LN_VEC_THREADS), 0, s, false, residual,    \
      static_cast<const T*>(delta), f1, g1, mult, static_cast<T*>(out), f2, g2, eps1, eps2, H)
    const bool two = H <= 2 * LN_VEC_THREADS * 4;
    if (dtype == DTYPE_F32) { if (two) ZB_RN(float, 2); else ZB_RN(float, LN_VEC_ITEMS); }
    else { if (two) ZB_RN(__nv_bfloat16, 2); else ZB_RN(__nv_bfloat16, LN_VEC_ITEMS); }
#undef ZB_RN
    return launch_result();
  }
  const size_t smem = static_cast<size_t>(H) * sizeof(float);
  const int threads = norm_threads(H);
  if (dtype == DTYPE_F32) {
    auto kernel = residual_layer_norm_kernel<float, RMS>;
    if (int rc = allow_shared(kernel, smem)) return rc;
    kernel<<<rows, threads, smem, s>>>(residual, static_cast<const float*>(delta), w1, b1, mult,
                                       static_cast<float*>(out), w2, b2, w_dtype, eps1, eps2, H);
  } else {
    auto kernel = residual_layer_norm_kernel<__nv_bfloat16, RMS>;
    if (int rc = allow_shared(kernel, smem)) return rc;
    kernel<<<rows, threads, smem, s>>>(residual, static_cast<const __nv_bfloat16*>(delta), w1, b1, mult,
                                       static_cast<__nv_bfloat16*>(out), w2, b2, w_dtype, eps1, eps2, H);
  }
  return launch_result();
}

ZB_API int zb_residual_layer_norm(float* residual, const void* delta, const void* w1, const void* b1, float mult,
                                  void* out, const void* w2, const void* b2, int w_dtype, float eps1, float eps2,
                                  int rows, int H, int dtype, void* stream) {
  return residual_norm_launch<false>(residual, delta, w1, b1, mult, out, w2, b2, w_dtype, eps1, eps2, rows, H, dtype, stream);
}

// residual += mult * RMSnorm(delta; w1); then out = RMSnorm(residual; w2), or with a null w2 the sum in delta's type.
ZB_API int zb_residual_rms_norm(float* residual, const void* delta, const void* w1, float mult, void* out,
                                const void* w2, int w_dtype, float eps1, float eps2, int rows, int H, int dtype,
                                void* stream) {
  return residual_norm_launch<true>(residual, delta, w1, nullptr, mult, out, w2, nullptr, w_dtype, eps1, eps2, rows, H, dtype, stream);
}

ZB_API int zb_embedding_f32(float* out, void* rounded, const void* table, const int* ids, float scale, int tokens,
                            int H, int V, int dtype, int* status, void* stream) {
  if (tokens < 0 || H <= 0 || V <= 0) return ERR_BAD_ARGUMENT;
  if (tokens == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if (dtype == DTYPE_F32)
    embedding_f32(out, static_cast<float*>(rounded), static_cast<const float*>(table), ids, scale, tokens, H, V, status, s);
  else
    embedding_f32(out, static_cast<__nv_bfloat16*>(rounded), static_cast<const __nv_bfloat16*>(table), ids, scale, tokens, H, V,
                  status, s);
  return launch_result();
}

ZB_API int zb_causal_conv_silu(void* out, const void* x, long long x_stride, float* state, long long slot_stride,
                               const int* slots, const int* row_q_start, const int* row_q_len, const int* token_row,
                               int tokens, int rows, const void* w,
                               const void* bias, int w_dtype, int C, int taps, int num_slots, int write_state, int dtype,
                               int* status, void* stream) {
  if (rows < 0 || C <= 0 || taps <= 0) return ERR_BAD_ARGUMENT;
  if (taps > CONV_MAX_TAPS) return ERR_UNSUPPORTED;
  if (rows == 0) return OK;
  ConvArgs a;
  a.out = out; a.x = x; a.x_stride = x_stride; a.state = state; a.slot_stride = slot_stride; a.slots = slots;
  a.row_q_start = row_q_start; a.row_q_len = row_q_len; a.w = w; a.bias = bias; a.w_dtype = w_dtype; a.C = C;
  a.taps = taps; a.num_slots = num_slots; a.write_state = write_state; a.status = status;
  auto s = static_cast<cudaStream_t>(stream);
  if (tokens <= 0) return OK;
  const dim3 grid((tokens + CONV_TOKENS - 1) / CONV_TOKENS, (C + 127) / 128), per_row((C + 127) / 128, rows);
  // Runs pay where requests bring several tokens (a step of single tokens has nothing to share) and from half a million values
  // on: below, runs of CONV_RUN tokens are too few CTAs.  4096 channels, 64 tokens: 8.2 us as runs, 6.2 a value at a time; 128:
  // 8.4 and 8.5; 256: 8.9 and 12.3; 2560 channels, 128 tokens: 8.1 and 7.2; 256: 8.4 and 9.4.  The sums are the same.
  auto aligned = [&](int vec) {
    const size_t bytes = vec * (dtype == DTYPE_F32 ? 4 : 2);
    return C % vec == 0 && x_stride % vec == 0 && w_dtype == DTYPE_F32 && reinterpret_cast<uintptr_t>(x) % bytes == 0 &&
           reinterpret_cast<uintptr_t>(out) % bytes == 0;
  };
  const bool runs = tokens >= 4 * rows && static_cast<long long>(tokens) * C >= 1 << 19 && aligned(2);
  if (dtype == DTYPE_F32) {
    if (runs) conv_run_launch<float>(a, token_row, tokens, aligned(4), s);
    else launch_dependent(causal_conv_silu_kernel<float>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
    if (write_state && taps > 1) launch_dependent(conv_state_update_kernel<float>, dim3(per_row), dim3(128), 0, s, false, a);
  } else {
    if (runs) conv_run_launch<__nv_bfloat16>(a, token_row, tokens, aligned(4), s);
    else launch_dependent(causal_conv_silu_kernel<__nv_bfloat16>, dim3(grid), dim3(128), 0, s, false, a, token_row, tokens);
    if (write_state && taps > 1) launch_dependent(conv_state_update_kernel<__nv_bfloat16>, dim3(per_row), dim3(128), 0, s, false, a);
  }
  return launch_result();
}

// The most key channels a head of the recurrence may have.
ZB_API int zb_state_scan_max_channels() { return 16 * SCAN_ROWS; }

// `z` (gated mode): decay logits [tokens, H * D] float32, overwritten with the decays.
ZB_API int zb_decayed_state_scan(float* out, const void* q, long long q_stride, const void* k, long long k_stride,
                                 const void* v, long long v_stride, float* z, long long z_stride,
                                 const void* z_bias, const void* dt, long long dt_stride, const void* dt_bias,
                                 const void* a_log, const void* skip, const float* decay, int w_dtype, float* state,
                                 long long slot_stride,
                                 const int* slots, const int* row_q_start, const int* row_q_len, int rows, int tokens,
                                 int H, int D, int V, int heads_per_group, int num_slots, int write_state,
                                 int below, float q_scale, float inv_tau, int mode, int dtype, int seg_len, float* ws_state,
                                 float* ws_decay, int* status, void* stream) {
  if (rows < 0 || tokens < 0 || H <= 0 || D <= 0 || V <= 0 || heads_per_group <= 0 || seg_len < 0 ||
      (seg_len > 0 && (ws_state == nullptr || ws_decay == nullptr)))
    return ERR_BAD_ARGUMENT;
  if (D > 16 * SCAN_ROWS) return ERR_UNSUPPORTED;
  if (below < 0 || (below > 0 && (mode != SCAN_STATE_SPACE || seg_len > 0))) return ERR_BAD_ARGUMENT;
  if (mode < SCAN_GATED || mode > SCAN_FIXED || (mode == SCAN_FIXED && decay == nullptr)) return ERR_BAD_ARGUMENT;
  if (rows == 0 || tokens == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if (mode == SCAN_GATED) {
    const long long count = static_cast<long long>(tokens) * H * D;
    launch_dependent(gated_decay_kernel, dim3(static_cast<unsigned>((count + 255) / 256)), dim3(256), 0, s, false, z,
        z_stride, z_bias, w_dtype, H * D, inv_tau, count);
  }
  ScanArgs a;
  a.q = q; a.q_stride = q_stride; a.k = k; a.k_stride = k_stride; a.v = v; a.v_stride = v_stride;
  a.z = z; a.z_stride = z_stride; a.dt = dt; a.dt_stride = dt_stride; a.dt_bias = dt_bias;
  a.decay = decay;
  a.a_log = a_log; a.skip = skip; a.w_dtype = w_dtype; a.state = state; a.slot_stride = slot_stride; a.out = out;
  a.slots = slots; a.row_q_start = row_q_start; a.row_q_len = row_q_len; a.H = H; a.D = D; a.V = V;
  a.heads_per_group = heads_per_group; a.num_slots = num_slots; a.write_state = write_state; a.q_scale = q_scale;
  a.below = below; a.status = status;
  a.seg_len = seg_len; a.segs = seg_len > 0 ? (tokens + seg_len - 1) / seg_len : 1;
  a.ws_state = ws_state; a.ws_decay = ws_decay;
  if (static_cast<long long>(rows) * a.segs > 65535) return ERR_UNSUPPORTED;
  const int warps = std::max(2, (D + SCAN_ROWS - 1) / SCAN_ROWS);
  const size_t smem = sizeof(float) * (3 * SCAN_CHUNK * warps * SCAN_ROWS + SCAN_CHUNK * SCAN_COLS +
                                       SCAN_CHUNK * warps * SCAN_COLS + 2 * SCAN_CHUNK);
  const dim3 grid((V + SCAN_COLS - 1) / SCAN_COLS, H, rows * a.segs);
#define ZB_SCAN(T, MODE)                                                                                       \
  {                                                                                                            \
    auto kernel = MODE == SCAN_STATE_SPACE && below > 0                                                        \
                      ? decayed_state_scan_kernel<T, MODE, MODE == SCAN_STATE_SPACE ? SCAN_PASS_SHORT : SCAN_PASS_OUTPUT> \
                      : decayed_state_scan_kernel<T, MODE, SCAN_PASS_OUTPUT>;                                  \
    if (int rc = allow_shared(kernel, smem)) return rc;                                                        \
    if (seg_len > 0) {                                                                                         \
      auto local = decayed_state_scan_kernel<T, MODE, SCAN_PASS_LOCAL>;                                        \
      if (int rc = allow_shared(local, smem)) return rc;                                                       \
      local<<<grid, warps * 32, smem, s>>>(a);                                                                 \
      const long long per = static_cast<long long>(H) * D * V;                                                 \
      scan_carry_kernel<<<dim3(static_cast<unsigned>((per + 255) / 256), rows), 256, 0, s>>>(                  \
          ws_state, ws_decay, state, slot_stride, slots, row_q_len, a.segs, seg_len, H, D, V, num_slots);      \
    }                                                                                                          \
    launch_dependent(kernel, grid, dim3(warps * 32), smem, s, false, a);                                       \
  }
  if (dtype == DTYPE_F32) {
    if (mode == SCAN_GATED) ZB_SCAN(float, SCAN_GATED)
    else if (mode == SCAN_FIXED) ZB_SCAN(float, SCAN_FIXED)
    else ZB_SCAN(float, SCAN_STATE_SPACE)
  } else {
    if (mode == SCAN_GATED) ZB_SCAN(__nv_bfloat16, SCAN_GATED)
    else if (mode == SCAN_FIXED) ZB_SCAN(__nv_bfloat16, SCAN_FIXED)
    else ZB_SCAN(__nv_bfloat16, SCAN_STATE_SPACE)
  }
#undef ZB_SCAN
  return launch_result();
}

// out [T, 2 heads * dim] float32 = the rotated q and k heads of x's rows (float32, `stride` apart), k times k_scale.
ZB_API int zb_rotate_qk(float* out, const float* x, long long stride, const float* freqs, int rot_dims, float k_scale,
                        const int* positions, int tokens, int heads, int dim, void* stream) {
  if (tokens < 0 || heads <= 0 || dim <= 0 || rot_dims < 0 || rot_dims > dim || rot_dims % 2 != 0 || stride < 2LL * heads * dim ||
      (rot_dims > 0 && freqs == nullptr) || rot_dims > 4096)
    return ERR_BAD_ARGUMENT;
  if (tokens == 0) return OK;
  const int vectors = rot_dims % 8 == 0 && dim % 4 == 0 && stride % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                      reinterpret_cast<uintptr_t>(out) % 16 == 0;
  rotate_qk_kernel<<<tokens, 256, sizeof(float2) * (rot_dims / 2 + 1), static_cast<cudaStream_t>(stream)>>>(
      out, x, stride, freqs, rot_dims, k_scale, positions, heads, dim, vectors);
  return launch_result();
}

ZB_API int zb_gated_group_rms_norm(void* out, const float* o, const void* gate, long long gate_stride, const void* w,
                                   int w_dtype, int w_len, int tokens, int width, int group, float eps, int gate_first,
                                   int gate_dtype, int dtype, void* stream) {
  if (tokens < 0 || width <= 0 || group <= 0 || width % group != 0 || w_len <= 0 || (dtype == DTYPE_F32 && gate_dtype != DTYPE_F32))
    return ERR_BAD_ARGUMENT;
  if (tokens == 0) return OK;
  const long long items = static_cast<long long>(tokens) * (width / group);
  const int warps = 4;
  const unsigned blocks = static_cast<unsigned>((items + warps - 1) / warps);
  auto s = static_cast<cudaStream_t>(stream);
  const int elem = dtype == DTYPE_F32 ? 4 : 2, gate_elem = gate_dtype == DTYPE_F32 ? 4 : 2;
  if (items <= INT_MAX && group % 4 == 0 && group <= GN_VEC_MAX && w_len % 4 == 0 && w_dtype == DTYPE_F32 && gate_stride % 4 == 0 &&
      reinterpret_cast<uintptr_t>(gate) % (4 * gate_elem) == 0 && reinterpret_cast<uintptr_t>(o) % 16 == 0 &&
      reinterpret_cast<uintptr_t>(out) % (4 * elem) == 0 && reinterpret_cast<uintptr_t>(w) % 16 == 0) {
    const float* wf = static_cast<const float*>(w);
    using bf16 = __nv_bfloat16;
    if (dtype == DTYPE_F32)
      gated_group_rms_norm_vec(static_cast<float*>(out), o, static_cast<const float*>(gate), gate_stride, wf, w_len, width, group,
                               eps, gate_first, static_cast<unsigned>(items), s);
    else if (gate_dtype == DTYPE_F32)
      gated_group_rms_norm_vec(static_cast<bf16*>(out), o, static_cast<const float*>(gate), gate_stride, wf, w_len, width, group,
                               eps, gate_first, static_cast<unsigned>(items), s);
    else
      gated_group_rms_norm_vec(static_cast<bf16*>(out), o, static_cast<const bf16*>(gate), gate_stride, wf, w_len, width, group,
                               eps, gate_first, static_cast<unsigned>(items), s);
    return launch_result();
  }
  if (dtype == DTYPE_F32)
    gated_group_rms_norm_kernel<float, float><<<blocks, warps * 32, 0, s>>>(
        static_cast<float*>(out), o, static_cast<const float*>(gate), gate_stride, w, w_dtype, w_len, width, group, eps,
        gate_first, tokens);
  else if (gate_dtype == DTYPE_F32)
    gated_group_rms_norm_kernel<__nv_bfloat16, float><<<blocks, warps * 32, 0, s>>>(
        static_cast<__nv_bfloat16*>(out), o, static_cast<const float*>(gate), gate_stride, w, w_dtype, w_len, width, group, eps,
        gate_first, tokens);
  else
    gated_group_rms_norm_kernel<__nv_bfloat16, __nv_bfloat16><<<blocks, warps * 32, 0, s>>>(
        static_cast<__nv_bfloat16*>(out), o, static_cast<const __nv_bfloat16*>(gate), gate_stride, w, w_dtype, w_len,
        width, group, eps, gate_first, tokens);
  return launch_result();
}

ZB_API int zb_scaled_sum(void* out, const void* a, const void* b, const float* bias, int width, float sa, float sb, long long n,
                         int in_dtype, int dtype, void* stream) {
  if (n < 0 || (bias != nullptr && (width <= 0 || n % width != 0))) return ERR_BAD_ARGUMENT;
  if (n == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  using bf16 = __nv_bfloat16;
  if (in_dtype == DTYPE_F32 && dtype == DTYPE_F32)
    scaled_sum(static_cast<float*>(out), static_cast<const float*>(a), static_cast<const float*>(b), bias, width, sa, sb, n, s);
  else if (in_dtype == DTYPE_F32)
    scaled_sum(static_cast<bf16*>(out), static_cast<const float*>(a), static_cast<const float*>(b), bias, width, sa, sb, n, s);
  else if (dtype == DTYPE_BF16)
    scaled_sum(static_cast<bf16*>(out), static_cast<const bf16*>(a), static_cast<const bf16*>(b), bias, width, sa, sb, n, s);
  else
    return ERR_BAD_ARGUMENT;
  return launch_result();
}
