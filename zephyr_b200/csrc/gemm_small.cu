// Y[M, N] = X[M, K] * W[N, K]^T for the few rows of a decode step (M <= 64), bfloat16 with float32
// accumulation: a weight streamer.  Every weight is read once, straight from global memory into
// tensor-core fragments by 16-byte loads (no shared-memory staging), so many loads are in flight
// per warp; the activations, a few KB, come from L2 the same way.
//
// The weight rows sit on the 16-row side of m16n8k16 and the tokens on the 8-column side (the
// product is computed as W X^T).  Inside a block of 32 consecutive k, lane t of a quad owns the 8
// consecutive values k = 8t .. 8t+7 of its row: one 16-byte load feeds two tensor-core products.
// The products see k in a permuted order, the same for both operands, so the sum is unchanged.
//
// One CTA owns 16 rows of W (or 32); its warps split K, and for matrices with few rows a cluster of
// up to 8 CTAs splits K further.  A decode step's product is bound by latency before it is by bandwidth: a warp has the loads
// of several blocks of 32 k in flight, whatever is left of its slice: four up to 16 rows, two from 17 to 32 and where a CTA takes
// 32 rows of W; above 32 rows four blocks of W alone, x at its use (with x ahead too, two blocks: 12288 x 4096, 64 rows: 92 us,
// now 47; 6144 x 2048: 29 and 17) (one block after the other, as a loop's remainder, 2048 x
// 6144 with 12 rows took 13.8 us; now 10.1, its bytes 3.8), and the CTAs of a cluster each finish a share of the tile with one
// round of remote reads (one CTA for all, 2048 x 2048: 9.8 us; now 6.1).  4096 x 2048: 10.2 -> 7.9, 12288 x 2048: 14.9 -> 14.1,
// 8192 x 4096, 12 rows: 16.9.  Partial sums meet in (distributed) shared memory and are added in
// a fixed order, so the result does not depend on timing.  ACT takes each sum through GELU's tanh form, a
// squared ReLU, or GELU times a value of the token's row of a table.  With SWIGLU the 16 rows are 8 gate
// rows followed by their 8 up rows, and the epilogue writes silu(gate) * up: the activation costs
// no extra pass over memory (reference: src/layer/mlp.cpp:29-36, src/layer/activation.cu:31-33).
#include <cooperative_groups.h>

#include "common.cuh"
#include "mma.cuh"

namespace zb {

namespace cg = cooperative_groups;

constexpr int ACT_TOKEN_GATE = 3;
constexpr int GS_MAX_MT = 8;      // token tiles of 8: M <= 64
constexpr int GS_MAX_KSPLIT = 8;
constexpr int GS_FETCH_AHEAD_CTAS = 4 * 148;

struct SmallGemmArgs {
  void* y;
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;
  int M, N, K;
  int cut_rows;                        // rows of the weight matrix, which with K say how K is cut: N, or M where the sides have changed
  long long ldx, ldw, ldy;
  long long ldn;                       // between two rows of w's outputs: 1, or what a transposed result takes (ungated, no activation)
  const __nv_bfloat16* token_rows;     // ACT_TOKEN_GATE: gelu(sum) * token_rows[token_ids[token] * token_stride + column]
  long long token_stride;
  const int* token_ids;
  int vocab;
  int* status;
  GateForm gate;      // with the gated epilogue: what becomes of a gate sum and its up sum
};

__device__ __forceinline__ uint4 load16_or_zero(const __nv_bfloat16* p, bool ok) {
  return ok ? *reinterpret_cast<const uint4*>(p) : make_uint4(0, 0, 0, 0);
}

template <typename T> __device__ __forceinline__ void store_out(T* p, float v);
template <> __device__ __forceinline__ void store_out<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void store_out<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

template <int RT, int WARPS, int MT, typename TOut, bool SWIGLU, int ACT>
__global__ void __launch_bounds__(WARPS * 32)
gemm_small_kernel(const SmallGemmArgs a) {
  constexpr bool X_AHEAD = MT <= 4;                 // (eight tiles of tokens ahead leave room for two blocks of W)
  constexpr int U = (RT == 1 && MT <= 2) || !X_AHEAD ? 4 : 2;     // blocks of k in flight
  constexpr int PER_WARP = RT * MT * 16 * 8;        // sums of a warp: [rt][mt][row][token]
  __shared__ float red[WARPS][PER_WARP];
  cg::cluster_group cluster = cg::this_cluster();
  const int ksplit = gridDim.y, krank = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * (16 * RT);

  const int total_blocks = (a.K + 31) / 32;
  const int slices = WARPS * ksplit, slice = krank * WARPS + warp;
  const int b_begin = static_cast<int>(static_cast<long long>(total_blocks) * slice / slices);
  const int b_end = static_cast<int>(static_cast<long long>(total_blocks) * (slice + 1) / slices);

  bool w_ok[2 * RT];
  const __nv_bfloat16* w_row[2 * RT];
#pragma unroll
  for (int r = 0; r < 2 * RT; ++r) {
    w_ok[r] = n0 + g + 8 * r < a.N;
    w_row[r] = a.w + static_cast<size_t>(w_ok[r] ? n0 + g + 8 * r : 0) * a.ldw + 8 * t;
  }
  const __nv_bfloat16* x_row[MT];
  bool x_ok[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    x_ok[mt] = mt * 8 + g < a.M;
    x_row[mt] = a.x + static_cast<size_t>(x_ok[mt] ? mt * 8 + g : 0) * a.ldx + 8 * t;
  }

  // While the kernel before this one still runs: the warp's rows of W are asked for as far as L2 (a fetch into the coherent cache
  // only: what the loads below bring is right whoever wrote it last).  CTAs behind the first round of them start when their
  // weights would be asked for anyway.  (A pass of 25 steps of 12 rows, 290 of these products and as many short kernels: 6.06 -> 5.86 ms
  // with all of them launched as dependents.)
  if (blockIdx.x * ksplit < GS_FETCH_AHEAD_CTAS) {
    const int row = n0 + lane % 16;
    const char* line = reinterpret_cast<const char*>(a.w + static_cast<size_t>(row) * a.ldw + b_begin * 32) + 128 * (lane / 16);
    const int bytes = (min(b_end * 32, a.K) - b_begin * 32) * 2;
#pragma unroll
    for (int rt = 0; rt < RT; ++rt)
      for (int at = 128 * (lane / 16); at < bytes; at += 256)
        if (row + 16 * rt < a.N)
          asm volatile("prefetch.global.L2 [%0];\n" ::"l"(line + static_cast<size_t>(rt) * 16 * a.ldw * 2 + (at - 128 * (lane / 16))));
  }
  wait_for_prior_grids();
  let_dependents_launch();

  float acc[RT][MT][4];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) acc[rt][mt][0] = acc[rt][mt][1] = acc[rt][mt][2] = acc[rt][mt][3] = 0.0f;

  for (int b = b_begin; b < b_end; b += U) {
    uint4 wv[U][2 * RT], xv[X_AHEAD ? U : 1][X_AHEAD ? MT : 1];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (b + u) * 32;
      const bool k_ok = b + u < b_end && k + 8 * t + 8 <= a.K;      // K is a multiple of 8: a chunk is whole or absent
#pragma unroll
      for (int r = 0; r < 2 * RT; ++r) wv[u][r] = load16_or_zero(w_row[r] + k, w_ok[r] && k_ok);
#pragma unroll
      for (int mt = 0; X_AHEAD && mt < MT; ++mt) xv[u][mt] = load16_or_zero(x_row[mt] + k, x_ok[mt] && k_ok);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        const uint4 wl = wv[u][2 * rt], wh = wv[u][2 * rt + 1];
        const unsigned a0[4] = {wl.x, wh.x, wl.y, wh.y};
        const unsigned a1[4] = {wl.z, wh.z, wl.w, wh.w};
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int k = (b + u) * 32;
          const uint4 x = X_AHEAD ? xv[X_AHEAD ? u : 0][X_AHEAD ? mt : 0]
                                  : load16_or_zero(x_row[mt] + k, x_ok[mt] && b + u < b_end && k + 8 * t + 8 <= a.K);
          mma_bf16_16816(acc[rt][mt], a0, x.x, x.y);
          mma_bf16_16816(acc[rt][mt], a1, x.z, x.w);
        }
      }
  }

#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float* at = &red[warp][(rt * MT + mt) * 128 + g * 8 + 2 * t];
      *reinterpret_cast<float2*>(at) = make_float2(acc[rt][mt][0], acc[rt][mt][1]);
      *reinterpret_cast<float2*>(at + 64) = make_float2(acc[rt][mt][2], acc[rt][mt][3]);
    }
  __syncthreads();
  // A CTA adds its warps' sums in their order; a cluster's CTAs each finish a share of the tile from the sums of all, in
  // the CTAs' order, which lie in (distributed) shared memory.
  if (ksplit > 1) {
    for (int e = threadIdx.x; e < PER_WARP; e += WARPS * 32) {
      float sum = red[0][e];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) sum += red[w][e];
      red[0][e] = sum;
    }
    cluster.sync();
  }
  auto total_of = [&](int e) {
    float sum;
    if (ksplit == 1) {
      sum = red[0][e];
#pragma unroll
      for (int w = 1; w < WARPS; ++w) sum += red[w][e];
    } else {
      float part[GS_MAX_KSPLIT];
#pragma unroll
      for (int c = 0; c < GS_MAX_KSPLIT; ++c) part[c] = c < ksplit ? *cluster.map_shared_rank(&red[0][e], c) : 0.0f;
      sum = part[0];
#pragma unroll
      for (int c = 1; c < GS_MAX_KSPLIT; ++c) sum += part[c];
    }
    return sum;
  };
  TOut* y = static_cast<TOut*>(a.y);
  for (int i = krank * WARPS * 32 + threadIdx.x; i < (SWIGLU ? PER_WARP / 2 : PER_WARP); i += ksplit * WARPS * 32) {
    const int r = (i / 8) % (SWIGLU ? 8 : 16), tile = i / (SWIGLU ? 64 : 128), mt = tile % MT, rt = tile / MT;
    const int token = mt * 8 + i % 8, row = n0 + 16 * rt + r;
    if (token >= a.M) continue;
    if (SWIGLU) {                          // rows 0..7 of a tile are gate rows, rows 8..15 the matching up rows
      if (row + 8 >= a.N) continue;
      float gate = total_of(tile * 128 + r * 8 + i % 8), up = total_of(tile * 128 + 64 + r * 8 + i % 8), v;
      if (a.gate.kind == GATE_BOUNDED) {
        if (a.gate.bias != nullptr) {
          gate += a.gate.bias[row];
          up += a.gate.bias[row + 8];
        }
        v = bounded_gate<false>(gate, up, a.gate);
      } else {
        v = (a.gate.kind == GATE_RELU ? fmaxf(gate, 0.0f) : gate / (1.0f + expf(-gate))) * up;
      }
      store_out<TOut>(y + static_cast<size_t>(token) * a.ldy + (blockIdx.x * RT + rt) * 8 + r, v);
    } else {
      if (row >= a.N) continue;
      const float sum = total_of(i);
      TOut* at = y + static_cast<size_t>(token) * a.ldy + static_cast<size_t>(row) * a.ldn;
      if (ACT == ACT_TOKEN_GATE) {
        const int id = a.token_ids[token];
        const bool ok = id >= 0 && id < a.vocab;
        if (!ok && row == 0) report(a.status, STATUS_TOKEN_OUT_OF_RANGE, id, token);
        const float e = ok ? __bfloat162float(a.token_rows[static_cast<long long>(id) * a.token_stride + row]) : 0.0f;
        store_out<TOut>(at, gelu_tanh(sum) * e);
      } else {
        store_out<TOut>(at, ACT == ACT_GELU ? gelu_tanh(sum) : ACT == ACT_RELU2 ? relu_squared(sum) : sum);
      }
    }
  }
  if (ksplit > 1) cluster.sync();           // nobody leaves while its shared memory may still be read
}

struct SmallGemmSplit {
  int warps, ksplit;           // of a CTA; CTAs that share K
};
// How K is cut, from the matrix alone: a row's sums are the same whatever rows it is computed with.  Eight warps a CTA and, up
// to two CTAs an SM, a cluster that shares K (a power of two up to 8, two blocks of k a warp or more): with every warp's loads
// in flight at once the latency of the last one, not the split, is what is left.  Above four such CTAs an SM a second wave
// begins, and four warps are the better CTA (32768 x 2048, 12 rows: 29.8 us against 33.4) until K gives each of them more
// than 32 blocks to walk (24576 x 4096: 56 us against 45).
static SmallGemmSplit small_gemm_split(int N, int K) {
  const int tiles = (N + 15) / 16, blocks = (K + 31) / 32;
  if (tiles > 4 * 148) return {blocks >= 128 ? 8 : 4, 1};
  int ksplit = 1;
  while (ksplit < GS_MAX_KSPLIT && tiles * ksplit < 2 * 148 && blocks >= 4 * 8 * ksplit) ksplit *= 2;
  return {8, ksplit};
}

template <int RT, int WARPS, int MT, typename TOut, bool SWIGLU, int ACT>
int small_gemm_launch(const SmallGemmArgs& a, int ksplit, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((a.N + 16 * RT - 1) / (16 * RT), ksplit, 1);
  config.blockDim = dim3(WARPS * 32, 1, 1);
  config.dynamicSmemBytes = 0;
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = 1;
  attribute[0].val.clusterDim.y = ksplit;
  attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = dependent_launch_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&config, gemm_small_kernel<RT, WARPS, MT, TOut, SWIGLU, ACT>, a) != cudaSuccess) return ERR_CUDA;
  return launch_result();
}

template <int MT, typename TOut, bool SWIGLU, int ACT>
int small_gemm_split_launch(const SmallGemmArgs& a, cudaStream_t stream) {
  const SmallGemmSplit s = small_gemm_split(a.cut_rows, a.K);
  if (s.warps == 8) return small_gemm_launch<1, 8, MT, TOut, SWIGLU, ACT>(a, s.ksplit, stream);
  // Up to 8 tokens and several waves of CTAs: 32 rows a CTA read the tokens half as often (151936 x 1024, 4 rows: 50 us
  // against 54; with 12 rows their registers cost more, 66 against 64).  The sums are the same.
  if (MT == 1) return small_gemm_launch<2, 4, 1, TOut, SWIGLU, ACT>(a, s.ksplit, stream);
  return small_gemm_launch<1, 4, MT, TOut, SWIGLU, ACT>(a, s.ksplit, stream);
}

template <typename TOut, bool SWIGLU, int ACT>
int small_gemm_dispatch(const SmallGemmArgs& a, cudaStream_t stream) {
  switch ((a.M + 7) / 8) {
    case 1: return small_gemm_split_launch<1, TOut, SWIGLU, ACT>(a, stream);
    case 2: return small_gemm_split_launch<2, TOut, SWIGLU, ACT>(a, stream);
    case 3: case 4: return small_gemm_split_launch<4, TOut, SWIGLU, ACT>(a, stream);
    default: return small_gemm_split_launch<8, TOut, SWIGLU, ACT>(a, stream);
  }
}

}  // namespace zb

using namespace zb;

// 1 if zb_gemm_small takes this problem.
ZB_API int zb_gemm_small_supported(int M, int N, int K) {
  return M >= 1 && M <= 8 * GS_MAX_MT && N >= 1 && K >= 8 && K % 8 == 0 ? 1 : 0;
}

// y = x w^T (swiglu = 0), or y[:, 8j + r] = silu(x w[16j + r]^T) * (x w[16j + 8 + r]^T) (swiglu = 1; 2: max(., 0) for silu;
// w holds gate and up rows interleaved in blocks of 8, y has N / 2 columns).
// x: [M, K] bfloat16 rows ldx apart (ldx, ldw multiples of 8, pointers 16-byte aligned);
// out_dtype: bfloat16 or float32.
static int small_gemm(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw,
                      long long ldy, int out_dtype, bool gated, const GateForm& gate, void* stream,
                      int act = ACT_NONE) {
  if (!zb_gemm_small_supported(M, N, K)) return ERR_UNSUPPORTED;
  if (ldx < K || ldw < K || ldx % 8 != 0 || ldw % 8 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(w) % 16 != 0 || (gated && N % 16 != 0))
    return ERR_BAD_ARGUMENT;
  SmallGemmArgs a = {};
  a.y = y;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.w = static_cast<const __nv_bfloat16*>(w);
  a.M = M; a.N = a.cut_rows = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldy = ldy; a.ldn = 1;
  a.gate = gate;
  auto s = static_cast<cudaStream_t>(stream);
  if (act == ACT_GELU)
    return out_dtype == DTYPE_F32 ? small_gemm_dispatch<float, false, ACT_GELU>(a, s)
                                  : small_gemm_dispatch<__nv_bfloat16, false, ACT_GELU>(a, s);
  if (act == ACT_RELU2)
    return out_dtype == DTYPE_F32 ? small_gemm_dispatch<float, false, ACT_RELU2>(a, s)
                                  : small_gemm_dispatch<__nv_bfloat16, false, ACT_RELU2>(a, s);
  if (gated)
    return out_dtype == DTYPE_F32 ? small_gemm_dispatch<float, true, ACT_NONE>(a, s)
                                  : small_gemm_dispatch<__nv_bfloat16, true, ACT_NONE>(a, s);
  return out_dtype == DTYPE_F32 ? small_gemm_dispatch<float, false, ACT_NONE>(a, s)
                                : small_gemm_dispatch<__nv_bfloat16, false, ACT_NONE>(a, s);
}

ZB_API int zb_gemm_small(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw,
                         long long ldy, int out_dtype, int swiglu, void* stream) {
  return small_gemm(y, x, w, M, N, K, ldx, ldw, ldy, out_dtype, swiglu != 0,
                    plain_gate(swiglu == 2 ? GATE_RELU : GATE_SILU), stream);
}

// y [rows, outputs] = x w^T for many rows and few outputs (a router's): the kernel's sides change places, x's rows are streamed as
// its matrix and w's are its few rows, and the result is written transposed.  K is cut as w alone says, so that a row's sums are the
// same as in a step of a few rows.  (Rows of 2048 x 18 outputs, float32 out, us, the
// library's product / here: 65 rows 6.3 / 3.9, 777 12.6 / 4.6, 2048 13 / 5.9, 5000 18.1 / 14.5, 8192 18.3 / 20; cut by the number of rows
// the last two took 11.2 and 12.3.)
ZB_API int zb_gemm_few_outputs(void* y, const void* x, const void* w, int rows, int outputs, int K, long long ldx, long long ldw,
                               long long ldy, int out_dtype, void* stream) {
  if (!zb_gemm_small_supported(outputs, rows, K)) return ERR_UNSUPPORTED;
  if (ldx < K || ldw < K || ldx % 8 != 0 || ldw % 8 != 0 || ldy < outputs || reinterpret_cast<uintptr_t>(x) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(w) % 16 != 0)
    return ERR_BAD_ARGUMENT;
  SmallGemmArgs a = {};
  a.y = y;
  a.x = static_cast<const __nv_bfloat16*>(w);
  a.w = static_cast<const __nv_bfloat16*>(x);
  a.M = a.cut_rows = outputs; a.N = rows; a.K = K; a.ldx = ldw; a.ldw = ldx; a.ldy = 1; a.ldn = ldy;
  auto s = static_cast<cudaStream_t>(stream);
  return out_dtype == DTYPE_F32 ? small_gemm_dispatch<float, false, ACT_NONE>(a, s) : small_gemm_dispatch<__nv_bfloat16, false, ACT_NONE>(a, s);
}

// y = act(x w^T); act: 1 gelu_tanh, 2 the square of max(., 0).
ZB_API int zb_gemm_small_act(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw,
                             long long ldy, int out_dtype, int act, void* stream) {
  if (act != ACT_GELU && act != ACT_RELU2) return ERR_BAD_ARGUMENT;
  return small_gemm(y, x, w, M, N, K, ldx, ldw, ldy, out_dtype, false, plain_gate(GATE_SILU), stream, act);
}

// y [M, N] bfloat16 = gelu_tanh(x w^T) times the values offset .. offset + N of the tokens' rows of `table` [vocab, stride].
ZB_API int zb_gemm_small_token_gate(void* y, const void* x, const void* w, const void* table, long long table_stride, int offset,
                                    const int* ids, int vocab, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                                    int* status, void* stream) {
  if (!zb_gemm_small_supported(M, N, K)) return ERR_UNSUPPORTED;
  if (ldx < K || ldw < K || ldx % 8 != 0 || ldw % 8 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(w) % 16 != 0 || offset < 0 || offset + N > table_stride || vocab <= 0)
    return ERR_BAD_ARGUMENT;
  SmallGemmArgs a = {};
  a.y = y;
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.w = static_cast<const __nv_bfloat16*>(w);
  a.M = M; a.N = a.cut_rows = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldy = ldy; a.ldn = 1;
  a.token_rows = static_cast<const __nv_bfloat16*>(table) + offset;
  a.token_stride = table_stride; a.token_ids = ids; a.vocab = vocab; a.status = status;
  return small_gemm_dispatch<__nv_bfloat16, false, ACT_TOKEN_GATE>(a, static_cast<cudaStream_t>(stream));
}

// The gated form with the bounded gate: y[:, 8j + r] from the sums of w's rows 16j + r (gate) and 16j + 8 + r
// (up), their biases (bias: float32 [N] in w's row order, or null), the bounds and the shifted product.
ZB_API int zb_gemm_small_bounded(void* y, const void* x, const void* w, const float* bias, float limit, float alpha,
                                 float shift, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                                 int out_dtype, void* stream) {
  if (!(limit > 0.0f)) return ERR_BAD_ARGUMENT;
  return small_gemm(y, x, w, M, N, K, ldx, ldw, ldy, out_dtype, true, GateForm{GATE_BOUNDED, bias, limit, alpha, shift, nullptr},
                    stream);
}
