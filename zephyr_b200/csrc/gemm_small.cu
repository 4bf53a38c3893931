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
// of several blocks of 32 k in flight, whatever is left of its slice: four up to 16 rows, two from 17 to 32 and where a CTA takes 32 rows of W;
// above 32 rows four blocks of W alone, x at its use (with x ahead too, two blocks: 12288 x 4096, 64 rows: 92 us,
// now 47; 6144 x 2048: 29 and 17) (one block after the other, as a loop's remainder, 2048 x
// 6144 with 12 rows took 13.8 us; now 10.1, its bytes 3.8), and the CTAs of a cluster each finish a share of the tile with one
// round of remote reads (one CTA for all, 2048 x 2048: 9.8 us; now 6.1).  4096 x 2048: 10.2 -> 7.9, 12288 x 2048: 14.9 -> 14.1,
// 8192 x 4096, 12 rows: 16.9.  Partial sums meet in (distributed) shared memory and are added in
// a fixed order, so the result does not depend on timing.  ACT takes each sum through GELU's tanh form, a
// squared ReLU, or GELU times a value of the token's row of a table.  With SWIGLU the 16 rows are 8 gate
// rows followed by their 8 up rows, and the epilogue writes silu(gate) * up: the activation costs
// no extra pass over memory (reference: src/layer/mlp.cpp:29-36, src/layer/activation.cu:31-33).  Matrices of many rows go through a
// persistent form with the same sums, gemm_small_stream_kernel below, where small_gemm_streams says so.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "mma.cuh"

namespace zb {

namespace cg = cooperative_groups;

constexpr int ACT_TOKEN_GATE = 3;
constexpr int GS_MAX_MT = 8;      // token tiles of 8: M <= 64
constexpr int GS_MAX_KSPLIT = 8;
constexpr int GS_FETCH_AHEAD_CTAS = 4 * 148;
constexpr int GS_STREAM_WARPS = 16;
constexpr size_t GS_STREAM_SMEM = 226 * 1024;

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

__device__ __forceinline__ void copy16_or_zero(unsigned to, const __nv_bfloat16* p, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(p), "r"(ok ? 16 : 0) : "memory");
}

template <typename T> __device__ __forceinline__ void store_out(T* p, float v);
template <> __device__ __forceinline__ void store_out<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void store_out<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}

// A tile's results from its sums: total_of(e) is the sum of entry e of [mt][row][token].
template <int MT, typename TOut, bool SWIGLU, int ACT, typename Total>
__device__ __forceinline__ void small_gemm_finish(const SmallGemmArgs& a, int n0, int first, int step, const Total& total_of) {
  TOut* y = static_cast<TOut*>(a.y);
  for (int i = first; i < MT * (SWIGLU ? 64 : 128); i += step) {
    const int r = (i / 8) % (SWIGLU ? 8 : 16), mt = i / (SWIGLU ? 64 : 128);
    const int token = mt * 8 + i % 8, row = n0 + r;
    if (token >= a.M) continue;
    if (SWIGLU) {                          // rows 0..7 of a tile are gate rows, rows 8..15 the matching up rows
      if (row + 8 >= a.N) continue;
      float gate = total_of(mt * 128 + r * 8 + i % 8), up = total_of(mt * 128 + 64 + r * 8 + i % 8), v;
      if (a.gate.kind == GATE_BOUNDED) {
        if (a.gate.bias != nullptr) {
          gate += a.gate.bias[row];
          up += a.gate.bias[row + 8];
        }
        v = bounded_gate<false>(gate, up, a.gate);
      } else {
        v = (a.gate.kind == GATE_RELU ? fmaxf(gate, 0.0f) : gate / (1.0f + expf(-gate))) * up;
      }
      store_out<TOut>(y + static_cast<size_t>(token) * a.ldy + n0 / 2 + r, v);
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
}

template <int RT, int WARPS, int MT, typename TOut, bool SWIGLU, int ACT>
__global__ void __launch_bounds__(WARPS * 32)
gemm_small_kernel(const SmallGemmArgs a) {
  constexpr bool X_AHEAD = MT <= 4;                 // (eight tiles of tokens ahead leave room for two blocks of W)
  constexpr int U = (RT == 1 && MT <= 2) || !X_AHEAD ? 4 : 2;     // blocks of k in flight
  constexpr int SUMS = MT * 16 * 8, PER_WARP = RT * SUMS;         // sums of a warp: [rt][mt][row][token]
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
      float* at = &red[warp][rt * SUMS + mt * 128 + g * 8 + 2 * t];
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
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
    small_gemm_finish<MT, TOut, SWIGLU, ACT>(a, n0 + 16 * rt, krank * WARPS * 32 + threadIdx.x, ksplit * WARPS * 32,
                                             [&](int e) { return total_of(rt * SUMS + e); });
  if (ksplit > 1) cluster.sync();           // nobody leaves while its shared memory may still be read
}

// The same sums with one CTA an SM that walks the tiles of 16 rows: a team of its 16 warps (SLICES of them, at most all) shares a
// tile, a warp one slice of K or SLICES / 16 of them, added in the order in which the kernel above adds its warps and its
// cluster's CTAs.  That kernel is bound by its waits: a warp asks for four blocks of k, waits for all of them and only then
// asks for more, and every tile fetches the few rows of x from L2 again, as many bytes as the tile has from 16 rows on.  Here x
// lies in shared memory once an SM, as fragments, and a warp's blocks pass through a ring of DEPTH of them that a lane fills
// with asynchronous copies of just the 16 bytes it will use itself, so that nobody has to be told of their arrival and 64 to
// 128 KB an SM are on their way all the time, also from one tile to the next (through registers, four blocks ahead, 32768 x
// 2048 with 12 rows took 28.1 us).  With X_RING, where x and four blocks a warp are more than shared memory, the rings bring
// x's pieces beside W's.  In us, the kernel above and this one (TB/s): 32768 x 2048, 1 row 25.5 and 22.2 (6.0),
// 12 rows 33.2 and 24.7 (5.4), 32 rows 44 and 29.8; 16384 x 2048, 8 rows 19.3 and 12.3, 12 rows 16.5 and 13.5; 24576 x 4096,
// 12 rows 46 and 38.4; 151936 x 1024, 12 rows 67 and 52 (6.0), one row 50.3 (with 32 rows a CTA) and 49.7; with X_RING 2048 x 8192, 12
// rows 12.1 and 9.6, 12288 x 4096, 32 rows 47.6 and 28.5.
template <int SLICES, int DEPTH, bool X_RING, int MT, typename TOut, bool SWIGLU, int ACT>
__global__ void __launch_bounds__(GS_STREAM_WARPS * 32, 1)
gemm_small_stream_kernel(const SmallGemmArgs a) {
  constexpr int TEAM = SLICES < GS_STREAM_WARPS ? SLICES : GS_STREAM_WARPS, TEAMS = GS_STREAM_WARPS / TEAM;
  constexpr int PER_WARP = SLICES / TEAM, GROUP = SLICES < 8 ? SLICES : 8, SUMS = MT * 128;
  constexpr int SLOT = X_RING ? 2 + MT : 2;       // 512-byte pieces of a ring's slot: two of W, with X_RING x's behind them
  extern __shared__ __align__(16) unsigned char gs_smem[];
  const int blocks = (a.K + 31) / 32;
  uint4* x_s = reinterpret_cast<uint4*>(gs_smem);                                  // [block of k][mt][lane]: fragments
  float* red = reinterpret_cast<float*>(x_s + (X_RING ? 0 : static_cast<size_t>(blocks) * MT * 32));      // [team][slice][SUMS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, team = warp / TEAM;
  uint4* ring = reinterpret_cast<uint4*>(red + TEAMS * SLICES * SUMS) + warp * DEPTH * SLOT * 32 + lane;   // [warps][DEPTH][SLOT][lane]
  const int g = lane >> 2, t = lane & 3;
  const int first_slice = warp % TEAM * PER_WARP;
  auto slice_begin = [&](int i) { return blocks * i / SLICES; };
  const int b_begin = slice_begin(first_slice), b_end = slice_begin(first_slice + PER_WARP);
  const int tiles = (a.N + 15) / 16, first_tile = team * gridDim.x + blockIdx.x, tile_step = TEAMS * gridDim.x;

  // While the kernel before this one still runs: the team's first tile, as far as L2 (as above).
  {
    const int row = first_tile * 16 + lane % 16;
    if (row < a.N) {
      const char* line = reinterpret_cast<const char*>(a.w + static_cast<size_t>(row) * a.ldw + b_begin * 32);
      const int bytes = (min(b_end * 32, a.K) - b_begin * 32) * 2;
      for (int at = 128 * (lane / 16); at < bytes; at += 256) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(line + at));
    }
  }
  wait_for_prior_grids();
  let_dependents_launch();

  // Cursor of the copies: `ahead` blocks in front of the products, across the team's tiles.
  int c_tile = first_tile, c_b = b_begin, c_slot = 0;
  const __nv_bfloat16 *lo, *hi;
  bool lo_ok, hi_ok;
  auto rows_of = [&]() {
    const int row = c_tile * 16 + g;
    lo_ok = c_tile < tiles && row < a.N;
    hi_ok = c_tile < tiles && row + 8 < a.N;
    lo = a.w + static_cast<size_t>(lo_ok ? row : 0) * a.ldw;
    hi = a.w + static_cast<size_t>(hi_ok ? row + 8 : 0) * a.ldw;
  };
  rows_of();
  const unsigned ring_at = smem_u32(ring);
  auto copy_next = [&]() {
    const int k = c_b * 32 + 8 * t;
    const bool k_ok = k + 8 <= a.K;
    const unsigned to = ring_at + c_slot * (SLOT * 512);
    copy16_or_zero(to, lo + (k_ok ? k : 0), lo_ok && k_ok);
    copy16_or_zero(to + 512, hi + (k_ok ? k : 0), hi_ok && k_ok);
#pragma unroll
    for (int mt = 0; X_RING && mt < MT; ++mt) {
      const bool ok = mt * 8 + g < a.M && k_ok && c_tile < tiles;
      copy16_or_zero(to + 1024 + mt * 512, a.x + (ok ? static_cast<size_t>(mt * 8 + g) * a.ldx + k : 0), ok);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    c_slot = c_slot + 1 == DEPTH ? 0 : c_slot + 1;
    if (++c_b >= b_end) {
      c_b = b_begin;
      c_tile += tile_step;
      rows_of();
    }
  };
#pragma unroll
  for (int u = 0; u < DEPTH; ++u) copy_next();
  for (int e = threadIdx.x; !X_RING && e < blocks * MT * 32; e += GS_STREAM_WARPS * 32) {
    const int k = e / (MT * 32) * 32 + 8 * (e % 4), m = e / 32 % MT * 8 + e % 32 / 4;
    x_s[e] = load16_or_zero(a.x + static_cast<size_t>(m < a.M ? m : 0) * a.ldx + k, m < a.M && k + 8 <= a.K);
  }
  if (!X_RING) __syncthreads();

  auto team_barrier = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + team), "n"(TEAM * 32) : "memory"); };
  int slot = 0;
  for (int tile = first_tile; tile < tiles; tile += tile_step) {
    if (tile != first_tile) team_barrier();               // the tile before has been read
    int b = b_begin;
#pragma unroll 1
    for (int i = 0; i < PER_WARP; ++i) {
      const int slice = first_slice + i;
      float acc[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.0f;
      const int end = slice_begin(slice + 1);
#pragma unroll 2
      for (; b < end; ++b) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(DEPTH - 1) : "memory");
        const uint4* now = ring + slot * (SLOT * 32);
        const uint4 wl = now[0], wh = now[32];
        slot = slot + 1 == DEPTH ? 0 : slot + 1;
        const unsigned a0[4] = {wl.x, wh.x, wl.y, wh.y}, a1[4] = {wl.z, wh.z, wl.w, wh.w};
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const uint4 x = X_RING ? now[64 + mt * 32] : x_s[(b * MT + mt) * 32 + lane];
          mma_bf16_16816(acc[mt], a0, x.x, x.y);
          mma_bf16_16816(acc[mt], a1, x.z, x.w);
        }
        copy_next();
      }
      float* mine = red + (team * SLICES + slice) * SUMS;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float* at = mine + mt * 128 + g * 8 + 2 * t;
        *reinterpret_cast<float2*>(at) = make_float2(acc[mt][0], acc[mt][1]);
        *reinterpret_cast<float2*>(at + 64) = make_float2(acc[mt][2], acc[mt][3]);
      }
    }
    team_barrier();
    const float* all = red + team * SLICES * SUMS;
    small_gemm_finish<MT, TOut, SWIGLU, ACT>(a, tile * 16, threadIdx.x % (TEAM * 32), TEAM * 32, [&](int e) {
      float total = 0.0f;                                 // the sums of eight slices in order, then those
#pragma unroll
      for (int s0 = 0; s0 < SLICES; s0 += GROUP) {
        float sum = all[s0 * SUMS + e];
#pragma unroll
        for (int i = 1; i < GROUP; ++i) sum += all[(s0 + i) * SUMS + e];
        total = s0 == 0 ? sum : total + sum;
      }
      return total;
    });
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// The streaming kernel's shared memory: x where the rings do not bring it, the slices' sums, the rings.
static size_t small_gemm_stream_smem(int K, int token_tiles, int slices, int depth, bool x_ring) {
  const size_t teams = slices < GS_STREAM_WARPS ? GS_STREAM_WARPS / slices : 1, pieces = x_ring ? 2 + token_tiles : 2;
  return ((x_ring ? 0 : static_cast<size_t>((K + 31) / 32) * token_tiles) + teams * slices * token_tiles +
          GS_STREAM_WARPS * depth * pieces) * 512;
}

struct SmallGemmSplit {
  int warps, ksplit;           // of a CTA; CTAs that share K
};

// Whether the streaming kernel takes a product (its sums are the other kernel's, so that this may look at the number of rows).  It
// starts later (x and the rings first) and then never waits for a whole burst of loads, so it is ahead where a warp of the other kernel walks
// several bursts or its CTAs come in more than one round, and behind where one burst or one full round brings all there is.  In us, the
// other kernel and this one, matrices from memory, launched one behind the other:
//   more than four tiles of 16 rows an SM (K cut among four warps, bursts of 512 values of k):
//     8 rows (32 rows of W a CTA, rounds of up to 14 tiles an SM): 65536 x 1024 24.0 and 23.5, 65536 x 512 14.0 and 12.8; 32768 x 1536 18.8
//     and 18.1, 16384 x 1024 9.4 and 7.7, 24576 x 1024 12.8 and 10.1, 32768 x 1024 12.1 and 12.7, but as the head of a decode step 15.5 and
//     15.2 with what follows it 3.7 us earlier (eight requests on four layers 15.68 and 15.52 ms a pass); 24576 x 768 9.4 and 8.5, 32768 x 768
//     9.1 and 10.2; 24576 x 512 7.0 and 7.1, 16384 x 512 4.5 and 5.6; 65536 x 256 8.2 and 8.8;
//     12 rows (rounds of up to 7 tiles an SM): 20480 x 256 5.9 and 5.2, 65536 x 256 13.0 and 10.6; 16384 x 1024 8.4 and 8.3, 12288 x 768
//     7.5 and 6.9, 16384 x 768 7.4 and 7.6, 10240 x 512 5.3 and 5.1, 12288 x 512 5.0 and 5.4, 16384 x 512 5.0 and 6.4;
//     32 rows: 24576 x 512 13.3 and 10.9, 24576 x 256 8.7 and 8.6 (24 rows 7.5 and 7.8); 16384 x 1024 11.6 and 10.6, 16384 x 768 9.2 and 9.3,
//     10240 x 512 6.8 and 6.3;
//   fewer tiles (eight warps, and clusters that share K; bursts of 1024):
//     8 rows: 4864 x 4096 12.5 and 11.0, 8192 x 3072 11.7 and 10.4, 8192 x 2048 7.7 and 8.2;
//     12 rows: 2048 x 2048 7.2 and 5.4, 2048 x 1536 4.0 and 4.6, 3072 x 1536 7.5 and 6.0, 4096 x 1024 7.2 and 4.9, 2048 x 1024 3.7 and 3.7, 4096 x 768
//     2.6 and 3.9; 4736 x 2048 5.4 and 7.3 (exactly two CTAs an SM of the other); 8192 x 512 4.8 and 4.4, 8192 x 768 5.2 and 5.6, 8192 x 1024
//     5.8 and 6.6, 8192 x 1536 8.1 and 7.9;
//     32 rows: 4096 x 1536 7.6 and 6.9, 4096 x 1024 5.8 and 6.2, 6144 x 1024 7.9 and 7.1, 6144 x 512 5.2 and 5.1 (24 rows 4.7 and 4.9), 8192 x 1024
//     7.9 and 8.4.
static bool small_gemm_streams(int N, int K, int token_tiles, const SmallGemmSplit& s) {
  const int tiles = (N + 15) / 16, slices = s.warps * s.ksplit;
  if (slices > 32) return false;
  if (tiles > 4 * 148) {
    if (token_tiles == 1) return tiles > 14 * 148 ? K >= 512 : K >= 1024 || (K >= 768 && tiles <= 12 * 148);
    if (token_tiles == 2) return tiles > 7 * 148 || K >= 1024 || (K >= 768 && tiles <= 6 * 148) || (K >= 512 && tiles <= 5 * 148);
    return K >= 1024 || (K >= 512 && (tiles > 7 * 148 || tiles <= 5 * 148));
  }
  if (token_tiles == 1) return tiles > 2 * 148 && K >= 3072;
  if (token_tiles == 2) {
    if (tiles < 2 * 148) return tiles >= 96 && (K >= 2048 || (K >= 1024 && tiles > 148));
    return tiles > 400 && (K >= 1536 || K <= 512);
  }
  return tiles > 200 && (K >= 1536 || (K >= 768 && tiles > 2 * 148 && tiles <= 400));
}
// How K is cut, from the matrix alone: a row's sums are the same whatever rows it is computed with.  Eight warps a CTA and, up
// to two CTAs an SM, a cluster that shares K (a power of two up to 8, two blocks of k a warp or more): with every warp's loads
// in flight at once the latency of the last one, not the split, is what is left.  Above four such CTAs an SM a second wave
// begins, and four warps are the better CTA (32768 x 2048, 12 rows: 29.8 us against 33.4) until K gives each of them more
// than 32 blocks to walk (24576 x 4096: 56 us against 45); the streaming kernel, which takes most of those, keeps the cut.
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

template <int SLICES, int DEPTH, bool X_RING, int MT, typename TOut, bool SWIGLU, int ACT>
int small_gemm_stream_launch(const SmallGemmArgs& a, cudaStream_t stream) {
  const size_t smem = small_gemm_stream_smem(a.K, MT, SLICES, DEPTH, X_RING);
  if (cuda_failed(cudaFuncSetAttribute(gemm_small_stream_kernel<SLICES, DEPTH, X_RING, MT, TOut, SWIGLU, ACT>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem))))
    return ERR_CUDA;
  return launch_dependent(gemm_small_stream_kernel<SLICES, DEPTH, X_RING, MT, TOut, SWIGLU, ACT>, dim3(std::min(148, (a.N + 15) / 16)),
                          dim3(GS_STREAM_WARPS * 32), smem, stream, false, a);
}

// As many blocks on their way as shared memory has room for beside all of x; x through the rings where that leaves none.
template <int SLICES, int MT, typename TOut, bool SWIGLU, int ACT>
int small_gemm_stream(const SmallGemmArgs& a, cudaStream_t stream) {
  constexpr int WITH_X = MT == 1 ? 8 : MT == 2 ? 6 : 4;
  if (small_gemm_stream_smem(a.K, MT, SLICES, 8, false) <= GS_STREAM_SMEM)
    return small_gemm_stream_launch<SLICES, 8, false, MT, TOut, SWIGLU, ACT>(a, stream);
  if constexpr (SLICES == 4 && MT <= 2) {        // K below 4096
    return small_gemm_stream_launch<SLICES, 4, false, MT, TOut, SWIGLU, ACT>(a, stream);
  } else {
    if (small_gemm_stream_smem(a.K, MT, SLICES, 4, false) <= GS_STREAM_SMEM)
      return small_gemm_stream_launch<SLICES, 4, false, MT, TOut, SWIGLU, ACT>(a, stream);
    return small_gemm_stream_launch<SLICES, WITH_X, true, MT, TOut, SWIGLU, ACT>(a, stream);
  }
}

template <int MT, typename TOut, bool SWIGLU, int ACT>
int small_gemm_split_launch(const SmallGemmArgs& a, cudaStream_t stream) {
  const SmallGemmSplit s = small_gemm_split(a.cut_rows, a.K);
  if constexpr (MT <= 4) {
    if (small_gemm_streams(a.cut_rows, a.K, MT, s)) {
      const int slices = s.warps * s.ksplit;
      if (slices == 4) return small_gemm_stream<4, MT, TOut, SWIGLU, ACT>(a, stream);
      if constexpr (MT > 1)
        if (slices == 16) return small_gemm_stream<16, MT, TOut, SWIGLU, ACT>(a, stream);
      if constexpr (MT == 2)
        if (slices == 32) return small_gemm_stream<32, MT, TOut, SWIGLU, ACT>(a, stream);
      return small_gemm_stream<8, MT, TOut, SWIGLU, ACT>(a, stream);
    }
  }
  if (s.warps == 8) return small_gemm_launch<1, 8, MT, TOut, SWIGLU, ACT>(a, s.ksplit, stream);
  // Up to 8 tokens 32 rows a CTA read the tokens half as often and are half as many CTAs (151936 x 1024, 4 rows: 50 us against 54; with 12
  // rows their registers cost more, 66 against 64).  The sums are the same.
  return small_gemm_launch<MT == 1 ? 2 : 1, 4, MT, TOut, SWIGLU, ACT>(a, s.ksplit, stream);
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

// 1 if zb_gemm_small streams this problem's matrix through its persistent kernel.
ZB_API int zb_gemm_small_streams(int M, int N, int K) {
  if (!zb_gemm_small_supported(M, N, K) || M > 32) return 0;
  return small_gemm_streams(N, K, M > 16 ? 4 : (M + 7) / 8, small_gemm_split(N, K)) ? 1 : 0;
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
