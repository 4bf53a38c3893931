// Y[M, N] = X[M, K] * W[N, K]^T of float32 matrices on the fifth-generation tensor cores, every product of two float32 values
// and their float32 sum, no TF32: the true 32-bit path's product for rows that start on 16-byte boundaries.
//
// A float32 value is the sum of three bfloat16 values, hi + mid + lo, to its last bit (each is what the ones before it leave,
// rounded to nearest), and the product of two bfloat16 values is exact in float32.  Six of the nine products of parts count:
// what mid lo, lo mid and lo lo would add is below 2^-25 of the whole.  The tensor cores cut a sum's last bits at every step, so
// the sums are kept short: hi hi is summed over 64 values of k in tensor memory, from zero each time, and those sums are added
// to the total in registers with float32's rounding; the other five, 2^-8 and less of it, are summed over all of K where a cut
// bit is 2^-8 of one of the total's.  Error against 64 bits (2-norm of the difference over the result's, normal values): 3.7e-8 at K = 16,
// 7.0e-8 at 64, 8.1e-8 at 256, 1.05e-7 at 1024, 1.5e-7 at 3072, 1.7e-7 at 4096, where multiply-adds in four chains had 7.4e-8, 8.4e-8,
// 1.5e-7, 2.9e-7, 5.0e-7 and 5.7e-7.  The order of all this is the same whatever M, N and the tile, so a row's result does not depend on
// the batch around it.
// Values are split times 2^39, with which the parts hold every bit of float32's smallest and no part of an output is below float32's
// range; a sum is taken back at its end.  A value from 2^88 on, or a sum from 2^50, leaves that range at its other end: outputs that
// are not finite are formed again by multiply-adds.
//
// A pair of SMs (tcgen05.mma.cta_group::2) = 256 rows of w, the tensor cores' row side, by NT rows of x, their columns; each CTA fetches 128
// and NT / 2 of them.  Per 64 values of k: sixteen warps (eight with 256 columns) fetch the rows as float32 (the next 64 on their way in
// registers meanwhile), split them and store the parts where the tensor cores read them (K-major, 128-byte swizzle); one thread issues
// the products of parts, the small ones first, hi hi behind the warps' having taken the sums of the 64 values before; the warps
// add those to theirs while the next products run.
// Bound by the tensor cores from 192 columns on (4096^3 598 us, 230 TFLOP/s and six times that of bfloat16
// products, 0.84 of the measured peak; with eight warps 700 us), below by the chain of a stage: fetch, split, 24 products of at least 50
// cycles, sums.  What it takes beside: 700 x 4096 x 1024 33 us (multiply-adds on CUDA cores 197; eight warps 44), 700 x 1024 x 2048 35
// (102; 40), 900 x 1024 x 3072 49 (189; 54), 8 x 151936 x 1024 163 (387; 201), one row x 4096 x 1024 17 (18; 20).  Four stages are little beside
// the kernel's start and end: one row x 1024 x 256 6.5 (5.3), x 2048 x 512 10.6 (9.8).  On single SMs (128 rows of w by 96) 62 us for the first,
// bound by the operands' way from L2.  The second SM's stages are announced by a thread of its own, which costs 1 to 3 %: its warps' own arrivals on the
// other SM's barrier do not come behind their stores, and arrivals with a release across the cluster, by the warps or by that thread, cost
// 500 cycles a stage (700 x 1024 x 2048 48 and 41 us).
// Every wait is bounded and reports instead of hanging; tensor memory is given back on every path.
#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"

ZB_API int zb_gemm_nt_simt(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                           int in_dtype, int out_dtype, void* stream);      // gemm_simt.cu

namespace zb {

constexpr int GF_BK = 64;                   // values of k a stage: one 128-byte row of a part
constexpr int GF_ROWS = 128;                // rows of w of a CTA
constexpr int GF_AHEAD = 4;                  // stages of w that L2 is asked for ahead
constexpr int GF_WAIT_LIMIT = 1 << 18;
constexpr int GF_W_PART = GF_ROWS * GF_BK * 2;

template <int NT> struct GemmF32Shape {
  // That fetch, split and sum (one of the four behind them issues the products): sixteen, whose waits overlap better than eight's
  // (700 x 4096 x 1024 in 192 columns 34.8 us against 42, 700 x 1024 x 2048 in 64 34.5 against 40), up to the columns whose sums their
  // registers hold.
  static constexpr int WARPS = NT <= 192 ? 16 : 8;
  static constexpr int THREADS = (WARPS + 4) * 32;
  // Of the 96 or 168 that the block is launched with: 512 x 104 + 128 x 64 = 640 x 96, 256 x 232 + 128 x 40 = 384 x 168.
  static constexpr int WORKER_REGISTERS = WARPS == 16 ? 104 : 232, OTHER_REGISTERS = WARPS == 16 ? 64 : 40;
  static constexpr int PASS = WARPS * 4;    // rows that the workers fetch at a time

  static constexpr int X_ROWS = NT / 2;     // of a CTA
  static constexpr int X_PART = X_ROWS * GF_BK * 2;
  static constexpr int STAGE_BYTES = 3 * (GF_W_PART + X_PART);
  static constexpr int SMEM_BYTES = 2 * STAGE_BYTES + 1024;
  static constexpr int TMEM_COLUMNS = NT <= 32 ? 64 : NT <= 64 ? 128 : NT <= 128 ? 256 : 512;      // the hi hi sums, the others
  static constexpr int COLUMNS = NT * 4 / WARPS;      // of a warp
  static constexpr int PER = (GF_ROWS + X_ROWS + PASS - 1) / PASS;      // 32-byte pieces a thread fetches of a stage
  static_assert(NT % 32 == 0 && NT <= 256 && COLUMNS % 8 == 0, "columns of tensor memory in runs of 8 a warp");
};

struct GemmF32Args {
  float* y;
  const float* x;
  const float* w;
  int M, N, K, tiles_m;
  long long ldx, ldw, ldy;
  int* status;
};

__device__ __forceinline__ void tmem_ld_run(unsigned at, unsigned (&v)[16]) { tmem_ld16(at, v); }
__device__ __forceinline__ void tmem_ld_run(unsigned at, unsigned (&v)[8]) { tmem_ld8(at, v); }
__device__ __forceinline__ void tmem_wait_ld_run(unsigned (&v)[16]) { tmem_wait_ld16(v); }
__device__ __forceinline__ void tmem_wait_ld_run(unsigned (&v)[8]) { tmem_wait_ld8(v); }

// One output by multiply-adds in ascending k.
__device__ __noinline__ float dot_f32(const float* x, const float* w, int K) {
  float sum = 0.0f;
  for (int k = 0; k < K; k += 4) {
    const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
    sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
  }
  return sum;
}

template <int NT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GemmF32Shape<NT>::THREADS, 1) gemm_f32_tc_kernel(const GemmF32Args a) {
  using Shape = GemmF32Shape<NT>;
  constexpr int COLUMNS = Shape::COLUMNS, PER = Shape::PER, X_PART = Shape::X_PART, WARPS = Shape::WARPS, PASS = Shape::PASS;
  extern __shared__ unsigned char gf_smem_raw[];
  __shared__ unsigned long long full[2], taken, done, own_full[2];      // own_full: of the second CTA's own warps
  __shared__ unsigned tmem_base_s;
  __shared__ volatile int failed;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gf_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = static_cast<int>(cluster_rank());
  const int pair = static_cast<int>(blockIdx.x >> 1);
  const int m0 = pair % a.tiles_m * NT, n0 = pair / a.tiles_m * (2 * GF_ROWS) + rank * GF_ROWS;
  const int blocks = (a.K + GF_BK - 1) / GF_BK;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&full[i], WARPS + 1);
      mbar_init(&own_full[i], WARPS);
    }
    mbar_init(&taken, 2 * WARPS);
    mbar_init(&done, 1);
    failed = 0;
    fence_barrier_init();
  }
  if (warp == WARPS) {
    tmem_alloc_pair(&tmem_base_s, Shape::TMEM_COLUMNS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                   // both CTAs' barriers and tensor memory are there
  tc_fence_after_sync();
  const unsigned tmem_base = tmem_base_s, tmem_low = tmem_base + Shape::TMEM_COLUMNS / 2;
  wait_for_prior_grids();
  let_dependents_launch();

  auto wait = [&](auto look, unsigned long long* bar, unsigned parity, int where) -> bool {
    bool ok = false;
    for (int i = 0; i < GF_WAIT_LIMIT && !ok; ++i) {
      ok = look(bar, parity);
      if (!ok && (i & 255) == 255 && failed) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0 && !failed) report(a.status, STATUS_BARRIER_TIMEOUT, where, static_cast<int>(blockIdx.x));
      failed = 1;
    }
    return ok;
  };
  auto landed = [&](unsigned long long* bar, unsigned parity, int where) { return wait(mbar_try_wait, bar, parity, where); };          // this CTA's own, or a commit's
  auto arrived = [&](unsigned long long* bar, unsigned parity, int where) { return wait(mbar_try_wait_cluster, bar, parity, where); };

  if (warp >= WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(Shape::OTHER_REGISTERS));
    if (warp == WARPS && rank == 0) {
      constexpr unsigned IDESC = tc_idesc_pair(NT);
      const bool leader = elect_one();
      for (int b = 0; b < blocks; ++b) {
        const unsigned stage = smem_u32(ring + (b & 1) * Shape::STAGE_BYTES);
        if (!arrived(&full[b & 1], b >> 1 & 1, b)) break;
        tc_fence_after_sync();
        const unsigned long long w_hi = desc_k_major(stage), w_mid = desc_k_major(stage + GF_W_PART), w_lo = desc_k_major(stage + 2 * GF_W_PART);
        const unsigned x_at = stage + 3 * GF_W_PART;
        const unsigned long long x_hi = desc_k_major(x_at), x_mid = desc_k_major(x_at + X_PART), x_lo = desc_k_major(x_at + 2 * X_PART);
        if (leader) {
#pragma unroll
          for (int k = 0; k < GF_BK / 16; ++k) {
            tc_mma_pair(tmem_low, w_lo + 2 * k, x_hi + 2 * k, IDESC, (b | k) != 0 ? 1u : 0u);
            tc_mma_pair(tmem_low, w_mid + 2 * k, x_mid + 2 * k, IDESC, 1u);
            tc_mma_pair(tmem_low, w_hi + 2 * k, x_lo + 2 * k, IDESC, 1u);
            tc_mma_pair(tmem_low, w_mid + 2 * k, x_hi + 2 * k, IDESC, 1u);
            tc_mma_pair(tmem_low, w_hi + 2 * k, x_mid + 2 * k, IDESC, 1u);
          }
        }
        if (b > 0 && !arrived(&taken, (b - 1) & 1, -1 - b)) break;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int k = 0; k < GF_BK / 16; ++k) tc_mma_pair(tmem_base, w_hi + 2 * k, x_hi + 2 * k, IDESC, k != 0 ? 1u : 0u);
          tc_commit_pair(&done);
        }
      }
    } else if (warp == WARPS + 1 && rank == 1) {
      // The second CTA's stages are announced by a thread that has seen all of its warps' stores arrive in its shared memory, where its tensor
      // core reads them: a warp's own arrival on the other CTA's barrier is no measure of that.
      const unsigned at = in_cta_of_rank(smem_u32(&full[0]), 0);
      for (int b = 0; b < blocks; ++b) {
        if (!landed(&own_full[b & 1], b >> 1 & 1, 2000000 + b)) break;
        if (lane == 0) mbar_arrive_at(at + 8 * (b & 1));
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(Shape::WORKER_REGISTERS));
    // Piece u of this thread: 8 values of k (4 c .. and 32 + 4 c .. of the stage's 64, side by side in both operands' shared memory)
    // of row tid / 8 + PASS u of the CTA's rows of w and, behind them, of x.
    const int c = tid & 7, r0 = tid >> 3, x0 = m0 + rank * Shape::X_ROWS;
    const float* const w_row = a.w + static_cast<long long>(n0 + r0) * a.ldw + 4 * c;
    const float* const x_row = a.x + static_cast<long long>(x0 + r0) * a.ldx + 4 * c;
    unsigned present = 0;              // bit u: its row lies within the matrix
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int r = r0 + PASS * u;
      if (PASS * u < GF_ROWS ? n0 + r < a.N : x0 + r - GF_ROWS < a.M && r - GF_ROWS < Shape::X_ROWS) present |= 1u << u;
    }
    float4 ahead[PER][2];
    // Up to 64 rows of x (in tiles of up to 64 columns) a stage is the time of its fetches, which is short from L2: w's rows are asked for that far
    // ahead.  (One row x 4096 x 1024 19.6 -> 17.3 us, 64 x 1024 x 2048 34 -> 31; with more rows it costs 2 to 5 %.)
    auto ask = [&](int b) {
      if (a.M > 64) return;
#pragma unroll
      for (int u = 0; u < (NT <= 64 ? GF_ROWS / PASS : 0); ++u)
        if (c < 2 && (present >> u & 1) && b * GF_BK + 32 * c < a.K)
          asm volatile("prefetch.global.L2 [%0];\n" ::"l"(w_row + PASS * u * a.ldw + b * GF_BK + 28 * c));
    };
    auto fetch = [&](int b) {
#pragma unroll
      for (int u = 0; u < PER; ++u)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int k = b * GF_BK + 32 * half;
          const float* row = PASS * u < GF_ROWS ? w_row + PASS * u * a.ldw : x_row + (PASS * u - GF_ROWS) * a.ldx;
          ahead[u][half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if ((present >> u & 1) && k + 4 * c < a.K) ahead[u][half] = *reinterpret_cast<const float4*>(row + k);
        }
    };
    auto store = [&](unsigned char* stage) {
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int r = r0 + PASS * u;
        const bool of_w = PASS * u < GF_ROWS;
        if (!of_w && PASS * u + PASS - 1 >= GF_ROWS + Shape::X_ROWS && r >= GF_ROWS + Shape::X_ROWS) continue;
        unsigned char* to = stage + (of_w ? r * 128 : 3 * GF_W_PART + (r - GF_ROWS) * 128) + ((c ^ (r & 7)) << 4);
        const int part = of_w ? GF_W_PART : X_PART;
        const float4 p = ahead[u][0], q = ahead[u][1];
        uint4 hi, mid, lo;
        three_parts_scaled(p.x, p.y, hi.x, mid.x, lo.x);
        three_parts_scaled(p.z, p.w, hi.y, mid.y, lo.y);
        three_parts_scaled(q.x, q.y, hi.z, mid.z, lo.z);
        three_parts_scaled(q.z, q.w, hi.w, mid.w, lo.w);
        *reinterpret_cast<uint4*>(to) = hi;
        *reinterpret_cast<uint4*>(to + part) = mid;
        *reinterpret_cast<uint4*>(to + 2 * part) = lo;
      }
    };
    // Sums: this thread's row of w (its lane of tensor memory) and a warp's share of the columns.
    const int quarter = warp & 3, column0 = (warp >> 2) * COLUMNS;
    const unsigned tmem_mine = (static_cast<unsigned>(32 * quarter) << 16) + column0;
    float sum[COLUMNS];
#pragma unroll
    for (int i = 0; i < COLUMNS; ++i) sum[i] = 0.0f;
    auto add = [&](unsigned from) {
      constexpr int RUN = COLUMNS % 16 == 0 && WARPS == 8 ? 16 : 8;
      unsigned v[2][RUN];
      tmem_ld_run(from + tmem_mine, v[0]);
#pragma unroll
      for (int i = 0; i < COLUMNS / RUN; ++i) {
        tmem_wait_ld_run(v[i & 1]);
        if (i + 1 < COLUMNS / RUN) tmem_ld_run(from + tmem_mine + RUN * (i + 1), v[(i + 1) & 1]);
#pragma unroll
        for (int e = 0; e < RUN; ++e) sum[RUN * i + e] += __uint_as_float(v[i & 1][e]);
      }
    };
    const unsigned taken_at = in_cta_of_rank(smem_u32(&taken), 0);
    auto take = [&](int b) -> bool {           // the hi hi sums of stage b
      if (!landed(&done, b & 1, 1000000 + b)) return false;
      tc_fence_after_sync();
      add(tmem_base);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_at(taken_at);      // (the sums are in registers, and tensor memory is all that is written behind it)
      return true;
    };
    fetch(0);
    for (int b = 1; b < GF_AHEAD; ++b) ask(b);
    bool ok = true;
    for (int b = 0; b < blocks && ok; ++b) {
      store(ring + (b & 1) * Shape::STAGE_BYTES);       // (free: the stage before last's sums have been taken)
      fence_proxy_async();              // the tensor cores read the parts through the asynchronous proxy
      __syncwarp();
      if (lane == 0) tc_mbar_arrive(rank == 0 ? &full[b & 1] : &own_full[b & 1]);
      fetch(b + 1);
      ask(b + GF_AHEAD);
      if (b > 0) ok = take(b - 1);
    }
    if (ok && take(blocks - 1)) {
      add(tmem_low);
      const int n = n0 + 32 * quarter + lane;
      float* to = a.y + n;
#pragma unroll
      for (int i = 0; i < COLUMNS; ++i) {
        const int m = m0 + column0 + i;
        if (n >= a.N || m >= a.M) continue;
        float v = sum[i] * PARTS_UNSCALE;
        if (!(fabsf(sum[i]) <= 3.4e38f)) v = dot_f32(a.x + m * a.ldx, a.w + n * a.ldw, a.K);
        to[m * a.ldy] = v;
      }
    }
  }

  // Both CTAs meet here on every path (the other's barriers, shared and tensor memory are used until then), and the warps that
  // took the tensor memory give it back.
  tc_fence_before_sync();
  __syncthreads();
  if (failed) let_copies_land();        // (the products in flight)
  __syncwarp();
  cluster_sync_all();
  if (warp == WARPS) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, Shape::TMEM_COLUMNS);
  }
}

template <int NT>
static int gemm_f32_launch(GemmF32Args a, cudaStream_t stream) {
  using Shape = GemmF32Shape<NT>;
  a.tiles_m = (a.M + NT - 1) / NT;
  const long long pairs = static_cast<long long>(a.tiles_m) * ((a.N + 2 * GF_ROWS - 1) / (2 * GF_ROWS));
  if (pairs >= (1LL << 30)) return ERR_UNSUPPORTED;
  auto kernel = gemm_f32_tc_kernel<NT>;
  if (cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM_BYTES))) return ERR_CUDA;
  return launch_dependent(kernel, dim3(static_cast<unsigned>(2 * pairs)), dim3(Shape::THREADS), Shape::SMEM_BYTES, stream, false, a);
}

}  // namespace zb

using namespace zb;

// y = x * w^T, all float32.  x: [M, K] rows ldx apart; w: [N, K] rows ldw apart; y: [M, N] rows ldy apart.  Rows on 16-byte boundaries
// (K, ldx and ldw multiples of 4) run on the tensor cores, others on multiply-adds (gemm_simt.cu).
ZB_API int zb_gemm_nt_f32(float* y, const float* x, const float* w, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                          int* status, void* stream) {
  if (M < 0 || N < 0 || K <= 0 || ldx < K || ldw < K || ldy < N) return ERR_BAD_ARGUMENT;
  if (M == 0 || N == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if ((M + 63LL) / 64 > 65535) return ERR_UNSUPPORTED;
  if (K % 4 != 0 || ldx % 4 != 0 || ldw % 4 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0 || reinterpret_cast<uintptr_t>(w) % 16 != 0)
    return zb_gemm_nt_simt(y, x, w, M, N, K, ldx, ldw, ldy, DTYPE_F32, DTYPE_F32, stream);
  GemmF32Args a;
  a.y = y; a.x = x; a.w = w; a.M = M; a.N = N; a.K = K; a.ldx = ldx; a.ldw = ldw; a.ldy = ldy; a.status = status;
  // The tile whose rounds over the pairs of SMs take the least time (us of a full round at K = 1024, whatever K's share of it):
  // 700 x 4096 x 1024 is one round of 64 pairs with 192 columns, 35 us (256: 49, 128: 48, 96: 45); 700 x 1024 x 2048 44 pairs with 64,
  // 35 (32: 59, 96: 36); 2048 x 6144 x 1024 four rounds with 192, 133 (256: 140, 128: 141), all at one time; 8 x 151936 x 1024 with 32, 163.
  struct Tile { int columns, us; };
  constexpr Tile tiles[] = {{32, 17}, {64, 19}, {96, 21}, {128, 23}, {160, 28}, {192, 32}, {256, 46}};
  const long long row_blocks = (N + 2LL * GF_ROWS - 1) / (2 * GF_ROWS);
  int best = 0;
  long long least = 0;
  for (const Tile& tile : tiles) {
    const long long time = ((M + tile.columns - 1LL) / tile.columns * row_blocks + 73) / 74 * tile.us;
    if (best != 0 && time >= least) continue;
    best = tile.columns;
    least = time;
  }
  switch (best) {
    case 256: return gemm_f32_launch<256>(a, s);
    case 192: return gemm_f32_launch<192>(a, s);
    case 160: return gemm_f32_launch<160>(a, s);
    case 128: return gemm_f32_launch<128>(a, s);
    case 96: return gemm_f32_launch<96>(a, s);
    case 64: return gemm_f32_launch<64>(a, s);
    default: return gemm_f32_launch<32>(a, s);
  }
}
