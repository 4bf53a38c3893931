// Y[M, N] = X[M, K] * W[N, K]^T on CUDA cores with float32 multiply-adds: the matrix product of
// the true 32-bit path.  No tensor cores, hence no TF32 or other reduced-precision mode: the
// reference's "float32" linear layers run in TF32 (deps/ttl/src/ops/matmul.cpp:269-271), which is
// exactly what this path exists to avoid.  The order in which an output's K products are summed does
// not depend on M, N or the tile it is made in (rows that start on 16-byte boundaries are summed in four
// chains, others in one, by the strides alone), so a row's result does not depend on the batch around it.  Inputs may be float32 or bfloat16 (read exactly); the output is float32 or the input type.
#include "common.cuh"

namespace zb {

// ---- any alignment, either input type: one chain of multiply-adds in ascending k ------------------
constexpr int GT = 64;      // output tile edge
constexpr int GK = 16;      // K slice
constexpr int GPAD = 4;

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_nt_simt_kernel(TOut* __restrict__ y, const TIn* __restrict__ x, const TIn* __restrict__ w, int M, int N, int K,
                    long long ldx, long long ldw, long long ldy) {
  __shared__ __align__(16) float xs[GK][GT + GPAD];
  __shared__ __align__(16) float ws[GK][GT + GPAD];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * GT, n0 = blockIdx.x * GT;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

  const int lr = threadIdx.x >> 2;          // row of the tile this thread loads (0..63)
  const int lc = (threadIdx.x & 3) * 4;     // first of its 4 columns of the K slice
  for (int k0 = 0; k0 < K; k0 += GK) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = k0 + lc + u;
      const int m = m0 + lr, n = n0 + lr;
      xs[lc + u][lr] = (m < M && k < K) ? to_float(x[static_cast<size_t>(m) * ldx + k]) : 0.0f;
      ws[lc + u][lr] = (n < N && k < K) ? to_float(w[static_cast<size_t>(n) * ldw + k]) : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&xs[k][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[k][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) y[static_cast<size_t>(m) * ldy + n] = from_float<TOut>(acc[i][j]);
    }
  }
}

template <typename TIn, typename TOut>
int gemm_launch(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw,
                long long ldy, cudaStream_t stream) {
  const dim3 grid((N + GT - 1) / GT, (M + GT - 1) / GT);
  if (grid.y > 65535) return ERR_UNSUPPORTED;
  gemm_nt_simt_kernel<TIn, TOut><<<grid, 256, 0, stream>>>((TOut*)y, (const TIn*)x, (const TIn*)w, M, N, K, ldx,
                                                           ldw, ldy);
  return launch_result();
}

// ---- float32 rows that start on 16-byte boundaries, K a multiple of 4 -----------------------------
// Bound by the reads of shared memory beside the multiply-adds, and at few tiles by latency.  A CTA makes a tile of
// BM x BN with VG groups of threads: the slices of VK values of k are dealt to the groups in turn, every group sums
// its own slices in ascending k, and the groups' sums are added in their order at the end.  That order is the same for
// all tile sizes.  Four groups give a CTA eight warps where one group would leave an SM two (88 tiles of 64 x 128 at
// 700 x 1024 x 2048: 137 us, 216 us with the kernel above, 293 us with one group on tiles of 128 x 128), and four
// short chains are closer to the exact sum than one long one (2.9e-7 against 5.7e-7 at K = 1024).
// A thread makes 4 GM x 4 GN outputs as groups of four rows and four columns, so a step of k is GM + GN 16-byte
// reads of shared memory for 8 GM GN paired multiply-adds.  A slice sits in one of two buffers, the next one on its way
// into registers; a lane loads 32 bytes of one row of x or w, neighbouring lanes neighbouring rows, and stores them
// transposed without bank conflicts.
// Measured (us, the kernel above in brackets): 700 x 4096 x 1024 199 (259), 2048 x 6144 x 1024 716 (1017),
// 900 x 1024 x 3072 189 (330).
constexpr int VK = 16;
constexpr int VG = 4;

__device__ __forceinline__ void group_sync(int group, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory");
}

template <int BM, int BN, int GM, int GN>
__global__ void __launch_bounds__(BM / (4 * GM) * (BN / (4 * GN)) * VG)
gemm_nt_vec_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ w, int M, int N, int K,
                   long long ldx, long long ldw, long long ldy) {
  constexpr int THREADS = BM / (4 * GM) * (BN / (4 * GN));     // of a group
  constexpr int ROWS = BM + BN, PIECES = ROWS * (VK / 8), PER = PIECES / THREADS;
  static_assert(PIECES % THREADS == 0 && ROWS % 32 == 0 && THREADS % 32 == 0, "whole pieces a thread");
  extern __shared__ __align__(16) float g_smem[];
  const int group = threadIdx.x / THREADS, tid = threadIdx.x % THREADS;
  float* s = g_smem + group * (2 * VK * ROWS);
  const int lane = tid & 31, warp = tid >> 5;
  constexpr int WX = BN / (4 * GN * 8);
  const int tx = warp % WX * 8 + (lane & 7), ty = warp / WX * 4 + (lane >> 3);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const float* src[PER];
  float4 staged[PER][2];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int p = tid + i * THREADS, r = p % ROWS, k = p / ROWS * 8;
    const bool of_x = r < BM;
    const int at = of_x ? m0 + r : n0 + r - BM;
    src[i] = at < (of_x ? M : N) ? (of_x ? x + at * ldx : w + at * ldw) + k : nullptr;
  }
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < PER; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int k = k0 + (tid + i * THREADS) / ROWS * 8 + 4 * half;
        staged[i][half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (src[i] != nullptr && k < K) staged[i][half] = *reinterpret_cast<const float4*>(src[i] + k0 + 4 * half);
      }
  };
  auto store = [&](int buffer) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int p = tid + i * THREADS, r = p % ROWS, k = p / ROWS * 8;
      float* to = s + (buffer * VK + k) * ROWS + r;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        to[(4 * half) * ROWS] = staged[i][half].x;
        to[(4 * half + 1) * ROWS] = staged[i][half].y;
        to[(4 * half + 2) * ROWS] = staged[i][half].z;
        to[(4 * half + 3) * ROWS] = staged[i][half].w;
      }
    }
  };
  float acc[4 * GM][4 * GN];
#pragma unroll
  for (int i = 0; i < 4 * GM; ++i)
#pragma unroll
    for (int j = 0; j < 4 * GN; ++j) acc[i][j] = 0.0f;
  fetch(group * VK);
  store(0);
  group_sync(group, THREADS);
  int buffer = 0;
  for (int k0 = group * VK; k0 < K; k0 += VG * VK) {
    const bool more = k0 + VG * VK < K;
    if (more) fetch(k0 + VG * VK);
#pragma unroll
    for (int k = 0; k < VK; ++k) {
      float a[4 * GM], b[4 * GN];
      const float* row = s + (buffer * VK + k) * ROWS;
#pragma unroll
      for (int g = 0; g < GM; ++g) *reinterpret_cast<float4*>(&a[4 * g]) = *reinterpret_cast<const float4*>(row + g * (BM / GM) + ty * 4);
#pragma unroll
      for (int g = 0; g < GN; ++g) *reinterpret_cast<float4*>(&b[4 * g]) = *reinterpret_cast<const float4*>(row + BM + g * (BN / GN) + tx * 4);
#pragma unroll
      for (int i = 0; i < 4 * GM; ++i) {
        unsigned long long twice;
        asm("mov.b64 %0, {%1, %1};" : "=l"(twice) : "f"(a[i]));
#pragma unroll
        for (int j = 0; j < 2 * GN; ++j) {
          unsigned long long& pair = *reinterpret_cast<unsigned long long*>(&acc[i][2 * j]);
          asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(pair) : "l"(twice), "l"(*reinterpret_cast<unsigned long long*>(&b[2 * j])));
        }
      }
    }
    if (more) store(buffer ^ 1);
    group_sync(group, THREADS);
    buffer ^= 1;
  }
  // The groups' tiles side by side, then their sums in group order.
  __syncthreads();
  float* part = g_smem + group * (BM * BN);
#pragma unroll
  for (int i = 0; i < 4 * GM; ++i)
#pragma unroll
    for (int g = 0; g < GN; ++g)
      *reinterpret_cast<float4*>(part + (i / 4 * (BM / GM) + ty * 4 + i % 4) * BN + g * (BN / GN) + tx * 4) =
          *reinterpret_cast<const float4*>(&acc[i][4 * g]);
  __syncthreads();
  const bool vectors = ldy % 4 == 0 && reinterpret_cast<uintptr_t>(y) % 16 == 0;
  for (int e = threadIdx.x; e < BM * BN / 4; e += THREADS * VG) {
    const int m = m0 + e / (BN / 4), n = n0 + e % (BN / 4) * 4;
    if (m >= M || n >= N) continue;
    float4 v = *reinterpret_cast<const float4*>(g_smem + e * 4);
#pragma unroll
    for (int g = 1; g < VG; ++g) {
      const float4 o = *reinterpret_cast<const float4*>(g_smem + g * (BM * BN) + e * 4);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    float* p = y + m * ldy + n;
    if (vectors && n + 3 < N) {
      *reinterpret_cast<float4*>(p) = v;
    } else {
      p[0] = v.x;
      if (n + 1 < N) p[1] = v.y;
      if (n + 2 < N) p[2] = v.z;
      if (n + 3 < N) p[3] = v.w;
    }
  }
}

template <int BM, int BN, int GM, int GN>
int gemm_vec_launch(float* y, const float* x, const float* w, int M, int N, int K, long long ldx, long long ldw, long long ldy,
                    cudaStream_t stream) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return ERR_UNSUPPORTED;
  constexpr int smem = 4 * VG * (2 * VK * (BM + BN) > BM * BN ? 2 * VK * (BM + BN) : BM * BN);
  auto kernel = gemm_nt_vec_kernel<BM, BN, GM, GN>;
  if (smem > 48 * 1024 && cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) return ERR_CUDA;
  kernel<<<grid, BM / (4 * GM) * (BN / (4 * GN)) * VG, smem, stream>>>(y, x, w, M, N, K, ldx, ldw, ldy);
  return launch_result();
}

}  // namespace zb

using namespace zb;

// y = x * w^T.  x: [M, K] rows ldx apart; w: [N, K] rows ldw apart; y: [M, N] rows ldy apart.
ZB_API int zb_gemm_nt_simt(void* y, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw,
                           long long ldy, int in_dtype, int out_dtype, void* stream) {
  if (M < 0 || N < 0 || K <= 0 || ldx < K || ldw < K || ldy < N) return ERR_BAD_ARGUMENT;
  if (M == 0 || N == 0) return OK;
  auto s = static_cast<cudaStream_t>(stream);
  if (in_dtype == DTYPE_F32 && out_dtype == DTYPE_F32) {
    const bool vectors = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(w) % 16 == 0;
    auto yf = static_cast<float*>(y);
    auto xf = static_cast<const float*>(x), wf = static_cast<const float*>(w);
    if (!vectors) return gemm_launch<float, float>(y, x, w, M, N, K, ldx, ldw, ldy, s);
    // The tile whose rounds over the SMs take the least time: a round costs (us at K = 1024, whatever K's share of
    // it) 65 with tiles of 64 x 128, 50 with 64 x 96, 44 with 64 x 64, 30 with 32 x 64 and 18 with 32 x 32, which are
    // one CTA an SM or as good as one.  (us, here / with the largest or the smallest tile alone: 700 x 6144 x 1024
    // 249 / 264; 700 x 1024 x 2048, one round of 64 x 96 instead of one of the largest on 88 SMs, 102 / 137;
    // 500 x 1024 x 2048 90 / 133, 300 x 1024 x 2048 89 / 100, 128 x 4096 x 1024 47 / 68, 64 x 4096 x 1024 32 / 36,
    // 1500 x 1024 x 2048 196 / 255, 8 x 151936 x 1024 388 / 430.)
    struct Tile { int m, n, us; };
    constexpr Tile tiles[5] = {{64, 128, 65}, {64, 96, 50}, {64, 64, 44}, {32, 64, 30}, {32, 32, 18}};
    int best = 0;
    long long least = 0;
    for (int t = 0; t < 5; ++t) {
      const int down = (M + tiles[t].m - 1) / tiles[t].m;
      if (t > 0 && down > 65535) continue;  // a grid holds no more
      const long long units = static_cast<long long>(down) * ((N + tiles[t].n - 1) / tiles[t].n);
      const long long time = (units + 147) / 148 * tiles[t].us;
      if (t == 0 || time < least) {
        best = t;
        least = time;
      }
    }
    switch (best) {
      case 0: return gemm_vec_launch<64, 128, 2, 4>(yf, xf, wf, M, N, K, ldx, ldw, ldy, s);
      case 1: return gemm_vec_launch<64, 96, 2, 3>(yf, xf, wf, M, N, K, ldx, ldw, ldy, s);
      case 2: return gemm_vec_launch<64, 64, 2, 2>(yf, xf, wf, M, N, K, ldx, ldw, ldy, s);
      case 3: return gemm_vec_launch<32, 64, 1, 2>(yf, xf, wf, M, N, K, ldx, ldw, ldy, s);
      default: return gemm_vec_launch<32, 32, 1, 1>(yf, xf, wf, M, N, K, ldx, ldw, ldy, s);
    }
  }
  if (in_dtype == DTYPE_BF16 && out_dtype == DTYPE_F32)
    return gemm_launch<__nv_bfloat16, float>(y, x, w, M, N, K, ldx, ldw, ldy, s);
  if (in_dtype == DTYPE_BF16 && out_dtype == DTYPE_BF16)
    return gemm_launch<__nv_bfloat16, __nv_bfloat16>(y, x, w, M, N, K, ldx, ldw, ldy, s);
  return ERR_BAD_ARGUMENT;
}
