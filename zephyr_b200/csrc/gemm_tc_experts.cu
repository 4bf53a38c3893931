// The products of a routed feed-forward on the fifth-generation tensor cores: y[place] = x[place] w[expert]^T for tokens sorted by
// expert, in one launch, with silu(gate) * up (or its likes) where the sums are read out.
//
// A product is bound by its experts' matrices, so their rows take the tensor core's row side, 256 on a pair of SMs
// (cta_group::2), and a run of one expert's tokens the other, up to 256: every matrix is fetched once, none of its rows is
// multiplied with a tile of padding, and a CTA fetches its 128 rows of w beside half of the run's rows of x.  (With the tokens on
// the 128-row side, tiles of 128 x 256, a run of 173 tokens was two tiles that each fetched w: 777 tokens, 4 of 16 experts, 2048
// wide, 3072 / 1536 rows: 67 and 38 us, bound by 590 and 295 MB from L2.  One SM a tile of 128 rows of w x run, 503 and
// 250 MB: 67 and 37; on pairs, 344 and 172 MB, 43
// and 26.  The matrices alone take 31 and 15 us at the copy rate; three rounds of 74 pairs for 2.6 rounds of work cost 14 %.)
// Persistent: a pair takes (256 rows of w, run) in turn, the runs of one expert next to each other in time.  Roles of a CTA's ten warps:
//   * warp 0, one thread: per 64 elements of K a tiled copy of its 128 rows of w and one for every 32 of its half of the run's rows
//     of x into the next stage of a ring (128-byte swizzle; what lies beyond a matrix comes as zeros, what lies beyond a run is
//     another run's and ends in columns that are not written), the bytes counted on the first CTA's barrier;
//   * warp 1 of the first CTA: four products 256 x run x 16 a stage into one of two accumulators in both CTAs' tensor memory, issued
//     by an elected lane;
//   * warps 2..9: a thread owns a row of w (its TMEM lane) and reads 32 tokens' sums at a time, every other 32 of them.  A warp's outputs for 32 tokens
//     go through shared memory to 16-byte stores.
// x [places, K], w [experts * N, K], y [places, N or N / 2], all bfloat16; N a multiple of 8 (16 where gated), K of 8.
// Every wait is bounded and reports instead of hanging; tensor memory is given back on every path.
#include "common.cuh"
#include "mma.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace zb {

bool matrix_tensor_map(const void* base, long long rows, int cols, long long ld, int box_rows, CUtensorMap* out,
                       int element_bytes);       // gemm_tc.cu

constexpr int GX_BK = 64;                 // elements of K per stage: one 128-byte swizzled row
constexpr int GX_THREADS = 320;
constexpr int GX_WAIT_LIMIT = 1 << 18;
constexpr int GX_MAX_STAGES = 10;
constexpr int GX_W_BYTES = 128 * GX_BK * 2;
constexpr int GX_X_BOX = 32;              // rows of x per copy
constexpr int GX_STAGING = 32 * 80;       // an epilogue warp's 32 tokens x 32 outputs, rows 80 bytes apart

// RUN: the longest run of a launch.  Shorter runs leave room for more stages.
template <int RUN> struct ExpertsShape {
  static constexpr int STAGE_BYTES = GX_W_BYTES + RUN / 2 * GX_BK * 2;
  static constexpr int STAGES = 200 * 1024 / STAGE_BYTES;               // 256: 6, 128: 8, 64: 10
  static_assert(STAGES <= GX_MAX_STAGES, "a barrier of each kind a stage");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 8 * GX_STAGING + 1024;
};

struct ExpertsTcArgs {
  CUtensorMap w_map;             // w as [experts * N][K]; box 64 x 128
  CUtensorMap x_map;             // x as [places][K]; box 64 x 32
  __nv_bfloat16* y;
  long long ldy;
  int N, K, row_blocks;          // row_blocks: of 256 rows of an expert's matrix
  const int* plan;               // [0] runs; then per run its expert, first place and number of places that count
  GateForm gate;
  int* status;
};

struct ExpertsShared {
  unsigned long long full[GX_MAX_STAGES], empty[GX_MAX_STAGES], acc_full[2], acc_empty[2];
  unsigned tmem_base;
  volatile int failed;
};

__device__ __forceinline__ bool gx_wait(ExpertsShared& sh, unsigned long long* bar, unsigned parity) {
  for (int i = 0; i < GX_WAIT_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255) == 255 && sh.failed) return false;
  }
  return false;
}

// GATED: w's rows come in blocks of 8 gates and their 8 ups; y has N / 2 columns.  SCALED: both sums of a place times
// gate.row_scale[place] first.
template <int RUN, bool GATED, bool SCALED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GX_THREADS, 1) gemm_tc_experts_kernel(const __grid_constant__ ExpertsTcArgs a) {
  using Shape = ExpertsShape<RUN>;
  extern __shared__ unsigned char gx_smem_raw[];
  __shared__ ExpertsShared sh;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(gx_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_blocks = (a.K + GX_BK - 1) / GX_BK;
  const int rank = static_cast<int>(cluster_rank()), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Shape::STAGES; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh.acc_full[b], 1);
      mbar_init(&sh.acc_empty[b], 16);               // eight epilogue warps in each CTA
    }
    sh.failed = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&sh.tmem_base, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                               // both CTAs' barriers and tensor memory are there
  tc_fence_after_sync();
  const unsigned tmem_base = sh.tmem_base;
  wait_for_prior_grids();
  let_dependents_launch();
  const int runs = a.plan[0], items = runs * a.row_blocks;
  // The product's columns: a run's places up to a multiple of 64, half of them in each CTA.
  auto half_columns = [](int rows) { return (rows + 63) / 64 * 32; };

  if (warp == 0) {
    // A copy a lane: lane 0 the rows of w, the lanes behind it 32 of the run's rows each (one lane issuing all of them one after the
    // other held the stages up: runs of 173, 2048 wide 47 us, of 250, 1024 wide 21.7; now 45 and 18.6.  Fewer stages change neither).
    int stage = 0;
    unsigned phase = 0;
    for (int item = pair; item < items; item += pairs) {
      const int* run = a.plan + 1 + 3 * (item % runs);
      const int half = half_columns(run[2]), boxes = half / GX_X_BOX, box = lane - 1;
      const int row = lane == 0 ? run[0] * a.N + item / runs * 256 + 128 * rank : run[1] + half * rank + box * GX_X_BOX;
      const unsigned offset = lane == 0 ? 0 : GX_W_BYTES + box * GX_X_BOX * GX_BK * 2;
      const CUtensorMap* map = lane == 0 ? &a.w_map : &a.x_map;
      bool ok = true;
      for (int kb = 0; kb < k_blocks; ++kb) {
        ok = __all_sync(0xffffffffu, gx_wait(sh, &sh.empty[stage], phase ^ 1));
        if (!ok) break;
        if (rank == 0 && lane == 0) mbar_arrive_expect_tx(&sh.full[stage], 2 * (GX_W_BYTES + boxes * GX_X_BOX * GX_BK * 2));
        if (lane <= boxes)
          tiled_copy_2d_g2s_pair(ring + stage * Shape::STAGE_BYTES + offset, map, kb * GX_BK, row, in_cta_of_rank(smem_u32(&sh.full[stage]), 0));
        if (++stage == Shape::STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        if (lane == 0 && !sh.failed) report(a.status, STATUS_COPY_TIMEOUT, item, stage);
        sh.failed = 1;
        break;
      }
    }
  } else if (warp == 1 && rank == 0) {
    const bool leader = elect_one();
    int stage = 0, acc = 0;
    unsigned phase = 0, acc_phase = 0;
    for (int item = pair; item < items; item += pairs) {
      const unsigned idesc = tc_idesc_pair(2 * half_columns(a.plan[3 + 3 * (item % runs)]));
      bool ok = __all_sync(0xffffffffu, gx_wait(sh, &sh.acc_empty[acc], acc_phase ^ 1));
      if (!ok && leader && !sh.failed) report(a.status, STATUS_BARRIER_TIMEOUT, item, -1);
      tc_fence_after_sync();
      const unsigned d = tmem_base + acc * 256;
      for (int kb = 0; kb < k_blocks && ok; ++kb) {
        ok = __all_sync(0xffffffffu, gx_wait(sh, &sh.full[stage], phase));
        if (!ok) {
          if (leader && !sh.failed) report(a.status, STATUS_COPY_TIMEOUT, item, -2 - kb);
          break;
        }
        tc_fence_after_sync();
        const unsigned slot = smem_u32(ring + stage * Shape::STAGE_BYTES);
        const unsigned long long w_desc = desc_k_major(slot), x_desc = desc_k_major(slot + GX_W_BYTES);
        if (leader) {
#pragma unroll
          for (int k = 0; k < GX_BK / 16; ++k) tc_mma_pair(d, w_desc + 2 * k, x_desc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          tc_commit_pair(&sh.empty[stage]);
          if (kb + 1 == k_blocks) tc_commit_pair(&sh.acc_full[acc]);
        }
        if (++stage == Shape::STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) {
        sh.failed = 1;
        break;
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  } else if (warp > 1) {
    const int quarter = warp & 3;                   // the TMEM lanes this warp may read: 32 quarter .. + 31
    unsigned char* staging = ring + Shape::STAGES * Shape::STAGE_BYTES + (warp - 2) * GX_STAGING;
    constexpr int OUTPUTS = GATED ? 16 : 32;        // of a warp, a token
    constexpr int PIECES = OUTPUTS / 8;             // 16-byte pieces of them
    const int width = GATED ? a.N / 2 : a.N;
    const bool holds_gate = (lane & 8) == 0;
    int acc = 0;
    unsigned acc_phase = 0;
    for (int item = pair; item < items; item += pairs) {
      const int* run = a.plan + 1 + 3 * (item % runs);
      const int place0 = run[1], rows = run[2];
      const int column0 = (item / runs * 256 + 128 * rank + 32 * quarter) / (GATED ? 2 : 1);
      if (!__all_sync(0xffffffffu, gx_wait(sh, &sh.acc_full[acc], acc_phase))) {
        if (lane == 0 && !sh.failed) report(a.status, STATUS_BARRIER_TIMEOUT, item, -3);
        sh.failed = 1;
        break;
      }
      tc_fence_after_sync();
      const unsigned tmem_row = tmem_base + (static_cast<unsigned>(32 * quarter) << 16) + acc * 256;
      for (int c = 32 * (warp > 5); c < rows; c += 64) {          // (columns beyond the product's are read and not used)
        unsigned v[32];
        tmem_ld32(tmem_row + c, v);
        tmem_wait_ld32(v);
        __nv_bfloat16* mine = reinterpret_cast<__nv_bfloat16*>(staging) + (GATED ? (lane >> 4) * 8 + (lane & 7) : lane);
        if (GATED) {
          // Lane l holds the gates, lane l + 8 their ups of 32 tokens: the first finishes 16 of them, the second the others.
          const float* scale = SCALED ? a.gate.row_scale + place0 + c + (holds_gate ? 0 : 16) : nullptr;
          auto finish = [&](auto activation) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const unsigned other = __shfl_xor_sync(0xffffffffu, holds_gate ? v[16 + i] : v[i], 8);
              float gate = __uint_as_float(holds_gate ? v[i] : other), up = __uint_as_float(holds_gate ? other : v[16 + i]);
              if (SCALED) {
                const float s = c + (holds_gate ? 0 : 16) + i < rows ? scale[i] : 0.0f;
                gate *= s;
                up *= s;
              }
              mine[((holds_gate ? 0 : 16) + i) * 40] = __float2bfloat16_rn(activation(gate, up));
            }
          };
          if (a.gate.kind == GATE_SILU) finish([](float gate, float up) { return silu_fast(gate) * up; });
          else if (a.gate.kind == GATE_RELU) finish([](float gate, float up) { return fmaxf(gate, 0.0f) * up; });
          else finish([&](float gate, float up) { return bounded_gate<true>(gate, up, a.gate); });
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) mine[i * 40] = __float2bfloat16_rn(__uint_as_float(v[i]));
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          const int token = i * (32 / PIECES) + lane / PIECES, piece = lane % PIECES;
          if (c + token < rows && column0 + piece * 8 < width)
            *reinterpret_cast<uint4*>(a.y + static_cast<size_t>(place0 + c + token) * a.ldy + column0 + piece * 8) =
                *reinterpret_cast<const uint4*>(staging + token * 80 + piece * 16);
        }
        __syncwarp();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_in_cluster(in_cta_of_rank(smem_u32(&sh.acc_empty[acc]), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  // Both CTAs meet here on every path (the other's barriers and tensor memory are used until then), and the warps that took the
  // tensor memory give it back.
  tc_fence_before_sync();
  __syncthreads();
  if (sh.failed) let_copies_land();                 // (they count on the first CTA's barriers)
  __syncwarp();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

template <int RUN, bool GATED, bool SCALED>
int experts_launch(const ExpertsTcArgs& a, int max_runs, int sms, cudaStream_t stream) {
  using Shape = ExpertsShape<RUN>;
  auto kernel = gemm_tc_experts_kernel<RUN, GATED, SCALED>;
  if (cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM_BYTES))) return ERR_CUDA;
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(GX_THREADS);
  config.dynamicSmemBytes = Shape::SMEM_BYTES;
  config.stream = stream;
  config.gridDim = dim3(2 * (sms / 2));
  int clusters = 0;                                 // how many pairs the device holds at once
  if (cuda_failed(cudaOccupancyMaxActiveClusters(&clusters, kernel, &config)) || clusters <= 0) return ERR_CUDA;
  const long long items = static_cast<long long>(max_runs) * a.row_blocks;
  config.gridDim = dim3(2 * static_cast<unsigned>(items < clusters ? items : clusters));
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = dependent_launch_enabled() ? 1 : 0;
  return cuda_failed(cudaLaunchKernelEx(&config, kernel, a)) ? ERR_CUDA : launch_result();
}
template <int RUN>
int experts_run_launch(const ExpertsTcArgs& a, int max_runs, bool gated, int sms, cudaStream_t stream) {
  if (!gated) return experts_launch<RUN, false, false>(a, max_runs, sms, stream);
  return a.gate.row_scale != nullptr ? experts_launch<RUN, true, true>(a, max_runs, sms, stream)
                                     : experts_launch<RUN, true, false>(a, max_runs, sms, stream);
}

}  // namespace zb

using namespace zb;

// The longest run for this many choices and experts: the smallest of the kernel's forms that holds the average run with room for
// its spread (a run that is longer all the same is cut in two, and its expert's matrix fetched twice).
ZB_API int zb_gemm_tc_experts_run(int choices, int experts) {
  const int average = experts > 0 ? (choices + experts - 1) / experts : 0;
  return average <= 48 ? 64 : average <= 104 ? 128 : 256;
}

// y = x w^T over the runs of `plan` (zb_route_align_runs with the same `run`).  kind: 0 the sums; 1 silu(gate) * up, 2 max(gate, 0) * up,
// 3 the bounded gate (`limit`, `alpha`, `shift`).  `row_scale`: null, or one float32 per place (kinds 1 and 2).
ZB_API int zb_gemm_tc_experts(void* y, const void* x, const void* w, const int* plan, int max_runs, int run, int places, int experts,
                              int N, int K, long long ldx, long long ldy, int kind, const float* row_scale, float limit, float alpha,
                              float shift, int* status, void* stream) {
  const bool gated = kind != 0;
  if (max_runs <= 0 || places <= 0 || experts <= 0 || N <= 0 || K <= 0 || plan == nullptr || kind < 0 || kind > 3 || (run != 64 && run != 128 && run != 256) ||
      N % (gated ? 16 : 8) != 0 || K % 8 != 0 || ldx % 8 != 0 || ldx < K || ldy % 8 != 0 || ldy < (gated ? N / 2 : N) ||
      (kind == 3 && (row_scale != nullptr || !(limit > 0.0f))) || (kind == 0 && row_scale != nullptr) ||
      reinterpret_cast<uintptr_t>(y) % 16 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0 || reinterpret_cast<uintptr_t>(w) % 16 != 0)
    return ERR_BAD_ARGUMENT;
  int device = 0, sms = 0;
  if (cuda_failed(cudaGetDevice(&device)) || cuda_failed(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device))) return ERR_CUDA;
  ExpertsTcArgs a;
  a.y = static_cast<__nv_bfloat16*>(y);
  a.ldy = ldy;
  a.N = N; a.K = K;
  a.row_blocks = (N + 255) / 256;
  a.plan = plan;
  a.gate = kind == 3 ? GateForm{GATE_BOUNDED, nullptr, limit, alpha, shift, nullptr} : plain_gate(kind == 2 ? GATE_RELU : GATE_SILU);
  a.gate.row_scale = row_scale;
  a.status = status;
  if (static_cast<long long>(experts) * N >= (1LL << 31)) return ERR_UNSUPPORTED;
  if (!matrix_tensor_map(w, static_cast<long long>(experts) * N, K, K, 128, &a.w_map, 2) ||
      !matrix_tensor_map(x, places, K, ldx, GX_X_BOX, &a.x_map, 2))
    return ERR_CUDA;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  return run == 64 ? experts_run_launch<64>(a, max_runs, gated, sms, s)
         : run == 128 ? experts_run_launch<128>(a, max_runs, gated, sms, s) : experts_run_launch<256>(a, max_runs, gated, sms, s);
}
