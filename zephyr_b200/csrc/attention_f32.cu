// Paged causal attention of the true 32-bit path for rows that bring several tokens: float32 multiply-adds on CUDA
// cores, as the general kernel (attention_simt.cu) does them, in tiles whose operands are used from registers.
//
// The general kernel reads one key value per lane and multiply-add from shared memory; here a CTA takes F_ROWS query
// rows (the (token, head) pairs of neighbouring tokens and one key/value head) against F_KEYS keys at a time, a thread
// 4 x 4 scores and 4 x D/16 outputs, so that a 16-byte read serves 8 to 11 multiply-adds, two of them an instruction.
// Bound at few tiles by the serial chain of the tile that sees most keys, alone on its SM: of 10 us a step of 64 keys the
// scores take 4, the weighted values 3, the rest barriers, exponentials and shuffles.  Two CTAs an SM are worth
// more than registers at long prompts (4000 tokens 1699 us, 2086 with one CTA of 212 registers).  Keys lie transposed
// ([channel][key]), values as they are; a warp owns eight rows across all keys, so the weights go from one product
// to the other inside a warp.  A weight of zero skips its value; a tile of which a warp sees every key needs no look at
// that.  Where a key lies in the cache is worked out once, by the lane that fetches it, and read from shared memory for
// its value (eight divisions and table reads a thread otherwise: 700 tokens 148 us against 125).  A lane sums the weights of its own
// keys and the lanes' sums meet at the end (125 us against 122).
// 700 tokens, 16 heads over 8 of 128: 122 us (one multiply-add an instruction and every value's place worked out 167, the
// general kernel 776); 4000 tokens 1678 (2241).  Every row with several tokens runs here, so that its result hangs on
// that row alone: two tokens behind a context of 600 take 97 us (136; the general kernel 328), two tokens of a new prompt,
// most of whose tile is empty, 16.6 (18.6; 16), eight rows of sixteen 23 (25; 37).
//
// Masks: causal, a window, a chunk (key and query in the same run of `chunk` positions); `sinks` join the softmax's
// denominators; `softcap` > 0 bounds the scaled scores.  Keys and values have one width, a multiple of 4 up to 128.
#include <initializer_list>
#include <type_traits>

#include "common.cuh"
#include "mma.cuh"

namespace zb {

constexpr int F_ROWS = 64;      // (token, head) pairs of a CTA
constexpr int F_KEYS = 64;      // keys of a tile
constexpr int F_THREADS = 256;

// to[0..3] += a * b[0..3], two multiply-adds an instruction.
__device__ __forceinline__ void multiply_add(float* to, float a, const float* b) {
  unsigned long long twice;
  asm("mov.b64 %0, {%1, %1};" : "=l"(twice) : "f"(a));
#pragma unroll
  for (int pair = 0; pair < 2; ++pair)
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(*reinterpret_cast<unsigned long long*>(to + 2 * pair))
        : "l"(twice), "l"(*reinterpret_cast<const unsigned long long*>(b + 2 * pair)));
}

struct AttentionF32Args {
  const float* q;           // [T, nh * d]
  float* out;               // [T, nh * d]
  const float* kv_cache;    // pages {[nkv][page_size][d] keys, the same of values}
  const int* block_table;   // [R, max_blocks]
  const int* tile_row;      // [n_tiles], by the number of keys a tile sees, fewest first
  const int* tile_q0;
  const int* row_q_start;
  const int* row_q_len;
  const int* row_ctx;
  int max_blocks, page_size, num_pages, num_rows, n_tiles;
  int nh, nkv, d, window, chunk, tile_tokens, cta_tokens, subs;
  float scale, softcap;
  const float* sinks;       // null, or [nh]
  int* status;
};

// D: the padded width, 64 or 128.
template <int D>
__global__ void __launch_bounds__(F_THREADS, 2) paged_attention_f32_kernel(const AttentionF32Args a) {
  extern __shared__ __align__(16) float f_smem[];
  float* q_s = f_smem;                        // [D][F_ROWS]
  float* k_s = q_s + D * F_ROWS;              // [D][F_KEYS]
  float* v_s = k_s + D * F_KEYS;              // [F_KEYS][D]
  float* p_s = v_s + F_KEYS * D;              // [F_KEYS][F_ROWS]
  auto base_s = reinterpret_cast<long long*>(p_s + F_KEYS * F_ROWS);   // [F_KEYS]: where a key begins in the cache, or -1
  constexpr int VG4 = D / 64;                 // groups of four output columns a thread
  constexpr int K_PER = F_KEYS * (D / 8) / F_THREADS;      // 32-byte pieces of a key tile a thread moves
  // The last tiles of the list see the most keys and run first.
  const int kvh = blockIdx.x % a.nkv, at = blockIdx.x / a.nkv;
  const int tile = a.n_tiles - 1 - at / a.subs, sub = a.subs - 1 - at % a.subs;
  const int row = a.tile_row[tile], q0 = a.tile_q0[tile] + sub * a.cta_tokens;
  if (row < 0 || row >= a.num_rows) {
    if (threadIdx.x == 0) report(a.status, STATUS_ROW_OUT_OF_RANGE, row, tile);
    return;
  }
  const int g = a.nh / a.nkv, d = a.d, tid = threadIdx.x;
  const int n_tok = min(min(a.cta_tokens, a.tile_tokens - sub * a.cta_tokens), a.row_q_len[row] - q0);
  if (n_tok <= 0) return;
  const int ctx = a.row_ctx[row], tok0 = a.row_q_start[row] + q0, rows = n_tok * g;
  const int tx = tid & 15, ty = tid >> 4;
  const int chunks = d / 4;                   // 16-byte pieces of a row

  // Queries, transposed: lanes take neighbouring rows.
  for (int e = tid; e < F_ROWS * (D / 4); e += F_THREADS) {
    const int r = e % F_ROWS, c = e / F_ROWS;
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (r < rows && c < chunks)
      x = *reinterpret_cast<const float4*>(a.q + (static_cast<size_t>(tok0 + r / g) * a.nh + kvh * g + r % g) * d + 4 * c);
    q_s[(4 * c) * F_ROWS + r] = x.x;
    q_s[(4 * c + 1) * F_ROWS + r] = x.y;
    q_s[(4 * c + 2) * F_ROWS + r] = x.z;
    q_s[(4 * c + 3) * F_ROWS + r] = x.w;
  }
  // Keys any row of this CTA may see: [lo, hi).
  const int hi = ctx + q0 + n_tok;
  int lo = a.window > 0 ? max(0, ctx + q0 - a.window + 1) : 0;
  if (a.chunk > 0) lo = max(lo, (ctx + q0) / a.chunk * a.chunk);
  const size_t page_elems = static_cast<size_t>(2) * a.nkv * a.page_size * d;
  const size_t value_part = static_cast<size_t>(a.nkv) * a.page_size * d;
  const int* table = a.block_table + static_cast<size_t>(row) * a.max_blocks;

  // Where position `pos` of this head begins in the cache; false outside [lo, hi) (its rows are zeros) or if its page
  // is none (reported).
  auto locate = [&](int pos, size_t& base) -> bool {
    if (pos < lo || pos >= hi) return false;
    const int block = pos / a.page_size;
    const int page = block < a.max_blocks ? table[block] : -1;
    if (page <= 0 || page >= a.num_pages) {
      report(a.status, STATUS_PAGE_OUT_OF_RANGE, page, tok0);
      return false;
    }
    base = page * page_elems + (static_cast<size_t>(kvh) * a.page_size + pos % a.page_size) * d;
    return true;
  };
  // A key tile on its way through registers: piece p is 8 channels (p / F_KEYS) of key p % F_KEYS.
  float4 staged[K_PER][2];
  auto fetch_keys = [&](int k0) {
    size_t base = 0;
    const int pos = k0 + tid % F_KEYS;        // F_THREADS is a multiple of F_KEYS: one key a thread
    const bool ok = locate(pos, base);
    const int turn = kv_swizzle(pos, chunks);
    if (tid < F_KEYS) base_s[tid] = ok ? static_cast<long long>(base) : -1;
#pragma unroll
    for (int i = 0; i < K_PER; ++i)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int c = (tid + i * F_THREADS) / F_KEYS * 2 + half;
        staged[i][half] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (ok && c < chunks) staged[i][half] = *reinterpret_cast<const float4*>(a.kv_cache + base + 4 * (c ^ turn));
      }
  };
  auto store_keys = [&]() {
#pragma unroll
    for (int i = 0; i < K_PER; ++i) {
      float* to = k_s + (tid + i * F_THREADS) / F_KEYS * 8 * F_KEYS + tid % F_KEYS;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        to[(4 * half) * F_KEYS] = staged[i][half].x;
        to[(4 * half + 1) * F_KEYS] = staged[i][half].y;
        to[(4 * half + 2) * F_KEYS] = staged[i][half].z;
        to[(4 * half + 3) * F_KEYS] = staged[i][half].w;
      }
    }
  };
  auto copy_values = [&](int k0) {
    constexpr int per_row = D / 4;
#pragma unroll
    for (int i = 0; i < F_KEYS * per_row / F_THREADS; ++i) {
      const int e = tid + i * F_THREADS, j = e / per_row, c = e % per_row;
      const long long base = base_s[j];
      const bool ok = c < chunks && base >= 0;
      cp_async_16(v_s + j * D + 4 * c, ok ? a.kv_cache + base + value_part + 4 * (c ^ kv_swizzle(k0 + j, chunks)) : a.kv_cache, ok);
    }
    cp_async_commit();
  };

  float m[4], l[4];
  alignas(16) float acc[4][4 * VG4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < 4 * VG4; ++c) acc[i][c] = 0.0f;
  }
  int qpos[4], first[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    qpos[i] = r < rows ? ctx + q0 + r / g : -1;
    first[i] = a.window > 0 ? max(0, qpos[i] - a.window + 1) : 0;
    if (a.chunk > 0) first[i] = max(first[i], qpos[i] / a.chunk * a.chunk);
  }
  const int begin = lo / F_KEYS * F_KEYS;
  fetch_keys(begin);
  for (int k0 = begin; k0 < hi; k0 += F_KEYS) {
    __syncthreads();                          // the tile before is read
    store_keys();
    copy_values(k0);
    __syncthreads();
    alignas(16) float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.0f;
#pragma unroll 16
    for (int c = 0; c < D; ++c) {
      alignas(16) float q4[4], k4[4];
      *reinterpret_cast<float4*>(q4) = *reinterpret_cast<const float4*>(q_s + c * F_ROWS + ty * 4);
      *reinterpret_cast<float4*>(k4) = *reinterpret_cast<const float4*>(k_s + c * F_KEYS + tx * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) multiply_add(s[i], q4[i], k4);
    }
    if (k0 + F_KEYS < hi) fetch_keys(k0 + F_KEYS);
    float corr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kp = k0 + tx * 4 + j;
        s[i][j] *= a.scale;
        if (a.softcap > 0.0f) s[i][j] = a.softcap * tanhf(s[i][j] / a.softcap);
        if (kp > qpos[i] || kp < first[i]) s[i][j] = -INFINITY;
        top = fmaxf(top, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float new_m = fmaxf(m[i], top);
      // (a row that has seen no key yet keeps zeros: its weights are exp(-inf) of a finite difference)
      const float from = new_m == -INFINITY ? 0.0f : new_m;
      corr[i] = expf(m[i] - from);
      float sum = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = expf(s[i][j] - from);
        sum += s[i][j];
      }
      l[i] = fmaf(l[i], corr[i], sum);
      m[i] = new_m;
    }
    bool dense = true;                        // every row of the warp sees every key of the tile
#pragma unroll
    for (int i = 0; i < 4; ++i) dense = dense && s[i][0] > 0.0f && s[i][1] > 0.0f && s[i][2] > 0.0f && s[i][3] > 0.0f;
    dense = __all_sync(0xffffffffu, dense);
    // Weights: a key's groups of four rows are turned by its group of four, so that a warp's stores meet all banks.
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(p_s + (tx * 4 + j) * F_ROWS + ((ty + tx) & 15) * 4) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4 * VG4; ++c) acc[i][c] *= corr[i];
    cp_async_wait<0>();
    __syncthreads();                          // the values have landed; the weights of a row stay within its warp
    auto weigh = [&](auto all) {
#pragma unroll 8
      for (int j = 0; j < F_KEYS; ++j) {
        float p4[4];
        *reinterpret_cast<float4*>(p4) = *reinterpret_cast<const float4*>(p_s + j * F_ROWS + ((ty + j / 4) & 15) * 4);
#pragma unroll
        for (int c = 0; c < VG4; ++c) {
          alignas(16) float v4[4];
          *reinterpret_cast<float4*>(v4) = *reinterpret_cast<const float4*>(v_s + j * D + c * 64 + tx * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (all.value || p4[i] != 0.0f) multiply_add(acc[i] + 4 * c, p4[i], v4);   // (what a row does not see may be anything)
        }
      }
    };
    if (dense) weigh(std::true_type());
    else weigh(std::false_type());
  }
  // A lane has summed the weights of its own keys.
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= rows) continue;
    const int head = kvh * g + r % g;
    float denominator = l[i], keep = 1.0f;
    if (a.sinks != nullptr) {
      // The sink joins the sum as one more exponential: rescale to the larger of the two maxima.
      const float sink = a.sinks[head], top = fmaxf(m[i], sink);
      keep = expf(m[i] - top);
      denominator = l[i] * keep + expf(sink - top);
    }
    const float inv = denominator > 0.0f ? keep / denominator : 0.0f;
    float* to = a.out + (static_cast<size_t>(tok0 + r / g) * a.nh + head) * d;
#pragma unroll
    for (int c = 0; c < VG4; ++c) {
      const int at_d = c * 64 + tx * 4;
      if (at_d < d)
        *reinterpret_cast<float4*>(to + at_d) = make_float4(acc[i][4 * c] * inv, acc[i][4 * c + 1] * inv, acc[i][4 * c + 2] * inv,
                                                            acc[i][4 * c + 3] * inv);
    }
  }
}

template <int D>
static int attention_f32_launch(const AttentionF32Args& a, cudaStream_t s) {
  constexpr int smem = static_cast<int>(sizeof(float)) * (D * F_ROWS + 2 * D * F_KEYS + F_KEYS * F_ROWS) + 8 * F_KEYS;
  auto kernel = paged_attention_f32_kernel<D>;
  if (cuda_failed(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))) return ERR_CUDA;
  kernel<<<dim3(a.n_tiles * a.subs * a.nkv), F_THREADS, smem, s>>>(a);
  return launch_result();
}

}  // namespace zb

using namespace zb;

// 1 if the kernel takes heads of this width and this many query heads per key/value head.
ZB_API int zb_paged_attention_f32_supported(int nh, int nkv, int d) {
  return nh > 0 && nkv > 0 && nh % nkv == 0 && nh / nkv <= F_ROWS && d > 0 && d % 4 == 0 && d <= 128;
}

// Tiles of `tile_tokens` tokens, each cut among CTAs of F_ROWS (token, head) pairs.  q, out and the cache start on
// 16-byte boundaries.
ZB_API int zb_paged_attention_f32(float* out, const float* q, const float* kv_cache, const int* block_table, int max_blocks,
                                  int page_size, int num_pages, int num_rows, const int* tile_row, const int* tile_q0, int n_tiles,
                                  int tile_tokens, const int* row_q_start, const int* row_q_len, const int* row_ctx, int nh, int nkv,
                                  int d, int window, int chunk, float scale, float softcap, const float* sinks, int* status,
                                  void* stream) {
  if (page_size <= 0 || max_blocks <= 0 || n_tiles < 0 || tile_tokens <= 0 || window < 0 || chunk < 0 || softcap < 0.0f)
    return ERR_BAD_ARGUMENT;
  for (const void* p : {static_cast<const void*>(out), static_cast<const void*>(q), static_cast<const void*>(kv_cache)})
    if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return ERR_BAD_ARGUMENT;
  if (!zb_paged_attention_f32_supported(nh, nkv, d)) return ERR_UNSUPPORTED;
  if (n_tiles == 0) return OK;
  AttentionF32Args a;
  a.q = q; a.out = out; a.kv_cache = kv_cache; a.block_table = block_table; a.tile_row = tile_row; a.tile_q0 = tile_q0;
  a.row_q_start = row_q_start; a.row_q_len = row_q_len; a.row_ctx = row_ctx; a.max_blocks = max_blocks; a.page_size = page_size;
  a.num_pages = num_pages; a.num_rows = num_rows; a.n_tiles = n_tiles; a.nh = nh; a.nkv = nkv; a.d = d; a.window = window;
  a.chunk = chunk; a.tile_tokens = tile_tokens; a.cta_tokens = F_ROWS / (nh / nkv);
  a.subs = (tile_tokens + a.cta_tokens - 1) / a.cta_tokens;
  a.scale = scale; a.softcap = softcap; a.sinks = sinks; a.status = status;
  if (static_cast<long long>(n_tiles) * a.subs * nkv > 0x7fffffffLL) return ERR_UNSUPPORTED;
  auto s = static_cast<cudaStream_t>(stream);
  return d <= 64 ? attention_f32_launch<64>(a, s) : attention_f32_launch<128>(a, s);
}
