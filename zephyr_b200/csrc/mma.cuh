// Warp-level tensor-core and asynchronous-copy primitives shared by the attention kernels:
// 16-byte cp.async with zero fill, ldmatrix, and the bf16 m16n8k16 multiply-accumulate.
//
// Fragment layouts of mma.m16n8k16 (lane = 4 * g + t, g = lane / 4, t = lane % 4):
//   A (16x16, row-major): a[0] = (row g,     cols 2t, 2t+1)    a[1] = (row g + 8, cols 2t, 2t+1)
//                         a[2] = (row g,     cols 2t+8, 2t+9)  a[3] = (row g + 8, cols 2t+8, 2t+9)
//   B (16x8, "col"):      b0   = (k 2t, 2t+1; n g)             b1   = (k 2t+8, 2t+9; n g)
//   C (16x8):             c[0], c[1] = (row g, cols 2t, 2t+1)  c[2], c[3] = (row g + 8, cols 2t, 2t+1)
#pragma once

#include "common.cuh"

namespace zb {

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem, bool valid) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int bytes = valid ? 16 : 0;       // 0 bytes read: the 16 destination bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], const void* smem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], const void* smem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
// (Lanes 0 to 15 give the rows' addresses.)
__device__ __forceinline__ void ldmatrix_x2_trans(unsigned (&r)[2], const void* smem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const unsigned*>(&h);
}

// a * b + c of two values in one instruction, each with one rounding.
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\nfma.rn.f32x2 a, a, b, c;\nmov.b64 {%0, %1}, a;\n}\n"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 mul_pair(float2 a, float2 b) {
  float2 r;
  asm("{\n.reg .b64 a, b;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmul.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}\n"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// x and y as three pairs of bfloat16 values whose sums they are (of a value below 2^-110 the bits below 2^-133 are lost), the largest first.  A
// value that would round to infinity keeps the largest bfloat16 as its first part; an infinity's parts are that, itself and a NaN.
__device__ __forceinline__ void three_parts(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
  const float2 minus = make_float2(-1.0f, -1.0f);
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;\n" : "=r"(hi) : "f"(y), "f"(x));
  float2 rest = fma_pair(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus, make_float2(x, y));
  mid = pack_bf16(rest.x, rest.y);
  rest = fma_pair(make_float2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), minus, rest);
  lo = pack_bf16(rest.x, rest.y);
}

// The same of x and y times 2^39 = PARTS_SCALE: all bits of every float32 value below 2^88, also of the smallest; a larger one gives a NaN.
// PARTS_UNSCALE takes a product of two such values back.
constexpr float PARTS_SCALE = 549755813888.0f, PARTS_UNSCALE = 3.308722450212111e-24f;        // 2^39, 2^-78
__device__ __forceinline__ void three_parts_scaled(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
  const float2 scaled = mul_pair(make_float2(x, y), make_float2(PARTS_SCALE, PARTS_SCALE));
  three_parts(scaled.x, scaled.y, hi, mid, lo);
}

// ---- mbarrier and bulk asynchronous copy (the TMA engine, untiled form) -------------------------
__device__ __forceinline__ unsigned smem_u32(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// Makes freshly initialised barriers visible to the asynchronous proxy before any copy names them.
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// Orders this thread's earlier generic-proxy accesses to shared memory before later asynchronous-proxy ones.  (And the compiler's: stores that
// it moved behind the fence would be seen by the tensor cores or the copy engine at some time or other.)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// One arrival that also announces `bytes` of copies to come.
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned done;
  asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return done != 0;
}
// A bounded wait: false if the phase did not complete within `limit` polls (nothing spins forever).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// For a CTA in which a wait has run out, before it leaves: time (0.2 ms, a copy takes some microseconds) for the asynchronous copies
// that are still on their way into its shared memory, which another CTA gets next.  (Not by their barriers: which phase is due there is what
// the failed wait has lost, and of the two parities one is always complete.)
__device__ __forceinline__ void let_copies_land() {
#pragma unroll 1
  for (int i = 0; i < 200; ++i) __nanosleep(1000);
}
// `bytes` (a multiple of 16) from global to this CTA's shared memory, both 16-byte aligned; completion
// is counted on `bar`.  This CTA's own shared memory is not multicast to anyone.
__device__ __forceinline__ void bulk_copy_g2s(void* smem_dst, const void* gmem_src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

}  // namespace zb
