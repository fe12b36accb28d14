// sm_103a tensor-core primitives: tcgen05 MMA with TMEM accumulators,
// shared-memory matrix descriptors, mbarriers with bounded waits.
//
// Operand layout used throughout (K-major, no swizzle): a tile of R rows x
// KC columns (bf16) is stored as core matrices of 8 rows x 8 columns
// (8 rows of 16 bytes, 128 contiguous bytes), ordered column-chunk major:
//   byte(r, k) = (k / 8) * (R * 16) + (r / 8) * 128 + (r % 8) * 16 + (k % 8) * 2
// so that, in the descriptor, the stride between the two 8-column core
// matrices of one K=16 step (leading byte offset) is R * 16 and the stride
// between 8-row groups (stride byte offset) is 128.  Step j of K=16 starts
// at byte 2 * j * R * 16.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace bgpu {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (r, k) in a K-major tile with R rows (R % 8 == 0)
__host__ __device__ __forceinline__ uint32_t kmajor_off(int r, int k, int R) {
  return (uint32_t)((k >> 3) * (R * 16) + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor (tcgen05 format: start, leading and stride
// byte offsets in 16-byte units, descriptor version 1 at bits 46-47, no
// swizzle)
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// its high word (stride byte offset 128 and the version), in place: the low
// word is start / 16 | (leading byte offset / 16) << 16
__host__ __device__ constexpr uint64_t smem_desc_hi() { return ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46); }

// instruction descriptor of kind::f16 with bf16 A and B (both K-major),
// f32 accumulator, shape M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4)                        // D format f32
         | (1u << 7)                      // A format bf16
         | (1u << 10)                     // B format bf16
         | ((uint32_t)(N >> 3) << 17)     // N / 8
         | ((uint32_t)(M >> 4) << 24);    // M / 16
}

// same with fp16 A and B
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// 16-bit slices: x ~= hi + lo with hi = round(x), lo = round(x - hi) in bf16
// (8-bit significand, f32 range) or fp16 (11-bit significand, range +-65504)
__device__ __forceinline__ void split16(float x, bool fp16, uint32_t& hi, uint32_t& lo) {
  if (fp16) {
    const __half h = __float2half_rn(x);
    hi = __half_as_ushort(h);
    lo = __half_as_ushort(__float2half_rn(x - __half2float(h)));
  } else {
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    hi = __bfloat16_as_ushort(h);
    lo = __bfloat16_as_ushort(__float2bfloat16_rn(x - __bfloat162float(h)));
  }
}
__device__ __forceinline__ void split16(double x, bool fp16, uint32_t& hi, uint32_t& lo) {
  if (fp16) {
    const __half h = __double2half(x);
    hi = __half_as_ushort(h);
    lo = __half_as_ushort(__double2half(x - (double)__half2float(h)));
  } else {
    const __nv_bfloat16 h = __double2bfloat16(x);
    hi = __bfloat16_as_ushort(h);
    lo = __bfloat16_as_ushort(__double2bfloat16(x - (double)__bfloat162float(h)));
  }
}

// ---- TMEM ----
// one full warp; writes the allocated base address to *dst (shared memory)
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// generic-proxy shared-memory writes become visible to the tensor core
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T  (issued by one thread)
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the mbarrier once all earlier tcgen05 operations of this thread finished
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// The same in code that a whole warp runs, carried out by the lane with `on`
// set (24 orbitals M=500, with the sums of phase 2 in registers and its pieces
// side by side: 1005 -> 801 us a product).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}
// x, the same in every lane, known to be so
__device__ __forceinline__ int uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ void mma_bf16_if(bool on, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"((uint32_t)on)
      : "memory");
}
__device__ __forceinline__ void mma_commit_if(bool on, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
      "r"((uint32_t)on)
      : "memory");
}

// 32 lanes x 16 columns of 32-bit: thread t of the warp gets lane (base lane + t).
// Load and wait are one statement: the registers hold the values only after the
// wait, and nothing made of them can be moved between the two.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- packed pairs of f32 (one instruction for two values, rounded each) ----
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// products rounded by themselves: a packed product that only feeds packed
// sums was contracted with them (the sums of a triplet state then moved by
// 1.5e-8, the rounding of the products)
__device__ __forceinline__ uint64_t scale2(float a, float lo, float hi) {
  return pack2(__fmul_rn(a, lo), __fmul_rn(a, hi));
}
// (double)x by integer operations (the conversion takes a slot of the FP64
// pipe, a sixteenth of the rate)
__device__ __forceinline__ double f32_to_f64(float x) {
  const uint32_t u = __float_as_uint(x), e = u & 0x7f800000u;
  if (e == 0u ? (u & 0x7fffffffu) != 0u : e == 0x7f800000u) return (double)x;  // subnormal, infinite or NaN
  const uint32_t hi = e ? ((u & 0x7fffffffu) >> 3) + 0x38000000u : 0u;
  return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)(u << 29));
}
// split16 of two values: hi and lo hold the slices of x (low half) and y
__device__ __forceinline__ void split16x2(uint64_t xy, bool fp16, uint32_t& hi, uint32_t& lo) {
  float x, y;
  unpack2(xy, x, y);
  uint64_t h;
  if (fp16) {
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    h = pack2(__half2float(__ushort_as_half((unsigned short)(hi & 0xffffu))),
              __half2float(__ushort_as_half((unsigned short)(hi >> 16))));
  } else {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    h = pack2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u));
  }
  unpack2(sub2(xy, h), x, y);
  if (fp16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(y), "f"(x));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(y), "f"(x));
}

// ---- mbarrier ----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// whether the phase has completed, without waiting (try_wait may suspend the thread)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
constexpr int kSpinPolls = 1000;  // polls of a wait before it looks at the clock
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase with the given parity to complete, for at most
// `limit_ns` nanoseconds; returns false if the limit was reached.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity))
    if (globaltimer_ns() - t0 > limit_ns) return false;
  return true;
}

// ---- bulk copies (global -> shared, completion counted on an mbarrier) ----
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// dst and src 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace tc
}  // namespace bgpu
