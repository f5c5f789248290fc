// Device arithmetic and data-movement helpers for sm_100a.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "btk_internal.h"

namespace btk {

// ---------------------------------------------------------------------------
// FP64 reciprocal square root and reciprocal for the pairwise kernels.
//
// Seed: the FP32 approximation rsqrt.approx.f32 / rcp.approx.f32 (one MUFU op)
// of the FP32 number that shares x's exponent and top 23 mantissa bits. The
// FP32 bit pattern is built from x's two words by integer re-biasing of the
// exponent (11-bit bias 1023 -> 8-bit bias 127: a 3-bit funnel shift of the
// high word with the top bits of the low word, then + 128 << 23 in the 9-bit
// field the shift leaves); the result is widened by the conversion
// instruction. Measured on the 1M potential + gradient solve (interaction
// kernel, ms): both ways in integers 125.2, widening by conversion 123.0,
// narrowing by conversion 125.9, widening by a 32 x 32 + 64-bit multiply-add
// 132, the FP64 seed rsqrt.approx.ftz.f64 with a cubic step 130. The seed's
// relative error e0 is at most 1.6e-7 (4e-8 rms).
//
// Refinement: one Newton step, which squares the relative error:
//   rsqrt: y' = y (3/2 - x y^2 / 2)          -> error 1.5 e0^2 <~ 4e-14
//   rcp:   e = 1 - x y,   y' = y + y e       -> error e0^2 <~ 4e-14     (2 FP64 ops)
// far below the 1e-12 agreement with the reference that the FP64 path keeps.
// The rsqrt step runs on w = sqrt(2 / x), the approximation at x / 2 (free in
// the re-biasing): x w^2 = 2, and w (6 - x w^2) = 4 sqrt(2) / sqrt(x) takes 3
// FP64 operations where y + (y / 2)(1 - x y^2) takes 4; the constant is
// taken out once per target (fp64_rescale).
//
// Domain: rsqrt x in [2^-125, 2^128), rcp x in [2^-126, 2^127]. The kernels
// guarantee the lower ends with eps^2 >= kSeedMin; callers with smaller eps
// use the guarded variants.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float fp32_seed_arg(double x, int shift = 0) {
  return __int_as_float(__funnelshift_l(__double2loint(x), __double2hiint(x), 3) + 0x40000000 + shift * 0x00800000);
}

// kRsqrtScale / sqrt(x).
__device__ __forceinline__ double rsqrt_fp64_scaled(double x) {
  float wf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(wf) : "f"(fp32_seed_arg(x, -1)));
  const double w = (double)wf;
  return w * fma(-x, w * w, 6.0);
}

// Same, extended to x = 0 (-> +inf, matching 1/sqrt(0)) and to x below the
// seed's range (rare: only with eps^2 < 2^-125 and near-coincident points).
__device__ __forceinline__ double rsqrt_fp64_scaled_guarded(double x) {
  if (x < kSeedMin) return x == 0.0 ? __longlong_as_double(0x7ff0000000000000LL) : kRsqrtScale / sqrt(x);
  return rsqrt_fp64_scaled(x);
}

// FP64 reciprocal of a positive x in the FP32 normal range (seed and Newton
// step as above).
__device__ __forceinline__ double rcp_fp64_pos(double x) {
  float yf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(fp32_seed_arg(x)));
  const double y = (double)yf;
  return fma(y, fma(-x, y, 1.0), y);
}

__device__ __forceinline__ double rcp_fp64_pos_guarded(double x) {
  if (x < kSeedMin) return x == 0.0 ? __longlong_as_double(0x7ff0000000000000LL) : 1.0 / x;
  return rcp_fp64_pos(x);
}

// ---------------------------------------------------------------------------
// FP64 natural logarithm of a positive x in [2^-1022, 2^1021), for the 2-D kernels
// (table-driven range reduction after Tang, ACM TOMS 16(4), 1990, with the
// reciprocal from the FP32 unit): x = 2^e f, f in [sqrt(1/2), sqrt(2)), so that
// e ln 2 and log f never cancel (e = 0 for every x near 1); c = 1/f rounded to 9
// mantissa bits, so u = x 2^-e c - 1 (one fma, exact to its rounding) is at most
// h = 2^-10 and log x = e ln 2 - log c + log(1 + u). c is 1 and the table's value 0
// where f is within 2^-11 of 1, so log x keeps its relative accuracy there. The
// last by its series to u^6, the sixth term folded into the others by
// u^4 = h^2 u^2 - h^4 / 8 (its Chebyshev polynomial left out): at most u^2 h^4 / 48
// is lost. -log c comes from a table over the values of c in shared memory
// (log_table_fill). 10 FP64 operations; the error is at most 2.6 roundings of the
// result (0.7 rms; test_gpu_log2d.py). With f in [1, 2) instead x just below 1
// lost up to 460. Non-finite x give non-finite results. yf: the FP32 reciprocal of
// f, for a caller that needs 1/x too (rcp_from_log).
// ---------------------------------------------------------------------------
constexpr int kLogTable = 515;
// c of table entry k, as the high word of a double, and entry 0 as FP32 bits.
constexpr int kLogHi = 0x3fe69800;
constexpr unsigned kLogFirst = 0x3f34c000u;

__device__ __forceinline__ void log_table_fill(double* table) {
  for (int k = threadIdx.x; k < kLogTable; k += blockDim.x) table[k] = -log(__hiloint2double(kLogHi + (k << 11), 0));
}

// The biased exponent e + 1023 of x = 2^e f, in place (sqrt(2) is 0x3ff6a09e...).
__device__ __forceinline__ int log_exponent(double x) { return (__double2hiint(x) + (0x00100000 - 0x0006a09e)) & 0x7ff00000; }

__device__ __forceinline__ double log_fp64_pos(double x, const double* table, float& yf) {
  const int eb = log_exponent(x);
  const unsigned fb = __funnelshift_l(__double2loint(x), __double2hiint(x) - eb, 3) + 0x3f800000u;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(__uint_as_float(fb)));
  const unsigned k = (__float_as_uint(yf) - (kLogFirst - 0x2000u)) >> 14;
  const double c = __hiloint2double((int)(k << 11) + (kLogHi + 0x3ff00000) - eb, 0);  // c 2^-e
  const double u = fma(x, c, -1.0), q = u * u;
  constexpr double h2 = 0x1p-20;
  const double a = fma(q, fma(u, 0.2, -0.25 - h2 / 6.0), fma(u, 1.0 / 3.0, -0.5 + h2 * h2 / 48.0));
  const double e = __hiloint2double(0x43300000, eb) - (4503599627370496.0 + 1023.0 * 1048576.0);  // 2^20 e
  return fma(e, 0.693147180559945309417 / 1048576.0, table[k]) + fma(q, a, u);
}

// 1 / x from log_fp64_pos's reciprocal: y 2^-e and one Newton step (rcp_fp64_pos).
__device__ __forceinline__ double rcp_from_log(double x, float yf) {
  const double f = (double)yf;
  const double y = __hiloint2double(__double2hiint(f) + 0x3ff00000 - log_exponent(x), __double2loint(f));
  return fma(y, fma(-x, y, 1.0), y);
}

// FP32 hardware approximations used by the mixed-precision kernels.
__device__ __forceinline__ float rsqrt_fp32(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_fp32(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// mbarrier + TMA bulk copies (cp.async.bulk, no tensor map, no multicast).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// Makes barrier initialisation visible to the async (TMA) proxy.
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: gives up after `limit` polls (each poll may itself suspend
// for a hardware-chosen interval) and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Global -> shared bulk copy completing on `bar`. dst, src 16-byte aligned,
// bytes a multiple of 16.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// ---------------------------------------------------------------------------
// tcgen05 (5th-generation tensor cores): TMEM allocation, shared-memory
// operand descriptors, UMMA issue, completion and TMEM loads, cta_group::1.
// ---------------------------------------------------------------------------
// Allocates ncols TMEM columns (a power of two >= 32) for the CTA; the whole
// warp executes it and the base address lands in *dst (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Orders this thread's generic-proxy shared-memory writes before the tensor
// cores (async proxy) read them.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Descriptor of a K-major operand tile in shared memory without swizzle: core
// matrices of 8 rows x 16 bytes (each row's 16 bytes contiguous), lbo = byte
// distance between the two 16-byte K halves of one 32-byte MMA K step, sbo =
// byte distance between consecutive groups of 8 rows; descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc_kmajor(const void* tile, uint32_t lbo, uint32_t sbo) {
  const uint32_t a = smem_addr(tile);
  return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16 with BF16 A and B (both K-major) and an
// FP32 accumulator, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16_f32(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D[tmem] = A * B^T (+ D when accumulate), issued by one thread.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  const uint32_t mask0 = 0, mask1 = 0, mask2 = 0, mask3 = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(mask0), "r"(mask1), "r"(mask2), "r"(mask3)
      : "memory");
}

// The mbarrier receives one arrival when every MMA this thread issued before
// has completed (its shared-memory reads included).
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

// 16 consecutive 32-bit TMEM columns of this thread's lane (warp w reads lanes
// 32w..32w+31; taddr carries the lane in bits 31..16), then waits for them.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  // the registers pass through the wait, so no use of them is scheduled before it
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

}  // namespace btk
