// Shared device helpers for libwn_b200: status codes, the device error word,
// and the sm_100a bulk-copy (TMA 1-D) + mbarrier primitives used to stage face
// tiles into shared memory.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace wn {

// Bits of the device error word (one int per device, cleared per call).
enum DeviceError : int {
  kErrWaitTimeout = 1,   // an mbarrier wait hit its iteration limit
  kErrBadLaunch = 2,     // a kernel found inconsistent launch parameters
};

// A bounded wait gives up after this many polls (each poll suspends the
// thread for up to the hardware time limit), i.e. well after any legitimate
// bulk copy has landed.
constexpr uint32_t kWaitPolls = 1u << 24;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

// Makes the initialised barriers visible to the async (bulk-copy) proxy.
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// 1-D bulk copy global -> this CTA's shared memory, completing on `bar`.
// Requirements (checked by the callers' layout): src and dst 16-byte aligned,
// bytes a multiple of 16. No cluster multicast anywhere in this library.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait on phase `parity`; false (and the error bit set) on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err) {
  for (uint32_t i = 0; i < kWaitPolls; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  if (err) atomicOr(err, kErrWaitTimeout);
  return false;
}

__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// 1 / sqrt(x) in FP64 from the hardware's approximation by one step of Halley's
// (third-order) iteration: with e = 1 - x y^2, y (1 + e/2 + 3 e^2/8) leaves a relative
// error of 5 e^3 / 16, below rounding for e < 2^-18 (measured: the approximation is
// within 2^-20.05, the result within 2^-52.7 over [2^-600, 2^600]). 5 FP64 operations
// and no branch; x = 0, a subnormal, infinity or NaN give NaN or infinity.
__device__ __forceinline__ double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// det and denom of a pair (wn_pair.cuh) with contracted products and rsqrt64's roots: 65
// FP64 operations instead of 115. True if denom is certain to be positive by a margin
// (above |a||b||c| / 4, and between 2^-300 and 2^300): then no branch of the angle is
// near, its error stays within a few roundings, and neither term's last bits decide
// anything. Else, and for anything not finite, the caller takes the bit-identical terms.
__device__ __forceinline__ bool pair_terms_far(double ox, double oy, double oz, double Ax,
                                               double Ay, double Az, double Bx, double By,
                                               double Bz, double Cx, double Cy, double Cz,
                                               double& det, double& denom) {
  const double ax = Ax - ox, ay = Ay - oy, az = Az - oz;
  const double bx = Bx - ox, by = By - oy, bz = Bz - oz;
  const double cx = Cx - ox, cy = Cy - oy, cz = Cz - oz;
  const double aa = fma(ax, ax, fma(ay, ay, az * az));
  const double bb = fma(bx, bx, fma(by, by, bz * bz));
  const double cc = fma(cx, cx, fma(cy, cy, cz * cz));
  const double la = aa * rsqrt64(aa), lb = bb * rsqrt64(bb), lc = cc * rsqrt64(cc);
  const double nx = fma(by, cz, -(bz * cy)), ny = fma(bz, cx, -(bx * cz)),
               nz = fma(bx, cy, -(by * cx));
  det = fma(ax, nx, fma(ay, ny, az * nz));
  const double lll = la * lb * lc;
  double d = fma(fma(ax, bx, fma(ay, by, az * bz)), lc, lll);
  d = fma(fma(bx, cx, fma(by, cy, bz * cz)), la, d);
  denom = fma(fma(cx, ax, fma(cy, ay, cz * az)), lb, d);
  const int hd = __double2hiint(denom);  // high words order positive numbers
  return hd > 0x2d300000 && hd < 0x52b00000 && hd > __double2hiint(lll) - 0x00200000;
}

}  // namespace wn
