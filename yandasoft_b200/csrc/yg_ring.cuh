// Device-side pieces that the gridding and degridding kernels share: the
// weighted visibility of a sample, and mbarrier / bulk-copy primitives of the
// shared-memory rings.
#pragma once
#include "yg_internal.h"

namespace yg {

// ---------------------------------------------------------------------------
// weights: rVis = phasor * conj(vis) * wt (* mfs), TableVisGridder.cc:775-806
// ---------------------------------------------------------------------------
__device__ __forceinline__ float noise_weight(float nre) {
  const float vn = __fmul_rn(nre, nre);
  return (vn > 0.f) ? (float)(1.0 / (double)vn) : 0.f;
}

__device__ __forceinline__ void phasor(double freq, double delay, float* pr, float* pi) {
  const double ph = __ddiv_rn(__dmul_rn(__dmul_rn(__dmul_rn(2.0, kPi), freq), delay), kC);
  *pr = (float)cos(ph);
  *pi = (float)sin(ph);
}

__device__ __forceinline__ void phasor_of(const VisArgs& v, long long row, int chan, float* pr, float* pi) {
  *pr = 1.f;
  *pi = 0.f;
  if (v.delay) phasor(v.freq[chan], v.delay[row], pr, pi);
}

// rVis = phasor * conj(vis) * wt (* mfs) (TableVisGridder.cc:775-806), wt
// (* mfs) for the PSF, wt for the preconditioner function; FP32 with explicit
// rounding.
__device__ __forceinline__ float2 weigh(const VisArgs& v, float2 vis, float wt, float pr, float pi, float m) {
  if (v.pcf) return make_float2(__fmul_rn(1.f, wt), __fmul_rn(0.f, wt));
  if (v.psf) return make_float2(__fmul_rn(__fmul_rn(1.f, wt), m), __fmul_rn(__fmul_rn(0.f, wt), m));
  const float vr = vis.x, vi = -vis.y;
  float rr = __fsub_rn(__fmul_rn(pr, vr), __fmul_rn(pi, vi));
  float ri = __fadd_rn(__fmul_rn(pr, vi), __fmul_rn(pi, vr));
  rr = __fmul_rn(__fmul_rn(rr, wt), m);
  ri = __fmul_rn(__fmul_rn(ri, wt), m);
  return make_float2(rr, ri);
}

// the weighted visibility of sample s, polarisation p
__device__ __forceinline__ float2 weighted_vis(const VisArgs& v, long long s, long long n, int p, float pr, float pi,
                                               float m) {
  const float wt = v.noise ? noise_weight(v.noise[s + n * p].x) : 1.f;
  return weigh(v, v.psf || v.pcf ? make_float2(0.f, 0.f) : v.vis[s + n * p], wt, pr, pi, m);
}

// samples of a ring segment
constexpr int kSeg = 32;

// bounded mbarrier waits: a wait gives up after 4 s on the global timer (and
// after 2^26 polls, should the timer not advance)
constexpr unsigned long long kWaitNs = 4000000000ull;
constexpr long long kWaitPolls = 1ll << 26;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// one-dimensional TMA bulk copy global -> shared, completion on the mbarrier
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// try_wait that may suspend the thread up to hint_ns while the phase is open
__device__ __forceinline__ bool mbar_try_wait_for(unsigned long long* bar, unsigned phase, unsigned hint_ns) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase), "r"(hint_ns)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// bounded wait; false when the limit was reached.  The bound is time, not a
// poll count: CTAs of many kernels sharing the SMs (the major-cycle graph runs
// instances side by side) can make an ordinary wait last many polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned phase) {
  if (mbar_try_wait(bar, phase)) return true;
  const unsigned long long t0 = global_ns();
  for (long long i = 0; i < kWaitPolls; ++i) {
    if (mbar_try_wait_for(bar, phase, 100000u)) return true;
    if (global_ns() - t0 > kWaitNs) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace yg
