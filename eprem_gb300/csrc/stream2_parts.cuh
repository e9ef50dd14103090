// stream2_parts.cuh -- what the FP32 streaming kernels share: the relaxation
// weight of a sub-cycle, exact power-of-two scalings, and the bounded waits
// and predicated stores of the halo hand-over between warps.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace eprem {

// The relaxation weight of one sub-cycle, f <- f (1 - om) + iso om with
// om = 1 - exp(-dtProp/tau).  For the sum over mu to be kept, 1 - om must be
// exact in float, so om is a multiple of 2^-24; rounding it there once moved
// the relaxation rate by up to 2^-25 / om (1e-4 at the 1536-stream case,
// whose om is 3e-4 - 1e-3), a bias that the diffusive tail of the
// distribution turns into 1e-3 of the flux 15 decades below its peak.  So
// om alternates between the two multiples around it (omlo and omlo +
// 2^-24) with an error-diffusion counter: over any run of sub-cycles the
// weights sum to the exact om times their number within 2^-24, and every
// single sub-cycle still keeps the sum.  Splitting the weight apart, f +
// om (iso - f), would do the same at one more packed operation per cell
// pair.  dith starts at 1/2 in every launch; phi is om 2^24 - omlo 2^24.
__device__ __forceinline__ float relax_weight(float omlo, float phi, float &dith) {
  dith += phi;
  const bool up = dith >= 1.f;
  dith = up ? dith - 1.f : dith;
  return up ? omlo + 0x1p-24f : omlo;
}

// The two power-of-two factors of ldexp_f(x, k), formed once for a row.
struct Pow2Pair {
  float a, b;
};
__device__ __forceinline__ Pow2Pair pow2_pair(int k) {
  const int k1 = k > 127 ? 127 : (k < -126 ? -126 : k);
  int k2 = k - k1;
  k2 = k2 > 127 ? 127 : (k2 < -126 ? -126 : k2);
  return Pow2Pair{pow2f(k1), pow2f(k2)};
}
__device__ __forceinline__ float scale2(float x, Pow2Pair p) { return (x * p.a) * p.b; }

// Bounded wait on a CTA mbarrier phase: at most kMirrorWaitLimit try_waits,
// each of which suspends the warp until the phase completes or about a
// microsecond has passed; false when the limit ran out.  (Publishing the
// warp-edge rows right after relaxing the edge nodes, before the others, and
// a few test_wait polls before suspending measured slower: 8.00 against
// 7.75 ms per 96-stream launch, the reordering spilling registers.)
constexpr int kMirrorWaitLimit = 1 << 20;
__device__ __forceinline__ bool halo_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
  for (int i = 0; i < kMirrorWaitLimit; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity), "r"(1000u)
        : "memory");
    if (done) return true;
  }
  return false;
}
// An arrival by the lanes where p holds, as a predicated instruction of the whole
// warp rather than a divergent branch.
__device__ __forceinline__ void halo_arrive_if(bool p, uint64_t *bar) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(bar);
  asm volatile(
      "{\n .reg .pred q;\n .reg .b64 st;\n setp.ne.u32 q, %0, 0;\n"
      " @q mbarrier.arrive.shared::cta.b64 st, [%1];\n}\n" ::"r"(p ? 1u : 0u),
      "r"(a)
      : "memory");
}
}  // namespace eprem
