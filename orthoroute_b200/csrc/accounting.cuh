// Device helpers shared by the accounting kernels and the routing loop.
#pragma once
#include "common.cuh"

namespace orsp {

// commit_path / clear_path on one edge (UPF:821-836): usage +-1 (never below
// 0) and present kept equal to it; atomic, so paths of a batch may share edges.
__device__ __forceinline__ int32_t apply_usage(int32_t *usage, float *present, int32_t e,
                                               int32_t sign) {
  int32_t left;
  if (sign >= 0) {
    left = atomicAdd(&usage[e], sign) + sign;
    if (present) atomicAdd(&present[e], 1.0f);
  } else {
    // clear_path: canonical count drops (never below 0) and
    // present = max(0, present - 1)
    int32_t old = __ldcg(&usage[e]);
    for (;;) {
      const int32_t nv = old > 0 ? old - 1 : 0;
      const int32_t prev = atomicCAS(&usage[e], old, nv);
      left = nv;
      if (prev == old) break;
      old = prev;
    }
    if (present) {
      unsigned *pp = (unsigned *)&present[e];
      unsigned ob = __ldcg(pp);
      for (;;) {
        float nv = __fsub_rn(__uint_as_float(ob), 1.0f);
        nv = nv > 0.0f ? nv : 0.0f;
        const unsigned prev = atomicCAS(pp, ob, __float_as_uint(nv));
        if (prev == ob) break;
        ob = prev;
      }
    }
  }
  return left;
}

// The edge-index jitter of the cost formulas, xp.arange(E, dtype=float32) %
// 9973 * 1e-6: the index is first rounded to float32 (exact below 2^24), the
// remainder is exact.  A rounded index below 2^31 is a 32-bit integer, whose
// remainder by a constant is a multiply and a subtract; fmodf's general
// reduction made update_costs compute-bound (226 us for 25.2 M edges; 99 us,
// 5.6 TB/s, with the integer form and four edges per thread).
__device__ __forceinline__ float index_jitter(int64_t e) {
  const float fi = __ll2float_rn(e);
  const float r = fi < 2147483648.0f ? (float)((uint32_t)fi % 9973u) : fmodf(fi, 9973.0f);
  return __fmul_rn(r, 1e-6f);
}

// Live-usage cost (classic PathFinder, the per-net refresh the reference's
// EdgeAccountant.update_present_cost_only (UPF:1045-1068) is meant for):
//   total = ((base*via_mult)*base_w) + pres_fac*max(0, (usage+1) - cap)
//           + hist_w*history [+ jitter]
// i.e. update_costs with present_ema replaced by the prospective usage if the
// net being routed takes the edge.  Applied to every edge (edges == nullptr)
// or to a list of edge ids (negative ids skipped; repeats are harmless).
__device__ __forceinline__ float live_cost_of(int64_t e, float base, int32_t usage, float cap, float hist,
                                              float pres_fac, float hist_w, float via_mult, float base_w,
                                              int jitter) {
  float over = __fsub_rn(__fadd_rn((float)usage, 1.0f), cap);
  over = over > 0.0f ? over : 0.0f;
  const float adjusted = __fmul_rn(__fmul_rn(base, via_mult), base_w);
  float total = __fadd_rn(__fadd_rn(adjusted, __fmul_rn(pres_fac, over)), __fmul_rn(hist_w, hist));
  if (jitter) total = __fadd_rn(total, index_jitter(e));
  return total;
}

__device__ __forceinline__ float live_cost(int64_t e, const float *base, const int32_t *usage,
                                           const float *cap, const float *hist, float pres_fac,
                                           float hist_w, float via_mult, float base_w, int jitter) {
  return live_cost_of(e, base[e], usage[e], cap[e], hist[e], pres_fac, hist_w, via_mult, base_w, jitter);
}

}  // namespace orsp
