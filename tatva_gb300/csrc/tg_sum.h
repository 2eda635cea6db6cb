// Sums of FP32 numbers to more than FP64's precision, in FP32 operations: what dots of FP32
// vectors are added in beyond the thread (DotAcc in tg_cg.cuh).
//
// A sum is three floats s + c + cc, each the running error of the one before (two-sums are
// exact), so an addition loses 2^-72 of the total; FP64 loses 2^-53, a pair of floats 2^-48.
// Why not FP64: an addition there takes 81 clocks on GB300 and 16 of the SM's FP64 pipe for a
// warp (a conversion from FP32 as long again), two-sums run at the FP32 rate.  The range is
// FP32's: callers scale by powers of two where totals may leave it.
// Plain C++, so that the arithmetic is tested on the host.
#pragma once

#ifdef __CUDACC__
#define TG_HD __host__ __device__ __forceinline__
#else
#define TG_HD inline
#endif

namespace tg {

// a becomes the rounded a + b; returns the exact rest
TG_HD float two_sum(float& a, float b) {
  const float s = a + b, t = s - a;
  const float e = (a - (s - t)) + (b - t);
  a = s;
  return e;
}

struct alignas(16) Sum3 {
  float s, c, cc;
  TG_HD static Sum3 of(float hi, float lo) { return {hi, lo, 0.f}; }
  TG_HD static Sum3 of(double v) {
    const float s = (float)v;
    const double a = v - (double)s;
    const float c = (float)a;
    return {s, c, (float)(a - (double)c)};
  }
  TG_HD double value() const { return (double)s + ((double)c + (double)cc); }
  TG_HD void add(const Sum3& o) {
    cc += o.cc;
    add(o.s, o.c);
  }
  // a float pair, as the threads' accumulators hold
  TG_HD void add(float hi, float lo) {
    const float e = two_sum(s, hi);
    const float d = two_sum(c, lo);
    cc += d + two_sum(c, e);
  }
  // the same value with s the nearest float to s + c, and c to the rest
  TG_HD void normalize() {
    float e = two_sum(s, c);
    cc = two_sum(e, cc);
    c = e;
  }
};

}  // namespace tg
