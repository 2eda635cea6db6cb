// CG building blocks shared by the vector kernels (linalg.cu) and the fused grid
// iteration (grid.cu): device-scalar slots, compensated FP32 dot accumulation, the
// fixed-order CTA reduction, 16-byte access and the last-arriving-CTA pattern.
#pragma once

#include "tg_common.cuh"
#include "tg_sum.h"

namespace tg {

constexpr int DOT_CHUNKS = 2048;
constexpr int DOT_THREADS = 256;
// SCAL_TOL2: the squared residual tolerance of the running CG; SCAL_DONE: set by the
// update when |r|^2 <= SCAL_TOL2 (the iteration's launches then return at once, so a
// captured block of iterations stops doing work when the solve has converged inside
// it); SCAL_ITERS: iterations performed.  Slots 5 and 7: true-residual norms.
constexpr int SCAL_RZ = 0, SCAL_PQ = 1, SCAL_ALPHA = 2, SCAL_BETA = 3, SCAL_RR = 4,
              SCAL_FLAG = 6, SCAL_TOL2 = 8, SCAL_DONE = 9, SCAL_ITERS = 10, SCAL_N = 12;

// 16-byte vector access of 4 consecutive values (4-aligned index, 16-byte aligned base)
__device__ __forceinline__ void ldv(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ldv(const double* p, double (&v)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0];
  const double2 b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void stv(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void stv(double* p, const double (&v)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// ------------------------------------------------------------------ dot accumulators
// FP32 vectors: each thread accumulates x_i y_i as an unevaluated pair (hi, lo) of
// floats -- the product is split exactly with an FMA and added with a two-sum, so the
// thread's partial keeps about 48 bits -- and only the per-thread partials enter the
// tree reduction, in FP64 or in three floats (Sum3).  (This GPU's FP64 rate is a small
// fraction of FP32: per-element FP64 conversions and multiply-adds made the dots several
// times slower than their memory traffic.)  FP64 vectors accumulate in FP64.
template <class T>
struct DotAcc;
template <>
struct DotAcc<float> {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float a, float b) {
    const float pr = a * b;
    const float pe = fmaf(a, b, -pr);
    const float s = hi + pr;
    const float bp = s - hi;
    const float err = (hi - (s - bp)) + (pr - bp);
    hi = s;
    lo += err + pe;
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};
template <>
struct DotAcc<double> {
  double v = 0.0;
  __device__ __forceinline__ void add(double a, double b) { v += a * b; }
  __device__ __forceinline__ double value() const { return v; }
};

// The scalars of a recursion on vectors of T and their sums over threads: Sum3 for FP32,
// FP64 for FP64.
template <class T>
struct Total;
template <>
struct Total<float> : Sum3 {
  __device__ static Total of(double v) { return {Sum3::of(v)}; }
  __device__ static Total of(float hi, float lo) { return {Sum3::of(hi, lo)}; }
  __device__ Total down(int o) const {
    return {{__shfl_down_sync(0xffffffffu, s, o), __shfl_down_sync(0xffffffffu, c, o),
             __shfl_down_sync(0xffffffffu, cc, o)}};
  }
  // of a total that another CTA stored
  __device__ static Total load(const Total* p) {
    const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
    return {{t.x, t.y, t.z}};
  }
  __device__ void store(Total* p) const {
    *reinterpret_cast<float4*>(p) = make_float4(s, c, cc, 0.f);
  }
  __device__ bool finite() const { return isfinite(s + c); }
  __device__ bool positive() const { return s + c > 0.f; }
  __device__ bool at_most(const Total& o) const {
    return (s - o.s) + ((c - o.c) + (cc - o.cc)) <= 0.f;
  }
  // this / o, rounded to FP32: an approximate quotient and the quotient of its exact
  // residual (a division in FP64 takes 580 clocks)
  __device__ float over(const Total& o) const {
    if (o.s < 0x1p-120f || o.s > 0x1p120f) return (float)(value() / o.value());
    const float q = __fdividef(s, o.s);
    if (!isfinite(q)) return q;
    const float r = fmaf(-q, o.s, s) + (fmaf(-q, o.c, c) + fmaf(-q, o.cc, cc));
    return q + __fdividef(r, o.s);
  }
};
template <>
struct Total<double> {
  double v;
  __device__ static Total of(double a) { return {a}; }
  __device__ double value() const { return v; }
  __device__ void add(const Total& o) { v += o.v; }
  __device__ void normalize() {}
  __device__ Total down(int o) const { return {__shfl_down_sync(0xffffffffu, v, o)}; }
  __device__ static Total load(const Total* p) { return {__ldcg(&p->v)}; }
  __device__ void store(Total* p) const { p->v = v; }
  __device__ bool finite() const { return isfinite(v); }
  __device__ bool positive() const { return v > 0.0; }
  __device__ bool at_most(const Total& o) const { return v <= o.v; }
  __device__ double over(const Total& o) const { return v / o.v; }
};
// a thread's sum
__device__ __forceinline__ Total<float> total_of(const DotAcc<float>& a) {
  return Total<float>::of(a.hi, a.lo);
}

// ------------------------------------------------------------------ reductions
// Sum of one value per thread of the CTA into out[k] (thread 0 writes): a fixed tree
// (shuffles inside each warp, then the warps' sums in warp order), so the result does
// not depend on timing.  Ends with a barrier: the CTA may call it again.
template <int K, int NT = DOT_THREADS>
__device__ __forceinline__ void block_reduce_store(double (&v)[K], double* __restrict__ out) {
  constexpr int NW = NT / 32;
  __shared__ double sh[K][NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0) sh[k][warp] = v[k];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double a = sh[k][0];
#pragma unroll
      for (int w = 1; w < NW; ++w) a += sh[k][w];
      out[k] = a;
    }
  }
  __syncthreads();
}

// The same for totals of FP32 vectors: warp k adds value k of all threads (a tree in every
// warp would be several times the instructions).  Ends with a barrier.
template <int K, int NT = DOT_THREADS>
__device__ __forceinline__ void block_sum(const Total<float> (&v)[K],
                                          Total<float>* __restrict__ out) {
  __shared__ Total<float> part[K][NT];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) part[k][threadIdx.x] = v[k];
  __syncthreads();
  if (w < K) {
    Total<float> t = part[w][lane];
#pragma unroll
    for (int j = 1; j < NT / 32; ++j) t.add(part[w][lane + 32 * j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t.add(t.down(o));
    if (lane == 0) t.store(out + w);
  }
  __syncthreads();
}

// Called by every thread after thread 0 stored this CTA's partials: true in the CTA
// that arrives last, which then sees every CTA's partials (read them with __ldcg).
// That CTA resets the ticket for the next launch.  An arrival counter, no waiting.
// Only thread 0's partial has to be visible before its arrival, so only thread 0
// fences: a fence in every thread waited for all of the CTA's output stores.
__device__ __forceinline__ bool last_cta(unsigned* ticket) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(ticket, 1u);
    last = (t == gridDim.x - 1);
    if (last) *ticket = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

}  // namespace tg
