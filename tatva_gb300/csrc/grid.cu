// Structured-brick linear-elastic Hex8 residual / HVP launches (the stencil and its
// tiling are in tg_grid.cuh).
#include "tg_grid.cuh"

namespace tg {

// pack the per-dof mask into one byte per node
__global__ void pack_node_mask_kernel(const uint8_t* __restrict__ fixed, int64_t n_nodes,
                                      uint8_t* __restrict__ out) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < n_nodes) out[g] = (uint8_t)mask_bits<MASK_DOF>(fixed, g);
}

// Jacobi diagonal of the brick's operator: per dof, the sum of the element matrix's
// diagonal entry over the cells that exist around the node (the element-by-element sum
// of the reference's Hessian diagonal); fixed dofs get 1, the identity rows of the
// Dirichlet-masked operator.
template <class T>
__global__ void grid_diag_kernel(const __grid_constant__ GridCoef<T> P,
                                 const uint8_t* __restrict__ fixed, T* __restrict__ y) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t plane = (int64_t)P.nx * P.ny;
  if (g >= plane * P.nz) return;
  const int x = (int)(g % P.nx), yy = (int)((g / P.nx) % P.ny), z = (int)(g / plane);
  const int bits = fixed ? mask_bits<MASK_DOF>(fixed, g) : 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    T sum = T(0);
#pragma unroll
    for (int o = 0; o < 8; ++o) {  // cell whose corner o is this node
      const int cx = x - (o & 1), cy = yy - ((o >> 1) & 1), cz = z - (o >> 2);
      if (cx >= 0 && cy >= 0 && cz >= 0 && cx < P.nx - 1 && cy < P.ny - 1 && cz < P.nz - 1)
        sum += P.ke[o][o][a][a];
    }
    y[3 * g + a] = (bits >> a & 1) ? T(1) : sum;
  }
}

// Device scalars and partials of the CG dot that a DOT launch produces.
struct GridDot {
  double* scal;    // SCAL_* slots: reads RZ and FLAG, writes PQ, ALPHA, FLAG
  double* part;    // one partial per CTA
  unsigned* ticket;  // zeroed arrival counter (reset by the last CTA)
};

// DOT: the launch also forms p.q of its input p and output q (every dof: the HVP's
// fixed rows are the identity, so they add p^2) -- per CTA in a fixed order, the CTAs'
// partials added by the CTA that arrives last in index order -- and stores
// alpha = rz / (p.q) for the CG update (breakdown flag when p.q <= 0 or not finite).
template <class T, int MODE, int MK, bool DOT>
__global__ void __launch_bounds__(grid_threads<T>(), grid_ctas_per_sm<T>())
    grid_le_kernel(const __grid_constant__ GridCoef<T> P, const T* __restrict__ in,
                   const T* __restrict__ vin, const uint8_t* __restrict__ fixed,
                   T* __restrict__ y, const GridDot D) {
  constexpr int NT = grid_threads<T>();
  __shared__ GridShared<T> sh;
  if constexpr (DOT) {
    if (D.scal[SCAL_DONE] != 0.0) return;  // the CG converged earlier in this block
  }
  GridDotAcc<T> dot;
  grid_cta<T, MODE, MK, DOT>(P, blockIdx.x, in, vin, fixed, y, sh, dot);
  if constexpr (DOT) {
    double v[1] = {dot.value()};
    block_reduce_store<1, NT>(v, D.part + blockIdx.x);
    if (!last_cta(D.ticket)) return;
    double w[1] = {0.0};
    for (int i = threadIdx.x; i < (int)gridDim.x; i += NT) w[0] += __ldcg(D.part + i);
    __shared__ double out[1];
    block_reduce_store<1, NT>(w, out);
    if (threadIdx.x == 0) {
      const double pq = out[0];
      D.scal[SCAL_PQ] = pq;
      const bool bad = !(pq > 0.0) || !isfinite(pq) || D.scal[SCAL_FLAG] != 0.0;
      if (bad) D.scal[SCAL_FLAG] = 1.0;
      D.scal[SCAL_ALPHA] = bad ? 0.0 : D.scal[SCAL_RZ] / pq;
    }
  }
}

template <class T>
static int launch_grid_le_t(const tg_block_plan* plan, int mode, const T* u, const T* v,
                            const uint8_t* fixed, T* y, double mu, double lam,
                            cudaStream_t st) {
  GridCoef<T> P;
  const int64_t n = grid_setup<T>(plan, mu, lam, P);
  if (n < 0) return set_error(TG_ERR_VALUE, "grid too large");
  if (n == 0) return TG_OK;
  if (mode == TG_MODE_DIAG) {
    const int64_t nn = (int64_t)P.nx * P.ny * P.nz;
    grid_diag_kernel<T><<<grid_for(nn, 256), 256, 0, st>>>(P, fixed, y);
    return launch_check("grid diagonal kernel");
  }
  const T* in = (mode == TG_MODE_HVP) ? v : u;
  const unsigned grid = (unsigned)n;
  const GridDot D{nullptr, nullptr, nullptr};
  constexpr int NT = grid_threads<T>();
  if (mode == TG_MODE_HVP) {
    if (fixed)
      grid_le_kernel<T, TG_MODE_HVP, MASK_DOF, false><<<grid, NT, 0, st>>>(P, in, v, fixed, y, D);
    else
      grid_le_kernel<T, TG_MODE_HVP, MASK_NONE, false><<<grid, NT, 0, st>>>(P, in, v, fixed, y, D);
  } else if (fixed) {
    grid_le_kernel<T, TG_MODE_RESIDUAL, MASK_DOF, false><<<grid, NT, 0, st>>>(P, in, v, fixed, y,
                                                                             D);
  } else {
    grid_le_kernel<T, TG_MODE_RESIDUAL, MASK_NONE, false><<<grid, NT, 0, st>>>(P, in, v, fixed, y,
                                                                              D);
  }
  return launch_check("grid linear-elastic kernel");
}

int64_t grid_cg_ctas(const tg_block_plan* plan) {
  GridCoef<float> P32;
  GridCoef<double> P64;
  const int64_t a = grid_setup<float>(plan, 1.0, 1.0, P32);
  const int64_t b = grid_setup<double>(plan, 1.0, 1.0, P64);
  return (a < 0 || b < 0) ? -1 : (a > b ? a : b);
}

// The grid CG's handling of fixed dofs: x = b there (the identity rows of the masked
// system) and a zero inverse diagonal, so that z, p and the updates of x and r are
// exactly zero on them and the HVP of p needs no input mask.
template <class T>
__global__ void grid_cg_fixed_kernel(int64_t n_nodes, const uint8_t* __restrict__ nmask,
                                     const T* __restrict__ b, T* __restrict__ x,
                                     T* __restrict__ dinv) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_nodes) return;
  const int m = nmask[g];
  if (!m) return;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (m >> d & 1) {
      x[3 * g + d] = b[3 * g + d];
      dinv[3 * g + d] = T(0);
    }
}

int grid_cg_fixed(int prec, int64_t n_nodes, const uint8_t* nmask, const void* b, void* x,
                  void* dinv, cudaStream_t st) {
  if (prec == TG_F32)
    grid_cg_fixed_kernel<float><<<grid_for(n_nodes, 256), 256, 0, st>>>(
        n_nodes, nmask, (const float*)b, (float*)x, (float*)dinv);
  else
    grid_cg_fixed_kernel<double><<<grid_for(n_nodes, 256), 256, 0, st>>>(
        n_nodes, nmask, (const double*)b, (double*)x, (double*)dinv);
  return launch_check("grid CG fixed dofs");
}

int pack_node_mask(const uint8_t* fixed, int64_t n_nodes, uint8_t* out, cudaStream_t st) {
  pack_node_mask_kernel<<<grid_for(n_nodes, 256), 256, 0, st>>>(fixed, n_nodes, out);
  return launch_check("pack node mask");
}

int launch_grid_hvp_dot(const tg_block_plan* plan, int prec, double mu, double lam,
                        const void* p, const uint8_t* node_mask, void* q, double* scal,
                        double* part, unsigned* ticket, cudaStream_t st) {
  auto go = [&](auto t) -> int {
    using T = decltype(t);
    GridCoef<T> P;
    const int64_t n = grid_setup<T>(plan, mu, lam, P);
    if (n <= 0) return set_error(TG_ERR_VALUE, "grid CG: empty or too large grid");
    const GridDot D{scal, part, ticket};
    const T* in = (const T*)p;
    constexpr int NT = grid_threads<T>();
    if (node_mask)  // p is zero on the fixed dofs (grid_cg_fixed): only the rows are masked
      grid_le_kernel<T, TG_MODE_HVP, MASK_NODE_OUT, true><<<(unsigned)n, NT, 0, st>>>(
          P, in, in, node_mask, (T*)q, D);
    else
      grid_le_kernel<T, TG_MODE_HVP, MASK_NONE, true><<<(unsigned)n, NT, 0, st>>>(
          P, in, in, node_mask, (T*)q, D);
    return launch_check("grid HVP with p.q");
  };
  return prec == TG_F32 ? go(0.f) : go(0.0);
}

// ------------------------------------------------------------------ persistent CG
// `iters` Jacobi-CG iterations in one cooperative launch.  Per iteration
//   A: q = A p (the grid's tiles and faces) with p.q           | grid barrier
//   B: alpha; r -= alpha q with r.z and r.r                     | grid barrier
//   C: beta, stopping test; x += alpha p, p = r dinv + beta p   | grid barrier
// One CTA per SM holds the groups that would be separate CTAs, so that a barrier joins 152
// arrivals and a dot 152 partials.  Every CTA adds the partials itself, in the same fixed
// order, so all of them hold the same scalars and take the same decisions, and none waits
// for one that sums up.  The sums and scalars of FP32 vectors keep more than FP64's 53 bits
// (Sum3); in float pairs, 48 bits, the iteration took as long.  Tiles and vector entries are
// taken by a fixed stride: the result depends on the number of CTAs alone.
// Three launches a step spent most of a small or mid-size brick's iteration between kernels
// and in the arrival counters and last-CTA sums of their dots.  The vectors that only their
// own thread touches (r, 1 / diag, x, and its p) stay in shared memory as far as they fit.
// CG in FP32, us an iteration, three launches -> one for 50 iterations -> vectors kept and one
// for up to 800: 16^3 20.8 -> 12.8 -> 12.2, 32^3 20.7 -> 14.4 -> 13.9, 64^3 28.4 -> 21.3 -> 19.7,
// 96^3 41.9 -> 38.6 -> 37.0.  At 64^3 the tiles take 11,500 clocks, the update 4,200, the
// direction 2,000 and an exchange about 7,000 (fences and loads across the dies).
// The barrier's wait ends after GRID_SPIN polls (a second or more); the kernel then reports
// SCAL_FLAG = 2 and returns.
constexpr unsigned GRID_SPIN = 1u << 22;
constexpr int CG_SMEM = 220 * 1024;  // of the 227 KB a CTA can have; the rest: the sums'
constexpr int CG_MAX_CTAS = DOT_CHUNKS / 4;  // partials: CTAs of A, then two per CTA of B
template <class T>
constexpr int cg_groups() { return grid_ctas_per_sm<T>(); }
template <class T>
constexpr int cg_threads() { return cg_groups<T>() * grid_threads<T>(); }

template <class T>
struct GridCg {
  T *x, *r, *p, *q;
  const T* dinv;
  const uint8_t* nmask;
  int64_t n;
  double *scal, *part;
  unsigned* count;  // zero before the launch
  int iters, n_items;
  int cached, slabs;  // vectors kept in shared memory (of r, dinv, x, p), entries / (4 grid NT)
};

// The scalars of the recursion are totals (tg_cg.cuh): three floats for FP32 vectors (an
// exchange is a chain of some 20 additions, 81 clocks each in FP64) and FP64 for FP64 vectors.
// The floats' range is FP32's, where the three-launch path adds the threads' sums in FP64:
// large totals are scaled down by more than the number of threads (CG_MAX_CTAS of them), so
// that a total overflows no earlier than one thread's sum does.
template <class T>
__device__ __forceinline__ T total_scale(double v) {
  return sizeof(T) == 4 && v > 0x1p60 ? T(0x1p-18) : T(1);
}
static_assert(CG_MAX_CTAS * cg_threads<float>() <= 1 << 18, "what total_scale allows for");
static_assert((int64_t)4 * CG_MAX_CTAS * GRID_CG_MAX_ITERS < (int64_t)1 << 31,
              "a launch's arrivals fit the barrier's counter");

// A thread's sum as it is handed to the warp that adds them up: a float pair or a double.
template <class T>
struct ThreadSum {
  float hi, lo;
  __device__ ThreadSum(const GridDotAcc<T>& a, float scale) : hi(a.hi * scale), lo(a.lo * scale) {}
  __device__ ThreadSum(const DotAcc<T>& a, float scale) : hi(a.hi * scale), lo(a.lo * scale) {}
  __device__ Total<T> total() const { return Total<T>::of(hi, lo); }
  __device__ void add_to(Total<T>& t) const { t.add(hi, lo); }
};
template <>
struct ThreadSum<double> {
  double v;
  __device__ ThreadSum(const GridDotAcc<double>& a, double) : v(a.v) {}
  __device__ ThreadSum(const DotAcc<double>& a, double) : v(a.v) {}
  __device__ Total<double> total() const { return {v}; }
  __device__ void add_to(Total<double>& t) const { t.v += v; }
};

// sum over the warp's lanes (lane 0)
template <class T>
__device__ __forceinline__ Total<T> warp_total(Total<T> a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a.add(a.down(o));
  return a;
}

__device__ __forceinline__ bool grid_arrive_wait(unsigned* count, unsigned target) {
  __threadfence();
  atomicAdd(count, 1u);
  unsigned seen, polls = 0;
  do {
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
  } while (seen < target && ++polls < GRID_SPIN);
  __threadfence();
  return seen >= target;
}

// What the threads share of a recursion: the scalars, thread 0's but for tol2, and what the
// exchanges decide.
template <class T>
struct CgShared {
  Total<T> rz, rz_old, pq, rr, tol2;
  T ratio;          // alpha, then beta
  bool ok[2], bad;  // the wait ended; a sum is not positive (A) or not finite (B)
  bool done;
};

// The K sums over all threads of all CTAs.  Warp k adds value k of its CTA's threads, stores
// the CTA's total, waits for the other CTAs' (K arrivals each: everything the CTA has written
// is then visible too) and adds those, in a fixed order: the same totals in every CTA.  (A tree
// in every warp was more instructions: 64^3 21.3 us an iteration, 16^3 13.1.)
// v: the thread's sums, handed over in `stage`, the shared memory of the groups' tiles.
// finish(k, w): lane 0 of warp k with value k's total.
template <class T, int K, int NT, class F>
__device__ __forceinline__ bool grid_sum(const ThreadSum<T> (&v)[K], GridShared<T>* stage,
                                         Total<T>* part, unsigned* count, unsigned target,
                                         CgShared<T>& S, F&& finish) {
  constexpr int NW = NT / 32, GT = grid_threads<T>();
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  auto slot = [&](int t, int kk) -> ThreadSum<T>& {
    return reinterpret_cast<ThreadSum<T>*>(stage + t / GT)[kk * GT + t % GT];
  };
#pragma unroll
  for (int kk = 0; kk < K; ++kk) slot(threadIdx.x, kk) = v[kk];
  __syncthreads();
  if (k < K) {
    Total<T> w = slot(lane, k).total();
#pragma unroll
    for (int j = 1; j < NW; ++j) slot(lane + 32 * j, k).add_to(w);
    w = warp_total<T>(w);
    bool here = true;
    if (lane == 0) {
      w.store(part + K * blockIdx.x + k);
      here = grid_arrive_wait(count, target);
    }
    here = __shfl_sync(0xffffffffu, (int)here, 0) != 0;
    w = Total<T>::of(0.0);
#pragma unroll 8
    for (int i = lane; i < (int)gridDim.x; i += 32) w.add(Total<T>::load(part + K * i + k));
    w = warp_total<T>(w);
    if (lane == 0) {
      w.normalize();
      S.ok[k] = here;
      finish(k, w);
    }
  }
  __syncthreads();
  return S.ok[0] && S.ok[K - 1];
}

// grid barrier alone
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned target) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) ok = grid_arrive_wait(count, target);
  __syncthreads();
  return ok;
}

// four entries of a vector from i on (zero beyond n), and back
template <class T>
__device__ __forceinline__ void ld4n(const T* p, int64_t i, int64_t n, T (&v)[4]) {
  if (i + 3 < n) {
    ldv(p + i, v);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k < n ? p[i + k] : T(0);
  }
}
template <class T>
__device__ __forceinline__ void st4n(T* p, int64_t i, int64_t n, const T (&v)[4]) {
  if (i + 3 < n) {
    stv(p + i, v);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (i + k < n) p[i + k] = v[k];
  }
}

template <class T, int MK>
__global__ void __launch_bounds__(cg_threads<T>(), 1)
    grid_cg_kernel(const __grid_constant__ GridCoef<T> P, const GridCg<T> G) {
  constexpr int NT = cg_threads<T>(), NG = cg_groups<T>();
  extern __shared__ __align__(16) unsigned char cg_smem[];
  GridShared<T>* sh = reinterpret_cast<GridShared<T>*>(cg_smem);  // one per group
  using S = Total<T>;
  static_assert(3 * CG_MAX_CTAS * sizeof(S) <= 2 * DOT_CHUNKS * sizeof(double), "partials fit");
  const int group = threadIdx.x / grid_threads<T>();
  S* part_a = reinterpret_cast<S*>(G.part);
  S* part_b = part_a + CG_MAX_CTAS;
  __shared__ CgShared<T> C;
  unsigned target = 0;
  const T sz = total_scale<T>(G.scal[SCAL_RZ]), sr = total_scale<T>(G.scal[SCAL_RR]);
  if (threadIdx.x == 0) {
    C.rz = S::of((double)sz * G.scal[SCAL_RZ]);
    C.rr = S::of((double)sr * G.scal[SCAL_RR]);
    C.tol2 = S::of((double)sr * G.scal[SCAL_TOL2]);
    C.pq = S::of(0.0);
    C.rz_old = C.rz;
  }
  T alpha = T(0), beta = T(0);
  double flag = G.scal[SCAL_FLAG];
  bool done = G.scal[SCAL_DONE] != 0.0;
  int it = 0;
  const int64_t i0 = 4 * ((int64_t)blockIdx.x * NT + threadIdx.x);
  const int64_t stride = 4 * (int64_t)gridDim.x * NT;
  // entries i0 + j stride + 0..3 are this thread's throughout: vectors 0 (r), 1 (dinv), 2 (x), 3
  // (p) in shared memory as far as they fit
  T* const cache = reinterpret_cast<T*>(sh + NG) + 4 * threadIdx.x;
  auto kept = [&](int v, int j) { return cache + ((size_t)v * G.slabs + j) * (4 * NT); };
  auto get = [&](int v, const T* g, int64_t i, int j, T (&o)[4]) {
    if (v < G.cached) ldv(kept(v, j), o);
    else ld4n(g, i, G.n, o);
  };
  auto put = [&](int v, T* g, int64_t i, int j, const T (&o)[4]) {
    if (v < G.cached) stv(kept(v, j), o);
    else st4n(g, i, G.n, o);
  };
  for (int j = 0; j < G.slabs; ++j) {
    const int64_t i = i0 + j * stride;
    T t[4];  // zero beyond n
    if (G.cached > 0) { ld4n(G.r, i, G.n, t); stv(kept(0, j), t); }
    if (G.cached > 1) { ld4n(G.dinv, i, G.n, t); stv(kept(1, j), t); }
    if (G.cached > 2) { ld4n(G.x, i, G.n, t); stv(kept(2, j), t); }
    if (G.cached > 3) { ld4n(G.p, i, G.n, t); stv(kept(3, j), t); }
  }
  while (it < G.iters && !done && flag == 0.0) {
    GridDotAcc<T> dot;
    for (int item = group * gridDim.x + blockIdx.x; item < G.n_items; item += NG * gridDim.x) {
      grid_cta<T, TG_MODE_HVP, MK, true, EPI_PLAIN, true>(P, item, G.p, G.p, G.nmask, G.q,
                                                          sh[group], dot);
      group_sync<T, true>();  // the next item restages the group's shared memory
    }
    {
      const ThreadSum<T> v[1] = {{dot, sz}};
      const bool met = grid_sum<T, 1, NT>(v, sh, part_a, G.count, target += gridDim.x, C,
                                          [&](int, const S& w) {
                                            C.pq = w;
                                            C.bad = !w.positive() || !w.finite();
                                            C.ratio = C.rz.over(w);
                                          });
      if (!met) {
        flag = 2.0;
        break;
      }
    }
    ++it;
    if (C.bad) {
      flag = 1.0;
      alpha = T(0);
      break;
    }
    alpha = C.ratio;
    DotAcc<T> a0, a1;
#pragma unroll 2
    for (int j = 0; j < G.slabs; ++j) {
      const int64_t i = i0 + j * stride;
      T rv[4], qv[4], dv[4];
      ld4n(G.q, i, G.n, qv);
      get(0, G.r, i, j, rv);
      get(1, G.dinv, i, j, dv);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        rv[k] = rv[k] - alpha * qv[k];
        a0.add(rv[k], rv[k] * dv[k]);
        a1.add(rv[k], rv[k]);
      }
      put(0, G.r, i, j, rv);
    }
    const ThreadSum<T> v[2] = {{a0, sz}, {a1, sr}};
    const bool met = grid_sum<T, 2, NT>(v, sh, part_b, G.count, target += 2 * gridDim.x, C,
                                        [&](int k, const S& w) {
                                          if (k == 0) {
                                            C.bad = !w.finite();
                                            C.ratio = w.over(C.rz);
                                            if (!C.bad) {
                                              C.rz_old = C.rz;
                                              C.rz = w;
                                            }
                                          } else {
                                            C.rr = w;
                                            C.done = w.at_most(C.tol2);
                                          }
                                        });
    if (!met) {
      flag = 2.0;
      break;
    }
    done = C.done;
    beta = C.ratio;
    if (C.bad) {
      flag = 1.0;
      beta = T(0);
    }
    const bool stop = done || flag != 0.0;  // the direction stays as it is
#pragma unroll 2
    for (int j = 0; j < G.slabs; ++j) {
      const int64_t i = i0 + j * stride;
      T xv[4], pv[4], rv[4], dv[4];
      get(2, G.x, i, j, xv);
      get(3, G.p, i, j, pv);
      get(0, G.r, i, j, rv);
      get(1, G.dinv, i, j, dv);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        xv[k] += alpha * pv[k];
        pv[k] = rv[k] * dv[k] + beta * pv[k];
      }
      put(2, G.x, i, j, xv);
      if (!stop) {
        st4n(G.p, i, G.n, pv);
        if (G.cached > 3) stv(kept(3, j), pv);
      }
    }
    if (stop || it == G.iters) break;
    if (!grid_barrier(G.count, target += gridDim.x)) {
      flag = 2.0;
      break;
    }
  }
  for (int j = 0; j < G.slabs; ++j) {
    const int64_t i = i0 + j * stride;
    T t[4];
    if (G.cached > 0) { ldv(kept(0, j), t); st4n(G.r, i, G.n, t); }
    if (G.cached > 2) { ldv(kept(2, j), t); st4n(G.x, i, G.n, t); }
  }
  if (it > 0 && blockIdx.x == 0 && threadIdx.x == 0) {  // every CTA has read the scalars
    const double z1 = C.rz.value() / (double)sz, z0 = C.rz_old.value() / (double)sz;
    G.scal[SCAL_PQ] = C.pq.value() / (double)sz;
    G.scal[SCAL_ALPHA] = (double)alpha;
    G.scal[SCAL_BETA] = flag == 0.0 ? z1 / z0 : 0.0;
    G.scal[SCAL_RZ] = z1;
    G.scal[SCAL_RR] = C.rr.value() / (double)sr;
    G.scal[SCAL_DONE] = done ? 1.0 : 0.0;
    G.scal[SCAL_ITERS] += (double)it;
  }
  // any CTA whose wait ran out reports it (the others' waits then run out too)
  if (threadIdx.x == 0 && flag != 0.0) G.scal[SCAL_FLAG] = flag;
}

bool grid_cg_persistent(const tg_block_plan* plan) {
  const int64_t n = 3 * (int64_t)plan->grid_nodes[0] * plan->grid_nodes[1] * plan->grid_nodes[2];
  return n <= GRID_CG_MAX_DOFS && !(plan->grid_flags & TG_GRID_SEPARATE_LAUNCHES);
}

int launch_grid_cg(const tg_block_plan* plan, int prec, double mu, double lam,
                   const uint8_t* node_mask, void* x, void* r, void* p, void* q, const void* dinv,
                   double* scal, double* part, unsigned* count, int iters, cudaStream_t st) {
  auto go = [&](auto t) -> int {
    using T = decltype(t);
    constexpr int NT = cg_threads<T>();
    GridCoef<T> P;
    const int64_t sms = grid_sm_count();
    const int64_t items = grid_setup<T>(plan, mu, lam, P, cg_groups<T>() * sms);
    if (items <= 0) return set_error(TG_ERR_VALUE, "grid CG: empty or too large grid");
    GridCg<T> G{(T*)x, (T*)r, (T*)p, (T*)q, (const T*)dinv, node_mask,
                3 * (int64_t)P.nx * P.ny * P.nz, scal, part, count, iters, (int)items, 0, 0};
    const void* kern = node_mask ? (const void*)grid_cg_kernel<T, MASK_NODE_OUT>
                                 : (const void*)grid_cg_kernel<T, MASK_NONE>;
    // one CTA per SM (all resident), none without work
    const int64_t vec = (G.n + 4 * NT - 1) / (4 * NT), want = items > vec ? items : vec;
    int64_t ctas = sms < want ? sms : want;
    ctas = ctas < CG_MAX_CTAS ? ctas : CG_MAX_CTAS;
    // the SM's shared memory holds as many of the vectors as fit
    constexpr int tiles = cg_groups<T>() * (int)sizeof(GridShared<T>);
    G.slabs = (int)((vec + ctas - 1) / ctas);
    const int64_t vbytes = (int64_t)G.slabs * 4 * NT * sizeof(T), room = CG_SMEM - tiles;
    G.cached = (int)(room / vbytes < 4 ? room / vbytes : 4);
    const int smem = tiles + (int)(G.cached * vbytes);
    TG_TRY(cuda_check(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CG_SMEM),
        "grid CG: shared memory"));
    TG_TRY(cuda_check(cudaMemsetAsync(count, 0, sizeof(unsigned), st), "grid CG: barrier"));
    void* args[] = {&P, &G};
    const cudaError_t e =
        cudaLaunchCooperativeKernel(kern, dim3((unsigned)ctas), dim3(NT), args, smem, st);
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
      cudaGetLastError();  // fewer SMs than the device reports: the caller's other path runs
      return TG_ERR_UNSUPPORTED;
    }
    return cuda_check(e, "grid CG: launch");
  };
  return prec == TG_F32 ? go(0.f) : go(0.0);
}

int launch_grid_le(const tg_block_plan* plan, int prec, int mode, const void* u, const void* v,
                   const uint8_t* fixed, void* y, double mu, double lam, cudaStream_t st) {
  if (mode != TG_MODE_HVP && mode != TG_MODE_RESIDUAL && mode != TG_MODE_DIAG)
    return TG_ERR_UNSUPPORTED;
  if (plan->grid_nodes[0] < 2 || plan->grid_nodes[1] < 2 || plan->grid_nodes[2] < 2)
    return TG_ERR_UNSUPPORTED;
  if (prec == TG_F32)
    return launch_grid_le_t<float>(plan, mode, (const float*)u, (const float*)v, fixed,
                                   (float*)y, mu, lam, st);
  return launch_grid_le_t<double>(plan, mode, (const double*)u, (const double*)v, fixed,
                                  (double*)y, mu, lam, st);
}

}  // namespace tg
