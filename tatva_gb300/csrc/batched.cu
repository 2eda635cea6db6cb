// Batched solves of many independent sparse SPD systems in one persistent launch.
//
// The reference has no batched solver: a user loops over meshes and calls
// jax.scipy.sparse.linalg.cg on each (README.md:93).  Here every system is one
// mesh's assembled, Dirichlet-reduced CSR matrix (tatva.sparse.jacfwd output,
// tatva/sparse/base.py:139-176), converted once to a per-system ELLPACK layout:
// column-major (entry k of local row i at k * n_rows + i) with 16-bit local column
// ids, so that one thread per row reads coalesced.
//
// Systems are taken from device counters (in the caller's order, largest first).  A system
// whose matrix fits beside the others' in half an SM's shared memory is solved by one CTA,
// a larger one by a cluster of four, each CTA with a quarter of the rows.  On chip for the
// whole solve: the FP32 matrix and the window of p that the CTA's rows touch in shared
// memory, the CG vectors of a thread's rows in its registers.  What does not fit (wide
// rows, systems of more than 10,000 rows) stays in global memory: the last entries of each
// row, then the vectors.  After the first dot of an iteration the CTAs of a cluster need
// only the rows that others' windows hold: z = D^-1 r of those rows travels with the
// second dot, and every CTA updates its copies of p itself -- two cluster barriers an
// iteration.
//
// Bound: the latency of an iteration (two sums over the CTA or cluster, the SpMV's
// dependent loads), 2.3 us for 289 rows, 3.3 us for 9,409 rows on a cluster; at full
// load the shared-memory loads (2.5 per entry).  768 unit squares of 8..96 cells a side:
// 28.5 -> 6.0 ms; 4,096 of them 59.7 -> 32.1; 4,096 of 6..24: 13.9 -> 1.8 (5.5, 29.8 and 1.6
// with sums in float pairs, 48 bits).  Before, one CTA
// streamed a system's matrix from the L2 and DRAM: 27 us an iteration for the largest, which
// the whole batch waited for, and FP64 sums in every warp, 7 us for the smallest.  Clusters
// of two: 10 ms, of eight: 14 (768 squares).
//
// Each system runs FP32 Jacobi-preconditioned CG on the residual direction
// r64 / |r64| and FP64 iterative refinement on the true residual b - A64 x, until
// |b - A64 x| <= rtol |b|.  Dots accumulate as exact-product float pairs in a thread and to
// more than FP64's 53 bits (three floats, tg_sum.h) beyond it, in a fixed order, so each
// system's result depends only on its own data and the block size -- not on which CTA took it,
// nor on what else ran.  Every loop is bounded by max_outer / max_inner; CTAs wait for others
// of their cluster only, at cluster barriers that all of it reach (every decision is taken on
// sums that are the same bits in each).
#include <cmath>
#include <map>
#include <mutex>

#include "tg_cg.cuh"
#include "tg_dispatch.cuh"

namespace tg {
namespace {

constexpr int BATCH_MAX_ROWS = 49152;  // p of one system in shared memory: 192 KB
constexpr int TEAM = 4;  // CTAs of a cluster
// shared memory of a CTA when `per_sm` of them share an SM (228 KB, of which Crew::Shared
// and 1 KB for the system are the CTA's own)
constexpr int batch_smem(int nt, int per_sm) { return 228 * 1024 / per_sm - 2048 - 16 * nt; }
// What one CTA solves alone: its FP32 matrix and p within half an SM's shared memory, its
// vectors within its registers (10 rows a thread at 256 threads).  768 squares of 8..96, with
// sums in float pairs: 5.6 ms with this limit, 5.9 with 80 KB, 7 with 54 KB (more work at
// cluster barriers).
constexpr int64_t SOLO_BYTES = 103 * 1024;
constexpr int SOLO_ROWS = 2560;
using Total32 = Total<float>;

struct BatchArgs {
  tg_batch_desc d;
  const double* b;
  double* x;
  float* q;
  float* r;
  float* dv;
  float* idiag;
  double* r64;
  unsigned* counter;  // [0] systems of a whole cluster, [1] systems of one CTA
  int smem_floats;
  double rtol, inner_rtol;
  int max_outer, max_inner;
  int32_t* iters;
  int32_t* outer;
  double* rel_res;
  int32_t* status;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// address of this CTA's shared-memory object in the CTA of rank `cta`
__device__ __forceinline__ unsigned remote(const void* p, int cta) {
  const unsigned l = (unsigned)__cvta_generic_to_shared(p);
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(l), "r"(cta));
  return a;
}
__device__ __forceinline__ void put(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void put(unsigned addr, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void put(unsigned addr, const Total32& v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.s),
               "f"(v.c), "f"(v.cc), "f"(0.f)
               : "memory");
}
__device__ __forceinline__ void put(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

// The CTAs that solve one system: the whole cluster (size TEAM) or this CTA alone.
template <int NT>
struct Crew {
  static constexpr int NW = NT / 32;
  struct Shared {
    float2 part[2][NT];        // the threads' partial sums
    Total32 total[2][2][TEAM]; // the CTAs' sums; two halves, used in turn
    double dtotal[2][TEAM];
    double scal[4];
    float ratio;  // alpha or NaN, then beta
    int state;    // of the residual: 0 goes on, 1 small enough, 2 not finite
    int lo[TEAM], hi[TEAM];  // window of every CTA
    int next;
  };
  Shared& S;
  int size, rank, flip;

  __device__ void sync() const {
    if (size > 1) cluster_sync(); else __syncthreads();
  }

  // Sums of K per-thread float pairs over the crew, in a fixed order and to more than FP64's
  // precision.  Warp k adds value k for the whole CTA: a tree in every warp was more
  // instructions than the rows of a mid-size system.  finish(k, sum): lane 0 of warp k with
  // value k's sum, the same in every CTA; what it leaves in S the threads read after the
  // call.  A CTA may be one sum ahead of the others (its total goes to the other half), not
  // two (the sync).  between(): work of the threads after warp K - 1 while those add.
  template <int K, class F, class G>
  __device__ __forceinline__ void sum(const float2 (&v)[K], F&& between, G&& finish) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) S.part[k][threadIdx.x] = v[k];
    __syncthreads();
    if (w < K) {
      const float2* in = S.part[w];
      Total32 t = Total32::of(in[lane].x, in[lane].y);
#pragma unroll
      for (int j = 1; j < NW; ++j) t.add(in[lane + 32 * j].x, in[lane + 32 * j].y);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t.add(t.down(o));
      if (size > 1) {
        t.s = __shfl_sync(0xffffffffu, t.s, 0);
        t.c = __shfl_sync(0xffffffffu, t.c, 0);
        t.cc = __shfl_sync(0xffffffffu, t.cc, 0);
        if (lane < TEAM) put(remote(S.total[flip][w] + rank, lane), t);
      } else if (lane == 0) {
        finish(w, t);
      }
    } else {
      between();
    }
    if (size > 1) {
      cluster_sync();
      if (w < K && lane == 0) {
        Total32 t = S.total[flip][w][0];
#pragma unroll
        for (int r = 1; r < TEAM; ++r) t.add(S.total[flip][w][r]);
        finish(w, t);
      }
      flip ^= 1;
    }
    __syncthreads();
  }
  // the same for one FP64 value per thread; every thread gets the sum
  __device__ __forceinline__ double sum(double v) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double* part = reinterpret_cast<double*>(S.part[0]);
    part[threadIdx.x] = v;
    __syncthreads();
    if (w == 0) {
      double t = part[lane];
#pragma unroll
      for (int j = 1; j < NW; ++j) t += part[lane + 32 * j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
      if (size > 1) {
        t = __shfl_sync(0xffffffffu, t, 0);
        if (lane < TEAM) put(remote(S.dtotal[flip] + rank, lane), t);
      } else if (lane == 0) {
        S.dtotal[flip][0] = t;
      }
    }
    sync();
    v = S.dtotal[flip][0];
    if (size > 1)
#pragma unroll
      for (int t = 1; t < TEAM; ++t) v += S.dtotal[flip][t];
    flip ^= 1;
    return v;
  }
};

// Systems larger than this go to a whole cluster.  Own size only: which other systems
// are in the batch changes nothing in a system's arithmetic.
__device__ __forceinline__ bool for_cluster(const tg_batch_desc& d, int sys) {
  const int64_t n = d.row_ofs[sys + 1] - d.row_ofs[sys];
  const int W = d.ell_width[sys];
  return n > 0 && n <= d.max_rows && W >= 0 &&
         (n > SOLO_ROWS || n * (6 * (int64_t)W + 4) > SOLO_BYTES);
}

// The next system (in `order`) of the wanted kind, n_systems when none is left; called
// by one whole warp.  Claims go through the counter; a warp that claims one of the other
// kind looks ahead and moves the counter past the stretch it has seen to hold no match.
__device__ int take(const tg_batch_desc& d, unsigned* counter, bool cluster) {
  const int lane = threadIdx.x & 31, N = d.n_systems;
  for (;;) {
    int k = 0;
    if (lane == 0) k = (int)min(atomicAdd(counter, 1u), (unsigned)N);
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k >= N || for_cluster(d, d.order[k]) == cluster) return k;
    int at = k + 1;
    unsigned hit = 0;
    for (; at < N; at += 32) {
      const bool m = at + lane < N && for_cluster(d, d.order[at + lane]) == cluster;
      hit = __ballot_sync(0xffffffffu, m);
      if (hit) break;
    }
    if (lane == 0) atomicMax(counter, (unsigned)(hit ? at + __ffs(hit) - 1 : N));
  }
}

// y = A p for the P row pairs (l, l + half), l = tid + j NT, of this thread: entries k < Ks
// of the rows from shared memory, the others (what did not fit) from global memory.
template <int NT, int P, int NR>
__device__ __forceinline__ void spmv(float (&y)[NR], const float* __restrict__ p,
                                     const float* __restrict__ sval,
                                     const uint32_t* __restrict__ scol, int m, int half, int Ks,
                                     int W, int n, int wlo, const float* __restrict__ v32,
                                     const uint16_t* __restrict__ col) {
  int l[P], t0 = threadIdx.x;
  asm volatile("" : "+r"(t0));
#pragma unroll
  for (int j = 0; j < P; ++j) {
    l[j] = min(t0 + j * NT, half - 1);
    y[2 * j] = y[2 * j + 1] = 0.f;
  }
#pragma unroll(P == 1 ? 2 : 1)
  for (int k = 0; k < Ks; ++k) {
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const uint32_t c = scol[l[j]];
      y[2 * j] = fmaf(sval[l[j]], p[c & 0xffffu], y[2 * j]);
      y[2 * j + 1] = fmaf(sval[l[j] + half], p[c >> 16], y[2 * j + 1]);
    }
    sval += m;
    scol += half;
  }
  for (int k = Ks; k < W; ++k) {
    const int64_t e = (int64_t)k * n;
#pragma unroll
    for (int j = 0; j < P; ++j) {
      const int h = min(l[j] + half, m - 1);
      y[2 * j] = fmaf(v32[e + l[j]], p[col[e + l[j]] - wlo], y[2 * j]);
      y[2 * j + 1] = fmaf(v32[e + h], p[col[e + h] - wlo], y[2 * j + 1]);
    }
  }
}
template <int NT, int P, int NR>
__device__ __forceinline__ void spmv_pairs(int np, float (&y)[NR], const float* p,
                                           const float* sval, const uint32_t* scol, int m, int half, int Ks, int W,
                                           int n, int wlo, const float* v32, const uint16_t* col) {
  if constexpr (P > 0) {
    if (np == P) return spmv<NT, P>(y, p, sval, scol, m, half, Ks, W, n, wlo, v32, col);
    if constexpr (P > 1)
      return spmv_pairs<NT, P - 1>(np, y, p, sval, scol, m, half, Ks, W, n, wlo, v32, col);
  }
}

// PP > 0: the CG vectors of this thread's rows live in registers (at most PP row pairs a
// thread); PP = 0: in shared memory if they fit there, else in the workspace.
template <int NT, int PP>
__device__ void solve_rows(const BatchArgs& a, int sys, float* smem, Crew<NT>& crew) {
  const int tid = threadIdx.x;
  const int n = (int)(a.d.row_ofs[sys + 1] - a.d.row_ofs[sys]);
  const int W = a.d.ell_width[sys];
  // this CTA's rows [f0, f0 + m); thread t has rows l and l + half, l = t, t + NT, ...
  const int chunk = (n + crew.size - 1) / crew.size;
  const int f0 = min(n, crew.rank * chunk), m = min(n, f0 + chunk) - f0, half = (m + 1) >> 1;
  const int np = max(0, (half - (tid & ~31) + NT - 1) / NT);  // of this warp
  // offsets, not pointers, and made opaque where they are used: kept as addresses they
  // drove the CG vectors out of the registers
  const int64_t g0 = a.d.row_ofs[sys] + f0, e0 = a.d.ell_ofs[sys] + f0;
  auto at_row = [&](auto* base) {
    int64_t o = g0;
    asm volatile("" : "+l"(o));
    return base + o;
  };
  auto at_entry = [&](auto* base) {
    int64_t o = e0;
    asm volatile("" : "+l"(o));
    return base + o;
  };
  // the columns that its rows touch: the window of p kept here
  int wlo = 0, whi = n - 1;
  if (crew.size > 1) {
    if (tid == 0) {
      crew.S.lo[crew.rank] = m ? f0 : n;  // no rows: an empty window above all
      crew.S.hi[crew.rank] = m ? f0 + m - 1 : n - 1;
    }
    __syncthreads();
    int lo = n, hi = -1;
    const uint16_t* __restrict__ col = at_entry(a.d.ell_col);
    for (int i = tid; i < m; i += NT)
      for (int k = 0; k < W; ++k) {
        const int c = col[(int64_t)k * n + i];
        lo = min(lo, c);
        hi = max(hi, c);
      }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((tid & 31) == 0 && hi >= 0) {
      atomicMin(&crew.S.lo[crew.rank], lo);
      atomicMax(&crew.S.hi[crew.rank], hi);
    }
    __syncthreads();
    wlo = crew.S.lo[crew.rank];
    whi = crew.S.hi[crew.rank];
    if (tid < TEAM && tid != crew.rank) {
      put(remote(&crew.S.lo[crew.rank], tid), wlo);
      put(remote(&crew.S.hi[crew.rank], tid), whi);
    }
  }
  // shared memory: the window of p, the CG vectors (PP = 0), then as many of the W
  // entries of every row as fit
  float* p = smem;
  float* pown = p + (f0 - wlo);
  const int nw = whi - wlo + 1;
  float* hz = p + nw;  // PP > 0: the direction's update z of the window's other rows
  int at = PP > 0 ? nw + (nw - m) : nw;
  const bool vs = PP == 0 && at + 4 * m <= a.smem_floats;
  float* mem[4];  // r, d, 1 / diagonal, q
  {
    float* const ws[4] = {at_row(a.r), at_row(a.dv), at_row(a.idiag), at_row(a.q)};
#pragma unroll
    for (int v = 0; v < 4; ++v) mem[v] = vs ? smem + at + v * m : ws[v];
    if (vs) at += 4 * m;
  }
  const int Ks = m ? min(W, (a.smem_floats - at) / (m + half)) : 0;
  float* sval = smem + at;
  uint32_t* scol = reinterpret_cast<uint32_t*>(sval + Ks * m);
  // the thread's values (PP > 0); a row that does not exist holds zeros throughout
  constexpr int NR = PP ? 2 * PP : 4;
  float vr[NR] = {}, vd[NR] = {}, vg[NR] = {}, vq[NR] = {}, vp[NR] = {};
  auto R = [&](int j, int i) -> float& {
    if constexpr (PP > 0) return vr[j];
    else return mem[0][i];
  };
  auto D = [&](int j, int i) -> float& {
    if constexpr (PP > 0) return vd[j];
    else return mem[1][i];
  };
  auto G = [&](int j, int i) -> float& {
    if constexpr (PP > 0) return vg[j];
    else return mem[2][i];
  };
  auto Q = [&](int j, int i) -> float& {
    if constexpr (PP > 0) return vq[j];
    else return mem[3][i];
  };
  auto Pv = [&](int j, int i) -> float& {
    if constexpr (PP > 0) return vp[j];
    else return pown[i];
  };
  // f(j, i, exists) for the thread's rows i; with PP > 0 also for its places j without a row
  auto each = [&](auto&& f) {
    if constexpr (PP > 0) {
      int t0 = tid;
      // indices and conditions made anew in each pass: kept, they drove the vectors out of
      // the registers
      asm volatile("" : "+r"(t0));
#pragma unroll
      for (int j = 0; j < PP; ++j) {
        if (j >= np) break;
        const int l = t0 + j * NT;
        f(2 * j, l, l < half);
        f(2 * j + 1, l + half, l + half < m && l < half);
      }
    } else {
#pragma unroll 2
      for (int i = tid; i < m; i += NT) f(0, i, true);
    }
  };

  // set-up: inverse diagonal, x = 0, r64 = b, |b|^2; the matrix
  double s2 = 0.0;
  bool bad = false;
  {
    const uint16_t* __restrict__ col = at_entry(a.d.ell_col);
    const float* __restrict__ v32 = at_entry(a.d.ell_val32);
    const double* __restrict__ b = at_row(a.b);
    double* __restrict__ x = at_row(a.x);
    double* __restrict__ r64 = at_row(a.r64);
    for (int l = tid; l < half; l += NT) {
      const int h = min(l + half, m - 1);
#pragma unroll 4
      for (int k = 0; k < Ks; ++k) {
        const int64_t e = (int64_t)k * n;
        sval[k * m + l] = v32[e + l];
        sval[k * m + h] = v32[e + h];
        scol[k * half + l] = (uint32_t)(col[e + l] - wlo) | ((uint32_t)(col[e + h] - wlo) << 16);
      }
    }
    each([&](int j, int i, bool ok) {
      float dg = 0.f;
      if (ok) {
#pragma unroll 1
        for (int k = 0; k < W; ++k) {
          const int64_t e = (int64_t)k * n + i;
          if (col[e] == f0 + i) dg += v32[e];
        }
        bad |= !(dg > 0.f);
        G(j, i) = 1.f / dg;
      }
    });
    for (int i = tid; i < m; i += NT) {
      x[i] = 0.0;
      const double bi = b[i];
      r64[i] = bi;
      s2 += bi * bi;
    }
  }
  s2 = crew.sum(s2);  // also publishes the windows
  const double nbad = crew.sum(bad ? 1.0 : 0.0);
  // scal: |b|, |r|, |r| / |b|, 1 / |r|
  double* const scal = crew.S.scal;
  if (tid == 0) scal[0] = scal[1] = sqrt(s2);
  __syncthreads();
  // What `pown` holds, to the CTAs whose windows have these rows: p into the window, or
  // z into hz (the window without that CTA's own rows).  By the warps from 2 on, after a
  // barrier on pown; warp w serves CTA w mod TEAM.
  constexpr int PW = (Crew<NT>::NW - 2) / TEAM ? (Crew<NT>::NW - 2) / TEAM : 1;
  auto publish = [&](bool z) {
    const int w = (tid >> 5) - 2;
    if (w < 0) return;
    for (int v = w; v < TEAM * PW; v += Crew<NT>::NW - 2) {
      const int t = v % TEAM;
      if (t == crew.rank) continue;
      const int lo = crew.S.lo[t], hi = crew.S.hi[t];
      const int skip = z ? hi - lo + 1 - (t < crew.rank ? chunk : 0) : 0;
      const unsigned dst = remote(p, t) + 4u * (unsigned)(f0 - lo + skip);
      const int last = min(m - 1, hi - f0);
      for (int i = max(0, lo - f0) + (v / TEAM) * 32 + (tid & 31); i <= last; i += 32 * PW)
        put(dst + 4u * (unsigned)i, pown[i]);
    }
  };
  int status = TG_OK, it_total = 0, n_outer = 0;
  if (nbad > 0.0) {
    status = TG_ERR_BREAKDOWN;  // a non-positive diagonal entry: not SPD
    if (tid == 0) scal[2] = 1.0;
  } else if (!(scal[0] > 0.0)) {
    if (tid == 0) scal[2] = 0.0;
  } else {
    for (;;) {
      if (tid == 0) {
        scal[2] = scal[1] / scal[0];
        scal[3] = 1.0 / scal[1];
      }
      __syncthreads();
      if (scal[2] <= a.rtol) break;
      if (n_outer >= a.max_outer) { status = TG_ERR_NOT_CONVERGED; break; }
      ++n_outer;
      // inner FP32 CG on A d = r64 / |r64|
      const double inv_rn = scal[3];
      DotAcc<float> rz_acc, rr_acc;
      const double* __restrict__ r64 = at_row(a.r64);
      each([&](int j, int i, bool ok) {
        const float ri = ok ? (float)(r64[i] * inv_rn) : 0.f;
        const float zi = ok ? ri * G(j, i) : 0.f;
        R(j, i) = ri;
        D(j, i) = 0.f;
        Pv(j, i) = zi;
        if (PP > 0 && ok) pown[i] = zi;
        rz_acc.add(ri, zi);
        rr_acc.add(ri, ri);
      });
      if (crew.size > 1) {
        __syncthreads();
        publish(false);
      }
      const float2 t2[2] = {{rz_acc.hi, rz_acc.lo}, {rr_acc.hi, rr_acc.lo}};
      Total32 kept;  // r.z in thread 0, the |r|^2 to stop at in thread 32
      crew.sum(t2, [] {}, [&](int k, const Total32& t) {  // also publishes p
        kept = t;
        if (k == 1) kept = Total32::of(a.inner_rtol * a.inner_rtol * t.value());
      });
      bool broke = false;
      for (int it = 0; it < a.max_inner; ++it) {
        DotAcc<float> pq_acc;
        if constexpr (PP > 0) {
          spmv_pairs<NT, PP>(np, vq, p, sval, scol, m, half, Ks, W, n, wlo, at_entry(a.d.ell_val32),
                             at_entry(a.d.ell_col));
          each([&](int j, int i, bool ok) {
            if (!ok) vq[j] = 0.f;
            pq_acc.add(vp[j], vq[j]);
          });
        } else {
          const uint16_t* __restrict__ col = at_entry(a.d.ell_col);
          const float* __restrict__ v32 = at_entry(a.d.ell_val32);
          for (int l0 = tid; l0 < half; l0 += 2 * NT) {
            const int l1 = min(l0 + NT, half - 1);
            float s[4] = {0.f, 0.f, 0.f, 0.f};
            const float* v = sval;
            const uint32_t* c = scol;
#pragma unroll 4
            for (int k = 0; k < Ks; ++k) {
              const uint32_t c0 = c[l0], c1 = c[l1];
              s[0] = fmaf(v[l0], p[c0 & 0xffffu], s[0]);
              s[1] = fmaf(v[l0 + half], p[c0 >> 16], s[1]);
              s[2] = fmaf(v[l1], p[c1 & 0xffffu], s[2]);
              s[3] = fmaf(v[l1 + half], p[c1 >> 16], s[3]);
              v += m;
              c += half;
            }
            const int h0 = min(l0 + half, m - 1), h1 = min(l1 + half, m - 1);
#pragma unroll 2
            for (int k = Ks; k < W; ++k) {
              const int64_t e = (int64_t)k * n;
              s[0] = fmaf(v32[e + l0], p[col[e + l0] - wlo], s[0]);
              s[1] = fmaf(v32[e + h0], p[col[e + h0] - wlo], s[1]);
              s[2] = fmaf(v32[e + l1], p[col[e + l1] - wlo], s[2]);
              s[3] = fmaf(v32[e + h1], p[col[e + h1] - wlo], s[3]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int i = (u < 2 ? l0 : l1) + (u & 1) * half;
              if (i < m && (u < 2 || l0 + NT < half)) {
                Q(u, i) = s[u];
                pq_acc.add(pown[i], s[u]);
              }
            }
          }
        }
        const float2 t1[1] = {{pq_acc.hi, pq_acc.lo}};
        crew.sum(t1, [] {}, [&](int, const Total32& t) {
          crew.S.ratio = t.positive() && t.finite() ? kept.over(t) : NAN;
        });
        ++it_total;
        const float alpha = crew.S.ratio;
        if (isnan(alpha)) { broke = true; break; }
        DotAcc<float> rz2, rr2;
        each([&](int j, int i, bool ok) {
          D(j, i) = fmaf(alpha, Pv(j, i), D(j, i));
          const float ri = fmaf(-alpha, Q(j, i), R(j, i));
          R(j, i) = ri;
          const float zi = ri * G(j, i);
          if constexpr (PP > 0) vq[j] = zi;  // A p is not needed any more
          rz2.add(ri, zi);
          rr2.add(ri, ri);
          if (PP > 0 && crew.size > 1 && ok) pown[i] = zi;  // p itself is in registers
        });
        const float2 t3[2] = {{rz2.hi, rz2.lo}, {rr2.hi, rr2.lo}};
        crew.sum(
            t3,
            [&] {
              if (PP > 0 && crew.size > 1) publish(true);
            },
            [&](int k, const Total32& t) {
              if (k == 0) {
                crew.S.ratio = t.over(kept);
                kept = t;
              } else {
                crew.S.state = !t.finite() ? 2 : (t.at_most(kept) ? 1 : 0);
              }
            });
        const int state = crew.S.state;
        if (state) {
          broke = state == 2;
          break;
        }
        const float beta = crew.S.ratio;
        each([&](int j, int i, bool ok) {
          const float pi = fmaf(beta, Pv(j, i), PP > 0 ? Q(j, i) : R(j, i) * G(j, i));
          Pv(j, i) = pi;
          if (PP > 0 && ok) pown[i] = pi;
        });
        if constexpr (PP > 0) {
          // the window's other rows: their p is updated here as in their own CTA
          if (crew.size > 1) {
            const int below = f0 - wlo;
            for (int i = tid; i < nw - m; i += NT) {
              float& pi = p[i < below ? i : i + m];
              pi = fmaf(beta, pi, hz[i]);
            }
          }
          __syncthreads();
        } else {
          __syncthreads();
          if (crew.size > 1) {
            publish(false);
            cluster_sync();
          }
        }
      }
      if (broke) { status = TG_ERR_BREAKDOWN; break; }
      // refinement: x += |r64| d, r64 = b - A64 x (FP64)
      double* x = at_row(a.x);
      each([&](int j, int i, bool ok) {
        if (ok) x[i] += scal[1] * (double)D(j, i);
      });
      if (crew.size > 1) __threadfence();
      crew.sync();
      double u2 = 0.0;
      const double* xs = x - f0;
      const uint16_t* __restrict__ col = at_entry(a.d.ell_col);
      const double* __restrict__ v64 = at_entry(a.d.ell_val64);
      const double* __restrict__ b = at_row(a.b);
      double* __restrict__ rs = at_row(a.r64);
      for (int i = tid; i < m; i += NT) {
        double s = b[i];
#pragma unroll 4
        for (int k = 0; k < W; ++k) {
          const int64_t e = (int64_t)k * n + i;
          s -= v64[e] * __ldcg(xs + col[e]);
        }
        rs[i] = s;
        u2 += s * s;
      }
      u2 = crew.sum(u2);
      if (tid == 0) scal[1] = sqrt(u2);
      __syncthreads();
      if (!isfinite(scal[1])) { status = TG_ERR_BREAKDOWN; break; }
    }
  }
  if (tid == 0 && crew.rank == 0) {
    a.iters[sys] = it_total;
    a.outer[sys] = n_outer;
    a.rel_res[sys] = scal[2];
    a.status[sys] = status;
  }
  crew.sync();  // shared memory is reused by the next system
}

template <int NT, int PP, bool ALL>
__device__ void solve_system(const BatchArgs& a, int sys, float* smem, Crew<NT>& crew) {
  const int n = (int)(a.d.row_ofs[sys + 1] - a.d.row_ofs[sys]);
  if (n < 0 || n > a.d.max_rows || a.d.ell_width[sys] < 0) {  // inconsistent: skip the system
    if (threadIdx.x == 0) {
      a.iters[sys] = 0;
      a.outer[sys] = 0;
      a.rel_res[sys] = 1.0;
      a.status[sys] = TG_ERR_VALUE;
    }
    __syncthreads();
    return;
  }
  if constexpr (ALL) {
    if ((n + crew.size - 1) / crew.size > 2 * NT * PP) return solve_rows<NT, 0>(a, sys, smem, crew);
  }
  solve_rows<NT, PP>(a, sys, smem, crew);
}

template <int NT, int PP, bool ALL, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) __cluster_dims__(TEAM, 1, 1)
    batch_solve_kernel(BatchArgs a) {
  extern __shared__ __align__(16) float smem[];
  __shared__ typename Crew<NT>::Shared S;
  const int me = (int)cluster_rank();
  {
    Crew<NT> crew{S, TEAM, me, 0};
    for (;;) {
      if (me == 0 && threadIdx.x < 32) {
        const int k = take(a.d, a.counter, true);
        if (threadIdx.x < TEAM) put(remote(&S.next, threadIdx.x), k);
      }
      cluster_sync();
      const int k = S.next;
      if (k >= a.d.n_systems) break;
      solve_system<NT, PP, ALL>(a, a.d.order[k], smem, crew);
    }
  }
  __syncthreads();
  Crew<NT> crew{S, 1, 0, 0};
  for (;;) {
    if (threadIdx.x < 32) {
      const int k = take(a.d, a.counter + 1, false);
      if (threadIdx.x == 0) S.next = k;
    }
    __syncthreads();
    const int k = S.next;
    if (k >= a.d.n_systems) break;
    solve_system<NT, PP, ALL>(a, a.d.order[k], smem, crew);
  }
}

// ELL conversion: thread per global row (row -> system by binary search on row_ofs)
__global__ void ell_from_csr_kernel(tg_batch_desc d, int64_t n_rows, const int32_t* __restrict__ indptr,
                                    const int32_t* __restrict__ indices,
                                    const double* __restrict__ data, uint16_t* col, float* v32,
                                    double* v64, int* bad) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_rows) return;
  int lo = 0, hi = d.n_systems;  // largest s with row_ofs[s] <= g
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (d.row_ofs[mid] <= g) lo = mid; else hi = mid;
  }
  const int s = lo;
  const int64_t r0 = d.row_ofs[s];
  const int n = (int)(d.row_ofs[s + 1] - r0);
  const int i = (int)(g - r0);
  const int W = d.ell_width[s];
  const int64_t e0 = d.ell_ofs[s];
  const int j0 = indptr[g], len = indptr[g + 1] - j0;
  if (len > W) { atomicExch(bad, 1); return; }
  for (int k = 0; k < W; ++k) {
    const int64_t e = e0 + (int64_t)k * n + i;
    if (k < len) {
      const int64_t c = (int64_t)indices[j0 + k] - r0;
      if (c < 0 || c >= n) {  // a coupling between two systems: not block diagonal
        atomicExch(bad, 2);
        col[e] = (uint16_t)i;
        v32[e] = 0.f;
        v64[e] = 0.0;
        continue;
      }
      col[e] = (uint16_t)c;
      v64[e] = data[j0 + k];
      v32[e] = (float)data[j0 + k];
    } else {
      col[e] = (uint16_t)i;
      v32[e] = 0.f;
      v64[e] = 0.0;
    }
  }
}

int desc_check(const tg_batch_desc* d) {
  if (!d) return set_error(TG_ERR_VALUE, "batch description must not be NULL");
  if (d->n_systems < 0) return set_error(TG_ERR_VALUE, "n_systems must be >= 0");
  if (d->max_rows < 0 || d->max_rows > BATCH_MAX_ROWS)
    return set_error(TG_ERR_UNSUPPORTED, "batched solve: a system has %d rows; at most %d are supported",
                     d->max_rows, BATCH_MAX_ROWS);
  if (d->n_systems > 0) {
    TG_TRY(check_ptr(d->row_ofs, "row_ofs"));
    TG_TRY(check_ptr(d->ell_ofs, "ell_ofs"));
    TG_TRY(check_ptr(d->ell_width, "ell_width"));
    TG_TRY(check_ptr(d->ell_col, "ell_col"));
    TG_TRY(check_ptr(d->ell_val32, "ell_val32"));
    TG_TRY(check_ptr(d->ell_val64, "ell_val64"));
  }
  return TG_OK;
}

}  // namespace
}  // namespace tg

using namespace tg;

extern "C" int tg_batch_ell_from_csr(const tg_batch_desc* desc, int64_t n_rows,
                                     const int32_t* indptr, const int32_t* indices,
                                     const double* data, int32_t* bad_flag, void* stream) {
  TG_TRY(desc_check(desc));
  if (n_rows < 0) return set_error(TG_ERR_VALUE, "n_rows must be >= 0");
  if (n_rows == 0) return TG_OK;
  TG_TRY(check_ptr(indptr, "indptr"));
  TG_TRY(check_ptr(indices, "indices"));
  TG_TRY(check_ptr(data, "data"));
  TG_TRY(check_ptr(bad_flag, "bad_flag"));
  ell_from_csr_kernel<<<grid_for(n_rows, 256), 256, 0, as_stream(stream)>>>(
      *desc, n_rows, indptr, indices, data, const_cast<uint16_t*>(desc->ell_col),
      const_cast<float*>(desc->ell_val32), const_cast<double*>(desc->ell_val64), bad_flag);
  return launch_check("tg_batch_ell_from_csr");
}

extern "C" size_t tg_batch_workspace_bytes(int64_t n_rows) {
  const size_t n = (size_t)(n_rows > 0 ? n_rows : 0);
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  return al(4 * n * sizeof(float)) + al(n * sizeof(double)) + 256;
}

extern "C" int tg_batch_solve(const tg_batch_desc* desc, int64_t n_rows, const double* b, double* x,
                              double rtol, double inner_rtol, int max_outer, int max_inner,
                              int threads, int ctas_per_sm, void* workspace, size_t workspace_bytes,
                              int32_t* iters, int32_t* outer, double* rel_res, int32_t* status,
                              void* stream) {
  TG_TRY(desc_check(desc));
  if (n_rows < 0) return set_error(TG_ERR_VALUE, "n_rows must be >= 0");
  if (!(rtol > 0.0) || !(inner_rtol > 0.0) || inner_rtol >= 1.0)
    return set_error(TG_ERR_VALUE, "need rtol > 0 and 0 < inner_rtol < 1");
  if (max_outer < 0 || max_inner <= 0) return set_error(TG_ERR_VALUE, "bad iteration limits");
  if (workspace_bytes < tg_batch_workspace_bytes(n_rows))
    return set_error(TG_ERR_WORKSPACE, "tg_batch_solve: workspace too small");
  if (desc->n_systems == 0) return TG_OK;
  TG_TRY(check_ptr(desc->order, "order"));
  TG_TRY(check_ptr(b, "b"));
  TG_TRY(check_ptr(x, "x"));
  TG_TRY(check_ptr(iters, "iters"));
  TG_TRY(check_ptr(outer, "outer"));
  TG_TRY(check_ptr(rel_res, "rel_res"));
  TG_TRY(check_ptr(status, "status"));
  TG_TRY(check_ptr(workspace, "workspace"));
  const size_t n = (size_t)n_rows;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  char* w = (char*)workspace;
  BatchArgs a;
  a.d = *desc;
  a.b = b;
  a.x = x;
  a.q = (float*)w;
  a.r = a.q + n;
  a.dv = a.r + n;
  a.idiag = a.dv + n;
  a.r64 = (double*)(w + al(4 * n * sizeof(float)));
  a.counter = (unsigned*)(w + al(4 * n * sizeof(float)) + al(n * sizeof(double)));
  a.rtol = rtol;
  a.inner_rtol = inner_rtol;
  a.max_outer = max_outer;
  a.max_inner = max_inner;
  a.iters = iters;
  a.outer = outer;
  a.rel_res = rel_res;
  a.status = status;
  cudaStream_t st = as_stream(stream);
  TG_TRY(cuda_check(cudaMemsetAsync(a.counter, 0, 2 * sizeof(unsigned), st),
                    "tg_batch_solve: counter reset"));
  int dev = 0, sms = 0;
  TG_TRY(cuda_check(cudaGetDevice(&dev), "cudaGetDevice"));
  TG_TRY(cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count"));
  auto go = [&](auto kern, int nt, int fit) -> int {
    // p of the largest system has to fit whatever its columns; a larger one takes the SM
    const size_t smem = std::max((size_t)batch_smem(nt, fit),
                                 ((size_t)desc->max_rows * sizeof(float) + 15) & ~(size_t)15);
    a.smem_floats = (int)(smem / sizeof(float));
    {
      // the attribute only grows: graphs captured with larger systems stay launchable
      static std::mutex mu;
      static std::map<std::pair<const void*, int>, size_t> attr;
      std::lock_guard<std::mutex> g(mu);
      size_t& cur = attr[std::make_pair((const void*)kern, dev)];
      if (smem > cur) {
        TG_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem),
                          "tg_batch_solve: shared memory attribute"));
        cur = smem;
      }
    }
    int per_sm = 0;
    TG_TRY(cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, smem),
                      "tg_batch_solve: occupancy"));
    if (per_sm <= 0)
      return set_error(TG_ERR_UNSUPPORTED, "tg_batch_solve: kernel does not fit on an SM");
    const int want = ctas_per_sm > 0 ? std::min(ctas_per_sm, per_sm) : per_sm;
    const int clusters = std::max(1, std::min(desc->n_systems, sms * want / TEAM));
    const int grid = clusters * TEAM;
    kern<<<grid, nt, smem, st>>>(a);
    return launch_check("tg_batch_solve");
  };
  // Many small systems (two or more for every CTA at four to an SM): few registers and
  // little shared memory, four CTAs of 256 on an SM instead of two.  With sums in float pairs,
  // 4,096 squares of 6..24: 1.6 ms, 2.2 with two to an SM; 700 of 6..31: 0.88 ms, 0.52 with
  // two (the largest systems then share an SM with fewer others).  The rows of a thread and
  // every sum are the same.
  const bool many = desc->n_systems >= 8 * sms;
  switch (threads) {
    case 128:
      return many && desc->max_rows <= 512 ? go(batch_solve_kernel<128, 2, false, 8>, 128, 8)
                                           : go(batch_solve_kernel<128, 10, true, 2>, 128, 2);
    case 256:
      return many && desc->max_rows <= 1024 ? go(batch_solve_kernel<256, 2, false, 4>, 256, 4)
                                            : go(batch_solve_kernel<256, 5, true, 2>, 256, 2);
    case 512: return go(batch_solve_kernel<512, 2, true, 2>, 512, 2);
    default: return set_error(TG_ERR_VALUE, "threads must be 128, 256 or 512");
  }
}
