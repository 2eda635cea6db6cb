// Colored compressed Hessian (K6) and its decompression into CSR values, and the CSR
// values straight from the element tangents (hessian_csr_kernel) on a mesh's own pattern.
//
// Reference (tatva/sparse/base.py):
//   colored_jacobian_batch (:230-270): Jc[:, c] = jvp(grad E, u, seed_c),
//        seed_c = (colors == c) as 1.0 / 0.0  (:259), Jc has shape (N, C) (:268-270)
//   compute_rows_cols (:108-136): rows = repeat(arange(N), diff(indptr)),
//        col_colors = colors[indices]
//   jacfwd decompression (:173): data = Jc[rows, col_colors]
//
// Jc is computed here from element tangents instead of C full HVPs:
//   Jc[i, c] = sum_e sum_{(b,k) in e : color(dof(b,k)) = c} K_e[(a,i), (b,k)]
// which equals sum_{j: color j = c} H[i, j] because every element-local dof pair is
// inside the pattern.  Node-centric: a thread owns one node's V rows of Jc and adds the
// row blocks of the node's incident (element, corner) pairs in incidence order
// (ascending element): deterministic, no atomics, no colouring of the elements.  With
// a distance-2 colouring each colour occurs at most once per row, so a row is a dense
// vector over the colours; the thread accumulates it in shared memory and the CTA
// writes its consecutive nodes' rows as one contiguous, coalesced block of Jc.
#include "tg_common.cuh"
#include "tg_dispatch.cuh"
#include "tg_hex.cuh"
#include "tg_materials.cuh"

namespace tg {

// One quadrature point's share of the row block of corner a.  For every law here the
// tangent block of corners (a, b) is
//   K_ab[i][k] = wd (mu delta_ik G_a.G_b + c1 g_a[k] g_b[i] + lam g_a[i] g_b[k])
// with the shape gradients G in the undeformed cell and g = G, c1 = mu (linear elastic),
// or g the gradients in the deformed cell and c1 = mu - lam ln J (Neo-Hookean: the two
// F^-T of each term of d2psi/dF2 take G to g); Poisson has the first term alone.  s: the
// first term, ca = wd c1 g_a, la = wd lam g_a.
template <int V, int COLS, class T>
__device__ __forceinline__ void add_tangent_block(T (&rb)[V][COLS], int b, T s, const T (&ca)[V],
                                                  const T (&la)[V], const T (&gb)[V]) {
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) {
      T v = rb[i][b * V + k];
      if constexpr (V > 1) v = fma(gb[k], la[i], fma(gb[i], ca[k], v));
      if (i == k) v += s;
      rb[i][b * V + k] = v;
    }
}

// coordinates and, where the law needs them, displacements of an element's nodes
template <int ET, int MAT, class T>
struct ElementNodes {
  static constexpr bool NH = MAT == TG_NEO_HOOKEAN;
  T X[Elem<ET>::NN][Elem<ET>::D], U[Elem<ET>::NN][NH ? 3 : 1];
  __device__ __forceinline__ void load(const T* __restrict__ coords, const T* __restrict__ u,
                                       const int (&nid)[Elem<ET>::NN]) {
    constexpr int D = Elem<ET>::D;
#pragma unroll
    for (int b = 0; b < Elem<ET>::NN; ++b)
#pragma unroll
      for (int d = 0; d < D; ++d) {
        X[b][d] = coords[(int64_t)nid[b] * D + d];
        if constexpr (NH) U[b][d] = u[(int64_t)nid[b] * 3 + d];
      }
  }
};

// Row block K_e[(a, i), (b, k)] (i, k < V, b < NN) of element e's tangent at u,
// rb[i][b V + k]
template <int ET, int MAT, class T>
__device__ __forceinline__ void element_row_block(
    ElementNodes<ET, MAT, T>& nodes, T p0, T p1, const T* __restrict__ eparam, int64_t e,
    int a, T (&rb)[LawDims<MAT, Elem<ET>::D>::V][Elem<ET>::NN * LawDims<MAT, Elem<ET>::D>::V]) {
  using E = Elem<ET>;
  constexpr int NN = E::NN, D = E::D, V = LawDims<MAT, D>::V;
  constexpr bool NH = MAT == TG_NEO_HOOKEAN;
  auto& X = nodes.X;  // (overwritten)
  auto& U = nodes.U;
  const T mu = eparam ? eparam[e] : p0, lam = MAT == TG_POISSON ? T(0) : p1;
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int c = 0; c < NN * V; ++c) rb[i][c] = T(0);
  if constexpr (E::SIMPLEX) {
    T J[D][D], R[D][D], G[NN][D], g[NN][D];
#pragma unroll
    for (int k = 0; k < D; ++k)
#pragma unroll
      for (int d = 0; d < D; ++d) J[k][d] = X[k + 1][d] - X[0][d];
    auto nodes_of = [&](const T (&Ri)[D][D], T (&out)[NN][D]) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        T s0 = T(0);
#pragma unroll
        for (int k = 0; k < D; ++k) {
          out[k + 1][d] = Ri[d][k];
          s0 -= Ri[d][k];
        }
        out[0][d] = s0;
      }
    };
    T wd, c1;
    if constexpr (NH) {
      T Du[3][3], j[3][3], r[3][3], rdet;
      wd = inv3(J, R, rdet) * E::template w<T>(0);
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          Du[k][d] = U[k + 1][d] - U[0][d];
          j[k][d] = J[k][d] + Du[k][d];
        }
      const T dj = inv3(j, r);
      c1 = wd * (mu - lam * log_volume_ratio(J, R, rdet, j, r, dj, Du));
      nodes_of(r, g);
    } else {
      wd = invD<T, D>(J, R) * E::template w<T>(0);
      c1 = wd * mu;
    }
    nodes_of(R, G);
    T Ga[D], ca[V], la[V];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      Ga[d] = G[0][d];
      T ga = NH ? g[0][d] : T(0);
#pragma unroll
      for (int b = 1; b < NN; ++b)
        if (b == a) {
          Ga[d] = G[b][d];
          if constexpr (NH) ga = g[b][d];
        }
      if (!NH) ga = Ga[d];
      if constexpr (V > 1) {
        ca[d] = c1 * ga;
        la[d] = wd * lam * ga;
      }
      Ga[d] *= wd * mu;
    }
#pragma unroll
    for (int b = 0; b < NN; ++b) {
      T s = Ga[0] * G[b][0];
#pragma unroll
      for (int d = 1; d < D; ++d) s = fma(Ga[d], G[b][d], s);
      T gb[V];
#pragma unroll
      for (int i = 0; i < V; ++i) gb[i] = NH ? g[b][i] : G[b][i];
      add_tangent_block<V, NN * V, T>(rb, b, s, ca, la, gb);
    }
  } else {
    // Hex8, modal form (tg_hex.cuh).  8 dN_b/dxi at a point are products of two of the
    // factors 1 +- x_l; the metric C = R^T R gives G_a.G_b without forming the G.
    hex_modes8<T, 3>(X);
    hex_scale_gauss<T, 3>(X);
    if constexpr (NH) {
      hex_modes8<T, 3>(U);
      hex_scale_gauss<T, 3>(U);
    }
    const T sa[3] = {T(E::s(a, 0)), T(E::s(a, 1)), T(E::s(a, 2))};
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
      T sx, sy;
      hex_pair_sides<T>(q & 3, sx, sy);
      const int up = q >> 2;
      const T sz = up ? T(1) : T(-1), gp = T(HEX_GAUSS);
      T J[3][3], R[3][3], r[3][3], rdet;
      HexPair<T, 3> pr;
      pr.set(X, sx, sy);
      pr.at(up, J);
      const T wd = inv3(J, R, rdet) * T(1.0 / 512);
      T c1 = wd * mu;
      if constexpr (NH) {
        T Du[3][3], j[3][3];
        pr.set(U, sx, sy);
        pr.at(up, Du);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
          for (int d = 0; d < 3; ++d) j[k][d] = J[k][d] + Du[k][d];
        const T dj = inv3(j, r);
        c1 = wd * (mu - lam * log_volume_ratio(J, R, rdet, j, r, dj, Du));
      }
      // f[l][side]: 1 + s x_l of the corners on that side along axis l
      const T f[3][2] = {{T(1) - sx * gp, T(1) + sx * gp},
                         {T(1) - sy * gp, T(1) + sy * gp},
                         {T(1) - sz * gp, T(1) + sz * gp}};
      T pa[3];  // 8 dN_a/dxi, corner a at run time
      {
        const T fa[3] = {fma(sa[0], sx * gp, T(1)), fma(sa[1], sy * gp, T(1)),
                         fma(sa[2], sz * gp, T(1))};
        pa[0] = sa[0] * fa[1] * fa[2];
        pa[1] = sa[1] * fa[0] * fa[2];
        pa[2] = sa[2] * fa[0] * fa[1];
      }
      T Ca[3], ca[V], la[V];  // wd mu C pa; c1 g_a, lam g_a
      {
        T Ga[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          Ga[d] = fma(R[d][2], pa[2], fma(R[d][1], pa[1], R[d][0] * pa[0]));
        const T m = wd * mu;
#pragma unroll
        for (int k = 0; k < 3; ++k)
          Ca[k] = m * fma(R[2][k], Ga[2], fma(R[1][k], Ga[1], R[0][k] * Ga[0]));
        if constexpr (V > 1) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const T ga = NH ? fma(r[d][2], pa[2], fma(r[d][1], pa[1], r[d][0] * pa[0])) : Ga[d];
            ca[d] = c1 * ga;
            la[d] = wd * lam * ga;
          }
        }
      }
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int b0 = E::s(b, 0) > 0, b1 = E::s(b, 1) > 0, b2 = E::s(b, 2) > 0;
        const T q0 = f[1][b1] * f[2][b2], q1 = f[0][b0] * f[2][b2], q2 = f[0][b0] * f[1][b1];
        const T pb[3] = {b0 ? q0 : -q0, b1 ? q1 : -q1, b2 ? q2 : -q2};
        const T s = fma(Ca[2], pb[2], fma(Ca[1], pb[1], Ca[0] * pb[0]));
        T gb[V];
        if constexpr (V > 1) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            if constexpr (NH)
              gb[d] = fma(r[d][2], pb[2], fma(r[d][1], pb[1], r[d][0] * pb[0]));
            else
              gb[d] = fma(R[d][2], pb[2], fma(R[d][1], pb[1], R[d][0] * pb[0]));
          }
        } else {
          gb[0] = T(0);
        }
        add_tangent_block<V, NN * V, T>(rb, b, s, ca, la, gb);
      }
    }
  }
}

// ------------------------------------------------------------------ straight into CSR
// The CSR values without the compressed matrix: thread = node, a warp's 32 nodes = one
// contiguous run of `data`.  The node's row block (V rows of V deg values, the order of
// the CSR rows) is accumulated in shared memory with word e of lane l at e 32 + l: every
// lane stays in its own bank whatever word it adds to, so the scattered adds never
// conflict.  slots[NP j + b]: position of corner b's node among the columns of incidence
// entry j's node (tg_csr_slots).  Sums run in incidence order (ascending element).
// What bounds it is on chip: about 250 arithmetic instructions and 36 shared-memory adds
// per (Tet4 element, corner) and the gathers of the element's nodes; the data is written
// once and neither column indices nor colours are read.  Kuhn 56^3 jittered, Neo-Hookean
// FP32 (1.05 M tets, 24 M values): 187 us, 201 without the loads run ahead; compressed Hessian
// and decompression, which it replaces on the mesh's own pattern, 717 + 125 us.
template <int ET>
constexpr int slot_pad() { return Elem<ET>::NN <= 4 ? 4 : 8; }
constexpr int CSR_WARPS = 2;   // warps per CTA, at most (csr_warps)
constexpr int CSR_SLAB = 16;   // row words a lane hands over at a time when writing

template <int ET, int MAT, class T>
__global__ void __launch_bounds__(32 * CSR_WARPS)
    hessian_csr_kernel(const T* __restrict__ coords, const int32_t* __restrict__ conn,
                       bool conn16, const T* __restrict__ u, T p0, T p1,
                       const T* __restrict__ eparam,
                       int64_t n_nodes, const int32_t* __restrict__ inc_ptr,
                       const int32_t* __restrict__ inc_idx, const uint16_t* __restrict__ slots,
                       const int32_t* __restrict__ indptr, int row_words, T* __restrict__ data) {
  using E = Elem<ET>;
  constexpr int NN = E::NN, V = LawDims<MAT, E::D>::V, NP = slot_pad<ET>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* acc = reinterpret_cast<T*>(smem_raw) + (size_t)warp * row_words * 32;
  const int64_t n = ((int64_t)blockIdx.x * (blockDim.x >> 5) + warp) * 32 + lane;
  const bool live = n < n_nodes;
  const int base = live ? __ldg(indptr + V * n) : 0;
  const int len = live ? __ldg(indptr + V * n + V) - base : 0;
  const int L = len / V;  // the length of each of the node's rows
  for (int k = 0; k < len; ++k) acc[k * 32 + lane] = T(0);
  const int j0 = live ? __ldg(inc_ptr + n) : 0, last = (live ? __ldg(inc_ptr + n + 1) : 0) - 1;
  // The loads of an incidence entry depend on one another (entry, node ids and slots,
  // coordinates), so they run ahead: the entry by two turns, ids and slots by one and, for
  // simplices, the coordinates from before the adds of the turn before.  At 11 warps an SM
  // (shared memory) their latency was a third of the time.  Scalar laws (a ninth of the adds
  // and of the shared memory, hence more warps) lose by it: Poisson 81.7 -> 84.8 us.
  constexpr bool AHEAD = V > 1, NODES_AHEAD = AHEAD && E::SIMPLEX;
  auto ids = [&](int ea, int (&nid)[NN]) {
    const int32_t* row = conn + (int64_t)(ea / NN) * NN;
    if (NN % 4 == 0 && conn16) {
#pragma unroll
      for (int b = 0; b < NN / 4; ++b) {
        const int4 c = __ldg(reinterpret_cast<const int4*>(row) + b);
        nid[4 * b] = c.x;
        nid[4 * b + 1] = c.y;
        nid[4 * b + 2] = c.z;
        nid[4 * b + 3] = c.w;
      }
    } else {
#pragma unroll
      for (int b = 0; b < NN; ++b) nid[b] = __ldg(row + b);
    }
  };
  if (j0 <= last) {
    int ea = 0, ea1 = 0, nid[NN];
    LconnRaw<NP> raw;
    ElementNodes<ET, MAT, T> nodes;
    if constexpr (AHEAD) {
      ea = __ldg(inc_idx + j0);
      ea1 = __ldg(inc_idx + min(j0 + 1, last));
      ids(ea, nid);
      raw.load(slots + (int64_t)j0 * NP);
    }
    if constexpr (NODES_AHEAD) nodes.load(coords, u, nid);
    for (int j = j0; j <= last; ++j) {
      if constexpr (!AHEAD) {
        ea = __ldg(inc_idx + j);
        raw.load(slots + (int64_t)j * NP);
        ids(ea, nid);
      }
      if constexpr (!NODES_AHEAD) nodes.load(coords, u, nid);
      int sl[NP], ea2 = 0;
      raw.unpack(sl);
      if constexpr (AHEAD) {
        ea2 = __ldg(inc_idx + min(j + 2, last));
        ids(ea1, nid);
        raw.load(slots + (int64_t)min(j + 1, last) * NP);
      }
      T rb[V][NN * V];
      element_row_block<ET, MAT, T>(nodes, p0, p1, eparam, ea / NN, ea % NN, rb);
      if constexpr (NODES_AHEAD) nodes.load(coords, u, nid);
#pragma unroll
      for (int b = 0; b < NN; ++b) {
        T* w = acc + (V * sl[b]) * 32 + lane;
        T t[V][V];
#pragma unroll
        for (int i = 0; i < V; ++i)
#pragma unroll
          for (int k = 0; k < V; ++k) t[i][k] = w[(i * L + k) * 32];
#pragma unroll
        for (int i = 0; i < V; ++i)
#pragma unroll
          for (int k = 0; k < V; ++k) w[(i * L + k) * 32] = t[i][k] + rb[i][b * V + k];
      }
      if constexpr (AHEAD) {
        ea = ea1;
        ea1 = ea2;
      }
    }
  }
  // write-out in slabs of CSR_SLAB words per node: each lane moves its slab from its own
  // bank to row l of a 32 x CSR_SLAB tile in the same place (columns XORed so that neither
  // side conflicts), then half a warp writes one node's slab
  int longest = len;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  const int half = lane >> 4, q = lane & 15;
  for (int s0 = 0; s0 < longest; s0 += CSR_SLAB) {
    T* tile = acc + s0 * 32;
    T v[CSR_SLAB];
#pragma unroll
    for (int k = 0; k < CSR_SLAB; ++k) v[k] = tile[k * 32 + lane];
    __syncwarp();
#pragma unroll
    for (int k = 0; k < CSR_SLAB; ++k) tile[lane * CSR_SLAB + (k ^ (lane >> 1))] = v[k];
    __syncwarp();
#pragma unroll 4
    for (int t = 0; t < 16; ++t) {
      const int m = 2 * t + half;
      const int bm = __shfl_sync(0xffffffffu, base, m), lm = __shfl_sync(0xffffffffu, len, m);
      if (s0 + q < lm) data[(int64_t)bm + s0 + q] = tile[m * CSR_SLAB + (q ^ (m >> 1))];
    }
  }
}

// Checks that a CSR pattern has the form hessian_csr_kernel writes and that a colouring
// separates its columns: per node, V rows of the same ascending columns in groups of V
// dofs of one node, all of different colours (then Jc[i, colour(j)] is H[i, j] alone).
// info[0] |= 1 where it does not; info[1]: the most columns (nodes) of a row.  CHECK_LANES
// lanes per node (rows of 7 to 81 columns); the colours seen so far as bits in shared memory.
// A node whose row is no longer than info[1] already was leaves it alone: one address, and
// most rows have the same length.
constexpr int SLOT_MAX_COLORS = 1024;
constexpr int CHECK_LANES = 8, CHECK_NODES = 128 / CHECK_LANES;
template <int V>
__global__ void __launch_bounds__(128)
    csr_pattern_check_kernel(int64_t n_nodes, int64_t nnz, const int32_t* __restrict__ indptr,
                             const int32_t* __restrict__ indices,
                             const int32_t* __restrict__ colors, int n_colors,
                             int32_t* __restrict__ info) {
  __shared__ unsigned seen[CHECK_NODES][SLOT_MAX_COLORS / 32 + 1];
  const int lane = threadIdx.x % CHECK_LANES, own = threadIdx.x / CHECK_LANES;
  const int64_t n = (int64_t)blockIdx.x * CHECK_NODES + own;
  for (int k = lane; k < SLOT_MAX_COLORS / 32; k += CHECK_LANES) seen[own][k] = 0u;
  __syncwarp();
  if (n >= n_nodes) return;
  const int64_t N = n_nodes * V;
  const int64_t r0 = __ldg(indptr + V * n);
  const int64_t L = __ldg(indptr + V * n + 1) - r0;
  bool good = r0 >= 0 && L >= 0 && L % V == 0 && r0 + V * L <= nnz && (n > 0 || r0 == 0);
  for (int i = 0; i < V; ++i)
    good = good && (__ldg(indptr + V * n + i + 1) - __ldg(indptr + V * n + i) == L);
  if (n == n_nodes - 1) good = good && r0 + V * L == nnz;
  if (good) {
    for (int64_t p = lane; p < L; p += CHECK_LANES) {
      const int64_t c = __ldg(indices + r0 + p);
      bool ok = c >= 0 && c < N;
      for (int i = 1; i < V; ++i) ok = ok && __ldg(indices + r0 + i * L + p) == c;
      if (p % V == 0) ok = ok && c % V == 0 && (p == 0 || __ldg(indices + r0 + p - 1) < c);
      else ok = ok && __ldg(indices + r0 + p - 1) == c - 1;
      if (ok) {
        const int col = __ldg(colors + c);
        ok = col >= 0 && col < n_colors;
        if (ok) ok = !(atomicOr(&seen[own][col >> 5], 1u << (col & 31)) >> (col & 31) & 1u);
      }
      good = good && ok;
    }
  }
  if (!good) atomicOr(info, 1);
  if (lane == 0 && good && (int)(L / V) > *(volatile int32_t*)(info + 1))
    atomicMax(info + 1, (int)(L / V));
}

// slots of the incidence entries (a thread per entry); info[0] |= 2 where a node of an
// element is not among the columns.  Runs after the check, on rows it found ascending.
// Bound: the chain of dependent loads of the searches; a thread per node went through them
// one after another.  Jacobian made and called once with this and the check, FP32 Poisson:
// Kuhn 40^3 292 -> 139 us, Tri3 400^2 275 -> 122 (the compressed Hessian's: 145 and 132).
template <int ET, int V>
__global__ void csr_slots_kernel(int64_t n_nodes, int64_t n_entries,
                                 const int32_t* __restrict__ conn,
                                 const int32_t* __restrict__ inc_ptr,
                                 const int32_t* __restrict__ inc_idx,
                                 const int32_t* __restrict__ indptr,
                                 const int32_t* __restrict__ indices,
                                 uint16_t* __restrict__ slots, int32_t* __restrict__ info) {
  constexpr int NN = Elem<ET>::NN, NP = slot_pad<ET>();
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n_entries || j >= __ldg(inc_ptr + n_nodes) || (*(volatile int32_t*)info & 1)) return;
  const int64_t ea = __ldg(inc_idx + j), n = __ldg(conn + ea);
  const int64_t r0 = __ldg(indptr + V * n);
  const int deg = (int)((__ldg(indptr + V * n + 1) - r0) / V);
  alignas(8) uint16_t row[NP];
#pragma unroll
  for (int b = 0; b < NP; ++b) {
    row[b] = 0;
    if (b >= NN) continue;
    const int64_t want = (int64_t)V * __ldg(conn + ea / NN * NN + b);
    int lo = 0, hi = deg;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(indices + r0 + (int64_t)V * mid) < want) lo = mid + 1;
      else hi = mid;
    }
    const bool found = lo < deg && lo < 65536 && __ldg(indices + r0 + (int64_t)V * lo) == want;
    if (!found) atomicOr(info, 2);
    row[b] = (uint16_t)(found ? lo : 0);
  }
#pragma unroll
  for (int b = 0; b < NP; b += 4)
    *reinterpret_cast<uint2*>(slots + j * NP + b) = *reinterpret_cast<const uint2*>(row + b);
}

// Thread t of the CTA owns node n0 + t.  ACC_SMEM: its V x C row block sits in shared
// memory at row t (stride V C + 1 words: conflict-free for the CTA's row-major write);
// otherwise (too many colours for shared memory) it accumulates in its own rows of
// Jc, which the caller zeroed.
template <int ET, int MAT, class T, bool ACC_SMEM>
__global__ void compressed_hessian_kernel(const T* __restrict__ coords,
                                          const int32_t* __restrict__ conn,
                                          const T* __restrict__ u, T p0, T p1,
                                          const T* __restrict__ eparam, int64_t n_nodes,
                                          const int32_t* __restrict__ inc_ptr,
                                          const int32_t* __restrict__ inc_idx,
                                          const int32_t* __restrict__ dof_colors, int n_colors,
                                          T* __restrict__ Jc) {
  using E = Elem<ET>;
  using L = Law<MAT, E::D, T>;
  constexpr int NN = E::NN, V = L::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  const int row_words = V * n_colors;
  const int stride = row_words + 1;
  const int64_t n0 = (int64_t)blockIdx.x * blockDim.x;
  const int64_t n = n0 + threadIdx.x;
  T* acc_row = ACC_SMEM ? sm + (int64_t)threadIdx.x * stride : Jc + n * row_words;
  if (ACC_SMEM)
    for (int k = 0; k < row_words; ++k) acc_row[k] = T(0);
  if (n < n_nodes) {
    for (int j = __ldg(inc_ptr + n); j < __ldg(inc_ptr + n + 1); ++j) {
      const int ea = __ldg(inc_idx + j);
      const int64_t e = ea / NN;
      const int a = ea - (int)(e * NN);
      T rb[V][NN * V];
      int nid[NN];
#pragma unroll
      for (int b = 0; b < NN; ++b) nid[b] = __ldg(conn + e * NN + b);
      ElementNodes<ET, MAT, T> nodes;
      nodes.load(coords, u, nid);
      element_row_block<ET, MAT, T>(nodes, p0, p1, eparam, e, a, rb);
#pragma unroll
      for (int b = 0; b < NN; ++b)
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const int col = __ldg(dof_colors + (int64_t)nid[b] * V + k);
#pragma unroll
          for (int i = 0; i < V; ++i) acc_row[i * n_colors + col] += rb[i][b * V + k];
        }
    }
  }
  if (ACC_SMEM) {
    __syncthreads();
    // rows of nodes n0 .. n0 + blockDim.x - 1 are one contiguous block of Jc
    const int64_t rows_here = (n_nodes - n0) < (int64_t)blockDim.x ? (n_nodes - n0) : blockDim.x;
    const int64_t total = rows_here * row_words;
    T* out = Jc + n0 * row_words;
    for (int64_t k = threadIdx.x; k < total; k += blockDim.x) {
      const int t = (int)(k / row_words);
      out[k] = sm[(int64_t)t * stride + (k - (int64_t)t * row_words)];
    }
  }
}

template <class T>
__global__ void fill_kernel(T* __restrict__ x, int64_t n, T val) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] = val;
}

__global__ void rows_cols_kernel(const int32_t* __restrict__ indptr,
                                 const int32_t* __restrict__ indices,
                                 const int32_t* __restrict__ colors, int64_t n_rows,
                                 int32_t* __restrict__ rows, int32_t* __restrict__ col_colors) {
  // one warp per row
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (w >= n_rows) return;
  const int k0 = indptr[w], k1 = indptr[w + 1];
  for (int k = k0 + lane; k < k1; k += 32) {
    rows[k] = (int32_t)w;
    col_colors[k] = __ldg(colors + __ldg(indices + k));
  }
}

template <class T>
__global__ void decompress_kernel(const T* __restrict__ Jc, int n_colors,
                                  const int32_t* __restrict__ rows,
                                  const int32_t* __restrict__ col_colors, int64_t nnz,
                                  T* __restrict__ data) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nnz) return;
  data[k] = Jc[(int64_t)__ldg(rows + k) * n_colors + __ldg(col_colors + k)];
}

template <class T>
__global__ void seeds_kernel(const int32_t* __restrict__ colors, int64_t n, int c0, int nc,
                             T* __restrict__ seeds) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * nc) return;
  const int j = (int)(t / n);
  const int64_t i = t % n;
  seeds[t] = (__ldg(colors + i) == c0 + j) ? T(1) : T(0);
}

template <class T>
__global__ void set_column_kernel(const T* __restrict__ col, int64_t n, int n_colors, int c,
                                  T* __restrict__ Jc) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) Jc[i * n_colors + c] = col[i];
}

template <class F>
int dispatch_mat2(int kind, F&& f) {
  switch (kind) {
    case TG_POISSON: return f(IntC<TG_POISSON>{});
    case TG_LINEAR_ELASTIC: return f(IntC<TG_LINEAR_ELASTIC>{});
    case TG_NEO_HOOKEAN: return f(IntC<TG_NEO_HOOKEAN>{});
    default: return set_error(TG_ERR_VALUE, "unknown material kind %d", kind);
  }
}

}  // namespace tg

using namespace tg;

extern "C" int tg_compressed_hessian(int elem, int prec, const tg_material* mat,
                                     const void* coords, int64_t n_nodes, const int32_t* conn,
                                     int64_t n_elems, const void* u, const int32_t* inc_ptr,
                                     const int32_t* inc_idx, const int32_t* dof_colors,
                                     int n_colors, void* Jc, void* stream) {
  TG_TRY(check_ptr(mat, "mat"));
  TG_TRY(check_sizes(n_elems, n_nodes, 1));
  TG_TRY(check_ptr(Jc, "Jc"));
  if (n_colors <= 0) return set_error(TG_ERR_VALUE, "n_colors must be positive");
  if (n_nodes == 0) return TG_OK;
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  if (n_elems > 0) {
    TG_TRY(check_ptr(coords, "coords"));
    TG_TRY(check_ptr(conn, "conn"));
    TG_TRY(check_ptr(inc_idx, "inc_idx"));
    TG_TRY(check_ptr(dof_colors, "dof_colors"));
  }
  cudaStream_t st = as_stream(stream);
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_mat2(mat->kind, [&](auto mk) -> int {
      constexpr int MAT = decltype(mk)::value;
      if constexpr (MAT == TG_NEO_HOOKEAN && Elem<ET>::D != 3) {
        return set_error(TG_ERR_UNSUPPORTED, "Neo-Hookean needs a 3D element");
      } else {
        return dispatch_prec(prec, [&](auto t) -> int {
          using T = decltype(t);
          constexpr int V = LawDims<MAT, Elem<ET>::D>::V;
          if (!Law<MAT, Elem<ET>::D, T>::LINEAR && n_elems > 0) TG_TRY(check_ptr(u, "u"));
          // threads per CTA (a multiple of 32, <= 128): the most resident threads per
          // SM that shared memory allows (each thread holds one node's row block)
          const size_t row_bytes = ((size_t)V * n_colors + 1) * sizeof(T);
          int dev = 0, sm_bytes = 0, cta_bytes = 0;
          TG_TRY(cuda_check(cudaGetDevice(&dev), "tg_compressed_hessian: device"));
          TG_TRY(cuda_check(cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev),
                            "tg_compressed_hessian: shared memory per SM"));
          TG_TRY(cuda_check(cudaDeviceGetAttribute(&cta_bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev),
                            "tg_compressed_hessian: shared memory per CTA"));
          int nt = 0, best = 0;
          for (int cand = 128; cand >= 32; cand -= 32) {
            const size_t need = (size_t)cand * row_bytes;
            if (need > (size_t)cta_bytes) continue;
            const int resident = (int)((size_t)sm_bytes / (need + 1024)) * cand;
            if (resident > best) {
              best = resident;
              nt = cand;
            }
          }
          if (nt == 0) nt = 32;
          const unsigned grid = (unsigned)((n_nodes + nt - 1) / nt);
          if (best > 0) {
            const size_t smem = (size_t)nt * row_bytes;
            auto kern = compressed_hessian_kernel<ET, MAT, T, true>;
            TG_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem),
                              "tg_compressed_hessian: shared memory"));
            kern<<<grid, nt, smem, st>>>((const T*)coords, conn, (const T*)u, (T)mat->p0,
                                         (T)mat->p1, (const T*)mat->elem_param, n_nodes, inc_ptr,
                                         inc_idx, dof_colors, n_colors, (T*)Jc);
          } else {
            const int64_t total = n_nodes * V * (int64_t)n_colors;
            fill_kernel<T><<<grid_for(total, 256), 256, 0, st>>>((T*)Jc, total, T(0));
            compressed_hessian_kernel<ET, MAT, T, false><<<grid, 32, 0, st>>>(
                (const T*)coords, conn, (const T*)u, (T)mat->p0, (T)mat->p1,
                (const T*)mat->elem_param, n_nodes, inc_ptr, inc_idx, dof_colors, n_colors,
                (T*)Jc);
          }
          return launch_check("tg_compressed_hessian");
        });
      }
    });
  });
}

// dofs per node of a law on an element (0: not available)
static int law_values(int elem, int kind) {
  if (kind == TG_POISSON) return 1;
  if (kind == TG_LINEAR_ELASTIC) return elem == TG_TRI3 ? 2 : 3;
  return (kind == TG_NEO_HOOKEAN && elem != TG_TRI3) ? 3 : 0;
}

extern "C" int tg_csr_slots(int elem, int n_vals, int64_t n_nodes, const int32_t* conn,
                            int64_t n_elems, const int32_t* inc_ptr, const int32_t* inc_idx,
                            const int32_t* indptr, const int32_t* indices, int64_t nnz,
                            const int32_t* colors, int n_colors, uint16_t* slots, int32_t* info,
                            void* stream) {
  TG_TRY(check_sizes(n_elems, n_nodes, n_vals));
  if (nnz < 0) return set_error(TG_ERR_VALUE, "negative size");
  if (n_vals > 3 || n_colors < 1 || n_colors > SLOT_MAX_COLORS)
    return set_error(TG_ERR_UNSUPPORTED, "tg_csr_slots: at most 3 values per node and %d colours",
                     SLOT_MAX_COLORS);
  if (n_nodes == 0 || n_elems == 0)
    return set_error(TG_ERR_UNSUPPORTED, "tg_csr_slots: empty mesh");
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(inc_idx, "inc_idx"));
  TG_TRY(check_ptr(indptr, "indptr"));
  TG_TRY(check_ptr(indices, "indices"));
  TG_TRY(check_ptr(colors, "colors"));
  TG_TRY(check_ptr(slots, "slots"));
  TG_TRY(check_ptr(info, "info"));
  if (reinterpret_cast<uintptr_t>(slots) % 16 != 0)
    return set_error(TG_ERR_VALUE, "tg_csr_slots: slots must be 16-byte aligned");
  cudaStream_t st = as_stream(stream);
  TG_TRY(cuda_check(cudaMemsetAsync(info, 0, 2 * sizeof(int32_t), st), "tg_csr_slots: info"));
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    auto go = [&](auto vc) -> int {
      constexpr int V = decltype(vc)::value;
      csr_pattern_check_kernel<V><<<grid_for(n_nodes, CHECK_NODES), 128, 0, st>>>(
          n_nodes, nnz, indptr, indices, colors, n_colors, info);
      const int64_t entries = n_elems * Elem<ET>::NN;
      csr_slots_kernel<ET, V><<<grid_for(entries, 128), 128, 0, st>>>(
          n_nodes, entries, conn, inc_ptr, inc_idx, indptr, indices, slots, info);
      return launch_check("tg_csr_slots");
    };
    if (n_vals == 1) return go(IntC<1>{});
    if (n_vals == 2) return go(IntC<2>{});
    return go(IntC<3>{});
  });
}

// shared-memory words per lane of a row block of max_deg columns
static int csr_row_words(int V, int max_deg) {
  return (V * V * max_deg + CSR_SLAB - 1) / CSR_SLAB * CSR_SLAB;
}

// Warps of a CTA of hessian_csr_kernel with `warp_bytes` of row blocks a warp: the ones that
// leave more warps on an SM.  FP64 Hex8 (65 KB a warp for three values: three CTAs of one warp
// where one of two fits), Linear-Elastic 22^3 1,316 us with two and 877 with one, 30^3 2,625 and
// 1,757, 48^3 10,504 and 7,017.  Where the count is about the same, FP64 Hex8 takes one, for a
// last wave in finer grains (Poisson 24^3 395 and 374, 30^3 729 and 664, 48^3 2,326 and 2,320),
// and the others two: an SM holds 32 CTAs at most (Tet4 Poisson 56^3 FP32 52 us and 67 with
// one, Hex8 Linear-Elastic 36^3 FP32 112 and 120).
static int csr_warps(int elem, int prec, size_t warp_bytes, int sm_bytes) {
  auto resident = [&](int w) {
    const int64_t ctas = sm_bytes / (int64_t)(w * warp_bytes + 1024);
    return w * (ctas < 32 ? ctas : 32);
  };
  const int64_t one = resident(1), two = resident(CSR_WARPS);
  return one > two || (one * 10 >= two * 9 && elem == TG_HEX8 && prec == TG_F64) ? 1 : CSR_WARPS;
}

extern "C" int tg_hessian_csr(int elem, int prec, const tg_material* mat, const void* coords,
                              int64_t n_nodes, const int32_t* conn, int64_t n_elems,
                              const void* u, const int32_t* inc_ptr, const int32_t* inc_idx,
                              const uint16_t* slots, const int32_t* indptr, int max_deg,
                              void* data, void* stream) {
  TG_TRY(check_ptr(mat, "mat"));
  TG_TRY(check_sizes(n_elems, n_nodes, 1));
  if (n_nodes == 0) return TG_OK;
  const int values = law_values(elem, mat->kind);
  if (values == 0) return set_error(TG_ERR_UNSUPPORTED, "Neo-Hookean needs a 3D element");
  TG_TRY(check_ptr(coords, "coords"));
  TG_TRY(check_ptr(conn, "conn"));
  TG_TRY(check_ptr(inc_ptr, "inc_ptr"));
  TG_TRY(check_ptr(inc_idx, "inc_idx"));
  TG_TRY(check_ptr(slots, "slots"));
  TG_TRY(check_ptr(indptr, "indptr"));
  TG_TRY(check_ptr(data, "data"));
  if (reinterpret_cast<uintptr_t>(slots) % 16 != 0)
    return set_error(TG_ERR_VALUE, "tg_hessian_csr: slots must be 16-byte aligned");
  int dev = 0, cta_bytes = 0, sm_bytes = 0;
  TG_TRY(cuda_check(cudaGetDevice(&dev), "tg_hessian_csr: device"));
  TG_TRY(cuda_check(
      cudaDeviceGetAttribute(&sm_bytes, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev),
      "tg_hessian_csr: shared memory per SM"));
  TG_TRY(cuda_check(cudaDeviceGetAttribute(&cta_bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev),
                    "tg_hessian_csr: shared memory per CTA"));
  const size_t word = prec == TG_F32 ? 4 : 8;
  if (max_deg < 1 || max_deg > 65536 ||
      (size_t)csr_row_words(values, max_deg) * 32 * CSR_WARPS * word > (size_t)cta_bytes)
    return set_error(TG_ERR_UNSUPPORTED, "tg_hessian_csr: rows of %d columns do not fit", max_deg);
  cudaStream_t st = as_stream(stream);
  return dispatch_elem(elem, [&](auto et) -> int {
    constexpr int ET = decltype(et)::value;
    return dispatch_mat2(mat->kind, [&](auto mk) -> int {
      constexpr int MAT = decltype(mk)::value;
      if constexpr (MAT == TG_NEO_HOOKEAN && Elem<ET>::D != 3) {
        return set_error(TG_ERR_UNSUPPORTED, "Neo-Hookean needs a 3D element");
      } else {
        return dispatch_prec(prec, [&](auto t) -> int {
          using T = decltype(t);
          constexpr int V = LawDims<MAT, Elem<ET>::D>::V;
          if (!Law<MAT, Elem<ET>::D, T>::LINEAR) TG_TRY(check_ptr(u, "u"));
          const int words = csr_row_words(V, max_deg);
          const int warps =
              csr_warps(elem, prec, (size_t)words * 32 * sizeof(T), sm_bytes);
          const size_t smem = (size_t)words * 32 * warps * sizeof(T);
          auto kern = hessian_csr_kernel<ET, MAT, T>;
          TG_TRY(cuda_check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem),
                            "tg_hessian_csr: shared memory"));
          kern<<<grid_for(n_nodes, 32 * warps), 32 * warps, smem, st>>>(
              (const T*)coords, conn, reinterpret_cast<uintptr_t>(conn) % 16 == 0, (const T*)u,
              (T)mat->p0, (T)mat->p1, (const T*)mat->elem_param, n_nodes, inc_ptr, inc_idx, slots,
              indptr, words, (T*)data);
          return launch_check("tg_hessian_csr");
        });
      }
    });
  });
}

extern "C" int tg_rows_cols(const int32_t* indptr, const int32_t* indices, const int32_t* colors,
                            int64_t n_rows, int64_t nnz, int32_t* rows, int32_t* col_colors,
                            void* stream) {
  if (n_rows < 0 || nnz < 0) return set_error(TG_ERR_VALUE, "negative size");
  if (n_rows == 0 || nnz == 0) return TG_OK;
  TG_TRY(check_ptr(indptr, "indptr"));
  TG_TRY(check_ptr(indices, "indices"));
  TG_TRY(check_ptr(colors, "colors"));
  TG_TRY(check_ptr(rows, "rows"));
  TG_TRY(check_ptr(col_colors, "col_colors"));
  rows_cols_kernel<<<grid_for(n_rows * 32, 256), 256, 0, as_stream(stream)>>>(
      indptr, indices, colors, n_rows, rows, col_colors);
  return launch_check("tg_rows_cols");
}

extern "C" int tg_decompress(int prec, const void* Jc, int n_colors, const int32_t* rows,
                             const int32_t* col_colors, int64_t nnz, void* data, void* stream) {
  if (nnz < 0 || n_colors <= 0) return set_error(TG_ERR_VALUE, "bad sizes for tg_decompress");
  if (nnz == 0) return TG_OK;
  TG_TRY(check_ptr(Jc, "Jc"));
  TG_TRY(check_ptr(rows, "rows"));
  TG_TRY(check_ptr(col_colors, "col_colors"));
  TG_TRY(check_ptr(data, "data"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    decompress_kernel<T><<<grid_for(nnz, 256), 256, 0, as_stream(stream)>>>(
        (const T*)Jc, n_colors, rows, col_colors, nnz, (T*)data);
    return launch_check("tg_decompress");
  });
}

extern "C" int tg_color_seeds(int prec, const int32_t* colors, int64_t n, int c0, int nc,
                              void* seeds, void* stream) {
  if (n < 0 || nc < 0) return set_error(TG_ERR_VALUE, "negative size");
  if (n == 0 || nc == 0) return TG_OK;
  TG_TRY(check_ptr(colors, "colors"));
  TG_TRY(check_ptr(seeds, "seeds"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    seeds_kernel<T><<<grid_for(n * nc, 256), 256, 0, as_stream(stream)>>>(colors, n, c0, nc,
                                                                            (T*)seeds);
    return launch_check("tg_color_seeds");
  });
}

extern "C" int tg_set_column(int prec, const void* col, int64_t n, int n_colors, int c, void* Jc,
                             void* stream) {
  if (n < 0 || n_colors <= 0 || c < 0 || c >= n_colors)
    return set_error(TG_ERR_VALUE, "bad arguments for tg_set_column");
  if (n == 0) return TG_OK;
  TG_TRY(check_ptr(col, "col"));
  TG_TRY(check_ptr(Jc, "Jc"));
  return dispatch_prec(prec, [&](auto t) -> int {
    using T = decltype(t);
    set_column_kernel<T><<<grid_for(n, 256), 256, 0, as_stream(stream)>>>((const T*)col, n,
                                                                          n_colors, c, (T*)Jc);
    return launch_check("tg_set_column");
  });
}
