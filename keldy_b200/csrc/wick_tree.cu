// The tree kernel of the Wick-determinant integrand (sm_100a): one warp per group of points.
//
// keldy's integrand (impurity_oneband/wick_direct.cpp:43-158) sums, over the 2^n Keldysh
// configurations a, (-1)^|a| det(s1_a) det(s2_a): s2_a is the n x n matrix of g0 between the
// vertices' chosen copies, s1_a the same with the two external points as one more row and
// column (corner 0). Three facts about those matrices carry the kernel.
//
// * With the vertices sorted by time, an entry between two vertices depends only on the
//   Keldysh index of the EARLIER one (the later point's branch does not matter: its row of
//   g0 is the same on both branches), the diagonal entry on neither, an external entry only
//   on its vertex's index.
// * Gaussian elimination of the vertices, earliest first, keeps that form: the correction
//   c_i r_j / p holds the eliminated vertex's column and row, which depend on its index alone.
//   So a node of the elimination tree with m vertices left is ONE (m+1) x (m+1) matrix S (the
//   backward copies), both children of a node share its pivot p, and the difference of an
//   entry's two copies is the same number at every node: S^f_ij = S_ij + delta_ij with delta
//   fixed per point. (A node of both copies, as in an elimination in the given order, is
//   (2m+1)^2 entries and two pivots.)
// * The last two vertices need no division. With X, Y the external entries of the latest
//   vertex, its two configurations differ only in them, so the external corner and the
//   square of the leaf's own terms cancel before anything is rounded:
//     sum_{a1} = -D^2 p2 p1' (X_f Y_f - X_b Y_b)', and p2 times each factor is a polynomial
//   of the 3 x 3 matrix's entries (leaf2).
//
// Cost: sum_m 2^(n-m) (m+1)^2 complex multiply-adds, ~15 * 2^n (the elimination in the given
// order with both copies, which this kernel replaced, took ~40 * 2^n).
//
// Work split: a level of 256 >> m nodes with m vertices left fills a warp from m = 8 (one
// node, one point) down to m = 3 (32 nodes, one per lane), whatever the order: order n starts
// at level n with 2^(8-n) points per warp. Levels 8..5 go through shared memory with the lanes
// of a node splitting its children; the last three vertices run in registers. Orders above 8
// walk the first n - 8 levels depth first, one node per level kept. Warps never wait for each
// other: no CTA barrier in the kernel.
#include <cuda_runtime.h>

#include "kb_device.cuh"
#include "kb_launch.h"
#include "kb_spline.cuh"

namespace kb {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Row width and node size of a node with m vertices left (m+1 rows): the row widths and sizes
// are chosen so that the eight lanes of a 128-bit shared-memory phase hit different banks in
// the levels' reads and writes.
__host__ __device__ constexpr int node_w(int m) { return m == 7 ? 9 : m + 1; }
__host__ __device__ constexpr int node_sz(int m) {
  return m == 1 ? 5 : m == 2 ? 9 : m == 3 ? 17 : m == 4 ? 26 : m == 5 ? 36 : m == 6 ? 49 : m == 7 ? 72 : (m + 1) * (m + 1);
}
// Complex entries of a warp's node buffers: level m's nodes start at NODES_ODD for odd m >= 5,
// at 0 otherwise; the point differences delta start after the buffers the order uses.
constexpr int NODES_ODD = 16 * 26;                     // behind the 16 nodes of level 4
constexpr int NODES_END = NODES_ODD + 8 * 36;          // behind the 8 nodes of level 5
constexpr int WARP_BUF = NODES_END + 272;              // delta of order 16: 16 * 17
__host__ __device__ constexpr int node_base(int m) { return (m & 1) && m >= 5 ? NODES_ODD : 0; }
__host__ __device__ constexpr int delta_base(int n) { return n >= 5 ? NODES_END : n == 4 ? NODES_ODD : 32 * 17; }
// delta of a point, in shells: vertex k (1 = latest) holds its k column entries (i, k), i < k,
// at k(k-1), then its k row entries (k, j), j < k, at k*k.
__host__ __device__ constexpr int delta_sz(int n) { return n < 8 ? n * (n + 1) + 1 : n * (n + 1); }
static_assert(delta_base(3) + 32 * delta_sz(3) <= WARP_BUF && delta_base(5) + 8 * delta_sz(5) <= WARP_BUF &&
                  delta_base(4) + 16 * delta_sz(4) <= WARP_BUF && delta_base(8) + 16 * 17 <= WARP_BUF,
              "differences fit behind the nodes");

template <bool SCALE>
struct WarpShared {
  double2 buf[WARP_BUF];
  double u[256];      // the group's vertex times, u[j * gp + p] (sorted, latest first)
  double2 fval[32];   // the group's values
  double2 D2[2][16];  // squared prefix determinant of every node (by parity of its level)
  double2 Dst[8];     // the same of the depth-first levels above 8
  int fl[32];         // a guarded pivot in the point's tree
  double fscale[SCALE ? 32 : 2];
};

__device__ __forceinline__ double2 cfma(double2 c, double2 a, double2 b) {
  return c2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// s + f d, f = 1 (the forward copy) or 0
__device__ __forceinline__ double2 copyof(double2 s, double2 d, double f) { return c2(fma(d.x, f, s.x), fma(d.y, f, s.y)); }

__device__ __forceinline__ int find_chunk_item(const long long *off, int n_items, long long c) {
  int lo = 0, hi = n_items; // off[lo] <= c < off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= c)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// ------------------------------------------------------------------ a group's set-up

// Sobol coordinates of points k0 .. k0+31 (lane = point): the Gray code of a point splits into
// its aligned block of 32 and its five low bits, so each coordinate is one warp-wide xor over
// the block's columns (two blocks at most) and five columns by the lane's own bits. The same
// number as sobol_coord.
__device__ __forceinline__ void sobol_group(const SobolDev &s, uint32_t k0, int N, int lg, int lane, double *u) {
  const uint32_t k = k0 + lane, b0 = k0 >> 5, b1 = b0 + 1;
  const uint32_t g0 = (b0 << 5) ^ (b0 << 4), g1 = (b1 << 5) ^ (b1 << 4);
  const uint32_t r = k & 31u, gr = r ^ (r >> 1);
  for (int j = 0; j < N; ++j) {
    const uint32_t *C = s.Csr + j * s.m;
    // column b of the matrix; Gray bit m (point 2^m) folds into column 0
    const uint32_t col = lane < s.m ? __ldg(C + lane) : (lane == s.m ? __ldg(C) : 0u);
    const uint32_t x0 = __reduce_xor_sync(FULL, ((g0 >> lane) & 1u) ? col : 0u);
    const uint32_t x1 = __reduce_xor_sync(FULL, ((g1 >> lane) & 1u) ? col : 0u);
    uint32_t cur = (k >> 5) == b0 ? x0 : x1;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
      const uint32_t cb = __shfl_sync(FULL, col, b);
      if ((gr >> b) & 1u) cur ^= cb;
    }
    if (lane < (1 << lg)) u[(j << lg) + lane] = 2.3283064365386963e-10 * (double)(cur ^ __ldg(s.shfr + j));
  }
}

// Points gp0 .. gp0+cnt-1 of an item: vertex times into u (not yet sorted), each lane's own
// point's Jacobian and domain flag. The product warpers, whose logarithms and exponentials
// dominate, run over (coordinate, point) pairs so that small groups fill the warp; a point's
// Jacobian is the product of its factors in coordinate order.
__device__ void setup_group(const Launch &L, const ItemDev &it, int N, int lg, long long gp0, int cnt, bool keep,
                            double *u, double *fac, int lane, double &jac, bool &dom) {
  jac = 1.0;
  int top = 0;
  const bool mine = lane < cnt;
  if (L.mode == IN_SOBOL) {
    top = it.chain_len;
    if (it.flow_x) { // Sobol points already mapped by the learned flow
      for (int j = 0; j < N; ++j)
        if (mine) u[(j << lg) + lane] = it.flow_x[(gp0 + lane) * N + j];
      if (mine) jac = it.flow_jac[gp0 + lane];
    } else {
      sobol_group(it.rng, it.k_first + (uint32_t)gp0, N, lg, lane, u);
      if (it.spline_knots) { // the separable spline flow in line
        const SplineKnots *kn = reinterpret_cast<const SplineKnots *>(it.spline_knots);
        __syncwarp();
        int lc = 0;
        while ((1 << lc) < cnt) ++lc;
        for (int e = lane; e < (N << lc); e += 32) {
          const int p = e & ((1 << lc) - 1), j = e >> lc;
          if (p >= cnt) continue;
          double der;
          u[(j << lg) + p] = spline_inverse(kn[j], u[(j << lg) + p], der);
          fac[(j << lg) + p] = der;
        }
        __syncwarp();
        if (mine)
          for (int j = 0; j < N; ++j) jac /= fac[(j << lg) + lane];
      }
      if (it.ar_spline && mine) jac = ar_spline_point(it.ar_spline, N, u + lane, 1 << lg);
    }
  } else {
    for (int j = 0; j < N; ++j)
      if (mine) u[(j << lg) + lane] = L.in[(gp0 + lane) * N + j];
    if (L.mode == IN_LI) top = it.chain_start;
  }
  __syncwarp();
  int lc = 0;
  while ((1 << lc) < cnt) ++lc;
  double cj = 1.0; // the chain's Jacobian
  for (int w = top - 1; w >= 0; --w) {
    const WarperDev &wd = it.chain[w];
    if (wd.kind == KB_WARPER_IDENTITY) continue;
    if (wd.kind == KB_WARPER_PLASMA_UV) {
      if (mine) cj *= warp_reverse_one(wd, N, u + lane, 1 << lg);
      __syncwarp();
      continue;
    }
    for (int e = lane; e < (N << lc); e += 32) {
      const int p = e & ((1 << lc) - 1), j = e >> lc;
      if (p >= cnt) continue;
      double &x = u[(j << lg) + p];
      double f;
      if (wd.kind == KB_WARPER_TABLE) {
        double t;
        f = table_reverse(wd.tab[wd.ntab == 1 ? 0 : j], x, t);
        x = t;
      } else {
        const double t = warper_Finv(wd, x);
        x = t;
        f = 1.0 / warper_f1(wd, t);
      }
      fac[(j << lg) + p] = f;
    }
    __syncwarp();
    if (mine) {
      double jw = 1.0;
      for (int j = 0; j < N; ++j) jw *= fac[(j << lg) + lane];
      cj *= jw;
    }
    __syncwarp();
  }
  jac *= cj;
  dom = it.f.A.spin == it.f.B.spin;
  if (mine && keep)
    for (int j = 0; j < N; ++j)
      if (u[(j << lg) + lane] < 0.0) dom = false;
}

// Bin of the earliest vertex time (binner_t::in_bounds and coord2index, binner.hpp:163-176:
// in [xmin, xmax], xmax itself in the last bin); -1: dropped. An index that rounds up to
// nbins just below xmax goes to the last bin.
__device__ __forceinline__ int earliest_bin(const Launch &L, const double *u, int stride, int N) {
  double t = u[0];
  for (int j = 1; j < N; ++j) t = fmin(t, u[j * stride]);
  if (!(L.bin_xmin <= t && t <= L.bin_xmax)) return -1;
  if (t == L.bin_xmax) return L.nbins - 1;
  return min((int)((t - L.bin_xmin) / L.bin_size), L.nbins - 1);
}

// Sorts a point's times (stride st), latest first; of equal times the higher vertex index
// counts as the later one on the contour (compare_3way's timesplit).
__device__ __forceinline__ void sort_times(double *u, int st, int N) {
  for (int i = 1; i < N; ++i) {
    const double v = u[i * st];
    int j = i - 1;
    while (j >= 0 && u[j * st] <= v) {
      u[(j + 1) * st] = u[j * st];
      --j;
    }
    u[(j + 1) * st] = v;
  }
}

// Root matrices and differences of np points (columns p0.. of u): entry (i, j), i != j, of
// position i (0: the external row A or column B, 1..N: the vertices, latest first) is one table
// lookup of g^< and g^> at one time difference: S = the copy of Keldysh index 1 (backward) of
// the pair's earlier vertex, delta = forward copy - S. Each lane starts GK lookups before it
// uses the first, so that their L2 round trips overlap.
template <bool CUBIC, int GK>
__device__ void build_roots(const ItemDev &it, int N, int np, const double *u, int st, unsigned dommask, double2 eq,
                            double2 *S, int ssz, int sw, double2 *dl, int dsz, int lane, bool &bad) {
  const ModelDev &m = it.model;
  const kb_gf_index &A = it.f.A, &B = it.f.B;
  const int spin = A.spin;
  const double2 *t00 = m.tab[spin][0][0];
  const double2 *trow = m.tab[spin][A.orbital][0];
  const double2 *tcol = m.tab[spin][0][B.orbital];
  const int per = N * (N + 1), total = np * per;
  // quotients by multiply-high with 2^32 / d rounded up (exact: r < 2^16, d <= 272); 0 = d is 1
  const unsigned mper = 0xFFFFFFFFu / (unsigned)per + 1u;
  const unsigned mn = N > 1 ? 0xFFFFFFFFu / (unsigned)N + 1u : 0u;
  for (int base = 0; base < total; base += 32 * GK) {
    int so[GK], dof[GK], ix[GK], how[GK]; // how: bit 0 forward copy is g^>, bit 1 backward copy is g^>, 4 none, 8 zero
    double wt[GK];
    const double2 *tb[GK];
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      const int r = base + 32 * k + lane;
      how[k] = 4;
      tb[k] = nullptr;
      ix[k] = so[k] = dof[k] = 0;
      wt[k] = 0.0;
      if (r >= total) continue;
      const int p = (int)__umulhi((unsigned)r, mper), q = r - p * per;
      const int i = mn ? (int)__umulhi((unsigned)q, mn) : q;
      const int jj = q - i * N, j = jj + (jj >= i ? 1 : 0);
      so[k] = p * ssz + i * sw + j;
      dof[k] = p * dsz + (i < j ? j * (j - 1) + i : i * i + j);
      if (!((dommask >> p) & 1u)) { // out of domain: identity, its value is discarded
        how[k] = 8;
        continue;
      }
      double dt;
      if (i == 0) {
        const double uj = u[(j - 1) * st + p];
        dt = A.time - uj;
        tb[k] = trow;
        // A later than the vertex (or at its time): forward g^>, backward g^<; earlier: A's branch decides
        how[k] = A.time < uj ? (A.k_idx ? 3 : 0) : 1;
      } else if (j == 0) {
        const double ui = u[(i - 1) * st + p];
        dt = ui - B.time;
        tb[k] = tcol;
        how[k] = ui > B.time ? (B.k_idx ? 0 : 3) : 2;
      } else {
        dt = u[(i - 1) * st + p] - u[(j - 1) * st + p];
        tb[k] = t00;
        how[k] = i < j ? 1 : 2;
      }
      if (tb[k] && !interp_index(m, dt, ix[k], wt[k])) {
        bad = true;
        ix[k] = 0;
        wt[k] = 0.0;
      }
    }
    double2 gl[GK], gg[GK];
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      if (tb[k] && CUBIC)
        interp_pair_cubic(tb[k], m.npts, ix[k], wt[k], gl[k], gg[k]);
      else if (tb[k])
        interp_pair(tb[k], ix[k], wt[k], gl[k], gg[k]);
      else
        gl[k] = gg[k] = c2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      if (how[k] == 4) continue;
      const double2 f = (how[k] & 1) ? gg[k] : gl[k], b = (how[k] & 2) ? gg[k] : gl[k];
      S[so[k]] = b;
      dl[dof[k]] = c2(f.x - b.x, f.y - b.y);
    }
  }
  // diagonals (equal contour points) and the external corner
  for (int e = lane; e < np * (N + 1); e += 32) {
    const int p = e / (N + 1), i = e - p * (N + 1);
    const bool in = (dommask >> p) & 1u;
    S[p * ssz + i * sw + i] = i == 0 ? c2(0.0, 0.0) : (in ? eq : c2(1.0, 0.0));
  }
}

// ------------------------------------------------------------------ the tree

// Level m (4 < m <= 8): the children of this lane's node. Nodes of a level, and the lanes
// of a node, are numbered so that a point's nodes stay in its own lanes: node lane >> (m-3),
// child lane >> (m-4), whose low bit is the copy of vertex m it eliminates (1: backward).
template <int m>
__device__ __forceinline__ void level(double2 *buf, const double2 *dl, const double2 *D2p, double2 *D2c, int lane,
                                      double floor_, bool &guard) {
  constexpr int W = node_w(m), WC = node_w(m - 1), LC = m - 4; // 2^LC lanes per child
  const int child = lane >> LC, l = lane & ((1 << LC) - 1);
  const double2 *S = buf + node_base(m) + (child >> 1) * node_sz(m);
  double2 *o = buf + node_base(m - 1) + child * node_sz(m - 1);
  const double2 *dc = dl + m * (m - 1), *dr = dl + m * m;
  const double f = (child & 1) ? 0.0 : 1.0;
  const double2 p = S[m * W + m];
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = crcp(p);
  if (l == 0) D2c[child] = cmul(D2p[child >> 1], cmul(p, p));
  if constexpr (m == 8) { // 8 x 8: half a row per lane
    const int i = l >> 1, j0 = (l & 1) * 4;
    const double2 Lf = cmul(copyof(S[i * W + m], dc[i], f), ip);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = j0 + q;
      o[i * WC + j] = cfms(S[i * W + j], Lf, copyof(S[m * W + j], dr[j], f));
    }
  } else if constexpr (m == 7) { // 7 x 7: a row per lane
    if (l < 7) {
      const double2 Lf = cmul(copyof(S[l * W + m], dc[l], f), ip);
#pragma unroll
      for (int j = 0; j < 7; ++j) o[l * WC + j] = cfms(S[l * W + j], Lf, copyof(S[m * W + j], dr[j], f));
    }
  } else if constexpr (m == 6) { // 6 x 6: a 3 x 3 block per lane
    const int i0 = (l >> 1) * 3, j0 = (l & 1) * 3;
    double2 r[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) r[j] = copyof(S[m * W + j0 + j], dr[j0 + j], f);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 Lf = cmul(copyof(S[(i0 + i) * W + m], dc[i0 + i], f), ip);
#pragma unroll
      for (int j = 0; j < 3; ++j) o[(i0 + i) * WC + j0 + j] = cfms(S[(i0 + i) * W + j0 + j], Lf, r[j]);
    }
  } else { // 5 x 5: rows 0, 1 or 3, 4 per lane, and its side of row 2
    const int i0 = l * 3, j0 = l * 2;
    double2 r[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) r[j] = copyof(S[m * W + j], dr[j], f);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const double2 Lf = cmul(copyof(S[(i0 + i) * W + m], dc[i0 + i], f), ip);
#pragma unroll
      for (int j = 0; j < 5; ++j) o[(i0 + i) * WC + j] = cfms(S[(i0 + i) * W + j], Lf, r[j]);
    }
    const double2 Lf = cmul(copyof(S[2 * W + m], dc[2], f), ip);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double2 rj = l ? r[j + 2] : r[j];
      o[2 * WC + j0 + j] = cfms(S[2 * W + j0 + j], Lf, rj);
    }
  }
}

// The last two vertices of a node T (3 x 3: external, latest vertex 1, vertex 2), all four
// configurations. With c = (T02, T12), r = (T20, T21) of vertex 2's copy, after its elimination
//   p2 p1' = T11 p2 - c1 r1 = q,  p2 (X_f Y_f - X_b Y_b) = p2 K - c0 r1 dY - c1 r0 dX,
// (X, Y = T01, T10; dX, dY their differences; K = X dY + dX (Y + dY)), and the two leaves of
// vertex 1 sum to -D^2 q times that: no division, the external corner drops out. Returns
// q_b (...)_b - q_f (...)_f. d2: vertex 2's differences {c0, c1, r0, r1}; g2 = d2[0] dY,
// h2 = dX d2[2]. SCALE: also the sum of |term| of the four leaves, without the factor D^2.
template <bool SCALE>
__device__ __forceinline__ double2 leaf2(const double2 (&T)[9], double2 dX, double2 dY, const double2 (&d2)[4],
                                         double2 g2, double2 h2, double &scale, double floor_, bool &guard) {
  const double2 K = cfma(cmul(T[1], dY), dX, cadd(T[3], dY));
  const double2 P = cmul(T[4], T[8]), Q = cmul(T[8], K);
  const double2 g = cmul(T[2], dY), h = cmul(dX, T[6]);
  const double2 tb = cmul(cfms(P, T[5], T[7]), cfms(cfms(Q, g, T[7]), h, T[5]));
  const double2 c1 = cadd(T[5], d2[1]), r1 = cadd(T[7], d2[3]);
  const double2 tf = cmul(cfms(P, c1, r1), cfms(cfms(Q, cadd(g, g2), r1), cadd(h, h2), c1));
  if constexpr (SCALE) {
    if (!(cabs1(T[8]) >= floor_)) guard = true;
    const double2 ip = crcp(T[8]);
#pragma unroll
    for (int a2 = 0; a2 < 2; ++a2) {
      const double2 c0 = a2 ? T[2] : cadd(T[2], d2[0]), r0 = a2 ? T[6] : cadd(T[6], d2[2]);
      const double2 k1 = a2 ? T[5] : c1, s1 = a2 ? T[7] : r1;
      const double2 q = cfms(P, k1, s1), sg = cfms(cmul(T[8], T[0]), c0, r0);
#pragma unroll
      for (int a1 = 0; a1 < 2; ++a1) {
        const double2 X = a1 ? T[1] : cadd(T[1], dX), Y = a1 ? T[3] : cadd(T[3], dY);
        const double2 xi = cfms(cmul(T[8], X), c0, s1), et = cfms(cmul(T[8], Y), k1, r0);
        scale += cabs(cmul(cmul(q, ip), cfms(cmul(q, sg), xi, et)));
      }
    }
  }
  return c2(tb.x - tf.x, tb.y - tf.y);
}

// The last three vertices of a node s (4 x 4, in registers), all eight configurations, times
// the node's D^2: vertex 3's elimination for both copies, then leaf2.
template <bool SCALE>
__device__ __forceinline__ double2 leaf3(const double2 (&s)[16], const double2 *dl, double2 D2, double floor_,
                                         bool &guard, double &scale) {
  const double2 p = s[15];
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = crcp(p);
  const double2 dX = dl[0], dY = dl[1];
  const double2 d2[4] = {dl[2], dl[3], dl[4], dl[5]};
  const double2 g2 = cmul(d2[0], dY), h2 = cmul(dX, d2[2]);
  double2 acc = c2(0.0, 0.0);
  double sc = 0.0;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    double2 r[3], T[9];
#pragma unroll
    for (int j = 0; j < 3; ++j) r[j] = a ? s[12 + j] : cadd(s[12 + j], dl[9 + j]);
    T[0] = c2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double2 Lf = cmul(a ? s[4 * i + 3] : cadd(s[4 * i + 3], dl[6 + i]), ip);
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (SCALE || i + j > 0) T[3 * i + j] = cfms(s[4 * i + j], Lf, r[j]);
    }
    const double2 v = leaf2<SCALE>(T, dX, dY, d2, g2, h2, sc, floor_, guard);
    acc = a ? c2(acc.x - v.x, acc.y - v.y) : v;
  }
  const double2 Dn = cmul(D2, cmul(p, p));
  if (SCALE) scale += sc * cabs(Dn);
  return cmul(Dn, acc);
}

// Level 4's child of this lane (child index = lane) in registers, then leaf3.
template <bool SCALE>
__device__ __forceinline__ double2 level4_leaves(const double2 *buf, const double2 *dl, const double2 *D2p, int lane,
                                                 double floor_, bool &guard, double &scale) {
  const double2 *S = buf + (lane >> 1) * node_sz(4);
  const double f = (lane & 1) ? 0.0 : 1.0;
  const double2 p = S[24];
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = crcp(p);
  double2 r[4], s[16];
#pragma unroll
  for (int j = 0; j < 4; ++j) r[j] = copyof(S[20 + j], dl[16 + j], f);
  s[0] = c2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double2 Lf = cmul(copyof(S[5 * i + 4], dl[12 + i], f), ip);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (SCALE || i + j > 0) s[4 * i + j] = cfms(S[5 * i + j], Lf, r[j]);
  }
  return leaf3<SCALE>(s, dl, cmul(D2p[lane >> 1], cmul(p, p)), floor_, guard, scale);
}

// The tree below the nodes of level min(n, 8) in the buffers (their D^2 set): this lane's
// value, with the sign of its copies of the vertices down to 4.
template <bool SCALE>
__device__ __forceinline__ double2 subtree(WarpShared<SCALE> &T, const double2 *dl, int n, int lane, double floor_,
                                           bool &guard, double &scale) {
  if (n >= 8) {
    level<8>(T.buf, dl, T.D2[0], T.D2[1], lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 7) {
    level<7>(T.buf, dl, T.D2[1], T.D2[0], lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 6) {
    level<6>(T.buf, dl, T.D2[0], T.D2[1], lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 5) {
    level<5>(T.buf, dl, T.D2[1], T.D2[0], lane, floor_, guard);
    __syncwarp();
  }
  double2 v;
  if (n >= 4) {
    v = level4_leaves<SCALE>(T.buf, dl, T.D2[0], lane, floor_, guard, scale);
  } else {
    double2 s[16];
    const double2 *S = T.buf + lane * node_sz(3);
#pragma unroll
    for (int e = 0; e < 16; ++e) s[e] = S[e];
    v = leaf3<SCALE>(s, dl, c2(1.0, 0.0), floor_, guard, scale);
  }
  const int lg = min(n, 8) - 3;
  if (__popc(lane & ((1 << lg) - 1)) & 1) v = c2(-v.x, -v.y);
  return v;
}

// One depth-first step above level 8: node S (m vertices left, m+1 wide) to its child of copy
// a, written to o (m wide). All lanes; the caller's __syncwarp follows.
__device__ __forceinline__ void step_down(const double2 *S, double2 *o, const double2 *dl, int m, int a, int lane,
                                          double2 D2, double2 &D2n, double floor_, bool &guard) {
  const int W = m + 1;
  const double2 p = S[m * W + m];
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = crcp(p);
  D2n = cmul(D2, cmul(p, p));
  const double f = a ? 0.0 : 1.0;
  const double2 *dc = dl + m * (m - 1), *dr = dl + m * m;
  const unsigned magic = 0xFFFFFFFFu / (unsigned)m + 1u; // e / m == umulhi(e, magic) for e < 2^16
  for (int e = lane; e < m * m; e += 32) {
    const int i = (int)__umulhi((unsigned)e, magic), j = e - i * m;
    const double2 Lf = cmul(copyof(S[i * W + m], dc[i], f), ip);
    o[e] = cfms(S[i * W + j], Lf, copyof(S[m * W + j], dr[j], f));
  }
}

// A group's points in passes of P, each point's value into T.fval (guarded: T.fl).
template <bool SCALE, bool ANY_CUBIC>
__device__ void group_values(WarpShared<SCALE> &T, const ItemDev &it, int n, int lgp, int cnt, unsigned dommask,
                             double2 eq, double2 *stack, int lane, bool &bad) {
  const double floor_ = it.model.pivot_floor;
  const int P = n <= 3 ? 32 : (n >= 8 ? 1 : 256 >> n);
  const int lg = n < 3 ? 0 : min(n, 8) - 3; // lanes per point
  const int st = 1 << lgp;
  double2 *dl0 = T.buf + delta_base(n);
  const int dsz = delta_sz(n);
  // orders above 8: the nodes of the depth-first levels, the deepest behind the differences in
  // shared memory when it fits, the others in global scratch
  double2 *node9 = nullptr;
  int soff = 0;
  if (n > 8) {
    const bool fits = n * (n + 1) + 100 <= WARP_BUF - NODES_END;
    for (int m = n; m > 9; --m) soff += (m + 1) * (m + 1);
    node9 = fits ? dl0 + n * (n + 1) : stack + soff;
  }
  for (int s0 = 0; s0 < cnt; s0 += P) {
    const int np = min(P, cnt - s0);
    const unsigned dm = (dommask >> s0) & (np >= 32 ? FULL : (1u << np) - 1u);
    if (P == 1 && !dm) {
      if (lane == 0) {
        T.fval[s0] = c2(0.0, 0.0);
        T.fl[s0] = 0;
        if (SCALE) T.fscale[s0] = 0.0;
      }
      continue;
    }
    double2 *root = n > 9 ? stack : (n == 9 ? node9 : T.buf + node_base(n));
    const int rsz = n > 8 ? 0 : node_sz(n), rw = n > 8 ? n + 1 : node_w(n);
    if (ANY_CUBIC && it.model.interp == 3)
      build_roots<true, 2>(it, n, np, T.u + s0, st, dm, eq, root, rsz, rw, dl0, dsz, lane, bad);
    else
      build_roots<false, 4>(it, n, np, T.u + s0, st, dm, eq, root, rsz, rw, dl0, dsz, lane, bad);
    if (n >= 4 && lane < 16) T.D2[n > 8 ? 0 : n & 1][lane] = c2(1.0, 0.0);
    __syncwarp();
    bool guard = false;
    double scale = 0.0;
    double2 v = c2(0.0, 0.0);
    if (n > 8) {
      const int K0 = n - 8;
      for (int sub = 0; sub < (1 << K0); ++sub) {
        // the levels whose copy changed since the last subtree, down to level 8
        const int first = sub == 0 ? 0 : K0 - 1 - (__ffs(sub) - 1);
        const double2 *src = stack;
        int off = 0;
        for (int d = 0; d < K0; ++d) {
          const int m = n - d;
          const double2 *S = m == 9 ? node9 : stack + off;
          off += (m + 1) * (m + 1);
          if (d < first) continue;
          double2 *o = m - 1 == 8 ? T.buf : (m - 1 == 9 ? node9 : stack + off);
          double2 D2n;
          step_down(S, o, dl0, m, (sub >> (K0 - 1 - d)) & 1, lane, d == 0 ? c2(1.0, 0.0) : T.Dst[d - 1], D2n, floor_,
                    guard);
          __syncwarp();
          if (lane == 0) {
            if (m - 1 == 8)
              T.D2[0][0] = D2n;
            else
              T.Dst[d] = D2n;
          }
          __syncwarp();
        }
        (void)src;
        const double2 w = subtree<SCALE>(T, dl0, 8, lane, floor_, guard, scale);
        v = (__popc(sub) & 1) ? c2(v.x - w.x, v.y - w.y) : cadd(v, w);
        __syncwarp();
      }
    } else if (n >= 3) {
      const int p = min(lane >> lg, np - 1); // idle lanes of a short pass repeat its last point's differences
      v = subtree<SCALE>(T, dl0 + p * dsz, n, lane, floor_, guard, scale);
    } else if (n == 2) {
      if (lane < np) {
        double2 s[9], d2[4];
        const double2 *S = T.buf + lane * node_sz(2), *dl = dl0 + lane * dsz;
#pragma unroll
        for (int e = 0; e < 9; ++e) s[e] = S[e];
#pragma unroll
        for (int e = 0; e < 4; ++e) d2[e] = dl[2 + e];
        if (!(cabs1(s[8]) >= floor_)) guard = true;
        v = leaf2<SCALE>(s, dl[0], dl[1], d2, cmul(d2[0], dl[1]), cmul(dl[0], d2[2]), scale, floor_, guard);
      }
    } else if (lane < np) { // order 1: -p (X_f Y_f - X_b Y_b)
      const double2 *S = T.buf + lane * node_sz(1), *dl = dl0 + lane * dsz;
      const double2 dX = dl[0], dY = dl[1];
      v = cmul(S[3], cfma(cmul(S[1], dY), dX, cadd(S[2], dY)));
      v = c2(-v.x, -v.y);
      if (SCALE) {
        const double2 xb = S[1], yb = S[2], xf = cadd(xb, dX), yf = cadd(yb, dY);
        scale = cabs(cmul(S[3], cfms(cmul(S[3], S[0]), xf, yf))) + cabs(cmul(S[3], cfms(cmul(S[3], S[0]), xb, yb)));
      }
    }
    for (int off = 1; off < (1 << lg); off <<= 1) {
      v.x += __shfl_xor_sync(FULL, v.x, off);
      v.y += __shfl_xor_sync(FULL, v.y, off);
      if (SCALE) scale += __shfl_xor_sync(FULL, scale, off);
    }
    const unsigned gm = __ballot_sync(FULL, guard);
    const int p = lane >> lg;
    if ((lane & ((1 << lg) - 1)) == 0 && p < np) {
      T.fval[s0 + p] = v;
      T.fl[s0 + p] = ((gm >> lane) & (lg == 5 ? FULL : (1u << (1 << lg)) - 1u)) != 0u;
      if (SCALE) T.fscale[s0 + p] = scale;
    }
    __syncwarp();
  }
}

__device__ __forceinline__ double2 cut_off(double2 f, double cutoff) { return cabs(f) < cutoff ? c2(0.0, 0.0) : f; }

// Persistent warps pull scheduling chunks (it.chunk_points points of one item) and walk them
// in groups of up to 32 points (16 above order 8): set-up, values, then the group's sum in a
// fixed shuffle order, so that results do not depend on which warp ran what.
// Bound: FP64 issue and shared-memory reads of the levels; 12 warps per SM at 168 registers.
template <bool EVAL, bool ANY_CUBIC, bool SCALE>
__global__ void __launch_bounds__(TREE_WARPS * 32, TREE_CTAS_PER_SM) tree_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpShared<SCALE> &T = reinterpret_cast<WarpShared<SCALE> *>(smem_raw)[warp];
  double2 *stack = reinterpret_cast<double2 *>(L.pts) + (size_t)(blockIdx.x * TREE_WARPS + warp) * TREE_STACK;
  bool bad = false;
  for (;;) {
    int c = 0;
    if (lane == 0) c = atomicAdd(L.chunk_counter, 1);
    c = __shfl_sync(FULL, c, 0);
    if (c >= L.n_chunks) break;
    const int item = find_chunk_item(L.chunk_offsets, L.n_items, c);
    const ItemDev &it = L.items[item];
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    const int ccount = (int)min((long long)it.chunk_points, (long long)it.n_points - cfirst);
    const int N = it.order;
    const bool keep = EVAL ? (L.keep_u_hypercube != 0) : true;
    const int lgp = N <= 8 ? 5 : 4;
    double2 eq = c2(0.0, 0.0);
    if (N > 0) {
      double2 gl, gg;
      int b0 = 0;
      g0_pair(it.model, it.model.tab[it.f.A.spin][0][0], 0.0, gl, gg, &b0);
      eq = c2(gl.x, gl.y - it.model.alpha);
    }
    if (!EVAL && L.nbins) {
      for (int b = lane; b < L.nbins; b += 32) {
        L.bin_sums[(size_t)c * L.nbins + b] = c2(0.0, 0.0);
        L.bin_counts[(size_t)c * L.nbins + b] = 0u;
      }
      __syncwarp();
    }
    double2 csum = c2(0.0, 0.0);
    unsigned ndom = 0, nfb = 0, ndrop = 0;
    unsigned long long fbm0 = 0, fbm1 = 0;
    for (int g0 = 0; g0 < ccount; g0 += 1 << lgp) {
      const int cnt = min(1 << lgp, ccount - g0);
      const bool mine = lane < cnt;
      double jac;
      bool dom;
      setup_group(L, it, N, lgp, cfirst + g0, cnt, keep, T.u, reinterpret_cast<double *>(T.buf), lane, jac, dom);
      int bin = -1;
      if (!EVAL && L.nbins && mine) bin = earliest_bin(L, T.u + lane, 1 << lgp, N);
      if (mine) sort_times(T.u + lane, 1 << lgp, N);
      const unsigned dommask = __ballot_sync(FULL, mine && dom);
      if (N > 0) {
        __syncwarp();
        group_values<SCALE, ANY_CUBIC>(T, it, N, lgp, cnt, dommask, eq, stack, lane, bad);
      } else if (mine) { // order 0: g0(A, B)
        kb_gf_index a = it.f.A, b = it.f.B;
        a.timesplit = b.timesplit = 0;
        int b0 = 0;
        const double2 v = dom ? g0_contour(it.model, a, b, 0, &b0) : c2(0.0, 0.0);
        bad = bad || b0;
        T.fval[lane] = v;
        T.fl[lane] = 0;
        if (SCALE) T.fscale[lane] = cabs(v);
      }
      __syncwarp();
      const double2 fv = mine ? T.fval[lane] : c2(0.0, 0.0);
      const bool ok = mine && dom;
      const bool fb = ok && (T.fl[lane] || !isfinite(fv.x) || !isfinite(fv.y));
      if (EVAL) {
        if (mine) {
          const long long o = cfirst + g0 + lane;
          const double2 f = ok ? cut_off(fv, it.f.cutoff) : c2(0.0, 0.0);
          L.out_val[o] = c2(f.x * jac, f.y * jac);
          if (L.out_jac) L.out_jac[o] = jac;
          if (L.out_dom) L.out_dom[o] = dom ? 1 : 0;
          if (SCALE) L.out_scale[o] = dom ? T.fscale[lane] * fabs(jac) : 0.0;
          if (L.out_flag) L.out_flag[o] = fb ? 1 : 0;
        }
        __syncwarp();
        continue;
      }
      double2 fj = c2(0.0, 0.0);
      if (ok && !fb) {
        const double2 f = cut_off(fv, it.f.cutoff);
        fj = c2(f.x * jac, f.y * jac);
      }
      if (L.nbins) {
        // each bin of the group: its lowest lane adds the bin's points in point order (guarded
        // points are counted here and added by the pivoted-LU pass)
        __syncwarp();
        T.fval[lane] = fj;
        const unsigned same = __match_any_sync(FULL, mine ? bin : -2);
        __syncwarp();
        if (mine && bin >= 0 && (same & ((1u << lane) - 1u)) == 0u) {
          double2 s = L.bin_sums[(size_t)c * L.nbins + bin];
          for (unsigned r = same; r; r &= r - 1) s = cadd(s, T.fval[__ffs(r) - 1]);
          L.bin_sums[(size_t)c * L.nbins + bin] = s;
          L.bin_counts[(size_t)c * L.nbins + bin] += __popc(same);
        }
        ndrop += __popc(__ballot_sync(FULL, mine && bin < 0));
        __syncwarp();
      }
      const unsigned fbm = __ballot_sync(FULL, fb);
      for (int off = 16; off > 0; off >>= 1) {
        fj.x += __shfl_xor_sync(FULL, fj.x, off);
        fj.y += __shfl_xor_sync(FULL, fj.y, off);
      }
      csum = cadd(csum, fj);
      ndom += __popc(dommask);
      nfb += __popc(fbm);
      // the guarded points' bits of the chunk: g0 is a multiple of 16
      if (g0 < 64)
        fbm0 |= (unsigned long long)fbm << g0;
      if (g0 > 32 && g0 < 64)
        fbm1 |= (unsigned long long)fbm >> (64 - g0);
      if (g0 >= 64) fbm1 |= (unsigned long long)fbm << (g0 - 64);
      __syncwarp();
    }
    if (!EVAL && lane == 0) {
      ChunkPartial pr;
      pr.sum_re = csum.x;
      pr.sum_im = csum.y;
      pr.n_in_domain = ndom;
      pr.n_fallback = nfb;
      pr.fb_mask[0] = fbm0;
      pr.fb_mask[1] = fbm1;
      L.partials[c] = pr;
      if (L.nbins) L.bin_dropped[c] = ndrop;
    }
  }
  if (__any_sync(FULL, bad) && lane == 0) atomicOr(L.err, 1);
}

template <bool SCALE>
constexpr size_t tree_smem() {
  return TREE_WARPS * sizeof(WarpShared<SCALE>);
}
static_assert(tree_smem<false>() <= (233472 / TREE_CTAS_PER_SM) - 1024, "four CTAs share an SM's shared memory");

template <bool EVAL, bool CUBIC, bool SCALE>
cudaError_t configure_one() {
  return cudaFuncSetAttribute(tree_kernel<EVAL, CUBIC, SCALE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)tree_smem<SCALE>());
}

} // namespace

cudaError_t configure_tree_kernels() {
  cudaError_t e = configure_one<false, false, false>();
  if (e == cudaSuccess) e = configure_one<false, true, false>();
  if (e == cudaSuccess) e = configure_one<true, true, false>();
  if (e == cudaSuccess) e = configure_one<true, true, true>();
  return e;
}

cudaError_t launch_tree(const Launch &L, int grid, cudaStream_t st) {
  constexpr int T = TREE_WARPS * 32;
  if (L.mode == IN_SOBOL) {
    if (L.any_cubic)
      tree_kernel<false, true, false><<<grid, T, tree_smem<false>(), st>>>(L);
    else
      tree_kernel<false, false, false><<<grid, T, tree_smem<false>(), st>>>(L);
  } else if (L.out_scale) {
    tree_kernel<true, true, true><<<grid, T, tree_smem<true>(), st>>>(L);
  } else {
    tree_kernel<true, true, false><<<grid, T, tree_smem<false>(), st>>>(L);
  }
  return cudaGetLastError();
}

} // namespace kb
