// keldy's kernel method (integrand_g_kernel, impurity_oneband/wick_kernel.cpp:42-138) on the
// time-ordered elimination tree, one warp per group of points (sm_100a).
//
// With the fixed point X in the external slot, s1_a = [[g_XX, r], [c, W_a]], W_a = the vertex matrix
// V_a of configuration a with the diagonal entry of vertex n-1 (keldy's entry (n, n)) set to 0,
// and vertex i's term is x_{i+1} (-1)^|a| det(V_a), x the first-row cofactors of s1_a. The terms of
// a point are summed per (vertex i, Keldysh index k): 2n sums. Since det(s1_a) is linear in the
// first row r, they are the derivatives of
//   Phi(r) = sum_a (-1)^|a| det(V_a) det(s1_a)
// with respect to r's 2n entries (one per vertex and copy), so one reverse pass over the tree of the
// direct integrand (wick_tree.cu, whose facts about the vertex matrix hold here) gives them all:
//
// * Forward: a node with m vertices left is V's Schur complement S (m x m, one function of every
//   entry: EntryKind), the columns C (the entries to X, copies as S's rows) and E (the unit vector e_q of the
//   zeroed vertex q), and the row Q = d e_q^T (d = the zeroed diagonal entry) with its two
//   corners: by Sherman-Morrison det(W) W^-1 c = det(V) [(1 - d z_q) y + d y_q z], y = V^-1 c,
//   z = V^-1 e_q, and the corners hold -d y_q and -d z_q. The row r itself is never formed.
// * Backward: h_j = the derivative of a node's share of Phi with respect to r_j (both copies
//   together), g with respect to r's entry in column E (its entry in column C drops out: the two
//   copies of the latest vertex cancel in it). Eliminating vertex m with copy a adds
//     t = -(1/p) (sum_{j<m} h_j S_mj^a + g E_m)
//   to sum (m, a) and to h_m; a node's h_j and g are its two children's summed.
//
// Cost ~25 * 2^n complex multiply-adds per point (carrying the eliminated rows to the leaves, as
// the Gauss-Jordan tree that this kernel replaced did, ~60 * 2^n). The lanes and levels are those
// of wick_tree.cu: 256 >> m nodes of level m per warp, from m = 8 (or the order) to m = 3 (one per
// lane), the last three vertices forward and backward in registers. All levels' nodes stay in
// shared memory for the way back.
//
// Bound: latency, at 8 warps per SM (255 registers; the nodes kept for the way back fill the shared
// memory). 2^20 points of order 8 8.9 ms (69 for the tree that it replaced), of order 5 1.6 (9.8);
// of 65,536 points of order 8 (0.67 ms) ncu shows the FP64 pipe 27 % busy, shared memory 52 %.
#include "kb_wick.cuh"

namespace kb {

namespace {

// Row width and node size with m vertices left: rows 0 (Q and its corners) to m, columns the m
// vertices, C, E. Sizes keep the half-warps' reads on different banks.
__host__ __device__ constexpr int km_w(int m) { return m + 2; }
__host__ __device__ constexpr int km_sz(int m) {
  return m == 1 ? 7 : m == 2 ? 13 : m == 3 ? 21 : m == 4 ? 31 : m == 6 ? 57 : m == 7 ? 73 : (m + 1) * (m + 2);
}
// Nodes of level m in a warp's buffer (levels 4 to 8, or the roots of orders 1 to 3), then delta.
constexpr int KN5 = 16 * 31, KN6 = KN5 + 8 * 42, KN7 = KN6 + 4 * 57, KN8 = KN7 + 2 * 73, KN_END = KN8 + 90;
constexpr int KM_BUF = KN_END + 100;
__host__ __device__ constexpr int km_base(int m) { return m == 8 ? KN8 : m == 7 ? KN7 : m == 6 ? KN6 : m == 5 ? KN5 : 0; }
__host__ __device__ constexpr int km_delta(int n) {
  return n >= 8 ? KN_END : n == 7 ? KN8 : n == 6 ? KN7 : n == 5 ? KN6 : n == 4 ? KN5 : 32 * 21;
}
// delta of a point, in shells: vertex k >= 2 holds its entries (i, k), i < k, at (k-1)(k-2), then its
// entries (k, j); behind all shells the n entries of column C.
__host__ __device__ constexpr int km_delta_sz(int n) { return n * n + (n < 8 && n % 2 == 0 ? 1 : 0); }
__host__ __device__ constexpr int km_pass(int n) { return n <= 3 ? 32 : n >= 8 ? 1 : 256 >> n; }
// Lookups in flight per lane (whole rounds of lanes for a pass's n^2 entries per point; 0: the orders above 8).
__host__ __device__ constexpr int km_flight(int n) {
  constexpr int FLIGHT[] = {4, 1, 4, 5, 4, 4, 5, 4, 2};
  return FLIGHT[n];
}
__host__ __device__ constexpr int km_group_lg(int n) { return n <= 3 ? 5 : 4; }
static_assert(km_delta(3) + 32 * km_delta_sz(3) <= KM_BUF && km_delta(4) + 16 * km_delta_sz(4) <= KM_BUF &&
                  km_delta(5) + 8 * km_delta_sz(5) <= KM_BUF && km_delta(6) + 4 * km_delta_sz(6) <= KM_BUF &&
                  km_delta(7) + 2 * km_delta_sz(7) <= KM_BUF && km_delta(10) + km_delta_sz(10) <= KM_BUF,
              "differences fit behind the nodes");

// The lookups of a pass, as wick_tree.cu's: the vertex pairs and column C.
constexpr int km_lookup_first(int n) {
  int s = 0;
  for (int k = 1; k < n; ++k) s += km_pass(k) * k * k;
  return s;
}
struct KmLookups {
  unsigned long long e[km_lookup_first(KM_MAX_ORDER + 1)];
  int first[KM_MAX_ORDER + 1];
  constexpr KmLookups() : e(), first() {
    int r = 0;
    for (int n = 1; n <= KM_MAX_ORDER; ++n) {
      first[n] = r;
      const int ssz = n > 8 ? 0 : km_sz(n), w = km_w(n), st = 1 << km_group_lg(n);
      for (int p = 0; p < km_pass(n); ++p)
        for (int i = 1; i <= n; ++i)
          for (int j = 0; j <= n; ++j) {
            if (i == j) continue;
            const unsigned long long ui = i * st + p, uj = (j ? j : n + 1) * st + p;
            const unsigned long long so = p * ssz + i * w + (j ? j - 1 : n);
            const int d = j == 0 ? n * (n - 1) + i - 1 : i < j ? (j - 1) * (j - 2) + i - 1 : (i - 1) * (i - 2) + i + j - 2;
            const unsigned long long dof = p * km_delta_sz(n) + d, kind = j == 0 ? 3 : i < j ? 0 : 1;
            e[r++] = ui | uj << 10 | so << 20 | dof << 32 | kind << 42;
          }
    }
  }
};
__device__ const KmLookups km_lookups = KmLookups();

struct KmShared {
  double2 buf[KM_BUF];
  double2 D2[32];    // signed squared prefix determinants: level 4's nodes at 0, 5's at 16, 6's at 24, 7's at 28, 8's at 30
  double2 out[2 * KM_MAX_ORDER]; // orders above 8: the point's sums over its subtrees
  ItemConst k;
  double u[192];     // the group's times, u[i * gp + p]: X, the vertices latest first, X
  double jac[32];
  unsigned char place[KM_MAX_ORDER * 16 + 32]; // vertex index of position i + 1: place[i * gp + p]
};

// Sorts a point's times (stride st), latest first, of equal times the higher vertex index, and notes
// which vertex each position holds.
__device__ __forceinline__ void sort_places(double *u, unsigned char *pl, int st, int N) {
  for (int i = 0; i < N; ++i) pl[i * st] = (unsigned char)i;
  for (int i = 1; i < N; ++i) {
    const double v = u[i * st];
    int j = i - 1;
    while (j >= 0 && u[j * st] <= v) {
      u[(j + 1) * st] = u[j * st];
      pl[(j + 1) * st] = pl[j * st];
      --j;
    }
    u[(j + 1) * st] = v;
    pl[(j + 1) * st] = (unsigned char)i;
  }
}

// The entries of a root that are no lookups: diagonals, column E, row Q, corners.
__device__ __forceinline__ void km_fixed_entries(const KmShared &T, int n, int np, int s0, int lgp, double2 *S, int ssz,
                                                 int lane) {
  const int w = km_w(n), per = 3 * n + 2;
  const unsigned mper = 0xFFFFFFFFu / (unsigned)per + 1u;
  const double2 eq = T.k.eq, z = c2(0.0, 0.0);
  for (int e = lane; e < np * per; e += 32) {
    const int p = (int)__umulhi((unsigned)e, mper), q = e - p * per;
    double2 *N = S + p * ssz;
    if (q >= 3 * n) { // corners
      N[q - 2 * n] = z;
      continue;
    }
    const int what = q >= 2 * n ? 2 : q >= n ? 1 : 0, i = q - what * n;
    const bool zeroed = T.place[(i << lgp) + s0 + p] == n - 1;
    if (what == 0)
      N[(i + 1) * w + i] = eq;
    else if (what == 1)
      N[(i + 1) * w + n + 1] = zeroed ? c2(1.0, 0.0) : z;
    else
      N[i] = zeroed ? eq : z;
  }
}

// Level m (5..8): the children of this lane's node (child lane >> (m-4), whose low bit is the copy of
// vertex m), 2^(m-4) lanes each: half a row, a row, a 3 x 4 block or three columns per lane.
template <int m>
__device__ __forceinline__ void km_level(double2 *buf, const double2 *dl, const double2 *dlC, const double2 *D2p,
                                         double2 *D2c, int lane, double floor_, bool &guard) {
  constexpr int W = km_w(m), WC = km_w(m - 1), LC = m - 4;
  const int child = lane >> LC, l = lane & ((1 << LC) - 1);
  const double2 *S = buf + km_base(m) + (child >> 1) * km_sz(m);
  double2 *o = buf + km_base(m - 1) + child * km_sz(m - 1);
  const double2 *dc = dl + (m - 1) * (m - 2), *dr = dc + m - 1; // entries (i, m) and (m, j)
  const double f = (child & 1) ? 0.0 : 1.0, fr = (child & 1) ? 1.0 : 0.0;
  const double2 p = S[m * W + m - 1], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  if (l == (1 << LC) - 1) {
    const double2 D = cmul(D2p[child >> 1], cmul(p, p));
    D2c[child] = (child & 1) ? c2(-D.x, -D.y) : D;
  }
  constexpr int ROWS = m == 8 || m == 7 ? 1 : m == 6 ? 3 : 5, COLS = m == 8 ? 5 : m == 7 ? 8 : m == 6 ? 4 : 3;
  const int i0 = m == 8 ? l >> 1 : m == 7 ? l : m == 6 ? 3 * (l >> 1) : 0;
  const int c0 = m == 8 ? 5 * (l & 1) : m == 7 ? 0 : m == 6 ? 4 * (l & 1) : 3 * l;
  if (m == 7 && l == 7) return;
  // child column c is column c of the node up to vertex m-1, then C and E
  double2 r[COLS];
#pragma unroll
  for (int q = 0; q < COLS; ++q) {
    const int c = min(c0 + q, m), src = c < m - 1 ? c : c + 1;
    const double2 d = c < m - 1 ? dr[c] : dlC[m - 1];
    r[q] = copyof(S[m * W + src], d, c == m ? 0.0 : fr);
  }
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    const int i = i0 + k; // row 0 is Q: no copies
    const double2 Lf = cmul(copyof(S[i * W + m - 1], dc[max(i, 1) - 1], i ? f : 0.0), ip);
#pragma unroll
    for (int q = 0; q < COLS; ++q) {
      const int c = c0 + q, src = c < m - 1 ? c : c + 1;
      if (c <= m) o[i * WC + c] = cfms(S[i * W + src], Lf, r[q]);
    }
  }
}

// The last two vertices of a node T (rows Q, 1, 2; columns 1, 2, C, E), signed D^2 = D2: adds its
// terms to o (sums (1, 0), (1, 1), (2, 0), (2, 1)) and its h_1, h_2, g to h. With vertex 1 left
// alone, p, C, E, Q, corners kc, ke: t_1^a = -+D^2 p ((1 + ke) C^a - kc E) without a division
// (C^1 = C^0 + dC_1), and h_1 = D^2 p (1 + ke) dC_1, g = -D^2 Q dC_1 (times the squared pivot p2's
// share of D^2).
__device__ __forceinline__ void km_leaf2(const double2 (&T)[12], double2 D2, double2 d12, double2 d21, double2 dC1,
                                         double2 dC2, double2 *o, double2 *h, double floor_, bool &guard) {
  const double2 p2 = T[9], ip = pivot_rcp(p2);
  if (!(cabs1(p2) >= floor_)) guard = true;
  const double2 Dn = cmul(D2, cmul(p2, p2));
  const double2 q = cmul(T[1], ip), E2 = T[11];
  const double2 ke = cfms(T[3], q, E2), one = c2(1.0 + ke.x, ke.y), nC1 = c2(-dC1.x, -dC1.y);
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const double sg = a ? -1.0 : 1.0;
    const double2 r1 = a ? cadd(T[8], d21) : T[8], c = a ? T[5] : cadd(T[5], d12), Cc = a ? cadd(T[10], dC2) : T[10];
    const double2 L = cmul(c, ip);
    const double2 p1 = cfms(T[4], L, r1), C1 = cfms(T[6], L, Cc), E1 = cfms(T[7], L, E2), Q1 = cfms(T[0], q, r1);
    const double2 kc = cfms(T[2], q, Cc);
    double2 w = cmul(Dn, p1);
    w = c2(sg * w.x, sg * w.y);
    const double2 u = cmul(w, cfms(cmul(one, C1), kc, E1)), v = cmul(w, cmul(one, nC1)); // -t_1^0, -h_1
    const double2 ge = cmul(cmul(c2(sg * Dn.x, sg * Dn.y), Q1), cmul(p1, nC1));
    const double2 t2 = cmul(ip, cfms(cmul(v, r1), ge, E2));
    o[0] = c2(o[0].x - u.x, o[0].y - u.y);
    o[1] = c2(o[1].x + (u.x - v.x), o[1].y + (u.y - v.y));
    o[2 + a] = cadd(o[2 + a], t2);
    h[0] = c2(h[0].x - v.x, h[0].y - v.y);
    h[1] = cadd(h[1], t2);
    h[2] = cadd(h[2], ge);
  }
}

// Level m on the way back: this lane's child's h (h_1 .. h_{m-1}) and g to its node's, and t, the
// term of its copy of vertex m.
template <int m>
__device__ __forceinline__ void km_back(const double2 *buf, const double2 *dl, int lane, double2 (&h)[8], double2 &g,
                                        double2 &t) {
  constexpr int W = km_w(m), LC = m - 4, bit = 1 << LC;
  const int child = lane >> LC;
  const double2 *S = buf + km_base(m) + (child >> 1) * km_sz(m) + m * W;
  const double2 *dr = dl + (m - 1) * (m - 2) + m - 1;
  const double f = (child & 1) ? 1.0 : 0.0; // (its row)
  const double2 ip = pivot_rcp(S[m - 1]);
  double2 s = cmul(g, S[m + 1]);
#pragma unroll
  for (int j = 0; j < m - 1; ++j) s = cfma(s, h[j], copyof(S[j], dr[j], f));
  t = cmul(c2(-s.x, -s.y), ip);
  h[m - 1] = t;
#pragma unroll
  for (int j = 0; j < m; ++j) {
    h[j].x += __shfl_xor_sync(FULL, h[j].x, bit);
    h[j].y += __shfl_xor_sync(FULL, h[j].y, bit);
  }
  g.x += __shfl_xor_sync(FULL, g.x, bit);
  g.y += __shfl_xor_sync(FULL, g.y, bit);
}

__device__ __forceinline__ double2 lane_sum(double2 v, int from, int to) { // over lane bits from .. to - 1
  for (int off = 1 << from; off < (1 << to); off <<= 1) {
    v.x += __shfl_xor_sync(FULL, v.x, off);
    v.y += __shfl_xor_sync(FULL, v.y, off);
  }
  return v;
}

// The tree below the roots of order n <= 8 in the buffer, or of level 8's node (n >= 8): every lane
// gets h_1 .. h_min(n,8) and g of its point's root; the point's sums of positions 1 .. min(n, 8) go
// to out[p * 2n + 2 (i-1) + k] (added there when `add`), for the np points of the pass.
__device__ __forceinline__ void km_subtree(KmShared &T, double2 *out, const double2 *dl, int n, int np, bool add, int lane,
                                           double floor_, bool &guard, double2 (&h)[8], double2 &g) {
  const int m0 = min(n, 8), lg = max(m0 - 3, 0);
  const double2 *dlC = dl + n * (n - 1);
  if (n >= 8) {
    km_level<8>(T.buf, dl, dlC, T.D2 + 30, T.D2 + 28, lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 7) {
    km_level<7>(T.buf, dl, dlC, T.D2 + 28, T.D2 + 24, lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 6) {
    km_level<6>(T.buf, dl, dlC, T.D2 + 24, T.D2 + 16, lane, floor_, guard);
    __syncwarp();
  }
  if (n >= 5) {
    km_level<5>(T.buf, dl, dlC, T.D2 + 16, T.D2, lane, floor_, guard);
    __syncwarp();
  }
  double2 o[6], hh[3], D2 = c2(1.0, 0.0);
#pragma unroll
  for (int q = 0; q < 6; ++q) o[q] = c2(0.0, 0.0);
  hh[0] = hh[1] = hh[2] = c2(0.0, 0.0);
  if (n >= 3) {
    double2 s[20];
    if (n == 3) {
#pragma unroll
      for (int e = 0; e < 20; ++e) s[e] = T.buf[lane * km_sz(3) + e];
    } else { // level 4's child of this lane
      constexpr int W = km_w(4);
      const double2 *S = T.buf + (lane >> 1) * km_sz(4);
      const double2 *dc = dl + 6, *dr = dl + 9;
      const double f = (lane & 1) ? 0.0 : 1.0, fr = (lane & 1) ? 1.0 : 0.0;
      const double2 p = S[4 * W + 3], ip = pivot_rcp(p);
      if (!(cabs1(p) >= floor_)) guard = true;
      D2 = cmul(T.D2[lane >> 1], cmul(p, p));
      if (lane & 1) D2 = c2(-D2.x, -D2.y);
      double2 r[5];
#pragma unroll
      for (int q = 0; q < 5; ++q)
        r[q] = q == 4 ? S[4 * W + 5] : copyof(S[4 * W + (q < 3 ? q : 4)], q < 3 ? dr[q] : dlC[3], fr);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 Lf = cmul(i ? copyof(S[i * W + 3], dc[i - 1], f) : S[3], ip);
#pragma unroll
        for (int q = 0; q < 5; ++q) s[i * 5 + q] = cfms(S[i * W + (q < 3 ? q : q + 1)], Lf, r[q]);
      }
    }
    // vertex 3
    const double2 p = s[17], ip = pivot_rcp(p);
    if (!(cabs1(p) >= floor_)) guard = true;
    const double2 Dn = cmul(D2, cmul(p, p)), q = cmul(s[2], ip), E3 = s[19];
    double2 h3 = c2(0.0, 0.0), t3f = c2(0.0, 0.0);
#pragma unroll 1
    for (int a = 0; a < 2; ++a) {
      const double f = a ? 0.0 : 1.0, fr = a ? 1.0 : 0.0, sg = a ? -1.0 : 1.0;
      double2 r[4], U[12];
      r[0] = copyof(s[15], dl[4], fr);
      r[1] = copyof(s[16], dl[5], fr);
      r[2] = copyof(s[18], dlC[2], fr);
      r[3] = E3;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double2 Lf = i ? cmul(copyof(s[i * 5 + 2], dl[2 + i - 1], f), ip) : q;
#pragma unroll
        for (int c = 0; c < 4; ++c) U[i * 4 + c] = cfms(s[i * 5 + (c < 2 ? c : c + 1)], Lf, r[c]);
      }
      double2 hc[3];
      hc[0] = hc[1] = hc[2] = c2(0.0, 0.0);
      km_leaf2(U, c2(sg * Dn.x, sg * Dn.y), dl[0], dl[1], dlC[0], dlC[1], o, hc, floor_, guard);
      const double2 t = cfma(cfma(cmul(hc[0], r[0]), hc[1], r[1]), hc[2], E3);
      const double2 t3 = cmul(c2(-t.x, -t.y), ip);
      if (a)
        o[5] = t3;
      else
        t3f = t3;
      h3 = cadd(h3, t3);
      hh[0] = cadd(hh[0], hc[0]);
      hh[1] = cadd(hh[1], hc[1]);
      hh[2] = cadd(hh[2], hc[2]);
    }
    o[4] = t3f;
    h[2] = h3;
  } else if (n == 2) {
    double2 U[12];
#pragma unroll
    for (int e = 0; e < 12; ++e) U[e] = T.buf[lane * km_sz(2) + e];
    km_leaf2(U, D2, dl[0], dl[1], dlC[0], dlC[1], o, hh, floor_, guard);
  } else { // order 1: t^a = -+p C^a (its corners are 0)
    const double2 *S = T.buf + lane * km_sz(1) + km_w(1);
    const double2 t0 = cmul(S[0], S[1]);
    o[0] = c2(-t0.x, -t0.y);
    o[1] = cmul(S[0], cadd(S[1], dlC[0]));
  }
  h[0] = hh[0];
  h[1] = hh[1];
  g = hh[2];
  double2 t4, t5, t6, t7, t8;
  t4 = t5 = t6 = t7 = t8 = c2(0.0, 0.0);
  if (n >= 4) km_back<4>(T.buf, dl, lane, h, g, t4);
  if (n >= 5) km_back<5>(T.buf, dl, lane, h, g, t5);
  if (n >= 6) km_back<6>(T.buf, dl, lane, h, g, t6);
  if (n >= 7) km_back<7>(T.buf, dl, lane, h, g, t7);
  if (n >= 8) km_back<8>(T.buf, dl, lane, h, g, t8);
  __syncwarp(); // the nodes are read: the sums may take their place
  const int l = lane & ((1 << lg) - 1), p = lane >> lg;
  double2 *po = out + p * 2 * n;
  const bool mine = p < np;
  auto put = [&](int e, double2 v, bool here) {
    if (mine && here) po[e] = add ? cadd(po[e], v) : v;
  };
  if (lg >= 3) {
    // the six sums of vertices 1 to 3: after three merging rounds lane l & 7 holds sum l & 7's part
    const double2 z = c2(0.0, 0.0);
    auto merge = [&](double2 a, double2 b, int bit) {
      const bool up = lane & bit;
      const double2 keep = up ? b : a, send = up ? a : b;
      return c2(keep.x + __shfl_xor_sync(FULL, send.x, bit), keep.y + __shfl_xor_sync(FULL, send.y, bit));
    };
    const double2 a = merge(o[0], o[1], 1), b = merge(o[2], o[3], 1), c = merge(o[4], o[5], 1);
    const double2 v = lane_sum(merge(merge(a, b, 2), merge(c, z, 2), 4), 3, lg);
    put(l, v, l < 6);
  } else {
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      const double2 v = lane_sum(o[q], 0, lg);
      put(q, v, l == 0 && q < 2 * n);
    }
  }
  // vertices 4 to 8: bit m-4 of the lane is the copy, the bits above are nodes
  if (n >= 4) put(6 + (l & 1), lane_sum(t4, 1, lg), l < 2);
  if (n >= 5) put(8 + ((l >> 1) & 1), lane_sum(t5, 2, lg), (l & ~2) == 0);
  if (n >= 6) put(10 + ((l >> 2) & 1), lane_sum(t6, 3, lg), (l & ~4) == 0);
  if (n >= 7) put(12 + ((l >> 3) & 1), lane_sum(t7, 4, lg), (l & ~8) == 0);
  if (n >= 8) put(14 + (l >> 4), t8, (l & ~16) == 0);
  __syncwarp();
}

// One step above level 8: node S (m vertices left) to its child of copy a at o, both (rows x (m+2)).
__device__ __forceinline__ void km_step_down(const double2 *S, double2 *o, const double2 *dl, const double2 *dlC, int m, int a,
                                             int lane, double2 D2, double2 &D2n, double floor_, bool &guard) {
  const int W = km_w(m), WC = km_w(m - 1);
  const double2 *dc = dl + (m - 1) * (m - 2), *dr = dc + m - 1;
  const double f = a ? 0.0 : 1.0, fr = a ? 1.0 : 0.0;
  const double2 p = S[m * W + m - 1], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  D2n = cmul(D2, cmul(p, p));
  if (a) D2n = c2(-D2n.x, -D2n.y);
  const int c = min(lane & 15, m), src = c < m - 1 ? c : c + 1; // a column per lane, every other row
  const double2 r = copyof(S[m * W + src], c < m - 1 ? dr[c] : dlC[m - 1], c == m ? 0.0 : fr);
#pragma unroll 5
  for (int i = lane >> 4; i < m; i += 2) {
    const double2 Lf = cmul(copyof(S[i * W + m - 1], dc[max(i, 1) - 1], i ? f : 0.0), ip);
    const double2 v = cfms(S[i * W + src], Lf, r);
    if ((lane & 15) <= m) o[i * WC + c] = v;
  }
}

// Orders 9 and 10: level 8's subtrees depth first, their h and g carried up through levels 9 and 10.
__device__ __noinline__ void km_deep(KmShared &T, double2 *stack, const double2 *dl, int n, int lane, double floor_, bool &guard) {
  const double2 *dlC = dl + n * (n - 1);
  const double2 *N10 = stack, *N9 = n == 9 ? stack : stack + km_sz(10);
  double2 h[8], g, H[9], G;
  for (int a10 = 0; a10 < (n == 10 ? 2 : 1); ++a10) {
    double2 D9 = c2(1.0, 0.0);
    if (n == 10) {
      km_step_down(N10, stack + km_sz(10), dl, dlC, 10, a10, lane, c2(1.0, 0.0), D9, floor_, guard);
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) H[j] = c2(0.0, 0.0);
    G = c2(0.0, 0.0);
    for (int a9 = 0; a9 < 2; ++a9) {
      double2 D8;
      km_step_down(N9, T.buf + km_base(8), dl, dlC, 9, a9, lane, D9, D8, floor_, guard);
      if (lane == 0) T.D2[30] = D8;
      __syncwarp();
      km_subtree(T, T.out, dl, n, 1, a10 + a9 > 0, lane, floor_, guard, h, g);
      const double2 *R = N9 + 9 * km_w(9), *dr = dl + 8 * 7 + 8;
      const double2 ip = pivot_rcp(R[8]);
      double2 s = cmul(g, R[10]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        s = cfma(s, h[j], copyof(R[j], dr[j], a9 ? 1.0 : 0.0));
        H[j] = cadd(H[j], h[j]);
      }
      const double2 t = cmul(c2(-s.x, -s.y), ip);
      H[8] = cadd(H[8], t);
      G = cadd(G, g);
      if (lane == 0) T.out[16 + a9] = a10 ? cadd(T.out[16 + a9], t) : t;
      __syncwarp();
    }
    if (n == 10) {
      const double2 *R = N10 + 10 * km_w(10), *dr = dl + 9 * 8 + 9;
      double2 s = cmul(G, R[11]);
#pragma unroll
      for (int j = 0; j < 9; ++j) s = cfma(s, H[j], copyof(R[j], dr[j], a10 ? 1.0 : 0.0));
      if (lane == 0) T.out[18 + a10] = cmul(c2(-s.x, -s.y), pivot_rcp(R[9]));
      __syncwarp();
    }
  }
}

// A group's passes: the points' sums, scaled by their Jacobians, to the bins, the sum or the output;
// returns the points for the pivoted-LU pass. ORDER: 1..8, 0 for the orders above: compiled per
// order, as the integrand's passes are.
template <int ORDER>
__device__ __forceinline__ unsigned km_passes(const Launch &L, KmShared &T, int order, bool symmetric, int cnt, unsigned inmask,
                                              unsigned dommask, long long first, int c, double2 *stack, int lane,
                                              double2 &csum, unsigned &ndrop) {
  const int N = ORDER ? ORDER : order, n2 = 2 * N, P = km_pass(N), lgp = km_group_lg(N), lg = max(min(N, 8) - 3, 0);
  const bool eval = L.mode != IN_SOBOL;
  const int nb = L.nbins * 2;
  const double floor_ = T.k.floor_;
  const int flip = T.k.greater; // the trees' copy 0 is Keldysh index 1
  double2 *dl0 = T.buf + km_delta(N);
  const int dsz = km_delta_sz(N);
  double2 *root = N > 8 ? stack : T.buf + km_base(N);
  const int rsz = N > 8 ? 0 : km_sz(N);
  double2 *out = N > 8 ? T.out : T.buf;
  unsigned guarded = symmetric ? 0u : dommask;
  for (int s0 = 0; s0 < cnt; s0 += P) {
    const int np = min(P, cnt - s0);
    const unsigned some = (inmask >> s0) & (np >= 32 ? FULL : (1u << np) - 1u);
    bool guard = false;
    unsigned good = 0; // points of the pass with values
    if (some && symmetric) {
      if (T.k.cubic)
        build_entries<true, 2>(T.k, np * N * N, T.u + s0, root, dl0, lane);
      else
        build_entries<false, km_flight(ORDER)>(T.k, np * N * N, T.u + s0, root, dl0, lane);
      km_fixed_entries(T, N, np, s0, lgp, root, rsz, lane);
      if (N <= 8 && N >= 4) T.D2[lane] = c2(1.0, 0.0);
      __syncwarp();
      double2 h[8], g;
      if (N > 8)
        km_deep(T, stack, dl0, N, lane, floor_, guard);
      else
        km_subtree(T, out, dl0 + min(lane >> lg, np - 1) * dsz, N, np, false, lane, floor_, guard, h, g);
      const unsigned gm = __ballot_sync(FULL, guard);
      const unsigned pm = lg == 5 ? gm : (gm >> ((lane << lg) & 31)) & ((1u << (1 << lg)) - 1u);
      // a value that is not finite goes to the pivoted-LU pass as a guarded one does
      bool nonfinite = false;
      if (lane < np)
        for (int q = 0; q < n2; ++q) {
          const double2 v = out[lane * n2 + q];
          nonfinite = nonfinite || !isfinite(v.x) || !isfinite(v.y);
        }
      const unsigned flagged = __ballot_sync(FULL, lane < np && (pm || nonfinite)) & some;
      guarded |= flagged << s0;
      good = some & ~flagged;
    }
    // every (point, position, index) of the pass: e = p 2N + 2 (i - 1) + k
    for (int e0 = 0; e0 < np * n2; e0 += 32) {
      const int e = e0 + lane;
      const bool have = e < np * n2;
      const int ee = have ? e : 0, p = ee / n2, q = ee - p * n2, i = q >> 1, kk = (q & 1) ^ flip; // idle lanes: the first
      const bool ok = have && ((good >> p) & 1u);
      const double j = (N & flip) ? -T.jac[s0 + p] : T.jac[s0 + p], t = T.u[((i + 1) << lgp) + s0 + p];
      double2 v = c2(0.0, 0.0); // (whatever the Jacobian of a point that is not evaluated)
      if (ok) v = c2(out[ee].x * j, out[ee].y * j);
      if (eval) {
        if (have && !((guarded >> (s0 + p)) & 1u))
          L.out_kvals[(first + s0 + p) * n2 + 2 * T.place[(i << lgp) + s0 + p] + kk] = v;
        continue;
      }
      if (L.km_fourier) {
        double sn, cs;
        sincos(L.km_omega * t, &sn, &cs);
        csum = cadd(csum, ok ? cmul(v, c2(cs, sn)) : c2(0.0, 0.0));
        continue;
      }
      int bin = -1;
      if (L.bin_xmin <= t && t <= L.bin_xmax)
        bin = t == L.bin_xmax ? L.nbins - 1 : min((int)((t - L.bin_xmin) / L.bin_size), L.nbins - 1);
      csum = cadd(csum, v);
      // each bin's lowest lane adds the lanes' terms in order
      const unsigned same = __match_any_sync(FULL, ok && bin >= 0 ? 2 * bin + kk : -1 - lane);
      double2 s = v;
      for (unsigned r = same & (same - 1u); __any_sync(FULL, r != 0u); r &= r - 1u) {
        const int from = r ? __ffs(r) - 1 : lane;
        const double2 w = c2(__shfl_sync(FULL, v.x, from), __shfl_sync(FULL, v.y, from));
        if (r) s = cadd(s, w);
      }
      if (ok && bin >= 0 && lane == __ffs(same) - 1) {
        const size_t b = (size_t)c * nb + 2 * bin + kk;
        L.bin_sums[b] = cadd(L.bin_sums[b], s);
        L.bin_counts[b] += (unsigned)__popc(same) << (N - 1);
      }
      ndrop += __popc(__ballot_sync(FULL, ok && bin < 0)) << (N - 1);
      __syncwarp();
    }
    __syncwarp();
  }
  return guarded;
}

// Persistent warps pull scheduling chunks and walk them in groups (32 points up to order 3, then 16):
// set-up, then passes of km_pass points, each pass's 2n sums per point to the outputs (IN_TIMES), the
// chunk's bins, or weighted by e^{i omega t} (km_fourier) to the chunk's sum. Points with a guarded
// pivot, and all points of models whose spins differ, are left to the pivoted-LU pass (fb_mask).
__global__ void __launch_bounds__(KM_WARPS * 32, KM_CTAS_PER_SM) km_tree_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  KmShared &T = reinterpret_cast<KmShared *>(smem_raw)[warp];
  double2 *stack = reinterpret_cast<double2 *>(L.pts) + (size_t)(blockIdx.x * KM_WARPS + warp) * KM_STACK;
  const bool eval = L.mode != IN_SOBOL;
  const int nb = L.nbins * 2;
  bool bad = false;
  int item = -1, next = first_chunk();
  for (;;) {
    const int c = __shfl_sync(FULL, next, 0);
    if (c >= L.n_chunks) break;
    next = later_chunk(L.chunk_counter, KM_WARPS, lane); // the chunk after this one, ahead of its use
    bool fresh = item < 0;
    if (fresh || c >= L.chunk_offsets[item + 1] || c < L.chunk_offsets[item]) {
      item = find_chunk_item(L.chunk_offsets, L.n_items, c, lane);
      fresh = true;
    }
    const ItemDev &it = L.items[item]; // (a copy as the integrand's kernel keeps doubles the spills: +20 %)
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    const int ccount = (int)min((long long)it.chunk_points, (long long)it.n_points - cfirst);
    const int N = it.order, lgp = km_group_lg(N), st = 1 << lgp;
    const bool keep = eval ? (L.keep_u_hypercube != 0) : true;
    const double rdelta = 1.0 / it.model.delta;
    __syncwarp();
    if (fresh) fill_item(T.k, it, rdelta, km_lookups.e + km_lookups.first[N], lane);
    if (!eval && L.nbins) {
      for (int b = lane; b < nb; b += 32) {
        L.bin_sums[(size_t)c * nb + b] = c2(0.0, 0.0);
        L.bin_counts[(size_t)c * nb + b] = 0u;
      }
    }
    __syncwarp();
    double2 csum = c2(0.0, 0.0);
    unsigned ndom = 0, nfb = 0, ndrop = 0;
    unsigned long long fbm[2] = {0, 0};
    for (int g0 = 0; g0 < ccount; g0 += st) {
      const int cnt = min(st, ccount - g0);
      const bool mine = lane < cnt;
      double *ul = T.u + st + lane;
      const GroupSetup su =
          setup_group(L.mode, L.in, it, N, lgp, cfirst + g0, cnt, keep, T.u + st, reinterpret_cast<double *>(T.buf), lane);
      const double jac = su.jac;
      const bool dom = su.dom;
      bool sorted = su.sorted;
      bool in = mine && dom;
      if (mine) {
        // (equal times need the vertices' order: the set-up's `sorted` lets them pass)
        for (int j = 1; j < N; ++j) sorted = sorted && ul[j << lgp] < ul[(j - 1) << lgp];
        if (sorted)
          for (int j = 0; j < N; ++j) T.place[(j << lgp) + lane] = (unsigned char)j;
        else
          sort_places(ul, T.place + lane, st, N);
        T.jac[lane] = jac;
      }
      if (in && it.spin_symmetric && !in_window(it, N, ul, st, rdelta)) {
        bad = true;
        in = false;
      }
      const unsigned dommask = __ballot_sync(FULL, mine && dom);
      const unsigned inmask = __ballot_sync(FULL, in);
      if (mine) {
        const double tX = it.f.A.time;
        T.u[lane] = T.u[((N + 1) << lgp) + lane] = tX;
        if (!in) // a point that is not evaluated still takes its place in a pass: at X's time, inside the window
          for (int j = 0; j < N; ++j) T.u[((j + 1) << lgp) + lane] = dom && !it.spin_symmetric ? ul[j << lgp] : tX;
      }
      __syncwarp();
      unsigned guarded;
      switch (N) {
        case 1: guarded = km_passes<1>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 2: guarded = km_passes<2>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 3: guarded = km_passes<3>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 4: guarded = km_passes<4>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 5: guarded = km_passes<5>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 6: guarded = km_passes<6>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 7: guarded = km_passes<7>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        case 8: guarded = km_passes<8>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop); break;
        default: guarded = km_passes<0>(L, T, N, it.spin_symmetric, cnt, inmask, dommask, cfirst + g0, c, stack, lane, csum, ndrop);
      }
      if (eval && mine) {
        const long long o = cfirst + g0 + lane;
        if (L.out_jac) L.out_jac[o] = jac;
        if (L.out_dom) L.out_dom[o] = dom ? 1 : 0;
      }
      guarded &= dommask;
      ndom += __popc(dommask);
      nfb += __popc(guarded);
      if (g0 < 64) fbm[0] |= (unsigned long long)guarded << g0; // (32 | g0 up to order 3, then 16 | g0: no carry)
      else fbm[1] |= (unsigned long long)guarded << (g0 - 64);
      __syncwarp();
    }
    csum = lane_sum(csum, 0, 5);
    if (lane == 0) {
      ChunkPartial pr;
      pr.sum_re = csum.x;
      pr.sum_im = csum.y;
      pr.n_in_domain = ndom;
      pr.n_fallback = nfb;
      pr.fb_mask[0] = fbm[0];
      pr.fb_mask[1] = fbm[1];
      L.partials[c] = pr;
      if (!eval && L.nbins) L.bin_dropped[c] = ndrop;
      if (eval && nfb) atomicAdd(L.n_flagged, (int)nfb);
    }
  }
  if (__any_sync(FULL, bad) && lane == 0) atomicOr(L.err, 1);
}

static_assert(KM_WARPS * sizeof(KmShared) <= 233472 / KM_CTAS_PER_SM - 1024, "the resident CTAs share an SM's shared memory");

} // namespace

cudaError_t configure_km_kernel() {
  return cudaFuncSetAttribute(km_tree_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KM_WARPS * (int)sizeof(KmShared));
}

cudaError_t launch_km_tree(const Launch &L, int grid, cudaStream_t st) {
  km_tree_kernel<<<grid, KM_WARPS * 32, KM_WARPS * sizeof(KmShared), st>>>(L);
  return cudaGetLastError();
}

} // namespace kb
