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
//   So a node of the elimination tree with m vertices left is ONE (m+1) x (m+1) matrix S (of every
//   entry the copy that starts as g^<, or of every entry g^>: EntryKind), both children of a node
//   share its pivot p, and the difference of an entry's two copies is the same number at every
//   node: S_ij + delta_ij with delta fixed per point. (A node of both copies, as in an elimination in the given order, is
//   (2m+1)^2 entries and two pivots.)
// * The last two vertices need no division. With X, Y the external entries of the latest
//   vertex, its two configurations differ only in them, so the external corner and the
//   square of the leaf's own terms cancel before anything is rounded:
//     sum_{a1} = -D^2 p2 p1' (X_0 Y_0 - X_1 Y_1)', and p2 times each factor is a polynomial
//   of the 3 x 3 matrix's entries (leaf2).
//
// Cost: sum_m 2^(n-m) (m+1)^2 complex multiply-adds, ~15 * 2^n (the elimination in the given
// order with both copies, which this kernel replaced, took ~40 * 2^n).
//
// Work split: a level of 256 >> m nodes with m vertices left fills a warp from m = 8 (one
// node, one point) down to m = 3 (32 nodes, one per lane), whatever the order: order n starts
// at level n with 2^(8-n) points per warp. Levels 8 to 5 go through shared memory with the lanes
// of a node splitting its children; the last five vertices run in registers. Orders above 8
// walk the levels above 9 depth first. Warps never wait for each other: no CTA barrier.
//
// Bound: latency. Order 8 (2^20 points): 3.17 ms (13.1 for the elimination in the given order, one
// CTA per sub-batch of points). Of 65,536 points (0.37 ms) ncu shows the FP64 pipe 39 % busy, 1,335
// instructions per point, shared memory 44 %; the stalls are shared-memory loads (2.2 cycles per
// issued instruction) and fixed latencies of dependent FP64 instructions (1.8) at 12 warps per SM.
// Measured when order 8 took 3.6 to 3.8 ms: splitting a level's nodes over fewer
// lanes with more registers (512 >> m nodes, 255 registers, 8 warps) took 4.6 ms, 15 warps at
// 128 registers 4.8 (spills), an elimination of both vertices 8 and 7 per step 4.1.
#include <cuda_runtime.h>

#include "kb_wick.cuh"

namespace kb {

namespace {

// Row width and node size of a node with m vertices left (m+1 rows). A 16-byte shared-memory read
// takes two cycles when each half-warp reads at most eight distinct words in different 16-byte
// banks and four when all words differ; the widths, the sizes and the lanes' blocks are chosen
// for that in the reads of levels 6 and 5.
__host__ __device__ constexpr int node_w(int m) { return m == 7 ? 9 : m == 6 ? 10 : m + 1; }
__host__ __device__ constexpr int node_sz(int m) {
  return m == 1 ? 5 : m == 2 ? 9 : m == 3 ? 17 : m == 4 ? 25 : m == 5 ? 37 : m == 6 ? 76 : m == 7 ? 72 : (m + 1) * (m + 1);
}
// Complex entries of a warp's buffers: the nodes of odd levels (and the roots of orders 1..4) at 0,
// those of levels 6 and 8 behind level 5's, then the point differences delta, then the nodes of
// levels 8 and 9 that orders above 8 keep.
constexpr int NODES6 = 8 * 37;
constexpr int NODES_END = NODES6 + 4 * 76;
constexpr int WARP_BUF = 960;
__host__ __device__ constexpr int node_base(int m) { return m == 6 || m == 8 ? NODES6 : 0; }
__host__ __device__ constexpr int delta_base(int n) { return n >= 6 ? NODES_END : n == 5 ? NODES6 : n == 4 ? 16 * 25 : 32 * 17; }
// delta of a point, in shells: vertex k (1 = latest) holds its k column entries (i, k), i < k,
// at k(k-1), then its k row entries (k, j), j < k, at k*k.
__host__ __device__ constexpr int delta_sz(int n) { return n < 8 ? n * (n + 1) + 1 : n * (n + 1); }
// Points of a pass (2^(n-3) lanes per point, at most one point per lane), and of a group.
__host__ __device__ constexpr int pass_points(int n) { return n <= 3 ? 32 : n >= 8 ? 1 : 256 >> n; }
// Points whose roots are built together: a pass's, but two of order 8 (72 entries a point leave the
// lanes' second and third lookup idle: 3.25 -> 3.16 ms). Lookups in flight per lane: with whole rounds
// of lanes for the build's entries (3 at every order: order 7's 112 took two rounds, 1.89 ms for 1.78;
// order 10 13.3 for 12.9).
__host__ __device__ constexpr int build_points(int n) { return n == 8 ? 2 : pass_points(n); }
__host__ __device__ constexpr int build_flight(int n) {
  constexpr int FLIGHT[] = {4, 2, 3, 6, 5, 4, 3, 4, 5}; // (0: the orders above 8)
  return FLIGHT[n];
}
// A root's place: its level's, order 8's two behind the differences.
__host__ __device__ constexpr int root_base(int n) { return n == 8 ? NODES_END + 2 * 72 : node_base(n); }
__host__ __device__ constexpr int group_lg(int n) { return n <= 8 ? 5 : 4; }
static_assert(delta_base(3) + 32 * delta_sz(3) <= WARP_BUF && delta_base(4) + 16 * delta_sz(4) <= WARP_BUF &&
                  delta_base(5) + 8 * delta_sz(5) <= WARP_BUF && delta_base(6) + 4 * delta_sz(6) <= WARP_BUF &&
                  delta_base(16) + delta_sz(16) <= WARP_BUF && root_base(8) + 2 * 81 <= WARP_BUF && ITEM_END <= WARP_BUF,
              "differences (and the set-up's factors) fit in a warp's buffers");
// The lookups of a pass: entry (p, i, j), i != j, of point p's root (position 0: external row A or
// column B; 1..n: the vertices, latest first). Fields: index of the times of positions i and j in
// the group's array, place in the roots and in the differences, kind (0: j the earlier vertex,
// 1: i the earlier, 2: row A, 3: column B).
constexpr int lookup_first(int n) { // entries of orders below n
  int s = 0;
  for (int k = 1; k < n; ++k) s += build_points(k) * k * (k + 1);
  return s;
}
struct LookupTable {
  unsigned long long e[lookup_first(MAX_ORDER + 1)];
  int first[MAX_ORDER + 1];
  constexpr LookupTable() : e(), first() {
    int r = 0;
    for (int n = 1; n <= MAX_ORDER; ++n) {
      first[n] = r;
      const int ssz = n > 8 ? 0 : n == 8 ? 81 : node_sz(n), w = n > 8 ? n + 1 : node_w(n), st = 1 << group_lg(n);
      for (int p = 0; p < build_points(n); ++p)
        for (int i = 0; i <= n; ++i)
          for (int j = 0; j <= n; ++j) {
            if (i == j) continue;
            const unsigned long long ui = i * st + p, uj = (j ? j : n + 1) * st + p;
            const unsigned long long so = p * ssz + i * w + j, dof = p * delta_sz(n) + (i < j ? j * (j - 1) + i : i * i + j);
            const unsigned long long kind = i == 0 ? 2 : j == 0 ? 3 : i < j ? 0 : 1;
            e[r++] = ui | uj << 10 | so << 20 | dof << 32 | kind << 42;
          }
    }
  }
};
__device__ const LookupTable lookups = LookupTable();

// What a warp keeps of its chunk from group to group: the same in all lanes, where a spilled register
// is 128 bytes and an L2 round trip (with the item's copy: order 1 0.18 -> 0.13 ms, order 2 0.25 -> 0.19).
struct ChunkState {
  double2 sum;
  unsigned long long fb0, fb1; // the guarded points' bits
  long long first;             // first point of the chunk within its item
  int chunk, item, count, order;
  unsigned ndom, nfb, ndrop;
};

template <bool SCALE>
struct WarpShared {
  double2 buf[WARP_BUF];
  double u[320];      // the group's times, u[i * gp + p]: A, the vertices latest first, B
  double2 fval[32];   // the group's values
  ItemConst k;
  double2 D2[24];     // squared prefix determinants: level 5's nodes at 0, 6's at 8, 7's and 8's at
                      // 12, the depth-first levels' above 8 at 16
  double cutoff;
  ChunkState s;
  double fscale[SCALE ? 32 : 1];
};

// Root matrices and differences of the np points of a pass (u: their times).
template <bool CUBIC, int GK>
__device__ __forceinline__ void build_roots(const ItemConst &K, int N, int np, const double *u, double2 *S, int ssz,
                                            int sw, double2 *dl, int lane) {
  build_entries<CUBIC, GK>(K, np * N * (N + 1), u, S, dl, lane);
  // diagonals (equal contour points) and the external corner
  const unsigned md = 0xFFFFFFFFu / (unsigned)(N + 1) + 1u; // e / (N + 1) by multiply-high
  const double2 eq = K.eq;
  for (int e = lane; e < np * (N + 1); e += 32) {
    const int p = (int)__umulhi((unsigned)e, md), i = e - p * (N + 1);
    S[p * ssz + i * (sw + 1)] = i == 0 ? c2(0.0, 0.0) : eq;
  }
}

// ------------------------------------------------------------------ the tree

// Nodes of a level, and the lanes of a node, are numbered so that a point's nodes stay in its
// own lanes: with m vertices left, node lane >> (m-3), whose low bit is the copy of vertex m+1
// that led to it (0: delta in its column, 1: delta in its row).

// Level 8 (node S, 9 x 9) to level 7: half a row of its child per lane.
__device__ __forceinline__ void level8(const double2 *S, double2 *buf, const double2 *dl, double2 D2, double2 *D2c,
                                       int lane, double floor_, bool &guard) {
  constexpr int W = node_w(8), WC = node_w(7);
  const int child = lane >> 4, l = lane & 15, i = l >> 1, j0 = (l & 1) * 4;
  const double2 *dc = dl + 56, *dr = dl + 64;
  const double f = child ? 0.0 : 1.0;
  const double2 p = S[8 * W + 8], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  if (l == 0) D2c[child] = cmul(D2, cmul(p, p));
  const double2 Lf = cmul(copyof(S[i * W + 8], dc[i], f), ip);
  double2 *o = buf + node_base(7) + child * node_sz(7) + i * WC + j0;
#pragma unroll
  for (int q = 0; q < 4; ++q) o[q] = cfms(S[i * W + j0 + q], Lf, copyof(S[8 * W + j0 + q], dr[j0 + q], 1.0 - f));
}

// Level 7 to level 6: a row of its child per lane.
__device__ __forceinline__ void level7(double2 *buf, const double2 *dl, const double2 *D2p, double2 *D2c, int lane, double floor_, bool &guard) {
  constexpr int W = node_w(7), WC = node_w(6);
  const int child = lane >> 3, i = lane & 7;
  const double2 *S = buf + node_base(7) + (child >> 1) * node_sz(7);
  const double2 *dc = dl + 42, *dr = dl + 49;
  const double f = (child & 1) ? 0.0 : 1.0;
  const double2 p = S[7 * W + 7], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  if (i < 7) {
    const double2 Lf = cmul(copyof(S[i * W + 7], dc[i], f), ip);
    double2 *o = buf + node_base(6) + child * node_sz(6) + i * WC;
#pragma unroll
    for (int j = 0; j < 7; ++j) o[j] = cfms(S[i * W + j], Lf, copyof(S[7 * W + j], dr[j], 1.0 - f));
  } else {
    D2c[child] = cmul(D2p[child >> 1], cmul(p, p));
  }
}

// Level 6 to level 5: a 3 x 3 block of its child per lane.
__device__ __forceinline__ void level6(double2 *buf, const double2 *dl, const double2 *D2p, double2 *D2c, int lane,
                                       double floor_, bool &guard) {
  constexpr int W = node_w(6), WC = node_w(5);
  const int child = lane >> 2, l = lane & 3, i0 = (l >> 1) * 3, j0 = (l & 1) * 3;
  const double2 *S = buf + node_base(6) + (child >> 1) * node_sz(6);
  const double2 *dc = dl + 30, *dr = dl + 36;
  const double f = (child & 1) ? 0.0 : 1.0;
  const double2 p = S[6 * W + 6], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  if (l == 0) D2c[child] = cmul(D2p[child >> 1], cmul(p, p));
  double2 r[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) r[j] = copyof(S[6 * W + j0 + j], dr[j0 + j], 1.0 - f);
  double2 *o = buf + node_base(5) + child * node_sz(5) + i0 * WC + j0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double2 Lf = cmul(copyof(S[(i0 + i) * W + 6], dc[i0 + i], f), ip);
#pragma unroll
    for (int j = 0; j < 3; ++j) o[i * WC + j] = cfms(S[(i0 + i) * W + j0 + j], Lf, r[j]);
  }
}

// The last two vertices of a node T (3 x 3: external, latest vertex 1, vertex 2), all four
// configurations. With c = (T02, T12), r = (T20, T21) of vertex 2's copy, after its elimination
//   p2 p1' = T11 p2 - c1 r1 = q,  p2 (X_0 Y_0 - X_1 Y_1) = p2 K + c0 r1 dY - c1 r0 dX,
// (X, Y = T01, T10; X_0 = X + dX, Y_1 = Y + dY; K = dX Y - X dY), and the two leaves of
// vertex 1 sum to -D^2 q times that: no division, the external corner drops out. Returns
// q_1 (...)_1 - q_0 (...)_0. d2: vertex 2's differences {c0, c1, r0, r1}; g2 = d2[0] dY,
// h2 = dX d2[2]. SCALE: also the sum of |term| of the four leaves, without the factor D^2.
template <bool SCALE>
__device__ __forceinline__ double2 leaf2(const double2 (&T)[9], double2 dX, double2 dY, const double2 (&d2)[4],
                                         double2 g2, double2 h2, double &scale, double floor_, bool &guard) {
  const double2 K = cfms(cmul(dX, T[3]), T[1], dY);
  const double2 P = cmul(T[4], T[8]), Q = cmul(T[8], K);
  const double2 g = cmul(T[2], dY), h = cmul(dX, T[6]);
  const double2 c1 = cadd(T[5], d2[1]), r1 = cadd(T[7], d2[3]);
  const double2 t1 = cmul(cfms(P, T[5], r1), cfms(cfma(Q, g, r1), cadd(h, h2), T[5]));
  const double2 t0 = cmul(cfms(P, c1, T[7]), cfms(cfma(Q, cadd(g, g2), T[7]), h, c1));
  if constexpr (SCALE) {
    if (!(cabs1(T[8]) >= floor_)) guard = true;
    const double2 ip = pivot_rcp(T[8]);
#pragma unroll
    for (int a2 = 0; a2 < 2; ++a2) {
      const double2 c0 = a2 ? T[2] : cadd(T[2], d2[0]), r0 = a2 ? cadd(T[6], d2[2]) : T[6];
      const double2 k1 = a2 ? T[5] : c1, s1 = a2 ? r1 : T[7];
      const double2 q = cfms(P, k1, s1), sg = cfms(cmul(T[8], T[0]), c0, r0);
#pragma unroll
      for (int a1 = 0; a1 < 2; ++a1) {
        const double2 X = a1 ? T[1] : cadd(T[1], dX), Y = a1 ? cadd(T[3], dY) : T[3];
        const double2 xi = cfms(cmul(T[8], X), c0, s1), et = cfms(cmul(T[8], Y), k1, r0);
        scale += cabs(cmul(cmul(q, ip), cfms(cmul(q, sg), xi, et)));
      }
    }
  }
  return c2(t1.x - t0.x, t1.y - t0.y);
}

// The last three vertices of a node s (4 x 4, in registers), all eight configurations, times
// the node's D^2: vertex 3's elimination for both copies, then leaf2.
template <bool SCALE>
__device__ __forceinline__ double2 leaf3(const double2 (&s)[16], const double2 *dl, double2 D2, double floor_,
                                         bool &guard, double &scale) {
  const double2 p = s[15];
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = pivot_rcp(p);
  const double2 dX = dl[0], dY = dl[1];
  const double2 d2[4] = {dl[2], dl[3], dl[4], dl[5]};
  const double2 g2 = cmul(d2[0], dY), h2 = cmul(dX, d2[2]);
  double2 acc = c2(0.0, 0.0);
  double sc = 0.0;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    double2 r[3], T[9];
#pragma unroll
    for (int j = 0; j < 3; ++j) r[j] = a ? cadd(s[12 + j], dl[9 + j]) : s[12 + j];
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

// Level 5 to this lane's node s of level 3 (index = lane), both eliminations in registers; returns
// its D^2. (Through level-4 nodes in shared memory, two lanes sharing each elimination, order 8 takes
// 6 % longer.)
template <bool SCALE>
__device__ __forceinline__ double2 level5(double2 (&s)[16], const double2 *buf, const double2 *dl, const double2 *D2p,
                                          int lane, double floor_, bool &guard) {
  constexpr int W = node_w(5);
  const double2 *S = buf + node_base(5) + (lane >> 2) * node_sz(5);
  const double f5 = (lane & 2) ? 0.0 : 1.0, f4 = (lane & 1) ? 0.0 : 1.0;
  const double2 p5 = S[5 * W + 5], i5 = pivot_rcp(p5);
  double2 r5[5], r4[4];
#pragma unroll
  for (int j = 0; j < 5; ++j) r5[j] = copyof(S[5 * W + j], dl[25 + j], 1.0 - f5);
  const double2 L54 = cmul(copyof(S[4 * W + 5], dl[24], f5), i5);
  const double2 p4 = cfms(S[4 * W + 4], L54, r5[4]), i4 = pivot_rcp(p4);
  if (!(cabs1(p5) >= floor_) || !(cabs1(p4) >= floor_)) guard = true;
#pragma unroll
  for (int j = 0; j < 4; ++j) r4[j] = copyof(cfms(S[4 * W + j], L54, r5[j]), dl[16 + j], 1.0 - f4);
  s[0] = c2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double2 L5 = cmul(copyof(S[i * W + 5], dl[20 + i], f5), i5);
    const double2 L4 = cmul(copyof(cfms(S[i * W + 4], L5, r5[4]), dl[12 + i], f4), i4);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (SCALE || i + j > 0) s[4 * i + j] = cfms(cfms(S[i * W + j], L5, r5[j]), L4, r4[j]);
  }
  const double2 pp = cmul(p5, p4);
  return cmul(D2p[lane >> 2], cmul(pp, pp));
}

// Order 4's child s of this lane (child index = lane) in registers; returns its D^2.
template <bool SCALE>
__device__ __forceinline__ double2 level4(double2 (&s)[16], const double2 *buf, const double2 *dl, const double2 *D2p,
                                          int lane, double floor_, bool &guard) {
  const double2 *S = buf + (lane >> 1) * node_sz(4);
  const double f = (lane & 1) ? 0.0 : 1.0;
  const double2 p = S[24], ip = pivot_rcp(p);
  if (!(cabs1(p) >= floor_)) guard = true;
  double2 r[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) r[j] = copyof(S[20 + j], dl[16 + j], 1.0 - f);
  s[0] = c2(0.0, 0.0);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double2 Lf = cmul(copyof(S[5 * i + 4], dl[12 + i], f), ip);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (SCALE || i + j > 0) s[4 * i + j] = cfms(S[5 * i + j], Lf, r[j]);
  }
  return cmul(D2p[lane >> 1], cmul(p, p));
}

// The tree below the roots of order n <= 8 in the buffers, or below the node of level 8 at
// T.buf[node8] with D^2 = D8 (orders 8 and up): this lane's value, with the sign of its copies of the
// vertices down to 4.
template <bool SCALE>
__device__ __forceinline__ double2 subtree(WarpShared<SCALE> &T, int node8, double2 D8, const double2 *dl, int n, int lane,
                                           double floor_, bool &guard, double &scale) {
  double2 s[16], D2 = c2(1.0, 0.0);
  if (n <= 3) {
    const double2 *S = T.buf + lane * node_sz(3);
#pragma unroll
    for (int e = 0; e < 16; ++e) s[e] = S[e];
  } else {
    if (n >= 8) {
      level8(T.buf + node8, T.buf, dl, D8, T.D2 + 12, lane, floor_, guard);
      __syncwarp();
    }
    if (n >= 7) level7(T.buf, dl, T.D2 + 12, T.D2 + 8, lane, floor_, guard);
    if (n >= 6) {
      __syncwarp();
      level6(T.buf, dl, T.D2 + 8, T.D2, lane, floor_, guard);
      __syncwarp();
    }
    if (n == 4)
      D2 = level4<SCALE>(s, T.buf, dl, T.D2, lane, floor_, guard);
    else
      D2 = level5<SCALE>(s, T.buf, dl, T.D2, lane, floor_, guard);
  }
  const double2 v = leaf3<SCALE>(s, dl, D2, floor_, guard, scale);
  const int lg = n <= 3 ? 0 : min(n, 8) - 3;
  return (__popc(lane & ((1 << lg) - 1)) & 1) ? c2(-v.x, -v.y) : v;
}

// One step above level 8: node S (m vertices left, m+1 wide) to its child of copy a, or PAIR: to both
// children (copy 0 by the lower half-warp at o, copy 1 by the upper one behind it), m wide. A column
// per lane; its rows' loads are issued together, as S may lie in global scratch. D2n: the
// children's D^2. The caller's __syncwarp follows.
template <bool PAIR>
__device__ __forceinline__ void step_down(const double2 *S, double2 *o, const double2 *dl, int m, int a, int lane,
                                          double2 D2, double2 &D2n, double floor_, bool &guard) {
  const int W = m + 1, j = lane & 15, half = lane >> 4;
  const double2 p = S[m * W + m];
  const double2 *dc = dl + m * (m - 1), *dr = dl + m * m;
  const double f = (PAIR ? half : a) ? 0.0 : 1.0;
  const int col = min(j, m - 1); // idle lanes repeat the last column's loads
  const double2 r = copyof(S[m * W + col], dr[col], 1.0 - f);
  if (!(cabs1(p) >= floor_)) guard = true;
  const double2 ip = pivot_rcp(p);
  D2n = cmul(D2, cmul(p, p));
  if (PAIR) o += half * m * m;
  constexpr int ROWS = 5, STEP = PAIR ? 1 : 2;
  for (int i0 = PAIR ? 0 : half; i0 < m; i0 += ROWS * STEP) {
    double2 c[ROWS], x[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const int i = min(i0 + k * STEP, m - 1);
      c[k] = copyof(S[i * W + m], dc[i], f);
      x[k] = S[i * W + col];
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const int i = i0 + k * STEP;
      if (i < m && j < m) o[i * m + j] = cfms(x[k], cmul(c[k], ip), r);
    }
  }
}

// a on lanes with bit `bit` clear, b on the others, each summed over the lane pair.
__device__ __forceinline__ double2 merge_lanes(double2 a, double2 b, int bit, int lane) {
  const bool up = lane & bit;
  const double2 keep = up ? b : a, send = up ? a : b;
  return c2(keep.x + __shfl_xor_sync(FULL, send.x, bit), keep.y + __shfl_xor_sync(FULL, send.y, bit));
}

// A group's points in passes, each point's value into T.fval; returns the points with a guarded
// pivot (bit per point of the group). ORDER: 1..8, 0 for the orders above. Compiled per order, as
// the places, strides and the levels that an order has are then constants: 2^20 points of order 8 3.54 ->
// 3.25 ms, of order 5 0.68 -> 0.61, and the orders above, without the branches of the others, 5 to
// 10 % less.
template <bool SCALE, bool ANY_CUBIC, int ORDER>
__device__ __forceinline__ unsigned group_values(WarpShared<SCALE> &T, int order, int cnt, unsigned inmask, double2 *stack,
                                                 int lane) {
  constexpr bool DEEP = ORDER == 0;
  const int n = DEEP ? order : ORDER;
  const double floor_ = T.k.floor_;
  const int P = pass_points(n);
  const int lg = n <= 3 ? 0 : min(n, 8) - 3; // lanes per point
  double2 *dl0 = T.buf + delta_base(DEEP ? 9 : n);
  const int dsz = delta_sz(n);
  // orders above 8: the depth-first levels' nodes, level 8's pair and then level 9's node behind the
  // differences in shared memory where they fit, the others in global scratch
  double2 *pair8 = nullptr, *node9 = nullptr;
  int pair_at = 0;
  if constexpr (DEEP) {
    int room = WARP_BUF - delta_base(n) - dsz;
    double2 *at = dl0 + dsz;
    int soff = 0;
    for (int m = n; m > 9; --m) soff += (m + 1) * (m + 1);
    pair8 = stack + TREE_STACK - 162;
    node9 = stack + soff;
    if (room >= 162) {
      pair8 = at;
      pair_at = (int)(at - T.buf);
      at += 162;
      room -= 162;
    }
    if (room >= 100) node9 = at;
  }
  const int K0 = max(n - 9, 0); // K0 depth-first levels above level 9
  double2 *root = DEEP ? (n > 9 ? stack : node9) : T.buf + root_base(n);
  const int rsz = DEEP ? 0 : n == 8 ? 81 : node_sz(n), rw = DEEP ? n + 1 : node_w(n);
  unsigned guarded = 0;
  double2 h0 = c2(0.0, 0.0), h1 = c2(0.0, 0.0); // values of earlier passes of a quad, not yet summed over lanes
  for (int s0 = 0, t = 0; s0 < cnt || (lg >= 2 && (t & 3)); s0 += P, ++t) {
    const int np = min(P, cnt - s0);
    const unsigned in = np <= 0 ? 0u : (inmask >> s0) & (np >= 32 ? FULL : (1u << np) - 1u);
    bool guard = false;
    double scale = 0.0;
    double2 v = c2(0.0, 0.0);
    const bool second = ORDER == 8 && (t & 1) && ((inmask >> (s0 - 1)) & 1u);
    if (in) {
      const int nb = ORDER == 8 ? min(2, cnt - s0) : np;
      if (second) { // built with the point before
      } else if (ANY_CUBIC && T.k.cubic)
        build_roots<true, 2>(T.k, n, nb, T.u + s0, root, rsz, rw, dl0, lane);
      else
        build_roots<false, build_flight(ORDER)>(T.k, n, nb, T.u + s0, root, rsz, rw, dl0, lane);
      if (!DEEP && n <= 7 && n >= 4) {
        if (n >= 5 && lane < 8) T.D2[n == 7 ? 12 + (lane & 1) : n == 6 ? 8 + (lane & 3) : lane] = c2(1.0, 0.0);
        if (n == 4 && lane < 16) T.D2[lane] = c2(1.0, 0.0);
      }
      __syncwarp();
      if (DEEP || n >= 3) {
        // orders above 8: 2^K0 subtrees of level 9's node, each its two children's; else one tree
        const double2 *dl = DEEP || n >= 8 ? dl0 + dsz * second : dl0 + min(lane >> lg, np - 1) * dsz; // (idle lanes: the last point's)
        double2 D8 = c2(1.0, 0.0);
        const int trees = DEEP ? 2 << K0 : 1;
        for (int tr = 0; tr < trees; ++tr) {
          int node8 = ORDER == 8 ? root_base(8) + 81 * second : node_base(8);
          if constexpr (DEEP) {
            if (pair_at) {
              node8 = pair_at + 81 * (tr & 1);
            }
            if ((tr & 1) == 0) {
              // the levels whose copy changed since the last subtree, down to level 9
              const int sub = tr >> 1, first = sub == 0 ? 0 : K0 - __ffs(sub);
              int off = 0;
              for (int d = 0; d <= K0; ++d) {
                const int m = n - d;
                const double2 *S = d == K0 ? node9 : stack + off;
                off += (m + 1) * (m + 1);
                if (d < first) continue;
                const double2 D2 = d == 0 ? c2(1.0, 0.0) : T.D2[15 + d];
                if (d == K0)
                  step_down<true>(S, pair8, dl0, 9, 0, lane, D2, D8, floor_, guard);
                else
                  step_down<false>(S, d + 1 == K0 ? node9 : stack + off, dl0, m, (sub >> (K0 - 1 - d)) & 1, lane, D2, D8,
                                   floor_, guard);
                if (lane == 0) T.D2[16 + d] = D8;
                __syncwarp();
              }
            }
            if (!pair_at) { // orders 14 to 16: level 8's node from global scratch
              for (int e = lane; e < 81; e += 32) T.buf[node_base(8) + e] = pair8[81 * (tr & 1) + e];
              __syncwarp();
            }
          }
          const double2 w = subtree<SCALE>(T, node8, D8, dl, DEEP ? 8 : n, lane, floor_, guard, scale);
          v = (__popc(tr) & 1) ? c2(v.x - w.x, v.y - w.y) : cadd(v, w);
          __syncwarp();
        }
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
      } else if (lane < np) { // order 1: -p (X_0 Y_0 - X_1 Y_1)
        const double2 *S = T.buf + lane * node_sz(1), *dl = dl0 + lane * dsz;
        const double2 dX = dl[0], dY = dl[1];
        v = cmul(S[3], cfms(cmul(S[1], dY), dX, S[2]));
        if (SCALE) {
          const double2 X = S[1], Y = S[2], z = cmul(S[3], S[0]);
          scale = cabs(cmul(S[3], cfms(z, cadd(X, dX), Y))) + cabs(cmul(S[3], cfms(z, X, cadd(Y, dY))));
        }
      }
      const unsigned gm = __ballot_sync(FULL, guard);
      if (gm) {
        const unsigned mine = lg == 5 ? gm : (gm >> ((lane << lg) & 31)) & ((1u << (1 << lg)) - 1u);
        guarded |= __ballot_sync(FULL, lane < np && mine) << s0;
      }
    }
    if (SCALE) {
      for (int off = 1; off < (1 << lg); off <<= 1) scale += __shfl_xor_sync(FULL, scale, off);
      if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < np) T.fscale[s0 + (lane >> lg)] = scale;
    }
    // sums over a point's lanes. Of four passes at a time (4 lanes per point and up): the first two
    // rounds leave the lanes of each residue mod 4 with one pass's value, the others sum those
    if (lg >= 2) {
      if ((t & 1) == 0) {
        h0 = v;
      } else if ((t & 3) == 1) {
        h1 = merge_lanes(h0, v, 1, lane);
      } else {
        v = merge_lanes(h1, merge_lanes(h0, v, 1, lane), 2, lane);
        for (int off = 4; off < (1 << lg); off <<= 1) {
          v.x += __shfl_xor_sync(FULL, v.x, off);
          v.y += __shfl_xor_sync(FULL, v.y, off);
        }
        const int q = (t - 3 + (lane & 3)) * P + (lane >> lg);
        if ((lane & ((1 << lg) - 4)) == 0 && q < cnt) T.fval[q] = v;
      }
    } else {
      if (lg == 1) {
        v.x += __shfl_xor_sync(FULL, v.x, 1);
        v.y += __shfl_xor_sync(FULL, v.y, 1);
      }
      if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < np) T.fval[s0 + (lane >> lg)] = v;
    }
    __syncwarp();
  }
  return guarded;
}

__device__ __forceinline__ double2 cut_off(double2 f, double cutoff) { return cutoff > 0.0 && cabs(f) < cutoff ? c2(0.0, 0.0) : f; }

// Order 0: g0(A, B).
__device__ __noinline__ double2 order0(const ItemDev &it, int *err) {
  kb_gf_index a = it.f.A, b = it.f.B;
  a.timesplit = b.timesplit = 0;
  int b0 = 0;
  const double2 v = g0_contour(it.model, a, b, 0, &b0);
  if (b0) atomicOr(err, 1);
  return v;
}

// Persistent warps pull scheduling chunks (it.chunk_points points of one item) and walk them
// in groups of up to 32 points (16 above order 8): set-up, values, then the group's sum in a
// fixed shuffle order, so that results do not depend on which warp ran what.
template <bool EVAL, bool ANY_CUBIC, bool SCALE>
__global__ void __launch_bounds__(TREE_WARPS * 32, TREE_CTAS_PER_SM) tree_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpShared<SCALE> &T = reinterpret_cast<WarpShared<SCALE> *>(smem_raw)[warp];
  double2 *stack = reinterpret_cast<double2 *>(L.pts) + (size_t)(blockIdx.x * TREE_WARPS + warp) * TREE_STACK;
  if (lane == 0) T.s.item = -1;
  int next = first_chunk();
  for (;;) {
    const int c = __shfl_sync(FULL, next, 0);
    if (c >= L.n_chunks) break;
    next = later_chunk(L.chunk_counter, TREE_WARPS, lane); // the chunk after this one, ahead of its use
    __syncwarp();
    int item = T.s.item;
    bool fresh = item < 0;
    if (fresh || c >= L.chunk_offsets[item + 1]) {
      item = find_chunk_item(L.chunk_offsets, L.n_items, c, lane);
      fresh = true;
    }
    const ItemDev &it = stage_item(T.buf, L.items + item, lane); // until group_values
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    if (lane == 0)
      T.s = ChunkState{c2(0.0, 0.0), 0, 0, cfirst, c, item, (int)min((long long)it.chunk_points, (long long)it.n_points - cfirst), it.order, 0, 0, 0};
    const int N = it.order;
    const bool keep = EVAL ? (L.keep_u_hypercube != 0) : true;
    const int lgp = group_lg(N);
    if (fresh) { // what the passes read of the item
      if (N > 0) fill_item(T.k, it, 1.0 / it.model.delta, lookups.e + lookups.first[N], lane);
      if (lane == 0) T.cutoff = it.f.cutoff;
    }
    if (!EVAL && L.nbins) {
      for (int b = lane; b < L.nbins; b += 32) {
        L.bin_sums[(size_t)c * L.nbins + b] = c2(0.0, 0.0);
        L.bin_counts[(size_t)c * L.nbins + b] = 0u;
      }
      __syncwarp();
    }
    __syncwarp();
    for (int g0 = 0; g0 < T.s.count; g0 += 1 << lgp) {
      const int cnt = min(1 << lgp, T.s.count - g0);
      const bool mine = lane < cnt;
      const int N = T.s.order;
      if (g0) stage_item(T.buf, L.items + T.s.item, lane);
      const GroupSetup su = setup_group(L.mode, L.in, it, N, lgp, T.s.first + g0, cnt, keep, T.u + (1 << lgp),
                                        reinterpret_cast<double *>(T.buf), lane);
      const double jac = su.jac;
      const bool dom = su.dom;
      int bin = -1;
      if (!EVAL && L.nbins && mine) bin = earliest_bin(L, T.u + (1 << lgp) + lane, 1 << lgp, N);
      const unsigned dommask = __ballot_sync(FULL, mine && dom);
      if (lane == 0) T.s.ndom += __popc(dommask);
      unsigned guarded = 0;
      if (N > 0) {
        bool in = mine && dom;
        double *ul = T.u + (1 << lgp) + lane;
        if (!su.sorted) sort_times(ul, 1 << lgp, N); // (the plasma warper's times come sorted)
        if (in && !in_window(it, N, ul, 1 << lgp, T.k.rdelta)) {
          atomicOr(L.err, 1);
          in = false;
        }
        if (mine) {
          // a point that is not evaluated still takes its place in a pass: at A's time, inside the window
          const double tA = it.f.A.time;
          if (!in)
            for (int j = 0; j < N; ++j) ul[j << lgp] = tA;
          T.u[lane] = tA;
          T.u[((N + 1) << lgp) + lane] = it.f.B.time;
        }
        const unsigned inmask = __ballot_sync(FULL, in);
        __syncwarp();
        switch (N) {
          case 1: guarded = group_values<SCALE, ANY_CUBIC, 1>(T, N, cnt, inmask, stack, lane); break;
          case 2: guarded = group_values<SCALE, ANY_CUBIC, 2>(T, N, cnt, inmask, stack, lane); break;
          case 3: guarded = group_values<SCALE, ANY_CUBIC, 3>(T, N, cnt, inmask, stack, lane); break;
          case 4: guarded = group_values<SCALE, ANY_CUBIC, 4>(T, N, cnt, inmask, stack, lane); break;
          case 5: guarded = group_values<SCALE, ANY_CUBIC, 5>(T, N, cnt, inmask, stack, lane); break;
          case 6: guarded = group_values<SCALE, ANY_CUBIC, 6>(T, N, cnt, inmask, stack, lane); break;
          case 7: guarded = group_values<SCALE, ANY_CUBIC, 7>(T, N, cnt, inmask, stack, lane); break;
          case 8: guarded = group_values<SCALE, ANY_CUBIC, 8>(T, N, cnt, inmask, stack, lane); break;
          default: guarded = group_values<SCALE, ANY_CUBIC, 0>(T, N, cnt, inmask, stack, lane);
        }
      } else if (mine) { // order 0: g0(A, B)
        const double2 v = dom ? order0(it, L.err) : c2(0.0, 0.0);
        T.fval[lane] = v;
        if (SCALE) T.fscale[lane] = cabs(v);
      }
      __syncwarp();
      double2 fv = mine ? T.fval[lane] : c2(0.0, 0.0);
      if (N & T.k.greater) fv = c2(-fv.x, -fv.y);
      const bool ok = mine && dom;
      const bool fb = ok && (((guarded >> lane) & 1u) || !isfinite(fv.x) || !isfinite(fv.y));
      if (EVAL) {
        if (mine) {
          const long long o = T.s.first + g0 + lane;
          const double2 f = ok ? cut_off(fv, T.cutoff) : c2(0.0, 0.0);
          L.out_val[o] = c2(f.x * jac, f.y * jac);
          if (L.out_jac) L.out_jac[o] = jac;
          if (L.out_dom) L.out_dom[o] = dom ? 1 : 0;
          if (SCALE) L.out_scale[o] = dom ? T.fscale[lane] * fabs(jac) : 0.0;
          if (L.out_flag) L.out_flag[o] = fb ? 1 : 0;
        }
        const unsigned nf = __popc(__ballot_sync(FULL, fb));
        if (nf && lane == 0) atomicAdd(L.n_flagged, (int)nf);
        __syncwarp();
        continue;
      }
      double2 fj = c2(0.0, 0.0);
      if (ok && !fb) {
        const double2 f = cut_off(fv, T.cutoff);
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
          const size_t o = (size_t)T.s.chunk * L.nbins + bin;
          double2 s = L.bin_sums[o];
          for (unsigned r = same; r; r &= r - 1) s = cadd(s, T.fval[__ffs(r) - 1]);
          L.bin_sums[o] = s;
          L.bin_counts[o] += __popc(same);
        }
        const unsigned nd = __popc(__ballot_sync(FULL, mine && bin < 0));
        if (lane == 0) T.s.ndrop += nd;
        __syncwarp();
      }
      const unsigned fbm = __ballot_sync(FULL, fb);
      for (int off = 16; off > 0; off >>= 1) {
        fj.x += __shfl_xor_sync(FULL, fj.x, off);
        fj.y += __shfl_xor_sync(FULL, fj.y, off);
      }
      if (lane == 0) {
        T.s.sum = cadd(T.s.sum, fj);
        T.s.nfb += __popc(fbm);
        // the guarded points' bits of the chunk: g0 is a multiple of 16
        if (g0 < 64) T.s.fb0 |= (unsigned long long)fbm << g0;
        if (g0 > 32 && g0 < 64) T.s.fb1 |= (unsigned long long)fbm >> (64 - g0);
        if (g0 >= 64) T.s.fb1 |= (unsigned long long)fbm << (g0 - 64);
      }
      __syncwarp();
    }
    if (!EVAL && lane == 0) {
      ChunkPartial pr;
      pr.sum_re = T.s.sum.x;
      pr.sum_im = T.s.sum.y;
      pr.n_in_domain = T.s.ndom;
      pr.n_fallback = T.s.nfb;
      pr.fb_mask[0] = T.s.fb0;
      pr.fb_mask[1] = T.s.fb1;
      L.partials[T.s.chunk] = pr;
      if (L.nbins) L.bin_dropped[T.s.chunk] = T.s.ndrop;
    }
  }
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
