// What the warp-per-group tree kernels share (wick_tree.cu, km_tree.cu): the set-up of a group of
// points (Sobol coordinates, flows, warper chain, domain), table positions, pivots.
#pragma once
#include "kb_device.cuh"
#include "kb_launch.h"
#include "kb_spline.cuh"

namespace kb {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// An entry in the column of its earlier vertex is g^> on that vertex's forward copy and g^< on the
// backward one, an entry in its row the opposite. A node keeps ONE function S of every entry, the same
// for the whole matrix (`base`), and delta = the other one - S: one copy of a vertex takes delta in its
// column and not in its row (copy 0 of the trees: forward where S is g^<), the other in its row and not
// in its column. The base is the function that is smaller at equal times. The other way round (or with
// one copy as the base of rows and columns alike) S + delta of a nearly empty or full level cancels:
// with |g^<| = 1e-3 |g^>| three digits were lost.
//
// What an entry's value is made of, by its kind: the table, and the functions as a word: the high word
// of delta's sign (+1, -1: delta is g^> - g^< or the opposite; 0: both copies are one function), bit 0:
// S is g^>, bit 1: there is no table. `alt`: for a vertex on the other side of the external time.
struct EntryKind {
  const double2 *tab;
  unsigned w, alt;
};

// What the passes read of their work item, kept in shared memory: with the kernel's shared memory
// most of the L1, a global load is often an L2 round trip.
struct ItemConst {
  EntryKind kind[4];
  double2 eq; // equal contour points
  double xmin, delta, rdelta, floor_;
  const unsigned long long *lookup;
  int last; // first mesh point of the last interval
  int cubic;
  int greater; // the base is g^>: the trees' copy 0 is the backward one, their sums have the sign (-1)^order
};

__device__ __forceinline__ double2 cfma(double2 c, double2 a, double2 b) {
  return c2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
// s + f d, f = 1 (the copy that takes the difference) or 0
__device__ __forceinline__ double2 copyof(double2 s, double2 d, double f) { return c2(fma(d.x, f, s.x), fma(d.y, f, s.y)); }

// 1 / a for a pivot: the squared modulus' reciprocal by one third-order Newton-Raphson (Householder)
// step from the hardware's 20-bit seed, y (1 + e + e^2) with e = 1 - x y: error e^3 < 2^-57 plus
// the last rounding. Three dependent multiply-adds and no special-case branch, where the IEEE
// quotient 1.0 / x takes a longer chain on each level's critical path. A zero, overflowed or
// not finite modulus gives a NaN or an infinity, which the guard catches.
__device__ __forceinline__ double2 pivot_rcp(double2 a) {
  const double x = fma(a.x, a.x, a.y * a.y);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  y = fma(y, fma(e, e, e), y);
  return c2(a.x * y, -a.y * y);
}

// The latency of a small call is a chain of round trips to the L2 (300 to 700 cycles each): what
// follows keeps their number down. 1,000 points of order 2: the kernel took 18,900 cycles, 11,000 of
// them in the item's search, constants and set-up (now 8,600; the kernel 16 -> 13 us between
// events).

// The warps take their first chunk by their place (first warps of all CTAs, then second ones) and
// later ones from the counter, each one chunk ahead of its use. (As plain PTX: atomicAdd's
// compiled form hands the result through a shuffle, which waits for it at once.)
__device__ __forceinline__ int first_chunk() { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }
__device__ __forceinline__ int later_chunk(int *counter, int warps, int lane) {
  int next = 0;
  if (lane == 0) asm volatile("atom.global.add.s32 %0, [%1], 1;" : "=r"(next) : "l"(counter) : "memory");
  return next + (int)gridDim.x * warps;
}

// The item of chunk c (the last with off[item] <= c), by all lanes: a 32nd of the list per round.
__device__ __forceinline__ int find_chunk_item(const long long *off, int n_items, long long c, int lane) {
  int lo = 0, len = n_items; // off[lo] <= c < off[lo + len]
  while (len > 1) {
    const int step = (len + 31) >> 5, p = lane * step;
    const unsigned le = __ballot_sync(FULL, p < len && off[lo + p] <= c);
    const int k = 31 - __clz(le);
    lo += k * step;
    len = min(step, len - k * step);
  }
  return lo;
}

// A copy of an item in a warp's buffers, behind the set-up's factors, for the set-up of a group: the
// some fifty reads of its fields there were L2 round trips (little L1 beside the shared memory, and
// the spilled registers go through it).
constexpr int ITEM_AT = 128; // complex entries: order << lg factors are at most 256 doubles
constexpr int ITEM_END = ITEM_AT + (int)(sizeof(ItemDev) + 15) / 16;
__device__ __forceinline__ const ItemDev &stage_item(double2 *buf, const ItemDev *src, int lane) {
  constexpr int WORDS = (int)sizeof(ItemDev) / 8, R = (WORDS + 31) / 32;
  static_assert(sizeof(ItemDev) % 8 == 0, "whole words");
  unsigned long long w[R];
  unsigned long long *dst = reinterpret_cast<unsigned long long *>(buf + ITEM_AT);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (32 * r + lane < WORDS) w[r] = reinterpret_cast<const unsigned long long *>(src)[32 * r + lane];
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (32 * r + lane < WORDS) dst[32 * r + lane] = w[r];
  __syncwarp();
  return *reinterpret_cast<const ItemDev *>(dst);
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
  for (int j0 = 0; j0 < N; j0 += 4) { // four coordinates' columns in flight
    uint32_t cols[4], sh[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = min(j0 + q, N - 1);
      const uint32_t *C = s.Csr + j * s.m;
      // column b of the matrix; Gray bit m (point 2^m) folds into column 0
      cols[q] = lane < s.m ? __ldg(C + lane) : (lane == s.m ? __ldg(C) : 0u);
      sh[q] = __ldg(s.shfr + j);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (j0 + q >= N) break;
      const uint32_t col = cols[q];
      const uint32_t x0 = __reduce_xor_sync(FULL, ((g0 >> lane) & 1u) ? col : 0u);
      const uint32_t x1 = __reduce_xor_sync(FULL, ((g1 >> lane) & 1u) ? col : 0u);
      uint32_t cur = (k >> 5) == b0 ? x0 : x1;
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        const uint32_t cb = __shfl_sync(FULL, col, b);
        if ((gr >> b) & 1u) cur ^= cb;
      }
      if (lane < (1 << lg)) u[((j0 + q) << lg) + lane] = 2.3283064365386963e-10 * (double)(cur ^ sh[q]);
    }
  }
}

// Points gp0 .. gp0+cnt-1 of an item: vertex times into u (not yet sorted), each lane's own
// point's Jacobian and domain flag. The product warpers, whose logarithms and exponentials
// dominate, run over (coordinate, point) pairs so that small groups fill the warp; a point's
// Jacobian is the product of its factors in coordinate order.
struct GroupSetup {
  double jac;
  bool dom, sorted; // inside the domain; the times latest first
};
__device__ __noinline__ GroupSetup setup_group(int mode, const double *in, const ItemDev &it, int N, int lg, long long gp0,
                                               int cnt, bool keep, double *u, double *fac, int lane) {
  double jac = 1.0;
  int top = 0;
  const bool mine = lane < cnt;
  if (mode == IN_SOBOL) {
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
      if (mine) u[(j << lg) + lane] = in[(gp0 + lane) * N + j];
    if (mode == IN_LI) top = it.chain_start;
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
      } else if (wd.kind == KB_WARPER_EXPONENTIAL) {
        // u = u_max - w log(1 + c0 l), so 1 / f1(u) = c1 exp(u / w) = c1 (1 + c0) / (1 + c0 l) without
        // the exponential (and without the rounding of u in its argument); c0 = exp(u_max / w) - 1
        // overflows from u_max = 710 w on: then u = -infinity, 1 / f1 = 0
        const double a = wd.c[0] * x;
        x = wd.u_max - wd.w * log1p(a);
        f = isinf(wd.c[0]) ? 1.0 / warper_f1(wd, x) : wd.c[1] * ((1.0 + wd.c[0]) / (1.0 + a));
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
  bool dom = it.f.A.spin == it.f.B.spin, sorted = true;
  if (mine && N > 0) { // (order 0 has no coordinates: u holds what an earlier kernel left there)
    double before = u[lane];
    if (keep && before < 0.0) dom = false;
    for (int j = 1; j < N; ++j) {
      const double x = u[(j << lg) + lane];
      if (keep && x < 0.0) dom = false;
      if (!(x <= before)) sorted = false;
      before = x;
    }
  }
  return GroupSetup{jac, dom, sorted};
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

// Sorts a point's times (stride st), latest first (of equal times the higher vertex index counts
// as the later one on the contour, compare_3way's timesplit: their order changes nothing here).
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

// dx / delta correctly rounded, from rdelta = 1 / delta rounded: the product and one residual step
// (Markstein's theorem).
__device__ __forceinline__ double mesh_position(double dx, double delta, double rdelta) {
  const double q = __dmul_rn(dx, rdelta);
  return fma(fma(-q, delta, dx), rdelta, q);
}

// Whether every lookup of a point (sorted times, stride st) lies inside the tabulated window, by
// interp_index's rule: positions whose whole part is 0 .. npts - 1 (2 t_max / delta itself may round
// above npts - 1). The mesh position grows with the time difference, so the extreme differences
// decide.
__device__ __forceinline__ bool in_window(const ItemDev &it, int N, const double *u, int st, double rdelta) {
  const ModelDev &m = it.model;
  const int spin = it.f.A.spin;
  const double hi = u[0], lo = u[(N - 1) * st];
  auto inside = [&](double x) {
    const double a = mesh_position(__dsub_rn(x, m.xmin), m.delta, rdelta);
    return a >= 0.0 && a < (double)m.npts;
  };
  bool ok = true;
  for (int j = 0; j < N; ++j) ok = ok && u[j * st] == u[j * st];
  if (N > 1 && m.tab[spin][0][0]) ok = ok && inside(hi - lo) && inside(lo - hi);
  if (m.tab[spin][it.f.A.orbital][0]) ok = ok && inside(it.f.A.time - lo) && inside(it.f.A.time - hi);
  if (m.tab[spin][0][it.f.B.orbital]) ok = ok && inside(hi - it.f.B.time) && inside(lo - it.f.B.time);
  return ok;
}

// What the lookups of an absent block read.
__device__ __align__(128) const double2 no_table[8] = {};

// An item's constants: a kind of entry per lane, the rest by lane 0.
__device__ __forceinline__ void fill_item(ItemConst &K, const ItemDev &it, double rdelta, const unsigned long long *lookup, int lane) {
  if (lane >= 4) return;
  const ModelDev &m = it.model;
  const int spin = it.f.A.spin;
  double2 gl, gg;
  int b0 = 0;
  g0_pair(m, m.tab[spin][0][0], 0.0, gl, gg, &b0);
  const bool greater = cabs1(gg) < cabs1(gl);
  // A earlier than the vertex: A's branch decides; B likewise; of two vertices the earlier one's index.
  const double2 *tab = m.tab[spin][lane == 2 ? it.f.A.orbital : 0][lane == 3 ? it.f.B.orbital : 0];
  const unsigned w = greater ? 0xBFF00001u : 0x3FF00000u, none = tab ? 0u : 2u;
  const unsigned alt = lane == 2 ? (it.f.A.k_idx ? 1u : 0u) : lane == 3 ? (it.f.B.k_idx ? 0u : 1u) : w;
  K.kind[lane] = EntryKind{tab ? tab : no_table, w | none, alt | none};
  if (lane) return;
  K.eq = c2(gl.x, gl.y - m.alpha);
  K.xmin = m.xmin;
  K.delta = m.delta;
  K.rdelta = rdelta;
  K.floor_ = m.pivot_floor;
  K.lookup = lookup;
  K.last = m.npts - 2;
  K.cubic = m.interp == 3;
  K.greater = greater;
}

// The first `total` entries of a pass's lookup list: S and delta (EntryKind); u: the group's times
// from the pass's first column. Each entry
// is one lookup of g^< and g^> at one time difference; each lane starts GK of them, without a
// branch between them, before it uses the first, so that their L2 round trips overlap. The
// gathers do not allocate in the little L1 that shared memory leaves, which then holds the
// entry list, the item and the Sobol matrices (order 8 -6 %, order 5 -13 %). The position's whole
// part comes from rounding a - 1/2 (at a mesh point either interval gives the mesh value).
template <bool CUBIC, int GK>
__device__ __forceinline__ void build_entries(const ItemConst &K, int total, const double *u, double2 *S, double2 *dl,
                                              int lane) {
  const double xmin = K.xmin, delta = K.delta, rdelta = K.rdelta;
  const int last = K.last;
  const unsigned long long *lt = K.lookup;
  for (int base = 0; base < total; base += 32 * GK) {
    unsigned lo[GK], hi[GK], word[GK];
    double wt[GK];
    const double2 *tb[GK];
#pragma unroll
    for (int k = 0; k < GK; ++k) { // idle lanes repeat the last entry
      const unsigned long long e = __ldg(lt + min(base + 32 * k + lane, total - 1));
      lo[k] = (unsigned)e;
      hi[k] = (unsigned)(e >> 32);
    }
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      const int kind = (hi[k] >> 10) & 3;
      const EntryKind ek = K.kind[kind];
      const double d = __dsub_rn(u[lo[k] & 1023], u[(lo[k] >> 10) & 1023]);
      // the other side: A earlier than the vertex (d < 0), the vertex later than B (d > 0)
      const unsigned dh = (unsigned)__double2hiint(d) ^ ((unsigned)kind << 31);
      word[k] = dh > 0x80000000u ? ek.alt : ek.w;
      const double a = mesh_position(__dsub_rn(d, xmin), delta, rdelta);
      const double t52 = __dadd_rn(a - 0.5, 6755399441055744.0); // 1.5 * 2^52: the sum's low word is the integer
      int ix = (int)min((unsigned)__double2loint(t52), (unsigned)last);
      if (CUBIC) ix = max(0, min(ix - 1, last - 2)); // first of the four mesh points
      wt[k] = a - (__hiloint2double(0x43380000, ix) - 6755399441055744.0);
      tb[k] = ek.tab + 2 * ((word[k] & 2u) ? 0 : ix);
    }
    double2 v[GK][CUBIC ? 8 : 4];
#pragma unroll
    for (int k = 0; k < GK; ++k)
#pragma unroll
      for (int e = 0; e < (CUBIC ? 4 : 2); ++e)
        asm volatile("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(v[k][2 * e].x), "=d"(v[k][2 * e].y), "=d"(v[k][2 * e + 1].x), "=d"(v[k][2 * e + 1].y)
                     : "l"(tb[k] + 2 * e));
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      double2 gl, gg;
      if (CUBIC) { // Lagrange through the four mesh points, as interp_pair_cubic
        const double x = wt[k], am = x - 1.0, bm = x - 2.0, cm = x - 3.0;
        const double n0 = am * bm * cm, n3 = x * am * bm;
        const double w[4] = {-mesh_position(n0, 6.0, 1.0 / 6.0), 0.5 * (x * bm * cm), -0.5 * (x * am * cm),
                             mesh_position(n3, 6.0, 1.0 / 6.0)};
        gl = gg = c2(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const double2 l = v[k][2 * e], g = v[k][2 * e + 1];
          gl = c2(fma(w[e], l.x, gl.x), fma(w[e], l.y, gl.y));
          gg = c2(fma(w[e], g.x, gg.x), fma(w[e], g.y, gg.y));
        }
      } else {
        const double w = wt[k];
        const double2 l0 = v[k][0], g0 = v[k][1], l1 = v[k][2], g1 = v[k][3];
        gl = c2(fma(w, l1.x - l0.x, l0.x), fma(w, l1.y - l0.y, l0.y));
        gg = c2(fma(w, g1.x - g0.x, g0.x), fma(w, g1.y - g0.y, g0.y));
      }
      const double sg = __hiloint2double(word[k] & 0xFFF00000u, 0);
      S[lo[k] >> 20] = (word[k] & 1u) ? gg : gl;
      dl[hi[k] & 1023] = c2(sg * (gg.x - gl.x), sg * (gg.y - gl.y));
    }
  }
}

} // namespace

} // namespace kb
