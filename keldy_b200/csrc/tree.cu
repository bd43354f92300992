// Wick-determinant integrand kernels (sm_100a).
//
// keldy's integrand (impurity_oneband/wick_direct.cpp:43-158) sums, over the 2^n
// Keldysh configurations a, (-1)^|a| det(s1_a) det(s2_a), where s1_a is the (n+1)^2
// matrix of g0 between the chosen vertex copies and the two external points (corner
// set to 0) and s2_a the n^2 matrix of the opposite spin. Every s1_a/s2_a is a
// principal submatrix of one (2n+1)^2 matrix G (vertex j forward = row 2j, backward =
// row 2j+1, external = row 2n).
//
// Direct kernel: keldy's own algorithm, one partial-pivot LU pair per configuration
// (pivot = first maximum of |re|+|im|, as LAPACK's zgetf2). It serves models whose
// spin-down tables differ from spin-up ones, points whose tree pivots fall below the
// guard, and cross-checks.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdio.h>

#include "kb_device.cuh"
#include "kb_launch.h"
#include "kb_spline.cuh"

namespace kb {

namespace {

constexpr int NT = CTA_THREADS;

__device__ __forceinline__ int find_item(const long long *off, int n_items, long long c) {
  int lo = 0, hi = n_items; // off[lo] <= c < off[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (off[mid] <= c)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The learned spline flow in line: the Sobol point x (stride `st`) to x_j = F_j^{-1}(x_j),
// returning the flow's Jacobian prod_j 1 / F_j'(x_j), formed as the flow's own map kernel
// forms it (same operations, same order).
__device__ __forceinline__ double spline_flow_point(const double *knots, int N, double *x, int st) {
  const SplineKnots *k = reinterpret_cast<const SplineKnots *>(knots);
  double jac = 1.0;
  for (int j = 0; j < N; ++j) {
    double der;
    x[j * st] = spline_inverse(k[j], x[j * st], der);
    jac /= der;
  }
  return jac;
}

// Inputs of point gp (by the calling thread): vertex times into x (stride st), Jacobian and domain
// flag (0: inside). keep: drop points with a negative time (keep_u_hypercube).
__device__ void load_point(const Launch &L, const ItemDev &it, int N, long long gp, double *x, int st, bool keep,
                           double &jac_out, int &flag_out) {
  double jac = 1.0;
  if (L.mode == IN_SOBOL) {
    if (it.flow_x) { // Sobol point already mapped by the learned flow
      for (int j = 0; j < N; ++j) x[j * st] = it.flow_x[gp * N + j];
      jac = it.flow_jac[gp];
    } else {
      uint32_t k = it.k_first + (uint32_t)gp;
      for (int j = 0; j < N; ++j) x[j * st] = sobol_coord(it.rng, k, j);
      if (it.spline_knots) jac = spline_flow_point(it.spline_knots, N, x, st);
      if (it.ar_spline) jac = ar_spline_point(it.ar_spline, N, x, st);
    }
    jac *= chain_reverse(it.chain, it.chain_len, 0, N, x, st);
  } else {
    long long src = L.index ? (long long)L.index[gp] : gp;
    for (int j = 0; j < N; ++j) x[j * st] = L.in[src * N + j];
    if (L.mode == IN_LI) jac = chain_reverse(it.chain, it.chain_start, 0, N, x, st);
  }
  int dom = 1;
  if (it.f.A.spin != it.f.B.spin) dom = 0;
  if (keep)
    for (int j = 0; j < N; ++j)
      if (x[j * st] < 0.0) dom = 0;
  jac_out = jac;
  flag_out = dom ? 0 : 1;
}

// Bin of the earliest vertex time (binner_t::in_bounds and coord2index, binner.hpp:163-176:
// in [xmin, xmax], xmax itself in the last bin); -1: dropped. An index that rounds up to
// nbins just below xmax goes to the last bin.
__device__ __forceinline__ int time_bin(const Launch &L, const double *u, int stride, int N) {
  double t = u[0];
  for (int j = 1; j < N; ++j) t = fmin(t, u[j * stride]);
  if (!(L.bin_xmin <= t && t <= L.bin_xmax)) return -1;
  if (t == L.bin_xmax) return L.nbins - 1;
  return min((int)((t - L.bin_xmin) / L.bin_size), L.nbins - 1);
}

// G (row-major, M = 2N+1) of a point inside the domain.
// Items: the N(N-1) ordered vertex pairs, the N external-row and N external-column entries
// (one table lookup each: g^< and g^> at one time difference), the N diagonal blocks (g(0))
// and the corner. Each thread computes the lookup positions of GK items before issuing
// their loads, so that GK L2 round trips overlap.
template <bool CUBIC, int GK>
__device__ void build_G(const ItemDev &it, int N, const double *u, double2 *G, int spin, int *bad) {
  const ModelDev &m = it.model;
  const int M = 2 * N + 1;
  const int npair = N * (N - 1), nlook = npair + 2 * N, total = nlook + N + 1;
  const kb_gf_index &A = it.f.A, &B = it.f.B;
  const double2 *t00 = m.tab[spin][0][0];
  const double2 *trow = m.tab[spin][A.orbital][0];
  const double2 *tcol = m.tab[spin][0][B.orbital];
  // q / (N - 1) as a multiply-high by 2^32 / (N - 1) rounded up (exact for the quotients here);
  // mn1 wraps to 0 for N - 1 = 1 (q / 1 = q)
  const unsigned mn1 = N > 1 ? 0xFFFFFFFFu / (unsigned)(N - 1) + 1u : 0u;
  auto pair = [&](int q, int &i, int &j) {
    i = mn1 ? (int)__umulhi((unsigned)q, mn1) : q;
    const int r = q - i * (N - 1);
    j = r + (r >= i ? 1 : 0);
  };
  for (int base = threadIdx.x; base < total; base += GK * blockDim.x) {
    int kind[GK], ix[GK];
    double wt[GK], dt[GK];
    const double2 *tb[GK];
#pragma unroll
    for (int k = 0; k < GK; ++k) {
      const int q = base + k * blockDim.x;
      kind[k] = 0; // 0: none, 1: pair, 2: row, 3: col, 4: diagonal, 5: corner
      tb[k] = nullptr;
      ix[k] = 0;
      wt[k] = 0.0;
      dt[k] = 0.0;
      if (q >= total) continue;
      if (q < npair) {
        int i, j;
        pair(q, i, j);
        kind[k] = 1;
        dt[k] = u[i] - u[j];
        tb[k] = t00;
      } else if (q < npair + N) {
        kind[k] = 2;
        dt[k] = A.time - u[q - npair];
        tb[k] = trow;
      } else if (q < nlook) {
        kind[k] = 3;
        dt[k] = u[q - npair - N] - B.time;
        tb[k] = tcol;
      } else if (q < nlook + N) {
        kind[k] = 4;
        tb[k] = t00;
      } else {
        kind[k] = 5;
      }
      if (tb[k] && !interp_index(m, dt[k], ix[k], wt[k])) {
        *bad = 1;
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
      const int q = base + k * blockDim.x;
      if (kind[k] == 1) {
        int i, j;
        pair(q, i, j);
        double2 *g = G + (2 * i) * M + 2 * j;
        const double d = dt[k];
        const bool later = (d != 0.0) ? (d > 0.0) : (i > j);
        g[0] = later ? gg[k] : gl[k];     // forward-forward
        g[M + 1] = later ? gl[k] : gg[k]; // backward-backward
        g[1] = gl[k];                     // forward-backward
        g[M] = gg[k];                     // backward-forward
      } else if (kind[k] == 2) {
        const int j = q - npair;
        double2 *row = G + (2 * N) * M + 2 * j;
        row[0] = compare_3way(A.time, A.k_idx, N, u[j], 0, j) > 0 ? gg[k] : gl[k];
        row[1] = compare_3way(A.time, A.k_idx, N, u[j], 1, j) > 0 ? gg[k] : gl[k];
      } else if (kind[k] == 3) {
        const int j = q - npair - N;
        double2 *col = G + (2 * j) * M + 2 * N;
        col[0] = compare_3way(u[j], 0, j, B.time, B.k_idx, N) > 0 ? gg[k] : gl[k];
        col[M] = compare_3way(u[j], 1, j, B.time, B.k_idx, N) > 0 ? gg[k] : gl[k];
      } else if (kind[k] == 4) {
        const int i = q - nlook;
        double2 *g = G + (2 * i) * M + 2 * i;
        const double2 eq = c2(gl[k].x, gl[k].y - m.alpha); // equal contour points, internal
        g[0] = eq;
        g[M + 1] = eq;
        g[1] = gl[k];
        g[M] = gg[k];
      } else if (kind[k] == 5) {
        G[(2 * N) * M + 2 * N] = c2(0.0, 0.0);
      }
    }
  }
}

// build_G with the model's interpolation.
__device__ void build_G_model(const ItemDev &it, int N, const double *u, double2 *G, int spin, int *bad) {
  if (it.model.interp == 3)
    build_G<true, 2>(it, N, u, G, spin, bad);
  else
    build_G<false, 2>(it, N, u, G, spin, bad);
}

__device__ __forceinline__ double2 apply_cutoff(double2 f, double cutoff) {
  return (cabs(f) < cutoff) ? c2(0.0, 0.0) : f;
}

// Zeroes chunk c's bins (all threads of the CTA; a barrier follows before their use).
__device__ __forceinline__ void clear_bins(const Launch &L, int c) {
  if (!L.nbins) return;
  for (int b = threadIdx.x; b < L.nbins; b += blockDim.x) {
    L.bin_sums[(size_t)c * L.nbins + b] = c2(0.0, 0.0);
    L.bin_counts[(size_t)c * L.nbins + b] = 0u;
  }
  if (threadIdx.x == 0) L.bin_dropped[c] = 0u;
}

// ---------------------------------------------------------------- direct kernel

struct DirectShared {
  double2 G1[(2 * MAX_ORDER + 1) * (2 * MAX_ORDER + 1)];
  double2 G2[(2 * MAX_ORDER + 1) * (2 * MAX_ORDER + 1)];
  double u[MAX_ORDER];
  double jac[1];
  int flag[1];
  double2 red[NT];
  double reds[NT];
};

// det of the n x n row-major matrix a (destroyed): partial pivoting on the first
// maximum of |re|+|im| in the column, multipliers with the pivot's reciprocal.
__device__ double2 lu_det(double2 *a, int n) {
  double2 det = c2(1.0, 0.0);
  bool neg = false;
  for (int k = 0; k < n; ++k) {
    int p = k;
    double best = cabs1(a[k * n + k]);
    for (int i = k + 1; i < n; ++i) {
      double v = cabs1(a[i * n + k]);
      if (v > best) {
        best = v;
        p = i;
      }
    }
    if (best == 0.0) return c2(0.0, 0.0);
    if (p != k) {
      for (int j = 0; j < n; ++j) {
        double2 t = a[k * n + j];
        a[k * n + j] = a[p * n + j];
        a[p * n + j] = t;
      }
      neg = !neg;
    }
    double2 piv = a[k * n + k];
    det = cmul(det, piv);
    double2 inv = crcp(piv);
    for (int i = k + 1; i < n; ++i) {
      double2 l = cmul(a[i * n + k], inv);
      for (int j = k + 1; j < n; ++j) a[i * n + j] = cfms(a[i * n + j], l, a[k * n + j]);
    }
  }
  return neg ? c2(-det.x, -det.y) : det;
}

// The integrand of one point (inputs in D.u / D.flag): keldy's algorithm.
__device__ __forceinline__ void direct_point(DirectShared &D, const ItemDev &it, int N, bool want_scale, double2 &f_out,
                             double &scale_out, int *bad) {
  const int tid = threadIdx.x;
  if (D.flag[0] & 1) {
    f_out = c2(0.0, 0.0);
    scale_out = 0.0;
    return;
  }
  if (N == 0) {
    if (tid == 0) {
      kb_gf_index a = it.f.A, b = it.f.B;
      a.timesplit = 0;
      b.timesplit = 0;
      D.red[0] = g0_contour(it.model, a, b, 0, bad);
      D.reds[0] = cabs(D.red[0]);
    }
    __syncthreads();
    f_out = D.red[0];
    scale_out = D.reds[0];
    __syncthreads();
    return;
  }
  const int M = 2 * N + 1;
  const int spin = it.f.A.spin;
  build_G_model(it, N, D.u, D.G1, spin, bad);
  const double2 *G2 = D.G1;
  if (!it.spin_symmetric) {
    build_G_model(it, N, D.u, D.G2, 1 - spin, bad);
    G2 = D.G2;
  }
  __syncthreads();
  double2 acc = c2(0.0, 0.0);
  double sc = 0.0;
  double2 m1[(MAX_ORDER + 1) * (MAX_ORDER + 1)];
  double2 m2[MAX_ORDER * MAX_ORDER];
  int pick[MAX_ORDER + 1];
  const unsigned nconf = 1u << N;
  for (unsigned cfg = tid; cfg < nconf; cfg += blockDim.x) {
    for (int i = 0; i < N; ++i) pick[i] = 2 * i + ((cfg >> i) & 1u);
    pick[N] = 2 * N;
    for (int i = 0; i <= N; ++i)
      for (int j = 0; j <= N; ++j) m1[i * (N + 1) + j] = D.G1[pick[i] * M + pick[j]];
    m1[N * (N + 1) + N] = c2(0.0, 0.0);
    for (int i = 0; i < N; ++i)
      for (int j = 0; j < N; ++j) m2[i * N + j] = G2[pick[i] * M + pick[j]];
    double2 d = cmul(lu_det(m1, N + 1), lu_det(m2, N));
    if (__popc(cfg) & 1)
      acc = c2(acc.x - d.x, acc.y - d.y);
    else
      acc = cadd(acc, d);
    if (want_scale) sc += cabs(d);
  }
  D.red[tid] = acc;
  D.reds[tid] = sc;
  __syncthreads();
  if (tid == 0) {
    double2 s = c2(0.0, 0.0);
    double ss = 0.0;
    for (int t = 0; t < (int)blockDim.x; ++t) {
      s = cadd(s, D.red[t]);
      ss += D.reds[t];
    }
    D.red[0] = s;
    D.reds[0] = ss;
  }
  __syncthreads();
  f_out = D.red[0];
  scale_out = D.reds[0];
  __syncthreads();
}

// Modes: IN_TIMES / IN_LI (every point, or the points of L.index), IN_SOBOL (per-chunk
// partial sums, as the tree kernel).
__global__ void __launch_bounds__(NT) direct_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DirectShared &D = *reinterpret_cast<DirectShared *>(smem_raw);
  __shared__ int s_chunk;
  __shared__ int s_bad;
  const int tid = threadIdx.x;
  if (tid == 0) s_bad = 0;
  const bool eval = L.mode != IN_SOBOL;
  for (;;) {
    if (tid == 0) s_chunk = atomicAdd(L.chunk_counter, 1);
    __syncthreads();
    const int c = s_chunk;
    if (c >= L.n_chunks) break;
    const int item = find_item(L.chunk_offsets, L.n_items, c);
    const ItemDev &it = L.items[item];
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    const long long total = eval ? (L.index ? (long long)L.n_index : it.n_points) : it.n_points;
    const int ccount = (int)min((long long)it.chunk_points, total - cfirst);
    const int N = it.order;
    const bool keep = eval ? (L.keep_u_hypercube != 0) : true;
    double2 csum = c2(0.0, 0.0);
    unsigned long long cdom = 0;
    if (!eval) {
      clear_bins(L, c);
      __syncthreads();
    }
    for (int p = 0; p < ccount; ++p) {
      long long gp = cfirst + p;
      if (tid == 0) load_point(L, it, N, gp, D.u, 1, keep, D.jac[0], D.flag[0]);
      __syncthreads();
      double2 f;
      double sc;
      direct_point(D, it, N, eval && L.out_scale != nullptr, f, sc, &s_bad);
      if (tid == 0) {
        bool dom = !(D.flag[0] & 1);
        double j = D.jac[0];
        f = dom ? apply_cutoff(f, it.f.cutoff) : c2(0.0, 0.0);
        if (eval) {
          long long o = L.index ? (long long)L.index[gp] : gp;
          L.out_val[o] = c2(f.x * j, f.y * j);
          if (L.out_jac) L.out_jac[o] = j;
          if (L.out_dom) L.out_dom[o] = dom ? 1 : 0;
          if (L.out_scale) L.out_scale[o] = dom ? sc * fabs(j) : 0.0;
          if (L.out_flag) L.out_flag[o] = 0;
        } else {
          csum.x += f.x * j;
          csum.y += f.y * j;
          cdom += dom ? 1 : 0;
          if (L.nbins) {
            const int bin = time_bin(L, D.u, 1, N);
            if (bin < 0) {
              L.bin_dropped[c]++;
            } else {
              L.bin_counts[(size_t)c * L.nbins + bin]++;
              double2 &bs = L.bin_sums[(size_t)c * L.nbins + bin];
              bs = c2(bs.x + f.x * j, bs.y + f.y * j);
            }
          }
        }
      }
      __syncthreads();
    }
    if (!eval && tid == 0) {
      ChunkPartial pr;
      pr.sum_re = csum.x;
      pr.sum_im = csum.y;
      pr.n_in_domain = cdom;
      pr.n_fallback = 0;
      pr.fb_mask[0] = pr.fb_mask[1] = 0;
      L.partials[c] = pr;
    }
  }
  if (tid == 0 && s_bad) atomicOr(L.err, 1);
}

// Of the chunks first + k * step, k = 0 .. NT - 1, the number k of the next one after `after` with
// guarded points (after = -1: look at all of them first); -1: none. All threads of the block.
__device__ __forceinline__ int next_guarded(const Launch &L, long long first, int step, int after, unsigned *found) {
  if (after < 0) {
    const long long c = first + (long long)threadIdx.x * step;
    const unsigned m =
        __ballot_sync(0xffffffffu, threadIdx.x < NT && c < L.n_chunks && L.partials[c].n_fallback != 0);
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && threadIdx.x < NT) found[threadIdx.x >> 5] = m;
    __syncthreads();
  }
  for (int k = after + 1; k < NT; k = (k | 31) + 1) {
    const unsigned m = found[k >> 5] >> (k & 31);
    if (m) return k + __ffs(m) - 1;
  }
  return -1;
}

// Points the tree marked in a chunk's fb_mask, evaluated with keldy's algorithm and
// added to that chunk's partial sum in point order. A cluster of FB_CTAS blocks per chunk: block r
// takes the guarded points r, r + FB_CTAS, ... of the chunk, sets them up at once (a thread per
// point) and leaves their values in block 0's shared memory, which adds them in point order. Where
// every point is guarded (a zero diagonal, alpha = Im g^<(0)) this pass is the call: 4,096
// points of order 6 take 674 us, with a block per chunk and each point set up by itself 1,135, in
// clusters of four blocks 677; 32,768 points 4.1 ms, in clusters of four 5.2.
constexpr int FB_CTAS = 2;
constexpr int FB_MINE = CHUNK_POINTS / FB_CTAS; // a block's points of a chunk, at most
static_assert(NT == CHUNK_POINTS, "a thread per point of a chunk");
// In the place of the other spin's matrix, which these points do not need (more shared memory would
// leave the factorisations' local arrays little L1).
struct GuardedShared {
  double u[MAX_ORDER * FB_MINE], jac[FB_MINE]; // this block's points
  int flag[FB_MINE];
  // block 0: values, Jacobians and bins of the cluster's points; two sets, so that one barrier per
  // chunk keeps the next chunk's values from those still being added
  double2 f[2 * CHUNK_POINTS];
  double j[2 * CHUNK_POINTS];
  int b[2 * CHUNK_POINTS];
};
static_assert(sizeof(GuardedShared) <= sizeof(DirectShared::G2), "the other spin's matrix holds the points");
__global__ void __launch_bounds__(NT, 4) __cluster_dims__(FB_CTAS, 1, 1) fallback_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DirectShared &D = *reinterpret_cast<DirectShared *>(smem_raw);
  __shared__ int s_bad;
  __shared__ unsigned s_found[NT / 32];
  GuardedShared &S = *reinterpret_cast<GuardedShared *>(D.G2);
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = threadIdx.x, rank = (int)cluster.block_rank();
  GuardedShared &S0 = *cluster.map_shared_rank(&S, 0);
  if (tid == 0) s_bad = 0;
  cluster.sync(); // block 0 runs
  // cluster b takes chunks b, b + clusters, ...; it looks at NT of them at once, as guarded points are
  // rare (one by one, 8,192 chunks without any took 14 us)
  const int step = gridDim.x / FB_CTAS;
  int k = -1, set = 0;
  for (long long c0 = blockIdx.x / FB_CTAS; c0 < L.n_chunks;) {
    k = next_guarded(L, c0, step, k, s_found);
    if (k < 0) {
      c0 += (long long)NT * step;
      continue;
    }
    const int c = (int)(c0 + (long long)k * step);
    const int item = find_item(L.chunk_offsets, L.n_items, c);
    const ItemDev &it = L.items[item];
    const int N = it.order;
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    const unsigned long long w0 = L.partials[c].fb_mask[0], w1 = L.partials[c].fb_mask[1], w = tid < 64 ? w0 : w1;
    const int low = __popcll(w0), total = low + __popcll(w1);
    const unsigned long long below = (1ull << (tid & 63)) - 1ull;
    const int q = __popcll(w & below) + (tid >= 64 ? low : 0); // this thread's point among the guarded ones
    __syncthreads();
    if (((w >> (tid & 63)) & 1ull) && q % FB_CTAS == rank) {
      const int p = q / FB_CTAS;
      load_point(L, it, N, cfirst + tid, S.u + p, FB_MINE, true, S.jac[p], S.flag[p]);
    }
    __syncthreads();
    for (int p = 0; p * FB_CTAS + rank < total; ++p) {
      if (tid < N) D.u[tid] = S.u[tid * FB_MINE + p];
      if (tid == 0) D.flag[0] = S.flag[p];
      __syncthreads();
      double2 f;
      double sc;
      direct_point(D, it, N, false, f, sc, &s_bad);
      if (tid == 0) {
        const int o = set * CHUNK_POINTS + p * FB_CTAS + rank;
        S0.f[o] = apply_cutoff(f, it.f.cutoff);
        S0.j[o] = S.jac[p];
        if (L.nbins) S0.b[o] = time_bin(L, D.u, 1, N);
      }
      __syncthreads();
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
      double2 sum = c2(L.partials[c].sum_re, L.partials[c].sum_im);
      for (int o = set * CHUNK_POINTS, e = o + total; o < e; ++o) {
        const double2 f = S.f[o];
        const double j = S.j[o];
        sum = c2(fma(f.x, j, sum.x), fma(f.y, j, sum.y)); // (explicit: with and without bins the same sums)
        if (L.nbins && S.b[o] >= 0) { // counted by the tree kernel; the value is added here
          double2 &bs = L.bin_sums[(size_t)c * L.nbins + S.b[o]];
          bs = c2(fma(f.x, j, bs.x), fma(f.y, j, bs.y));
        }
      }
      L.partials[c].sum_re = sum.x;
      L.partials[c].sum_im = sum.y;
    }
    set ^= 1;
  }
  if (tid == 0 && s_bad) atomicOr(L.err, 1);
}

// acc[item] += sum of the item's chunk partials: each thread adds every RT-th chunk in order, the
// warps' sums go by a fixed xor-shuffle pattern, then warp by warp (deterministic). With
// contiguous runs per thread (uncoalesced, 128 threads) 8,192 partials took 29 us.
constexpr int RT = 512;
__global__ void __launch_bounds__(RT) reduce_kernel(Launch L, kb_accum *acc) {
  __shared__ double s_re[RT / 32], s_im[RT / 32];
  __shared__ unsigned long long s_dom[RT / 32], s_fb[RT / 32];
  const int item = blockIdx.x;
  const long long c0 = L.chunk_offsets[item], c1 = L.chunk_offsets[item + 1];
  double re = 0.0, im = 0.0;
  unsigned long long dom = 0, fb = 0;
  kb_accum a;
  if (threadIdx.x == 0) { // read ahead of the sums
    a = acc[item];
    a.n_points += (uint64_t)L.items[item].n_points;
  }
#pragma unroll 4
  for (long long c = c0 + threadIdx.x; c < c1; c += RT) {
    const ChunkPartial &pr = L.partials[c];
    re += pr.sum_re;
    im += pr.sum_im;
    dom += pr.n_in_domain;
    fb += pr.n_fallback;
  }
  for (int off = 16; off > 0; off >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, off);
    im += __shfl_xor_sync(0xffffffffu, im, off);
    dom += __shfl_xor_sync(0xffffffffu, dom, off);
    fb += __shfl_xor_sync(0xffffffffu, fb, off);
  }
  if ((threadIdx.x & 31) == 0) {
    const int w = threadIdx.x >> 5;
    s_re[w] = re;
    s_im[w] = im;
    s_dom[w] = dom;
    s_fb[w] = fb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int t = 1; t < RT / 32; ++t) {
      re += s_re[t];
      im += s_im[t];
      dom += s_dom[t];
      fb += s_fb[t];
    }
    a.sum_re += re;
    a.sum_im += im;
    a.n_in_domain += dom;
    a.n_fallback += fb;
    acc[item] = a;
  }
}

// ------------------------------------------------------------ kernel method
// keldy's integrand_g_kernel (impurity_oneband/wick_kernel.cpp:42-138) as keldy computes it: with
// the fixed point X in the external slot, for every Keldysh configuration a the matrix s1 (X first,
// then the vertex copies picked by a; keldy zeroes its entry (n, n)) is factored with partial
// pivoting and the first row of its cofactor matrix is found by solving s1 x = det(s1) e_0
// (first_row_expansion, det_expansion.hpp:44-74). Vertex i's term is x_{i+1} (-1)^|a| det(s2_a),
// accumulated at (vertex time, a_i). For points with a guarded pivot in the tree form
// (km_tree.cu) and models whose spins differ.
constexpr int KM_THREADS = 256;
struct KernelShared {
  double2 G1[(2 * KM_MAX_ORDER + 1) * (2 * KM_MAX_ORDER + 1)];
  double2 G2[(2 * KM_MAX_ORDER) * (2 * KM_MAX_ORDER)];
  double u[KM_MAX_ORDER];
  double jac[1];
  int flag[1];
  double2 X[KM_THREADS][KM_MAX_ORDER];
  double2 S[2 * KM_MAX_ORDER];
};

// LU with partial pivoting (first maximum of |re|+|im|) of the m x m matrix a, then the
// solve a x = det(a) e_0 (row interchanges, unit-lower then upper substitution).
__device__ void first_row_cofactors(double2 *a, int m, double2 *x) {
  int piv[KM_MAX_ORDER + 1];
  double2 det = c2(1.0, 0.0);
  bool neg = false;
  for (int k = 0; k < m; ++k) {
    int p = k;
    double best = cabs1(a[k * m + k]);
    for (int i = k + 1; i < m; ++i) {
      const double v = cabs1(a[i * m + k]);
      if (v > best) {
        best = v;
        p = i;
      }
    }
    piv[k] = p;
    if (p != k) {
      for (int j = 0; j < m; ++j) {
        const double2 t = a[k * m + j];
        a[k * m + j] = a[p * m + j];
        a[p * m + j] = t;
      }
      neg = !neg;
    }
    const double2 pv = a[k * m + k];
    det = cmul(det, pv);
    if (best == 0.0) continue;
    const double2 inv = crcp(pv);
    for (int i = k + 1; i < m; ++i) {
      const double2 l = cmul(a[i * m + k], inv);
      a[i * m + k] = l;
      for (int j = k + 1; j < m; ++j) a[i * m + j] = cfms(a[i * m + j], l, a[k * m + j]);
    }
  }
  if (neg) det = c2(-det.x, -det.y);
  for (int i = 0; i < m; ++i) x[i] = c2(0.0, 0.0);
  x[0] = det;
  for (int k = 0; k < m; ++k)
    if (piv[k] != k) {
      const double2 t = x[k];
      x[k] = x[piv[k]];
      x[piv[k]] = t;
    }
  for (int i = 1; i < m; ++i)
    for (int j = 0; j < i; ++j) x[i] = cfms(x[i], a[i * m + j], x[j]);
  for (int i = m - 1; i >= 0; --i) {
    for (int j = i + 1; j < m; ++j) x[i] = cfms(x[i], a[i * m + j], x[j]);
    x[i] = cmul(x[i], crcp(a[i * m + i]));
  }
}

// The 2n sums of one point (inputs in K.u, K.flag): thread t < 2n returns sum (i = t/2, k = t%2).
__device__ double2 kernel_point(KernelShared &K, const ItemDev &it, int N, int *bad) {
  const int tid = threadIdx.x;
  const kb_gf_index X = it.f.A;
  const int spin = X.spin;
  const int M1 = 2 * N + 1, M2 = 2 * N;
  for (int e = tid; e < M1 * M1 + M2 * M2; e += blockDim.x) {
    const bool first = e < M1 * M1;
    const int q = first ? e : e - M1 * M1, M = first ? M1 : M2;
    const int r = q / M, c = q - r * M;
    kb_gf_index a, b;
    const int sp = first ? spin : 1 - spin;
    if (first && r == 2 * N) {
      a = X;
      a.timesplit = N;
    } else {
      a.time = K.u[r % N];
      a.spin = sp;
      a.k_idx = r >= N ? 1 : 0;
      a.timesplit = r % N;
      a.orbital = 0;
    }
    if (first && c == 2 * N) {
      b = X;
      b.timesplit = N;
    } else {
      b.time = K.u[c % N];
      b.spin = sp;
      b.k_idx = c >= N ? 1 : 0;
      b.timesplit = c % N;
      b.orbital = 0;
    }
    const double2 g = g0_contour(it.model, a, b, (first && r == 2 * N && c == 2 * N) ? 0 : 1, bad);
    if (first)
      K.G1[q] = g;
    else
      K.G2[q] = g;
  }
  __syncthreads();
  const unsigned nconf = 1u << N;
  const int ti = tid >> 1, tk = tid & 1;
  double2 acc = c2(0.0, 0.0);
  for (unsigned base = 0; base < nconf; base += blockDim.x) {
    const unsigned cfg = base + tid;
    if (cfg < nconf) {
      double2 m1[(KM_MAX_ORDER + 1) * (KM_MAX_ORDER + 1)], m2[KM_MAX_ORDER * KM_MAX_ORDER];
      double2 x[KM_MAX_ORDER + 1];
      int pick[KM_MAX_ORDER + 1];
      pick[0] = 2 * N;
      for (int i = 0; i < N; ++i) pick[i + 1] = i + (int)((cfg >> i) & 1u) * N;
      for (int r = 0; r <= N; ++r)
        for (int c = 0; c <= N; ++c) m1[r * (N + 1) + c] = K.G1[pick[r] * M1 + pick[c]];
      m1[N * (N + 1) + N] = c2(0.0, 0.0);
      for (int r = 0; r < N; ++r)
        for (int c = 0; c < N; ++c) m2[r * N + c] = K.G2[pick[r + 1] * M2 + pick[c + 1]];
      first_row_cofactors(m1, N + 1, x);
      double2 d2 = lu_det(m2, N);
      if (__popc(cfg) & 1) d2 = c2(-d2.x, -d2.y);
      for (int i = 0; i < N; ++i) K.X[tid][i] = cmul(x[i + 1], d2);
    }
    __syncthreads();
    if (tid < 2 * N) {
      const unsigned cnt = min((unsigned)blockDim.x, nconf - base);
      for (unsigned c = 0; c < cnt; ++c)
        if ((int)(((base + c) >> ti) & 1u) == tk) acc = cadd(acc, K.X[c][ti]);
    }
    __syncthreads();
  }
  return acc;
}

// The points the tree form marked (fb_mask of the chunks' partials), one by one: their 2n sums to
// out_kvals (IN_TIMES), or times their Jacobian to the chunk's bins and sum.
// Two blocks per SM (without the bound on the registers: one), the points set up KM_STAGE at a time:
// 65,536 points of order 2 of a model whose spins differ 4.4 -> 1.6 ms.
constexpr int KM_STAGE = 16;
__global__ void __launch_bounds__(KM_THREADS, 2) km_fallback_kernel(Launch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KernelShared &K = *reinterpret_cast<KernelShared *>(smem_raw);
  __shared__ int s_bad;
  __shared__ unsigned s_found[NT / 32];
  __shared__ double s_u[KM_MAX_ORDER * KM_STAGE], s_jac[KM_STAGE];
  __shared__ int s_flag[KM_STAGE];
  const int tid = threadIdx.x;
  if (tid == 0) s_bad = 0;
  __syncthreads();
  const bool eval = L.mode != IN_SOBOL;
  const bool keep = eval ? (L.keep_u_hypercube != 0) : true;
  const int nb = L.nbins * 2;
  const long long step = gridDim.x;
  int k = -1;
  for (long long c0 = blockIdx.x; c0 < L.n_chunks;) {
    k = next_guarded(L, c0, gridDim.x, k, s_found);
    if (k < 0) {
      c0 += NT * step;
      continue;
    }
    const int c = (int)(c0 + k * step);
    ChunkPartial pr = L.partials[c];
    const int item = find_item(L.chunk_offsets, L.n_items, c);
    const ItemDev &it = L.items[item];
    const int N = it.order, n2 = 2 * N;
    const unsigned half = 1u << (N - 1);
    const long long cfirst = (long long)(c - L.chunk_offsets[item]) * it.chunk_points;
    for (int bit = 0; bit < it.chunk_points; ++bit) {
      const unsigned long long w = pr.fb_mask[bit >> 6] >> (bit & 63);
      if (bit % KM_STAGE == 0) {
        __syncthreads();
        if (tid < KM_STAGE && ((w >> tid) & 1ull))
          load_point(L, it, N, cfirst + bit + tid, s_u + tid, KM_STAGE, keep, s_jac[tid], s_flag[tid]);
      }
      if (!(w & 1ull)) continue;
      __syncthreads();
      const int p = bit % KM_STAGE;
      if (tid < N) K.u[tid] = s_u[tid * KM_STAGE + p];
      if (tid == 0) {
        K.jac[0] = s_jac[p];
        K.flag[0] = s_flag[p];
      }
      __syncthreads();
      const double2 s = kernel_point(K, it, N, &s_bad);
      if (tid < n2) K.S[tid] = s;
      __syncthreads();
      const double j = K.jac[0];
      if (eval) {
        if (tid < n2) L.out_kvals[(cfirst + bit) * n2 + tid] = c2(s.x * j, s.y * j);
      } else if (tid == 0) {
        for (int i = 0; i < N; ++i) {
          if (L.km_fourier) {
            double sn, cs;
            sincos(L.km_omega * K.u[i], &sn, &cs);
            const double2 v = cmul(cadd(K.S[2 * i], K.S[2 * i + 1]), c2(cs, sn));
            pr.sum_re += v.x * j;
            pr.sum_im += v.y * j;
            continue;
          }
          const int bin = time_bin(L, K.u + i, 1, 1);
          if (bin < 0) L.bin_dropped[c] += 2 * half;
          for (int q = 0; q < 2; ++q) {
            const double2 v = c2(K.S[2 * i + q].x * j, K.S[2 * i + q].y * j);
            pr.sum_re += v.x;
            pr.sum_im += v.y;
            if (bin < 0) continue;
            const size_t b = (size_t)c * nb + 2 * bin + q;
            L.bin_sums[b] = cadd(L.bin_sums[b], v);
            L.bin_counts[b] += half;
          }
        }
      }
    }
    __syncthreads();
    if (tid == 0) L.partials[c] = pr;
    __syncthreads();
  }
  if (tid == 0 && s_bad) atomicOr(L.err, 1);
}

// Block (item, y) sums bins 32 y .. 32 y + 31 of an item over its chunks: lane = bin, warp w every
// BW-th chunk in order, then the warps' sums in order (deterministic). (One thread per bin walking
// all chunks took 0.2 ms for 2,048 chunks of 100 bins.)
constexpr int BW = 32;
__global__ void __launch_bounds__(32 * BW) reduce_bins_kernel(Launch L, double2 *sums, unsigned long long *counts,
                                                              unsigned long long *dropped) {
  __shared__ double2 s_sum[BW][32];
  __shared__ unsigned long long s_cnt[BW][32], s_drop[BW];
  const int item = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long c0 = L.chunk_offsets[item], c1 = L.chunk_offsets[item + 1];
  const int nb = L.nbins * max(1, L.bin_cols), b = blockIdx.y * 32 + lane;
  double2 s = c2(0.0, 0.0);
  unsigned long long n = 0, d = 0;
  if (b < nb) {
#pragma unroll 4
    for (long long c = c0 + w; c < c1; c += BW) {
      s = cadd(s, L.bin_sums[(size_t)c * nb + b]);
      n += L.bin_counts[(size_t)c * nb + b];
    }
  }
  if (blockIdx.y == 0) {
    for (long long c = c0 + threadIdx.x; c < c1; c += 32 * BW) d += L.bin_dropped[c];
    for (int off = 16; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
    if (lane == 0) s_drop[w] = d;
  }
  s_sum[w][lane] = s;
  s_cnt[w][lane] = n;
  __syncthreads();
  if (w == 0) {
    for (int k = 1; k < BW; ++k) {
      s = cadd(s, s_sum[k][lane]);
      n += s_cnt[k][lane];
    }
    if (b < nb) {
      sums[(size_t)item * nb + b] = s;
      counts[(size_t)item * nb + b] = n;
    }
    if (blockIdx.y == 0 && lane == 0) {
      for (int k = 1; k < BW; ++k) d += s_drop[k];
      dropped[item] = d;
    }
  }
}

} // namespace

// The launchers rely on configure_kernels() having set the kernels' shared-memory limits
// on the launching device: kb_context_create calls it, with the context's device current,
// for every context (the attribute belongs to each device's context, not to the process).
cudaError_t launch_km_fallback(const Launch &L, int grid, cudaStream_t st) {
  km_fallback_kernel<<<grid, KM_THREADS, (int)sizeof(KernelShared), st>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_reduce_bins(const Launch &L, double2 *sums, unsigned long long *counts,
                               unsigned long long *dropped, cudaStream_t st) {
  if (L.n_items == 0 || L.nbins == 0) return cudaSuccess;
  const int nb = L.nbins * (L.bin_cols > 1 ? L.bin_cols : 1);
  reduce_bins_kernel<<<dim3((unsigned)L.n_items, (unsigned)((nb + 31) / 32)), 32 * BW, 0, st>>>(L, sums, counts, dropped);
  return cudaGetLastError();
}

cudaError_t configure_kernels() {
  cudaError_t e = configure_tree_kernels();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(direct_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DirectShared));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(fallback_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DirectShared));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(km_fallback_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KernelShared));
  if (e == cudaSuccess) e = configure_km_kernel();
  return e;
}

static size_t direct_smem_bytes() { return sizeof(DirectShared); }

cudaError_t launch_direct(const Launch &L, int grid, cudaStream_t st) {
  direct_kernel<<<grid, NT, direct_smem_bytes(), st>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_fallback(const Launch &L, int grid, cudaStream_t st) {
  fallback_kernel<<<(grid + FB_CTAS - 1) / FB_CTAS * FB_CTAS, NT, direct_smem_bytes(), st>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const Launch &L, kb_accum *acc_dev, cudaStream_t st) {
  if (L.n_items == 0) return cudaSuccess;
  reduce_kernel<<<L.n_items, RT, 0, st>>>(L, acc_dev);
  return cudaGetLastError();
}

} // namespace kb
