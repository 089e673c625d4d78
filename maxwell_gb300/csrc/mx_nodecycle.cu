// The node V-cycle on the coarse levels in one launch (vcycle_node2d,
// node2d.c:1352-1389; sweeps node2d.c:629-1138, transfers 1140-1273).
//
// A CTA takes one vector of one k-point through whole V-cycles of the levels
// n0 .. n0 << top with every level's x and b in shared memory; only the top
// level's b and x touch global memory.  On these levels the launches of the
// row kernels were bound by their own latency: four launches of 5 to 12 us per
// sweep for a few microseconds of arithmetic, sixteen sweeps' worth per level
// pair and cycle.
//
// A sweep takes a warp per row.  Along a row x_t = x_{t-1} / 8 + beta_t in
// sweep coordinates (mx_stencil.cu); a lane takes LR consecutive positions,
// sums its own run and receives the carry of the runs before it by a
// shuffle scan with factor 8^-LR, cut where 8^-terms is below the arithmetic's
// rounding.  With beta_t = 3/8 b_t + (x_{t+1} + six neighbours of rows j-1,
// j+1) / 8 the old value across the seam that starts the row and the new one
// that ends it enter like a seventh neighbour.  Rows of a group are
// independent; row 0 only touches row 1 of the odd rows and row n-1 only row
// n-2 of the even ones, so one warp takes each such pair in sequence and a
// sweep is two phases with a barrier each.
//
// Bound by the latency of a phase (shared loads, scan, barrier), FP64 blocks by
// the FP64 rate of the K m SMs it would occupy: few FP64 vectors take a
// cluster of CTAs each, which share the rows and nodes of a phase; every CTA
// keeps a copy of the levels and writes its part to all of them.  One cycle of the levels 64 .. 8,
// 8 k-points x 16 c64 vectors: 66 us against about 460 us in 62 launches; five
// cycles from 64 of 4 x 12 FP64 vectors 1.6 ms against 9.9 ms.
#include <cooperative_groups.h>

#include <type_traits>

#include "mx_common.cuh"
#include "mx_internal.h"

using namespace mx;

namespace {

constexpr int NCT = 512;   // threads: 16 warps

template <typename R> struct Terms { static constexpr int value = 19; };   // 8^-19 < 2^-53
template <> struct Terms<float> { static constexpr int value = 9; };       // 8^-9 < 2^-24

__device__ __forceinline__ float up_r(float v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ double up_r(double v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
__device__ __forceinline__ dd up_r(dd v, int d) { return dd_make(up_r(v.hi, d), up_r(v.lo, d)); }
__device__ __forceinline__ float from0(float v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ double from0(double v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ dd from0(dd v) { return dd_make(from0(v.hi), from0(v.lo)); }
template <typename R> __device__ __forceinline__ cx<R> up_c(cx<R> v, int d) { return mkc(up_r(v.re, d), up_r(v.im, d)); }

// The CTAs of a cluster that share a vector: each holds every level, does a
// part of the rows and nodes and writes its results to all copies
template <bool CLU> struct Team {
  unsigned size, rank;
  __device__ __forceinline__ void sync() const {
    if constexpr (CLU) asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
    else __syncthreads();
  }
  template <typename T> __device__ __forceinline__ void put(T* p, const T& v) const {
    if constexpr (CLU) {
      for (unsigned q = 0; q < size; q++) *cooperative_groups::this_cluster().map_shared_rank(p, q) = v;
    } else {
      *p = v;
    }
  }
};

// one row of one sweep by a warp; EDGE: row 0 or n-1, whose neighbour rows
// cross the seam
template <typename R, int LR, bool EDGE, typename TM>
__device__ void gs_row(int n, int j, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm, const TM& team) {
  const int lane = threadIdx.x & 31, t0 = lane * LR;
  const R eighth = rc<R>(0.125f), c38 = rc<R>(0.375f);
  const cx<R>* Xm = X + (j == 0 ? n - 1 : j - 1) * n;
  const cx<R>* Xp = X + (j == n - 1 ? 0 : j + 1) * n;
  cx<R>* Xc = X + j * n;
  const cx<R>* Bc = B + j * n;
  // factors of the values one position before the first and after the last
  const cx<R> pm = back ? sm.xf : conjc(sm.xf), pp = back ? conjc(sm.xf) : sm.xf;
  auto at = [&](int t) { return back ? n - 1 - t : t; };
  cx<R> w[LR + 2], y[LR];
#pragma unroll
  for (int p = 0; p < LR + 2; p++) {
    const int t = t0 - 1 + p;
    w[p] = czero<R>();
    if (t <= n) {
      const int i = at(t < 0 ? n - 1 : t == n ? 0 : t);
      cx<R> a = Xm[i], c = Xp[i];
      if (EDGE && j == 0) a = conjc(sm.yf) * a;
      if (EDGE && j == n - 1) c = sm.yf * c;
      w[p] = a + c;
      if (t < 0) w[p] = pm * (w[p] + Xc[i]);   // with the row's old value across the seam
    }
  }
#pragma unroll
  for (int q = 0; q < LR; q++) {
    const int t = t0 + q;
    y[q] = czero<R>();
    if (t < n) {
      cx<R> s = w[q] + w[q + 1];
      if (t < n - 1) s += w[q + 2] + Xc[at(t + 1)];
      else s += pp * w[q + 2];
      y[q] = scal(c38, Bc[at(t)]) + scal(eighth, s);
    }
  }
  // the row's first new value, which its last position sees across the seam
  const cx<R> x0 = mkc(from0(y[0].re), from0(y[0].im));
  if (t0 < n && t0 + LR >= n) {
    const cx<R> z = scal(eighth, pp * x0);
#pragma unroll
    for (int q = 0; q < LR; q++)
      if (t0 + q == n - 1) y[q] += z;
  }
#pragma unroll
  for (int q = 1; q < LR; q++) y[q] += scal(eighth, y[q - 1]);
  // inclusive scan of the runs' ends
  cx<R> s = y[LR - 1];
  R f = eighth;
#pragma unroll
  for (int q = 1; q < LR; q++) f = f * eighth;
#pragma unroll
  for (int off = 1; off * LR < Terms<R>::value; off *= 2) {
    const cx<R> u = up_c(s, off);
    if (lane >= off) s += scal(f, u);
    f = f * f;
  }
  cx<R> carry = up_c(s, 1);
  if (lane == 0) carry = czero<R>();
#pragma unroll
  for (int q = 0; q < LR; q++) {
    carry = scal(eighth, carry);
    if (t0 + q < n) team.put(Xc + at(t0 + q), y[q] + carry);
  }
}

// one sweep by the CTA; ends at a barrier
template <typename R, int LR, typename TM>
__device__ void sweep(int n, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm, const TM& team) {
  const int warp = (threadIdx.x >> 5) * team.size + team.rank, nw = NCT / 32 * team.size;
#pragma unroll 1
  for (int ph = 0; ph < 2; ph++) {
    // forward: row 0 and the odd rows, then the even rows and row n-1;
    // backward the reverse
    const bool odd = (ph == 0) != (back != 0);
    if (warp == 0) {
      const int edge = odd ? 0 : n - 1, next = odd ? 1 : n - 2;
      if (ph == 0) {
        gs_row<R, LR, true>(n, edge, back, X, B, sm, team);
        __syncwarp();
        gs_row<R, LR, false>(n, next, back, X, B, sm, team);
      } else {
        gs_row<R, LR, false>(n, next, back, X, B, sm, team);
        __syncwarp();
        gs_row<R, LR, true>(n, edge, back, X, B, sm, team);
      }
    } else {
      // the group's other rows: 3, 5 .. n-3 or 2, 4 .. n-4
      for (int r = warp - 1; r < n / 2 - 2; r += nw - 1) gs_row<R, LR, false>(n, (odd ? 3 : 2) + 2 * r, back, X, B, sm, team);
    }
    team.sync();
  }
}

template <typename R, typename TM>
__device__ void smooth(int n, int nu, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm, const TM& team) {
  for (int q = 0; q < nu; q++) {
    if (n <= 32) sweep<R, 1>(n, back, X, B, sm, team);
    else if (n <= 64) sweep<R, 2>(n, back, X, B, sm, team);
    else sweep<R, 3>(n, back, X, B, sm, team);
  }
}

// bc = restriction of b - L x, xc = 0
template <typename R, typename TM>
__device__ void restrict_residual(int n, const cx<R>* X, const cx<R>* B, cx<R>* Xc, cx<R>* Bc, const Seam<R>& sm,
                                  const Sc& third_s, const TM& team) {
  const int nc = n / 2;
  const R third = sget<R>(third_s), half = rc<R>(0.5f), nine = rc<R>(9.0f);
  for (int e = threadIdx.x + team.rank * NCT; e < nc * nc; e += NCT * team.size) {
    const int I = e % nc, J = e / nc, fi = 2 * I, fj = 2 * J;
    cx<R> out;
    auto body = [&](const auto& V, const auto& W) {
      // rows fj-2 .. fj+2: sums h of three neighbours at columns fi-1 .. fi+1
      cx<R> h[3][3], mid[3], acc[3];
#pragma unroll
      for (int q = 0; q < 5; q++) {
        const int j = fj - 2 + q;
        const cx<R> a = V(fi - 2, j), b = V(fi - 1, j), c = V(fi, j), d = V(fi + 1, j), g = V(fi + 2, j);
        const cx<R> bc = b + c, cd = c + d;
        cx<R>* hq = h[q % 3];
        hq[0] = a + bc; hq[1] = bc + d; hq[2] = cd + g;
        if (q >= 2) {
          // d = b - L x on row j - 1, L x = (9 x - the sum of nine) / 3 (with
          // 3 x and a third of the sum apart, the rounded third would shift
          // a smooth x by its own relative error)
#pragma unroll
          for (int p = 0; p < 3; p++) {
            const cx<R> s9 = h[0][p] + h[1][p] + h[2][p];
            const cx<R> r = W(fi - 1 + p, j - 1) + scal(third, s9 - scal(nine, mid[p]));
            if (q == 2) acc[p] = scal(half, r);
            else if (q == 3) acc[p] += r;
            else acc[p] += scal(half, r);
          }
        }
        mid[0] = b; mid[1] = c; mid[2] = d;
      }
      out = acc[1] + scal(half, acc[0] + acc[2]);
    };
    if (I > 0 && J > 0 && I < nc - 1 && J < nc - 1) {
      body([&](int i, int j) { return X[j * n + i]; }, [&](int i, int j) { return B[j * n + i]; });
    } else {
      auto wrapped = [&](const cx<R>* P) {
        return [&, P](int i, int j) {
          cx<R> p;
          const bool w = sm.wrap(i, j, p);
          const cx<R> v = P[j * n + i];
          return w ? p * v : v;
        };
      };
      body(wrapped(X), wrapped(B));
    }
    team.put(Bc + e, out);
    team.put(Xc + e, czero<R>());
  }
  team.sync();
}

// x += P xc, bilinear
template <typename R, typename TM>
__device__ void prolong(int n, cx<R>* X, const cx<R>* Xc, const Seam<R>& sm, const TM& team) {
  const int nc = n / 2;
  const R half = rc<R>(0.5f);
  for (int e = threadIdx.x + team.rank * NCT; e < nc * nc; e += NCT * team.size) {
    const int I = e % nc, J = e / nc;
    const bool wi = I == nc - 1, wj = J == nc - 1;
    const int I1 = wi ? 0 : I + 1, J1 = wj ? 0 : J + 1;
    cx<R> c00 = Xc[e], c10 = Xc[J * nc + I1], c01 = Xc[J1 * nc + I], c11 = Xc[J1 * nc + I1];
    if (wi) { c10 = sm.xf * c10; c11 = sm.xf * c11; }
    if (wj) { c01 = sm.yf * c01; c11 = sm.yf * c11; }
    cx<R>* p0 = X + 2 * J * n + 2 * I;
    cx<R>* p1 = p0 + n;
    const cx<R> h0 = scal(half, c00 + c10), h1 = scal(half, c01 + c11);
    team.put(p0, p0[0] + c00);
    team.put(p0 + 1, p0[1] + h0);
    team.put(p1, p1[0] + scal(half, c00 + c01));
    team.put(p1 + 1, p1[1] + scal(half, h0 + h1));
  }
  team.sync();
}

// x = Ainv b on the coarsest level: N rows, the columns split over NCT / N
// groups of threads; part: NCT values of shared memory
template <typename R, typename MS>
__device__ void coarse_solve(int N, const MS* __restrict__ ainv, cx<R>* X, const cx<R>* B, cx<R>* part) {
  const int groups = NCT / N, r = threadIdx.x % N, g = threadIdx.x / N;
  if (g < groups) {
    cx<R> acc = czero<R>();
    for (int c = g; c < N; c += groups) acc += Store<MS, R>::ld(ainv + (size_t) c * N + r) * B[c];
    part[g * N + r] = acc;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < N; q += NCT) {
    cx<R> acc = part[q];
    for (int h = 1; h < groups; h++) acc += part[h * N + q];
    X[q] = acc;
  }
  __syncthreads();
}

template <typename S, typename R, typename MS, bool CLU>
__global__ void __launch_bounds__(NCT) k_node_vcycle(int n0, int top, int m, int K, int nu, int cycles, int zero,
                                                   int planar, const double* __restrict__ ph, Sc third,
                                                   const MS* __restrict__ ainv, const S* __restrict__ b, S* x) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const unsigned cl = CLU ? gridDim.x / (unsigned) (K * m) : 1u;
  const Team<CLU> team{cl, CLU ? blockIdx.x % cl : 0u};
  const int kv = blockIdx.x / team.size, v = kv % m, k = kv / m, n = n0 << top, nn = n * n;
  // level l: x, then b; the top level first
  cx<R>* part = reinterpret_cast<cx<R>*>(sm_raw);
  cx<R>* X = part + NCT;
  auto level = [&](int l) {
    cx<R>* p = X;
    for (int q = top; q > l; q--) p += 2 * (n0 << q) * (n0 << q);
    return p;
  };
  const Seam<R> sm0 = seam_load<R>(ph, K, k, n);
  // element e of vector v: [k][e][v], or [k][v][e] where planar
  const size_t at0 = (size_t) k * nn * m + (planar ? (size_t) v * nn : (size_t) v), es = planar ? 1 : m;
  const S* bk = b + at0;
  S* xk = x + at0;
  for (int e = threadIdx.x; e < nn; e += NCT) {
    X[nn + e] = Store<S, R>::ld(bk + e * es);
    X[e] = zero ? czero<R>() : Store<S, R>::ld(xk + e * es);
  }
  team.sync();
  for (int c = 0; c < cycles; c++) {
#pragma unroll 1
    for (int l = top; l > 0; l--) {
      const int nl = n0 << l;
      cx<R>*Xl = level(l), *Xc = level(l - 1);
      Seam<R> sm = sm0;
      sm.n = nl;
      smooth<R>(nl, nu, 0, Xl, Xl + nl * nl, sm, team);
      restrict_residual<R>(nl, Xl, Xl + nl * nl, Xc, Xc + nl * nl / 4, sm, third, team);
    }
    {
      cx<R>* X0 = level(0);
      coarse_solve<R, MS>(n0 * n0, ainv + (size_t) k * n0 * n0 * n0 * n0, X0, X0 + n0 * n0, part);
    }
#pragma unroll 1
    for (int l = 1; l <= top; l++) {
      const int nl = n0 << l;
      cx<R>* Xl = level(l);
      Seam<R> sm = sm0;
      sm.n = nl;
      prolong<R>(nl, Xl, level(l - 1), sm, team);
      smooth<R>(nl, nu, 1, Xl, Xl + nl * nl, sm, team);
    }
  }
  for (int e = threadIdx.x + team.rank * NCT; e < nn; e += NCT * team.size) Store<S, R>::st(xk + e * es, X[e]);
}

// ------------------------------------------------------------------
// The fine levels: all that a V-cycle does with a level on one side of the
// coarse correction in one pass over memory, for c64 vectors stored one after
// the other ([k][v][j][i], planar).
//   PRE   x' = nu forward sweeps on x (or zero) and b, and the restriction of
//         b - L x' (node2d.c:1352-1389's first half of a level)
//   POST  x' = nu backward sweeps on x + P xc and b
// A CTA takes a band of B rows of one vector, with the rows around it that
// the band's final values depend on: a phase (half a sweep) uses up one row on
// each side, the residual and its restriction one and two more.  Row 0 is
// swept before the odd rows and row n-1 after the even ones, which lets a
// dependence run two rows in one phase across the seam; bands start at row 0
// or 8 and more, and end at row n or n - 8 and less, where the same halo
// holds.  The result goes to another vector, since neighbour bands read the
// old one.  Rows beyond the seam are loaded with their phase, so only the
// columns wrap.  x sits in shared memory (two CTAs per SM), b comes through L2
// for every sweep.  A warp sweeps a row in segments of 128 columns, four per
// lane: run of four, shuffle scan of the runs with factor 8^-4, carry from the
// segment before.
//
// Traffic per side: x and b read with B + 11 (PRE) or B + 8 rows for B, x
// written once, against 2 nu + .. passes of the separate kernels (a sweep 4
// arrays, residual and restriction 2.25).  Bound by the barriers of the
// phases and by issue (54 % of issue slots in PRE, 49 % in POST; 0.85 and 0.84
// GB of DRAM traffic at 512^2).  8 k-points x 16 vectors, nu = 2: PRE 0.456 ms
// at 512^2 (0.411 from zero) against 0.69 for two sweeps and residual with
// restriction, 0.117 from zero against 0.25 at 256^2; POST 0.357 against 0.56
// for prolongation and two sweeps.
// ------------------------------------------------------------------
constexpr int NBT = 512;

__device__ __forceinline__ cx<float> dn_c(cx<float> v, int d) {
  return mkc(__shfl_down_sync(0xffffffffu, v.re, d), __shfl_down_sync(0xffffffffu, v.im, d));
}
__device__ __forceinline__ cx<float> at_c(cx<float> v, int src) {
  return mkc(__shfl_sync(0xffffffffu, v.re, src), __shfl_sync(0xffffffffu, v.im, src));
}
struct Two {
  cx<float> a, b;   // columns c, c + 1
};
__device__ __forceinline__ Two ld2(const float2* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return Two{mkc(v.x, v.y), mkc(v.z, v.w)};
}
__device__ __forceinline__ void st2(float2* p, Two t) {
  *reinterpret_cast<float4*>(p) = make_float4(t.a.re, t.a.im, t.b.re, t.b.im);
}
__device__ __forceinline__ cx<float> ld1(const float2* p) { return mkc(p->x, p->y); }

// A row in shared memory: segments of 128 columns, the column pairs 4l, 4l+1
// of the lanes first, then the pairs 4l+2, 4l+3, so that a lane's four columns
// are two conflict-free 16-byte accesses.
__device__ __forceinline__ int pcol(int c) { return (c & ~127) + ((c & 2) << 5) + ((c & 124) >> 1) + (c & 1); }
struct Four {
  cx<float> v[4];
};
__device__ __forceinline__ Four ld4(const float2* p, int second) {
  const Two a = ld2(p), b = ld2(p + second);
  return Four{{a.a, a.b, b.a, b.b}};
}
__device__ __forceinline__ void st4(float2* p, int second, const Four& t) {
  st2(p, Two{t.v[0], t.v[1]});
  st2(p + second, Two{t.v[2], t.v[3]});
}
__device__ __forceinline__ cx<float> pick(bool c, cx<float> a, cx<float> b) { return mkc(c ? a.re : b.re, c ? a.im : b.im); }
// 8^-4d, the carry's weight in lane d of a segment (below FP32's rounding past 3)
__device__ __forceinline__ float pow84(int d) { return d < 4 ? __int_as_float((127 - 12 * d) << 23) : 0.0f; }

// one row of one sweep by a warp; Xm, Xc, Xp: rows j-1, j, j+1 in shared
// memory, bp: the phase of b's row where phased
template <bool BACK>
__device__ __forceinline__ void band_row(int n, const float2* Xm, float2* Xc, const float2* Xp,
                                         const float2* __restrict__ B, bool phased, cx<float> bp, cx<float> xf) {
  const int lane = threadIdx.x & 31, nseg = (n + 127) / 128, pl = pcol(n - 1);
  const cx<float> xfc = conjc(xf);
  // the sums of rows j-1 and j+1 in the columns across the seam, and the
  // row's old value there that starts the recurrence
  const cx<float> wl = xfc * (ld1(Xm + pl) + ld1(Xp + pl)), wr = xf * (ld1(Xm) + ld1(Xp));
  const cx<float> old = BACK ? xf * ld1(Xc) : xfc * ld1(Xc + pl);
  cx<float> carry = czero<float>(), first = czero<float>();
#pragma unroll 1
  for (int q = 0; q < nseg; q++) {
    const int sg = BACK ? nseg - 1 - q : q, c = 128 * sg + 4 * lane, at = 128 * sg + 2 * lane;
    const bool in = c < n, end = c + 4 == n;
    Four bb = ld4(B + (in ? c : 0), 2);
    const Four m4 = ld4(Xm + at, 64), p4 = ld4(Xp + at, 64), o4 = ld4(Xc + at, 64);
    // the columns next to the segment (any column where there is none)
    const int cl = sg > 0 ? pcol(128 * sg - 1) : 0, cr = sg + 1 < nseg ? 128 * (sg + 1) : 0;
    const cx<float> el = sg > 0 ? ld1(Xm + cl) + ld1(Xp + cl) : wl, er = ld1(Xm + cr) + ld1(Xp + cr);
    cx<float> w[4], y[4];
#pragma unroll
    for (int t = 0; t < 4; t++) w[t] = m4.v[t] + p4.v[t];
    const cx<float> lft = pick(lane == 0, el, up_c(w[3], 1));
    const cx<float> rgt = pick(end, wr, pick(lane == 31, er, dn_c(w[0], 1)));
    const cx<float> s01 = w[0] + w[1], s12 = w[1] + w[2], s23 = w[2] + w[3];
    y[0] = lft + s01;
    y[1] = s01 + w[2];
    y[2] = s12 + w[3];
    y[3] = s23 + rgt;
    // the old value of the next position (at the row's end the new first one,
    // added below), the old value across the seam at the first
    if (!BACK) {
      const cx<float> nx = pick(lane == 31, ld1(Xc + cr), dn_c(o4.v[0], 1));
      y[0] += o4.v[1];
      y[1] += o4.v[2];
      y[2] += o4.v[3];
      if (!end) y[3] += nx;
      if (c == 0) y[0] += old;
    } else {
      const cx<float> nx = pick(lane == 0, ld1(Xc + cl), up_c(o4.v[3], 1));
      y[3] += o4.v[2];
      y[2] += o4.v[1];
      y[1] += o4.v[0];
      if (c > 0) y[0] += nx;
      if (end) y[3] += old;
    }
    if (phased) {
#pragma unroll
      for (int t = 0; t < 4; t++) bb.v[t] = bp * bb.v[t];
    }
#pragma unroll
    for (int t = 0; t < 4; t++) y[t] = scal(0.375f, bb.v[t]) + scal(0.125f, y[t]);
    if (!in) y[0] = y[1] = y[2] = y[3] = czero<float>();
    // the first new value of the row and its way round to the last position
    if (q == 0) first = BACK ? xfc * at_c(y[3], ((n - 4) & 127) / 4) : xf * at_c(y[0], 0);
    if (BACK ? c == 0 : end) y[BACK ? 0 : 3] += scal(0.125f, first);
    cx<float> s;
    if (!BACK) {
#pragma unroll
      for (int t = 1; t < 4; t++) y[t] += scal(0.125f, y[t - 1]);
      s = y[3];
    } else {
#pragma unroll
      for (int t = 2; t >= 0; t--) y[t] += scal(0.125f, y[t + 1]);
      s = y[0];
    }
    // scan of the runs: 16 positions back
    float f = 1.0f / 4096.0f;
#pragma unroll
    for (int off = 1; off < 4; off *= 2) {
      const cx<float> u = BACK ? dn_c(s, off) : up_c(s, off);
      const float g = (BACK ? lane + off < 32 : lane >= off) ? f : 0.0f;
      s += scal(g, u);
      f *= f;
    }
    // the value before the lane's run: the neighbour lane's, and what the end
    // of the segment before contributes
    const int dl = BACK ? 31 - lane : lane;
    const cx<float> prev = BACK ? dn_c(s, 1) : up_c(s, 1);
    const cx<float> cin = scal(dl == 0 ? 0.0f : 1.0f, prev) + scal(pow84(dl), carry);
    carry = at_c(s, BACK ? 0 : 31);
#pragma unroll
    for (int t = 0; t < 4; t++) {
      constexpr float w8[4] = {0.125f, 0.015625f, 0.001953125f, 0.000244140625f};
      y[t] += scal(w8[BACK ? 3 - t : t], cin);
    }
    __syncwarp();
    if (in) st4(Xc + at, 64, Four{{y[0], y[1], y[2], y[3]}});
    __syncwarp();
  }
}

template <bool POST>
__global__ void __launch_bounds__(NBT, 2)
    k_node_band(int n, int m, int K, int B, int nu, const double* __restrict__ ph, float third,
                const float2* __restrict__ b, const float2* __restrict__ xin, const float2* __restrict__ xc,
                float2* __restrict__ xout, float2* __restrict__ bc) {
  extern __shared__ __align__(16) float2 sx[];
  const int nb = (n + B - 1) / B, kv = blockIdx.x / nb, k = kv / m, nn = n * n, nc = n / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = NBT / 32, nseg = (n + 127) / 128, NS = nseg * 128;
  const int J0 = (int) (blockIdx.x - kv * nb) * B, J1 = J0 + B < n ? J0 + B : n;
  // rows lo .. hi in shared memory (beyond 0 .. n-1 across the seam)
  const int lo = J0 - 2 * nu - (POST ? 0 : 2), hi = J1 - 1 + 2 * nu + (POST ? 0 : 1);
  const Seam<float> sm = seam_load<float>(ph, K, k, n);
  const float2* bv = b + (size_t) kv * nn;
  auto row_at = [&](int r) { return r < 0 ? r + n : r >= n ? r - n : r; };
  auto X = [&](int r) { return sx + (r - lo) * NS; };
  // ---- load (and prolongate into) the rows
  for (int r = lo + warp; r <= hi; r += nw) {
    const int j = row_at(r);
    const bool out = j != r;
    const cx<float> rp = r < 0 ? conjc(sm.yf) : sm.yf;
    const float2* src = xin ? xin + (size_t) kv * nn + (size_t) j * n : nullptr;
    const float2 *c0 = nullptr, *c1 = nullptr;
    cx<float> p0 = mkc(1.0f, 0.0f), p1 = p0;
    if (POST) {
      // coarse rows J and J + 1 with the phases of rows outside the cell
      const int J = r >= 0 ? r / 2 : -((1 - r) / 2), J2 = J + 1;
      const float2* cv = xc + (size_t) kv * nc * nc;
      c0 = cv + (size_t) (J < 0 ? J + nc : J >= nc ? J - nc : J) * nc;
      c1 = cv + (size_t) (J2 < 0 ? J2 + nc : J2 >= nc ? J2 - nc : J2) * nc;
      if (J < 0) p0 = conjc(sm.yf);
      if (J >= nc) p0 = sm.yf;
      if (J2 < 0) p1 = conjc(sm.yf);
      if (J2 >= nc) p1 = sm.yf;
    }
    for (int c = 4 * lane, at = 2 * lane; c < n; c += 128, at += 128) {
      Four t{{czero<float>(), czero<float>(), czero<float>(), czero<float>()}};
      if (src) {
        t = ld4(src + c, 2);
        if (out)
#pragma unroll
          for (int q = 0; q < 4; q++) t.v[q] = rp * t.v[q];
      }
      if (POST) {
        // coarse columns I, I + 1, I + 2
        const int I = c / 2, I2 = I + 2 < nc ? I + 2 : 0;
        const Two a0 = ld2(c0 + I);
        cx<float> v0 = p0 * a0.a, v1 = p0 * a0.b, v2 = p0 * ld1(c0 + I2);
        if (r & 1) {
          const Two a1 = ld2(c1 + I);
          v0 = scal(0.5f, v0 + p1 * a1.a);
          v1 = scal(0.5f, v1 + p1 * a1.b);
          v2 = scal(0.5f, v2 + p1 * ld1(c1 + I2));
        }
        if (I2 == 0) v2 = sm.xf * v2;
        t.v[0] += v0;
        t.v[1] += scal(0.5f, v0 + v1);
        t.v[2] += v1;
        t.v[3] += scal(0.5f, v1 + v2);
      }
      st4(X(r) + at, 64, t);
    }
  }
  __syncthreads();
  // ---- the sweeps
  auto sweep_row = [&](int r) {
    const int j = row_at(r);
    band_row<POST>(n, X(r - 1), X(r), X(r + 1), bv + (size_t) j * n, j != r, r < 0 ? conjc(sm.yf) : sm.yf, sm.xf);
  };
#pragma unroll 1
  for (int p = 1; p <= 2 * nu; p++) {
    // forward: odd rows with row 0, then even rows with row n-1; backward the
    // reverse.  A row next to a special one takes it along, in the sweep's order.
    const bool odd = POST ? (p & 1) == 0 : (p & 1) == 1;
    const bool before = POST ? !odd : odd;   // the special row comes before its neighbour
    const int a = lo + p, e = hi - p, f0 = a + (((a & 1) != 0) != odd);
#pragma unroll 1
    for (int r = f0 + 2 * warp; r <= e; r += 2 * nw) {
      const int j = row_at(r);
      if (j == (odd ? n - 1 : 0)) continue;   // (the other phase's)
      const bool next = j == (odd ? 1 : n - 2);
      const int sp = odd ? r - 1 : r + 1;
      const bool chain = next && sp >= a && sp <= e;
      // up to two rows in turn, through one copy of the sweep's code
#pragma unroll 1
      for (int q = 0; q < 1 + (int) chain; q++) {
        sweep_row(chain && (q == 0) == before ? sp : r);
        __syncwarp();
      }
    }
    // a special row that comes first, with its neighbour outside the range
    if (before && warp == nw - 1)
#pragma unroll 1
      for (int q = 0; q < 2; q++) {
        const int sp = odd ? q * n : q * n - 1, nbr = odd ? sp + 1 : sp - 1;
        if (sp >= a && sp <= e && !(nbr >= a && nbr <= e)) sweep_row(sp);
      }
    __syncthreads();
  }
  // ---- results
  float2* xo = xout + (size_t) kv * nn;
  for (int r = J0 + warp; r < J1; r += nw)
    for (int c = 4 * lane, at = 2 * lane; c < n; c += 128, at += 128) st4(xo + (size_t) r * n + c, 2, ld4(X(r) + at, 64));
  if (!POST) {
    // coarse rows J0/2 .. J1/2 - 1, the row in one or two parts.  t(c) =
    // d(c, fj) + (d(c, fj-1) + d(c, fj+1)) / 2 with d = b - (9 x - the sum of
    // nine) / 3; the coarse value is t(2I) + (t(2I-1) + t(2I+1)) / 2.  With h
    // the sums of three columns, the x part of 3 t is row by row
    // h/2, 3/2 (h - 3x), 2h - 9x, 3/2 (h - 3x), h/2: its partial sums stay small.
    const int C0 = J0 / 2, parts = nseg > 1 ? 2 : 1, per = (nseg + parts - 1) / parts;
    for (int tsk = warp; tsk < parts * (J1 - J0) / 2; tsk += nw) {
      const int J = C0 + tsk / parts, sa = (tsk % parts) * per, sb = sa + per < nseg ? sa + per : nseg, fj = 2 * J;
      constexpr float wh[5] = {0.5f, 1.5f, 2.0f, 1.5f, 0.5f}, wx[5] = {0.0f, 4.5f, 9.0f, 4.5f, 0.0f};
      auto bphase = [&](int r) { return r < 0 ? conjc(sm.yf) : sm.yf; };
      // t in the column before the part
      cx<float> left = czero<float>();
      {
        const int c = sa > 0 ? 128 * sa - 1 : n - 1, pc = pcol(c), pm = pcol(c - 1), pp = c + 1 < n ? pcol(c + 1) : 0;
        cx<float> acc = czero<float>();
#pragma unroll
        for (int q = 0; q < 5; q++) {
          const int r = fj - 2 + q;
          cx<float> g = ld1(X(r) + pp);
          if (c + 1 == n) g = sm.xf * g;
          const cx<float> x0 = ld1(X(r) + pc), h = ld1(X(r) + pm) + x0 + g;
          acc += scal(wh[q], h) - scal(wx[q], x0);
          if (q > 0 && q < 4) {
            const int j = row_at(r);
            cx<float> d = ld1(bv + (size_t) j * n + c);
            if (j != r) d = bphase(r) * d;
            left += scal(q == 2 ? 1.0f : 0.5f, d);
          }
        }
        left += scal(third, acc);
        if (sa == 0) left = conjc(sm.xf) * left;
      }
#pragma unroll 1
      for (int sg = sa; sg < sb; sg++) {
        const int c = 128 * sg + 4 * lane, at = 128 * sg + 2 * lane;
        const int cl = sg > 0 ? pcol(128 * sg - 1) : pcol(n - 1), cr = sg + 1 < nseg ? 128 * (sg + 1) : 0;
        const bool in = c < n, end = c + 4 == n;
        Four acc{{czero<float>(), czero<float>(), czero<float>(), czero<float>()}}, t4 = acc;
#pragma unroll
        for (int q = 0; q < 5; q++) {
          const int r = fj - 2 + q;
          const float2* Xr = X(r);
          const Four x4 = ld4(Xr + at, 64);
          cx<float> el = ld1(Xr + cl), er = ld1(Xr + cr);
          if (sg == 0) el = conjc(sm.xf) * el;
          const cx<float> l = pick(lane == 0, el, up_c(x4.v[3], 1));
          cx<float> g = pick(lane == 31, er, dn_c(x4.v[0], 1));
          if (end) g = sm.xf * ld1(Xr);
          const cx<float> s01 = x4.v[0] + x4.v[1], s23 = x4.v[2] + x4.v[3];
          acc.v[0] += scal(wh[q], l + s01) - scal(wx[q], x4.v[0]);
          acc.v[1] += scal(wh[q], s01 + x4.v[2]) - scal(wx[q], x4.v[1]);
          acc.v[2] += scal(wh[q], x4.v[1] + s23) - scal(wx[q], x4.v[2]);
          acc.v[3] += scal(wh[q], s23 + g) - scal(wx[q], x4.v[3]);
          if (q > 0 && q < 4) {
            const int j = row_at(r);
            Four d = ld4(bv + (size_t) j * n + (in ? c : 0), 2);
            if (j != r)
#pragma unroll
              for (int u = 0; u < 4; u++) d.v[u] = bphase(r) * d.v[u];
#pragma unroll
            for (int u = 0; u < 4; u++) t4.v[u] += scal(q == 2 ? 1.0f : 0.5f, d.v[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) acc.v[u] = t4.v[u] + scal(third, acc.v[u]);
        const cx<float> l = pick(lane == 0, left, up_c(acc.v[3], 1));
        left = at_c(acc.v[3], 31);
        if (in)
          st2(bc + (size_t) kv * nc * nc + (size_t) J * nc + c / 2,
              Two{acc.v[0] + scal(0.5f, l + acc.v[1]), acc.v[2] + scal(0.5f, acc.v[1] + acc.v[3])});
      }
    }
  }
}

// [k][e][v] <-> [k][v][e] in tiles of 64 elements x m vectors, both sides in
// 16-byte accesses where m is even (nn is)
__global__ void __launch_bounds__(256) k_planar(int nn, int m, int to, const float2* __restrict__ src,
                                                float2* __restrict__ dst) {
  __shared__ float2 t[32 * 65];   // [v][e], a vector's elements 65 apart
  const int k = blockIdx.y, e0 = blockIdx.x * 64, ne = nn - e0 < 64 ? nn - e0 : 64, len = ne * m;
  const size_t base = (size_t) k * nn * m;
  const float2* si = src + base + (size_t) e0 * m;
  float2* di = dst + base + (size_t) e0 * m;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (to) {
    if (m % 2 == 0)
      for (int q = 2 * threadIdx.x; q < len; q += 512) {
        const int e = q / m, v = q - e * m;
        const float4 f = *reinterpret_cast<const float4*>(si + q);
        t[v * 65 + e] = make_float2(f.x, f.y);
        t[(v + 1) * 65 + e] = make_float2(f.z, f.w);
      }
    else
      for (int q = threadIdx.x; q < len; q += 256) t[(q % m) * 65 + q / m] = si[q];
    __syncthreads();
    for (int v = w; v < m; v += 8) {
      const int e = 2 * lane;
      if (e < ne) {
        const float2 a = t[v * 65 + e], c = t[v * 65 + e + 1];
        *reinterpret_cast<float4*>(dst + base + (size_t) v * nn + e0 + e) = make_float4(a.x, a.y, c.x, c.y);
      }
    }
  } else {
    for (int v = w; v < m; v += 8) {
      const int e = 2 * lane;
      if (e < ne) {
        const float4 f = *reinterpret_cast<const float4*>(src + base + (size_t) v * nn + e0 + e);
        t[v * 65 + e] = make_float2(f.x, f.y);
        t[v * 65 + e + 1] = make_float2(f.z, f.w);
      }
    }
    __syncthreads();
    if (m % 2 == 0)
      for (int q = 2 * threadIdx.x; q < len; q += 512) {
        const int e = q / m, v = q - e * m;
        const float2 a = t[v * 65 + e], c = t[(v + 1) * 65 + e];
        *reinterpret_cast<float4*>(di + q) = make_float4(a.x, a.y, c.x, c.y);
      }
    else
      for (int q = threadIdx.x; q < len; q += 256) di[q] = t[(q % m) * 65 + q / m];
  }
}

// rows per band: as many as two CTAs per SM hold, fewer (down to 8) where the
// batch leaves SMs without a CTA; even, the last band not below 8 rows
int band_rows(int n, int vecs, int halo) {
  int B = (110 * 1024) / ((n + 127) / 128 * 128 * 8) - halo;
  const int want = (int) (((size_t) n * vecs + 607) / 608);   // four CTAs per SM
  if (B > want) B = want;
  if (B > n / 2) B = n / 2;
  B &= ~1;
  if (B < 8) B = 8;
  for (int q = B; q >= 8; q -= 2)
    if (n % q == 0 || n % q >= 8) return q;
  while (n % B != 0 && n % B < 8) B += 2;
  return B;
}

size_t cycle_smem(int n0, int top, int prec) {
  const size_t es = prec == MX_C64 ? 8 : 16;
  size_t s = NCT;
  for (int l = top; l >= 0; l--) s += 2 * (size_t) (n0 << l) * (n0 << l);
  return s * es;
}

template <typename S, typename R, typename MS>
int run(int n0, int top, int m, int K, int nu, int cycles, int zero, int planar, const double* ph, const void* ainv, int prec,
        const void* b, void* x, cudaStream_t st) {
  const size_t smem = cycle_smem(n0, top, prec);
  // FP64 vectors over a cluster of CTAs where SMs are left for it: cycle of
  // levels 64 .. 8 of 48 vectors 510 us on one CTA each, 380 on two; of 16,
  // 509, 379 and on four 348; of one, 502, 374 and 342.  Three CTAs for 48 no
  // longer run side by side (693 us).  Levels 32 .. 8: 197 and 180; 16, 8: 87
  // and 89.  c64 and float-float do not wait for the arithmetic unit: 63 -> 95
  // and 331 -> 371 us on two.
  int cl = 1;
  if (prec == MX_C128 && n0 << top >= 32) cl = K * m <= 16 ? 4 : K * m <= 64 ? 2 : 1;
  auto kern = k_node_vcycle<S, R, MS, false>;
  if constexpr (std::is_same<R, double>::value)
    if (cl > 1) kern = k_node_vcycle<S, R, MS, true>;
  allow_smem(kern);
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = cl;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned) K * m * cl);
  cfg.blockDim = dim3(NCT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = cl > 1;
  return (int) cudaLaunchKernelEx(&cfg, kern, n0, top, m, K, nu, cycles, zero, planar, ph, make_sc(1.0 / 3.0),
                                  (const MS*) ainv, (const S*) b, (S*) x);
}

}  // namespace

// Every level whose chain of levels fits into a CTA's shared memory, up to 96
// nodes a side (three positions per lane): c64 64 and 96, FP64 64.  The coarse
// solve wants n0^2 <= NCT / 2 rows.
extern "C" int mxk_node_vcycle_top(int n0, int top, int prec) {
  if (n0 < 4 || (n0 & 1) || n0 > 16) return 0;
  int l = 0;
  while (l < top && (n0 << (l + 1)) <= 96 && cycle_smem(n0, l + 1, prec) <= 200 * 1024) l++;
  return l;
}

// A CTA per vector: past the batch that the SMs hold at once the launch takes a
// multiple of its time, while the row kernels it replaces only then begin to
// fill the GPU.  The limits by the highest level's nodes a side, n; one launch
// against theirs, ms, cycles from 16 and 32 to 4 nodes, from 64 to 8, and of
// FP64 and float-float from 80 and 96, whose highest level is 40 and 48:
// c64    2048 vectors 0.33/0.36, 0.50/0.60, 0.76/1.01, from 96 to 12 1.60/1.71;
//        3072 0.49/0.39, 0.74/0.68, 1.13/1.30, 2.38/2.07;
//        4096 0.64/0.40, 0.97/0.70, 1.46/1.43
// FP64   1024 vectors 0.90/0.92, 1.66/1.84, 3.49/4.10;
//        1280 1.15/0.98, 2.12/2.38, 4.48/5.41, 6.57/7.13, 9.09/9.37;
//        1536 1.40/0.99, 2.59/2.44, 5.47/5.82, 8.14/8.30, 10.2/9.92
// cdd    448 vectors 0.55/0.64, 0.80/1.08, 1.08/1.57, 1.71/1.86, 2.37/2.45;
//        512 0.70/0.65, 1.02/1.08, 1.39/1.59, 2.19/2.16, 2.69/2.50;
//        640 0.86/0.65, 1.25/1.10, 1.71/1.85
// (Under a level that takes bands the launch serves every batch: the bands'
// planar vectors need it, and they gain more than it loses.)
extern "C" int mxk_node_vcycle_pays(int n, int vecs, int prec) {
  // (a multiple of 32 or 64: rows that fill their lanes)
  if (prec == MX_C64) return vecs <= (n % 64 ? 2048 : 3072);
  if (prec == MX_C128) return vecs <= (n < 32 ? 1024 : 1280);
  return vecs <= (n % 32 ? 448 : 512);
}

extern "C" int mxk_node_vcycle(int n0, int top, int m, int K, int nu, int cycles, int zero, int planar,
                               const double* ph, const double* ainv, const void* ainv_c64, int prec, const void* b, void* x, mx_stream s) {
  cudaStream_t st = (cudaStream_t) s;
  if (prec == MX_C64) {
    if (ainv_c64) return run<float2, float, float2>(n0, top, m, K, nu, cycles, zero, planar, ph, ainv_c64, prec, b, x, st);
    return run<float2, float, double2>(n0, top, m, K, nu, cycles, zero, planar, ph, ainv, prec, b, x, st);
  }
  if (prec == MX_C128) return run<double2, double, double2>(n0, top, m, K, nu, cycles, zero, planar, ph, ainv, prec, b, x, st);
  return run<cdd, dd, double2>(n0, top, m, K, nu, cycles, zero, planar, ph, ainv, prec, b, x, st);
}

// c64 levels of 100 to 512 nodes a side (a row of more columns would leave the
// bands mostly halo), at most two sweeps each way
extern "C" int mxk_node_band_ok(int n, int m, int nu, int prec) {
  return prec == MX_C64 && n > 96 && n <= 512 && n % 4 == 0 && nu >= 1 && nu <= 2 && m <= 32;
}

extern "C" int mxk_node_band_pre(int n, int m, int K, int nu, const double* ph, const void* b, const void* xin, void* xout,
                                 void* bc, mx_stream s) {
  const int halo = 4 * nu + 3, B = band_rows(n, K * m, halo), nb = (n + B - 1) / B;
  const size_t smem = (size_t) (B + halo) * ((n + 127) / 128 * 128) * sizeof(float2);
  allow_smem(k_node_band<false>);
  k_node_band<false><<<(unsigned) nb * K * m, NBT, smem, (cudaStream_t) s>>>(
      n, m, K, B, nu, ph, (float) (1.0 / 3.0), (const float2*) b, (const float2*) xin, nullptr, (float2*) xout, (float2*) bc);
  MX_CHECK_LAUNCH();
  return 0;
}

extern "C" int mxk_node_band_post(int n, int m, int K, int nu, const double* ph, const void* b, const void* xin,
                                  const void* xc, void* xout, mx_stream s) {
  const int halo = 4 * nu, B = band_rows(n, K * m, halo), nb = (n + B - 1) / B;
  const size_t smem = (size_t) (B + halo) * ((n + 127) / 128 * 128) * sizeof(float2);
  allow_smem(k_node_band<true>);
  k_node_band<true><<<(unsigned) nb * K * m, NBT, smem, (cudaStream_t) s>>>(
      n, m, K, B, nu, ph, (float) (1.0 / 3.0), (const float2*) b, (const float2*) xin, (const float2*) xc, (float2*) xout,
      nullptr);
  MX_CHECK_LAUNCH();
  return 0;
}

extern "C" int mxk_node_planar(int n, int m, int K, int to, const void* src, void* dst, mx_stream s) {
  const int nn = n * n;
  k_planar<<<dim3((nn + 63) / 64, K), 256, 0, (cudaStream_t) s>>>(nn, m, to, (const float2*) src, (float2*) dst);
  MX_CHECK_LAUNCH();
  return 0;
}
