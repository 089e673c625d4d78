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
// Bound by the latency of a phase (shared loads, scan, barrier; FP64 blocks by
// the FP64 rate of the K m SMs it occupies).  One cycle of the levels 64 .. 8,
// 8 k-points x 16 c64 vectors: 66 us against about 460 us in 62 launches; five
// cycles from 64 of 4 x 12 FP64 vectors 2.2 ms against 9.9 ms.
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

// one row of one sweep by a warp; EDGE: row 0 or n-1, whose neighbour rows
// cross the seam
template <typename R, int LR, bool EDGE>
__device__ void gs_row(int n, int j, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm) {
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
    if (t0 + q < n) Xc[at(t0 + q)] = y[q] + carry;
  }
}

// one sweep by the CTA; ends at a barrier
template <typename R, int LR>
__device__ void sweep(int n, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm) {
  const int warp = threadIdx.x >> 5, nw = NCT / 32;
#pragma unroll 1
  for (int ph = 0; ph < 2; ph++) {
    // forward: row 0 and the odd rows, then the even rows and row n-1;
    // backward the reverse
    const bool odd = (ph == 0) != (back != 0);
    if (warp == 0) {
      const int edge = odd ? 0 : n - 1, next = odd ? 1 : n - 2;
      if (ph == 0) {
        gs_row<R, LR, true>(n, edge, back, X, B, sm);
        __syncwarp();
        gs_row<R, LR, false>(n, next, back, X, B, sm);
      } else {
        gs_row<R, LR, false>(n, next, back, X, B, sm);
        __syncwarp();
        gs_row<R, LR, true>(n, edge, back, X, B, sm);
      }
    } else {
      // the group's other rows: 3, 5 .. n-3 or 2, 4 .. n-4
      for (int r = warp - 1; r < n / 2 - 2; r += nw - 1) gs_row<R, LR, false>(n, (odd ? 3 : 2) + 2 * r, back, X, B, sm);
    }
    __syncthreads();
  }
}

template <typename R>
__device__ void smooth(int n, int nu, int back, cx<R>* X, const cx<R>* B, const Seam<R>& sm) {
  for (int q = 0; q < nu; q++) {
    if (n <= 32) sweep<R, 1>(n, back, X, B, sm);
    else if (n <= 64) sweep<R, 2>(n, back, X, B, sm);
    else sweep<R, 3>(n, back, X, B, sm);
  }
}

// bc = restriction of b - L x, xc = 0
template <typename R>
__device__ void restrict_residual(int n, const cx<R>* X, const cx<R>* B, cx<R>* Xc, cx<R>* Bc, const Seam<R>& sm,
                                  const Sc& third_s) {
  const int nc = n / 2;
  const R third = sget<R>(third_s), half = rc<R>(0.5f), nine = rc<R>(9.0f);
  for (int e = threadIdx.x; e < nc * nc; e += NCT) {
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
    Bc[e] = out;
    Xc[e] = czero<R>();
  }
  __syncthreads();
}

// x += P xc, bilinear
template <typename R>
__device__ void prolong(int n, cx<R>* X, const cx<R>* Xc, const Seam<R>& sm) {
  const int nc = n / 2;
  const R half = rc<R>(0.5f);
  for (int e = threadIdx.x; e < nc * nc; e += NCT) {
    const int I = e % nc, J = e / nc;
    const bool wi = I == nc - 1, wj = J == nc - 1;
    const int I1 = wi ? 0 : I + 1, J1 = wj ? 0 : J + 1;
    cx<R> c00 = Xc[e], c10 = Xc[J * nc + I1], c01 = Xc[J1 * nc + I], c11 = Xc[J1 * nc + I1];
    if (wi) { c10 = sm.xf * c10; c11 = sm.xf * c11; }
    if (wj) { c01 = sm.yf * c01; c11 = sm.yf * c11; }
    cx<R>* p0 = X + 2 * J * n + 2 * I;
    cx<R>* p1 = p0 + n;
    const cx<R> h0 = scal(half, c00 + c10), h1 = scal(half, c01 + c11);
    p0[0] += c00;
    p0[1] += h0;
    p1[0] += scal(half, c00 + c01);
    p1[1] += scal(half, h0 + h1);
  }
  __syncthreads();
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

template <typename S, typename R, typename MS>
__global__ void __launch_bounds__(NCT) k_node_vcycle(int n0, int top, int m, int K, int nu, int cycles, int zero,
                                                   const double* __restrict__ ph, Sc third,
                                                   const MS* __restrict__ ainv, const S* __restrict__ b, S* x) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const int v = blockIdx.x % m, k = blockIdx.x / m, n = n0 << top, nn = n * n;
  // level l: x, then b; the top level first
  cx<R>* part = reinterpret_cast<cx<R>*>(sm_raw);
  cx<R>* X = part + NCT;
  auto level = [&](int l) {
    cx<R>* p = X;
    for (int q = top; q > l; q--) p += 2 * (n0 << q) * (n0 << q);
    return p;
  };
  const Seam<R> sm0 = seam_load<R>(ph, K, k, n);
  const S* bk = b + (size_t) k * nn * m + v;
  S* xk = x + (size_t) k * nn * m + v;
  for (int e = threadIdx.x; e < nn; e += NCT) {
    X[nn + e] = Store<S, R>::ld(bk + (size_t) e * m);
    X[e] = zero ? czero<R>() : Store<S, R>::ld(xk + (size_t) e * m);
  }
  __syncthreads();
  for (int c = 0; c < cycles; c++) {
#pragma unroll 1
    for (int l = top; l > 0; l--) {
      const int nl = n0 << l;
      cx<R>*Xl = level(l), *Xc = level(l - 1);
      Seam<R> sm = sm0;
      sm.n = nl;
      smooth<R>(nl, nu, 0, Xl, Xl + nl * nl, sm);
      restrict_residual<R>(nl, Xl, Xl + nl * nl, Xc, Xc + nl * nl / 4, sm, third);
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
      prolong<R>(nl, Xl, level(l - 1), sm);
      smooth<R>(nl, nu, 1, Xl, Xl + nl * nl, sm);
    }
  }
  for (int e = threadIdx.x; e < nn; e += NCT) Store<S, R>::st(xk + (size_t) e * m, X[e]);
}

size_t cycle_smem(int n0, int top, int prec) {
  const size_t es = prec == MX_C64 ? 8 : 16;
  size_t s = NCT;
  for (int l = top; l >= 0; l--) s += 2 * (size_t) (n0 << l) * (n0 << l);
  return s * es;
}

template <typename S, typename R, typename MS>
int run(int n0, int top, int m, int K, int nu, int cycles, int zero, const double* ph, const void* ainv, int prec,
        const void* b, void* x, cudaStream_t st) {
  const size_t smem = cycle_smem(n0, top, prec);
  cudaFuncSetAttribute(k_node_vcycle<S, R, MS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
  k_node_vcycle<S, R, MS><<<(unsigned) K * m, NCT, smem, st>>>(n0, top, m, K, nu, cycles, zero, ph, make_sc(1.0 / 3.0),
                                                               (const MS*) ainv, (const S*) b, (S*) x);
  MX_CHECK_LAUNCH();
  return 0;
}

}  // namespace

// Every level whose chain of levels fits into a CTA's shared memory, up to 96
// nodes a side (three positions per lane): c64 64 and 96, FP64 64.  Measured
// as above for 64; with 1 to 512 vectors in the batch the launches it
// replaces cost more.  The coarse solve wants n0^2 <= NCT / 2 rows.
extern "C" int mxk_node_vcycle_top(int n0, int top, int prec) {
  if (n0 < 4 || (n0 & 1) || n0 > 16) return 0;
  int l = 0;
  while (l < top && (n0 << (l + 1)) <= 96 && cycle_smem(n0, l + 1, prec) <= 200 * 1024) l++;
  return l;
}

extern "C" int mxk_node_vcycle(int n0, int top, int m, int K, int nu, int cycles, int zero, const double* ph,
                               const double* ainv, const void* ainv_c64, int prec, const void* b, void* x, mx_stream s) {
  cudaStream_t st = (cudaStream_t) s;
  if (prec == MX_C64) {
    if (ainv_c64) return run<float2, float, float2>(n0, top, m, K, nu, cycles, zero, ph, ainv_c64, prec, b, x, st);
    return run<float2, float, double2>(n0, top, m, K, nu, cycles, zero, ph, ainv, prec, b, x, st);
  }
  if (prec == MX_C128) return run<double2, double, double2>(n0, top, m, K, nu, cycles, zero, ph, ainv, prec, b, x, st);
  return run<cdd, dd, double2>(n0, top, m, K, nu, cycles, zero, ph, ainv, prec, b, x, st);
}
