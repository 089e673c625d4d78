// Batched small dense complex linear algebra in FP64 (one CTA per k-point).
// These matrices are small (at n0 = 8 the inverses of 64 nodes and of 128
// edges, the coarse eigenproblem's matrix of 64 cells; Ritz systems of at most
// 3m = 96 columns); the Jacobi sweeps of the coarse eigenproblem and the Ritz
// step do most of their rotations in FP32 and finish in FP64 (jacobi_mixed).
// They replace the reference's LAPACK calls (linalg.c:48-317):
//   mxk_hpd_inverse    zpotrf + ztrsm pairs of the coarse-grid solves
//   mxk_coarse_pairs   zhegv of the coarse start, through the cells' matrix
//   mxk_heev           zheev (cyclic Jacobi with Brent-Luk parallel ordering)
//   mxk_rayleigh_ritz  zhegv of the Ritz step, as Cholesky-QR of the Gram
//                      matrix with column dropping followed by Jacobi
// Matrices are column-major, complex stored as (re, im) double pairs.
#include "mx_common.cuh"
#include "mx_internal.h"

#include <math.h>

using namespace mx;

namespace {

constexpr int DT = 256;   // threads per CTA

struct Z {
  double re, im;
};
__device__ __forceinline__ Z zmk(double a, double b) { Z z; z.re = a; z.im = b; return z; }
__device__ __forceinline__ Z zadd(Z a, Z b) { return zmk(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ Z zsub(Z a, Z b) { return zmk(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ Z zmul(Z a, Z b) { return zmk(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re); }
__device__ __forceinline__ Z zcmul(Z a, Z b) { return zmk(a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re); }  // conj(a) b
__device__ __forceinline__ Z zconj(Z a) { return zmk(a.re, -a.im); }
__device__ __forceinline__ Z zscal(double s, Z a) { return zmk(s * a.re, s * a.im); }
__device__ __forceinline__ double zabs2(Z a) { return a.re * a.re + a.im * a.im; }
__device__ __forceinline__ Z zdiv(Z a, Z b) {
  double d = zabs2(b);
  return zmk((a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d);
}

#define AT(M, ld, i, j) (reinterpret_cast<Z*>(M)[(size_t) (j) * (ld) + (i)])

__device__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    t = warp_sum(t);
  }
  __syncthreads();
  if (threadIdx.x == 0) sh[0] = t;
  __syncthreads();
  t = sh[0];
  __syncthreads();
  return t;
}

// ------------------------------------------------------------------
// Gauss-Jordan inverse of a Hermitian positive definite matrix (no
// pivoting is needed for HPD input)
// ------------------------------------------------------------------
__global__ void k_hpd_inverse(int N, double* a, int* info) {
  extern __shared__ double sm[];
  Z* f = reinterpret_cast<Z*>(sm);
  Z* rowp = f + N;
  double* A = a + (size_t) blockIdx.x * 2 * N * N;
  int bad = 0;
  for (int p = 0; p < N; p++) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) f[i] = AT(A, N, i, p);
    __syncthreads();
    Z piv = f[p];
    if (!(piv.re > 0.0)) bad = p + 1;
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      Z v = j == p ? zmk(1.0, 0.0) : AT(A, N, p, j);
      rowp[j] = zdiv(v, piv);
    }
    __syncthreads();
    for (size_t e = threadIdx.x; e < (size_t) N * N; e += blockDim.x) {
      int i = (int) (e % N), j = (int) (e / N);
      if (i == p) AT(A, N, i, j) = rowp[j];
      else {
        Z v = j == p ? zmk(0.0, 0.0) : AT(A, N, i, j);
        AT(A, N, i, j) = zsub(v, zmul(f[i], rowp[j]));
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && info) info[blockIdx.x] = bad;
}

// The same for matrices whose lower triangle fits into shared memory, by the
// symmetric sweep operator: with d = a_pp, a_ij -= a_ip a_pj / d, a_ip /= d,
// a_pp = -1 / d keep the matrix Hermitian, and sweeping every p leaves -A^-1.
// Half the arithmetic of the Gauss-Jordan step, which the FP64 unit of one SM
// bounds, no index division per entry and no round trip to L2.  A warp takes
// whole columns (packed, column j from its diagonal on).  Orders 128 and 64
// (n0 = 8), together: 5.2 -> 3.1 ms.
constexpr int SWT = 512;
__host__ __device__ inline size_t sweep_smem(int N) { return ((size_t) N * (N + 1) / 2 + 2 * (size_t) N) * sizeof(Z); }

__global__ void __launch_bounds__(SWT) k_hpd_inverse_sweep(int N, double* a, int* info) {
  extern __shared__ double sm[];
  Z* f = reinterpret_cast<Z*>(sm);
  Z* g = f + N;
  Z* L = g + N;
  double* A = a + (size_t) blockIdx.x * 2 * N * N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = SWT / 32;
  auto col = [&](int j) { return L + j * N - j * (j + 1) / 2; };   // col(j)[i] = a_ij, i >= j
  for (int j = warp; j < N; j += nw)
    for (int i = j + lane; i < N; i += 32) col(j)[i] = AT(A, N, i, j);
  __syncthreads();
  int bad = 0;
  for (int p = 0; p < N; p++) {
    const double d = col(p)[p].re;
    if (!(d > 0.0)) bad = p + 1;
    if ((int) threadIdx.x < N) {
      const int i = threadIdx.x;
      const double inv = 1.0 / d;
      const Z v = i >= p ? col(p)[i] : zconj(col(i)[p]);
      f[i] = v;
      g[i] = i == p ? zmk(-inv, 0.0) : zmk(v.re * inv, v.im * inv);
    }
    __syncthreads();
    for (int j = warp; j < N; j += nw) {
      Z* c = col(j);
      if (j == p) {
        for (int i = j + lane; i < N; i += 32) c[i] = g[i];
      } else {
        const Z gj = g[j];
        for (int i = j + lane; i < N; i += 32) {
          const Z v = zsub(c[i], zcmul(gj, f[i]));
          c[i] = i == p ? zconj(gj) : v;
        }
      }
    }
    __syncthreads();
  }
  for (int j = warp; j < N; j += nw)
    for (int i = j + lane; i < N; i += 32) {
      const Z v = col(j)[i];
      AT(A, N, i, j) = zmk(-v.re, i == j ? 0.0 : -v.im);
      if (i > j) AT(A, N, j, i) = zmk(-v.re, v.im);
    }
  if (threadIdx.x == 0 && info) info[blockIdx.x] = bad;
}

// ------------------------------------------------------------------
// y_k = Ainv_k x_k on a level-0 block: the block of one k-point is a
// row-major N x m matrix (dense row r at offset r*m)
// ------------------------------------------------------------------
// The inverse is read as MS (double2, or its float2 rounding for FP32 solves).
template <typename S, typename R, typename MS>
__global__ void k_coarse_apply(int N, int m, const MS* __restrict__ ainv, const S* __restrict__ x,
                               S* __restrict__ y) {
  int k = blockIdx.y;
  const MS* Ai = ainv + (size_t) k * N * N;
  const S* xk = x + (size_t) k * N * m;
  S* yk = y + (size_t) k * N * m;
  size_t t = (size_t) blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t) N * m) return;
  int v = (int) (t % m), r = (int) (t / m);
  cx<R> acc = czero<R>();
  for (int c = 0; c < N; c++)
    acc += Store<MS, R>::ld(Ai + (size_t) c * N + r) * Store<S, R>::ld(xk + (size_t) c * m + v);
  Store<S, R>::st(yk + (size_t) r * m + v, acc);
}

// ------------------------------------------------------------------
// Cyclic Jacobi for a Hermitian N x N matrix (full storage), eigenvectors
// accumulated in Zm; Brent-Luk round-robin ordering lets the N/2 rotations of
// one round run concurrently.  Rotation of the pair (p,q) with a_pq = g e,
// g = |a_pq|, d = a_qq - a_pp, h = sqrt(d^2 + 4 g^2): cos(2 theta) = |d| / h,
// c = cos theta, s = sgn(d) g / (h c), V = [[c, s e], [-s conj(e), c]] on
// (p,q); A <- V^H A V, Z <- Z V.
//
// A CTA works alone on its matrix, so what bounds it is the FP64 rate of one
// SM (2 FMA per clock; a warp instruction takes 64 cycles whatever its active
// lanes).  Hence: the 2 x 2 blocks of A (pair s against pair t <= s) are
// rotated from both sides in one pass and mirrored, half the arithmetic of a
// column pass and a row pass and a barrier less; an angle costs three
// reciprocal square roots instead of three square roots and five divisions;
// eigenvalues are sorted by rank in parallel.
// Rayleigh-Ritz step of 8 k-points, before and after: 48 columns 4.39 -> 2.52
// ms, 36 columns 1.35 -> 0.80 ms, the coarse eigenproblem of 128 columns (its
// matrices in global memory) 85 -> 54 ms.
// ------------------------------------------------------------------
template <typename T> struct Cx {
  T re, im;
};
__device__ __forceinline__ float rsq(float v) { return rsqrtf(v); }
__device__ __forceinline__ double rsq(double v) { return rsqrt(v); }
#define AM(M, i, j) (M[(size_t) (j) * ld + (i)])

// rotation data of one CTA: half = (N + 1) / 2 pairs
template <typename T> struct Rot {
  T *c, *s, *er, *ei;
  int *p, *q;
};
template <typename T> __device__ __forceinline__ Rot<T> rot_data(double* shd, int* shi, int half) {
  T* t = reinterpret_cast<T*>(shd);
  return Rot<T>{t, t + half, t + 2 * half, t + 3 * half, shi, shi + half};
}

// (x, y) -> (c x - s conj(e) y, s e x + c y): the columns p, q of a row
template <typename T>
__device__ __forceinline__ void rot_right(T c, T s, T xr, T xi, Cx<T>& x, Cx<T>& y) {
  const T sr = s * xr, si = s * xi;
  const Cx<T> a = x, b = y;
  x.re = c * a.re - sr * b.re - si * b.im;
  x.im = c * a.im - sr * b.im + si * b.re;
  y.re = sr * a.re - si * a.im + c * b.re;
  y.im = sr * a.im + si * a.re + c * b.im;
}

// sweeps until one makes no rotation: a pair is left alone when |a_pq|^2 is
// below tol |a_pp a_qq| or below tolf |A|_F^2 (Rutishauser's test; a block of
// equal or zero eigenvalues would otherwise be rotated forever)
template <typename T>
__device__ void jacobi_sweeps(int N, int ld, Cx<T>* A, Cx<T>* Zm, double* shd, int* shi, double* red, T tol, T tolf,
                              int max_sweeps) {
  const int Np = N + (N & 1), half = Np / 2;   // padded to even with a dummy index N
  const Rot<T> R = rot_data<T>(shd, shi, half);
  double fro = 0.0;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const Cx<T> a = AM(A, e % N, e / N);
    fro += (double) a.re * a.re + (double) a.im * a.im;
  }
  const T tf = tolf * (T) block_sum(fro, red);
  const int nblk = half * (half + 1) / 2;
  const int bq = (int) blockDim.x / N, br = (int) blockDim.x % N;
  const int s0 = (int) threadIdx.x / N, i0 = (int) threadIdx.x % N;
  for (int sweep = 0; sweep < max_sweeps; sweep++) {
    int rotated = 0;
    for (int r = 0; r < Np - 1; r++) {
      for (int s = threadIdx.x; s < half; s += blockDim.x) {
        const int a = s == 0 ? 0 : 1 + (s - 1 + r) % (Np - 1);
        const int b = 1 + (Np - 2 - s + r) % (Np - 1);
        const int p = a < b ? a : b, q = a < b ? b : a;
        T c = 1, sv = 0, xr = 1, xi = 0;
        if (q < N) {
          const Cx<T> apq = AM(A, p, q);
          const T app = AM(A, p, p).re, aqq = AM(A, q, q).re;
          const T g2 = apq.re * apq.re + apq.im * apq.im, w = app * aqq;
          if (g2 > tol * (w < 0 ? -w : w) && g2 > tf) {
            rotated = 1;
            const T d = aqq - app, ad = d < 0 ? -d : d;
            const T rg = rsq(g2), rh = rsq(d * d + 4 * g2);
            const T u = (T) 0.5 + (T) 0.5 * ad * rh, ru = rsq(u);
            c = u * ru;
            sv = g2 * rg * rh * ru;
            if (d < 0) sv = -sv;
            xr = apq.re * rg;
            xi = apq.im * rg;
          }
        }
        R.p[s] = p; R.q[s] = q; R.c[s] = c; R.s[s] = sv; R.er[s] = xr; R.ei[s] = xi;
      }
      __syncthreads();
      // A <- V^H A V by blocks of rows (p_s, q_s) and columns (p_t, q_t), t <= s
      for (int e = threadIdx.x; e < nblk; e += blockDim.x) {
        int s = (int) ((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
        while (s * (s + 1) / 2 > e) s--;
        while ((s + 1) * (s + 2) / 2 <= e) s++;
        const int t = e - s * (s + 1) / 2;
        const T ss = R.s[s], st = R.s[t];
        if (ss == 0 && st == 0) continue;
        const int p = R.p[s], q = R.q[s], u = R.p[t], v = R.q[t];
        const bool hq = q < N, hv = v < N;   // the dummy index has no entries
        Cx<T> pu = AM(A, p, u), pv = {0, 0}, qu = {0, 0}, qv = {0, 0};
        if (hv) pv = AM(A, p, v);
        if (hq) qu = AM(A, q, u);
        if (hq && hv) qv = AM(A, q, v);
        if (st != 0) {
          const T ct = R.c[t], xr = R.er[t], xi = R.ei[t];
          rot_right(ct, st, xr, xi, pu, pv);
          rot_right(ct, st, xr, xi, qu, qv);
        }
        if (ss != 0) {   // rows: conjugated e
          const T cs = R.c[s], xr = R.er[s], xi = -R.ei[s];
          rot_right(cs, ss, xr, xi, pu, qu);
          rot_right(cs, ss, xr, xi, pv, qv);
        }
        if (s == t) { pu.im = 0; qv.im = 0; }
        AM(A, p, u) = pu;
        if (hv) AM(A, p, v) = pv;
        if (hq) AM(A, q, u) = qu;
        if (hq && hv) AM(A, q, v) = qv;
        if (s != t) {
          AM(A, u, p) = Cx<T>{pu.re, -pu.im};
          if (hv) AM(A, v, p) = Cx<T>{pv.re, -pv.im};
          if (hq) AM(A, u, q) = Cx<T>{qu.re, -qu.im};
          if (hq && hv) AM(A, v, q) = Cx<T>{qv.re, -qv.im};
        }
      }
      // Z <- Z V: the (rotation s, row i) items e = s N + i are dealt to the
      // threads in strides of blockDim.x, with (s, i) advanced incrementally
      for (int s = s0, i = i0; s < half;
           s += bq + (i + br >= N), i = i + br >= N ? i + br - N : i + br) {
        const T sv = R.s[s];
        if (sv == 0) continue;
        const int p = R.p[s], q = R.q[s];
        Cx<T> x = AM(Zm, i, p), y = AM(Zm, i, q);
        rot_right(R.c[s], sv, R.er[s], R.ei[s], x, y);
        AM(Zm, i, p) = x;
        AM(Zm, i, q) = y;
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
}

// eigenvalues (the diagonal of A) ascending into w, the columns of Zm in the
// same order; A is overwritten.  An eigenvalue that is NaN keeps its place and
// the numbers ascend around it: the ranks are a permutation in any case.
__device__ void sort_eigen(int N, int ld, Cx<double>* A, Cx<double>* Zm, double* w, int* rank) {
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double wi = AM(A, i, i).re;
    int r = 0, nans = 0;
    for (int j = 0; j < N; j++) {
      const double wj = AM(A, j, j).re;
      r += wj < wi || (wj == wi && j < i);
      nans += wj != wj;
    }
    if (wi != wi) r = i;
    else if (nans)
      for (int j = 0; j < N && j <= r; j++) r += AM(A, j, j).re != AM(A, j, j).re;
    rank[i] = r;
    w[r] = wi;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) AM(A, e % N, rank[e / N]) = AM(Zm, e % N, e / N);
  __syncthreads();
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) AM(Zm, e % N, e / N) = AM(A, e % N, e / N);
  __syncthreads();
}

// FP64 eigendecomposition; A completed from its lower triangle
__device__ void jacobi_cta(int N, int ld, double* A, double* Zm, double* w, double* shd, int* shi, int max_sweeps) {
  const int half = (N + 1) / 2 + 1;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    int i = e % N, j = e / N;
    AT(Zm, ld, i, j) = zmk(i == j ? 1.0 : 0.0, 0.0);
    if (i < j) AT(A, ld, i, j) = zconj(AT(A, ld, j, i));
    if (i == j) AT(A, ld, i, i).im = 0.0;
  }
  __syncthreads();
  jacobi_sweeps<double>(N, ld, reinterpret_cast<Cx<double>*>(A), reinterpret_cast<Cx<double>*>(Zm), shd, shi,
                        shd + 4 * half, 1e-32, 1e-30, max_sweeps);
  sort_eigen(N, ld, reinterpret_cast<Cx<double>*>(A), reinterpret_cast<Cx<double>*>(Zm), w, shi);
}

// ------------------------------------------------------------------
// Mixed-precision Jacobi.  FP64 arithmetic on GB300 runs at a small fraction
// of the FP32 rate and a CTA's Jacobi sweeps are bound by it, so the sweeps
// that do the bulk of the work run in FP32: they bring the off-diagonal
// part down to about 1e-6 of the matrix.  Their accumulated rotations Zf are
// then made unitary to FP64 precision by one Newton-Schulz step
// Q = Z (3I - Z^H Z) / 2, the matrix is transformed exactly in FP64,
// A' = Q^H A Q (same eigenvalues as A), and FP64 sweeps finish A' -- one or
// two, Jacobi converging quadratically -- accumulating into Q.
// ------------------------------------------------------------------

// C = op(X) Y for N x N complex FP64 matrices (leading dimension ld), op =
// conjugate transpose when cx; herm: C is Hermitian, half of it is computed
__device__ void zgemm_cta(int N, int ld, double* X, bool cx, double* Y, double* C, bool herm) {
  const int items = herm ? N * (N + 1) / 2 : N * N;
  for (int e = threadIdx.x; e < items; e += blockDim.x) {
    int i = e % N, j = e / N;
    if (herm) {
      i = (int) ((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
      while (i * (i + 1) / 2 > e) i--;
      while ((i + 1) * (i + 2) / 2 <= e) i++;
      j = e - i * (i + 1) / 2;
    }
    Z s = zmk(0.0, 0.0);
    if (cx)
      for (int l = 0; l < N; l++) {
        const Z a = AT(X, ld, l, i), b = AT(Y, ld, l, j);
        s.re = fma(a.re, b.re, fma(a.im, b.im, s.re));
        s.im = fma(a.re, b.im, fma(-a.im, b.re, s.im));
      }
    else
      for (int l = 0; l < N; l++) {
        const Z a = AT(X, ld, i, l), b = AT(Y, ld, l, j);
        s.re = fma(a.re, b.re, fma(-a.im, b.im, s.re));
        s.im = fma(a.re, b.im, fma(a.im, b.re, s.im));
      }
    AT(C, ld, i, j) = s;
    if (herm && i != j) AT(C, ld, j, i) = zconj(s);
  }
  __syncthreads();
}

// Eigen-decomposition of the Hermitian A (lower triangle used; overwritten)
// into w (ascending) and Zm.  Buffers: F (N*N complex doubles of space: the
// FP32 copies, later Q) and G (N*N complex doubles); all with leading
// dimension ld.
__device__ void jacobi_mixed(int N, int ld, double* A, double* Zm, double* w, double* shd, int* shi, double* F,
                             double* G) {
  const int half = (N + 1) / 2 + 1;
  double* red = shd + 4 * half;
  Cx<float>* Af = reinterpret_cast<Cx<float>*>(F);
  Cx<float>* Zf = Af + (size_t) ld * N;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    int i = e % N, j = e / N;
    Z a = i >= j ? AT(A, ld, i, j) : zconj(AT(A, ld, j, i));
    if (i == j) a.im = 0.0;
    if (i <= j) AT(A, ld, i, j) = a;   // complete the FP64 matrix as well
    AM(Af, i, j) = Cx<float>{(float) a.re, (float) a.im};
    AM(Zf, i, j) = Cx<float>{i == j ? 1.0f : 0.0f, 0.0f};
  }
  __syncthreads();
  // to where FP32 can no longer resolve the couplings
  jacobi_sweeps<float>(N, ld, Af, Zf, shd, shi, red, 1e-12f, 1e-12f, 30);
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const Cx<float> z = AM(Zf, e % N, e / N);
    AT(Zm, ld, e % N, e / N) = zmk((double) z.re, (double) z.im);
  }
  __syncthreads();
  // Q = Z (3I - Z^H Z) / 2 into F
  zgemm_cta(N, ld, Zm, true, Zm, G, true);
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    int i = e % N, j = e / N;
    Z g = AT(G, ld, i, j);
    AT(G, ld, i, j) = zmk((i == j ? 1.5 : 0.0) - 0.5 * g.re, -0.5 * g.im);
  }
  __syncthreads();
  zgemm_cta(N, ld, Zm, false, G, F, false);
  // A' = Q^H A Q, then the FP64 sweeps accumulate onto Q
  zgemm_cta(N, ld, A, false, F, G, false);
  zgemm_cta(N, ld, F, true, G, A, true);
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) AT(Zm, ld, e % N, e / N) = AT(F, ld, e % N, e / N);
  __syncthreads();
  jacobi_sweeps<double>(N, ld, reinterpret_cast<Cx<double>*>(A), reinterpret_cast<Cx<double>*>(Zm), shd, shi, red,
                        1e-32, 1e-30, 20);
  sort_eigen(N, ld, reinterpret_cast<Cx<double>*>(A), reinterpret_cast<Cx<double>*>(Zm), w, shi);
}

__global__ void k_heev(int N, double* a, double* zwork, double* w, int* info) {
  extern __shared__ double sm[];
  int half = (N + 1) / 2 + 1;
  double* A = a + (size_t) blockIdx.x * 2 * N * N;
  double* Zm = zwork + (size_t) blockIdx.x * 2 * N * N;
  jacobi_cta(N, N, A, Zm, w + (size_t) blockIdx.x * N, sm, reinterpret_cast<int*>(sm + 4 * half + 32), 60);
  for (size_t e = threadIdx.x; e < (size_t) N * N; e += blockDim.x)
    reinterpret_cast<Z*>(A)[e] = reinterpret_cast<Z*>(Zm)[e];
  if (threadIdx.x == 0 && info) info[blockIdx.x] = 0;
}

// odd leading dimension of the Ritz work matrices
__host__ __device__ inline int ritz_ld(int ns) { return ns | 1; }

// ------------------------------------------------------------------
// Rayleigh-Ritz from Gram matrices (see mx_internal.h)
// workspace per k: 5 * ns * ns complex doubles
// ------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_rayleigh_ritz(int ns, int m, const double* __restrict__ ga, const double* __restrict__ gm,
                                const int* __restrict__ sel, double drop, double theta_min, double* coef,
                                double* theta, int* info, double* work, int in_smem) {
  extern __shared__ double sm[];
  int k = blockIdx.x;
  int half = (ns + 1) / 2 + 1;
  double* shd = sm;                                  // jacobi rotation data: 4*half + 32
  double* d = shd + 4 * half + 32;                   // ns
  double* wv = d + ns;                               // ns
  double* rd = wv + ns;                              // ns
  int* shi = reinterpret_cast<int*>(rd + ns);        // 2*half
  int* idx = shi + 2 * half;                         // ns
  int* kept = idx + ns;                              // ns
  int* cnt = kept + ns;                              // 2
  const double* GA = ga + (size_t) k * 2 * ns * ns;
  const double* GM = gm + (size_t) k * 2 * ns * ns;
  // work matrices: in shared memory for the Ritz systems (ns <= 48), in
  // global memory for the coarse-grid eigenproblem
  // every work matrix has the odd leading dimension ld >= ns: a row of a
  // column-major matrix then falls into distinct shared-memory banks
  const int ld = ritz_ld(ns);
  const size_t msz = (size_t) 2 * ld * ns;           // doubles per work matrix
  double* W0;
  if (in_smem) {
    uintptr_t p0 = reinterpret_cast<uintptr_t>(cnt + 2);
    W0 = reinterpret_cast<double*>((p0 + 15) & ~(uintptr_t) 15);
  } else {
    W0 = work + (size_t) k * 5 * msz;
  }
  double* W1 = W0 + msz;                             // T = D R^-1
  double* W2 = W1 + msz;                             // G_A T, then projected A
  double* W3 = W2 + msz;                             // Jacobi eigenvectors
  double* GS = in_smem ? W3 + msz : nullptr;         // G_A on the selected columns
  // work of the mixed Jacobi: W0 (free once T is formed) and GS, or in global
  // memory a fifth matrix
  double* GB = in_smem ? GS : W3 + msz;
  if (threadIdx.x == 0) {
    int na = 0;
    for (int i = 0; i < ns; i++)
      if (!sel || sel[(size_t) k * ns + i]) idx[na++] = i;
    cnt[0] = na;
  }
  __syncthreads();
  int na = cnt[0];
  for (int i = threadIdx.x; i < na; i += blockDim.x) {
    double g = reinterpret_cast<const Z*>(GM)[(size_t) idx[i] * ns + idx[i]].re;
    d[i] = g > 0.0 ? 1.0 / sqrt(g) : 0.0;
  }
  __syncthreads();
  for (size_t e = threadIdx.x; e < (size_t) na * na; e += blockDim.x) {
    int i = (int) (e % na), j = (int) (e / na);
    Z g = reinterpret_cast<const Z*>(GM)[(size_t) idx[j] * ns + idx[i]];
    AT(W0, ld, i, j) = zscal(d[i] * d[j], g);
  }
  __syncthreads();
  // right-looking Cholesky with column dropping: W0 -> R (upper), kept flags,
  // the reciprocals of R's diagonal in rd
  for (int j = 0; j < na; j++) {
    if (threadIdx.x == 0) {
      const double piv = AT(W0, ld, j, j).re;
      const bool keep = piv > drop && d[j] > 0.0;
      kept[j] = keep;
      rd[j] = keep ? rsqrt(piv) : 0.0;
      AT(W0, ld, j, j) = zmk(piv * rd[j], 0.0);
    }
    __syncthreads();
    const bool keep = kept[j];
    const double rj = rd[j];
    for (int l = j + 1 + threadIdx.x; l < na; l += blockDim.x) AT(W0, ld, j, l) = zscal(rj, AT(W0, ld, j, l));
    __syncthreads();
    if (keep)
      for (int e = threadIdx.x; e < (na - j - 1) * (na - j - 1); e += blockDim.x) {
        int i = j + 1 + e % (na - j - 1), l = j + 1 + e / (na - j - 1);
        if (i <= l) AT(W0, ld, i, l) = zsub(AT(W0, ld, i, l), zcmul(AT(W0, ld, j, i), AT(W0, ld, j, l)));
      }
    __syncthreads();
  }
  // compact the kept indices
  if (threadIdx.x == 0) {
    int r = 0;
    for (int j = 0; j < na; j++)
      if (kept[j]) kept[r++] = j;
    cnt[1] = r;
  }
  __syncthreads();
  int r = cnt[1];
  if (r < m) {
    if (threadIdx.x == 0) info[k] = -1 - r;
    return;
  }
  // T (na x r) = D R[kept,kept]^-1: the rows from the last one up, each taken
  // out of the rows above it at once
  for (int e = threadIdx.x; e < na * r; e += blockDim.x) AT(W1, ld, e % na, e / na) = zmk(0.0, 0.0);
  __syncthreads();
  for (int c = threadIdx.x; c < r; c += blockDim.x) AT(W1, ld, kept[c], c) = zmk(1.0, 0.0);
  __syncthreads();
  for (int a = r - 1; a >= 0; a--) {
    const int ia = kept[a];
    const double ra = rd[ia];
    for (int c = a + threadIdx.x; c < r; c += blockDim.x) AT(W1, ld, ia, c) = zscal(ra, AT(W1, ld, ia, c));
    __syncthreads();
    const int nc = r - a;
    for (int e = threadIdx.x; e < a * nc; e += blockDim.x) {
      const int ib = kept[e / nc], c = a + e % nc;
      AT(W1, ld, ib, c) = zsub(AT(W1, ld, ib, c), zmul(AT(W0, ld, ib, ia), AT(W1, ld, ia, c)));
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < na * r; e += blockDim.x) {
    const int i = e % na;
    AT(W1, ld, i, e / na) = zscal(d[i], AT(W1, ld, i, e / na));
  }
  __syncthreads();
  // W3 <- G_A T  (na x r), then W2 <- T^H W3 (r x r)
  if (GS) {
    for (size_t e = threadIdx.x; e < (size_t) na * na; e += blockDim.x) {
      int i = (int) (e % na), l = (int) (e / na);
      AT(GS, ld, i, l) = reinterpret_cast<const Z*>(GA)[(size_t) idx[l] * ns + idx[i]];
    }
    __syncthreads();
  }
  for (size_t e = threadIdx.x; e < (size_t) na * r; e += blockDim.x) {
    int i = (int) (e % na), c = (int) (e / na);
    Z s = zmk(0.0, 0.0);
    if (GS)
      for (int l = 0; l < na; l++) s = zadd(s, zmul(AT(GS, ld, i, l), AT(W1, ld, l, c)));
    else
      for (int l = 0; l < na; l++)
        s = zadd(s, zmul(reinterpret_cast<const Z*>(GA)[(size_t) idx[l] * ns + idx[i]], AT(W1, ld, l, c)));
    AT(W3, ld, i, c) = s;
  }
  __syncthreads();
  // (Hermitian: the lower triangle, which jacobi_mixed completes)
  for (int e = threadIdx.x; e < r * (r + 1) / 2; e += blockDim.x) {
    int a = (int) ((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
    while (a * (a + 1) / 2 > e) a--;
    while ((a + 1) * (a + 2) / 2 <= e) a++;
    const int c = e - a * (a + 1) / 2;
    Z s = zmk(0.0, 0.0);
    for (int l = 0; l < na; l++) s = zadd(s, zcmul(AT(W1, ld, l, a), AT(W3, ld, l, c)));
    AT(W2, ld, a, c) = s;
  }
  __syncthreads();
  jacobi_mixed(r, ld, W2, W3, wv, shd, shi, W0, GB);
  // Ritz values at or below theta_min are spurious (null-space) modes and
  // are passed over, as exp_bloch2d.c:546-551 does for its coarse start
  if (threadIdx.x == 0) {
    int f = 0;
    while (f < r && !(wv[f] > theta_min)) f++;
    cnt[0] = f;
  }
  __syncthreads();
  int first = cnt[0];
  if (r - first < m) {
    if (threadIdx.x == 0) info[k] = -1 - (r - first);
    return;
  }
  for (size_t e = threadIdx.x; e < (size_t) ns * m; e += blockDim.x) {
    int i = (int) (e % ns), j = (int) (e / ns);
    reinterpret_cast<Z*>(coef)[(size_t) k * ns * m + (size_t) j * ns + i] = zmk(0.0, 0.0);
  }
  __syncthreads();
  for (size_t e = threadIdx.x; e < (size_t) na * m; e += blockDim.x) {
    int i = (int) (e % na), j = (int) (e / na);
    Z s = zmk(0.0, 0.0);
    for (int l = 0; l < r; l++) s = zadd(s, zmul(AT(W1, ld, i, l), AT(W3, ld, l, first + j)));
    reinterpret_cast<Z*>(coef)[(size_t) k * ns * m + (size_t) j * ns + idx[i]] = s;
  }
  for (int j = threadIdx.x; j < m; j += blockDim.x) theta[(size_t) k * m + j] = wv[first + j];
  if (threadIdx.x == 0) info[k] = r;
}

size_t jacobi_smem(int N) {
  int half = (N + 1) / 2 + 1;
  return sizeof(double) * (4 * half + 32) + sizeof(int) * 2 * half;
}

}  // namespace

extern "C" int mxk_hpd_inverse(int N, int K, double* a, int* info, mx_stream s) {
  const size_t smem = sweep_smem(N);
  // The sweep for orders up to 160, but not where small matrices outnumber the
  // SMs: a warp takes a column of theirs, and the FP64 unit, which all of an
  // SM's matrices share, works for idle lanes (Gauss-Jordan against sweep, us:
  // 300 matrices of order 16 51 / 64, of 32 164 / 171, of 48 445 / 446; 3000 of
  // 8 88 / 138, of 32 1300 / 1430; 64 of 32 125 / 102).
  if (smem <= 208 * 1024 && !(N <= 32 && K > 152)) {
    allow_smem(k_hpd_inverse_sweep);
    k_hpd_inverse_sweep<<<K, SWT, smem, (cudaStream_t) s>>>(N, a, info);
  } else {
    k_hpd_inverse<<<K, DT, 2 * N * sizeof(Z), (cudaStream_t) s>>>(N, a, info);
  }
  MX_CHECK_LAUNCH();
  return 0;
}

template <typename S, typename R, typename MS>
static int L_coarse_apply(int N, int m, int K, const void* ainv, const void* x, void* y, cudaStream_t st) {
  dim3 g((unsigned) (((size_t) N * m + 127) / 128), K);
  k_coarse_apply<S, R, MS><<<g, 128, 0, st>>>(N, m, (const MS*) ainv, (const S*) x, (S*) y);
  MX_CHECK_LAUNCH();
  return 0;
}

extern "C" int mxk_coarse_apply(int N, int m, int K, const double* ainv, const void* ainv_c64, int prec,
                                const void* x, void* y, mx_stream s) {
  cudaStream_t st = (cudaStream_t) s;
  if (prec == MX_C64) {
    if (ainv_c64) return L_coarse_apply<float2, float, float2>(N, m, K, ainv_c64, x, y, st);
    return L_coarse_apply<float2, float, double2>(N, m, K, ainv, x, y, st);
  }
  if (prec == MX_C128) return L_coarse_apply<double2, double, double2>(N, m, K, ainv, x, y, st);
  return L_coarse_apply<cdd, dd, double2>(N, m, K, ainv, x, y, st);
}

extern "C" int mxk_heev(int N, int K, double* a, double* zwork, double* w, int* info, mx_stream s) {
  k_heev<<<K, DT, jacobi_smem(N), (cudaStream_t) s>>>(N, a, zwork, w, info);
  MX_CHECK_LAUNCH();
  return 0;
}

extern "C" size_t mxk_ritz_work_doubles(int ns) { return (size_t) 10 * ritz_ld(ns) * ns; }

extern "C" int mxk_rayleigh_ritz(int ns, int m, int K, const double* ga, const double* gm, const int* sel,
                                 double drop, double theta_min, double* coef, double* theta, int* info,
                                 double* work, mx_stream s) {
  size_t smem = jacobi_smem(ns) + sizeof(int) * (2 * ns + 4) + sizeof(double) * (3 * ns + 2);
  int in_smem = ns <= 48;
  if (in_smem) smem += 16 + sizeof(double) * 2 * (size_t) ritz_ld(ns) * ns * 5;
  if (smem > 48 * 1024) allow_smem(k_rayleigh_ritz);   // (the rotation data alone from order 939 on)
  int threads = in_smem ? 512 : 1024;
  k_rayleigh_ritz<<<K, threads, smem, (cudaStream_t) s>>>(ns, m, ga, gm, sel, drop, theta_min, coef, theta, info,
                                                         work, in_smem);
  MX_CHECK_LAUNCH();
  return 0;
}

// ------------------------------------------------------------------
// The lowest eigenpairs of the coarse pencil (A, M), A = C^H D^2 C with the
// cell curls C (nc = n0^2 rows) and D^2 = n0^2 kappa >= 0.  The nonzero
// eigenvalues of M^-1 A are those of the nc x nc Hermitian matrix
//   B = D C M^-1 C^H D,   e = M^-1 C^H D y / sqrt(lambda) M-normalised,
// half the order of the edge matrices, and M^-1 is known: M couples the
// x-edges of a column (the y-edges of a row) as (1, 4, 1) / 6 on a line
// closed by the Bloch factor f, whose Green's function is
//   G(d) = sqrt(3) (r^d / (1 - conj(f) r^n) + f r^(n-d) / (1 - f r^n)),
//   0 <= d < n, r = sqrt(3) - 2, G(d - n) = conj(f) G(d).
// Hence B(c, c') = D_c D_c' (same column: Hy(j - j') + same row: Hx(i - i')),
// H(d) = 2 G(d) - G(d-1) - G(d+1) = 6 (G(d) - [d = 0]).
// A CTA per k-point; its matrices lie in shared memory up to nc = 64 (but for
// one product), and the eigenvectors are written as the level-0 block.  8
// k-points, n0 = 8: 4.6 ms against 54 ms for the pencil of order 128.
// ------------------------------------------------------------------
namespace {
__device__ __forceinline__ Z green(const Z* G, Z f, int n, int d) {
  return d < 0 ? zcmul(f, G[d + n]) : G[d];
}

template <typename S>
__global__ void __launch_bounds__(512) k_coarse_pairs(int n, int m, int K, const double* __restrict__ ph,
                                                    const double* __restrict__ kappa, double* work, int in_smem,
                                                    S* __restrict__ E, double* __restrict__ mu, int* info) {
  extern __shared__ __align__(16) double smp[];
  const int k = blockIdx.x, nc = n * n, half = (nc + 1) / 2 + 1, ld = ritz_ld(nc);
  const size_t msz = (size_t) 2 * ld * nc;
  double* M0 = in_smem ? smp : work + (size_t) k * 4 * msz;
  double *A = M0, *Zm = M0 + msz, *F = M0 + 2 * msz;
  double* G = in_smem ? work + (size_t) k * msz : M0 + 3 * msz;
  double* shd = in_smem ? smp + 3 * msz : smp;
  double* w = shd + 4 * half + 32;
  double* D = w + nc;
  Z* Gx = reinterpret_cast<Z*>(D + nc);   // (nc is even: 16-byte aligned)
  Z* Gy = Gx + n;
  int* shi = reinterpret_cast<int*>(Gy + n);
  __shared__ int first_s;
  const Seam<double> seam = seam_load<double>(ph, K, k, n);
  const Z fx = zmk(seam.xf.re, seam.xf.im), fy = zmk(seam.yf.re, seam.yf.im);
  const double s3 = sqrt(3.0), r = s3 - 2.0;
  if (threadIdx.x < 2 * n) {
    const int d = threadIdx.x % n;
    const Z f = threadIdx.x < n ? fx : fy;
    double rd = 1.0, rn = 1.0, rnd = 1.0;   // r^d, r^n, r^(n-d)
    for (int q = 0; q < n; q++) {
      rn *= r;
      if (q < d) rd *= r;
      if (q < n - d) rnd *= r;
    }
    const Z a = zdiv(zmk(rd, 0.0), zmk(1.0 - f.re * rn, f.im * rn));
    const Z b = zdiv(zscal(rnd, f), zmk(1.0 - f.re * rn, -f.im * rn));
    (threadIdx.x < n ? Gx : Gy)[d] = zscal(s3, zadd(a, b));
  }
  for (int c = threadIdx.x; c < nc; c += blockDim.x) D[c] = n * sqrt(kappa[c]);
  __syncthreads();
  for (int e = threadIdx.x; e < nc * nc; e += blockDim.x) {
    const int c = e % nc, q = e / nc, i = c % n, j = c / n, i2 = q % n, j2 = q / n;
    Z b = zmk(0.0, 0.0);
    if (i == i2) b = zadd(b, green(Gy, fy, n, j - j2));
    if (j == j2) b = zadd(b, green(Gx, fx, n, i - i2));
    if (c == q) b.re -= 2.0;
    AT(A, ld, c, q) = zscal(6.0 * D[c] * D[q], b);
  }
  __syncthreads();
  jacobi_mixed(nc, ld, A, Zm, w, shd, shi, F, G);
  // pass over the zero eigenvalues (exp_bloch2d.c:546-551)
  if (threadIdx.x == 0) {
    int f = 0;
    while (f < nc && fabs(w[f]) < 1e-8) f++;
    first_s = f;
    info[k] = f + m <= nc ? 0 : -1;
  }
  __syncthreads();
  const int first = first_s;
  if (first + m > nc) return;
  Lay L{n, m, K};
  for (int e = threadIdx.x; e < 2 * nc * m; e += blockDim.x) {
    const int v = e % m, site = e / m % nc, p = e / (m * nc), i = site % n, j = site / n, col = first + v;
    Z s = zmk(0.0, 0.0);
    for (int q = 0; q < n; q++) {
      // column i, row q of the cells for x-edges; column q, row j for y-edges
      const int c = p == 0 ? q * n + i : j * n + q;
      const Z g = p == 0 ? zsub(green(Gy, fy, n, j - q), green(Gy, fy, n, j - q - 1))
                         : zsub(green(Gx, fx, n, i - q - 1), green(Gx, fx, n, i - q));
      s = zadd(s, zmul(g, zscal(D[c], AT(Zm, ld, c, col))));
    }
    const double sc = rsqrt(w[col]);
    Store<S, double>::st(E + L.edge(k, p, j, i, v), mkc(sc * s.re, sc * s.im));
  }
  for (int v = threadIdx.x; v < m; v += blockDim.x) mu[(size_t) k * m + v] = 1.0 + w[first + v];
}
}  // namespace

extern "C" size_t mxk_coarse_pairs_work_doubles(int n) {
  return (size_t) 2 * ritz_ld(n * n) * n * n * (n <= 8 ? 1 : 4);
}

extern "C" int mxk_coarse_pairs(int n, int m, int K, const double* ph, const double* kappa, double* work, int prec_e,
                                void* E, double* mu, int* info, mx_stream s) {
  if (n < 4 || (n & 1)) return (int) cudaErrorInvalidValue;
  const int nc = n * n, half = (nc + 1) / 2 + 1, in_smem = n <= 8;
  const size_t smem = sizeof(double) * (4 * half + 32 + 2 * nc + 4 * n + (in_smem ? (size_t) 6 * ritz_ld(nc) * nc : 0))
                      + sizeof(int) * 2 * half;
  if (prec_e == MX_CDD) {
    allow_smem(k_coarse_pairs<cdd>);
    k_coarse_pairs<cdd><<<K, 512, smem, (cudaStream_t) s>>>(n, m, K, ph, kappa, work, in_smem, (cdd*) E, mu, info);
  } else if (prec_e == MX_C128) {
    allow_smem(k_coarse_pairs<double2>);
    k_coarse_pairs<double2><<<K, 512, smem, (cudaStream_t) s>>>(n, m, K, ph, kappa, work, in_smem, (double2*) E, mu,
                                                                info);
  } else return (int) cudaErrorInvalidValue;
  MX_CHECK_LAUNCH();
  return 0;
}

// ------------------------------------------------------------------
// Cholesky-QR coefficients: for the Hermitian positive definite mass Gram
// G = X^H M X of m vectors, G = R^H R with R upper triangular and a positive
// real diagonal, and coef = R^{-1}; X coef is then M-orthonormal and its
// first j columns span the first j columns of X (the function of the
// reference's Householder orthonormalisation, orthonormalize_edge2d,
// edge2d.c:6264-6296).  info[k] = 0, or j+1 if column j is (numerically)
// dependent on the columns before it.
// ------------------------------------------------------------------
namespace {
__global__ void k_chol_qr_coef(int m, const double* __restrict__ gm, double* __restrict__ coef, int* info) {
  extern __shared__ double smc[];
  Z* R = reinterpret_cast<Z*>(smc);          // m x m column-major
  __shared__ int bad;
  const double* G = gm + (size_t) blockIdx.x * 2 * m * m;
  double* C = coef + (size_t) blockIdx.x * 2 * m * m;
  for (int e = threadIdx.x; e < m * m; e += blockDim.x) R[e] = reinterpret_cast<const Z*>(G)[e];
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int j = 0; j < m; j++) {
    // row j of R: R_jj = sqrt(G_jj - sum |R_ij|^2), R_jc = (G_jc - sum conj(R_ij) R_ic) / R_jj
    __shared__ double djj;
    if (threadIdx.x == 0) {
      double g = R[j * m + j].re, d = g;
      for (int i = 0; i < j; i++) d -= zabs2(R[j * m + i]);
      // column j counts as dependent when the part of it outside the span
      // of the columns before it has less than 1e-5 of its M-norm
      if (!(d > 1e-10 * g) && !bad) bad = j + 1;
      djj = d > 0.0 ? sqrt(d) : 1.0;
    }
    __syncthreads();
    for (int c = j + 1 + threadIdx.x; c < m; c += blockDim.x) {
      Z s = R[c * m + j];
      for (int i = 0; i < j; i++) s = zsub(s, zcmul(R[j * m + i], R[c * m + i]));
      R[c * m + j] = zscal(1.0 / djj, s);
    }
    __syncthreads();
    if (threadIdx.x == 0) R[j * m + j] = zmk(djj, 0.0);
    __syncthreads();
  }
  // coef = R^{-1}, one column per thread (back substitution)
  for (int c = threadIdx.x; c < m; c += blockDim.x) {
    for (int i = m - 1; i > c; i--) AT(C, m, i, c) = zmk(0.0, 0.0);
    AT(C, m, c, c) = zmk(1.0 / R[c * m + c].re, 0.0);
    for (int i = c - 1; i >= 0; i--) {
      Z s = zmk(0.0, 0.0);
      for (int q = i + 1; q <= c; q++) s = zadd(s, zmul(R[q * m + i], AT(C, m, q, c)));
      AT(C, m, i, c) = zscal(-1.0 / R[i * m + i].re, s);
    }
  }
  if (threadIdx.x == 0 && info) info[blockIdx.x] = bad;
}
}  // namespace

extern "C" int mxk_chol_qr_coef(int m, int K, const double* gm, double* coef, int* info, mx_stream s) {
  if (m < 1 || m > 64) return (int) cudaErrorInvalidValue;
  size_t smem = sizeof(double) * 2 * (size_t) m * m;
  allow_smem(k_chol_qr_coef);
  k_chol_qr_coef<<<K, 64, smem, (cudaStream_t) s>>>(m, gm, coef, info);
  MX_CHECK_LAUNCH();
  return 0;
}
