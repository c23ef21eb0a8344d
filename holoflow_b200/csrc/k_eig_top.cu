// The r largest eigenpairs of a batch of symmetric n x n float64 matrices (n <= 128, r <= 16).
//
// The clutter filter W = (I - V_r V_r^T) D needs only the top clutter_rank eigenvectors of each
// window's Gram matrix, and the full cyclic Jacobi solve (k_pca.cu) spends O(n^3) shared-memory
// traffic per sweep over ~11 sweeps.  Here one CTA per matrix (128, 256 or 512 threads for n up to 32,
// 64 or 128) runs:
//  1. Householder reduction to tridiagonal form, A = Q T Q^T (Golub & Van Loan, Matrix
//     Computations, 4th ed., Alg. 8.3.1), with the matrix in registers: a half-warp per four rows, a
//     thread holding n / 16 columns of them.  Two barriers per step: p = beta A v (the four rows' sums
//     are reduced and scattered over the half-warp together) with per-warp partials of p^T v; then the
//     rank-2 update, after which the half-warp of row k + 1 builds the next house vector from its
//     registers and writes it where the back-transformation reads it;
//  2. the r largest eigenvalues of T by Sturm-sequence multisection (Wilkinson): a warp evaluates 32
//     shifts at once and the bracket shrinks 33x per round (four chains per lane take 8 rounds for 11,
//     but twice the time: the FP64 pipe takes a warp's instruction every two cycles);
//  3. their eigenvectors of T by inverse iteration (Wilkinson): two solves with the tridiagonal
//     LU factorisation of T - lambda I with partial pivoting, pivots floored at eps ||T||, from
//     distinct starting vectors, orthonormalised (modified Gram-Schmidt) within clusters of close
//     eigenvalues after each solve;
//  4. back-transformation V_r = Q Y by the reflectors in reverse order, four per step, a warp per
//     column.
// Bound: one CTA on one SM.  A step's vectors cross shared memory, whose 128 bytes per cycle every
// thread shares: with four threads per row, each reading whole quarters of v and p, those reads alone
// took 800 (n = 64) to 3000 (n = 128) cycles per step; 4 x (n / 16) tiles read a third of that.  The
// rest is latency: dependent FP64 operations (9 cycles), shuffles, barriers.  So the library's square
// root and two divisions per house vector became float-seeded third-order Newton steps (the matrix is
// scaled to entries below 1), sums run pairwise, independent chains run side by side, values a chain
// needs are loaded ahead of it, and finished rows and columns are skipped.
// Measured, 8 matrices, r = 4, before -> now: n = 32 86 -> 50 us, 64 172 -> 99, 128 396 -> 254 (at n = 64:
// reduction 51 us, eigenvalues 14, factors and inverse iteration 20, back-transformation 6).
// Accuracy: two solves per eigenvector (one with lambda to the rounding of ||T|| gains about 1e15; a third
// changed no residual) and brackets that stop at 2^-54 ||T|| (the reduction has perturbed T by more).
// Over Gram, decaying, cluttered and clustered spectra of n = 8 .. 128, r = 4, the residuals
// ||A v - lambda v|| / ||A|| are 2.9e-16 .. 7.2e-16 in the median of a kind and at most 1.8e-15; the
// shared-memory kernel before, with three solves, brackets relative to lambda and the library's square roots
// and divisions, had 2.1e-16 .. 6.5e-16 and at most 2.0e-15.  The eigenvalues' errors agree (at most
// 5.3e-15 ||A|| for both), and the filter matrix made from them is float32.
// The eigenvalues ascend in evals[n - r .. n - 1] and the vectors go to the matching columns of
// evecs ([n][n], column = eigenvalue index, as the Jacobi solver lays them out); the other entries
// are not written.  info = 0, or 1 when the input is not finite.
#include <cfloat>

#include "k_pca.cuh"

namespace hf {

namespace {

constexpr int kEigMaxN = 128;
constexpr int kEigMaxR = 16;
constexpr int kEigRed  = 20; // reduction slots (up to 16 warps)

// Stride of the per-eigenvalue vectors, = 1 (mod 16) doubles, so the lanes of the inverse iteration
// (one per eigenvalue, r <= 16) address distinct bank pairs.
__host__ __device__ inline int eig_ldy(int n) { return 16 * ((n + 15) / 16) + 1; }
// Threads of a CTA: a half-warp per four rows.
__host__ __device__ inline int eig_threads(int n) { return n <= 32 ? 128 : (n <= 64 ? 256 : 512); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Number of eigenvalues of the tridiagonal (d, e) below x: sign changes of the leading minors
// p_j = (d_j - x) p_(j-1) - e_(j-1)^2 p_(j-2) of T - x I.  T is scaled to ||T|| < 1, |d_j - x| is kept at
// or above 2^-60 and e2 at or above 2^-120 (perturbations far below the rounding of T), so four steps
// change a minor by less than 2^+-301 relative to the pair before them: the pair is rescaled by 2^+-300
// between groups of four and no sign is lost.  Zero counts as positive: the minor after a zero has the
// sign opposite to the one before it, so the pair still counts one change.
__device__ __forceinline__ int sturm_count(const double *d, const double *e2, int n, double x) {
  double p = d[0] - x, pm = 1.0;
  int    cnt = (unsigned)__double2hiint(p) >> 31;
  double dj[4], ej[4]; // (the arrays hold eight entries beyond n)
#pragma unroll
  for (int jj = 0; jj < 4; ++jj)
    dj[jj] = d[1 + jj], ej[jj] = e2[jj];
  for (int j0 = 1; j0 < n; j0 += 4) {
    double dn[4], en[4]; // the next group's entries, loaded ahead of the chain
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
      dn[jj] = d[j0 + 4 + jj], en[jj] = e2[j0 + 3 + jj];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      double    dx = dj[jj] - x;
      const int hi = __double2hiint(dx);
      if ((hi & 0x7FFFFFFF) < 0x3C300000) // |dx| < 2^-60
        dx = __hiloint2double((hi & 0x80000000) | 0x3C300000, 0);
      const double q = fma(dx, p, -(ej[jj] * pm));
      cnt += (unsigned)(__double2hiint(q) ^ __double2hiint(p)) >> 31;
      pm = p;
      p  = q;
    }
    // by the larger exponent: above 2^300 or below 2^-300
    const int    ex = max(__double2hiint(p) & 0x7FF00000, __double2hiint(pm) & 0x7FF00000);
    const double f =
        __hiloint2double(ex > (1323 << 20) ? (723 << 20) : (ex < (723 << 20) ? (1323 << 20) : (1023 << 20)), 0);
    p *= f;
    pm *= f;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
      dj[jj] = dn[jj], ej[jj] = en[jj];
  }
  return cnt;
}

// Hardware approximations (relative error below 2^-21) that seed the Newton steps.
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 1 / sqrt(t) and 1 / t for t in the normal float range, to double precision: a float32 seed
// (relative error below 2^-21) and one third-order Newton step, e -> O(e^3).
__device__ __forceinline__ double rsqrt_seeded(double t, float seed) {
  const double y = (double)seed, a = t * y, e = fma(-a, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double rcp_seeded(double t, float seed) {
  const double r = (double)seed, e = fma(-t, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

__device__ __forceinline__ double reciprocal(double x) {
  return fabs(x) > 1e-30 && fabs(x) < 1e30 ? rcp_seeded(x, rcp_approx((float)x)) : 1.0 / x;
}

template <int NT, int PER_SM>
__global__ void __launch_bounds__(NT, PER_SM) eig_top_kernel(const double *a_in, double *evecs, double *evals, int *info,
                                                        int n, int r) {
  constexpr int kWarps = NT / 32;
  constexpr int RM     = NT / 4;          // rows the CTA can hold
  constexpr int M      = RM / 32;         // column pairs per thread: columns 2 tc, 2 tc + 1 (+ 32 m)
  constexpr int NC     = RM / 32;         // entries of a vector per lane
  extern __shared__ __align__(16) double esm[];
  double   *R    = esm;                   // [n][RM] house vectors, zero up to their own index
  double   *pw   = R + n * RM;            // [RM] p = beta A v
  double   *beta = pw + RM;               // [n]
  double   *d    = beta + n;              // [n] diagonal of T
  double   *e    = d + n;                 // [n] subdiagonal of T (e[n-1] = 0)
  double   *e2   = e + n;                 // [n + 8] e^2, scaled by sc^2
  double   *ds   = e2 + n + 8;            // [n + 8] d, scaled by sc (||T|| sc <= 1)
  double   *lam  = ds + n + 8;            // [kEigMaxR] eigenvalues, descending
  const int ldy  = eig_ldy(n);            // per-vector stride: lane t's entries in bank pair t
  double   *Y    = lam + kEigMaxR;        // [kEigMaxR][ldy] eigenvectors of T, then of A
  double   *lu   = Y + kEigMaxR * ldy;    // [4][kEigMaxR][ldy] LU factors of each shift
  double   *red  = lu + 4 * kEigMaxR * ldy; // [kEigRed] reductions and scalars

  const int     tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int     i0 = 4 * (tid >> 4), tc = lane & 15; // the half-warp's first row; this thread's columns
  const double *src = a_in + (int64_t)blockIdx.x * n * n;
  double        a[4][2 * M], big = 0.0; // symmetric part, and its largest magnitude
  bool          finite = true;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int c = 0; c < 2 * M; ++c) {
      const int i = i0 + q, j = 2 * tc + (c & 1) + 32 * (c >> 1);
      a[q][c]     = i < n && j < n ? 0.5 * (src[i * n + j] + src[j * n + i]) : 0.0;
      finite      = finite && isfinite(a[q][c]);
      big         = fmax(big, fabs(a[q][c]));
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (lane == 0)
    red[warp] = big;
  if (__syncthreads_or(!finite)) { // not finite: report, leave the outputs alone
    if (tid == 0 && info != nullptr)
      info[blockIdx.x] = 1;
    return;
  }
  // scale by a power of two to a largest entry in [1/2, 1): exact, and the house vectors' squared
  // norms stay in the float range that seeds their square roots
  big = red[0];
#pragma unroll
  for (int q = 1; q < kWarps; ++q)
    big = fmax(big, red[q]);
  int ex = 0;
  frexp(big, &ex);
  {
    const double f1 = ldexp(1.0, -ex / 2), f2 = ldexp(1.0, -ex - (-ex / 2));
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 2 * M; ++c)
        a[q][c] = a[q][c] * f1 * f2;
  }

  // ---- 1. Householder tridiagonalisation ------------------------------------------------------
  // House vector of step k by the half-warp of row k, from the entries x beyond the diagonal:
  // v = x + sign(x_0) ||x|| e_0, beta = 2 / v^T v = 1 / (t + |x_0| ||x||) with t = ||x||^2.
  const auto house = [&](int k) {
    const unsigned half = 0xFFFFu << (lane & 16);
    double         x[2 * M], sa = 0.0, sb = 0.0, xs = 0.0, xd = 0.0;
#pragma unroll
    for (int c = 0; c < 2 * M; ++c) {
      const int j = 2 * tc + (c & 1) + 32 * (c >> 1);
      x[c] = (k & 2) ? ((k & 1) ? a[3][c] : a[2][c]) : ((k & 1) ? a[1][c] : a[0][c]);
      xs   = j == k + 1 ? x[c] : xs; // the owner of entry k + 1 / k
      xd   = j == k ? x[c] : xd;
      x[c] = j > k + 1 ? x[c] : 0.0;
      if (c & 1)
        sb = fma(x[c], x[c], sb);
      else
        sa = fma(x[c], x[c], sa);
    }
    const double x0 = __shfl_sync(half, xs, (lane & 16) + (((k + 1) & 31) >> 1));
    double       s  = sa + sb;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
      s += __shfl_xor_sync(half, s, o);
    double v0 = 0.0, b = 0.0, alpha = x0;
    if (s > 0.0) {
      const double t = fma(x0, x0, s);
      double       mu;
      if (t > 1e-30) { // t <= n: in the float range
        const float tf = (float)t, yf = rsqrt_approx(tf);
        mu = t * rsqrt_seeded(t, yf);
        b  = rcp_seeded(fma(fabs(x0), mu, t), rcp_approx(fmaf(fabsf((float)x0), tf * yf, tf)));
      } else {
        mu = sqrt(t);
        b  = 1.0 / fma(fabs(x0), mu, t);
      }
      if (isfinite(b)) { // (a norm whose square underflows leaves the row as it is: v = 0, H = I)
        v0    = x0 + copysign(mu, x0);
        alpha = -copysign(mu, x0);
      } else {
        b = 0.0;
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int j  = 2 * tc + 32 * m;
      double2   vv = b != 0.0 ? make_double2(x[2 * m], x[2 * m + 1]) : make_double2(0.0, 0.0);
      vv.x = j == k + 1 ? v0 : vv.x;
      vv.y = j + 1 == k + 1 ? v0 : vv.y;
      *reinterpret_cast<double2 *>(R + k * RM + j) = vv;
    }
    if (tc == ((k & 31) >> 1)) {
      beta[k] = b;
      d[k]    = xd;
      e[k]    = alpha;
    }
  };
  const int ip = i0 + ((lane >> 2) & 3); // the row whose p this lane ends up with
  if (i0 == 0 && n >= 3)
    house(0);
  __syncthreads();
  for (int k = 0; k + 2 < n; ++k) {
    const double  b = beta[k], *v = R + k * RM;
    const bool    live = 8 * warp + 7 > k; // the warp has unfinished rows
    const double  vi = v[ip];
    double        s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (live && 32 * m + 31 > k) { // v is zero up to entry k
        const double2 vv = *reinterpret_cast<const double2 *>(v + 2 * tc + 32 * m);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          s[q] = fma(a[q][2 * m + 1], vv.y, fma(a[q][2 * m], vv.x, s[q]));
      }
    // sums over the half-warp: lanes with bit 3 keep rows 2, 3, then bit 2 picks one of the two
    const bool   b3 = lane & 8, b2 = lane & 4;
    const double u0 = (b3 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, b3 ? s[0] : s[2], 8);
    const double u1 = (b3 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, b3 ? s[1] : s[3], 8);
    double       pi = (b2 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b2 ? u0 : u1, 4);
    pi += __shfl_xor_sync(0xffffffffu, pi, 2);
    pi += __shfl_xor_sync(0xffffffffu, pi, 1);
    pi = ip > k ? b * pi : 0.0; // the finished rows take no update
    if ((lane & 3) == 0)
      pw[ip] = pi;
    double pv = pi * vi; // the warp's eight rows
    pv += __shfl_xor_sync(0xffffffffu, pv, 4);
    pv += __shfl_xor_sync(0xffffffffu, pv, 8);
    pv += __shfl_xor_sync(0xffffffffu, pv, 16);
    if (lane == 0)
      red[warp] = pv;
    __syncthreads();
    // A' = A - v p^T - p v^T + kk v v^T with kk = beta p^T v, that is A - v p^T - (p - kk v) v^T
    if (live) {
      double dp[kWarps];
#pragma unroll
      for (int q = 0; q < kWarps; ++q)
        dp[q] = red[q];
#pragma unroll
      for (int h = kWarps / 2; h > 0; h >>= 1)
#pragma unroll
        for (int q = 0; q < h; ++q)
          dp[q] += dp[q + h];
      const double  kk = b * dp[0];
      const double2 va = *reinterpret_cast<const double2 *>(v + i0), vb = *reinterpret_cast<const double2 *>(v + i0 + 2);
      const double2 pa = *reinterpret_cast<const double2 *>(pw + i0), pb = *reinterpret_cast<const double2 *>(pw + i0 + 2);
      const double  vr[4] = {va.x, va.y, vb.x, vb.y};
      const double  pk[4] = {fma(-kk, va.x, pa.x), fma(-kk, va.y, pa.y), fma(-kk, vb.x, pb.x), fma(-kk, vb.y, pb.y)};
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (32 * m + 31 > k) {
          const double2 vv = *reinterpret_cast<const double2 *>(v + 2 * tc + 32 * m);
          const double2 pp = *reinterpret_cast<const double2 *>(pw + 2 * tc + 32 * m);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            a[q][2 * m]     = fma(-pk[q], vv.x, fma(-vr[q], pp.x, a[q][2 * m]));
            a[q][2 * m + 1] = fma(-pk[q], vv.y, fma(-vr[q], pp.y, a[q][2 * m + 1]));
          }
        }
      if (i0 == ((k + 1) & ~3) && k + 3 < n)
        house(k + 1);
    }
    __syncthreads();
  }
  // the last two rows
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int c = 0; c < 2 * M; ++c) {
      const int i = i0 + q, j = 2 * tc + (c & 1) + 32 * (c >> 1);
      if (i < n && i >= n - 2 && j == i)
        d[i] = a[q][c];
      if (i < n && i >= n - 2 && j == i + 1 && j < n)
        e[i] = a[q][c];
    }
  if (tid == 0)
    e[n - 1] = 0.0;
  __syncthreads();
    // Gershgorin bounds and ||T|| (warp 0)
  if (warp == 0) {
    double lo = DBL_MAX, hi = -DBL_MAX, nrm = 0.0;
    for (int i = lane; i < n; i += 32) {
      const double rad = fabs(e[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0);
      lo               = fmin(lo, d[i] - rad);
      hi               = fmax(hi, d[i] + rad);
      nrm              = fmax(nrm, fabs(d[i]) + rad);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo  = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi  = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
    }
    if (lane == 0) {
      const double pad = 2.0 * DBL_EPSILON * nrm + DBL_MIN;
      int          ex  = 0;
      frexp(nrm, &ex);
      red[0] = lo - pad;
      red[1] = hi + pad;
      red[2] = nrm;
      red[3] = nrm > 0.0 ? ldexp(1.0, -ex) : 1.0; // sc: a power of two with ||T|| sc < 1
    }
  }
  __syncthreads();
  const double sc = red[3];
  // the Sturm sequences run on T sc (exactly scaled), padded to whole groups of four by steps that
  // change no sign
  for (int i = tid; i < n + 8; i += NT) {
    const double es = i + 1 < n ? e[i] * sc : 0.0;
    ds[i]           = i < n ? d[i] * sc : 2.0;
    e2[i]           = i + 1 < n ? fmax(es * es, 0x1p-120) : 0.0;
  }
  __syncthreads();

  // ---- 2. eigenvalues n-1, n-2, ..., n-r by multisection, a warp each: 32 shifts per round, until
  //         the bracket is below the rounding of ||T|| ---------------------------------------------
  for (int t = warp; t < r; t += kWarps) {
    const int idx = n - 1 - t; // ascending index: count(a) <= idx < count(b)
    double    a = red[0] * sc, b = red[1] * sc;
    for (int round = 0; round < 24; ++round) {
      const double   w = (b - a) * (1.0 / 33.0);
      const int      c = sturm_count(ds, e2, n, fma(w, (double)(lane + 1), a));
      const unsigned m = __ballot_sync(0xffffffffu, c > idx);
      const int      f = m ? __ffs(m) - 1 : 32; // the first shift with more than idx eigenvalues below
      const double   na = f == 0 ? a : fma(w, (double)f, a);
      const double   nb = f == 32 ? b : fma(w, (double)(f + 1), a);
      a                 = na;
      b                 = nb;
      if (b - a <= fmax(2.0 * DBL_EPSILON * fmax(fabs(a), fabs(b)), 0x1p-54))
        break;
    }
    if (lane == 0)
      lam[t] = 0.5 * (a + b) * (1.0 / sc); // 1 / sc is a power of two: exact
  }
  __syncthreads();

  // ---- 3. eigenvectors of T by inverse iteration: eigenvalue t in warp t % kWarps, whose lane 0 runs
  //         the LU factorisation and the solves while the warp normalises; close eigenvalues are
  //         orthogonalised in descending order between block barriers ----------------------------
  {
    const double  nrm  = red[2];
    const double  tiny = DBL_EPSILON * nrm + DBL_MIN; // pivot floor
    const double  clus = 1e-7 * nrm + 8.0 * DBL_MIN;  // eigenvalues closer than this share a cluster
    constexpr int kPer = (kEigMaxR + kWarps - 1) / kWarps; // eigenvalues per warp
    uint32_t      swp[kPer][kEigMaxN / 32];            // row j and j+1 exchanged at step j
    for (int u = 0; u < kPer; ++u) {
      const int t = warp + kWarps * u;
#pragma unroll
      for (int q = 0; q < kEigMaxN / 32; ++q)
        swp[u][q] = 0u;
      if (t >= r)
        continue;
      double *y = Y + t * ldy;
      double *u0 = lu + (0 * kEigMaxR + t) * ldy, *u1 = lu + (1 * kEigMaxR + t) * ldy,
             *u2 = lu + (2 * kEigMaxR + t) * ldy, *ml = lu + (3 * kEigMaxR + t) * ldy;
      if (lane == 0) {
        // Gaussian elimination of M = T - lambda I with partial pivoting.  The working row holds the
        // entries (a0, a1) of columns j, j+1 (its column-(j+2) entry is always 0); row j+1 of M is
        // (e_j, d_{j+1} - lambda, e_{j+1}) on columns j, j+1, j+2.  U gets (u0, u1, u2) per row.
        const double lm = lam[t];
        double       a0 = d[0] - lm, a1 = n > 1 ? e[0] : 0.0;
        for (int j = 0; j + 1 < n; ++j) {
          const double b0 = e[j], b1 = d[j + 1] - lm, b2 = j + 2 < n ? e[j + 1] : 0.0;
          const bool   keep = fabs(a0) >= fabs(b0);
          const double piv  = keep ? (fabs(a0) < tiny ? copysign(tiny, a0) : a0) : b0;
          const double l    = (keep ? b0 : a0) * reciprocal(piv);
          u0[j] = piv, ml[j] = l;
          u1[j] = keep ? a1 : b1, u2[j] = keep ? 0.0 : b2;
          if (!keep)
            swp[u][j >> 5] |= 1u << (j & 31);
          a0 = keep ? fma(-l, a1, b1) : fma(-l, b1, a1);
          a1 = keep ? b2 : -l * b2;
        }
        u0[n - 1] = fabs(a0) < tiny ? copysign(tiny, a0) : a0;
      }
      __syncwarp();
      for (int j = lane; j < n; j += 32) { // U's rows over their pivots: one fused step per entry
        const double ip = reciprocal(u0[j]);
        u0[j] = ip;
        u1[j] = j + 1 < n ? u1[j] * ip : 0.0;
        u2[j] = j + 2 < n ? u2[j] * ip : 0.0;
        y[j]  = 1.0 + 0.01 * (double)(((j * 7 + t * 13) % 17) - 8); // start: nonzero, distinct per t
      }
    }
    bool clustered = false; // any two of the r eigenvalues closer than clus
    for (int q = 1; q < r; ++q)
      clustered |= fabs(lam[q] - lam[q - 1]) <= clus;
    for (int it = 0; it < 2; ++it) {
      for (int u = 0; u < kPer; ++u) {
        const int t = warp + kWarps * u;
        if (t >= r)
          continue;
        double       *y  = Y + t * ldy;
        const double *u0 = lu + (0 * kEigMaxR + t) * ldy, *u1 = lu + (1 * kEigMaxR + t) * ldy,
                     *u2 = lu + (2 * kEigMaxR + t) * ldy, *ml = lu + (3 * kEigMaxR + t) * ldy;
        __syncwarp();
        if (lane == 0) { // solve M y' = y in place, the running entry carried in a register; eight
                         // entries are loaded ahead of the chain and stored behind it
          constexpr int kCh = 8;
          double        c   = y[0];
          for (int j0 = 0; j0 + 1 < n; j0 += kCh) {
            double nx[kCh], l[kCh], o[kCh];
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 + i + 1 < n)
                nx[i] = y[j0 + i + 1], l[i] = ml[j0 + i];
            const uint32_t sw = swp[u][j0 >> 5] >> (j0 & 31);
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 + i + 1 < n) {
                const bool ex2 = (sw >> i) & 1u; // rows j, j+1 exchanged
                o[i] = ex2 ? nx[i] : c;
                c    = ex2 ? fma(-l[i], nx[i], c) : fma(-l[i], c, nx[i]);
              }
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 + i + 1 < n)
                y[j0 + i] = o[i];
          }
          double c1 = c * u0[n - 1], c2 = 0.0; // y[j+1], y[j+2] of the back substitution
          y[n - 1]  = c1;
          for (int j0 = n - 2; j0 >= 0; j0 -= kCh) {
            double yy[kCh], a1[kCh], a2[kCh];
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 - i >= 0)
                yy[i] = y[j0 - i] * u0[j0 - i], a1[i] = u1[j0 - i], a2[i] = u2[j0 - i];
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 - i >= 0) {
                yy[i] = fma(-a1[i], c1, fma(-a2[i], c2, yy[i]));
                c2    = c1;
                c1    = yy[i];
              }
#pragma unroll
            for (int i = 0; i < kCh; ++i)
              if (j0 - i >= 0)
                y[j0 - i] = yy[i];
          }
        }
        __syncwarp();
        // scale by the largest entry first (the solve grows y by up to 1 / (eps ||T||)), then
        // normalise
        double mx = 0.0;
        for (int i = lane; i < n; i += 32)
          mx = fmax(mx, fabs(y[i]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (mx > 0.0) {
          const double im = 1.0 / mx;
          double       ss = 0.0;
          for (int i = lane; i < n; i += 32) {
            const double yi = y[i] * im;
            y[i]            = yi;
            ss              = fma(yi, yi, ss);
          }
          const double inv = 1.0 / sqrt(warp_sum(ss));
          for (int i = lane; i < n; i += 32)
            y[i] *= inv;
        }
      }
      if (!clustered)
        continue;
      __syncthreads();
      // modified Gram-Schmidt within clusters, in descending eigenvalue order, by the warp of s2
      for (int s2 = 1; s2 < r; ++s2) {
        if (warp == s2 % kWarps) {
          double *y   = Y + s2 * ldy;
          bool    any = false;
          for (int q = 0; q < s2; ++q) {
            if (fabs(lam[q] - lam[s2]) > clus)
              continue;
            const double *yq = Y + q * ldy;
            double        dt = 0.0;
            for (int i = lane; i < n; i += 32)
              dt = fma(yq[i], y[i], dt);
            dt = warp_sum(dt);
            for (int i = lane; i < n; i += 32)
              y[i] = fma(-dt, yq[i], y[i]);
            __syncwarp();
            any = true;
          }
          if (any) {
            double ss = 0.0;
            for (int i = lane; i < n; i += 32)
              ss = fma(y[i], y[i], ss);
            ss = warp_sum(ss);
            if (ss > 0.0) {
              const double inv = 1.0 / sqrt(ss);
              for (int i = lane; i < n; i += 32)
                y[i] *= inv;
            }
          }
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();

  // ---- 4. back-transformation V = Q Y by the reflectors in descending order, four at a time: the
  //         dot products of a block with y run side by side, and the products of its reflectors with
  //         each other (in G) carry the sequential order.  A warp per column, entries lane + 32 c -----
  double *G = lu; // [blocks][6]: v_k . v_(k-1), v_k . v_(k-2), v_(k-1) . v_(k-2), then those with v_(k-3)
  const auto reflector = [&](int k, double (&v)[NC]) { // 0 before k = 0
#pragma unroll
    for (int c = 0; c < NC; ++c)
      v[c] = k >= 0 ? R[k * RM + lane + 32 * c] : 0.0;
  };
  const int nblk = (max(n - 2, 0) + 3) / 4;
  for (int bl = warp; bl < nblk; bl += kWarps) {
    const int k = n - 3 - 4 * bl;
    double    v[4][NC], g[6];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      reflector(k - q, v[q]);
#pragma unroll
    for (int q = 1; q < 4; ++q)
#pragma unroll
      for (int h = 0; h < q; ++h) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
          s = fma(v[q][c], v[h][c], s);
        g[q * (q - 1) / 2 + h] = warp_sum(s);
      }
    if (lane < 6) {
      double x = g[0];
#pragma unroll
      for (int q = 1; q < 6; ++q)
        x = lane == q ? g[q] : x;
      G[6 * bl + lane] = x;
    }
  }
  __syncthreads();
  for (int t = warp; t < r; t += kWarps) {
    const double *ys = Y + t * ldy;
    double        y[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int i = lane + 32 * c;
      y[c]        = i < n ? ys[i] : 0.0;
    }
    for (int bl = 0; bl < nblk; ++bl) {
      const int k = n - 3 - 4 * bl;
      double    v[4][NC], s[4], cf[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        reflector(k - q, v[q]);
        s[q] = 0.0;
#pragma unroll
        for (int c = 0; c < NC; ++c)
          s[q] = fma(v[q][c], y[c], s[q]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
#pragma unroll
      for (int q = 0; q < 4; ++q) { // coefficient of reflector k - q after the ones before it
        double x = s[q];
#pragma unroll
        for (int h = 0; h < q; ++h)
          x = fma(-cf[h], G[6 * bl + q * (q - 1) / 2 + h], x);
        cf[q] = k - q >= 0 ? beta[k - q] * x : 0.0;
      }
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          y[c] = fma(-cf[q], v[q][c], y[c]);
    }
    const int idx = n - 1 - t;
    double   *vec = evecs + (int64_t)blockIdx.x * n * n;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int i = lane + 32 * c;
      if (i < n)
        vec[i * n + idx] = y[c];
    }
    if (lane == 0)
      evals[(int64_t)blockIdx.x * n + idx] = ldexp(lam[t], ex);
  }
  if (tid == 0 && info != nullptr)
    info[blockIdx.x] = 0;
}

} // namespace

size_t eig_top_smem_bytes(int n) {
  return ((size_t)(n + 1) * (eig_threads(n) / 4) + 5 * (size_t)n + 16 + kEigMaxR + 5 * (size_t)kEigMaxR * eig_ldy(n) +
          kEigRed) * sizeof(double) + 16;
}

bool eig_top_supported(int n, int r) { return n >= 1 && n <= kEigMaxN && r >= 1 && r <= kEigMaxR && r <= n; }

int launch_eig_top(const double *a, double *evecs, double *evals, int *info, int n, int r, int64_t batch,
                   cudaStream_t s) {
  HF_CHECK_ARG(eig_top_supported(n, r) && batch >= 1, "eig_top: order must be in [1, 128] and 1 <= r <= min(16, n)");
  const size_t smem = eig_top_smem_bytes(n);
  const int    nt   = eig_threads(n);
  auto         kern = nt == 128 ? eig_top_kernel<128, 1> : (nt == 512 ? eig_top_kernel<512, 1> : eig_top_kernel<256, 1>);
  // more matrices than SMs: two CTAs per SM within 128 registers each take longer apiece and less in all.
  // 600 matrices of 50, r = 4: 370 -> 246 us (284 with the shared-memory kernel before), 149 of them 149 ->
  // 92; the others fit one CTA (n > 64) or several (n <= 32) as they are.
  if (nt == 256 && batch > sm_count())
    kern = eig_top_kernel<256, 2>;
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)batch, nt, smem, s>>>(a, evecs, evals, info, n, r);
  note_launch();
  return launch_status("eig_top_kernel");
}

} // namespace hf
