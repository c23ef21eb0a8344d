// Shared-memory FFT of any length, for transform sides that are no four-step length (32 N1).
//
// A Stockham auto-sort sequence of stages, one per radix p of a factorisation of n planned on the
// host.
//  - Factors 4, 2, 3, 5 are merged pairwise into the composite radices 6, 8, 9, 10, 12, 15, 16
//    (one shared-memory pass and barrier fewer per pair).
//  - Primes 3..17 take register butterflies in the symmetric form; a composite radix takes a
//    register Cooley-Tukey split; a larger prime takes the symmetric form as a dense product tiled
//    over rows and outputs.
//  - Odd radices come first: the first stage (Ns = 1) stores with stride p, which is conflict-free
//    for odd p and up to p-way conflicting for even p; by the time the even radices store, their
//    runs of Ns consecutive entries cover the banks.
// A stage of radix p over sub-transforms of span Ns reads x[j + r n/p], twiddles input r by
// w_n^(r m (j mod Ns)) with m = n / (Ns p), takes the p-point DFT and writes output q to
// ((j / Ns) Ns p + j mod Ns) + q Ns.  The twiddles are read from the table: as products of powers they
// took the same time but their roundings were most of the transform's error (600 x 800 Fresnel moments
// 2.8e-7 against 0.8e-7 from float64).  Index divisions are multiply-high divisions by invariant integers.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "hf_common.cuh"
#include "twiddles.inc"

namespace hf {
namespace {

constexpr int kFftStages = 16;

// Division by a run-time invariant d as a multiply-high and a shift (Granlund and Montgomery,
// "Division by invariant integers using multiplication", 1994, round-up variant): with
// l = ceil(log2 d), m = ceil(2^(31+l) / d) < 2^32 and x < 2^31, x / d = umulhi(x, m) >> (l - 1).
struct FastDiv {
  uint32_t d, m;
  int      s;
};

FastDiv make_div(uint32_t d) {
  if (d <= 1)
    return {1u, 0u, 0};
  int l = 0;
  while ((1u << l) < d)
    ++l;
  const uint64_t p = 31 + (uint64_t)l;
  return {d, (uint32_t)(((1ull << p) + d - 1) / d), (int)(p - 32)};
}

__device__ __forceinline__ int fdiv(int x, const FastDiv &f) {
  return f.d == 1 ? x : (int)(__umulhi((uint32_t)x, f.m) >> f.s);
}

struct Stage {
  int     p, Ns, m, nb; // radix, span of the sub-transforms before the stage, n / (Ns p), n / p
  FastDiv by_nb, by_Ns;
};

struct GPlan {
  int     n, nst;
  FastDiv by_n;
  Stage   st[kFftStages];
};

bool make_plan(int n, GPlan &pl, int max_n) {
  if (n < 2 || n > max_n)
    return false;
  std::memset(&pl, 0, sizeof(pl));
  pl.n = n, pl.nst = 0, pl.by_n = make_div((uint32_t)n);
  int rem = n, Ns = 1;
  auto push = [&](int p) {
    Stage &st = pl.st[pl.nst++];
    st.p = p, st.Ns = Ns, st.m = n / (Ns * p), st.nb = n / p;
    st.by_nb = make_div((uint32_t)st.nb), st.by_Ns = make_div((uint32_t)Ns);
    Ns *= p;
  };
  // prime-power factors first (4 before 2), then pairs of the small ones merged into one
  // register radix (6, 8, 9, 10, 12, 15, 16): one shared-memory pass and barrier fewer per pair
  std::vector<int> f;
  for (int p : {4, 2, 3, 5, 7, 11, 13, 17})
    while (rem % p == 0)
      f.push_back(p), rem /= p;
  for (int p = 19; rem > 1; p += 2)
    while (rem % p == 0)
      f.push_back(p), rem /= p;
  auto mergeable = [](int a, int b) {
    const int c = a * b;
    return (a <= 5 && b <= 5) && (c == 6 || c == 8 || c == 9 || c == 10 || c == 12 || c == 15 || c == 16);
  };
  std::vector<int> radices;
  for (size_t i = 0; i < f.size(); ++i) {
    size_t best = f.size();
    if (f[i] <= 5)
      for (size_t k = i + 1; k < f.size(); ++k)
        if (f[k] > 0 && mergeable(f[i], f[k]) && (best == f.size() || f[i] * f[k] > f[i] * f[best]))
          best = k;
    if (f[i] == 0)
      continue;
    if (best < f.size()) {
      radices.push_back(f[i] * f[best]);
      f[best] = 0;
    } else {
      radices.push_back(f[i]);
    }
  }
  if ((int)radices.size() > kFftStages)
    return false;
  std::stable_sort(radices.begin(), radices.end(), [](int a, int b) {
    return (a % 2 != b % 2) ? a % 2 > b % 2 : (a % 2 ? a > b : a < b);
  });
  for (int p : radices)
    push(p);
  return true;
}

// Relative time of the stages over `rows` rows with `threads` threads.  A thread takes whole butterflies,
// so a stage lasts as many rounds as ceil(rows nb / threads), each about as long as one butterfly: 16
// rows of 204 = 17 x 12 take 2 rounds of the 12-point stage for 272 butterflies, 15 rows take 1.
double plan_time(const GPlan &pl, int rows, int threads) {
  double t = 0.0;
  for (int i = 0; i < pl.nst; ++i) {
    const int    p = pl.st[i].p, rounds = (rows * pl.st[i].nb + threads - 1) / threads;
    const bool   prime = p == 7 || p == 11 || p == 13 || p >= 17;
    t += rounds * (100.0 + 20.0 * p + (prime ? 1.0 * p * p : 4.0 * p)); // barrier, loads and stores, arithmetic
  }
  return t;
}

// The number of rows (a multiple of `step` up to `most`) that a CTA of `threads` transforms fastest, per row.
int plan_rows(const GPlan &pl, int step, int most, int threads) {
  int    best = step;
  double rate = 0.0;
  for (int rows = step; rows <= most; rows += step) { // 400: filling the tables, launching
    const double v = rows / (400.0 + plan_time(pl, rows, threads) + 30.0 * rows * pl.n / threads);
    if (v > rate)
      best = rows, rate = v;
  }
  return best;
}

// exp(-2 pi i k / P), 0 <= k < P a compile-time constant after unrolling: an operand in constant memory
template <int P> __device__ __forceinline__ float2 root(int k);
#define HF_ROOT(P)                                                                                 \
  template <> __device__ __forceinline__ float2 root<P>(int k) { return c_root##P[k]; }
HF_ROOT(3) HF_ROOT(5) HF_ROOT(6) HF_ROOT(7) HF_ROOT(8) HF_ROOT(9) HF_ROOT(10) HF_ROOT(11) HF_ROOT(12) HF_ROOT(13)
HF_ROOT(15) HF_ROOT(16) HF_ROOT(17)
#undef HF_ROOT

// v exp(-2 pi i k / P)
template <int P> __device__ __forceinline__ float2 mul_root(float2 v, int k) {
  if (k == 0)
    return v;
  if (4 * k == P)
    return make_float2(v.y, -v.x);
  if (2 * k == P)
    return make_float2(-v.x, -v.y);
  if (4 * k == 3 * P)
    return make_float2(-v.y, v.x);
  return cmul(v, root<P>(k));
}

__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// P-point DFT in registers.  2 and 4 take the exact butterflies; an odd P takes the symmetric form
// Y[q] = v0 + sum_r (v_r + v_{P-r}) cos(2 pi q r / P) - i sum_r (v_r - v_{P-r}) sin(2 pi q r / P),
// r = 1 .. (P-1)/2, with Y[P-q] the same with +i: ((P-1)/2)^2 complex-by-real products for both.
// The constants come from the root tables (reading them from the length-n table took a shared load and
// an index each, and their registers).
template <int P> struct Split { // P = A B with A the radix taken first (0: P is 2, 4 or prime)
  static constexpr int A = P % 4 == 0 && P > 4 ? 4 : (P % 2 == 0 && P > 4 ? 2 : (P % 3 == 0 && P > 3 ? 3 : 0));
  static constexpr int B = A ? P / A : 0;
};

template <int P> __device__ __forceinline__ void dft_small(float2 (&v)[P]);

// Composite P = A B in registers (Cooley-Tukey): B DFTs of length A over v[i2 + B i1], the inner
// twiddles w_P^(i2 k1), A DFTs of length B; output k1 + A k2.
template <int P> __device__ __forceinline__ void dft_composite(float2 (&v)[P]) {
  constexpr int A = Split<P>::A, B = Split<P>::B;
  float2        u[P];
#pragma unroll
  for (int i2 = 0; i2 < B; ++i2) {
    float2 t[A];
#pragma unroll
    for (int i1 = 0; i1 < A; ++i1)
      t[i1] = v[i2 + B * i1];
    dft_small<A>(t);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1)
      u[i2 * A + k1] = mul_root<P>(t[k1], (i2 * k1) % P);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 t[B];
#pragma unroll
    for (int i2 = 0; i2 < B; ++i2)
      t[i2] = u[i2 * A + k1];
    dft_small<B>(t);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2)
      v[k1 + A * k2] = t[k2];
  }
}

// Outputs q and P - q of the symmetric form.
template <int P>
__device__ __forceinline__ void odd_pair(float2 v0, const float2 (&a)[(P + 1) / 2], const float2 (&b)[(P + 1) / 2], int q,
                                         float2 &yq, float2 &yp) {
  float2 sc = v0, ss = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 1; r <= (P - 1) / 2; ++r) {
    const float2 w = root<P>((q * r) % P); // (cos, -sin)
    sc             = cfma2(a[r], make_float2(w.x, w.x), sc);
    ss             = cfma2(b[r], make_float2(w.y, w.y), ss);
  }
  yq = make_float2(sc.x - ss.y, sc.y + ss.x); // sc + i ss
  yp = make_float2(sc.x + ss.y, sc.y - ss.x);
}

template <int P> __device__ __forceinline__ void dft_small(float2 (&v)[P]) {
  if constexpr (Split<P>::A != 0) {
    dft_composite<P>(v);
  } else if constexpr (P == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b), v[1] = csub(a, b);
  } else if constexpr (P == 4) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 a2 = cadd(v[1], v[3]), a3 = csub(v[1], v[3]);
    const float2 r = make_float2(a3.y, -a3.x); // -i a3
    v[0] = cadd(a0, a2), v[2] = csub(a0, a2);
    v[1] = cadd(a1, r), v[3] = csub(a1, r);
  } else {
    constexpr int H = (P - 1) / 2;
    float2        a[H + 1], b[H + 1];
    const float2  v0 = v[0];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      a[r] = cadd(v[r], v[P - r]), b[r] = csub(v[r], v[P - r]);
      v[0] = cadd(v[0], a[r]);
    }
#pragma unroll
    for (int q = 1; q <= H; ++q)
      odd_pair<P>(v0, a, b, q, v[q], v[P - q]);
  }
}

// Work buffers of a transform: element i of row `row` at row * rs + i * es.  Rows one after the other
// (ROWS: rs = pitch, es = 1), or interleaved (columns of a strip as they lie in memory: rs = 1, es = the
// padded number of columns, which by_es divides by), where neighbouring threads take neighbouring
// columns of one butterfly, so no stage has bank conflicts.
template <bool IL> struct Layout {
  int     rs, es, rows;
  FastDiv by_es;
  __device__ __forceinline__ int stride() const { return IL ? es : 1; }
  __device__ __forceinline__ int total(int per_row) const { return (IL ? es : rows) * per_row; }
  // work item t of per_row items (by_per divides by per_row) for each row -> (row, item of the row)
  __device__ __forceinline__ void split(int t, const FastDiv &by_per, int per_row, int &row, int &j) const {
    if constexpr (IL)
      j = fdiv(t, by_es), row = t - j * es;
    else
      row = fdiv(t, by_per), j = t - row * per_row;
  }
};

__device__ __forceinline__ Layout<false> row_layout(int pitch, int rows) { return {pitch, 1, rows, {}}; }
__device__ __forceinline__ Layout<true> strip_layout(const FastDiv &by_cols) { return {1, (int)by_cols.d, 0, by_cols}; }

// Odd P: the symmetric form of dft_small, with the inputs folded into a_r = v_r + v_(P-r) and
// b_r = v_r - v_(P-r) as they are loaded (the twiddle of input P - r is w^P conj(w^r)) and each
// output pair stored as soon as it is formed, so no P-element array stays live.
template <int P, bool IL>
__device__ void stage_bfly_odd(const float2 *x, float2 *y, const Layout<IL> &lay, const Stage &st, const float2 *tw) {
  constexpr int H  = (P - 1) / 2;
  const int     Ns = st.Ns, total = lay.total(st.nb), es = lay.stride(), nb = st.nb * es, Nss = Ns * es;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int row, j;
    lay.split(t, st.by_nb, st.nb, row, j);
    const int     jb = fdiv(j, st.by_Ns), k = j - jb * Ns;
    const int     e  = st.m * k;
    const float2 *xr = x + row * lay.rs + j * es;
    float2       *yr = y + row * lay.rs + (jb * Ns * P + k) * es;
    const float2  v0 = xr[0];
    float2        a[H + 1], b[H + 1];
    float2        y0 = v0;
    if (e > 0) {
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const float2 t = cmul(xr[r * nb], tw[r * e]);
        const float2 u = cmul(xr[(P - r) * nb], tw[(P - r) * e]);
        a[r]           = cadd(t, u);
        b[r]           = csub(t, u);
        y0             = cadd(y0, a[r]);
      }
    } else {
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const float2 vr = xr[r * nb], vp = xr[(P - r) * nb];
        a[r] = cadd(vr, vp), b[r] = csub(vr, vp);
        y0   = cadd(y0, a[r]);
      }
    }
    yr[0] = y0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      float2 yq, yp;
      odd_pair<P>(v0, a, b, q, yq, yp);
      yr[q * Nss]       = yq;
      yr[(P - q) * Nss] = yp;
    }
  }
}

template <int P, bool IL>
__device__ void stage_bfly(const float2 *x, float2 *y, const Layout<IL> &lay, const Stage &st, const float2 *tw) {
  if constexpr (P % 2 == 1 && Split<P>::A == 0) {
    stage_bfly_odd<P>(x, y, lay, st, tw);
    return;
  }
  const int Ns = st.Ns, total = lay.total(st.nb), es = lay.stride(), nb = st.nb * es, Nss = Ns * es;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int row, j;
    lay.split(t, st.by_nb, st.nb, row, j);
    const int     jb = fdiv(j, st.by_Ns), k = j - jb * Ns;
    const int     e  = st.m * k; // twiddle of input r: w_n^(r m k) = (w_n^(m k))^r
    const float2 *xr = x + row * lay.rs + j * es;
    float2       *yr = y + row * lay.rs + (jb * Ns * P + k) * es;
    float2        v[P];
#pragma unroll
    for (int r = 0; r < P; ++r)
      v[r] = xr[r * nb];
    if (e > 0)
#pragma unroll
      for (int r = 1; r < P; ++r)
        v[r] = cmul(v[r], tw[r * e]);
    dft_small<P>(v);
#pragma unroll
    for (int q = 0; q < P; ++q)
      yr[q * Nss] = v[q];
  }
}

// A prime radix beyond the register butterflies, in the symmetric form (see stage_bfly_odd): first
// the twiddled inputs are folded in place, a_r = v_r + v_(p-r) at r and b_r = v_r - v_(p-r) at p - r;
// then each thread sums RB rows x kDenseQ output pairs (q, p - q), so a pair's cosine and sine are
// loaded once for RB rows and a row's a_r, b_r once for kDenseQ pairs.  The p-term sums per output
// it replaces loaded one sample and one twiddle per complex product.
// Both buffers need room for `rows` rounded up to a multiple of RB.
constexpr int kDenseQ = 4;
template <int RB, bool IL>
__device__ void stage_dense(float2 *x, float2 *y, const Layout<IL> &lay, const Stage &st, const float2 *tw, int n) {
  const int p = st.p, nb = st.nb, Ns = st.Ns, H = (p - 1) / 2, step = n / p, es = lay.stride(), rs = lay.rs;
  const int rows = IL ? lay.es : lay.rows;
  {
    const int total = rows * nb * H; // (row, r, j): j fastest, or the row where rows are interleaved
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      int row, r, j;
      if constexpr (IL) {
        const int u = fdiv(t, lay.by_es), v = fdiv(u, st.by_nb);
        row = t - u * rows, j = u - v * nb, r = 1 + v;
      } else {
        const int u = fdiv(t, st.by_nb);
        j = t - u * nb, row = u / H, r = 1 + u - row * H;
      }
      const int k = j - fdiv(j, st.by_Ns) * Ns;
      float2   *xr = x + row * rs + j * es;
      const float2 vr = cmul(xr[r * nb * es], tw[st.m * k * r]);
      const float2 vp = cmul(xr[(p - r) * nb * es], tw[st.m * k * (p - r)]);
      xr[r * nb * es] = cadd(vr, vp), xr[(p - r) * nb * es] = csub(vr, vp);
    }
  }
  __syncthreads();
  const int nrb = (rows + RB - 1) / RB, cols = nrb * nb, groups = (H + 1 + kDenseQ - 1) / kDenseQ;
  for (int t = threadIdx.x; t < cols * groups; t += blockDim.x) {
    const int     qg = t / cols, c = t - qg * cols;
    const int     rb = fdiv(c, st.by_nb), j = c - rb * nb;
    const int     q0 = qg * kDenseQ;
    const float2 *xr = x + rb * RB * rs + j * es;
    float2        sc[RB][kDenseQ], ss[RB][kDenseQ];
    int           e[kDenseQ], de[kDenseQ];
#pragma unroll
    for (int i = 0; i < kDenseQ; ++i)
      e[i] = 0, de[i] = min(q0 + i, H) * step;
#pragma unroll
    for (int b = 0; b < RB; ++b)
#pragma unroll
      for (int i = 0; i < kDenseQ; ++i)
        sc[b][i] = xr[b * rs], ss[b][i] = make_float2(0.f, 0.f);
    for (int r = 1; r <= H; ++r) {
      float2 w[kDenseQ];
#pragma unroll
      for (int i = 0; i < kDenseQ; ++i) {
        e[i] += de[i];
        e[i] -= e[i] >= n ? n : 0;
        w[i] = tw[e[i]]; // (cos, -sin) of 2 pi q r / p
      }
#pragma unroll
      for (int b = 0; b < RB; ++b) {
        const float2 av = xr[b * rs + r * nb * es], bv = xr[b * rs + (p - r) * nb * es];
#pragma unroll
        for (int i = 0; i < kDenseQ; ++i) {
          sc[b][i] = cfma2(av, make_float2(w[i].x, w[i].x), sc[b][i]);
          ss[b][i] = cfma2(bv, make_float2(w[i].y, w[i].y), ss[b][i]);
        }
      }
    }
    const int jb = fdiv(j, st.by_Ns), k = j - jb * Ns, base = (jb * Ns * p + k) * es;
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float2 *yr = y + (rb * RB + b) * rs + base;
#pragma unroll
      for (int i = 0; i < kDenseQ; ++i) {
        const int q = q0 + i;
        if (q > H)
          continue;
        // sc + i ss for q, sc - i ss for p - q
        const float2 yq = make_float2(sc[b][i].x - ss[b][i].y, sc[b][i].y + ss[b][i].x);
        const float2 yp = make_float2(sc[b][i].x + ss[b][i].y, sc[b][i].y - ss[b][i].x);
        yr[q * Ns * es] = yq;
        if (q > 0)
          yr[(p - q) * Ns * es] = yp;
      }
    }
  }
}

// Transforms the rows of `a`, ping-ponging with `b` (both with room for the rows rounded up to a multiple
// of RB); returns the buffer that holds the result.  Every thread of the CTA calls it; the rows must be
// in `a` and visible.  Forward; the inverse is swap(forward(swap(x))) with swap(v) = (v.y, v.x), which
// the callers apply as they load and store (flip).
__device__ __forceinline__ float2 flip(float2 v, bool inv) { return inv ? make_float2(v.y, v.x) : v; }
template <int RB, bool IL>
__device__ float2 *fft_smem(float2 *a, float2 *b, const Layout<IL> &lay, const GPlan &pl, const float2 *tw) {
  for (int s = 0; s < pl.nst; ++s) {
    const Stage &st = pl.st[s];
    switch (st.p) {
    case 2: stage_bfly<2>(a, b, lay, st, tw); break;
    case 3: stage_bfly<3>(a, b, lay, st, tw); break;
    case 4: stage_bfly<4>(a, b, lay, st, tw); break;
    case 5: stage_bfly<5>(a, b, lay, st, tw); break;
    case 7: stage_bfly<7>(a, b, lay, st, tw); break;
    case 11: stage_bfly<11>(a, b, lay, st, tw); break;
    case 13: stage_bfly<13>(a, b, lay, st, tw); break;
    case 17: stage_bfly<17>(a, b, lay, st, tw); break;
    case 6: stage_bfly<6>(a, b, lay, st, tw); break;
    case 8: stage_bfly<8>(a, b, lay, st, tw); break;
    case 9: stage_bfly<9>(a, b, lay, st, tw); break;
    case 10: stage_bfly<10>(a, b, lay, st, tw); break;
    case 12: stage_bfly<12>(a, b, lay, st, tw); break;
    case 15: stage_bfly<15>(a, b, lay, st, tw); break;
    case 16: stage_bfly<16>(a, b, lay, st, tw); break;
    default: stage_dense<RB>(a, b, lay, st, tw, pl.n); break;
    }
    __syncthreads();
    float2 *t = a;
    a = b, b = t;
  }
  return a;
}

} // namespace
} // namespace hf
