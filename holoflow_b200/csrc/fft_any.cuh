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
// w_n^(r m (j mod Ns)) with m = n / (Ns p) (the powers by recurrence from one table load), takes
// the p-point DFT and writes output q to ((j / Ns) Ns p + j mod Ns) + q Ns.  Index divisions are
// multiply-high divisions by invariant integers.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "hf_common.cuh"

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

__device__ __forceinline__ float2 twid(const float2 *tw, int e, bool inv) {
  const float2 w = tw[e];
  return inv ? make_float2(w.x, -w.y) : w;
}

__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// P-point DFT in registers.  2 and 4 take the exact butterflies; an odd P takes the symmetric form
// Y[q] = v0 + sum_r (v_r + v_{P-r}) cos(2 pi q r / P) - i sum_r (v_r - v_{P-r}) sin(2 pi q r / P),
// r = 1 .. (P-1)/2, with Y[P-q] the same with +i: ((P-1)/2)^2 complex-by-real products for both.
// cos and sin of 2 pi m / P come from the length-n table at m n / P.
template <int P> struct Split { // P = A B with A the radix taken first (0: P is 2, 4 or prime)
  static constexpr int A = P % 4 == 0 && P > 4 ? 4 : (P % 2 == 0 && P > 4 ? 2 : (P % 3 == 0 && P > 3 ? 3 : 0));
  static constexpr int B = A ? P / A : 0;
};

template <int P> __device__ __forceinline__ void dft_small(float2 (&v)[P], bool inv, const float2 *tw, int step);

// Composite P = A B in registers (Cooley-Tukey): B DFTs of length A over v[i2 + B i1], the inner
// twiddles w_P^(i2 k1) (table entries (i2 k1) n / P), A DFTs of length B; output k1 + A k2.
template <int P> __device__ __forceinline__ void dft_composite(float2 (&v)[P], bool inv, const float2 *tw, int step) {
  constexpr int A = Split<P>::A, B = Split<P>::B;
  float2        u[P];
#pragma unroll
  for (int i2 = 0; i2 < B; ++i2) {
    float2 t[A];
#pragma unroll
    for (int i1 = 0; i1 < A; ++i1)
      t[i1] = v[i2 + B * i1];
    dft_small<A>(t, inv, tw, step * B);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1)
      u[i2 * A + k1] = (i2 == 0 || k1 == 0) ? t[k1] : cmul(t[k1], twid(tw, ((i2 * k1) % P) * step, inv));
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 t[B];
#pragma unroll
    for (int i2 = 0; i2 < B; ++i2)
      t[i2] = u[i2 * A + k1];
    dft_small<B>(t, inv, tw, step * A);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2)
      v[k1 + A * k2] = t[k2];
  }
}

template <int P> __device__ __forceinline__ void dft_small(float2 (&v)[P], bool inv, const float2 *tw, int step) {
  if constexpr (Split<P>::A != 0) {
    dft_composite<P>(v, inv, tw, step);
  } else if constexpr (P == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b), v[1] = csub(a, b);
  } else if constexpr (P == 4) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 a2 = cadd(v[1], v[3]), a3 = csub(v[1], v[3]);
    const float2 r = inv ? make_float2(-a3.y, a3.x) : make_float2(a3.y, -a3.x); // (+i or -i) a3
    v[0] = cadd(a0, a2), v[2] = csub(a0, a2);
    v[1] = cadd(a1, r), v[3] = csub(a1, r);
  } else {
    constexpr int H = (P - 1) / 2;
    float2        a[H + 1], b[H + 1];
    float         cs[H + 1], sn[H + 1];
    float2        y0 = v[0];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      a[r] = cadd(v[r], v[P - r]), b[r] = csub(v[r], v[P - r]);
      y0   = cadd(y0, a[r]);
      const float2 w = tw[r * step]; // (cos, -sin) of 2 pi r / P
      cs[r] = w.x, sn[r] = -w.y;
    }
    float2 out[P];
    out[0] = y0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      float2 sc = v[0], ss = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const int   mm = (q * r) % P;
        const float c  = mm <= H ? cs[mm] : cs[P - mm];
        const float sv = mm <= H ? sn[mm] : -sn[P - mm];
        sc.x = fmaf(a[r].x, c, sc.x), sc.y = fmaf(a[r].y, c, sc.y);
        ss.x = fmaf(b[r].x, sv, ss.x), ss.y = fmaf(b[r].y, sv, ss.y);
      }
      const float2 yq = make_float2(sc.x + ss.y, sc.y - ss.x); // sc - i ss
      const float2 yp = make_float2(sc.x - ss.y, sc.y + ss.x); // sc + i ss
      out[q]     = inv ? yp : yq;
      out[P - q] = inv ? yq : yp;
    }
#pragma unroll
    for (int q = 0; q < P; ++q)
      v[q] = out[q];
  }
}

// Odd P: the symmetric form of dft_small, with the inputs folded into a_r = v_r + v_(P-r) and
// b_r = v_r - v_(P-r) as they are loaded (the twiddle of input P - r is w^P conj(w^r)) and each
// output pair stored as soon as it is formed, so no P-element array stays live.
template <int P>
__device__ void stage_bfly_odd(const float2 *x, float2 *y, int pitch, int rows, const Stage &st, const float2 *tw,
                               int n, bool inv) {
  constexpr int H  = (P - 1) / 2;
  const int     nb = st.nb, Ns = st.Ns, total = rows * nb, step = n / P;
  float         cs[H + 1], sn[H + 1];
#pragma unroll
  for (int r = 1; r <= H; ++r) {
    const float2 w = tw[r * step]; // (cos, -sin) of 2 pi r / P
    cs[r] = w.x, sn[r] = -w.y;
  }
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int     row = fdiv(t, st.by_nb), j = t - row * nb;
    const int     jb = fdiv(j, st.by_Ns), k = j - jb * Ns;
    const int     e  = st.m * k;
    const float2 *xr = x + row * pitch;
    float2       *yr = y + row * pitch;
    const float2  v0 = xr[j];
    float2        a[H + 1], b[H + 1];
    float2        y0 = v0;
    if (e > 0) {
      const float2 w1 = twid(tw, e, inv);
      float2       wr = w1, wh = w1;
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        if (r > 1)
          wr = cmul(wr, w1);
        if (r == H)
          wh = wr;
        a[r] = cmul(xr[j + r * nb], wr);
      }
      const float2 wp = cmul(cmul(wh, wh), w1); // w^P
      wr              = w1;
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        if (r > 1)
          wr = cmul(wr, w1);
        const float2 u = cmul(xr[j + (P - r) * nb], cmul(wp, make_float2(wr.x, -wr.y)));
        b[r]           = csub(a[r], u);
        a[r]           = cadd(a[r], u);
        y0             = cadd(y0, a[r]);
      }
    } else {
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const float2 vr = xr[j + r * nb], vp = xr[j + (P - r) * nb];
        a[r] = cadd(vr, vp), b[r] = csub(vr, vp);
        y0   = cadd(y0, a[r]);
      }
    }
    const int base = jb * Ns * P + k;
    yr[base]       = y0;
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      float2 sc = v0, ss = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const int   mm = (q * r) % P;
        const float c  = mm <= H ? cs[mm] : cs[P - mm];
        const float sv = mm <= H ? sn[mm] : -sn[P - mm];
        sc.x = fmaf(a[r].x, c, sc.x), sc.y = fmaf(a[r].y, c, sc.y);
        ss.x = fmaf(b[r].x, sv, ss.x), ss.y = fmaf(b[r].y, sv, ss.y);
      }
      const float2 yq = make_float2(sc.x + ss.y, sc.y - ss.x); // sc - i ss
      const float2 yp = make_float2(sc.x - ss.y, sc.y + ss.x); // sc + i ss
      yr[base + q * Ns]       = inv ? yp : yq;
      yr[base + (P - q) * Ns] = inv ? yq : yp;
    }
  }
}

template <int P>
__device__ void stage_bfly(const float2 *x, float2 *y, int pitch, int rows, const Stage &st, const float2 *tw, int n,
                           bool inv) {
  if constexpr (P % 2 == 1 && Split<P>::A == 0) {
    stage_bfly_odd<P>(x, y, pitch, rows, st, tw, n, inv);
    return;
  }
  const int nb = st.nb, Ns = st.Ns, total = rows * nb, step = n / P;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int     row = fdiv(t, st.by_nb), j = t - row * nb;
    const int     jb = fdiv(j, st.by_Ns), k = j - jb * Ns;
    const int     e  = st.m * k; // twiddle of input r: w_n^(r m k) = (w_n^(m k))^r
    const float2 *xr = x + row * pitch;
    float2       *yr = y + row * pitch;
    float2        v[P];
#pragma unroll
    for (int r = 0; r < P; ++r)
      v[r] = xr[j + r * nb];
    if (e > 0) {
      const float2 w1 = twid(tw, e, inv);
      float2       wr = w1;
#pragma unroll
      for (int r = 1; r < P; ++r) {
        v[r] = cmul(v[r], wr);
        if (r + 1 < P)
          wr = cmul(wr, w1);
      }
    }
    dft_small<P>(v, inv, tw, step);
    const int base = jb * Ns * P + k;
#pragma unroll
    for (int q = 0; q < P; ++q)
      yr[base + q * Ns] = v[q];
  }
}

// A prime radix beyond the register butterflies, in the symmetric form (see stage_bfly_odd): first
// the twiddled inputs are folded in place, a_r = v_r + v_(p-r) at r and b_r = v_r - v_(p-r) at p - r;
// then each thread sums RB rows x kDenseQ output pairs (q, p - q), so a pair's cosine and sine are
// loaded once for RB rows and a row's a_r, b_r once for kDenseQ pairs.  The p-term sums per output
// it replaces loaded one sample and one twiddle per complex product.
// Both buffers need room for `rows` rounded up to a multiple of RB.
constexpr int kDenseQ = 4;
template <int RB>
__device__ void stage_dense(float2 *x, float2 *y, int pitch, int rows, const Stage &st, const float2 *tw, int n,
                            bool inv) {
  const int p = st.p, nb = st.nb, Ns = st.Ns, H = (p - 1) / 2, step = n / p;
  if (rows * nb > 0) {
    const int total = rows * nb * H; // (row, r, j), j fastest
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      const int u = fdiv(t, st.by_nb), j = t - u * nb, row = u / H, r = 1 + u - row * H;
      const int k = j - fdiv(j, st.by_Ns) * Ns;
      float2   *xr = x + row * pitch + j;
      const float2 vr = cmul(xr[r * nb], twid(tw, st.m * k * r, inv));
      const float2 vp = cmul(xr[(p - r) * nb], twid(tw, st.m * k * (p - r), inv));
      xr[r * nb] = cadd(vr, vp), xr[(p - r) * nb] = csub(vr, vp);
    }
  }
  __syncthreads();
  const int nrb = (rows + RB - 1) / RB, cols = nrb * nb, groups = (H + 1 + kDenseQ - 1) / kDenseQ;
  for (int t = threadIdx.x; t < cols * groups; t += blockDim.x) {
    const int     qg = t / cols, c = t - qg * cols;
    const int     rb = fdiv(c, st.by_nb), j = c - rb * nb;
    const int     q0 = qg * kDenseQ;
    const float2 *xr = x + rb * RB * pitch + j;
    float2        sc[RB][kDenseQ], ss[RB][kDenseQ];
    int           e[kDenseQ], de[kDenseQ];
#pragma unroll
    for (int i = 0; i < kDenseQ; ++i)
      e[i] = 0, de[i] = min(q0 + i, H) * step;
#pragma unroll
    for (int b = 0; b < RB; ++b)
#pragma unroll
      for (int i = 0; i < kDenseQ; ++i)
        sc[b][i] = xr[b * pitch], ss[b][i] = make_float2(0.f, 0.f);
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
        const float2 av = xr[b * pitch + r * nb], bv = xr[b * pitch + (p - r) * nb];
#pragma unroll
        for (int i = 0; i < kDenseQ; ++i) {
          sc[b][i] = cfma2(av, make_float2(w[i].x, w[i].x), sc[b][i]);
          ss[b][i] = cfma2(bv, make_float2(w[i].y, w[i].y), ss[b][i]);
        }
      }
    }
    const int jb = fdiv(j, st.by_Ns), k = j - jb * Ns, base = jb * Ns * p + k;
#pragma unroll
    for (int b = 0; b < RB; ++b) {
      float2 *yr = y + (rb * RB + b) * pitch + base;
#pragma unroll
      for (int i = 0; i < kDenseQ; ++i) {
        const int q = q0 + i;
        if (q > H)
          continue;
        // with s = -ss the pair is sc - i s (forward q) and sc + i s
        const float2 yq = make_float2(sc[b][i].x - ss[b][i].y, sc[b][i].y + ss[b][i].x);
        const float2 yp = make_float2(sc[b][i].x + ss[b][i].y, sc[b][i].y - ss[b][i].x);
        yr[q * Ns] = inv ? yp : yq;
        if (q > 0)
          yr[(p - q) * Ns] = inv ? yq : yp;
      }
    }
  }
}

// Transforms `rows` rows of `a` (pitch `pitch`), ping-ponging with `b` (both with room for `rows`
// rounded up to a multiple of RB); returns the buffer that holds the result.  Every thread of the CTA calls it; the rows must be in `a` and visible.
template <int RB>
__device__ float2 *fft_rows_smem(float2 *a, float2 *b, int pitch, int rows, const GPlan &pl, const float2 *tw, bool inv) {
  for (int s = 0; s < pl.nst; ++s) {
    const Stage &st = pl.st[s];
    switch (st.p) {
    case 2: stage_bfly<2>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 3: stage_bfly<3>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 4: stage_bfly<4>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 5: stage_bfly<5>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 7: stage_bfly<7>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 11: stage_bfly<11>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 13: stage_bfly<13>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 17: stage_bfly<17>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 6: stage_bfly<6>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 8: stage_bfly<8>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 9: stage_bfly<9>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 10: stage_bfly<10>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 12: stage_bfly<12>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 15: stage_bfly<15>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    case 16: stage_bfly<16>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    default: stage_dense<RB>(a, b, pitch, rows, st, tw, pl.n, inv); break;
    }
    __syncthreads();
    float2 *t = a;
    a = b, b = t;
  }
  return a;
}

} // namespace
} // namespace hf
