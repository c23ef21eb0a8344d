// Row and column passes of the 2-D transforms for lengths that are no four-step length (32 N1):
// camera sides such as 480, 600, 800, odd crops, primes.  Any length 2 <= n <= kAnyMaxN whose two
// work buffers fit in shared memory; the direct O(n^2) sums of k_fft2d.cu remain for the rest.
//
// Bound: the direct sums evaluated a sine and a cosine per product, 25.8 ms of rows and 15.3 ms of
// columns for 2 windows x 10 planes of 600 x 800; the passes here take 96 and 81 us (0.31 GB of planes
// read and written, 1.7 TB/s: shared-memory and barrier bound).  A CTA transforms R rows (or a strip of
// C columns) in shared memory with the staged FFT of fft_any.cuh, so a pass reads and writes each plane
// once; the CTAs are persistent over the row groups (strips), so the twiddle table w_n^e is built once
// per CTA.  The rows stay one after the other: interleaved as the columns are, they took 94 us against 91 (with
// twiddles by powers, before the table took their place at the same time).
#include <algorithm>

#include "fft_any.cuh"
#include "k_fft2d.cuh"

namespace hf {
namespace {

constexpr int    kAnyThreads = 256;
constexpr int    kAnyMaxN    = 8192;
constexpr int    kAnyRB      = 4;          // rows per thread of a dense stage
constexpr int    kAnyMaxRows = 16;
constexpr size_t kAnySmem    = 112 * 1024; // two CTAs per SM
constexpr size_t kAnySmemMax = 220 * 1024; // one CTA per SM (long transforms)

// w_n^e for e < n.  The angle is reduced to a quadrant q and a fraction r / n of it in exact
// integers, |r| <= n / 2, so its float32 rounding is at most 2^-26 of a quadrant's half.
__device__ __forceinline__ void any_twiddles(float2 *tw, int n) {
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int q = (8 * e + n) / (2 * n), r = 4 * e - q * n; // e / n = (q + r / n) / 4
    float     s, c;
    sincospif(0.5f * (float)r / (float)n, &s, &c);
    const float2 w = (q & 1) ? make_float2(-s, c) : make_float2(c, s); // times i for odd q
    tw[e]          = (q & 2) ? make_float2(-w.x, w.y) : make_float2(w.x, -w.y); // sign, conjugate
  }
}

__global__ void __launch_bounds__(kAnyThreads, 2) any_rows_kernel(const __grid_constant__ RowPass a,
                                                               const __grid_constant__ GPlan pl, int R, int64_t nrows) {
  extern __shared__ __align__(16) float2 sm[];
  __shared__ int64_t s_in[kAnyMaxRows], s_pre[kAnyMaxRows], s_out[kAnyMaxRows];
  const int n   = pl.n, Rp = (R + kAnyRB - 1) / kAnyRB * kAnyRB;
  float2   *tw = sm, *b0 = sm + n, *b1 = b0 + (size_t)Rp * n;
  any_twiddles(tw, n);
  for (int64_t row0 = (int64_t)blockIdx.x * R; row0 < nrows; row0 += (int64_t)gridDim.x * R) {
    const int rows = (int)min((int64_t)R, nrows - row0);
    __syncthreads(); // the previous group's rows are stored
    for (int r = threadIdx.x; r < rows; r += blockDim.x) {
      const int64_t row = row0 + r, rest = row / a.H;
      const int     y = (int)(row - rest * a.H), w = (int)(rest / a.nplanes), ir = y - a.oy;
      const int     plane = (int)(rest - (int64_t)w * a.nplanes);
      s_in[r]  = ir >= 0 && ir < a.IH ? w * a.in_win + plane * a.in_plane + (int64_t)ir * a.in_row : INT64_MIN;
      s_pre[r] = (int64_t)y * n;
      s_out[r] = w * a.out_win + plane * a.out_plane + (int64_t)y * a.out_row;
    }
    __syncthreads();
    constexpr int U = 4; // independent loads in flight per thread
    for (int t0 = threadIdx.x; t0 < rows * n; t0 += U * kAnyThreads) {
      float2 v[U], L[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * kAnyThreads;
        v[u]        = make_float2(0.f, 0.f);
        L[u]        = make_float2(1.f, 0.f);
        if (t >= rows * n)
          continue;
        const int r = fdiv(t, pl.by_n), i = t - r * n, ic = i - a.ox;
        if (s_in[r] == INT64_MIN || ic < 0 || ic >= a.IW)
          continue;
        const int64_t off = s_in[r] + (int64_t)ic * a.in_col;
        v[u] = a.in_real ? make_float2(__ldg(reinterpret_cast<const float *>(a.in) + off), 0.f)
                         : __ldg(reinterpret_cast<const float2 *>(a.in) + off);
        if (a.pre != nullptr)
          L[u] = __ldg(a.pre + s_pre[r] + i);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * kAnyThreads;
        if (t < rows * n)
          b0[t] = flip(a.pre != nullptr ? cmul(v[u], L[u]) : v[u], a.inverse != 0);
      }
    }
    __syncthreads();
    const float2 *res = fft_smem<kAnyRB>(b0, b1, row_layout(n, rows), pl, tw);
    for (int t = threadIdx.x; t < rows * n; t += blockDim.x) {
      const int r = fdiv(t, pl.by_n), i = t - r * n;
      a.out[s_out[r] + i] = flip(res[t], a.inverse != 0);
    }
  }
}

// |v| without overflow or underflow of the squares (hypotf outside their safe range).
__device__ __forceinline__ float any_abs(float2 v) {
  const float s = fmaf(v.x, v.x, v.y * v.y);
  return s >= 1e-30f && s <= 1e37f ? __fsqrt_rn(s) : hypotf(v.x, v.y);
}

// A strip of C (a power of two) columns of one plane, interleaved in shared memory as they lie in it.
__global__ void __launch_bounds__(kAnyThreads, 2) any_cols_kernel(const __grid_constant__ ColPass a,
                                                               const __grid_constant__ GPlan pl, FastDiv by_C, int nstrip,
                                                               int64_t nwork, int magnitude) {
  extern __shared__ __align__(16) float2 sm[];
  const int n = pl.n, C = (int)by_C.d, lc = 31 - __clz(C);
  float2   *tw = sm, *b0 = sm + n, *b1 = b0 + (size_t)C * n;
  any_twiddles(tw, n);
  for (int64_t wk = blockIdx.x; wk < nwork; wk += gridDim.x) {
    const int64_t img = wk / nstrip;
    const int     x0 = (int)(wk - img * nstrip) * C, cw = min(C, a.W - x0);
    const int     w = (int)(img / a.nplanes), plane = (int)(img - (int64_t)w * a.nplanes);
    const float2 *in = a.in + w * a.in_win + plane * a.in_plane + x0;
    __syncthreads(); // the table is built; the previous strip is stored
    constexpr int U = 8;
    for (int t0 = threadIdx.x; t0 < n * C; t0 += U * kAnyThreads) {
      float2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * kAnyThreads, y = t >> lc, c = t & (C - 1);
        v[u] = t < n * C && c < cw ? __ldg(in + (int64_t)y * a.in_row + c) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int t = t0 + u * kAnyThreads;
        if (t < n * C)
          b0[t] = flip(v[u], a.inverse != 0);
      }
    }
    __syncthreads();
    const float2 *res = fft_smem<kAnyRB>(b0, b1, strip_layout(by_C), pl, tw);
    const int64_t o0  = w * a.out_win + plane * a.out_plane;
    for (int t = threadIdx.x; t < n * C; t += blockDim.x) {
      const int y = t >> lc, c = t & (C - 1);
      if (c >= cw)
        continue;
      const float2  v = flip(res[t], a.inverse != 0);
      const int64_t o = o0 + (int64_t)y * a.out_row + (int64_t)(x0 + c) * a.out_col;
      if (magnitude)
        reinterpret_cast<float *>(a.out)[o] = any_abs(v);
      else
        reinterpret_cast<float2 *>(a.out)[o] =
            a.post != nullptr ? cmul(v, __ldg(a.post + (int64_t)y * a.W + x0 + c)) : v;
    }
  }
}

size_t any_smem(int n, int rows, int pitch) {
  return (size_t)n * sizeof(float2) + 2 * (size_t)((rows + kAnyRB - 1) / kAnyRB * kAnyRB) * pitch * sizeof(float2);
}

// Persistent grid of a kernel with `smem` bytes per CTA.
template <typename K> int any_grid(K kern, size_t smem, int64_t work, unsigned *grid) {
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  HF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kAnyThreads, smem));
  *grid = (unsigned)std::min<int64_t>(work, (int64_t)std::max(1, per_sm) * sm_count());
  return HF_OK;
}

} // namespace

// 2 <= n whose buffers for one group of kAnyRB rows fit (n <= 3128).
bool fft_any_length(int n) { return n >= 2 && n <= kAnyMaxN && any_smem(n, kAnyRB, n | 1) <= kAnySmemMax; }

int launch_row_any(const RowPass &a, int nwin, cudaStream_t s) {
  GPlan pl;
  if (!make_plan(a.N, pl, kAnyMaxN))
    return fail(HF_ERR_UNSUPPORTED, "row pass: no plan for this length");
  int R = kAnyMaxRows; // at most as many rows as leave two CTAs per SM
  while (R > kAnyRB && any_smem(a.N, R, a.N) > kAnySmem)
    R -= kAnyRB;
  R = plan_rows(pl, 1, R, kAnyThreads);
  const int64_t nrows = (int64_t)nwin * a.nplanes * a.H;
  const size_t  smem  = any_smem(a.N, R, a.N);
  unsigned      grid  = 0;
  HF_TRY(any_grid(any_rows_kernel, smem, (nrows + R - 1) / R, &grid));
  any_rows_kernel<<<grid, kAnyThreads, smem, s>>>(a, pl, R, nrows);
  note_launch();
  return launch_status("any_rows_kernel");
}

int launch_col_any(const ColPass &a, int magnitude, int nwin, cudaStream_t s) {
  GPlan pl;
  if (!make_plan(a.H, pl, kAnyMaxN))
    return fail(HF_ERR_UNSUPPORTED, "column pass: no plan for this length");
  int C = 16; // at least 4 columns, so that a row of the strip is a whole 32-byte sector
  while (C > kAnyRB && any_smem(a.H, C, a.H) > kAnySmem)
    C /= 2;
  const int     nstrip = (a.W + C - 1) / C;
  const int64_t nwork  = (int64_t)nwin * a.nplanes * nstrip;
  const size_t  smem   = any_smem(a.H, C, a.H);
  unsigned      grid   = 0;
  HF_TRY(any_grid(any_cols_kernel, smem, nwork, &grid));
  any_cols_kernel<<<grid, kAnyThreads, smem, s>>>(a, pl, make_div((uint32_t)C), nstrip, nwork, magnitude);
  note_launch();
  return launch_status("any_cols_kernel");
}

} // namespace hf
