// Angular spectrum columns: forward column FFT, transfer function, inverse column FFT of every band
// plane, in place in HBM (the TF sandwich between the forward and the inverse row passes).
//
// Bound: one read and one write of the planes (1.64 GB for 4 windows x 28 planes of 768^2 placed in
// 1024^2) against two transforms per column.  A CTA owns a strip of kTfC columns of one window and
// walks its planes, two CTAs per SM:
//  - the next plane's strip arrives by cp.async (16-byte pieces, zero outside the rows the placement
//    fills, which the row pass therefore neither transforms nor writes) while this one is transformed;
//  - thread (n2, c) takes the column's samples n2 + 32 n1, N1-point DFT, twiddles from a [N1][32]
//    table, exchange in the landed stage at k1 * (32 C + C) + n2 * C + c (conflict-free both ways);
//  - thread (k1, c) takes the 32-point DFT, multiplies by its 32 transfer-function values, which stay
//    in registers for every plane of the strip, and runs the transposed steps back: inverse 32-point
//    DFT, twiddles from the transposed table, the same exchange positions, inverse N1-point DFT.
// It replaces strips of 8 columns in one CTA per SM with loads into registers, swizzled twiddle
// look-ups and the transfer function read per plane: 1440 us for those 4 windows, 559 us here (2.9 TB/s;
// 8 warps per SM wait on their shared-memory exchanges).
#include <algorithm>

#include "fft_core.cuh"
#include "k_fft2d.cuh"

namespace hf {
namespace {

constexpr int kTfC = 4; // columns per strip

template <int N1> struct TfGeom {
  static constexpr int    N     = 32 * N1;
  static constexpr int    XRow  = 32 * kTfC + kTfC;          // exchange row (one k1) in float2
  static constexpr int    Slot  = N1 * XRow;                 // >= N * kTfC
  static constexpr size_t smem  = sizeof(float2) * (2 * (size_t)Slot + 2 * (size_t)N);
};

template <int N1>
__global__ void __launch_bounds__(32 * kTfC, 2) col_tf_kernel(ColPass a, int nplanes_z) {
  using G             = TfGeom<N1>;
  constexpr int N     = G::N, C = kTfC, NT = 32 * C;
  extern __shared__ __align__(16) float2 sm2[];
  float2 *stage = sm2, *tw = sm2 + 2 * G::Slot, *twt = tw + N; // twiddles [k1][n2] and [n2][k1]
  const int tid = threadIdx.x, n2 = tid / C, c = tid % C, k1 = n2;
  const int strip = blockIdx.x, w = blockIdx.z, p0 = blockIdx.y, pstep = nplanes_z;
  const int col   = strip * C + c;
  const float2 *in = a.in + w * a.in_win + strip * C;
  const auto fetch = [&](int plane, int s) { // rows of C columns as 16-byte pieces, zero outside the valid rows
    if (plane < a.nplanes) {
      const float2 *src = in + (int64_t)plane * a.in_plane;
      float2       *dst = stage + s * G::Slot;
#pragma unroll 4
      for (int i = tid; i < N * C / 2; i += NT) {
        const int      row = i / (C / 2), h = i % (C / 2);
        const bool     ok  = row >= a.row_lo && row < a.row_hi;
        const uint32_t d   = (uint32_t)__cvta_generic_to_shared(dst + row * C + 2 * h);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d),
                     "l"(src + (ok ? (int64_t)row * a.in_row : 0) + 2 * h), "r"(ok ? 16 : 0)
                     : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(p0, 0);
  fetch(p0 + pstep, 1);
  for (int i = tid; i < N; i += NT) {
    float sv, cv;
    sincospif(-2.0f * (float)((i >> 5) * (i & 31)) / (float)N, &sv, &cv);
    tw[i]                          = make_float2(cv, sv);
    twt[(i & 31) * N1 + (i >> 5)] = make_float2(cv, sv);
  }
  float2 tf[32]; // rows k1 + N1 k2 of the transfer function
  if (k1 < N1) {
#pragma unroll
    for (int k2 = 0; k2 < 32; ++k2)
      tf[k2] = __ldg(a.tf + (int64_t)(k1 + N1 * k2) * a.W + col);
  }
  int s = 0;
  for (int plane = p0; plane < a.nplanes; plane += pstep, s ^= 1) {
    float2 *st = stage + s * G::Slot;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads(); // every thread's copies of this plane have landed
    float2 x[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1)
      x[n1] = st[(n2 + 32 * n1) * C + c];
    __syncthreads(); // the strip is in registers: the stage becomes the exchange
    dft_reg<N1, false>(x);
#pragma unroll
    for (int k = 0; k < N1; ++k)
      st[k * G::XRow + n2 * C + c] = k == 0 ? x[k] : cmul(x[k], tw[k * 32 + n2]);
    __syncthreads();
    if (k1 < N1) {
      float2 y[32];
#pragma unroll
      for (int j = 0; j < 32; ++j)
        y[j] = st[k1 * G::XRow + j * C + c];
      dft_reg<32, false>(y);
#pragma unroll
      for (int k2 = 0; k2 < 32; ++k2)
        y[k2] = cmul(y[k2], tf[k2]);
      dft_reg<32, true>(y); // index k2 of the spectrum -> kb
#pragma unroll
      for (int kb = 0; kb < 32; ++kb) {
        float2 v = y[kb];
        if (kb != 0) {
          const float2 t = twt[kb * N1 + k1];
          v              = cmul(v, make_float2(t.x, -t.y));
        }
        st[k1 * G::XRow + kb * C + c] = v; // the positions this thread read
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N1; ++k)
      x[k] = st[k * G::XRow + n2 * C + c];
    __syncthreads(); // the stage is read: it takes the plane after next
    fetch(plane + 2 * pstep, s);
    dft_reg<N1, true>(x);
    float2 *dst = reinterpret_cast<float2 *>(a.out) + w * a.out_win + (int64_t)plane * a.out_plane + col;
#pragma unroll
    for (int ka = 0; ka < N1; ++ka)
      dst[(int64_t)(n2 + 32 * ka) * a.out_row] = x[ka];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int N1> int launch_tf(const ColPass &a, int nwin, cudaStream_t s) {
  HF_CUDA(cudaFuncSetAttribute(col_tf_kernel<N1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TfGeom<N1>::smem));
  const int strips = a.W / kTfC;
  // a strip's planes stay in one CTA (its transfer function and tables are loaded once) unless that
  // leaves SMs idle: then they are split until two CTAs per SM have work
  const int64_t want = (2LL * sm_count() + (int64_t)strips * nwin - 1) / ((int64_t)strips * nwin);
  const int     pz   = (int)std::max<int64_t>(1, std::min<int64_t>(a.nplanes, want));
  col_tf_kernel<N1><<<dim3(strips, pz, nwin), 32 * kTfC, TfGeom<N1>::smem, s>>>(a, pz);
  note_launch();
  return launch_status("col_tf_kernel");
}

// Column transform to complex planes (optionally times a [H][W] factor) or magnitudes, over the same
// strips and loads.  G = max(1, 32 / N1) planes at a time, so that short columns have a 32-point DFT for
// every thread in the second stage; the magnitudes take one range test per 32 values (abs32).  Strips of 8
// columns, one plane at a time with loads into registers and a hypotf call per value, took 40 us for 20
// planes of 512^2 (63 MB), 28 us here.
template <int N1, bool INV, bool MAG>
__global__ void __launch_bounds__(32 * kTfC, 2) col_strip_kernel(ColPass a) {
  using T             = TfGeom<N1>;
  constexpr int N     = T::N, C = kTfC, NT = 32 * C, G = N1 < 32 ? 32 / N1 : 1;
  extern __shared__ __align__(16) float2 sm2[];
  float2 *stage = sm2, *tw = sm2 + 2 * G * T::Slot; // [2][G][Slot], [k1][n2]
  const int tid = threadIdx.x, n2 = tid / C, c = tid % C, k1 = n2 % N1, g2 = n2 / N1;
  const int strip = blockIdx.x, w = blockIdx.z, col = strip * C + c;
  const int ngroups = (a.nplanes + G - 1) / G;
  const float2 *in = a.in + w * a.in_win + strip * C;
  const auto fetch = [&](int grp, int s) {
    if (grp < ngroups)
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (grp * G + g < a.nplanes) {
          const float2 *src = in + (int64_t)(grp * G + g) * a.in_plane;
          const uint32_t d  = (uint32_t)__cvta_generic_to_shared(stage + (size_t)(s * G + g) * T::Slot);
#pragma unroll 4
          for (int i = tid; i < N * C / 2; i += NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i),
                         "l"(src + (int64_t)(i / (C / 2)) * a.in_row + 2 * (i % (C / 2)))
                         : "memory");
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(blockIdx.y, 0);
  fetch(blockIdx.y + gridDim.y, 1);
  for (int i = tid; i < N; i += NT) {
    float sv, cv;
    sincospif((INV ? 2.0f : -2.0f) * (float)((i >> 5) * (i & 31)) / (float)N, &sv, &cv);
    tw[i] = make_float2(cv, sv);
  }
  int s = 0;
  for (int grp = blockIdx.y; grp < ngroups; grp += gridDim.y, s ^= 1) {
    float2   *st = stage + (size_t)s * G * T::Slot;
    const int np = min(G, a.nplanes - grp * G);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads(); // every thread's copies of this group have landed
    float2 x[G][N1];
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (g < np)
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1)
          x[g][n1] = st[g * T::Slot + (n2 + 32 * n1) * C + c];
    __syncthreads(); // the strips are in registers: the stage becomes the exchange
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (g < np) {
        dft_reg<N1, INV>(x[g]);
#pragma unroll
        for (int k = 0; k < N1; ++k)
          st[g * T::Slot + k * T::XRow + n2 * C + c] = k == 0 ? x[g][k] : cmul(x[g][k], tw[k * 32 + n2]);
      }
    __syncthreads();
    float2     y[32];
    const bool on = g2 < np;
    if (on) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        y[j] = st[g2 * T::Slot + k1 * T::XRow + j * C + c];
    }
    __syncthreads(); // the exchange is read: the stage takes the group after next
    fetch(grp + 2 * gridDim.y, s);
    if (on) {
      dft_reg<32, INV>(y);
      const int64_t o = w * a.out_win + (int64_t)(grp * G + g2) * a.out_plane + (int64_t)col * a.out_col;
      if constexpr (MAG) {
        abs32(y);
        float *dst = reinterpret_cast<float *>(a.out) + o;
#pragma unroll
        for (int k2 = 0; k2 < 32; ++k2)
          dst[(int64_t)(k1 + N1 * k2) * a.out_row] = y[k2].x;
      } else {
        float2 *dst = reinterpret_cast<float2 *>(a.out) + o;
        if (a.post != nullptr) {
#pragma unroll
          for (int k2 = 0; k2 < 32; ++k2)
            y[k2] = cmul(y[k2], __ldg(a.post + (int64_t)(k1 + N1 * k2) * a.W + col));
        }
#pragma unroll
        for (int k2 = 0; k2 < 32; ++k2)
          dst[(int64_t)(k1 + N1 * k2) * a.out_row] = y[k2];
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

template <int N1, bool INV> int launch_strip(const ColPass &a, bool magnitude, int nwin, cudaStream_t s) {
  constexpr int  G    = N1 < 32 ? 32 / N1 : 1;
  constexpr size_t sm = sizeof(float2) * (2 * (size_t)G * TfGeom<N1>::Slot + TfGeom<N1>::N);
  auto kern = magnitude ? col_strip_kernel<N1, INV, true> : col_strip_kernel<N1, INV, false>;
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  // three CTAs per SM's worth of work, each over as many groups as that leaves it
  const int     strips = a.W / kTfC, ngroups = (a.nplanes + G - 1) / G;
  const int64_t want   = (3LL * sm_count() + (int64_t)strips * nwin - 1) / ((int64_t)strips * nwin);
  const int     gy     = (int)std::max<int64_t>(1, std::min<int64_t>(ngroups, want));
  kern<<<dim3(strips, gy, nwin), 32 * kTfC, sm, s>>>(a);
  note_launch();
  return launch_status("col_strip_kernel");
}

template <bool INV> int launch_strip_len(const ColPass &a, bool magnitude, int nwin, cudaStream_t s) {
  switch (a.H) {
  case 64: return launch_strip<2, INV>(a, magnitude, nwin, s);
  case 128: return launch_strip<4, INV>(a, magnitude, nwin, s);
  case 256: return launch_strip<8, INV>(a, magnitude, nwin, s);
  case 512: return launch_strip<16, INV>(a, magnitude, nwin, s);
  case 768: return launch_strip<24, INV>(a, magnitude, nwin, s);
  case 1024: return launch_strip<32, INV>(a, magnitude, nwin, s);
  default: return fail(HF_ERR_UNSUPPORTED, "column strips need H <= 1024");
  }
}

} // namespace

bool col_strip_supported(const ColPass &a) {
  return fft_fast_length(a.H) && a.H <= 1024 && a.W % kTfC == 0 && (reinterpret_cast<uintptr_t>(a.in) & 15) == 0 &&
         a.in_win % 2 == 0 && a.in_plane % 2 == 0 && a.in_row % 2 == 0;
}

int launch_col_strip(const ColPass &a, bool magnitude, int nwin, cudaStream_t s) {
  return a.inverse ? launch_strip_len<true>(a, magnitude, nwin, s) : launch_strip_len<false>(a, magnitude, nwin, s);
}

bool col_tf_supported(const ColPass &a) { return col_strip_supported(a) && a.inverse == 0 && a.out_col == 1; }

int launch_col_tf(const ColPass &a, int nwin, cudaStream_t s) {
  switch (a.H) {
  case 64: return launch_tf<2>(a, nwin, s);
  case 128: return launch_tf<4>(a, nwin, s);
  case 256: return launch_tf<8>(a, nwin, s);
  case 512: return launch_tf<16>(a, nwin, s);
  case 768: return launch_tf<24>(a, nwin, s);
  case 1024: return launch_tf<32>(a, nwin, s);
  default: return fail(HF_ERR_UNSUPPORTED, "transfer-function column pass needs H <= 1024");
  }
}

} // namespace hf
