// Temporal band DFT: per pixel S_k = scale * sum_t x_t W[t][k] for k < nz, written as complex
// planes [nz][P] (optionally multiplied by a per-pixel lens).
//
// W is the T x nz complex matrix a window's SVD clutter filter and its band DFT reduce to,
// W = (I - V V^T) D[:, z0:z1]  (D the unnormalised DFT, V the removed eigenvectors), so this one
// kernel stands for RFFT/FFT along T + Slice + Copy (holonp/src/rfft.cu:150-160,
// fft.cu:234-252, graph_builder.cc:264-267) and for the filter, and Fresnel's lens multiply
// (the load callback of fresnel_diffraction.cu:262-303) is fused into its store.
//
// Plain form: FP32 CUDA-core FMAs, and their rate is the bound: T nz complex-by-real products per
// pixel, 60 GFLOP for 8 windows of 64 x 1024^2 at nz = 28 (0.83 ms at 72 TFLOP/s).
//  - A thread holds NB bins x 4 pixels of complex sums; (re, im) is one packed fp32x2 FMA, so a
//    frame costs 4 NB packed FMAs against NB / 2 broadcast loads of W, two loads of samples and
//    about 20 instructions of unpacking.  7 bins x 8 pixels with scalar FMAs and integer-to-float
//    conversions took 2.82 ms for those 8 windows.
//  - Integer samples are taken as x - m (exact; no conversion instruction) with m the pixel's own level,
//    the middle one of its first, middle and last sample, and m sum_t W is added at the end: the running
//    sums stay as small as the pixel's changes.  One level for every pixel (the middle of the format's
//    range) lost the dark ones: for 12-bit samples around 5 of T = 64, the error of a bin is 3e-5 of its rms
//    with 2048, 1.5e-7 with raw samples and 1.2e-7 with the pixel's level; in mid-range clutter 3e-7, 6e-7 and
//    1.4e-7.
//  - 128 threads per CTA, three CTAs per SM (about 170 registers each): 128 / KG lanes x 4 pixels by
//    KG bin groups.  The CTAs are persistent over the pixel tiles of a window, so W is staged once,
//    and the next tile's samples stream in by cp.async while this one is summed (long windows, whose two
//    tiles do not fit beside W, hold one).
#include <algorithm>

#include "frames.cuh"
#include "host/band_geom.hh"
#include "k_band.cuh"

namespace hf {

namespace {

template <int FMT> struct FmtBytes;
template <> struct FmtBytes<HF_MONO12P> { static constexpr int num = 3, den = 2; };
template <> struct FmtBytes<HF_U16> { static constexpr int num = 2, den = 1; };
template <> struct FmtBytes<HF_U8> { static constexpr int num = 1, den = 1; };
template <> struct FmtBytes<HF_F32> { static constexpr int num = 4, den = 1; };

constexpr float kMagic = 8388608.f; // 2^23: 2^23 + v is the float with v < 2^23 in its low bits

// Samples 4 g .. 4 g + 3 of a staged row: integers v as 2^23 + v, floats as they are.
template <int FMT> __device__ __forceinline__ void load4(const uint8_t *row, int g, float (&x)[kBandPX]) {
  const auto lift = [](uint32_t v) { return __uint_as_float(0x4B000000u | v); };
  if constexpr (FMT == HF_MONO12P) { // 48 bits from bit 0 (even g) or 16 (odd g) of two words
    const uint32_t *w  = reinterpret_cast<const uint32_t *>(row) + 3 * (g >> 1) + (g & 1);
    const uint32_t  a = w[0], b = w[1], sh = (g & 1) * 16;
    const uint32_t  lo = __funnelshift_r(a, b, sh), hi = b >> sh;
    x[0] = lift(lo & 0xFFFu);
    x[1] = lift((lo >> 12) & 0xFFFu);
    x[2] = lift(__funnelshift_r(lo, hi, 24) & 0xFFFu);
    x[3] = lift((hi >> 4) & 0xFFFu);
  } else if constexpr (FMT == HF_U16) {
    const uint2 v = reinterpret_cast<const uint2 *>(row)[g];
    x[0] = lift(v.x & 0xFFFFu), x[1] = lift(v.x >> 16);
    x[2] = lift(v.y & 0xFFFFu), x[3] = lift(v.y >> 16);
  } else if constexpr (FMT == HF_U8) {
    const uint32_t v = reinterpret_cast<const uint32_t *>(row)[g];
    x[0] = lift(v & 0xFFu), x[1] = lift((v >> 8) & 0xFFu);
    x[2] = lift((v >> 16) & 0xFFu), x[3] = lift(v >> 24);
  } else { // F32
    const float4 v = reinterpret_cast<const float4 *>(row)[g];
    x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
  }
}

// Entry (t, k) of window w's matrix: the supplied W, or the DFT bin exp(-2 pi i t (z0+k) / T).
__device__ __forceinline__ float2 wmat_entry(const BandArgs &a, int w, int t, int k) {
  if (a.wmat != nullptr)
    return a.wmat[(int64_t)w * a.wmat_stride + (int64_t)t * a.nz + k];
  const int m = (int)(((int64_t)t * (a.z0 + k)) % a.T);
  float     s, c;
  sincospif(-2.0f * (float)m / (float)a.T, &s, &c);
  return make_float2(c, s);
}

// Copies `bytes` bytes of a row into shared memory (16-byte aligned), zero beyond `valid`.  `unit` is
// the common alignment of every row of the tile: 16 and 4 go by cp.async, less byte by byte.
__device__ __forceinline__ void stage_tile(uint8_t *dst, const uint8_t *base, const int64_t *foff, int T, int bytes,
                                           int valid, int unit) {
  if (unit >= 4) {
    const int per = bytes / unit;
    for (int i = threadIdx.x; i < T * per; i += kBandThr) {
      const int      t = i / per, o = (i - t * per) * unit, n = max(0, min(unit, valid - o));
      const uint8_t *src = base + foff[t] + (n > 0 ? o : 0);
      const uint32_t d   = (uint32_t)__cvta_generic_to_shared(dst + t * bytes + o);
      if (unit == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    }
  } else {
    constexpr int U = 8; // loads in flight per thread
    for (int i0 = threadIdx.x; i0 < T * bytes; i0 += U * kBandThr) {
      uint8_t v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * kBandThr, t = i / bytes, o = i - t * bytes;
        v[u]        = i < T * bytes && o < valid ? __ldg(base + foff[t] + o) : 0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i0 + u * kBandThr < T * bytes)
          dst[i0 + u * kBandThr] = v[u];
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int FMT, int NB, int STAGES>
__global__ void __launch_bounds__(kBandThr, 3) band_dft_fp32_kernel(BandArgs a, int KG, int nzpad, int unit, int vec) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int  num = FmtBytes<FMT>::num, den = FmtBytes<FMT>::den;
  constexpr bool kLevel = FMT != HF_F32;
  const int     w       = blockIdx.y;
  const int     tile_px = kBandThr * kBandPX / KG, bytes = tile_px * num / den;
  uint8_t *stage = smem;                                                            // [STAGES][T][bytes]
  float2  *w_sh  = reinterpret_cast<float2 *>(smem + STAGES * (size_t)a.T * bytes); // [T][nzpad]
  float2  *wsum  = w_sh + (size_t)a.T * nzpad;                                  // [nzpad] sum_t W
  int64_t *foff  = reinterpret_cast<int64_t *>(wsum + nzpad);                    // [T] frame offsets
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int t = tid; t < a.T; t += kBandThr)
    foff[t] = a.ring.frame(w, t) - a.ring.base;
  __syncthreads();
  const int64_t ntiles = (a.P + tile_px - 1) / tile_px;
  const auto    fetch  = [&](int64_t tile, int s) {
    if (tile >= ntiles) {
      asm volatile("cp.async.commit_group;" ::: "memory");
      return;
    }
    const int64_t p0 = tile * tile_px;
    const int     np = (int)min((int64_t)tile_px, a.P - p0);
    stage_tile(stage + (size_t)s * a.T * bytes, a.ring.base + p0 * num / den, foff, a.T, bytes, np * num / den, unit);
  };
  fetch(blockIdx.x, 0);
  for (int i = tid; i < a.T * nzpad; i += kBandThr) {
    const int t = i / nzpad, k = i % nzpad;
    w_sh[i]     = k < a.nz ? wmat_entry(a, w, t, k) : make_float2(0.f, 0.f);
  }
  __syncthreads();
  for (int k = tid; k < nzpad; k += kBandThr) {
    double sr = 0.0, si = 0.0;
    if constexpr (kLevel)
      for (int t = 0; t < a.T; ++t)
        sr += (double)w_sh[t * nzpad + k].x, si += (double)w_sh[t * nzpad + k].y;
    wsum[k] = make_float2((float)sr, (float)si);
  }

  const int kgi = warp % KG, g = (warp / KG) * 32 + lane; // bin group, 4-pixel group of the tile
  int       s   = 0;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, s ^= STAGES - 1) {
    if constexpr (STAGES == 2) {
      fetch(tile + gridDim.x, s ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    const uint8_t *rows = stage + (size_t)s * a.T * bytes;
    const int64_t  p0   = tile * tile_px + (int64_t)g * kBandPX;
    float          m[kBandPX]; // 2^23 + the pixel's level
    if constexpr (kLevel) {
      float m1[kBandPX], m2[kBandPX];
      load4<FMT>(rows, g, m);
      load4<FMT>(rows + (a.T / 2) * bytes, g, m1);
      load4<FMT>(rows + (a.T - 1) * bytes, g, m2);
#pragma unroll
      for (int p = 0; p < kBandPX; ++p)
        m[p] = fmaxf(fminf(m[p], m1[p]), fminf(fmaxf(m[p], m1[p]), m2[p]));
    }
    for (int kc = kgi * NB; kc < a.nz; kc += KG * NB) {
      float2 acc[NB][kBandPX];
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int p = 0; p < kBandPX; ++p)
          acc[b][p] = make_float2(0.f, 0.f);
      const float4 *wr = reinterpret_cast<const float4 *>(w_sh + kc);
#pragma unroll 2
      for (int t = 0; t < a.T; ++t) {
        float x[kBandPX];
        load4<FMT>(rows + t * bytes, g, x);
        if constexpr (kLevel)
#pragma unroll
          for (int p = 0; p < kBandPX; ++p)
            x[p] -= m[p];
#pragma unroll
        for (int b = 0; b < NB; b += 2) {
          const float4 wv = wr[t * (nzpad / 2) + b / 2];
#pragma unroll
          for (int p = 0; p < kBandPX; ++p) {
            acc[b][p]     = cfma2(make_float2(x[p], x[p]), make_float2(wv.x, wv.y), acc[b][p]);
            acc[b + 1][p] = cfma2(make_float2(x[p], x[p]), make_float2(wv.z, wv.w), acc[b + 1][p]);
          }
        }
      }
      if (p0 >= a.P)
        continue;
      float2 L[kBandPX];
#pragma unroll
      for (int p = 0; p < kBandPX; ++p)
        L[p] = a.lens != nullptr && p0 + p < a.P ? __ldg(a.lens + p0 + p) : make_float2(1.f, 0.f);
      float2 *out = a.out + (int64_t)w * a.out_win + p0;
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int k = kc + b;
        if (k >= a.nz)
          break;
        float2 v[kBandPX];
#pragma unroll
        for (int p = 0; p < kBandPX; ++p) {
          if constexpr (kLevel)
            acc[b][p] = cfma2(make_float2(m[p] - kMagic, m[p] - kMagic), wsum[k], acc[b][p]);
          v[p] = cscale(acc[b][p], a.scale);
          if (a.lens != nullptr)
            v[p] = cmul(v[p], L[p]);
        }
        float2 *o = out + (int64_t)k * a.out_plane;
        if (vec && p0 + kBandPX <= a.P) {
          reinterpret_cast<float4 *>(o)[0] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
          reinterpret_cast<float4 *>(o)[1] = make_float4(v[2].x, v[2].y, v[3].x, v[3].y);
        } else {
#pragma unroll
          for (int p = 0; p < kBandPX; ++p)
            if (p0 + p < a.P)
              o[p] = v[p];
        }
      }
    }
    __syncthreads(); // this tile's rows are read: the stage takes the tile after next (one stage: the next)
    if constexpr (STAGES == 1)
      fetch(tile + gridDim.x, 0);
  }
}

// One thread per pixel; any format (complex frames included), any P.
template <int FMT> __global__ void band_dft_simple_kernel(BandArgs a) {
  const int     w = blockIdx.y;
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.P)
    return;
  float2      *outp = a.out + (int64_t)w * a.out_win + p;
  const float2 L = a.lens ? a.lens[p] : make_float2(1.f, 0.f);
  for (int k0 = 0; k0 < a.nz; k0 += 8) {
    float2 acc[8];
#pragma unroll
    for (int b = 0; b < 8; ++b)
      acc[b] = make_float2(0.f, 0.f);
    for (int t = 0; t < a.T; ++t) {
      const uint8_t *fr = a.ring.frame(w, t);
      float2 x;
      if constexpr (FMT == HF_CF32)
        x = reinterpret_cast<const float2 *>(fr)[p];
      else
        x = make_float2(sample<FMT>(fr, p), 0.f);
#pragma unroll
      for (int b = 0; b < 8; ++b)
        if (k0 + b < a.nz)
          acc[b] = cadd(acc[b], cmul(x, wmat_entry(a, w, t, k0 + b)));
    }
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if (k0 + b < a.nz) {
        float2 v = cscale(acc[b], a.scale);
        if (a.lens)
          v = cmul(v, L);
        outp[(int64_t)(k0 + b) * a.out_plane] = v;
      }
  }
}

template <int FMT, int NB> int launch_nb(const BandArgs &a, const BandGeom &g, int unit, int vec, int nwin, cudaStream_t s) {
  auto kern = g.stages == 2 ? band_dft_fp32_kernel<FMT, NB, 2> : band_dft_fp32_kernel<FMT, NB, 1>;
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
  const int     tile_px = kBandThr * kBandPX / g.KG;
  const int64_t ntiles  = (a.P + tile_px - 1) / tile_px;
  const int     per_sm  = std::max(1, std::min(3, (int)(kBandSmem / g.smem)));
  const int64_t ctas    = std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)per_sm * sm_count() / nwin));
  kern<<<dim3((unsigned)ctas, nwin), kBandThr, g.smem, s>>>(a, g.KG, g.nzpad, unit, vec);
  note_launch();
  return launch_status("band_dft_fp32_kernel");
}

template <int FMT> int launch_fp32(const BandArgs &a, int nwin, cudaStream_t s) {
  const BandGeom g = band_geom(a.T, a.nz, FmtBytes<FMT>::num, FmtBytes<FMT>::den);
  if (g.smem > kBandSmem)
    return HF_ERR_UNSUPPORTED;
  const uintptr_t rows = reinterpret_cast<uintptr_t>(a.ring.base) | (uintptr_t)a.ring.frame_bytes;
  const int       unit = rows % 16 == 0 ? 16 : (rows % 4 == 0 ? 4 : 1);
  const int       vec  = reinterpret_cast<uintptr_t>(a.out) % 16 == 0 && a.out_plane % 2 == 0 && a.out_win % 2 == 0;
  switch (g.NB) {
  case 4: return launch_nb<FMT, 4>(a, g, unit, vec, nwin, s);
  case 6: return launch_nb<FMT, 6>(a, g, unit, vec, nwin, s);
  case 8: return launch_nb<FMT, 8>(a, g, unit, vec, nwin, s);
  case 10: return launch_nb<FMT, 10>(a, g, unit, vec, nwin, s);
  case 12: return launch_nb<FMT, 12>(a, g, unit, vec, nwin, s);
  default: return launch_nb<FMT, 14>(a, g, unit, vec, nwin, s);
  }
}

template <int FMT> int launch_simple(const BandArgs &a, int nwin, cudaStream_t s) {
  dim3 grid((unsigned)((a.P + 127) / 128), nwin);
  band_dft_simple_kernel<FMT><<<grid, 128, 0, s>>>(a);
  note_launch();
  return launch_status("band_dft_simple_kernel");
}

} // namespace

int launch_band_dft(const BandArgs &a, int fmt, int nwin, cudaStream_t s) {
  HF_CHECK_ARG(a.T > 0 && a.P > 0 && a.nz > 0 && nwin > 0, "band_dft: empty problem");
  int rc = HF_ERR_UNSUPPORTED; // (windows whose samples or W exceed shared memory, and complex frames)
  switch (fmt) {
  case HF_MONO12P: rc = launch_fp32<HF_MONO12P>(a, nwin, s); break;
  case HF_U16: rc = launch_fp32<HF_U16>(a, nwin, s); break;
  case HF_U8: rc = launch_fp32<HF_U8>(a, nwin, s); break;
  case HF_F32: rc = launch_fp32<HF_F32>(a, nwin, s); break;
  default: break;
  }
  if (rc != HF_ERR_UNSUPPORTED)
    return rc;
  switch (fmt) {
  case HF_MONO12P: return launch_simple<HF_MONO12P>(a, nwin, s);
  case HF_U16: return launch_simple<HF_U16>(a, nwin, s);
  case HF_U8: return launch_simple<HF_U8>(a, nwin, s);
  case HF_F32: return launch_simple<HF_F32>(a, nwin, s);
  case HF_CF32: return launch_simple<HF_CF32>(a, nwin, s);
  default: return fail(HF_ERR_INVALID, "band_dft: unsupported input dtype");
  }
}

} // namespace hf
