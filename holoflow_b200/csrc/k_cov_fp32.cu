// Gram matrix of a window's frames on the CUDA cores, any T <= 128, any sample format and any row
// alignment: 16-bit and float frames, and 8/12-bit frames the tensor-core kernel cannot address.  Sums in
// FP32 for the frames that cov_sums_fp32 names (T = 32, 64, 128 in aligned rows), in float64 for the rest,
// where integer samples give the exact matrix (up to 2^53).
//
// Bound: T (T + 1) / 2 products per pixel on the FMA pipe, against shared-memory reads of the
// operands.  A thread sums an 8 x 8 block of the upper triangle: four 16-byte reads feed 64 FMAs, which
// keeps the two pipes level; the 4 x 4 blocks before read 2 for 16.  The blocks of one pixel occupy
// U = NB (NB + 1) / 2 threads (NB = ceil(T / 8)) and the CTA's 256 threads work on 256 / U pixels at
// once.  Samples are staged four frames of one pixel per thread, so the transposed 16-byte stores are
// conflict-free (row stride = 1 mod 8 chunks).
//  - FP32: staged as x - shift, exact; the shift is undone in float64 by the reduction, from exact
//    integer frame sums (summed from the staged tile: 64-bit shared atomics per sample quad took half of
//    the kernel).  Two CTAs of 256 threads per SM (the registers of 288 threads fit once, whose load
//    latency nothing covers: 165 us).  Measured, 2 windows of 32 x 600 x 800 16-bit frames, kernel +
//    reduction: 331 -> 94 us.
//  - float64: staged as x and widened as it is read; the block takes 128 registers, so one CTA per SM, and
//    three times the loads in flight cover for the second (12-bit frames spill with them).  Measured, 2 windows
//    of 50 x 600 x 800 16-bit frames: 275 us (in FP32 180; float64 needs 96 at its pipe's rate), 16 of 50 x 16384
//    91 with the reduction, 2551 with a thread per entry.
#include <algorithm>

#include "host/cov_split.hh"
#include "k_pca.cuh"

namespace hf {

namespace {

constexpr int kCovThr = 256;

struct CovGeom {
  int NB, U, G, PX, XS; // 8-frame blocks, upper blocks, pixel groups, pixels per tile, row stride
  int lh;               // 2^lh lanes add the groups' sums of an entry
  int nxs;              // floats of the tile (and of the final block rows, 8 sums per thread)
  size_t smem;
};

CovGeom cov_geom(int T) {
  CovGeom g{};
  g.NB = (T + 7) / 8, g.U = g.NB * (g.NB + 1) / 2, g.G = kCovThr / g.U, g.XS = 8 * g.NB + 4;
  // the multiple of 32 pixels (whole warps stage one frame quad) that wastes least over the groups
  double best = 1e9;
  for (int px = 64; px <= 256; px += 32) {
    const double waste = (double)((px + g.G - 1) / g.G * g.G) / px;
    if ((size_t)px * g.XS * sizeof(float) <= 48 * 1024 && waste < best - 1e-9)
      best = waste, g.PX = px;
  }
  for (g.lh = 0; g.lh < 5 && (2 << g.lh) * g.U * 8 <= kCovThr;)
    ++g.lh;
  g.nxs  = std::max(g.PX * g.XS, 2 * 8 * kCovThr);
  g.smem = (size_t)g.nxs * sizeof(float) + 128 * (sizeof(int64_t) + sizeof(unsigned long long));
  return g;
}

template <int FMT> __device__ __forceinline__ uint32_t raw_sample(const uint8_t *frame, int64_t p) {
  if constexpr (FMT == HF_F32)
    return __float_as_uint(__ldg(reinterpret_cast<const float *>(frame) + p));
  else if constexpr (FMT == HF_U16)
    return __ldg(reinterpret_cast<const uint16_t *>(frame) + p);
  else if constexpr (FMT == HF_U8)
    return __ldg(frame + p);
  else {
    const int64_t  q  = (p >> 1) * 3;
    const uint32_t b0 = __ldg(frame + q + (p & 1)), b1 = __ldg(frame + q + (p & 1) + 1);
    return (p & 1) ? (b0 >> 4) | (b1 << 4) : b0 | ((b1 & 0xFu) << 8);
  }
}

// A staged sample as an operand.  For float64 sums integers stay integers in the tile and become 2^52 + v by
// their bits, 2^52 taken off: one instruction of the FP64 pipe instead of a conversion (308 -> 288 us for those 2 windows).
template <int FMT, typename Acc> __device__ __forceinline__ Acc widen(float x) {
  if constexpr (FMT != HF_F32 && sizeof(Acc) == 8)
    return __hiloint2double(0x43300000, __float_as_int(x)) - 4503599627370496.0;
  else
    return (Acc)x;
}

// Acc: float, or double with shift = 0 and no frame sums.
template <int FMT, typename Acc>
__global__ void __launch_bounds__(kCovThr, sizeof(Acc) == 4 ? 2 : 1)
    cov_cores_kernel(FrameRing ring, int T, int64_t P, float shift, CovGeom g, Acc *partial, double *sums) {
  constexpr bool kShift = FMT != HF_F32 && sizeof(Acc) == 4;
  constexpr bool kRaw   = !kShift; // the tile holds the samples' bits
  extern __shared__ __align__(16) float xs[]; // [PX][XS]
  int64_t            *foff = reinterpret_cast<int64_t *>(xs + g.nxs);                // [128]
  unsigned long long *ssum = reinterpret_cast<unsigned long long *>(foff + 128);     // [128]
  const int tid = threadIdx.x, w = blockIdx.y;
  const int grp = tid / g.U, blk = tid % g.U;
  int       bi = 0, rem = blk; // upper-triangle block index -> (bi, bj), bi <= bj
  while (rem >= g.NB - bi) {
    rem -= g.NB - bi;
    ++bi;
  }
  const int bj = bi + rem;
  Acc       acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      acc[i][j] = Acc(0);
  int64_t fsum[4] = {0, 0, 0, 0}; // this warp's share of the sums of frames lane + 32 c
  if (tid < 128) {
    foff[tid] = ring.frame(w, min(tid, T - 1)) - ring.base;
    ssum[tid] = 0ull;
  }
  __syncthreads();

  const int64_t ntiles = (P + g.PX - 1) / g.PX;
  const int     items  = 2 * g.NB * g.PX; // (frame quad, pixel), pixel fastest
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t p0 = tile * g.PX;
    constexpr int V = sizeof(Acc) == 4 || FMT == HF_MONO12P ? 4 : 12; // frame quads in flight per thread
    for (int i0 = tid & ~31; i0 < items; i0 += V * kCovThr) { // whole warps: PX is a multiple of 32
      uint32_t v[V][4];
#pragma unroll
      for (int u = 0; u < V; ++u) { // unconditional loads (clamped addresses), so that all are in flight
        if (V > 4 && i0 + u * kCovThr >= items)
          break; // (a whole warp's; of 4 at most 3 repeat the last items)
        const int     it = min(i0 + u * kCovThr, items - 32), tq = it / g.PX, p = it - tq * g.PX + (tid & 31);
        const int64_t pc = min(p0 + p, P - 1);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          v[u][q] = raw_sample<FMT>(ring.base + foff[4 * tq + q], pc);
      }
#pragma unroll
      for (int u = 0; u < V; ++u) {
        const int it = i0 + u * kCovThr, tq = it / g.PX, p = it - tq * g.PX + (tid & 31);
        if (it < items) {
          float x[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float c = kRaw ? __uint_as_float(v[u][q])
                                 : __uint_as_float(0x4B000000u | v[u][q]) - (8388608.f + shift);
            x[q]          = p0 + p < P && 4 * tq + q < T ? c : 0.f;
          }
          *reinterpret_cast<float4 *>(xs + p * g.XS + 4 * tq) = make_float4(x[0], x[1], x[2], x[3]);
        }
      }
    }
    __syncthreads();
    if constexpr (kShift) { // frame sums: a tile's (at most 256 values below 2^16) are exact in FP32
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = (tid & 31) + 32 * c;
        if (32 * c < 8 * g.NB) {
          float s0 = 0.f, s1 = 0.f;
          if (t < 8 * g.NB)
            for (int p = tid >> 5; p < g.PX; p += 2 * (kCovThr / 32)) {
              s0 += xs[p * g.XS + t];
              s1 += p + kCovThr / 32 < g.PX ? xs[(p + kCovThr / 32) * g.XS + t] : 0.f;
            }
          fsum[c] += (int64_t)(s0 + s1);
        }
      }
    }
    if (grp < g.G) {
      const float *xa = xs + 8 * bi, *xb = xs + 8 * bj;
      for (int p = grp; p < g.PX; p += g.G) {
        const float4 a0 = *reinterpret_cast<const float4 *>(xa + p * g.XS), a1 = *reinterpret_cast<const float4 *>(xa + p * g.XS + 4);
        const float4 b0 = *reinterpret_cast<const float4 *>(xb + p * g.XS), b1 = *reinterpret_cast<const float4 *>(xb + p * g.XS + 4);
        const Acc    va[8] = {widen<FMT, Acc>(a0.x), widen<FMT, Acc>(a0.y), widen<FMT, Acc>(a0.z), widen<FMT, Acc>(a0.w),
                              widen<FMT, Acc>(a1.x), widen<FMT, Acc>(a1.y), widen<FMT, Acc>(a1.z), widen<FMT, Acc>(a1.w)};
        const Acc    vb[8] = {widen<FMT, Acc>(b0.x), widen<FMT, Acc>(b0.y), widen<FMT, Acc>(b0.z), widen<FMT, Acc>(b0.w),
                              widen<FMT, Acc>(b1.x), widen<FMT, Acc>(b1.y), widen<FMT, Acc>(b1.z), widen<FMT, Acc>(b1.w)};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[i][j] = fma(va[i], vb[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  // the groups' sums of a block row, added in float64 through shared memory (row i of every block at
  // a time), one partial per CTA
  Acc *rows = reinterpret_cast<Acc *>(xs);
  const int64_t pidx = ((int64_t)w * gridDim.x + blockIdx.x) * g.U * 64;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (grp < g.G)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        rows[tid * 8 + j] = acc[i][j];
    __syncthreads();
    if constexpr (sizeof(Acc) == 4) {
      for (int e = tid; e < g.U * 8; e += kCovThr) {
        double s = 0.0;
        for (int q = 0; q < g.G; ++q)
          s += (double)rows[q * g.U * 8 + e];
        partial[pidx + (e >> 3) * 64 + 8 * i + (e & 7)] = (Acc)s;
      }
    } else { // few blocks have many groups (256 at T <= 8: 64 windows of 1024 pixels 44 us in all, 27 by lanes)
      for (int k0 = 0; k0 < (g.U * 8) << g.lh; k0 += kCovThr) { // whole warps take part in the shuffles
        const int  k = k0 + tid, e = k >> g.lh, h = k & ((1 << g.lh) - 1);
        const bool in = e < g.U * 8;
        Acc        s = Acc(0);
        if (in)
          for (int q = h; q < g.G; q += 1 << g.lh)
            s += rows[q * g.U * 8 + e];
        for (int o = (1 << g.lh) >> 1; o > 0; o >>= 1)
          s += __shfl_xor_sync(0xffffffffu, s, o);
        if (in && h == 0)
          partial[pidx + (e >> 3) * 64 + 8 * i + (e & 7)] = s;
      }
    }
    __syncthreads();
  }
  if constexpr (kShift) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      atomicAdd(&ssum[(tid & 31) + 32 * c], (unsigned long long)fsum[c]);
    __syncthreads();
    for (int t = tid; t < T; t += kCovThr) // of x - shift
      sums[((int64_t)w * gridDim.x + blockIdx.x) * T + t] = (double)(long long)ssum[t];
  }
}

// Float64 reduction of the CTA partials in a fixed order (S interleaved slices per entry, added pairwise);
// undoes the shift exactly.  `blocked`: partials are the 8 x 8 upper blocks of cov_cores_kernel, else whole
// [T][T] matrices of which the upper triangle is read.
template <typename Acc, int S>
__global__ void __launch_bounds__(256) cov_reduce_kernel(const Acc *partial, const double *sums, int nblk, int nsum,
                                                         int T, int64_t P, double shift, int blocked, double *gram) {
  constexpr int E = 256 / S; // entries per CTA
  __shared__ double red[3][S][E];
  const int w = blockIdx.y, lane = threadIdx.x % E, slice = threadIdx.x / E;
  const int NB = (T + 7) / 8, per = blocked ? NB * (NB + 1) / 2 * 64 : T * T;
  const int e = blockIdx.x * E + lane;
  int       i = T, j = T;
  if (e < per) {
    if (blocked) {
      int bi = 0, rem = e >> 6;
      while (rem >= NB - bi) {
        rem -= NB - bi;
        ++bi;
      }
      i = 8 * bi + ((e >> 3) & 7), j = 8 * (bi + rem) + (e & 7);
    } else {
      i = e / T, j = e % T;
    }
  }
  const bool ok = i < T && j < T && i <= j;
  double     s = 0.0, si = 0.0, sj = 0.0;
  if (ok) {
    const Acc *pp = partial + (int64_t)w * nblk * per + e;
    for (int b = slice; b < nblk; b += S)
      s += (double)pp[(int64_t)b * per];
    if (shift != 0.0) {
      const double *sp = sums + (int64_t)w * nsum * T;
      for (int b = slice; b < nsum; b += S)
        si += sp[(int64_t)b * T + i], sj += sp[(int64_t)b * T + j];
    }
  }
  red[0][slice][lane] = s, red[1][slice][lane] = si, red[2][slice][lane] = sj;
  __syncthreads();
  if (slice != 0 || !ok)
    return;
  double t[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if constexpr (S == 8)
      t[q] = ((red[q][0][lane] + red[q][1][lane]) + (red[q][2][lane] + red[q][3][lane])) +
             ((red[q][4][lane] + red[q][5][lane]) + (red[q][6][lane] + red[q][7][lane]));
    else
      t[q] = red[q][0][lane];
  }
  // x_i x_j = c_i c_j + s (c_i + c_j) + s^2 with c = x - s; the sums are of c (blocked) or of x
  const double sq = shift * shift * (double)P;
  const double v  = shift != 0.0 ? t[0] + (shift * (t[1] + t[2]) + (blocked ? sq : -sq)) : t[0];
  gram[(int64_t)w * T * T + i * T + j] = v;
  gram[(int64_t)w * T * T + j * T + i] = v;
}

template <typename Acc>
int launch_reduce(const Acc *partial, const double *sums, int nblk, int nsum, int T, int64_t P, double shift, int blocked,
                  double *gram, int nwin, cudaStream_t s) {
  const int NB = (T + 7) / 8, per = blocked ? NB * (NB + 1) / 2 * 64 : T * T;
  // 8 slices keep the loads of a window's hundreds of partials in flight; where few partials meet more
  // CTAs than run at once, a thread per entry takes them all: 64 windows of T = 128 with 5 partials 48 -> 9.4
  // us, 16 with 18 18 -> 7.2; below that line 16 windows of T = 64 with 18 take 5.9 sliced, 6.8 not
  const bool sliced = nblk >= 32 || (int64_t)((per + 31) / 32) * nwin <= 8LL * sm_count();
  auto       kern   = sliced ? cov_reduce_kernel<Acc, 8> : cov_reduce_kernel<Acc, 1>;
  const int  E      = sliced ? 32 : 256;
  kern<<<dim3((per + E - 1) / E, nwin), 256, 0, s>>>(partial, sums, nblk, nsum, T, P, shift, blocked, gram);
  note_launch();
  return launch_status("cov_reduce_kernel");
}

int64_t cov_tiles(int T, int64_t P) { return (P + cov_geom(T).PX - 1) / cov_geom(T).PX; }

int cov_ctas(int T, int64_t P, int nwin) { return (int)cov_split(sm_count(), cov_tiles(T, P), nwin); }

template <int FMT, typename Acc>
int launch_sums(const FrameRing &ring, int T, int64_t P, int nwin, void *ws, double *gram, int max_ctas, cudaStream_t s) {
  const CovGeom g     = cov_geom(T);
  const int     ctas  = max_ctas > 0 ? std::min(max_ctas, cov_ctas(T, P, nwin)) : cov_ctas(T, P, nwin);
  const float   shift = FMT == HF_F32 || sizeof(Acc) == 8 ? 0.f : (FMT == HF_U8 ? 128.f : 2048.f);
  auto         *sums  = reinterpret_cast<double *>(ws); // 8-byte aligned first, then the partials
  auto         *part  = reinterpret_cast<Acc *>(sums + (sizeof(Acc) == 8 ? 0 : (size_t)nwin * ctas * T));
  auto          kern  = cov_cores_kernel<FMT, Acc>;
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
  kern<<<dim3(ctas, nwin), kCovThr, g.smem, s>>>(ring, T, P, shift, g, part, sums);
  note_launch();
  HF_TRY(launch_status("cov_cores_kernel"));
  return launch_reduce<Acc>(part, sums, ctas, ctas, T, P, (double)shift, 1, gram, nwin, s);
}

template <int FMT>
int launch_fmt(const FrameRing &ring, int T, int64_t P, int nwin, void *ws, double *gram, int max_ctas, cudaStream_t s) {
  return cov_sums_fp32(ring, T, P) ? launch_sums<FMT, float>(ring, T, P, nwin, ws, gram, max_ctas, s)
                                   : launch_sums<FMT, double>(ring, T, P, nwin, ws, gram, max_ctas, s);
}

} // namespace

int launch_cov_finalize(const float *partial, const double *sums, int nblk, int nsum, int T, int64_t P, double shift,
                        double *gram, int nwin, cudaStream_t s) {
  return launch_reduce<float>(partial, sums, nblk, nsum, T, P, shift, 0, gram, nwin, s);
}

bool cov_cores_supported(int T) { return T >= 1 && T <= 128; }

size_t cov_cores_workspace_bytes(int T, int64_t P, int max_windows) {
  // float64 partials of the blocks; FP32 ones with the T frame sums take less
  const size_t cta = (size_t)cov_geom(T).U * 64 * sizeof(double);
  return (size_t)cov_split_most(sm_count(), cov_tiles(T, P), max_windows) * cta + 256;
}

int launch_cov_cores(const FrameRing &ring, int fmt, int T, int64_t P, int nwin, void *ws, double *gram, int max_ctas,
                     cudaStream_t s) {
  HF_CHECK_ARG(cov_cores_supported(T), "covariance: at most 128 frames");
  switch (fmt) {
  case HF_MONO12P: return launch_fmt<HF_MONO12P>(ring, T, P, nwin, ws, gram, max_ctas, s);
  case HF_U16: return launch_fmt<HF_U16>(ring, T, P, nwin, ws, gram, max_ctas, s);
  case HF_U8: return launch_fmt<HF_U8>(ring, T, P, nwin, ws, gram, max_ctas, s);
  case HF_F32: return launch_fmt<HF_F32>(ring, T, P, nwin, ws, gram, max_ctas, s);
  default: return fail(HF_ERR_INVALID, "covariance: unsupported input dtype");
  }
}

} // namespace hf
