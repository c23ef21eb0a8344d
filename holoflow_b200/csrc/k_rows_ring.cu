// Four-step row passes fed by a ring of asynchronous copies: the row pass of complex, unit-stride
// planes (the Fresnel lens and the angular spectrum's placement fused into it) and the angular
// spectrum's last pass, inverse rows + |.| + M0/M1/M2 over the band.
//
// Bound: HBM.  A row of 1024 points is 8 KB in and 8 KB out for about 1000 warp instructions, so the
// passes run at memory speed only while loads are in flight during the transforms.  With loads
// straight into registers the SM held 8 warps that each waited for their own row (4.0-5.0 TB/s; 1.2
// TB/s where placement made every load conditional).  Here a warp owns two row slots: while it
// transforms one row in place, the copies of its next row land in the other, and nothing but its own
// cp.async groups is waited for.  Rows run plane by plane at one image row, so the warps of a CTA
// read the same lens row.  8 windows x 28 planes of 1024^2 with the lens: 753 -> 637 us (5.9 TB/s); 4
// windows x 56 planes of 1024 x 1536: 1430 -> 1161 us; 4 windows x 28 planes of 768^2 placed in 1024^2:
// 1240 -> 221 us; inverse rows and moments of those: 487 -> 383 us.
#include <algorithm>

#include "fft_core.cuh"
#include "k_fft2d.cuh"

namespace hf {
namespace {

// Most warps per CTA (one CTA per SM): two slots each within shared memory, registers within 64 K.
template <int N1> constexpr int ring_warps(bool moments) {
  return moments ? 8 : (N1 >= 48 ? 8 : (N1 >= 24 ? 12 : 16));
}

// Warps per CTA of a launch: the rows in as few rounds as `most` warps on every SM need, spread over all
// SMs and the rounds.  (512 rows of 512 in CTAs of 16 warps kept 32 SMs busy and took 6.2 us, 2304 rows of
// 768 filled 1.3 rounds of 12 warps and took 11.2: 4.1 and 9.5 here; 5120 rows of 512 11.8 -> 10.1.)
int ring_launch_warps(int64_t nrows, int most) {
  const int64_t per_round = (int64_t)most * sm_count(), rounds = (nrows + per_round - 1) / per_round;
  return (int)std::min<int64_t>(most, (nrows + rounds * sm_count() - 1) / (rounds * sm_count()));
}

template <int N1> constexpr size_t ring_smem(int warps) {
  return sizeof(float2) * ((size_t)N1 * 32 + 2 * (size_t)warps * XBuf<N1>::kSize);
}

// Starts the copies of a row into `slot` (two elements per lane and copy), zero outside
// [ox, ox + IW); a null `src` is a row of zeros.  One commit group per call.
template <int N1>
__device__ __forceinline__ void ring_fetch(float2 *slot, const float2 *src, int ox, int IW, int lane) {
#pragma unroll
  for (int i = 0; i < N1 / 2; ++i) {
    const int      col = 2 * (lane + 32 * i), ic = col - ox;
    const bool     ok  = src != nullptr && ic >= 0 && ic < IW;
    const uint32_t d   = (uint32_t)__cvta_generic_to_shared(slot + col);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(ok ? src + ic : src), "r"(ok ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void ring_skip() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// The older of the two groups in flight has landed, for every lane.
__device__ __forceinline__ void ring_wait() {
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncwarp();
}

template <int N1, bool INV>
__global__ void __launch_bounds__(32 * ring_warps<N1>(false), 1) row_ring_kernel(RowPass a, int64_t nrows) {
  constexpr int N = N1 * 32;
  const int     NW = blockDim.x >> 5;
  extern __shared__ __align__(16) float2 smf2[];
  TwTable tw{smf2, N};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2   *slots = smf2 + N + 2 * warp * XBuf<N1>::kSize;
  // work item -> (window, image row, plane), plane fastest; only rows inside the placed input
  const float2 *in = reinterpret_cast<const float2 *>(a.in);
  const auto decode = [&](int64_t it, int &w, int &ir, int &plane) {
    const int64_t rest = it / a.nplanes;
    plane = (int)(it - rest * a.nplanes);
    w     = (int)(rest / a.IH);
    ir    = (int)(rest - (int64_t)w * a.IH);
  };
  const auto fetch = [&](int64_t it, int s) {
    if (it >= nrows) {
      ring_skip();
      return;
    }
    int w, ir, plane;
    decode(it, w, ir, plane);
    ring_fetch<N1>(slots + s * XBuf<N1>::kSize, in + w * a.in_win + plane * a.in_plane + (int64_t)ir * a.in_row, a.ox,
                   a.IW, lane);
  };
  const int64_t stride = (int64_t)gridDim.x * NW;
  int64_t       it     = (int64_t)blockIdx.x * NW + warp;
  fetch(it, 0);
  fetch(it + stride, 1);
  tw.fill(threadIdx.x, blockDim.x);
  __syncthreads();
  for (int s = 0; it < nrows; it += stride, s ^= 1) {
    int w, ir, plane;
    decode(it, w, ir, plane);
    const int r    = ir + a.oy;
    float2   *slot = slots + s * XBuf<N1>::kSize;
    float2    x[N1];
    if (a.pre != nullptr) {
      const float2 *pr = a.pre + (int64_t)r * N + lane;
      float2        pv[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        pv[n1] = __ldg(pr + 32 * n1);
      ring_wait();
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        x[n1] = cmul(slot[lane + 32 * n1], pv[n1]);
    } else {
      ring_wait();
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        x[n1] = slot[lane + 32 * n1];
    }
    __syncwarp(); // the row is in registers: its slot becomes the exchange
    four_step_a<N1, INV>(x, lane, tw, slot);
    __syncwarp();
    float2 *orow = a.out + w * a.out_win + plane * a.out_plane + (int64_t)r * a.out_row;
    for (int k1 = lane; k1 < N1; k1 += 32) {
      float2 y[32];
      four_step_b<N1, INV>(y, k1, slot);
#pragma unroll
      for (int k2 = 0; k2 < 32; ++k2)
        orow[k1 + N1 * k2] = y[k2];
    }
    __syncwarp(); // the exchange is read: the slot takes the row after next
    fetch(it + 2 * stride, s);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// A warp owns one image row of a window for every plane and keeps the three sums of its 32 outputs
// per lane in registers (they were read, added to and written back in shared memory per plane).
template <int N1, bool INV>
__global__ void __launch_bounds__(32 * ring_warps<N1>(true), 1) row_moments_ring_kernel(ColPass a, MomentSpec m,
                                                                                       int64_t nrows) {
  constexpr int N = N1 * 32;
  const int     NW = blockDim.x >> 5;
  extern __shared__ __align__(16) float2 smf2[];
  TwTable tw{smf2, N};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2   *slots = smf2 + N + 2 * warp * XBuf<N1>::kSize;
  tw.fill(threadIdx.x, blockDim.x);
  __syncthreads();
  for (int64_t it = (int64_t)blockIdx.x * NW + warp; it < nrows; it += (int64_t)gridDim.x * NW) {
    const int     w = (int)(it / a.H), r = (int)(it - (int64_t)w * a.H);
    const float2 *src = a.in + w * a.in_win + (int64_t)r * a.in_row;
    ring_fetch<N1>(slots, src, 0, N, lane);
    if (m.nz > 1)
      ring_fetch<N1>(slots + XBuf<N1>::kSize, src + a.in_plane, 0, N, lane);
    else
      ring_skip();
    float2 acc0[16], acc1[16], acc2[16]; // outputs k2 = 2 i, 2 i + 1 as packed pairs
#pragma unroll
    for (int i = 0; i < 16; ++i)
      acc0[i] = acc1[i] = acc2[i] = make_float2(0.f, 0.f);
    for (int k = 0; k < m.nz; ++k) {
      float2 *slot = slots + (k & 1) * XBuf<N1>::kSize;
      ring_wait();
      float2 x[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1)
        x[n1] = slot[lane + 32 * n1];
      __syncwarp();
      four_step_a<N1, INV>(x, lane, tw, slot);
      __syncwarp();
      if (lane < N1) {
        float2 y[32];
        four_step_b<N1, INV>(y, lane, slot);
        abs32(y);
        const float2 f1 = make_float2(m.w1[k], m.w1[k]), f2 = make_float2(m.w2[k], m.w2[k]);
#pragma unroll
        for (int i = 0; i < 16; ++i) { // the reference's float32 sequence in band order
          const float2 mag = make_float2(y[2 * i].x, y[2 * i + 1].x);
          acc0[i] = cadd(acc0[i], mag);
          acc1[i] = cadd(acc1[i], pmul2(f1, mag));
          acc2[i] = cadd(acc2[i], pmul2(f2, mag));
        }
      }
      __syncwarp(); // the exchange is read: the slot takes the plane after next
      if (k + 2 < m.nz)
        ring_fetch<N1>(slot, src + (int64_t)(k + 2) * a.in_plane, 0, N, lane);
      else
        ring_skip();
    }
    if (lane < N1) {
      const float nzf = (float)m.nz;
      float      *out = reinterpret_cast<float *>(a.out) + w * a.out_win;
      const int   rr  = m.fftshift ? (r + a.H / 2) % a.H : r;
      int         mi  = 0;
#pragma unroll
      for (int mo = 0; mo < 3; ++mo) {
        if (!(m.mask & (1 << mo)))
          continue;
        const float2 *acc = mo == 0 ? acc0 : (mo == 1 ? acc1 : acc2);
        float        *orow = out + mi * a.out_plane + (int64_t)rr * a.out_row;
#pragma unroll
        for (int k2 = 0; k2 < 32; ++k2) {
          const int i  = lane + N1 * k2;
          const int cc = m.fftshift ? (i + N / 2) % N : i;
          orow[cc] = __fdiv_rn((k2 & 1) ? acc[k2 >> 1].y : acc[k2 >> 1].x, nzf);
        }
        ++mi;
      }
    }
  }
}

template <int N1, bool INV> int launch_ring(const RowPass &a, int nwin, cudaStream_t s) {
  const int64_t nrows = (int64_t)nwin * a.nplanes * a.IH;
  const int     NW    = ring_launch_warps(nrows, ring_warps<N1>(false));
  const size_t  smem  = ring_smem<N1>(NW);
  HF_CUDA(cudaFuncSetAttribute(row_ring_kernel<N1, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int     grid  = (int)std::min<int64_t>((nrows + NW - 1) / NW, sm_count());
  row_ring_kernel<N1, INV><<<grid, 32 * NW, smem, s>>>(a, nrows);
  note_launch();
  return launch_status("row_ring_kernel");
}

template <int N1, bool INV> int launch_moments_ring(const ColPass &a, const MomentSpec &m, int nwin, cudaStream_t s) {
  const int64_t nrows = (int64_t)nwin * a.H;
  int           NW    = ring_launch_warps(nrows, ring_warps<N1>(true));
  NW += NW > 4 ? NW & 1 : 0; // 1024 rows of 256, 10 planes: 29.2 us with 7 warps, 27.0 with 8
  const size_t  smem  = ring_smem<N1>(NW);
  HF_CUDA(cudaFuncSetAttribute(row_moments_ring_kernel<N1, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int     grid  = (int)std::min<int64_t>((nrows + NW - 1) / NW, sm_count());
  row_moments_ring_kernel<N1, INV><<<grid, 32 * NW, smem, s>>>(a, m, nrows);
  note_launch();
  return launch_status("row_moments_ring_kernel");
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

#define HF_RING_N1(n, CALL)                                                                        \
  switch ((n) / 32) {                                                                              \
  case 2: { constexpr int N1 = 2; CALL; }                                                          \
  case 4: { constexpr int N1 = 4; CALL; }                                                          \
  case 8: { constexpr int N1 = 8; CALL; }                                                          \
  case 16: { constexpr int N1 = 16; CALL; }                                                        \
  case 24: { constexpr int N1 = 24; CALL; }                                                        \
  case 32: { constexpr int N1 = 32; CALL; }                                                        \
  default: break;                                                                                  \
  }

} // namespace

// Complex rows of unit stride whose two-element chunks are 16-byte aligned in every row; with rows
// outside the placed input only where the caller does not need them written.
bool row_ring_supported(const RowPass &a) {
  return fft_fast_length(a.N) && !a.in_real && a.in_col == 1 && aligned16(a.in) && a.in_win % 2 == 0 &&
         a.in_plane % 2 == 0 && a.in_row % 2 == 0 && a.ox % 2 == 0 && a.IW % 2 == 0 && a.IH <= a.H &&
         a.ox + a.IW <= a.N && a.oy + a.IH <= a.H && (a.IH == a.H || a.rows_only);
}

int launch_row_ring(const RowPass &a, int nwin, cudaStream_t s) {
  if (a.N == 1536)
    return a.inverse ? launch_ring<48, true>(a, nwin, s) : launch_ring<48, false>(a, nwin, s);
  if (a.inverse) {
    HF_RING_N1(a.N, return (launch_ring<N1, true>(a, nwin, s)))
  } else {
    HF_RING_N1(a.N, return (launch_ring<N1, false>(a, nwin, s)))
  }
  return fail(HF_ERR_UNSUPPORTED, "row pass: unsupported row length");
}

// Rows of at most 1024 points (32 outputs per lane).
bool row_moments_ring_supported(const ColPass &a) {
  return fft_fast_length(a.W) && a.W <= 1024 && aligned16(a.in) && a.in_win % 2 == 0 && a.in_plane % 2 == 0 &&
         a.in_row % 2 == 0;
}

int launch_row_moments_ring(const ColPass &a, const MomentSpec &m, int nwin, cudaStream_t s) {
  if (a.inverse) {
    HF_RING_N1(a.W, return (launch_moments_ring<N1, true>(a, m, nwin, s)))
  } else {
    HF_RING_N1(a.W, return (launch_moments_ring<N1, false>(a, m, nwin, s)))
  }
  return fail(HF_ERR_UNSUPPORTED, "row moments: unsupported row length");
}

} // namespace hf
