// Chosen form, raw band planes on the tensor cores, in row segments.
//
// The fused pass (k_tc_band.cu) needs a whole image row in shared memory and TMEM because it runs
// the row FFT; that fixes T = 64, W <= 1024 and Nz <= 32.  Without the row FFT no full row is
// needed, so this pass covers the other shapes of the path: T = 32, 64 or 128 frames, any width
// that is a multiple of 128, up to 64 band bins, and every propagation (the angular spectrum and
// the autofocus need the band planes before any lens).  It stores
//   S[p][k] = sum_t (x_t[p] - 2048) (Wh + Wl)[t][k] + 2048 sum_t (Wh + Wl)[t][k]
// for each pixel p of a segment of `seg` 128-pixel tiles of one row, with Wh = f16(W) and
// Wl = f16(W - Wh) as in the fused pass: A = the segment's samples x - 2048 (exact in f16 for
// 12-bit data), MN-major [T][128] per tile; B = Wh / Wl as real/imaginary rows, K-major in 64-frame
// atoms; tcgen05.mma M = 128, N = 16 ceil(2 Nz / 16), K = 16, f32 accumulators in TMEM (tile j ->
// columns j * ncol .. j * ncol + N - 1, ncol the power of two >= N).  The later passes (row FFT
// with the lens, column FFT and moments, or the angular spectrum) read the planes as the plain
// band DFT leaves them.
//
// Warp roles (384 threads, one CTA per SM, persistent over segments taken from a counter):
//   warps 0-3  : unpack the segment into A, rebuild B per window, and (thread 0) issue the MMAs once
//                the epilogue has released TMEM.  The packed samples arrive by cp.async one whole
//                segment ahead, into a ring whose slots each thread fills and empties itself;
//                segments alternate between two halves of TMEM, so the MMAs of the next one run
//                while the epilogue still reads this one;
//   warps 4-11 : epilogue; warp 4 + 4h + q reads TMEM lane quarter q of the tiles j = h (mod 2),
//                adds the DC correction and stores each bin's 32 pixels as one coalesced row.
// mbarriers per half: `full` (MMAs of a segment complete: TMEM readable, A/B reusable) and `free` (the
// 8 epilogue warps finished reading it), with bounded waits as in the fused pass.
//
// Bound: HBM, 4.0 GB for 4 windows of 128 x 1024 x 1536 at 56 bins (620 us at the copy rate).  With the
// samples staged through registers, one round of 24 KB ahead, the loaders took 13 us per 512-pixel
// segment and the epilogue, which could not start on the next one before they were done, 7: 1466 us in
// all, 981 now (4.1 TB/s; 4 windows of 64 x 768^2 at 28 bins 266 -> 213).  The ring keeps 49 KB in
// flight all the time and hides the loads completely; what is left is the epilogue's stores and the
// hand-over of A between segments.
//
// One launch can serve several acquisitions of the same window length and sample format (the
// batched uneven acquisitions): each is a job with its own ring, W, planes and geometry, and the
// units of all jobs form one work list, (job, window, row, segment) in order, taken from the one
// counter.
#include <algorithm>
#include <initializer_list>

#include <cuda_fp16.h>

#include "k_tc_band.cuh"
#include "tc_band_common.cuh"
#include "tc_common.cuh"

namespace hf {

namespace {

using tcb::GroupLoad;
using tcb::mbar_arrive;
using tcb::mbar_arrive_cnt;
using tcb::named_bar;
using tcb::wait_or_abort;

constexpr int kSegLoaders  = 128; // warps 0-3
constexpr int kSegEpilogue = 256; // warps 4-11
constexpr int kSegThr      = kSegLoaders + kSegEpilogue;
constexpr int kSegCols     = 256; // TMEM columns of a segment: two segments in turn
constexpr int kSegTF       = 256; // tiles x frames of a segment: A holds 256 bytes of f16 for each
constexpr int kSegItems    = kSegTF * 4 / kSegLoaders; // a loader's items of 32 samples per segment
// The loaders' ring: one slot more than a segment's items; a slot's pitch is an odd multiple of 16
// bytes, so that neighbouring threads' 16-byte reads touch different banks.
template <int FMT> struct SegRing {
  static constexpr int kPitch = FMT == HF_MONO12P ? 48 : 80;
  static constexpr int kSlots = kSegItems + 1;
  static constexpr int kBytes = kSlots * kSegLoaders * kPitch;
};
constexpr int kSegABytes   = kSegTF * 256;
constexpr int kUnitSlots   = 4; // unit indexes kept: one ahead of the loaders, one behind
constexpr int kSegMaxN     = 128;    // MMA N (Nz <= 64)

struct SegGeom {
  int N;    // MMA N, 16 ceil(2 Nz / 16)
  int ncol; // TMEM columns per tile: the power of two >= N (>= 32)
  int seg;  // tiles per segment
  int spr;  // segments per row
};

// One acquisition of a launch.
struct SegJob {
  FrameRing     ring;
  const float2 *wmat;
  int64_t       wmat_stride;
  float2       *out;
  int64_t       out_win, out_plane, out_row;
  int64_t       unit0; // first unit of this job in the launch's work list
  int           H, W, nz, nwin;
  float         shift;
  SegGeom       g;
};

struct SegJobs {
  int     njob;
  int     bpart_max; // bytes of one W part at the largest N of the launch
  int64_t nunits;    // units of all jobs
  int    *status;
  int    *counter;
  SegJob  job[kMaxSegJobs];
};

// Job of unit u (the jobs' first units ascend).
__device__ __forceinline__ int job_of(const SegJobs &J, int64_t u) {
  int ji = 0;
  while (ji + 1 < J.njob && u >= J.job[ji + 1].unit0)
    ++ji;
  return ji;
}

template <int FMT, int T>
__global__ void __launch_bounds__(kSegThr, 1) band_seg_tc_kernel(const __grid_constant__ SegJobs J) {
  constexpr int KA   = (T + 63) / 64; // 64-frame K atoms of B
  constexpr int KS   = T / 16;        // k-steps per W part
  constexpr int TILE = T * 256;       // A tile bytes: [T][128] f16
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // aligned by pointer arithmetic on the shared array, so every derived pointer stays a shared-space
  // pointer
  uint8_t  *smem   = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t  *sA     = smem;                                        // g.seg tiles
  using RG         = SegRing<FMT>;
  uint8_t  *sB     = sA + kSegABytes;                            // hi [KA][N][128 B], then lo
  uint8_t  *ring   = sB + 2 * J.bpart_max;                        // [kSlots][kSegLoaders][kPitch] packed samples
  float    *colsum = reinterpret_cast<float *>(ring + RG::kBytes); // [4][128], windows in turn
  int64_t  *foff   = reinterpret_cast<int64_t *>(colsum + 512);   // [2][128] frame offsets, by window parity
  int64_t  *unitbuf = foff + 256;                                 // [kUnitSlots] unit of iteration k
  uint64_t *mbar   = reinterpret_cast<uint64_t *>(unitbuf + kUnitSlots); // full[2], free[2]
  uint32_t *tslot  = reinterpret_cast<uint32_t *>(mbar + 4);
  int      *abort_flag = reinterpret_cast<int *>(tslot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&mbar[i], 2); // the MMA commit + the issuing thread's release arrive
      tc::mbar_init(&mbar[2 + i], kSegEpilogue / 32);
    }
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0)
    tc::tmem_alloc(tslot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase  = *tslot;
  volatile int  *abortv = abort_flag;
  const int64_t  nunits = J.nunits;
  // segment k uses TMEM half k & 1 and the barriers of that half, in phase (k >> 1) & 1
  uint64_t *const full = mbar, *const free_ = mbar + 2;
  const auto      phase = [](int k) { return (uint32_t)((k >> 1) & 1); };

  if (tid < kSegLoaders) {
    // ------------------------------------------------------------------ loader / MMA warps
    using GL         = GroupLoad<FMT>;
    constexpr int IT = kSegItems;
    int           k = 0, cur_ji = -1, cur_w = -1, wpar = 1; // window of B and its DC corrections
    int           nxt_ji = -1, nxt_w = -1, npar = 1;        // window of the segment being fetched
    int           fill = 0, drain = 0;                      // this thread's ring slots
    uint8_t      *mine = ring + (size_t)tid * RG::kPitch;
    // a segment of the work list: job, window, row, first tile, tiles
    struct Seg {
      int ji, w, r, j0, nt;
    };
    const auto decode = [&](int64_t u) {
      Seg           q;
      q.ji              = job_of(J, u);
      const SegJob &a   = J.job[q.ji];
      const int64_t uj  = u - a.unit0;
      q.w               = (int)(uj / ((int64_t)a.H * a.g.spr));
      const int64_t rem = uj - (int64_t)q.w * a.H * a.g.spr;
      q.r               = (int)(rem / a.g.spr);
      q.j0              = (int)(rem - (int64_t)q.r * a.g.spr) * a.g.seg;
      q.nt              = min(a.g.seg, a.W / 128 - q.j0);
      return q;
    };
    // work item `it` of a segment = (tile, frame t, 32-pixel group); consecutive threads take the four
    // groups of one frame row, so each quad reads 128 contiguous pixels.  One commit group per call.
    const auto fetch = [&](const Seg &q, const int64_t *fo, int it) {
      if (it < q.nt * T * 4) {
        const SegJob  &a = J.job[q.ji];
        const int      j = it / (T * 4), t = (it >> 2) % T, grp = it & 3;
        const uint8_t *src = a.ring.base + fo[t] + ((int64_t)q.r * a.W + 128 * (q.j0 + j) + 32 * grp) * GL::kBytes / 32;
        const uint32_t dst = tc::smem_u32(mine + (size_t)fill * kSegLoaders * RG::kPitch);
#pragma unroll
        for (int i = 0; i < GL::kBytes / 16; ++i)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(src + 16 * i) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      fill = fill + 1 == RG::kSlots ? 0 : fill + 1;
    };
    const auto offsets = [&](const Seg &q, int64_t *fo) { // frame offsets of the segment's window
      const SegJob &a = J.job[q.ji];
      for (int t = tid; t < T; t += kSegLoaders)
        fo[t] = a.ring.frame(q.w, t) - a.ring.base;
    };
    if (tid == 0)
      unitbuf[0] = atomicAdd(J.counter, 1);
    named_bar(1, kSegLoaders);
    Seg nxt{};
    if (unitbuf[0] < nunits) { // the first segment's samples
      nxt    = decode(unitbuf[0]);
      nxt_ji = nxt.ji, nxt_w = nxt.w, npar = 0;
      offsets(nxt, foff);
      named_bar(1, kSegLoaders);
#pragma unroll
      for (int i = 0; i < IT; ++i)
        fetch(nxt, foff, i * kSegLoaders + tid);
    }
    for (;; ++k) {
      const int64_t u = unitbuf[k % kUnitSlots];
      if (tid == 0)
        unitbuf[(k + 1) % kUnitSlots] = u < nunits ? (int64_t)atomicAdd(J.counter, 1) : nunits;
      if (k > 0) // MMAs of the previous segment done: A and B may be overwritten
        wait_or_abort(&full[(k - 1) & 1], phase(k - 1), abortv, J.status, 31);
      named_bar(1, kSegLoaders);
      if (u >= nunits) { // no segments left: complete this phase empty so that the epilogue ends too
        if (tid == 0) {
          // only after the epilogue has released the half's last segment (see the fused pass)
          if (k > 1)
            wait_or_abort(&free_[k & 1], phase(k - 2), abortv, J.status, 34);
          mbar_arrive_cnt(&full[k & 1], 2);
        }
        break;
      }
      const Seg     cur = nxt;
      const SegJob &a   = J.job[cur.ji];
      const SegGeom g   = a.g;
      const int     bpart = KA * g.N * 128, nt = cur.nt;
      const bool    new_w = cur.w != cur_w || cur.ji != cur_ji;
      const int64_t un    = unitbuf[(k + 1) % kUnitSlots];
      const bool    more  = un < nunits;
      if (more)
        nxt = decode(un);
      const bool nxt_new = more && (nxt.w != nxt_w || nxt.ji != nxt_ji);
      if (nxt_new) {
        nxt_ji = nxt.ji, nxt_w = nxt.w, npar ^= 1;
        offsets(nxt, foff + npar * 128);
      }
      if (new_w) { // per window: B = (Wh, Wl) rows n = 2 bin + {re, im}
        cur_ji = cur.ji;
        cur_w  = cur.w;
        wpar   = (wpar + 1) & 3;
        const float2 *wm = a.wmat + (int64_t)cur.w * a.wmat_stride;
        for (int e = tid; e < g.N * (T / 8); e += kSegLoaders) {
          const int n = e / (T / 8), c8 = e % (T / 8); // one 16-byte chunk = 8 frames
          __half    hv[8], lv[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int t = 8 * c8 + i;
            float     v = 0.f;
            if ((n >> 1) < a.nz) {
              const float2 z = __ldg(wm + (int64_t)t * a.nz + (n >> 1));
              v              = (n & 1) ? z.y : z.x;
            }
            hv[i] = __float2half_rn(v);
            lv[i] = __float2half_rn(v - __half2float(hv[i]));
          }
          const int off = (c8 >> 3) * g.N * 128 + n * 128 + (((c8 & 7) ^ (n & 7)) << 4);
          *reinterpret_cast<uint4 *>(sB + off)         = *reinterpret_cast<const uint4 *>(hv);
          *reinterpret_cast<uint4 *>(sB + bpart + off) = *reinterpret_cast<const uint4 *>(lv);
        }
      }
      if (nxt_new)
        named_bar(1, kSegLoaders); // its frame offsets are visible to every loader
      // A: tile j = pixels [128 (j0 + j), +128) of row r; element (m, t) at
      //    (m/64)*(128 T) + (t/8)*1024 + (t%8)*128 + ((m%64/8) ^ (t%8))*16 + (m%8)*2.
      //    Item i of the next segment is fetched before item i of this one is unpacked.
      {
        const float magic = 8388608.f + a.shift; // x - shift exactly: (2^23 + x) - (2^23 + shift)
#pragma unroll 2
        for (int i = 0; i < IT; ++i) {
          const int it = i * kSegLoaders + tid;
          if (more)
            fetch(nxt, foff + npar * 128, it);
          else
            asm volatile("cp.async.commit_group;" ::: "memory");
          asm volatile("cp.async.wait_group %0;" ::"n"(IT) : "memory"); // this thread's item i has landed
          const uint4 *src = reinterpret_cast<const uint4 *>(mine + (size_t)drain * kSegLoaders * RG::kPitch);
          drain            = drain + 1 == RG::kSlots ? 0 : drain + 1;
          if (it >= nt * T * 4)
            continue;
          const int j = it / (T * 4), t = (it >> 2) % T, grp = it & 3;
          uint32_t  raw[GL::kWords], v[32];
#pragma unroll
          for (int q = 0; q < GL::kWords / 4; ++q) {
            const uint4 x = src[q];
            raw[4 * q] = x.x, raw[4 * q + 1] = x.y, raw[4 * q + 2] = x.z, raw[4 * q + 3] = x.w;
          }
          GL::unpack(raw, v);
          uint8_t *tile = sA + j * TILE;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int m0 = 32 * grp + 8 * q;
            __half2   h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              h[e] = __floats2half2_rn(__uint_as_float(0x4B000000u | v[8 * q + 2 * e]) - magic,
                                       __uint_as_float(0x4B000000u | v[8 * q + 2 * e + 1]) - magic);
            const int chunk = (m0 & 63) >> 3;
            uint8_t  *dst   = tile + (m0 >> 6) * (T * 128) + (t >> 3) * 1024 + (t & 7) * 128 + ((chunk ^ (t & 7)) << 4);
            *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(h);
          }
        }
      }
      named_bar(1, kSegLoaders); // A (and B) complete
      if (new_w && tid < g.N) { // DC correction of the shifted samples: shift * sum_t (hi + lo)[t][n]
        float sacc = 0.f;
        for (int t = 0; t < T; ++t) {
          const int c   = (t & 63) >> 3;
          const int off = (t >> 6) * g.N * 128 + tid * 128 + ((c ^ (tid & 7)) << 4) + (t & 7) * 2;
          sacc += __half2float(*reinterpret_cast<const __half *>(sB + off)) +
                  __half2float(*reinterpret_cast<const __half *>(sB + bpart + off));
        }
        colsum[wpar * 128 + tid] = a.shift * sacc;
      }
      tc::fence_proxy_async_smem();
      named_bar(1, kSegLoaders);
      if (tid == 0) {
        if (k > 1) // the epilogue has read segment k - 2 out of this half
          wait_or_abort(&free_[k & 1], phase(k - 2), abortv, J.status, 32);
        tc::fence_after_sync();
        if (!*abortv) {
          const uint32_t idesc = tc::idesc_f16(128, g.N, true, false);
          for (int j = 0; j < nt; ++j)
#pragma unroll
            for (int s = 0; s < 2 * KS; ++s) { // k-steps 0..KS-1 with W hi, then the same with W lo
              const int      part = s / KS, ks = s % KS;
              const uint64_t ad   = tc::sw128_desc(tc::smem_u32(sA + j * TILE + ks * 2048), T * 128, 1024);
              const uint64_t bd =
                  tc::sw128_desc(tc::smem_u32(sB + part * bpart + (ks >> 2) * g.N * 128 + (ks & 3) * 32), 16, 1024);
              tc::mma_f16(tbase + (uint32_t)((k & 1) * kSegCols + j * g.ncol), ad, bd, idesc, s > 0 ? 1u : 0u);
            }
        }
        tc::mma_commit(&full[k & 1]);
        mbar_arrive(&full[k & 1]); // release: the unit index, B and the DC correction are in place
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int e = warp - 4, q = warp & 3, half = e >> 2;
    int       k = 0, cur_ji = -1, cur_w = -1, wpar = 1;
    for (;; ++k) {
      wait_or_abort(&full[k & 1], phase(k), abortv, J.status, 33);
      tc::fence_after_sync();
      const int64_t u = unitbuf[k % kUnitSlots];
      if (u >= nunits || *abortv)
        break;
      const int     ji   = job_of(J, u);
      const SegJob &a    = J.job[ji];
      const SegGeom g    = a.g;
      const int     ngrp = (2 * a.nz + 7) / 8; // 8-column groups = 4 bins
      const int64_t uj   = u - a.unit0;
      const int     w    = (int)(uj / ((int64_t)a.H * g.spr));
      const int64_t rem  = uj % ((int64_t)a.H * g.spr);
      const int     r = (int)(rem / g.spr), sg = (int)(rem % g.spr);
      const int     j0 = sg * g.seg, nt = min(g.seg, a.W / 128 - j0);
      if (w != cur_w || ji != cur_ji) {
        cur_ji = ji;
        cur_w  = w;
        wpar   = (wpar + 1) & 3;
      }
      const float *cs   = colsum + wpar * 128;
      float2      *orow = a.out + (int64_t)w * a.out_win + (int64_t)r * a.out_row + 32 * q + lane;
      for (int j = half; j < nt; j += 2) {
        float2 *op = orow + 128 * (j0 + j);
        for (int g0 = 0; g0 < ngrp; g0 += 4) { // four TMEM loads in flight, one wait
          uint32_t  v[4][8];
          const int ng = min(4, ngrp - g0);
#pragma unroll
          for (int gi = 0; gi < 4; ++gi)
            if (gi < ng)
              tc::tmem_ld8(tbase + ((uint32_t)(32 * q) << 16) + (uint32_t)((k & 1) * kSegCols + j * g.ncol + 8 * (g0 + gi)), v[gi]);
          tc::tmem_wait_ld();
#pragma unroll
          for (int gi = 0; gi < 4; ++gi)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const int bin = 4 * (g0 + gi) + b;
              if (gi < ng && bin < a.nz)
                op[(int64_t)bin * a.out_plane] =
                    cadd(make_float2(__uint_as_float(v[gi][2 * b]), __uint_as_float(v[gi][2 * b + 1])),
                         reinterpret_cast<const float2 *>(cs)[bin]);
            }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&free_[k & 1]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, 512);
  }
}

// seg_cap > 0 caps the tiles per segment (the autotuner's tile parameter); 0 takes the most that A
// and TMEM hold.
SegGeom seg_geom(int T, int W, int nz, int seg_cap) {
  SegGeom g{};
  g.N    = 16 * ((2 * nz + 15) / 16);
  g.ncol = g.N <= 32 ? 32 : (g.N <= 64 ? 64 : 128);
  g.seg  = std::min({kSegCols / g.ncol, kSegTF / T, W / 128});
  if (seg_cap > 0)
    g.seg = std::min(g.seg, seg_cap);
  g.spr  = (W / 128 + g.seg - 1) / g.seg;
  return g;
}

template <int FMT, int T> int launch_t(SegJobs &J, int max_ctas, cudaStream_t s) {
  const size_t smem = 1024 + (size_t)kSegABytes + 2 * (size_t)J.bpart_max + SegRing<FMT>::kBytes + 512 * 4 +
                      256 * 8 + kUnitSlots * 8 + 4 * 8 + 16;
  HF_CUDA(cudaFuncSetAttribute(band_seg_tc_kernel<FMT, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int cap  = max_ctas > 0 ? std::min(max_ctas, sm_count()) : sm_count();
  const int grid = (int)std::min<int64_t>(J.nunits, cap);
  HF_CUDA(cudaMemsetAsync(J.counter, 0, sizeof(int), s));
  band_seg_tc_kernel<FMT, T><<<grid, kSegThr, smem, s>>>(J);
  note_launch();
  return launch_status("band_seg_tc_kernel");
}

} // namespace

bool band_seg_tc_supported(int fmt, int T, int W, int nz, int64_t frame_bytes) {
  return (fmt == HF_MONO12P || fmt == HF_U16) && (T == 32 || T == 64 || T == 128) && W >= 128 && W % 128 == 0 &&
         nz >= 1 && 2 * nz <= kSegMaxN && frame_bytes % 16 == 0;
}

int launch_band_seg_tc_multi(const BandRowsArgs *jobs, int njobs, int fmt, int seg_cap, int max_ctas, int *counter,
                             int *status, cudaStream_t s) {
  HF_CHECK_ARG(jobs != nullptr && njobs >= 1 && njobs <= kMaxSegJobs, "band segments: 1 to 16 jobs per launch");
  HF_CHECK_ARG(counter != nullptr, "band segments: unit counter missing");
  const int T = jobs[0].T;
  SegJobs   J{};
  J.njob = njobs, J.status = status, J.counter = counter;
  for (int i = 0; i < njobs; ++i) {
    const BandRowsArgs &a = jobs[i];
    HF_CHECK_ARG(a.T == T, "band segments: the jobs of one launch share the window length");
    HF_CHECK_ARG(band_seg_tc_supported(fmt, a.T, a.W, a.nz, a.ring.frame_bytes),
                 "band segments (tensor core): unsupported shape");
    HF_CHECK_ARG(((uintptr_t)a.ring.base & 15) == 0, "band segments (tensor core): ring must be 16-byte aligned");
    HF_CHECK_ARG(a.nwin >= 1 && a.H >= 1, "band segments: empty job");
    SegJob &j = J.job[i];
    j.ring = a.ring, j.wmat = a.wmat, j.wmat_stride = a.wmat_stride, j.out = a.out;
    j.out_win = a.out_win, j.out_plane = a.out_plane, j.out_row = a.out_row;
    j.H = a.H, j.W = a.W, j.nz = a.nz, j.nwin = a.nwin, j.shift = a.shift;
    j.g     = seg_geom(T, a.W, a.nz, seg_cap);
    j.unit0 = J.nunits;
    J.nunits += (int64_t)a.nwin * a.H * j.g.spr;
    J.bpart_max = std::max(J.bpart_max, ((T + 63) / 64) * j.g.N * 128);
  }
  switch (T) {
  case 32: return fmt == HF_MONO12P ? launch_t<HF_MONO12P, 32>(J, max_ctas, s) : launch_t<HF_U16, 32>(J, max_ctas, s);
  case 64: return fmt == HF_MONO12P ? launch_t<HF_MONO12P, 64>(J, max_ctas, s) : launch_t<HF_U16, 64>(J, max_ctas, s);
  default:
    return fmt == HF_MONO12P ? launch_t<HF_MONO12P, 128>(J, max_ctas, s) : launch_t<HF_U16, 128>(J, max_ctas, s);
  }
}

int launch_band_seg_tc(const BandRowsArgs &a, int fmt, cudaStream_t s) {
  return launch_band_seg_tc_multi(&a, 1, fmt, 0, a.max_ctas, a.row_counter, a.status, s);
}

} // namespace hf
