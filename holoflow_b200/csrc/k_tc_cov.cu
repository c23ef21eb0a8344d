// Tensor-core (tcgen05) Gram matrix of a window's frames: exact integers for samples of at most 12
// bits (both forms), f16 operands for 16-bit samples (the chosen form), described first.
//
// G' = (X - 2048)^T (X - 2048) with X = [T][P] 12-bit samples: (x - 2048) is exact in f16, the
// products are exact in the f32 accumulator, and the shift is undone in float64 by the shared
// finalize kernel (k_cov_fp32.cu) from exact integer frame sums.  Per CTA: a ring of 4 shared-memory
// stages of 128 pixels x T frames in the canonical K-major 128-byte-swizzled layout (rows = frames,
// K = pixels).  All threads unpack the next stage while the tensor core consumes the previous ones;
// one thread issues M = N = T, K = 16 MMAs (A and B are the same tile) into a TMEM accumulator and
// commits each stage to its mbarrier, which gates the stage's reuse.
#include <cuda_fp16.h>

#include "k_pca.cuh"
#include "tc_common.cuh"

namespace hf {

namespace {

constexpr int kTcPX     = 128; // pixels per stage (two K-subtiles of 64)
constexpr int kTcStages = 4;

template <int FMT> struct TcBpp;
template <> struct TcBpp<HF_MONO12P> { static constexpr int num = 3, den = 2; };
template <> struct TcBpp<HF_U16> { static constexpr int num = 2, den = 1; };
template <> struct TcBpp<HF_U8> { static constexpr int num = 1, den = 1; };

template <int T> // 16-bit samples
__global__ void __launch_bounds__(128) cov_tc_kernel(CovArgs a, int *status) {
  constexpr int SUB   = T * 128;       // bytes of one 64-pixel K-subtile (T rows x 128 B)
  constexpr int STAGE = 2 * SUB;       // 128 pixels
  constexpr int NCOL  = T == 64 ? 64 : 128;
  constexpr int TPT   = T * 16 / 128;  // (frame, 8-pixel group) items per thread per stage
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment of the swizzle atoms
  uint8_t  *smem  = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u); // stays a shared-space pointer
  uint64_t *mbar  = reinterpret_cast<uint64_t *>(smem + kTcStages * STAGE);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + kTcStages);
  unsigned long long *ssum = reinterpret_cast<unsigned long long *>(tslot + 2);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int w   = blockIdx.y;
  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s)
      tc::mbar_init(&mbar[s], 1);
    tc::mbar_fence_init();
  }
  for (int t = tid; t < T; t += blockDim.x)
    ssum[t] = 0ull;
  if (warp == 0)
    tc::tmem_alloc(tslot, NCOL);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;
  constexpr uint32_t idesc = tc::idesc_f16(T, T, false, false);

  // this thread's fixed (frame, group) items: t = tid/16 + 8k, g = tid % 16
  const int g = tid & 15;
  uint32_t  isum[TPT];
#pragma unroll
  for (int k = 0; k < TPT; ++k)
    isum[k] = 0u;

  const int64_t ntiles = (a.P + kTcPX - 1) / kTcPX;
  int           nj     = 0;
  bool          ok     = true;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++nj) {
    const int s = nj % kTcStages;
    bool      w_ok = true;
    if (nj >= kTcStages)
      w_ok = tc::mbar_wait_bounded(&mbar[s], (uint32_t)((nj / kTcStages) - 1) & 1u, status, 1);
    ok = __syncthreads_and(w_ok) != 0; // uniform: every thread leaves together on a timeout
    if (!ok)
      break;
    uint8_t      *st = smem + s * STAGE;
    const int64_t p  = tile * kTcPX + g * 8;
    const bool    valid = p < a.P;
#pragma unroll
    for (int k = 0; k < TPT; ++k) {
      const int t = (tid >> 4) + 8 * k;
      uint32_t  v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (valid) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(a.ring.frame(w, t) + 2 * p);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t wv = __ldg(src + i);
          v[2 * i]     = wv & 0xFFFFu;
          v[2 * i + 1] = wv >> 16;
        }
      }
      __half2 h[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        isum[k] += valid ? v[2 * i] + v[2 * i + 1] : 0u;
        const float x0 = valid ? (float)v[2 * i] - a.shift : 0.f;
        const float x1 = valid ? (float)v[2 * i + 1] - a.shift : 0.f;
        h[i] = __floats2half2_rn(x0, x1);
      }
      const int sub = g >> 3, c = g & 7;
      uint4    *dst = reinterpret_cast<uint4 *>(st + sub * SUB + t * 128 + ((c ^ (t & 7)) << 4));
      *dst = *reinterpret_cast<const uint4 *>(h);
    }
    tc::fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int sub = 0; sub < 2; ++sub)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint64_t d = tc::sw128_desc(tc::smem_u32(st + sub * SUB + ks * 32), 16, 1024);
          tc::mma_f16(tbase, d, d, idesc, (nj > 0 || sub > 0 || ks > 0) ? 1u : 0u);
        }
      tc::mma_commit(&mbar[s]);
    }
  }
  // drain: the last commit covers every MMA issued before it
  if (nj > 0 && ok) {
    const int last = nj - 1;
    ok = tc::mbar_wait_bounded(&mbar[last % kTcStages], (uint32_t)(last / kTcStages) & 1u, status, 2);
  }
  ok = __syncthreads_and(ok) != 0;
  tc::fence_after_sync();
#pragma unroll
  for (int k = 0; k < TPT; ++k)
    atomicAdd(&ssum[(tid >> 4) + 8 * k], (unsigned long long)isum[k]);

  const int64_t pidx = ((int64_t)w * a.nblk + blockIdx.x) * T * T;
  if constexpr (T == 64) {
    // M = 64 accumulator: row m sits in TMEM lane 32*(m/16) + m%16 (the lower half of each
    // 32-lane subpartition), columns 0..63 hold N = 0..63
    uint32_t r0[32], r1[32];
    tc::tmem_ld32(tbase + ((uint32_t)(32 * warp) << 16), r0);
    tc::tmem_ld32(tbase + ((uint32_t)(32 * warp) << 16) + 32, r1);
    tc::tmem_wait_ld();
    const int i = tid & 31;
    if (i < 16) {
      const int m = 16 * warp + i;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        a.partial[pidx + m * T + c]      = (nj > 0 && ok) ? __uint_as_float(r0[c]) : 0.f;
        a.partial[pidx + m * T + 32 + c] = (nj > 0 && ok) ? __uint_as_float(r1[c]) : 0.f;
      }
    }
  } else {
    const int m = 32 * warp + (tid & 31);
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      uint32_t r[32];
      tc::tmem_ld32(tbase + ((uint32_t)(32 * warp) << 16) + 32 * cb, r);
      tc::tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < 32; ++c)
        a.partial[pidx + m * T + 32 * cb + c] = (nj > 0 && ok) ? __uint_as_float(r[c]) : 0.f;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  for (int t = tid; t < T; t += blockDim.x)
    a.sums[((int64_t)w * gridDim.x + blockIdx.x) * T + t] = (double)ssum[t];
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, NCOL);
  }
}

// ------------------------------------------------------------------------------------------------
// Exact integer variant for samples of at most 12 bits: x = 16 h + l with h in [0, 255], l in [0, 15]
// (both unsigned bytes).  The stage of a 128-pixel tile holds 2 rows (h, l) per frame, K-major; kind::i8
// MMAs accumulate D = Z Z^T of a window's 2T rows Z in 32-bit TMEM columns, and
// G = 256 HH + 16 (HL + LH) + LL is folded into a per-window int64 accumulator with integer atomics
// (exact, so the result does not depend on their order).  An entry of D grows by at most 255^2 per pixel
// and the accumulators wrap, so a CTA of up to 65536 pixels leaves each one exact as an unsigned number.
//  - A CTA owns a group of up to G consecutive windows, i.e. the frames w0*hop + [0, F) with
//    F = T + (G - 1) hop, and stages every frame of the group once per tile.  G = 4 for T = 64
//    windows that overlap on an 8-frame grid (hop 8..32); G = 1 otherwise (T = 32, 64, 128).
//  - Operand rows come in 8-frame pairs of swizzle atoms, [h of frames 8p..8p+7][l of the same
//    frames], so window wl's 2T operand rows are the consecutive atoms from pair wl*hop/8: one
//    descriptor offset selects them.  T = 32 is one M = N = 64 MMA per K-step and T = 64 one
//    M = N = 128; T = 128 takes M = 128 twice, N = 256 for the first 64 frames' rows and N = 128
//    (the last 64 frames' columns) for the rest, since D is symmetric.
//  - Packed samples travel global -> shared through a ring of per-warp cp.async copies, D tiles deep;
//    each warp unpacks exactly the bytes it copied, so no block barrier guards the raw ring.  The lanes
//    copy the warp's 8 frame runs in order: lanes that copied their own 32 pixels, 48 bytes apart,
//    asked for every sector twice (3 % slower).
//  - The split is byte selects and masks on the packed stream (two pixels are b0 | (b1 & 15) << 8 and
//    b1 >> 4 | b2 << 4, so l and h are the halves of b0, b1 and b2 as it is): 12 instructions per 8
//    pixels.  The order of the pixels along K is free as long as every frame has the same.  Splitting at
//    6 bits around 2048, with the frame sums that undoing the shift needs, took 50 and bound the kernel.
// Measured, loads through registers between block barriers -> copy ring -> byte split: one 64 x 1024^2
// window 97 -> 48 -> 41 us (15 us of bytes), eight at hop 16 152 -> 149 -> 123, four of 128 x 1024 x 1536
// 718 -> 400 -> 274 (82 us of bytes read once; their products alone take 137 at the nominal int8 rate).
// Operand row r of a window holds frame 8 (r / 16) + r % 8, kind h when (r / 8) is even; the h-row
// and l-row of a frame sit 8 lanes apart in one warp and are folded with a shuffle before the
// integer atomics, which cover the upper triangle.
// Warp roles: the producer warps fill the stages and arrive (one arrival per warp) on the stage's
// `full` barrier; the last warp waits on it, issues the stage's MMAs and commits them to the
// stage's `free` barrier, so no producer waits for the others between tiles.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int FMT, int T, int G, int HOP8> struct GroupCov {
  static constexpr int F    = T + (G - 1) * 8 * HOP8;      // frames of a full group
  static constexpr int NT   = 4 * F;                       // one (frame, 32-pixel run) per thread
  static constexpr int RB   = FMT == HF_MONO12P ? 48 : 32; // packed bytes of a 32-pixel run
  static constexpr int D    = F <= 128 ? 4 : 3;            // raw ring depth (tiles)
  static constexpr int S    = F <= 136 ? 3 : 2;            // operand stages
  static constexpr int STG  = 256 * F;                     // 2F rows x 128 B
  static constexpr int NTHR = NT + 32;                     // producers + the MMA warp
  static constexpr int WCOL = 2 * T * (T == 128 ? 2 : 1);  // TMEM columns per window
  // CTAs per SM: one for the groups and T = 128 (their TMEM), else as many as shared memory holds
  static constexpr int PER_SM = G > 1 || T == 128 ? 1 : (T == 64 ? 2 : 4);
  static constexpr size_t smem = 1024 + (size_t)S * STG + (size_t)D * NT * RB + 2 * S * 8 + 16;
  static_assert(smem <= 227 * 1024 && PER_SM * WCOL * G <= 512, "Gram kernel resources");
};

// Bounded mbarrier wait that also gives up once another thread has raised `abort`; the first
// thread to time out records `code` in the status word and raises it.
__device__ __forceinline__ bool wait_or_abort(uint64_t *mbar, uint32_t parity, volatile int *abort, int *status,
                                              int code) {
  const uint64_t t0 = tc::globaltimer_ns();
  for (uint32_t i = 0; i < tc::kWaitLimit; ++i) {
    if (tc::mbar_try_wait(mbar, parity))
      return true;
    if ((i & 255u) == 255u && (*abort || tc::globaltimer_ns() - t0 > tc::kWaitNs))
      break;
  }
  if (!*abort && status)
    atomicCAS(status, 0, code);
  *abort = 1;
  return false;
}

template <int FMT, int T, int NG, int HOP8>
__global__ void __launch_bounds__(GroupCov<FMT, T, NG, HOP8>::NTHR, GroupCov<FMT, T, NG, HOP8>::PER_SM)
    cov_tc_group_kernel(FrameRing ring, int64_t P, int nwin, uint32_t ncols, unsigned long long *acc, int *status) {
  using G                = GroupCov<FMT, T, NG, HOP8>;
  constexpr int HOP      = 8 * HOP8;
  constexpr int M        = T == 32 ? 64 : 128; // MMA rows
  constexpr int NMB      = 2 * T / M;          // M-blocks
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t  *smem  = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u); // stays a shared-space pointer
  uint8_t  *raw   = smem + G::S * G::STG;
  uint64_t *mbar  = reinterpret_cast<uint64_t *>(raw + (size_t)G::D * G::NT * G::RB); // [S] free
  uint64_t *fullb = mbar + G::S;                                                        // [S] full
  uint32_t *tslot = reinterpret_cast<uint32_t *>(fullb + G::S);
  int      *abort_flag = reinterpret_cast<int *>(tslot + 1);
  volatile int *abortv = abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int w0  = NG * blockIdx.y;
  const int g   = min(NG, nwin - w0);  // windows of this group
  const int Fg  = T + (g - 1) * HOP;   // frames of this group
  const bool producer = tid < G::NT;   // the last warp issues the MMAs
  if (tid == 0) {
    for (int s = 0; s < G::S; ++s) {
      tc::mbar_init(&mbar[s], 1);              // the MMA commit of the stage's tile
      tc::mbar_init(&fullb[s], G::NT / 32);    // one arrival per producer warp
    }
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 0)
    tc::tmem_alloc(tslot, ncols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *tslot;

  const int      f      = tid >> 2, grp = tid & 3;
  const bool     active = f < Fg;
  uint8_t       *myraw  = raw + (size_t)tid * G::RB;
  // this thread's rows in the stage: frame f -> pair f / 8, row f % 8 of the pair's h and l atoms
  const int rr = f & 7, pr = f >> 3;

  const int64_t ntiles = (P + kTcPX - 1) / kTcPX;
  // A warp's 32 runs are 8 frames x 128 pixels; its lanes copy them in order, 16 bytes each
  constexpr int  CI = G::RB / 16;
  const uint8_t *csrc[CI];
#pragma unroll
  for (int i = 0; i < CI; ++i) {
    const int c = 32 * i + lane;
    csrc[i]     = active ? ring.frame(w0, 8 * warp + c / (4 * CI)) + 16 * (c % (4 * CI)) : nullptr;
  }
  auto issue = [&](int64_t tile, int slot) {
    uint8_t *dst = raw + (size_t)slot * G::NT * G::RB + (size_t)warp * 32 * G::RB + 16 * lane;
    if (active && tile < ntiles)
#pragma unroll
      for (int i = 0; i < CI; ++i) {
        const int run = (32 * i + lane) % (4 * CI) / CI; // of this frame, 32 pixels each
        if (tile * kTcPX + 32 * run < P)
          cp_async16(dst + 512 * i, csrc[i] + tile * (kTcPX * TcBpp<FMT>::num / TcBpp<FMT>::den));
      }
    cp_async_commit();
  };
  int      nj = 0;
  bool     ok = true;
  if (producer) {
#pragma unroll
  for (int d = 0; d < G::D - 1; ++d)
    issue(blockIdx.x + (int64_t)d * gridDim.x, d);
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++nj) {
    const int s = nj % G::S;
    issue(tile + (int64_t)(G::D - 1) * gridDim.x, (nj + G::D - 1) % G::D);
    bool w_ok = true;
    if (nj >= G::S) // the MMAs that read this stage S tiles ago are done
      w_ok = wait_or_abort(&mbar[s], (uint32_t)((nj / G::S) - 1) & 1u, abortv, status, 5);
    cp_async_wait<G::D - 1>();
    __syncwarp(); // the warp's copies of this tile have landed
    const bool valid = active && tile * kTcPX + grp * 32 < P;
    if (w_ok && active) {
      uint32_t hw[8], lw[8];
      if (valid) {
        const uint4 *src = reinterpret_cast<const uint4 *>(myraw + (size_t)(nj % G::D) * G::NT * G::RB);
        uint32_t     wv[G::RB / 4];
#pragma unroll
        for (int i = 0; i < G::RB / 16; ++i) {
          const uint4 v = src[i];
          wv[4 * i] = v.x, wv[4 * i + 1] = v.y, wv[4 * i + 2] = v.z, wv[4 * i + 3] = v.w;
        }
        if constexpr (FMT == HF_MONO12P) {
#pragma unroll
          for (int q = 0; q < 4; ++q) { // 8 pixels from 3 words: every third byte of the 12
            const uint32_t a0 = wv[3 * q], a1 = wv[3 * q + 1], a2 = wv[3 * q + 2];
            const uint32_t b0 = __byte_perm(__byte_perm(a0, a1, 0x0630), a2, 0x5210);
            const uint32_t b1 = __byte_perm(__byte_perm(a0, a1, 0x0741), a2, 0x6210);
            const uint32_t b2 = __byte_perm(__byte_perm(a0, a1, 0x0052), a2, 0x7410);
            lw[2 * q]     = b0 & 0x0F0F0F0Fu; // the four even pixels, then the four odd ones
            hw[2 * q]     = ((b0 >> 4) & 0x0F0F0F0Fu) | ((b1 << 4) & 0xF0F0F0F0u);
            lw[2 * q + 1] = (b1 >> 4) & 0x0F0F0F0Fu;
            hw[2 * q + 1] = b2;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            lw[i] = wv[i] & 0x0F0F0F0Fu;
            hw[i] = (wv[i] >> 4) & 0x0F0F0F0Fu;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          hw[i] = lw[i] = 0u;
      }
      uint8_t *hrow = smem + s * G::STG + pr * 2048 + rr * 128;
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        const int c = 2 * grp + hc;
        *reinterpret_cast<uint4 *>(hrow + ((c ^ rr) << 4)) =
            make_uint4(hw[4 * hc], hw[4 * hc + 1], hw[4 * hc + 2], hw[4 * hc + 3]);
        *reinterpret_cast<uint4 *>(hrow + 1024 + ((c ^ rr) << 4)) =
            make_uint4(lw[4 * hc], lw[4 * hc + 1], lw[4 * hc + 2], lw[4 * hc + 3]);
      }
    }
    tc::fence_proxy_async_smem(); // this thread's stage writes before the async proxy reads them
    __syncwarp();
    if (lane == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(&fullb[s])) : "memory");
    if (__any_sync(0xFFFFFFFFu, !w_ok || *abortv)) {
      ok = false;
      break;
    }
  }
  cp_async_wait<0>(); // no copy may land in shared memory after the CTA has left
  } else {
    // MMA warp: issue each stage's MMAs as soon as every producer warp has filled it
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++nj) {
      const int s = nj % G::S;
      if (!wait_or_abort(&fullb[s], (uint32_t)(nj / G::S) & 1u, abortv, status, 7)) {
        ok = false;
        break;
      }
      if (lane == 0) {
        tc::fence_after_sync();
        const uint8_t *st = smem + s * G::STG;
        for (int wl = 0; wl < g; ++wl) {
          const uint32_t z = tc::smem_u32(st + wl * HOP8 * 2048); // the window's first operand row
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
#pragma unroll
            for (int mb = 0; mb < NMB; ++mb) { // block mb against the columns from its own first row on
              const uint64_t d = tc::sw128_desc(z + mb * M * 128 + ks * 32, 16, 1024);
              tc::mma_i8(tbase + G::WCOL * wl + mb * 2 * T, d, d, tc::idesc_u8(M, 2 * T - mb * M, false, false),
                         (nj > 0 || ks > 0) ? 1u : 0u);
            }
        }
        tc::mma_commit(&mbar[s]);
      }
      __syncwarp();
    }
    if (nj > 0 && ok) { // drain: the last commit covers every MMA issued before it
      const int last = nj - 1;
      ok = wait_or_abort(&mbar[last % G::S], (uint32_t)(last / G::S) & 1u, abortv, status, 6);
    }
  }
  ok = __syncthreads_and(ok && !*abortv) != 0;
  tc::fence_after_sync();

  constexpr int NQ = G::NT / 128; // complete warp quads: each reads all 128 TMEM lanes
  if (nj > 0 && ok && warp < 4 * NQ) {
    const int q  = warp & 3;
    // operand row of this lane within its M-block; M = 64 keeps row m in TMEM lane 32 (m / 16) + m % 16
    const int       r    = M == 64 ? 16 * q + (lane & 15) : 32 * q + lane;
    const bool      is_h = ((r >> 3) & 1) == 0;
    const long long wh   = is_h ? 256 : 16, wlw = is_h ? 16 : 1;
    for (int it = warp >> 2; it < g * NMB; it += NQ) {
      const int wl = it / NMB, mb = it % NMB;
      const int a  = 8 * (r >> 4) + (r & 7) + 64 * mb; // this row's frame
      unsigned long long *aw = acc + (int64_t)(w0 + wl) * T * T + a * T;
#pragma unroll
      for (int cb = 0; cb < 2 * T / 32; ++cb) {
        if (cb >= (2 * T - mb * M) / 32)
          break;
        uint32_t v[32];
        tc::tmem_ld32(tbase + ((uint32_t)(32 * q) << 16) + G::WCOL * wl + mb * 2 * T + 32 * cb, v);
        tc::tmem_wait_ld();
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            // columns 16 half + c (h of frame b) and 16 half + 8 + c (l of frame b)
            const int b = 16 * cb + 8 * half + c + 64 * mb;
            long long e = wh * (long long)v[16 * half + c] + wlw * (long long)v[16 * half + 8 + c];
            e += __shfl_xor_sync(0xFFFFFFFFu, e, 8);
            if (is_h && a <= b && (M == 128 || lane < 16))
              atomicAdd(&aw[b], (unsigned long long)e);
          }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tbase, ncols);
  }
}

// int64 accumulator (upper triangle) -> float64 Gram.
__global__ void cov_i8_finalize_kernel(const unsigned long long *acc, int T, double *gram) {
  const int w = blockIdx.y;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= T * T)
    return;
  const int i = e / T, j = e % T;
  gram[(int64_t)w * T * T + e] = (double)acc[(int64_t)w * T * T + min(i, j) * T + max(i, j)];
}

template <int T>
int launch_tc(const FrameRing &ring, int64_t P, int nwin, void *ws, double *gram, int *status,
              cudaStream_t s) {
  const size_t smem = 1024 + (size_t)kTcStages * 2 * T * 128 + kTcStages * 8 + 8 + T * 8;
  const int64_t ntiles = (P + kTcPX - 1) / kTcPX;
  const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>(3LL * sm_count() / nwin, ntiles));
  CovArgs a;
  a.ring    = ring;
  a.T       = T;
  a.P       = P;
  a.shift   = 2048.f;
  a.nblk    = ctas;
  a.partial = reinterpret_cast<float *>(ws);
  a.sums    = reinterpret_cast<double *>(reinterpret_cast<uint8_t *>(ws) +
                                      (size_t)nwin * ctas * T * T * sizeof(float));
  HF_CUDA(cudaFuncSetAttribute(cov_tc_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cov_tc_kernel<T><<<dim3(ctas, nwin), 128, smem, s>>>(a, status);
  note_launch();
  HF_TRY(launch_status("cov_tc_kernel"));
  return launch_cov_finalize(a.partial, a.sums, a.nblk, ctas, T, P, (double)a.shift, gram, nwin, s);
}

template <int FMT, int T, int NG, int HOP8>
int launch_tc_group(const FrameRing &ring, int64_t P, int nwin, void *ws, double *gram, int *status,
                    cudaStream_t s) {
  using G               = GroupCov<FMT, T, NG, HOP8>;
  const int     ngroups = (nwin + NG - 1) / NG;
  const int64_t ntiles  = (P + kTcPX - 1) / kTcPX;
  // the CTAs of all groups fit the SMs at once, the SMs split evenly between the groups: one wave, or as
  // many full ones as keep a CTA at 512 tiles (65536 pixels, the accumulators' range)
  const int64_t min_ctas = (ntiles + 511) / 512, slots = (int64_t)G::PER_SM * sm_count();
  int64_t       waves    = 1;
  while (waves * slots / ngroups < min_ctas)
    ++waves;
  const int ctas = (int)std::max<int64_t>(min_ctas, std::min<int64_t>(std::max<int64_t>(1, waves * slots / ngroups), ntiles));
  uint32_t ncols = 32; // a power of two
  while (ncols < (uint32_t)(G::WCOL * std::min(nwin, NG)))
    ncols *= 2;
  auto *acc = reinterpret_cast<unsigned long long *>(ws);
  HF_CUDA(cudaMemsetAsync(acc, 0, (size_t)nwin * T * T * sizeof(unsigned long long), s));
  auto kern = cov_tc_group_kernel<FMT, T, NG, HOP8>;
  HF_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem));
  kern<<<dim3(ctas, ngroups), G::NTHR, G::smem, s>>>(ring, P, nwin, ncols, acc, status);
  note_launch();
  HF_TRY(launch_status("cov_tc_group_kernel"));
  cov_i8_finalize_kernel<<<dim3((T * T + 255) / 256, nwin), 256, 0, s>>>(acc, T, gram);
  note_launch();
  return launch_status("cov_i8_finalize_kernel");
}

// T = 64 windows that overlap on an 8-frame grid stage each frame once per group of four; the other
// shapes take one window per CTA.
template <int FMT>
int launch_i8(const FrameRing &ring, int T, int64_t P, int nwin, void *ws, double *gram, int *status, cudaStream_t s) {
  if (T == 32)
    return launch_tc_group<FMT, 32, 1, 0>(ring, P, nwin, ws, gram, status, s);
  if (T == 128)
    return launch_tc_group<FMT, 128, 1, 0>(ring, P, nwin, ws, gram, status, s);
  if (nwin >= 2 && ring.hop % 8 == 0)
    switch (ring.hop / 8) {
    case 1: return launch_tc_group<FMT, 64, 4, 1>(ring, P, nwin, ws, gram, status, s);
    case 2: return launch_tc_group<FMT, 64, 4, 2>(ring, P, nwin, ws, gram, status, s);
    case 3: return launch_tc_group<FMT, 64, 4, 3>(ring, P, nwin, ws, gram, status, s);
    case 4: return launch_tc_group<FMT, 64, 4, 4>(ring, P, nwin, ws, gram, status, s);
    default: break;
    }
  return launch_tc_group<FMT, 64, 1, 0>(ring, P, nwin, ws, gram, status, s);
}

} // namespace

size_t cov_tc_workspace_bytes(int T, int64_t P, int nwin) {
  const int64_t ntiles = (P + kTcPX - 1) / kTcPX;
  const int64_t ctas   = std::max<int64_t>(1, std::min<int64_t>((3LL * sm_count() + nwin - 1) / nwin, ntiles));
  const size_t f16 = (size_t)(nwin * ctas) * T * T * sizeof(float) + (size_t)(nwin * ctas) * T * sizeof(double) + 256;
  const size_t i8  = (size_t)nwin * T * T * sizeof(unsigned long long) + 256;
  return std::max(f16, i8);
}

bool cov_tc_exact(int fmt) { return fmt == HF_MONO12P || fmt == HF_U8; }

bool cov_tc_supported(int fmt, int T, int64_t P, int64_t frame_bytes) {
  if (cov_tc_exact(fmt)) // 16-byte loads of 32-pixel runs
    return (T == 32 || T == 64 || T == 128) && P % 32 == 0 && frame_bytes % 16 == 0;
  return fmt == HF_U16 && (T == 64 || T == 128) && P % 8 == 0 && frame_bytes % 4 == 0;
}

int launch_covariance_tc(const FrameRing &ring, int fmt, int T, int64_t P, int nwin, void *ws,
                         double *gram, int *status, cudaStream_t s) {
  HF_CHECK_ARG(cov_tc_supported(fmt, T, P, ring.frame_bytes), "tensor-core covariance: unsupported shape");
  // samples of at most 12 bits: exact int8 split; 16-bit samples: f16 operands
  if (fmt == HF_MONO12P)
    return launch_i8<HF_MONO12P>(ring, T, P, nwin, ws, gram, status, s);
  if (fmt == HF_U8)
    return launch_i8<HF_U8>(ring, T, P, nwin, ws, gram, status, s);
  return T == 64 ? launch_tc<64>(ring, P, nwin, ws, gram, status, s)
                 : launch_tc<128>(ring, P, nwin, ws, gram, status, s);
}

} // namespace hf
