// PCA / SVD clutter filter kernels: Gram matrix of a window's frames, FP64 Jacobi
// eigendecomposition, the filter+DFT matrix of the band, and the PCA projection.
//
// Reference: PcaTask::execute (holotask/src/syncs/pca.cc:68-119) computes C = X^T X with
// cublasGemmEx (FP16 tensor-core compute), an ascending eigendecomposition with cuSolverDx heev
// (pca_heev.cc:35-133) and the projection X V[:, begin:end].  Here the Gram matrix comes from
// k_cov_fp32.cu or k_tc_cov.cu; the eigensolver is FP64 throughout.
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <string>

#include "k_pca.cuh"

namespace hf {

namespace {

// Any T, no workspace (more than 128 frames, or callers that have or may use none): a CTA per window and
// 8 x 8 block of the upper triangle, its threads over the pixels, float64 accumulation, no shift, the
// threads' sums added pairwise.  Bound: a block's 16 rows are read once per block, from L2.  A thread per
// entry over all pixels took 319 us for 4 windows of 50 x 4096 16-bit pixels, here 15.
constexpr int kDirThr = 256;
template <int FMT>
__global__ void __launch_bounds__(kDirThr, 1) cov_direct_kernel(FrameRing ring, int T, int64_t P, double *gram) {
  __shared__ double red[kDirThr / 32][64];
  const int NB = (T + 7) / 8, w = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int       bi = 0, rem = blockIdx.x;
  while (rem >= NB - bi) {
    rem -= NB - bi;
    ++bi;
  }
  const int      bj = bi + rem;
  const uint8_t *fa[8], *fb[8]; // (rows beyond T repeat the last one and are not written)
#pragma unroll
  for (int i = 0; i < 8; ++i)
    fa[i] = ring.frame(w, min(8 * bi + i, T - 1)), fb[i] = ring.frame(w, min(8 * bj + i, T - 1));
  double acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      acc[i][j] = 0.0;
  for (int64_t p = tid; p < P; p += kDirThr) {
    double a[8], b[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      a[i] = (double)sample<FMT>(fa[i], p), b[i] = (double)sample<FMT>(fb[i], p);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        acc[i][j] = fma(a[i], b[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      double s = acc[i][j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0)
        red[warp][8 * i + j] = s;
    }
  __syncthreads();
  const int i = 8 * bi + (tid >> 3), j = 8 * bj + (tid & 7);
  if (tid < 64 && i <= j && j < T) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kDirThr / 32; ++q)
      s += red[q][tid];
    gram[(int64_t)w * T * T + (int64_t)i * T + j] = s;
    gram[(int64_t)w * T * T + (int64_t)j * T + i] = s;
  }
}

template <int FMT>
int launch_cov_direct_fmt(const FrameRing &ring, int T, int64_t P, int nwin, double *gram, cudaStream_t s) {
  const int64_t NB = (T + 7) / 8;
  cov_direct_kernel<FMT><<<dim3((unsigned)(NB * (NB + 1) / 2), nwin), kDirThr, 0, s>>>(ring, T, P, gram);
  note_launch();
  return launch_status("cov_direct_kernel");
}

int launch_cov_direct(const FrameRing &ring, int fmt, int T, int64_t P, int nwin, double *gram, cudaStream_t s) {
  switch (fmt) {
  case HF_MONO12P: return launch_cov_direct_fmt<HF_MONO12P>(ring, T, P, nwin, gram, s);
  case HF_U16: return launch_cov_direct_fmt<HF_U16>(ring, T, P, nwin, gram, s);
  case HF_U8: return launch_cov_direct_fmt<HF_U8>(ring, T, P, nwin, gram, s);
  case HF_F32: return launch_cov_direct_fmt<HF_F32>(ring, T, P, nwin, gram, s);
  default: return fail(HF_ERR_INVALID, "covariance: unsupported input dtype");
  }
}

// ------------------------------------------------------------------------------------------------
// Jacobi
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void pair_of(int r, int k, int n, int &p, int &q) {
  if (k == 0) {
    p = n - 1;
    q = r;
  } else {
    p = (r + k) % (n - 1);
    q = (r - k + (n - 1)) % (n - 1);
  }
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
}

// Packed upper-triangle index of the symmetric matrix (i <= j).
__device__ __forceinline__ int sym_idx(int i, int j, int np) {
  if (i > j) {
    const int t = i;
    i = j;
    j = t;
  }
  return i * np - (i * (i - 1)) / 2 + (j - i);
}

// Parallel cyclic Jacobi (round-robin pairing, np/2 disjoint rotations per step).  The matrix is
// kept as a packed upper triangle and the rotation accumulator transposed (Vt[p][:] = V[:, p]),
// both in shared memory (194 KB at n = 128).  Every thread owns a fixed set of 2x2 blocks (k, l)
// and accumulator entries for the whole solve, so a step is: rotations of the np/2 pairs,
// barrier, block and accumulator updates, barrier.
constexpr int kJacobiThreads = 1024;
constexpr int kJacobiMaxBlk  = 3;  // 2x2 blocks per thread: ceil(65*64/2 / 1024)
constexpr int kJacobiMaxV    = 8;  // accumulator entries per thread: 64*128 / 1024

__global__ void __launch_bounds__(kJacobiThreads) jacobi_kernel(const double *a_in, double *evecs,
                                                                double *evals, int *info, int n) {
  extern __shared__ __align__(16) double dsm[];
  const int np   = n + (n & 1);
  const int half = np / 2;
  const int npk  = np * (np + 1) / 2;
  double   *A    = dsm;                                    // packed [npk]
  double   *Vt   = A + npk;                                // [np][np]
  double   *cs   = Vt + np * np;                           // [half][2]
  int      *pq   = reinterpret_cast<int *>(cs + 2 * half); // [half][2]
  int      *flag = pq + 2 * half;
  const int tid = threadIdx.x, nt = blockDim.x;
  const double *src = a_in + (int64_t)blockIdx.x * n * n;

  for (int e = tid; e < np * np; e += nt) {
    const int i = e / np, j = e % np;
    Vt[e] = i == j ? 1.0 : 0.0;
    if (i <= j) {
      double v = 0.0;
      if (i < n && j < n)
        v = 0.5 * (src[i * n + j] + src[j * n + i]);
      else if (i == j)
        v = -DBL_MAX; // padding entry of an odd order: sorts first and is dropped
      A[sym_idx(i, j, np)] = v;
    }
  }
  // absolute rotation threshold: entries below 2^-52 of the trace (the matrix is a Gram matrix,
  // so the trace bounds its norm) are at the rounding level of the largest eigenvalues and cannot
  // be reduced further by two-sided rotations
  __syncthreads(); // the cooperative load of A above must be complete
  if (tid == 0) {
    double tr = 0.0;
    for (int i = 0; i < n; ++i)
      tr += fabs(A[sym_idx(i, i, np)]);
    cs[0] = tr * 2.220446049250313e-16;
  }
  __syncthreads();
  const double tol_abs = cs[0];
  __syncthreads();
  // this thread's fixed work items
  const int nblocks = half * (half + 1) / 2;
  int       bk[kJacobiMaxBlk], bl[kJacobiMaxBlk], nb = 0;
  for (int e = tid; e < nblocks && nb < kJacobiMaxBlk; e += nt) {
    int k = 0, rem = e;
    while (rem >= half - k) {
      rem -= half - k;
      ++k;
    }
    bk[nb] = k;
    bl[nb] = k + rem;
    ++nb;
  }
  int vk[kJacobiMaxV], vj[kJacobiMaxV], nv = 0;
  for (int f = tid; f < half * np && nv < kJacobiMaxV; f += nt) {
    vk[nv] = f / np;
    vj[nv] = f % np;
    ++nv;
  }
  __syncthreads();

  const int max_sweeps = 40;
  int       sweep      = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (tid == 0)
      flag[0] = 0;
    __syncthreads();
    for (int r = 0; r < np - 1; ++r) {
      if (tid < half) {
        int p, q;
        pair_of(r, tid, np, p, q);
        const double app = A[sym_idx(p, p, np)], aqq = A[sym_idx(q, q, np)];
        const double apq = A[sym_idx(p, q, np)];
        double       c = 1.0, s = 0.0;
        const bool   pad = (p >= n) || (q >= n);
        if (!pad && fabs(apq) > tol_abs && fabs(apq) > 1e-15 * sqrt(fabs(app * aqq))) {
          // t = tan(phi) of the annihilating rotation, the smaller root of t^2 + 2 theta t - 1 = 0
          // with theta = d / (2 apq), d = aqq - app, written with one square root and one division
          const double d  = aqq - app;
          const double a2 = 2.0 * apq;
          const double t  = (d >= 0.0 ? a2 : -a2) / (fabs(d) + sqrt(fma(d, d, a2 * a2)));
          c = rsqrt(fma(t, t, 1.0));
          s = t * c;
          flag[0] = 1;
        }
        cs[2 * tid]     = c;
        cs[2 * tid + 1] = s;
        pq[2 * tid]     = p;
        pq[2 * tid + 1] = q;
      }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < kJacobiMaxBlk; ++b) {
        if (b >= nb)
          break;
        const int    k = bk[b], l = bl[b];
        const double ck = cs[2 * k], sk = cs[2 * k + 1], cl = cs[2 * l], sl = cs[2 * l + 1];
        if (sk == 0.0 && sl == 0.0)
          continue;
        const int pk = pq[2 * k], qk = pq[2 * k + 1], pl = pq[2 * l], ql = pq[2 * l + 1];
        const int i00 = sym_idx(pk, pl, np), i01 = sym_idx(pk, ql, np);
        const int i10 = sym_idx(qk, pl, np), i11 = sym_idx(qk, ql, np);
        const double b00 = A[i00], b01 = A[i01], b10 = A[i10], b11 = A[i11];
        // M = B J_l ;  B' = J_k^T M   with J = [[c, s], [-s, c]]
        const double m00 = cl * b00 - sl * b01, m01 = sl * b00 + cl * b01;
        const double m10 = cl * b10 - sl * b11, m11 = sl * b10 + cl * b11;
        const double n00 = ck * m00 - sk * m10, n01 = ck * m01 - sk * m11;
        const double n10 = sk * m00 + ck * m10, n11 = sk * m01 + ck * m11;
        if (k == l) { // diagonal block: i01 == i10 is the annihilated entry
          A[i00] = n00;
          A[i11] = n11;
          A[i01] = 0.0;
        } else {
          A[i00] = n00;
          A[i01] = n01;
          A[i10] = n10;
          A[i11] = n11;
        }
      }
#pragma unroll
      for (int v = 0; v < kJacobiMaxV; ++v) {
        if (v >= nv)
          break;
        const int    k = vk[v], j = vj[v];
        const double c = cs[2 * k], s = cs[2 * k + 1];
        if (s != 0.0) {
          const int    p = pq[2 * k], q = pq[2 * k + 1];
          const double vp = Vt[p * np + j], vq = Vt[q * np + j];
          Vt[p * np + j] = c * vp - s * vq;
          Vt[q * np + j] = s * vp + c * vq;
        }
      }
      __syncthreads();
    }
    const int any = flag[0];
    __syncthreads();
    if (any == 0)
      break;
  }
  // ascending rank sort (ties by index) and write out
  double *ev  = evals + (int64_t)blockIdx.x * n;
  double *vec = evecs + (int64_t)blockIdx.x * n * n;
  for (int i = tid; i < np; i += nt) {
    const double li   = A[sym_idx(i, i, np)];
    int          rank = 0;
    for (int j = 0; j < np; ++j) {
      const double lj = A[sym_idx(j, j, np)];
      rank += (lj < li) || (lj == li && j < i);
    }
    if (np != n)
      rank -= 1;
    if (i < n) {
      ev[rank] = li;
      for (int t = 0; t < n; ++t)
        vec[t * n + rank] = Vt[i * np + t];
    }
  }
  if (tid == 0 && info != nullptr)
    info[blockIdx.x] = (sweep >= max_sweeps) ? sweep : 0;
}

// W = (I - V V^T) D[:, bins]; one CTA per window.  bins = [z0, z1), followed for the two-sided
// method by [T - z1, T - z0) (graph_builder.cc:270-287: the positive then the negative band).
__device__ __forceinline__ int band_bin(int kk, int z0, int z1, int T) {
  const int nzh = z1 - z0;
  return kk < nzh ? z0 + kk : T - z1 + (kk - nzh);
}

// One CTA per matrix.  The T roots exp(-2 pi i m / T) come from a table built once and the projections
// V^T D run as kBmLanes partial sums per (vector, bin), added pairwise.  Evaluating a sine and a cosine
// per product and one serial sum per entry took 36 us at T = 64, Nz = 28 (7 now) and 74 at T = 128,
// Nz = 56 (18 now).
constexpr int kBmThr   = 512;
constexpr int kBmLanes = 8;
__global__ void __launch_bounds__(kBmThr) band_matrix_kernel(const double *evecs, int T, int rank, int z0, int z1,
                                                             int two_sided, int staged, float2 *wmat) {
  extern __shared__ __align__(16) double bsm[];
  const int     nz  = (z1 - z0) * (two_sided ? 2 : 1);
  const double *V   = evecs + (int64_t)blockIdx.x * T * T + (T - rank);
  double       *cr  = bsm;                     // [rank][nz] re
  double       *ci  = cr + rank * nz;          // [rank][nz] im
  double       *rc  = ci + rank * nz, *rs = rc + T; // [T] cos, sin of -2 pi m / T (staged)
  double       *vst = rs + T;                  // [T][rank] the removed eigenvectors (staged)
  const double *vs  = staged ? vst : V;
  const int     ldv = staged ? rank : T;
  if (staged) {
    for (int m = threadIdx.x; m < T; m += kBmThr)
      sincospi(-2.0 * (double)m / (double)T, &rs[m], &rc[m]);
    for (int e = threadIdx.x; e < T * rank; e += kBmThr) {
      const int t = e / rank, m = e - t * rank;
      vst[e]      = V[t * T + m];
    }
    __syncthreads();
  }
  const auto root = [&](int i, double &c, double &s) {
    if (staged)
      c = rc[i], s = rs[i];
    else
      sincospi(-2.0 * (double)i / (double)T, &s, &c);
  };
  const int work = rank * nz * kBmLanes;
  for (int e0 = 0; e0 < work; e0 += kBmThr) { // whole warps take part in the shuffles
    const int  e  = e0 + threadIdx.x, q = e % kBmLanes, o = e / kBmLanes;
    const bool in = e < work;
    double     sr = 0.0, si = 0.0;
    if (in) {
      const int m = o / nz, bin = band_bin(o - m * nz, z0, z1, T);
      for (int t = q; t < T; t += kBmLanes) {
        const double v = vs[t * ldv + m];
        double       c, sn;
        root((t * bin) % T, c, sn);
        sr = fma(v, c, sr);
        si = fma(v, sn, si);
      }
    }
#pragma unroll
    for (int s = kBmLanes / 2; s > 0; s >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, s);
      si += __shfl_xor_sync(0xffffffffu, si, s);
    }
    if (in && q == 0)
      cr[o] = sr, ci[o] = si;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < T * nz; e += kBmThr) {
    const int t = e / nz, kk = e - t * nz;
    double    wr, wi;
    root((t * band_bin(kk, z0, z1, T)) % T, wr, wi);
    for (int m = 0; m < rank; ++m) {
      const double v = vs[t * ldv + m];
      wr = fma(-v, cr[m * nz + kk], wr);
      wi = fma(-v, ci[m * nz + kk], wi);
    }
    wmat[(int64_t)blockIdx.x * T * nz + e] = make_float2((float)wr, (float)wi);
  }
}

__global__ void pca_project_kernel(const float *in, int T, int64_t P, const double *evecs,
                                   int begin, int ncomp, float *out) {
  extern __shared__ float vsh[]; // [T][ncomp]
  const int64_t b = blockIdx.y;
  const double *V = evecs + b * T * T;
  for (int e = threadIdx.x; e < T * ncomp; e += blockDim.x)
    vsh[e] = (float)V[(e / ncomp) * T + begin + (e % ncomp)];
  __syncthreads();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P)
    return;
  const float *x = in + b * T * P + p;
  for (int c0 = 0; c0 < ncomp; c0 += 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int t = 0; t < T; ++t) {
      const float xv = x[(int64_t)t * P];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < ncomp)
          acc[j] = fmaf(xv, vsh[t * ncomp + c0 + j], acc[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c0 + j < ncomp)
        out[(b * ncomp + c0 + j) * P + p] = acc[j];
  }
}

} // namespace

size_t cov_workspace_bytes(int T, int64_t P, int max_windows) {
  return cov_cores_supported(T) ? cov_cores_workspace_bytes(T, P, max_windows) : 256;
}

int launch_covariance(const FrameRing &ring, int fmt, int T, int64_t P, int nwin, void *ws,
                      double *gram, cudaStream_t s) {
  HF_CHECK_ARG(T > 0 && P > 0 && nwin > 0, "covariance: empty problem");
  if (ws != nullptr && cov_cores_supported(T))
    return launch_cov_cores(ring, fmt, T, P, nwin, ws, gram, 0, s);
  return launch_cov_direct(ring, fmt, T, P, nwin, gram, s);
}

int launch_jacobi(const double *a, double *evecs, double *evals, int *info, int n, int64_t batch,
                  cudaStream_t s) {
  HF_CHECK_ARG(n >= 1 && n <= 128 && batch >= 1, "jacobi: order must be in [1, 128]");
  const int    np   = n + (n & 1);
  const size_t smem = (size_t)(np * (np + 1) / 2) * 8 + (size_t)np * np * 8 + (size_t)np * 8 +
                      (size_t)np * 4 + 16;
  HF_CUDA(cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  jacobi_kernel<<<(unsigned)batch, kJacobiThreads, smem, s>>>(a, evecs, evals, info, n);
  note_launch();
  return launch_status("jacobi_kernel");
}

int launch_band_matrix(const double *evecs, int64_t batch, int T, int rank, int z0, int z1,
                       float2 *wmat, cudaStream_t s, bool two_sided) {
  HF_CHECK_ARG(T > 0 && z0 >= 0 && z1 > z0 && z1 <= T && rank >= 0 && rank <= T, "band matrix: bad range");
  const size_t proj = (size_t)2 * std::max(rank, 1) * (z1 - z0) * (two_sided ? 2 : 1) * sizeof(double);
  // the table and the eigenvectors are staged where they fit (every plan of rank <= 60 at T = 128)
  const size_t stage  = ((size_t)2 * T + (size_t)T * rank) * sizeof(double);
  const int    staged = proj + stage <= 200 * 1024;
  const size_t smem   = proj + (staged ? stage : 0);
  HF_CUDA(cudaFuncSetAttribute(band_matrix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  band_matrix_kernel<<<(unsigned)batch, kBmThr, smem, s>>>(evecs, T, rank, z0, z1, two_sided ? 1 : 0, staged,
                                                                wmat);
  note_launch();
  return launch_status("band_matrix_kernel");
}

int launch_pca_project(const float *in, int64_t batch, int T, int64_t P, const double *evecs,
                       int begin, int end, float *out, cudaStream_t s) {
  HF_CHECK_ARG(begin >= 0 && end > begin && end <= T, "pca projection: bad component range");
  const int    ncomp = end - begin;
  const size_t smem  = (size_t)T * ncomp * sizeof(float);
  HF_CUDA(cudaFuncSetAttribute(pca_project_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  pca_project_kernel<<<dim3((unsigned)((P + 255) / 256), (unsigned)batch), 256, smem, s>>>(
      in, T, P, evecs, begin, ncomp, out);
  note_launch();
  return launch_status("pca_project_kernel");
}

// ------------------------------------------------------------------------------------------------
// Gram matrices with a fixed, library-owned workspace (hf_covariance_noalloc).
//
// The workspace is a file-scope device array, so the module loader reserves it once per device
// and the call itself never allocates.  Its device address is looked up once per device (with
// that device current) and cached.  The kernel writes every partial and per-frame sum the
// reduction reads before it is read, so nothing in the array has to start at zero.  Every call
// on a device uses the same array: calls whose work overlaps in time race on it.
// ------------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_cov_scratch[HF_COVARIANCE_NOALLOC_SCRATCH_BYTES];

namespace {
constexpr int kMaxScratchDevices = 64;
std::mutex    g_scratch_mu;
void         *g_scratch_ptr[kMaxScratchDevices] = {};

int scratch_address(void **ptr) {
  int dev = 0;
  HF_CUDA(cudaGetDevice(&dev));
  HF_CHECK_ARG(dev >= 0 && dev < kMaxScratchDevices, "hf_covariance_noalloc: device ordinal above 63");
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_ptr[dev] == nullptr) {
    void             *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_cov_scratch);
    if (e != cudaSuccess)
      return cuda_status(e, "hf_covariance_noalloc: cudaGetSymbolAddress of the fixed workspace");
    g_scratch_ptr[dev] = p;
  }
  *ptr = g_scratch_ptr[dev];
  return HF_OK;
}

// One CTA's partials as the batch limit counts them (the kernel needs no more).
size_t fixed_cta_bytes(int T) {
  const int G = T == 32 ? 4 : (T == 64 ? 2 : 1);
  return (size_t)G * T * T * sizeof(float) + (size_t)T * sizeof(double);
}
} // namespace

int launch_covariance_fixed_scratch(const FrameRing &ring, int fmt, int T, int64_t P, int nwin, double *gram,
                                    cudaStream_t s) {
  HF_CHECK_ARG(T > 0 && P > 0 && nwin > 0, "covariance: empty problem");
  // only the FP32 sums use the workspace, which calls that overlap in time would share
  if (!cov_sums_fp32(ring, T, P))
    return launch_cov_direct(ring, fmt, T, P, nwin, gram, s);
  const size_t fit = (HF_COVARIANCE_NOALLOC_SCRATCH_BYTES - 256) / ((size_t)nwin * fixed_cta_bytes(T));
  if (fit < 1)
    return fail(HF_ERR_INVALID,
                "hf_covariance_noalloc: batch " + std::to_string(nwin) + " at T = " + std::to_string(T) +
                    " needs more than the fixed " +
                    std::to_string(HF_COVARIANCE_NOALLOC_SCRATCH_BYTES >> 20) +
                    " MiB workspace; split the batch or use hf_covariance with a workspace");
  void *ws = nullptr;
  HF_TRY(scratch_address(&ws));
  return launch_cov_cores(ring, fmt, T, P, nwin, ws, gram, (int)std::min<size_t>(fit, (size_t)1 << 20), s);
}

} // namespace hf
