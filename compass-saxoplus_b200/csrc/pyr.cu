// High-resolution pyramid wavefront sensor with modulation.
//
// Reference: SutraWfs_PyrHR::comp_generic / comp_modulation
// (libsutra/src.cpp/sutra_wfs_pyr_pyrhr.cpp:379-627) and its kernels
// (libsutra/src.cu/sutra_wfs.cu: pyrgetpup_krnl :1191-1233, submask_krnl and
// submaskpyr_krnl :1864-1958, pyr_bimg_krnl :1580-1630, pyrfact_krnl
// :2164-2241; abs2_krnl with a factor, sutra_utils.cu:118-142).  Per
// modulation point the reference fills the padded pupil field, runs a cuFFT
// inverse transform, multiplies by the field stop and the pyramid phase mask,
// runs a forward transform and accumulates the weighted |.|^2; then the
// high-resolution image is convolved with the pixel transfer function (FFT,
// x sinc, FFT), binned by nrebin and normalised to nphot.
//
// Here the npts modulation planes (npts x nfft^2 complex, 50 MB at 512^2 x 24:
// resident in the 126 MB L2) go through three fused passes, each with the
// transforms in registers (fft.cuh), so a plane crosses memory once per pass
// and shared memory only between the radix-8 passes:
//   rows   inverse transform along x of the ntot pupil rows only (the other
//          rows of the padded field are zero), field and modulation tilt
//          formed on the fly, straight into the registers;
//   cols   per group of columns: inverse transform along y, field stop x
//          pyramid mask, forward transform along y; a CTA keeps the columns'
//          mask and the twiddles in registers over its modulation points;
//   accum  per row y: forward transform along x of every modulation plane, the
//          weighted |.|^2 summed in registers by groups of threads (points g,
//          g + G, ...), then over the groups; the complete row goes on to the
//          pixel transfer function's first transform in the same kernel.
// The pixel transfer function's column and second row transforms follow, the
// last one bins its rows, and one kernel normalises and adds the Philox photon /
// readout noise of the SH sensor (same sampler, same streams).

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "aob_objects.hpp"
#include "fft.cuh"

namespace aob {

constexpr int PYR_MAX_REBIN = 8;
constexpr int PYR_THREADS = 512;      // binning: threads per CTA, at most
// accum: threads per CTA, at most -- two CTAs of 256 on an SM overlap one's last steps
// (the sum over its groups and one group's transform) with the other's planes: 83.1 us
// for the 512 x 512 image, its slopes and commands, 89.2 with CTAs of 512, 82.7 with
// 128, which nfft 2048 (256 threads a sequence) does not allow
constexpr int PYR_ACC_THREADS = 256;
constexpr int PYR_ROW_THREADS = 256;

struct PyrArgs {
  int ntot, off, npts;
  const float *phase, *pupil;
  float mic2rad;
  const float *cx, *cy, *w;
  const float *submask;
  const float2 *phalfxy;
  const float *sincar;
  int early;         // the tables' addresses have stayed inside the library
  const float2 *tw;  // N/2 forward twiddles (global)
  float2 *work;      // npts x N x N
  float2 *conv;      // N x N
  float *hrimg;      // N x N
  float *binimg;     // nb x nb
  float *partial;    // nb row sums
  float *focal_work; // npts x N x N, w_p |field stop x focal field|^2 (null: not computed)
  int nrebin, nb;
};

// complex multiply
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.y * b.x + a.x * b.y);
}

// 1. rows of the padded pupil field, inverse transform along x; a group of
//    N / 8 threads takes one pupil row of one modulation point: work[p][yb][:].
template <int N>
__global__ void __launch_bounds__(PYR_ROW_THREADS) pyr_rows_kernel(PyrArgs A) {
  constexpr int T = N / 8, SEQ = PYR_ROW_THREADS / T, BS = fft_smem_elems(N);
  __shared__ float2 s[SEQ * 2 * BS];
  const int g = threadIdx.x / T, j = threadIdx.x % T;
  const int q = blockIdx.x * SEQ + g;
  const bool active = q < A.npts * A.ntot;
  const int p = active ? q / A.ntot : 0, yb = active ? q - p * A.ntot : 0;
  FftTw<N> W;
  dep_launch();
  W.load(A.tw, j);
  dep_wait();
  const float cxp = A.cx[p], cyp = A.cy[p];
  const float yy = (float)yb - A.ntot / 2.0f;
  float2 v[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int x = j + T * m - A.off;
    v[m] = make_float2(0.f, 0.f);
    if (active && x >= 0 && x < A.ntot) {
      const int id = x + yb * A.ntot;
      const float xx = (float)x - A.ntot / 2.0f;
      float sn, cs;
      sincosf(A.phase[id] * A.mic2rad + (cxp * xx + cyp * yy), &sn, &cs);
      const float a = A.pupil[id];
      v[m] = make_float2(cs * a, sn * a);
    }
  }
  fft_regs<N, 1, BS, true>(v, W, j, s + g * 2 * BS, GroupSync<T>{g});
  if (active) {
    float2 *row = A.work + ((size_t)p * N + yb) * N;
#pragma unroll
    for (int m = 0; m < 8; ++m) row[j + T * m] = v[m];
  }
}

// columns per CTA: 8 (64-byte segments), fewer where 8 would pass 512 threads
constexpr int pyr_cols(int n) { return n <= 512 ? 8 : 4096 / n; }

// 2. per unit -- a group of columns of one modulation plane: inverse transform
//    along y (rows outside the pupil are zero), x field stop, x pyramid phase mask
//    (submask_krnl, submaskpyr_krnl), forward transform along y.  In place in
//    work[p].  A CTA takes an equal run of units, a column group's planes one after
//    the other, so that it loads the mask once per group and no SM waits for a
//    last wave (1536 units at nfft 512 and 24 points: 11 on the fullest of 148 SMs).
//    Bound: instruction issue (about 300 per thread and transform) with one
//    512-thread CTA per SM at these registers; the next unit's loads go out
//    before the current one's transforms.  The whole image and its slopes at nfft
//    512, 24 points, with a 1600-actuator command matrix: 83 us per pass, 181 us
//    when every radix-8 pass went through shared memory and every point was
//    read and written with bank conflicts.
template <int N, bool FOCAL>
__global__ void __launch_bounds__(N / 8 * pyr_cols(N)) pyr_cols_kernel(PyrArgs A) {
  extern __shared__ float2 sm[];
  constexpr int T = N / 8, CB = pyr_cols(N), BS = fft_smem_elems(N) * CB;
  const int c = threadIdx.x % CB, j = threadIdx.x / CB;
  float2 *s = sm + c;
  FftTw<N> W;
  dep_launch();
  W.load(A.tw, j);
  const int64_t units = (int64_t)(N / CB) * A.npts;  // unit = group * npts + point
  int u = (int)(blockIdx.x * units / gridDim.x);
  const int u1 = (int)((blockIdx.x + 1) * units / gridDim.x);
  float2 mask[8];
  auto load_mask = [&](int x) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const size_t g = x + (size_t)(j + T * m) * N;
      const float msk = A.submask[g];
      mask[m] = A.phalfxy[g];
      if (!FOCAL) mask[m] = make_float2(mask[m].x * msk, mask[m].y * msk);
    }
  };
  auto load = [&](float2(&v)[8], int unit) {
    const int g = unit / A.npts;
    const float2 *base = A.work + (size_t)(unit - g * A.npts) * N * N + g * CB + c;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      const int yb = j + T * m - A.off;
      v[m] = (yb >= 0 && yb < A.ntot) ? __ldcg(base + (size_t)yb * N) : make_float2(0.f, 0.f);
    }
  };
  int group = u / A.npts;
  // the mask is uploaded by the host and asked for ahead of the wait, until its address has
  // been handed out (aob_pyr_buffer): a kernel of the caller may then write it
  if (!A.early) dep_wait();
  load_mask(group * CB + c);
  dep_wait();
  // rows [0, ntot) hold the input and are overwritten by the output: every
  // thread of the column has its input in registers by the first barrier
  float2 nxt[8];
  load(nxt, u);
  for (; u < u1; ++u) {
    const int g0 = u / A.npts, p = u - g0 * A.npts;
    if (g0 != group) {
      group = g0;
      load_mask(group * CB + c);
    }
    const int x = group * CB + c;
    float2 v[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = nxt[m];
    if (u + 1 < u1) load(nxt, u + 1);
    fft_regs<N, CB, BS, true>(v, W, j, s, CtaSync{});
    if (fft_odd_exchanges(N)) __syncthreads();
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      if (FOCAL) {
        // the focal plane image (compute_pyrfocalplane): abs2_krnl with the point's weight
        const size_t g = x + (size_t)(j + T * m) * N;
        const float msk = A.submask[g];
        v[m] = make_float2(v[m].x * msk, v[m].y * msk);
        A.focal_work[(size_t)p * N * N + g] = A.w[p] * (v[m].x * v[m].x + v[m].y * v[m].y);
      }
      v[m] = cmul(v[m], mask[m]);
    }
    fft_regs<N, CB, BS, false>(v, W, j, s, CtaSync{});
    float2 *base = A.work + (size_t)p * N * N + x;
#pragma unroll
    for (int m = 0; m < 8; ++m) __stcg(base + (size_t)(j + T * m) * N, v[m]);
    if (fft_odd_exchanges(N)) __syncthreads();
  }
}

// 3. per row y: forward transform along x of every modulation plane, hrimg[y][x]
//    = sum_p w_p |.|^2 (abs2_krnl with the modulation weight) -- group g of the
//    CTA sums points g, g + G, ..., the groups are added in order -- then the
//    pixel transfer function's inverse transform along x of that row.
template <int N>
__global__ void __launch_bounds__(PYR_ACC_THREADS) pyr_accum_kernel(PyrArgs A) {
  extern __shared__ float2 sm[];
  constexpr int T = N / 8, BS = fft_smem_elems(N);
  const int g = threadIdx.x / T, j = threadIdx.x % T, G = blockDim.x / T;
  const int y = blockIdx.x;
  const GroupSync<T> sync{g};
  float2 *s = sm + g * 2 * BS;
  FftTw<N> W;
  dep_launch();
  W.load(A.tw, j);
  dep_wait();
  float acc[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) acc[m] = 0.f;
  float2 nxt[8];
  auto load = [&](int p) {
#pragma unroll
    for (int m = 0; m < 8; ++m)
      nxt[m] = p < A.npts ? __ldcg(A.work + ((size_t)p * N + y) * N + j + T * m) : make_float2(0.f, 0.f);
  };
  load(g);
  // (every group makes the same number of passes: groups of one warp share its barrier)
  for (int p = g, r = (A.npts + G - 1) / G; r > 0; --r, p += G) {
    float2 v[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = nxt[m];
    const float w = p < A.npts ? A.w[p] : 0.f;
    if (r > 1) load(p + G);
    fft_regs<N, 1, BS, false>(v, W, j, s, sync);
    if (fft_odd_exchanges(N)) sync();
    if (p < A.npts) {
#pragma unroll
      for (int m = 0; m < 8; ++m) acc[m] += w * (v[m].x * v[m].x + v[m].y * v[m].y);
    }
  }
  __syncthreads();  // the exchange buffers are free: the groups' sums, then the row
  float *red = reinterpret_cast<float *>(sm);
#pragma unroll
  for (int m = 0; m < 8; ++m) red[g * N + j + T * m] = acc[m];
  __syncthreads();
  for (int x = threadIdx.x; x < N; x += blockDim.x) {
    float t = red[x];
    for (int q = 1; q < G; ++q) t += red[q * N + x];
    A.hrimg[(size_t)y * N + x] = t;
    red[x] = t;
  }
  __syncthreads();
  float2 v[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = make_float2(red[j + T * m], 0.f);
  __syncthreads();
  // the first group takes the row on (with groups of less than a warp, that warp's)
  if (threadIdx.x < (T < 32 ? 32 : T)) {
    fft_regs<N, 1, BS, true>(v, W, j, s, sync);
    if (g == 0) {
#pragma unroll
      for (int m = 0; m < 8; ++m) A.conv[(size_t)y * N + j + T * m] = v[m];
    }
  }
}

// 4. pixel transfer function, columns: inverse transform along y, x sinc, forward
//    transform along y.  Fewer columns per CTA than in the modulation planes: one
//    image has to spread over the whole GPU.
constexpr int pyr_conv_cols(int n) { return n <= 1024 ? 4 : 2; }
template <int N>
__global__ void __launch_bounds__(N / 8 * pyr_conv_cols(N)) pyr_conv_cols_kernel(PyrArgs A) {
  extern __shared__ float2 sm[];
  constexpr int T = N / 8, CB = pyr_conv_cols(N), BS = fft_smem_elems(N) * CB;
  const int c = threadIdx.x % CB, j = threadIdx.x / CB;
  const int x = blockIdx.x * CB + c;
  float2 *s = sm + c;
  float2 v[8];
  float msk[8];
  FftTw<N> W;
  dep_launch();
  W.load(A.tw, j);
  if (!A.early) dep_wait();  // (see pyr_cols_kernel)
#pragma unroll
  for (int m = 0; m < 8; ++m) msk[m] = A.sincar[x + (size_t)(j + T * m) * N];
  dep_wait();
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = A.conv[x + (size_t)(j + T * m) * N];
  fft_regs<N, CB, BS, true>(v, W, j, s, CtaSync{});
  if (fft_odd_exchanges(N)) __syncthreads();
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = make_float2(v[m].x * msk[m], v[m].y * msk[m]);
  fft_regs<N, CB, BS, false>(v, W, j, s, CtaSync{});
#pragma unroll
  for (int m = 0; m < 8; ++m) A.conv[x + (size_t)(j + T * m) * N] = v[m];
}

// 5. a few rows per CTA (a multiple of nrebin): forward transform along x, real part,
//    binning (pyr_bimg_krnl order: x offset outer, y offset inner, then / nrebin^2)
//    and the row sums of the binned image for the normalisation.
template <int N>
__global__ void __launch_bounds__(PYR_THREADS) pyr_bin_kernel(PyrArgs A, int rows) {
  extern __shared__ float2 sm[];
  constexpr int T = N / 8, BS = fft_smem_elems(N);
  const int g = threadIdx.x / T, j = threadIdx.x % T, G = blockDim.x / T;
  const GroupSync<T> sync{g};
  float2 *s = sm + g * 2 * BS;
  float *real = reinterpret_cast<float *>(sm + G * 2 * BS);  // rows x N
  const int y0 = blockIdx.x * rows;
  FftTw<N> W;
  dep_launch();
  W.load(A.tw, j);
  dep_wait();
  for (int r = g; r < rows; r += G) {  // rows is a multiple of G
    float2 v[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = A.conv[(size_t)(y0 + r) * N + j + T * m];
    fft_regs<N, 1, BS, false>(v, W, j, s, sync);
    if (fft_odd_exchanges(N)) sync();
#pragma unroll
    for (int m = 0; m < 8; ++m) real[r * N + j + T * m] = v[m].x;
  }
  __syncthreads();
  const int nbr = rows / A.nrebin;
  const float div = (float)(A.nrebin * A.nrebin);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int br = threadIdx.x >> 5; br < nbr; br += nw) {  // a warp per binned row
    float sum = 0.f;
    for (int bx = lane; bx < A.nb; bx += 32) {
      float o = 0.f;
      for (int ii = 0; ii < A.nrebin; ++ii)
        for (int jj = 0; jj < A.nrebin; ++jj) o = o + real[(br * A.nrebin + jj) * N + bx * A.nrebin + ii];
      o = o / div;
      A.binimg[(size_t)(blockIdx.x * nbr + br) * A.nb + bx] = o;
      sum += o;
    }
    sum = warp_sum(sum);
    if (lane == 0) A.partial[blockIdx.x * nbr + br] = sum;
  }
}

// 6. normalisation to nphot (sum of the row sums in row order) and noise.
__global__ void pyr_norm_noise_kernel(float *binimg, const float *partial, int nb, float nphot, int noise_mode,
                                      float noise, uint32_t frame, uint32_t k0, uint32_t k1) {
  dep_sync();
  __shared__ float s_fact;
  __shared__ float rk[AOB_POISSON_INV_KMAX + 1];
  if (noise_mode >= 1)
    for (int i = threadIdx.x; i <= AOB_POISSON_INV_KMAX; i += blockDim.x) rk[i] = i ? __frcp_rn((float)i) : 0.f;
  if (threadIdx.x < 32) {
    // the row sums in a fixed order: lane-strided partial sums, then a butterfly
    float s = 0.f;
    for (int r = threadIdx.x; r < nb; r += 32) s += partial[r];
    s = warp_sum(s);
    if (threadIdx.x == 0) s_fact = nphot / s;
  }
  __syncthreads();
  const float fact = s_fact;
  const int n2 = nb * nb;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
    float v = binimg[i] * fact;
    if (noise_mode >= 1) {
      const U4 w0 = philox4x32_10(U4{(uint32_t)i, frame, TAG_POISSON, 0u}, k0, k1);
      v = v < AOB_POISSON_INV_MAX_MEAN ? poisson_inversion(v, w0, rk) : poisson_ptrs(v, w0, (uint32_t)i, frame, k0, k1);
      if (noise_mode >= 2) v = v + noise * gauss_sample(w0);
    }
    binimg[i] = v;
  }
}

// focal plane: the per-point images summed in point order from zero, as the
// reference accumulates d_pyrfocalplane (sutra_wfs_pyr_pyrhr.cpp:398-401,501-506)
__global__ void pyr_focal_sum_kernel(float *focal, const float *work, int npts, int64_t n2) {
  dep_sync();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n2; i += (int64_t)gridDim.x * blockDim.x) {
    float acc = 0.f;
    for (int p = 0; p < npts; ++p) acc += work[(size_t)p * n2 + i];
    focal[i] = acc;
  }
}

template <class K>
static void pyr_smem(K kern, size_t bytes) {
  smem_opt_in(reinterpret_cast<const void *>(kern), (int)std::max<size_t>(bytes, 48 * 1024));
}

template <int N>
static void pyr_launch(const PyrArgs &A, int device, cudaStream_t s) {
  constexpr int T = N / 8, BS = fft_smem_elems(N);
  const int nsm = num_sms(device);
  {
    constexpr int SEQ = PYR_ROW_THREADS / T;
    launch_after(pyr_rows_kernel<N>, (A.npts * A.ntot + SEQ - 1) / SEQ, PYR_ROW_THREADS, 0, s, A);
    AOB_LAUNCH_CHECK("pyr_rows_kernel");
  }
  {
    constexpr int CB = pyr_cols(N), threads = T * CB, groups = N / CB;
    const size_t sm = sizeof(float2) * 2 * BS * CB;
    auto kern = A.focal_work ? pyr_cols_kernel<N, true> : pyr_cols_kernel<N, false>;
    pyr_smem(kern, sm);
    const int slots = nsm * std::max(1, 512 / threads);
    const int grid = (int)std::min<int64_t>(slots, (int64_t)groups * A.npts);
    launch_after(kern, grid, threads, sm, s, A);
    AOB_LAUNCH_CHECK("pyr_cols_kernel");
  }
  {
    // groups of threads per row: one per point, in whole warps, up to PYR_ACC_THREADS
    const int unit = T < 32 ? 32 / T : 1;
    const int G = std::min(PYR_ACC_THREADS / T, (A.npts + unit - 1) / unit * unit);
    const size_t sm = std::max(sizeof(float2) * 2 * BS * G, sizeof(float) * N * G);
    pyr_smem(pyr_accum_kernel<N>, sm);
    launch_after(pyr_accum_kernel<N>, N, G * T, sm, s, A);
    AOB_LAUNCH_CHECK("pyr_accum_kernel");
  }
  {
    constexpr int CB = pyr_conv_cols(N);
    const size_t sm = sizeof(float2) * 2 * BS * CB;
    pyr_smem(pyr_conv_cols_kernel<N>, sm);
    launch_after(pyr_conv_cols_kernel<N>, N / CB, T * CB, sm, s, A);
    AOB_LAUNCH_CHECK("pyr_conv_cols_kernel");
  }
  {
    // as few rows per CTA as the binning and a whole warp allow (a power of two)
    const int rows = std::max({A.nrebin, 2, 32 / T});
    const int G = std::min(rows, PYR_THREADS / T);
    const size_t sm = sizeof(float2) * 2 * BS * G + sizeof(float) * N * rows;
    pyr_smem(pyr_bin_kernel<N>, sm);
    launch_after(pyr_bin_kernel<N>, N / rows, G * T, sm, s, A, rows);
    AOB_LAUNCH_CHECK("pyr_bin_kernel");
  }
}

}  // namespace aob

using namespace aob;

aob_pyr::aob_pyr(int device_, int nxsub_, int nvalid_, int npix_, int nphase_, int nrebin_, int nfft_, int ntot_,
                 int npts_, float pdiam_, float nphot_, float nphot4imat_)
    : device(device_), nxsub(nxsub_), nvalid(nvalid_), npix(npix_), nphase(nphase_), nrebin(nrebin_), nfft(nfft_),
      ntot(ntot_), npts(npts_), pdiam(pdiam_), nphot(nphot_), nphot4imat(nphot4imat_) {
  AOB_REQUIRE(nvalid > 0 && nrebin > 0 && ntot > 0 && npts > 0, "pyr: sizes must be > 0");
  AOB_REQUIRE(nfft >= 64 && nfft <= 2048 && (nfft & (nfft - 1)) == 0,
              "pyr: nfft must be a power of two in [64, 2048]");
  AOB_REQUIRE(nrebin <= PYR_MAX_REBIN && (nrebin & (nrebin - 1)) == 0,
              "pyr: nrebin must be a power of two <= 8 (the binning rows tile nfft)");
  AOB_REQUIRE(ntot <= nfft, "pyr: the phase grid (ntot) must fit in nfft");
  AOB_REQUIRE(nfft % nrebin == 0, "pyr: nfft must be a multiple of nrebin");
  while ((1 << logn) < nfft) ++logn;
  AOB_CUDA(cudaSetDevice(device));
  phase.alloc((int64_t)ntot * ntot);
  pupil.alloc((int64_t)ntot * ntot);
  const int64_t n2 = (int64_t)nfft * nfft;
  submask.alloc(n2);
  sincar.alloc(n2);
  phalfxy.alloc(n2);
  conv.alloc(n2);
  hrimg.alloc(n2);
  binimg.alloc((int64_t)nbin() * nbin());
  partial.alloc(nbin());
  validsubsx.alloc(4 * (int64_t)nvalid);
  validsubsy.alloc(4 * (int64_t)nvalid);
  fluxPerSub.alloc(nvalid);
}

void aob_pyr::set_modulation(const float *h_cx, const float *h_cy, const float *h_w, int n) {
  AOB_REQUIRE(h_cx && h_cy && n > 0, "pyr.set_modulation: null points");
  AOB_CUDA(cudaSetDevice(device));
  npts = n;
  cx.alloc(n);
  cy.alloc(n);
  weights.alloc(n);
  cx.upload(h_cx, n);
  cy.upload(h_cy, n);
  std::vector<float> one(n, 1.f);
  weights.upload(h_w ? h_w : one.data(), n);
  work.alloc((int64_t)npts * nfft * nfft);
}

void aob_pyr::load_arrays(const float2 *h_halfxy, const float *h_cx, const float *h_cy, const float *h_w,
                          const float *h_sincar, const float *h_submask, const int32_t *h_vsx, const int32_t *h_vsy,
                          const float *h_flux) {
  AOB_REQUIRE(h_halfxy && h_sincar && h_submask && h_vsx && h_vsy, "pyr.load_arrays: a required array is NULL");
  const int nb = nbin();
  for (int i = 0; i < 4 * nvalid; ++i)
    AOB_REQUIRE(h_vsx[i] >= 0 && h_vsx[i] < nb && h_vsy[i] >= 0 && h_vsy[i] < nb,
                "pyr.load_arrays: valid pixel outside the binned image");
  set_modulation(h_cx, h_cy, h_w, npts);
  const int64_t n2 = (int64_t)nfft * nfft;
  phalfxy.upload(h_halfxy, n2);
  sincar.upload(h_sincar, n2);
  submask.upload(h_submask, n2);
  validsubsx.upload(h_vsx, 4 * (int64_t)nvalid);
  validsubsy.upload(h_vsy, 4 * (int64_t)nvalid);
  if (h_flux) fluxPerSub.upload(h_flux, nvalid);
  loaded = true;
}

void aob_pyr::comp_image(bool with_noise, cudaStream_t s) {
  AOB_REQUIRE(loaded, "pyr.comp_image: load_arrays has not been called");
  AOB_CUDA(cudaSetDevice(device));
  PyrArgs A{};
  A.ntot = ntot;
  A.off = (int)((nfft - ntot) / 2.0f);
  A.npts = npts;
  A.phase = phase.p;
  A.pupil = pupil.p;
  A.mic2rad = 2.0f * (float)M_PI / lambda_um;
  A.cx = cx.p;
  A.cy = cy.p;
  A.w = weights.p;
  A.submask = submask.p;
  A.phalfxy = phalfxy.p;
  A.sincar = sincar.p;
  A.early = !tables_out;
  A.tw = fft_twiddles(device, nfft);
  A.work = work.p;
  A.conv = conv.p;
  A.hrimg = hrimg.p;
  A.binimg = binimg.p;
  A.partial = partial.p;
  A.nrebin = nrebin;
  A.nb = nbin();
  const int64_t n2 = (int64_t)nfft * nfft;
  A.focal_work = nullptr;
  if (compute_focalplane) {
    if (focal_work.n != npts * n2) focal_work.alloc(npts * n2);
    if (focalplane.n != n2) focalplane.alloc(n2);
    A.focal_work = focal_work.p;
  }
  switch (nfft) {
    case 64: pyr_launch<64>(A, device, s); break;
    case 128: pyr_launch<128>(A, device, s); break;
    case 256: pyr_launch<256>(A, device, s); break;
    case 512: pyr_launch<512>(A, device, s); break;
    case 1024: pyr_launch<1024>(A, device, s); break;
    default: pyr_launch<2048>(A, device, s); break;
  }
  if (compute_focalplane) {
    launch_after(pyr_focal_sum_kernel, (int)std::min<int64_t>((n2 + 255) / 256, 8 * num_sms(device)), 256, 0, s,
        focalplane.p, focal_work.p, npts, n2);
    AOB_LAUNCH_CHECK("pyr_focal_sum_kernel");
  }
  const float nz = with_noise ? noise : -1.f;
  const int noise_mode = nz > 0 ? 2 : (nz > -1 ? 1 : 0);
  const int nb2 = nbin() * nbin();
  launch_after(pyr_norm_noise_kernel, std::min((nb2 + 255) / 256, 4 * num_sms(device)), 256, 0, s,
      binimg.p, partial.p, nbin(), nphot, noise_mode, nz, (uint32_t)frame, (uint32_t)((uint64_t)seed & 0xffffffffu),
      (uint32_t)((uint64_t)seed >> 32));
  AOB_LAUNCH_CHECK("pyr_norm_noise_kernel");
  if (noise_mode) ++frame;
  ++image_gen;
}
