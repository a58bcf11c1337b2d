// Batched complex 2-D FFT for power-of-two sizes (8 .. 2048), single
// precision, in place.  Used for the target PSF and the SH field stop.
//
// Row pass: T = N / 8 threads per row, 256 threads per CTA; column pass: up to 8
// adjacent columns per CTA (64-byte row segments).  Both hold the transform
// in registers (fft.cuh) and read and write global memory once.  Twiddles come
// from a table computed in double on the host.  Sign convention of cuFFT: forward
// = exp(-2 pi i k m / n), inverse = exp(+2 pi i k m / n), both unnormalised.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "aob_objects.hpp"
#include "fft.cuh"

namespace aob {

namespace {
struct TwiddleKey {
  int device, n;
  bool operator<(const TwiddleKey &o) const { return device != o.device ? device < o.device : n < o.n; }
};
std::map<TwiddleKey, DevBuf<float2> *> g_tw;
std::mutex g_tw_mu;
}  // namespace

const float2 *fft_twiddles(int device, int n) {
  std::lock_guard<std::mutex> lk(g_tw_mu);
  auto it = g_tw.find({device, n});
  if (it != g_tw.end()) return it->second->p;
  std::vector<float2> h(n / 2);
  for (int m = 0; m < n / 2; ++m) {
    const double a = 2.0 * M_PI * (double)m / (double)n;
    h[m] = make_float2((float)std::cos(a), (float)-std::sin(a));  // forward twiddles
  }
  auto *b = new DevBuf<float2>(n / 2);
  b->upload(h.data(), n / 2);
  g_tw[{device, n}] = b;  // kept for the lifetime of the process
  return b->p;
}

constexpr int FFT_ROW_THREADS = 256;

template <int N, bool INV>
__global__ void __launch_bounds__(FFT_ROW_THREADS) fft_rows_kernel(float2 *data, int64_t nrows, const float2 *tw) {
  constexpr int T = N / 8, SEQ = FFT_ROW_THREADS / T, BS = fft_smem_elems(N);
  __shared__ float2 s[BS > 0 ? SEQ * 2 * BS : 1];
  const int g = threadIdx.x / T, j = threadIdx.x % T;
  const int64_t r = (int64_t)blockIdx.x * SEQ + g;
  float2 *row = data + r * N;
  float2 v[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = r < nrows ? row[j + T * m] : make_float2(0.f, 0.f);
  FftTw<N> W;
  W.load(tw, j);
  fft_regs<N, 1, BS, INV>(v, W, j, s + g * 2 * BS, GroupSync<T>{g});
  if (r < nrows) {
#pragma unroll
    for (int m = 0; m < 8; ++m) row[j + T * m] = v[m];
  }
}

// columns per CTA: 8, fewer where 8 would pass 512 threads
constexpr int fft_cols(int n) { return n <= 512 ? 8 : 4096 / n; }

template <int N, bool INV>
__global__ void __launch_bounds__(N / 8 * fft_cols(N)) fft_cols_kernel(float2 *data, const float2 *tw) {
  extern __shared__ float2 scol[];
  constexpr int T = N / 8, CB = fft_cols(N), BS = fft_smem_elems(N) * CB;
  constexpr int groups = N / CB;
  const int img = blockIdx.x / groups;
  const int c = threadIdx.x % CB, j = threadIdx.x / CB;
  float2 *base = data + (size_t)img * N * N + (blockIdx.x - img * groups) * CB + c;
  float2 v[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = base[(size_t)(j + T * m) * N];
  FftTw<N> W;
  W.load(tw, j);
  fft_regs<N, CB, BS, INV>(v, W, j, scol + c, CtaSync{});
#pragma unroll
  for (int m = 0; m < 8; ++m) base[(size_t)(j + T * m) * N] = v[m];
}

template <int N, bool INV>
static void fft2d_n(float2 *data, int batch, const float2 *tw, cudaStream_t s) {
  constexpr int SEQ = FFT_ROW_THREADS / (N / 8);
  const int64_t nrows = (int64_t)N * batch;
  fft_rows_kernel<N, INV><<<(unsigned)((nrows + SEQ - 1) / SEQ), FFT_ROW_THREADS, 0, s>>>(data, nrows, tw);
  AOB_LAUNCH_CHECK("fft_rows_kernel");
  constexpr int sm = (int)sizeof(float2) * 2 * fft_smem_elems(N) * fft_cols(N);
  smem_opt_in(reinterpret_cast<const void *>(fft_cols_kernel<N, INV>), std::max(sm, 48 * 1024));
  fft_cols_kernel<N, INV><<<(unsigned)(N / fft_cols(N) * batch), N / 8 * fft_cols(N), sm, s>>>(data, tw);
  AOB_LAUNCH_CHECK("fft_cols_kernel");
}

void fft2d(float2 *data, int n, int batch, bool inverse, int device, cudaStream_t s) {
  AOB_REQUIRE(n >= 8 && n <= 2048 && (n & (n - 1)) == 0, "fft2d: n must be a power of two in [8, 2048]");
  const float2 *tw = fft_twiddles(device, n);
  auto go = [&](auto size) {
    constexpr int N = decltype(size)::value;
    inverse ? fft2d_n<N, true>(data, batch, tw, s) : fft2d_n<N, false>(data, batch, tw, s);
  };
  switch (n) {
    case 8: go(std::integral_constant<int, 8>{}); break;
    case 16: go(std::integral_constant<int, 16>{}); break;
    case 32: go(std::integral_constant<int, 32>{}); break;
    case 64: go(std::integral_constant<int, 64>{}); break;
    case 128: go(std::integral_constant<int, 128>{}); break;
    case 256: go(std::integral_constant<int, 256>{}); break;
    case 512: go(std::integral_constant<int, 512>{}); break;
    case 1024: go(std::integral_constant<int, 1024>{}); break;
    default: go(std::integral_constant<int, 2048>{}); break;
  }
}

}  // namespace aob

extern "C" int aob_fft2d_c64(void *data, int n, int batch, int inverse, int device, void *stream) {
  try {
    if (!data) throw aob::Error("aob_fft2d_c64: null data");
    AOB_CUDA(cudaSetDevice(device));
    aob::fft2d(static_cast<float2 *>(data), n, batch, inverse != 0, device, reinterpret_cast<cudaStream_t>(stream));
    return AOB_OK;
  } catch (const std::exception &e) {
    aob::set_last_error(e.what());
    return AOB_ERR;
  }
}
