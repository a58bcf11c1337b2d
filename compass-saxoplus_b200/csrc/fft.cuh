// Complex FFTs held in registers (device code) and the batched in-place 2-D
// transform (fft.cu).
#pragma once

#include <cuda_runtime.h>

namespace aob {

// ---------------------------------------------------------------------------
// A length-N transform (N a power of two, 8 .. 2048) by a group of T = N / 8
// threads, thread j holding elements j + T m in v[m] (m < 8), natural order in
// and out: Stockham radix-8 passes, a last radix-2 or radix-4 pass when N is not
// a power of 8 (Govindaraju et al., "High performance discrete Fourier transforms
// on graphics processors", SC'08).  The first pass's inputs and the last pass's
// outputs are the thread's own elements, so a transform touches shared memory
// only between passes (twice for N = 512) and global memory is read and
// written straight from registers, T consecutive elements at a time.
//   pass with sub-transform length NS: butterfly j takes elements j + r N / R,
//   multiplies by W_(NS R)^(r (j mod NS)) and gives (j / NS) NS R + j mod NS + r NS.
// cuFFT sign convention (forward exp(-2 pi i k m / N)), unnormalised.

__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * w, or a * conj(w) for the inverse transform
template <bool INV>
__device__ __forceinline__ float2 c_mulw(float2 a, float2 w) {
  return INV ? make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y)
             : make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 c_rot(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft2(float2 &a, float2 &b) {
  const float2 t = a;
  a = c_add(t, b);
  b = c_sub(t, b);
}
template <bool INV>
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c, float2 &d) {
  const float2 t0 = c_add(a, c), t1 = c_sub(a, c);
  const float2 t2 = c_add(b, d), t3 = c_rot<INV>(c_sub(b, d));
  a = c_add(t0, t2);
  c = c_sub(t0, t2);
  b = c_add(t1, t3);
  d = c_sub(t1, t3);
}
template <bool INV>
__device__ __forceinline__ void dft8(float2 (&v)[8]) {
  dft4<INV>(v[0], v[2], v[4], v[6]);
  dft4<INV>(v[1], v[3], v[5], v[7]);
  const float h = 0.70710678118654752f;  // cos(pi / 4)
  const float sg = INV ? 1.f : -1.f;
  // odd outputs times W8^k: W8 = exp(-/+ i pi / 4)
  const float2 o1 = make_float2(h * (v[3].x - sg * v[3].y), h * (v[3].y + sg * v[3].x));
  const float2 o2 = c_rot<INV>(v[5]);
  const float2 o3 = make_float2(h * (-v[7].x - sg * v[7].y), h * (-v[7].y + sg * v[7].x));
  const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
  v[0] = c_add(e0, o0);
  v[4] = c_sub(e0, o0);
  v[1] = c_add(e1, o1);
  v[5] = c_sub(e1, o1);
  v[2] = c_add(e2, o2);
  v[6] = c_sub(e2, o2);
  v[3] = c_add(e3, o3);
  v[7] = c_sub(e3, o3);
}

constexpr int fft_passes(int n) { return n <= 8 ? 1 : (n <= 64 ? 2 : (n <= 512 ? 3 : 4)); }
// Padded position of element i in shared memory: one slot skipped every eight, so
// that the strided writes after a radix-8 pass fall on different banks.
__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 3); }
constexpr int fft_smem_elems(int n) { return n > 8 ? n + n / 8 : 0; }  // per sequence and buffer

// The twiddles of thread j's butterflies in the passes after the first, read once
// from the table tw (exp(-2 pi i m / N), m < N / 2) and kept in registers.
template <int N>
struct FftTw {
  static constexpr int P = fft_passes(N) - 1;
  float2 w[P > 0 ? 7 * P : 1];
  static __device__ __forceinline__ float2 at(const float2 *tw, int m) {
    float2 r = __ldg(tw + (m & (N / 2 - 1)));
    if (m >= N / 2) r = make_float2(-r.x, -r.y);
    return r;
  }
  template <int NS, int I>
  __device__ __forceinline__ void fill(const float2 *tw, int j) {
    if constexpr (NS < N) {
      constexpr int R = NS * 8 <= N ? 8 : N / NS;
      if constexpr (R == 8) {
        const int k = j & (NS - 1);
#pragma unroll
        for (int r = 1; r < 8; ++r) w[7 * I + r - 1] = at(tw, r * k * (N / (NS * 8)));
      } else {  // NS R = N: butterflies j + q T, exponent r (j + q T)
#pragma unroll
        for (int q = 0; q < 8 / R; ++q)
#pragma unroll
          for (int r = 1; r < R; ++r) w[7 * I + q * (R - 1) + r - 1] = at(tw, r * (j + q * (N / 8)));
      }
      fill<NS * 8, I + 1>(tw, j);
    }
  }
  __device__ __forceinline__ void load(const float2 *tw, int j) { fill<8, 0>(tw, j); }
};

// The passes after the first.  s: this sequence's exchange buffers (two, fft_smem_elems
// long, element i at s[fft_pad(i) * CS], the second BS floats2 behind the first); sync():
// barrier over the threads that share them.
template <int N, int CS, int BS, bool INV, int NS, int I, class Sync>
__device__ __forceinline__ void fft_tail(float2 (&v)[8], const FftTw<N> &W, int j, float2 *s, const Sync &sync) {
  if constexpr (NS < N) {
    constexpr int T = N / 8, PS = NS / 8;  // PS: sub-transform length of the pass before
    constexpr int R = NS * 8 <= N ? 8 : N / NS;
    float2 *b = s + (I & 1) * BS;
    const int k = j & (PS - 1);
    const int d = (j - k) * 8 + k;
#pragma unroll
    for (int r = 0; r < 8; ++r) b[fft_pad(d + r * PS) * CS] = v[r];
    sync();
#pragma unroll
    for (int m = 0; m < 8; ++m) v[m] = b[fft_pad(j + T * m) * CS];
    if constexpr (R == 8) {
#pragma unroll
      for (int r = 1; r < 8; ++r) v[r] = c_mulw<INV>(v[r], W.w[7 * I + r - 1]);
      dft8<INV>(v);
    } else if constexpr (R == 4) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int r = 1; r < 4; ++r) v[q + 2 * r] = c_mulw<INV>(v[q + 2 * r], W.w[7 * I + q * 3 + r - 1]);
        dft4<INV>(v[q], v[q + 2], v[q + 4], v[q + 6]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q + 4] = c_mulw<INV>(v[q + 4], W.w[7 * I + q]);
        dft2<INV>(v[q], v[q + 4]);
      }
    }
    fft_tail<N, CS, BS, INV, NS * 8, I + 1>(v, W, j, s, sync);
  }
}

// One transform.  Exchanges alternate between the two buffers, one barrier each: a
// buffer is written again only after a barrier that followed its last reads.  That
// also holds from one transform to the next when their number is even; after an odd
// number (fft_odd_exchanges) the caller synchronises before the next transform.
template <int N, int CS, int BS, bool INV, class Sync>
__device__ __forceinline__ void fft_regs(float2 (&v)[8], const FftTw<N> &W, int j, float2 *s, const Sync &sync) {
  dft8<INV>(v);
  fft_tail<N, CS, BS, INV, 8, 0>(v, W, j, s, sync);
}
constexpr bool fft_odd_exchanges(int n) { return ((fft_passes(n) - 1) & 1) != 0; }

// Barrier over one group of T consecutive threads of the CTA (a warp or less: the
// warp; more: named barrier 1 + group; a CTA has at most 15 such groups).
template <int T>
struct GroupSync {
  int group;
  __device__ __forceinline__ void operator()() const {
    if constexpr (T <= 32)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(T) : "memory");
  }
};
struct CtaSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// n x n transforms of ``batch`` contiguous images (x fastest), in place.
void fft2d(float2 *data, int n, int batch, bool inverse, int device, cudaStream_t s);
const float2 *fft_twiddles(int device, int n);
}  // namespace aob
