// Interaction matrix of a DM seen by a SH sensor, every actuator poked in one
// batch.
//
// The reference's SutraRtc::do_imat (libsutra/src.cpp/sutra_rtc.cpp:150-292)
// loops over the actuators: comp_oneactu (push), raytrace to the sensor,
// comp_image, do_centroids, then the same with the pull, and the column
// (s_push - s_pull) / (2 push).
//
// A poke moves only the sub-apertures whose phase window meets the actuator's
// influence patch: at 40 x 40 sub-apertures and 41 x 41 actuators about 32 of
// 1248.  The others see a flat phase on the push and on the pull, so their
// entries are the difference of a slope from itself.  One CTA takes one
// actuator: it lists the sub-apertures that the patch reaches, writes the
// entries of all the others, and forms the push and pull images of the listed
// ones (the stages of sh_core.cuh) with the phase evaluated from the patch
// where it is needed, so neither DM shapes, phases nor slopes go through
// memory.  Every value has the arithmetic of the corresponding separate call,
// so the matrix equals the poke-by-poke one bit for bit.
//
// Bound: issue of the sensor stages (about 86,000 images at that size).  One call
// takes 0.245 ms (B200, warm); forming all 3.4 M images from DM shapes and phases
// in memory took 22 ms (14.7 ms images, 2.8 ms shapes, 0.65 ms tracing, the rest
// 1.5 GB of scratch).

#include <algorithm>

#include "aob_objects.hpp"
#include "sh_core.cuh"
#include "sim.hpp"

namespace aob {

constexpr int IMAT_THREADS = 256;
constexpr int IMAT_LIST = 512;  // sub-apertures of one actuator listed at a time
// images per batch, at most: 51 KB of shared memory at 40 x 40 (the registers, 80 a thread, allow
// three CTAs on an SM)
constexpr int IMAT_ITEMS = 16;

struct ImatArgs {
  const float *influ;
  const int32_t *i1, *j1;
  int isz, dim;
  float xoff, yoff, push;
  const float *flat;  // slopes of the flat phase (2 nvalid, the sensor's order)
  float *imat;        // nslope x nact, column-major
};

// Items 2 j (push) and 2 j + 1 (pull) of listed sub-aperture j; a < 0: every item
// is a sub-aperture of its own under a flat phase.
struct ImatSource {
  static constexpr bool LISTED = true;
  const ImatArgs &A;
  const int *list;
  float2 *slopes;
  int a, npup, first;  // first: item of the batch's s = 0
  int i1, j1;
  __device__ int sub(int s) const { return list[a < 0 ? first + s : (first + s) >> 1]; }
  // the DM screen with actuator a's command only: dm_shape_kernel's 0 + com * influ
  __device__ float screen(int x, int y, float com) const {
    const int u = x - i1, v = y - j1;
    const bool in = u >= 0 && u < A.isz && v >= 0 && v < A.isz && x < A.dim && y < A.dim;
    return in ? com * __ldg(A.influ + u + v * A.isz + (size_t)a * A.isz * A.isz) : 0.f;
  }
  __device__ float phase(int s, int X, int Y) const {
    if (a < 0) return 0.f;
    const float xref = ray_position(X, npup, A.xoff), yref = ray_position(Y, npup, A.yoff);
    const int i = (int)xref, j = (int)yref;
    float acc = 0.f;
    if (i >= 0 && j >= 0 && i + 1 < A.dim && j + 1 < A.dim) {
      const float com = ((first + s) & 1) ? -A.push : A.push;
      acc += ray_bilinear(xref - i, yref - j, screen(i, j, com), screen(i + 1, j, com), screen(i, j + 1, com),
                          screen(i + 1, j + 1, com));
    }
    return acc;
  }
  __device__ void store(int s, float x, float y) const { slopes[first + s] = make_float2(x, y); }
  // whether the phase window [x0, x0 + pd) x [y0, y0 + pd) reads the patch
  __device__ bool reaches(int x0, int y0, int pd) const {
    auto at = [](int i, int n, float off) { return (int)ray_position(i, n, off); };
    return at(x0 + pd - 1, npup, A.xoff) >= i1 - 1 && at(x0, npup, A.xoff) <= i1 + A.isz - 1 &&
           at(y0 + pd - 1, npup, A.yoff) >= j1 - 1 && at(y0, npup, A.yoff) <= j1 + A.isz - 1;
  }
};

// shared memory behind the sensor's tables and work area: the list, then two slopes per entry
constexpr size_t IMAT_LIST_BYTES = IMAT_LIST * (sizeof(int) + 2 * sizeof(float2));

template <int NFFT, int PD>
__device__ __forceinline__ void imat_images(const ShKernelArgs &P, ImatSource &src, int nitems, int S,
                                            unsigned char *smem, const ShSmem &L) {
  const Team T{(int)threadIdx.x, (int)blockDim.x, 0};
  for (int f = 0; f < nitems; f += S) {
    src.first = f;
    sh_batch<NFFT, PD, TEAM_CTA, NoHook, false, false, ImatSource>(P, 0, 1, min(S, nitems - f), smem, smem + L.hdr, L,
                                                                   T, NoHook{}, src);
  }
}

// The slopes of the flat phase, sub-apertures blockIdx.x * IMAT_ITEMS and on.
template <int NFFT, int PD>
__global__ void __launch_bounds__(IMAT_THREADS) imat_flat_kernel(ShKernelArgs P, ImatArgs A, int S, float *flat) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int pd = PD > 0 ? PD : P.pdiam;
  const ShSmem L(NFFT, P.nu, P.nv, pd, P.nrebin2 * P.npix * P.npix, P.npix * P.npix, S);
  float2 *slopes = reinterpret_cast<float2 *>(smem + ShSmem::align16(L.bytes()));
  int *list = reinterpret_cast<int *>(slopes + 2 * IMAT_LIST);
  sh_load_tables<NFFT>(P, smem, threadIdx.x, blockDim.x);
  const int k0 = blockIdx.x * IMAT_ITEMS, n = min(IMAT_ITEMS, P.nvalid - k0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) list[i] = k0 + i;
  __syncthreads();
  ImatSource src{A, list, slopes, -1, P.npup, 0, 0, 0};
  imat_images<NFFT, PD>(P, src, n, S, smem, L);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int k = k0 + i;
    flat[P.c_order ? 2 * k : k] = slopes[i].x;
    flat[P.c_order ? 2 * k + 1 : k + P.nvalid] = slopes[i].y;
  }
}

template <int NFFT, int PD>
__global__ void __launch_bounds__(IMAT_THREADS) imat_kernel(ShKernelArgs P, ImatArgs A, int S) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_n;
  const int pd = PD > 0 ? PD : P.pdiam;
  const ShSmem L(NFFT, P.nu, P.nv, pd, P.nrebin2 * P.npix * P.npix, P.npix * P.npix, S);
  float2 *slopes = reinterpret_cast<float2 *>(smem + ShSmem::align16(L.bytes()));
  int *list = reinterpret_cast<int *>(slopes + 2 * IMAT_LIST);
  sh_load_tables<NFFT>(P, smem, threadIdx.x, blockDim.x);
  const int a = blockIdx.x;
  ImatSource src{A, list, slopes, a, P.npup, 0, __ldg(A.i1 + a), __ldg(A.j1 + a)};
  const int nvalid = P.nvalid;
  float *col = A.imat + (int64_t)a * 2 * nvalid;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  // s_n only hands out places in the list; how many there are, each thread counts for
  // itself from the barrier's sum, so that every thread comes to the same decision
  // whatever the other warps have gone on to append.
  int n = 0;
  for (int base = 0; base < nvalid; base += IMAT_THREADS) {
    const int k = base + (int)threadIdx.x;
    bool reached = false;
    if (k < nvalid) {
      reached = src.reaches(__ldg(P.puppixx + k), __ldg(P.puppixy + k), pd);
      if (reached) {
        list[atomicAdd(&s_n, 1)] = k;  // (the order within the list does not matter to any value)
      } else {
        const int ix = P.c_order ? 2 * k : k, iy = P.c_order ? 2 * k + 1 : k + nvalid;
        const float fx = __ldg(A.flat + ix), fy = __ldg(A.flat + iy);
        col[ix] = (fx - fx) / (2.f * A.push);
        col[iy] = (fy - fy) / (2.f * A.push);
      }
    }
    n += __syncthreads_count(reached);
    if (n + IMAT_THREADS > IMAT_LIST || base + IMAT_THREADS >= nvalid) {
      imat_images<NFFT, PD>(P, src, 2 * n, S, smem, L);
      for (int j = threadIdx.x; j < n; j += IMAT_THREADS) {
        const int m = list[j];
        const float2 sp = slopes[2 * j], sm = slopes[2 * j + 1];
        col[P.c_order ? 2 * m : m] = (sp.x - sm.x) / (2.f * A.push);
        col[P.c_order ? 2 * m + 1 : m + nvalid] = (sp.y - sm.y) / (2.f * A.push);
      }
      n = 0;
      if (threadIdx.x == 0) s_n = 0;
      __syncthreads();
    }
  }
}

template <int NFFT, int PD>
static void launch_imat(const ShKernelArgs &P, const ImatArgs &A, int nact, int S, size_t sm, float *flat,
                        cudaStream_t s) {
  const int lim = (int)std::max<size_t>(sm, 48 * 1024);
  smem_opt_in(reinterpret_cast<const void *>(imat_flat_kernel<NFFT, PD>), lim);
  smem_opt_in(reinterpret_cast<const void *>(imat_kernel<NFFT, PD>), lim);
  imat_flat_kernel<NFFT, PD><<<(P.nvalid + IMAT_ITEMS - 1) / IMAT_ITEMS, IMAT_THREADS, sm, s>>>(P, A, S, flat);
  AOB_LAUNCH_CHECK("imat_flat_kernel");
  imat_kernel<NFFT, PD><<<nact, IMAT_THREADS, sm, s>>>(P, A, S);
  AOB_LAUNCH_CHECK("imat_kernel");
}
template <int NFFT>
static void launch_imat_pd(const ShKernelArgs &P, const ImatArgs &A, int nact, int S, size_t sm, float *flat,
                           cudaStream_t s) {
  switch (P.pdiam) {
    case 4: launch_imat<NFFT, 4>(P, A, nact, S, sm, flat, s); break;
    case 6: launch_imat<NFFT, 6>(P, A, nact, S, sm, flat, s); break;
    case 8: launch_imat<NFFT, 8>(P, A, nact, S, sm, flat, s); break;
    default: launch_imat<NFFT, 0>(P, A, nact, S, sm, flat, s); break;
  }
}

}  // namespace aob

using namespace aob;

extern "C" int aob_imat_build(aob_sh *w, aob_centro *c, aob_dm *dm, float xoff, float yoff, float push, int chunk,
                              float *dev_imat, void *stream) {
  try {
    if (!w || !c || !dm || !dev_imat) throw Error("aob_imat_build: null handle or pointer");
    AOB_REQUIRE(w->device == c->device && w->device == dm->device, "aob_imat_build: objects on different devices");
    AOB_REQUIRE(push != 0.f, "aob_imat_build: push must be non-zero");
    AOB_REQUIRE(!w->fs_n, "aob_imat_build: sensors with a field stop are not supported");
    AOB_CUDA(cudaSetDevice(w->device));
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    ShKernelArgs P;
    aob_centro *fc = w->make_args(false, nullptr, nullptr, P);
    AOB_REQUIRE(fc == c, "aob_imat_build: attach the CoG-family centroider to the sensor first");
    // the reference forms the calibration images with nphot4imat photons
    // (SutraRtc::comp_images_imat, sutra_rtc.cpp:380-395); 0 keeps nphot
    if (w->nphot4imat > 0.f) P.nphot = w->nphot4imat;
    const int nact = dm->nact;
    // (chunk is a limit on the scratch that earlier forms needed; only its check is left)
    AOB_REQUIRE((chunk > 0 ? std::min(chunk, nact) : nact) <= 32767,
                "aob_imat_build: at most 32767 actuators per chunk");
    DevBuf<float> flat(2 * (int64_t)w->nvalid);
    ImatArgs A{};
    A.influ = dm->influ.p;
    A.i1 = dm->i1.p;
    A.j1 = dm->j1.p;
    A.isz = dm->influsize;
    A.dim = dm->dim;
    A.xoff = xoff;
    A.yoff = yoff;
    A.push = push;
    A.flat = flat.p;
    A.imat = dev_imat;
    // images per batch: as many as leave room for several CTAs on an SM
    int S = IMAT_ITEMS;
    while (S > 1 && w->smem_bytes(S) + IMAT_LIST_BYTES > 56 * 1024) --S;
    const size_t sm = ShSmem::align16(w->smem_bytes(S)) + IMAT_LIST_BYTES;
    if (w->nfft == 16)
      launch_imat_pd<16>(P, A, nact, S, sm, flat.p, s);
    else if (w->nfft == 32)
      launch_imat_pd<32>(P, A, nact, S, sm, flat.p, s);
    else
      launch_imat_pd<64>(P, A, nact, S, sm, flat.p, s);
    // the scratch is released below: wait for the launches that read it
    AOB_CUDA(cudaStreamSynchronize(s));
    return AOB_OK;
  } catch (const std::exception &e) {
    set_last_error(e.what());
    return AOB_ERR;
  }
}
