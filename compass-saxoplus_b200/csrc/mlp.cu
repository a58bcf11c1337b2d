// Learned reconstructor: a 3-layer MLP from slopes to DM commands
// (in -> h1 -> h2 -> out, GELU on the hidden layers) plus a linear skip path
// in -> out, y = W3 h2 + b3 + Ws x.  With Ws set to the least-squares command
// matrix and W3 = 0 the untrained network is the LS reconstructor; training
// learns the non-linear correction on top of it.  Trained on the GPU with
// the project's own BF16 tensor-core GEMMs (tcgen05 / TMEM in mlp_tc.cuh, or
// mma.sync in mlp_gemm.cuh) and Adam, run in the
// loop by three batch-1 GEMV kernels, and backed by the least-squares MVM:
// when the norm of the predicted commands exceeds a threshold the step uses
// the LS commands instead.  There is no counterpart in the reference.
//
// Numerics: weights are FP32 masters with BF16 copies; inputs and hidden
// activations are rounded to BF16, every product is accumulated in FP32.
// The network works on scaled quantities: x = slopes * in_scale,
// commands = y * out_scale.  All dimensions are padded to multiples of 8
// (padding weights stay zero).

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "aob_objects.hpp"
#include "mlp_gemm.cuh"
#include "mlp_tc.cuh"
#include "mvm_core.cuh"
#include "mlp_fused.cuh"

namespace aob {

__global__ void f32_to_bf16_kernel(const float *src, __nv_bfloat16 *dst, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i]);
}

// x [batch][nin] float -> xb [batch][pin] bf16 of x * scale, zero padding.  A thread
// takes groups of four elements, two groups' loads in flight (16-byte loads when
// every row starts on 16 bytes).  Bound: DRAM (x is read once).
__global__ void __launch_bounds__(256)
    mlp_input_kernel(const float *x, int nin, int pin, int64_t ngrp, int vec, float scale, __nv_bfloat16 *xb) {
  dep_sync();
  const int gpr = pin / 4;  // groups per row
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g0 < ngrp; g0 += 2 * stride) {
    float4 v[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int64_t g = g0 + k * stride;
      v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g < ngrp) {
        const int64_t b = g / gpr;
        const int i = 4 * (int)(g - b * gpr);
        const float *row = x + b * nin + i;
        if (vec) {
          if (i < nin) v[k] = __ldcs(reinterpret_cast<const float4 *>(row));
        } else {
          if (i < nin) v[k].x = __ldcs(row);
          if (i + 1 < nin) v[k].y = __ldcs(row + 1);
          if (i + 2 < nin) v[k].z = __ldcs(row + 2);
          if (i + 3 < nin) v[k].w = __ldcs(row + 3);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int64_t g = g0 + k * stride;
      if (g >= ngrp) break;
      __nv_bfloat162 q[2] = {__floats2bfloat162_rn(v[k].x * scale, v[k].y * scale),
                             __floats2bfloat162_rn(v[k].z * scale, v[k].w * scale)};
      *reinterpret_cast<uint2 *>(xb + 4 * g) = *reinterpret_cast<const uint2 *>(q);
    }
  }
}

// (after the mma.sync GEMMs; the tcgen05 GEMM stores the scaled outputs itself)
__global__ void mlp_output_kernel(const float *y, int nout, int pout, int batch, float scale, float *out) {
  for (int b = blockIdx.x; b < batch; b += gridDim.x)
    for (int o = threadIdx.x; o < nout; o += blockDim.x) out[(int64_t)b * nout + o] = y[(int64_t)b * pout + o] * scale;
}

// Mean-squared error on the scaled outputs: d = y - t / out_scale; the loss
// gradient 2 d / (batch * nout) goes to dy (bf16).  A block takes 32 adjacent
// columns and a chunk of rows (8 at a time, four rows' loads in flight per
// thread); it leaves the column sums of the rounded gradient over its rows (the
// output bias's gradient) and its sum of d^2, both added up by mlp_finish_kernel.
constexpr int LOSS_ROWS = 64;  // rows per block
__global__ void __launch_bounds__(256)
    mlp_loss_kernel(const float *y, const float *t, int nout, int pout, int batch, float inv_out_scale,
                    __nv_bfloat16 *dy, float *colpart, float *part) {
  dep_sync();
  __shared__ float red[8][33], red2[8];
  const float g = 2.f / ((float)batch * (float)nout);
  // (one grid dimension: the chunks of a large batch pass the 65535 of the others)
  const int ncb = (pout + 31) / 32, chunk = blockIdx.x / ncb;
  const int c = ((int)blockIdx.x - chunk * ncb) * 32 + threadIdx.x;
  const int r0 = chunk * LOSS_ROWS + threadIdx.y, r1 = min(batch, (chunk + 1) * LOSS_ROWS);
  float csum = 0.f, acc = 0.f;
  if (c < pout)
    for (int b0 = r0; b0 < r1; b0 += 32) {
      float yv[4], tv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int b = b0 + 8 * k;
        const bool in = b < r1 && c < nout;
        yv[k] = in ? __ldcs(y + (int64_t)b * pout + c) : 0.f;
        tv[k] = in ? __ldcs(t + (int64_t)b * nout + c) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int b = b0 + 8 * k;
        if (b >= r1) break;
        const float d = c < nout ? yv[k] - tv[k] * inv_out_scale : 0.f;
        const __nv_bfloat16 q = __float2bfloat16_rn(g * d);
        dy[(int64_t)b * pout + c] = q;
        csum += __bfloat162float(q);
        acc += d * d;
      }
    }
  red[threadIdx.y][threadIdx.x] = csum;
  acc = warp_sum(acc);  // (a row of threads is a warp)
  if (threadIdx.x == 0) red2[threadIdx.y] = acc;
  __syncthreads();
  if (threadIdx.y == 0) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += red[k][threadIdx.x];
    if (c < pout) colpart[(int64_t)chunk * pout + c] = v;
    if (threadIdx.x == 0) {
      v = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) v += red2[k];
      part[blockIdx.x] = v;
    }
  }
}

// Partial column sums of d [batch][cols] (cols even) over row chunks, for the
// mma.sync path (the tcgen05 GEMM's epilogue leaves them itself): block 64
// columns x 8 row lanes, two adjacent columns per thread, four rows in flight.
constexpr int COLSUM_CHUNKS = 16;
__global__ void mlp_colsum_part_kernel(const __nv_bfloat16 *d, int batch, int cols, float *part) {
  __shared__ float red[8][2][33];
  const int c = 2 * (blockIdx.x * 32 + threadIdx.x);
  const int rchunk = (batch + gridDim.y - 1) / gridDim.y;
  const int r0 = blockIdx.y * rchunk, r1 = min(batch, r0 + rchunk);
  float s0 = 0.f, s1 = 0.f;
  if (c < cols)
    for (int b0 = r0 + threadIdx.y; b0 < r1; b0 += 32) {
      __nv_bfloat162 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int b = b0 + 8 * k;
        v[k] = b < r1 ? *reinterpret_cast<const __nv_bfloat162 *>(d + (int64_t)b * cols + c)
                      : __floats2bfloat162_rn(0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (b0 + 8 * k >= r1) break;
        const float2 f = __bfloat1622float2(v[k]);
        s0 += f.x;
        s1 += f.y;
      }
    }
  red[threadIdx.y][0][threadIdx.x] = s0;
  red[threadIdx.y][1][threadIdx.x] = s1;
  __syncthreads();
  if (threadIdx.y < 2) {
    const int cc = c + threadIdx.y;
    if (cc < cols) {
      float t = 0.f;
      for (int y = 0; y < 8; ++y) t += red[y][threadIdx.y][threadIdx.x];
      part[(int64_t)blockIdx.y * cols + cc] = t;
    }
  }
}

// The small sums of a backward pass in one launch: the three bias gradients from
// their partial column sums, and the loss.  A block adds up 32 columns of one
// layer (8 lanes of parts, lane order fixed); the last block the loss.  (One thread
// adding the loss's 1184 partial sums took 18 us.)
struct FinishArgs {
  const float *part[3];
  float *out[3];
  int nparts[3], cols[3], block0[4];  // layer l: blocks block0[l] .. block0[l + 1]
  const float *loss_part;
  int nloss;
  float denom;
  float *loss;  // or null
};
__global__ void __launch_bounds__(256) mlp_finish_kernel(const __grid_constant__ FinishArgs A) {
  dep_sync();
  __shared__ float red[8][33];
  if ((int)blockIdx.x == A.block0[3]) {
    float s = 0.f;
    for (int i = threadIdx.y * 32 + threadIdx.x; i < A.nloss; i += 256) s += A.loss_part[i];
    s = warp_sum(s);
    if (threadIdx.x == 0) red[0][threadIdx.y] = s;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
      s = 0.f;
      for (int w = 0; w < 8; ++w) s += red[0][w];
      *A.loss = s / A.denom;
    }
    return;
  }
  int l = 0;
  while (l < 2 && (int)blockIdx.x >= A.block0[l + 1]) ++l;
  const int cols = A.cols[l], c = ((int)blockIdx.x - A.block0[l]) * 32 + threadIdx.x;
  float s = 0.f;
  if (c < cols)
    for (int y = threadIdx.y; y < A.nparts[l]; y += 8) s += A.part[l][(int64_t)y * cols + c];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < cols) {
    s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[k][threadIdx.x];
    A.out[l][c] = s;
  }
}

// Adam (Kingma & Ba 2015) on the FP32 masters of every layer, four values per
// thread; refreshes the BF16 copies.  One launch over the concatenated arrays
// (all sizes are multiples of 8).  Bound: DRAM, 30 bytes per parameter.
constexpr int ADAM_SEGS = 7;
struct AdamArgs {
  float *w[ADAM_SEGS], *m[ADAM_SEGS], *v[ADAM_SEGS];
  const float *g[ADAM_SEGS];
  __nv_bfloat16 *wb[ADAM_SEGS];  // or null
  int64_t end[ADAM_SEGS];        // groups of four up to and including this array
  float lr, b1, b2, eps, c1, c2;
};
__global__ void __launch_bounds__(256) mlp_adam_kernel(const __grid_constant__ AdamArgs A) {
  dep_sync();
  const int64_t total = A.end[ADAM_SEGS - 1];
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    int l = 0;
    while (q >= A.end[l]) ++l;
    const int64_t i = q - (l ? A.end[l - 1] : 0);
    float4 g4 = __ldcs(reinterpret_cast<const float4 *>(A.g[l]) + i);
    float4 m4 = reinterpret_cast<const float4 *>(A.m[l])[i];
    float4 v4 = reinterpret_cast<const float4 *>(A.v[l])[i];
    float4 w4 = reinterpret_cast<const float4 *>(A.w[l])[i];
    const float *g = &g4.x;
    float *m = &m4.x, *v = &v4.x, *w = &w4.x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m[k] = A.b1 * m[k] + (1.f - A.b1) * g[k];
      v[k] = A.b2 * v[k] + (1.f - A.b2) * g[k] * g[k];
      w[k] = w[k] - A.lr * (m[k] / A.c1) / (sqrtf(v[k] / A.c2) + A.eps);
    }
    reinterpret_cast<float4 *>(A.m[l])[i] = m4;
    reinterpret_cast<float4 *>(A.v[l])[i] = v4;
    reinterpret_cast<float4 *>(A.w[l])[i] = w4;
    if (A.wb[l]) {
      __nv_bfloat162 b[2] = {__floats2bfloat162_rn(w[0], w[1]), __floats2bfloat162_rn(w[2], w[3])};
      reinterpret_cast<uint2 *>(A.wb[l])[i] = *reinterpret_cast<const uint2 *>(b);
    }
  }
}

// Partial dot product of one bf16 row (nchunk 16-byte chunks) with x (float,
// shared memory) over the chunks lane, lane + 32, ...: GEMV_U loads in flight.
constexpr int GEMV_U = 8;
__device__ __forceinline__ float gemv_row(const uint4 *row, const float *x, int nchunk, int lane) {
  float acc = 0.f;
  for (int c0 = lane; c0 < nchunk; c0 += 32 * GEMV_U) {
    uint4 q[GEMV_U];
#pragma unroll
    for (int u = 0; u < GEMV_U; ++u) {
      const int c = c0 + 32 * u;
      q[u] = c < nchunk ? __ldg(row + c) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < GEMV_U; ++u) {
      const int c = c0 + 32 * u;
      if (c < nchunk) {
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&q[u]);
        const float4 x0 = *reinterpret_cast<const float4 *>(x + 8 * c);
        const float4 x1 = *reinterpret_cast<const float4 *>(x + 8 * c + 4);
        const float2 f0 = __bfloat1622float2(h[0]), f1 = __bfloat1622float2(h[1]);
        const float2 f2 = __bfloat1622float2(h[2]), f3 = __bfloat1622float2(h[3]);
        acc = fmaf(f0.x, x0.x, acc);
        acc = fmaf(f0.y, x0.y, acc);
        acc = fmaf(f1.x, x0.z, acc);
        acc = fmaf(f1.y, x0.w, acc);
        acc = fmaf(f2.x, x1.x, acc);
        acc = fmaf(f2.y, x1.y, acc);
        acc = fmaf(f3.x, x1.z, acc);
        acc = fmaf(f3.y, x1.w, acc);
      }
    }
  }
  return acc;
}

// One layer for a single input vector: y[r] = act(W[r] . bf16(x * xscale) + b[r]) * yscale
// for r < rows_real (0 in the padding).  One warp per row, 16-byte weight loads.
// With Ws set, y[r] also gets + Ws[r] . bf16(xs_in * xs_scale) (the skip path).
__global__ void mlp_gemv_kernel(const __nv_bfloat16 *W, const float *bias, const float *x, int nin_real, int ld,
                                float xscale, int rows, int rows_real, int gelu, float yscale, float *y,
                                const __nv_bfloat16 *Ws, const float *xs_in, int nskip_real, int lds,
                                float xs_scale) {
  extern __shared__ float xs[];
  float *xk = xs + ld;  // skip input
  for (int k = threadIdx.x; k < ld; k += blockDim.x) xs[k] = k < nin_real ? bf16_round(x[k] * xscale) : 0.f;
  if (Ws)
    for (int k = threadIdx.x; k < lds; k += blockDim.x) xk[k] = k < nskip_real ? bf16_round(xs_in[k] * xs_scale) : 0.f;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int nchunk = ld / 8;
  for (int r = blockIdx.x * nw + warp; r < rows; r += gridDim.x * nw) {
    const float acc = warp_sum(gemv_row(reinterpret_cast<const uint4 *>(W + (int64_t)r * ld), xs, nchunk, lane));
    const float sk = Ws ? warp_sum(gemv_row(reinterpret_cast<const uint4 *>(Ws + (int64_t)r * lds), xk, lds / 8, lane))
                        : 0.f;
    if (lane == 0) {
      float v = acc + bias[r] + sk;
      if (gelu) v = gelu_f(v);
      y[r] = r < rows_real ? v * yscale : 0.f;
    }
  }
}

// Reconstruction choice: predicted commands c = y; when ||c|| <= threshold the
// step uses them (err = -c, integrator applied here, LS MVM skipped), otherwise
// the LS MVM runs and the fallback counter is bumped.  One CTA.
__global__ void mlp_select_kernel(const float *y, int n, float threshold, float gain, const float *mgain, float *err,
                                  float *com, uint32_t *use_ls, uint32_t *fallbacks) {
  __shared__ float red[1024];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += y[i] * y[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  const bool fallback = !(sqrtf(red[0]) <= threshold);
  if (threadIdx.x == 0) {
    *use_ls = fallback ? 1u : 0u;
    if (fallback) *fallbacks += 1u;
  }
  if (!fallback)
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const float e = -y[i];
      err[i] = e;
      com[i] = gain * (e * mgain[i]) + com[i];
    }
}

// 2-D bf16 tensor map for the tcgen05 GEMM: inner (contiguous) extent, outer
// extent, row stride in elements; box 64 (inner, 128 bytes) x box_outer, 128-byte
// swizzle, zero fill outside the matrix.
// (the driver entry point is looked up through the runtime, so the library
// does not link the driver library itself and still loads on machines without it)
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    AOB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    AOB_REQUIRE(p != nullptr && q == cudaDriverEntryPointSuccess, "mlp gemm: cuTensorMapEncodeTiled not available");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

static void encode_map(CUtensorMap *m, const void *base, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_outer) {
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64u, box_outer};
  cuuint32_t es[2] = {1u, 1u};
  const CUresult r = encode_tiled_fn()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides,
                                       box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  AOB_REQUIRE(r == CUDA_SUCCESS, "mlp gemm: tensor map encoding failed (" + std::to_string((int)r) + ")");
}

// One product of a tcgen05 launch: the operands' layouts, an optional second product
// added in the same accumulator (same M, N and layouts), the epilogue's extra outputs.
struct TcOp {
  GemmArgs P;
  bool a_km, b_kn;
  const GemmArgs *P2 = nullptr;
  bool slices = false;  // K accumulated in slices (a weight gradient's K is the batch)
  float *colpart = nullptr;
  float *out = nullptr;
  int out_n = 0;
  float out_scale = 1.f;
};

// Launch up to TC_MAX_PROBS products of equal tile width as one list of tiles.
// Tile width: the one with the smallest cost = rounds of tiles over the pairs of SMs
// x (stages x time per stage + the tile's set-up), then one epilogue that nothing
// overlaps.  A stage takes about 0.1 us plus the part that grows with the width
// (0.3 us at 256); narrow tiles win where a product has few, wide ones where it
// has many.  An N-contiguous B is loaded in boxes of 64, so its tiles are 128 or
// 256 wide.
static void tc_gemm(const TcOp *ops, int n, int device, uint32_t *status, cudaStream_t s) {
  AOB_REQUIRE(n >= 1 && n <= TC_MAX_PROBS, "mlp gemm: bad product count");
  const int pairs = std::max(1, num_sms(device) / 2);
  int nk = 0;
  bool boxes = false;
  for (int i = 0; i < n; ++i) {
    const GemmArgs &P = ops[i].P;
    AOB_REQUIRE(P.M > 0 && P.N > 0 && P.K > 0, "mlp gemm: empty product");
    AOB_REQUIRE(P.lda % 8 == 0 && P.ldb % 8 == 0 && ((ops[i].a_km && ops[i].b_kn) || P.K % 8 == 0),
                "mlp gemm: contiguous dimensions must be multiples of 8");
    int k = (P.K + TC_BK - 1) / TC_BK;
    if (ops[i].P2) {
      AOB_REQUIRE(n == 1, "mlp gemm: a second operand pair goes with a single product");
      AOB_REQUIRE(ops[i].P2->M == P.M && ops[i].P2->N == P.N && ops[i].P2->K > 0 && ops[i].P2->lda % 8 == 0 &&
                      ops[i].P2->ldb % 8 == 0,
                  "mlp gemm: the second product must have the first's shape");
      k += (ops[i].P2->K + TC_BK - 1) / TC_BK;
    }
    AOB_REQUIRE(P.N % 2 == 0 && P.ldc % 2 == 0 && P.ldp % 2 == 0 && !P.accumulate &&
                    (P.epi == MG_EPI_NONE ? P.Cf && !P.Cb
                     : P.epi == MG_EPI_GELU ? P.bias && P.pre_out && P.Cb && !P.Cf
                                            : P.pre_in && P.Cb && !P.Cf && !P.bias && ops[i].colpart),
                "mlp gemm: outputs that the epilogue does not have");
    AOB_REQUIRE(!ops[i].slices || (P.epi == MG_EPI_NONE && !P.bias && !ops[i].out && !ops[i].P2),
                "mlp gemm: K slices go with a plain product");
    AOB_REQUIRE(P.epi == ops[0].P.epi && ops[i].slices == ops[0].slices,
                "mlp gemm: the products of a launch have the same epilogue");
    nk = std::max(nk, k);
    boxes |= ops[i].b_kn;
  }
  auto tiles_of = [&](int bn) {
    int64_t t = 0;
    for (int i = 0; i < n; ++i)
      t += (int64_t)((ops[i].P.M + TC_BM - 1) / TC_BM) * ((ops[i].P.N + bn - 1) / bn);
    return t;
  };
  int bn = TC_MAX_BN;
  double best = 1e30;
  for (int w = TC_MAX_BN; w >= 64; w -= 32) {
    if (boxes && w != 256 && w != 128) continue;
    const double rounds = (double)((tiles_of(w) + pairs - 1) / pairs);
    const double cost = rounds * (nk * (0.1 + 0.0008 * w) + 0.5) + 1.0 + 0.01 * w;
    if (cost < best) {
      best = cost;
      bn = w;
    }
  }
  TcArgs T{};
  TcMaps M;
  T.nprob = n;
  T.bn = bn;
  T.status = status;
  int64_t tiles = 0;
  auto maps = [bn](const GemmArgs &Q, bool a_km, bool b_kn, CUtensorMap *m) {
    if (a_km)
      encode_map(&m[0], Q.A, (uint64_t)Q.M, (uint64_t)Q.K, (uint64_t)Q.lda, 64u);
    else
      encode_map(&m[0], Q.A, (uint64_t)Q.K, (uint64_t)Q.M, (uint64_t)Q.lda, (uint32_t)TC_ROWS);
    if (b_kn)
      encode_map(&m[1], Q.B, (uint64_t)Q.N, (uint64_t)Q.K, (uint64_t)Q.ldb, 64u);
    else
      encode_map(&m[1], Q.B, (uint64_t)Q.K, (uint64_t)Q.N, (uint64_t)Q.ldb, (uint32_t)(bn / 2));
  };
  for (int i = 0; i < n; ++i) {
    const TcOp &O = ops[i];
    TcProb &Q = T.prob[i];
    Q.P = O.P;
    Q.a_mn = O.a_km ? 1 : 0;
    Q.b_mn = O.b_kn ? 1 : 0;
    Q.K2 = O.P2 ? O.P2->K : 0;
    Q.tiles_m = (O.P.M + TC_BM - 1) / TC_BM;
    Q.tile0 = (int)tiles;
    Q.colpart = O.colpart;
    Q.out = O.out;
    Q.out_n = O.out_n;
    Q.out_scale = O.out_scale;
    tiles += (int64_t)Q.tiles_m * ((O.P.N + bn - 1) / bn);
    maps(O.P, O.a_km, O.b_kn, &M.m[2 * i]);
    if (O.P2) maps(*O.P2, O.a_km, O.b_kn, &M.m[2]);
  }
  AOB_REQUIRE(tiles < (int64_t)1 << 30, "mlp gemm: too many tiles");
  T.ntiles = (int)tiles;
  for (int i = n == 1 && ops[0].P2 ? 2 : n; i < TC_MAX_PROBS; ++i) {
    M.m[2 * i] = M.m[0];
    M.m[2 * i + 1] = M.m[1];
  }
  const int epi = ops[0].P.epi;
  auto kern = ops[0].slices          ? tc_gemm_kernel<TC_EPI_SLICES>
              : epi == MG_EPI_GELU   ? tc_gemm_kernel<MG_EPI_GELU>
              : epi == MG_EPI_DGELU  ? tc_gemm_kernel<MG_EPI_DGELU>
                                     : tc_gemm_kernel<MG_EPI_NONE>;
  smem_opt_in(reinterpret_cast<const void *>(kern), (int)TC_SMEM_BYTES);
  launch_after(kern, 2 * (int)std::min<int64_t>(tiles, pairs), TC_THREADS, TC_SMEM_BYTES, s, M, T);
  AOB_LAUNCH_CHECK("tc_gemm_kernel");
}

// The mma.sync kernel.
template <bool A_KM, bool B_KN>
static void gemm(const GemmArgs &P, cudaStream_t s) {
  AOB_REQUIRE(P.M > 0 && P.N > 0 && P.K > 0, "mlp gemm: empty product");
  AOB_REQUIRE(P.lda % 8 == 0 && P.ldb % 8 == 0 && ((A_KM && B_KN) || P.K % 8 == 0),
              "mlp gemm: contiguous dimensions must be multiples of 8");
  dim3 grid((P.N + MG_BN - 1) / MG_BN, (P.M + MG_BM - 1) / MG_BM);
  mlp_gemm_kernel<A_KM, B_KN><<<grid, MG_THREADS, 0, s>>>(P);
  AOB_LAUNCH_CHECK("mlp_gemm_kernel");
}

static int grid_for(int64_t n, int device) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8 * num_sms(device)));
}

}  // namespace aob

using namespace aob;

static int pad8(int v) { return (v + 7) / 8 * 8; }

aob_mlp::aob_mlp(int device_, int nin_, int nh1_, int nh2_, int nout_)
    : device(device_), nin(nin_), nh1(nh1_), nh2(nh2_), nout(nout_) {
  AOB_REQUIRE(nin > 0 && nh1 > 0 && nh2 > 0 && nout > 0, "mlp: sizes must be > 0");
  pin = pad8(nin);
  ph1 = pad8(nh1);
  ph2 = pad8(nh2);
  pout = pad8(nout);
  AOB_CUDA(cudaSetDevice(device));
  for (int l = 0; l < 4; ++l) {
    const int64_t nw = (int64_t)rows(l) * cols(l);
    w[l].alloc(nw);
    mw[l].alloc(nw);
    vw[l].alloc(nw);
    gw[l].alloc(nw);
    wb[l].alloc(nw);
    if (l < 3) {
      b[l].alloc(rows(l));
      mb[l].alloc(rows(l));
      vb[l].alloc(rows(l));
      gb[l].alloc(rows(l));
    }
  }
  ix.alloc(pin);
  ih1.alloc(ph1);
  ih2.alloc(ph2);
  iy.alloc(pout);
  use_ls.alloc(1);
  fallbacks.alloc(1);
  tc_status.alloc(1);
}

static void real_dims(const aob_mlp &m, int l, int &rr, int &cr) {
  rr = l == 0 ? m.nh1 : (l == 1 ? m.nh2 : m.nout);
  cr = l == 0 ? m.nin : (l == 1 ? m.nh1 : (l == 2 ? m.nh2 : m.nin));
}

void aob_mlp::set_params(int l, const float *wh, const float *bh) {
  AOB_REQUIRE(l >= 0 && l < 4 && wh && (bh || l == 3), "mlp.set_params: bad layer or null arrays");
  AOB_CUDA(cudaSetDevice(device));
  int rr, cr;
  real_dims(*this, l, rr, cr);
  std::vector<float> W((size_t)rows(l) * cols(l), 0.f), B(rows(l), 0.f);
  for (int r = 0; r < rr; ++r) {
    for (int c = 0; c < cr; ++c) W[(size_t)r * cols(l) + c] = wh[(size_t)r * cr + c];
    if (bh) B[r] = bh[r];
  }
  w[l].upload(W.data(), (int64_t)W.size());
  AOB_CUDA(cudaMemset(mw[l].p, 0, mw[l].bytes()));
  AOB_CUDA(cudaMemset(vw[l].p, 0, vw[l].bytes()));
  if (l < 3) {
    b[l].upload(B.data(), (int64_t)B.size());
    AOB_CUDA(cudaMemset(mb[l].p, 0, mb[l].bytes()));
    AOB_CUDA(cudaMemset(vb[l].p, 0, vb[l].bytes()));
  }
  f32_to_bf16_kernel<<<grid_for(w[l].n, device), 256>>>(w[l].p, reinterpret_cast<__nv_bfloat16 *>(wb[l].p), w[l].n);
  AOB_LAUNCH_CHECK("f32_to_bf16_kernel");
  AOB_CUDA(cudaDeviceSynchronize());
  t = 0;
}

void aob_mlp::get_params(int l, float *wh, float *bh) {
  AOB_REQUIRE(l >= 0 && l < 4, "mlp.get_params: bad layer");
  AOB_CUDA(cudaSetDevice(device));
  AOB_CUDA(cudaDeviceSynchronize());
  int rr, cr;
  real_dims(*this, l, rr, cr);
  std::vector<float> W((size_t)rows(l) * cols(l)), B(rows(l), 0.f);
  AOB_CUDA(cudaMemcpy(W.data(), w[l].p, w[l].bytes(), cudaMemcpyDeviceToHost));
  if (l < 3) AOB_CUDA(cudaMemcpy(B.data(), b[l].p, b[l].bytes(), cudaMemcpyDeviceToHost));
  if (wh)
    for (int r = 0; r < rr; ++r)
      for (int c = 0; c < cr; ++c) wh[(size_t)r * cr + c] = W[(size_t)r * cols(l) + c];
  if (bh)
    for (int r = 0; r < rr; ++r) bh[r] = B[r];
}

void aob_mlp::ensure_batch(int batch) {
  AOB_REQUIRE(batch > 0, "mlp: batch must be > 0");
  if (batch <= cap) return;
  AOB_CUDA(cudaSetDevice(device));
  cap = batch;
  xb.alloc((int64_t)cap * pin);
  z1.alloc((int64_t)cap * ph1);
  h1b.alloc((int64_t)cap * ph1);
  z2.alloc((int64_t)cap * ph2);
  h2b.alloc((int64_t)cap * ph2);
  y.alloc((int64_t)cap * pout);
  dy.alloc((int64_t)cap * pout);
  dz2.alloc((int64_t)cap * ph2);
  dz1.alloc((int64_t)cap * ph1);
  // partial sums: the loss kernel's blocks, and the bias gradients' (a row per 32
  // samples, the output layer's per LOSS_ROWS; COLSUM_CHUNKS rows on the mma.sync path)
  const int nchunk = (cap + LOSS_ROWS - 1) / LOSS_ROWS, rparts = std::max((cap + 31) / 32, COLSUM_CHUNKS);
  const int64_t np[4] = {(int64_t)rparts * ph1, (int64_t)rparts * ph2, (int64_t)nchunk * pout,
                         (int64_t)nchunk * ((pout + 31) / 32)};
  parts.alloc(np[0] + np[1] + np[2] + np[3]);  // (one allocation: they are on the path of a first forward)
  colpart[0] = parts.p;
  for (int l = 1; l < 3; ++l) colpart[l] = colpart[l - 1] + np[l - 1];
  loss_part = colpart[2] + np[2];
}

static __nv_bfloat16 *bf(aob::DevBuf<uint16_t> &b) { return reinterpret_cast<__nv_bfloat16 *>(b.p); }

void aob_mlp::forward(const float *x, int batch, float *y_out, cudaStream_t s) {
  AOB_CUDA(cudaSetDevice(device));
  ensure_batch(batch);
  {
    const int64_t ngrp = (int64_t)batch * (pin / 4);
    const int vec = nin % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    launch_after(mlp_input_kernel, (int)std::max<int64_t>(1, std::min<int64_t>((ngrp + 511) / 512, 8 * num_sms(device))), 256, 0, s,
        x, nin, pin, ngrp, vec, in_scale, bf(xb));
    AOB_LAUNCH_CHECK("mlp_input_kernel");
  }
  // h1 = GELU(x W1^T + b1), h2 = GELU(h1 W2^T + b2), y = h2 W3^T + b3 + x Ws^T (the skip path)
  const GemmArgs P1{batch, ph1, pin, bf(xb), pin, bf(wb[0]), pin, b[0].p, MG_EPI_GELU, nullptr, z1.p, ph1,
                    nullptr, bf(h1b), ph1, 0};
  const GemmArgs P2{batch, ph2, ph1, bf(h1b), ph1, bf(wb[1]), ph1, b[1].p, MG_EPI_GELU, nullptr, z2.p, ph2,
                    nullptr, bf(h2b), ph2, 0};
  const GemmArgs P3{batch, pout, ph2, bf(h2b), ph2, bf(wb[2]), ph2, b[2].p, MG_EPI_NONE, nullptr, nullptr, 0,
                    y.p, nullptr, pout, 0};
  GemmArgs PS{batch, pout, pin, bf(xb), pin, bf(wb[3]), pin, nullptr, MG_EPI_NONE, nullptr, nullptr, 0,
              y.p, nullptr, pout, 1};
  if (gemm_kind == 1) {
    TcOp O{P1, false, false};
    tc_gemm(&O, 1, device, tc_status.p, s);
    O.P = P2;
    tc_gemm(&O, 1, device, tc_status.p, s);
    O.P = P3;  // one K loop over [h2 | x]
    O.P2 = &PS;
    O.out = y_out;
    O.out_n = nout;
    O.out_scale = out_scale;
    tc_gemm(&O, 1, device, tc_status.p, s);
    return;
  }
  gemm<false, false>(P1, s);
  gemm<false, false>(P2, s);
  gemm<false, false>(P3, s);
  gemm<false, false>(PS, s);
  if (y_out) {
    mlp_output_kernel<<<std::min(batch, 8 * num_sms(device)), 256, 0, s>>>(y.p, nout, pout, batch, out_scale,
                                                                              y_out);
    AOB_LAUNCH_CHECK("mlp_output_kernel");
  }
}

// Gradients of the MSE after forward() on the same batch.
void aob_mlp::backward(const float *target, int batch, float *loss, cudaStream_t s) {
  AOB_REQUIRE(batch <= cap, "mlp.backward: run forward on this batch first");
  AOB_CUDA(cudaSetDevice(device));
  const int nchunk = (batch + LOSS_ROWS - 1) / LOSS_ROWS;
  const int64_t lgrid = (int64_t)nchunk * ((pout + 31) / 32);
  AOB_REQUIRE(lgrid <= INT32_MAX, "mlp.backward: batch too large");
  launch_after(mlp_loss_kernel, (unsigned)lgrid, dim3(32, 8), 0, s, y.p, target, nout, pout, batch, 1.f / out_scale, bf(dy), colpart[2],
               loss_part);
  AOB_LAUNCH_CHECK("mlp_loss_kernel");
  // data gradients: dz2 = (dy W3) * GELU'(z2), dz1 = (dz2 W2) * GELU'(z1)
  const GemmArgs D2{batch, ph2, pout, bf(dy), pout, bf(wb[2]), ph2, nullptr, MG_EPI_DGELU, z2.p, nullptr, ph2,
                    nullptr, bf(dz2), ph2, 0};
  const GemmArgs D1{batch, ph1, ph2, bf(dz2), ph2, bf(wb[1]), ph1, nullptr, MG_EPI_DGELU, z1.p, nullptr, ph1,
                    nullptr, bf(dz1), ph1, 0};
  // weight gradients: dW3 = dy^T h2, dW2 = dz2^T h1, dW1 = dz1^T x, dWs = dy^T x
  const GemmArgs G3{pout, ph2, batch, bf(dy), pout, bf(h2b), ph2, nullptr, MG_EPI_NONE, nullptr, nullptr, 0,
                    gw[2].p, nullptr, ph2, 0};
  const GemmArgs G2{ph2, ph1, batch, bf(dz2), ph2, bf(h1b), ph1, nullptr, MG_EPI_NONE, nullptr, nullptr, 0,
                    gw[1].p, nullptr, ph1, 0};
  const GemmArgs G1{ph1, pin, batch, bf(dz1), ph1, bf(xb), pin, nullptr, MG_EPI_NONE, nullptr, nullptr, 0,
                    gw[0].p, nullptr, pin, 0};
  const GemmArgs GS{pout, pin, batch, bf(dy), pout, bf(xb), pin, nullptr, MG_EPI_NONE, nullptr, nullptr, 0,
                    gw[3].p, nullptr, pin, 0};
  int rparts;
  if (gemm_kind == 1) {
    rparts = (batch + 31) / 32;
    TcOp O{D2, false, true};
    O.colpart = colpart[1];
    tc_gemm(&O, 1, device, tc_status.p, s);
    O.P = D1;
    O.colpart = colpart[0];
    tc_gemm(&O, 1, device, tc_status.p, s);
    // (a batch of one slice needs no sums)
    const bool slices = batch > TC_SLICE * TC_BK;
    const TcOp W[4] = {{GS, true, true, nullptr, slices},
                       {G1, true, true, nullptr, slices},
                       {G3, true, true, nullptr, slices},
                       {G2, true, true, nullptr, slices}};
    tc_gemm(W, 4, device, tc_status.p, s);
  } else {
    rparts = COLSUM_CHUNKS;
    auto colsum = [&](const __nv_bfloat16 *d, int cols, float *part) {
      mlp_colsum_part_kernel<<<dim3((cols / 2 + 31) / 32, COLSUM_CHUNKS), dim3(32, 8), 0, s>>>(d, batch, cols, part);
      AOB_LAUNCH_CHECK("mlp_colsum_part_kernel");
    };
    gemm<true, true>(G3, s);
    gemm<false, true>(D2, s);
    colsum(bf(dz2), ph2, colpart[1]);
    gemm<true, true>(G2, s);
    gemm<false, true>(D1, s);
    colsum(bf(dz1), ph1, colpart[0]);
    gemm<true, true>(G1, s);
    gemm<true, true>(GS, s);
  }
  FinishArgs F{};
  const int cols[3] = {ph1, ph2, pout}, parts[3] = {rparts, rparts, nchunk};
  for (int l = 0; l < 3; ++l) {
    F.part[l] = colpart[l];
    F.out[l] = gb[l].p;
    F.nparts[l] = parts[l];
    F.cols[l] = cols[l];
    F.block0[l + 1] = F.block0[l] + (cols[l] + 31) / 32;
  }
  F.loss_part = loss_part;
  F.nloss = (int)lgrid;
  F.denom = (float)batch * (float)nout;
  F.loss = loss;
  launch_after(mlp_finish_kernel, F.block0[3] + (loss ? 1 : 0), dim3(32, 8), 0, s, F);
  AOB_LAUNCH_CHECK("mlp_finish_kernel");
}

void aob_mlp::adam(float lr, cudaStream_t s) {
  AOB_CUDA(cudaSetDevice(device));
  ++t;
  AdamArgs A{};
  A.lr = lr;
  A.b1 = beta1;
  A.b2 = beta2;
  A.eps = eps;
  A.c1 = 1.f - std::pow(beta1, (float)t);
  A.c2 = 1.f - std::pow(beta2, (float)t);
  int64_t end = 0;
  for (int q = 0; q < ADAM_SEGS; ++q) {
    const bool weight = q < 4;
    const int l = weight ? q : q - 4;
    A.w[q] = weight ? w[l].p : b[l].p;
    A.m[q] = weight ? mw[l].p : mb[l].p;
    A.v[q] = weight ? vw[l].p : vb[l].p;
    A.g[q] = weight ? gw[l].p : gb[l].p;
    A.wb[q] = weight ? bf(wb[l]) : nullptr;
    end += (weight ? w[l].n : b[l].n) / 4;
    A.end[q] = end;
  }
  launch_after(mlp_adam_kernel, (int)std::max<int64_t>(1, std::min<int64_t>((end + 255) / 256, 8 * num_sms(device))), 256, 0, s, A);
  AOB_LAUNCH_CHECK("mlp_adam_kernel");
}

void aob_mlp::infer(const float *x, float *y_out, cudaStream_t s) {
  AOB_CUDA(cudaSetDevice(device));
  const int threads = 256, nw = threads / 32;
  auto layer = [&](int l, const float *in, int nin_real, float xscale, int nrows_real, int gelu, float yscale,
                   float *out, bool skip) {
    const int rws = rows(l), ld = cols(l);
    const int grid = std::max(1, std::min((rws + nw - 1) / nw, 4 * num_sms(device)));
    const size_t sm = sizeof(float) * (ld + (skip ? pin : 0));
    mlp_gemv_kernel<<<grid, threads, sm, s>>>(bf(wb[l]), b[l].p, in, nin_real, ld, xscale, rws, nrows_real, gelu,
                                              yscale, out, skip ? bf(wb[3]) : nullptr, x, nin, pin, in_scale);
    AOB_LAUNCH_CHECK("mlp_gemv_kernel");
  };
  layer(0, x, nin, in_scale, nh1, 1, 1.f, ih1.p, false);
  layer(1, ih1.p, ph1, 1.f, nh2, 1, 1.f, ih2.p, false);
  layer(2, ih2.p, ph2, 1.f, nout, 0, out_scale, y_out ? y_out : iy.p, true);
}


// ---------------------------------------------------------------------------
// the fused control step (mlp_fused_kernel) is in mlp_fused.cuh

using namespace aob;

// One control step through the fused kernel; false when the configuration
// does not fit it (shared memory, co-residency), in which case the caller runs
// the multi-kernel path.
// The arguments of the fused control step for controller ls on a grid of one CTA
// per SM, and its shared-memory bytes; false when it does not fit.
bool aob_mlp::fused_args(aob_ls *ls, float threshold, MlpFusedArgs &A, size_t &smem_bytes) {
  if (fused_mode == 1) return false;
  if (ls->mvm_kind == 2) return false;  // the fallback reproduces the bulk-copy MVM only
  ls->ensure_packed(ls->prec);
  const int G = num_sms(device);
  auto per = [G](int n) { return (n + G - 1) / G; };
  const int esize = ls->prec == AOB_PREC_F32 ? 4 : (ls->prec == AOB_PREC_BF16 ? 2 : 1);
  const int V = 16 / esize;
  const int ld_ls = (ls->nslope + V - 1) / V * V;
  A = MlpFusedArgs{};
  A.W1 = bf(wb[0]);
  A.W2 = bf(wb[1]);
  A.W3 = bf(wb[2]);
  A.Ws = bf(wb[3]);
  A.b1 = b[0].p;
  A.b2 = b[1].p;
  A.b3 = b[2].p;
  A.pin = pin;
  A.ph1 = ph1;
  A.ph2 = ph2;
  A.pout = pout;
  A.nin = nin;
  A.nh1 = nh1;
  A.nh2 = nh2;
  A.nout = nout;
  A.in_scale = in_scale;
  A.out_scale = out_scale;
  A.threshold = threshold;
  A.x = ls->centroids.p;
  A.h1 = ih1.p;
  A.h2 = ih2.p;
  A.y = iy.p;
  if (partial.n < G) partial.alloc(G);
  if (gbar.n < GRID_WORDS) gbar.alloc(GRID_WORDS);
  A.partial = partial.p;
  A.n1 = per(ph1);
  A.n2 = per(ph2);
  A.n3 = per(pout);
  A.nls = per(nout);
  A.gain = ls->gain;
  A.mgain = ls->gains.p;
  A.err = ls->err.p;
  A.com = ls->com();
  A.use_ls = use_ls.p;
  A.fallbacks = fallbacks.p;
  A.status = ls->status.p;
  A.gbar = gbar.p;
  A.lsmat = ls->prec == AOB_PREC_F32 ? (const void *)ls->cm_f32.p
                                     : (ls->prec == AOB_PREC_BF16 ? (const void *)ls->cm_bf16.p : (const void *)ls->cm_fp8.p);
  A.rscale = ls->prec == AOB_PREC_FP8 ? ls->row_scale.p : nullptr;
  A.ld_ls = ld_ls;
  AOB_REQUIRE((int64_t)std::max(pin, pout) * G < (int64_t)1 << 32, "mlp: sizes beyond the row-split range");
  const MlpFusedSmem L(pin, ph1, ph2, A.n1, A.n2, A.n3, A.nls, swizzled_slope_floats(ld_ls, V));
  if (L.bytes > 227 * 1024 || A.nls > MLP_FUSED_THREADS) return false;
  smem_bytes = L.bytes;
  return true;
}

bool aob_mlp::comp_com_fused(aob_ls *ls, float threshold, cudaStream_t s) {
  MlpFusedArgs A{};
  size_t smem = 0;
  if (!fused_args(ls, threshold, A, smem)) return false;
  const int G = num_sms(device);
  auto launch = [&](auto kern) {
    try {
      smem_opt_in(reinterpret_cast<const void *>(kern), (int)smem);  // only ever raised, per device
    } catch (const std::exception &) {
      cudaGetLastError();
      return false;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, MLP_FUSED_THREADS, smem) != cudaSuccess ||
        per_sm < 1) {
      cudaGetLastError();
      return false;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(MLP_FUSED_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    AOB_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
    AOB_LAUNCH_CHECK("mlp_fused_kernel");
    return true;
  };
  if (ls->prec == AOB_PREC_F32) return launch(mlp_fused_kernel<float>);
  if (ls->prec == AOB_PREC_BF16) return launch(mlp_fused_kernel<__nv_bfloat16>);
  return launch(mlp_fused_kernel<__nv_fp8_e4m3>);
}

// ---------------------------------------------------------------------------
extern "C" {

#define MLP_TRY try {
#define MLP_END                     \
  return AOB_OK;                    \
  }                                 \
  catch (const std::exception &e) { \
    aob::set_last_error(e.what());  \
    return AOB_ERR;                 \
  }
#define MLP_NEED(p) \
  if (!(p)) throw aob::Error(std::string(__func__) + ": null handle or pointer")
static inline cudaStream_t MS(void *p) { return reinterpret_cast<cudaStream_t>(p); }

int aob_mlp_create(aob_mlp **out, int device, int nin, int nh1, int nh2, int nout) {
  MLP_TRY MLP_NEED(out);
  *out = nullptr;
  AOB_CUDA(cudaSetDevice(device));
  *out = new aob_mlp(device, nin, nh1, nh2, nout);
  MLP_END
}
int aob_mlp_destroy(aob_mlp *m) {
  MLP_TRY if (m) {
    cudaSetDevice(m->device);
    delete m;
  }
  MLP_END
}
int aob_mlp_set_params(aob_mlp *m, int layer, const float *w, const float *b) {
  MLP_TRY MLP_NEED(m);
  m->set_params(layer, w, b);
  MLP_END
}
int aob_mlp_get_params(aob_mlp *m, int layer, float *w, float *b) {
  MLP_TRY MLP_NEED(m);
  m->get_params(layer, w, b);
  MLP_END
}
int aob_mlp_set_scales(aob_mlp *m, float in_scale, float out_scale) {
  MLP_TRY MLP_NEED(m);
  if (!(out_scale != 0.f)) throw aob::Error("mlp.set_scales: out_scale must be non-zero");
  m->in_scale = in_scale;
  m->out_scale = out_scale;
  MLP_END
}
int aob_mlp_forward(aob_mlp *m, const float *dev_x, int batch, float *dev_y, void *stream) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(dev_x);
  m->forward(dev_x, batch, dev_y, MS(stream));
  MLP_END
}
int aob_mlp_backward(aob_mlp *m, const float *dev_target, int batch, float *dev_loss, void *stream) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(dev_target);
  m->backward(dev_target, batch, dev_loss, MS(stream));
  MLP_END
}
int aob_mlp_train_step(aob_mlp *m, const float *dev_x, const float *dev_target, int batch, float lr,
                       float *dev_loss, void *stream) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(dev_x);
  MLP_NEED(dev_target);
  m->forward(dev_x, batch, nullptr, MS(stream));
  m->backward(dev_target, batch, dev_loss, MS(stream));
  m->adam(lr, MS(stream));
  MLP_END
}
int aob_mlp_infer(aob_mlp *m, const float *dev_x, float *dev_y, void *stream) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(dev_x);
  m->infer(dev_x, dev_y, MS(stream));
  MLP_END
}
int aob_mlp_comp_com(aob_mlp *m, aob_ls *ls, float threshold, void *stream) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(ls);
  if (ls->nslope != m->nin || ls->nactu != m->nout) throw aob::Error("mlp.comp_com: sizes differ from the controller's");
  if (ls->kind != AOB_CTRL_LS) throw aob::Error("mlp.comp_com: the LS fallback needs an LS controller");
  if (ls->open_loop) return AOB_OK;
  AOB_CUDA(cudaSetDevice(m->device));
  cudaStream_t s = MS(stream);
  if (m->comp_com_fused(ls, threshold, s)) return AOB_OK;
  m->infer(ls->centroids.p, m->iy.p, s);
  mlp_select_kernel<<<1, 1024, 0, s>>>(m->iy.p, m->nout, threshold, ls->gain, ls->gains.p, ls->err.p, ls->com(),
                                       m->use_ls.p, m->fallbacks.p);
  AOB_LAUNCH_CHECK("mlp_select_kernel");
  ls->comp_com(s, nullptr, m->use_ls.p);
  MLP_END
}
int aob_mlp_set_gemm(aob_mlp *m, int kind) {
  MLP_TRY MLP_NEED(m);
  if (kind < 0 || kind > 1) throw aob::Error("mlp.set_gemm: kind must be 0 or 1");
  m->gemm_kind = kind;
  MLP_END
}
int aob_mlp_gemm_status(aob_mlp *m, uint32_t *status, int reset) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(status);
  AOB_CUDA(cudaSetDevice(m->device));
  AOB_CUDA(cudaMemcpy(status, m->tc_status.p, sizeof(uint32_t), cudaMemcpyDeviceToHost));
  if (reset) AOB_CUDA(cudaMemset(m->tc_status.p, 0, sizeof(uint32_t)));
  MLP_END
}
int aob_mlp_set_mode(aob_mlp *m, int mode) {
  MLP_TRY MLP_NEED(m);
  if (mode < 0 || mode > 1) throw aob::Error("mlp.set_mode: mode must be 0 or 1");
  m->fused_mode = mode;
  MLP_END
}
int aob_mlp_fallbacks(aob_mlp *m, uint32_t *count, int reset) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(count);
  AOB_CUDA(cudaSetDevice(m->device));
  AOB_CUDA(cudaMemcpy(count, m->fallbacks.p, sizeof(uint32_t), cudaMemcpyDeviceToHost));
  if (reset) AOB_CUDA(cudaMemset(m->fallbacks.p, 0, sizeof(uint32_t)));
  MLP_END
}
int aob_mlp_buffer(aob_mlp *m, const char *which, void **dev_ptr, int64_t *nelem) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(which);
  MLP_NEED(dev_ptr);
  const std::string w(which);
  void *p = nullptr;
  int64_t n = 0;
  auto pick = [&](const char *name, aob::DevBuf<float> *arr) {
    for (int l = 0; l < 3; ++l)
      if (w == std::string(name) + std::to_string(l + 1)) {
        p = arr[l].p;
        n = arr[l].n;
      }
  };
  pick("W", m->w);
  if (w == "Ws") {
    p = m->w[3].p;
    n = m->w[3].n;
  } else if (w == "dWs") {
    p = m->gw[3].p;
    n = m->gw[3].n;
  }
  pick("b", m->b);
  pick("dW", m->gw);
  pick("db", m->gb);
  if (w == "y") {
    p = m->y.p;
    n = m->y.n;
  }
  if (!p) throw aob::Error("mlp.buffer: unknown buffer '" + w + "'");
  *dev_ptr = p;
  if (nelem) *nelem = n;
  MLP_END
}
int aob_mlp_get_dims(aob_mlp *m, int *padded4) {
  MLP_TRY MLP_NEED(m);
  MLP_NEED(padded4);
  padded4[0] = m->pin;
  padded4[1] = m->ph1;
  padded4[2] = m->ph2;
  padded4[3] = m->pout;
  MLP_END
}

}  // extern "C"
