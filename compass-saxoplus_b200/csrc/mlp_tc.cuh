// BF16 GEMM on the fifth-generation tensor cores (tcgen05) for the learned
// reconstructor's batched products.  Same contract as mlp_gemm_kernel (GemmArgs:
// A stored M x K ("MK") or K x M ("KM"), B stored N x K ("NK") or K x N
// ("KN"), the same epilogue), so the three products of a training step run
// without transposed copies: K-major operands use the K-major shared-memory
// descriptor, M- or N-contiguous ones the MN-major descriptor.
//
// Two CTAs (a cluster, cta_group::2) form one 256 x bn tile: each loads its own
// 128 rows of A and bn / 2 rows of B, 32 KB for a 64-deep stage at bn = 256,
// two thirds of what two separate 128 x 256 tiles need from L2 and half of what
// four 128 x 128 tiles do.  Bound: that traffic -- with either tile the SMs draw
// 9 - 10 TB/s from L2 (0.42 us per stage at 256 x 256, 1.28 PFLOP/s in the main
// loop; 128 x 128 tiles reached 0.68).  A training step at batch 4096 (2496 -> 1024
// -> 1024 -> 1377) takes 309 us, 503 us with 128 x 128 tiles, split K and a launch
// per bias and parameter array.
// Pairs are persistent: pair p takes tiles p, p + pairs, ... of a list of up to
// TC_MAX_PROBS products, so the four weight gradients of a training step
// (independent, K = the batch) fill the GPU in one launch.  Their K is accumulated in
// slices of TC_SLICE stages that the epilogue adds in registers: in one run the
// accumulator's rounding grows with the batch (against float64 sums of the same bfloat16
// values 9e-6 at batch 4096 and 1e-4 at 20,000; 3e-7 at either in slices, 1 to 8 us of a
// step).
// Per CTA, 18 warps:
//  * warp 0, one lane: TMA producer -- 2-D tensor loads with 128-byte swizzle
//    (K-major tile: one box of 64 (K) x rows; MN-major: boxes of 64 (M or N) x
//    64 (K)) into a 5-stage ring; both CTAs' loads complete on the "full"
//    mbarrier of the leader (cluster rank 0);
//  * warp 1: allocates the TMEM (two 256-column FP32 accumulators); one lane of
//    the leader issues tcgen05.mma.cta_group::2.kind::f16 (M 256, N bn, K 16) and
//    commits each stage to both CTAs' "empty" mbarriers, and each finished
//    tile to both CTAs' accumulator barriers;
//  * 16 warps: the epilogue of a tile (or slice) while the next one is multiplied -- a warp
//    reads the TMEM lanes of its quadrant (warp & 3) in chunks of 16 columns,
//    transposes each through shared memory and applies bias / GELU / GELU' with
//    row accesses of whole sectors.
// A second operand pair (A2, B2, same layouts, its own K) can follow the first
// in the same K loop, so y = h2 W3^T + x Ws^T is one GEMM with no read-back of
// the output.
// Every mbarrier wait is bounded: on expiry a status bit is set, nothing of the
// tile is stored, and the CTA goes to its end, where it waits (bounded) for its loads and
// the pair's MMAs in flight and frees its TMEM.  No load uses multicast.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "aob_common.cuh"
#include "mlp_gemm.cuh"

namespace aob {

constexpr int TC_BM = 256, TC_ROWS = 128, TC_MAX_BN = 256, TC_BK = 64, TC_STAGES = 5;
constexpr int TC_EPI_WARPS = 16, TC_THREADS = 64 + 32 * TC_EPI_WARPS;
constexpr int TC_TILE_BYTES = TC_ROWS * TC_BK * 2;  // one operand tile of a CTA and stage (16 KB)
constexpr int TC_STAGE_BYTES = 2 * TC_TILE_BYTES;
constexpr int TC_MAX_PROBS = 4;
// K stages of one slice of a weight gradient (512 samples): the tensor cores' FP32
// accumulator loses a little at every addition, in proportion to its sum, so a long K is
// accumulated in slices, added in order in registers.
constexpr int TC_SLICE = 8;
constexpr uint32_t TC_MAX_POLLS = 1u << 22;
enum : uint32_t { ERR_TC_TIMEOUT = 8u };

struct TcProb {
  GemmArgs P;
  int a_mn, b_mn;    // 1: the operand's M (N) index is the contiguous one (KM / KN)
  int K2;            // > 0: a second product A2 B2^T over K2, summed in the same accumulator
  int tiles_m;       // tiles along M; the tile index runs over M first
  int tile0;         // first tile of this product in the launch's list
  float *colpart;    // column sums of the bf16 output over each 32 rows (or null): [row / 32][ldc]
  float *out;        // the output scaled by out_scale, without padding (or null): [M][out_n]
  int out_n;
  float out_scale;
};
struct TcArgs {
  int nprob, ntiles, bn;
  uint32_t *status;  // error word (bounded waits that expired)
  TcProb prob[TC_MAX_PROBS];
};
// operand maps of product i at 2 i (A), 2 i + 1 (B); a second operand pair (single products) at 2, 3
struct TcMaps {
  CUtensorMap m[2 * TC_MAX_PROBS];
};

constexpr int TC_STAGING_PITCH = 18;  // a warp's 32 x 16 chunk: 8-byte accesses, conflict-free writes
constexpr int TC_STAGING_FLOATS = 32 * TC_STAGING_PITCH;
// shared memory bytes of the kernel (stages, epilogue staging, barriers, 1024-byte alignment slack)
constexpr size_t TC_SMEM_BYTES =
    (size_t)TC_STAGES * TC_STAGE_BYTES + sizeof(float) * TC_STAGING_FLOATS * TC_EPI_WARPS + 1024 + 256;

// UMMA shared-memory matrix descriptor: start address, leading / stride byte
// offsets (16-byte units), descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// instruction descriptor of kind::f16: BF16 x BF16 -> F32, M = 256 (the pair), N = bn
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int a_mn, int b_mn, int bn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// cluster address of this shared-memory address in the CTA of the given rank
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// 2-D tensor load into this CTA's shared memory, completing on ``bar`` (a cluster address)
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  const uint32_t z = 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(z));
}

// arrives on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
  const uint16_t both = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_addr(bar)),
      "h"(both)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The tile of a launch's list: its product and coordinates.
struct TcTile {
  int i, mt, nt, nk1, nk;
  __device__ TcTile(const TcArgs &T, int t) {
    i = 0;
    while (i + 1 < T.nprob && t >= T.prob[i + 1].tile0) ++i;
    const TcProb &Q = T.prob[i];
    const int u = t - Q.tile0;
    nt = u / Q.tiles_m;
    mt = u - nt * Q.tiles_m;
    nk1 = (Q.P.K + TC_BK - 1) / TC_BK;
    nk = nk1 + (Q.K2 > 0 ? (Q.K2 + TC_BK - 1) / TC_BK : 0);
  }
};

// The epilogue of one warp: its 32 rows from m0 on, 16-column chunks part, part + 4,
// ... of the tile's bn columns from n0 on.  Each chunk goes TMEM -> registers
// (thread = row) -> shared memory -> registers (lane: two columns of rows lane / 8,
// + 4, ...), so global accesses are whole sectors, two values each.  The product's
// parameters are copied to registers before the loops: read from the parameter
// bank through a run-time index they cost more than the arithmetic (70 us per
// product against 10).
//   EPI none: Cf (+ bias), the scaled copy out; GELU: bias, pre_out, Cb; GELU': Cb
//   and its column sums over the warp's rows.
template <int EPI>
__device__ __forceinline__ void tc_epilogue(const TcProb &Q, int m0, int n0, int bn, int part, uint32_t taddr,
                                            float *stage, int lane) {
  const int M = Q.P.M, N = Q.P.N, ldc = Q.P.ldc, ldp = Q.P.ldp, out_n = Q.out_n;
  // (written by kernels that this one may overlap: coherent loads, __ldca, and not the
  // read-only path)
  const float *bias = Q.P.bias;
  const float *pre_in = Q.P.pre_in;
  float *__restrict__ pre_out = Q.P.pre_out;
  float *__restrict__ Cf = Q.P.Cf;
  __nv_bfloat16 *__restrict__ Cb = Q.P.Cb;
  float *__restrict__ out = Q.out;
  float *__restrict__ colpart = Q.colpart;
  const float oscale = Q.out_scale;
  const int cp = 2 * (lane & 7), rq = lane >> 3;  // column pair, row offset
  const bool full = m0 + 32 <= M;
#pragma unroll 1
  for (int c = part; c < bn / 16 && n0 + c * 16 < N; c += TC_EPI_WARPS / 4) {
    const int cn = n0 + c * 16 + cp;
    const bool in = cn < N;  // (N is even: both columns or neither)
    // the chunk's global inputs go out ahead of its TMEM read and the transpose
    float2 x[8];
    if (EPI == MG_EPI_DGELU) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = m0 + 4 * i + rq;
        x[i] = (in && (full || m < M)) ? __ldca(reinterpret_cast<const float2 *>(pre_in + (size_t)m * ldp + cn))
                                       : make_float2(0.f, 0.f);
      }
    }
    float2 bv = make_float2(0.f, 0.f);
    if (EPI != MG_EPI_DGELU && bias && in) bv = __ldca(reinterpret_cast<const float2 *>(bias + cn));
    uint32_t r[16];
    tmem_ld16(taddr + (uint32_t)(c * 16), r);
#pragma unroll
    for (int j = 0; j < 16; j += 2)
      *reinterpret_cast<float2 *>(stage + lane * TC_STAGING_PITCH + j) =
          make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
    __syncwarp();
    float2 csum = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + rq, m = m0 + row;
      float2 v = *reinterpret_cast<const float2 *>(stage + row * TC_STAGING_PITCH + cp);
      if (!in || !(full || m < M)) continue;
      const size_t o = (size_t)m * ldc + cn;
      if (EPI == MG_EPI_DGELU) {
        v.x *= gelu_grad_f(x[i].x);
        v.y *= gelu_grad_f(x[i].y);
      } else {
        v.x += bv.x;
        v.y += bv.y;
      }
      if (EPI == MG_EPI_GELU) {
        *reinterpret_cast<float2 *>(pre_out + (size_t)m * ldp + cn) = v;
        v.x = gelu_f(v.x);
        v.y = gelu_f(v.y);
      }
      if (EPI == MG_EPI_NONE) {
        *reinterpret_cast<float2 *>(Cf + o) = v;
        if (out) {
          if (cn < out_n) out[(size_t)m * out_n + cn] = v.x * oscale;
          if (cn + 1 < out_n) out[(size_t)m * out_n + cn + 1] = v.y * oscale;
        }
      } else {
        const __nv_bfloat162 q = __floats2bfloat162_rn(v.x, v.y);
        *reinterpret_cast<__nv_bfloat162 *>(Cb + o) = q;
        if (EPI == MG_EPI_DGELU) {
          const float2 f = __bfloat1622float2(q);
          csum.x += f.x;
          csum.y += f.y;
        }
      }
    }
    if (EPI == MG_EPI_DGELU) {
#pragma unroll
      for (int o = 8; o < 32; o <<= 1) {
        csum.x += __shfl_xor_sync(0xffffffffu, csum.x, o);
        csum.y += __shfl_xor_sync(0xffffffffu, csum.y, o);
      }
      if (rq == 0 && in && m0 < M) *reinterpret_cast<float2 *>(colpart + (size_t)(m0 / 32) * ldc + cn) = csum;
    }
    __syncwarp();
  }
}

// One warp's chunks of a tile whose K was accumulated in slices: tc_epilogue's chunks,
// held in registers while the slices are added, then stored.
struct TcSums {
  static constexpr int CHUNKS = TC_MAX_BN / 16 / (TC_EPI_WARPS / 4);
  float v[CHUNKS][16];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k)
#pragma unroll
      for (int j = 0; j < 16; ++j) v[k][j] = 0.f;
  }
  __device__ __forceinline__ void add(uint32_t taddr, int part, int bn) {
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = part + k * (TC_EPI_WARPS / 4);
      if (c >= bn / 16) break;
      uint32_t r[16];
      tmem_ld16(taddr + (uint32_t)(c * 16), r);
#pragma unroll
      for (int j = 0; j < 16; ++j) v[k][j] += __uint_as_float(r[j]);
    }
  }
  __device__ __forceinline__ void store(const TcProb &Q, int m0, int n0, int bn, int part, float *stage, int lane) const {
    const int M = Q.P.M, N = Q.P.N, ldc = Q.P.ldc;
    const int cp = 2 * (lane & 7), rq = lane >> 3;
    float *C = Q.P.Cf + (size_t)(m0 + rq) * ldc + n0 + cp;
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const int c = part + k * (TC_EPI_WARPS / 4);
      if (c >= bn / 16 || n0 + c * 16 >= N) break;
#pragma unroll
      for (int j = 0; j < 16; j += 2)
        *reinterpret_cast<float2 *>(stage + lane * TC_STAGING_PITCH + j) = make_float2(v[k][j], v[k][j + 1]);
      __syncwarp();
      const bool in = n0 + c * 16 + cp < N;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 x = *reinterpret_cast<const float2 *>(stage + (4 * i + rq) * TC_STAGING_PITCH + cp);
        if (in && m0 + 4 * i + rq < M) *reinterpret_cast<float2 *>(C + (size_t)(4 * i) * ldc + c * 16) = x;
      }
      __syncwarp();
    }
  }
};

// EPI: the products' epilogue (all of a launch have the same), or TC_EPI_SLICES: plain
// products accumulated TC_SLICE stages at a time.  A kernel each: with all in one body the
// sums in registers made the other epilogues spill (61.9 -> 65.0 us the forward pass).
constexpr int TC_EPI_SLICES = 3;
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
    tc_gemm_kernel(const __grid_constant__ TcMaps maps, const __grid_constant__ TcArgs T) {
  extern __shared__ __align__(1024) unsigned char tc_raw[];
  unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  float *staging = reinterpret_cast<float *>(sm + TC_STAGES * TC_STAGE_BYTES);
  uint64_t *full = reinterpret_cast<uint64_t *>(staging + TC_STAGING_FLOATS * TC_EPI_WARPS);
  uint64_t *empty = full + TC_STAGES;
  uint64_t *accfull = empty + TC_STAGES, *accempty = accfull + 2, *drained = accempty + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(drained + 1);
  dep_launch();
  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accfull[b], 1);
      mbar_init(&accempty[b], 2 * TC_EPI_WARPS);
    }
    mbar_init(drained, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync();  // both CTAs' barriers exist before either's loads, MMAs or arrivals
  tc_fence_after();
  dep_wait();
  const uint32_t tmem = *tslot;
  const int bn = T.bn, bh = bn / 2;
  bool ok = true;
  // the other lanes of the two role warps wait at the warp barrier (not in a
  // polling loop that would share the warp's issue slots with the role lane)
  if (warp == 0) {
    if (lane == 0) {
      // ---- TMA producer ----
      // (stage and phase run along: one thread's instructions are on the path of
      // every stage -- with a division by a run-time stage count they cost 0.2 us)
      int it = 0, s = 0;
      uint32_t phase = 1;  // parity of the hand-back before this use of the ring
      const uint32_t lead = cluster_addr(smem_addr(full), 0);
      for (int t = pair; ok && t < T.ntiles; t += npairs) {
        const TcTile X(T, t);
        const bool a_mn = T.prob[X.i].a_mn, b_mn = T.prob[X.i].b_mn;
        const int m0 = X.mt * TC_BM + (int)rank * TC_ROWS, n0 = X.nt * bn + (int)rank * bh;
        for (int kt = 0; kt < X.nk; ++kt, ++it) {
          if (it >= TC_STAGES && !mbar_wait(&empty[s], phase, TC_MAX_POLLS)) {
            ok = false;
            break;
          }
          unsigned char *sa = sm + s * TC_STAGE_BYTES, *sb = sa + TC_TILE_BYTES;
          if (rank == 0) mbar_expect_tx(&full[s], 2u * (uint32_t)(TC_TILE_BYTES + bh * TC_BK * 2));
          const uint32_t bar = lead + 8u * (uint32_t)s;
          const bool second = kt >= X.nk1;
          const CUtensorMap *ma = &maps.m[second ? 2 : 2 * X.i], *mb = ma + 1;
          const int k0 = (second ? kt - X.nk1 : kt) * TC_BK;
          if (a_mn) {
            tma_load_2d(sa, ma, m0, k0, bar);
            tma_load_2d(sa + TC_TILE_BYTES / 2, ma, m0 + 64, k0, bar);
          } else {
            tma_load_2d(sa, ma, k0, m0, bar);
          }
          if (b_mn) {
            for (int h = 0; h < bh; h += 64) tma_load_2d(sb + h * TC_BK * 2, mb, n0 + h, k0, bar);
          } else {
            tma_load_2d(sb, mb, k0, n0, bar);
          }
          if (++s == TC_STAGES) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
      // the last stages' hand-backs have arrived before the CTA may end
      for (int k = max(0, it - TC_STAGES); ok && k < it; ++k)
        ok = mbar_wait(&empty[k % TC_STAGES], (uint32_t)(k / TC_STAGES) & 1u, TC_MAX_POLLS);
      // a wait that expired: its loads may still be landing (a load takes microseconds)
      if (!ok)
        for (int k = 0; k < 1000; ++k) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // ---- MMA issuer ----
      int n = 0, s = 0;
      uint32_t phase = 0;
      for (int t = pair; ok && t < T.ntiles; t += npairs) {
        const TcTile X(T, t);
        const int a_mn = T.prob[X.i].a_mn, b_mn = T.prob[X.i].b_mn;
        const uint32_t idesc = umma_idesc_bf16(a_mn, b_mn, bn);
        // K-major: 16 elements = 32 bytes along the swizzled row; MN-major: 16 rows of 128
        // bytes (descriptor addresses count 16 bytes)
        const uint64_t da0 = umma_desc_sw128(smem_addr(sm), a_mn ? TC_TILE_BYTES / 2 : 16, 1024);
        const uint64_t db0 = umma_desc_sw128(smem_addr(sm) + TC_TILE_BYTES, b_mn ? TC_TILE_BYTES / 2 : 16, 1024);
        const uint32_t ka = a_mn ? 128 : 2, kb = b_mn ? 128 : 2;
        // (n counts slices: each takes the other accumulator)
        const int ks = EPI == TC_EPI_SLICES ? TC_SLICE : X.nk;
        for (int k0 = 0; ok && k0 < X.nk; k0 += ks, ++n) {
          const uint32_t acc = tmem + (uint32_t)(n & 1) * TC_MAX_BN;
          if (n >= 2 && !mbar_wait(&accempty[n & 1], (uint32_t)(n / 2 - 1) & 1u, TC_MAX_POLLS)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int k1 = min(X.nk, k0 + ks);
          for (int kt = k0; kt < k1; ++kt) {
            if (!mbar_wait(&full[s], phase, TC_MAX_POLLS)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t off = (uint64_t)(s * (TC_STAGE_BYTES / 16));
#pragma unroll
            for (int k = 0; k < TC_BK / 16; ++k)
              umma_bf16(acc, da0 + off + k * ka, db0 + off + k * kb, idesc, (kt > k0 || k > 0) ? 1u : 0u);
            umma_commit_pair(&empty[s]);
            if (++s == TC_STAGES) {
              s = 0;
              phase ^= 1u;
            }
          }
          if (ok) umma_commit_pair(&accfull[n & 1]);
        }
      }
      umma_commit_pair(drained);
    }
    __syncwarp();
  } else {
    // ---- epilogue ----
    const int quad = warp & 3, part = (warp - 2) >> 2;
    float *stage = staging + (warp - 2) * TC_STAGING_FLOATS;
    int n = 0;
    // the accumulator of slice n is finished; its columns of this warp's lanes
    auto finished = [&]() {
      ok = mbar_wait(&accfull[n & 1], (uint32_t)(n / 2) & 1u, TC_MAX_POLLS);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      return tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(n & 1) * TC_MAX_BN;
    };
    auto hand_back = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_addr(&accempty[n & 1]), 0));
      ++n;
    };
    for (int t = pair; ok && t < T.ntiles; t += npairs) {
      const TcTile X(T, t);
      const TcProb &Q = T.prob[X.i];
      const int m0 = X.mt * TC_BM + (int)rank * TC_ROWS + quad * 32, n0 = X.nt * bn;
      if constexpr (EPI == TC_EPI_SLICES) {
        TcSums sums;
        sums.clear();
        for (int k0 = 0; k0 < X.nk; k0 += TC_SLICE) {
          const uint32_t taddr = finished();
          if (!ok) break;
          sums.add(taddr, part, bn);
          hand_back();
        }
        if (ok) sums.store(Q, m0, n0, bn, part, stage, lane);
      } else {
        const uint32_t taddr = finished();
        if (!ok) break;
        tc_epilogue<EPI>(Q, m0, n0, bn, part, taddr, stage, lane);
        hand_back();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {  // every MMA that was issued has completed, also where a wait above has expired
    if (lane == 0) ok = mbar_wait(drained, 0, TC_MAX_POLLS) && ok;
    __syncwarp();
  }
  cluster_sync();  // the pair's MMAs, loads and arrivals are done (or its bounded waits have expired)
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  if (!ok && lane == 0 && T.status) atomicOr(T.status, (uint32_t)ERR_TC_TIMEOUT);
}

}  // namespace aob
