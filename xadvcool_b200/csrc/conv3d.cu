// 3-D convolutions of the warm-start surrogate as BF16 tensor-core implicit GEMMs with FP32 accumulation.
//
// Layout: activations channels-last, x fastest: act[n][z][y][x][c] (BF16); weights w[tap][co][ci] (BF16,
// ci fastest), tap = (dz+1)*9 + (dy+1)*3 + (dx+1) for a 3x3x3 kernel (tap 0 only for 1x1x1); zero padding.
//
//   forward   out[v][co] = act( bias[co] + sum_{tap,ci} w[tap][co][ci] * in[v + off(tap)][ci] )
//             GEMM M = voxels, N = Co, K = taps * Ci, on tcgen05 (128 voxels x Co per CTA, accumulator in TMEM).
//   data grad the forward kernel applied to d_out with the flipped, transposed weights
//             w'[26 - tap][ci][co] = w[tap][co][ci] (the adjoint of a zero-padded convolution).
//   weight grad dw[tap][co][ci] = sum_v d_out[v][co] * in[v + off(tap)][ci]
//             GEMM M = taps * Co, N = Ci, K = voxels on tcgen05, split over voxel chunks; partials reduced in a
//             fixed order.
//
// Ci and Co must be multiples of 16 (the model pads its 3 input channels and 5 output channels to 16).
#include <cuda.h>
#include <cuda_bf16.h>

#include <array>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>

#include "xac_internal.cuh"

namespace xac {
namespace {

struct ConvShape {
  int N, D, H, W;  // batch, z, y, x
  int Ci, Co;
  int ksize;  // 1 or 3
};



__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

// ---- shared pieces of the tcgen05 kernels ----------------------------------------------------------------
constexpr int kTcM = 128;
constexpr uint32_t kTcSpin = 1u << 22;
__device__ unsigned int g_conv_status;  // bit 0: a wait ran out

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = kTcSpin) {
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  atomicOr(&g_conv_status, 1u);
  return false;
}
// bounded wait that also ends when another role of the CTA gave up; one that runs out raises the CTA's abort flag
__device__ __forceinline__ bool mbar_wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_v) {
  for (uint32_t i = 0; i < kTcSpin; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (*abort_v) return false;
  }
  atomicOr(&g_conv_status, 1u);
  *abort_v = 1;
  return false;
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// tiled TMA loads: the innermost coordinate is a multiple of 16 channels (32 bytes); boxes may start or end outside
// the tensor, where they read zeros
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], "
      "[%7];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: no swizzle (layout type 0 in bits 61..63), descriptor version 1
constexpr uint32_t kSwizzle128 = 2, kSwizzle64 = 4, kSwizzle32 = 6;
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both K-major, N = n, M = 128
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcM >> 4) << 24);
}
// a, b: descriptors as low and high words
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                       uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %6, 0;\n\tmov.b64 a, {%1, %2};\n\t"
      "mov.b64 b, {%3, %4};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}"
      ::"r"(tmem_d), "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accum));
}
// one lane of a converged warp, the same one each time; the compiler then knows that the code under it runs in a
// single thread and keeps the MMA operands in uniform registers without a loop around every instruction
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- forward / data grad on the 5th-generation tensor cores (tcgen05) ------------------------------------
// Bound: for Co <= 64 the tensor core's reads of the activation operand from shared memory (4 KB per 128 voxels x 16
// channels: 39 cycles an MMA for Co = 16, 48 for 64, where the products alone would take 8 and 32). The kernel
// before this one copied that operand from L2 once per tap, one 16-byte copy per thread, and one thread issued its
// MMAs from a loop. Here a plane of input voxels with its halo is copied once and the 27 taps read it in place:
//
//   * A unit of work is a tile of bx x by voxels of one z plane (x Co, or a slice of nb channels of it). Its input is
//     three z planes of by + 2 rows of P = bx + 2 voxels; TMA boxes fill the part outside the volume with zeros.
//   * A plane lies in shared memory as Ci / KB blocks of [R voxels][KB channels] (K-major, swizzle of the row size:
//     KB = 64, 32, 16 channels are 128, 64, 32 bytes), so the A operand of tap (dz,dy,dx) is the plane's rows
//     m + dy*P + dx, m = y*P + x: the same bytes from another start address.
//   * The accumulator rows m run over the flattened tile, mt blocks of 128 rows; rows with x >= bx are halo columns
//     and are dropped by the epilogue (2 of P).
//   * A CTA walks a contiguous range of units, z fastest. When its planes are kept (march) a plane is copied once
//     for the three units that read it, into a ring of NS planes; the tap order has dz outermost, so the oldest
//     plane is free after the first third of a unit and the next one is on its way during the rest.
//   * Weights: all of them resident where they fit beside the planes, otherwise a ring of stages of one tap (all of its
//     channels where Ci / KB is at most 3, else KB of them).
//
// The products of an output are added in the order tap, then channel, whatever the tile.
//
// Measured on a B200, the kernel before -> this one (same bits): 16 -> 16 channels at 32x128x152 217 -> 35 us, at batch 4
// 808 -> 113 (the MMAs alone 77), 48 -> 16 2203 -> 270, 96 -> 32 at 16x64x76 755 -> 131, 192 -> 64 at 8x32x38 357 -> 74.
//
// Roles: warps 0-15 epilogue, 16-19 issue the MMAs (warp 16 + k those of the accumulator blocks k, k + 4, ...), 20
// copies input planes and 21 weights. Accumulators are double-buffered in tensor memory where they fit, so the epilogue
// of a unit runs under the MMAs of the next.
// Every wait is bounded: a wait that runs out sets g_conv_status and the CTA's abort flag, every role leaves its
// loop, and the CTA waits (bounded) for its copies and MMAs in flight, frees its tensor memory and returns.
constexpr int kFwdThreads = 704;
constexpr int kEpiWarps = 16;
constexpr int kMmaWarps = 4;
constexpr int kMaxPlanes = 4;
constexpr int kMaxBStages = 8;

struct FwdPlan {
  int bx, by, P, nxt, nyt;  // tile, row length with halo, tiles along x and y
  int mt, R;                // blocks of 128 accumulator rows; voxels of a stored plane
  int NS, march;            // planes in the ring; 1: planes are kept from one z to the next
  int nb, nsplit;           // output channels of a unit, slices of Co
  int KB, G;                // channels of a block, blocks of a weight stage
  int bs, resident;         // weight stages held, 1: all weights held
  int nbuf;                 // accumulator buffers
  uint32_t ncols;           // tensor-memory columns allocated
  long long units;
  int ctas;
  size_t smem;
};

// barriers, by number
struct FwdBars {
  uint32_t b0;
  __device__ __forceinline__ uint32_t afull(int i) const { return b0 + 8u * i; }
  __device__ __forceinline__ uint32_t aempty(int i) const { return b0 + 8u * (kMaxPlanes + i); }
  __device__ __forceinline__ uint32_t bfull(int i) const { return b0 + 8u * (2 * kMaxPlanes + i); }
  __device__ __forceinline__ uint32_t bempty(int i) const { return b0 + 8u * (2 * kMaxPlanes + kMaxBStages + i); }
  __device__ __forceinline__ uint32_t cfull(int i) const { return b0 + 8u * (2 * kMaxPlanes + 2 * kMaxBStages + i); }
  __device__ __forceinline__ uint32_t cempty(int i) const {
    return b0 + 8u * (2 * kMaxPlanes + 2 * kMaxBStages + 2 + i);
  }
  __device__ __forceinline__ uint32_t done() const { return b0 + 8u * (2 * kMaxPlanes + 2 * kMaxBStages + 4); }
  static constexpr int kCount = 2 * kMaxPlanes + 2 * kMaxBStages + 5;
};

struct MmaRole {
  uint32_t tmem;
  uint32_t a, b, hi;           // descriptors of the first plane and weight stage (low words), their high word
  uint32_t plane16, bblk16;    // sizes of a plane and of a weight block in 16-byte units
  FwdBars bar;
  int nd, nst, taps;           // stages of a tap
  volatile int* abort_v;
};

// KC steps of 16 channels (32 bytes apart) for NT accumulator blocks; a, b: low words of the descriptors
template <int KC, int NT>
__device__ __forceinline__ void issue_stage(uint32_t d, uint32_t dstep, uint32_t a, uint32_t b, uint32_t hi,
                                            uint32_t idesc, uint32_t accum) {
  constexpr uint32_t kBlock = kMmaWarps * kTcM * KC * 2;  // four blocks of 128 rows of KC * 32 bytes, in 16 bytes
#pragma unroll
  for (int c = 0; c < KC; ++c)
#pragma unroll
    for (int t = 0; t < NT; ++t)
      tc_mma(d + (uint32_t)t * dstep, a + (uint32_t)(2 * c) + (uint32_t)t * kBlock, hi, b + (uint32_t)(2 * c), hi, idesc,
             c == 0 ? accum : 1u);
}

// one weight stage: G blocks of KC steps; ablk, bblk: distances of the blocks
template <int KC, int G, int NT>
__device__ __forceinline__ void issue_tap(uint32_t d, uint32_t dstep, uint32_t a, uint32_t ablk, uint32_t b,
                                          uint32_t bblk, uint32_t hi, uint32_t idesc, uint32_t accum) {
#pragma unroll
  for (int g = 0; g < G; ++g)
    issue_stage<KC, NT>(d, dstep, a + (uint32_t)g * ablk, b + (uint32_t)g * bblk, hi, idesc, g == 0 ? accum : 1u);
}

// The MMAs of one warp over the CTA's units (the whole warp waits, one lane issues). An MMA in a loop of its own
// costs its thread 180-250 cycles, in straight-line code 45-120, so the taps of a plane (or of a row of it) are
// unrolled where the weights are resident, and four warps issue side by side.
template <int KC, int G, int NT>
__device__ __forceinline__ void mma_role(const MmaRole& m, const ConvShape& s, const FwdPlan& pl, int t0, int issuer,
                                         long long u_begin, long long u_end) {
  constexpr uint32_t kRow = KC * 2;  // a voxel's row in 16-byte units
  const int nb = pl.nb, P = pl.P, D = s.D, nd = m.nd, nst = m.nst;
  const uint32_t idesc = tc_idesc(nb);
  const uint32_t abase = m.a + (uint32_t)(t0 * kTcM) * kRow, ablk = (uint32_t)pl.R * kRow;
  const uint32_t bblk = pl.resident ? (uint32_t)m.taps * m.bblk16 : m.bblk16;
  const uint32_t dstep = (uint32_t)(kMmaWarps * nb);
  int seq0 = 0, cnt = 0, st = 0;
  uint32_t bpar = 0;
  if (pl.resident) {
    if (!mbar_wait_or_abort(m.bar.bfull(0), 0, m.abort_v)) return;
    tc_fence_after();
  }
  for (long long u = u_begin; u < u_end;) {
    const int z0 = (int)(u % D);
    const int nz = (int)((u_end - u < D - z0) ? u_end - u : D - z0);
    for (int i = 0; i < nz; ++i, ++cnt) {
      const int buf = cnt % pl.nbuf;
      if (cnt >= pl.nbuf && !mbar_wait_or_abort(m.bar.cempty(buf), ((cnt / pl.nbuf) - 1) & 1, m.abort_v)) return;
      tc_fence_after();
      const uint32_t acc = m.tmem + (uint32_t)((buf * pl.mt + t0) * nb);
      for (int dz = 0; dz < nd; ++dz) {
        const int sq = seq0 + (pl.march ? i + dz : i * nd + dz), slot = sq % pl.NS;
        if (!mbar_wait_or_abort(m.bar.afull(slot), (sq / pl.NS) & 1, m.abort_v)) return;
        tc_fence_after();
        const uint32_t arow = abase + (uint32_t)slot * m.plane16;
        if (pl.resident && nst == 1 && nd == 3) {
          if (issuer) {
            constexpr int kRows = KC * G * NT <= 4 ? 3 : 1;  // rows of taps in one straight run
#pragma unroll 1
            for (int dy0 = 0; dy0 < 3; dy0 += kRows) {
#pragma unroll
              for (int k = 0; k < 3 * kRows; ++k) {
                const int dy = dy0 + k / 3, dx = k % 3;
                issue_tap<KC, G, NT>(acc, dstep, arow + (uint32_t)(dy * P + dx) * kRow, ablk,
                                     m.b + (uint32_t)(dz * 9 + dy * 3 + dx) * m.bblk16, bblk, m.hi, idesc,
                                     (dz > 0 || dy > 0 || dx > 0) ? 1u : 0u);
              }
            }
          }
        } else {
          for (int dyx = 0; dyx < nd * nd; ++dyx) {
            const uint32_t a = arow + (uint32_t)(dyx / nd * P + dyx % nd) * kRow;
            for (int k = 0; k < nst; ++k) {
              if (!pl.resident) {
                if (!mbar_wait_or_abort(m.bar.bfull(st), bpar, m.abort_v)) return;
                tc_fence_after();
              }
              if (issuer) {
                const int blk = pl.resident ? k * G * m.taps + dz * nd * nd + dyx : st * G;
                issue_tap<KC, G, NT>(acc, dstep, a + (uint32_t)(k * G) * ablk, ablk,
                                     m.b + (uint32_t)blk * m.bblk16, bblk, m.hi, idesc,
                                     (dz > 0 || dyx > 0 || k > 0) ? 1u : 0u);
                if (!pl.resident) tc_commit(m.bar.bempty(st));
              }
              if (++st == pl.bs) {
                st = 0;
                bpar ^= 1u;
              }
            }
          }
        }
        if (issuer && (!pl.march || dz == 0 || i == nz - 1)) tc_commit(m.bar.aempty(slot));
        __syncwarp();
      }
      if (issuer) tc_commit(m.bar.cfull(buf));
      __syncwarp();
    }
    seq0 += pl.march ? nz + nd - 1 : nz * nd;
    u += nz;
  }
}

// strip = (slice of Co, batch item, y tile, x tile)
struct Strip {
  int n0, n, y0, x0;
};
__device__ __forceinline__ Strip strip_of(long long strip, const FwdPlan& pl, const ConvShape& s) {
  Strip t;
  unsigned v = (unsigned)strip;
  t.x0 = (int)(v % pl.nxt) * pl.bx;
  v /= pl.nxt;
  t.y0 = (int)(v % pl.nyt) * pl.by;
  v /= pl.nyt;
  t.n = (int)(v % s.N);
  t.n0 = (int)(v / s.N) * pl.nb;
  return t;
}

__global__ void __launch_bounds__(kFwdThreads, 1) conv_fwd_kernel(const __grid_constant__ CUtensorMap tin,
                                                                  const __grid_constant__ CUtensorMap tw,
                                                                  const float* __restrict__ bias, ConvShape s, int act,
                                                                  FwdPlan pl, __nv_bfloat16* __restrict__ out_bf16,
                                                                  float* __restrict__ out_f32) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[FwdBars::kCount];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int Co = s.Co, kr = s.ksize >> 1, nd = s.ksize, taps = nd * nd * nd, nb = pl.nb, P = pl.P, D = s.D;
  const int nkc = s.Ci / pl.KB;
  const int nmw = pl.mt < kMmaWarps ? pl.mt : kMmaWarps;  // warps that issue MMAs
  const uint32_t row_bytes = (uint32_t)pl.KB * 2u;
  const uint32_t plane_bytes = (uint32_t)nkc * pl.R * row_bytes, bblk_bytes = (uint32_t)nb * row_bytes;
  const uint32_t bstage_bytes = (uint32_t)pl.G * bblk_bytes;
  const uint32_t a0 = smem_addr(smem), b0 = a0 + pl.NS * plane_bytes;
  const FwdBars bar{smem_addr(bars)};

  if (tid == 0) {
    for (int i = 0; i < kMaxPlanes; ++i) {
      mbar_init(bar.afull(i), 1);
      mbar_init(bar.aempty(i), nmw);
    }
    for (int i = 0; i < kMaxBStages; ++i) {
      mbar_init(bar.bfull(i), 1);
      mbar_init(bar.bempty(i), nmw);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar.cfull(i), nmw);
      mbar_init(bar.cempty(i), 32 * kEpiWarps);
    }
    mbar_init(bar.done(), nmw);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                 "r"(pl.ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abort_v = &abort_flag;
  const long long u_begin = pl.units * blockIdx.x / gridDim.x, u_end = pl.units * (blockIdx.x + 1) / gridDim.x;

  if (warp == kEpiWarps + kMmaWarps) {
    // ---- input planes: one thread starts the boxes of a plane, one per block of KB channels
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)nkc * (uint32_t)(P * (pl.by + 2 * kr)) * row_bytes;
      int slot = 0, seq = 0;
      uint32_t par = 1;  // parity of the wait for room: passes at once in the first round
      auto load_plane = [&](const Strip& t, int z) -> bool {
        if (!mbar_wait_or_abort(bar.aempty(slot), par, abort_v)) return false;
        mbar_expect_tx(bar.afull(slot), bytes);
        for (int k = 0; k < nkc; ++k)
          tma_load_5d(a0 + (uint32_t)slot * plane_bytes + (uint32_t)(k * pl.R) * row_bytes, &tin, k * pl.KB, t.x0 - kr,
                      t.y0 - kr, z, t.n, bar.afull(slot));
        ++seq;
        if (++slot == pl.NS) {
          slot = 0;
          par ^= 1u;
        }
        return true;
      };
      bool ok = true;
      for (long long u = u_begin; ok && u < u_end;) {
        const long long strip = u / D;
        const int z0 = (int)(u - strip * D);
        const int nz = (int)((u_end - u < D - z0) ? u_end - u : D - z0);
        const Strip t = strip_of(strip, pl, s);
        if (pl.march) {
          for (int i = 0; ok && i < nz + 2 * kr; ++i) ok = load_plane(t, z0 - kr + i);
        } else {
          for (int z = z0; ok && z < z0 + nz; ++z)
            for (int d = 0; ok && d < nd; ++d) ok = load_plane(t, z - kr + d);
        }
        u += nz;
      }
      // an abort may leave copies that no role waits for: each lands before the block's memory goes back
      for (int k = seq > pl.NS ? seq - pl.NS : 0; k < seq; ++k) mbar_wait(bar.afull(k % pl.NS), (k / pl.NS) & 1);
    }
  } else if (warp == kEpiWarps + kMmaWarps + 1) {
    // ---- weights: all of them at once, or the stages of one unit again and again (with the unit's slice of Co)
    if (lane == 0) {
      if (pl.resident) {
        mbar_expect_tx(bar.bfull(0), (uint32_t)(taps * nkc) * bblk_bytes);
        for (int k = 0; k < nkc; ++k)
          tma_load_3d(b0 + (uint32_t)(k * taps) * bblk_bytes, &tw, k * pl.KB, 0, 0, bar.bfull(0));
        mbar_wait(bar.bfull(0), 0);
      } else {
        int st = 0;
        long long seq = 0;
        uint32_t par = 1;
        bool ok = true;
        for (long long u = u_begin; ok && u < u_end; ++u) {
          const Strip t = strip_of(u / D, pl, s);
          for (int tap = 0; ok && tap < taps; ++tap)
            for (int k = 0; k < nkc; k += pl.G) {
              if (!mbar_wait_or_abort(bar.bempty(st), par, abort_v)) {
                ok = false;
                break;
              }
              mbar_expect_tx(bar.bfull(st), bstage_bytes);
              for (int g = 0; g < pl.G; ++g)
                tma_load_3d(b0 + (uint32_t)st * bstage_bytes + (uint32_t)g * bblk_bytes, &tw, (k + g) * pl.KB, t.n0, tap,
                            bar.bfull(st));
              ++seq;
              if (++st == pl.bs) {
                st = 0;
                par ^= 1u;
              }
            }
        }
        for (long long k = seq > pl.bs ? seq - pl.bs : 0; k < seq; ++k)
          mbar_wait(bar.bfull((int)(k % pl.bs)), (uint32_t)(k / pl.bs) & 1u);
      }
    }
  } else if (warp >= kEpiWarps) {
    // ---- MMA issue: accumulator blocks t0, t0 + 4, ...
    const int t0 = warp - kEpiWarps;
    if (t0 < nmw) {
      const uint64_t desc = smem_desc(0, 16u, 8u * row_bytes) |
                            ((uint64_t)(pl.KB == 64 ? kSwizzle128 : (pl.KB == 32 ? kSwizzle64 : kSwizzle32)) << 61);
      const uint32_t dlo = (uint32_t)desc, dhi = (uint32_t)(desc >> 32);
      const MmaRole m{tmem, dlo + (a0 >> 4), dlo + (b0 >> 4), dhi, plane_bytes >> 4, bblk_bytes >> 4, bar, nd,
                      nkc / pl.G, taps, abort_v};
      const int nt = (pl.mt - t0 + kMmaWarps - 1) / kMmaWarps, kc = pl.KB >> 4;
      const int issuer = elect_one() ? 1 : 0;
#define XAC_ROLE(KC, GG)                                                    \
  if (kc == KC && pl.G == GG) {                                             \
    if (nt == 1) mma_role<KC, GG, 1>(m, s, pl, t0, issuer, u_begin, u_end); \
    else mma_role<KC, GG, 2>(m, s, pl, t0, issuer, u_begin, u_end);         \
  }
      XAC_ROLE(1, 1) XAC_ROLE(2, 1) XAC_ROLE(4, 1) XAC_ROLE(1, 3) XAC_ROLE(2, 3) XAC_ROLE(4, 2) XAC_ROLE(4, 3)
#undef XAC_ROLE
      // arrives when every MMA issued has finished
      if (issuer) tc_commit(bar.done());
    }
  } else {
    // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4)..; blocks x 16-column groups go round the warps
    int cnt = 0;
    const int quad = warp & 3;
    for (long long u = u_begin; u < u_end; ++u, ++cnt) {
      const int buf = cnt % pl.nbuf;
      if (!mbar_wait_or_abort(bar.cfull(buf), (cnt / pl.nbuf) & 1, abort_v)) break;
      tc_fence_after();
      const long long strip = u / D;
      const int z = (int)(u - strip * D);
      const Strip t = strip_of(strip, pl, s);
      const int groups = nb >> 4;
      for (int it = warp >> 2; it < pl.mt * groups; it += kEpiWarps / 4) {
        const int b = it / groups, c0 = (it - b * groups) << 4;
        const int m = b * kTcM + quad * 32 + lane;
        const int y = m / P, x = m - y * P;
        const int gy = t.y0 + y, gx = t.x0 + x;
        const bool valid = x < pl.bx && y < pl.by && gy < s.H && gx < s.W;
        const long long o = ((((long long)t.n * D + z) * s.H + gy) * s.W + gx) * Co + t.n0;
        {
          float v[16];
          __syncwarp();
          tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((buf * pl.mt + b) * nb + c0), v);
          if (!valid) continue;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float yv = v[i] + (bias ? __ldg(bias + t.n0 + c0 + i) : 0.0f);
            v[i] = act == 1 ? gelu(yv) : yv;
          }
          if (out_bf16) {
            uint4 pk[2];
            uint32_t* pw = reinterpret_cast<uint32_t*>(pk);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
              pw[i] = *reinterpret_cast<uint32_t*>(&b2);
            }
            uint4* dst = reinterpret_cast<uint4*>(out_bf16 + o + c0);
            dst[0] = pk[0];
            dst[1] = pk[1];
          } else {
            float4* dst = reinterpret_cast<float4*>(out_f32 + o + c0);
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          }
        }
      }
      tc_fence_before();
      mbar_arrive(bar.cempty(buf));
    }
  }
  // Every MMA issued has finished before the tensor memory goes back. The warps that work to the end wait on done, so its
  // limit counts from the end of their own work; those that are idle or end early stand at the barrier, where a long launch
  // is no failure. (With the MMA warps alone on done: 16 -> 16 channels at 32x128x152 34.93 us, against 34.83.)
  __syncwarp();
  if (warp < kEpiWarps + nmw) mbar_wait(bar.done(), 0);
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(pl.ncols));
  }
}

// ---- weight grad on the tensor cores (tcgen05) --------------------------------------------------------
// dw[tap][co][ci] = sum_v d_out[v][co] * in[v + off(tap)][ci]: GEMMs with K = voxels. Bound: the operands' reads from
// shared memory (32 bytes per M row and per N column for 16 voxels, 128 B/clk). The kernel before this one gathered d_out
// from L2 once per tap and voxel; here a tile of d_out and its input planes are copied once by TMA, and every tap is
// another start address in them:
//
//   * A unit is a tile of bx x by voxels of one z plane, as in the forward kernel: d_out's rows r = y*P + x (P = bx + 2;
//     the two columns after the tile and the rows around it are zeros), the input's three planes with their halo. Both lie
//     in shared memory as [rows][KB channels] with the row-size swizzle, which is the MN-major layout with K = rows.
//   * MMA step: 16 rows. B holds the three dy taps of a block of KBx input channels: N groups P rows apart, N = 3 KBx.
//     A holds up to three dx taps: M groups of KBd output channels one row apart (D[k + g] against X[k + s] is tap dx =
//     s - g), so 16 output channels fill M = 64 and 32 fill M = 128; 64 channels take two dx taps in M = 128 and the third
//     in M = 64; more take one.
//   * One accumulator of a (dz, dx set) is an `Au`. blockIdx.y selects a set of them that fits the 512 columns,
//     blockIdx.z the block of input channels and of at most 128 output channels, blockIdx.x a range of units.
//   * Rounding: an accumulator takes at most 256 steps (4096 rows) before it is added, in FP32 on the CUDA cores, to the
//     CTA's partial in global memory (the tensor core's own additions truncate); wgrad_reduce_kernel adds the partials
//     of the CTAs in a fixed order.
//
// Measured on a B200 with the reductions and db, the kernels before -> these, batch 4: 16 -> 16 channels at 32x128x152
// 1327 -> 97 us, 48 -> 16 1777 -> 215, 32 -> 32 at 16x64x76 428 -> 43, 192 -> 64 at 8x32x38 259 -> 62; relative error against
// 64-bit sums 4.8e-6 -> 4.0e-6, 4.7e-6 -> 4.2e-6, 4.7e-6 -> 2.4e-6, 4.2e-6 -> 2.6e-6.
//
// Roles: warps 0-7 epilogue, 8-11 MMAs (Au a on warp 8 + a % 4), 12 copies. Waits are bounded as in the forward kernel.
constexpr int kWgThreads = 416;
constexpr int kWgEpiWarps = 8;
constexpr int kWgMaxSteps = 256;  // MMA steps of an accumulator before it is flushed
constexpr int kWgMaxAu = 9;
constexpr int kWgLead = 8;  // zero rows before d_out's tile

struct Au {
  int dz;   // plane
  int M;    // 64 or 128
  int dx0;  // dx tap of M group 0; group g is dx0 - g
  int ndx;  // dx taps held
};
struct WgPlan {
  int bx, by, P, nxt, nyt;
  int rows_mode;  // 1: d_out is copied row by row (the tile is narrower than the volume: its halo stays zero)
  int RX, RD;     // rows of a stored input plane / d_out tile block
  int NX, march;  // input planes in the ring; 1: kept from one z to the next
  int KBx, KBd, cb, nblk, mblk;  // channels of a block; output channels of a CTA; blocks of Ci; of Co
  int nstack;     // dy taps in N
  int nau, ngr, first[kWgMaxAu + 1];
  Au au[kWgMaxAu];
  int nsteps, upc, nbuf;  // steps of a unit, units of an accumulation, accumulator buffers
  uint32_t ncols;
  long long units;
  int ctas;
  size_t smem;
};

struct WgBars {
  uint32_t b0;
  __device__ __forceinline__ uint32_t xfull(int i) const { return b0 + 8u * i; }
  __device__ __forceinline__ uint32_t xempty(int i) const { return b0 + 8u * (kMaxPlanes + i); }
  __device__ __forceinline__ uint32_t dfull(int i) const { return b0 + 8u * (2 * kMaxPlanes + i); }
  __device__ __forceinline__ uint32_t dempty(int i) const { return b0 + 8u * (2 * kMaxPlanes + 2 + i); }
  __device__ __forceinline__ uint32_t cfull(int i) const { return b0 + 8u * (2 * kMaxPlanes + 4 + i); }
  __device__ __forceinline__ uint32_t cempty(int i) const { return b0 + 8u * (2 * kMaxPlanes + 6 + i); }
  __device__ __forceinline__ uint32_t done() const { return b0 + 8u * (2 * kMaxPlanes + 8); }
  static constexpr int kCount = 2 * kMaxPlanes + 9;
};

__host__ __device__ constexpr uint32_t swizzle_of(int kb) {
  return kb == 64 ? kSwizzle128 : (kb == 32 ? kSwizzle64 : kSwizzle32);
}

__global__ void __launch_bounds__(kWgThreads, 1) conv_wgrad_kernel(const __grid_constant__ CUtensorMap tin,
                                                                   const __grid_constant__ CUtensorMap tdo, ConvShape s,
                                                                   const __grid_constant__ WgPlan pl,
                                                                   float* __restrict__ partial) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t bars[WgBars::kCount];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int kr = s.ksize >> 1, nd = s.ksize, taps = nd * nd * nd, P = pl.P, D = s.D;
  const int blk = blockIdx.z % pl.nblk, m0 = (int)(blockIdx.z / pl.nblk) * 128;
  const int cb = s.Co - m0 < pl.cb ? s.Co - m0 : pl.cb, ndb = cb / pl.KBd;  // this CTA's output channels, in blocks
  const int au0 = pl.first[blockIdx.y], au1 = pl.first[blockIdx.y + 1];
  const int dlo = pl.au[au0].dz, ndz = pl.au[au1 - 1].dz - dlo + 1;  // planes used
  const int N = pl.KBx * pl.nstack, naus = au1 - au0;
  const int nmw = naus < kMmaWarps ? naus : kMmaWarps;
  const uint32_t xrow = (uint32_t)pl.KBx * 2u, drow = (uint32_t)pl.KBd * 2u;
  const uint32_t dslot = (uint32_t)(pl.cb / pl.KBd) * pl.RD * drow, xslot = (uint32_t)pl.RX * xrow;
  const uint32_t d0 = smem_addr(smem), x0 = d0 + 2u * dslot;
  const WgBars bar{smem_addr(bars)};

  // rows that no copy writes (before, between and after the tiles) are read against zeros: they must be finite
  for (uint32_t i = tid * 16u; i < (uint32_t)pl.smem; i += kWgThreads * 16u)
    *reinterpret_cast<uint4*>(smem + i) = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async();
  if (tid == 0) {
    for (int i = 0; i < kMaxPlanes; ++i) {
      mbar_init(bar.xfull(i), 1);
      mbar_init(bar.xempty(i), nmw);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar.dfull(i), 1);
      mbar_init(bar.dempty(i), nmw);
      mbar_init(bar.cfull(i), nmw);
      mbar_init(bar.cempty(i), 32 * kWgEpiWarps);
    }
    mbar_init(bar.done(), nmw);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                 "r"(pl.ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abort_v = &abort_flag;
  const long long u_begin = pl.units * blockIdx.x / gridDim.x, u_end = pl.units * (blockIdx.x + 1) / gridDim.x;
  // unit = ((n * nyt + y tile) * nxt + x tile) * D + z
  struct Tile {
    int n, y0, x0;
  };
  auto tile_of = [&](long long strip) {
    Tile t;
    unsigned v = (unsigned)strip;
    t.x0 = (int)(v % pl.nxt) * pl.bx;
    v /= pl.nxt;
    t.y0 = (int)(v % pl.nyt) * pl.by;
    t.n = (int)(v / pl.nyt);
    return t;
  };

  if (warp == kWgEpiWarps + kMmaWarps) {
    if (lane == 0) {
      const uint32_t xbytes = (uint32_t)(P * (pl.by + 2 * kr)) * xrow;
      const uint32_t dbytes = (uint32_t)(ndb * pl.by * (pl.rows_mode ? pl.bx : P)) * drow;
      int xs = 0, ds = 0, xseq = 0, dseq = 0;
      uint32_t xpar = 1, dpar = 1;
      auto load_x = [&](const Tile& t, int z) -> bool {
        if (!mbar_wait_or_abort(bar.xempty(xs), xpar, abort_v)) return false;
        mbar_expect_tx(bar.xfull(xs), xbytes);
        tma_load_5d(x0 + (uint32_t)xs * xslot, &tin, blk * pl.KBx, t.x0 - kr, t.y0 - kr, z, t.n, bar.xfull(xs));
        ++xseq;
        if (++xs == pl.NX) {
          xs = 0;
          xpar ^= 1u;
        }
        return true;
      };
      auto load_d = [&](const Tile& t, int z) -> bool {
        if (!mbar_wait_or_abort(bar.dempty(ds), dpar, abort_v)) return false;
        mbar_expect_tx(bar.dfull(ds), dbytes);
        for (int k = 0; k < ndb; ++k) {
          const uint32_t dst = d0 + (uint32_t)ds * dslot + (uint32_t)(k * pl.RD + kWgLead) * drow;
          if (pl.rows_mode) {
            for (int y = 0; y < pl.by; ++y)
              tma_load_5d(dst + (uint32_t)(y * P) * drow, &tdo, m0 + k * pl.KBd, t.x0, t.y0 + y, z, t.n, bar.dfull(ds));
          } else {
            tma_load_5d(dst, &tdo, m0 + k * pl.KBd, 0, t.y0, z, t.n, bar.dfull(ds));
          }
        }
        ++dseq;
        if (++ds == 2) {
          ds = 0;
          dpar ^= 1u;
        }
        return true;
      };
      bool ok = true;
      for (long long u = u_begin; ok && u < u_end;) {
        const long long strip = u / D;
        const int z0 = (int)(u - strip * D);
        const int nz = (int)((u_end - u < D - z0) ? u_end - u : D - z0);
        const Tile t = tile_of(strip);
        for (int i = 0; ok && i < nz; ++i) {
          ok = load_d(t, z0 + i);
          for (int d = (pl.march && i > 0) ? ndz - 1 : 0; ok && d < ndz; ++d) ok = load_x(t, z0 + i + dlo + d - kr);
        }
        u += nz;
      }
      // as in the forward kernel: each copy lands before the block's memory goes back
      for (int k = xseq > pl.NX ? xseq - pl.NX : 0; k < xseq; ++k) mbar_wait(bar.xfull(k % pl.NX), (k / pl.NX) & 1);
      for (int k = dseq > 2 ? dseq - 2 : 0; k < dseq; ++k) mbar_wait(bar.dfull(k & 1), (k >> 1) & 1);
    }
  } else if (warp >= kWgEpiWarps) {
    const int t0 = warp - kWgEpiWarps;
    if (t0 < nmw) {
      // SBO: the next 8 rows; LBO: the next M / N group (one row on where it is another dx tap, a block on otherwise)
      const uint64_t ad = smem_desc(d0, ndb == 1 ? drow : (uint32_t)pl.RD * drow, 8u * drow) |
                          ((uint64_t)swizzle_of(pl.KBd) << 61);
      const uint64_t bd = smem_desc(x0, (uint32_t)P * xrow, 8u * xrow) | ((uint64_t)swizzle_of(pl.KBx) << 61);
      const uint32_t ahi = (uint32_t)(ad >> 32), bhi = (uint32_t)(bd >> 32);
      const uint32_t astep = drow, bstep = xrow;  // 16 rows in 16-byte units
      const int issuer = elect_one() ? 1 : 0;
      int cnt = 0, buf = 0, ds = 0, xseq0 = 0, unit = 0;
      uint32_t dpar = 0;
      bool ok = true;
      for (long long u = u_begin; ok && u < u_end;) {
        const int z0 = (int)(u % D);
        const int nz = (int)((u_end - u < D - z0) ? u_end - u : D - z0);
        for (int i = 0; ok && i < nz; ++i, ++unit) {
          const bool first = unit % pl.upc == 0, last = unit % pl.upc == pl.upc - 1 || u + i == u_end - 1;
          if (first) {
            buf = cnt % pl.nbuf;
            if (cnt >= pl.nbuf && !mbar_wait_or_abort(bar.cempty(buf), ((cnt / pl.nbuf) - 1) & 1, abort_v)) ok = false;
            ++cnt;
          }
          if (ok) ok = mbar_wait_or_abort(bar.dfull(ds), dpar, abort_v);
          for (int d = 0; ok && d < ndz; ++d) {
            const int sq = xseq0 + (pl.march ? i + d : i * ndz + d), slot = sq % pl.NX;
            if (!mbar_wait_or_abort(bar.xfull(slot), (sq / pl.NX) & 1, abort_v)) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (issuer) {
              for (int a = t0; a < naus; a += kMmaWarps) {
                const Au& au = pl.au[au0 + a];
                if (au.dz != dlo + d) continue;
                const uint32_t idesc = (tc_idesc(N) & ~(31u << 24)) | ((uint32_t)(au.M >> 4) << 24) | (1u << 15) | (1u << 16);
                const uint32_t acc = tmem + (uint32_t)((buf * naus + a) * N);
                // M group g reads D[k + g] with X[k + dx0]: k starts at -(ndx - 1)
                uint32_t alo = (uint32_t)ad + ((uint32_t)ds * dslot + (uint32_t)(kWgLead - (au.ndx - 1)) * drow) / 16u;
                uint32_t blo = (uint32_t)bd + ((uint32_t)slot * xslot + (uint32_t)(au.dx0 - (au.ndx - 1)) * xrow) / 16u;
                uint32_t accum = first ? 0u : 1u;
#pragma unroll 2
                for (int j = 0; j < pl.nsteps; j += 4) {
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    tc_mma(acc, alo + (uint32_t)k * astep, ahi, blo + (uint32_t)k * bstep, bhi, idesc, accum);
                    accum = 1u;
                  }
                  alo += 4u * astep;
                  blo += 4u * bstep;
                }
              }
              if (!pl.march || d == 0 || i == nz - 1) tc_commit(bar.xempty(slot));
            }
            __syncwarp();
          }
          if (ok && issuer) {
            tc_commit(bar.dempty(ds));
            if (last) tc_commit(bar.cfull(buf));
          }
          __syncwarp();
          ds ^= 1;
          if (ds == 0) dpar ^= 1u;
        }
        xseq0 += pl.march ? nz + ndz - 1 : nz * ndz;
        u += nz;
      }
      if (issuer) tc_commit(bar.done());
    }
  } else {
    // ---- flush: accumulator rows of M = 64 lie in the first 16 lanes of each warp quadrant, of M = 128 in all 32
    const int quad = warp & 3, groups = N >> 4;
    const long long nu = u_end - u_begin;
    const int flushes = (int)((nu + pl.upc - 1) / pl.upc);
    float* base = partial + (long long)blockIdx.x * taps * s.Co * s.Ci;
    for (int f = 0; f < flushes; ++f) {
      const int buf = f % pl.nbuf;
      if (!mbar_wait_or_abort(bar.cfull(buf), (f / pl.nbuf) & 1, abort_v)) break;
      tc_fence_after();
      for (int it = warp >> 2; it < naus * groups; it += kWgEpiWarps / 4) {
        const int a = it / groups, c0 = (it - a * groups) << 4;
        const Au& au = pl.au[au0 + a];
        float v[16];
        __syncwarp();
        tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)((buf * naus + a) * N + c0), v);
        const int m = au.M == 64 ? quad * 16 + lane : quad * 32 + lane;
        const int g = ndb == 1 ? m / pl.KBd : 0, co = ndb == 1 ? m - g * pl.KBd : m;
        if (au.M == 64 && lane >= 16) continue;
        if (g >= au.ndx || co >= cb) continue;
        const int dy = c0 / pl.KBx, ci = blk * pl.KBx + c0 - dy * pl.KBx;
        const int tap = nd == 3 ? au.dz * 9 + dy * 3 + au.dx0 - g : 0;
        float4* dst = reinterpret_cast<float4*>(base + ((long long)tap * s.Co + m0 + co) * s.Ci + ci);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float4 p = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          if (f > 0) {
            const float4 o = dst[i];
            p = make_float4(o.x + p.x, o.y + p.y, o.z + p.z, o.w + p.w);
          }
          dst[i] = p;
        }
      }
      tc_fence_before();
      mbar_arrive(bar.cempty(buf));
    }
  }
  __syncwarp();
  if (warp < kWgEpiWarps + nmw) mbar_wait(bar.done(), 0);
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(pl.ncols));
  }
}

// db[co] = sum over voxels of d_out. Bound: one read of d_out. A thread takes 8 channels (16 bytes) of every
// stride-th voxel; the block's sums per channel go to one row of partials, which a second pass adds in order.
constexpr int kBiasBlocks = 592;
__global__ void __launch_bounds__(256) bias_grad_partial_kernel(const __nv_bfloat16* __restrict__ dout, long long V, int Co,
                                                                float* __restrict__ partial) {
  __shared__ float part[256][9];
  const int oct = Co >> 3, lanes = 256 / oct, o = threadIdx.x % oct, g = threadIdx.x / oct;
  float a[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
  if (g < lanes) {
    const uint4* src = reinterpret_cast<const uint4*>(dout) + o;
#pragma unroll 4
    for (long long v = (long long)blockIdx.x * lanes + g; v < V; v += (long long)gridDim.x * lanes) {
      const uint4 q = __ldg(src + v * oct);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[2 * i] += __uint_as_float(w[i] << 16);
        a[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) part[threadIdx.x][i] = a[i];
  __syncthreads();
  if ((int)threadIdx.x < Co) {
    const int co = threadIdx.x;
    float t = 0.0f;
    for (int k = 0; k < lanes; ++k) t += part[k * oct + (co >> 3)][co & 7];
    partial[(long long)blockIdx.x * Co + co] = t;
  }
}

// dw[tap][co][ci] over the voxels u of the input, d_out[u - off(tap)] a zero outside the volume; the caller's segment takes
// its eighth of them, 64 voxels at a time in FP32 (products are exact there), the rest in FP64. A NaN stays one and is looked
// for after each 64, so that their loads overlap: one infinity in a d_out of 16 channels at 4x32x128x152 costs 50 ms, NaN
// everywhere 3 (one voxel at a time in FP64: 94 and 6; without either the weight gradient takes 0.1).
__device__ __noinline__ double wgrad_direct(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ dout,
                                            const ConvShape& s, long long e, int seg) {
  const int ci = (int)(e % s.Ci), co = (int)(e / s.Ci % s.Co), tap = (int)(e / s.Ci / s.Co), nd = s.ksize, kr = nd >> 1;
  const int dz = tap / (nd * nd) - kr, dy = tap / nd % nd - kr, dx = tap % nd - kr;
  const long long V = (long long)s.N * s.D * s.H * s.W, end = V * (seg + 1) / 8;
  long long u = V * seg / 8;
  int x = (int)(u % s.W), y = (int)(u / s.W % s.H), z = (int)(u / s.W / s.H % s.D);
  const long long off = ((long long)dz * s.H + dy) * s.W + dx;
  const __nv_bfloat16* a = in + u * s.Ci + ci;
  const __nv_bfloat16* d = dout + (u - off) * s.Co + co;
  int left = (int)(end - u);
  double t = 0.0;
  while (left > 0 && t == t) {
    const int n = left < 64 ? left : 64;
    left -= n;
    float c = 0.0f;
#pragma unroll 4
    for (int k = 0; k < n; ++k, a += s.Ci, d += s.Co) {
      const bool inside = (unsigned)(z - dz) < (unsigned)s.D && (unsigned)(y - dy) < (unsigned)s.H &&
                          (unsigned)(x - dx) < (unsigned)s.W;
      c = fmaf(inside ? __bfloat162float(*d) : 0.0f, __bfloat162float(*a), c);
      if (++x == s.W) {
        x = 0;
        if (++y == s.H) {
          y = 0;
          if (++z == s.D) z = 0;
        }
      }
    }
    t += (double)c;
  }
  return t;
}

// The partial sums of both, one launch. dw[e] = sum of the CTAs' partials: a block sums 32 values, 8 segments of the CTAs
// each in order, then the segments in order. The blocks after those take db: a warp per channel, 32 strided sums
// of the bias partials, then a fixed tree.
// The tiles multiply d_out by the zeros around the input and the input by the zeros around d_out, and an infinity times
// those is a NaN in taps that do not use the voxel. Such a sum is never finite, so a value that is not is summed anew.
__global__ void __launch_bounds__(256, 8) wgrad_reduce_kernel(const float* __restrict__ partial, int n, long long count,
                                                           float* __restrict__ dw, const float* __restrict__ bias_partial,
                                                           int bias_rows, const __nv_bfloat16* __restrict__ in,
                                                           const __nv_bfloat16* __restrict__ dout,
                                                           const __grid_constant__ ConvShape s,
                                                           float* __restrict__ db) {
  __shared__ float part[8][33];
  const int Co = s.Co;
  const int x = threadIdx.x & 31, seg = threadIdx.x >> 5;
  const long long dw_blocks = (count + 31) / 32;
  if (blockIdx.x >= dw_blocks) {
    const int c = (int)(blockIdx.x - dw_blocks) * 8 + seg;
    if (c >= Co) return;
    float t = 0.0f;
    for (int b = x; b < bias_rows; b += 32) t += bias_partial[(long long)b * Co + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (x == 0) db[c] = t;
    return;
  }
  const long long e = blockIdx.x * 32ll + x;
  float t = 0.0f;
  if (e < count) {
    const int k0 = n * seg / 8, k1 = n * (seg + 1) / 8;
#pragma unroll 8
    for (int k = k0; k < k1; ++k) t += partial[(long long)k * count + e];
  }
  part[seg][x] = t;
  __syncthreads();
  bool finite = true;
  if (seg == 0 && e < count) {
    for (int k = 1; k < 8; ++k) t += part[k][x];
    dw[e] = t;
    finite = isfinite(t);
  }
  if (__syncthreads_and(finite)) return;
  __shared__ double direct[8][33];
  __shared__ int redo[32];
  if (seg == 0) redo[x] = !finite;
  __syncthreads();
  if (redo[x]) direct[seg][x] = wgrad_direct(in, dout, s, e, seg);
  __syncthreads();
  if (!finite) {
    double sum = 0.0;
    for (int k = 0; k < 8; ++k) sum += direct[k][x];
    dw[e] = (float)sum;
  }
}

int check_shape(const ConvShape& s) {
  XAC_REQUIRE(s.N > 0 && s.D > 0 && s.H > 0 && s.W > 0, "conv3d: bad volume");
  XAC_REQUIRE((long long)s.N * s.D * s.H * s.W < (1LL << 31), "conv3d: volume must stay below 2^31 voxels");
  XAC_REQUIRE(s.Ci % 16 == 0 && s.Co % 16 == 0 && s.Ci <= 256 && s.Co <= 256 && s.Ci >= 16 && s.Co >= 16,
              "conv3d: channels must be multiples of 16 with Ci, Co <= 256 (got %d -> %d)", s.Ci, s.Co);
  XAC_REQUIRE(s.ksize == 1 || s.ksize == 3, "conv3d: kernel size must be 1 or 3");
  return XAC_OK;
}


// ---- host: the forward tile ---------------------------------------------------------------------------------
// The tile is a pure function of the shape: the cheapest of all tiles that fit, by a model of one CTA's time (the
// longest CTA decides): MMAs at the measured rate (39 cycles for 128 voxels x 16 channels x Co = 16, 48 for 64, 64 for 128)
// against the bytes copied from L2 at about 22 B/clk per SM, plus a fixed cost per unit and per CTA. It picks the
// slice of Co, the tile, the plane ring and resident or streamed weights.
constexpr size_t kSmemLimit = 231000;  // dynamic shared memory of a CTA (227 KB less the static part)

int sm_count(int* out) {
  int dev = 0;
  XAC_CUDA(cudaGetDevice(&dev));
  XAC_CUDA(cudaDeviceGetAttribute(out, cudaDevAttrMultiProcessorCount, dev));
  return XAC_OK;
}

// Raises a kernel's dynamic shared-memory limit once per device (the attribute belongs to the device's context).
enum { kFwdSlot = 0, kWgSlot = 1, kSlots = 2 };
int allow_smem(const void* fn, int slot) {
  static std::atomic<unsigned long long> done[kSlots];  // a bit per device
  int dev = 0;
  XAC_CUDA(cudaGetDevice(&dev));
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit && (done[slot].load() & bit)) return XAC_OK;
  XAC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
  done[slot].fetch_or(bit);
  return XAC_OK;
}

// TMA map of a packed BF16 tensor (innermost dimension first), read in boxes whose innermost extent is the swizzle span
// (128, 64 or 32 bytes). The encoder comes from the driver, once.
int bf16_map(CUtensorMap* m, const void* base, int rank, const cuuint64_t* dims, const cuuint32_t* box) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static std::atomic<Encode> fn{nullptr};
  Encode f = fn.load();
  if (!f) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    XAC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    XAC_REQUIRE(p && q == cudaDriverEntryPointSuccess, "conv3d: the driver has no cuTensorMapEncodeTiled");
    f = (Encode)p;
    fn.store(f);
  }
  XAC_REQUIRE(((uintptr_t)base & 15u) == 0, "conv3d: operands must be 16-byte aligned");
  cuuint64_t strides[4];
  cuuint32_t ones[5] = {1, 1, 1, 1, 1};
  cuuint64_t bytes = 2;
  for (int k = 0; k + 1 < rank; ++k) strides[k] = bytes *= dims[k];
  const CUtensorMapSwizzle sw = box[0] == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
                                : box[0] == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                                               : CU_TENSOR_MAP_SWIZZLE_32B;
  const CUresult e = f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides,
                       box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  XAC_REQUIRE(e == CUDA_SUCCESS, "conv3d: cuTensorMapEncodeTiled failed (%d)", (int)e);
  return XAC_OK;
}

bool search_fwd_plan(const ConvShape& s, int sms, FwdPlan* best) {
  const int kr = s.ksize / 2, taps = s.ksize * s.ksize * s.ksize;
  double best_cost = INFINITY;
  for (int split = 1; split <= s.Co / 16; ++split) {
    if (s.Co % (16 * split)) continue;
    const int nb = s.Co / split;
    const int min_nxt = (s.W + 253) / 254;
    int last_bx = -1;
    // x tiles: every count at first, then steps of an eighth, down to tiles of 8 voxels (256 channels need <= 27)
    for (int nxt = min_nxt; nxt == min_nxt || (s.W + nxt - 1) / nxt >= 8; nxt += nxt < 8 ? 1 : nxt / 8) {
      const int bx = (s.W + nxt - 1) / nxt, P = bx + 2 * kr;
      if (bx == last_bx) continue;
      last_bx = bx;
      for (int by = 1; by <= s.H; ++by) {
        const int mt = ((by - 1) * P + bx + kTcM - 1) / kTcM;
        if (mt * nb > 512 || mt > 2 * kMmaWarps) break;
        if (P > 256 || by + 2 * kr > 256) break;  // a TMA box
        const int R = (mt * kTcM + 2 * kr * (P + 1) + 7) / 8 * 8;  // whole swizzle atoms
        const size_t plane = (size_t)R * s.Ci * 2;
        if (2 * plane > kSmemLimit) break;
        for (int ring = 2; ring <= kMaxPlanes; ++ring) {
          const int march = kr == 1 && ring >= 3;
          if (kr == 0 && ring == kMaxPlanes) continue;
          // weights: resident; streamed by taps; streamed by blocks
          for (int mode = split == 1 ? 0 : 1; mode < 3; ++mode) {
            const int resident = mode == 0, big = mode < 2;
            FwdPlan p{};
            p.KB = 64;
            while (s.Ci % p.KB) p.KB >>= 1;
            const int nkc = s.Ci / p.KB;
            p.G = nkc <= 3 && big ? nkc : 1;
            if (p.G == 2 && p.KB != 64) p.G = 1;
            const size_t stage = (size_t)p.KB * p.G * nb * 2;
            const int stages = taps * (nkc / p.G);
            p.bs = resident ? stages : kMaxBStages;
            while (!resident && p.bs > 3 && ring * plane + p.bs * stage > kSmemLimit) --p.bs;
            p.smem = ring * plane + p.bs * stage;
            if (p.smem > kSmemLimit) continue;
            p.bx = bx;
            p.by = by;
            p.P = P;
            p.nxt = (s.W + bx - 1) / bx;
            p.nyt = (s.H + by - 1) / by;
            p.mt = mt;
            p.R = R;
            p.NS = ring;
            p.march = march;
            p.nb = nb;
            p.nsplit = split;
            p.resident = resident;
            p.nbuf = 2 * mt * nb <= 512 ? 2 : 1;
            p.ncols = 32;
            while ((int)p.ncols < p.nbuf * mt * nb) p.ncols <<= 1;
            p.units = (long long)s.N * s.D * p.nyt * p.nxt * split;
            p.ctas = (int)(p.units < sms ? p.units : sms);
            const double per = (double)((p.units + p.ctas - 1) / p.ctas);
            const double hw = 35.0 + nb * 0.24, one = nb / 2.0 > hw ? nb / 2.0 : hw;  // cycles of an MMA
            // one warp's straight-line issue, and the turn of its loop over stages
            const int steps = p.KB / 16 * p.G, nt = (mt + kMmaWarps - 1) / kMmaWarps;
            const double turn = resident && nkc == p.G && kr == 1 ? (steps * nt <= 4 ? 150.0 / 9 : 150.0 / 3) : 250.0;
            const double issue = 100.0 * steps * nt + turn, stage_hw = mt * one * steps;
            const double mma = stages * (stage_hw > issue ? stage_hw : issue);
            const double run = per < s.D ? per : s.D;  // planes of one z walk
            const double planes = march ? (run + 2) / run : s.ksize;
            const double bytes = planes * (by + 2 * kr) * P * s.Ci * 2.0 + (resident ? 0.0 : taps * s.Ci * nb * 2.0);
            const double epi = 300.0 + mt * (nb / 16) * 40.0;
            const double mem = bytes / 22.0;
            double unit = mma > mem ? mma + 0.2 * mem : mem + 0.2 * mma;
            unit = p.nbuf == 2 ? (unit > epi ? unit : epi) + 200.0 : unit + epi + 200.0;
            const double cost = per * unit + 3000.0 + (resident ? taps * s.Ci * nb * 2.0 / 32.0 : 0.0);
            if (cost < best_cost) {
              best_cost = cost;
              *best = p;
            }
          }
        }
      }
    }
  }
  return std::isfinite(best_cost);
}

// Plans kept by shape (the search takes 20 to 300 us on a host core, most for wide volumes of few channels); the map is
// emptied when it holds 256.
int fwd_plan(const ConvShape& s, FwdPlan* out) {
  static std::mutex mu;
  static std::map<std::array<int, 8>, FwdPlan> plans;
  int sms = 0;
  int r = sm_count(&sms);
  if (r != XAC_OK) return r;
  const std::array<int, 8> key = {s.N, s.D, s.H, s.W, s.Ci, s.Co, s.ksize, sms};
  try {
    std::lock_guard<std::mutex> g(mu);
    auto it = plans.find(key);
    if (it == plans.end()) {
      FwdPlan p;
      XAC_REQUIRE(search_fwd_plan(s, sms, &p), "conv3d: no tile for %d -> %d channels", s.Ci, s.Co);
      if (plans.size() >= 256) plans.clear();
      it = plans.emplace(key, p).first;
    }
    *out = it->second;
  } catch (...) {  // no C++ exception crosses the C boundary
    set_error("conv3d: host allocation failed");
    return XAC_ENOMEM;
  }
  return XAC_OK;
}

// ---- host: the weight gradient's tile ---------------------------------------------------------------------------
// A pure function of the shape (148 CTAs are assumed, whatever the device: the partial buffer's size is part of the ABI).
constexpr int kWgCtas = 148;

bool search_wg_plan(const ConvShape& s, WgPlan* best) {
  const int kr = s.ksize / 2, nd = s.ksize;
  WgPlan b{};
  b.KBx = b.KBd = 64;
  while (s.Ci % b.KBx) b.KBx >>= 1;
  while (s.Co % b.KBd) b.KBd >>= 1;
  b.nblk = s.Ci / b.KBx;
  b.cb = s.Co < 128 ? s.Co : 128;
  b.mblk = (s.Co + 127) / 128;
  b.nstack = nd;
  const int N = b.KBx * b.nstack, M1 = s.Co <= 64 ? 64 : 128;
  for (int dz = 0; dz < nd; ++dz) {
    if (nd == 1) {
      b.au[b.nau++] = {0, M1, 0, 1};
    } else if (s.Co == 16 || s.Co == 32) {
      b.au[b.nau++] = {dz, s.Co == 16 ? 64 : 128, 2, 3};
    } else if (s.Co == 64) {
      b.au[b.nau++] = {dz, 128, 2, 2};
      b.au[b.nau++] = {dz, 64, 0, 1};
    } else {
      for (int dx = 0; dx < 3; ++dx) b.au[b.nau++] = {dz, M1, dx, 1};
    }
  }
  // accumulator sets of at most 512 columns, as even as their number allows
  const int cap = 512 / N;
  b.ngr = (b.nau + cap - 1) / cap;
  for (int g = 0; g <= b.ngr; ++g) b.first[g] = b.nau * g / b.ngr;
  int most = 0, planes = 0;
  double mma = 0.0;  // cycles of a step, in the longest set
  for (int g = 0; g < b.ngr; ++g) {
    const int n = b.first[g + 1] - b.first[g];
    double c = 0.0;
    for (int a = b.first[g]; a < b.first[g + 1]; ++a) {
      const double rd = (b.au[a].M + N) / 4.0 + 8.0, math = N / 2.0;
      c += rd > math ? rd : math;
    }
    const double issue = 60.0 * ((n + kMmaWarps - 1) / kMmaWarps);
    if (c < issue) c = issue;
    if (c > mma) mma = c;
    if (n > most) most = n;
    const int pz = b.au[b.first[g + 1] - 1].dz - b.au[b.first[g]].dz + 1;
    if (pz > planes) planes = pz;
  }
  b.nbuf = 2 * most * N <= 512 ? 2 : 1;
  b.ncols = 32;
  while ((int)b.ncols < b.nbuf * most * N) b.ncols <<= 1;
  const int sets = b.ngr * b.nblk * b.mblk;
  double best_cost = INFINITY;
  const int pitches[] = {0, 256, 128, 64, 48, 32, 24, 16, 8};  // 0: the whole row of the volume
  for (int pitch : pitches) {
    WgPlan p = b;
    p.rows_mode = pitch != 0;
    p.P = pitch ? pitch : s.W + 2 * kr;
    p.bx = p.P - 2 * kr;
    if (p.P > 256 || (pitch && p.bx >= s.W)) continue;
    p.nxt = (s.W + p.bx - 1) / p.bx;
    for (p.by = 1; p.by <= s.H && p.by + 2 * kr <= 256; ++p.by) {
      p.nsteps = ((p.by * p.P + 2 * kr + 15) / 16 + 3) / 4 * 4;
      if (p.nsteps > kWgMaxSteps) break;
      // the last step's rows, the farthest M group and dy tap stay inside a block
      p.RD = (kWgLead + p.nsteps * 16 + 8 + 7) / 8 * 8;
      p.RX = (p.nsteps * 16 + 2 + 2 * kr * p.P + 7) / 8 * 8;
      if (p.RX < (p.by + 2 * kr) * p.P) p.RX = ((p.by + 2 * kr) * p.P + 7) / 8 * 8;
      p.nyt = (s.H + p.by - 1) / p.by;
      const size_t dtile = (size_t)p.RD * p.cb * 2, plane = (size_t)p.RX * p.KBx * 2;
      for (p.NX = 2; p.NX <= kMaxPlanes; ++p.NX) {
        p.march = p.NX > planes || (p.NX == planes && planes == 3);
        if (planes == 1) p.march = 0;
        p.smem = 2 * dtile + p.NX * plane;
        // M groups past the last block read on from the second tile: keep them inside
        const size_t reach = dtile + (size_t)(128 / p.KBd) * p.RD * p.KBd * 2;
        if (p.smem < reach) p.smem = reach;
        if (p.smem > kSmemLimit) break;
        p.upc = kWgMaxSteps / p.nsteps;
        p.units = (long long)s.N * s.D * p.nyt * p.nxt;
        const long long room = kWgCtas / sets > 0 ? kWgCtas / sets : 1;
        p.ctas = (int)(p.units < room ? p.units : room);
        const double waves = (double)((p.ctas * sets + kWgCtas - 1) / kWgCtas);
        const double per = (double)((p.units + p.ctas - 1) / p.ctas), run = per < s.D ? per : s.D;
        const double loads = p.march ? (run + planes - 1) / run : planes;
        const double mem = (p.by * p.P * p.cb * 2.0 + loads * (p.by + 2 * kr) * p.P * p.KBx * 2.0) / 22.0;
        const double work = mma * p.nsteps;
        const double flush = 500.0 + most * (N / 16) * 60.0;
        const double unit = (work > mem ? work + 0.2 * mem : mem + 0.2 * work) + 200.0 + (p.nbuf == 1 ? flush / p.upc : 0.0);
        const double cost = waves * (per * unit + 5000.0 + flush);
        if (cost < best_cost) {
          best_cost = cost;
          *best = p;
        }
      }
    }
  }
  return std::isfinite(best_cost);
}

int wg_plan(const ConvShape& s, WgPlan* out) {
  static std::mutex mu;
  static std::map<std::array<int, 7>, WgPlan> plans;
  const std::array<int, 7> key = {s.N, s.D, s.H, s.W, s.Ci, s.Co, s.ksize};
  try {
    std::lock_guard<std::mutex> g(mu);
    auto it = plans.find(key);
    if (it == plans.end()) {
      WgPlan p;
      XAC_REQUIRE(search_wg_plan(s, &p), "conv3d: no weight-gradient tile for %d -> %d channels", s.Ci, s.Co);
      if (plans.size() >= 256) plans.clear();
      it = plans.emplace(key, p).first;
    }
    *out = it->second;
  } catch (...) {  // no C++ exception crosses the C boundary
    set_error("conv3d: host allocation failed");
    return XAC_ENOMEM;
  }
  return XAC_OK;
}

}  // namespace
}  // namespace xac

using namespace xac;

extern "C" {

int xac_conv3d_forward(const void* in, int N, int D, int H, int W, int Ci, const void* weight, const float* bias,
                       int Co, int ksize, int activation, void* out_bf16, float* out_f32, void* stream) {
  ConvShape s{N, D, H, W, Ci, Co, ksize};
  int r = check_shape(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(in && weight && (out_bf16 || out_f32) && !(out_bf16 && out_f32),
              "xac_conv3d_forward: give exactly one output");
  XAC_REQUIRE(activation == 0 || activation == 1, "xac_conv3d_forward: activation must be 0 (none) or 1 (GELU)");
  FwdPlan pl;
  r = fwd_plan(s, &pl);
  if (r != XAC_OK) return r;
  r = allow_smem((const void*)conv_fwd_kernel, kFwdSlot);
  if (r != XAC_OK) return r;
  CUtensorMap tin, tw;
  const int kr = ksize / 2;
  {
    const cuuint64_t dims[5] = {(cuuint64_t)Ci, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N};
    const cuuint32_t box[5] = {(cuuint32_t)pl.KB, (cuuint32_t)pl.P, (cuuint32_t)(pl.by + 2 * kr), 1, 1};
    r = bf16_map(&tin, in, 5, dims, box);
    if (r != XAC_OK) return r;
    const cuuint32_t taps = (cuuint32_t)(ksize * ksize * ksize);
    const cuuint64_t wdims[3] = {(cuuint64_t)Ci, (cuuint64_t)Co, taps};
    const cuuint32_t wbox[3] = {(cuuint32_t)pl.KB, (cuuint32_t)pl.nb, pl.resident ? taps : 1u};
    r = bf16_map(&tw, weight, 3, wdims, wbox);
    if (r != XAC_OK) return r;
  }
  conv_fwd_kernel<<<pl.ctas, kFwdThreads, pl.smem, as_stream(stream)>>>(tin, tw, bias, s, activation, pl,
                                                                        (__nv_bfloat16*)out_bf16, out_f32);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

// partial must hold xac_conv3d_partial_floats() floats; dw receives taps * Co * Ci floats, db Co floats
int xac_conv3d_weight_grad(const void* in, int N, int D, int H, int W, int Ci, const void* dout, int Co, int ksize,
                           float* partial, float* dw, float* db, void* stream) {
  ConvShape s{N, D, H, W, Ci, Co, ksize};
  int r = check_shape(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(in && dout && partial && dw, "xac_conv3d_weight_grad: null pointer");
  const long long V = (long long)N * D * H * W;
  const int taps = ksize == 3 ? 27 : 1, kr = ksize / 2;
  WgPlan pl;
  r = wg_plan(s, &pl);
  if (r != XAC_OK) return r;
  r = allow_smem((const void*)conv_wgrad_kernel, kWgSlot);
  if (r != XAC_OK) return r;
  CUtensorMap tin, tdo;
  {
    const cuuint64_t dims[5] = {(cuuint64_t)Ci, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N};
    const cuuint32_t box[5] = {(cuuint32_t)pl.KBx, (cuuint32_t)pl.P, (cuuint32_t)(pl.by + 2 * kr), 1, 1};
    r = bf16_map(&tin, in, 5, dims, box);
    if (r != XAC_OK) return r;
    const cuuint64_t ddims[5] = {(cuuint64_t)Co, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)N};
    const cuuint32_t dbox[5] = {(cuuint32_t)pl.KBd, (cuuint32_t)(pl.rows_mode ? pl.bx : pl.P),
                                (cuuint32_t)(pl.rows_mode ? 1 : pl.by), 1, 1};
    r = bf16_map(&tdo, dout, 5, ddims, dbox);
    if (r != XAC_OK) return r;
  }
  cudaStream_t st = as_stream(stream);
  conv_wgrad_kernel<<<dim3((unsigned)pl.ctas, (unsigned)pl.ngr, (unsigned)(pl.nblk * pl.mblk)), kWgThreads, pl.smem, st>>>(
      tin, tdo, s, pl, partial);
  const long long count = (long long)taps * Co * Ci;
  float* bias_partial = partial + pl.ctas * count;
  const int lanes = 256 / (Co / 8);
  const int rows = (int)((V + lanes - 1) / lanes < kBiasBlocks ? (V + lanes - 1) / lanes : kBiasBlocks);
  if (db)
    bias_grad_partial_kernel<<<rows, 256, 0, st>>>((const __nv_bfloat16*)dout, V, Co, bias_partial);
  wgrad_reduce_kernel<<<(unsigned)((count + 31) / 32) + (db ? (Co + 7) / 8 : 0), 256, 0, st>>>(
      partial, pl.ctas, count, dw, bias_partial, rows, (const __nv_bfloat16*)in, (const __nv_bfloat16*)dout, s, db);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

// Test-only: the convolution kernels' mbarrier wait on a barrier that nothing completes must give up after
// `limit` polls and set g_conv_status (read and cleared by xac_conv3d_status).
static __global__ void test_conv_wait_timeout_kernel(uint32_t limit) {
  __shared__ __align__(8) uint64_t bar;
  const uint32_t b = smem_addr(&bar);
  if (threadIdx.x == 0) {
    mbar_init(b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mbar_wait(b, 0, limit);
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(b) : "memory");
  }
}

int xac_test_conv_plan(int N, int D, int H, int W, int Ci, int Co, int ksize, int sms, long long* fwd, long long* wg) {
  XAC_REQUIRE(fwd && wg && sms > 0, "xac_test_conv_plan: bad arguments");
  const ConvShape s{N, D, H, W, Ci, Co, ksize};
  int r = check_shape(s);
  if (r != XAC_OK) return r;
  FwdPlan f;
  WgPlan w;
  XAC_REQUIRE(search_fwd_plan(s, sms, &f) && search_wg_plan(s, &w), "xac_test_conv_plan: no tile");
  const long long a[] = {f.units, f.ctas, f.march, f.NS, f.resident, f.bs, f.nbuf, f.mt};
  const long long b[] = {w.units, w.ctas, w.march, w.NX, w.upc, w.nbuf, w.rows_mode};
  for (int k = 0; k < 8; ++k) fwd[k] = a[k];
  for (int k = 0; k < 7; ++k) wg[k] = b[k];
  return XAC_OK;
}

int xac_test_conv_wait_timeout(unsigned limit, void* stream) {
  XAC_REQUIRE(limit > 0 && limit <= (1u << 20), "xac_test_conv_wait_timeout: limit %u out of (0, 2^20]", limit);
  cudaStream_t s = as_stream(stream);
  test_conv_wait_timeout_kernel<<<1, 32, 0, s>>>(limit);
  XAC_CUDA(cudaGetLastError());
  XAC_CUDA(cudaStreamSynchronize(s));
  return XAC_OK;
}

int xac_conv3d_status(int* flags) {
  XAC_REQUIRE(flags, "xac_conv3d_status: null pointer");
  unsigned int v = 0, zero = 0;
  XAC_CUDA(cudaMemcpyFromSymbol(&v, g_conv_status, sizeof(v)));
  XAC_CUDA(cudaMemcpyToSymbol(g_conv_status, &zero, sizeof(zero)));
  *flags = (int)v;
  return XAC_OK;
}

int xac_conv3d_partial_floats(int N, int D, int H, int W, int Ci, int Co, int ksize, long long* count) {
  XAC_REQUIRE(count, "xac_conv3d_partial_floats: null pointer");
  const ConvShape s{N, D, H, W, Ci, Co, ksize};
  int r = check_shape(s);
  if (r != XAC_OK) return r;
  WgPlan pl;
  r = wg_plan(s, &pl);
  if (r != XAC_OK) return r;
  *count = (long long)pl.ctas * (ksize == 3 ? 27 : 1) * Co * Ci + (long long)kBiasBlocks * Co;
  return XAC_OK;
}

}  // extern "C"
