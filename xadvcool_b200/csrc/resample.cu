// The surrogate's changes of resolution on channels-last BF16 volumes [N][D][H][W][C], one pass each: 2x average pooling
// and its gradient, and nearest 2x upsampling joined to the skip volume's channels (benchmark/models/unet3d.py:11-125).
// The gradient of the upsampling stays a tensor operation: the order of its sums decides how BF16 values round.
//
// What bounds them: memory, one read of each input and one write of each output. A thread takes an octet of channels (16
// bytes) of one coarse voxel, or of one fine voxel of the joined volume; eight values are added in FP32 and rounded to
// BF16 once. Where their exponents lie within 13 bits of one another the sum is exact in any order; others round by the
// order, and gave the tensor operations' bits on the cases measured. The tensor operations this replaces wrote FP32 copies of
// the fine volume and the upsampled volume on its own: a training step's gradients at batch 4 10.8 -> 9.7 ms, a prediction
// 2.97 -> 2.69.
#include <cuda_bf16.h>

#include "xac_internal.cuh"

namespace xac {
namespace {

constexpr int kBlock = 256;

struct Coarse {  // coarse voxels; the fine volume has twice the extents
  unsigned N, D, H, W;
};

__device__ __forceinline__ void add8(const uint4& r, float (&v)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] += __uint_as_float(w[k] << 16);
    v[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8], float scale) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * k] * scale, v[2 * k + 1] * scale);
    w[k] = *reinterpret_cast<const uint32_t*>(&p);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// voxel v of the coarse volume -> its first fine voxel
__device__ __forceinline__ unsigned fine_of(unsigned v, const Coarse& c) {
  const unsigned x = v % c.W;
  v /= c.W;
  const unsigned y = v % c.H;
  v /= c.H;  // n * D + z: the fine volume's planes are twice as many
  return (v * 2 * (2 * c.H) + 2 * y) * (2 * c.W) + 2 * x;
}
__device__ __forceinline__ unsigned fine_step(int k, const Coarse& c) {
  return (((k >> 2) & 1) * (2 * c.H) + ((k >> 1) & 1)) * (2 * c.W) + (k & 1);
}

__global__ void __launch_bounds__(kBlock) pool_kernel(const uint4* __restrict__ x, Coarse c, unsigned oct, unsigned count,
                                                      uint4* __restrict__ out) {
  const unsigned i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= count) return;
  const unsigned o = i % oct, f = fine_of(i / oct, c);
  uint4 r[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) r[k] = __ldg(x + (size_t)(f + fine_step(k, c)) * oct + o);
  float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 8; ++k) add8(r[k], v);
  out[i] = pack8(v, 0.125f);
}

__global__ void __launch_bounds__(kBlock) pool_grad_kernel(const uint4* __restrict__ dout, Coarse c, unsigned oct, unsigned count,
                                                           uint4* __restrict__ dx) {
  const unsigned i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= count) return;
  const unsigned o = i % oct, f = fine_of(i / oct, c);
  float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  add8(__ldg(dout + i), v);
  const uint4 r = pack8(v, 0.125f);
#pragma unroll
  for (int k = 0; k < 8; ++k) dx[(size_t)(f + fine_step(k, c)) * oct + o] = r;
}

// out[fine][0..Ca) = low[coarse], out[fine][Ca..Ca+Cb) = skip[fine]
__global__ void __launch_bounds__(kBlock) upcat_kernel(const uint4* __restrict__ low, const uint4* __restrict__ skip, Coarse c,
                                                       unsigned oa, unsigned ob, unsigned count, uint4* __restrict__ out) {
  const unsigned i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= count) return;
  const unsigned oct = oa + ob, o = i % oct, f = i / oct;
  if (o >= oa) {
    out[i] = __ldg(skip + (size_t)f * ob + (o - oa));
    return;
  }
  unsigned v = f;
  const unsigned x = v % (2 * c.W) / 2;
  v /= 2 * c.W;
  const unsigned y = v % (2 * c.H) / 2;
  v /= 2 * c.H;  // n * 2D + z
  out[i] = __ldg(low + (size_t)((v / 2 * c.H + y) * c.W + x) * oa + o);
}

bool aligned16(const void* a, const void* b, const void* c) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15u) == 0;
}
// the kernels index octets and voxels of the fine volume in 32 bits
int check(int N, int D, int H, int W, int Ca, int Cb, const char* who) {
  XAC_REQUIRE(N >= 1 && D >= 1 && H >= 1 && W >= 1, "%s: extents must be positive", who);
  XAC_REQUIRE(Ca >= 8 && Ca % 8 == 0 && Cb >= 0 && Cb % 8 == 0, "%s: channels must be a multiple of 8", who);
  const double fine = 8.0 * N * D * H * W * ((Ca + (double)Cb) / 8.0);
  XAC_REQUIRE(fine <= 1073741824.0, "%s: at most 2^33 values", who);
  return XAC_OK;
}

}  // namespace
}  // namespace xac

using namespace xac;

extern "C" {

int xac_pool2(const void* in, int N, int D, int H, int W, int C, int backward, void* out, void* stream) {
  int r = check(N, D, H, W, C, 0, "xac_pool2");
  if (r != XAC_OK) return r;
  XAC_REQUIRE(in && out && aligned16(in, out, nullptr), "xac_pool2: 16-byte aligned volumes are needed");
  const Coarse c{(unsigned)N, (unsigned)D, (unsigned)H, (unsigned)W};
  const unsigned oct = C / 8, count = c.N * c.D * c.H * c.W * oct;
  (backward ? pool_grad_kernel : pool_kernel)<<<grid_for(count, kBlock), kBlock, 0, as_stream(stream)>>>((const uint4*)in, c, oct,
                                                                                                     count, (uint4*)out);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

int xac_upcat2(const void* low, const void* skip, int N, int D, int H, int W, int Ca, int Cb, void* out, void* stream) {
  int r = check(N, D, H, W, Ca, Cb, "xac_upcat2");
  if (r != XAC_OK) return r;
  XAC_REQUIRE(Cb >= 8 && low && skip && out && aligned16(low, skip, out),
              "xac_upcat2: 16-byte aligned volumes are needed");
  const Coarse c{(unsigned)N, (unsigned)D, (unsigned)H, (unsigned)W};
  const unsigned count = 8 * c.N * c.D * c.H * c.W * ((Ca + Cb) / 8);
  upcat_kernel<<<grid_for(count, kBlock), kBlock, 0, as_stream(stream)>>>((const uint4*)low, (const uint4*)skip, c, Ca / 8, Cb / 8,
                                                                         count, (uint4*)out);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

}  // extern "C"
