// GroupNorm + GELU of the surrogate's units on channels-last BF16 volumes [N][V][C] once a group's mean and 1/std are
// known (the unit of benchmark/models/unet3d.py:11-26): the forward values, and the backward sums and values.
//
// What bounds it: memory. Forward reads the volume and writes it once; the tensor operations this replaces wrote six
// FP32 volumes. Backward reads the volume and the incoming gradient twice, writes the two FP32 volumes whose sums are the
// groups' (added by the caller) and the result; the tensor operations wrote more than ten FP32 volumes.
// 16 channels at 32x128x152, one sample: forward 237 -> 127 us, 105 of them the statistics (tensor operations in
// both); backward 430 -> 199. A training step's gradients at batch 4: 19.6 -> 10.8 ms; a prediction: 3.6 -> 2.9.
// A thread owns one octet of channels (16-byte loads) and walks voxels, so its channels' scale, shift, mean and
// 1/std stay in registers. Every multiply and add of a value is rounded by itself, in the tensor operations' order, so
// that the BF16 results are theirs: a result that rounds the other way is carried through all later layers. The
// channels' sums run in FP32 over 8 voxels, then in FP64, in a fixed order.
#include <cuda_bf16.h>

#include "xac_internal.cuh"

namespace xac {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxC = 256;
constexpr int kChunk = 8;          // voxels a thread sums in FP32 before the FP64 sums take over
constexpr int kTargetBlocks = 1184;  // 148 SMs x 8 resident blocks of 256 threads

struct NormShape {
  int N;
  long long V;
  int C, G;
  int oct() const { return C / 8; }
  int vpb() const { return kThreads / oct(); }  // voxels of one pass of a block
};

// blocks of a sample: passes of kChunk voxels a thread, no more blocks than fill the GPU once
int stat_blocks(const NormShape& s) {
  const long long per = (long long)s.vpb() * kChunk;
  const long long need = (s.V + per - 1) / per;
  const long long most = (kTargetBlocks + s.N - 1) / s.N;
  return (int)(need < most ? need : most);
}
// voxels a thread takes in the elementwise passes: up to 8 (the registers' set-up is spread over them), fewer where the
// volume would not fill the GPU
int apply_iters(const NormShape& s) {
  const long long it = s.V * s.N / ((long long)s.vpb() * kTargetBlocks);
  return it < 1 ? 1 : (it > 8 ? 8 : (int)it);
}
unsigned apply_blocks(const NormShape& s, int iters) {
  const long long per = (long long)s.vpb() * iters;
  return (unsigned)((s.V + per - 1) / per);
}

__device__ __forceinline__ void unpack8(const uint4& r, float (&v)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = __uint_as_float(w[k] << 16);
    v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    w[k] = *reinterpret_cast<const uint32_t*>(&p);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float gelu(float z) {
  return __fmul_rn(__fmul_rn(z, 0.5f), __fadd_rn(1.0f, erff(__fmul_rn(z, 0.70710678118654752f))));
}
// Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_slope(float z) {
  const float cdf = __fmul_rn(0.5f, __fadd_rn(1.0f, erff(__fmul_rn(z, 0.70710678118654752f))));
  const float pdf = __fmul_rn(expf(__fmul_rn(__fmul_rn(-0.5f, z), z)), 0.39894228040143268f);
  return __fadd_rn(cdf, __fmul_rn(z, pdf));
}

// a warp's lanes that hold the same octet, added in a fixed tree
__device__ __forceinline__ double octet_sum(double v, int oct) {
  for (int d = 16; d >= oct; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// the registers of a thread's octet
struct OctetParams {
  float mean[2], rstd[2], g[8], s[8];
  __device__ __forceinline__ void load(const float* mu, const float* rs, const float* gamma, const float* beta, int n, int o,
                                       int C, int G) {
    const int cg = C / G;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      mean[q] = mu[n * G + (o * 8 + q * 4) / cg];
      rstd[q] = rs[n * G + (o * 8 + q * 4) / cg];
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      g[c] = gamma[o * 8 + c];
      s[c] = beta[o * 8 + c];
    }
  }
  __device__ __forceinline__ float centred(float y, int c) const { return __fadd_rn(y, -mean[c / 4]); }
  __device__ __forceinline__ float h(float centred, int c) const { return __fmul_rn(centred, rstd[c / 4]); }
  __device__ __forceinline__ float z(float h, int c) const { return __fadd_rn(__fmul_rn(h, g[c]), s[c]); }
};

__global__ void __launch_bounds__(kThreads) norm_act_kernel(const __nv_bfloat16* __restrict__ y, const float* __restrict__ mean,
                                                            const float* __restrict__ rstd,
                                                            const float* __restrict__ gamma, const float* __restrict__ beta,
                                                            long long V, int C, int G, int iters,
                                                            __nv_bfloat16* __restrict__ out) {
  const int oct = C / 8, o = threadIdx.x % oct, vpb = kThreads / oct, n = blockIdx.y;
  OctetParams P;
  P.load(mean, rstd, gamma, beta, n, o, C, G);
  const uint4* p = reinterpret_cast<const uint4*>(y + (long long)n * V * C) + o;
  uint4* w = reinterpret_cast<uint4*>(out + (long long)n * V * C) + o;
  long long v = (long long)blockIdx.x * vpb * iters + threadIdx.x / oct;
#pragma unroll 4
  for (int k = 0; k < iters; ++k, v += vpb) {
    if (v >= V) break;
    float x[8];
    unpack8(__ldg(p + v * oct), x);
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = gelu(P.z(P.h(P.centred(x[c], c), c), c));
    w[v * oct] = pack8(x);
  }
}

// dz = d_out gelu'(z), dh = dz gamma: direct = dh rstd and slope = dh (y - mean) of each value, and
// partial[n][block][channel] = (sum dz, sum dz h)
__global__ void __launch_bounds__(kThreads) norm_grad_terms_kernel(const __nv_bfloat16* __restrict__ y,
                                                                   const __nv_bfloat16* __restrict__ dout,
                                                                   const float* __restrict__ mean, const float* __restrict__ rstd,
                                                                   const float* __restrict__ gamma,
                                                                   const float* __restrict__ beta, long long V, int C, int G,
                                                                   float4* __restrict__ direct, float4* __restrict__ slope,
                                                                   double2* __restrict__ partial) {
  const int oct = C / 8, o = threadIdx.x % oct, vpb = kThreads / oct, n = blockIdx.y;
  OctetParams P;
  P.load(mean, rstd, gamma, beta, n, o, C, G);
  const uint4* py = reinterpret_cast<const uint4*>(y + (long long)n * V * C) + o;
  const uint4* pd = reinterpret_cast<const uint4*>(dout + (long long)n * V * C) + o;
  const long long step = (long long)gridDim.x * vpb;
  double A[8], B[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) A[c] = B[c] = 0.0;
  for (long long v0 = (long long)blockIdx.x * vpb + threadIdx.x / oct; v0 < V; v0 += step * kChunk) {
    float a[8], b[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = b[c] = 0.0f;
#pragma unroll 2
    for (int k = 0; k < kChunk; ++k) {
      const long long v = v0 + k * step;
      if (v >= V) break;
      float x[8], d[8];
      unpack8(__ldg(py + v * oct), x);
      unpack8(__ldg(pd + v * oct), d);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float e = P.centred(x[c], c), h = P.h(e, c), dz = __fmul_rn(d[c], gelu_slope(P.z(h, c)));
        const float dh = __fmul_rn(dz, P.g[c]);
        a[c] += dz;
        b[c] = fmaf(dz, h, b[c]);
        x[c] = __fmul_rn(dh, P.rstd[c / 4]);
        d[c] = __fmul_rn(dh, e);
      }
      const long long at = (((long long)n * V + v) * oct + o) * 2;
      direct[at] = make_float4(x[0], x[1], x[2], x[3]);
      direct[at + 1] = make_float4(x[4], x[5], x[6], x[7]);
      slope[at] = make_float4(d[0], d[1], d[2], d[3]);
      slope[at + 1] = make_float4(d[4], d[5], d[6], d[7]);
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      A[c] += a[c];
      B[c] += b[c];
    }
  }
  __shared__ double2 sh[kWarps][kMaxC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const double s = octet_sum(A[c], oct), t = octet_sum(B[c], oct);
    if (lane < oct) sh[warp][lane * 8 + c] = make_double2(s, t);
  }
  __syncthreads();
  if ((int)threadIdx.x < C) {
    double s = 0.0, t = 0.0;
    for (int w = 0; w < kWarps; ++w) {
      s += sh[w][threadIdx.x].x;
      t += sh[w][threadIdx.x].y;
    }
    partial[((long long)n * gridDim.x + blockIdx.x) * C + threadIdx.x] = make_double2(s, t);
  }
}

// A block per channel: over the blocks (a warp per sample in turn), then over the samples
__global__ void __launch_bounds__(kThreads) norm_grad_finish_kernel(const double2* __restrict__ partial, int blocks, int N, int C,
                                                                    float* __restrict__ dgamma, float* __restrict__ dbeta) {
  const int c = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ double2 part[kWarps];
  double A = 0.0, B = 0.0;
  for (int n = warp; n < N; n += kWarps) {
    double s = 0.0, t = 0.0;
#pragma unroll 4
    for (int b = lane; b < blocks; b += 32) {
      const double2 v = partial[((long long)n * blocks + b) * C + c];
      s += v.x;
      t += v.y;
    }
    for (int d = 16; d; d >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, d);
      t += __shfl_xor_sync(0xffffffffu, t, d);
    }
    A += s;
    B += t;
  }
  if (lane == 0) part[warp] = make_double2(A, B);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) {
      A += part[w].x;
      B += part[w].y;
    }
    dbeta[c] = (float)A;
    dgamma[c] = (float)B;
  }
}

// dy = (dh rstd + k2 (y - mean)) + k1: k2[n][g] and k1[n][g] are the gradient's parts through the variance and the mean.
// dh is computed again (4 bytes a value) rather than kept (6).
__global__ void __launch_bounds__(kThreads) norm_grad_kernel(const __nv_bfloat16* __restrict__ y,
                                                             const __nv_bfloat16* __restrict__ dout,
                                                             const float* __restrict__ mean, const float* __restrict__ rstd,
                                                             const float* __restrict__ gamma, const float* __restrict__ beta,
                                                             const float* __restrict__ k1, const float* __restrict__ k2,
                                                             long long V, int C, int G, int iters,
                                                             __nv_bfloat16* __restrict__ dy) {
  const int oct = C / 8, o = threadIdx.x % oct, vpb = kThreads / oct, n = blockIdx.y, cg = C / G;
  OctetParams P;
  P.load(mean, rstd, gamma, beta, n, o, C, G);
  float2 m[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int g = n * G + (o * 8 + q * 4) / cg;
    m[q] = make_float2(k1[g], k2[g]);
  }
  const long long base = (long long)n * V * C;
  const uint4* py = reinterpret_cast<const uint4*>(y + base) + o;
  const uint4* pd = reinterpret_cast<const uint4*>(dout + base) + o;
  uint4* w = reinterpret_cast<uint4*>(dy + base) + o;
  long long v = (long long)blockIdx.x * vpb * iters + threadIdx.x / oct;
#pragma unroll 2
  for (int k = 0; k < iters; ++k, v += vpb) {
    if (v >= V) break;
    float x[8], d[8];
    unpack8(__ldg(py + v * oct), x);
    unpack8(__ldg(pd + v * oct), d);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float e = P.centred(x[c], c), dz = __fmul_rn(d[c], gelu_slope(P.z(P.h(e, c), c)));
      const float direct = __fmul_rn(__fmul_rn(dz, P.g[c]), P.rstd[c / 4]);
      x[c] = __fadd_rn(__fadd_rn(direct, __fmul_rn(m[c / 4].y, e)), m[c / 4].x);
    }
    w[v * oct] = pack8(x);
  }
}

int check(const NormShape& s) {
  XAC_REQUIRE(s.N >= 1 && s.N <= 65535 && s.V >= 1 && s.V <= (1ll << 31), "norm_act: batch 1..65535, 1..2^31 voxels");
  XAC_REQUIRE(s.C >= 8 && s.C <= kMaxC && (s.C & (s.C - 1)) == 0, "norm_act: channels must be a power of two, 8..256");
  XAC_REQUIRE(s.G >= 1 && s.C % s.G == 0 && (s.C / s.G) % 4 == 0, "norm_act: a group must hold a multiple of 4 channels");
  return XAC_OK;
}
bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

}  // namespace
}  // namespace xac

using namespace xac;

extern "C" {

int xac_norm_act_scratch_doubles(int N, long long V, int C, int G, long long* count) {
  NormShape s{N, V, C, G};
  int r = check(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(count, "xac_norm_act_scratch_doubles: null pointer");
  *count = 2ll * N * stat_blocks(s) * C;
  return XAC_OK;
}

int xac_norm_act_forward(const void* y, int N, long long V, int C, int G, const float* mean, const float* rstd,
                         const float* gamma, const float* beta, void* out, void* stream) {
  NormShape s{N, V, C, G};
  int r = check(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(y && mean && rstd && gamma && beta && out, "xac_norm_act_forward: null pointer");
  XAC_REQUIRE(aligned16(y) && aligned16(out), "xac_norm_act_forward: volumes must be 16-byte aligned");
  const int iters = apply_iters(s);
  norm_act_kernel<<<dim3(apply_blocks(s, iters), N), kThreads, 0, as_stream(stream)>>>(
      (const __nv_bfloat16*)y, mean, rstd, gamma, beta, V, C, G, iters, (__nv_bfloat16*)out);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

int xac_norm_act_grad_terms(const void* y, const void* d_out, int N, long long V, int C, int G, const float* mean,
                            const float* rstd, const float* gamma, const float* beta, double* scratch, float* direct,
                            float* slope, float* dgamma, float* dbeta, void* stream) {
  NormShape s{N, V, C, G};
  int r = check(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(y && d_out && mean && rstd && gamma && beta && scratch && direct && slope && dgamma && dbeta,
              "xac_norm_act_grad_terms: null pointer");
  XAC_REQUIRE(aligned16(y) && aligned16(d_out) && aligned16(direct) && aligned16(slope) && aligned16(scratch),
              "xac_norm_act_grad_terms: volumes and scratch must be 16-byte aligned");
  cudaStream_t st = as_stream(stream);
  const int blocks = stat_blocks(s);
  norm_grad_terms_kernel<<<dim3(blocks, N), kThreads, 0, st>>>((const __nv_bfloat16*)y, (const __nv_bfloat16*)d_out, mean, rstd,
                                                               gamma, beta, V, C, G, (float4*)direct, (float4*)slope,
                                                               (double2*)scratch);
  norm_grad_finish_kernel<<<C, kThreads, 0, st>>>((const double2*)scratch, blocks, N, C, dgamma, dbeta);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

int xac_norm_act_backward(const void* y, const void* d_out, int N, long long V, int C, int G, const float* mean,
                          const float* rstd, const float* gamma, const float* beta, const float* k1, const float* k2, void* dy,
                          void* stream) {
  NormShape s{N, V, C, G};
  int r = check(s);
  if (r != XAC_OK) return r;
  XAC_REQUIRE(y && d_out && mean && rstd && gamma && beta && k1 && k2 && dy, "xac_norm_act_backward: null pointer");
  XAC_REQUIRE(aligned16(y) && aligned16(d_out) && aligned16(dy), "xac_norm_act_backward: volumes must be 16-byte aligned");
  const int iters = apply_iters(s);
  norm_grad_kernel<<<dim3(apply_blocks(s, iters), N), kThreads, 0, as_stream(stream)>>>(
      (const __nv_bfloat16*)y, (const __nv_bfloat16*)d_out, mean, rstd, gamma, beta, k1, k2, V, C, G, iters, (__nv_bfloat16*)dy);
  XAC_CUDA(cudaGetLastError());
  return XAC_OK;
}

}  // extern "C"
