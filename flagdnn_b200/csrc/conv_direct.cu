// Direct convolution on CUDA cores: one thread per output element, any dtype
// (f16 / bf16 / f32 accumulate in fp32, f64 in fp64), any groups, dilation and
// element strides.  It serves the parts of conv2d's surface the tensor-core
// kernel does not take: grouped and depthwise convolutions, fp64, geometry
// outside the TMA im2col limits, and problems too small to fill the machine
// (the reference covers these with its depthwise and fp64 kernels,
// src/flag_dnn/ops/conv2d.py:2613-2800, 3276-3460).  Index arithmetic follows
// src/flag_dnn/graph/kernels/fused_conv.py:249-299.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "conv_internal.h"

namespace fdnn {
namespace {

template <typename T> struct Acc { using type = float; };
template <> struct Acc<double> { using type = double; };

template <typename T, typename A> __device__ __forceinline__ A ld(const T* p) { return static_cast<A>(*p); }
template <> __device__ __forceinline__ float ld<__half, float>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float ld<__nv_bfloat16, float>(const __nv_bfloat16* p) { return __bfloat162float(*p); }

template <typename T, typename A> __device__ __forceinline__ T cvt(A v) { return static_cast<T>(v); }
template <> __device__ __forceinline__ __half cvt<__half, float>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 cvt<__nv_bfloat16, float>(float v) { return __float2bfloat16_rn(v); }

// Scale, bias, residual, activation, one rounding.
template <typename T, typename A>
__device__ __forceinline__ void finish(const DirectParams& p, A acc, int k, long long y_idx) {
  if (p.scale != nullptr) acc *= ld<T, A>(static_cast<const T*>(p.scale) + k);
  if (p.bias != nullptr) acc += ld<T, A>(static_cast<const T*>(p.bias) + k);
  if (p.residual != nullptr) acc += ld<T, A>(static_cast<const T*>(p.residual) + y_idx);
  if (p.act == FDNN_ACT_RELU) {
    acc = (acc < A(0)) ? A(0) : acc;  // keeps NaN, like torch.relu
  } else if (p.act == FDNN_ACT_GELU) {
    acc = A(0.5) * acc * (A(1) + erf(acc * A(0.70710678118654752440)));
  } else if (p.act == FDNN_ACT_GELU_TANH) {
    const A u = A(0.79788456080286535588) * (acc + A(0.044715) * acc * acc * acc);
    acc = A(0.5) * acc * (A(1) + tanh(u));
  }
  static_cast<T*>(p.y)[y_idx] = cvt<T, A>(acc);
}

template <typename T>
__global__ void __launch_bounds__(256)
conv_direct_kernel(const DirectParams p, const bool k_fastest) {
  using A = typename Acc<T>::type;
  const long long total = (long long)p.N * p.K * p.OH * p.OW;
  const T* x = static_cast<const T*>(p.x);
  const T* w = static_cast<const T*>(p.w);
  const int cg = p.C / p.groups;
  const int kg = p.K / p.groups;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    int n, k, oh, ow;
    long long t = idx;
    if (k_fastest) {  // channels-last output: neighbouring threads write neighbouring channels
      k = int(t % p.K); t /= p.K;
      ow = int(t % p.OW); t /= p.OW;
      oh = int(t % p.OH); t /= p.OH;
      n = int(t);
    } else {
      ow = int(t % p.OW); t /= p.OW;
      oh = int(t % p.OH); t /= p.OH;
      k = int(t % p.K); t /= p.K;
      n = int(t);
    }
    const int g = k / kg;
    A acc = A(0);
    const T* xg = x + n * p.x_s[0] + (long long)(g * cg) * p.x_s[1];
    const T* wk = w + k * p.w_s[0];
    for (int r = 0; r < p.R; ++r) {
      const int ih = oh * p.stride_h + r * p.dil_h - p.pad_top;
      if (ih < 0 || ih >= p.H) continue;
      for (int s = 0; s < p.S; ++s) {
        const int iw = ow * p.stride_w + s * p.dil_w - p.pad_left;
        if (iw < 0 || iw >= p.W) continue;
        const T* xp = xg + ih * p.x_s[2] + iw * p.x_s[3];
        const T* wp = wk + r * p.w_s[2] + s * p.w_s[3];
        for (int c = 0; c < cg; ++c) {
          acc += ld<T, A>(xp + c * p.x_s[1]) * ld<T, A>(wp + c * p.w_s[1]);
        }
      }
    }
    finish<T, A>(p, acc, k, n * p.y_s[0] + k * p.y_s[1] + oh * p.y_s[2] + ow * p.y_s[3]);
  }
}

// The same for long reductions over few outputs: the eight warps of a block share the 32 outputs its lanes stand for and
// take an eighth of the reduction each (a contiguous stretch of (r, s, c), c innermost); the first warp adds the eight
// partial sums in order.  One thread per output is a serial chain of C * R * S loads and FMAs, some 45 ns each: 73 us for
// 1368 of them (4 x 152 x 7 x 13 -> 48 channels 3x3), whatever else the GPU could do meanwhile.
constexpr int kSplitWarps = 8;
template <typename T>
__global__ void __launch_bounds__(kSplitWarps * 32)
conv_direct_split_kernel(const DirectParams p, const bool k_fastest) {
  using A = typename Acc<T>::type;
  __shared__ A part[kSplitWarps][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const long long total = (long long)p.N * p.K * p.OH * p.OW;
  const long long idx = blockIdx.x * 32LL + lane;
  const int cg = p.C / p.groups, kg = p.K / p.groups;
  int n = 0, k = 0, oh = 0, ow = 0;
  A acc = A(0);
  if (idx < total) {
    long long t = idx;
    if (k_fastest) {
      k = int(t % p.K); t /= p.K;
      ow = int(t % p.OW); t /= p.OW;
      oh = int(t % p.OH); t /= p.OH;
    } else {
      ow = int(t % p.OW); t /= p.OW;
      oh = int(t % p.OH); t /= p.OH;
      k = int(t % p.K); t /= p.K;
    }
    n = int(t);
    const T* xg = static_cast<const T*>(p.x) + n * p.x_s[0] + (long long)(k / kg * cg) * p.x_s[1];
    const T* wk = static_cast<const T*>(p.w) + k * p.w_s[0];
    const long long red = (long long)cg * p.R * p.S;
    long long i = red * slice / kSplitWarps;
    const long long end = red * (slice + 1) / kSplitWarps;
    while (i < end) {
      const int tap = int(i / cg), c0 = int(i - (long long)tap * cg);
      const int c1 = int(end - i < cg - c0 ? c0 + (end - i) : cg);
      i += c1 - c0;
      const int r = tap / p.S, s = tap - r * p.S;
      const int ih = oh * p.stride_h + r * p.dil_h - p.pad_top, iw = ow * p.stride_w + s * p.dil_w - p.pad_left;
      if (ih < 0 || ih >= p.H || iw < 0 || iw >= p.W) continue;
      const T* xp = xg + ih * p.x_s[2] + iw * p.x_s[3];
      const T* wp = wk + r * p.w_s[2] + s * p.w_s[3];
#pragma unroll 4
      for (int c = c0; c < c1; ++c) acc += ld<T, A>(xp + c * p.x_s[1]) * ld<T, A>(wp + c * p.w_s[1]);
    }
  }
  part[slice][lane] = acc;
  __syncthreads();
  if (slice != 0 || idx >= total) return;
  for (int i = 1; i < kSplitWarps; ++i) acc += part[i][lane];
  finish<T, A>(p, acc, k, n * p.y_s[0] + k * p.y_s[1] + oh * p.y_s[2] + ow * p.y_s[3]);
}

template <typename T>
cudaError_t go(const DirectParams& p, cudaStream_t stream) {
  const long long total = (long long)p.N * p.K * p.OH * p.OW;
  long long blocks = (total + 255) / 256;
  if (blocks > 148LL * 64) blocks = 148LL * 64;
  if (blocks < 1) blocks = 1;
  const bool k_fastest = p.y_s[1] == 1 && p.K > 1;
  // split where a thread per output would leave the chip idle (under half a wave of threads) on chains worth splitting
  if ((long long)p.C / p.groups * p.R * p.S >= 96 && total <= 148LL * 1024) {
    conv_direct_split_kernel<T><<<unsigned((total + 31) / 32), kSplitWarps * 32, 0, stream>>>(p, k_fastest);
    return cudaGetLastError();
  }
  conv_direct_kernel<T><<<int(blocks), 256, 0, stream>>>(p, k_fastest);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_direct(int dtype, const DirectParams& p, cudaStream_t stream) {
  switch (dtype) {
    case FDNN_F16: return go<__half>(p, stream);
    case FDNN_BF16: return go<__nv_bfloat16>(p, stream);
    case FDNN_F32: return go<float>(p, stream);
    case FDNN_F64: return go<double>(p, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fdnn
