// Pooling next to the convolution path: max_pool2d (the layer after a ResNet
// stem) and adaptive_avg_pool2d (the one before its classifier).  Both are
// HBM-bound maps with a small window, so the kernels are about access order,
// not arithmetic: a thread's linear index walks y in y's own memory order
// (channel fastest for channels-last, width fastest for NCHW), and dense
// channels-last 16-bit tensors move 8 channels (16 bytes) per thread.
//
// Semantics follow torch.nn.functional.max_pool2d / adaptive_avg_pool2d, which
// the reference's operators are tested against
// (src/flag_dnn/ops/max_pool2d.py:174-243, tests/test_max_pool2d.py:49-58;
// src/flag_dnn/ops/adaptive_avg_pool2d.py:456-480): -inf padding, NaN wins a
// maximum, indices are ih * W + iw of the first maximum in scan order; an
// adaptive window is [floor(o * L / O), ceil((o + 1) * L / O)), summed in fp32
// (fp64 for doubles) and divided by its size.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>

#include "conv_convert.cuh"
#include "conv_internal.h"
#include "pool_stretch.h"

namespace fdnn {
namespace {

template <typename T>
struct Acc {
  using type = float;
};
template <>
struct Acc<double> {
  using type = double;
};

template <typename T>
__device__ __forceinline__ typename Acc<T>::type up(T v) {
  if constexpr (sizeof(T) == 2) return to_f32<T>(v);
  else return v;
}
template <typename T>
__device__ __forceinline__ T down(typename Acc<T>::type v) {
  if constexpr (sizeof(T) == 2) return from_f32<T>(v);
  else return static_cast<T>(v);
}

// linear index -> (n, c, oh, ow) in y's memory order.  I is unsigned 32-bit whenever the output has fewer
// than 2^31 elements: four 64-bit divisions per element are what such a kernel would otherwise spend
// its time on.
template <typename I>
__device__ __forceinline__ void unravel(I i, const PoolParams& p, bool c_fastest, int& n, int& c, int& oh,
                                        int& ow) {
  if (c_fastest) {
    c = int(i % I(p.C)); i /= I(p.C);
    ow = int(i % I(p.OW)); i /= I(p.OW);
    oh = int(i % I(p.OH)); n = int(i / I(p.OH));
  } else {
    ow = int(i % I(p.OW)); i /= I(p.OW);
    oh = int(i % I(p.OH)); i /= I(p.OH);
    c = int(i % I(p.C)); n = int(i / I(p.C));
  }
}

template <typename T, typename I>
__global__ void max_pool2d_kernel(const PoolParams p) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.x);
  T* y = static_cast<T*>(p.y);
  const bool c_fastest = p.y_s[1] == 1 && p.C > 1;
  const long long total = (long long)p.N * p.C * p.OH * p.OW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int n, c, oh, ow;
    unravel<I>(I(i), p, c_fastest, n, c, oh, ow);
    const T* xc = x + n * p.x_s[0] + c * p.x_s[1];
    A best = -INFINITY;
    long long best_at = -1;
    for (int r = 0; r < p.kh; ++r) {
      const int ih = oh * p.sh - p.ph + r * p.dh;
      if (ih < 0 || ih >= p.H) continue;
      for (int s = 0; s < p.kw; ++s) {
        const int iw = ow * p.sw - p.pw + s * p.dw;
        if (iw < 0 || iw >= p.W) continue;
        const A v = up<T>(xc[ih * p.x_s[2] + iw * p.x_s[3]]);
        const long long pos = (long long)ih * p.W + iw;
        if (best_at < 0) best_at = pos;  // the window's first element, as torch starts
        if (v > best || v != v) {
          best = v;
          best_at = pos;
        }
      }
    }
    const long long at = n * p.y_s[0] + c * p.y_s[1] + oh * p.y_s[2] + ow * p.y_s[3];
    y[at] = down<T>(best);
    if (p.idx != nullptr) p.idx[at] = best_at;
  }
}

// Maximum of two packed pairs; a NaN on either side wins (and is the canonical one).
template <typename T>
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b);
template <>
__device__ __forceinline__ uint32_t max2<__half>(uint32_t a, uint32_t b) {
  const __half2 r = __hmax2_nan(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <>
__device__ __forceinline__ uint32_t max2<__nv_bfloat16>(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmax2_nan(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <typename T>
__device__ __forceinline__ uint4 max8(const uint4& a, const uint4& b) {
  return make_uint4(max2<T>(a.x, b.x), max2<T>(a.y, b.y), max2<T>(a.z, b.z), max2<T>(a.w, b.w));
}
template <typename T>
__device__ __forceinline__ uint4 lowest8() {   // -inf in every lane
  const uint32_t v = pack2(from_f32<T>(-INFINITY), from_f32<T>(-INFINITY));
  return make_uint4(v, v, v, v);
}

// Dense channels-last 16-bit tensors, C % 8 == 0, no indices: 8 channels per thread.  Maxima are taken on packed 16-bit
// pairs (nothing is rounded by a maximum): widening every element to fp32 and comparing there took 98 us on
// 128 x 64 x 112 x 112 bf16, 2.6 TB/s, bound by instruction issue.
template <typename T, typename I>
__global__ void max_pool2d_nhwc8_kernel(const PoolParams p) {
  const int c8 = p.C / 8;
  const long long total = (long long)p.N * p.OH * p.OW * c8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    I t = I(i);
    const int cv = int(t % I(c8)); t /= I(c8);
    const int ow = int(t % I(p.OW)); t /= I(p.OW);
    const int oh = int(t % I(p.OH));
    const int n = int(t / I(p.OH));
    const T* xc = static_cast<const T*>(p.x) + n * p.x_s[0] + cv * 8;
    uint4 best = lowest8<T>();
    for (int r = 0; r < p.kh; ++r) {
      const int ih = oh * p.sh - p.ph + r * p.dh;
      if (ih < 0 || ih >= p.H) continue;
      for (int s = 0; s < p.kw; ++s) {
        const int iw = ow * p.sw - p.pw + s * p.dw;
        if (iw < 0 || iw >= p.W) continue;
        best = max8<T>(best, __ldg(reinterpret_cast<const uint4*>(xc + ih * p.x_s[2] + iw * p.x_s[3])));
      }
    }
    T* yc = static_cast<T*>(p.y) + n * p.y_s[0] + oh * p.y_s[2] + ow * p.y_s[3] + cv * 8;
    *reinterpret_cast<uint4*>(yc) = best;
  }
}

// 3x3 windows at stride 2 (the pooling after a ResNet stem), same tensors: a thread owns two output rows of a column,
// whose windows share an input row, and asks for all fifteen pixels before it compares.
template <typename T, typename I>
__global__ void __launch_bounds__(256)
max_pool2d_nhwc8_3x3s2_kernel(const PoolParams p) {
  const int c8 = p.C / 8, ohp = (p.OH + 1) / 2;
  const long long total = (long long)p.N * ohp * p.OW * c8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    I t = I(i);
    const int cv = int(t % I(c8)); t /= I(c8);
    const int ow = int(t % I(p.OW)); t /= I(p.OW);
    const int oh = 2 * int(t % I(ohp));
    const int n = int(t / I(ohp));
    const int ih0 = oh * 2 - p.ph, iw0 = ow * 2 - p.pw;
    const T* xc = static_cast<const T*>(p.x) + n * p.x_s[0] + cv * 8;
    const bool two = oh + 1 < p.OH;
    uint4 q[5][3];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int ih = ih0 + r, iw = iw0 + s;
        const bool ok = ih >= 0 && ih < p.H && iw >= 0 && iw < p.W && (r < 3 || two);
        q[r][s] = ok ? __ldg(reinterpret_cast<const uint4*>(xc + ih * p.x_s[2] + iw * p.x_s[3])) : lowest8<T>();
      }
    uint4 row[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) row[r] = max8<T>(max8<T>(q[r][0], q[r][1]), q[r][2]);
    T* yc = static_cast<T*>(p.y) + n * p.y_s[0] + oh * p.y_s[2] + ow * p.y_s[3] + cv * 8;
    *reinterpret_cast<uint4*>(yc) = max8<T>(max8<T>(row[0], row[1]), row[2]);
    if (two) *reinterpret_cast<uint4*>(yc + p.y_s[2]) = max8<T>(max8<T>(row[2], row[3]), row[4]);
  }
}

__device__ __forceinline__ int win_start(int o, int in, int out) { return int(((long long)o * in) / out); }
__device__ __forceinline__ int win_end(int o, int in, int out) { return int(((long long)(o + 1) * in + out - 1) / out); }

template <typename T, typename I>
__global__ void adaptive_avg_pool2d_kernel(const PoolParams p) {
  using A = typename Acc<T>::type;
  const T* x = static_cast<const T*>(p.x);
  T* y = static_cast<T*>(p.y);
  const bool c_fastest = p.y_s[1] == 1 && p.C > 1;
  const long long total = (long long)p.N * p.C * p.OH * p.OW;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int n, c, oh, ow;
    unravel<I>(I(i), p, c_fastest, n, c, oh, ow);
    const int h0 = win_start(oh, p.H, p.OH), h1 = win_end(oh, p.H, p.OH);
    const int w0 = win_start(ow, p.W, p.OW), w1 = win_end(ow, p.W, p.OW);
    const T* xc = x + n * p.x_s[0] + c * p.x_s[1];
    A sum = 0;
    for (int ih = h0; ih < h1; ++ih)
      for (int iw = w0; iw < w1; ++iw) sum += up<T>(xc[ih * p.x_s[2] + iw * p.x_s[3]]);
    y[n * p.y_s[0] + c * p.y_s[1] + oh * p.y_s[2] + ow * p.y_s[3]] = down<T>(sum / A((h1 - h0) * (w1 - w0)));
  }
}

template <typename T, typename I>
__global__ void adaptive_avg_pool2d_nhwc8_kernel(const PoolParams p) {
  const int c8 = p.C / 8;
  const long long total = (long long)p.N * p.OH * p.OW * c8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    I t = I(i);
    const int cv = int(t % I(c8)); t /= I(c8);
    const int ow = int(t % I(p.OW)); t /= I(p.OW);
    const int oh = int(t % I(p.OH));
    const int n = int(t / I(p.OH));
    const int h0 = win_start(oh, p.H, p.OH), h1 = win_end(oh, p.H, p.OH);
    const int w0 = win_start(ow, p.W, p.OW), w1 = win_end(ow, p.W, p.OW);
    const T* xc = static_cast<const T*>(p.x) + n * p.x_s[0] + cv * 8;
    float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int ih = h0; ih < h1; ++ih)
      for (int iw = w0; iw < w1; ++iw) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(xc + ih * p.x_s[2] + iw * p.x_s[3]));
        const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] += to_f32<T>(e[j]);
      }
    const float inv = float((h1 - h0) * (w1 - w0));
    uint4 out;
    out.x = pack2(from_f32<T>(sum[0] / inv), from_f32<T>(sum[1] / inv));
    out.y = pack2(from_f32<T>(sum[2] / inv), from_f32<T>(sum[3] / inv));
    out.z = pack2(from_f32<T>(sum[4] / inv), from_f32<T>(sum[5] / inv));
    out.w = pack2(from_f32<T>(sum[6] / inv), from_f32<T>(sum[7] / inv));
    T* yc = static_cast<T*>(p.y) + n * p.y_s[0] + oh * p.y_s[2] + ow * p.y_s[3] + cv * 8;
    *reinterpret_cast<uint4*>(yc) = out;
  }
}

// The same for few outputs over large windows (a network's last pooling on a small batch): the eight warps of a block
// share 32 channel vectors and take an eighth of the window each; the first adds the eight fp32 sums in order.  One
// thread per output reads its window serially: 11 us for two images of 2048 x 6 x 6.
template <typename T>
__global__ void __launch_bounds__(256)
adaptive_avg_pool2d_nhwc8_split_kernel(const PoolParams p) {
  __shared__ float part[8][32][9];   // rows of nine: no bank conflicts
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int c8 = p.C / 8;
  const long long total = (long long)p.N * p.OH * p.OW * c8;
  const long long i = blockIdx.x * 32LL + lane;
  float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int n = 0, oh = 0, ow = 0, cv = 0;
  long long count = 1;                 // a window can have more pixels than an int counts
  if (i < total) {
    long long t = i;
    cv = int(t % c8); t /= c8;
    ow = int(t % p.OW); t /= p.OW;
    oh = int(t % p.OH);
    n = int(t / p.OH);
    const int h0 = win_start(oh, p.H, p.OH), h1 = win_end(oh, p.H, p.OH);
    const int w0 = win_start(ow, p.W, p.OW), w1 = win_end(ow, p.W, p.OW);
    const int ww = w1 - w0;
    count = (long long)(h1 - h0) * ww;
    const long long k0 = stretch_begin(count, slice, 8), k1 = stretch_begin(count, slice + 1, 8);
    int ih = h0 + int(k0 / ww), iw = w0 + int(k0 % ww);
    const T* xc = static_cast<const T*>(p.x) + n * p.x_s[0] + cv * 8;
#pragma unroll 4
    for (long long k = k0; k < k1; ++k) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(xc + ih * p.x_s[2] + iw * p.x_s[3]));
      if (++iw == w1) {
        iw = w0;
        ++ih;
      }
      const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[j] += to_f32<T>(e[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) part[slice][lane][j] = sum[j];
  __syncthreads();
  if (slice != 0 || i >= total) return;
  for (int k = 1; k < 8; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] += part[k][lane][j];
  const float inv = float(count);
  uint4 out;
  out.x = pack2(from_f32<T>(sum[0] / inv), from_f32<T>(sum[1] / inv));
  out.y = pack2(from_f32<T>(sum[2] / inv), from_f32<T>(sum[3] / inv));
  out.z = pack2(from_f32<T>(sum[4] / inv), from_f32<T>(sum[5] / inv));
  out.w = pack2(from_f32<T>(sum[6] / inv), from_f32<T>(sum[7] / inv));
  T* yc = static_cast<T*>(p.y) + n * p.y_s[0] + oh * p.y_s[2] + ow * p.y_s[3] + cv * 8;
  *reinterpret_cast<uint4*>(yc) = out;
}

bool nhwc8_ok(const PoolParams& p, int es) {
  auto a16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (es != 2 || p.C % 8 != 0 || p.idx != nullptr) return false;
  if (p.x_s[1] != 1 || p.y_s[1] != 1 || !a16(p.x) || !a16(p.y)) return false;
  for (int i : {0, 2, 3})
    if (p.x_s[i] % 8 != 0 || p.y_s[i] % 8 != 0) return false;
  return true;
}

int grid_for(long long work) {
  long long blocks = (work + 255) / 256;
  if (blocks > 148LL * 256) blocks = 148LL * 256;
  return int(blocks < 1 ? 1 : blocks);
}

}  // namespace

#define FDNN_POOL_GO(KERNEL, T)                                            \
  do {                                                                    \
    if (small) KERNEL<T, uint32_t><<<g, 256, 0, stream>>>(p);             \
    else KERNEL<T, unsigned long long><<<g, 256, 0, stream>>>(p);         \
  } while (0)

cudaError_t launch_max_pool2d(int dtype, const PoolParams& p, cudaStream_t stream) {
  const long long total = (long long)p.N * p.C * p.OH * p.OW;
  if (total == 0) return cudaSuccess;
  const bool small = total < (1ll << 31);
  const int es = dtype == FDNN_F64 ? 8 : (dtype == FDNN_F32 ? 4 : 2);
  if (nhwc8_ok(p, es) && p.kh == 3 && p.kw == 3 && p.sh == 2 && p.sw == 2 && p.dh == 1 && p.dw == 1) {
    const int g = grid_for(total / 16 + 1);
    if (dtype == FDNN_F16) FDNN_POOL_GO(max_pool2d_nhwc8_3x3s2_kernel, __half);
    else FDNN_POOL_GO(max_pool2d_nhwc8_3x3s2_kernel, __nv_bfloat16);
    return cudaGetLastError();
  }
  if (nhwc8_ok(p, es)) {
    const int g = grid_for(total / 8);
    if (dtype == FDNN_F16) FDNN_POOL_GO(max_pool2d_nhwc8_kernel, __half);
    else FDNN_POOL_GO(max_pool2d_nhwc8_kernel, __nv_bfloat16);
    return cudaGetLastError();
  }
  const int g = grid_for(total);
  switch (dtype) {
    case FDNN_F16: FDNN_POOL_GO(max_pool2d_kernel, __half); break;
    case FDNN_BF16: FDNN_POOL_GO(max_pool2d_kernel, __nv_bfloat16); break;
    case FDNN_F32: FDNN_POOL_GO(max_pool2d_kernel, float); break;
    case FDNN_F64: FDNN_POOL_GO(max_pool2d_kernel, double); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_adaptive_avg_pool2d(int dtype, const PoolParams& p, cudaStream_t stream) {
  const long long total = (long long)p.N * p.C * p.OH * p.OW;
  if (total == 0) return cudaSuccess;
  const bool small = total < (1ll << 31);
  const int es = dtype == FDNN_F64 ? 8 : (dtype == FDNN_F32 ? 4 : 2);
  // windows of 16 pixels and more (on average), fewer outputs than half of the threads the device holds
  if (nhwc8_ok(p, es) && (long long)p.H * p.W >= 16LL * p.OH * p.OW && total / 8 <= 148LL * 1024) {
    const unsigned g = unsigned((total / 8 + 31) / 32);
    if (dtype == FDNN_F16) adaptive_avg_pool2d_nhwc8_split_kernel<__half><<<g, 256, 0, stream>>>(p);
    else adaptive_avg_pool2d_nhwc8_split_kernel<__nv_bfloat16><<<g, 256, 0, stream>>>(p);
    return cudaGetLastError();
  }
  if (nhwc8_ok(p, es)) {
    const int g = grid_for(total / 8);
    if (dtype == FDNN_F16) FDNN_POOL_GO(adaptive_avg_pool2d_nhwc8_kernel, __half);
    else FDNN_POOL_GO(adaptive_avg_pool2d_nhwc8_kernel, __nv_bfloat16);
    return cudaGetLastError();
  }
  const int g = grid_for(total);
  switch (dtype) {
    case FDNN_F16: FDNN_POOL_GO(adaptive_avg_pool2d_kernel, __half); break;
    case FDNN_BF16: FDNN_POOL_GO(adaptive_avg_pool2d_kernel, __nv_bfloat16); break;
    case FDNN_F32: FDNN_POOL_GO(adaptive_avg_pool2d_kernel, float); break;
    case FDNN_F64: FDNN_POOL_GO(adaptive_avg_pool2d_kernel, double); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
#undef FDNN_POOL_GO

}  // namespace fdnn
