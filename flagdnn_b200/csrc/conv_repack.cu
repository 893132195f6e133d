// Relayout kernels feeding the implicit-GEMM path.
//
// The tensor-core kernel reads activations as NHWC with 16-byte aligned pixel
// rows and filters as [K, R, S, C] with the same channel padding.  Tensors that
// already look like that are consumed in place; everything else (NCHW inputs,
// channel counts that are not a multiple of 16 bytes, fp32 tensors that must be
// split into TF32 halves) passes through one of these kernels first.  The
// filter relayout is the counterpart of the reference's one-time weight packers
// (src/flag_dnn/ops/conv2d.py:193-276).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "conv_internal.h"
#include "sm100_ptx.cuh"

namespace fdnn {
namespace {

// First statement of every kernel here: the next launch of the stream may be set up as soon as all blocks of this one
// run, and nothing of this one touches memory before the launch in front of it is complete (programmatic dependent
// launch, as in the tensor-core kernels: relayout and main kernel are a few microseconds each on small layers).
__device__ __forceinline__ void chain_launches() {
  griddep_launch_dependents();
  griddep_wait();
}
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int threads, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = launch_overlap_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// fp32 -> (hi, lo) with hi = x rounded to TF32 and lo = (x - hi) rounded to
// TF32; hi + lo carries about 21 mantissa bits of x.
__device__ __forceinline__ void split_tf32(float v, float& hi, float& lo) {
  uint32_t h, l;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
  hi = __uint_as_float(h);
  const float rem = v - hi;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(rem));
  lo = __uint_as_float(l);
}

template <typename T>
__device__ __forceinline__ void put(T* dst, long long plane, long long i, T v) {
  if constexpr (std::is_same<T, float>::value) {
    float hi, lo;
    split_tf32(v, hi, lo);
    dst[i] = hi;
    dst[plane + i] = lo;
  } else {
    dst[i] = v;
  }
}

// Generic gather: one thread per destination element, channel fastest.
template <typename T>
__global__ void __launch_bounds__(256)
repack_x_generic(const T* __restrict__ x, long long sn, long long sc, long long sh, long long sw,
                 int N, int C, int H, int W, int c_pad, T* __restrict__ dst, long long plane) {
  chain_launches();
  const long long total = (long long)N * H * W * c_pad;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int c = int(t % c_pad); t /= c_pad;
    const int w = int(t % W); t /= W;
    const int h = int(t % H); t /= H;
    const int n = int(t);
    const T v = (c < C) ? x[n * sn + c * sc + h * sh + w * sw] : T(0.0f);
    put<T>(dst, plane, i, v);
  }
}

// A filter [K, C, R, S] (any strides) as [K, R, S, c_pad]: a thread takes a run of TAPS taps of one input channel of one
// filter, so that a warp reads PyTorch's [K][C][R][S] by contiguous stretches and writes 32 channels of a tap at a time.
// Ten at a time by itself (a 3x3 filter's at once), five in the launch that relays x out.  (Threads that walked all taps of
// their channel left a filter of few channels and many taps to a few warps: 16 -> 16 31x31 63 us, a call on 2 x 64 x 64 NCHW
// 246 us and now 189; conv1d 64 -> 64 of 31 taps on 16 x 2000 28.9 and 20.7.)
template <typename T>
struct PackJob {
  const T* w;
  long long sk, sc, sr, ss;
  int K, C, R, S, c_pad;
  T* dst;
  long long plane;
  int blocks;          // of 256 threads
};
constexpr int kPackTaps = 10, kPackTapsRelayout = 5;
template <typename T, int TAPS>
__device__ __forceinline__ void pack_taps(const PackJob<T>& j, int block) {
  const int taps = j.R * j.S, runs = (taps + TAPS - 1) / TAPS;
  const long long total = (long long)j.K * runs * j.c_pad;
  for (long long i = block * 256LL + threadIdx.x; i < total; i += j.blocks * 256LL) {
    const long long i2 = i / j.c_pad;
    const int c = int(i - i2 * j.c_pad), k = int(i2 / runs), t0 = int(i2 - (long long)k * runs) * TAPS;
    const T* src = j.w + k * j.sk + c * j.sc;
    const long long at = ((long long)k * taps + t0) * j.c_pad + c;
    int r = t0 / j.S, s = t0 - r * j.S;
    T v[TAPS];
#pragma unroll
    for (int u = 0; u < TAPS; ++u) {
      v[u] = (t0 + u < taps && c < j.C) ? src[r * j.sr + s * j.ss] : T(0.0f);
      if (++s == j.S) {
        s = 0;
        ++r;
      }
    }
#pragma unroll
    for (int u = 0; u < TAPS; ++u)
      if (t0 + u < taps) put<T>(j.dst, j.plane, at + (long long)u * j.c_pad, v[u]);
  }
}

// Row-major [C][P] -> [P][c_pad] transposition, the relayout of a tensor whose pixels (or filters) are contiguous:
// NCHW activations (one matrix per image, or per image row when rows are padded), and filters whose K dimension is
// contiguous (mm's second operand).  `mat_stride` elements separate consecutive matrices, `sc` its rows.
//
// Bound by memory traffic: a block moves one tile of 64 columns x 128 bytes of channels through shared memory, so
// that reads are 128 bytes of pixels and writes 128 bytes of channels per quarter warp, 16 bytes per lane (VEC = 1;
// sources whose rows are not 16-byte aligned, VEC = 0, are read one element per lane, 64 contiguous bytes per warp,
// eight loads in flight).  The version with 32 x 32 tiles and one element per lane on both sides that this replaces
// moved 1.2 TB/s on 32 x 128 x 28 x 28 bf16 (10.8 us) and 1.8 TB/s on 30 x 728 x 91 x 32 (142 us).
//
// 16-bit types keep channel pairs as 32-bit words ([64 columns][32 words], rows of 33 words): a lane reads 8 columns
// of two channels and joins them, the writer reads four neighbouring words.
// PACK: the launch's first blocks pack the layer's filter instead (one launch for both where a call brings a filter that is
// not kept packed; as the last blocks they ended 0.8 us after the others, 128 -> 128 3x3 on 32 x 28 x 28).
// The tiles wait for memory, so that blocks per SM count where there are many: eight where the transposition itself lets them
// in, six for reads by element.  Unbounded, every block holds the 50 to 67 registers of the packing ones: 64 -> 64 1x1 on
// 32 x 56 x 56 fp32 23.9 us, now 18.6 (17.1 without a filter to pack), 64 channels of 8 x 112 x 112 39.6 and 34.2 (33.2), bf16 14.5
// and 13.2 (11.7).  FEW: with up to four blocks per SM registers are loads in flight instead (calls of conv1d 136 -> 327 of 5
// taps on 3 x 1265 11.1 us, bounded 12.9; 56 -> 24 5x5 on 94 x 8 x 21 11.0 and 12.3; 256 -> 512 1x1 on 64 x 7 x 7, nothing to pack,
// 9.0 and 10.5).
template <typename T, bool VEC, bool PACK, bool FEW>
__global__ void __launch_bounds__(256, FEW ? 1 : VEC ? 8 : 6)
transpose_repack(const T* __restrict__ x, long long mat_stride, long long mat_stride2, int mats2, long long sc, int mats,
                 int C, int P, int c_pad, T* __restrict__ dst, long long plane, const PackJob<T> pack) {
  chain_launches();
  const int first = PACK ? pack.blocks : 0, blocks = int(gridDim.x) - first;
  if constexpr (PACK) {
    if (int(blockIdx.x) < first) {
      pack_taps<T, kPackTapsRelayout>(pack, int(blockIdx.x));
      return;
    }
  }
  constexpr int kCh = 128 / int(sizeof(T));   // channels per tile: 64 or 32
  constexpr int kVec = 16 / int(sizeof(T));   // elements per 16 bytes
  __shared__ uint32_t tile[64][33];
  const int p_tiles = (P + 63) / 64, c_tiles = (c_pad + kCh - 1) / kCh;
  const long long total = (long long)mats * p_tiles * c_tiles;
  const int tid = threadIdx.x;
  for (long long b = int(blockIdx.x) - first; b < total; b += blocks) {
    // channel tiles innermost: the blocks that share an output row's cache lines run together
    const int ct = int(b % c_tiles);
    const long long b2 = b / c_tiles;
    const int pt = int(b2 % p_tiles);
    const int mat = int(b2 / p_tiles);
    const int p0 = pt * 64, c0 = ct * kCh;
    const T* src = x + (mat / mats2) * mat_stride + (mat % mats2) * mat_stride2;
    if constexpr (sizeof(T) == 2) {
      if constexpr (VEC) {
        const int pv = (tid & 7) * 8, cp = tid >> 3;          // 8 columns of the channel pair cp
        const int c = c0 + 2 * cp, p = p0 + pv;
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (p < P) {                                           // P is a multiple of 8
          if (c < C) lo = __ldg(reinterpret_cast<const uint4*>(src + c * sc + p));
          if (c + 1 < C) hi = __ldg(reinterpret_cast<const uint4*>(src + (c + 1) * sc + p));
        }
        const uint32_t a[4] = {lo.x, lo.y, lo.z, lo.w}, d[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          tile[pv + 2 * i][cp] = __byte_perm(a[i], d[i], 0x5410);
          tile[pv + 2 * i + 1][cp] = __byte_perm(a[i], d[i], 0x7632);
        }
      } else {
        const int px = tid & 63, cq = tid >> 6;                // 64 columns x 4 channel pairs per round
        const uint16_t* s16 = reinterpret_cast<const uint16_t*>(src) + p0 + px;
        const bool p_ok = p0 + px < P;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint16_t v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int c = c0 + 2 * (cq + 4 * (half * 4 + (i >> 1))) + (i & 1);
            v[i] = (p_ok && c < C) ? __ldg(s16 + c * sc) : uint16_t(0);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
            tile[px][cq + 4 * (half * 4 + i)] = uint32_t(v[2 * i]) | (uint32_t(v[2 * i + 1]) << 16);
        }
      }
    } else {
      if constexpr (VEC) {
        const int pv = (tid & 7) * 4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int cl = tid >> 3, c = c0 + cl, p = p0 + pv + h * 32;
          float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (p < P && c < C) q = __ldg(reinterpret_cast<const float4*>(src + c * sc + p));   // P is a multiple of 4
          tile[pv + h * 32 + 0][cl] = __float_as_uint(q.x);
          tile[pv + h * 32 + 1][cl] = __float_as_uint(q.y);
          tile[pv + h * 32 + 2][cl] = __float_as_uint(q.z);
          tile[pv + h * 32 + 3][cl] = __float_as_uint(q.w);
        }
      } else {
        const int px = tid & 63, cq = tid >> 6;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int c = c0 + cq + 4 * i;
          v[i] = (p0 + px < P && c < C) ? __ldg(reinterpret_cast<const float*>(src) + c * sc + p0 + px) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) tile[px][cq + 4 * i] = __float_as_uint(v[i]);
      }
    }
    __syncthreads();
    T* out = dst + (long long)mat * P * c_pad;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int cg = tid & 7, pl = (tid >> 3) + h * 32;        // 16 bytes of channels of one column
      const int p = p0 + pl, c = c0 + cg * kVec;
      if (p < P && c < c_pad) {                                // c_pad is a multiple of kVec
        uint32_t w4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w4[i] = tile[pl][cg * 4 + i];
        T* o = out + (long long)p * c_pad + c;
        if constexpr (sizeof(T) == 2) {
          *reinterpret_cast<uint4*>(o) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
        } else {
          float4 hi, lo;
          split_tf32(__uint_as_float(w4[0]), hi.x, lo.x);
          split_tf32(__uint_as_float(w4[1]), hi.y, lo.y);
          split_tf32(__uint_as_float(w4[2]), hi.z, lo.z);
          split_tf32(__uint_as_float(w4[3]), hi.w, lo.w);
          *reinterpret_cast<float4*>(o) = hi;
          *reinterpret_cast<float4*>(o + plane) = lo;
        }
      }
    }
    __syncthreads();
  }
}

// Channel-contiguous sources (channels-last with a channel count or pixel pitch that is not a multiple of 16 bytes,
// and fp32 channels-last): one lane writes 16 bytes of channels of one pixel, reading them as UNIT-byte pieces (the
// widest the source's alignment allows: consecutive lanes read consecutive pieces).  Bound by memory traffic; one
// element per thread with three 64-bit divisions each, as before, took 24 us for 24 x 45 x 37 pixels of 100 channels.
// UNIT == 16 / 8 / 4 / 2 bytes.  Pixels are evenly spaced (`sw` elements apart) in memory.
template <typename T, int UNIT>
__global__ void __launch_bounds__(256)
repack_rows(const T* __restrict__ x, long long sw, long long pixels, int C, int c_pad, T* __restrict__ dst,
            long long plane) {
  chain_launches();
  constexpr int kVec = 16 / int(sizeof(T));
  const unsigned vecs = unsigned(c_pad / kVec);
  const long long total = pixels * vecs;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long p = i / vecs;
    const int c = int(i - p * vecs) * kVec;
    const char* src = reinterpret_cast<const char*>(x + p * sw + c);
    const int left = (C - c) * int(sizeof(T));                 // bytes of real channels from here on
    uint32_t w4[4] = {0u, 0u, 0u, 0u};
    if (left >= 16) {
      if constexpr (UNIT == 16) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(src));
        w4[0] = q.x; w4[1] = q.y; w4[2] = q.z; w4[3] = q.w;
      } else if constexpr (UNIT == 8) {
        const uint2 q0 = __ldg(reinterpret_cast<const uint2*>(src)), q1 = __ldg(reinterpret_cast<const uint2*>(src) + 1);
        w4[0] = q0.x; w4[1] = q0.y; w4[2] = q1.x; w4[3] = q1.y;
      } else if constexpr (UNIT == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w4[j] = __ldg(reinterpret_cast<const uint32_t*>(src) + j);
      } else {
        const uint16_t* s16 = reinterpret_cast<const uint16_t*>(src);
        uint16_t v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __ldg(s16 + j);
#pragma unroll
        for (int j = 0; j < 4; ++j) w4[j] = uint32_t(v[2 * j]) | (uint32_t(v[2 * j + 1]) << 16);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {                            // the ragged last piece, element by element
        if constexpr (sizeof(T) == 4) {
          if (4 * j < left) w4[j] = __ldg(reinterpret_cast<const uint32_t*>(src) + j);
        } else {
          const uint16_t* s16 = reinterpret_cast<const uint16_t*>(src);
          if (4 * j < left) w4[j] = __ldg(s16 + 2 * j);
          if (4 * j + 2 < left) w4[j] |= uint32_t(__ldg(s16 + 2 * j + 1)) << 16;
        }
      }
    }
    T* o = dst + p * c_pad + c;
    if constexpr (sizeof(T) == 2) {
      *reinterpret_cast<uint4*>(o) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
    } else {
      float4 hi, lo;
      split_tf32(__uint_as_float(w4[0]), hi.x, lo.x);
      split_tf32(__uint_as_float(w4[1]), hi.y, lo.y);
      split_tf32(__uint_as_float(w4[2]), hi.z, lo.z);
      split_tf32(__uint_as_float(w4[3]), hi.w, lo.w);
      *reinterpret_cast<float4*>(o) = hi;
      *reinterpret_cast<float4*>(o + plane) = lo;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) pack_w_kernel(const PackJob<T> job) {
  chain_launches();
  pack_taps<T, kPackTaps>(job, int(blockIdx.x));
}

// Low-channel input relayout: one thread per stored pixel (4 channels = 8 bytes).
template <typename T>
__global__ void __launch_bounds__(256)
repack_x_lowc_kernel(const T* __restrict__ x, long long sn, long long sc, long long sh, long long sw,
                     int N, int C, int H, int W, int pad_left, int w_pad, T* __restrict__ dst) {
  chain_launches();
  const long long total = (long long)N * H * w_pad;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int j = int(t % w_pad); t /= w_pad;
    const int h = int(t % H); t /= H;
    const int n = int(t);
    const int w = j - pad_left;
    T v[4] = {T(0.0f), T(0.0f), T(0.0f), T(0.0f)};
    if (w >= 0 && w < W) {
      const T* src = x + n * sn + h * sh + w * sw;
      for (int c = 0; c < C; ++c) v[c] = src[c * sc];
    }
    uint2 packed;
    packed.x = uint32_t(*reinterpret_cast<uint16_t*>(&v[0])) | (uint32_t(*reinterpret_cast<uint16_t*>(&v[1])) << 16);
    packed.y = uint32_t(*reinterpret_cast<uint16_t*>(&v[2])) | (uint32_t(*reinterpret_cast<uint16_t*>(&v[3])) << 16);
    reinterpret_cast<uint2*>(dst)[i] = packed;
  }
}

// Fast path of the low-channel relayout for a dense 3-channel NHWC source with
// 16-byte aligned rows and W % 8 == 0: one thread turns 8 pixels (48 bytes, three
// aligned 16-byte loads) into 8 four-channel pixels (64 bytes, four aligned stores).
__global__ void __launch_bounds__(256)
repack_x_lowc_c3_kernel(const uint16_t* __restrict__ x, long long sn, long long sh, int N, int H, int W,
                        int pad_left, int w_pad, uint16_t* __restrict__ dst) {
  chain_launches();
  const int w8s = W / 8;
  const long long total = (long long)N * H * w8s;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int w8 = int(t % w8s); t /= w8s;
    const int h = int(t % H); t /= H;
    const int n = int(t);
    const uint4* src = reinterpret_cast<const uint4*>(x + n * sn + h * sh + w8 * 24);
    uint32_t in[12];
    const uint4 a = src[0], b = src[1], c = src[2];
    in[0] = a.x; in[1] = a.y; in[2] = a.z; in[3] = a.w;
    in[4] = b.x; in[5] = b.y; in[6] = b.z; in[7] = b.w;
    in[8] = c.x; in[9] = c.y; in[10] = c.z; in[11] = c.w;
    auto get16 = [&in](int e) -> uint32_t { return (in[e >> 1] >> (16 * (e & 1))) & 0xffffu; };
    uint16_t* row = dst + (((long long)n * H + h) * w_pad) * 4;
    uint4* out = reinterpret_cast<uint4*>(row + (long long)(pad_left + 8 * w8) * 4);
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // two pixels per 16-byte store
      const int p0 = 2 * q, p1 = 2 * q + 1;
      uint4 v;
      v.x = get16(3 * p0) | (get16(3 * p0 + 1) << 16);
      v.y = get16(3 * p0 + 2);
      v.z = get16(3 * p1) | (get16(3 * p1 + 1) << 16);
      v.w = get16(3 * p1 + 2);
      out[q] = v;
    }
    if (w8 == 0) {
      for (int j = 0; j < pad_left; ++j) reinterpret_cast<uint2*>(row)[j] = make_uint2(0u, 0u);
    }
    if (w8 == w8s - 1) {
      for (int j = pad_left + W; j < w_pad; ++j) reinterpret_cast<uint2*>(row)[j] = make_uint2(0u, 0u);
    }
  }
}

// Few-channel input relayout for pixel windows: [N][H][w_pad][8], `pad_left` zero pixels, the image row, zeros to the end;
// channels beyond C are zero.  One lane per stored pixel: 16-byte stores, reads coalesced along W (NCHW) or C * W (NHWC).
__global__ void __launch_bounds__(256)
repack_x_windows_kernel(const uint16_t* __restrict__ x, long long sn, long long sc, long long sh, long long sw, unsigned rows,
                        int C, int H, int W, int pad_left, int w_pad, uint4* __restrict__ dst) {
  chain_launches();
  const unsigned j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= unsigned(w_pad)) return;
  const int w = int(j) - pad_left;
  for (unsigned row = blockIdx.y; row < rows; row += gridDim.y) {
    uint32_t v[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    if (w >= 0 && w < W) {
      const unsigned n = row / unsigned(H), h = row - n * unsigned(H);
      const uint16_t* src = x + n * sn + h * sh + w * sw;
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < C) v[c] = __ldg(src + c * sc);
    }
    dst[(long long)row * w_pad + j] = make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
pack_w_lowc_kernel(const T* __restrict__ w, long long sk, long long sc, long long sr, long long ss, int K,
                   int C, int R, int S, int stride_w, int chans, int shift_elems, T* __restrict__ dst) {
  chain_launches();
  const long long total = 4LL * K * R * 64;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int e = int(t % 64); t /= 64;
    const int r = int(t % R); t /= R;
    const int row = int(t);          // q * K + k
    const int q = row / K, k = row - q * K;
    // element = shift_elems + chans * (stride_w * q + tap) + channel
    const int rel = e - shift_elems - chans * stride_w * q;
    const int s = rel >= 0 ? rel / chans : -1;
    const int c = rel >= 0 ? rel - s * chans : 0;
    T v = T(0.0f);
    if (rel >= 0 && c < C && s < S) v = w[k * sk + c * sc + r * sr + s * ss];
    dst[i] = v;
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
pack_w_grouped_kernel(const T* __restrict__ w, long long sk, long long sc, long long sr, long long ss, int K,
                      int C, int R, int S, int stride_w, int q, int c_pad, T* __restrict__ dst) {
  chain_launches();
  const int sv = S + (q - 1) * stride_w;
  const long long total = (long long)q * K * R * sv * c_pad;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int c = int(t % c_pad); t /= c_pad;
    const int j = int(t % sv); t /= sv;
    const int r = int(t % R); t /= R;
    const int row = int(t);          // g * K + k
    const int g = row / K, k = row - g * K;
    const int s = j - g * stride_w;
    T v = T(0.0f);
    if (c < C && s >= 0 && s < S) v = w[k * sk + c * sc + r * sr + s * ss];
    dst[i] = v;
  }
}

int grid_for(long long work_items, int per_block) {
  long long blocks = (work_items + per_block - 1) / per_block;
  if (blocks > 148LL * 32) blocks = 148LL * 32;
  if (blocks < 1) blocks = 1;
  return int(blocks);
}

template <typename T>
PackJob<T> pack_job(const FilterPack& f, int run) {
  PackJob<T> j = {static_cast<const T*>(f.w), f.strides[0], f.strides[1], f.strides[2], f.strides[3], f.K, f.C, f.R, f.S, f.c_pad,
                  static_cast<T*>(f.dst), (long long)f.K * f.R * f.S * f.c_pad, 0};
  j.blocks = grid_for((long long)f.K * f.c_pad * ((f.R * f.S + run - 1) / run), 256);
  return j;
}

// Transposition of `mats` matrices: matrix i starts at (i / mats2) * ms + (i % mats2) * ms2.
template <typename T>
cudaError_t transpose_t(const T* x, long long ms, long long ms2, int mats2, long long sc, int mats, int C, int P,
                        int c_pad, T* dst, long long plane, cudaStream_t stream, FilterPack* pack = nullptr) {
  constexpr int v = 16 / int(sizeof(T));
  auto mult = [](long long extent, long long stride) { return extent <= 1 || stride % v == 0; };
  const bool vec = P % v == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && mult(C, sc) && mult(mats / mats2, ms) &&
                   mult(mats2, ms2);
  const long long tiles = (long long)mats * ((P + 63) / 64) * ((c_pad + 128 / int(sizeof(T)) - 1) / (128 / int(sizeof(T))));
  PackJob<T> job = {};
  if (pack != nullptr) job = pack_job<T>(*pack, kPackTapsRelayout);
  const int grid = grid_for(tiles, 1) + job.blocks;
  auto pick = [vec](auto packing, auto few) {
    constexpr bool P = decltype(packing)::value, F = decltype(few)::value;
    return vec ? transpose_repack<T, true, P, F> : transpose_repack<T, false, P, F>;
  };
  const bool few = grid <= 4 * current_sm_count();
  auto* kernel = pack == nullptr ? (few ? pick(std::false_type{}, std::true_type{}) : pick(std::false_type{}, std::false_type{}))
                                 : (few ? pick(std::true_type{}, std::true_type{}) : pick(std::true_type{}, std::false_type{}));
  launch_chained(kernel, dim3(grid), 256, stream, x, ms, ms2, mats2, sc, mats, C, P, c_pad, dst, plane, job);
  const cudaError_t e = cudaGetLastError();
  if (pack != nullptr) pack->done = e == cudaSuccess;
  return e;
}

// Rows of channels: `pixels` pixels `sw` elements apart.
template <typename T>
cudaError_t rows_t(const T* x, long long sw, long long pixels, int C, int c_pad, T* dst, long long plane,
                   cudaStream_t stream) {
  const int grid = grid_for(pixels * (c_pad / (16 / int(sizeof(T)))), 256);
  const uintptr_t a = reinterpret_cast<uintptr_t>(x) | (pixels > 1 ? uintptr_t(sw) * sizeof(T) : uintptr_t(0));
  if (a % 16 == 0) launch_chained(repack_rows<T, 16>, dim3(grid), 256, stream, x, sw, pixels, C, c_pad, dst, plane);
  else if (a % 8 == 0) launch_chained(repack_rows<T, 8>, dim3(grid), 256, stream, x, sw, pixels, C, c_pad, dst, plane);
  else if (a % 4 == 0) launch_chained(repack_rows<T, 4>, dim3(grid), 256, stream, x, sw, pixels, C, c_pad, dst, plane);
  else if constexpr (sizeof(T) == 2) launch_chained(repack_rows<T, 2>, dim3(grid), 256, stream,
      x, sw, pixels, C, c_pad, dst, plane);
  else return cudaErrorInvalidValue;   // fp32 elements are 4-byte aligned
  return cudaGetLastError();
}

template <typename T>
cudaError_t pack_w_t(const void* w, const long long s[4], int K, int C, int R, int S, int c_pad, void* dst, long long plane,
                     cudaStream_t stream);

// Which kernel relays a tensor out: pixels contiguous in memory (W innermost; whole planes when rows are not padded,
// else row by row) -> transposition; channels contiguous and pixels evenly spaced -> rows; anything else -> the
// element-wise gather.  Extents of one carry no stride.
template <typename T>
cudaError_t repack_x_t(const void* x, const long long x_s[4], int N, int C, int H, int W, int c_pad,
                       void* dst, long long plane, cudaStream_t stream, FilterPack* pack) {
  long long s[4] = {x_s[0], x_s[1], x_s[2], x_s[3]};
  if (W == 1) {   // a column of pixels is a row of them
    W = H; H = 1;
    s[3] = s[2];
  }
  const T* src = static_cast<const T*>(x);
  T* out = static_cast<T*>(dst);
  if (s[3] == 1 && W > 1 && s[1] != 1) {
    const bool plane_rows = H == 1 || s[2] == W;
    if (plane_rows && (long long)H * W < (1LL << 30))
      return transpose_t<T>(src, s[0], 0, 1, s[1], N, C, H * W, c_pad, out, plane, stream, pack);
    if ((long long)N * H < (1LL << 30))
      return transpose_t<T>(src, s[0], s[2], H, s[1], N * H, C, W, c_pad, out, plane, stream, pack);
  }
  if (pack != nullptr) {   // a launch of its own, and the first one: the shorter of the two is not left for the end
    const cudaError_t e = pack_w_t<T>(pack->w, pack->strides, pack->K, pack->C, pack->R, pack->S, pack->c_pad, pack->dst,
                                      (long long)pack->K * pack->R * pack->S * pack->c_pad, stream);
    if (e != cudaSuccess) return e;
    pack->done = true;
  }
  if ((s[1] == 1 || C == 1) && !(C == 1 && s[3] == 1)) {
    const long long sw = W > 1 ? s[3] : (H > 1 ? s[2] : s[0]);
    const bool even = (W == 1 || H == 1 || s[2] == W * sw) && ((long long)W * H == 1 || N == 1 || s[0] == (long long)W * H * sw);
    if (even) return rows_t<T>(src, sw, (long long)N * H * W, C, c_pad, out, plane, stream);
  }
  const long long total = (long long)N * H * W * c_pad;
  launch_chained(repack_x_generic<T>, dim3(grid_for(total, 256)), 256, stream,
      src, s[0], s[1], s[2], s[3], N, C, H, W, c_pad, out, plane);
  return cudaGetLastError();
}

// Filters: K contiguous and one tap (mm's second operand, [C][K] row-major) -> transposition; otherwise tap by
// tap.
template <typename T>
cudaError_t pack_w_t(const void* w, const long long s[4], int K, int C, int R, int S, int c_pad,
                     void* dst, long long plane, cudaStream_t stream) {
  const T* src = static_cast<const T*>(w);
  T* out = static_cast<T*>(dst);
  if (R * S == 1 && s[0] == 1 && K > 1 && s[1] != 1)
    return transpose_t<T>(src, 0, 0, 1, s[1], 1, C, K, c_pad, out, plane, stream);
  FilterPack f = {w, {s[0], s[1], s[2], s[3]}, K, C, R, S, c_pad, dst, false};
  const PackJob<T> job = pack_job<T>(f, kPackTaps);
  launch_chained(pack_w_kernel<T>, dim3(job.blocks), 256, stream, job);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_repack_x(int dtype, const void* x, const long long x_s[4], int N, int C, int H,
                            int W, int c_pad, void* dst, long long plane_elems,
                            cudaStream_t stream, FilterPack* pack) {
  switch (dtype) {
    case FDNN_F16: return repack_x_t<__half>(x, x_s, N, C, H, W, c_pad, dst, plane_elems, stream, pack);
    case FDNN_BF16: return repack_x_t<__nv_bfloat16>(x, x_s, N, C, H, W, c_pad, dst, plane_elems, stream, pack);
    case FDNN_F32: return repack_x_t<float>(x, x_s, N, C, H, W, c_pad, dst, plane_elems, stream, pack);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_repack_x_lowc(int dtype, const void* x, const long long x_s[4], int N, int C, int H,
                                 int W, int pad_left, int w_pad, void* dst, cudaStream_t stream) {
  const bool fast = (dtype == FDNN_F16 || dtype == FDNN_BF16) && C == 3 && x_s[1] == 1 && x_s[3] == 3 &&
                    W % 8 == 0 && pad_left % 2 == 0 && x_s[2] % 8 == 0 && (N <= 1 || x_s[0] % 8 == 0) &&
                    (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  if (fast) {
    const long long items = (long long)N * H * (W / 8);
    launch_chained(repack_x_lowc_c3_kernel, dim3(grid_for(items, 256)), 256, stream,
        static_cast<const uint16_t*>(x), x_s[0], x_s[2], N, H, W, pad_left, w_pad, static_cast<uint16_t*>(dst));
    return cudaGetLastError();
  }
  const long long total = (long long)N * H * w_pad;
  const int grid = grid_for(total, 256);
  if (dtype == FDNN_F16) {
    launch_chained(repack_x_lowc_kernel<__half>, dim3(grid), 256, stream,
        static_cast<const __half*>(x), x_s[0], x_s[1], x_s[2], x_s[3], N, C, H, W, pad_left, w_pad,
        static_cast<__half*>(dst));
  } else if (dtype == FDNN_BF16) {
    launch_chained(repack_x_lowc_kernel<__nv_bfloat16>, dim3(grid), 256, stream,
        static_cast<const __nv_bfloat16*>(x), x_s[0], x_s[1], x_s[2], x_s[3], N, C, H, W, pad_left, w_pad,
        static_cast<__nv_bfloat16*>(dst));
  } else {
    return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_repack_x_windows(const void* x, const long long x_s[4], int N, int C, int H, int W, int pad_left,
                                    int w_pad, void* dst, cudaStream_t stream) {
  const int threads = w_pad >= 256 ? 256 : (w_pad + 31) / 32 * 32;
  const long long rows = (long long)N * H;
  const dim3 grid(unsigned((w_pad + threads - 1) / threads), unsigned(rows < 32768 ? rows : 32768));
  launch_chained(repack_x_windows_kernel, grid, threads, stream,
      static_cast<const uint16_t*>(x), x_s[0], x_s[1], x_s[2], x_s[3], unsigned(rows), C, H, W, pad_left, w_pad,
      static_cast<uint4*>(dst));
  return cudaGetLastError();
}

cudaError_t launch_pack_w_lowc(int dtype, const void* w, const long long w_s[4], int K, int C, int R,
                               int S, int stride_w, int chans, int shift_elems, void* dst, cudaStream_t stream) {
  const long long total = 4LL * K * R * 64;
  const int grid = grid_for(total, 256);
  if (dtype == FDNN_F16) {
    launch_chained(pack_w_lowc_kernel<__half>, dim3(grid), 256, stream,
        static_cast<const __half*>(w), w_s[0], w_s[1], w_s[2], w_s[3], K, C, R, S, stride_w, chans, shift_elems,
        static_cast<__half*>(dst));
  } else if (dtype == FDNN_BF16) {
    launch_chained(pack_w_lowc_kernel<__nv_bfloat16>, dim3(grid), 256, stream,
        static_cast<const __nv_bfloat16*>(w), w_s[0], w_s[1], w_s[2], w_s[3], K, C, R, S, stride_w, chans,
        shift_elems, static_cast<__nv_bfloat16*>(dst));
  } else {
    return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_pack_w_grouped(int dtype, const void* w, const long long w_s[4], int K, int C, int R,
                                  int S, int stride_w, int q, int c_pad, void* dst, cudaStream_t stream) {
  const long long total = (long long)q * K * R * (S + (q - 1) * stride_w) * c_pad;
  const int grid = grid_for(total, 256);
  if (dtype == FDNN_F16) {
    launch_chained(pack_w_grouped_kernel<__half>, dim3(grid), 256, stream,
        static_cast<const __half*>(w), w_s[0], w_s[1], w_s[2], w_s[3], K, C, R, S, stride_w, q, c_pad,
        static_cast<__half*>(dst));
  } else if (dtype == FDNN_BF16) {
    launch_chained(pack_w_grouped_kernel<__nv_bfloat16>, dim3(grid), 256, stream,
        static_cast<const __nv_bfloat16*>(w), w_s[0], w_s[1], w_s[2], w_s[3], K, C, R, S, stride_w, q, c_pad,
        static_cast<__nv_bfloat16*>(dst));
  } else {
    return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// A grouped filter [K][C/G][R][S] (any strides) written as the dense channels-last filter [K][R][S][C] of the
// same convolution: filter k keeps its group's C/G channels at their place among the C input channels and is zero
// everywhere else (a block-diagonal GEMM operand).
template <typename T>
__global__ void densify_w_kernel(const T* __restrict__ w, long long s0, long long s1, long long s2, long long s3, int K,
                                 int C, int R, int S, int groups, T* __restrict__ dense) {
  chain_launches();
  const long long total = (long long)K * R * S * C;
  const int cg = C / groups, kg = K / groups;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i;
    const int c = int(t % C); t /= C;
    const int s = int(t % S); t /= S;
    const int r = int(t % R); t /= R;
    const int k = int(t);
    const int local = c - (k / kg) * cg;
    T v = static_cast<T>(0.0f);
    if (local >= 0 && local < cg) v = w[k * s0 + local * s1 + r * s2 + s * s3];
    dense[i] = v;
  }
}

template <typename T>
cudaError_t densify_w_t(const void* w, const long long w_s[4], int K, int C, int R, int S, int groups, void* dense,
                        cudaStream_t stream) {
  const long long total = (long long)K * R * S * C;
  long long blocks = (total + 255) / 256;
  if (blocks > 148LL * 16) blocks = 148LL * 16;
  if (blocks < 1) blocks = 1;
  launch_chained(densify_w_kernel<T>, dim3(int(blocks)), 256, stream,
      static_cast<const T*>(w), w_s[0], w_s[1], w_s[2], w_s[3], K, C, R, S, groups, static_cast<T*>(dense));
  return cudaGetLastError();
}

cudaError_t launch_densify_w(int dtype, const void* w, const long long w_s[4], int K, int C, int R, int S, int groups,
                             void* dense, cudaStream_t stream) {
  switch (dtype) {
    case FDNN_F16: return densify_w_t<__half>(w, w_s, K, C, R, S, groups, dense, stream);
    case FDNN_BF16: return densify_w_t<__nv_bfloat16>(w, w_s, K, C, R, S, groups, dense, stream);
    case FDNN_F32: return densify_w_t<float>(w, w_s, K, C, R, S, groups, dense, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_pack_w(int dtype, const void* w, const long long w_s[4], int K, int C, int R,
                          int S, int c_pad, void* dst, long long plane_elems, cudaStream_t stream) {
  switch (dtype) {
    case FDNN_F16: return pack_w_t<__half>(w, w_s, K, C, R, S, c_pad, dst, plane_elems, stream);
    case FDNN_BF16: return pack_w_t<__nv_bfloat16>(w, w_s, K, C, R, S, c_pad, dst, plane_elems, stream);
    case FDNN_F32: return pack_w_t<float>(w, w_s, K, C, R, S, c_pad, dst, plane_elems, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fdnn
