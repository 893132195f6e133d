// Depthwise convolution of dense NCHW tensors: whole planes through a ring in shared memory.
//
// A block takes groups of consecutive (image, channel) planes, which lie one after another in x and in y: one bulk copy
// brings a group in while the one before is computed, one bulk copy takes its outputs out.  A thread owns a strip of PX
// neighbouring output columns of a band of output rows of TWO planes and walks down the band: every input row is read
// once (a 16-byte piece and the columns beside it), widened once, and added to the ceil(K / stride) output rows it
// belongs to, whose accumulators stay in registers; the same column of the two planes shares an fma.rn.f32x2.  (Pairs of
// neighbouring columns need a second, shifted set of pairs: 117 instructions beside the 36 multiplications of a row of
// eight outputs, 75.6 us.)
//
// What bounds depthwise_rowvec_kernel, which reads its windows from global memory: three reads and widenings of every
// input, 34 instructions per output, and waiting for its own loads with few in flight.  64 channels of 256 x 56 x 56,
// 3x3, bf16: 78.5 us there, 74.6 here, of 31.8 us for the bytes at 6458 GB/s.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>
#include <type_traits>

#include "conv_convert.cuh"
#include "conv_epilogue.cuh"
#include "conv_internal.h"
#include "f32x2.cuh"
#include "sm100_ptx.cuh"

namespace fdnn {
namespace {

// Threads per block: 3x3 layers take some 120 registers, 5x5 layers up to 250.  Two blocks of 256 threads per SM beat one of
// 512 where rows are whole 16-byte pieces (64 channels of 256 x 56 x 56: 74.6 and 84.1 us) and lose or tie elsewhere, with
// half the shared memory each (77 channels of 50 x 110 x 110 do not fit).
template <int K, int BLOCKS> constexpr int kThreadsOf = K == 3 && BLOCKS == 1 ? 512 : 256;
constexpr int smem_of(int blocks) { return 226 * 1024 / blocks - (blocks > 1 ? 1024 : 0); }
constexpr int kMaxStages = 6;

struct RingParams {
  const void* x;
  const void* w;
  const void* bias;
  const void* scale;
  void* y;
  int C, H, W, OH, OW;
  long long planes;              // N * C
  long long w_s0, w_s2, w_s3;
  int group;                     // planes per group
  int strips, bands, band_rows;
  int stages, outs;              // ring slots, output buffers
  int in_bytes, out_bytes;       // of a slot and of an output buffer (multiples of 128)
  int act;
  uint32_t* status;
  long long wait_limit;
};

// VB bytes of a row's elements of both planes (at a and b), as pairs; zeros where they do not exist.
template <typename T, int VB>
__device__ __forceinline__ void load_pairs(uint32_t a, uint32_t b, bool ok, F2* v) {
  if constexpr (VB == 16) {
    uint4 p = make_uint4(0u, 0u, 0u, 0u), q = p;
    if (ok) {
      p = lds_v4(a);
      q = lds_v4(b);
    }
    const uint32_t pw[4] = {p.x, p.y, p.z, p.w}, qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (sizeof(T) == 4) {
        v[i] = f2_make(pw[i], qw[i]);
      } else {
        float p0, p1, q0, q1;
        unpack2<T>(pw[i], p0, p1);
        unpack2<T>(qw[i], q0, q1);
        v[2 * i] = f2_make(__float_as_uint(p0), __float_as_uint(q0));
        v[2 * i + 1] = f2_make(__float_as_uint(p1), __float_as_uint(q1));
      }
    }
  } else {
    uint32_t p = 0u, q = 0u;
    if (ok) {
      p = VB == 4 ? lds_u32(a) : uint32_t(lds_u16(a));
      q = VB == 4 ? lds_u32(b) : uint32_t(lds_u16(b));
    }
    if constexpr (sizeof(T) == 4) {
      v[0] = f2_make(p, q);
    } else {
      float p0, p1, q0, q1;
      unpack2<T>(p, p0, p1);
      unpack2<T>(q, q0, q1);
      v[0] = f2_make(__float_as_uint(p0), __float_as_uint(q0));
      if constexpr (VB == 4) v[1] = f2_make(__float_as_uint(p1), __float_as_uint(q1));
    }
  }
}

// One plane's finished outputs of a row to shared memory; `left` of them exist.
template <typename T, int PX>
__device__ __forceinline__ void store_strip(uint32_t a, const float (&f)[PX], int act, int unit, int left) {
  if constexpr (sizeof(T) == 4) {
    uint32_t h[PX];
#pragma unroll
    for (int q = 0; q < PX; ++q) h[q] = __float_as_uint(act == 1 ? relu_keep_nan(f[q]) : f[q]);
    if (unit == 16) {
      if constexpr (PX == 4) sts_v4(a, make_uint4(h[0], h[1], h[2], h[3]));
      else sts_v2(a, make_uint2(h[0], h[1]));
    } else {
#pragma unroll
      for (int q = 0; q < PX; ++q)
        if (q < left) sts_u32(a + 4 * q, h[q]);
    }
  } else {
    uint32_t h[PX / 2];
#pragma unroll
    for (int q = 0; q < PX / 2; ++q) h[q] = act == 1 ? round_pack2_relu<T>(f[2 * q], f[2 * q + 1]) : round_pack2<T>(f[2 * q], f[2 * q + 1]);
    if (unit == 16) {
      if constexpr (PX == 8) sts_v4(a, make_uint4(h[0], h[1], h[2], h[3]));
      else sts_v2(a, make_uint2(h[0], h[1]));
    } else if (unit == 4) {
#pragma unroll
      for (int q = 0; q < PX / 2; ++q)
        if (2 * q < left) sts_u32(a + 4 * q, h[q]);
    } else {
#pragma unroll
      for (int q = 0; q < PX; ++q)
        if (q < left) sts_u16(a + 2 * q, uint16_t(h[q / 2] >> (16 * (q % 2))));
    }
  }
}

// K x K taps at stride ST; PX outputs of a row per thread; VB: rows start on this many bytes (16, 4 or one element).
template <typename T, int K, int ST, int PX, int VB, int BLOCKS>
__global__ void __launch_bounds__(kThreadsOf<K, BLOCKS>, BLOCKS)
depthwise_ring_kernel(const RingParams p) {
  constexpr int kEs = int(sizeof(T));
  constexpr int kThreads = kThreadsOf<K, BLOCKS>;
  constexpr int kPad = K / 2;
  constexpr int kIn = PX * ST;                    // input columns of a strip's own
  constexpr int kSpan = (PX - 1) * ST + K;        // columns its outputs read, from kPad to its left
  constexpr int kLive = (K + ST - 1) / ST;        // output rows an input row belongs to, at most
  constexpr int kPeriod = kLive * ST;
  static_assert(kIn * kEs == 16, "a strip's own columns are one piece");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint8_t* out = smem + p.stages * p.in_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(out + p.outs * p.out_bytes);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(full + kMaxStages);
  const long long plane_in = (long long)p.H * p.W * kEs, plane_out = (long long)p.OH * p.OW * kEs;
  const long long groups = (p.planes + p.group - 1) / p.group;
  const uint8_t* x = static_cast<const uint8_t*>(p.x);
  uint8_t* y = static_cast<uint8_t*>(p.y);

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) mbar_init(&full[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  auto planes_of = [&](long long g) { return int(p.planes - g * p.group < p.group ? p.planes - g * p.group : p.group); };
  auto ask = [&](long long g, int slot) {   // the last group's bytes past a multiple of 16 are read below
    const uint32_t bytes = uint32_t(planes_of(g) * plane_in) & ~15u;
    mbar_arrive_expect_tx(&full[slot], bytes);
    if (bytes != 0) bulk_load_1d(smem + slot * p.in_bytes, x + g * p.group * plane_in, bytes, &full[slot]);
  };
  int asked = 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      const long long g = blockIdx.x + (long long)s * gridDim.x;
      if (g < groups) {
        ask(g, s);
        ++asked;
      }
    }
  }
  const int per_plane = p.strips * p.bands;
  // how a strip's outputs go to shared memory: as one unit, by words, or one by one
  const int unit = p.OW % PX == 0 ? 16 : (kEs == 4 || p.OW % 2 == 0) ? 4 : 2;
  int slot = 0, buf = 0;
  uint32_t phase = 0;
  int done = 0;
  for (long long g = blockIdx.x; g < groups; g += gridDim.x, ++done, buf ^= p.outs - 1) {
    const int here = planes_of(g);
    uint8_t* in = smem + slot * p.in_bytes;
    const bool landed = mbar_wait_bounded(&full[slot], phase, abort_flag, p.status, kIncidentDepthwiseWait, p.wait_limit);
    {
      const int bytes = int(here * plane_in), left = bytes & 15;
      if (int(threadIdx.x) < left / kEs) {
        const int at = (bytes & ~15) + int(threadIdx.x) * kEs;
        *reinterpret_cast<T*>(in + at) = *reinterpret_cast<const T*>(x + g * p.group * plane_in + at);
      }
    }
    if (p.outs == 1 && threadIdx.x == 0) bulk_wait_group_read0();   // the only output buffer has been read
    if (__syncthreads_and(landed) == 0) break;
    for (int task = threadIdx.x; task < (here + 1) / 2 * per_plane; task += kThreads) {
      const int pair = task / per_plane;
      const int rest = task - pair * per_plane;
      const int band = rest / p.strips;
      const int strip = rest - band * p.strips;
      const int pl0 = 2 * pair, pl1 = 2 * pair + 1 < here ? 2 * pair + 1 : pl0;   // the last plane of an odd count: with itself
      const long long first = g * p.group + pl0;
      const int c0 = int(first % p.C), c1 = pl1 == pl0 ? c0 : (c0 + 1 == p.C ? 0 : c0 + 1);
      const T *w0 = static_cast<const T*>(p.w) + c0 * p.w_s0, *w1 = static_cast<const T*>(p.w) + c1 * p.w_s0;
      F2 wt[K * K];
#pragma unroll
      for (int i = 0; i < K * K; ++i) {
        const long long at = (i / K) * p.w_s2 + (i % K) * p.w_s3;
        wt[i] = f2_make(__float_as_uint(to_f32<T>(__ldg(w0 + at))), __float_as_uint(to_f32<T>(__ldg(w1 + at))));
      }
      auto per_channel = [&](const void* v, float none) {
        const T* t = static_cast<const T*>(v);
        return t == nullptr ? f2_make(__float_as_uint(none), __float_as_uint(none))
                            : f2_make(__float_as_uint(to_f32<T>(t[c0])), __float_as_uint(to_f32<T>(t[c1])));
      };
      const F2 sc2 = per_channel(p.scale, 1.0f), bi2 = per_channel(p.bias, 0.0f);
      const int oh0 = band * p.band_rows;
      const int rows_out = p.OH - oh0 < p.band_rows ? p.OH - oh0 : p.band_rows;
      const int rows_in = (rows_out - 1) * ST + K;
      const int col0 = strip * kIn;                             // first own column; the windows start kPad to its left
      const int row_bytes = p.W * kEs;
      const int ih0 = oh0 * ST - kPad;
      // row t of the band, own columns of the first plane; the second plane lies `apart` bytes on
      uint32_t a = smem_u32(in) + uint32_t(pl0 * int(plane_in) + ih0 * row_bytes + col0 * kEs);
      const uint32_t apart = uint32_t(pl1 - pl0) * uint32_t(plane_in);
      uint32_t o = smem_u32(out) + uint32_t(buf * p.out_bytes + pl0 * int(plane_out) + (oh0 * p.OW + strip * PX) * kEs);
      const uint32_t o_apart = uint32_t(pl1 - pl0) * uint32_t(plane_out), o_row = uint32_t(p.OW * kEs);
      const int left = p.OW - strip * PX;
      F2 acc[kLive][PX];
#pragma unroll
      for (int l = 0; l < kLive; ++l)
#pragma unroll
        for (int q = 0; q < PX; ++q) acc[l][q] = 0ull;
      for (int t0 = 0; t0 < rows_in; t0 += kPeriod) {
#pragma unroll
        for (int u = 0; u < kPeriod; ++u) {
          const int t = t0 + u;
          if (t < rows_in) {
            if (unsigned(ih0 + t) < unsigned(p.H)) {
              F2 v[kPad + kIn + K];                             // columns col0 - kPad ..
#pragma unroll
              for (int j = 0; j < kPad; ++j)
                load_pairs<T, kEs>(a - (kPad - j) * kEs, a + apart - (kPad - j) * kEs, col0 - kPad + j >= 0, v + j);
#pragma unroll
              for (int j = 0; j < kIn; j += VB / kEs)
                load_pairs<T, VB>(a + j * kEs, a + apart + j * kEs, VB == 16 || col0 + j < p.W, v + kPad + j);
#pragma unroll
              for (int j = kIn; j < kSpan - kPad; ++j)
                load_pairs<T, kEs>(a + j * kEs, a + apart + j * kEs, col0 + j < p.W, v + kPad + j);
#pragma unroll
              for (int s = 0; s < K; ++s) {
#pragma unroll
                for (int q = 0; q < PX; ++q) {
#pragma unroll
                  for (int r = 0; r < K; ++r) {
                    if ((u - r + kPeriod * K) % ST == 0) {      // row r of the window belongs to output row (t - r) / ST
                      const int l = ((u - r + kPeriod * K) / ST) % kLive;
                      acc[l][q] = f2_fma(v[q * ST + s], wt[r * K + s], acc[l][q]);
                    }
                  }
                }
              }
            }
            a += row_bytes;
            if ((u - (K - 1) + kPeriod * K) % ST == 0) {         // the window's last row: an output row is complete
              const int l = ((u - (K - 1) + kPeriod * K) / ST) % kLive;
              if (t >= K - 1) {
                float f0[PX], f1[PX];
#pragma unroll
                for (int q = 0; q < PX; ++q) f2_split(f2_fma(acc[l][q], sc2, bi2), f0[q], f1[q]);
                store_strip<T, PX>(o, f0, p.act, unit, left);
                if (pl1 != pl0) store_strip<T, PX>(o + o_apart, f1, p.act, unit, left);
                o += o_row;
              }
#pragma unroll
              for (int q = 0; q < PX; ++q) acc[l][q] = 0ull;
            }
          }
        }
      }
    }
    // outputs out, the slot free, and (with two buffers) the one the next group writes to read by its store
    fence_proxy_async_smem();
    if (p.outs == 2 && threadIdx.x == 0) bulk_wait_group_read0();
    __syncthreads();
    const int bytes = int(here * plane_out);
    uint8_t* dst = y + g * p.group * plane_out;
    const uint8_t* src = out + buf * p.out_bytes;
    if (threadIdx.x == 0) {
      if (bytes >= 16) bulk_store_1d(dst, src, uint32_t(bytes) & ~15u);
      bulk_commit_group();
      const long long ahead = g + (long long)p.stages * gridDim.x;
      if (ahead < groups) {
        ask(ahead, slot);
        ++asked;
      }
    }
    if (int(threadIdx.x) < (bytes & 15) / kEs) {
      const int at = (bytes & ~15) + int(threadIdx.x) * kEs;
      *reinterpret_cast<T*>(dst + at) = *reinterpret_cast<const T*>(src + at);
    }
    if (++slot == p.stages) {
      slot = 0;
      phase ^= 1u;
    }
  }
  if (threadIdx.x == 0) {
    bulk_wait_group0();
    if (*abort_flag) {   // after an incident: give the copies in flight time to land
      volatile uint32_t never = 0;
      for (int i = done; i < asked; ++i)
        mbar_wait_bounded(&full[i % p.stages], uint32_t(i / p.stages) & 1u, &never, p.status, kIncidentDrainWait, kWaitLimitCycles / 16);
    }
  }
}

long long gcd(long long a, long long b) { return b == 0 ? a : gcd(b, a % b); }

// Planes a group is a multiple of: groups start on 16 bytes in x and in y, and hold pairs.
long long group_unit(const DirectParams& p, int es) {
  const long long in = 16 / gcd((long long)p.H * p.W * es, 16), out = 16 / gcd((long long)p.OH * p.OW * es, 16);   // powers of two
  const long long unit = in > out ? in : out;
  return unit < 2 ? 2 : unit;
}
long long slot_bytes(const DirectParams& p, int es, long long planes, bool out) {
  return (planes * (out ? (long long)p.OH * p.OW : (long long)p.H * p.W) * es + 127) / 128 * 128;
}
constexpr long long kFixedBytes = (kMaxStages + 2) * 8 + 128;

// How a launch divides the work, or group 0 where no group fits: the cheapest split by rounds of a block's threads times
// the rows a thread walks, over the groups an SM gets.  A handful of candidates: it runs on every call.
struct RingSplit {
  int group, bands, band_rows, strips, stages, outs, in_bytes, out_bytes;
  size_t smem;
};
RingSplit ring_split(const DirectParams& p, int es, int px, int k, int st, int threads, int per_sm) {
  const int limit = smem_of(per_sm), blocks = current_sm_count() * per_sm;
  RingSplit best = {};
  const long long unit = group_unit(p, es), planes = (long long)p.N * p.C;
  const int strips = (p.OW + px - 1) / px;
  double best_cost = 1e300;
  for (long long g = unit; g <= 256; g += g / 4 < unit ? unit : g / 4 / unit * unit) {
    const long long in_b = slot_bytes(p, es, g, false), out_b = slot_bytes(p, es, g, true);
    if (2 * in_b + out_b + kFixedBytes > limit) break;
    const double per_block = double(((planes + g - 1) / g + blocks - 1) / blocks);
    for (int outs = 1; outs <= 2; ++outs) {
      const long long fixed = outs * out_b + kFixedBytes;
      if (2 * in_b + fixed > limit) continue;
      const int stages = (limit - fixed) / in_b > 2 ? 3 : 2;
      for (int rounds = 1; rounds <= 3; ++rounds) {
        long long bands = rounds * threads / (g / 2 * strips);
        if (bands > p.OH) bands = p.OH;
        if (bands < 1) bands = 1;
        const int rows = int((p.OH + bands - 1) / bands);
        bands = (p.OH + rows - 1) / rows;
        const long long tasks = g / 2 * bands * strips;
        const double cost = per_block * (double((tasks + threads - 1) / threads) * ((rows - 1) * st + k + 3) + (outs == 1 ? 4 : 2)) *
                            (stages > 2 ? 1.0 : 1.05);
        if (cost < best_cost) {
          best_cost = cost;
          best = {int(g), int(bands), rows, strips, stages, outs, int(in_b), int(out_b), size_t(stages * in_b + fixed)};
        }
      }
    }
  }
  return best;
}

template <typename T, int K, int ST, int VB, int BLOCKS>
cudaError_t launch_ring_k(const DirectParams& d, uint32_t* status, long long wait_limit, cudaStream_t stream) {
  constexpr int kEs = int(sizeof(T)), kPx = 16 / kEs / ST;
  const RingSplit s = ring_split(d, kEs, kPx, K, ST, kThreadsOf<K, BLOCKS>, BLOCKS);
  if (s.group == 0) return cudaErrorInvalidValue;
  RingParams p = {};
  p.x = d.x; p.w = d.w; p.bias = d.bias; p.scale = d.scale; p.y = d.y;
  p.C = d.C; p.H = d.H; p.W = d.W; p.OH = d.OH; p.OW = d.OW;
  p.planes = (long long)d.N * d.C;
  p.w_s0 = d.w_s[0]; p.w_s2 = d.w_s[2]; p.w_s3 = d.w_s[3];
  p.group = s.group; p.strips = s.strips; p.bands = s.bands; p.band_rows = s.band_rows;
  p.stages = s.stages; p.outs = s.outs; p.in_bytes = s.in_bytes; p.out_bytes = s.out_bytes;
  p.act = d.act;
  p.status = status;
  p.wait_limit = wait_limit;
  const long long groups = (p.planes + p.group - 1) / p.group;
  long long grid = (long long)current_sm_count() * BLOCKS;
  if (grid > groups) grid = groups;
  auto* kernel = depthwise_ring_kernel<T, K, ST, kPx, VB, BLOCKS>;
  static std::atomic<bool> ready[64];       // per device: shared-memory limit raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!ready[dev & 63].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_of(BLOCKS));
    if (e != cudaSuccess) return e;
    ready[dev & 63].store(true, std::memory_order_release);
  }
  kernel<<<unsigned(grid), kThreadsOf<K, BLOCKS>, s.smem, stream>>>(p);
  return cudaGetLastError();
}

// Layers that depthwise_ring_ok takes for two blocks per SM.
template <typename T>
bool two_blocks(const DirectParams& d) {
  return sizeof(T) == 2 && d.R == 3 && d.stride_w == 1 && d.W * int(sizeof(T)) % 16 == 0;
}

template <typename T, int K, int ST>
cudaError_t launch_ring_vb(const DirectParams& d, uint32_t* status, long long limit, cudaStream_t stream) {
  constexpr int kEs = int(sizeof(T));
  if constexpr (kEs == 2 && K == 3 && ST == 1) {
    if (two_blocks<T>(d)) return launch_ring_k<T, K, ST, 16, 2>(d, status, limit, stream);
  }
  if (d.W * kEs % 16 == 0) return launch_ring_k<T, K, ST, 16, 1>(d, status, limit, stream);
  if (d.W * kEs % 4 == 0) return launch_ring_k<T, K, ST, 4, 1>(d, status, limit, stream);
  return launch_ring_k<T, K, ST, kEs, 1>(d, status, limit, stream);
}

template <typename T>
cudaError_t launch_ring_t(const DirectParams& d, uint32_t* status, long long limit, cudaStream_t stream) {
  if (d.R == 3) return d.stride_w == 1 ? launch_ring_vb<T, 3, 1>(d, status, limit, stream) : launch_ring_vb<T, 3, 2>(d, status, limit, stream);
  return d.stride_w == 1 ? launch_ring_vb<T, 5, 1>(d, status, limit, stream) : launch_ring_vb<T, 5, 2>(d, status, limit, stream);
}

// Bytes of x from which this kernel is ahead of the other NCHW kernels, or none.  A ring starts later than a kernel that reads
// where it stands, and has nothing to overlap while a block has a group or two; what there is to gain depends on how wide the
// others can read (rows on 16, 8 or fewer bytes) and on the multiplications per input.  2200 layers of 7 to 112 columns and 1 to
// 136 MiB were timed on both: with these lines 26 take over 5 % longer than on the other (1.36 times at most); with one line at
// a megabyte 420 did (up to 1.9).  The others and this one, us, 3x3 bf16 unless said otherwise:
//   stride 1  rows off 8 bytes     6 x 512 x 14 x 14 5.4 and 5.0, 34 x 100 x 25 x 25 13.0 and 8.3, 168 x 512 x 14 x 14 62.4 and 34.9
//             rows on 8 bytes      3 x 256 x 28 x 28 3.8 and 5.0, 11 x 256 x 28 x 28 9.3 and 7.8
//             rows on 16 bytes     81 x 384 x 24 x 24 31.6 and 36.0, 162 x 384 x 24 x 24 71.7 and 60.8; 45 x 256 x 56 x 56 56.1 and
//                                  57.9, 89 x 256 x 56 x 56 105.9 and 103.9; 5x5 on 144 x 32 x 56 x 56 45.5 and 47.3
//             fp32                 3 x 512 x 14 x 14 3.6 and 4.5, 12 x 256 x 27 x 27 12.3 and 8.0; rows on 16 bytes 115 and 127
//   stride 2  16 bits              3 x 240 x 28 x 28 3.0 and 4.0, 45 x 240 x 28 x 28 12.7 and 11.0; 5x5 with rows on 16 bytes
//                                  32 x 512 x 16 x 16 7.8 and 10.0, 41 x 128 x 40 x 40 18.5 and 13.1
//             fp32                 7 x 96 x 57 x 57 6.6 and 9.6; 5x5 on 15 x 192 x 27 x 27 8.4 and 6.7
constexpr long long kNever = 1LL << 62, kMiB = 1 << 20;
long long ring_least_bytes(const DirectParams& p, int es) {
  const int row = p.W * es, area = p.H * p.W;
  if (p.stride_w == 1) {
    if (row % 16 == 0) return es == 4 || p.R == 5 ? kNever : area > 576 ? 96 * kMiB : row == 32 ? 24 * kMiB : 44 * kMiB;
    return es == 4 ? 19 * kMiB / 10 : row % 8 == 0 ? 3 * kMiB : kMiB;
  }
  if (p.W < 8) return kNever;
  if (row % 16 == 0) return p.R == 3 || row < 48 ? kNever : es == 2 && area <= 3136 ? 11 * kMiB / 2 : 7 * kMiB;
  if (es == 2) return row % 8 != 0 ? 3 * kMiB : p.R == 3 ? 15 * kMiB / 4 : 14 * kMiB / 5;
  if (p.R == 5) return area <= 2500 ? 11 * kMiB / 2 : kNever;
  return area > 2025 || (row % 8 == 0 && area > 400) ? 48 * kMiB : 13 * kMiB / 2;
}

}  // namespace

// Dense NCHW planes one after another, "same" padding of an unrolled filter, two groups of planes in shared memory, and a
// layer this is ahead on.
bool depthwise_ring_ok(int dtype, const DirectParams& p) {
  const int es = dtype == FDNN_F32 ? 4 : 2;
  if (p.dil_h != 1 || p.dil_w != 1 || p.stride_h != p.stride_w || p.R != p.S || (p.R != 3 && p.R != 5) ||
      (p.stride_w != 1 && p.stride_w != 2) || p.pad_left != p.R / 2 || p.pad_top != p.R / 2 || p.residual != nullptr || p.act > 1)
    return false;
  if (((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.y)) & 15u) != 0) return false;
  auto dense = [](const long long* s, int n, int c, int h, int w) {
    return (w <= 1 || s[3] == 1) && (h <= 1 || s[2] == w) && (c <= 1 || s[1] == (long long)h * w) && (n <= 1 || s[0] == (long long)c * h * w);
  };
  if (!dense(p.x_s, p.N, p.C, p.H, p.W) || !dense(p.y_s, p.N, p.C, p.OH, p.OW)) return false;
  // every strip's own columns begin inside the row: what lies past its end is padding
  if (p.OW > (p.W + p.stride_w - 1) / p.stride_w || p.OH > (p.H + p.stride_h - 1) / p.stride_h) return false;
  if ((long long)p.H * p.W > (1 << 20)) return false;
  const long long planes = (long long)p.N * p.C, unit = group_unit(p, es);
  if (planes * p.H * p.W * es < ring_least_bytes(p, es)) return false;
  // Planes that start off 16 bytes come in groups of up to eight, of which an SM holds two or three where planes are large:
  // too few groups leave SMs idle, and a second round that is nearly empty costs as much as the first.
  const long long groups = (planes + unit - 1) / unit, sms = current_sm_count(), rounds = (groups + sms - 1) / sms;
  if (p.stride_w == 2 || (es == 4 && p.R == 3)) {
    if (100 * groups < 57 * rounds * sms) return false;
  } else if (10 * groups < (es == 4 ? 5 : 3) * sms) {
    return false;
  }
  const int per_sm = es == 2 && p.R == 3 && p.stride_w == 1 && p.W * es % 16 == 0 ? 2 : 1;
  const int slots = p.stride_w == 2 && p.R == 3 ? 3 : 2;   // (186 x 64 x 75 x 75, two slots: 1.37 times as long)
  return slots * slot_bytes(p, es, unit, false) + slot_bytes(p, es, unit, true) + kFixedBytes <= smem_of(per_sm);
}

cudaError_t launch_depthwise_ring(int dtype, const DirectParams& d, uint32_t* status, long long wait_limit, cudaStream_t stream) {
  switch (dtype) {
    case FDNN_F16: return launch_ring_t<__half>(d, status, wait_limit, stream);
    case FDNN_BF16: return launch_ring_t<__nv_bfloat16>(d, status, wait_limit, stream);
    case FDNN_F32: return launch_ring_t<float>(d, status, wait_limit, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fdnn
