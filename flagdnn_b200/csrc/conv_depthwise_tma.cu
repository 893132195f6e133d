// Depthwise convolution on channels-last tensors: input rows staged by the TMA unit, output rows built up in registers.
//
// A depthwise layer moves two bytes in and two out per 2 * R * S flops: its floor is memory traffic.  The kernel that
// reads its window with per-thread loads (conv_depthwise.cu) is bound by instruction issue instead: bounds checks and
// 64-bit addresses for every pixel, and every pixel widened to fp32 once per output row that uses it (3x for 3x3),
// 27 instructions per output on 3x3.  Here
//   * a warp owns 64 channels (two per lane: one 128-byte row of shared memory per pixel, read without bank conflicts)
//     of PW neighbouring output columns, and walks down a band of output rows;
//   * a few input rows of the strip are one tiled tensor copy ((PW - 1) * stride + S pixels x 64 channels each); pixels and
//     channels outside the tensor arrive as zeros, which is the padding, so the arithmetic has no branches.  Each warp
//     has a ring of copies of its own, filled by its lane 0 (no block-wide synchronisation), and the ring runs on
//     across units, so that copies stay in flight while a unit ends and the next begins;
//   * an input row is widened once and added to every output row it belongs to: ceil(R / stride) rows of accumulators
//     live in registers, in rotation (the loop is unrolled by their number), with the taps beside them; arithmetic on
//     pairs of channels (fma.rn.f32x2), in the order of the taps, as the other depthwise kernels have it.
// Measured against that kernel, bf16 / fp32, us: 256 x 64 x 56 x 56 3x3 74.7 -> 64.1 / 100.8 -> 81.0; 64 x 512 x 28 x 28
// 44.6 -> 34.6 / 61.7 -> 43.2; 128 x 1024 x 7 x 7 23.8 -> 12.4 / 27.8 -> 12.1; 3 x 952 x 18 x 18 stride 2 12.2 -> 3.6 /
// 11.4 -> 3.5; 64 x 144 x 56 x 56 5x5 104 -> 89 / 120 -> 105.  What bounds it now is instruction issue again (half of the
// slots at 16 warps per SM, the most its registers allow), then the copies.
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

constexpr int kDtWarps = 4;        // warps per block
constexpr int kDtChunk = 64;       // channels per warp

struct DwTmaParams {
  int N, C, H, W, OH, OW;
  int pad_top, pad_left;
  long long w_s0, w_s2, w_s3;      // filter strides: channel, row, column
  long long y_sn, y_sh, y_sw;
  const void* w;
  const void* bias;
  const void* scale;
  const void* residual;            // y's strides, or nullptr
  void* y;
  int act;
  int owg, bands, band_rows;       // column groups per row, bands per image, output rows per band
  unsigned units;                  // N * bands * owg
  uint32_t* status;
  long long wait_limit;
};

template <typename T, int KR, int KS, int ST, int PW>
struct DwTmaCfg {
  static constexpr int kSpan = (PW - 1) * ST + KS;                        // input columns of a strip
  static constexpr int kPixBytes = kDtChunk * int(sizeof(T));
  static constexpr int kRowBytes = kSpan * kPixBytes;
  static constexpr int kLive = (KR + ST - 1) / ST;                        // output rows an input row belongs to
  static constexpr int kPeriod = kLive * ST;                              // rows after which the accumulators' roles repeat
  // Rows per copy, a divisor of the period: a copy of one 16-bit row (8 to 17 pixels of 128 bytes) takes the TMA unit
  // about 170 clocks however short it is, and that bounded the kernel.
  static constexpr int kRows = sizeof(T) == 4 ? 1 : (ST == 2 ? 2 : kPeriod);
  static constexpr int kCopyBytes = kRows * kRowBytes;
  static constexpr int kSlot = (kCopyBytes + 127) / 128 * 128;
  // copies in flight per warp: two to eight, within a quarter of an SM's shared memory (fp32: half of that measured best)
  static constexpr int kFit = (sizeof(T) == 4 ? 32 : 54) * 1024 / (kDtWarps * kSlot);
  static constexpr int kRing = kFit < 2 ? 2 : (kFit > 8 ? 8 : kFit);
  static constexpr int kSmem = kDtWarps * kRing * kSlot + kDtWarps * kRing * 8 + 16 + 128;
};

// Where the copies are: unit and row of the strip, advanced one row at a time.
struct DwCursor {
  unsigned unit;
  int row, rows;                   // next input row of the unit (copies bring kRows of them), input rows it has
  int n, oh0, ow0;                 // image, first output row, first output column
};

template <int KR, int ST, int PW>
__device__ __forceinline__ void cursor_open(DwCursor& c, const DwTmaParams& p) {
  const unsigned colg = c.unit % unsigned(p.owg), rest = c.unit / unsigned(p.owg);
  const unsigned band = rest % unsigned(p.bands);
  c.n = int(rest / unsigned(p.bands));
  c.oh0 = int(band) * p.band_rows;
  c.ow0 = int(colg) * PW;
  const int out_rows = min(p.band_rows, p.OH - c.oh0);
  c.rows = (out_rows - 1) * ST + KR;
  c.row = 0;
}

// PLAIN: no residual and no activation beyond ReLU.  The other epilogues' code (an erf and a tanh per output of the
// unrolled loop) would evict the loop from the instruction cache.
template <typename T, int KR, int KS, int ST, int PW, bool PLAIN>
__global__ void __launch_bounds__(kDtWarps * 32, 4)
depthwise_tma_kernel(const __grid_constant__ CUtensorMap tmX, const DwTmaParams p) {
  using Cfg = DwTmaCfg<T, KR, KS, ST, PW>;
  constexpr int kLive = Cfg::kLive, kRing = Cfg::kRing, kPeriod = Cfg::kPeriod;
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // carved by offsets from an aligned 32-bit shared address
  const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base_ptr + kDtWarps * kRing * Cfg::kSlot) + warp * kRing;
  volatile uint32_t* abort_flag = reinterpret_cast<uint32_t*>(base_ptr + kDtWarps * kRing * (Cfg::kSlot + 8));
  const uint32_t ring = base + warp * kRing * Cfg::kSlot;
  uint8_t* ring_ptr = base_ptr + warp * kRing * Cfg::kSlot;

  if (threadIdx.x == 0) *abort_flag = 0;
  if (lane == 0) {
    for (int i = 0; i < kRing; ++i) mbar_init(&bars[i], 1);
    fence_barrier_init();
  }
  __syncthreads();

  const int c0 = blockIdx.y * kDtChunk;
  const int ch = c0 + 2 * lane;
  const bool ch_ok = ch < p.C;             // C is even: both channels of a lane exist, or neither
  const unsigned stride_units = gridDim.x * kDtWarps;
  DwCursor ahead;                          // the next row to ask for
  ahead.unit = blockIdx.x * kDtWarps + warp;
  if (ahead.unit >= p.units) return;       // no warp waits for another from here on
  cursor_open<KR, ST, PW>(ahead, p);
  DwCursor cur = ahead;

  // taps, scale and bias of this lane's two channels
  F2 wt[KR * KS];
  F2 sc, bi;
  {
    const T* w = static_cast<const T*>(p.w) + (long long)ch * p.w_s0;
#pragma unroll
    for (int r = 0; r < KR; ++r)
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const T* t = w + r * p.w_s2 + s * p.w_s3;
        const float lo = ch_ok ? to_f32<T>(t[0]) : 0.0f, hi = ch_ok ? to_f32<T>(t[p.w_s0]) : 0.0f;
        wt[r * KS + s] = f2_make(__float_as_uint(lo), __float_as_uint(hi));
      }
    const T* gs = static_cast<const T*>(p.scale);
    const T* gb = static_cast<const T*>(p.bias);
    const bool s_ok = gs != nullptr && ch_ok, b_ok = gb != nullptr && ch_ok;
    sc = f2_make(__float_as_uint(s_ok ? to_f32<T>(gs[ch]) : 1.0f), __float_as_uint(s_ok ? to_f32<T>(gs[ch + 1]) : 1.0f));
    bi = f2_make(__float_as_uint(b_ok ? to_f32<T>(gb[ch]) : 0.0f), __float_as_uint(b_ok ? to_f32<T>(gb[ch + 1]) : 0.0f));
  }

  uint32_t put = 0, puts = 0, gets = 0;    // ring slot of the next copy; copies asked for; copies taken
  auto ask = [&]() {                       // one more copy into the ring, if any is left
    if (ahead.unit >= p.units) return;
    if (lane == 0) {
      mbar_arrive_expect_tx(&bars[put], uint32_t(Cfg::kCopyBytes));
      tma_load_4d(ring_ptr + put * Cfg::kSlot, &tmX, &bars[put], c0, ahead.ow0 * ST - p.pad_left,
                  ahead.oh0 * ST - p.pad_top + ahead.row, ahead.n);
    }
    ++puts;
    if (++put == uint32_t(kRing)) put = 0;
    ahead.row += Cfg::kRows;               // a unit's last copy may bring rows that nobody reads
    if (ahead.row >= ahead.rows) {
      ahead.unit += stride_units;
      if (ahead.unit < p.units) cursor_open<KR, ST, PW>(ahead, p);
    }
  };
  for (int i = 0; i < kRing; ++i) ask();

  uint32_t slot = 0, phase = 0;
  bool alive = true;
  const int act = p.act;
  while (cur.unit < p.units) {
    F2 acc[kLive][PW];
#pragma unroll
    for (int l = 0; l < kLive; ++l)
#pragma unroll
      for (int q = 0; q < PW; ++q) acc[l][q] = 0ull;
    T* y_unit = static_cast<T*>(p.y) + cur.n * p.y_sn + ch;
    const T* res_unit = static_cast<const T*>(p.residual) + cur.n * p.y_sn + ch;   // read only when there is one
    for (int t0 = 0; t0 < cur.rows && alive; t0 += kPeriod) {
#pragma unroll
      for (int u = 0; u < kPeriod; ++u) {
        if (t0 + u < cur.rows && alive) {  // uniform
          if (u % Cfg::kRows == 0) {
            if (!mbar_wait_bounded(&bars[slot], phase, abort_flag, p.status, kIncidentDepthwiseWait, p.wait_limit)) alive = false;
            alive = __all_sync(0xffffffffu, alive);
            ++gets;
          }
          if (alive) {
            const uint32_t src = ring + slot * Cfg::kSlot + (u % Cfg::kRows) * Cfg::kRowBytes + lane * 2 * int(sizeof(T));
#pragma unroll
            for (int j = 0; j < Cfg::kSpan; ++j) {
              F2 xv;
              if constexpr (sizeof(T) == 4) {
                const uint2 q2 = lds_v2(src + j * Cfg::kPixBytes);
                xv = f2_make(q2.x, q2.y);
              } else {
                float lo, hi;
                unpack2<T>(lds_u32(src + j * Cfg::kPixBytes), lo, hi);
                xv = f2_make(__float_as_uint(lo), __float_as_uint(hi));
              }
#pragma unroll
              for (int r = 0; r < KR; ++r) {
                if ((u - r + kPeriod * KR) % ST == 0) {          // row r of the window belongs to output row (t - r) / ST
                  const int l = ((u - r + kPeriod * KR) / ST) % kLive;
#pragma unroll
                  for (int q = 0; q < PW; ++q) {
                    const int s = j - q * ST;                     // constants once unrolled
                    if (s >= 0 && s < KS) acc[l][q] = f2_fma(xv, wt[r * KS + s], acc[l][q]);
                  }
                }
              }
            }
            if (u % Cfg::kRows == Cfg::kRows - 1 || t0 + u == cur.rows - 1) {
              __syncwarp();                // every lane has read the slot: it may be filled again
              if (++slot == uint32_t(kRing)) {
                slot = 0;
                phase ^= 1u;
              }
              ask();
            }
            if ((u - (KR - 1) + kPeriod * KR) % ST == 0) {        // the window's last row: an output row is complete
              const int l = ((u - (KR - 1) + kPeriod * KR) / ST) % kLive;
              const int o = (t0 + u - (KR - 1)) / ST;
              if (t0 + u >= KR - 1 && ch_ok) {
                T* yp = y_unit + (cur.oh0 + o) * p.y_sh + cur.ow0 * p.y_sw;
                const T* rp = PLAIN ? nullptr : res_unit + (cur.oh0 + o) * p.y_sh + cur.ow0 * p.y_sw;
                const int left = p.OW - cur.ow0;
#pragma unroll
                for (int q = 0; q < PW; ++q) {
                  if (q < left) {
                    float a, b;
                    f2_split(f2_fma(acc[l][q], sc, bi), a, b);
                    if constexpr (!PLAIN) {
                      if (p.residual != nullptr) {
                        a += to_f32<T>(rp[0]);
                        b += to_f32<T>(rp[1]);
                      }
                      if (act > 1) { a = apply_activation(a, act); b = apply_activation(b, act); }
                      rp += p.y_sw;
                    }
                    if constexpr (sizeof(T) == 4) {
                      if (act == 1) { a = relu_keep_nan(a); b = relu_keep_nan(b); }
                      __stcs(reinterpret_cast<float2*>(yp), make_float2(a, b));
                    } else {
                      __stcs(reinterpret_cast<uint32_t*>(yp), act == 1 ? round_pack2_relu<T>(a, b) : round_pack2<T>(a, b));
                    }
                  }
                  yp += p.y_sw;
                }
              }
#pragma unroll
              for (int q = 0; q < PW; ++q) acc[l][q] = 0ull;
            }
          }
        }
      }
    }
    if (!alive) break;
    cur.unit += stride_units;
    if (cur.unit < p.units) cursor_open<KR, ST, PW>(cur, p);
  }
  if (!alive && lane == 0) {
    // after an incident: the copies still in flight land before the block gives its shared memory back
    volatile uint32_t never = 0;
    for (uint32_t i = gets > 0 ? gets - 1 : 0; i < puts; ++i)
      mbar_wait_bounded(&bars[i % kRing], (i / kRing) & 1u, &never, p.status, kIncidentDrainWait, kWaitLimitCycles / 16);
  }
}

template <typename T, int KR, int KS, int ST, int PW, bool PLAIN>
cudaError_t launch_tma_one(const DirectParams& d, uint32_t* status, long long wait_limit,
                           cudaStream_t stream) {
  using Cfg = DwTmaCfg<T, KR, KS, ST, PW>;
  constexpr int dtype = std::is_same<T, float>::value ? FDNN_F32 : (std::is_same<T, __half>::value ? FDNN_F16 : FDNN_BF16);
  alignas(64) CUtensorMap tm;
  if (!encode_depthwise_map(&tm, dtype, d, kDtChunk, Cfg::kSpan, Cfg::kRows)) return cudaErrorInvalidValue;
  static std::atomic<int> ready[64];       // per device: shared-memory limit raised, resident blocks per SM
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  auto* kernel = depthwise_tma_kernel<T, KR, KS, ST, PW, PLAIN>;
  int per_sm = ready[dev & 63].load(std::memory_order_acquire);
  if (per_sm == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kDtWarps * 32, Cfg::kSmem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    ready[dev & 63].store(per_sm, std::memory_order_release);
  }
  DwTmaParams p = {};
  p.N = d.N; p.C = d.C; p.H = d.H; p.W = d.W; p.OH = d.OH; p.OW = d.OW;
  p.pad_top = d.pad_top; p.pad_left = d.pad_left;
  p.w_s0 = d.w_s[0]; p.w_s2 = d.w_s[2]; p.w_s3 = d.w_s[3];
  p.y_sn = d.y_s[0]; p.y_sh = d.y_s[2]; p.y_sw = d.y_s[3];
  p.w = d.w; p.bias = d.bias; p.scale = d.scale; p.residual = d.residual; p.y = d.y; p.act = d.act;
  p.status = status;
  p.wait_limit = wait_limit;
  const int chunks = (d.C + kDtChunk - 1) / kDtChunk;
  p.owg = (d.OW + PW - 1) / PW;
  // Band height: the one with the least work on the busiest warp (units per warp, rounded up, times the input rows of a
  // unit), taller bands first among equals, since a band re-reads R - stride rows of its neighbour.
  long long warps = (long long)current_sm_count() * per_sm * kDtWarps / chunks;
  if (warps < kDtWarps) warps = kDtWarps;
  long long best = -1;
  for (int bands = 1; bands <= d.OH; ++bands) {
    const int rows = (d.OH + bands - 1) / bands;
    if ((d.OH + rows - 1) / rows != bands) continue;
    const long long units = (long long)d.N * bands * p.owg;
    const long long cost = (units + warps - 1) / warps * ((rows - 1) * ST + KR + 1);
    if (best < 0 || cost < best) {
      best = cost;
      p.bands = bands;
      p.band_rows = rows;
    }
    if (units > 64 * warps) break;
  }
  p.units = unsigned((long long)d.N * p.bands * p.owg);
  long long gx = ((long long)p.units + kDtWarps - 1) / kDtWarps;
  if (gx > warps / kDtWarps) gx = warps / kDtWarps;
  kernel<<<dim3(unsigned(gx), unsigned(chunks)), kDtWarps * 32, Cfg::kSmem, stream>>>(tm, p);
  return cudaGetLastError();
}

template <typename T, bool PLAIN>
cudaError_t launch_tma_t(const DirectParams& d, uint32_t* status, long long limit, cudaStream_t stream) {
  if (d.R == 3 && d.stride_w == 1) return launch_tma_one<T, 3, 3, 1, 8, PLAIN>(d, status, limit, stream);
  if (d.R == 3) return launch_tma_one<T, 3, 3, 2, 8, PLAIN>(d, status, limit, stream);
  if (d.stride_w == 1) return launch_tma_one<T, 5, 5, 1, 4, PLAIN>(d, status, limit, stream);
  return launch_tma_one<T, 5, 5, 2, 4, PLAIN>(d, status, limit, stream);
}

template <typename T>
cudaError_t launch_tma_any(const DirectParams& d, uint32_t* status, long long limit, cudaStream_t stream) {
  if (d.residual == nullptr && d.act <= FDNN_ACT_RELU) return launch_tma_t<T, true>(d, status, limit, stream);
  return launch_tma_t<T, false>(d, status, limit, stream);
}

}  // namespace

bool depthwise_tma_ok(const DirectParams& d) {
  const bool unrolled = d.dil_h == 1 && d.dil_w == 1 && d.stride_h == d.stride_w && d.R == d.S && (d.R == 3 || d.R == 5) &&
                        (d.stride_w == 1 || d.stride_w == 2);
  // a chunk of 64 channels that is mostly padding wastes the lanes that hold it
  const int chunks = (d.C + kDtChunk - 1) / kDtChunk;
  return unrolled && d.C % 2 == 0 && 4 * d.C >= 3 * chunks * kDtChunk && chunks <= 65535;
}

cudaError_t launch_depthwise_tma(int dtype, const DirectParams& d, uint32_t* status, long long wait_limit,
                                 cudaStream_t stream) {
  switch (dtype) {
    case FDNN_F16: return launch_tma_any<__half>(d, status, wait_limit, stream);
    case FDNN_BF16: return launch_tma_any<__nv_bfloat16>(d, status, wait_limit, stream);
    case FDNN_F32: return launch_tma_any<float>(d, status, wait_limit, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fdnn
