// C-ABI front end: descriptor validation, planning (which kernel, which tile,
// how much scratch), tensor-map encoding and launches.  See
// include/flagdnn_b200.h for the contract of every exported function.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <atomic>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>

#include "conv_internal.h"

namespace fdnn {
namespace {

thread_local std::string g_last_error;

int fail(int status, const std::string& msg) {
  g_last_error = msg;
  return status;
}

int fail_cuda(const char* what, cudaError_t e) {
  // Clear the sticky-free error so later, unrelated calls do not see it.
  cudaGetLastError();
  return fail(FDNN_CUDA_ERROR, std::string(what) + ": " + cudaGetErrorString(e));
}

int elem_size(int dtype) {
  switch (dtype) {
    case FDNN_F16:
    case FDNN_BF16: return 2;
    case FDNN_F32: return 4;
    case FDNN_F64: return 8;
    default: return 0;
  }
}

int conv_out_dim(int in, int pad_before, int pad_after, int dil, int kernel, int stride) {
  // floor division on a possibly negative numerator, as Python's // does
  const long long num = (long long)in + pad_before + pad_after - (long long)dil * (kernel - 1) - 1;
  long long q = num / stride;
  if ((num % stride != 0) && ((num < 0) != (stride < 0))) --q;
  return int(q + 1);
}

// Same checks, in the same order, as _check_conv2d_inputs
// (src/flag_dnn/ops/conv2d.py:90-135); dtype/device equality of the tensors is
// the caller's business because this ABI carries a single dtype.
int validate(const fdnn_conv_desc* d) {
  if (d == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (elem_size(d->dtype) == 0) return fail(FDNN_NOT_SUPPORTED, "Unsupported dtype");
  if (d->groups <= 0) return fail(FDNN_BAD_PARAM, "groups must be a positive integer");
  if (d->stride_h <= 0 || d->stride_w <= 0) return fail(FDNN_BAD_PARAM, "stride must be positive");
  if (d->dil_h <= 0 || d->dil_w <= 0) return fail(FDNN_BAD_PARAM, "dilation must be positive");
  if (d->pad_top < 0 || d->pad_bottom < 0 || d->pad_left < 0 || d->pad_right < 0)
    return fail(FDNN_BAD_PARAM, "negative padding is not supported");
  if (d->n < 0 || d->c <= 0 || d->h < 0 || d->w < 0 || d->k <= 0 || d->r <= 0 || d->s <= 0)
    return fail(FDNN_BAD_PARAM, "tensor extents must be positive");
  if (d->c % d->groups != 0 || d->k % d->groups != 0)
    return fail(FDNN_BAD_PARAM, "channels must be divisible by groups");
  return FDNN_OK;
}

// SM count of the current device, looked up once per device ordinal (148 when no device is visible).
int sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return 148;
  }
  const int hit = cached[dev].load(std::memory_order_relaxed);
  if (hit > 0) return hit;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0) {
    cached[dev].store(sms, std::memory_order_relaxed);
    return sms;
  }
  cudaGetLastError();
  return 148;
}

bool aligned16(const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int round_up(int v, int m) { return (v + m - 1) / m * m; }

// Channels a relaid-out pixel or a packed filter tap is stored with.  The kernels copy 128 bytes of channels at a time;
// a pitch that leaves those pieces unaligned makes most of them straddle two cache lines, and the copies, which bound
// long reductions, slow down accordingly, so that channels fill whole 128-byte lines (or an even share of one):
// zeros are never computed with more often than before, since a block of 128 bytes was always multiplied whole.
int padded_channels(int dtype, int c) {
  const int es = elem_size(dtype);
  for (int bytes = 16; bytes < 128; bytes *= 2)
    if (c * es <= bytes) return bytes / es;
  return round_up(c, 128 / es);
}

// The same for the relaid-out activations, except where only rows of 16-byte multiples keep them within the built-in
// scratch of fdnn_conv2d_fwd_static_scratch: that call takes every problem whose tightest layout fits.
int padded_x_channels(const fdnn_conv_desc* d) {
  const int es = elem_size(d->dtype), wide = padded_channels(d->dtype, d->c), tight = round_up(d->c, 16 / es);
  const long long per_channel = (long long)(d->dtype == FDNN_F32 ? 2 : 1) * d->n * d->h * d->w * es;
  const bool fits = per_channel * tight <= FDNN_STATIC_SCRATCH_BYTES;
  return fits && per_channel * wide > FDNN_STATIC_SCRATCH_BYTES ? tight : wide;
}

// Can the tensor-core path express this geometry?  Limits are those of the
// im2col tensor map: box corners in [-128, 127], tap offsets <= 255,
// traversal strides <= 8.
bool igemm_geometry_ok(const fdnn_conv_desc* d) {
  if (d->dtype == FDNN_F64 || d->groups != 1) return false;
  if (d->stride_h > 8 || d->stride_w > 8) return false;
  if (d->pad_left > 128 || d->pad_top > 128) return false;
  const int up_w = d->pad_right - (d->s - 1) * d->dil_w;
  const int up_h = d->pad_bottom - (d->r - 1) * d->dil_h;
  if (up_w < -128 || up_w > 127 || up_h < -128 || up_h > 127) return false;
  if ((d->s - 1) * d->dil_w > 255 || (d->r - 1) * d->dil_h > 255) return false;
  return true;
}

// Tile width asked for through FDNN_ALGO_FLAG_TILE_N_* (0: none; fp32 tiles stop at 128 columns).
int forced_tile_n(const fdnn_conv_desc* d) {
  const int code = (d->algo & FDNN_ALGO_FLAG_TILE_N_MASK) >> 10;
  if (code == 0) return 0;
  const int bn = 32 << code;
  return (d->dtype == FDNN_F32 && bn > 128) ? 128 : bn;
}

int choose_tile_n(int dtype, int m_tiles, int kout, int sms) {
  const int max_bn = (dtype == FDNN_F32) ? 128 : 256;
  int best = 64;
  double best_cost = 1e300;
  for (int bn = 64; bn <= max_bn; bn *= 2) {
    if (bn > 64 && bn / 2 >= kout) break;  // a tile twice as wide as the problem is pure waste
    const long long tiles = (long long)m_tiles * ((kout + bn - 1) / bn);
    const long long waves = (tiles + sms - 1) / sms;
    // Measured on B200: a 128-wide tile costs about 0.8 of a 256-wide one (the
    // activation tile and the per-step overheads do not shrink with N).
    const double cost = double(waves) * (bn + 384);
    if (cost <= best_cost) {
      best_cost = cost;
      best = bn;
    }
  }
  return best;
}

// Stride between consecutive output pixels when y is one dense [M, K] matrix
// (channels contiguous, pixels / rows / images evenly spaced), else 0.
long long y_pixel_stride(const fdnn_conv_desc* d, int oh, int ow) {
  const int gran = 16 / elem_size(d->dtype);
  long long row = round_up(d->k, gran);
  if (ow > 1) row = d->y_strides[3];
  else if (oh > 1) row = d->y_strides[2];
  else if (d->n > 1) row = d->y_strides[0];
  const bool dense = (d->k == 1 || d->y_strides[1] == 1) && row >= d->k && row % gran == 0 &&
                     (ow <= 1 || oh <= 1 || d->y_strides[2] == (long long)ow * row) &&
                     ((long long)oh * ow <= 1 || d->n <= 1 || d->y_strides[0] == (long long)oh * ow * row);
  return dense ? row : 0;
}

bool y_is_dense_nhwc(const fdnn_conv_desc* d, int oh, int ow, const void* y) {
  return y_pixel_stride(d, oh, ow) > 0 && aligned16(y);
}

// The least scratch a relayout of x works with: rows of 16-byte multiples.  Callers that size their buffer so (it was the
// only layout once) get that one instead of the line-sized rows or the window mode the plan asks scratch for.
long long tight_x_bytes(const fdnn_conv_desc* d) {
  const int es = elem_size(d->dtype);
  return (long long)(d->dtype == FDNN_F32 ? 2 : 1) * d->n * d->h * d->w * round_up(d->c, 16 / es) * es;
}

// How the single-CTA kernel's epilogue writes a y that has no TMA map (see epilogue_store_strided): along channels
// when they are contiguous, with the widest unit that every pixel's start is a multiple of; along pixels when every image's
// pixels are (NCHW); otherwise element by element.
void choose_strided_store(const fdnn_conv_desc& d, int oh, int ow, const void* y, IgemmParams* p) {
  const int es = elem_size(d.dtype);
  const long long sn = d.y_strides[0], sk = d.y_strides[1], sh = d.y_strides[2], sw = d.y_strides[3];
  const uintptr_t base = reinterpret_cast<uintptr_t>(y);
  auto fits = [es](long long extent, long long stride, int unit) { return extent <= 1 || stride * es % unit == 0; };
  p->y_mode = 0;
  p->y_unit = es;
  if (d.k > 1 && sk == 1) {
    p->y_mode = 2;
    for (int unit = 16; unit > es; unit /= 2) {
      if (base % unit == 0 && fits(d.n, sn, unit) && fits(oh, sh, unit) && fits(ow, sw, unit)) {
        p->y_unit = unit;
        break;
      }
    }
    return;
  }
  const bool pixels = ow > 1 ? (sw == 1 && (oh == 1 || sh == ow)) : (oh == 1 || sh == 1);
  if (pixels) p->y_mode = 1;
}

// Low-channel mode (C <= 4, e.g. the 7x7 stride-2 stem): four neighbouring
// output pixels of a row form one GEMM row with 4*K columns; its operand is a
// 16-pixel window (64 elements = 128 bytes) of the input repacked to 4 channels,
// so a filter row costs one fat TMA row instead of S thin ones.
struct LowChannel {
  bool ok;
  int ow4, ohs, rows_per_tile, tiles_per_image, w_pad;
  int lpad;  // zero pixels stored left of each row: the conv's left padding rounded up to even (16-byte pixels pairs)
  // Fused variant for a dense 3-channel NHWC input and an even W-stride (the 7x7 stride-2 stem), CTA pairs
  // only: no relayout pass and no fourth channel.  A quad's window starts every 4 * stride_w * 3 elements,
  // which is a multiple of 16 bytes; per tile two warps copy the input rows it needs, shifted by
  // `lead_chunks` zero pieces and zero-padded, into a small per-CTA scratch slot that the window copies
  // read.  48 elements of a window hold data (three MMAs per filter row instead of four).
  bool fused3;
  int raw_rows;      // input rows per tile
  int row_chunks;    // 16-byte pieces per scratch row
  int lead_chunks;   // zero pieces before the row's own first piece
  int shift_elems;   // window element at which the quad's first pixel's first tap sits
  long long slot_bytes;
};

bool dense_nhwc3(const fdnn_conv_desc* d) {
  return d->c == 3 && d->x_strides[1] == 1 && (d->w <= 1 || d->x_strides[3] == 3) &&
         (d->h <= 1 || d->x_strides[2] == 3LL * d->w) && (d->n <= 1 || d->x_strides[0] == 3LL * d->w * d->h);
}

LowChannel low_channel_geometry(const fdnn_conv_desc* d, int oh, int ow, const void* y, bool pair_kernel = false) {
  LowChannel g = {};
  const bool is16 = elem_size(d->dtype) == 2;
  if (!is16 || d->groups != 1 || d->c > 4 || d->dil_w != 1 || ow < 4 || ow % 4 != 0 || ow / 4 > 128) return g;
  g.lpad = round_up(d->pad_left, 2);
  if (d->stride_w > 8 || d->stride_h > 8 || 3 * d->stride_w + (d->s - 1) + (g.lpad - d->pad_left) > 15 || d->k % 2 != 0) return g;
  if (oh <= 0 || d->pad_top > 255 || d->pad_left > 255) return g;
  if (y_pixel_stride(d, oh, ow) != d->k || !aligned16(y)) return g;  // a quad's 4*K outputs must be contiguous
  g.ow4 = ow / 4;
  g.ohs = 128 / g.ow4;
  if (g.ohs > oh) g.ohs = oh;
  if (g.ohs * d->stride_h > 256) g.ohs = 256 / d->stride_h;
  g.rows_per_tile = g.ohs * g.ow4;
  g.tiles_per_image = (oh + g.ohs - 1) / g.ohs;
  const int need = d->stride_w * 4 * (g.ow4 - 1) + 16;
  g.w_pad = round_up(need > g.lpad + d->w ? need : g.lpad + d->w, 2);
  g.ok = true;
  if (pair_kernel && dense_nhwc3(d) && d->stride_w % 2 == 0 && (3 * d->w) % 8 == 0 && d->r <= igemm_pair_max_resident_steps() &&
      4 * d->k <= 256) {
    const int lead_elems = round_up(3 * d->pad_left, 8);              // zeros before the row, whole 16-byte pieces
    g.shift_elems = lead_elems - 3 * d->pad_left;
    g.lead_chunks = lead_elems / 8;
    g.raw_rows = (g.ohs - 1) * d->stride_h + (d->r - 1) * d->dil_h + 1;
    const int span = g.shift_elems + 3 * (3 * d->stride_w + d->s);    // window elements that hold data
    const int row_elems = round_up(12 * d->stride_w * (g.ow4 - 1) + 64, 8);
    g.row_chunks = row_elems / 8;
    g.slot_bytes = round_up(g.raw_rows * row_elems * 2, 256);
    g.fused3 = span <= 48 && g.raw_rows <= 64 && g.slot_bytes <= 64 * 1024;
  }
  return g;
}

// Window mode for other layers of fewer than 8 channels (a stem on NCHW tensors, or with an output width that is no
// multiple of four): one GEMM row is one output pixel, its operand for a filter row the S x 8 stored values its taps
// read, 16 * S contiguous bytes of the input relaid out as [N][H][w_pad][8] with the padding stored.  Windows of
// neighbouring pixels overlap (a tiled map whose window stride is smaller than its length), the packed filter
// [K, R, S, 8] is read as [K, R, S * 8], and a reduction takes R steps instead of R * S copies of 16-byte rows, each of
// which costs the TMA unit as much as a 128-byte one (12 x 170 x 170 x 3 -> 32, 7x7 stride 2, NCHW bf16: 155 us).
// Elements past S * 8 are out of the map's bounds and arrive as zeros.
struct PixelWindows {
  bool ok;
  int ohs, rows_per_tile, tiles_per_image, w_pad;
  long long scratch;
};
PixelWindows pixel_windows(const fdnn_conv_desc* d, int oh, int ow) {
  PixelWindows g = {};
  if (elem_size(d->dtype) != 2 || d->groups != 1 || d->c >= 8 || d->dil_w != 1 || d->s < 3 || d->s > 8) return g;
  if (oh < 1 || ow < 1 || ow > 128 || d->stride_h > 8 || d->pad_top > 127 || (d->algo & FDNN_ALGO_FLAG_OUT_F32) != 0) return g;
  g.ohs = 128 / ow;
  if (g.ohs > oh) g.ohs = oh;
  if (g.ohs * d->stride_h > 256) g.ohs = 256 / d->stride_h;
  g.rows_per_tile = g.ohs * ow;
  g.tiles_per_image = (oh + g.ohs - 1) / g.ohs;
  if ((long long)d->n * g.tiles_per_image * 128 > 2000000000LL || (long long)d->n * d->h > 2000000000LL) return g;
  const int need = d->stride_w * (ow - 1) + 8;
  g.w_pad = need > d->pad_left + d->w ? need : d->pad_left + d->w;
  g.scratch = (long long)d->n * d->h * g.w_pad * 16;
  // half-empty tiles (few pixels per image, or rows just over 64 pixels) still take R steps instead of R * S; a call
  // that fits the built-in scratch the other way keeps fitting it
  const long long tight = (long long)d->n * d->h * d->w * 16;
  g.ok = g.rows_per_tile * d->s >= 128 * 2 && !(g.scratch > FDNN_STATIC_SCRATCH_BYTES && tight <= FDNN_STATIC_SCRATCH_BYTES);
  return g;
}

// Output-pixel grouping for narrow layers.  A reduction step of a narrow tile brings
// almost as many operand bytes as one of a wide tile (24 / 32 / 48 KB for 64 / 128 / 256
// columns), and an MMA of 64 columns runs at two thirds of the full rate, so a layer with
// K <= 128 output channels uses a fraction of the machine.  Grouping Q neighbouring
// output pixels of a row into one GEMM row turns the layer into an equivalent
// convolution with Q*K output channels, a filter widened to S + (Q-1)*stride_w
// taps (zero where a pixel does not reach) and a W-stride of Q*stride_w.  Its y,
// [N, OH, OW/Q, Q*K] in NHWC, is the same memory as the real [N, OH, OW, K].
// The wider filter costs (S + (Q-1)*stride_w) / S more MMA steps per row, the
// Q-fold wider tile makes each step Q times as productive.
int choose_pixel_group(const fdnn_conv_desc* d, int oh, int ow, const void* y) {
  if (elem_size(d->dtype) != 2 || d->groups != 1 || d->dil_w != 1 || d->c < 8) return 1;
  if (d->r * d->s < 4) return 1;                       // 1x1 / thin filters are bandwidth-bound anyway
  if (y_pixel_stride(d, oh, ow) != d->k || !aligned16(y)) return 1;
  if (2.0 * d->n * oh * ow * d->k * d->c * d->r * d->s < 4.0e9) return 1;  // only layers that fill the machine
  int best = 1;
  double best_cost = double(d->s);
  for (int q = 2; q <= 4; q *= 2) {
    if (q * d->k > 256 || ow % q != 0 || q * d->stride_w > 8) break;
    const int s_virtual = d->s + (q - 1) * d->stride_w;
    if (s_virtual - 1 > 255 || d->pad_right + (q - 1) * d->stride_w - (s_virtual - 1) < -128) break;
    const double cost = double(s_virtual) / q;        // MMA steps per output pixel, relative
    if (cost < 0.85 * best_cost) {
      best = q;
      best_cost = cost;
    }
  }
  return best;
}

// The equivalent convolution of a pixel-grouped layer (filter strides describe the packed [Q*K][R][S'][Cpad]).
fdnn_conv_desc grouped_desc(const fdnn_conv_desc* d, int q, int oh, int ow) {
  fdnn_conv_desc v = *d;
  const int c_pad = padded_channels(d->dtype, d->c);
  v.k = q * d->k;
  v.s = d->s + (q - 1) * d->stride_w;
  v.stride_w = q * d->stride_w;
  v.pad_right = d->pad_right + (q - 1) * d->stride_w;
  v.w_strides[0] = (int64_t)d->r * v.s * c_pad;
  v.w_strides[1] = 1;
  v.w_strides[2] = (int64_t)v.s * c_pad;
  v.w_strides[3] = c_pad;
  v.y_strides[0] = (int64_t)oh * ow * d->k;
  v.y_strides[1] = 1;
  v.y_strides[2] = (int64_t)ow * d->k;
  v.y_strides[3] = (int64_t)q * d->k;
  return v;
}

// A one-tap filter whose K dimension is contiguous (mm's second operand, [C][K] row-major with rows of 16-byte
// multiples) is read in place: the tensor core takes an MN-major operand as well.  It saves the transposing copy of every
// call, the filter moved twice.  Calls with the copy and without, bf16: 8192 x 4096 @ 4096 x 4096 190.1 and 177.5 us,
// 1024 x 4096 @ 4096 x 4096 42.1 and 29.8, 2048 cubed 23.8 and 18.8, 8192 x 512 @ 512 x 512 8.45 and 8.35.  (While the
// thread that issues the MMAs was the bottleneck, large products ran 10 to 20 % slower on such an operand.)
bool filter_mn_major(const fdnn_conv_desc* d, const void* w) {
  return elem_size(d->dtype) == 2 && d->r * d->s == 1 && d->k > 1 && d->c > 1 && d->w_strides[0] == 1 &&
         d->w_strides[1] % 8 == 0 && d->w_strides[1] >= d->k && aligned16(w) && (d->algo & 0xff) != FDNN_ALGO_IGEMM_PAIR;
}

// Below kSmallFlops a 16-bit layer still runs on the tensor-core kernel when its reduction is more than a few dozen
// products long: the direct kernel walks it serially (kernels of one 64 x 14 x 14 image, 64 filters 3x3, bf16: NCHW
// 25.9 -> 8.2 us, channels-last 83.2 -> 4.9), and both round an fp32 sum once.  fp32 layers stay on exact products there.
// Such a call needs what the tensor-core plan asks for (packed filter, scratch); without it, fwd_impl runs the direct
// kernel as before, and the scratch stays within the built-in one of fdnn_conv2d_fwd_static_scratch.
// Fewer than eight channels only in window mode (see pixel_windows): without it a reduction takes R * S copies of 16-byte
// rows (3 -> 16 channels 11x11 on 32 x 32 NCHW: 35 us against the direct kernel's 20).
constexpr double kSmallFlops = 2.0e7;
bool small_on_tensor_cores(const fdnn_conv_desc* d, int oh, int ow, double flops) {
  return elem_size(d->dtype) == 2 && d->c * d->r * d->s >= 64 && flops >= 2.0e5 &&
         (d->c >= 8 || pixel_windows(d, oh, ow).ok) &&
         (long long)d->n * d->h * d->w * padded_x_channels(d) * 2 <= FDNN_STATIC_SCRATCH_BYTES;
}

// Reduction splitting on CTA pairs: T tiles of K reduction steps on P pairs.  Whole tiles cost
// ceil(T / P) * K steps on the busiest pair, an even split ceil(T * K / P) plus the exchange of one partial
// tile (about three steps' worth of time).  Ranges shorter than 12 steps are not split (boundaries snap to
// tile edges within kStreamKMinFrag steps, and every pair must keep a non-empty range).
constexpr int kStreamKMinFrag = 4;
struct StreamK {
  bool worth;
};
StreamK plan_stream_k(long long tiles, long long k_steps, int pairs, bool filter_resident) {
  StreamK r = {false};
  if (tiles <= 0 || pairs <= 0 || filter_resident) return r;
  const long long total = tiles * k_steps;
  const long long whole = (tiles + pairs - 1) / pairs * k_steps;
  const long long even = (total + pairs - 1) / pairs;
  if (even < 12) return r;
  r.worth = double(even + 3) <= 0.95 * double(whole);
  return r;
}

// Grouped layers that are not depthwise run as one tensor-core launch per group on strided views of x, w and y
// (group g reads channels g*C/G.. of x, filters g*K/G.. of w and writes channels g*K/G.. of y), when the per-group
// channel counts keep every group's pointers 16-byte aligned like the first group's, so that all groups get the
// same plan.  The reference times such layers beside the dense ones (benchmark/test_conv2d_perf.py:48-49).
bool group_loop_ok(const fdnn_conv_desc* d) {
  if (d->groups <= 1 || d->groups > 64 || d->dtype == FDNN_F64) return false;
  if ((d->algo & 0xff) == FDNN_ALGO_DIRECT || (d->algo & FDNN_ALGO_FLAG_OUT_F32) != 0) return false;
  const int es = elem_size(d->dtype);
  const int cg = d->c / d->groups, kg = d->k / d->groups;
  return cg >= 8 && (cg * es) % 16 == 0 && (kg * es) % 16 == 0;
}

// With few groups the layer runs faster as ONE dense convolution whose filter is block-diagonal (zeros outside each
// filter's own channels): G times the MMAs, but full 256-column tiles, pixel grouping and CTA pairs instead of G
// launches on narrow per-group tiles (measured on 64 -> 128 3x3 in two groups at 56 x 56, 256 images: 329 us for
// the per-group launches).  The dense filter lives at the front of the packed-filter buffer.
bool group_dense_ok(const fdnn_conv_desc* d) {
  if (d->groups < 2 || d->groups > 8 || d->dtype == FDNN_F64) return false;
  if ((d->algo & 0xff) == FDNN_ALGO_DIRECT || (d->algo & FDNN_ALGO_FLAG_OUT_F32) != 0) return false;
  return d->c / d->groups >= 2 && (long long)d->k * d->c * d->r * d->s <= (1LL << 28);
}

long long dense_filter_bytes(const fdnn_conv_desc* d) {
  const long long b = (long long)d->k * d->r * d->s * d->c * elem_size(d->dtype);
  return (b + 255) / 256 * 256;
}

fdnn_conv_desc dense_group_desc(const fdnn_conv_desc* d) {
  fdnn_conv_desc v = *d;
  v.groups = 1;
  v.w_strides[0] = (int64_t)d->r * d->s * d->c;
  v.w_strides[1] = 1;
  v.w_strides[2] = (int64_t)d->s * d->c;
  v.w_strides[3] = d->c;
  return v;
}

// The taps of a five-dimensional im2col map: corners within [-16, 15], offsets up to 31.
bool batch_geometry_ok(const fdnn_conv_desc* d) {
  const int up_w = d->pad_right - (d->s - 1) * d->dil_w, up_h = d->pad_bottom - (d->r - 1) * d->dil_h;
  return d->pad_left <= 16 && d->pad_top <= 16 && up_w >= -16 && up_w <= 15 && up_h >= -16 && up_h <= 15 &&
         (d->s - 1) * d->dil_w <= 31 && (d->r - 1) * d->dil_h <= 31;
}

// Unless a tensor-core kernel was asked for, a grouped layer takes one of those routes only if the dense layer it turns
// into is not a small one, or if all its groups together are not (they then run in one launch, see group_batch).
bool worth_grouping(const fdnn_conv_desc* d, const fdnn_conv_plan& inner, double flops) {
  if ((d->algo & 0xff) != FDNN_ALGO_AUTO || inner.flops >= kSmallFlops) return true;
  if (elem_size(d->dtype) != 2 || d->algo != FDNN_ALGO_AUTO || d->groups <= 8 || flops < kSmallFlops || !batch_geometry_ok(d))
    return false;
  const long long per_group = (long long)d->n * d->h * d->w * (d->c / d->groups) * 2;
  return inner.workspace_bytes == 0 || per_group * 8 <= FDNN_STATIC_SCRATCH_BYTES;   // eight groups and more at a time
}

// Whether a layer of this many operations ran on the direct kernel before small ones had another choice: it still does
// for callers that bring neither packed filter nor scratch.
bool small_layer(const fdnn_conv_desc* d, double flops) {
  if (d->groups > 1 && group_dense_ok(d) && flops * d->groups >= kSmallFlops) return false;
  return flops / d->groups < kSmallFlops;
}

fdnn_conv_desc one_group_desc(const fdnn_conv_desc* d) {
  fdnn_conv_desc sub = *d;
  sub.c = d->c / d->groups;
  sub.k = d->k / d->groups;
  sub.groups = 1;
  return sub;
}

struct GroupBatch {    // see group_batch below
  int tile_n;          // 0: does not apply
  fdnn_conv_plan one;
};
GroupBatch group_batch(const fdnn_conv_desc* d, const void* x, const void* w, const void* y, const fdnn_conv_plan& plan,
                       bool dense);

// w in place: [K, R, S, C]-like memory, taps evenly spaced.  A stride over an extent of one carries no information.
bool filter_in_place(const fdnn_conv_desc* d, const void* w) {
  const int es = elem_size(d->dtype), gran = 16 / es, cg = d->c / d->groups;
  auto stride_ok = [gran](long long extent, long long stride) { return extent <= 1 || stride % gran == 0; };
  return es == 2 && (cg == 1 || d->w_strides[1] == 1) && stride_ok(d->k, d->w_strides[0]) &&
         stride_ok(d->s, d->w_strides[3]) && (d->s <= 1 || d->w_strides[3] >= cg) &&
         (d->r <= 1 || (d->s > 1 ? d->w_strides[2] == (long long)d->s * d->w_strides[3]
                                 : d->w_strides[2] % gran == 0)) &&
         aligned16(w);
}

int make_plan(const fdnn_conv_desc* d, const void* x, const void* w, const void* y,
              fdnn_conv_plan* plan, bool allow_group = true) {
  int st = validate(d);
  if (st != FDNN_OK) return st;
  if (plan == nullptr) return fail(FDNN_BAD_PARAM, "plan is NULL");
  std::memset(plan, 0, sizeof(*plan));
  const int es = elem_size(d->dtype);
  const int oh = conv_out_dim(d->h, d->pad_top, d->pad_bottom, d->dil_h, d->r, d->stride_h);
  const int ow = conv_out_dim(d->w, d->pad_left, d->pad_right, d->dil_w, d->s, d->stride_w);
  if (oh < 0 || ow < 0) return fail(FDNN_BAD_PARAM, "computed output size is negative");
  plan->oh = oh;
  plan->ow = ow;
  const double m = double(d->n) * oh * ow;
  const int cg = d->c / d->groups;
  plan->flops = 2.0 * m * d->k * cg * d->r * d->s;
  plan->bytes = es * (double(d->n) * d->c * d->h * d->w + double(d->k) * cg * d->r * d->s + d->k + m * d->k);

  if (group_dense_ok(d)) {
    const fdnn_conv_desc v = dense_group_desc(d);
    fdnn_conv_plan pv;
    // the dense filter will sit 256-byte aligned at the front of the packed buffer: plan it as readable in place
    if (make_plan(&v, x, nullptr, y, &pv, allow_group) == FDNN_OK && pv.algo != FDNN_ALGO_DIRECT && worth_grouping(d, pv, plan->flops)) {
      const double flops = plan->flops, bytes = plan->bytes;
      *plan = pv;
      plan->flops = flops;   // the layer's own work, not the block-diagonal GEMM's
      plan->bytes = bytes;
      plan->w_packed = 1;
      plan->packed_weight_bytes = dense_filter_bytes(d) + pv.packed_weight_bytes;
      if (allow_group && w != nullptr) {
        // The forward call will run all groups in one launch on w itself: no filter to pack, which for this route is G
        // times the size of w.  (With a NULL w the caller's filter is not known, and a packed one serves any.)
        const GroupBatch own = group_batch(d, x, w, y, *plan, true);
        const long long per_group = (long long)d->n * d->h * d->w * cg * es;
        if (own.tile_n != 0 && !own.one.w_packed && (!own.one.x_repacked || plan->workspace_bytes >= 2 * per_group)) {
          plan->w_packed = 0;
          plan->packed_weight_bytes = 0;
        }
      }
      return FDNN_OK;
    }
  }
  if (group_loop_ok(d)) {
    const fdnn_conv_desc sub = one_group_desc(d);
    fdnn_conv_plan ps;
    if (make_plan(&sub, x, w, y, &ps, allow_group) == FDNN_OK && ps.algo != FDNN_ALGO_DIRECT && worth_grouping(d, ps, plan->flops)) {
      const double flops = plan->flops, bytes = plan->bytes;
      *plan = ps;              // every group runs this plan; scratch is shared, the packed filters are not
      plan->flops = flops;
      plan->bytes = bytes;
      plan->launches = ps.launches * d->groups;
      plan->packed_weight_bytes = ps.packed_weight_bytes * d->groups;
      // room to relay several groups out at a time, within what the built-in scratch holds (see group_batch)
      const long long per_group = (long long)d->n * d->h * d->w * sub.c * es;
      if (ps.workspace_bytes > 0 && es == 2 && ps.workspace_bytes < FDNN_STATIC_SCRATCH_BYTES && per_group > 0) {
        long long some = FDNN_STATIC_SCRATCH_BYTES / per_group;
        if (some > d->groups) some = d->groups;
        if (some * per_group > plan->workspace_bytes) plan->workspace_bytes = some * per_group;
      }
      return FDNN_OK;
    }
  }

  const bool geom_ok = igemm_geometry_ok(d) && m > 0 && m < 2.0e9;
  int algo = d->algo & 0xff;
  const bool split_allowed = (d->algo & FDNN_ALGO_FLAG_STREAM_K) != 0;
  const bool out_f32 = (d->algo & FDNN_ALGO_FLAG_OUT_F32) != 0;
  if (out_f32) {
    if (es != 2) return fail(FDNN_BAD_PARAM, "a float32 output is an option of f16 / bf16 operands");
    if (algo == FDNN_ALGO_DIRECT || algo == FDNN_ALGO_IGEMM_PAIR || !igemm_geometry_ok(d))
      return fail(FDNN_NOT_SUPPORTED, "a float32 output from 16-bit operands runs on the single-CTA tensor-core path only");
    algo = FDNN_ALGO_IGEMM;
    plan->bytes += 2.0 * m * d->k;  // y is four bytes per element
  }
  if ((algo == FDNN_ALGO_IGEMM || algo == FDNN_ALGO_IGEMM_PAIR) && !geom_ok)
    return fail(FDNN_NOT_SUPPORTED, "implicit-GEMM path does not support this problem");
  const bool want_auto = algo == FDNN_ALGO_AUTO;
  if (want_auto) algo = (geom_ok && (plan->flops >= kSmallFlops || small_on_tensor_cores(d, oh, ow, plan->flops))) ? FDNN_ALGO_IGEMM : FDNN_ALGO_DIRECT;
  if (algo != FDNN_ALGO_IGEMM && algo != FDNN_ALGO_DIRECT && algo != FDNN_ALGO_IGEMM_PAIR)
    return fail(FDNN_BAD_PARAM, "unknown algo");
  plan->algo = algo;

  if (algo == FDNN_ALGO_DIRECT) {
    long long total = (long long)d->n * d->k * oh * ow;
    long long blocks = (total + 255) / 256;
    if (blocks > 148LL * 64) blocks = 148LL * 64;
    if (blocks < 1) blocks = 1;
    plan->grid = int(blocks);
    plan->block = 256;
    plan->launches = 1;
    return FDNN_OK;
  }

  LowChannel lc = low_channel_geometry(d, oh, ow, y);
  if (out_f32) lc.ok = false;   // quads and pixel groups rely on y's 16-bit layout
  // A quad multiplies each pixel's window by the zeros its neighbours' taps leave, so that an infinite pixel turns outputs
  // that do not read it into NaN.  Small layers, which the direct kernel computes tap by tap, keep that apart, as pixel
  // windows do (3 -> 16 channels 5x5 on 32 x 32: quads 5.8 us, windows 5.9, direct 11.9; 11x11, too wide for windows: 6.9
  // against 19.9 on the direct kernel).
  if (want_auto && plan->flops < kSmallFlops) lc.ok = false;
  if (lc.ok) {
    const int sms_lc = sm_count();
    const int m_tiles_lc = d->n * lc.tiles_per_image;
    const int n_gemm = 4 * d->k;
    plan->low_channel = 1;
    plan->c_padded = 4;
    plan->x_repacked = 1;
    plan->w_packed = 1;
    plan->workspace_bytes = (long long)d->n * d->h * lc.w_pad * 4 * es;
    plan->packed_weight_bytes = (long long)n_gemm * d->r * 64 * es;
    plan->tile_m = 128;
    plan->tile_k = 64;
    plan->tile_n = choose_tile_n(d->dtype, m_tiles_lc, n_gemm, sms_lc);
    if (forced_tile_n(d) != 0) plan->tile_n = forced_tile_n(d);
    plan->stages = igemm_stages(d->dtype, plan->tile_n);
    plan->smem_bytes = igemm_smem_bytes(d->dtype, plan->tile_n);
    const long long tiles_lc = (long long)m_tiles_lc * ((n_gemm + plan->tile_n - 1) / plan->tile_n);
    plan->grid = int(tiles_lc < sms_lc ? tiles_lc : sms_lc);
    plan->block = igemm_threads();
    plan->launches = 2;
    // CTA pairs keep their half of the quad filter resident: 216 vs 225 us on the 7x7 stride-2 stem
    const long long pair_tiles_lc = (long long)((m_tiles_lc + 1) / 2) * ((n_gemm + 255) / 256);
    if (algo == FDNN_ALGO_IGEMM_PAIR ||
        (want_auto && sms_lc % 2 == 0 && n_gemm >= 256 && pair_tiles_lc >= sms_lc / 2)) {
      plan->algo = FDNN_ALGO_IGEMM_PAIR;
      plan->tile_m = 256;
      plan->tile_n = 256;
      plan->stages = igemm_pair_stages();
      plan->smem_bytes = igemm_pair_smem_bytes();
      plan->block = igemm_pair_threads();
      const long long pairs = pair_tiles_lc < sms_lc / 2 ? pair_tiles_lc : sms_lc / 2;
      plan->grid = int(2 * pairs);
      lc = low_channel_geometry(d, oh, ow, y, true);
      if (lc.fused3) {
        // dense 3-channel input: no relayout pass; two small scratch slots per CTA instead of a copy of x
        plan->low_channel = 2;
        plan->c_padded = 3;
        plan->x_repacked = 0;
        plan->tile_k = 48;
        plan->workspace_bytes = (long long)plan->grid * 2 * lc.slot_bytes;
        plan->launches = 1;
      }
    }
    return FDNN_OK;
  }

  if (allow_group && !out_f32 && (d->algo & FDNN_ALGO_FLAG_NO_PIXEL_GROUP) == 0) {
    const int q = choose_pixel_group(d, oh, ow, y);
    if (q > 1) {
      fdnn_conv_desc v = grouped_desc(d, q, oh, ow);
      v.algo = d->algo;
      fdnn_conv_plan pv;
      if (make_plan(&v, x, nullptr, y, &pv, false) == FDNN_OK && pv.algo != FDNN_ALGO_DIRECT && pv.ow * q == ow) {
        const double flops = plan->flops, bytes = plan->bytes;
        *plan = pv;
        plan->pixel_group = q;
        plan->oh = oh;
        plan->ow = ow;
        plan->flops = flops;
        plan->bytes = bytes;
        plan->w_packed = 1;
        plan->packed_weight_bytes = (long long)v.k * v.r * v.s * padded_channels(d->dtype, d->c) * es;
        return FDNN_OK;
      }
    }
  }

  const int gran = 16 / es;  // channels per 16 bytes
  const bool is16 = es == 2;
  // A stride over an extent of one carries no information (torch reports
  // arbitrary values there), so only strides of real extents are constrained.
  auto stride_ok = [gran](long long extent, long long stride) { return extent <= 1 || stride % gran == 0; };
  // x in place: channel-contiguous, every other stride a multiple of 16 bytes
  const bool x_inplace = is16 && (d->c == 1 || d->x_strides[1] == 1) && stride_ok(d->n, d->x_strides[0]) &&
                         stride_ok(d->h, d->x_strides[2]) && stride_ok(d->w, d->x_strides[3]) &&
                         (d->w <= 1 || d->x_strides[3] >= d->c) && aligned16(x);
  const bool w_inplace = filter_in_place(d, w);
  const int c_pad = padded_channels(d->dtype, d->c);
  plan->c_padded = c_pad;
  plan->x_repacked = x_inplace ? 0 : 1;
  const bool w_direct = w_inplace || filter_mn_major(d, w);
  plan->w_packed = w_direct ? 0 : 1;
  const int planes = (d->dtype == FDNN_F32) ? 2 : 1;
  if (!x_inplace) plan->workspace_bytes = (long long)planes * d->n * d->h * d->w * padded_x_channels(d) * es;
  if (!w_direct) plan->packed_weight_bytes = (long long)planes * d->k * d->r * d->s * c_pad * es;
  plan->tile_m = 128;
  plan->tile_k = 128 / es;
  const int m_tiles = int(((long long)m + 127) / 128);
  const int sms = sm_count();
  plan->tile_n = choose_tile_n(d->dtype, m_tiles, d->k, sms);
  if (forced_tile_n(d) != 0) plan->tile_n = forced_tile_n(d);
  plan->stages = igemm_stages(d->dtype, plan->tile_n);
  plan->smem_bytes = igemm_smem_bytes(d->dtype, plan->tile_n);
  const long long tiles = (long long)m_tiles * ((d->k + plan->tile_n - 1) / plan->tile_n);
  plan->grid = int(tiles < sms ? tiles : sms);
  plan->block = igemm_threads();
  plan->launches = 1 + plan->x_repacked;

  if (plan->x_repacked && algo == FDNN_ALGO_IGEMM) {
    const PixelWindows pw = pixel_windows(d, oh, ow);
    if (pw.ok) {
      const long long window_tiles = (long long)d->n * pw.tiles_per_image;
      plan->workspace_bytes = pw.scratch;
      plan->tile_n = choose_tile_n(d->dtype, int(window_tiles), d->k, sms);
      if (forced_tile_n(d) != 0) plan->tile_n = forced_tile_n(d);
      plan->stages = igemm_stages(d->dtype, plan->tile_n);
      plan->smem_bytes = igemm_smem_bytes(d->dtype, plan->tile_n);
      const long long all = window_tiles * ((d->k + plan->tile_n - 1) / plan->tile_n);
      plan->grid = int(all < sms ? all : sms);
      return FDNN_OK;
    }
  }

  // CTA pairs: 16-bit types writing a dense NHWC y.  Worth it when the layer is
  // wide enough for 256-channel tiles and has at least one full wave of pairs.
  const bool pair_ok = is16 && !out_f32 && y_is_dense_nhwc(d, oh, ow, y) && (sms % 2 == 0);
  if (algo == FDNN_ALGO_IGEMM_PAIR && !pair_ok)
    return fail(FDNN_NOT_SUPPORTED, "the CTA-pair kernel needs f16/bf16 tensors and a dense channels-last output");
  const long long pair_tiles = (long long)((m_tiles + 1) / 2) * ((d->k + 255) / 256);
  const long long k_steps = (long long)d->r * d->s * ((c_pad + 63) / 64);
  const int pairs_all = sms / 2;
  const bool resident = d->k <= 256 && k_steps <= igemm_pair_max_resident_steps();
  const bool sk_on = split_allowed && plan_stream_k(pair_tiles, k_steps, pairs_all, resident).worth;
  // Measured on the ResNet-50 layers (python -m flagdnn_b200.tune): with at least 16 reduction steps pairs win
  // whenever every pair has a tile; with 32 or more steps they still win with half the pairs idle (a pair reads
  // each operand byte from L2 once for two tiles: 512 -> 512 3x3 stride 2 at 128 images 38.5 -> 32.1 us).
  const bool pairs_fill = pair_tiles >= pairs_all || (k_steps >= 32 && 2 * pair_tiles >= pairs_all);
  if (algo == FDNN_ALGO_IGEMM_PAIR || (want_auto && pair_ok && d->k >= 256 && k_steps >= 16 && (pairs_fill || sk_on))) {
    plan->algo = FDNN_ALGO_IGEMM_PAIR;
    plan->tile_m = 256;
    plan->tile_n = 256;
    plan->stages = igemm_pair_stages();
    plan->smem_bytes = igemm_pair_smem_bytes();
    plan->block = igemm_pair_threads();
    const long long pairs = (pair_tiles < pairs_all && !sk_on) ? pair_tiles : pairs_all;
    plan->grid = int(2 * pairs);
    if (sk_on) {
      plan->stream_k = 1;
      plan->streamk_bytes = FDNN_STREAMK_FLAG_BYTES + (long long)plan->grid * 128 * 256 * 4;
    }
  }
  return FDNN_OK;
}

// One activation copy per filter row (conv_rows_sm100.cu): whether a call that its plan sends to a tensor-core kernel runs
// there instead, and on which tiles.  The layouts of x and of the packed filter stay those of the plan.  Measured kernels,
// a copy per tap against this (bf16, channels-last, 3x3, microseconds): 256 -> 256 on 256 x 14 x 14 46.1 and 40.7, on
// 128 images 31.1 and 22.7, on one 10.3 and 9.0; 64 -> 64 on 128 x 56 x 56 (four pixels per row before) 49.9 and 32.2;
// 128 -> 128 on 128 x 28 x 28 34.7 and 25.1; 512 -> 512 on 128 x 7 x 7, an eighth of the walk rows no output, 30.5 and 27.6;
// 104 -> 152 on 24 x 45 x 37 40.6 and 25.7; NCHW 64 -> 64 on 128 x 56 x 56 60.1 and 38.0; two groups 64 -> 128 on
// 256 x 56 x 56 (block-diagonal before) 122 and 72; sixteen groups of 32 on 16 x 28 x 28 27.9 and 15.0.
//   Where it loses: few steps in all (64 -> 128 on 8 x 28 x 28 5.5 and 5.9: smaller tiles start sooner); where pair tiles fill a
// round and a bit (200 -> 200 5x5 on 20 x 31 x 29 NCHW: 141 tiles of 128 x 256 in one round against 152 in three, 42 and 50);
// and where the taps of a filter row do not fit a slot of the filter ring, so that every tap is waited for by itself
// (86 columns, 7x7 on 81 x 28 x 28 x 201 183 and 219).  So both sides are counted in clocks of the busiest SM: rounds of tiles,
// each as long as its steps of four MMAs (fp32: twelve) or as its drain, whichever is longer, and 1700 for the launch.
//                              a copy per tap                          here
//   step, columns 64/128/256   365 / 510 / 650, pairs 690              225 / 290 / 600 (570 where there are
//                                                                      more rounds); a tap by itself 600
//   fp32                       800 / 1100                              600 / 830
//   drain                      1500 / 3000 / 5000 through the TMA      2000 / 3000 / 4400 by sectors of 32 bytes
//                              unit, 6500 / 10000 / 11500 along        2700 / 5300 / 9200 along channels
//                              channels, 2000 / 3500 / 5500 pixels     1500 / 2800 / 4000 pixels
//   pixels off 128-byte lines  1100 per copy up to 192 bytes, wider    1100 per copy up to 192 bytes
//                              ones 1.05 (64 columns) or 1.15 times;
//                              64-byte ones 1100 from three rounds on
// The constants are fitted to 1600 layers timed on the copy per tap and on all three widths here: 29 are over 4 % slower than on
// the copy per tap (by 1.3 times at most); with one step time for all and 1350 for any pixel off a line it was 75 of 1200
// (34 x 66 x 8 x 824 -> 288 80 and 105, 87 x 14 x 14 x 440 -> 184 5x5 65 and 81).
struct RowsMode {
  int tile_n;          // 0: no
  int pitch;           // walk rows per image row
  int m_tiles, n_tiles, grid;
  int blk_groups;      // groups per 64-channel block (1: not grouped)
};
// Every output pixel starts on a 32-byte boundary and its channels fill 32-byte pieces.
bool sector_aligned(const fdnn_conv_desc& d, int oh, int ow, const void* y) {
  const int gran = 32 / elem_size(d.dtype);
  return d.k % gran == 0 && (reinterpret_cast<uintptr_t>(y) & 31u) == 0 && (d.n <= 1 || d.y_strides[0] % gran == 0) &&
         (oh <= 1 || d.y_strides[2] % gran == 0) && (ow <= 1 || d.y_strides[3] % gran == 0);
}
RowsMode rows_mode(const fdnn_conv_desc* d, const fdnn_conv_plan& plan, const void* y) {
  RowsMode g = {};
  const int oh = plan.oh, ow = plan.ow;
  const int es = elem_size(d->dtype);
  if (es > 4 || d->algo != FDNN_ALGO_AUTO || d->stride_w != 1 || d->s < 2 || (d->s - 1) * d->dil_w > kRowsCopy - 128) return g;
  fdnn_conv_desc one = *d;
  one.groups = 1;
  const int cg = d->c / d->groups, kg = d->k / d->groups;
  if (!igemm_geometry_ok(&one) || oh < 1 || ow < 1 || cg < 8 || d->k < 8) return g;
  // y along channels, or along the pixels of every image
  const bool pixels = (ow == 1 || d->y_strides[3] == 1) && (oh == 1 || d->y_strides[2] == ow);
  if (d->y_strides[1] != 1 && !pixels) return g;
  g.pitch = d->w + (d->pad_left > d->pad_right ? d->pad_left : d->pad_right);
  if (g.pitch - d->w - d->pad_left > 127 || ow > g.pitch) return g;
  const long long walk = (long long)d->n * oh * g.pitch;
  if (walk > 2000000000LL) return g;
  const int sms = sm_count();
  if (sms % 2 != 0) return g;
  g.m_tiles = int((walk + 127) / 128);
  g.blk_groups = 1;
  if (d->groups > 1) {
    if (es != 2 || (cg != 16 && cg != 32) || d->c % 64 != 0 || kg % 32 != 0 || d->y_strides[1] != 1 ||
        !sector_aligned(*d, oh, ow, y))
      return g;
    g.blk_groups = 64 / cg;
    const int bn = g.blk_groups * kg;
    if (bn != 64 && bn != 128 && bn != 256) return g;
    g.tile_n = bn;
    g.n_tiles = d->c / 64;
  } else {
    // clocks of the busiest SM (see above)
    const long long pixel = es * (plan.x_repacked ? padded_x_channels(d) : d->x_strides[3]);
    const bool off_lines = d->w > 1 && pixel % 128 != 0 && pixel != 64;
    const double copy = off_lines && pixel <= 192 ? 1100 : 0;
    const double steps = double(d->r) * ((d->c * es + 127) / 128);
    const int q = plan.pixel_group > 1 ? plan.pixel_group : 1;
    const bool pair = plan.algo == FDNN_ALGO_IGEMM_PAIR;
    auto column_class = [](int columns) { return columns == 64 ? 0 : columns == 128 ? 1 : 2; };
    auto rounds = [](long long tiles, int units) { return double((tiles + units - 1) / units); };
    auto longer = [](double x, double z) { return x > z ? x : z; };
    static constexpr double kStep[3] = {365, 510, 650}, kDrainTma[3] = {1500, 3000, 5000}, kDrainOther[3] = {6500, 10000, 11500}, kDrainPixels[3] = {2000, 3500, 5500};
    static constexpr double kTap[3] = {225, 290, 600}, kSectors[3] = {2000, 3000, 4400}, kChannels[3] = {2700, 5300, 9200},
                            kPixels[3] = {1500, 2800, 4000};
    const int now_class = column_class(plan.tile_n);
    const long long m_now = ((long long)d->n * oh * ow / q + plan.tile_m - 1) / plan.tile_m;
    const long long tiles_now = m_now * (((long long)q * d->k + plan.tile_n - 1) / plan.tile_n);
    const double rounds_now = rounds(tiles_now, pair ? sms / 2 : sms);
    double step = pair ? 690 : es == 4 ? (now_class == 0 ? 800 : 1100) : kStep[now_class];
    step = longer(step, pixel == 64 && d->w > 1 && q == 1 && rounds_now >= 3 ? 1100 : copy);
    if (off_lines && pixel > 192) step *= !pair && now_class == 0 ? 1.05 : 1.15;
    const double* drain_now = y_is_dense_nhwc(d, oh, ow, y) ? kDrainTma : d->y_strides[1] != 1 ? kDrainPixels : kDrainOther;
    double best_cost = rounds_now * longer(steps * (d->s + (q - 1) * d->stride_w) * step, drain_now[now_class]);
    const double* drain = d->y_strides[1] != 1 ? kPixels : sector_aligned(*d, oh, ow, y) ? kSectors : kChannels;
    for (int bn = 64; bn <= (es == 2 ? 256 : 128); bn *= 2) {
      if (bn > 64 && bn / 2 >= d->k) break;
      RowsParams ring = {};
      ring.R = d->r;
      ring.S = d->s;
      ring.halves = es == 4 ? 2 : 1;
      ring.c_blocks = int((d->c * es + 127) / 128);
      ring.n_tiles = (d->k + bn - 1) / bn;
      ring.b_bytes = ring.halves * (bn / 2) * 128;
      rows_stages(&ring);
      const long long tiles = (long long)((g.m_tiles + 1) / 2) * ring.n_tiles;
      const double all_rounds = rounds(tiles, sms / 2);
      double tap = es == 4 ? (bn == 64 ? 600 : 830) : bn == 256 && all_rounds > 1 ? 570 : kTap[column_class(bn)];
      if (ring.b_taps != d->s && bn < 256) tap = longer(tap, 600);
      tap = longer(tap, copy / d->s);
      const double cost = 1700 + all_rounds * longer(steps * d->s * tap, drain[column_class(bn)]);
      if (cost < best_cost) {
        best_cost = cost;
        g.tile_n = bn;
      }
    }
    if (g.tile_n == 0) return g;
    g.n_tiles = (d->k + g.tile_n - 1) / g.tile_n;
  }
  const long long tiles = (long long)((g.m_tiles + 1) / 2) * g.n_tiles;
  g.grid = 2 * int(tiles < sms / 2 ? tiles : sms / 2);
  return g;
}

// ... of a layer without groups, or of one with them and its filters where rows_filter finds them.
bool rows_layer_ok(const fdnn_conv_desc& d, const fdnn_conv_plan& plan) {
  return plan.algo != FDNN_ALGO_DIRECT && plan.low_channel == 0 && !(plan.x_repacked && d.c < 8);
}

// The filter as the kernels of conv_rows_sm100.cu read it.
struct FilterView {
  const void* base;
  int c, s_pitch, c_step;      // channels per tap, taps per filter row, first channel of group g: g * c_step
  long long s_tap, s_k;
};
// A grouped layer's filters: in place, or in the dense filter in front of the packed one.  False: neither.
bool rows_group_filter(const fdnn_conv_desc& d, const void* w, const void* w_packed, FilterView* f) {
  const int cg = d.c / d.groups;
  if (w != nullptr && filter_in_place(&d, w)) {
    *f = {w, cg, d.s, 0, d.s > 1 ? d.w_strides[3] : d.w_strides[2], d.w_strides[0]};
    return true;
  }
  if (!group_dense_ok(&d) || w_packed == nullptr || !aligned16(w_packed)) return false;
  *f = {w_packed, d.c, d.s, cg, d.c, (long long)d.r * d.s * d.c};
  return true;
}

// Several groups of a grouped 16-bit layer in one launch of the single-CTA kernel (see IgemmParams::groups), where that
// beats the route its plan names.  `group_batch` fills `one` with the plan of a single group on that kernel and
// answers how many column tiles of which width the launch would have, or 0 tiles when it does not apply:
//   * One launch per group costs 6 to 10 us each, however small the group (32 groups of 24 -> 48 channels 3x3 on
//     3 x 21 x 21: 242 us channels-last, 460 us NCHW, against 17.6 and 25 us in one).  A group that runs on CTA pairs
//     or groups its pixels fills the chip by itself and keeps its own launch.
//   * The block-diagonal dense layer multiplies G times as much, on wider tiles (256 channels in four groups on
//     16 x 56 x 56: 44.9 -> 28.2 us; 64 -> 128 in two groups on 256 x 56 x 56 stays dense: 125 us).
// Every group's channels start on 16 bytes in x, w and y, as for one launch per group, and the taps fit a
// five-dimensional im2col map.
GroupBatch group_batch(const fdnn_conv_desc* d, const void* x, const void* w, const void* y, const fdnn_conv_plan& plan,
                       bool dense) {
  GroupBatch g;
  g.tile_n = 0;
  if (!group_loop_ok(d) || d->algo != FDNN_ALGO_AUTO || elem_size(d->dtype) != 2) return g;
  if (!batch_geometry_ok(d)) return g;
  fdnn_conv_desc sub = one_group_desc(d);
  if (filter_mn_major(&sub, w)) return g;   // read MN-major, group by group
  fdnn_conv_plan own;
  if (make_plan(&sub, x, w, y, &own) != FDNN_OK || own.pixel_group > 1 || own.low_channel != 0 ||
      own.algo == FDNN_ALGO_IGEMM_PAIR)
    return g;
  sub.algo = FDNN_ALGO_IGEMM;
  if (make_plan(&sub, x, w, y, &g.one, false) != FDNN_OK || g.one.algo != FDNN_ALGO_IGEMM || g.one.low_channel != 0) return g;
  const int sms = sm_count();
  const long long m_tiles = ((long long)d->n * g.one.oh * g.one.ow + 127) / 128;
  if (m_tiles * d->groups > 1 << 28) return g;
  const int bn = choose_tile_n(d->dtype, int(m_tiles * d->groups), sub.k, sms);
  if (dense) {
    // relative cost of a launch: rounds x steps x what a step costs (as in choose_tile_n); a pair tile keeps two CTAs busy
    const long long tiles = m_tiles * d->groups * ((sub.k + bn - 1) / bn);
    const double batch = double((tiles + sms - 1) / sms) * d->r * d->s * ((sub.c + 63) / 64) * (bn + 384);
    const int q = plan.pixel_group > 1 ? plan.pixel_group : 1;
    const long long mt = ((long long)d->n * g.one.oh * g.one.ow / q + plan.tile_m - 1) / plan.tile_m;
    const long long nt = ((long long)q * d->k + plan.tile_n - 1) / plan.tile_n;
    const double whole = double((mt * nt * (plan.tile_m / 128) + sms - 1) / sms) * d->r * (d->s + (q - 1) * d->stride_w) *
                         ((d->c + 63) / 64) * (plan.tile_n + 384);
    // groups whose channels do not start on 64-byte boundaries pay more per copy (86 x 21 x 21, 80 channels in two groups of
    // 40: 22 us dense, 31 us in one launch at 0.73 of its cost)
    if (batch > ((sub.c * elem_size(d->dtype)) % 64 == 0 ? 0.7 : 0.5) * whole) return g;
  }
  g.tile_n = bn;
  return g;
}

// ------------------------------------------------------- tensor map encoding
PFN_cuTensorMapEncodeTiled g_encode_tiled = nullptr;
PFN_cuTensorMapEncodeIm2col g_encode_im2col = nullptr;
std::once_flag g_driver_once;
bool g_driver_ok = false;
int g_driver_version = 0;

void load_driver_entry_points() {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  bool ok = true;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || fn == nullptr)
    ok = false;
  g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
  fn = nullptr;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || fn == nullptr)
    ok = false;
  g_encode_im2col = reinterpret_cast<PFN_cuTensorMapEncodeIm2col>(fn);
  cudaDriverGetVersion(&g_driver_version);
  cudaGetLastError();
  g_driver_ok = ok;
}

// Encoded tensor maps are remembered per thread, keyed by every argument of the encode call: a layer that is run
// again on the same buffers (the steady state of an eager loop or of a compiled plan) costs a table lookup
// instead of a driver call per map.  512 entries, four-way set-associative; a miss simply re-encodes.
struct MapKey {
  uint64_t w[30];
};
struct MapSlot {
  MapKey key;
  alignas(64) CUtensorMap map;
  uint32_t stamp;
  bool used;
};
constexpr int kMapSets = 128, kMapWays = 4;
std::atomic<long long> g_map_hits{0}, g_map_misses{0};

// Four chains side by side: one multiply after another over the whole key took a fifth of a microsecond per launch.
inline uint64_t map_key_hash(const MapKey& k) {
  constexpr int kWords = int(sizeof(k.w) / sizeof(k.w[0]));
  uint64_t h[4] = {0x9e3779b97f4a7c15ull, 0xbf58476d1ce4e5b9ull, 0x94d049bb133111ebull, 0xff51afd7ed558ccdull};
  for (int i = 0; i < kWords; ++i) h[i & 3] = (h[i & 3] ^ k.w[i]) * 0x9fb21c651e98df25ull;
  uint64_t v = h[0] ^ (h[1] >> 31) ^ (h[2] << 17) ^ (h[3] >> 13);
  v ^= v >> 32;
  v *= 0xff51afd7ed558ccdull;
  return v ^ (v >> 32);
}

template <typename Encode>
CUresult memo_lookup(CUtensorMap* tm, const MapKey& key, Encode&& encode) {
  // sets of four entries; within a set the entry used longest ago is replaced
  thread_local std::unique_ptr<MapSlot[]> slots;   // on the heap, made on a thread's first call
  thread_local uint32_t tick = 0;
  if (!slots) slots.reset(new MapSlot[kMapSets * kMapWays]());
  MapSlot* set = &slots[(map_key_hash(key) % kMapSets) * kMapWays];
  ++tick;
  MapSlot* victim = &set[0];
  for (int w = 0; w < kMapWays; ++w) {
    MapSlot& slot = set[w];
    if (slot.used && std::memcmp(&slot.key, &key, sizeof key) == 0) {
      *tm = slot.map;
      slot.stamp = tick;
      g_map_hits.fetch_add(1, std::memory_order_relaxed);
      return CUDA_SUCCESS;
    }
    if (!slot.used || (victim->used && int32_t(slot.stamp - victim->stamp) < 0)) victim = &slot;
  }
  g_map_misses.fetch_add(1, std::memory_order_relaxed);
  const CUresult r = encode();
  if (r == CUDA_SUCCESS) {
    victim->key = key;
    victim->map = *tm;
    victim->used = true;
    victim->stamp = tick;
  }
  return r;
}

CUresult memo_encode_tiled(CUtensorMap* tm, CUtensorMapDataType dt, cuuint32_t rank, void* base, const cuuint64_t* dims,
                           const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* estr,
                           CUtensorMapInterleave il, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2,
                           CUtensorMapFloatOOBfill oob) {
  MapKey k{};
  int n = 0;
  k.w[n++] = 1;
  k.w[n++] = uint64_t(dt) | uint64_t(rank) << 8 | uint64_t(il) << 16 | uint64_t(sw) << 24 | uint64_t(l2) << 32 |
             uint64_t(oob) << 40;
  k.w[n++] = reinterpret_cast<uint64_t>(base);
  for (cuuint32_t i = 0; i < rank && i < 5; ++i) k.w[n++] = dims[i];
  for (cuuint32_t i = 0; i + 1 < rank && i < 4; ++i) k.w[n++] = strides[i];
  for (cuuint32_t i = 0; i < rank && i < 5; ++i) k.w[n++] = uint64_t(box[i]) | uint64_t(estr[i]) << 32;
  return memo_lookup(tm, k, [&]() { return g_encode_tiled(tm, dt, rank, base, dims, strides, box, estr, il, sw, l2, oob); });
}

CUresult memo_encode_im2col(CUtensorMap* tm, CUtensorMapDataType dt, cuuint32_t rank, void* base,
                            const cuuint64_t* dims, const cuuint64_t* strides, const int* lower, const int* upper,
                            cuuint32_t channels_per_pixel, cuuint32_t pixels_per_column, const cuuint32_t* estr,
                            CUtensorMapInterleave il, CUtensorMapSwizzle sw, CUtensorMapL2promotion l2,
                            CUtensorMapFloatOOBfill oob) {
  MapKey k{};
  int n = 0;
  k.w[n++] = 2;
  k.w[n++] = uint64_t(dt) | uint64_t(rank) << 8 | uint64_t(il) << 16 | uint64_t(sw) << 24 | uint64_t(l2) << 32 |
             uint64_t(oob) << 40;
  k.w[n++] = reinterpret_cast<uint64_t>(base);
  k.w[n++] = uint64_t(channels_per_pixel) | uint64_t(pixels_per_column) << 32;
  for (cuuint32_t i = 0; i < rank && i < 5; ++i) k.w[n++] = dims[i];
  for (cuuint32_t i = 0; i + 1 < rank && i < 4; ++i) k.w[n++] = strides[i];
  for (cuuint32_t i = 0; i + 2 < rank && i < 3; ++i) k.w[n++] = uint64_t(uint32_t(lower[i])) | uint64_t(uint32_t(upper[i])) << 32;
  for (cuuint32_t i = 0; i < rank && i < 5; ++i) k.w[n++] = estr[i];
  return memo_lookup(tm, k, [&]() {
    return g_encode_im2col(tm, dt, rank, base, dims, strides, lower, upper, channels_per_pixel, pixels_per_column, estr,
                           il, sw, l2, oob);
  });
}

CUtensorMapDataType tm_dtype(int dtype) {
  switch (dtype) {
    case FDNN_F16: return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    case FDNN_BF16: return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    default: return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  }
}

// Activation map: NHWC tensor seen as (C, W, H, N); one copy brings 128 output
// pixels x one 128-byte channel block for a single filter tap.  With a walk pitch (see conv_rows_sm100.cu) it walks
// through rows of that many pixels, padding included, and brings kRowsCopy of them.
int encode_activation_map(CUtensorMap* tm, int dtype, const void* base, int C, int W, int H, int N,
                          long long sw, long long sh, long long sn, const fdnn_conv_desc* d, int groups = 1,
                          int walk_pitch = 0) {
  const int es = elem_size(dtype);
  cuuint64_t dims[4] = {cuuint64_t(C), cuuint64_t(W), cuuint64_t(H), cuuint64_t(N)};
  cuuint64_t strides[3] = {cuuint64_t(sw) * es, cuuint64_t(sh) * es, cuuint64_t(sn) * es};
  int lower[2] = {-d->pad_left, -d->pad_top};
  int upper[2] = {d->pad_right - (d->s - 1) * d->dil_w, d->pad_bottom - (d->r - 1) * d->dil_h};
  if (walk_pitch > 0) upper[0] = walk_pitch - W - d->pad_left;   // the taps to the right are further rows of the copy
  cuuint32_t trav[4] = {1, cuuint32_t(d->stride_w), cuuint32_t(d->stride_h), 1};
  const cuuint32_t channels_per_pixel = 128 / es;
  const cuuint32_t pixels_per_column = walk_pitch > 0 ? kRowsCopy : 128;
  // several groups in one launch: C channels per group, the images as the walk's third dimension, the groups behind them
  cuuint64_t dims5[5] = {cuuint64_t(C), cuuint64_t(W), cuuint64_t(H), cuuint64_t(N), cuuint64_t(groups)};
  cuuint64_t strides5[4] = {strides[0], strides[1], strides[2], cuuint64_t(C) * es};
  int lower5[3] = {lower[0], lower[1], 0};
  int upper5[3] = {upper[0], upper[1], 0};
  cuuint32_t trav5[5] = {1, cuuint32_t(d->stride_w), cuuint32_t(d->stride_h), 1, 1};
  CUresult r = groups > 1
      ? memo_encode_im2col(tm, tm_dtype(dtype), 5, const_cast<void*>(base), dims5, strides5, lower5, upper5,
                           channels_per_pixel, pixels_per_column, trav5, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
      : memo_encode_im2col(tm, tm_dtype(dtype), 4, const_cast<void*>(base), dims, strides, lower,
                               upper, channels_per_pixel, pixels_per_column, trav,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeIm2col failed with CUresult %d", int(r));
    return fail(FDNN_CUDA_ERROR, buf);
  }
  // Drivers up to CUDA 13.1 encode im2col maps of tensors smaller than 128 KiB
  // with a flag (bit 21 of the second 64-bit word) that makes the copy misread
  // them; the flag has to be cleared by hand for such tensors.
#ifndef FDNN_NO_SMALL_IM2COL_FIX
  if (g_driver_version <= 13010) {
    const long long extent =
        ((long long)(N - 1) * sn + (long long)(H - 1) * sh + (long long)(W - 1) * sw + (long long)C * groups) * es;
    if (extent < 131072) reinterpret_cast<uint64_t*>(tm)[1] &= ~(1ull << 21);
  }
#endif
  return FDNN_OK;
}

// Filter map: [K, R*S, C] seen as (C, R*S, K); one copy brings tile_n output
// channels x one 128-byte channel block of one tap.
int encode_filter_map(CUtensorMap* tm, int dtype, const void* base, int C, int taps, int K,
                      long long s_tap, long long s_k, int tile_n) {
  const int es = elem_size(dtype);
  cuuint64_t dims[3] = {cuuint64_t(C), cuuint64_t(taps), cuuint64_t(K)};
  cuuint64_t strides[2] = {cuuint64_t(s_tap) * es, cuuint64_t(s_k) * es};
  cuuint32_t box[3] = {cuuint32_t(128 / es), 1, cuuint32_t(tile_n)};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = memo_encode_tiled(tm, tm_dtype(dtype), 3, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed with CUresult %d", int(r));
    return fail(FDNN_CUDA_ERROR, buf);
  }
  return FDNN_OK;
}

// Output map: dense NHWC y seen as a row-major [M, K] matrix; one store writes
// 32 pixels x 128 bytes of channels.
int encode_output_map(CUtensorMap* tm, int dtype, void* base, int K, long long M, long long row_stride, int groups = 1) {
  const int es = elem_size(dtype);
  // three-dimensional so that the low-channel mode can share the store path: (channel, row, image = 1); with several
  // groups in one launch (channel of the group, row, group)
  cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(M), cuuint64_t(groups)};
  cuuint64_t strides[2] = {cuuint64_t(row_stride) * es,
                           groups > 1 ? cuuint64_t(K) * es : cuuint64_t(row_stride) * es * cuuint64_t(M)};
  cuuint32_t box[3] = {cuuint32_t(128 / es), 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = memo_encode_tiled(tm, tm_dtype(dtype), 3, base, dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled (output) failed with CUresult %d", int(r));
    return fail(FDNN_CUDA_ERROR, buf);
  }
  return FDNN_OK;
}

// The residual tensor (laid out like a dense NHWC y) with one box per output tile: 128 rows x box_cols
// channels, no swizzle.  The producers use it for L2 prefetches only; nothing is copied to shared memory.
int encode_residual_map(CUtensorMap* tm, int dtype, const void* base, int K, long long M, long long row_stride,
                        int box_cols, int groups = 1) {
  const int es = elem_size(dtype);
  cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(M), cuuint64_t(groups)};
  cuuint64_t strides[2] = {cuuint64_t(row_stride) * es,
                           groups > 1 ? cuuint64_t(K) * es : cuuint64_t(row_stride) * es * cuuint64_t(M)};
  cuuint32_t box[3] = {cuuint32_t(box_cols), 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = memo_encode_tiled(tm, tm_dtype(dtype), 3, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled (residual) failed with CUresult %d", int(r));
    return fail(FDNN_CUDA_ERROR, buf);
  }
  return FDNN_OK;
}

__device__ uint32_t g_status_word;

std::once_flag g_prepare_once[64];
cudaError_t g_prepare_result[64];
}  // namespace

long long default_wait_limit_cycles() { return 4000000000LL; }  // kWaitLimitCycles of sm100_ptx.cuh

bool launch_overlap_enabled() {
  static const bool on = []() {
    const char* v = std::getenv("FLAGDNN_B200_LAUNCH_OVERLAP");
    return !(v != nullptr && v[0] == '0' && v[1] == '\0');
  }();
  return on;
}

namespace {
std::atomic<long long*> g_prof_buffer[64];  // per device ordinal; set through fdnn_debug_set_profile_buffer

long long* prof_buffer_of_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  return g_prof_buffer[dev].load(std::memory_order_relaxed);
}
std::atomic<long long> g_wait_limit{0};  // 0: the default limit; set through fdnn_debug_set_wait_limit
std::atomic<int> g_skip_copies{0};

void fill_debug_params(IgemmParams* p) {
  const long long limit = g_wait_limit.load(std::memory_order_relaxed);
  p->wait_limit = limit > 0 ? limit : default_wait_limit_cycles();
  p->skip_copies = g_skip_copies.load(std::memory_order_relaxed);
}
uint32_t* g_status_ptr[64];  // device address of g_status_word, looked up once per device

}  // namespace

int current_sm_count() { return sm_count(); }

// x of a depthwise layer as (channel, column, row, image), boxes of `chunk` channels x `span` pixels x `rows` rows; what lies outside
// arrives as zeros, which is the padding.
bool encode_depthwise_map(CUtensorMap* tm, int dtype, const DirectParams& p, int chunk, int span, int rows) {
  const int es = elem_size(dtype);
  // a stride over an extent of one says nothing: any multiple of 16 bytes will do
  const long long any = (long long)(p.C * es + 15) / 16 * 16;
  const long long sw = p.W > 1 ? p.x_s[3] * es : any, sh = p.H > 1 ? p.x_s[2] * es : any, sn = p.N > 1 ? p.x_s[0] * es : any;
  cuuint64_t dims[4] = {cuuint64_t(p.C), cuuint64_t(p.W), cuuint64_t(p.H), cuuint64_t(p.N)};
  cuuint64_t strides[3] = {cuuint64_t(sw), cuuint64_t(sh), cuuint64_t(sn)};
  cuuint32_t box[4] = {cuuint32_t(chunk), cuuint32_t(span), cuuint32_t(rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return memo_encode_tiled(tm, tm_dtype(dtype), 4, const_cast<void*>(p.x), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

uint32_t* device_status_word() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<uint32_t*>(p);
}

}  // namespace fdnn

namespace fdnn {
namespace {

int encode_tiled(CUtensorMap* tm, int dtype, const void* base, int rank, const cuuint64_t* dims,
                 const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t* estr, const char* what) {
  CUresult r = memo_encode_tiled(tm, tm_dtype(dtype), rank, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[160];
    std::snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled (%s) failed with CUresult %d", what, int(r));
    return fail(FDNN_CUDA_ERROR, buf);
  }
  return FDNN_OK;
}

// Low-channel forward: repack x to [N][H][w_pad][4], then run the implicit-GEMM
// kernel with pixel quads as rows (see LowChannel above).
int fwd_low_channel(const fdnn_conv_desc& d, const fdnn_conv_plan& plan, int dev, const void* x,
                    const void* w_packed, const void* bias, const void* scale, int activation, void* y,
                    void* workspace, cudaStream_t stream) {
  const int es = elem_size(d.dtype);
  const bool fused3 = plan.low_channel == 2;
  const LowChannel lc = low_channel_geometry(&d, plan.oh, plan.ow, y, fused3);
  if (!lc.ok || lc.fused3 != fused3) return fail(FDNN_BAD_PARAM, "low-channel plan no longer applies to these buffers");
  cudaError_t e = cudaSuccess;
  if (!fused3) {
    e = launch_repack_x_lowc(d.dtype, x, reinterpret_cast<const long long*>(d.x_strides), d.n, d.c, d.h, d.w, lc.lpad,
                             lc.w_pad, workspace, stream);
    if (e != cudaSuccess) return fail_cuda("low-channel repack launch", e);
  }

  const int n_gemm = 4 * d.k;
  alignas(64) CUtensorMap tmA, tmB, tmY, tmY2;
  if (fused3) {
    // windows of 64 elements every 4 output pixels' worth of input, over the per-CTA scratch slots:
    // (element, quad, row of the slot, slot)
    cuuint64_t dims[4] = {64, cuuint64_t(lc.ow4), cuuint64_t(lc.raw_rows), cuuint64_t(plan.grid) * 2};
    cuuint64_t strides[3] = {cuuint64_t(d.stride_w) * 4 * 3 * es, cuuint64_t(lc.row_chunks) * 16, cuuint64_t(lc.slot_bytes)};
    cuuint32_t box[4] = {64, cuuint32_t(lc.ow4), cuuint32_t(lc.ohs * d.stride_h), 1};
    cuuint32_t estr[4] = {1, 1, cuuint32_t(d.stride_h), 1};
    int st = encode_tiled(&tmA, d.dtype, workspace, 4, dims, strides, box, estr, "low-channel scratch windows");
    if (st != FDNN_OK) return st;
  } else {
    // windows of 64 elements that start every 4 output pixels' worth of input (overlapping rows)
    cuuint64_t dims[4] = {64, cuuint64_t(lc.ow4), cuuint64_t(d.h), cuuint64_t(d.n)};
    cuuint64_t strides[3] = {cuuint64_t(d.stride_w) * 4 * 4 * es, cuuint64_t(lc.w_pad) * 4 * es,
                             cuuint64_t(d.h) * lc.w_pad * 4 * es};
    cuuint32_t box[4] = {64, cuuint32_t(lc.ow4), cuuint32_t(lc.ohs * d.stride_h), 1};
    cuuint32_t estr[4] = {1, 1, cuuint32_t(d.stride_h), 1};
    int st = encode_tiled(&tmA, d.dtype, workspace, 4, dims, strides, box, estr, "low-channel activations");
    if (st != FDNN_OK) return st;
  }
  const int b_box_rows = plan.algo == FDNN_ALGO_IGEMM_PAIR ? 128 : plan.tile_n;
  {
    cuuint64_t dims[3] = {64, cuuint64_t(d.r), cuuint64_t(n_gemm)};
    cuuint64_t strides[2] = {cuuint64_t(64) * es, cuuint64_t(d.r) * 64 * es};
    cuuint32_t box[3] = {64, 1, cuuint32_t(b_box_rows)};
    cuuint32_t estr[3] = {1, 1, 1};
    int st = encode_tiled(&tmB, d.dtype, w_packed, 3, dims, strides, box, estr, "low-channel filter");
    if (st != FDNN_OK) return st;
  }
  const int tail_rows = lc.rows_per_tile % 32;
  {
    // y as (4*K channels of a quad, quads of one image, images)
    cuuint64_t dims[3] = {cuuint64_t(n_gemm), cuuint64_t(plan.oh) * lc.ow4, cuuint64_t(d.n)};
    cuuint64_t strides[2] = {cuuint64_t(n_gemm) * es, cuuint64_t(plan.oh) * lc.ow4 * n_gemm * es};
    cuuint32_t estr[3] = {1, 1, 1};
    cuuint32_t box[3] = {64, 32, 1};
    int st = encode_tiled(&tmY, d.dtype, y, 3, dims, strides, box, estr, "low-channel output");
    if (st != FDNN_OK) return st;
    cuuint32_t box2[3] = {64, cuuint32_t(tail_rows > 0 ? tail_rows : 32), 1};
    st = encode_tiled(&tmY2, d.dtype, y, 3, dims, strides, box2, estr, "low-channel output tail");
    if (st != FDNN_OK) return st;
  }

  IgemmParams p = {};
  p.Kout = n_gemm;
  p.k_real = d.k;
  p.OH = plan.oh; p.OW = plan.ow;
  p.stride_h = d.stride_h; p.stride_w = d.stride_w; p.pad_top = d.pad_top; p.pad_left = d.pad_left;
  p.dil_h = d.dil_h; p.dil_w = 1;
  p.R = d.r; p.S = 1; p.c_blocks = 1;
  p.m_tiles = d.n * lc.tiles_per_image;
  p.M = p.m_tiles * 128;
  p.n_tiles = (n_gemm + plan.tile_n - 1) / plan.tile_n;
  p.groups = 1;
  p.group_n_tiles = p.n_tiles;
  p.bias = bias; p.scale = scale; p.y = y;
  p.act = activation;
  p.vec_store = 0;
  p.tma_store = 1;
  p.lowc = 1;
  p.rows_per_tile = lc.rows_per_tile;
  p.tiles_per_image = lc.tiles_per_image;
  p.ohs = lc.ohs;
  p.a_tx_bytes = lc.rows_per_tile * 128;
  p.k16_per_step = 4;
  if (fused3) {
    p.fused3 = 1;
    p.x3 = x;
    p.scratch3 = workspace;
    p.x_h = d.h;
    p.x_row_chunks = 3 * d.w / 8;
    p.x_unaligned = (reinterpret_cast<uintptr_t>(x) & 15u) != 0 ? 1 : 0;
    p.raw_rows = lc.raw_rows;
    p.row_chunks = lc.row_chunks;
    p.lead_chunks = lc.lead_chunks;
    p.slot_elems = int(lc.slot_bytes / es);
    p.k16_per_step = 3;
  }
  p.prof = prof_buffer_of_current_device();
  fill_debug_params(&p);
  p.status = g_status_ptr[dev];
  if (p.status == nullptr) return fail(FDNN_CUDA_ERROR, "status word address unavailable");
  if (plan.algo == FDNN_ALGO_IGEMM_PAIR) {
    p.b_resident = (n_gemm <= 256 && d.r <= igemm_pair_max_resident_steps()) ? 1 : 0;
    e = launch_igemm_pair(d.dtype, tmA, tmB, tmY, tmY2, tmY, tmY, p, plan.grid, stream);
  } else {
    // the single-CTA kernel has no fifth 16-bit map slot: the tail map travels in the unused tmA2 slot
    e = launch_igemm(d.dtype, plan.tile_n, tmA, tmY2, tmB, tmB, tmY, tmY, tmY, p, plan.grid, stream);
  }
  if (e != cudaSuccess) return fail_cuda("low-channel igemm launch", e);
  return FDNN_OK;
}

// ---- which layout a packed filter buffer holds.  fdnn_conv2d_pack_weight notes it per buffer address so
// that fdnn_conv2d_fwd can refuse a buffer that was packed for another plan (another descriptor, or a y
// whose alignment selects a different path) instead of reading it with the wrong geometry.
struct PackedLayout {
  int kind;            // 1: [K,R,S,Cpad] (x2 planes for f32), 2 / 4: low-channel quads (4 / 3 stored channels), 3: pixel-grouped
  int a, b;            // kind 1: c_pad, dtype; kind 2: stride_w, left shift; kind 3: pixel group, stride_w
  int k, c, r, s;
  bool operator==(const PackedLayout& o) const {
    return kind == o.kind && a == o.a && b == o.b && k == o.k && c == o.c && r == o.r && s == o.s;
  }
};

PackedLayout packed_layout_of(const fdnn_conv_desc& d, const fdnn_conv_plan& plan) {
  PackedLayout l = {1, plan.c_padded, d.dtype, d.k, d.c, d.r, d.s};
  if (plan.pixel_group > 1) {
    l.kind = 3; l.a = plan.pixel_group; l.b = d.stride_w;
  } else if (plan.low_channel == 2) {
    l.kind = 4; l.a = d.stride_w; l.b = round_up(3 * d.pad_left, 8) - 3 * d.pad_left;
  } else if (plan.low_channel) {
    l.kind = 2; l.a = d.stride_w; l.b = round_up(d.pad_left, 2) - d.pad_left;
  }
  return l;
}

const char* packed_layout_name(int kind) {
  return kind == 2   ? "low-channel quad layout (4 stored channels)"
         : kind == 4 ? "low-channel quad layout (3 stored channels)"
         : kind == 3 ? "pixel-grouped layout"
                     : "[K,R,S,Cpad] layout";
}

struct PackedRecord {
  const void* ptr;
  int dev;
  PackedLayout layout;
};
constexpr int kPackedRecords = 512;
std::mutex g_packed_mutex;
PackedRecord g_packed[kPackedRecords];
unsigned g_packed_next = 0;

void remember_packed(const void* ptr, int dev, const PackedLayout& layout) {
  std::lock_guard<std::mutex> lock(g_packed_mutex);
  for (int i = 0; i < kPackedRecords; ++i) {
    if (g_packed[i].ptr == ptr && g_packed[i].dev == dev) {
      g_packed[i].layout = layout;
      return;
    }
  }
  g_packed[g_packed_next % kPackedRecords] = {ptr, dev, layout};
  ++g_packed_next;
}

bool find_packed(const void* ptr, int dev, PackedLayout* out) {
  std::lock_guard<std::mutex> lock(g_packed_mutex);
  for (int i = 0; i < kPackedRecords; ++i) {
    if (g_packed[i].ptr == ptr && g_packed[i].dev == dev) {
      *out = g_packed[i].layout;
      return true;
    }
  }
  return false;
}

// The first record that contradicts `want` among `count` buffers of `stride` bytes laid one after another from `ptr` (the
// packed filters of a layer's groups); false if none does.
bool find_other_layout(const void* ptr, long long stride, int count, int dev, const PackedLayout& want, PackedLayout* have) {
  const uintptr_t base = reinterpret_cast<uintptr_t>(ptr);
  std::lock_guard<std::mutex> lock(g_packed_mutex);
  for (int i = 0; i < kPackedRecords; ++i) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(g_packed[i].ptr);
    if (at < base || g_packed[i].dev != dev || (at - base) % uintptr_t(stride) != 0 || (at - base) / uintptr_t(stride) >= uintptr_t(count))
      continue;
    if (!(g_packed[i].layout == want)) {
      *have = g_packed[i].layout;
      return true;
    }
  }
  return false;
}

int fail_layout(const PackedLayout& have, const PackedLayout& want) {
  char buf[320];
  std::snprintf(buf, sizeof buf,
                "the packed filter holds the %s of a %dx%dx%dx%d filter, this call reads the %s of a "
                "%dx%dx%dx%d filter (other descriptor, or a y whose 16-byte alignment differs from the one "
                "given to fdnn_conv2d_pack_weight): pack again for this call",
                packed_layout_name(have.kind), have.k, have.c, have.r, have.s, packed_layout_name(want.kind),
                want.k, want.c, want.r, want.s);
  return fail(FDNN_BAD_PARAM, buf);
}

int current_device_or_minus1() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return dev;
}

}  // namespace
}  // namespace fdnn

using namespace fdnn;

extern "C" {

int fdnn_abi_version(void) { return FDNN_ABI_VERSION; }

const char* fdnn_status_string(int status) {
  switch (status) {
    case FDNN_OK: return "ok";
    case FDNN_BAD_PARAM: return "bad parameter";
    case FDNN_NOT_SUPPORTED: return "not supported";
    case FDNN_ARCH_MISMATCH: return "device is not sm_100";
    case FDNN_WORKSPACE_TOO_SMALL: return "workspace too small";
    case FDNN_CUDA_ERROR: return "CUDA error";
    case FDNN_DEVICE_TIMEOUT: return "a bounded device-side wait ran out";
    default: return "unknown status";
  }
}

const char* fdnn_last_error(void) { return g_last_error.c_str(); }

int fdnn_conv2d_query(const fdnn_conv_desc* desc, const void* x, const void* w, const void* y,
                      fdnn_conv_plan* plan) {
  return make_plan(desc, x, w, y, plan);
}

int fdnn_conv2d_main_kernel(const fdnn_conv_desc* desc, const void* x, const void* w, const void* y, fdnn_conv_kernel* kernel) {
  if (kernel == nullptr) return fail(FDNN_BAD_PARAM, "kernel is NULL");
  fdnn_conv_plan plan;
  const int st = make_plan(desc, x, w, y, &plan);
  if (st != FDNN_OK) return st;
  *kernel = {};
  if (plan.algo == FDNN_ALGO_DIRECT) return FDNN_OK;
  const RowsMode rows = rows_mode(desc, plan, y);
  FilterView f;
  // a packed filter is 16-byte aligned wherever it lies
  const bool have = desc->groups > 1 ? rows_group_filter(*desc, w, reinterpret_cast<const void*>(uintptr_t(256)), &f)
                                     : rows_layer_ok(*desc, plan);
  if (rows.tile_n != 0 && have) {
    *kernel = {FDNN_KERNEL_ROWS, 256, rows.tile_n, rows.grid};
  } else {
    *kernel = {plan.algo == FDNN_ALGO_IGEMM_PAIR ? FDNN_KERNEL_PAIR : FDNN_KERNEL_IGEMM, plan.tile_m, plan.tile_n, plan.grid};
  }
  return FDNN_OK;
}

// note: whether the buffer outlives the call and its layout is remembered
static int pack_weight(const fdnn_conv_desc* desc, const void* w, const void* y, void* packed, int64_t packed_bytes, void* stream,
                       bool note) {
  fdnn_conv_desc d;
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (validate(desc) == FDNN_OK && group_dense_ok(desc)) {
    fdnn_conv_plan whole;
    int gst = make_plan(desc, nullptr, reinterpret_cast<const void*>(uintptr_t(1)), y, &whole);
    const fdnn_conv_desc v = dense_group_desc(desc);
    fdnn_conv_plan pv;
    if (gst == FDNN_OK && whole.algo != FDNN_ALGO_DIRECT && make_plan(&v, nullptr, nullptr, y, &pv) == FDNN_OK &&
        pv.algo != FDNN_ALGO_DIRECT) {
      if (w == nullptr || packed == nullptr) return fail(FDNN_BAD_PARAM, "w and packed must not be NULL");
      if (packed_bytes < whole.packed_weight_bytes)
        return fail(FDNN_WORKSPACE_TOO_SMALL, "packed filter buffer too small");
      if ((reinterpret_cast<uintptr_t>(packed) & 15u) != 0)
        return fail(FDNN_BAD_PARAM, "the packed filter buffer of a grouped layer must be 16-byte aligned");
      cudaError_t e = launch_densify_w(desc->dtype, w, reinterpret_cast<const long long*>(desc->w_strides), desc->k,
                                       desc->c, desc->r, desc->s, desc->groups, packed,
                                       static_cast<cudaStream_t>(stream));
      if (e != cudaSuccess) return fail_cuda("densify launch", e);
      if (pv.w_packed) {
        // the dense plan wants its own layout (pixel groups, padded channels): packed behind the dense filter
        const long long off = dense_filter_bytes(desc);
        return pack_weight(&v, packed, y, static_cast<char*>(packed) + off, packed_bytes - off, stream, note);
      }
      return FDNN_OK;
    }
  }
  if (validate(desc) == FDNN_OK && group_loop_ok(desc)) {
    // one packed filter per group, back to back
    fdnn_conv_plan whole;
    int gst = make_plan(desc, nullptr, reinterpret_cast<const void*>(uintptr_t(1)), y, &whole);
    if (gst == FDNN_OK && whole.algo != FDNN_ALGO_DIRECT) {
      if (w == nullptr || packed == nullptr) return fail(FDNN_BAD_PARAM, "w and packed must not be NULL");
      if (packed_bytes < whole.packed_weight_bytes)
        return fail(FDNN_WORKSPACE_TOO_SMALL, "packed filter buffer too small");
      const fdnn_conv_desc sub = one_group_desc(desc);
      const int es = elem_size(desc->dtype);
      const long long per_group = whole.packed_weight_bytes / desc->groups;
      for (int g = 0; g < desc->groups; ++g) {
        const char* wg = static_cast<const char*>(w) + (long long)g * sub.k * desc->w_strides[0] * es;
        const char* yg = y == nullptr ? nullptr : static_cast<const char*>(y) + (long long)g * sub.k * desc->y_strides[1] * es;
        gst = pack_weight(&sub, wg, yg, static_cast<char*>(packed) + g * per_group, per_group, stream, note);
        if (gst != FDNN_OK) return gst;
      }
      return FDNN_OK;
    }
  }
  d = *desc;
  // Planned as fdnn_conv2d_fwd will plan (same algo request; an unaligned filter pointer so that the answer
  // is "packed"; the y it will write, whose alignment decides between the generic [K,R,S,Cpad] layout and
  // the low-channel / pixel-grouped ones).  Where that plan is the direct kernel, which reads the filter
  // unpacked, the layout of the single-CTA tensor-core path is written.
  if ((d.algo & 0xff) == FDNN_ALGO_DIRECT) d.algo = FDNN_ALGO_IGEMM;
  fdnn_conv_plan plan;
  int st = make_plan(&d, nullptr, reinterpret_cast<const void*>(uintptr_t(1)), y, &plan);
  if (st == FDNN_OK && plan.algo == FDNN_ALGO_DIRECT) {
    d.algo = FDNN_ALGO_IGEMM;
    st = make_plan(&d, nullptr, reinterpret_cast<const void*>(uintptr_t(1)), y, &plan);
  }
  if (st != FDNN_OK) return st;
  // a grouped filter [K, C / groups, R, S] is packed group by group or made dense above, never as one of C channels
  if (d.groups > 1 && d.algo != desc->algo) return pack_weight(&d, w, y, packed, packed_bytes, stream, note);
  if (d.groups > 1) return fail(FDNN_NOT_SUPPORTED, "no packed layout for this grouped filter");
  if (w == nullptr || packed == nullptr) return fail(FDNN_BAD_PARAM, "w and packed must not be NULL");
  if (packed_bytes < plan.packed_weight_bytes)
    return fail(FDNN_WORKSPACE_TOO_SMALL, "packed filter buffer too small");
  cudaError_t e;
  const char* what = "pack_weight launch";
  if (plan.pixel_group > 1) {
    e = launch_pack_w_grouped(d.dtype, w, reinterpret_cast<const long long*>(d.w_strides), d.k, d.c, d.r, d.s,
                              d.stride_w, plan.pixel_group, plan.c_padded, packed,
                              static_cast<cudaStream_t>(stream));
  } else if (plan.low_channel == 2) {
    const int shift_elems = round_up(3 * d.pad_left, 8) - 3 * d.pad_left;
    e = launch_pack_w_lowc(d.dtype, w, reinterpret_cast<const long long*>(d.w_strides), d.k, d.c, d.r, d.s,
                           d.stride_w, 3, shift_elems, packed, static_cast<cudaStream_t>(stream));
  } else if (plan.low_channel) {
    const int shift = round_up(d.pad_left, 2) - d.pad_left;
    e = launch_pack_w_lowc(d.dtype, w, reinterpret_cast<const long long*>(d.w_strides), d.k, d.c, d.r, d.s,
                           d.stride_w, 4, 4 * shift, packed, static_cast<cudaStream_t>(stream));
  } else {
    const long long plane = (long long)d.k * d.r * d.s * plan.c_padded;
    e = launch_pack_w(d.dtype, w, reinterpret_cast<const long long*>(d.w_strides), d.k, d.c, d.r, d.s,
                      plan.c_padded, packed, plane, static_cast<cudaStream_t>(stream));
  }
  if (e != cudaSuccess) return fail_cuda(what, e);
  if (note) remember_packed(packed, current_device_or_minus1(), packed_layout_of(d, plan));
  return FDNN_OK;
}

int fdnn_conv2d_pack_weight(const fdnn_conv_desc* desc, const void* w, const void* y, void* packed,
                            int64_t packed_bytes, void* stream) {
  return pack_weight(desc, w, y, packed, packed_bytes, stream, true);
}

static int fwd_impl(const fdnn_conv_desc* desc, const void* x, const void* w, const void* w_packed,
                    const void* bias, const void* scale, const void* residual, int activation, void* y,
                    void* workspace, int64_t workspace_bytes, void* stream_v, bool allow_group, int k_real,
                    void* sk_scratch = nullptr, int64_t sk_bytes = 0, const GroupBatch* batch = nullptr,
                    FilterPack* pack = nullptr);
static int pack_filter(int dtype, FilterPack* f, cudaStream_t stream);

int fdnn_conv2d_fwd(const fdnn_conv_desc* desc, const void* x, const void* w, const void* w_packed,
                    const void* bias, const void* scale, int activation, void* y, void* workspace,
                    int64_t workspace_bytes, void* stream_v) {
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  return fwd_impl(desc, x, w, w_packed, bias, scale, nullptr, activation, y, workspace, workspace_bytes, stream_v,
                  true, desc->k);
}

int fdnn_conv2d_fwd_residual(const fdnn_conv_desc* desc, const void* x, const void* w, const void* w_packed,
                             const void* bias, const void* scale, const void* residual, int activation, void* y,
                             void* workspace, int64_t workspace_bytes, void* stream_v) {
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15u) != (reinterpret_cast<uintptr_t>(y) & 15u))
    return fail(FDNN_NOT_SUPPORTED, "the residual must have y's alignment modulo 16 bytes");
  return fwd_impl(desc, x, w, w_packed, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v,
                  true, desc->k);
}

int fdnn_conv2d_fwd_ex(const fdnn_conv_desc* desc, const void* x, const void* w, const void* w_packed,
                       const void* bias, const void* scale, const void* residual, int activation, void* y,
                       void* workspace, int64_t workspace_bytes, void* streamk_scratch, int64_t streamk_bytes,
                       void* stream_v) {
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15u) != (reinterpret_cast<uintptr_t>(y) & 15u))
    return fail(FDNN_NOT_SUPPORTED, "the residual must have y's alignment modulo 16 bytes");
  if (streamk_scratch != nullptr && (reinterpret_cast<uintptr_t>(streamk_scratch) & 255u) != 0)
    return fail(FDNN_BAD_PARAM, "the reduction-splitting scratch must be 256-byte aligned");
  return fwd_impl(desc, x, w, w_packed, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v,
                  true, desc->k, streamk_scratch, streamk_bytes);
}

int fdnn_conv2d_fwd_unpacked(const fdnn_conv_desc* desc, const void* x, const void* w, void* packed, int64_t packed_bytes,
                             const void* bias, const void* scale, const void* residual, int activation, void* y,
                             void* workspace, int64_t workspace_bytes, void* stream_v) {
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (residual != nullptr && (reinterpret_cast<uintptr_t>(residual) & 15u) != (reinterpret_cast<uintptr_t>(y) & 15u))
    return fail(FDNN_NOT_SUPPORTED, "the residual must have y's alignment modulo 16 bytes");
  fdnn_conv_plan plan;
  int st = make_plan(desc, x, w, y, &plan);
  if (st != FDNN_OK) return st;
  if (plan.algo == FDNN_ALGO_DIRECT || !plan.w_packed)
    return fwd_impl(desc, x, w, nullptr, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v, true, desc->k);
  if (w == nullptr || packed == nullptr) return fail(FDNN_BAD_PARAM, "w and packed must not be NULL");
  if (packed_bytes < plan.packed_weight_bytes) return fail(FDNN_WORKSPACE_TOO_SMALL, "packed filter buffer too small");
  // a buffer inside the workspace is scratch like the rest of it: the workspace ends where it begins, nothing is remembered
  const uintptr_t base = reinterpret_cast<uintptr_t>(workspace), at = reinterpret_cast<uintptr_t>(packed);
  const bool kept = workspace == nullptr || at < base || at - base >= uintptr_t(workspace_bytes > 0 ? workspace_bytes : 0);
  if (!kept) workspace_bytes = int64_t(at - base);
  FilterPack pack = {w, {desc->w_strides[0], desc->w_strides[1], desc->w_strides[2], desc->w_strides[3]}, desc->k, desc->c, desc->r,
                     desc->s, plan.c_padded, packed, false};
  if (desc->groups > 1 || plan.low_channel || plan.pixel_group > 1) {
    st = pack_weight(desc, w, y, packed, packed_bytes, stream_v, kept);
    if (st != FDNN_OK) return st;
    pack.done = true;
    return fwd_impl(desc, x, w, packed, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v, true, desc->k,
                    nullptr, 0, nullptr, kept ? nullptr : &pack);
  }
  st = fwd_impl(desc, x, w, packed, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v, true, desc->k,
                nullptr, 0, nullptr, &pack);
  // a small layer that ran without it (no scratch, or few channels and a residual) has it packed all the same, for later calls
  if (!kept) return st;
  if (st == FDNN_OK && aligned16(packed)) st = pack_filter(desc->dtype, &pack, static_cast<cudaStream_t>(stream_v));
  if (pack.done) remember_packed(packed, current_device_or_minus1(), packed_layout_of(*desc, plan));
  return st;
}

// One-time set-up of the current device for kernels that use tensor maps and bounded waits.
static int prepare_device(int* device) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return fail_cuda("cudaGetDevice", e);
  if (dev < 0 || dev >= 64) return fail(FDNN_BAD_PARAM, "device ordinal out of range");
  std::call_once(g_prepare_once[dev], [dev]() {
    int major = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    g_prepare_result[dev] = (major == 10) ? igemm_prepare_device() : cudaErrorNoKernelImageForDevice;
    if (g_prepare_result[dev] == cudaSuccess) g_prepare_result[dev] = igemm_pair_prepare_device();
    if (g_prepare_result[dev] == cudaSuccess) g_prepare_result[dev] = rows_prepare_device();
    g_status_ptr[dev] = device_status_word();
  });
  if (g_prepare_result[dev] == cudaErrorNoKernelImageForDevice)
    return fail(FDNN_ARCH_MISMATCH, "the implicit-GEMM kernels are built for sm_100a only");
  if (g_prepare_result[dev] != cudaSuccess) return fail_cuda("kernel attribute setup", g_prepare_result[dev]);
  std::call_once(g_driver_once, load_driver_entry_points);
  if (!g_driver_ok) return fail(FDNN_CUDA_ERROR, "driver entry points for tensor maps not found");
  *device = dev;
  return FDNN_OK;
}

static int pack_filter(int dtype, FilterPack* f, cudaStream_t stream) {
  if (f == nullptr || f->done) return FDNN_OK;
  const cudaError_t e = launch_pack_w(dtype, f->w, f->strides, f->K, f->C, f->R, f->S, f->c_pad, f->dst,
                                      (long long)f->K * f->R * f->S * f->c_pad, stream);
  f->done = e == cudaSuccess;
  return f->done ? FDNN_OK : fail_cuda("pack_weight launch", e);
}

// Rewrites x into the scratch as dense NHWC where the plan says so, and says how the kernels see it.
struct ActivationView {
  const void* base;
  int c;                       // channels that may be read
  long long sw, sh, sn, plane; // element strides; offset of the second plane (fp32)
};
// pack: the layer's filter, packed in the same launch where that is possible, else in one before it.
static int relayout_x(const fdnn_conv_desc& d, const fdnn_conv_plan& plan, bool by_groups, const void* x, void* workspace,
                      int64_t workspace_bytes, cudaStream_t stream, ActivationView* a, FilterPack* pack) {
  const int es = elem_size(d.dtype);
  // Extent-one dimensions get a harmless aligned stride (theirs may be anything).
  a->base = x;
  a->c = by_groups ? d.c / d.groups : d.c;
  a->sw = d.w > 1 ? d.x_strides[3] : plan.c_padded;
  a->sh = d.h > 1 ? d.x_strides[2] : plan.c_padded;
  a->sn = d.n > 1 ? d.x_strides[0] : plan.c_padded;
  a->plane = 0;
  if (!plan.x_repacked) return pack_filter(d.dtype, pack, stream);
  int x_pad = by_groups ? d.c : padded_x_channels(&d);   // groups side by side, 16-byte multiples each
  if (!by_groups && (long long)(d.dtype == FDNN_F32 ? 2 : 1) * d.n * d.h * d.w * x_pad * es > workspace_bytes)
    x_pad = round_up(d.c, 16 / es);
  a->plane = (long long)d.n * d.h * d.w * x_pad;
  cudaError_t e = launch_repack_x(d.dtype, x, reinterpret_cast<const long long*>(d.x_strides), d.n, d.c, d.h, d.w, x_pad,
                                  workspace, a->plane, stream, pack != nullptr && !pack->done ? pack : nullptr);
  if (e != cudaSuccess) return fail_cuda("repack_x launch", e);
  a->base = workspace;
  a->sw = x_pad;
  a->sh = (long long)d.w * x_pad;
  a->sn = (long long)d.h * d.w * x_pad;
  if (!by_groups) a->c = x_pad;
  return FDNN_OK;
}

static int fwd_rows(const fdnn_conv_desc& d, const fdnn_conv_plan& plan, const RowsMode& rows, int dev, const void* x,
                    const FilterView& f, FilterPack* pack, const void* bias, const void* scale, int activation, void* y,
                    void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  ActivationView a;
  fdnn_conv_desc whole = d;    // a block of channels is copied whatever groups it holds
  whole.groups = 1;
  int st = relayout_x(whole, plan, false, x, workspace, workspace_bytes, stream, &a, pack);
  if (st != FDNN_OK) return st;
  const int cg = d.c / d.groups, kg = d.k / d.groups, es = elem_size(d.dtype);
  alignas(64) CUtensorMap tmA, tmA2, tmB;
  st = encode_activation_map(&tmA, d.dtype, a.base, a.c, d.w, d.h, d.n, a.sw, a.sh, a.sn, &whole, 1, rows.pitch);
  if (st != FDNN_OK) return st;
  tmA2 = tmA;
  if (es == 4) {
    st = encode_activation_map(&tmA2, d.dtype, static_cast<const char*>(a.base) + a.plane * es, a.c, d.w, d.h, d.n, a.sw, a.sh,
                               a.sn, &whole, 1, rows.pitch);
    if (st != FDNN_OK) return st;
  }
  const bool blk = rows.blk_groups > 1;
  RowsParams p = {};
  p.M = d.n * plan.oh * rows.pitch;
  p.Kout = d.k;
  p.OH = plan.oh; p.OW = plan.ow;
  p.P = rows.pitch;
  p.stride_h = d.stride_h; p.pad_top = d.pad_top; p.pad_left = d.pad_left; p.dil_h = d.dil_h; p.dil_w = d.dil_w;
  p.R = d.r; p.S = d.s;
  p.s_pitch = f.s_pitch;
  p.halves = es == 4 ? 2 : 1;
  p.c_blocks = blk ? 1 : (d.c * es + 127) / 128;
  p.m_tiles = rows.m_tiles;
  p.n_tiles = rows.n_tiles;
  p.blk_groups = rows.blk_groups;
  p.kg = kg;
  p.blk_c_step = f.c_step;
  p.b_bytes = blk ? rows.blk_groups * (kg / 2) * cg * 2 : p.halves * (rows.tile_n / 2) * 128;
  rows_stages(&p);
  {
    // (channel, filter, tap, half): one box per group (of a block of channels) and slot
    cuuint64_t dims[4] = {cuuint64_t(f.c), cuuint64_t(d.k), cuuint64_t(d.r) * f.s_pitch, 2};
    cuuint64_t strides[3] = {cuuint64_t(f.s_k) * es, cuuint64_t(f.s_tap) * es, cuuint64_t(d.k) * d.r * f.s_pitch * f.c * es};
    cuuint32_t box[4] = {cuuint32_t(blk ? cg : 128 / es), cuuint32_t(blk ? kg / 2 : rows.tile_n / 2), cuuint32_t(p.b_taps), 2};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = memo_encode_tiled(&tmB, tm_dtype(d.dtype), es == 4 ? 4 : 3, const_cast<void*>(f.base), dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   !blk ? CU_TENSOR_MAP_SWIZZLE_128B : cg == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FDNN_CUDA_ERROR, "cuTensorMapEncodeTiled (filter rows) failed with CUresult " + std::to_string(int(r)));
  }
  p.y_sn = d.y_strides[0]; p.y_sk = d.y_strides[1]; p.y_sh = d.y_strides[2]; p.y_sw = d.y_strides[3];
  IgemmParams unit = {};
  choose_strided_store(d, plan.oh, plan.ow, y, &unit);
  p.y_unit = d.y_strides[1] == 1 && sector_aligned(d, plan.oh, plan.ow, y) ? 32 : unit.y_unit;
  p.bias = bias; p.scale = scale; p.y = y;
  p.act = activation;
  IgemmParams dbg = {};
  fill_debug_params(&dbg);
  p.wait_limit = dbg.wait_limit;
  p.skip_copies = dbg.skip_copies;
  p.status = g_status_ptr[dev];
  if (p.status == nullptr) return fail(FDNN_CUDA_ERROR, "status word address unavailable");
  alignas(64) CUtensorMap tmY = tmA;
  const long long row = y_pixel_stride(&d, plan.oh, plan.ow);
  if (row > 0 && aligned16(y)) {
    st = encode_output_map(&tmY, d.dtype, y, d.k, (long long)d.n * plan.oh * plan.ow, row);
    if (st != FDNN_OK) return st;
    p.y_rows = 1;
  }
  cudaError_t e = launch_rows(d.dtype, rows.tile_n, tmA, tmA2, tmB, tmY, p, rows.grid, stream);
  if (e != cudaSuccess) return fail_cuda("rows launch", e);
  return FDNN_OK;
}

// k_real: length of bias / scale (differs from desc->k only for the equivalent convolution of a
// pixel-grouped layer, whose GEMM column j uses entry j % k_real).  pack: this call writes w_packed itself, or has (done).
static int fwd_impl(const fdnn_conv_desc* desc, const void* x, const void* w, const void* w_packed,
                    const void* bias, const void* scale, const void* residual, int activation, void* y,
                    void* workspace, int64_t workspace_bytes, void* stream_v, bool allow_group, int k_real,
                    void* sk_scratch, int64_t sk_bytes, const GroupBatch* batch, FilterPack* pack) {
  fdnn_conv_plan plan;
  // A caller that hands over a packed filter wants it used even when w itself
  // would qualify for in-place reads; plan accordingly.
  int st = FDNN_OK;
  if (batch != nullptr) {
    plan = batch->one;   // `desc` is a run of groups of a layer, all in one launch
    plan.tile_n = batch->tile_n;
  } else {
    st = make_plan(desc, x, w_packed != nullptr ? reinterpret_cast<const void*>(uintptr_t(1)) : w, y, &plan, allow_group);
    if (st != FDNN_OK) return st;
  }
  if (activation < FDNN_ACT_NONE || activation > FDNN_ACT_GELU_TANH)
    return fail(FDNN_BAD_PARAM, "unknown activation");
  if ((desc->algo & 0xff) == FDNN_ALGO_AUTO && plan.algo != FDNN_ALGO_DIRECT && small_layer(desc, plan.flops) &&
      allow_group && batch == nullptr && w != nullptr &&
      ((plan.w_packed && w_packed == nullptr) || (plan.workspace_bytes > 0 && (workspace == nullptr || workspace_bytes < plan.workspace_bytes)) ||
       (desc->c < 8 && residual != nullptr))) {
    // a small layer whose caller brought neither packed filter nor scratch, or one that was planned as pixel windows, which
    // carry no residual (see small_on_tensor_cores)
    fdnn_conv_desc direct = *desc;
    direct.algo = FDNN_ALGO_DIRECT;
    return fwd_impl(&direct, x, w, nullptr, bias, scale, residual, activation, y, nullptr, 0, stream_v, allow_group, k_real);
  }
  const fdnn_conv_desc& d = *desc;
  if (d.n == 0 || plan.oh == 0 || plan.ow == 0) return FDNN_OK;  // empty output: nothing to launch
  if (x == nullptr || y == nullptr || (w == nullptr && w_packed == nullptr))
    return fail(FDNN_BAD_PARAM, "x, w and y must not be NULL");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

  if (batch == nullptr && d.groups > 1 && plan.algo != FDNN_ALGO_DIRECT && allow_group && residual == nullptr) {
    const RowsMode rows = rows_mode(&d, plan, y);
    FilterView f = {};
    if (rows.tile_n != 0 && rows_group_filter(d, w, w_packed, &f) && (plan.x_repacked == 0 || (workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255u) == 0 &&
        workspace_bytes >= tight_x_bytes(&d)))) {
      int dev = 0;
      st = prepare_device(&dev);
      if (st != FDNN_OK) return st;
      return fwd_rows(d, plan, rows, dev, x, f, nullptr, bias, scale, activation, y, workspace, workspace_bytes, stream);
    }
  }
  if (batch == nullptr && d.groups > 1 && plan.algo != FDNN_ALGO_DIRECT && allow_group) {
    const bool dense = group_dense_ok(&d);
    // where the filter of a group lies: in w itself, or (one launch per group) one after another in the packed buffer
    const GroupBatch own = group_batch(&d, x, w, y, plan, dense);
    const int es = elem_size(d.dtype);
    const bool from_packed = own.tile_n != 0 && (own.one.w_packed || w == nullptr);
    const long long per_group = (long long)d.n * d.h * d.w * (d.c / d.groups) * es;
    long long run = d.groups;                     // groups per launch: as many as the scratch holds relaid out
    if (own.tile_n != 0 && own.one.x_repacked) run = workspace != nullptr && per_group > 0 ? workspace_bytes / per_group : 0;
    if (run > d.groups) run = d.groups;
    if (own.tile_n != 0 && run > 1 && !(from_packed && (dense || w_packed == nullptr))) {
      // what a launch per group checks for each of them: here once, before the first relayout writes to the scratch
      if (own.one.x_repacked && (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
        return fail(FDNN_BAD_PARAM, "workspace must be 256-byte aligned");
      fdnn_conv_desc part = d;
      const long long cg = d.c / d.groups, kg = d.k / d.groups;
      const long long filter_bytes = kg * d.r * d.s * own.one.c_padded * es;
      if (from_packed && pack == nullptr) {
        PackedLayout have;
        const PackedLayout want = packed_layout_of(one_group_desc(&d), own.one);
        if (find_other_layout(w_packed, filter_bytes, d.groups, current_device_or_minus1(), want, &have))
          return fail_layout(have, want);
      }
      auto at = [es](const void* base, long long elems) -> const void* {
        return base == nullptr ? nullptr : static_cast<const char*>(base) + elems * es;
      };
      GroupBatch b = own;
      b.one.w_packed = from_packed ? 1 : 0;
      for (int g0 = 0; g0 < d.groups; g0 += int(run)) {
        part.groups = int(run < d.groups - g0 ? run : d.groups - g0);
        part.c = int(cg * part.groups);
        part.k = int(kg * part.groups);
        st = fwd_impl(&part, at(x, g0 * cg * d.x_strides[1]), at(w, g0 * kg * d.w_strides[0]),
                      from_packed ? static_cast<const char*>(w_packed) + g0 * filter_bytes : nullptr, at(bias, g0 * kg),
                      at(scale, g0 * kg), at(residual, g0 * kg * d.y_strides[1]), activation,
                      const_cast<void*>(at(y, g0 * kg * d.y_strides[1])), workspace, workspace_bytes, stream_v, false,
                      int(kg), nullptr, 0, &b);
        if (st != FDNN_OK) return st;
      }
      return FDNN_OK;
    }
  }
  if (batch == nullptr && d.groups > 1 && plan.algo != FDNN_ALGO_DIRECT && group_dense_ok(&d)) {
    // one dense convolution with the block-diagonal filter the pack step left at the front of w_packed
    if (w_packed == nullptr && !plan.w_packed)   // planned as one launch on w; only the scratch can have kept it from that
      return fail(FDNN_WORKSPACE_TOO_SMALL, "workspace smaller than plan.workspace_bytes");
    if (w_packed == nullptr)
      return fail(FDNN_BAD_PARAM, "a grouped layer on the dense route needs its packed filter; w_packed is NULL");
    const fdnn_conv_desc v = dense_group_desc(&d);
    fdnn_conv_plan pv;
    st = make_plan(&v, x, nullptr, y, &pv, allow_group);
    if (st != FDNN_OK) return st;
    const void* inner = pv.w_packed ? static_cast<const char*>(w_packed) + dense_filter_bytes(&d) : nullptr;
    return fwd_impl(&v, x, w_packed, inner, bias, scale, residual, activation, y, workspace, workspace_bytes, stream_v,
                    allow_group, k_real, sk_scratch, sk_bytes, nullptr, pack);
  }
  if (batch == nullptr && d.groups > 1 && plan.algo != FDNN_ALGO_DIRECT) {
    // one launch per group on views of the tensors (see group_loop_ok); the groups share the scratch, which the
    // stream's order makes safe
    const fdnn_conv_desc sub = one_group_desc(&d);
    const int es = elem_size(d.dtype);
    const long long per_group = plan.packed_weight_bytes / d.groups;
    auto at = [es](const void* base, long long elems) -> const void* {
      return base == nullptr ? nullptr : static_cast<const char*>(base) + elems * es;
    };
    for (int g = 0; g < d.groups; ++g) {
      const long long k0 = (long long)g * sub.k;
      st = fwd_impl(&sub, at(x, (long long)g * sub.c * d.x_strides[1]), at(w, k0 * d.w_strides[0]),
                    w_packed == nullptr ? nullptr : static_cast<const char*>(w_packed) + g * per_group,
                    at(bias, k0), at(scale, k0), at(residual, k0 * d.y_strides[1]), activation,
                    const_cast<void*>(at(y, k0 * d.y_strides[1])), workspace, workspace_bytes, stream_v, allow_group,
                    sub.k, sk_scratch, sk_bytes, nullptr, pack);
      if (st != FDNN_OK) return st;
    }
    return FDNN_OK;
  }

  if (plan.algo == FDNN_ALGO_DIRECT) {
    if (w == nullptr) return fail(FDNN_BAD_PARAM, "the direct path reads the unpacked filter; w is NULL");
    DirectParams p;
    p.N = d.n; p.C = d.c; p.H = d.h; p.W = d.w; p.K = d.k; p.R = d.r; p.S = d.s;
    p.OH = plan.oh; p.OW = plan.ow;
    p.stride_h = d.stride_h; p.stride_w = d.stride_w; p.pad_top = d.pad_top; p.pad_left = d.pad_left;
    p.dil_h = d.dil_h; p.dil_w = d.dil_w; p.groups = d.groups;
    for (int i = 0; i < 4; ++i) {
      p.x_s[i] = d.x_strides[i];
      p.w_s[i] = d.w_strides[i];
      p.y_s[i] = d.y_strides[i];
    }
    p.x = x; p.w = w; p.bias = bias; p.scale = scale; p.residual = residual; p.y = y;
    p.act = activation;
    int dw = (d.algo & 0xff) == FDNN_ALGO_AUTO ? depthwise_kind(d.dtype, p) : 0;  // a forced "direct" stays direct
    if (dw == 6 || dw == 9) {
      int dev = 0;
      if (prepare_device(&dev) == FDNN_OK && g_status_ptr[dev] != nullptr) {
        const long long set = g_wait_limit.load(std::memory_order_relaxed), limit = set > 0 ? set : default_wait_limit_cycles();
        cudaError_t e = dw == 9 ? launch_depthwise_ring(d.dtype, p, g_status_ptr[dev], limit, stream)
                                : launch_depthwise_tma(d.dtype, p, g_status_ptr[dev], limit, stream);
        if (e == cudaSuccess) return FDNN_OK;
        if (e != cudaErrorInvalidValue) return fail_cuda("depthwise launch", e);
        cudaGetLastError();
      }
      dw = dw == 9 ? 2 : 1;   // no tensor map over this x: the kernel that reads it with plain loads
    }
    cudaError_t e = dw != 0 ? launch_depthwise(d.dtype, p, dw, stream) : launch_direct(d.dtype, p, stream);
    if (e != cudaSuccess) return fail_cuda("direct conv launch", e);
    return FDNN_OK;
  }

  // ---- tensor-core path
  int dev = 0;
  st = prepare_device(&dev);
  if (st != FDNN_OK) return st;
  cudaError_t e = cudaSuccess;

  if (plan.w_packed && w_packed == nullptr)
    return fail(FDNN_BAD_PARAM, "this problem needs a packed filter (fdnn_conv2d_pack_weight); w_packed is NULL");
  if (plan.workspace_bytes > 0 && batch == nullptr) {
    const long long least = plan.x_repacked && !plan.low_channel ? tight_x_bytes(&d) : plan.workspace_bytes;
    if (workspace == nullptr || workspace_bytes < (least < plan.workspace_bytes ? least : plan.workspace_bytes))
      return fail(FDNN_WORKSPACE_TOO_SMALL, "workspace smaller than plan.workspace_bytes");
    if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
      return fail(FDNN_BAD_PARAM, "workspace must be 256-byte aligned");
  }
  if (plan.w_packed && (reinterpret_cast<uintptr_t>(w_packed) & 15u) != 0)
    return fail(FDNN_BAD_PARAM, "packed filter must be 16-byte aligned");
  if (plan.w_packed && allow_group && pack == nullptr) {
    // the buffer must hold the layout this plan reads (allow_group is false only for the inner call of
    // a pixel-grouped layer, whose buffer was checked by the outer one; with `pack` this call writes it)
    PackedLayout have;
    const PackedLayout want = packed_layout_of(d, plan);
    if (find_packed(w_packed, dev, &have) && !(have == want)) return fail_layout(have, want);
  }

  if (batch == nullptr && residual == nullptr && allow_group && k_real == d.k && rows_layer_ok(d, plan)) {
    const RowsMode rows = rows_mode(&d, plan, y);
    if (rows.tile_n != 0) {
      const int c_pad = plan.c_padded;
      FilterView f = {w, d.c, d.s, 0, d.s > 1 ? d.w_strides[3] : d.w_strides[2], d.k > 1 ? d.w_strides[0] : c_pad};
      if (plan.w_packed) {
        // a filter packed for Q grouped pixels starts with the filter of the first one, its taps in front of each row
        const int s_pitch = plan.pixel_group > 1 ? d.s + (plan.pixel_group - 1) * d.stride_w : d.s;
        f = {w_packed, c_pad, s_pitch, 0, c_pad, (long long)d.r * s_pitch * c_pad};
      }
      return fwd_rows(d, plan, rows, dev, x, f, pack, bias, scale, activation, y, workspace, workspace_bytes, stream);
    }
  }
  if (plan.pixel_group > 1) {
    // run the equivalent convolution; its filter is the packed buffer, consumed in place
    const fdnn_conv_desc v = grouped_desc(&d, plan.pixel_group, plan.oh, plan.ow);
    return fwd_impl(&v, x, w_packed, nullptr, bias, scale, residual, activation, y, workspace, workspace_bytes,
                    stream_v, false, d.k, sk_scratch, sk_bytes);
  }
  if (plan.low_channel && residual != nullptr)
    return fail(FDNN_NOT_SUPPORTED, "the low-channel path takes no residual; add it in a separate step");
  if (plan.low_channel) return fwd_low_channel(d, plan, dev, x, w_packed, bias, scale, activation, y, workspace, stream);

  const int es = elem_size(d.dtype);
  const int c_pad = plan.c_padded;
  const long long any_stride = c_pad;
  const int groups = batch != nullptr ? d.groups : 1;
  const int k_group = d.k / groups;
  PixelWindows windows = {};
  if (plan.algo == FDNN_ALGO_IGEMM && plan.x_repacked && plan.w_packed && residual == nullptr && batch == nullptr)
    windows = pixel_windows(&d, plan.oh, plan.ow);
  if (windows.scratch > workspace_bytes) windows.ok = false;
  ActivationView a = {};
  if (windows.ok) {
    st = pack_filter(d.dtype, pack, stream);
    if (st != FDNN_OK) return st;
    e = launch_repack_x_windows(x, reinterpret_cast<const long long*>(d.x_strides), d.n, d.c, d.h, d.w, d.pad_left,
                                windows.w_pad, workspace, stream);
    if (e != cudaSuccess) return fail_cuda("repack_x launch", e);
    a.base = workspace;
  } else {
    st = relayout_x(d, plan, batch != nullptr, x, workspace, workspace_bytes, stream, &a, pack);
    if (st != FDNN_OK) return st;
  }
  const bool b_mn = !plan.w_packed && filter_mn_major(&d, w);
  const void* b_base = w;
  long long b_stap = d.s > 1 ? d.w_strides[3] : (d.r > 1 ? d.w_strides[2] : any_stride);
  long long b_sk = d.k > 1 ? d.w_strides[0] : any_stride;
  int b_c = d.c / groups;
  long long b_plane = 0;
  if (plan.w_packed) {
    b_base = w_packed;
    b_stap = c_pad;
    b_sk = (long long)d.r * d.s * c_pad;
    b_c = c_pad;
    b_plane = (long long)d.k * d.r * d.s * c_pad;
  }

  alignas(64) CUtensorMap tmA, tmA2, tmB, tmB2;
  if (windows.ok) {
    cuuint64_t dims[4] = {cuuint64_t(d.s) * 8, cuuint64_t(plan.ow), cuuint64_t(d.h), cuuint64_t(d.n)};
    cuuint64_t strides[3] = {cuuint64_t(d.stride_w) * 16, cuuint64_t(windows.w_pad) * 16, cuuint64_t(d.h) * windows.w_pad * 16};
    cuuint32_t box[4] = {64, cuuint32_t(plan.ow), cuuint32_t(windows.ohs * d.stride_h), 1};
    cuuint32_t estr[4] = {1, 1, cuuint32_t(d.stride_h), 1};
    st = encode_tiled(&tmA, d.dtype, a.base, 4, dims, strides, box, estr, "pixel windows");
  } else {
    st = encode_activation_map(&tmA, d.dtype, a.base, a.c, d.w, d.h, d.n, a.sw, a.sh, a.sn, &d, groups);
  }
  if (st != FDNN_OK) return st;
  const int b_box_rows = plan.algo == FDNN_ALGO_IGEMM_PAIR ? 128 : plan.tile_n;  // each CTA of a pair stages half
  if (b_mn) {
    cuuint64_t dims[3] = {cuuint64_t(d.k), cuuint64_t(d.c), 1};
    cuuint64_t strides[2] = {cuuint64_t(d.w_strides[1]) * es, cuuint64_t(d.w_strides[1]) * es * cuuint64_t(d.c)};
    cuuint32_t box[3] = {64, 64, 1};   // kMnBoxElems filters x one reduction step
    cuuint32_t estr[3] = {1, 1, 1};
    st = encode_tiled(&tmB, d.dtype, b_base, 3, dims, strides, box, estr, "filter, K contiguous");
  } else if (windows.ok) {
    st = encode_filter_map(&tmB, d.dtype, b_base, d.s * 8, d.r, d.k, (long long)d.s * 8, b_sk, b_box_rows);
  } else {
    st = encode_filter_map(&tmB, d.dtype, b_base, b_c, d.r * d.s, d.k, b_stap, b_sk, b_box_rows);
  }
  if (st != FDNN_OK) return st;
  if (d.dtype == FDNN_F32) {
    st = encode_activation_map(&tmA2, d.dtype, static_cast<const char*>(a.base) + a.plane * es, a.c, d.w,
                               d.h, d.n, a.sw, a.sh, a.sn, &d);
    if (st != FDNN_OK) return st;
    st = encode_filter_map(&tmB2, d.dtype, static_cast<const char*>(b_base) + b_plane * es, b_c,
                           d.r * d.s, d.k, b_stap, b_sk, plan.tile_n);
    if (st != FDNN_OK) return st;
  } else {
    tmA2 = tmA;
    tmB2 = tmB;
  }

  IgemmParams p = {};
  p.M = d.n * plan.oh * plan.ow;
  p.Kout = k_group;
  p.k_real = k_real;
  p.groups = groups;
  p.k16_per_step = 4;
  p.lowc = 0;
  p.rows_per_tile = 128;
  p.OH = plan.oh; p.OW = plan.ow;
  p.stride_h = d.stride_h; p.stride_w = d.stride_w; p.pad_top = d.pad_top; p.pad_left = d.pad_left;
  p.dil_h = d.dil_h; p.dil_w = d.dil_w;
  p.R = d.r; p.S = d.s;
  p.c_blocks = (c_pad + plan.tile_k - 1) / plan.tile_k;
  p.m_tiles = (p.M + 127) / 128;
  if (windows.ok) {
    p.lowc = 1;
    p.S = 1;
    p.c_blocks = 1;
    p.rows_per_tile = windows.rows_per_tile;
    p.tiles_per_image = windows.tiles_per_image;
    p.ohs = windows.ohs;
    p.a_tx_bytes = windows.rows_per_tile * 128;
    p.m_tiles = d.n * windows.tiles_per_image;
  }
  p.group_n_tiles = (k_group + plan.tile_n - 1) / plan.tile_n;
  p.n_tiles = groups * p.group_n_tiles;
  if (batch != nullptr) {
    const long long tiles = (long long)p.m_tiles * p.n_tiles;
    plan.grid = int(tiles < sm_count() ? tiles : sm_count());
  }
  p.y_sn = d.y_strides[0]; p.y_sk = d.y_strides[1]; p.y_sh = d.y_strides[2]; p.y_sw = d.y_strides[3];
  p.bias = bias; p.scale = scale; p.y = y;
  p.residual = residual;
  p.act = activation;
  p.b_mn = b_mn ? 1 : 0;
  const bool out_f32 = (d.algo & FDNN_ALGO_FLAG_OUT_F32) != 0;
  if (out_f32 && residual != nullptr) return fail(FDNN_NOT_SUPPORTED, "no residual with a float32 output from 16-bit operands");
  p.out_f32 = out_f32 ? 1 : 0;
  p.vec_store = (out_f32 && d.y_strides[1] == 1 && d.y_strides[0] % 4 == 0 && d.y_strides[2] % 4 == 0 &&
                 d.y_strides[3] % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0)
                    ? 1
                    : 0;
  // y as one [M, K] matrix: consecutive output pixels are row_stride apart
  alignas(64) CUtensorMap tmY;
  p.tma_store = 0;
  {
    const long long row = out_f32 ? 0 : y_pixel_stride(&d, plan.oh, plan.ow);
    if (row > 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0) {
      if (windows.ok) {
        // (channel, pixel of the image, image), and the box of a tile's last rows in the unused slot of the fp32 map
        cuuint64_t dims[3] = {cuuint64_t(d.k), cuuint64_t(plan.oh) * plan.ow, cuuint64_t(d.n)};
        cuuint64_t strides[2] = {cuuint64_t(row) * es, cuuint64_t(row) * es * plan.oh * plan.ow};
        cuuint32_t estr[3] = {1, 1, 1};
        cuuint32_t box[3] = {64, 32, 1};
        st = encode_tiled(&tmY, d.dtype, y, 3, dims, strides, box, estr, "window output");
        if (st != FDNN_OK) return st;
        const int tail = windows.rows_per_tile % 32;
        box[1] = cuuint32_t(tail > 0 ? tail : 32);
        st = encode_tiled(&tmA2, d.dtype, y, 3, dims, strides, box, estr, "window output tail");
      } else {
        st = encode_output_map(&tmY, d.dtype, y, k_group, p.M, row, groups);
      }
      if (st != FDNN_OK) return st;
      p.tma_store = 1;
      p.y_row = row;
    } else {
      tmY = tmA;
    }
  }
  if (!p.tma_store && !out_f32) choose_strided_store(d, plan.oh, plan.ow, y, &p);
  alignas(64) CUtensorMap tmR = tmY;
  alignas(64) CUtensorMap tmRbox = tmY;
  if (residual != nullptr && p.tma_store) {
    const int box_cols = plan.algo == FDNN_ALGO_IGEMM_PAIR ? 256 : plan.tile_n;
    st = encode_residual_map(&tmR, d.dtype, residual, k_group, p.M, p.y_row, box_cols, groups);
    if (st != FDNN_OK) return st;
    // the same tensor once more, boxed and swizzled like y: the epilogue warps copy from it
    st = encode_output_map(&tmRbox, d.dtype, const_cast<void*>(residual), k_group, p.M, p.y_row, groups);
    if (st != FDNN_OK) return st;
  }
  p.prof = prof_buffer_of_current_device();
  fill_debug_params(&p);
  p.status = g_status_ptr[dev];
  if (p.status == nullptr) return fail(FDNN_CUDA_ERROR, "status word address unavailable");
  if (plan.algo == FDNN_ALGO_IGEMM_PAIR) {
    if (!p.tma_store) return fail(FDNN_NOT_SUPPORTED, "the CTA-pair kernel needs a dense channels-last output");
    p.b_resident = (d.k <= 256 && !b_mn && d.r * d.s * p.c_blocks <= igemm_pair_max_resident_steps()) ? 1 : 0;
    // reduction splitting when the caller brought the scratch for it
    if (plan.stream_k && !p.b_resident && sk_scratch != nullptr && sk_bytes >= plan.streamk_bytes &&
        (reinterpret_cast<uintptr_t>(sk_scratch) & 255u) == 0) {
      p.stream_k = 1;
      p.sk_min_frag = kStreamKMinFrag;
      p.sk_flags = static_cast<uint32_t*>(sk_scratch);
      p.sk_slots = reinterpret_cast<float*>(static_cast<char*>(sk_scratch) + FDNN_STREAMK_FLAG_BYTES);
    }
    e = launch_igemm_pair(d.dtype, tmA, tmB, tmY, tmY, tmR, tmRbox, p, plan.grid, stream);
  } else {
    e = launch_igemm(d.dtype, plan.tile_n, tmA, tmA2, tmB, tmB2, tmY, tmR, tmRbox, p, plan.grid, stream);
  }
  if (e != cudaSuccess) return fail_cuda("igemm launch", e);
  return FDNN_OK;
}

int fdnn_debug_set_profile_buffer(void* device_buffer_16_int64) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(FDNN_CUDA_ERROR, "no current device");
  g_prof_buffer[dev].store(static_cast<long long*>(device_buffer_16_int64), std::memory_order_relaxed);
  return FDNN_OK;
}

int fdnn_debug_set_wait_limit(int64_t wait_limit_cycles, int skip_copies) {
  if (wait_limit_cycles < 0) return fail(FDNN_BAD_PARAM, "wait limit must not be negative");
  g_wait_limit.store(wait_limit_cycles, std::memory_order_relaxed);
  g_skip_copies.store(skip_copies != 0 ? 1 : 0, std::memory_order_relaxed);
  return FDNN_OK;
}

int fdnn_debug_tensor_map_counters(int64_t* reused, int64_t* encoded) {
  if (reused != nullptr) *reused = g_map_hits.load(std::memory_order_relaxed);
  if (encoded != nullptr) *encoded = g_map_misses.load(std::memory_order_relaxed);
  return FDNN_OK;
}

static int pool_params(const fdnn_pool_desc* d, const void* x, void* y, PoolParams* p, bool max_pool) {
  if (d == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  if (d->dtype < FDNN_F16 || d->dtype > FDNN_F64) return fail(FDNN_BAD_PARAM, "unknown dtype");
  if (d->n < 0 || d->c < 0 || d->h < 0 || d->w < 0 || d->oh < 0 || d->ow < 0)
    return fail(FDNN_BAD_PARAM, "negative extent");
  if (max_pool) {
    if (d->kernel_h <= 0 || d->kernel_w <= 0 || d->stride_h <= 0 || d->stride_w <= 0 || d->dil_h <= 0 ||
        d->dil_w <= 0 || d->pad_h < 0 || d->pad_w < 0)
      return fail(FDNN_BAD_PARAM, "kernel, stride and dilation must be positive, padding non-negative");
    if (2 * d->pad_h > d->kernel_h || 2 * d->pad_w > d->kernel_w)
      return fail(FDNN_BAD_PARAM, "pad should be at most half of effective kernel size");
  }
  const long long total = (long long)d->n * d->c * d->oh * d->ow;
  if (total > 0 && (x == nullptr || y == nullptr)) return fail(FDNN_BAD_PARAM, "x and y must not be NULL");
  p->N = d->n; p->C = d->c; p->H = d->h; p->W = d->w; p->OH = d->oh; p->OW = d->ow;
  p->kh = d->kernel_h; p->kw = d->kernel_w; p->sh = d->stride_h; p->sw = d->stride_w;
  p->ph = d->pad_h; p->pw = d->pad_w; p->dh = d->dil_h; p->dw = d->dil_w;
  for (int i = 0; i < 4; ++i) {
    p->x_s[i] = d->x_strides[i];
    p->y_s[i] = d->y_strides[i];
  }
  p->x = x; p->y = y; p->idx = nullptr;
  return FDNN_OK;
}

int fdnn_max_pool2d_fwd(const fdnn_pool_desc* desc, const void* x, void* y, int64_t* indices, void* stream) {
  PoolParams p;
  int st = pool_params(desc, x, y, &p, true);
  if (st != FDNN_OK) return st;
  p.idx = reinterpret_cast<long long*>(indices);
  cudaError_t e = launch_max_pool2d(desc->dtype, p, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail_cuda("max_pool2d launch", e);
  return FDNN_OK;
}

int fdnn_adaptive_avg_pool2d_fwd(const fdnn_pool_desc* desc, const void* x, void* y, void* stream) {
  PoolParams p;
  int st = pool_params(desc, x, y, &p, false);
  if (st != FDNN_OK) return st;
  if ((long long)desc->n * desc->c * desc->oh * desc->ow > 0 && (desc->h == 0 || desc->w == 0))
    return fail(FDNN_BAD_PARAM, "adaptive pooling needs a non-empty input plane");
  cudaError_t e = launch_adaptive_avg_pool2d(desc->dtype, p, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail_cuda("adaptive_avg_pool2d launch", e);
  return FDNN_OK;
}

int fdnn_device_status(uint32_t* word) {
  uint32_t v = 0;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return fail_cuda("cudaDeviceSynchronize", e);
  e = cudaMemcpyFromSymbol(&v, g_status_word, sizeof v);
  if (e != cudaSuccess) return fail_cuda("read status word", e);
  if (word != nullptr) *word = v;
  if (v != 0) {
    const uint32_t zero = 0;
    cudaMemcpyToSymbol(g_status_word, &zero, sizeof zero);
    return fail(FDNN_DEVICE_TIMEOUT, "a kernel gave up a bounded wait (incident " + std::to_string(v) + ")");
  }
  return FDNN_OK;
}

// ------------------------------------------------------------- host buffers
static long long span_elems(const int64_t s[4], long long a, long long b, long long c, long long e) {
  if (a == 0 || b == 0 || c == 0 || e == 0) return 0;
  return (a - 1) * s[0] + (b - 1) * s[1] + (c - 1) * s[2] + (e - 1) * s[3] + 1;
}
static long long align256(long long v) { return (v + 255) / 256 * 256; }

struct HostArena {
  long long x, w, bias, scale, y, packed, ws, total;
  long long x_bytes, w_bytes, y_bytes, k_bytes;
  fdnn_conv_plan plan;
};

static int host_arena_layout(const fdnn_conv_desc* d, HostArena* a) {
  fdnn_conv_desc q = *d;
  // Device copies start 256-byte aligned, so alignment never forces a repack.
  int st = make_plan(&q, nullptr, reinterpret_cast<const void*>(uintptr_t(256)), nullptr, &a->plan);
  if (st != FDNN_OK) return st;
  const int es = elem_size(d->dtype);
  a->x_bytes = span_elems(d->x_strides, d->n, d->c, d->h, d->w) * es;
  a->w_bytes = span_elems(d->w_strides, d->k, d->c / d->groups, d->r, d->s) * es;
  a->y_bytes = span_elems(d->y_strides, d->n, d->k, a->plan.oh, a->plan.ow) * es;
  a->k_bytes = (long long)d->k * es;
  long long off = 0;
  a->x = off; off += align256(a->x_bytes);
  a->w = off; off += align256(a->w_bytes);
  a->bias = off; off += align256(a->k_bytes);
  a->scale = off; off += align256(a->k_bytes);
  a->y = off; off += align256(a->y_bytes);
  a->packed = off; off += align256(a->plan.packed_weight_bytes);
  a->ws = off; off += align256(a->plan.workspace_bytes);
  a->total = off;
  return FDNN_OK;
}

int fdnn_conv2d_host_arena_bytes(const fdnn_conv_desc* desc, int64_t* bytes) {
  if (desc == nullptr || bytes == nullptr) return fail(FDNN_BAD_PARAM, "NULL argument");
  HostArena a;
  int st = host_arena_layout(desc, &a);
  if (st != FDNN_OK) return st;
  *bytes = a.total;
  return FDNN_OK;
}

int fdnn_conv2d_fwd_host(const fdnn_conv_desc* desc, const void* x_host, const void* w_host,
                         const void* bias_host, const void* scale_host, int activation, void* y_host,
                         void* dev_arena, int64_t arena_bytes, void* stream_v) {
  if (desc == nullptr) return fail(FDNN_BAD_PARAM, "descriptor is NULL");
  HostArena a;
  int st = host_arena_layout(desc, &a);
  if (st != FDNN_OK) return st;
  if (a.y_bytes == 0) return FDNN_OK;
  if (x_host == nullptr || w_host == nullptr || y_host == nullptr)
    return fail(FDNN_BAD_PARAM, "x, w and y must not be NULL");
  if (dev_arena == nullptr || arena_bytes < a.total)
    return fail(FDNN_WORKSPACE_TOO_SMALL, "device arena smaller than fdnn_conv2d_host_arena_bytes");
  if ((reinterpret_cast<uintptr_t>(dev_arena) & 255u) != 0)
    return fail(FDNN_BAD_PARAM, "device arena must be 256-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  char* base = static_cast<char*>(dev_arena);
  cudaError_t e;
  e = cudaMemcpyAsync(base + a.x, x_host, a.x_bytes, cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return fail_cuda("copy x", e);
  e = cudaMemcpyAsync(base + a.w, w_host, a.w_bytes, cudaMemcpyHostToDevice, stream);
  if (e != cudaSuccess) return fail_cuda("copy w", e);
  if (bias_host != nullptr) {
    e = cudaMemcpyAsync(base + a.bias, bias_host, a.k_bytes, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return fail_cuda("copy bias", e);
  }
  if (scale_host != nullptr) {
    e = cudaMemcpyAsync(base + a.scale, scale_host, a.k_bytes, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return fail_cuda("copy scale", e);
  }
  const void* packed = nullptr;
  if (a.plan.algo != FDNN_ALGO_DIRECT && a.plan.w_packed) {
    st = fdnn_conv2d_pack_weight(desc, base + a.w, base + a.y, base + a.packed, a.plan.packed_weight_bytes, stream);
    if (st != FDNN_OK) return st;
    packed = base + a.packed;
  }
  st = fdnn_conv2d_fwd(desc, base + a.x, base + a.w, packed, bias_host ? base + a.bias : nullptr,
                       scale_host ? base + a.scale : nullptr, activation, base + a.y, base + a.ws,
                       a.plan.workspace_bytes, stream);
  if (st != FDNN_OK) return st;
  e = cudaMemcpyAsync(y_host, base + a.y, a.y_bytes, cudaMemcpyDeviceToHost, stream);
  if (e != cudaSuccess) return fail_cuda("copy y", e);
  e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail_cuda("stream sync", e);
  return FDNN_OK;
}

}  // extern "C"
