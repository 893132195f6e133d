// Epilogue shared by the implicit-GEMM kernels when y is dense NHWC: one warp
// drains its 32 accumulator rows from tensor memory, applies per-channel scale,
// bias and the activation in fp32, rounds once, stages 32 rows x 128 bytes in shared
// memory and hands each box to a TMA store.  The arithmetic is that of the
// reference's fused kernel (src/flag_dnn/graph/kernels/fused_conv.py:297-310),
// plus an optional residual tensor added in fp32 before the activation.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "conv_convert.cuh"
#include "sm100_ptx.cuh"
#include "stream_k.cuh"

namespace fdnn {

// max(a, 0) that returns NaN for NaN, like torch.relu (plain max would return 0).
__device__ __forceinline__ float relu_keep_nan(float a) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(0.0f));
  return r;
}

// Two fp32 values -> max(., 0) -> one rounding -> a packed 16-bit pair, in one conversion instruction
// (cvt.rn.relu): saves the two separate maximum instructions per pair in a drain loop that is bound by
// instruction issue on short-reduction layers.  NaN stays NaN (the canonical one), like torch.relu.
template <typename T>
__device__ __forceinline__ uint32_t round_pack2_relu(float a, float b);
template <>
__device__ __forceinline__ uint32_t round_pack2_relu<__half>(float a, float b) {
  uint32_t r;
  asm("cvt.rn.relu.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));  // first source operand lands in the high half
  return r;
}
template <>
__device__ __forceinline__ uint32_t round_pack2_relu<__nv_bfloat16>(float a, float b) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}

// Epilogue activation by its FDNN_ACT_* code: none, ReLU, GELU (erf form, torch's default) or GELU's tanh
// approximation (torch's approximate="tanh").  All keep NaN.
__device__ __forceinline__ float apply_activation(float v, int act) {
  if (act == 1) return relu_keep_nan(v);
  if (act == 2) return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
  if (act == 3) {
    const float u = 0.79788456080286536f * (v + 0.044715f * v * v * v);
    return 0.5f * v * (1.0f + tanhf(u));
  }
  return v;
}

// The same for kernels that exist once with GELU and once without (GELU = false: none or ReLU).  erf and tanh, inlined for
// every value of an unrolled epilogue, are 110 KB of a tensor-core kernel's 180 KB of code; spread between the instructions
// of the other activations they made the drain loop miss the instruction cache, most of all where layers of different
// kernels alternate (in a ResNet-50 of 128 images: 64 -> 256 1x1 at 56 x 56 60.4 -> 51.0 us, 64 -> 64 3x3 37.9 -> 35.3;
// an 8192 x 4096 x 4096 product 177.1 -> 173.2).
template <bool GELU>
__device__ __forceinline__ float activate(float v, int act) {
  if constexpr (GELU) return apply_activation(v, act);
  return act == 1 ? relu_keep_nan(v) : v;
}

template <typename T>
__device__ __forceinline__ uint32_t round_pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t round_pack2<__half>(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t round_pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Two packed 16-bit values -> fp32 (identity for fp32 words is handled by the caller).
template <typename T>
__device__ __forceinline__ void unpack2(uint32_t w, float& a, float& b);
template <>
__device__ __forceinline__ void unpack2<__half>(uint32_t w, float& a, float& b) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  a = f.x;
  b = f.y;
}
template <>
__device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& a, float& b) {
  a = __uint_as_float(w << 16);
  b = __uint_as_float(w & 0xffff0000u);
}
template <>
__device__ __forceinline__ void unpack2<float>(uint32_t w, float& a, float& b) {
  a = __uint_as_float(w);
  b = 0.0f;
}

// How an epilogue warp gets its residual values: the TMA unit copies the 32-row x 128-byte box of the residual
// tensor (seen exactly like y, same swizzle) straight into the staging buffer the outputs will leave from; the
// lane then reads its own row, adds, and writes the finished row back in place.  With two staging buffers the
// box of the next column group is on its way while this one is computed.
struct ResidualFetch {
  const CUtensorMap* tm;          // nullptr: no residual for this warp's rows
  uint64_t* bars;                 // this warp's mbarriers, one per staging buffer
  uint32_t* phases;               // bit b: the parity bars[b] completes next
  volatile uint32_t* abort_flag;  // bounded waits, as everywhere in the kernels
  uint32_t* status_word;
  long long wait_limit;
  // With three staging buffers a box is on its way one group ahead, across tiles as well: `requested` counts the boxes asked
  // for (as store_seq counts the boxes staged); the warp's next tile, if it has one with columns of its own.
  uint32_t requested;
  bool next;
  int next_n0, next_row, next_img;
};

// t_row     tensor-memory address of this warp's lane quarter, first column of the tile
// n0        first GEMM column of the tile; kout: number of valid GEMM columns overall
// s_scale / s_bias  this warp's fp32 copies for columns n0 .. n0+BN-1
// my_out    this warp's NBUF 4 KB staging buffers (1024-byte aligned; two or three are used in rotation so
//           that a box can still be leaving through the TMA unit while the next one is staged;
//           with one, the other warp of the lane quarter fills that gap)
// tm_full / tm_tail  output maps with a 32-row box and a box of the tile's ragged last rows
// st_row, st_img     y coordinates (row, image) of the warp's first row; st_rows: valid rows (<= 0: none)
// store_seq          running count of this warp's staged boxes (selects the staging buffer)
// use_scale          false when the launch has no per-channel scale (s_scale then holds ones and is not read)
// RES                a residual tensor (same layout as y) is added before the activation
// rf                 how the residual box reaches the staging buffer (see ResidualFetch; the producer asked for
//                    the tile's residual values to be brought into L2 a main loop earlier)
// sk_slot0 / sk_count / sk_slot_stride / sk_row / sk_pc0
//                    reduction splitting: the accumulator holds only the tile's last reduction steps; add the
//                    fp32 partial sums of sk_count other CTAs first (slots sk_slot0, sk_slot0 - sk_slot_stride,
//                    ... in that order; this lane's row sk_row, this warp's first 16-byte piece sk_pc0)
template <typename T, int BN, bool RES, int NBUF, bool GELU>
__device__ __forceinline__ void epilogue_store_tile(uint32_t t_row, int n0, int kout, int act,
                                                    const float* s_scale, const float* s_bias,
                                                    uint8_t* my_out, int lane, const CUtensorMap* tm_full,
                                                    const CUtensorMap* tm_tail, int st_row, int st_img,
                                                    int st_rows, uint32_t& store_seq,
                                                    ResidualFetch* rf = nullptr, bool use_scale = true,
                                                    const float* sk_slot0 = nullptr, int sk_count = 0,
                                                    long long sk_slot_stride = 0, int sk_row = 0, int sk_pc0 = 0) {
  constexpr int kPerStore = 128 / int(sizeof(T));  // channels per staged row: 64 (16-bit) or 32 (fp32)
  constexpr int kLoads = kPerStore / 32;
  int groups = (kout - n0 + kPerStore - 1) / kPerStore;
  if (groups > BN / kPerStore) groups = BN / kPerStore;
  if (groups <= 0) return;
  uint32_t raw[kLoads][32];
#pragma unroll
  for (int l = 0; l < kLoads; ++l) tmem_ld_32x32b_x32(t_row + l * 32, raw[l]);
#pragma unroll 1
  for (int g = 0; g < groups; ++g) {
    const uint32_t slot = NBUF == 1 ? 0u : store_seq % uint32_t(NBUF);   // alternates across groups AND tiles
    uint8_t* buf = my_out + slot * (32 * 128);
    ++store_seq;
    if constexpr (RES && NBUF == 3) {
      const bool have = rf != nullptr && rf->tm != nullptr && st_rows > 0;   // uniform across the warp
      if (have) {
        auto request = [&](uint32_t to, int col, int row, int img) {
          mbar_arrive_expect_tx(&rf->bars[to], 32 * 128);
          tma_load_3d(my_out + to * (32 * 128), rf->tm, &rf->bars[to], col, row, img);
        };
        const bool first = rf->requested != store_seq;     // not asked for during the group before
        const bool more = g + 1 < groups || rf->next;
        if (lane == 0) {
          if (first) {
            bulk_wait_group_read0();
            request(slot, n0 + g * kPerStore, st_row, st_img);
          } else {
            bulk_wait_group_read1();   // the box staged two groups ago has left the buffer asked for here
          }
          if (more) {
            const bool here = g + 1 < groups;
            request(slot == 2 ? 0u : slot + 1u, here ? n0 + (g + 1) * kPerStore : rf->next_n0, here ? st_row : rf->next_row,
                    here ? st_img : rf->next_img);
          }
        }
        rf->requested = store_seq + (more ? 1u : 0u);
        __syncwarp();
        mbar_wait_bounded(&rf->bars[slot], (*rf->phases >> slot) & 1u, rf->abort_flag, rf->status_word, kIncidentResidualWait,
                          rf->wait_limit);
        *rf->phases ^= 1u << slot;
      } else if (lane == 0) {
        bulk_wait_group_read1();
      }
    } else if constexpr (RES) {
      const bool have = rf != nullptr && rf->tm != nullptr && st_rows > 0;   // uniform across the warp
      const uint32_t b = NBUF == 2 ? ((store_seq - 1u) & 1u) : 0u;
      if (lane == 0) {
        bulk_wait_group_read0();   // every staged box has left: both buffers may be written
        if (have) {
          if (g == 0 || NBUF == 1) {
            mbar_arrive_expect_tx(&rf->bars[b], 32 * 128);
            tma_load_3d(buf, rf->tm, &rf->bars[b], n0 + g * kPerStore, st_row, st_img);
          }
          if (NBUF == 2 && g + 1 < groups) {
            mbar_arrive_expect_tx(&rf->bars[b ^ 1u], 32 * 128);
            tma_load_3d(my_out + (b ^ 1u) * (32 * 128), rf->tm, &rf->bars[b ^ 1u], n0 + (g + 1) * kPerStore, st_row,
                        st_img);
          }
        }
      }
      __syncwarp();
      if (have) {
        mbar_wait_bounded(&rf->bars[b], (*rf->phases >> b) & 1u, rf->abort_flag, rf->status_word,
                          kIncidentResidualWait, rf->wait_limit);
        *rf->phases ^= 1u << b;
      }
    }
    tmem_ld_wait();
    for (int c = 0; c < sk_count; ++c) {  // uniform across the launch's owner tiles; zero otherwise
      const float* slot = sk_slot0 - c * sk_slot_stride;
#pragma unroll
      for (int l = 0; l < kLoads; ++l) {
        float4 part[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) part[j] = sk_load_piece(slot, sk_pc0 + g * (kPerStore / 4) + l * 8 + j, sk_row);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          raw[l][4 * j + 0] = __float_as_uint(__uint_as_float(raw[l][4 * j + 0]) + part[j].x);
          raw[l][4 * j + 1] = __float_as_uint(__uint_as_float(raw[l][4 * j + 1]) + part[j].y);
          raw[l][4 * j + 2] = __float_as_uint(__uint_as_float(raw[l][4 * j + 2]) + part[j].z);
          raw[l][4 * j + 3] = __float_as_uint(__uint_as_float(raw[l][4 * j + 3]) + part[j].w);
        }
      }
    }
    uint32_t row[32];  // the 128 bytes this lane contributes
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      const float4* sc4 = reinterpret_cast<const float4*>(s_scale + g * kPerStore + l * 32);
      const float4* bi4 = reinterpret_cast<const float4*>(s_bias + g * kPerStore + l * 32);
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4) {
        // without a per-channel scale the multiplier is 1 and its shared-memory read is skipped (uniform
        // branch): -13 % on a 64 -> 256 1x1 layer; packing scale and bias into one word per column instead
        // saves the same reads but pays them back in unpacking instructions
        const float4 sc = use_scale ? sc4[j4] : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        const float4 bi = bi4[j4];
        float v0 = fmaf(__uint_as_float(raw[l][4 * j4 + 0]), sc.x, bi.x);
        float v1 = fmaf(__uint_as_float(raw[l][4 * j4 + 1]), sc.y, bi.y);
        float v2 = fmaf(__uint_as_float(raw[l][4 * j4 + 2]), sc.z, bi.z);
        float v3 = fmaf(__uint_as_float(raw[l][4 * j4 + 3]), sc.w, bi.w);
        if constexpr (RES) {
          if constexpr (std::is_same<T, float>::value) {
            const uint4 mine = *reinterpret_cast<const uint4*>(buf + lane * 128 + ((j4 ^ (lane & 7)) << 4));
            v0 += __uint_as_float(mine.x);
            v1 += __uint_as_float(mine.y);
            v2 += __uint_as_float(mine.z);
            v3 += __uint_as_float(mine.w);
          } else {
            // 16-byte piece l*4 + j4/2 of the row holds the eight values of two passes of this loop
            const uint2 mine = *reinterpret_cast<const uint2*>(
                buf + lane * 128 + (((l * 4 + (j4 >> 1)) ^ (lane & 7)) << 4) + ((j4 & 1) << 3));
            float r0, r1, r2, r3;
            unpack2<T>(mine.x, r0, r1);
            unpack2<T>(mine.y, r2, r3);
            v0 += r0;
            v1 += r1;
            v2 += r2;
            v3 += r3;
          }
        }
        if constexpr (std::is_same<T, float>::value) {
          v0 = activate<GELU>(v0, act);   // uniform across the launch
          v1 = activate<GELU>(v1, act);
          v2 = activate<GELU>(v2, act);
          v3 = activate<GELU>(v3, act);
          row[4 * j4 + 0] = __float_as_uint(v0);
          row[4 * j4 + 1] = __float_as_uint(v1);
          row[4 * j4 + 2] = __float_as_uint(v2);
          row[4 * j4 + 3] = __float_as_uint(v3);
        } else if (act == 1) {  // ReLU folded into the rounding conversion
          row[l * 16 + 2 * j4 + 0] = round_pack2_relu<T>(v0, v1);
          row[l * 16 + 2 * j4 + 1] = round_pack2_relu<T>(v2, v3);
        } else {
          if constexpr (GELU) {
            v0 = apply_activation(v0, act);
            v1 = apply_activation(v1, act);
            v2 = apply_activation(v2, act);
            v3 = apply_activation(v3, act);
          }
          row[l * 16 + 2 * j4 + 0] = round_pack2<T>(v0, v1);
          row[l * 16 + 2 * j4 + 1] = round_pack2<T>(v2, v3);
        }
      }
    }
    // the accumulator columns of the next group travel while this one is stored
    if (g + 1 < groups) {
#pragma unroll
      for (int l = 0; l < kLoads; ++l) tmem_ld_32x32b_x32(t_row + (g + 1) * kPerStore + l * 32, raw[l]);
    }
    if constexpr (!RES) {
      if (lane == 0) {
        // the box staged NBUF groups ago has left this buffer
        if constexpr (NBUF == 2) bulk_wait_group_read1(); else bulk_wait_group_read0();
      }
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      // 128-byte swizzle: the 16-byte pieces of neighbouring rows land in different banks
      *reinterpret_cast<uint4*>(buf + lane * 128 + ((q ^ (lane & 7)) << 4)) =
          make_uint4(row[4 * q], row[4 * q + 1], row[4 * q + 2], row[4 * q + 3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      // committed even when empty so that "all but the latest group" always means the other buffer
      if (st_rows > 0) tma_store_3d(st_rows >= 32 ? tm_full : tm_tail, buf, n0 + g * kPerStore, st_row, st_img);
      bulk_commit_group();
    }
  }
}

// Epilogue for a channels-last y the TMA unit cannot write (its strides or base are not multiples of 16 bytes): the same
// arithmetic, and 32 rows x 128 bytes are staged in shared memory all the same, as [pixel][64 columns], but the warp then
// writes them itself, with lanes along the channels and `unit` bytes per lane, the widest the alignment of y allows.
// Where 16-bit rows may start at odd elements (unit 2), each run is written as the 4-byte words it covers whole, plus a
// 2-byte element at either end.  (One 2-byte store per value straight from the registers, each lane in a row of its own:
// 24 x 45 x 37 pixels, 104 -> 150 channels bf16 3x3, 106 us.)
constexpr int kYScattered = 0, kYPixels = 1, kYChannels = 2;   // how y is written: element by element, along pixels or channels
struct StridedOut {
  void* y;                 // element type of the operands
  const void* res;         // residual with y's strides, or nullptr
  long long y_off;         // this lane's pixel: element offset of the (group's) first channel
  int unit;                // bytes per lane and store
  bool row_ok;             // this lane's row exists
};

template <typename U> __device__ __forceinline__ U lds_unit(uint32_t a);
template <> __device__ __forceinline__ uint32_t lds_unit<uint32_t>(uint32_t a) { return lds_u32(a); }
template <> __device__ __forceinline__ uint2 lds_unit<uint2>(uint32_t a) { return lds_v2(a); }
template <> __device__ __forceinline__ uint4 lds_unit<uint4>(uint32_t a) { return lds_v4(a); }

// The writers of a staged group.  Each reads a batch of units from shared memory before it stores the first: with load
// and store of one unit after another the warp waits a shared-memory round trip per store (21 k clocks per 128 x 256 tile
// instead of the few thousand its stores take).
//
// [pixel][128 bytes of columns], swizzled, U units along columns; row r's element offset is lane r's y_off.
template <typename U, int ES>
__device__ __forceinline__ void strided_channels(char* out, uint32_t sbuf, int lane, int nc, uint32_t rows_ok, long long y_off) {
  constexpr int kLanes = 128 / int(sizeof(U)), kPer = 32 / kLanes, kBatch = 8;
  const int byte0 = (lane % kLanes) * int(sizeof(U));
  const bool full = byte0 + int(sizeof(U)) <= nc * ES;
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += kPer * kBatch) {
    U v[kBatch];
    long long off[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int r = (r0 + i * kPer + lane / kLanes) & 31;
      v[i] = lds_unit<U>(sbuf + r * 128 + ((((byte0 >> 4) ^ (r & 7)) << 4) | (byte0 & 15)));
      off[i] = __shfl_sync(0xffffffffu, y_off, r);
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int r = r0 + i * kPer + lane / kLanes;
      if (r >= 32 || !((rows_ok >> r) & 1u)) continue;
      char* dst = out + off[i] * ES + byte0;
      if (full) {
        *reinterpret_cast<U*>(dst) = v[i];
      } else {   // the last columns: element by element
        for (int b = 0; byte0 + b < nc * ES; b += ES) {
          const int byte = byte0 + b;
          const uint32_t a = sbuf + r * 128 + ((((byte >> 4) ^ (r & 7)) << 4) | (byte & 15));
          if constexpr (ES == 2) *reinterpret_cast<uint16_t*>(dst + b) = lds_u16(a);
          else *reinterpret_cast<uint32_t*>(dst + b) = lds_u32(a);
        }
      }
    }
  }
}

// The same for 16-bit rows that may start at odd elements: one row per store, as whole words and two ends: word l
// of a row that starts on a word boundary; else the halves either side of the boundary after it, and the last lane, whose
// neighbour wraps to word 0, writes the first element.
__device__ __forceinline__ void strided_odd_channels(char* out, uint32_t sbuf, int lane, int nc, uint32_t rows_ok, long long y_off) {
  uint16_t* y = reinterpret_cast<uint16_t*>(out);
  auto word = [&](int r, int w) { return sbuf + r * 128 + ((((w >> 2) ^ (r & 7)) << 4) | ((w & 3) << 2)); };
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += 8) {
    uint32_t lo[8], hi[8];
    long long off[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      off[i] = __shfl_sync(0xffffffffu, y_off, r0 + i);
      lo[i] = lds_u32(word(r0 + i, lane));
      hi[i] = lds_u32(word(r0 + i, (lane + 1) & 31));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (!((rows_ok >> (r0 + i)) & 1u)) continue;
      uint16_t* run = y + off[i];
      const bool par = (reinterpret_cast<uintptr_t>(run) & 2u) != 0;
      const int a = 2 * lane + (par ? 1 : 0);
      const uint32_t v = par ? __byte_perm(lo[i], hi[i], 0x5432) : lo[i];
      if (a + 1 < nc) *reinterpret_cast<uint32_t*>(run + a) = v;
      else if (a < nc) run[a] = uint16_t(v);
      if (par && lane == 31) run[0] = uint16_t(hi[i]);
    }
  }
}

// NBUF staging buffers of 4 KB per warp.
template <typename T, int BN, bool RES, int NBUF, bool GELU>
__device__ __forceinline__ void epilogue_store_strided(uint32_t t_row, int n0, int kout, int act, const float* s_scale,
                                                       const float* s_bias, uint8_t* my_out, int lane,
                                                       const StridedOut& o, uint32_t& store_seq) {
  constexpr int kEs = int(sizeof(T));
  constexpr int kCols = 128 / kEs;                 // columns per group: 64 (16-bit) or 32 (fp32)
  constexpr int kLoads = kCols / 32;
  int groups = (kout - n0 + kCols - 1) / kCols;
  if (groups > BN / kCols) groups = BN / kCols;
  if (groups <= 0) return;
  char* y = static_cast<char*>(o.y);
  const uint32_t rows_ok = __ballot_sync(0xffffffffu, o.row_ok);
#pragma unroll 1
  for (int g = 0; g < groups; ++g) {
    uint32_t raw[kLoads][32];
#pragma unroll
    for (int l = 0; l < kLoads; ++l) tmem_ld_32x32b_x32(t_row + g * kCols + l * 32, raw[l]);
    uint8_t* buf = my_out + (NBUF == 2 ? (store_seq & 1u) * (32 * 128) : 0u);
    ++store_seq;
    const int col0 = n0 + g * kCols;
    const int nc = kout - col0 < kCols ? kout - col0 : kCols;    // columns of this group that exist
    tmem_ld_wait();
    uint32_t row[32];
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      float v[32];
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4) {
        const float4 sc = reinterpret_cast<const float4*>(s_scale + g * kCols + l * 32)[j4];
        const float4 bi = reinterpret_cast<const float4*>(s_bias + g * kCols + l * 32)[j4];
        v[4 * j4 + 0] = fmaf(__uint_as_float(raw[l][4 * j4 + 0]), sc.x, bi.x);
        v[4 * j4 + 1] = fmaf(__uint_as_float(raw[l][4 * j4 + 1]), sc.y, bi.y);
        v[4 * j4 + 2] = fmaf(__uint_as_float(raw[l][4 * j4 + 2]), sc.z, bi.z);
        v[4 * j4 + 3] = fmaf(__uint_as_float(raw[l][4 * j4 + 3]), sc.w, bi.w);
      }
      if constexpr (RES) {
        if (o.res != nullptr && o.row_ok) {
          const T* res = static_cast<const T*>(o.res) + o.y_off + col0 + l * 32;
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (l * 32 + j < nc) v[j] += to_f32<T>(res[j]);
        }
      }
      if constexpr (GELU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = apply_activation(v[j], act);
      }
      if constexpr (kEs == 4) {
#pragma unroll
        for (int j = 0; j < 32; ++j) row[j] = __float_as_uint(act == 1 ? relu_keep_nan(v[j]) : v[j]);
      } else if (act == 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) row[l * 16 + j] = round_pack2_relu<T>(v[2 * j], v[2 * j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) row[l * 16 + j] = round_pack2<T>(v[2 * j], v[2 * j + 1]);
      }
    }
    const uint32_t sbuf = smem_u32(buf);
    if constexpr (NBUF == 1) __syncwarp();   // the group before has been read
#pragma unroll
    for (int q = 0; q < 8; ++q)   // 16-byte pieces swizzled by row, as for the TMA store
      sts_v4(sbuf + lane * 128 + ((q ^ (lane & 7)) << 4), make_uint4(row[4 * q], row[4 * q + 1], row[4 * q + 2], row[4 * q + 3]));
    __syncwarp();
    char* out = y + (long long)col0 * kEs;
    if (kEs == 2 && o.unit == 2) strided_odd_channels(out, sbuf, lane, nc, rows_ok, o.y_off);
    else if (o.unit == 16) strided_channels<uint4, kEs>(out, sbuf, lane, nc, rows_ok, o.y_off);
    else if (o.unit == 8) strided_channels<uint2, kEs>(out, sbuf, lane, nc, rows_ok, o.y_off);
    else strided_channels<uint32_t, kEs>(out, sbuf, lane, nc, rows_ok, o.y_off);
  }
}

// fp32 values before they are stored: ReLU behind one branch for all of them, and every value computed here.  With a select per
// value between the stores, and nothing to keep the scale's and the bias's reads from sinking between them too, a
// 64 -> 64 1x1 layer on 32 x 56 x 56 NCHW took 26.6 us, now 16.5; 64 -> 256 on 16 x 56 x 56 28.7 and 21.5.  (Rounding to 16 bits
// holds the values together by itself: the same there 12.7 -> 13.1 us, 128 -> 128 3x3 on 32 x 28 x 28.)
__device__ __forceinline__ void finish_f32(float (&v)[32], int act) {
  if (act == 1) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = relu_keep_nan(v[j]);
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) asm volatile("" : "+f"(v[j]));
}

// Epilogue for y along channels whose pixels start on 32-byte boundaries (16-bit: a multiple of 16 channels, or views that
// keep that): a lane writes its own pixel from the registers, 16 channels (fp32: 8; one whole 32-byte sector) per store,
// without staging.  y: the lane's pixel, first column of the warp's share; ok: the pixel exists.
// read_done() is called once, when the accumulator has been read and before its last columns are stored.
template <typename T, int WC, bool GELU, typename Done>
__device__ __forceinline__ void epilogue_store_sectors(uint32_t t_row, int n0, int kout, int act, const float* s_scale,
                                                       const float* s_bias, bool use_scale, T* y, bool ok, Done&& read_done) {
  int chunks = (kout - n0 + 31) / 32;
  if (chunks > WC / 32) chunks = WC / 32;
  if (chunks <= 0) {
    read_done();
    return;
  }
  uint32_t raw[32];
  tmem_ld_32x32b_x32(t_row, raw);
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    tmem_ld_wait();
    float v[32];
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
      const float4 sc = use_scale ? reinterpret_cast<const float4*>(s_scale + c * 32)[j4] : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      const float4 bi = reinterpret_cast<const float4*>(s_bias + c * 32)[j4];
      v[4 * j4 + 0] = fmaf(__uint_as_float(raw[4 * j4 + 0]), sc.x, bi.x);
      v[4 * j4 + 1] = fmaf(__uint_as_float(raw[4 * j4 + 1]), sc.y, bi.y);
      v[4 * j4 + 2] = fmaf(__uint_as_float(raw[4 * j4 + 2]), sc.z, bi.z);
      v[4 * j4 + 3] = fmaf(__uint_as_float(raw[4 * j4 + 3]), sc.w, bi.w);
    }
    if constexpr (sizeof(T) == 4) finish_f32(v, act);
    if (c + 1 < chunks) tmem_ld_32x32b_x32(t_row + (c + 1) * 32, raw);   // travels while this chunk is rounded and stored
    else read_done();
    if constexpr (GELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = apply_activation(v[j], act);
    }
    if constexpr (sizeof(T) == 4) {
      uint32_t row[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) row[j] = __float_as_uint(v[j]);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (ok && n0 + c * 32 + i * 8 + 8 <= kout) stg_v8(y + c * 32 + i * 8, row + i * 8);
    } else {
      uint32_t row[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) row[j] = act == 1 ? round_pack2_relu<T>(v[2 * j], v[2 * j + 1]) : round_pack2<T>(v[2 * j], v[2 * j + 1]);
      if (ok) {
        if (n0 + c * 32 + 16 <= kout) stg_v8(y + c * 32, row);
        if (n0 + c * 32 + 32 <= kout) stg_v8(y + c * 32 + 16, row + 8);
      }
    }
  }
}

// Epilogue for y along pixels (NCHW): a lane writes its own pixel of one channel after another, neighbouring lanes
// neighbouring pixels, straight from the registers.  A 64-byte run per store reaches 2.6 (any alignment) to 4 TB/s over the
// chip; staging the rows to store wider units cost more in latency than it saved (64 -> 64 3x3 on 128 x 56 x 56, 16 bytes
// per lane 60.1 us, 4 bytes 62.9, straight from the registers 38.0).
//   y, res: the lane's pixel, first column of the warp's share (res: nullptr or a tensor with y's strides); sk: elements
//   between channels; read_done() is called once, when the accumulator has been read and before its last columns are stored
template <typename T, int WC, bool RES, bool GELU, typename Done>
__device__ __forceinline__ void epilogue_store_pixels(uint32_t t_row, int n0, int kout, int act, const float* s_scale,
                                                      const float* s_bias, bool use_scale, T* y, const T* res, long long sk,
                                                      bool ok, Done&& read_done) {
  int chunks = (kout - n0 + 31) / 32;
  if (chunks > WC / 32) chunks = WC / 32;
  if (chunks <= 0) {
    read_done();
    return;
  }
  uint32_t raw[32];
  tmem_ld_32x32b_x32(t_row, raw);
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    const int nc = kout - n0 - c * 32;
    float r[RES ? 32 : 1];
    if constexpr (RES) {
      if (res != nullptr && ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < nc) r[j] = to_f32<T>(res[j * sk]);
        res += 32 * sk;
      }
    }
    tmem_ld_wait();
    float v[32];
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
      const float4 sc = use_scale ? reinterpret_cast<const float4*>(s_scale + c * 32)[j4] : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      const float4 bi = reinterpret_cast<const float4*>(s_bias + c * 32)[j4];
      v[4 * j4 + 0] = fmaf(__uint_as_float(raw[4 * j4 + 0]), sc.x, bi.x);
      v[4 * j4 + 1] = fmaf(__uint_as_float(raw[4 * j4 + 1]), sc.y, bi.y);
      v[4 * j4 + 2] = fmaf(__uint_as_float(raw[4 * j4 + 2]), sc.z, bi.z);
      v[4 * j4 + 3] = fmaf(__uint_as_float(raw[4 * j4 + 3]), sc.w, bi.w);
    }
    if constexpr (sizeof(T) == 4 && !RES) finish_f32(v, act);
    if (c + 1 < chunks) tmem_ld_32x32b_x32(t_row + (c + 1) * 32, raw);   // travels while this chunk is rounded and stored
    else read_done();
    if constexpr (RES) {
      if (res != nullptr && ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < nc) v[j] += r[j];
      }
    }
    if constexpr (GELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = apply_activation(v[j], act);
    }
    if constexpr (sizeof(T) == 4) {
      if (ok) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (j < nc) *y = RES && act == 1 ? relu_keep_nan(v[j]) : v[j];
          y += sk;
        }
      }
    } else {
      uint32_t row[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) row[j] = act == 1 ? round_pack2_relu<T>(v[2 * j], v[2 * j + 1]) : round_pack2<T>(v[2 * j], v[2 * j + 1]);
      uint16_t* y16 = reinterpret_cast<uint16_t*>(y);
      if (ok) {
        if (nc >= 32) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            y16[0] = uint16_t(row[j]);
            y16[sk] = uint16_t(row[j] >> 16);
            y16 += 2 * sk;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (2 * j < nc) y16[0] = uint16_t(row[j]);
            if (2 * j + 1 < nc) y16[sk] = uint16_t(row[j] >> 16);
            y16 += 2 * sk;
          }
        }
      }
      y = reinterpret_cast<T*>(y16);
    }
  }
}

// Contributor side of reduction splitting: this warp's 32 rows x WC raw fp32 accumulator columns go to the
// CTA's slot (piece pc0 onwards, row `row`) instead of through the epilogue.
template <int WC>
__device__ __forceinline__ void epilogue_dump_partial(uint32_t t_row, float* slot, int pc0, int row) {
  uint32_t raw[2][32];
  tmem_ld_32x32b_x32(t_row, raw[0]);
#pragma unroll
  for (int c = 0; c < WC / 32; ++c) {
    tmem_ld_wait();
    if (c + 1 < WC / 32) tmem_ld_32x32b_x32(t_row + (c + 1) * 32, raw[(c + 1) & 1]);
#pragma unroll
    for (int j = 0; j < 8; ++j) sk_store_piece(slot, pc0 + c * 8 + j, row, &raw[c & 1][4 * j]);
  }
}

}  // namespace fdnn
