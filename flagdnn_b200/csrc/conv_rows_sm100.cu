// Implicit-GEMM convolution forward on CTA pairs for layers of W-stride 1 whose filters are two taps wide or more:
// the activations of a filter row are copied once and serve every tap of that row.
//
// A GEMM row is a pixel of the output in a row pitch P = W + max(left, right padding) >= OW ("walk" rows: the positions
// an im2col copy of that width walks through, padding included).  In that numbering the operand of tap s is the operand
// of tap 0 moved down by s * dil_w rows, across image rows and images alike: what tap s reads past the end of an image
// row is the padding in front of the next one.  So one im2col copy of 128 + 8 walk rows x 64 channels per filter row and
// channel block is staged, and the MMAs of tap s read it from row s * dil_w on: a shared-memory descriptor may start on
// any 128-byte row, because the 128-byte swizzle is a function of the address alone.  The P - OW walk rows per image row
// that are no output are computed and not stored (1 in 15 at 14 columns, 1 in 57 at 56).
//
// What this buys: the kernels that copy the activations anew for every tap are bound by their operand stream from L2
// (32 KB per CTA and step of four 256 x 256 x 16 MMAs, 512 clocks, at 55 to 70 bytes per clock and SM) and by what the
// copies and the MMAs together ask of shared memory (64 + 64 of 128 bytes per clock).  With three taps per copy a step
// brings 16 + 5.7 KB; with the whole filter resident (short reductions into one column tile) 5.7 KB.  Narrow layers
// run on tiles of 64 or 128 columns as they are, without the zeros that grouping their pixels multiplies with.
//
// Few large groups (BLK): a block of 64 channels holds 64 / (channels per group) groups.  The copies of the activations
// stay whole blocks, and each 16-channel slice of a step multiplies the columns of its own group only; the filter tile
// of a group has rows of 32 or 64 bytes (32- or 64-byte swizzle).  Against the block-diagonal dense filter that is half
// (a quarter) of the MMAs and of the filter bytes.
//
// Roles as in conv_igemm_pair_sm100.cu: warp 0 copies, warp 1 of the leader issues, warps 4..11 drain.  32 walk rows that
// are 32 pixels leave as boxes through the TMA unit; where rows fall out in between, each lane stores its own pixel.
//
// Measured on the way (64 -> 64 3x3 on 128 x 56 x 56, bf16): 64.4 us with a branch and 64-bit descriptors between the MMAs
// (470 to 690 clocks per step of four, whatever its width; resident operands: 172 for 64 columns); 45.2 with the
// descriptors built in place and one wait for the three taps of a filter row; 41.4 with 32-byte stores from the registers
// instead of staging (4.8 k clocks per 32 rows x 64 columns and warp); 31.4 with one hand-over of the accumulator per
// warp, at CTA scope: a release at cluster scope by every thread waited for the stores before it.  What bounds it now is
// shared memory: the MMAs read 5 KB per 43 clocks beside 52 KB of copies per tile.  256 -> 256 on 256 x 14 x 14 keeps the
// tensor pipe busy for 52 k of its 67 k clocks (counters, at 1.65 GHz) and brings 336 MB from L2 where a copy per tap brings 462.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "conv_convert.cuh"
#include "conv_epilogue.cuh"
#include "conv_internal.h"
#include "sm100_ptx.cuh"

namespace fdnn {
namespace {

constexpr int kRows = 128;                                  // walk rows per CTA and tile (pair tile: 256)
constexpr int kACopyRows = kRowsCopy;                       // rows of an activation copy: taps up to 8 rows apart
constexpr int kABytes = kACopyRows * 128;                   // 17 KB, a multiple of the swizzle's 1 KB
constexpr int kRingBytes = 184 * 1024;
constexpr int kMaxA = 8, kMaxB = 16;                        // ring slots
constexpr int kEpiWarps = 8;
constexpr int kFirstEpiWarp = 4;
constexpr int kThreads = 32 * (kFirstEpiWarp + kEpiWarps);
constexpr int kRegsLean = 128, kRegsEpilogue = 184;
static_assert(128 * kRegsLean + 32 * kEpiWarps * kRegsEpilogue <= kThreads * (65536 / kThreads / 8 * 8),
              "register reallocation exceeds the launch allocation");
constexpr int kOutBytes = kEpiWarps * 32 * 128;             // one 4 KB staging buffer per warp
constexpr int kBars = 2 * kMaxA + 2 * kMaxB + 6;

template <int BN>
struct Cfg {
  // 256 and 128 columns: two warps per tensor-memory lane quarter, half of the columns each; 64 columns (one staged group):
  // the two sets of four warps take alternate tiles
  static constexpr int kSets = BN == 64 ? 2 : 1;
  static constexpr int kWarpCols = BN == 64 ? 64 : BN / 2;
  static constexpr int kEpiBytes = kEpiWarps * 2 * kWarpCols * int(sizeof(float));
  static constexpr int kSmem = kRingBytes + kOutBytes + kEpiBytes + kBars * 8 + 16 + 1024;
  static_assert(kSmem <= 227 * 1024, "shared memory budget");
};

// BLK: groups per 64-channel block (1: not grouped).  STORE: how y is written.
constexpr int kStoreSectors = 0;    // along channels, whole 32-byte sectors per lane
constexpr int kStoreChannels = 1;   // along channels, any alignment
constexpr int kStorePixels = 2;     // along pixels
// GELU: the activation is one of the GELU forms (p.act > 1).
template <typename T, int BN, int BLK, int STORE, bool GELU>
__global__ void __launch_bounds__(kThreads, 1)
conv_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA2,
                 const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmY, const RowsParams p) {
  using C = Cfg<BN>;
  constexpr bool kSplit = std::is_same<T, float>::value;
  constexpr uint32_t kFmt = std::is_same<T, __half>::value ? 0u : kSplit ? 2u : 1u;
  constexpr int kBlock = 128 / int(sizeof(T));      // channels per copy
  constexpr int kAStage = (kSplit ? 2 : 1) * kABytes;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // activation ring, then the filter: a ring of one tap and channel block per slot, or all of them
  uint8_t* a_ring = smem;
  uint8_t* b_ring = smem + p.a_stages * kAStage;
  uint8_t* out_stage = smem + kRingBytes;
  float* epi_stage = reinterpret_cast<float*>(out_stage + kOutBytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + kOutBytes + C::kEpiBytes);
  uint64_t* a_full = bars;                       // used in the leader only
  uint64_t* a_empty = bars + kMaxA;              // each CTA's own
  uint64_t* b_full = bars + 2 * kMaxA;           // leader only
  uint64_t* b_empty = bars + 2 * kMaxA + kMaxB;  // each CTA's own
  uint64_t* tmem_full = bars + 2 * kMaxA + 2 * kMaxB;    // [2], each CTA's own
  uint64_t* tmem_empty = tmem_full + 2;                  // [2], leader only
  uint64_t* drain_bar = tmem_full + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 5);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();       // 0 = leader

  griddep_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kMaxA; ++i) {
      mbar_init(&a_full[i], 1);
      mbar_init(&a_empty[i], 1);
    }
    for (int i = 0; i < kMaxB; ++i) {
      mbar_init(&b_full[i], 1);
      mbar_init(&b_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * (kEpiWarps / C::kSets));   // epilogue warps of both CTAs that drain this buffer
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if constexpr (kSplit) tma_prefetch_desc(&tmA2);
    if (p.y_rows) tma_prefetch_desc(&tmY);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 2 * BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int total_tiles = ((p.m_tiles + 1) / 2) * p.n_tiles;
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int steps = p.R * p.c_blocks;            // activation copies per tile

  if (warp < kFirstEpiWarp) {
  warpgroup_reg_dec<kRegsLean>();
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    const bool lead = elect_one();
    griddep_wait();      // from here on global memory is read: the launch before this one must be complete
    if (!p.skip_copies) {
      bool alive = true;
      uint32_t as = 0, aphase = 0, bs = 0, bphase = 0;
      const uint32_t a_full0 = map_to_cta(smem_u32(&a_full[0]), 0), b_full0 = map_to_cta(smem_u32(&b_full[0]), 0);
      const int ohp = p.OH * p.P;
      // one filter slot: b_taps taps of a channel block, [tap][filter][channels]
      auto copy_filter = [&](uint8_t* dst, uint32_t bar, int n_tile, int c0, int tap) {
        if constexpr (BLK > 1) {
          // group after group of the channel block: kg / 2 filters of this CTA, cg channels each
          const int part = p.b_slot / BLK;
          for (int g = 0; g < BLK; ++g) {
            const int group = n_tile * BLK + g;
            tma_load_3d_pair(dst + g * part, &tmB, bar, group * p.blk_c_step, group * p.kg + int(rank) * (p.kg / 2), tap);
          }
        } else if constexpr (kSplit) {   // both halves, one behind the other
          tma_load_4d_pair(dst, &tmB, bar, c0, n_tile * BN + int(rank) * (BN / 2), tap, 0);
        } else {
          tma_load_3d_pair(dst, &tmB, bar, c0, n_tile * BN + int(rank) * (BN / 2), tap);
        }
      };
      if (p.b_resident && pair_id < total_tiles && lead) {   // n_tiles == 1, slots of a whole filter row
        if (rank == 0) mbar_arrive_expect_tx(&b_full[0], uint32_t(2 * steps * p.b_slot));
        uint8_t* dst = b_ring;
        for (int r = 0; r < p.R; ++r)
          for (int cb = 0; cb < p.c_blocks; ++cb, dst += p.b_slot) copy_filter(dst, b_full0, 0, cb * kBlock, r * p.s_pitch);
      }
      __syncwarp();
      for (int tile = pair_id; tile < total_tiles && alive; tile += num_pairs) {
        const int m_pair = tile / p.n_tiles;
        const int n_tile = tile - m_pair * p.n_tiles;
        const int m0 = (2 * m_pair + int(rank)) * kRows;     // first walk row (may lie past the end: zeros arrive)
        const int img = m0 / ohp;
        const int rem = m0 - img * ohp;
        const int oh0 = rem / p.P;
        const int w_base = rem - oh0 * p.P - p.pad_left;
        const int h_base = oh0 * p.stride_h - p.pad_top;
        int r = 0, cb = 0;
        for (int kit = 0; kit < steps; ++kit) {
          if (!mbar_wait_warp(&a_empty[as], aphase ^ 1u, abort_flag, p.status, kIncidentProducerWait, p.wait_limit)) {
            alive = false;
            break;
          }
          const int c0 = BLK > 1 ? n_tile * 64 : cb * kBlock;
          if (lead) {
            if (rank == 0) mbar_arrive_expect_tx(&a_full[as], uint32_t(2 * kAStage));
            uint8_t* dst = a_ring + as * kAStage;
            const uint16_t off_h = static_cast<uint16_t>(r * p.dil_h);
            tma_load_im2col_4d_pair(dst, &tmA, a_full0 + as * 8, c0, w_base, h_base, img, 0, off_h);
            if constexpr (kSplit) tma_load_im2col_4d_pair(dst + kABytes, &tmA2, a_full0 + as * 8, c0, w_base, h_base, img, 0, off_h);
          }
          __syncwarp();
          if (++as == uint32_t(p.a_stages)) {
            as = 0;
            aphase ^= 1u;
          }
          if (!p.b_resident) {
            for (int s = 0; s < p.S; s += p.b_taps) {
              if (!mbar_wait_warp(&b_empty[bs], bphase ^ 1u, abort_flag, p.status, kIncidentProducerWait, p.wait_limit)) {
                alive = false;
                break;
              }
              if (lead) {
                if (rank == 0) mbar_arrive_expect_tx(&b_full[bs], uint32_t(2 * p.b_slot));
                copy_filter(b_ring + bs * p.b_slot, b_full0 + bs * 8, n_tile, c0, r * p.s_pitch + s);
              }
              __syncwarp();
              if (++bs == uint32_t(p.b_stages)) {
                bs = 0;
                bphase ^= 1u;
              }
            }
            if (!alive) break;
          }
          if (++cb == p.c_blocks) {
            cb = 0;
            ++r;
          }
        }
      }
      if (lead && (!alive || *abort_flag)) {
        // After an incident: give copies already issued time to land.
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
      }
      __syncwarp();
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------- issuer (leader only): the whole warp walks, one lane issues
    const bool lead = elect_one();
    uint32_t as = 0, aphase = 0, bs = 0, bphase = 0, tcount = 0;
    bool alive = true;
    if (p.b_resident && pair_id < total_tiles)
      alive = mbar_wait_warp(&b_full[0], 0u, abort_flag, p.status, kIncidentMmaWaitFull, p.wait_limit);
    const uint32_t a0 = sw128_desc_lo(smem_u32(a_ring)), b0 = smem_u32(b_ring);
    const uint32_t a_empty0 = smem_u32(&a_empty[0]), b_empty0 = smem_u32(&b_empty[0]), full0 = smem_u32(&tmem_full[0]);
    constexpr uint32_t kIdesc = make_idesc(kFmt, 2 * kRows, BN);
    const uint32_t blk_idesc = make_idesc(kFmt, 2 * kRows, uint32_t(p.kg));
    const uint32_t tap_step = uint32_t(p.dil_w) * (128 / 16);    // descriptor units from one tap's rows to the next one's
    const uint32_t b_step = uint32_t(p.b_slot / p.b_taps) / (kSplit ? 32 : 16);   // ... and from its filters to the next one's
    // The loop holds the waits, the MMAs and the commits and little else: with a branch on the number of 16-channel slices
    // and 64-bit descriptors carried from tap to tap a step of four MMAs took 470 clocks whatever its width.
    auto walk = [&](auto res_tag, uint32_t d_tmem) {
      constexpr bool kRes = decltype(res_tag)::value;
      uint32_t b_at = b0;
      uint32_t acc = 0;
      auto taps = [&](uint32_t a_lo, uint32_t b_addr, int n) {
        if constexpr (BLK > 1) {
          // slice k of 16 channels belongs to group k * BLK / 4 and touches its columns only
          constexpr uint32_t kBHi = BLK == 2 ? kSw64DescHi : kSw32DescHi;
          const uint32_t part = uint32_t(p.b_slot / BLK) / 16, kg = uint32_t(p.kg);
          uint32_t b_lo = sw128_desc_lo(b_addr);
          for (int t = 0; t < n; ++t, a_lo += tap_step, b_lo += b_step / BLK) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              constexpr int kPer = 4 / BLK;                          // slices per group
              mma_f16_pair_lo<kSw128DescHi, kBHi>(d_tmem + uint32_t(k / kPer) * kg, a_lo + k * 2, b_lo + (k / kPer) * part + (k % kPer) * 2,
                                                  blk_idesc, k % kPer == 0 ? acc : 1u);
            }
            acc = 1;
          }
        } else if constexpr (kSplit) {
          // fp32 as three products of TF32 halves, smallest first
          constexpr uint32_t kALow = kABytes / 16;
          const uint32_t b_low = uint32_t(p.b_slot) / 32;
          uint32_t b_lo = sw128_desc_lo(b_addr);
          for (int t = 0; t < n; ++t, a_lo += tap_step, b_lo += b_step) {
#pragma unroll
            for (uint32_t k = 0; k < 8; k += 2) {
              mma_tf32<true>(d_tmem, a_lo + kALow + k, b_lo + k, kIdesc, k == 0 ? acc : 1u);
              mma_tf32<true>(d_tmem, a_lo + k, b_lo + b_low + k, kIdesc, 1u);
              mma_tf32<true>(d_tmem, a_lo + k, b_lo + k, kIdesc, 1u);
            }
            acc = 1;
          }
        } else {
          uint32_t b_lo = sw128_desc_lo(b_addr);
          for (int t = 0; t < n; ++t, a_lo += tap_step, b_lo += b_step) {
            mma4_f16_pair(d_tmem, a_lo, b_lo, kIdesc, acc);
            acc = 1;
          }
        }
      };
      for (int kit = 0; kit < steps; ++kit) {
        if (!mbar_wait_warp(&a_full[as], aphase, abort_flag, p.status, kIncidentMmaWaitFull, p.wait_limit)) return false;
        tc_fence_after();
        const uint32_t a_lo = a0 + as * (kAStage / 16);
        if constexpr (kRes) {
          if (lead) {
            taps(a_lo, b_at, p.S);
            tc_commit_both(a_empty0 + as * 8);
          }
          b_at += p.b_slot;
        } else {
          for (int s = 0; s < p.S; s += p.b_taps) {
            if (!mbar_wait_warp(&b_full[bs], bphase, abort_flag, p.status, kIncidentMmaWaitFull, p.wait_limit)) return false;
            tc_fence_after();
            if (lead) {
              taps(a_lo + s * tap_step, b0 + bs * p.b_slot, p.b_taps);
              tc_commit_both(b_empty0 + bs * 8);
              if (s + p.b_taps >= p.S) tc_commit_both(a_empty0 + as * 8);
            }
            __syncwarp();
            if (++bs == uint32_t(p.b_stages)) {
              bs = 0;
              bphase ^= 1u;
            }
          }
        }
        __syncwarp();
        acc = 1;
        if (++as == uint32_t(p.a_stages)) {
          as = 0;
          aphase ^= 1u;
        }
      }
      return true;
    };
    for (int tile = pair_id; tile < total_tiles && alive; tile += num_pairs, ++tcount) {
      const uint32_t buf = tcount & 1u;
      alive = mbar_wait_warp(&tmem_empty[buf], ((tcount >> 1) & 1u) ^ 1u, abort_flag, p.status, kIncidentMmaWaitTmem, p.wait_limit);
      if (!alive) break;
      tc_fence_after();
      alive = p.b_resident ? walk(std::true_type{}, tmem_base + buf * BN) : walk(std::false_type{}, tmem_base + buf * BN);
      if (alive && lead) tc_commit_both(full0 + buf * 8);
      __syncwarp();
    }
    if (lead && (!alive || *abort_flag)) {
      volatile uint32_t never = 0;
      tc_commit_pair(smem_u32(drain_bar));
      mbar_wait_bounded(drain_bar, 0u, &never, p.status, kIncidentDrainWait, kWaitLimitCycles / 16);
    }
    __syncwarp();
  }
  } else {
  warpgroup_reg_inc<kRegsEpilogue>();
  {
    // ------------------------------------------------------------ epilogue
    constexpr int WC = C::kWarpCols;
    const int ew = warp & 3;
    const int half = (warp - kFirstEpiWarp) >> 2;
    const int col_off = C::kSets == 2 ? 0 : half * WC;       // this warp's first column of the tile
    float* s_scale = epi_stage + (warp - kFirstEpiWarp) * 2 * WC;
    float* s_bias = s_scale + WC;
    const T* g_bias = static_cast<const T*>(p.bias);
    const T* g_scale = static_cast<const T*>(p.scale);
    uint8_t* my_out = out_stage + (warp - kFirstEpiWarp) * 32 * 128;
    const uint32_t tempty_leader = map_to_cta(smem_u32(&tmem_empty[0]), 0);
    const int ohp = p.OH * p.P;
    int staged_n_tile = -1;
    uint32_t tcount = 0, store_seq = 0;
    // The first pass is a rehearsal that stores nothing: it brings the drain loop's instructions in while the launch before
    // this one still runs, instead of after the first accumulator is complete (0.5 to 1 us of a launch: one 128 x 28 x 28
    // image 6.6 -> 6.1 us, 128 -> 128 3x3 in a ResNet-50 of 128 images 27.6 -> 26.1).
    bool rehearsal = !GELU;
    if (GELU) griddep_wait();
    for (int tile = pair_id; tile < total_tiles; tile += num_pairs, ++tcount) {
      if (C::kSets == 2 && !rehearsal && (tcount & 1u) != uint32_t(half)) continue;
      const int m_pair = tile / p.n_tiles;
      const int n_tile = tile - m_pair * p.n_tiles;
      const int n0 = n_tile * BN + col_off;
      const uint32_t buf = tcount & 1u;
      if (!rehearsal && n_tile != staged_n_tile) {
        __syncwarp();
        for (int j = lane; j < WC; j += 32) {
          const int col = n0 + j;
          s_scale[j] = (g_scale != nullptr && col < p.Kout) ? to_f32<T>(g_scale[col]) : 1.0f;
          s_bias[j] = (g_bias != nullptr && col < p.Kout) ? to_f32<T>(g_bias[col]) : 0.0f;
        }
        __syncwarp();
        staged_n_tile = n_tile;
      }
      const int m0 = (2 * m_pair + int(rank)) * kRows + ew * 32;
      const int m = m0 + lane;
      long long y_off = 0;
      bool row_ok = false;
      int real = 0;             // index of the output pixel
      if (m < p.M) {
        const int img = m / ohp;
        const int rem = m - img * ohp;
        const int oh = rem / p.P;
        const int ow = rem - oh * p.P;
        row_ok = ow < p.OW;
        real = (img * p.OH + oh) * p.OW + ow;
        y_off = img * p.y_sn + oh * p.y_sh + ow * p.y_sw;
      }
      if (!rehearsal) {
        bool ok = mbar_wait_bounded(&tmem_full[buf], (tcount >> 1) & 1u, abort_flag, p.status, kIncidentEpilogueWait, p.wait_limit);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
      }
      // With GELU every drain takes the same way out: two copies of erf and tanh for all values, by turns, outgrow the instruction
      // cache (64 -> 64 3x3 on 32 x 56 x 56 27.3 us by turns, 16.3 so; four groups 128 -> 256 on 85 x 56 x 56 192 and 105).
      const bool boxes = STORE == kStoreSectors && !kSplit && !GELU && p.y_rows && __all_sync(0xffffffffu, row_ok);
      row_ok = row_ok && !rehearsal;
      const uint32_t t_row = tmem_base + (uint32_t(ew * 32) << 16) + buf * BN + col_off;
      auto read_done = [&]() {   // one arrival per warp, before the last stores and without waiting for the earlier ones
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && !rehearsal) mbar_arrive_remote(tempty_leader + buf * 8);
      };
      if (boxes) {
        // 32 pixels one after another: boxes through the TMA unit
        const int pixel = __shfl_sync(0xffffffffu, real, 0);
        epilogue_store_tile<T, WC, false, 1, GELU>(t_row, n0, p.Kout, p.act, s_scale, s_bias, my_out, lane, &tmY, &tmY, pixel, 0,
                                                   rehearsal ? 0 : 32, store_seq, nullptr, g_scale != nullptr);
        read_done();
      } else if constexpr (STORE == kStoreSectors) {
        epilogue_store_sectors<T, WC, GELU>(t_row, n0, p.Kout, p.act, s_scale, s_bias, g_scale != nullptr,
                                      static_cast<T*>(p.y) + y_off + n0, row_ok, read_done);
      } else if constexpr (STORE == kStorePixels) {
        epilogue_store_pixels<T, WC, false, GELU>(t_row, n0, p.Kout, p.act, s_scale, s_bias, g_scale != nullptr,
                                            static_cast<T*>(p.y) + y_off + n0 * p.y_sk, nullptr, p.y_sk, row_ok, read_done);
      } else {
        StridedOut so = {};
        so.y = p.y;
        so.y_off = y_off;
        so.unit = p.y_unit;
        so.row_ok = row_ok;
        epilogue_store_strided<T, WC, false, 1, GELU>(t_row, n0, p.Kout, p.act, s_scale, s_bias, my_out, lane, so, store_seq);
        read_done();
      }
      if (rehearsal) {
        rehearsal = false;
        griddep_wait();   // from here on global memory is read and written
        tile -= num_pairs;
        --tcount;
      }
    }
    if (STORE == kStoreSectors && p.y_rows && lane == 0) bulk_wait_group0();   // stores must be done before the CTA retires
  }
  }

  // Neither CTA may retire while its partner can still signal its barriers or the leader's MMAs can still read its
  // shared memory.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * BN);
  }
}

// The kernels a layer may run on: 32-byte stores for all of them, the other stores for layers that are not grouped.
template <typename T, int BN, int BLK, int STORE>
cudaError_t launch_one(const CUtensorMap& tmA, const CUtensorMap& tmA2, const CUtensorMap& tmB, const CUtensorMap& tmY,
                       const RowsParams& p, int grid, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg<BN>::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // set-up may overlap the previous launch's tail
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = launch_overlap_enabled() ? 2 : 1;
  auto* kernel = p.act > 1 ? conv_rows_kernel<T, BN, BLK, STORE, true> : conv_rows_kernel<T, BN, BLK, STORE, false>;
  return cudaLaunchKernelEx(&cfg, kernel, tmA, tmA2, tmB, tmY, p);
}

template <typename T, int BN>
cudaError_t launch_bn(const CUtensorMap& tmA, const CUtensorMap& tmA2, const CUtensorMap& tmB, const CUtensorMap& tmY,
                      const RowsParams& p, int grid, cudaStream_t stream) {
  if (p.blk_groups == 1) {
    if (p.y_sk != 1) return launch_one<T, BN, 1, kStorePixels>(tmA, tmA2, tmB, tmY, p, grid, stream);
    if (p.y_unit == 32) return launch_one<T, BN, 1, kStoreSectors>(tmA, tmA2, tmB, tmY, p, grid, stream);
    return launch_one<T, BN, 1, kStoreChannels>(tmA, tmA2, tmB, tmY, p, grid, stream);
  }
  if constexpr (sizeof(T) == 2) {
    if (p.y_sk != 1 || p.y_unit != 32) return cudaErrorInvalidValue;
    if (p.blk_groups == 2) return launch_one<T, BN, 2, kStoreSectors>(tmA, tmA2, tmB, tmY, p, grid, stream);
    if constexpr (BN > 64) {   // four groups of 32 filters or more
      if (p.blk_groups == 4) return launch_one<T, BN, 4, kStoreSectors>(tmA, tmA2, tmB, tmY, p, grid, stream);
    }
  }
  return cudaErrorInvalidValue;
}

template <typename T, int BN>
cudaError_t prepare_bn() {
  auto opt_in = [](auto blk, auto store) {
    auto* plain = conv_rows_kernel<T, BN, decltype(blk)::value, decltype(store)::value, false>;
    auto* gelu = conv_rows_kernel<T, BN, decltype(blk)::value, decltype(store)::value, true>;
    cudaError_t e = cudaFuncSetAttribute(plain, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::kSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gelu, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::kSmem);
    return e;
  };
  cudaError_t e = opt_in(std::integral_constant<int, 1>{}, std::integral_constant<int, kStoreSectors>{});
  if (e == cudaSuccess) e = opt_in(std::integral_constant<int, 1>{}, std::integral_constant<int, kStoreChannels>{});
  if (e == cudaSuccess) e = opt_in(std::integral_constant<int, 1>{}, std::integral_constant<int, kStorePixels>{});
  if constexpr (sizeof(T) == 2) {
    if (e == cudaSuccess) e = opt_in(std::integral_constant<int, 2>{}, std::integral_constant<int, kStoreSectors>{});
    if constexpr (BN > 64) {
      if (e == cudaSuccess) e = opt_in(std::integral_constant<int, 4>{}, std::integral_constant<int, kStoreSectors>{});
    }
  }
  return e;
}

template <typename T>
cudaError_t launch_t(int tile_n, const CUtensorMap& tmA, const CUtensorMap& tmA2, const CUtensorMap& tmB, const CUtensorMap& tmY,
                     const RowsParams& p, int grid, cudaStream_t stream) {
  if (tile_n == 64) return launch_bn<T, 64>(tmA, tmA2, tmB, tmY, p, grid, stream);
  if (tile_n == 128) return launch_bn<T, 128>(tmA, tmA2, tmB, tmY, p, grid, stream);
  if constexpr (sizeof(T) == 2) {
    if (tile_n == 256) return launch_bn<T, 256>(tmA, tmA2, tmB, tmY, p, grid, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t rows_prepare_device() {
  cudaError_t e = prepare_bn<__half, 64>();
  if (e == cudaSuccess) e = prepare_bn<__half, 128>();
  if (e == cudaSuccess) e = prepare_bn<__half, 256>();
  if (e == cudaSuccess) e = prepare_bn<__nv_bfloat16, 64>();
  if (e == cudaSuccess) e = prepare_bn<__nv_bfloat16, 128>();
  if (e == cudaSuccess) e = prepare_bn<__nv_bfloat16, 256>();
  if (e == cudaSuccess) e = prepare_bn<float, 64>();
  if (e == cudaSuccess) e = prepare_bn<float, 128>();
  return e;
}

// Splits the operand region: the whole filter where it leaves room for four activation copies or more and there is one
// column tile, else two rings.  A filter slot holds the taps of a filter row where two of the rows' worth fit three times
// over (one wait and one commit for twelve MMAs), else one tap.
void rows_stages(RowsParams* p) {
  const int copy = kABytes * p->halves, row = p->S * p->b_bytes, filter = p->R * p->c_blocks * row;
  p->b_resident = p->n_tiles == 1 && filter <= kRingBytes - 4 * copy ? 1 : 0;
  if (p->b_resident) {
    p->b_taps = p->S;
    p->b_slot = row;
    p->b_stages = 0;
    p->a_stages = (kRingBytes - filter) / copy;
    if (p->a_stages > kMaxA) p->a_stages = kMaxA;
    return;
  }
  p->b_taps = kRingBytes / (copy + row) >= 3 ? p->S : 1;
  p->b_slot = p->b_taps * p->b_bytes;
  // the producer runs ahead by as many taps as the filter ring holds; activation copies cover as many, and one more
  for (p->a_stages = 2;; ++p->a_stages) {
    p->b_stages = (kRingBytes - p->a_stages * copy) / p->b_slot;
    if (p->b_stages > kMaxB) p->b_stages = kMaxB;
    if (p->a_stages == kMaxA || (p->a_stages - 1) * p->S >= p->b_stages * p->b_taps) break;
  }
}

cudaError_t launch_rows(int dtype, int tile_n, const CUtensorMap& tmA, const CUtensorMap& tmA2, const CUtensorMap& tmB,
                        const CUtensorMap& tmY, const RowsParams& p, int grid, cudaStream_t stream) {
  if (dtype == FDNN_F16) return launch_t<__half>(tile_n, tmA, tmA2, tmB, tmY, p, grid, stream);
  if (dtype == FDNN_BF16) return launch_t<__nv_bfloat16>(tile_n, tmA, tmA2, tmB, tmY, p, grid, stream);
  if (dtype == FDNN_F32) return launch_t<float>(tile_n, tmA, tmA2, tmB, tmY, p, grid, stream);
  return cudaErrorInvalidValue;
}

}  // namespace fdnn
