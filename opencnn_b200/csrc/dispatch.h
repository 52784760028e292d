// How a problem is cut up and which kernel computes it: arithmetic on sizes alone, so that it can be compiled and tested without a GPU.
// Included by abi.cu, which checks the block sizes below against the kernels'.
#pragma once
#include "../../include/opencnn_b200.h"

namespace {

constexpr int kColumns = 32;             // columns (images) of a block
constexpr int kFp32Filters = 64;         // filters of a tile of the fp32 kernel
constexpr int kTcFilters = 128;          // of the single-CTA and the CTA-pair kernel
constexpr int kImgRowFilters = 64;       // of the image-rows kernel
constexpr int kStepBf16 = 16, kStepTf32 = 8;   // channels per K-step

// Rows of 2x2-output tiles that a launch computes.
struct TileRows { int first, count; };
TileRows all_rows(int H) { return {0, (H + 1) / 2}; }


// Blocks of 32 columns of a problem (see ocb::ColumnQuad), with every tile's images filled up to a multiple of 32 or packed.
struct Columns {
  int quads_per_tile;
  long long blocks;
};
Columns columns_of(int N, TileRows rows, int W, bool packed) {
  Columns c;
  c.quads_per_tile = packed ? N / 4 : (N + kColumns - 1) / kColumns * (kColumns / 4);
  c.blocks = ((long long)rows.count * ((W + 1) / 2) * c.quads_per_tile + 7) / 8;
  return c;
}

// ---- fp32 ----
// An SM's items are item, item + grid, ...: the first SM has most.  The last round of this schedule is usually only partly filled; cutting its
// whole tiles in two (one item per consumer group) pays if the halves still fit on the SMs (see item_tile in wino_fp32.cuh), and the
// tiles of a last filter block with at most 32 filters are such halves already.  A half takes about 0.55 of a tile.
// wholes: tiles for both groups; split: the last of these, which are two items each.
struct Fp32Schedule {
  long long blocks, tiles, wholes, split, cost;
  bool packed;
};
Fp32Schedule schedule_columns(const Columns &columns, int K, int sms, bool packed) {
  const auto rounds = [&](long long items) { return (items + sms - 1) / sms; };
  const int last = K % kFp32Filters;
  Fp32Schedule s;
  s.packed = packed;
  s.blocks = columns.blocks;
  s.tiles = s.blocks * ((K + kFp32Filters - 1) / kFp32Filters);
  s.wholes = s.tiles - (last && last <= kFp32Filters / 2 ? s.blocks : 0);
  const auto cost = [&](long long split) { return 11 * rounds(s.tiles + split) + 9 * rounds(s.wholes - split); };
  const long long rest = s.wholes % sms;
  s.split = cost(rest) < cost(0) ? rest : 0;
  s.cost = cost(s.split);
  return s;
}
// A ragged batch is packed where that shortens the schedule by more than the 4 to 7 % that the copies of its crossing blocks cost the main
// loop: 48x748x352x18x7 405 -> 363 us, but 28x24x396x7x7, one round either way, 10.9 -> 12.3.
Fp32Schedule schedule_fp32(int N, TileRows rows, int W, int K, int sms) {
  const Fp32Schedule filled = schedule_columns(columns_of(N, rows, W, false), K, sms, false);
  if (N % kColumns == 0) return filled;
  const Fp32Schedule packed = schedule_columns(columns_of(N, rows, W, true), K, sms, true);
  return 106 * packed.cost < 100 * filled.cost ? packed : filled;
}

// ---- tensor cores ----
// Which tensor-core kernel a problem gets: the one with the least estimated time.  All give the same bits.  An SM (or a CTA
// pair) works through its tiles one after the other, so a kernel takes
//     start + rounds x (round + step x K-steps),   K-steps = channels / 16 (BF16) or 8 (TF32),
// and a problem much larger than L2 no less than its bytes at the rate the kernel's stores and loads were seen to reach.  The constants are
// least squares through the fused kernels' times, back to back, at 260 random sizes per type (8 to 256 images, 64 to 1024
// filters, 1 to 1024 channels, maps of 4 to 112); the estimates are 4 to 6 % off in the mean.  At 350 other random sizes per type the
// kernel chosen by them was 0.15 % behind the fastest one in the mean, and 13 % at most.  Both sides of it, us,
// single : pair : stacked : image rows:
//   few K-steps or rounds      128x32x128x28x28  BF16 22.6 : 22.6 : - : 25.2    TF32 28.7 : 24.8 : - : 28.7
//                              128x64x64x14x14   BF16 12.3 : 14.4 : 10.3 : 12.3  TF32 16.4 : 15.0 : 14.4 : 12.3
//   64 filters                 128x64x64x56x56   BF16 81.8 : 82.7 : 71.1 : 65.9  TF32 123 : 103 : 111 : 71.8
//                              256x32x64x112x112 BF16 813 : 413 : 392 : 267      TF32 552 : 477 : 490 : 300
//                              128x512x64x14x14  BF16 41.1 : 39.0 : 39.1 : 29.4  TF32 76.4 : 50.8 : 60.5 : 40.0
//   more filters, deep         128x256x256x14x14 BF16 41.0 : 33.4 : - : 43.0    TF32 62.5 : 43.0 : - : 57.4
//                              64x1024x1024x14x14 BF16 279 : 196 : - : 276      TF32 512 : 322 : - : 459
//   more filters, large output 96x4x128x99x99    BF16 174 : 131 : - : 122       TF32 188 : 131 : - : 111
// Packed columns (single-CTA kernel, batch not a multiple of 32), filled up : packed
//                              8x66x192x38x38    BF16 24.6 : 18.6               TF32 34.9 : 20.5
//                              48x83x64x9x39     BF16 14.3 : 14.6               TF32 18.7 : 20.4
struct KernelCost {
  double start, round, step;    // us
  double rate;                  // MB per us
};
constexpr double kL2Bound = 200.0;   // MB of input and output from which on the rate counts
struct TcCosts { KernelCost single, single64, pair, stacked, image_rows, packed, packed64; };   // single64: at most 64 filters
constexpr TcCosts kTcCosts[2] = {   // BF16, TF32
    {{5.8, 1.29, 0.672, 2.9}, {4.9, 1.16, 0.57, 2.9}, {6.8, 1.53, 0.487, 4.1}, {5.2, 1.63, 1.043, 4.1}, {7.1, 1.61, 0.741, 4.5}, {6.6, 1.27, 0.826, 2.9}, {6.4, 0.99, 0.65, 2.9}},
    {{5.3, 1.32, 0.576, 2.9}, {5, 1.32, 0.557, 2.9}, {6.8, 1.6, 0.338, 4.2}, {5.2, 1.79, 0.883, 4.1}, {7.1, 1.61, 0.493, 5.1}, {6.2, 1.34, 0.603, 2.9}, {6, 1.15, 0.591, 2.9}},
};

struct TcChoice { int kernel; bool packed; };
// sms: SMs; clusters: CTA pairs that fit on the device at once.
TcChoice choose_tc_kernel(bool bf16, int N, int C, TileRows rows, int W, int K, int sms, int clusters) {
  const TcCosts &costs = kTcCosts[bf16 ? 0 : 1];
  const int step = bf16 ? kStepBf16 : kStepTf32;
  const double k_steps = (C + step - 1) / step, mb = 8e-6 * N * rows.count * W * ((double)C + K);
  TcChoice best = {OPENCNN_TC_AUTO, false};
  double best_time = 0;
  const auto consider = [&](int kernel, bool packed, const KernelCost &c, long long tiles, int at_once) {
    if (at_once <= 0) return;             // (no two CTAs of this size can be co-scheduled as a cluster)
    double t = c.start + (double)((tiles + at_once - 1) / at_once) * (c.round + c.step * k_steps);
    if (mb > kL2Bound && t < mb / c.rate) t = mb / c.rate;
    if (best.kernel != OPENCNN_TC_AUTO && t >= best_time) return;
    best_time = t;
    best = {kernel, packed};
  };
  const long long blocks = columns_of(N, rows, W, false).blocks, wide = (K + kTcFilters - 1) / kTcFilters;
  consider(OPENCNN_TC_SINGLE_CTA, false, K <= 64 ? costs.single64 : costs.single, blocks * wide, sms);
  if (N % kColumns) consider(OPENCNN_TC_SINGLE_CTA, true, K <= 64 ? costs.packed64 : costs.packed, columns_of(N, rows, W, true).blocks * wide, sms);
  consider(OPENCNN_TC_PAIR_LOCAL, false, costs.pair, (blocks + 1) / 2 * wide, clusters);
  if (K <= 64) consider(OPENCNN_TC_STACKED_BLOCKS, false, costs.stacked, (blocks + 1) / 2, sms);
  consider(OPENCNN_TC_IMAGE_ROWS, false, costs.image_rows, (blocks + 3) / 4 * (K / kImgRowFilters), clusters);
  return best;
}

}  // namespace
