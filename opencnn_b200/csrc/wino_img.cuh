// Tensor-core Winograd kernel with the images in the accumulator rows (BF16 or TF32 operands), on CTA pairs
// (tcgen05.mma.cta_group::2): for layers with few filters or few channels.
//
// Same operator as wino_tc.cuh (it replaces the reference's Winograd_kernel,
// src/convolutionForward_32x64x8.cu:169-262, with the contraction on the tensor cores; the reference
// has no tensor-core path).  wino_pair.cuh has filters as the M dimension and 128 of them per pair, of which a layer with 64
// filters leaves half empty; and its accumulator rows are filters, so a warp's stores go to 32 output planes at once.  Here
//     D[xi] (128 image columns x 64 filters)  +=  V[xi] (128 x KC) * U[xi] (KC x 64),   M = 128, N = 64 over two SMs:
// CTA r transforms the patches of blocks 4q + 2r and 4q + 2r + 1 of 32 columns (see ColumnQuad), loads the filters
// 32*r .. 32*r+31 of the tile's 64, and its tensor memory receives
//     lanes  0-63   its 64 columns x filters  0-31 of the tile      32 accumulator columns per position
//     lanes 64-127  the same 64 columns x filters 32-63
// (the M = 128 data-path layout of cta_group::2).  Each SM computes the same 64 x 64 share as in wino_pair.cuh for half the
// filters and twice the patches, and an epilogue warp stores whole 128-byte lines: 32 images of one filter.
//
// Barriers and roles are those of wino_pair.cuh: the patches' ring is each CTA's own; "filter slice landed" and "V written"
// are barriers of the leading CTA, the tensor core's commits reach both, a drained accumulator column is reported to the
// leader, all waits are bounded, and a thread whose wait gave up reports nothing more to the leader.
//
// What bounds it: on shallow layers the latency of a tile's own patches, of which the ring holds two K-steps, and the epilogue
// warps' stores; both cost about their DRAM time on top of the rest (128x64x64x56x56 BF16 64 us: without stores 45, without patch
// loads 46, without the transform 58, without MMAs 58; TF32 69: 56, 61, 64, 62).  On deep ones the ring of two filter slices, the
// transform and the MMAs' hand-off (128x512x64x14x14 BF16 27.5 us: without the transform 22.6, without MMAs 25.3, without stores or
// patch loads 26 to 27): 0.72 us per K-step in BF16, 0.48 in TF32, where the tensor pipe needs 0.26.
#pragma once
#include "wino_pair.cuh"

namespace ocb {

template <int DT> struct ImgCfg {
  static constexpr int kKC = DT == kTcBf16 ? 16 : 8;                       // channels per K-step
  static constexpr uint32_t kRawBytes = kKC * 16 * kTcN * 4;               // one block: [c][4 h][4 w][32 columns] fp32
  static constexpr uint32_t kUBytes = 16 * 1024;                           // 16 positions x (32 filters x one K-step)
  static constexpr uint32_t kVBytes = 16 * 2048;                           // 16 positions x (64 columns x one K-step)
  static constexpr int kRawStages = DT == kTcBf16 ? 4 : 8;
  static constexpr int kUStages = 2;
  static constexpr int kVStages = 2;
  // Transform warps: four per block of columns, a thread one channel and column pair (BF16, 16 channels: two).  In TF32 a second set of
  // eight takes every other K-step (256x32x64x112x112 325 -> 302 us); in BF16 that gains nothing on shallow layers, and the registers
  // are better spent on an epilogue that reads 16 accumulator columns at a time (276 -> 266, 128x512x64x14x14 30.8 -> 29.0).
  static constexpr int kBlockWarps = 4;
  static constexpr int kTransformWarps = DT == kTcBf16 ? 8 : 16, kFirstEpilogueWarp = kPairFirstTransformWarp + kTransformWarps;
  static constexpr int kThreads = (kFirstEpilogueWarp + kTcEpilogueWarps) * 32;
  static constexpr int kEpilogueLoad = DT == kTcBf16 ? 16 : 8;       // accumulator columns per load
  static constexpr int kLaunchRegs = DT == kTcBf16 ? 96 : 72, kIssueRegs = DT == kTcBf16 ? 64 : 72,
                       kTransformRegs = 48, kEpilogueRegs = DT == kTcBf16 ? 160 : 120;
  static_assert(4 * kIssueRegs + kTransformWarps * kTransformRegs + kTcEpilogueWarps * kEpilogueRegs <= kThreads / 32 * kLaunchRegs,
                "setmaxnreg budgets exceed the registers the CTA was launched with");
  static constexpr size_t kSmemBytes = (size_t)kRawStages * kRawBytes + (size_t)kUStages * kUBytes +
                                       (size_t)kVStages * kVBytes + 512;
  static_assert(kSmemBytes <= 232448, "shared memory");
  // Transform groups of a block that take K-steps in turn.  A group has to come back to the same stages (see PairCfg::kGroups).
  static constexpr int kStepGroups = kTransformWarps / kBlockWarps / 2;
  static_assert(kRawStages % (2 * kStepGroups) == 0 && kVStages % kStepGroups == 0, "ring depths are multiples of the group count");
};
constexpr int kImgFilters = 64;                  // per tile
// Transformed values of a column pair in the operand layout: as finish_v_bf16 / finish_v_tf32, but a position holds 64 columns
// (2 KB).  BF16: rows of 128 bytes, 128-byte swizzle (16-byte chunk index ^= c & 7).  TF32: the two blocks' rows of 128 bytes
// are 1 KB apart.
template <int DT>
__device__ __forceinline__ void finish_v_wide(const uint64_t (&d)[16], uint8_t *__restrict__ vst, int block, int c, int np) {
  uint64_t b[16];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    b[j] = sub2(d[j], d[8 + j]);
    b[4 + j] = add2(d[4 + j], d[8 + j]);
    b[8 + j] = sub2(d[8 + j], d[4 + j]);
    b[12 + j] = sub2(d[4 + j], d[12 + j]);
  }
  const int n = 2 * np;
  uint8_t *dst = DT == kTcBf16 ? vst + c * 128 + ((((4 * block + (np >> 2)) ^ c) & 7) << 4) + ((np & 3) << 2)
                               : vst + block * 1024 + c * 128 + ((((n >> 3) ^ c) & 3) << 5) + ((n & 7) << 2);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint64_t o[4];
    o[0] = sub2(b[4 * i + 0], b[4 * i + 2]);
    o[1] = add2(b[4 * i + 1], b[4 * i + 2]);
    o[2] = sub2(b[4 * i + 2], b[4 * i + 1]);
    o[3] = sub2(b[4 * i + 1], b[4 * i + 3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      unpack2(o[j], lo, hi);
      if (DT == kTcBf16) *reinterpret_cast<uint32_t *>(dst + (4 * i + j) * 2048) = pack_bf16x2(lo, hi);
      else               *reinterpret_cast<float2 *>(dst + (4 * i + j) * 2048) = make_float2(round_tf32_rne(lo), round_tf32_rne(hi));
    }
  }
}

// Epilogue of one warp: 32 columns (its tensor-memory lanes; `q` is the quad of this lane's, `n` its image) x 16 filters
// (accumulator columns from `tcol`, filters from `k0`).  The same operations in the same order as tc_epilogue; every store is
// 32 lanes of one output row.
template <int W, class Release>
__device__ __forceinline__ void img_epilogue(uint32_t tcol, bool active, const WinoParams &p, int k0, const ColumnQuad &q, int n,
                                             Release release) {
  float y[4][4][4];                                                  // [filter quad][output position][filter]
  read_accumulators<W>(tcol, active, y, release);
  if (active && q.valid) {
    const int oh0 = 2 * q.ty, ow0 = 2 * q.tx;
    const bool row1 = (oh0 + 1) < p.H, col1 = (ow0 + 1) < p.W;
    const size_t dW = (size_t)p.N, dH = (size_t)p.W * p.N, plane = (size_t)p.H * dH;
    float *dst = p.y + (size_t)k0 * plane + ((size_t)oh0 * p.W + ow0) * p.N + n;
#pragma unroll
    for (int f = 0; f < 16; ++f) {
      const float(&o)[4][4] = y[f >> 2];
      dst[0] = o[0][f & 3];
      if (col1) dst[dW] = o[1][f & 3];
      if (row1) dst[dH] = o[2][f & 3];
      if (row1 && col1) dst[dH + dW] = o[3][f & 3];
      dst += plane;
    }
  }
}

// p.k_blocks counts 64-filter blocks, p.blocks blocks of 32 columns, p.total_tiles pair tiles (k_blocks times a quarter of
// those).
template <int DT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(ImgCfg<DT>::kThreads, 1)
wino_img_kernel(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_u, const WinoParams p) {
  using Cfg = ImgCfg<DT>;
  constexpr int SR = Cfg::kRawStages, SU = Cfg::kUStages, SV = Cfg::kVStages, KC = Cfg::kKC;
  extern __shared__ __align__(1024) uint8_t ismem[];
  uint8_t *raw_s = ismem;
  uint8_t *v_s = raw_s + SR * Cfg::kRawBytes;
  uint8_t *u_s = v_s + SV * Cfg::kVBytes;
  uint64_t *bars = reinterpret_cast<uint64_t *>(u_s + SU * Cfg::kUBytes);
  uint64_t *raw_full = bars, *raw_empty = raw_full + SR, *u_full = raw_empty + SR, *u_empty = u_full + SU,
           *v_ready = u_empty + SU, *v_empty = v_ready + SV;
  uint64_t *acc_full = v_empty + SV, *mma_done = acc_full + 1, *acc_empty = acc_full + 3;   // mma_done[2], acc_empty[4]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 7);
  volatile int *dead = reinterpret_cast<volatile int *>(acc_full + 8);
  uint64_t *nowhere = acc_full + 9;                    // [4]: nobody waits for these; where a thread that gave up arrives
  static_assert(SV <= 4 && (2 * SR + 2 * SU + 2 * SV + 13) * 8 <= 512, "barriers");

  const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;   // warp: uniform, as the compiler can see
  const uint32_t rank = cluster_ctarank();
  const int cid = (int)blockIdx.x >> 1, n_clusters = (int)gridDim.x >> 1;
  const int my_tiles = (p.total_tiles - cid + n_clusters - 1) / n_clusters;
  const int quads = (p.blocks + 3) / 4;                // pair tiles per filter block
  const int cpt = p.chunks_per_tile;
  const int total_steps = my_tiles * cpt;

  if (tid == 0) {
    *dead = 0;
    for (int s = 0; s < SR; ++s) {
      mbar_init(smem_u32(raw_full + s), 1);
      mbar_init(smem_u32(raw_empty + s), Cfg::kBlockWarps);
    }
    for (int s = 0; s < SU; ++s) {
      mbar_init(smem_u32(u_full + s), 1);                              // leader only: its loader, with both CTAs' bytes
      mbar_init(smem_u32(u_empty + s), 2);                             // one commit per issuing warp
    }
    for (int s = 0; s < SV; ++s) {
      mbar_init(smem_u32(v_ready + s), 2 * 8);       // leader only: the transform warps of both CTAs
      mbar_init(smem_u32(v_empty + s), 2);
    }
    mbar_init(smem_u32(acc_full), 2);
    for (int j = 0; j < 4; ++j) mbar_init(smem_u32(acc_empty + j), 2 * kTcEpilogueWarps);   // leader only
    for (int j = 0; j < 4; ++j) mbar_init(smem_u32(nowhere + j), 1);
    mbar_init(smem_u32(mma_done + 0), 1);
    mbar_init(smem_u32(mma_done + 1), 1);
    mbar_fence_init();
  }
  __syncwarp();
  if (warp == kPairMmaWarp) tmem_alloc_512_pair(smem_u32(tmem_slot));
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                     // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp >= Cfg::kFirstEpilogueWarp) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::kEpilogueRegs));
    // ===================================== epilogue ============================================
    const int quarter = warp & 3;                                        // TMEM lanes this warp may read
    const int sub = (warp - Cfg::kFirstEpilogueWarp) >> 2;                // 0 / 1: which 16 of the quarter's 32 filters
    const uint32_t tcol = tmem_base + ((uint32_t)(quarter * 32) << 16) + 16 * sub;
    uint32_t acc_empty0 = map_to_rank(smem_u32(acc_empty), 0);
    for (int seq = 0; seq < my_tiles; ++seq) {
      const int t = cid + seq * n_clusters, kb = t / quads;
      const int block = 4 * (t - kb * quads) + 2 * (int)rank + (quarter & 1);
      const ColumnQuad q = column_quad(p, 8 * block + (lane >> 2));
      mbar_wait_reporting(smem_u32(acc_full), seq & 1, dead, p.status, acc_empty0, smem_u32(nowhere));
      tc_fence_after();
      img_epilogue<Cfg::kEpilogueLoad>(tcol, block < p.blocks, p, kb * kImgFilters + 32 * (quarter >> 1) + 16 * sub, q, q.n + (lane & 3),
                   [&](int j) { mbar_arrive_cluster(acc_empty0 + 8 * j); });
    }
  } else if (warp >= kPairFirstTransformWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kTransformRegs));
    // ===================================== input transform =====================================
    const int t = (tid - 32 * kPairFirstTransformWarp) % (32 * Cfg::kBlockWarps), np = t & 15;   // column pair
    // BF16: the two channels of a warp are four apart, so that their 64-byte halves of a row lie in different banks.
    const int c = DT == kTcBf16 ? (t >> 5) + 4 * ((t >> 4) & 1) : t >> 4;
    uint32_t v_ready0 = map_to_rank(smem_u32(v_ready), 0);
    // Groups of kBlockWarps: one for each block of a K-step (TF32: of every other K-step).
    const int group = (warp - kPairFirstTransformWarp) / Cfg::kBlockWarps, b = group & 1;
    constexpr int kStepGroups = Cfg::kStepGroups;
    for (int g = group >> 1; g < total_steps; g += kStepGroups) {
      const int sv = g % SV, r = 2 * g + b, sr = r % SR;
      const uint32_t use = g / SV;
      mbar_wait_reporting(smem_u32(raw_full + sr), (r / SR) & 1, dead, p.status, v_ready0, smem_u32(nowhere));
      const float *raw = reinterpret_cast<const float *>(raw_s + sr * Cfg::kRawBytes);
      uint8_t *vst = v_s + sv * Cfg::kVBytes;
      const auto wait_for_stage = [&] {              // V stage free again
        if (use > 0) mbar_wait_reporting(smem_u32(v_empty + sv), (use - 1) & 1, dead, p.status, v_ready0, smem_u32(nowhere));
      };
      if (KC == 8) {
        uint64_t d[16];
        load_patch_pair(raw, c, np, d);
        wait_for_stage();                            // (before the load: 36 -> 40 us on 128x128x64x28x28)
        finish_v_wide<DT>(d, vst, b, c, np);
      } else {
        wait_for_stage();
#pragma unroll 1                                     // (unrolled, the second patch's registers spill: 266 -> 277 us on 256x32x64x112x112)
        for (int i = 0; i < KC; i += 8) {
          uint64_t d[16];
          load_patch_pair(raw, c + i, np, d);
          finish_v_wide<DT>(d, vst, b, c + i, np);
        }
      }
      fence_proxy_async_smem();          // V is read by the tensor core through the async proxy
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(raw_empty + sr));     // behind the fence: TMA refills the stage
        mbar_arrive_cluster(v_ready0 + 8 * sv);
      }
    }
    // the leader's commits arrive here until the end: do not leave before the last ones have
    for (int i = total_steps > SV ? total_steps - SV : 0; i < total_steps; ++i)
      mbar_wait(smem_u32(v_empty + i % SV), (i / SV) & 1, dead, p.status);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kIssueRegs));
    if (warp == 0) {
      // ===================================== patches =============================================
        load_patches<KC, SR, 2>(p, &tm_in, raw_s, raw_full, raw_empty, my_tiles, dead,
                           [&](int seq, int i) { return 4 * ((cid + seq * n_clusters) % quads) + 2 * (int)rank + i; });
    } else if (warp == 1) {
      // ===================================== filter slices =======================================
      {
        if (elect_one()) tma_prefetch_descriptor(&tm_u);
        grid_dependency_wait();   // U is all that the kernel before this one writes
        int g = 0;
        bool ok = true;
        for (int seq = 0; seq < my_tiles && ok; ++seq) {
          const int kb = (cid + seq * n_clusters) / quads;
          for (int ci = 0; ci < cpt; ++ci, ++g) {
            const int s = g % SU;
            const uint32_t use = g / SU;
            if (use > 0 && !mbar_wait_warp(smem_u32(u_empty + s), (use - 1) & 1, dead, p.status)) { ok = false; break; }
            if (!elect_one()) continue;
            if (rank == 0) mbar_arrive_expect_tx(smem_u32(u_full + s), 2 * Cfg::kUBytes);
            // U viewed as {32 filters, channel, block of 32 filters, position}
            tma_load_4d_pair(smem_u32(u_s + s * Cfg::kUBytes), &tm_u, map_to_rank(smem_u32(u_full + s), 0), 0, ci * KC,
                             2 * kb + (int)rank, 0);
          }
        }
        // The slices land before the MMAs that read them, whose completion is what these phases stand for.  (After a
        // give-up nothing completes them: their limit, in both CTAs of the pair, is the time the copies get to land.)
        for (int i = g > SU ? g - SU : 0; i < g; ++i) mbar_wait_drain(smem_u32(u_empty + i % SU), (i / SU) & 1);
      }
    } else {
      // ============================ MMA issuers (leader: two warps, two position columns each) ===
      if (rank == 0) {
        const int me = warp - kPairMmaWarp;
        const int col0 = 2 * me;                         // columns col0, col0 + 1 of the 4x4 positions, column by column
        constexpr uint32_t fmt = DT == kTcBf16 ? 1u : 2u;
        // fp32 accumulate, both operands MN-major, M = 128 and N = 64 over the pair
        constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 15) | (1u << 16) |
                                   ((uint32_t)(kImgFilters >> 3) << 17) | ((uint32_t)(4 * kTcN >> 4) << 24);
        // A: this CTA's 64 columns, as U of wino_pair.cuh.  B: its 32 filters, as V there.  The peer's lie at the same offsets.
        const uint64_t a_desc0 = DT == kTcBf16 ? smem_desc(smem_u32(v_s), 2048, 1024, 2) : smem_desc(smem_u32(v_s), 1024, 512, 1);
        const uint64_t b_desc0 = DT == kTcBf16 ? smem_desc(smem_u32(u_s), 512, 512, 4) : smem_desc(smem_u32(u_s), 1024, 512, 1);
        int ci = 0, seq = 0;
        for (int g = 0; g < total_steps; ++g) {
          const int su = g % SU, sv = g % SV;
          // A wait that gave up: stop issuing (the operands or the accumulators are not ready).
          if (!mbar_wait_warp(smem_u32(u_full + su), (g / SU) & 1, dead, p.status)) break;
          if (!mbar_wait_warp(smem_u32(v_ready + sv), (g / SV) & 1, dead, p.status)) break;
          tc_fence_after();
          const uint64_t ad = a_desc0 + (uint64_t)(sv * (Cfg::kVBytes >> 4)) + (uint64_t)(col0 * (2048 >> 4)),
                         bd = b_desc0 + (uint64_t)(su * (Cfg::kUBytes >> 4)) + (uint64_t)(col0 * (1024 >> 4));
          const uint32_t accumulate = ci > 0 ? 1u : 0u, d0 = tmem_base + col0 * kTcN;
          bool ok = true;
#pragma unroll
          for (int xo = 0; xo < 8; ++xo) {
            const int xr = 4 * (xo & 3) + (xo >> 2);     // position relative to col0: row xo & 3, column xo >> 2
            if ((xo & 3) == 0 && ci == 0 && seq > 0) {   // first write to a column of a new tile: drained in both CTAs?
              if (!mbar_wait_warp(smem_u32(acc_empty + col0 + (xo >> 2)), (seq - 1) & 1, dead, p.status)) { ok = false; break; }
              tc_fence_after();
            }
            if (elect_one()) tc_mma_pair<DT>(d0 + xr * kTcN, ad + (uint64_t)(xr * (2048 >> 4)), bd + (uint64_t)(xr * (1024 >> 4)), idesc,
                            accumulate);
          }
          if (!ok) break;
          if (elect_one()) tc_commit_both(smem_u32(v_empty + sv));
          if (elect_one()) tc_commit_both(smem_u32(u_empty + su));
          if (++ci == cpt) {
            if (elect_one()) tc_commit_both(smem_u32(acc_full));              // tile finished
            ci = 0;
            ++seq;
          }
        }
        // Tensor memory is freed at the end of the kernel: every MMA this thread issued must have completed by then.
        if (elect_one()) tc_commit_pair_local(smem_u32(mma_done + me));
        mbar_wait_drain(smem_u32(mma_done + me), 0);
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                     // nobody still reads or signals the other CTA's shared memory
  if (warp == kPairMmaWarp) {
    tc_fence_after();
    tmem_dealloc_512_pair(tmem_base);
  }
  __syncwarp();
  cluster_sync_all();                     // both halves of the allocation are given back by running CTAs
}

}  // namespace ocb
