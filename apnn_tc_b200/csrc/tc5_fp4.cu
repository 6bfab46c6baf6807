// Flat convolution (and, with one tap, GEMM) on e2m1 operands: tcgen05 kind::mxf4 on CTA pairs.
//
// Operands are nibble rows as expand_nibbles_kernel writes them (two elements per byte): levels 0..3 and -1 / +1 are e2m1
// values, all products and partial sums small integers, exact in the fp32 accumulator below 2^24 (the host checks).
//
// The filter is the M operand: a tile is 256 output channels (128 TMEM lanes per CTA) x up to 224 flattened padded pixels
// (TMEM columns).  That orientation is what lets the 4-bit path fit: with pixels as columns the tile width is free, two
// 224-column accumulators and the scale factors share the 512 TMEM columns, and the width can be chosen so that the tiles
// fill whole waves (a 256-channel tile of the other orientation leaves no room for the second accumulator).  It also
// makes the epilogue cheap: a thread owns one channel, so its thresholds are three registers; 32 pixels of levels are
// two words that a 32 x 32 bit transposition over the warp (five shuffles) turns into the packed words of one pixel per
// lane; int32 rows and residuals are 128 contiguous bytes per warp access without staging.
//
// Positions are the flattened padded pixels q = (b*Hp + h)*Wp + w; tap (ti, tj) reads rows q + (ti+in_off)*Wp + tj+in_off
// of the flattened image.  Per K block (BKB bytes of channels) each CTA loads one box of NP/2 + (R-1)*(Wp+1) rows (its
// half of the tile's pixels plus the rows the taps reach) that all taps read through row-shifted descriptors, and its 128
// filter rows of every tap, R taps per ring stage.
//
// What it gives (B200, conv alone, thresholds -> nibble rows; int8 kernel in brackets): 128 x 28x28, 512 -> 512 channels 76 us
// (150), 128 x 56x56, 256 -> 256 86 (155), 128 -> 256 74 (115), 128 x 14x14, 512 -> 512 26 (45); 8 x 16x16, 1024 -> 1024
// 13.3 (24).
// What bounds it: per tap and 128-byte K block 4 MMAs of 256 x NP x 64 (2 NP clk) against 16 KiB of filter per SM from L2
// (about 54 B/clk arrive, 300 clk); below NP = 160 the feed, above it the tensor pipe.
//
// Synchronisation as in the int8 pair convolution: full barriers in the leader, empty barriers per CTA by multicast commit,
// tmem_empty in the leader (every epilogue warp of both CTAs).  All waits are time-bounded.  The loads carry no cluster multicast.
#include <cstdlib>
#include <cstring>

#include "api_internal.h"
#include "fp4_epilogue.cuh"
#include "tc5_common.cuh"
#include "tc5_gemm.h"

namespace apnn {

namespace {

using namespace tc5;
using namespace fp4;

constexpr int TILE_CH = 2 * HALF;       // channels of a pair's tile
constexpr int MAX_NP = 224;             // pixels of a tile: a multiple of 32
constexpr uint32_t SF_COL = 2 * MAX_NP; // 32 TMEM columns of scale factors, every byte ue8m0 1.0 (0x7F)
// Epilogue warps per CTA: each drains every (warps / 4)-th 32-pixel chunk of its TMEM lane quarter.  They are bound by
// latency (two per scheduler issue 0.3 instructions per clock).  128 x 56x56, 128 -> 256 channels (one 64-byte K block: the
// epilogue is the longer side): 78 us with 8 warps, 71 with 12 or 16; 256 -> 256 (MMAs longer): 86 with 8, 88 with 12, 91
// with 16, whose TMEM reads come between the MMAs.  The general epilogue (int32 rows: 178 against 159 us) takes 12.
constexpr int epi_warps(int EPI, int BKB) { return EPI == 1 && BKB == 128 ? 8 : 12; }
constexpr int threads_of(int EPI, int BKB) { return 32 * (2 + epi_warps(EPI, BKB)); }
constexpr int MAX_NA = 8, MAX_NB = 8;   // ring depths
constexpr int BAR_BYTES = 512;
constexpr int ROWS_BYTES = epi_warps(0, 64) * 64 * 4;   // per epilogue warp: the output rows of a chunk's 32 pixels
constexpr int SMEM_LIMIT = 232448;

// Arrival that says "this warp's TMEM loads are complete" (they are: tcgen05.wait::ld has returned).  Nothing else is
// published by it, so it is relaxed: a release at cluster scope waits for every output store the warp has in flight
// (128 x 56x56, 256 -> 256 channels: 95 -> 86 us).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// pair_mask: the two CTAs of this pair as bits of the cluster rank
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint16_t pair_mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(pair_mask)
      : "memory");
}
__device__ __forceinline__ void tc_mma_mxf4_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t sf_tmem, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sf_tmem), "r"(sf_tmem + 16u), "r"(accumulate)
      : "memory");
}

// EPI: the epilogue family of finish_chunk.
//
// SPLIT: a problem with fewer tiles than SM pairs and a long K (the fully connected layers) is launched as clusters of
// p.splits pairs that share one tile.  Each pair sums its part of the K blocks in its own TMEM; then 32-pixel chunk c goes
// to pair c % splits: the others store their partial sums of it into that pair's idle operand ring (distributed shared
// memory, one 16 KiB slot per source and chunk), and after a cluster barrier the owner adds the slots to its own sums --
// integers below 2^24, so the order does not matter -- and runs the ordinary epilogue on the chunk.
template <int RR, int BKB, int EPI, bool SPLIT>
__global__ void __launch_bounds__(threads_of(EPI, BKB), 1)
tc5_conv_fp4_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Fp4Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  constexpr uint32_t TAP_BYTES = HALF * BKB;
  constexpr uint32_t STAGE_BYTES = RR * TAP_BYTES;
  const uint32_t wring = base + (uint32_t)p.na * p.a_buf;
  const uint32_t bars = base + p.ring_bytes;
  auto xfull_bar = [&](int i) { return bars + 8u * i; };
  auto xempty_bar = [&](int i) { return bars + 8u * (MAX_NA + i); };
  auto wfull_bar = [&](int s) { return bars + 8u * (2 * MAX_NA + s); };
  auto wempty_bar = [&](int s) { return bars + 8u * (2 * MAX_NA + MAX_NB + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * MAX_NA + 2 * MAX_NB + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * MAX_NA + 2 * MAX_NB + 2 + a); };
  const uint32_t tmem_slot = bars + 8u * (2 * MAX_NA + 2 * MAX_NB + 4);
  static_assert(8 * (2 * MAX_NA + 2 * MAX_NB + 4) + 4 <= BAR_BYTES, "barrier block");
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t rank = crank & 1u;          // 0 = the pair's leader
  const uint32_t leader = SPLIT ? crank & ~1u : 0u;
  const int split = SPLIT ? (int)(crank >> 1) : 0;
  const int pair = SPLIT ? (int)blockIdx.x / (2 * p.splits) : (int)blockIdx.x >> 1;   // the pair's, or cluster's, first tile
  const int num_pairs = SPLIT ? (int)gridDim.x / (2 * p.splits) : (int)gridDim.x >> 1;
  const int cb0 = SPLIT ? split * p.cblocks / p.splits : 0;
  const int cb1 = SPLIT ? (split + 1) * p.cblocks / p.splits : p.cblocks;

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.na; i++) {
      mbar_init(xfull_bar(i), 1);
      mbar_init(xempty_bar(i), 1);
    }
    for (int s = 0; s < p.nb; s++) {
      mbar_init(wfull_bar(s), 1);
      mbar_init(wempty_bar(s), 1);
    }
    for (int a = 0; a < 2; a++) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 2 * epi_warps(EPI, BKB));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  if (warp >= 2 && warp < 6) {
    const uint32_t t0 = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + SF_COL;
#pragma unroll
    for (int i = 0; i < 4; i++) tmem_fill8(t0 + 8 * i, 0x7F7F7F7Fu);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers and scale factors exist before anything remote uses them
  tc_fence_after();
  // everything above overlapped the previous kernel's tail; from here on its results are visible
  grid_dependency_wait();
  if (threadIdx.x == 0 && blockIdx.x == 0) *p.error_flag = 0;

  const int num_tiles = p.tiles_m * p.tiles_n;

  if (warp == 0) {
    // ---------------- TMA producer (one per CTA) ----------------
    if (lane == 0) {
      int ia = 0, sb = 0;
      uint32_t pha = 0, phb = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        const int tm = tile / p.tiles_n, tn = tile - tm * p.tiles_n;
        const int q0 = tm * p.np + (int)rank * (p.np >> 1) + p.in_off * p.wp + p.in_off;
        const int wrow = tn * TILE_CH + (int)rank * HALF;
        for (int cb = cb0; cb < cb1 && ok; cb++) {
          if (!mbar_wait(xempty_bar(ia), pha ^ 1u)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(xfull_bar(ia), 2 * p.a_bytes);   // both CTAs' bytes
          tma_load_2d_pair(base + (uint32_t)ia * p.a_buf, &map_x, cb * BKB, q0, map_to_cta(xfull_bar(ia), leader));
          if (++ia == p.na) { ia = 0; pha ^= 1u; }
          int kcol = cb * BKB;
          if (p.w_resident && tile != pair) continue;
          for (int ti = 0; ti < RR; ti++) {
            if (!mbar_wait(wempty_bar(sb), phb ^ 1u)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(wfull_bar(sb), 2 * STAGE_BYTES);
            const uint32_t full = map_to_cta(wfull_bar(sb), leader);
#pragma unroll
            for (int tj = 0; tj < RR; tj++, kcol += p.cin_bytes)
              tma_load_2d_pair(wring + (uint32_t)sb * STAGE_BYTES + tj * TAP_BYTES, &map_w, kcol, wrow, full);
            if (++sb == p.nb) { sb = 0; phb ^= 1u; }
          }
        }
      }
      if (!ok) atomicExch(p.error_flag, 1);
    }
    if constexpr (SPLIT) {   // the two cluster barriers of the exchange (every thread takes part)
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (lane == 0 && rank == 0) {
      int ia = 0, sb = 0;
      uint32_t pha = 0, phb = 0;
      uint32_t tl = 0;
      bool ok = true;
      const uint32_t sf = tmem_base + SF_COL;
      const uint16_t pair_mask = (uint16_t)(3u << leader);
      const uint32_t row_step = (uint32_t)p.wp * (BKB / 16);
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, tl++) {
        const uint32_t acc = tl & 1u;
        const uint32_t aph = (tl >> 1) & 1u;
        if (!mbar_wait(tempty_bar(acc), aph ^ 1u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * MAX_NP;
        uint32_t enable = 0;
        for (int cb = cb0; cb < cb1 && ok; cb++) {
          if (!mbar_wait(xfull_bar(ia), pha)) { ok = false; break; }
          tc_fence_after();
          const uint64_t x0 = make_smem_desc_k<BKB>(base + (uint32_t)ia * p.a_buf);
#pragma unroll
          for (int ti = 0; ti < RR; ti++) {
            if (!p.w_resident || tl == 0) {
              if (!mbar_wait(wfull_bar(sb), phb)) { ok = false; break; }
              tc_fence_after();
            }
            // tap (ti, tj) reads the box from row ti*Wp + tj on: descriptors shifted by whole rows
            const uint64_t xdesc = x0 + ti * row_step;
            const uint64_t wdesc = make_smem_desc_k<BKB>(wring + (uint32_t)sb * STAGE_BYTES);
#pragma unroll
            for (int tj = 0; tj < RR; tj++) {
#pragma unroll
              for (int k = 0; k < BKB / 32; k++) {
                tc_mma_mxf4_pair(d_tmem, wdesc + tj * (TAP_BYTES / 16) + 2u * k, xdesc + tj * (BKB / 16) + 2u * k, p.idesc, sf,
                                 enable);
                enable = 1u;
              }
            }
            if (!p.w_resident) tc_commit_pair(wempty_bar(sb), pair_mask);   // frees the filter stage in both CTAs
            if (++sb == p.nb) { sb = 0; phb ^= 1u; }
          }
          if (ok) tc_commit_pair(xempty_bar(ia), pair_mask);   // frees the pixel box in both CTAs
          if (++ia == p.na) { ia = 0; pha ^= 1u; }
        }
        if (ok) tc_commit_pair(tfull_bar(acc), pair_mask);   // accumulators complete in both CTAs
      }
      if (!ok) atomicExch(p.error_flag, 2);
    }
    if constexpr (SPLIT) {
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    // ---------------- epilogue warps of both CTAs ----------------
    const int quarter = warp & 3;          // TMEM lanes 32*quarter .. +31 are the ones this warp may read
    const int part = (warp - 2) >> 2;      // this warp drains the 32-pixel chunks part, part + PARTS, ...
    constexpr int PARTS = epi_warps(EPI, BKB) / 4;
    const int nl = (1 << p.out_bits) - 1;
    uint32_t tl = 0;
    bool ok = true;
    int thr_tn = -1;
    ChannelThresholds thr;
    int* rows_s = reinterpret_cast<int*>(smem_raw + (bars + BAR_BYTES - raw)) + (warp - 2) * 64;   // rows, then dense rows
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, tl++) {
      const int tm = tile / p.tiles_n, tn = tile - tm * p.tiles_n;
      const int ch0 = tn * TILE_CH + (int)rank * HALF + quarter * 32;   // this warp's 32 channels
      if (EPI != 0 && tn != thr_tn) {
        if (ch0 + lane < p.N) thr.load(p.thresholds + (long long)(ch0 + lane) * nl, nl);
        thr_tn = tn;
      }
      const uint32_t acc = tl & 1u;
      const uint32_t aph = (tl >> 1) & 1u;
      const bool acc_ok = mbar_wait(tfull_bar(acc), aph);
      if (!acc_ok) ok = false;
      if (!SPLIT && !acc_ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * MAX_NP;
      // 16-byte groups of 4 pixels, group g of channel row r of slot n at ((8 n + g) * 128 + r) * 16
      const uint32_t slot_row = base + (uint32_t)(quarter * 32 + lane) * 16u;
      if constexpr (SPLIT) {
        __syncwarp();
        cluster_sync_all();   // every accumulator of the cluster is complete, every operand ring idle
        if (acc_ok) {
#pragma unroll 1
          for (int c = part; c * 32 < p.np; c += PARTS) {
            const int owner = c % p.splits;
            if (owner == split) continue;
            uint32_t x[32];
            tmem_ld32(taddr + c * 32, x);
            tmem_ld_wait();
            const uint32_t dst = map_to_cta(slot_row, (uint32_t)(2 * owner) | rank) +
                                 (uint32_t)((c / p.splits) * p.splits + split) * (HALF * 128u);
#pragma unroll
            for (int g = 0; g < 8; g++) st_cluster_v4(dst + (uint32_t)(g * HALF * 16), x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
          }
        }
        __syncwarp();
        cluster_sync_all();   // every slot has landed
        if (!ok) break;
      }
      if (ch0 < p.N) {
        uint32_t v[32];
        // this warp's chunks: every PARTS-th one (SPLIT: of the pair's own)
        const int c_first = SPLIT ? split + p.splits * part : part, c_step = SPLIT ? p.splits * PARTS : PARTS;
        if (!SPLIT && c_first * 32 < p.np) tmem_ld32(taddr + c_first * 32, v);
#pragma unroll 1
        for (int c = c_first; c * 32 < p.np; c += c_step) {
          const int c_next = c + c_step;
          if constexpr (SPLIT) tmem_ld32(taddr + c * 32, v);
          // this lane's pixel of the chunk, worked out while the load is in flight
          const PixelRow px = pixel_row(p, (long long)tm * p.np + c * 32 + lane);
          tmem_ld_wait();
          if constexpr (SPLIT) {
            for (int o = 0; o < p.splits; o++) {
              if (o == split) continue;
              const uint32_t src = slot_row + (uint32_t)((c / p.splits) * p.splits + o) * (HALF * 128u);
#pragma unroll
              for (int g = 0; g < 8; g++) add_shared_v4(v + 4 * g, src + (uint32_t)(g * HALF * 16));
            }
          }
          finish_chunk<EPI>(p, v, px, lane, ch0, thr, nl, rows_s, [&] {
            if (!SPLIT && c_next * 32 < p.np) tmem_ld32(taddr + c_next * 32, v);
          });
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), leader));   // the leader's barrier
    }
    if (!ok && lane == 0) atomicExch(p.error_flag, 3);
  }

  // ---------------- tear-down ----------------
  tc_fence_before();
  __syncthreads();
  grid_launch_dependents();   // the next kernel of the stream may start its prologue
  cluster_sync_all();         // the peer (SPLIT: the cluster) may not leave while the leader's MMAs or arrivals can still reach it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
}

// byte rows [rows][pitch], boxes of span bytes x box_rows rows, swizzle span = span (128 or 64)
bool make_rows_map(CUtensorMap* map, const void* base, long long rows, long long pitch, int box_rows, int span) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch};
  cuuint32_t box[2] = {(cuuint32_t)span, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int box_rows_of(int R, int Wp, int np) { return (np / 2 + (R - 1) * (Wp + 1) + 7) / 8 * 8; }

struct Fp4Plan {
  int np;          // 0: not applicable
  int splits;      // pairs of a cluster that share a tile's K
  long long clk;   // estimated SM clocks
  long long waves; // tiles of a pair
};
int fp4_cluster_capacity(int splits, int span);

// Tile width and K split: waves x (MMAs of a tile, or its operand bytes at the rate L2 delivers, whichever is longer; or
// its epilogue) plus the set-up, the last tile's epilogue and the exchange of a split.  Widths are multiples of 32 (whole
// epilogue chunks), the pixel box at most 256 rows; a split problem is one wave of resident clusters, and is taken when it
// saves a tenth.
Fp4Plan plan_np(long long flat_rows, int COUT, int R, int Wp, int kbytes_per_tap, int span, int sms) {
  Fp4Plan best = {0, 1, 0, 0};
  const long long cblocks = kbytes_per_tap / span;
  const long long tiles_n = (COUT + TILE_CH - 1) / TILE_CH;
  const int pairs = sms / 2;
  for (int splits = 1; splits <= 4 && splits * 2 <= cblocks + (splits == 1 ? 1 : 0); splits *= 2) {
    Fp4Plan here = {0, splits, 0, 0};
    const int resident = splits > 1 ? fp4_cluster_capacity(splits, span) : 0;
    for (int np = MAX_NP; np >= 32; np -= 32) {
      const int rows = box_rows_of(R, Wp, np);
      if (rows > 256) continue;
      const long long tiles = ((flat_rows + np - 1) / np) * tiles_n;
      if (splits > 1 && (tiles * splits > pairs || tiles > resident)) continue;
      const long long waves = (tiles + pairs - 1) / pairs;
      const long long kb = (cblocks + splits - 1) / splits;   // K blocks of one pair
      const long long mma = kb * R * R * np * 2 * span / 128;
      const long long feed = kb * span * ((long long)R * R * HALF + rows) / 54;
      const long long epi = 9LL * np;   // measured: about 2000 clk for 224 pixels
      long long per = mma > feed ? mma : feed;
      if (splits > 1) {   // one wave that streams the filter: about 3900 B/clk over the chip (7.3 TB/s, little L2 reuse)
        const long long stream = ((flat_rows + np - 1) / np) * COUT * R * R * kbytes_per_tap / 3900;
        if (per < stream) per = stream;
      }
      const long long clk = waves * (per > epi ? per : epi) + epi / splits + 6000 + (splits > 1 ? 2000 : 0);
      if (here.np == 0 || clk < here.clk) here = {np, splits, clk, waves};
    }
    if (here.np && (best.np == 0 || here.clk * 10 <= best.clk * 9)) best = here;
  }
  return best;
}

template <int RR, int BKB, int EPI, bool SPLIT>
cudaError_t launch_fp4(cudaStream_t s, const CUtensorMap& map_x, const CUtensorMap& map_w, Fp4Params& p, int pairs) {
  constexpr int stage = RR * HALF * BKB;
  // ring depths: filter stages take what two pixel boxes leave (one tap: as many boxes as filter tiles)
  const int room = SMEM_LIMIT - 1024 - BAR_BYTES - ROWS_BYTES;
  int na = 2, nb;
  if (RR == 1) {
    na = room / ((int)p.a_buf + stage);
    if (na > MAX_NA) na = MAX_NA;
    nb = na;
  } else {
    nb = (room - 2 * (int)p.a_buf) / stage;
    if (nb > MAX_NB) nb = MAX_NB;
    if (BKB == 64 && nb > 6) nb = 6;
    na = (room - nb * stage) / (int)p.a_buf;
    if (na > 4) na = 4;
  }
  if (na < 1 || nb < 2) return cudaErrorInvalidConfiguration;
  p.w_resident = !SPLIT && p.tiles_n == 1 && p.cblocks == 1 && nb >= RR;
  if (p.w_resident) {   // stage ti of every tile is slot ti; the boxes get the rest
    nb = RR;
    na = (room - nb * stage) / (int)p.a_buf;
    if (na > MAX_NA) na = MAX_NA;
  }
  p.na = na;
  p.nb = nb;
  int ring = na * (int)p.a_buf + nb * stage;
  const int exchange = SPLIT ? (p.np / 32 + p.splits - 1) / p.splits * p.splits * HALF * 128 : 0;
  if (ring < exchange) ring = exchange;
  if (ring > room) return cudaErrorInvalidConfiguration;
  p.ring_bytes = (uint32_t)ring;
  const int smem = 1024 + BAR_BYTES + ROWS_BYTES + (int)p.ring_bytes;
  cudaError_t e = ensure_max_smem(reinterpret_cast<const void*>(tc5_conv_fp4_kernel<RR, BKB, EPI, SPLIT>), SMEM_LIMIT);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * pairs * (SPLIT ? p.splits : 1), 1, 1);
  cfg.blockDim = dim3(threads_of(EPI, BKB), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = SPLIT ? 2 * p.splits : 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1 + (unsigned)pdl_attribute(attr + 1);
  return cudaLaunchKernelEx(&cfg, tc5_conv_fp4_kernel<RR, BKB, EPI, SPLIT>, map_x, map_w, p);
}

// How many clusters of `splits` pairs the device holds at once.
int fp4_cluster_capacity(int splits, int span) {
  const void* kernel = span == 128 ? reinterpret_cast<const void*>(tc5_conv_fp4_kernel<1, 128, 1, true>)
                                   : reinterpret_cast<const void*>(tc5_conv_fp4_kernel<1, 64, 1, true>);
  return cluster_capacity(kernel, threads_of(1, span), SMEM_LIMIT, 2 * splits);
}

template <int RR, int SPAN>
cudaError_t launch_kind(cudaStream_t s, const CUtensorMap& map_x, const CUtensorMap& map_w, Fp4Params& p, int pairs, int kind) {
  if (p.splits > 1) {   // residuals of a split problem take the general epilogue
    if (kind == 1) return launch_fp4<RR, SPAN, 1, true>(s, map_x, map_w, p, pairs);
    return launch_fp4<RR, SPAN, 0, true>(s, map_x, map_w, p, pairs);
  }
  if (kind == 1) return launch_fp4<RR, SPAN, 1, false>(s, map_x, map_w, p, pairs);
  if (kind == 2) return launch_fp4<RR, SPAN, 2, false>(s, map_x, map_w, p, pairs);
  return launch_fp4<RR, SPAN, 0, false>(s, map_x, map_w, p, pairs);
}

}  // namespace

static bool fp4_takes(int B, int Hin, int Win, int CIN, int R, int in_halo, int out_halo) {
  if (CIN % 128 != 0 || (R != 1 && R != 3) || (long long)R * R * CIN * 9 >= (1ll << 24)) return false;
  const long long flat_rows = (long long)B * (Hin + 2 * in_halo) * (Win + 2 * in_halo);
  const long long out_rows = (long long)B * (Hin + 2 * out_halo) * (Win + 2 * out_halo);
  return flat_rows < 0x7fffff00LL && out_rows < 0x7fffff00LL;
}

// Shapes tc5_conv_fp4 takes, and its cost estimate in SM clocks (0: not taken).
long long tc5_conv_fp4_clocks(int B, int Hin, int Win, int CIN, int COUT, int R, int in_halo, int out_halo) {
  if (!fp4_takes(B, Hin, Win, CIN, R, in_halo, out_halo)) return 0;
  const int Hp = Hin + 2 * in_halo, Wp = Win + 2 * in_halo;
  const Fp4Plan pl = plan_np((long long)B * Hp * Wp, COUT, R, Wp, CIN / 2, CIN % 256 == 0 ? 128 : 64, device_sm_count());
  return pl.np ? pl.clk : 0;
}

// Time of the expand pass and tc5_conv_fp4 together, for the choice between this path and int8 (i8_path_us), in us; negative
// for shapes it does not take.  Fitted to 1826 convolutions (1x1 and 3x3, 128 .. 1024 channels to 96 .. 1024, maps of 4 to
// 120) and 992 GEMMs timed on both paths, standard deviation 9 %: launches; 0.19 ns per 1000 elements expanded; per
// tile 0.5 us and its K blocks, whose 64-byte rows (CIN % 256 != 0) arrive at half the rate; the last tile's epilogue, 32
// pixels of a warp at a time.  thr2: thresholds of at most two bits, no residuals.
double tc5_conv_fp4_us(int B, int Hin, int Win, int CIN, int COUT, int R, int in_halo, int out_halo, bool thr2, long long* waves) {
  if (!fp4_takes(B, Hin, Win, CIN, R, in_halo, out_halo)) return -1.0;
  const int Hp = Hin + 2 * in_halo, Wp = Win + 2 * in_halo;
  const long long flat_rows = (long long)B * Hp * Wp;
  const int span = CIN % 256 == 0 ? 128 : 64;
  const Fp4Plan pl = plan_np(flat_rows, COUT, R, Wp, CIN / 2, span, device_sm_count());
  if (pl.np == 0) return -1.0;
  if (waves) *waves = pl.waves;
  const double elements = (double)(flat_rows + (long long)COUT * R * R) * CIN;
  const int kblocks = (CIN / 2 / span + pl.splits - 1) / pl.splits;
  const double bytes = (double)span * (R * R * HALF + box_rows_of(R, Wp, pl.np));   // operand bytes of a K block
  const double block_ns = span == 128 ? 362.0 + (R == 1 ? 0.0 : 0.0098 * bytes) : 106.0 + (R == 1 ? 0.0224 : 0.0140) * bytes;
  const int parts = epi_warps(thr2 ? 1 : 0, span) / 4;
  const int chunks = (pl.np / 32 + parts - 1) / parts;   // of a warp
  return 3.3 + 0.19e-6 * elements + pl.waves * (0.53 + 1e-3 * kblocks * block_ns) + chunks * (thr2 ? 1.45 : 2.83) / pl.splits +
         (pl.splits > 1 ? 3.4 : 0.0);
}

apnn_status tc5_conv_fp4(cudaStream_t s, const uint8_t* X4, const uint8_t* W4, void* Out, int B, int Hin, int Win, int CIN,
                         int COUT, int R, const apnn_epilogue* epi, int* status_flag) {
  const int pad = (R - 1) / 2;
  const int in_halo = (epi && epi->in_halo) ? epi->in_halo : pad;
  const int Hp = Hin + 2 * in_halo, Wp = Win + 2 * in_halo;
  const long long flat_rows = (long long)B * Hp * Wp;
  const int span = CIN % 256 == 0 ? 128 : 64;
  const int sms = device_sm_count();
  const Fp4Plan pl = plan_np(flat_rows, COUT, R, Wp, CIN / 2, span, sms);
  if (pl.np == 0 || flat_rows >= 0x7fffff00LL) return APNN_ERR_UNSUPPORTED;
  const int box_rows = box_rows_of(R, Wp, pl.np);
  CUtensorMap map_x, map_w;
  if (!make_rows_map(&map_x, X4, flat_rows, CIN / 2, box_rows, span) ||
      !make_rows_map(&map_w, W4, COUT, (long long)R * R * (CIN / 2), HALF, span))
    return cuda_fail(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
  Fp4Params p;
  memset(&p, 0, sizeof(p));
  p.out = Out;
  p.N = COUT;
  p.cin_bytes = CIN / 2;
  p.cblocks = CIN / 2 / span;
  p.np = pl.np;
  p.tiles_m = (int)((flat_rows + pl.np - 1) / pl.np);
  p.tiles_n = (COUT + TILE_CH - 1) / TILE_CH;
  p.out_mode = epi ? epi->out_mode : APNN_OUT_INT32;
  p.out_halo = epi ? epi->out_halo : 0;
  p.out_plane_words = (long long)B * (Hin + 2 * p.out_halo) * (Win + 2 * p.out_halo) * (COUT / 32);
  if (epi) {
    p.thresholds = epi->thresholds;
    p.residual_in = epi->residual_in;
    p.residual_out = epi->residual_out;
    p.out_bits = epi->out_bits;
    p.rows_out = epi->out_i8;
    p.affine_scale = epi->affine_scale;
    p.affine_bias = epi->affine_bias;
    p.res16_in = epi->residual_i16 & 1;
    p.res16_out = (epi->residual_i16 >> 1) & 1;
  }
  set_image(p, B, Hin, Win, Hp, Wp);
  p.in_off = in_halo - pad;
  p.a_bytes = (uint32_t)(box_rows * span);
  p.a_buf = (p.a_bytes + 1023u) & ~1023u;
  p.error_flag = status_flag;
  // block-scaled instruction descriptor: a / b format e2m1 (1) at bits 7 and 10, both K-major, N >> 3 at bit 17,
  // scale format ue8m0 (1) at bit 23, M >> 4 at bit 24, scale-factor ids 0
  p.idesc = (1u << 7) | (1u << 10) | ((uint32_t)(pl.np >> 3) << 17) | (1u << 23) | ((uint32_t)(TILE_CH >> 4) << 24);
  const long long tiles = (long long)p.tiles_m * p.tiles_n;
  if (tiles > 0x7fffffffLL) return APNN_ERR_UNSUPPORTED;
  const int pairs = (int)(tiles < sms / 2 ? tiles : sms / 2);
  const bool thr2 = p.out_mode == APNN_OUT_THRESHOLDS && p.out_bits <= 2;
  const bool residuals = p.residual_in || p.residual_out;
  const bool all16 = (!p.residual_in || p.res16_in) && (!p.residual_out || p.res16_out);
  const int kind = thr2 && !residuals ? 1 : thr2 && all16 && 9LL * R * R * CIN + 32768 < (1ll << 24) ? 2 : 0;
  cudaError_t e;
  p.splits = pl.splits;
  if (R == 3) e = span == 128 ? launch_kind<3, 128>(s, map_x, map_w, p, pairs, kind) : launch_kind<3, 64>(s, map_x, map_w, p, pairs, kind);
  else e = span == 128 ? launch_kind<1, 128>(s, map_x, map_w, p, pairs, kind) : launch_kind<1, 64>(s, map_x, map_w, p, pairs, kind);
  if (e != cudaSuccess) return cuda_fail(e, "tc5_conv_fp4 launch");
  return APNN_OK;
}

// D[m][n] over nibble rows A4 [M][K/2], B4 [N][K/2]: one tap, the rows of A as pixels and the rows of B as channels.
long long tc5_gemm_fp4_flat_clocks(int M, int N, int K) { return tc5_conv_fp4_clocks(1, 1, M, K, N, 1, 0, 0); }
apnn_status tc5_gemm_fp4_flat(cudaStream_t s, const uint8_t* A4, const uint8_t* B4, void* D, int M, int N, int K,
                              const apnn_epilogue* epi, int* status_flag) {
  return tc5_conv_fp4(s, A4, B4, D, 1, 1, M, K, N, 1, epi, status_flag);
}

}  // namespace apnn
