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
#include "tc5_common.cuh"
#include "tc5_gemm.h"

namespace apnn {

namespace {

using namespace tc5;

constexpr int HALF = 128;               // channels of one CTA
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

struct Fp4Params {
  void* out;
  const int32_t* thresholds;
  const int32_t* residual_in;
  int32_t* residual_out;
  int N, cblocks, cin_bytes;
  int np, tiles_m, tiles_n;
  int out_mode, out_bits;
  int rows_out;                // 0: packed planes, 1: int8 rows, 2: e2m1 nibble rows
  int res16_in, res16_out;
  long long out_plane_words;
  int wp, hpwp, in_off;
  int Bn, Ho, Wo, out_halo;
  unsigned long long magic_hpwp, magic_wp;   // n / d == (n * magic) >> shift for 0 <= n < 2^31
  int shift_hpwp, shift_wp;
  uint32_t a_bytes;            // bytes of one CTA's pixel box
  uint32_t a_buf;              // its buffer, a multiple of 1024
  int na, nb;                  // ring depths: pixel boxes, filter stages
  int w_resident;              // one channel tile and one K block: the R filter stages are loaded once and stay
  uint32_t idesc;
  int* error_flag;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// Arrival that says "this warp's TMEM loads are complete" (they are: tcgen05.wait::ld has returned).  Nothing else is
// published by it, so it is relaxed: a release at cluster scope waits for every output store the warp has in flight
// (128 x 56x56, 256 -> 256 channels: 95 -> 86 us).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA tile load of a CTA pair: data lands in this CTA, the bytes complete on the leader's barrier
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
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
__device__ __forceinline__ void tmem_fill8(uint32_t taddr, uint32_t v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(v) : "memory");
}

// 32 x 32 bit transposition over the warp: bit b of lane a <-> bit a of lane b.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const uint32_t low = s == 16 ? 0x0000FFFFu : s == 8 ? 0x00FF00FFu : s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    const bool up = (lane & s) != 0;
    const uint32_t rot = __funnelshift_l(y, y, up ? 32 - s : s);
    const uint32_t keep = up ? ~low : low;
    x = (x & keep) | (rot & ~keep);
  }
  return x;
}

// Bit j of each result: v[j] (a float integer) lies below the threshold whose negation nt holds (twice).  The sign bit of
// v + nt is that bit: one packed addition per two values, one PRMT that replicates two sign bits into bytes and one masked
// OR -- compare-and-set through predicates ran at 6 clk per instruction with the two warps a scheduler has here (13-cycle
// predicate latency): 128 x 56x56, 256 -> 256 channels went from 127 to 109 us with this form and the early reload below.
__device__ __forceinline__ uint32_t below_bits(const uint32_t (&v)[32], unsigned long long nt) {
  uint32_t w[2] = {0u, 0u};
#pragma unroll
  for (int h = 0; h < 2; h++) {   // elements 16h + i and 16h + 8 + i share a PRMT
    uint32_t e[16];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      unsigned long long x, d;
      asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "r"(v[16 * h + i]), "r"(v[16 * h + i + 1]));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(nt));
      asm("mov.b64 {%0, %1}, %2;" : "=r"(e[i]), "=r"(e[i + 1]) : "l"(d));
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      uint32_t s;
      asm("prmt.b32 %0, %1, %2, 0xFBFB;" : "=r"(s) : "r"(e[i]), "r"(e[i + 8]));
      w[h] |= s & (0x0101u << (16 * h + i));
    }
  }
  return w[0] | w[1];
}
// -t in both halves; a zero threshold stays +0, so that +0 and -0 sums both land on its upper side
__device__ __forceinline__ unsigned long long negated2(float t) {
  const uint32_t u = t == 0.0f ? 0u : __float_as_uint(-t);
  return ((unsigned long long)u << 32) | u;
}

// Level words of one pixel (bit 31 - c = channel c of the 32-channel group, one word per bit) -> the pixel's 16 bytes of
// e2m1 nibbles, in expand_nibbles_kernel's order: nibble i of word q holds the element at bit 4i + q.
__device__ __forceinline__ uint4 nibbles_of(uint32_t p0, uint32_t p1) {
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t t0 = (p0 >> q) & 0x11111111u, t1 = (p1 >> q) & 0x11111111u;
    o[q] = (t1 << 2) | ((t0 & ~t1) << 1) | (t0 & t1);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void store_32(uint8_t* dst, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Accesses of one pixel's row, left out when row < 0: predicated instructions (as `if`s they became a branch each, and the
// int32 epilogue of 128 x 56x56, 256 channels took 160 us instead of 119).
__device__ __forceinline__ void st_row32(int32_t* base, int row, int pitch, uint32_t x) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p st.global.b32 [%0], %1;\n\t}" ::"l"(base + (long long)row * pitch), "r"(x),
               "r"(row)
               : "memory");
}
__device__ __forceinline__ void st_row16(int16_t* base, int row, int pitch, uint32_t x) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\t@p st.global.b16 [%0], %1;\n\t}" ::"l"(base + (long long)row * pitch),
               "h"((uint16_t)x), "r"(row)
               : "memory");
}
__device__ __forceinline__ int ld_row32(const int32_t* base, int row, int pitch) {
  int x;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.b32 %0, [%1];\n\t}"
               : "=r"(x)
               : "l"(base + (long long)row * pitch), "r"(row));
  return x;
}
__device__ __forceinline__ int ld_row16(const int16_t* base, int row, int pitch) {
  int x;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.nc.s16 %0, [%1];\n\t}"
               : "=r"(x)
               : "l"(base + (long long)row * pitch), "r"(row));
  return x;
}

struct PixelRow {
  int row;     // output row, ring included; -1 when the position is not an output pixel
  int dense;   // output row without the ring (index of the residual tensors)
};
__device__ __forceinline__ PixelRow pixel_row(const Fp4Params& p, long long pos) {
  PixelRow r = {-1, -1};
  if (pos >= 0x7fffffffLL) return r;
  const uint32_t n = (uint32_t)pos;
  const int b = (int)(((unsigned long long)n * p.magic_hpwp) >> p.shift_hpwp);
  const uint32_t rem = n - (uint32_t)b * (uint32_t)p.hpwp;
  const int ho = (int)(((unsigned long long)rem * p.magic_wp) >> p.shift_wp);
  const int wo = (int)(rem - (uint32_t)ho * (uint32_t)p.wp);
  if (b < p.Bn && ho < p.Ho && wo < p.Wo) {
    r.row = (b * (p.Ho + 2 * p.out_halo) + ho + p.out_halo) * (p.Wo + 2 * p.out_halo) + wo + p.out_halo;
    r.dense = (b * p.Ho + ho) * p.Wo + wo;
  }
  return r;
}

// EPI 1: thresholds of at most two bits -> planes, int8 rows or nibble rows, no residuals; 2: the same with int16 residuals
// in and / or out, added as floats (the host checks that the sums stay below 2^24); 0: everything else.
template <int RR, int BKB, int EPI>
__global__ void __launch_bounds__(threads_of(EPI, BKB), 1)
tc5_conv_fp4_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Fp4Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  constexpr uint32_t TAP_BYTES = HALF * BKB;
  constexpr uint32_t STAGE_BYTES = RR * TAP_BYTES;
  const uint32_t wring = base + (uint32_t)p.na * p.a_buf;
  const uint32_t bars = wring + (uint32_t)p.nb * STAGE_BYTES;
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
  const uint32_t rank = cluster_ctarank();   // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

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
        for (int cb = 0; cb < p.cblocks && ok; cb++) {
          if (!mbar_wait(xempty_bar(ia), pha ^ 1u)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(xfull_bar(ia), 2 * p.a_bytes);   // both CTAs' bytes
          tma_load_2d_pair(base + (uint32_t)ia * p.a_buf, &map_x, cb * BKB, q0, map_to_cta(xfull_bar(ia), 0));
          if (++ia == p.na) { ia = 0; pha ^= 1u; }
          int kcol = cb * BKB;
          if (p.w_resident && tile != pair) continue;
          for (int ti = 0; ti < RR; ti++) {
            if (!mbar_wait(wempty_bar(sb), phb ^ 1u)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(wfull_bar(sb), 2 * STAGE_BYTES);
            const uint32_t full = map_to_cta(wfull_bar(sb), 0);
#pragma unroll
            for (int tj = 0; tj < RR; tj++, kcol += p.cin_bytes)
              tma_load_2d_pair(wring + (uint32_t)sb * STAGE_BYTES + tj * TAP_BYTES, &map_w, kcol, wrow, full);
            if (++sb == p.nb) { sb = 0; phb ^= 1u; }
          }
        }
      }
      if (!ok) atomicExch(p.error_flag, 1);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (lane == 0 && rank == 0) {
      int ia = 0, sb = 0;
      uint32_t pha = 0, phb = 0;
      uint32_t tl = 0;
      bool ok = true;
      const uint32_t sf = tmem_base + SF_COL;
      const uint32_t row_step = (uint32_t)p.wp * (BKB / 16);
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, tl++) {
        const uint32_t acc = tl & 1u;
        const uint32_t aph = (tl >> 1) & 1u;
        if (!mbar_wait(tempty_bar(acc), aph ^ 1u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * MAX_NP;
        uint32_t enable = 0;
        for (int cb = 0; cb < p.cblocks && ok; cb++) {
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
            if (!p.w_resident) tc_commit_pair(wempty_bar(sb));   // frees the filter stage in both CTAs
            if (++sb == p.nb) { sb = 0; phb ^= 1u; }
          }
          if (ok) tc_commit_pair(xempty_bar(ia));   // frees the pixel box in both CTAs
          if (++ia == p.na) { ia = 0; pha ^= 1u; }
        }
        if (ok) tc_commit_pair(tfull_bar(acc));   // accumulators complete in both CTAs
      }
      if (!ok) atomicExch(p.error_flag, 2);
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
    // the float comparison is exact: |value| < 2^24 is a float, and rounding a larger threshold keeps its side.  A missing
    // threshold is +inf (its negation -inf).
    unsigned long long nt1 = 0ull, nt2 = 0xff800000ff800000ull, nt3 = nt2;
    int* rows_s = reinterpret_cast<int*>(smem_raw + (bars + BAR_BYTES - raw)) + (warp - 2) * 64;   // rows, then dense rows
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, tl++) {
      const int tm = tile / p.tiles_n, tn = tile - tm * p.tiles_n;
      const int ch0 = tn * TILE_CH + (int)rank * HALF + quarter * 32;   // this warp's 32 channels
      const int ch = ch0 + lane;
      if (EPI != 0 && tn != thr_tn) {
        if (ch < p.N) {
          const int32_t* T = p.thresholds + (long long)ch * nl;
          nt1 = negated2((float)__ldg(T));
          if (nl > 1) {
            nt2 = negated2((float)__ldg(T + 1));
            nt3 = negated2((float)__ldg(T + 2));
          }
        }
        thr_tn = tn;
      }
      const uint32_t acc = tl & 1u;
      const uint32_t aph = (tl >> 1) & 1u;
      if (!mbar_wait(tfull_bar(acc), aph)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * MAX_NP;
      if (ch0 < p.N) {
        uint32_t v[32];
        if (part * 32 < p.np) tmem_ld32(taddr + part * 32, v);
#pragma unroll 1
        for (int c = part; c * 32 < p.np; c += PARTS) {
          const int c_next = c + PARTS;
          // this lane's pixel of the chunk, worked out while the load is in flight
          const PixelRow px = pixel_row(p, (long long)tm * p.np + c * 32 + lane);
          tmem_ld_wait();
          if constexpr (EPI != 0) {
            if constexpr (EPI == 2) {
              // accesses are 32 consecutive channels of one pixel; the 32 pixels' rows come from shared memory.  Integers
              // become floats, and back, through the low mantissa bits of 1.5 * 2^23.
              __syncwarp();
              rows_s[32 + lane] = px.dense;
              __syncwarp();
              const int4* row4 = reinterpret_cast<const int4*>(rows_s) + 8;
              constexpr float MAGIC = 12582912.0f;   // 1.5 * 2^23
              if (ch < p.N && p.residual_in != nullptr) {
                const int16_t* R = reinterpret_cast<const int16_t*>(p.residual_in) + ch;
                auto add = [&](uint32_t& x, int r) {
                  x = __float_as_uint(__uint_as_float(x) + (__int_as_float(0x4B400000 + r) - MAGIC));
                };
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[g];
                  add(v[4 * g], ld_row16(R, d.x, p.N));
                  add(v[4 * g + 1], ld_row16(R, d.y, p.N));
                  add(v[4 * g + 2], ld_row16(R, d.z, p.N));
                  add(v[4 * g + 3], ld_row16(R, d.w, p.N));
                }
              }
              if (ch < p.N && p.residual_out != nullptr) {
                int16_t* R = reinterpret_cast<int16_t*>(p.residual_out) + ch;
                auto sat = [](uint32_t x) {
                  return __float_as_uint(fminf(fmaxf(__uint_as_float(x), -32768.0f), 32767.0f) + MAGIC);
                };
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[g];
                  st_row16(R, d.x, p.N, sat(v[4 * g]));
                  st_row16(R, d.y, p.N, sat(v[4 * g + 1]));
                  st_row16(R, d.z, p.N, sat(v[4 * g + 2]));
                  st_row16(R, d.w, p.N, sat(v[4 * g + 3]));
                }
              }
            }
            const uint32_t b1 = below_bits(v, nt1), b2 = below_bits(v, nt2), b3 = below_bits(v, nt3);
            if (c_next * 32 < p.np) tmem_ld32(taddr + c_next * 32, v);   // in flight during the rest of this chunk
            // level = number of thresholds reached, as two bit words; then one word pair per pixel
            const uint32_t p0 = __brev(transpose_bits(~(b1 ^ b2 ^ b3), lane));
            const uint32_t p1 = __brev(transpose_bits(~((b1 & b2) | (b1 & b3) | (b2 & b3)), lane));
            if (px.row >= 0) {
              if (p.rows_out == 2) {
                *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + (((long long)px.row * p.N + ch0) >> 1)) = nibbles_of(p0, p1);
              } else if (p.rows_out == 1) {
                uint32_t r[8];
#pragma unroll
                for (int q = 0; q < 8; q++) r[q] = ((p0 >> q) & 0x01010101u) | (((p1 >> q) & 0x01010101u) << 1);
                store_32(reinterpret_cast<uint8_t*>(p.out) + (long long)px.row * p.N + ch0, r);
              } else {
                uint32_t* O = reinterpret_cast<uint32_t*>(p.out) + (long long)px.row * (p.N >> 5) + (ch0 >> 5);
                O[0] = p0;
                if (p.out_bits > 1) O[p.out_plane_words] = p1;
              }
            }
            __syncwarp();
          } else {
            const bool ch_ok = ch < p.N;
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = (uint32_t)__float2int_rn(__uint_as_float(v[j]));
            // every access below is 32 consecutive channels of one pixel; the 32 pixels' rows come from shared memory
            __syncwarp();
            rows_s[lane] = px.row;
            rows_s[32 + lane] = px.dense;
            __syncwarp();
            const int4* row4 = reinterpret_cast<const int4*>(rows_s);
            if (ch_ok && p.residual_in != nullptr) {
              if (p.res16_in) {
                const int16_t* R = reinterpret_cast<const int16_t*>(p.residual_in) + ch;
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[8 + g];
                  v[4 * g] += (uint32_t)ld_row16(R, d.x, p.N);
                  v[4 * g + 1] += (uint32_t)ld_row16(R, d.y, p.N);
                  v[4 * g + 2] += (uint32_t)ld_row16(R, d.z, p.N);
                  v[4 * g + 3] += (uint32_t)ld_row16(R, d.w, p.N);
                }
              } else {
                const int32_t* R = p.residual_in + ch;
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[8 + g];
                  v[4 * g] += (uint32_t)ld_row32(R, d.x, p.N);
                  v[4 * g + 1] += (uint32_t)ld_row32(R, d.y, p.N);
                  v[4 * g + 2] += (uint32_t)ld_row32(R, d.z, p.N);
                  v[4 * g + 3] += (uint32_t)ld_row32(R, d.w, p.N);
                }
              }
            }
            if (ch_ok && p.residual_out != nullptr) {
              if (p.res16_out) {
                int16_t* R = reinterpret_cast<int16_t*>(p.residual_out) + ch;
                auto sat = [](uint32_t x) { return (uint32_t)min(max((int)x, -32768), 32767); };
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[8 + g];
                  st_row16(R, d.x, p.N, sat(v[4 * g]));
                  st_row16(R, d.y, p.N, sat(v[4 * g + 1]));
                  st_row16(R, d.z, p.N, sat(v[4 * g + 2]));
                  st_row16(R, d.w, p.N, sat(v[4 * g + 3]));
                }
              } else {
                int32_t* R = p.residual_out + ch;
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[8 + g];
                  st_row32(R, d.x, p.N, v[4 * g]);
                  st_row32(R, d.y, p.N, v[4 * g + 1]);
                  st_row32(R, d.z, p.N, v[4 * g + 2]);
                  st_row32(R, d.w, p.N, v[4 * g + 3]);
                }
              }
            }
            if (p.out_mode == OUT_INT32) {
              int32_t* D = reinterpret_cast<int32_t*>(p.out) + ch;
              if (ch_ok) {
#pragma unroll
                for (int g = 0; g < 8; g++) {
                  const int4 d = row4[g];
                  st_row32(D, d.x, p.N, v[4 * g]);
                  st_row32(D, d.y, p.N, v[4 * g + 1]);
                  st_row32(D, d.z, p.N, v[4 * g + 2]);
                  st_row32(D, d.w, p.N, v[4 * g + 3]);
                }
              }
            } else {
              // packed modes need N % 32 == 0: all 32 channels of the warp exist
              if (p.out_mode == OUT_THRESHOLDS) {
                uint32_t lv[32];
#pragma unroll
                for (int j = 0; j < 32; j++) lv[j] = 0u;
                const int32_t* T = p.thresholds + (long long)ch * nl;
#pragma unroll 1
                for (int t = 0; t < nl; t++) {
                  const int thr = __ldg(T + t);
#pragma unroll
                  for (int j = 0; j < 32; j++) lv[j] += ((int)v[j] >= thr) ? 1u : 0u;
                }
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] = lv[j];
              }
              uint32_t r[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
              uint32_t first = 0u, second = 0u;
#pragma unroll 1
              for (int b = 0; b < p.out_bits; b++) {
                uint32_t w = 0u;
#pragma unroll
                for (int j = 0; j < 32; j++) w |= ((v[j] >> b) & 1u) << j;
                const uint32_t plane = __brev(transpose_bits(w, lane));
                if (p.rows_out == 1) {
#pragma unroll
                  for (int q = 0; q < 8; q++) r[q] |= ((plane >> q) & 0x01010101u) << b;
                } else if (p.rows_out == 2) {
                  if (b == 0) first = plane;
                  else second = plane;
                } else if (px.row >= 0) {
                  reinterpret_cast<uint32_t*>(p.out)[b * p.out_plane_words + (long long)px.row * (p.N >> 5) + (ch0 >> 5)] = plane;
                }
              }
              if (px.row >= 0) {
                if (p.rows_out == 1) store_32(reinterpret_cast<uint8_t*>(p.out) + (long long)px.row * p.N + ch0, r);
                else if (p.rows_out == 2)
                  *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(p.out) + (((long long)px.row * p.N + ch0) >> 1)) =
                      nibbles_of(first, second);
              }
            }
            __syncwarp();   // lanes that skipped a store rejoin before the warp-wide TMEM load
            if (c_next * 32 < p.np) tmem_ld32(taddr + c_next * 32, v);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), 0));   // the leader's barrier
    }
    if (!ok && lane == 0) atomicExch(p.error_flag, 3);
  }

  // ---------------- tear-down ----------------
  tc_fence_before();
  __syncthreads();
  grid_launch_dependents();   // the next kernel of the stream may start its prologue
  cluster_sync_all();         // the peer may not leave while the leader's MMAs or arrivals can still reach it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512));
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// byte rows [rows][pitch], boxes of span bytes x box_rows rows, swizzle span = span (128 or 64)
bool make_rows_map(CUtensorMap* map, const void* base, long long rows, long long pitch, int box_rows, int span) {
  EncodeTiledFn fn = reinterpret_cast<EncodeTiledFn>(tensor_map_encoder());
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch};
  cuuint32_t box[2] = {(cuuint32_t)span, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// floor(n / d) == (n * magic) >> shift for every 0 <= n < 2^31 (d >= 1): with L = ceil(log2 d),
// magic = floor(2^(31+L) / d) + 1 and shift = 31 + L; magic <= 2^32, the product stays below 2^63.
void division_magic(int d, unsigned long long* magic, int* shift) {
  int L = 0;
  while ((1ll << L) < d) L++;
  *shift = 31 + L;
  *magic = ((1ull << (31 + L)) / (unsigned long long)d) + 1ull;
}

int box_rows_of(int R, int Wp, int np) { return (np / 2 + (R - 1) * (Wp + 1) + 7) / 8 * 8; }

struct Fp4Plan {
  int np;          // 0: not applicable
  long long clk;   // estimated SM clocks
};
// Tile width: waves x (MMAs of a tile, or the filter bytes they need at the rate L2 delivers, whichever is longer) plus
// the set-up and the last tile's epilogue.  Widths are multiples of 32 (whole epilogue chunks), the pixel box at most 256 rows.
Fp4Plan plan_np(long long flat_rows, int COUT, int R, int Wp, int kbytes_per_tap, int span, int sms) {
  Fp4Plan best = {0, 0};
  const long long taps = (long long)R * R * (kbytes_per_tap / span);   // filter tiles of `span` bytes
  const long long tiles_n = (COUT + TILE_CH - 1) / TILE_CH;
  const int pairs = sms / 2;
  for (int np = MAX_NP; np >= 32; np -= 32) {
    const int rows = box_rows_of(R, Wp, np);
    if (rows > 256) continue;
    const long long tiles = ((flat_rows + np - 1) / np) * tiles_n;
    const long long waves = (tiles + pairs - 1) / pairs;
    const long long mma = taps * np * 2 * span / 128;
    const long long feed = (taps * HALF * span + (long long)(kbytes_per_tap / span) * rows * span) / 54;
    const long long epi = 9LL * np;   // measured: about 2000 clk for 224 pixels
    const long long per = mma > feed ? mma : feed;
    const long long clk = waves * (per > epi ? per : epi) + epi + 6000;
    if (best.np == 0 || clk < best.clk) best = {np, clk};
  }
  return best;
}

template <int RR, int BKB, int EPI>
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
  p.w_resident = p.tiles_n == 1 && p.cblocks == 1 && nb >= RR;
  if (p.w_resident) {   // stage ti of every tile is slot ti; the boxes get the rest
    nb = RR;
    na = (room - nb * stage) / (int)p.a_buf;
    if (na > MAX_NA) na = MAX_NA;
  }
  p.na = na;
  p.nb = nb;
  const int smem = 1024 + BAR_BYTES + ROWS_BYTES + na * (int)p.a_buf + nb * stage;
  cudaError_t e = ensure_max_smem(reinterpret_cast<const void*>(tc5_conv_fp4_kernel<RR, BKB, EPI>), SMEM_LIMIT);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(threads_of(EPI, BKB), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1 + (unsigned)pdl_attribute(attr + 1);
  return cudaLaunchKernelEx(&cfg, tc5_conv_fp4_kernel<RR, BKB, EPI>, map_x, map_w, p);
}

}  // namespace

// Shapes tc5_conv_fp4 takes, and its cost estimate in SM clocks (0: not taken).
long long tc5_conv_fp4_clocks(int B, int Hin, int Win, int CIN, int COUT, int R, int in_halo, int out_halo) {
  if (CIN % 128 != 0 || (R != 1 && R != 3) || (long long)R * R * CIN * 9 >= (1ll << 24)) return 0;
  const int Hp = Hin + 2 * in_halo, Wp = Win + 2 * in_halo;
  const long long flat_rows = (long long)B * Hp * Wp;
  const long long out_rows = (long long)B * (Hin + 2 * out_halo) * (Win + 2 * out_halo);
  if (flat_rows >= 0x7fffff00LL || out_rows >= 0x7fffff00LL) return 0;
  const Fp4Plan pl = plan_np(flat_rows, COUT, R, Wp, CIN / 2, CIN % 256 == 0 ? 128 : 64, device_sm_count());
  return pl.np ? pl.clk : 0;
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
    p.res16_in = epi->residual_i16 & 1;
    p.res16_out = (epi->residual_i16 >> 1) & 1;
  }
  p.wp = Wp;
  p.hpwp = Hp * Wp;
  division_magic(p.hpwp, &p.magic_hpwp, &p.shift_hpwp);
  division_magic(p.wp, &p.magic_wp, &p.shift_wp);
  p.in_off = in_halo - pad;
  p.Bn = B;
  p.Ho = Hin;
  p.Wo = Win;
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
#define APNN_FP4_CASE(RR, SPAN) \
  (kind == 1   ? launch_fp4<RR, SPAN, 1>(s, map_x, map_w, p, pairs) \
   : kind == 2 ? launch_fp4<RR, SPAN, 2>(s, map_x, map_w, p, pairs) \
               : launch_fp4<RR, SPAN, 0>(s, map_x, map_w, p, pairs))
  if (R == 3) e = span == 128 ? APNN_FP4_CASE(3, 128) : APNN_FP4_CASE(3, 64);
  else e = span == 128 ? APNN_FP4_CASE(1, 128) : APNN_FP4_CASE(1, 64);
#undef APNN_FP4_CASE
  if (e != cudaSuccess) return cuda_fail(e, "tc5_conv_fp4 launch");
  return APNN_OK;
}

}  // namespace apnn
