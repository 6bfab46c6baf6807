// GEMM of operands of at most two bits straight from their packed planes, one launch: the small and medium problems, where
// the expand pass and the second launch cost more than the contraction.
//
// The planes are read once per tile, spread to e2m1 nibbles in registers and written to shared memory in the layout the
// tensor core reads; tcgen05 kind::mxf4 (unit scale factors, exact integer sums below 2^24) does the rest.  A CTA owns 128
// rows of X (the output columns n, one TMEM lane each: "channels" of the shared epilogue) x up to 224 rows of W (the output
// rows m, TMEM columns: "pixels"), one tile per CTA; with few tiles and a long K a cluster of `splits` CTAs shares a tile,
// each CTA sums its part of K, and 32-row chunk c of the partial sums meets in CTA c % splits through distributed shared
// memory.
//
// A producer thread brings the planes in by TMA, 1024 k of every row per box (128-byte rows: a box costs the copy engine a
// few clocks per row, so narrow boxes would be the bound), two boxes in flight.  Eight warps spread them, K block by K block
// of 256 elements, into the 128-byte-swizzled operand stages and run the epilogue at the end; they have no global access of
// their own in flight, which their proxy fences would wait for (with private cp.async rings instead of the boxes a K block
// took 1400 clk).  One more thread issues the MMAs.  The operands need no cluster, so all those barriers are local.
//
// What bounds it: launch, first box, exchange and epilogue, 4 to 5 us together; then the spreading, about 0.5 us per K block
// (128 x 4096 x 9216, thresholds: 13.4 us, 33.5 on the warp-level kernel; 64 x 128 x 128: 3.7 against 7.5).
#include <cstdlib>
#include <cstring>

#include "api_internal.h"
#include "core_launch.h"
#include "fp4_epilogue.cuh"
#include "tc5_common.cuh"
#include "tc5_gemm.h"

namespace apnn {

namespace {

using namespace tc5;
using namespace fp4;

constexpr int MAX_NP = 224;
constexpr uint32_t SF_COL = MAX_NP;     // 32 TMEM columns of scale factors behind the accumulator
constexpr uint32_t TMEM_COLS = 256;
constexpr int WORKERS = 8;              // warps that spread and then run the epilogue
constexpr int THREADS = 32 * (WORKERS + 2);
constexpr int KB = 256;                 // elements of K per block: one 128-byte row of nibbles
constexpr int CH_BYTES = HALF * 128;    // one stage of the channel operand
constexpr int BOX_BLOCKS = 4;           // K blocks per box of packed planes
constexpr int RAW_STAGES = 2;           // boxes in flight
constexpr int BAR_BYTES = 256;
constexpr int MAX_STAGES = 4;
constexpr int ROWS_BYTES = WORKERS * 64 * 4;
constexpr int SMEM_LIMIT = 232448;

struct PlanesParams {
  Fp4Params o;              // output side; M as pixels (one image row), N as channels
  int px_signed, ch_signed; // one plane holding -1 / +1
  int kblocks;
  int stages;
  uint32_t stage_bytes;
  uint32_t raw_off;         // boxes of packed planes behind the stages
  uint32_t raw_bytes;       // of one box pair: channel planes, then pixel planes
  uint32_t bars_off;
};

__device__ __forceinline__ void tc_mma_mxf4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t sf_tmem,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(sf_tmem), "r"(sf_tmem + 16u), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// One 32-k word of BITS planes -> 16 bytes of nibbles in expand_nibbles_kernel's order (both operands share it).
template <int BITS>
__device__ __forceinline__ uint4 spread_nibbles(uint32_t w0, uint32_t w1, bool is_signed) {
  if constexpr (BITS == 2) {
    return nibbles_of(w0, w1);
  } else {
    uint32_t o[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t t = (w0 >> q) & 0x11111111u;
      // level 0 / 1 -> 0000 / 0010; bit 0 / 1 of a signed operand -> 1010 / 0010
      o[q] = is_signed ? 0xAAAAAAAAu ^ (t << 3) : t << 1;
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int PXB, int CHB, int EPI, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
tc5_planes_kernel(const __grid_constant__ CUtensorMap map_px, const __grid_constant__ CUtensorMap map_ch,
                  const __grid_constant__ PlanesParams q) {
  const Fp4Params& p = q.o;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + q.bars_off;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
  auto rfull_bar = [&](int s) { return bars + 8u * (2 * MAX_STAGES + s); };
  auto rempty_bar = [&](int s) { return bars + 8u * (2 * MAX_STAGES + RAW_STAGES + s); };
  const uint32_t tfull_bar = bars + 8u * (2 * MAX_STAGES + 2 * RAW_STAGES);
  const uint32_t tmem_slot = bars + 8u * (2 * MAX_STAGES + 2 * RAW_STAGES + 1);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - raw));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int split = SPLIT ? (int)cluster_ctarank() : 0;
  const int splits = SPLIT ? p.splits : 1;
  const int tile = (int)blockIdx.x / splits;
  const int tm = tile / p.tiles_n, tn = tile - tm * p.tiles_n;
  const int kb0 = SPLIT ? split * q.kblocks / splits : 0;
  const int kb1 = SPLIT ? (split + 1) * q.kblocks / splits : q.kblocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < q.stages; s++) {
      mbar_init(full_bar(s), WORKERS);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < RAW_STAGES; s++) {
      mbar_init(rfull_bar(s), 1);
      mbar_init(rempty_bar(s), WORKERS);
    }
    mbar_init(tfull_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // nothing global is touched before this wait (programmatic dependent launch)
  grid_dependency_wait();
  if (threadIdx.x == 0 && blockIdx.x == 0) *p.error_flag = 0;
  bool ok = true;

  if (warp == WORKERS + 1) {
    // ---------------- producer of packed planes ----------------
    __syncthreads();
    if (lane == 0) {
      int rs = 0;
      uint32_t rph = 0;
      for (int kb = kb0; kb < kb1; kb += BOX_BLOCKS) {
        if (!mbar_wait(rempty_bar(rs), rph ^ 1u)) { ok = false; break; }
        const uint32_t dst = base + q.raw_off + (uint32_t)rs * q.raw_bytes;
        mbar_expect_tx(rfull_bar(rs), q.raw_bytes);   // zero fill outside the operands counts too
        tma_load_3d(dst, &map_ch, kb * (KB / 8), tn * HALF, 0, rfull_bar(rs));
        tma_load_3d(dst + CHB * HALF * 128, &map_px, kb * (KB / 8), tm * p.np, 0, rfull_bar(rs));
        if (++rs == RAW_STAGES) { rs = 0; rph ^= 1u; }
      }
      if (!ok) atomicExch(p.error_flag, 1);
    }
    if constexpr (SPLIT) {
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  } else if (warp == WORKERS) {
    // ---------------- MMA issuer ----------------
    __syncthreads();   // the scale factors are in TMEM
    tc_fence_after();
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait(full_bar(s), ph)) { ok = false; break; }
        tc_fence_after();
        const uint64_t adesc = make_smem_desc(base + (uint32_t)s * q.stage_bytes);
        const uint64_t bdesc = make_smem_desc(base + (uint32_t)s * q.stage_bytes + CH_BYTES);
#pragma unroll
        for (int k = 0; k < 4; k++)
          tc_mma_mxf4(tmem_base, adesc + 2u * k, bdesc + 2u * k, p.idesc, tmem_base + SF_COL, (kb != kb0 || k != 0) ? 1u : 0u);
        tc_commit(empty_bar(s));
        if (++s == q.stages) { s = 0; ph ^= 1u; }
      }
      if (ok) tc_commit(tfull_bar);
      else atomicExch(p.error_flag, 2);
    }
    if constexpr (SPLIT) {
      __syncwarp();
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    // ---------------- workers: spread, then epilogue ----------------
    // pieces of this thread per K block: 128 k (half a block) of one channel row and of up to two pixel rows
    const int t = threadIdx.x;
    const int r0 = t >> 1, half = t & 1;
    bool px_used[2];
#pragma unroll
    for (int i = 0; i < 2; i++) px_used[i] = r0 + i * HALF < p.np;
    if (warp < 4) {   // scale factors, while the first bits arrive
      const uint32_t t0 = tmem_base + ((uint32_t)(warp * 32) << 16) + SF_COL;
#pragma unroll
      for (int i = 0; i < 4; i++) tmem_fill8(t0 + 8 * i, 0x7F7F7F7Fu);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    int s = 0, rs = 0;
    uint32_t ph = 0, rph = 0;
    const uint32_t px_plane = (uint32_t)p.np * 128u;
    for (int kb = kb0; kb < kb1; kb++) {
      const int sub = (kb - kb0) & (BOX_BLOCKS - 1);
      if (sub == 0) ok = mbar_wait(rfull_bar(rs), rph);
      // 16-byte chunk j of a row of the box lives at chunk j ^ (row & 7), as in the operand stages below
      uint4 c[CHB], x[2][PXB];
      const uint32_t chunk = (uint32_t)r0 * 128u + ((((uint32_t)(2 * sub + half)) ^ (uint32_t)(r0 & 7)) << 4);
      uint32_t src = base + q.raw_off + (uint32_t)rs * q.raw_bytes + chunk;
#pragma unroll
      for (int b = 0; b < CHB; b++, src += HALF * 128) c[b] = ld_shared_v4(src);
#pragma unroll
      for (int b = 0; b < PXB; b++, src += px_plane)
#pragma unroll
        for (int i = 0; i < 2; i++)
          if (px_used[i]) x[i][b] = ld_shared_v4(src + i * HALF * 128);
      if (sub == BOX_BLOCKS - 1) {   // the box is in registers
        __syncwarp();
        if (lane == 0) mbar_arrive(rempty_bar(rs));
        if (++rs == RAW_STAGES) { rs = 0; rph ^= 1u; }
      }
      if (ok) ok = mbar_wait(empty_bar(s), ph ^ 1u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      // 16-byte chunk j of a 128-byte row lives at chunk j ^ (row & 7) (128-byte swizzle); r0 and r0 + 128 agree in row & 7
      const uint32_t stage = base + (uint32_t)s * q.stage_bytes;
      const uint32_t row_s = stage + (uint32_t)r0 * 128u;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t at = (((uint32_t)(4 * half + k)) ^ (uint32_t)(r0 & 7)) << 4;
        auto word = [&](const uint4& v) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; };
        st_shared_v4(row_s + at, spread_nibbles<CHB>(word(c[0]), word(c[CHB - 1]), q.ch_signed != 0));
#pragma unroll
        for (int i = 0; i < 2; i++)
          if (px_used[i])
            st_shared_v4(row_s + CH_BYTES + i * HALF * 128 + at,
                         spread_nibbles<PXB>(word(x[i][0]), word(x[i][PXB - 1]), q.px_signed != 0));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> tensor-core reads
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(s));
      if (++s == q.stages) { s = 0; ph ^= 1u; }
    }

    // ---------------- epilogue ----------------
    const int quarter = warp & 3, part = warp >> 2;
    constexpr int PARTS = WORKERS / 4;
    const int nl = (1 << p.out_bits) - 1;
    const int ch0 = tn * HALF + quarter * 32;
    int* rows_s = reinterpret_cast<int*>(smem_raw + (bars + BAR_BYTES - raw)) + warp * 64;
    ChannelThresholds thr;
    if (EPI != 0 && ch0 + lane < p.N) thr.load(p.thresholds + (long long)(ch0 + lane) * nl, nl);
    if (ok) ok = mbar_wait(tfull_bar, 0u);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    // 16-byte groups of 4 pixels, group g of channel row r of slot n at ((8 n + g) * 128 + r) * 16
    const uint32_t slot_row = base + (uint32_t)(quarter * 32 + lane) * 16u;
    if constexpr (SPLIT) {
      __syncwarp();
      cluster_sync_all();   // every accumulator of the cluster is complete, all operand memory idle
      if (ok) {
#pragma unroll 1
        for (int c = part; c * 32 < p.np; c += PARTS) {
          const int owner = c % splits;
          if (owner == split) continue;
          uint32_t x[32];
          tmem_ld32(taddr + c * 32, x);
          tmem_ld_wait();
          const uint32_t dst = map_to_cta(slot_row, (uint32_t)owner) + (uint32_t)((c / splits) * splits + split) * (HALF * 128u);
#pragma unroll
          for (int g = 0; g < 8; g++) st_cluster_v4(dst + (uint32_t)(g * HALF * 16), x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
        }
      }
      __syncwarp();
      cluster_sync_all();   // every slot has landed
    }
    if (ok && ch0 < p.N) {
      const int c_step = splits * PARTS;
#pragma unroll 1
      for (int c = split + splits * part; c * 32 < p.np; c += c_step) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(taddr + c * 32, v);
        const PixelRow px = pixel_row(p, (long long)tm * p.np + c * 32 + lane);
        tmem_ld_wait();
        if constexpr (SPLIT) {
          for (int o = 0; o < splits; o++) {
            if (o == split) continue;
            const uint32_t src = slot_row + (uint32_t)((c / splits) * splits + o) * (HALF * 128u);
#pragma unroll
            for (int g = 0; g < 8; g++) add_shared_v4(v + 4 * g, src + (uint32_t)(g * HALF * 16));
          }
        }
        finish_chunk<EPI>(p, v, px, lane, ch0, thr, nl, rows_s, [] {});
      }
    }
    if (!ok && lane == 0) atomicExch(p.error_flag, 3);
  }

  tc_fence_before();
  __syncthreads();
  grid_launch_dependents();
  if (warp == WORKERS) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
  }
}

struct PlanesPlan {
  int np, splits;
  double us;   // estimated time, launch included
};
// Shared memory besides the operand stages.
int fixed_bytes(int pxb, int chb, int np) { return 1024 + BAR_BYTES + ROWS_BYTES + RAW_STAGES * (chb * HALF + pxb * np) * 128; }
int stages_of(int pxb, int chb, int np) {
  const int n = (SMEM_LIMIT - fixed_bytes(pxb, chb, np)) / (CH_BYTES + np * 128);
  return n < MAX_STAGES ? n : MAX_STAGES;
}
// Tile width and K split of the shortest estimated time; a split needs all its clusters resident.  The estimate is fitted to
// 2531 timed one-wave problems of w1a1, w1a2, w2a1 and w2a2 (standard deviation 9 %, split ones 4 %): per K block of 256 the
// planes to fetch and spread and the pixel columns to multiply; 32-pixel chunks of the epilogue, a warp's share of them
// one after the other; of a split the partial sums a warp sends away (1.2 us per chunk) and, per chunk kept, those it adds
// (0.46 us for each other CTA).  When sending cost a constant instead, wide tiles split eight ways were chosen: w1a1, 512 x
// 512 x 4096 took 12.7 us on 192 columns and 8 CTAs, 8.3 on 64 and 4.
PlanesPlan plan_planes(int pxb, int chb, int M, int N, int K, int sms) {
  PlanesPlan best = {0, 1, 0.0};
  const int kblocks = (K + KB - 1) / KB;
  const long long tiles_n = (N + HALF - 1) / HALF;
  for (int splits = 1; splits <= 8; splits *= 2) {
    if (splits > 1 && kblocks < 2 * splits) break;
    const int resident = splits == 1 ? 0 : cluster_capacity(reinterpret_cast<const void*>(tc5_planes_kernel<2, 2, 1, true>), THREADS, SMEM_LIMIT, splits);
    for (int np = 32; np <= MAX_NP; np += 32) {
      if (stages_of(pxb, chb, np) < 2) continue;
      const long long tiles = (((long long)M + np - 1) / np) * tiles_n;
      if (splits > 1 && tiles > resident) continue;
      const long long waves = (tiles * splits + sms - 1) / sms;
      const int chunks = np / 32, per_warp = WORKERS / 4;
      const int kept = ((chunks + splits - 1) / splits + per_warp - 1) / per_warp;
      const int sent = (chunks * (splits - 1) + splits * per_warp - 1) / (splits * per_warp);
      const double block = 0.22 + 0.0009 * np + 0.113 * (pxb * np + chb * HALF) / HALF;
      const double tile = ((kblocks + splits - 1) / splits) * block + kept * (1.13 + 0.46 * (splits - 1)) + 1.18 * sent;
      const double us = waves * (2.5 + tile);   // a further wave pays its set-up and first loads again
      if (best.np == 0 || us < best.us) best = {np, splits, us};
    }
  }
  return best;
}

template <int PXB, int CHB, int EPI, bool SPLIT>
cudaError_t launch_planes(cudaStream_t s, const CUtensorMap& map_px, const CUtensorMap& map_ch, PlanesParams& q, int tiles) {
  q.stage_bytes = (uint32_t)(CH_BYTES + q.o.np * 128);
  q.stages = stages_of(PXB, CHB, q.o.np);
  if (q.stages < 2) return cudaErrorInvalidConfiguration;
  q.raw_bytes = (uint32_t)((CHB * HALF + PXB * q.o.np) * 128);
  q.raw_off = (uint32_t)q.stages * q.stage_bytes;
  q.bars_off = q.raw_off + RAW_STAGES * q.raw_bytes;
  const int exchange = SPLIT ? (q.o.np / 32 + q.o.splits - 1) / q.o.splits * q.o.splits * HALF * 128 : 0;
  if ((int)q.bars_off < exchange) q.bars_off = (uint32_t)exchange;   // the exchange reuses stages and boxes
  const int smem = 1024 + (int)q.bars_off + BAR_BYTES + ROWS_BYTES;
  if (smem > SMEM_LIMIT) return cudaErrorInvalidConfiguration;
  cudaError_t e = ensure_max_smem(reinterpret_cast<const void*>(tc5_planes_kernel<PXB, CHB, EPI, SPLIT>), SMEM_LIMIT);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(tiles * (SPLIT ? q.o.splits : 1)), 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int na = pdl_attribute(attr);
  if (SPLIT) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)q.o.splits;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    na++;
  }
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned)na;
  return cudaLaunchKernelEx(&cfg, tc5_planes_kernel<PXB, CHB, EPI, SPLIT>, map_px, map_ch, q);
}

// planes [bits][rows][K/8 bytes]; box = 128 bytes x box_rows rows x all planes, 128-byte swizzle, zero fill outside
bool make_planes_map(CUtensorMap* map, const void* planes, long long rows, int K, int bits, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  const cuuint64_t row = (cuuint64_t)K / 8;
  cuuint64_t dims[3] = {row, (cuuint64_t)rows, (cuuint64_t)bits};
  cuuint64_t strides[2] = {row, row * (cuuint64_t)rows};
  cuuint32_t box[3] = {128, (cuuint32_t)box_rows, (cuuint32_t)bits};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(planes), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int PXB, int CHB>
cudaError_t launch_bits(cudaStream_t s, const CUtensorMap& mp, const CUtensorMap& mc, PlanesParams& q, int tiles, bool thr2) {
  if (q.o.splits > 1)
    return thr2 ? launch_planes<PXB, CHB, 1, true>(s, mp, mc, q, tiles) : launch_planes<PXB, CHB, 0, true>(s, mp, mc, q, tiles);
  return thr2 ? launch_planes<PXB, CHB, 1, false>(s, mp, mc, q, tiles) : launch_planes<PXB, CHB, 0, false>(s, mp, mc, q, tiles);
}

}  // namespace

bool tc5_gemm_planes_takes(int wbits, int xbits, int K) {
  return wbits >= 1 && wbits <= 2 && xbits >= 1 && xbits <= 2 && K % 128 == 0 && (long long)K * 9 < (1ll << 24);
}

// Whether the kernel is the fastest way to run the problem (us: this kernel / warp-level / expand pass and tcgen05).  It
// needs one wave of tiles with at most 24 K blocks each (thresholds, 128 x 4096 x 9216: 13.4 / 33.5 / 21.9; 2048 x 1024 x
// 1024: 6.7 / 30.0 / 9.6; 8192 x 64 x 2048: 8.6 / 12.2 / 11.8; two waves, 2048 x 2048 x 512: 10.5 / 27.3 / 9.6; 25 to 40 K
// blocks 0.82 to 1.3 times as fast as the best other way).  Packed outputs then always gain (64 x 1024 x 1024: 5.0 / 8.7 /
// 6.8): the warp-level epilogue takes about 4 us.  For int32 the warp-level kernel keeps the smallest (64 x 1024 x 1024: 5.2 / 4.5; 1024 x 1024 x 512: 4.9 / 5.6).
bool tc5_gemm_planes_preferred(int wbits, int xbits, int M, int N, int K, bool packed_out) {
  static const bool fp4_on = [] { const char* v = getenv("APNN_FP4"); return !(v && v[0] == '0'); }();
  if (!fp4_on || !tc5_gemm_planes_takes(wbits, xbits, K)) return false;
  const int sms = device_sm_count();
  const PlanesPlan pl = plan_planes(wbits, xbits, M, N, K, sms);
  const long long tiles = (((long long)M + pl.np - 1) / pl.np) * ((N + HALF - 1) / HALF);
  const int blocks = ((K + KB - 1) / KB + pl.splits - 1) / pl.splits;
  if (tiles * pl.splits > sms || blocks > 24) return false;
  if (packed_out) return true;
  return pl.us < core_gemm_us(wbits, xbits, M, N, K, sms);
}

apnn_status tc5_gemm_planes(cudaStream_t s, int wbits, int xbits, const uint32_t* W, const uint32_t* X, void* D, int M, int N,
                            int K, const apnn_epilogue* epi, int* status_flag) {
  const PlanesPlan pl = plan_planes(wbits, xbits, M, N, K, device_sm_count());
  CUtensorMap map_px, map_ch;
  if (!make_planes_map(&map_px, W, M, K, wbits, pl.np) || !make_planes_map(&map_ch, X, N, K, xbits, HALF))
    return cuda_fail(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
  PlanesParams q;
  memset(&q, 0, sizeof(q));
  const int sign = epi ? epi->signed_operand : APNN_SIGN_NONE;
  q.px_signed = sign == APNN_SIGN_W;
  q.ch_signed = sign == APNN_SIGN_X;
  q.kblocks = (K + KB - 1) / KB;
  Fp4Params& p = q.o;
  p.out = D;
  p.N = N;
  p.np = pl.np;
  p.splits = pl.splits;
  p.tiles_m = (M + pl.np - 1) / pl.np;
  p.tiles_n = (N + HALF - 1) / HALF;
  p.out_mode = epi ? epi->out_mode : APNN_OUT_INT32;
  p.out_plane_words = (long long)M * (N / 32);
  if (epi) {
    p.thresholds = epi->thresholds;
    p.residual_in = epi->residual_in;
    p.residual_out = epi->residual_out;
    p.out_bits = epi->out_bits;
  }
  set_image(p, 1, 1, M, 1, M);
  p.error_flag = status_flag;
  // block-scaled instruction descriptor: e2m1 operands, N >> 3 at bit 17, ue8m0 scales, M = 128
  p.idesc = (1u << 7) | (1u << 10) | ((uint32_t)(pl.np >> 3) << 17) | (1u << 23) | ((uint32_t)(HALF >> 4) << 24);
  const long long tiles = (long long)p.tiles_m * p.tiles_n;
  if (tiles * pl.splits > 0x7fffffffLL) return APNN_ERR_UNSUPPORTED;
  const bool thr2 = p.out_mode == APNN_OUT_THRESHOLDS && p.out_bits <= 2 && !p.residual_in && !p.residual_out;
  cudaError_t e = wbits == 1 ? (xbits == 1 ? launch_bits<1, 1>(s, map_px, map_ch, q, (int)tiles, thr2) : launch_bits<1, 2>(s, map_px, map_ch, q, (int)tiles, thr2))
                             : (xbits == 1 ? launch_bits<2, 1>(s, map_px, map_ch, q, (int)tiles, thr2) : launch_bits<2, 2>(s, map_px, map_ch, q, (int)tiles, thr2));
  if (e != cudaSuccess) return cuda_fail(e, "tc5_gemm_planes launch");
  return APNN_OK;
}

}  // namespace apnn
