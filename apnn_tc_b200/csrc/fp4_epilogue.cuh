// What the kernels on e2m1 operands share: parameters of the output side, the mapping of positions to output rows, and the
// epilogue of 32 channels x 32 pixels held one channel per lane.
#pragma once
#include <cstdint>

#include "apnn_device.cuh"
#include "tc5_common.cuh"

namespace apnn {
namespace fp4 {

constexpr int HALF = 128;   // channels of one CTA = TMEM lanes

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
  int splits;                  // SPLIT: pairs of a cluster that share a tile, each with its part of the K blocks
  uint32_t ring_bytes;         // shared memory of the rings (or of the partial-sum exchange, if larger)
  const float* affine_scale;   // OUT_FLOAT: out = float(value) * scale[ch] + bias[ch]
  const float* affine_bias;
  int w_resident;              // one channel tile and one K block: the R filter stages are loaded once and stay
  uint32_t idesc;
  int* error_flag;
};

// B images of H x W output positions inside Hp x Wp stored ones.
inline void set_image(Fp4Params& p, int B, int H, int W, int Hp, int Wp) {
  p.Bn = B;
  p.Ho = H;
  p.Wo = W;
  p.wp = Wp;
  p.hpwp = Hp * Wp;
  tc5::division_magic(p.hpwp, &p.magic_hpwp, &p.shift_hpwp);
  tc5::division_magic(p.wp, &p.magic_wp, &p.shift_wp);
}

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void add_shared_v4(uint32_t* v, uint32_t addr) {
  uint32_t x, y, z, w;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(addr));
  v[0] = __float_as_uint(__uint_as_float(v[0]) + __uint_as_float(x));
  v[1] = __float_as_uint(__uint_as_float(v[1]) + __uint_as_float(y));
  v[2] = __float_as_uint(__uint_as_float(v[2]) + __uint_as_float(z));
  v[3] = __float_as_uint(__uint_as_float(v[3]) + __uint_as_float(w));
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
  // code bits: 0 = both, 1 = the low bit alone, 2 = the high bit; each plane is shifted once per word and masked in place
  constexpr uint32_t M = 0x11111111u;
  const uint32_t a = p0 & p1, c = p0 & ~p1;
  return make_uint4((a & M) | ((c << 1) & (M << 1)) | ((p1 << 2) & (M << 2)), ((a >> 1) & M) | (c & (M << 1)) | ((p1 << 1) & (M << 2)),
                    ((a >> 2) & M) | ((c >> 1) & (M << 1)) | (p1 & (M << 2)),
                    ((a >> 3) & M) | ((c >> 2) & (M << 1)) | ((p1 >> 1) & (M << 2)));
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

// Negated thresholds of one channel (two-bit threshold epilogues), each in both halves of a 64-bit register; a missing one
// is -inf.  The float comparison is exact: |value| < 2^24 is a float, and rounding a larger threshold keeps its side.
struct ChannelThresholds {
  unsigned long long nt1 = 0ull, nt2 = 0xff800000ff800000ull, nt3 = 0xff800000ff800000ull;
  __device__ __forceinline__ void load(const int32_t* T, int nl) {
    nt1 = negated2((float)__ldg(T));
    if (nl > 1) {
      nt2 = negated2((float)__ldg(T + 1));
      nt3 = negated2((float)__ldg(T + 2));
    }
  }
};

// The epilogue of one chunk: v[j] = sum (a float integer) of channel ch0 + lane and pixel j, px = output row of this lane's
// pixel; rows_s: 64 words of shared memory of this warp; reload() runs as soon as v is dead (the next TMEM load).
// EPI 1: thresholds of at most two bits -> planes, int8 rows or nibble rows, no residuals; 2: the same with int16 residuals
// in and / or out, added as floats (the host checks that the sums stay below 2^24); 0: everything else.
template <int EPI, class Reload>
__device__ __forceinline__ void finish_chunk(const Fp4Params& p, uint32_t (&v)[32], const PixelRow& px, int lane, int ch0,
                                             const ChannelThresholds& thr, int nl, int* rows_s, Reload&& reload) {
  const int ch = ch0 + lane;
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
    const uint32_t b1 = below_bits(v, thr.nt1), b2 = below_bits(v, thr.nt2), b3 = below_bits(v, thr.nt3);
    reload();   // in flight during the rest of this chunk
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
    if (p.out_mode == OUT_FLOAT) {
      // two separately rounded operations per element (the CPU check computes the same two)
      const float sc = ch_ok ? __ldg(p.affine_scale + ch) : 0.0f, bi = ch_ok ? __ldg(p.affine_bias + ch) : 0.0f;
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__fadd_rn(__fmul_rn((float)(int)v[j], sc), bi));
    }
    if (p.out_mode == OUT_INT32 || p.out_mode == OUT_FLOAT) {
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
    reload();
  }
}

}  // namespace fp4
}  // namespace apnn
