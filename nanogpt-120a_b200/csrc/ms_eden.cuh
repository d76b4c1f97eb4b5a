// MS-EDEN device math shared by the tiled kernels (ms_eden_tile.cu) and the generic ones (quant_kernels.cu).
// Include only from translation units compiled with -fmad=false: one rounding per operation.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.h"

namespace nvfp4 {

// utils/quartet.rs:1-12: global scale of an MS-EDEN operand from the amax of its source.
__device__ __forceinline__ float ms_eden_scale_of_amax(float a) {
  const float so = (17.0f / 16.0f) * 0.93f;
  return (a == 0.0f) ? 1.0f : a * so / (256.0f * 6.0f);
}

// nz(decode(encode_e4m3(v))) for v >= 0: the value of the nearest E4M3 code (ties to the even
// code, saturating at 448), with zero mapped to one.  Inside the normal range [2^-6, 448) this is
// a round-to-nearest-even of the f32 mantissa at bit 20 and never zero (checked against the CPU
// restatement for every seventh f32 in the range); outside it the conversions are used.
__device__ __forceinline__ float e4m3_rounded_value_nz(float v) {
  const uint32_t bits = __float_as_uint(v);
  if (bits - 0x3c800000u < 0x43e00000u - 0x3c800000u)
    return __uint_as_float((bits + 0x0007ffffu + ((bits >> 20) & 1u)) & 0xfff00000u);
  return nz(e4m3_value(cvt_e4m3(v)));
}

// pack/scale.rs:7-30 of utils/nvfp4/quant/kernels/ms_eden.
__device__ __forceinline__ uint32_t stochastic_e4m3_scale(float value, uint32_t seed, uint32_t group) {
  // Values inside the normal E4M3 range [2^-6, 448) -- every block scale of a tensor whose groups
  // are within 2^14 of its amax -- need no conversions at all: the lower neighbour keeps the top
  // three mantissa bits, its code is (exponent, those bits) rebased, the upper neighbour is the
  // next code, and p = (value - down) / (up - down) is exactly the low 20 mantissa bits / 2^20.
  // The draw is 24 hash bits / 2^24, so `draw < p` is an integer comparison.  Identical to the
  // general path below for every value in the range (checked against the CPU restatement over
  // 7.7 million values including every grid point and its neighbours).
  const uint32_t vbits = __float_as_uint(value);
  if (vbits - 0x3c800000u < 0x43e00000u - 0x3c800000u) {
    const uint32_t draw = hash_u32(seed ^ group) & 0x00ffffffu;
    return (vbits >> 20) - 960u + (draw < ((vbits & 0x000fffffu) << 4) ? 1u : 0u);
  }
  const uint32_t cb = cvt_e4m3(value);
  const float cur = e4m3_value(cb);
  const bool above = cur > value;
  // Only the neighbour on the far side of `value` is needed: the code below when the nearest
  // code lies above the value, the code above otherwise (clamped like the reference's prev / next).
  const uint32_t ob = above ? (cb == 0 ? 0u : cb - 1u) : (cb == 255u ? 255u : cb + 1u);
  const float other = e4m3_value(ob);
  const float up = above ? cur : other;
  const float down = above ? other : cur;
  const uint32_t up_bits = above ? cb : ob;
  const uint32_t down_bits = above ? ob : cb;
  // p = (value - down) / (up - down).  Two E4M3 codes one step apart differ by +-2^e with
  // -9 <= e <= 5 unless one of them is the NaN code or the step was clamped, so the difference is
  // a power of two, zero or NaN.  For a power of two the quotient equals the product with the
  // exact reciprocal (both round the same real number); for zero the reference takes p = 0 and
  // for NaN the quotient is NaN: either way the draw is not below p and the lower code is kept.
  const uint32_t dbits = __float_as_uint(up - down);
  const uint32_t mag = dbits & 0x7fffffffu;
  const bool pow2 = (mag & 0x007fffffu) == 0u && mag - 0x00800000u <= 0x7e000000u - 0x00800000u;
  const float p = (value - down) * __uint_as_float((0x7f000000u - mag) | (dbits & 0x80000000u));
  return (pow2 && random_unit_f32(seed, group) < p) ? up_bits : down_bits;
}

// a / b by the IEEE division instruction, issued unconditionally (the compiler would otherwise
// wrap it in a branch where its result is selected away, and a branch per group costs more
// than the quotient).
__device__ __forceinline__ float div_rn_always(float a, float b) {
  float r;
  asm volatile("div.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// In-register 32-point Walsh-Hadamard butterfly in the reference's order
// (pack/hadamard.rs:6-19): stride 1,2,4,8,16; low lane a+b, high lane a-b; then * 1/sqrt(32).
// The chunk is held as 16 packed pairs P[i] = (u[i], u[i+16]): strides 1..8 act between
// registers on both halves at once (packed add / sub), stride 16 inside each register.
__device__ __forceinline__ void hadamard32_x2(f32x2_t (&P)[16]) {
#pragma unroll
  for (int stride = 1; stride < 16; stride <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if ((i & stride) == 0) {
        const f32x2_t a = P[i], b = P[i | stride];
        P[i] = add2(a, b);
        P[i | stride] = sub2(a, b);
      }
    }
  }
  const f32x2_t c = pack2(0.17677669f, 0.17677669f);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float lo, hi;
    unpack2(P[i], lo, hi);
    P[i] = mul2(pack2(lo + hi, lo - hi), c);  // after this: low lane = group 0, high lane = group 1
  }
}

// Two rotated 16-groups at once, one per packed lane (they may belong to one chunk or to two
// different chunks): block scale, RTN nibbles, EDEN correction and the stochastic scale byte
// of each (pack/payload.rs:15-69).  H points at the 16 packed values.  Returns the two scale
// bytes (low lane in bits 0..7) and the 8 nibble bytes of each lane.
__device__ __forceinline__ uint32_t ms_eden_group_lanes(const f32x2_t* H, float safe_gs, float so, float inv6,
                                                        uint32_t scale_seed, uint32_t group_lo, uint32_t group_hi,
                                                        uint2& nib_lo, uint2& nib_hi) {
  float ga0 = 0.0f, ga1 = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float a0, a1, b0, b1;
    unpack2(H[i], a0, a1);
    unpack2(H[i + 1], b0, b1);
    ga0 = max3_abs(ga0, a0, b0);
    ga1 = max3_abs(ga1, a1, b1);
  }
  const float s0a = e4m3_rounded_value_nz(ga0 * so * inv6);
  const float s0b = e4m3_rounded_value_nz(ga1 * so * inv6);
  const f32x2_t inv = pack2(inv_scale(s0a, safe_gs), inv_scale(s0b, safe_gs));
  f32x2_t x[16];
  float xa[16], xb[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    x[i] = mul2(H[i], inv);
    unpack2(x[i], xa[i], xb[i]);
  }
  nib_lo = make_uint2(cvt_e2m1x8(xa[0], xa[1], xa[2], xa[3], xa[4], xa[5], xa[6], xa[7]),
                      cvt_e2m1x8(xa[8], xa[9], xa[10], xa[11], xa[12], xa[13], xa[14], xa[15]));
  nib_hi = make_uint2(cvt_e2m1x8(xb[0], xb[1], xb[2], xb[3], xb[4], xb[5], xb[6], xb[7]),
                      cvt_e2m1x8(xb[8], xb[9], xb[10], xb[11], xb[12], xb[13], xb[14], xb[15]));
  float qa0[8], qa1[8], qb0[8], qb1[8];  // decoded nibbles: lane a / b, elements 0..7 / 8..15
  e2m1x8_values(nib_lo.x, qa0);
  e2m1x8_values(nib_lo.y, qa1);
  e2m1x8_values(nib_hi.x, qb0);
  e2m1x8_values(nib_hi.y, qb1);
  // first level of the xor-8 butterfly sums formed on the spot: entry i = e[i] + e[i + 8]
  f32x2_t num8[8], den8[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    num8[i] = add2(mul2_rounded(x[i], x[i]), mul2_rounded(x[i + 8], x[i + 8]));
    den8[i] = add2(mul2_rounded(x[i], pack2(qa0[i], qb0[i])), mul2_rounded(x[i + 8], pack2(qa1[i], qb1[i])));
  }
  float num_a, num_b, den_a, den_b;
  unpack2(add2(add2(add2(num8[0], num8[4]), add2(num8[2], num8[6])), add2(add2(num8[1], num8[5]), add2(num8[3], num8[7]))),
          num_a, num_b);
  unpack2(add2(add2(add2(den8[0], den8[4]), add2(den8[2], den8[6])), add2(add2(den8[1], den8[5]), add2(den8[3], den8[7]))),
          den_a, den_b);
  const float qa = div_rn_always(num_a, den_a), qb = div_rn_always(num_b, den_b);
  const float sa = nz(s0a * (den_a == 0.0f ? 1.0f : qa));
  const float sb = nz(s0b * (den_b == 0.0f ? 1.0f : qb));
  return stochastic_e4m3_scale(sa, scale_seed, group_lo) | (stochastic_e4m3_scale(sb, scale_seed, group_hi) << 8);
}

// Both 16-groups of one rotated chunk (low lane = group 0, high lane = group 1).
__device__ __forceinline__ uint32_t ms_eden_groups_x2(const f32x2_t (&H)[16], float safe_gs, float so, float inv6,
                                                      uint32_t scale_seed, uint32_t group0, uint4& packed) {
  uint2 lo, hi;
  const uint32_t sb = ms_eden_group_lanes(&H[0], safe_gs, so, inv6, scale_seed, group0, group0 + 1, lo, hi);
  packed = make_uint4(lo.x, lo.y, hi.x, hi.y);
  return sb;
}

// Where one orientation of an MS-EDEN result goes.
struct MsEdenOut {
  uint8_t* fp4;
  uint8_t* scales;
  float* global_scales;
  float* chunk_amax;      // optional
  uint32_t rows;          // valid output rows
  uint32_t dst_row_len;   // output K (multiple of 32)
  uint32_t scale_seed;
  uint32_t group_offset;  // added to the flat group id of the scale RNG
  uint32_t group_row_stride;  // 16-groups per row in the scale RNG's index space (dst_row_len / 16 unless sharded)
  uint32_t sign_offset;   // added to the K index of the sign hash
  int packed;             // scale bytes in the packed tile layout
};

struct MsEdenParams {
  const void* x;
  const uint8_t* src_bytes;
  const uint8_t* src_scales;
  const float* src_global;
  int src_packed;  // NVFP4 sources: scale bytes in the packed tile layout
  uint32_t a;      // F32_ROWS: src_row_len; transposed kinds: source_rows
  uint32_t b;      // transposed kinds: source_cols
  const float* global_scale_dev;
  float global_scale_host;
  int use_host_scale;
  float scale_override;
  uint32_t sign_seed;
  MsEdenOut out;
};

// Finishes one chunk whose signed inputs are in P (P[i] = (u[i], u[i+16])): rotation, two
// groups, stores.
__device__ __forceinline__ void ms_eden_emit_chunk(f32x2_t (&P)[16], const MsEdenOut& o, float gs, float so,
                                                   uint32_t row, uint32_t chunk_in_row) {
  const uint64_t chunk = static_cast<uint64_t>(row) * (o.dst_row_len >> 5) + chunk_in_row;
  hadamard32_x2(P);
  if (o.chunk_amax) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float lo, hi;
      unpack2(P[i], lo, hi);
      m = max3_abs(m, lo, hi);
    }
    o.chunk_amax[chunk] = m;
  }
  const float safe_gs = nz(gs);
  const float inv6 = inv_scale(6.0f, safe_gs);
  const uint32_t group0 = row * o.group_row_stride + chunk_in_row * 2u + o.group_offset;
  uint4 nibbles;
  const uint32_t sb = ms_eden_groups_x2(P, safe_gs, so, inv6, o.scale_seed, group0, nibbles);
  *reinterpret_cast<uint4*>(o.fp4 + chunk * 16) = nibbles;
  // two consecutive k-groups of one k-atom: adjacent bytes in either layout, 2-byte aligned
  const size_t off = o.packed ? packed_scale_offset(row, chunk_in_row * 2, o.dst_row_len >> 6) : chunk * 2;
  *reinterpret_cast<uint16_t*>(o.scales + off) = static_cast<uint16_t>(sb);
  if (chunk_in_row == 0) o.global_scales[row] = gs;
}

// Signed input pair (u[i], u[i+16]) from two values and the chunk's 32 sign bits.
__device__ __forceinline__ f32x2_t signed_pair(float lo, float hi, uint32_t neg_mask, int i) {
  const uint32_t a = __float_as_uint(lo) ^ ((neg_mask << (31 - i)) & 0x80000000u);
  const uint32_t b = __float_as_uint(hi) ^ ((neg_mask << (15 - i)) & 0x80000000u);
  return pack2(__uint_as_float(a), __uint_as_float(b));
}

// One launch of a tiled kernel (ms_eden_tile.cu, and ms_eden_tile_kernel of quant_kernels.cu).
struct MsEdenTileParams {
  const void* x;
  const uint8_t* src_bytes;
  const uint8_t* src_scales;
  const float* src_global;
  int src_packed;
  uint32_t src_rows, src_cols;
  const float* global_scale_dev;
  float global_scale_host;
  int use_host_scale;
  float scale_override;
  uint32_t sign_seed;
  MsEdenOut t;  // transposed operand: rows = src_cols, K = src_rows (padded)
  MsEdenOut r;  // row operand (pair mode): rows = src_rows, K = src_cols (padded)
  float* col_sum_partials;  // pair mode, optional: [row tiles][src_cols] column sums of each tile
  // whole-tile pair kernel, optional: take the global scale from the source amax (every thread
  // evaluates the same two operations) and publish it, instead of a one-thread kernel in between
  // (amax_count: so many partial maxima, of which NaN drop out and none counts as less than zero; 0: one word as it stands)
  const float* amax_in;
  float* gs_out;
  uint32_t amax_count = 0;
  uint4* zero = nullptr;  // pair kernel, optional: words to clear
  uint64_t zero_words = 0;
  uint32_t opaque_zero = 0;  // always 0; keeps the assembler from seeing through a pack / unpack pair (ms_eden_tile.cu)
};

bool ms_eden_pair_has_tile_form(const void* x, int dtype, uint32_t cols);
int launch_ms_eden_pair_tiles(cudaStream_t s, const MsEdenTileParams& p, int dtype, bool beside_others);
bool ms_eden_nvfp4_has_tile_form(const uint8_t* bytes, const uint8_t* scales, uint32_t cols);
int launch_ms_eden_nvfp4_tiles(cudaStream_t s, const MsEdenTileParams& p, bool rowwise);

}  // namespace nvfp4
