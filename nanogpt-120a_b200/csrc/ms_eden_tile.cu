// Tiled MS-EDEN quantizers of the linear backward for sm_100a: dY (f32 / bf16) in both orientations from one
// read of it, and the transposed operand of an NVFP4 matrix (X^T, W^T).
//
// Same bytes as the generic kernels of quant_kernels.cu (one thread per 32-chunk, utils/nvfp4/quant/kernels/
// ms_eden/**), organised for the rate at which instructions issue: in the pair kernel the schedulers issue on 67 % of the
// cycles, the FMA pipe is busy 61 % of them and the ALU 37 %, HBM 25 %.  Measured costs per warp instruction and scheduler are
// 1 cycle for scalar FP32 (mixed f32 += bf16 * bf16 included, either half of a word), 2 for the packed f32x2 forms, and 2 for
// integer, logic and conversion instructions, one for the rest.  Alone, a butterfly stage beside two conversions takes 5.3
// cycles instead of 8 (beside two three-input maxima 7.7), but these kernels take the sum: of the 47.5 cycles of a scheduler for
// an element of each lane the pair kernel's FP32 accounts for 26.8, integer, logic and conversions for 17.4 and the rest for 3;
// the transposer's 31 are 14.5, 12.4 and 4.  So fewer and cheaper operations are what helps:
//  * a bf16 source is widened, sign-flipped and taken through the first butterfly stage by mixed-precision FMAs,
//    x * (+-1) + u (exact product, one rounding), which read either half of a word;
//  * the E2M1 codes are widened with add.f32.f16 instead of cvt.f32.f16;
//  * the reciprocal of a block scale, 1 / (s * gs + eps), depends on the scale byte only: a table per CTA;
//  * every range check of a chunk (corrected scale inside the normal E4M3 range, finite quotients) is folded into one
//    predicate at the end; of a chunk that fails it the pair kernel computes the scale bytes by the general code from what the
//    straight line left (general_scales), and quantizes it again from the source only for infinite sums and NaN; the
//    transposer quantizes it again from the staged values;
//    The common path is one straight line, so the chains of the 16-groups overlap; with a branch per check they did not;
//  * output addresses are a pointer per tile plus an offset per thread; the row operand leaves in 32-byte stores;
//  * warps share nothing but the table, so that they drift apart and the FP32 of one runs beside the conversions of another:
//    with a barrier per tile all began their butterflies together.
// Measured at 32768 x 2304 bf16, both orientations and column sums: 117 -> 106 us (with a barrier per tile and the upper halves
// masked out by logic instructions 117, without the logic instructions 115); HBM would allow 36 us.  In a long step the board's
// power limit takes the gain back in clock rate (1927 -> 1852 MHz): there the count of operations is what is left.
#include <atomic>

#include "ms_eden.cuh"

namespace nvfp4 {

namespace {

constexpr int kTileRows = 128, kTileCols = 64;

constexpr uint32_t kScaleCodes = 256;  // every E4M3 byte: a negative global scale or scale override gives negative codes

__device__ __forceinline__ void cp_async_16(uint32_t smem_addr, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(gmem) : "memory");
}
// bytes = 0 fills the 16 bytes with zeros without reading memory
__device__ __forceinline__ void cp_async_16_or_zero(uint32_t smem_addr, const void* gmem, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds_64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts_128(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void set_lane(f32x2_t& p, int lane, float v) {
  float lo, hi;
  unpack2(p, lo, hi);
  p = lane == 0 ? pack2(v, hi) : pack2(lo, v);
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 lds_128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// x * s + c, x and s (+-1) bf16 in the low or high halves of 32-bit words: the product is exact, so this is the sum's one
// rounding.
__device__ __forceinline__ float signed_bf16_lo(uint32_t x, uint32_t s, float c) {
  float r;
  asm("{ .reg .b16 a, b, u, v; mov.b32 {a, u}, %1; mov.b32 {b, v}, %2; fma.rn.f32.bf16 %0, a, b, %3; }"
      : "=f"(r)
      : "r"(x), "r"(s), "f"(c));
  return r;
}
__device__ __forceinline__ float signed_bf16_hi(uint32_t x, uint32_t s, float c) {
  float r;
  asm("{ .reg .b16 a, b, u, v; mov.b32 {a, u}, %1; mov.b32 {b, v}, %2; fma.rn.f32.bf16 %0, u, v, %3; }"
      : "=f"(r)
      : "r"(x), "r"(s), "f"(c));
  return r;
}
__device__ __forceinline__ float add_bf16_lo(uint32_t x, float c) {
  float r;
  asm("{ .reg .b16 a, u; mov.b32 {a, u}, %1; add.rn.f32.bf16 %0, a, %2; }" : "=f"(r) : "r"(x), "f"(c));
  return r;
}
__device__ __forceinline__ float add_bf16_hi(uint32_t x, float c) {
  float r;
  asm("{ .reg .b16 a, u; mov.b32 {a, u}, %1; add.rn.f32.bf16 %0, u, %2; }" : "=f"(r) : "r"(x), "f"(c));
  return r;
}
__device__ __forceinline__ float widen_f16_lo(uint32_t x) {
  float r;
  asm("{ .reg .b16 a, u; mov.b32 {a, u}, %1; add.rn.f32.f16 %0, a, %2; }" : "=f"(r) : "r"(x), "f"(-0.0f));
  return r;
}
__device__ __forceinline__ float widen_f16_hi(uint32_t x) {
  float r;
  asm("{ .reg .b16 a, u; mov.b32 {a, u}, %1; add.rn.f32.f16 %0, u, %2; }" : "=f"(r) : "r"(x), "f"(-0.0f));
  return r;
}

// Stochastic E4M3 code of a value in [2^-6, 448): lower neighbour plus one with probability (low 20 mantissa bits) /
// 2^20, drawn as 24 hash bits < low bits * 16 (ms_eden.cuh: stochastic_e4m3_scale, same comparison shifted up by 8).
__device__ __forceinline__ uint32_t stochastic_code(uint32_t value_bits, uint32_t seed, uint32_t group) {
  const uint32_t draw = hash_u32(seed ^ group) << 8;
  return (value_bits >> 20) - 960u + (draw < (value_bits << 12) ? 1u : 0u);
}

// Stride-1 butterfly of the signed values of two bf16 words (a, b) with sign words (sa, sb): low halves ...
__device__ __forceinline__ void first_stage_lo(uint32_t a, uint32_t b, uint32_t sa, uint32_t sb, float& sum, float& diff) {
  const float ub = signed_bf16_lo(b, sb, -0.0f);
  sum = signed_bf16_lo(a, sa, ub);
  diff = signed_bf16_lo(a, sa, -ub);
}
// ... and high halves.
__device__ __forceinline__ void first_stage_hi(uint32_t a, uint32_t b, uint32_t sa, uint32_t sb, float& sum, float& diff) {
  const float ub = signed_bf16_hi(b, sb, -0.0f);
  sum = signed_bf16_hi(a, sa, ub);
  diff = signed_bf16_hi(a, sa, -ub);
}

// Two chunks of one thread, one per packed lane.
struct PairCode {
  uint4 lo, hi;      // nibble bytes of the low-lane and the high-lane chunk
  uint32_t scales;   // scale bytes: low-lane chunk in bits 0..15, high-lane chunk in bits 16..31 (group 0, group 1)
  float amax_lo, amax_hi;
  bool ok;           // false: some corrected scale lies outside the straight-line path's range, `scales` is not valid
  float corrected[4];  // corrected scale of each group, in the order of the scale bytes, ...
  uint32_t blocks;     // ... and the E4M3 code of its block scale: what general_scales needs
};

// One 16-group of both chunks; H: its 16 rotated values.  Returns the two scale bytes (low lane in bits 0..7, high lane
// in bits 8..15).
__device__ __forceinline__ uint32_t ms_eden_group(const f32x2_t* H, uint32_t inv_table, float so, float inv6,
                                                  uint32_t scale_seed, uint32_t opaque_zero, uint32_t group_lo, uint32_t group_hi, uint2& nib_lo,
                                                  uint2& nib_hi, float& ga_lo, float& ga_hi, bool& ok, uint32_t& block_codes,
                                                  float& corrected_lo, float& corrected_hi) {
  ga_lo = ga_hi = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    float a0, a1, b0, b1;
    unpack2(H[i], a0, a1);
    unpack2(H[i + 1], b0, b1);
    ga_lo = max3_abs(ga_lo, a0, b0);
    ga_hi = max3_abs(ga_hi, a1, b1);
  }
  // block scale code: nearest E4M3 value, ties to even, saturating at 448
  uint16_t codes;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(codes) : "f"(ga_hi * so * inv6), "f"(ga_lo * so * inv6));
  const uint2 t0 = lds_64(inv_table + (codes & 0xffu) * 8), t1 = lds_64(inv_table + (static_cast<uint32_t>(codes) >> 8) * 8);
  const f32x2_t inv = pack2(__uint_as_float(t0.x), __uint_as_float(t1.x));
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
  float qa0[8], qa1[8], qb0[8], qb1[8];
  e2m1x8_unpacked(nib_lo.x, opaque_zero, qa0);
  e2m1x8_unpacked(nib_lo.y, opaque_zero, qa1);
  e2m1x8_unpacked(nib_hi.x, opaque_zero, qb0);
  e2m1x8_unpacked(nib_hi.y, opaque_zero, qb1);
  // sums of x^2 and x q in the order of the reference's xor-8,4,2,1 butterfly
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
  // The quotient needs no range check of its own, whatever the global scale and the scale override make of x: an E2M1
  // value is 0 up to |x| = 1/4 and at least 1/2 beyond, so den is 0 or at least 1/8, and where the sums stay finite den is
  // below 2^71, its reciprocal far inside the normal range.  den = 0 and infinite sums end as NaN, which the range check
  // of the product catches like every product outside [2^-6, 448).
  corrected_lo = __uint_as_float(t0.y) * div_in_range(num_a, den_a);
  corrected_hi = __uint_as_float(t1.y) * div_in_range(num_b, den_b);
  block_codes = codes;
  const uint32_t s0 = __float_as_uint(corrected_lo), s1 = __float_as_uint(corrected_hi);
  ok = ok && s0 - 0x3c800000u < 0x43e00000u - 0x3c800000u && s1 - 0x3c800000u < 0x43e00000u - 0x3c800000u;
  return stochastic_code(s0, scale_seed, group_lo) | (stochastic_code(s1, scale_seed, group_hi) << 8);
}

// Two rotated-and-quantized 32-chunks: P[k] = signed input k of the low-lane and of the high-lane chunk, after the
// stride-1 butterfly stage.
// inv_table: shared-memory address of (1 / (s * gs + eps), s) over the E4M3 codes.
__device__ __forceinline__ PairCode ms_eden_chunk_pair(f32x2_t (&P)[32], uint32_t inv_table, float so, float inv6,
                                                       uint32_t scale_seed, uint32_t opaque_zero, uint32_t group_lo, uint32_t group_hi) {
#pragma unroll
  for (int stride = 2; stride < 32; stride <<= 1) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if ((i & stride) == 0) {
        const f32x2_t a = P[i], b = P[i | stride];
        P[i] = add2(a, b);
        P[i | stride] = sub2(a, b);
      }
    }
  }
  const f32x2_t c = pack2(0.17677669f, 0.17677669f);
#pragma unroll
  for (int i = 0; i < 32; ++i) P[i] = mul2(P[i], c);
  PairCode r;
  r.ok = true;
  uint2 lo0, lo1, hi0, hi1;
  float a0, a1, b0, b1;
  uint32_t codes0, codes1;
  const uint32_t g0 = ms_eden_group(&P[0], inv_table, so, inv6, scale_seed, opaque_zero, group_lo, group_hi, lo0, hi0, a0, b0, r.ok,
                                    codes0, r.corrected[0], r.corrected[2]);
  const uint32_t g1 = ms_eden_group(&P[16], inv_table, so, inv6, scale_seed, opaque_zero, group_lo + 1, group_hi + 1, lo1, hi1, a1,
                                    b1, r.ok, codes1, r.corrected[1], r.corrected[3]);
  r.blocks = __byte_perm(codes0, codes1, 0x5140);
  r.lo = make_uint4(lo0.x, lo0.y, lo1.x, lo1.y);
  r.hi = make_uint4(hi0.x, hi0.y, hi1.x, hi1.y);
  r.scales = __byte_perm(g0, g1, 0x5140);  // low lane: g0, g1; high lane: g0, g1
  r.amax_lo = max_f32(a0, a1);
  r.amax_hi = max_f32(b0, b1);
  return r;
}

// The four scale bytes of a thread's two chunks whatever their corrected scales are: below 2^-6, saturating, negative, zero
// groups.  The nibbles of the straight-line path hold for those too, so nothing else has to be done again.  A group has
// den = 0 exactly where all its nibbles are zero (ms_eden_group); its correction is one.  `lost`: a sum was infinite or an
// input NaN, the chunks need the generic code.  By value and not inlined, so that it costs the straight-line path no
// registers.  dY of a cross-entropy over 32000 columns comes this way in 21 to 94 % of its chunks, masked tokens and dead units
// in all of theirs: the linear backward of 8192 tokens x 32000 takes 676 us with normal dY, 752 to 788 with that gradient
// (logits N(0, 0.02) to N(0, 6)), against 1725 to 2190 when each thread quantized such chunks again.
struct GeneralScales {
  uint32_t bytes;
  bool lost;
};
__device__ __noinline__ GeneralScales general_scales(float4 corrected, uint32_t blocks, uint4 lo, uint4 hi, uint32_t scale_seed,
                                                     uint32_t group_lo, uint32_t group_hi) {
  const float c[4] = {corrected.x, corrected.y, corrected.z, corrected.w};
  const uint32_t nibbles[4] = {lo.x | lo.y, lo.z | lo.w, hi.x | hi.y, hi.z | hi.w};
  GeneralScales r = {0u, false};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float v = nz((nibbles[i] & 0x77777777u) ? c[i] : nz(e4m3_value((blocks >> (8 * i)) & 0xffu)));
    r.bytes |= stochastic_e4m3_scale(v, scale_seed, (i < 2 ? group_lo : group_hi) + (i & 1)) << (8 * i);
    r.lost = r.lost || v != v;
  }
  return r;
}
__device__ __forceinline__ GeneralScales general_scales(const PairCode& code, uint32_t scale_seed, uint32_t group_lo, uint32_t group_hi) {
  return general_scales(make_float4(code.corrected[0], code.corrected[1], code.corrected[2], code.corrected[3]), code.blocks, code.lo,
                        code.hi, scale_seed, group_lo, group_hi);
}

// A chunk again by the generic code, any values (infinite sums, NaN), from the source: `valid` values `step` elements apart,
// zeros behind them, K index k0 ...
template <typename T>
__device__ __noinline__ void requantize(const T* src, uint32_t step, uint32_t valid, uint32_t sign_seed, uint32_t k0,
                                        const MsEdenOut* o, float gs, float so, uint32_t row, uint32_t chunk_in_row) {
  f32x2_t P[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    uint32_t v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t k = i + 16 * h;
      v[h] = k < valid ? __float_as_uint(load_as_f32<T>(src, static_cast<size_t>(k) * step)) : 0u;
      v[h] ^= random_sign_negative(sign_seed, k0 + k) ? 0x80000000u : 0u;
    }
    P[i] = pack2(__uint_as_float(v[0]), __uint_as_float(v[1]));
  }
  ms_eden_emit_chunk(P, *o, gs, so, row, chunk_in_row);
}

// The same for values that are staged with their signs.
__device__ __noinline__ void requantize_staged(uint32_t src, uint32_t step, const MsEdenOut* o, float gs, float so, uint32_t row,
                                               uint32_t chunk_in_row) {
  f32x2_t P[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) P[i] = pack2(lds_f32(src + i * step), lds_f32(src + (i + 16) * step));
  ms_eden_emit_chunk(P, *o, gs, so, row, chunk_in_row);
}

// Where a role's chunks of one tile go: byte pointers of the tile (the same for every thread of a warp) and offsets
// inside it (the same for every tile of a thread), so that a chunk costs no index arithmetic.
struct ChunkOffsets {
  uint32_t nibbles, scales, group;
};
__device__ __forceinline__ uint8_t* tile_nibbles(const MsEdenOut& o, uint32_t row0, uint32_t chunk0) {
  return o.fp4 + (static_cast<size_t>(row0) * (o.dst_row_len >> 5) + chunk0) * 16;
}
__device__ __forceinline__ uint8_t* tile_scales(const MsEdenOut& o, uint32_t row0, uint32_t chunk0) {
  return o.scales + (o.packed ? packed_scale_offset(row0, chunk0 * 2, o.dst_row_len >> 6)
                              : (static_cast<size_t>(row0) * (o.dst_row_len >> 5) + chunk0) * 2);
}
// row, chunk: inside the tile (row0 a multiple of 64, row0 % 128 + row < 128, chunk0 even)
__device__ __forceinline__ ChunkOffsets chunk_offsets(const MsEdenOut& o, uint32_t row, uint32_t chunk) {
  const uint32_t cpr = o.dst_row_len >> 5;
  ChunkOffsets r;
  r.nibbles = (row * cpr + chunk) * 16;
  r.scales = o.packed ? (row & 31u) * 16 + (row >> 5) * 4 + (chunk >> 1) * 512 + (chunk & 1u) * 2 : (row * cpr + chunk) * 2;
  r.group = row * o.group_row_stride + chunk * 2 + o.group_offset;
  return r;
}
// Pad rows of a packed scale plane, up to a multiple of 128, hold 1.0.  `behind`: the tile also covers the 64 rows
// behind it (the last 64-column tile of a transposed operand).
__device__ __forceinline__ void store_pad_scales(const MsEdenOut& o, uint32_t row, uint32_t chunk_in_row, bool behind) {
  const uint32_t padded = (o.rows + 127u) & ~127u;
  for (uint32_t r = row; r < padded && r <= row + 64u; r += 64u)
    if (r >= o.rows && (r == row || behind))
      *reinterpret_cast<uint16_t*>(o.scales + packed_scale_offset(r, chunk_in_row * 2, o.dst_row_len >> 6)) = 0x3838;
}
// A transposed operand's column pair: two output rows, one chunk each.
__device__ __forceinline__ void store_column_scales(uint32_t bytes, uint8_t* scales, const ChunkOffsets& row_step, bool second) {
  *reinterpret_cast<uint16_t*>(scales) = static_cast<uint16_t>(bytes);
  if (second) *reinterpret_cast<uint16_t*>(scales + row_step.scales) = static_cast<uint16_t>(bytes >> 16);
}
__device__ __forceinline__ void store_column_pair(const PairCode& c, uint8_t* nibbles, uint8_t* scales, const ChunkOffsets& row_step,
                                                  bool first, bool second) {
  if (!first) return;  // `second` implies `first`
  *reinterpret_cast<uint4*>(nibbles) = c.lo;
  if (second) *reinterpret_cast<uint4*>(nibbles + row_step.nibbles) = c.hi;
  store_column_scales(c.scales, scales, row_step, second);
}

// The tiles of a persistent CTA: tile, tile + gridDim.x, ... as (row, column) of the tile grid without a division
// per tile.
struct TileWalk {
  uint32_t ty, tx, dy, dx, tiles_x;
  __device__ __forceinline__ TileWalk(uint32_t tiles_x_)
      : ty(blockIdx.x / tiles_x_), tx(blockIdx.x % tiles_x_), dy(gridDim.x / tiles_x_), dx(gridDim.x % tiles_x_), tiles_x(tiles_x_) {}
  __device__ __forceinline__ void advance() {
    ty += dy;
    tx += dx;
    if (tx >= tiles_x) {
      tx -= tiles_x;
      ++ty;
    }
  }
};

// (1 / (s * gs + eps), s) for every E4M3 code, zero standing for one, by the same operations as inv_scale.
__device__ __forceinline__ void fill_inv_table(float2* table, float safe_gs) {
  for (uint32_t i = threadIdx.x; i < kScaleCodes; i += blockDim.x) {
    const float s = e4m3_value(i);
    table[i] = make_float2(inv_scale(s, safe_gs), nz(s));
  }
}

__device__ __forceinline__ float tile_global_scale(const MsEdenTileParams& p) {
  if (!p.amax_in) return p.use_host_scale ? p.global_scale_host : after_prior(p.global_scale_dev)[0];
  const float* const in = after_prior(p.amax_in);
  float amax;
  if (p.amax_count <= 1) {
    amax = p.amax_count == 0 ? in[0] : max_f32(in[0], 0.0f);  // a single partial maximum by the rule of several
  } else {  // partial maxima, non-negative: the pass before neither waited for a cleared word nor added to it
    __shared__ uint32_t amax_bits;
    if (threadIdx.x == 0) amax_bits = 0u;
    __syncthreads();
    float m = 0.0f;
    for (uint32_t i = threadIdx.x; i < p.amax_count; i += blockDim.x) m = max_f32(m, in[i]);
    const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31u) == 0) atomicMax(&amax_bits, w);
    __syncthreads();
    amax = __uint_as_float(amax_bits);
  }
  const float gs = ms_eden_scale_of_amax(amax);
  if (blockIdx.x == 0 && threadIdx.x == 0) p.gs_out[0] = gs;
  return gs;
}

}  // namespace

// ---- dY in both orientations ------------------------------------------------------------------

// What a warp stages of a tile: 32 source rows of 64 values, 16 bytes of padding per row (conflict-free 16-byte reads along
// rows and 2- or 4-byte reads down columns).
constexpr int kBlockRows = 32;
template <typename T>
struct PairBlock {
  static constexpr bool kBf16 = sizeof(T) == 2;
  static constexpr int kPitch = kTileCols * static_cast<int>(sizeof(T)) + 16;
  static constexpr int kBytes = kBlockRows * kPitch;
  static constexpr int kPiecesPerRow = kTileCols * static_cast<int>(sizeof(T)) / 16;
  static constexpr int kSignWords = kBf16 ? 32 : kTileCols;
};

// Warps 0-3: the transposed operand, columns 2 * lane and 2 * lane + 1, rows 32 * warp ... of the CTA's tile.  Warps 4-7: the
// row operand, row 32 * (warp - 4) + lane, both of its chunks.  The roles are separate code, so that neither pays for
// selecting the other's addresses.  Every warp stages its rows and its signs for itself, and loads the next tile's as soon as
// it holds this one's in registers: no barrier ties the warps together (but the column sums, once per tile, those of the
// transposed role), so that the butterfly of one, all FP32, runs beside the conversions of another.
// `rows` and `cols` need not be whole tiles in the kEdge form (zero fill on the way in, guards on the way out, pad rows of
// the packed scale planes written with 1.0).
template <typename T, bool kColSum, bool kEdge>
__global__ void __launch_bounds__(256, 2)
    ms_eden_pair_kernel(const __grid_constant__ MsEdenTileParams p, uint32_t tiles_x, uint32_t tile_count) {
  wait_for_prior_then_allow_next();
  using PB = PairBlock<T>;
  constexpr bool kBf16 = PB::kBf16;
  constexpr uint32_t kSize = sizeof(T);
  extern __shared__ __align__(16) uint8_t pair_stage[];  // [8][PB::kBytes]
  // Random signs of a warp's rows (transposed role) or columns (row role).  bf16 sources: +-1 in bf16 for each half of a word;
  // the K positions of the transposed operand share one sign for both halves (two columns), those of the row operand have one
  // each.  f32 sources: the bare sign bit.
  __shared__ __align__(16) uint32_t sign_words[8][PB::kSignWords];
  __shared__ __align__(8) float quarter_sum[2][4][kTileCols];
  __shared__ float2 inv_table[kScaleCodes];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const T* x = after_prior(static_cast<const T*>(p.x));
  const uint32_t stage = static_cast<uint32_t>(__cvta_generic_to_shared(pair_stage)) + warp * PB::kBytes;
  const uint32_t signs = static_cast<uint32_t>(__cvta_generic_to_shared(sign_words[warp]));
  const uint32_t table = static_cast<uint32_t>(__cvta_generic_to_shared(inv_table));
  const uint32_t row_in_tile = (warp & 3u) * kBlockRows;  // of the warp's first row

  // 16-byte pieces, row-major over the block, kPiecesPerRow passes of kPassRows rows
  constexpr uint32_t kPassRows = 32 / PB::kPiecesPerRow;
  const uint32_t piece_row = lane / PB::kPiecesPerRow, piece_col = lane % PB::kPiecesPerRow * (16 / kSize);
  const uint32_t piece_dst = stage + piece_row * PB::kPitch + piece_col * kSize;
  const size_t piece_off = static_cast<size_t>(row_in_tile + piece_row) * p.src_cols + piece_col;
  const size_t pass_stride = static_cast<size_t>(kPassRows) * p.src_cols;
  auto issue_block = [&](uint32_t ty, uint32_t tx) {
    const T* src = x + static_cast<size_t>(ty) * kTileRows * p.src_cols + tx * kTileCols + piece_off;
#pragma unroll
    for (uint32_t k = 0; k < PB::kPiecesPerRow; ++k) {
      const uint32_t dst = piece_dst + k * kPassRows * PB::kPitch;
      if (kEdge) {
        const bool inside = ty * kTileRows + row_in_tile + piece_row + k * kPassRows < p.src_rows &&
                            tx * kTileCols + piece_col < p.src_cols;  // columns come in whole 16-byte pieces
        cp_async_16_or_zero(dst, inside ? src + k * pass_stride : x, inside ? 16u : 0u);
      } else {
        cp_async_16(dst, src + k * pass_stride);
      }
    }
  };

  TileWalk next(tiles_x);
  uint32_t buf = 0;
  if (blockIdx.x < tile_count) issue_block(next.ty, next.tx);  // in flight while the scale is derived
  const float gs = tile_global_scale(p), safe_gs = nz(gs);
  fill_inv_table(inv_table, safe_gs);
  const float inv6 = inv_scale(6.0f, safe_gs);

  const uint32_t src = stage + (warp < 4 ? lane * 2 * kSize : lane * PB::kPitch);
  const ChunkOffsets at = warp < 4 ? chunk_offsets(p.t, 2 * lane, warp) : chunk_offsets(p.r, row_in_tile + lane, 0);
  const ChunkOffsets row_step = {(p.t.dst_row_len >> 5) * 16, p.t.packed ? 16u : (p.t.dst_row_len >> 5) * 2, p.t.group_row_stride};
  const bool wide_rows = (p.r.dst_row_len & 63u) == 0 && (reinterpret_cast<uintptr_t>(p.r.fp4) & 31u) == 0 &&
                         (reinterpret_cast<uintptr_t>(p.r.scales) & 3u) == 0;

  for (uint64_t i = blockIdx.x * 256u + tid; i < p.zero_words; i += gridDim.x * 256u) p.zero[i] = make_uint4(0u, 0u, 0u, 0u);

  __syncthreads();  // the table
#pragma unroll 1
  for (uint32_t tile = blockIdx.x; tile < tile_count; tile += gridDim.x, buf ^= 1) {
    const uint32_t ty = next.ty, r0 = ty * kTileRows, c0 = next.tx * kTileCols;
    next.advance();
    const bool more = tile + gridDim.x < tile_count;
    if (warp < 4) {
      const bool neg = random_sign_negative(p.sign_seed, r0 + row_in_tile + lane + p.t.sign_offset);
      sign_words[warp][lane] = kBf16 ? (neg ? 0xbf80bf80u : 0x3f803f80u) : (neg ? 0x80000000u : 0u);
      if (r0 == 0 && warp < 2 && (!kEdge || c0 + tid < p.t.rows)) p.t.global_scales[c0 + tid] = gs;
    } else {
      const uint32_t col = c0 + (kBf16 ? 2 * lane : lane) + p.r.sign_offset;
      const bool neg0 = random_sign_negative(p.sign_seed, col), neg1 = random_sign_negative(p.sign_seed, col + (kBf16 ? 1u : 32u));
      if (kBf16) {
        sign_words[warp][lane] = (neg0 ? 0xbf80u : 0x3f80u) | (neg1 ? 0xbf800000u : 0x3f800000u);
      } else {
        sign_words[warp][lane] = neg0 ? 0x80000000u : 0u;
        sign_words[warp][lane + PB::kSignWords - 32] = neg1 ? 0x80000000u : 0u;
      }
      const uint32_t row = r0 + row_in_tile + lane;
      if (c0 == 0 && (!kEdge || row < p.r.rows)) p.r.global_scales[row] = gs;
    }
    cp_async_wait_all();
    __syncwarp();

    f32x2_t P[32];
    if (warp < 4) {
      float sum_lo = 0.0f, sum_hi = 0.0f;
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const uint4 sv = lds_128(signs + g * 16);
        const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
        for (int k = 0; k < 4; k += 2) {
          const int pos = 4 * g + k;
          if (kBf16) {
            const uint32_t wa = lds_u32(src + pos * PB::kPitch), wb = lds_u32(src + (pos + 1) * PB::kPitch);
            float sl, dl, sh, dh;
            first_stage_lo(wa, wb, sw[k], sw[k + 1], sl, dl);
            first_stage_hi(wa, wb, sw[k], sw[k + 1], sh, dh);
            P[pos] = pack2(sl, sh);
            P[pos + 1] = pack2(dl, dh);
            if (kColSum) {
              sum_lo = add_bf16_lo(wb, add_bf16_lo(wa, sum_lo));
              sum_hi = add_bf16_hi(wb, add_bf16_hi(wa, sum_hi));
            }
          } else {
            const uint2 wa = lds_64(src + pos * PB::kPitch), wb = lds_64(src + (pos + 1) * PB::kPitch);
            const f32x2_t ua = pack2(__uint_as_float(wa.x ^ sw[k]), __uint_as_float(wa.y ^ sw[k]));
            const f32x2_t ub = pack2(__uint_as_float(wb.x ^ sw[k + 1]), __uint_as_float(wb.y ^ sw[k + 1]));
            P[pos] = add2(ua, ub);
            P[pos + 1] = sub2(ua, ub);
            if (kColSum) {
              sum_lo = (sum_lo + __uint_as_float(wa.x)) + __uint_as_float(wb.x);
              sum_hi = (sum_hi + __uint_as_float(wa.y)) + __uint_as_float(wb.y);
            }
          }
        }
      }
      __syncwarp();
      if (more) issue_block(next.ty, next.tx);
      // dbias partials: four sequential 32-row sums per column, added below in the order ((q0 + q1) + q2) + q3
      if (kColSum) *reinterpret_cast<float2*>(&quarter_sum[buf][warp][2 * lane]) = make_float2(sum_lo, sum_hi);
      const uint32_t group = at.group + c0 * p.t.group_row_stride + (r0 >> 4);
      const PairCode code =
          ms_eden_chunk_pair(P, table, p.scale_override, inv6, p.t.scale_seed, p.opaque_zero, group, group + row_step.group);
      const uint32_t row = c0 + 2 * lane, chunk_in_row = (r0 >> 5) + warp;
      bool first = true, second = true;
      if (kEdge) {
        const bool k_inside = chunk_in_row * 32u < p.t.dst_row_len;
        if (p.t.packed && k_inside) {
          store_pad_scales(p.t, row, chunk_in_row, c0 + kTileCols >= p.src_cols);
          store_pad_scales(p.t, row + 1, chunk_in_row, c0 + kTileCols >= p.src_cols);
        }
        first = k_inside && row < p.t.rows;
        second = k_inside && row + 1 < p.t.rows;
      }
      uint8_t* const scales = tile_scales(p.t, c0, r0 >> 5) + at.scales;
      store_column_pair(code, tile_nibbles(p.t, c0, r0 >> 5) + at.nibbles, scales, row_step, first, second);
      if (!code.ok && first) {
        const GeneralScales g = general_scales(code, p.t.scale_seed, group, group + row_step.group);
        store_column_scales(g.bytes, scales, row_step, second);
        const uint32_t k0 = r0 + warp * kBlockRows, valid = kEdge ? p.src_rows - min(p.src_rows, k0) : 32u;
#pragma unroll 1
        for (uint32_t h = g.lost ? 0u : 2u; h < (second ? 2u : 1u); ++h)
          requantize<T>(x + static_cast<size_t>(k0) * p.src_cols + row + h, p.src_cols, valid, p.sign_seed, k0 + p.t.sign_offset, &p.t,
                        gs, p.scale_override, row + h, chunk_in_row);
      }
      if (kColSum) {
        // two buffers: a warp that is here again has passed the barrier of the tile between, behind the sums of this one
        __syncwarp();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (warp < 2 && (!kEdge || c0 + tid < p.src_cols))
          p.col_sum_partials[static_cast<size_t>(ty) * p.src_cols + c0 + tid] =
              ((quarter_sum[buf][0][tid] + quarter_sum[buf][1][tid]) + quarter_sum[buf][2][tid]) + quarter_sum[buf][3][tid];
      }
    } else {
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        constexpr int kPerLoad = 16 / static_cast<int>(kSize);
#pragma unroll
        for (int g = 0; g < 32 / kPerLoad; ++g) {
          const uint4 v = lds_128(src + half * 32 * kSize + g * 16);
          const uint4 s = lds_128(signs + half * (kBf16 ? 64 : 128) + g * 16);
          const uint32_t vw[4] = {v.x, v.y, v.z, v.w}, sw[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (kBf16) {  // K positions 2j (low half) and 2j + 1 (high half)
              const int pos = 8 * g + 2 * k;
              const float ub = signed_bf16_hi(vw[k], sw[k], -0.0f);
              set_lane(P[pos], half, signed_bf16_lo(vw[k], sw[k], ub));
              set_lane(P[pos + 1], half, signed_bf16_lo(vw[k], sw[k], -ub));
            } else if ((k & 1) == 0) {
              const float ua = __uint_as_float(vw[k] ^ sw[k]), ub = __uint_as_float(vw[k + 1] ^ sw[k + 1]);
              set_lane(P[4 * g + k], half, __fadd_rn(ua, ub));
              set_lane(P[4 * g + k + 1], half, __fsub_rn(ua, ub));
            }
          }
        }
      }
      __syncwarp();
      if (more) issue_block(next.ty, next.tx);
      const uint32_t group = at.group + r0 * p.r.group_row_stride + (c0 >> 4);
      const PairCode code = ms_eden_chunk_pair(P, table, p.scale_override, inv6, p.r.scale_seed, p.opaque_zero, group, group + 2);
      uint8_t* const nibbles = tile_nibbles(p.r, r0, c0 >> 5) + at.nibbles;
      uint8_t* const scales = tile_scales(p.r, r0, c0 >> 5) + at.scales;
      const uint32_t row = r0 + row_in_tile + lane, chunk_in_row = c0 >> 5;
      const bool inside = !kEdge || row < p.r.rows, second = !kEdge || (chunk_in_row + 1) * 32u < p.r.dst_row_len;
      if (kEdge && p.r.packed) {
        store_pad_scales(p.r, row, chunk_in_row, false);
        if (second) store_pad_scales(p.r, row, chunk_in_row + 1, false);
      }
      if (inside) {
        if (wide_rows) {  // 32 nibble bytes in one store, four scale bytes in one
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(nibbles), "r"(code.lo.x),
                       "r"(code.lo.y), "r"(code.lo.z), "r"(code.lo.w), "r"(code.hi.x), "r"(code.hi.y), "r"(code.hi.z), "r"(code.hi.w)
                       : "memory");
          *reinterpret_cast<uint32_t*>(scales) = code.scales;
        } else {
          *reinterpret_cast<uint4*>(nibbles) = code.lo;
          *reinterpret_cast<uint16_t*>(scales) = static_cast<uint16_t>(code.scales);
          if ((chunk_in_row + 1) * 32u < p.r.dst_row_len) {
            *reinterpret_cast<uint4*>(nibbles + 16) = code.hi;
            *reinterpret_cast<uint16_t*>(scales + 2) = static_cast<uint16_t>(code.scales >> 16);
          }
        }
        if (!code.ok) {
          const GeneralScales g = general_scales(code, p.r.scale_seed, group, group + 2);
          *reinterpret_cast<uint16_t*>(scales) = static_cast<uint16_t>(g.bytes);
          if (second) *reinterpret_cast<uint16_t*>(scales + 2) = static_cast<uint16_t>(g.bytes >> 16);
#pragma unroll 1
          for (uint32_t h = g.lost ? 0u : 2u; h < (second ? 2u : 1u); ++h) {
            const uint32_t k0 = c0 + 32 * h, valid = kEdge ? p.src_cols - min(p.src_cols, k0) : 32u;
            requantize<T>(x + static_cast<size_t>(row) * p.src_cols + k0, 1, valid, p.sign_seed, k0 + p.r.sign_offset, &p.r, gs,
                          p.scale_override, row, chunk_in_row + h);
          }
        }
      }
    }
    __syncwarp();
  }
}

// ---- the transposed operand of an NVFP4 matrix ------------------------------------------------

// A CTA decodes a [128 rows x 64 columns] tile to signed f32, one row per thread, then every thread takes two adjacent
// 32-chunks down a column pair.  Decoding is (q * s) * g as utils/nvfp4/tensor.rs:48-57 evaluates it: q * s in f16 (exact:
// E2M1 times E4M3 has six significant bits and lies between 2^-10 and 2688), then one rounding; the random sign of a K
// position is folded into its row's g, (q s)(-g) == -((q s) g).  Each thread's row of the next tile is in flight in
// registers during the current one.  A warp decodes the 32 rows whose chunks it takes, so that no barrier ties the warps
// together.
constexpr int kNvPitch = kTileCols * 4 + 16;

template <bool kRowwise, bool kEdge>
__global__ void __launch_bounds__(128, 4)
    ms_eden_nvfp4_transpose_kernel(const __grid_constant__ MsEdenTileParams p, uint32_t tiles_x, uint32_t tile_count) {
  wait_for_prior_then_allow_next();
  const uint8_t* const src_bytes = after_prior(p.src_bytes);
  const uint8_t* const src_scales = after_prior(p.src_scales);
  const float* const src_global = after_prior(p.src_global);
  __shared__ __align__(16) uint8_t nv_stage[kTileRows * kNvPitch];
  __shared__ float2 inv_table[kScaleCodes];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const float gs = tile_global_scale(p), safe_gs = nz(gs);
  fill_inv_table(inv_table, safe_gs);
  const float inv6 = inv_scale(6.0f, safe_gs);
  const uint32_t table = static_cast<uint32_t>(__cvta_generic_to_shared(inv_table));
  const float tensor_global = kRowwise ? 0.0f : src_global[0];
  // this thread's chunks: columns 2 * lane and 2 * lane + 1, rows 32 * warp ... of the tile
  const ChunkOffsets at = chunk_offsets(p.t, 2 * lane, warp);
  const ChunkOffsets row_step = {(p.t.dst_row_len >> 5) * 16, p.t.packed ? 16u : (p.t.dst_row_len >> 5) * 2, p.t.group_row_stride};

  // thread = one row of the tile: 32 nibble bytes, 4 scale bytes, one global scale, fetched one tile ahead
  uint4 raw[2];
  uint32_t raw_scales;
  float raw_global;
  auto load_tile = [&](uint32_t ty, uint32_t tx) {
    const uint32_t r = ty * kTileRows + tid;
    raw[0] = raw[1] = make_uint4(0u, 0u, 0u, 0u);
    raw_scales = 0;
    raw_global = kRowwise ? 1.0f : tensor_global;
    if (!kEdge || r < p.src_rows) {
      if (kRowwise) raw_global = __ldg(src_global + r);
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t c = tx * kTileCols + 32 * h;
        if (!kEdge || c < p.src_cols) {  // columns come in whole 32s
          const size_t index = static_cast<size_t>(r) * p.src_cols + c;
          raw[h] = __ldg(reinterpret_cast<const uint4*>(src_bytes + (index >> 1)));
          const size_t sidx = p.src_packed ? packed_scale_offset(r, c >> 4, p.src_cols >> 6) : index >> 4;
          raw_scales |= static_cast<uint32_t>(__ldg(reinterpret_cast<const uint16_t*>(src_scales + sidx))) << (16 * h);
        }
      }
    }
  };

  const uint32_t stage = static_cast<uint32_t>(__cvta_generic_to_shared(nv_stage));
  TileWalk next(tiles_x);
  if (blockIdx.x < tile_count) load_tile(next.ty, next.tx);
  __syncthreads();  // the table
#pragma unroll 1
  for (uint32_t tile = blockIdx.x; tile < tile_count; tile += gridDim.x) {
    const uint32_t r0 = next.ty * kTileRows, c0 = next.tx * kTileCols;
    next.advance();
    {
      const float g = random_sign_negative(p.sign_seed, r0 + tid + p.t.sign_offset) ? -raw_global : raw_global;
      const uint32_t dst = stage + tid * kNvPitch;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t words[4] = {raw[h].x, raw[h].y, raw[h].z, raw[h].w};
        uint32_t scales_f16;
        asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(scales_f16) : "h"(static_cast<uint16_t>(raw_scales >> (16 * h))));
        const __half2 both = *reinterpret_cast<const __half2*>(&scales_f16);
        const __half2 s[2] = {__low2half2(both), __high2half2(both)};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          float u[8];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t h2;
            asm("{ .reg .b8 t; cvt.u8.u32 t, %1; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(h2) : "r"(__byte_perm(words[w], 0u, 0x4440u | k)));
            const __half2 v = __hmul2(*reinterpret_cast<__half2*>(&h2), s[w >> 1]);
            u[2 * k] = __fmul_rn(widen_f16_lo(*reinterpret_cast<const uint32_t*>(&v)), g);
            u[2 * k + 1] = __fmul_rn(widen_f16_hi(*reinterpret_cast<const uint32_t*>(&v)), g);
          }
          sts_128(dst + h * 128 + w * 32, u[0], u[1], u[2], u[3]);
          sts_128(dst + h * 128 + w * 32 + 16, u[4], u[5], u[6], u[7]);
        }
      }
      if (r0 == 0 && tid < kTileCols && (!kEdge || c0 + tid < p.t.rows)) p.t.global_scales[c0 + tid] = gs;
    }
    if (tile + gridDim.x < tile_count) load_tile(next.ty, next.tx);
    __syncwarp();

    const uint32_t src = stage + warp * 32 * kNvPitch + lane * 8;
    f32x2_t P[32];
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
      const uint2 wa = lds_64(src + k * kNvPitch), wb = lds_64(src + (k + 1) * kNvPitch);
      const f32x2_t ua = pack2(__uint_as_float(wa.x), __uint_as_float(wa.y)), ub = pack2(__uint_as_float(wb.x), __uint_as_float(wb.y));
      P[k] = add2(ua, ub);
      P[k + 1] = sub2(ua, ub);
    }
    const uint32_t group = at.group + c0 * p.t.group_row_stride + (r0 >> 4);
    const PairCode code = ms_eden_chunk_pair(P, table, p.scale_override, inv6, p.t.scale_seed, p.opaque_zero, group, group + row_step.group);
    const uint32_t row = c0 + 2 * lane, chunk_in_row = (r0 >> 5) + warp;
    bool first = true, second = true;
    if (kEdge) {
      const bool k_inside = chunk_in_row * 32u < p.t.dst_row_len;
      if (p.t.packed && k_inside) {
        store_pad_scales(p.t, row, chunk_in_row, c0 + kTileCols >= p.src_cols);
        store_pad_scales(p.t, row + 1, chunk_in_row, c0 + kTileCols >= p.src_cols);
      }
      first = k_inside && row < p.t.rows;
      second = k_inside && row + 1 < p.t.rows;
    }
    uint8_t* const scales = tile_scales(p.t, c0, r0 >> 5) + at.scales;
    store_column_pair(code, tile_nibbles(p.t, c0, r0 >> 5) + at.nibbles, scales, row_step, first, second);
    if (p.t.chunk_amax) {
      const size_t chunk = static_cast<size_t>(row) * (p.t.dst_row_len >> 5) + chunk_in_row;
      if (first) p.t.chunk_amax[chunk] = code.amax_lo;
      if (second) p.t.chunk_amax[chunk + (p.t.dst_row_len >> 5)] = code.amax_hi;
    }
    if (!code.ok && first) {
      // the generic code, from the signed values still staged (general_scales takes the kernel from 120 to 121 registers a
      // thread, and one GPT-2-small layer at 8192 tokens with it from 541 to 545 us)
      for (uint32_t h = 0; h < (second ? 2u : 1u); ++h)
        requantize_staged(src + h * 4, kNvPitch, &p.t, gs, p.scale_override, row + h, chunk_in_row);
    }
    __syncwarp();
  }
}

// ---- launchers --------------------------------------------------------------------------------

namespace {

// The opt-in to more than 48 KB of shared memory is a per-device attribute of a kernel.
template <auto kKernel>
int opt_in_shared(int bytes) {
  static std::atomic<int> attr_state[64];  // per kernel and device ordinal: 0 = not set, 1 = set, -(error) = failed
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return static_cast<int>(cudaErrorInvalidDevice);
  int st = attr_state[dev].load(std::memory_order_acquire);
  if (st == 0) {
    const cudaError_t e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    st = e == cudaSuccess ? 1 : -static_cast<int>(e);
    attr_state[dev].store(st, std::memory_order_release);
  }
  return st < 0 ? -st : 0;
}

template <typename T, bool kColSum, bool kEdge>
int launch_pair(cudaStream_t s, const MsEdenTileParams& p, bool beside_others) {
  constexpr int kStage = 8 * PairBlock<T>::kBytes;
  const int rc = opt_in_shared<ms_eden_pair_kernel<T, kColSum, kEdge>>(kStage);
  if (rc) return rc;
  const uint32_t tiles_x = (p.src_cols + kTileCols - 1) / kTileCols;
  const uint32_t tiles = tiles_x * ((p.src_rows + kTileRows - 1) / kTileRows);
  const uint32_t resident = 148u * 2u;
  // With a tile for every resident CTA this kernel takes every register of the chip.  Started early, its CTAs sit there waiting
  // for the amax before it while the transposers of the other stream, enqueued earlier, may find no room until it ends.  A
  // backward call behind another kernel, L2 cold, dY 8192 x 2304 bf16: 92 us started early, 105 with some side streams (which
  // of them differs from process to process), 87 otherwise; 1000 x 3072 53 and 67 against 52.  Calls back to back gain 1 to 3
  // us from the early start below 5000 tokens and lose 1 to 2 above.  With fewer CTAs (512 x 3072: 192) there is room for
  // both streams.
  if (beside_others && tiles >= resident) {
    ms_eden_pair_kernel<T, kColSum, kEdge><<<resident, 256, kStage, s>>>(p, tiles_x, tiles);
    count_launch();
    return static_cast<int>(cudaGetLastError());
  }
  return launch_chained(ms_eden_pair_kernel<T, kColSum, kEdge>, tiles < resident ? tiles : resident, 256, kStage, s, p, tiles_x,
                        tiles);
}

template <typename T>
int launch_pair_of(cudaStream_t s, const MsEdenTileParams& p, bool edge, bool beside_others) {
  if (p.col_sum_partials)
    return edge ? launch_pair<T, true, true>(s, p, beside_others) : launch_pair<T, true, false>(s, p, beside_others);
  return edge ? launch_pair<T, false, true>(s, p, beside_others) : launch_pair<T, false, false>(s, p, beside_others);
}

}  // namespace

// Whole 16-byte pieces per row is all the pair kernel needs; whole 128 x 128 blocks (no pad rows in either scale
// plane) take the form without guards.
bool ms_eden_pair_has_tile_form(const void* x, int dtype, uint32_t cols) {
  return (reinterpret_cast<uintptr_t>(x) & 15u) == 0 && cols % (dtype == NVFP4_DTYPE_BF16 ? 8u : 4u) == 0;
}
int launch_ms_eden_pair_tiles(cudaStream_t s, const MsEdenTileParams& p, int dtype, bool beside_others) {
  const bool edge = p.src_rows % 128 != 0 || p.src_cols % 128 != 0 || p.t.dst_row_len != p.src_rows ||
                    p.r.dst_row_len != p.src_cols;
  return dtype == NVFP4_DTYPE_BF16 ? launch_pair_of<__nv_bfloat16>(s, p, edge, beside_others)
                                   : launch_pair_of<float>(s, p, edge, beside_others);
}

bool ms_eden_nvfp4_has_tile_form(const uint8_t* bytes, const uint8_t* scales, uint32_t cols) {
  return (reinterpret_cast<uintptr_t>(bytes) & 15u) == 0 && (reinterpret_cast<uintptr_t>(scales) & 1u) == 0 && cols % 32 == 0;
}
template <bool kRowwise, bool kEdge>
static int launch_nvfp4(cudaStream_t s, const MsEdenTileParams& p) {
  const uint32_t tiles_x = (p.src_cols + kTileCols - 1) / kTileCols;
  const uint32_t tiles = tiles_x * ((p.src_rows + kTileRows - 1) / kTileRows);
  const uint32_t resident = 148u * 4u;
  return launch_chained(ms_eden_nvfp4_transpose_kernel<kRowwise, kEdge>, tiles < resident ? tiles : resident, 128, 0, s, p,
                        tiles_x, tiles);
}
int launch_ms_eden_nvfp4_tiles(cudaStream_t s, const MsEdenTileParams& p, bool rowwise) {
  const bool edge = p.src_rows % 128 != 0 || p.src_cols % 128 != 0 || p.t.dst_row_len != p.src_rows;
  if (rowwise) return edge ? launch_nvfp4<true, true>(s, p) : launch_nvfp4<true, false>(s, p);
  return edge ? launch_nvfp4<false, true>(s, p) : launch_nvfp4<false, false>(s, p);
}

}  // namespace nvfp4
