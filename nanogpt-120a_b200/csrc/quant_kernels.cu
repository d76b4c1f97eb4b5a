// Bandwidth kernels of the NVFP4 projection path for sm_100a: amax reductions, the
// four-six quantizer, the MS-EDEN quantizer (row, transposed, NVFP4-source variants),
// decode, scale-plane packing, padding, post-ops and the bias gradient.
//
// Compiled with -fmad=false: the arithmetic below must round exactly like the
// reference's device code (one rounding per operation, no contraction).
//
// Work decomposition differs from the reference on purpose.  The reference gives each
// element its own lane and reduces 16-groups with shuffles; here one thread owns a whole
// 16-group (four-six) or 32-chunk (MS-EDEN) in registers, loads it with 128-bit
// transactions and writes nibbles as 8/16-byte words.  The reduction trees are evaluated
// in the same order as the reference's xor butterflies, so the bytes are identical.

#include <cstdlib>
#include <atomic>
#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "ms_eden.cuh"

namespace nvfp4 {

// ============================================================================
// amax
// ============================================================================

template <typename T>
struct VecTraits;
template <>
struct VecTraits<float> {
  static constexpr int kPerVec = 4;
};
template <>
struct VecTraits<__nv_bfloat16> {
  static constexpr int kPerVec = 8;
};

template <typename T>
__device__ __forceinline__ float vec_amax(const T* p);  // 16-byte aligned, kPerVec elements
template <>
__device__ __forceinline__ float vec_amax<float>(const float* p) {
  float4 t = __ldg(reinterpret_cast<const float4*>(p));
  return max_f32(max_f32(fabsf(t.x), fabsf(t.y)), max_f32(fabsf(t.z), fabsf(t.w)));
}
template <>
__device__ __forceinline__ float vec_amax<__nv_bfloat16>(const __nv_bfloat16* p) {
  uint4 t = __ldg(reinterpret_cast<const uint4*>(p));
  uint32_t w[4] = {t.x, t.y, t.z, t.w};
  float m = 0.0f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    m = max_f32(m, fabsf(__uint_as_float(w[j] << 16)));
    m = max_f32(m, fabsf(__uint_as_float(w[j] & 0xffff0000u)));
  }
  return m;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v = max_f32(v, __shfl_xor_sync(0xffffffffu, v, s));
  return v;
}

// One warp per row.  utils/nvfp4/quant/kernels/row_amax.rs:43-64 (max is order independent).
template <typename T>
__global__ void __launch_bounds__(256) row_amax_kernel(const T* __restrict__ x, float* __restrict__ out,
                                                        uint32_t rows, uint32_t row_len) {
  wait_for_prior_then_allow_next();
  x = after_prior(x);
  const uint32_t row = blockIdx.x * 8 + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* p = x + static_cast<size_t>(row) * row_len;
  constexpr int V = VecTraits<T>::kPerVec;
  float m = 0.0f;
  const bool aligned = (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
  uint32_t done = 0;
  if (aligned) {
    const uint32_t vecs = row_len / V;
    for (uint32_t v = lane; v < vecs; v += 32) m = max_f32(m, vec_amax<T>(p + static_cast<size_t>(v) * V));
    done = vecs * V;
  }
  for (uint32_t c = done + lane; c < row_len; c += 32) m = max_f32(m, fabsf(load_as_f32<T>(p, c)));
  m = warp_max(m);
  if (lane == 0) out[row] = m;
}

// Block max of per-warp values followed by ONE atomic max per CTA into out[0] (which the
// launcher zeroes first; non-negative floats order like their bit patterns).
__device__ __forceinline__ void cta_atomic_max(float warp_value, float* out) {
  __shared__ float partial[8];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) partial[w] = warp_value;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) r = max_f32(r, partial[i]);
    atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(r));
  }
}

// The CTA's maximum to its slot of `partials` where the consumer reduces them (no zeroing launch, no atomics), else one
// atomic max into out[0].
__device__ __forceinline__ void cta_publish_max(float warp_value, float* out, float* partials) {
  if (!partials) {
    cta_atomic_max(warp_value, out);
    return;
  }
  __shared__ float partial[8];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float m = warp_max(warp_value);
  if (lane == 0) partial[w] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) r = max_f32(r, partial[i]);
    partials[blockIdx.x] = r;
  }
}

// amax of one full, 16-byte aligned 1024-value chunk, 32 lanes cooperating (result in every lane).
// bf16: the maximum is taken on packed bf16 pairs (exact -- a maximum rounds nothing -- and NaN
// operands are dropped like max.f32 drops them), four instructions per eight values.
template <typename T>
__device__ __forceinline__ float chunk_amax_1024(const T* p, uint32_t lane);
template <>
__device__ __forceinline__ float chunk_amax_1024<float>(const float* p, uint32_t lane) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = max_f32(m, vec_amax<float>(p + (static_cast<size_t>(i) * 32 + lane) * 4));
  return warp_max(m);
}
template <>
__device__ __forceinline__ float chunk_amax_1024<__nv_bfloat16>(const __nv_bfloat16* p, uint32_t lane) {
  uint4 t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = __ldg(reinterpret_cast<const uint4*>(p) + i * 32 + lane);
  __nv_bfloat162 m = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w[4] = {t[i].x, t[i].y, t[i].z, t[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[j])));
  }
  return warp_max(max_f32(__low2float(m), __high2float(m)));
}

// Tensor amax: warps stride over 1024-value chunks (chunk amax written when requested).
// utils/nvfp4/quant/kernels/row_amax.rs:67-101.
template <typename T>
__global__ void __launch_bounds__(256) tensor_amax_kernel(const T* __restrict__ x, float* __restrict__ chunk_amax,
                                                           float* __restrict__ out, float* __restrict__ partials,
                                                           uint64_t n) {
  wait_for_prior_then_allow_next();
  x = after_prior(x);
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * 8;
  const uint64_t chunks = (n + 1023) / 1024;
  float running = 0.0f;
  for (uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); chunk < chunks; chunk += warps) {
    const uint64_t base = chunk * 1024;
    const T* p = x + base;
    float m = 0.0f;
    if (base + 1024 <= n && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
      m = chunk_amax_1024<T>(p, lane);
    } else {
      const uint32_t count = static_cast<uint32_t>(min(static_cast<uint64_t>(1024), n - base));
      for (uint32_t i = lane; i < count; i += 32) m = max_f32(m, fabsf(load_as_f32<T>(p, i)));
      m = warp_max(m);
    }
    if (lane == 0 && chunk_amax) chunk_amax[chunk] = m;
    running = max_f32(running, m);
  }
  cta_publish_max(running, out, partials);
}

// amax of a decoded NVFP4 tensor [n/cols][cols], warps striding over 1024-value chunks.
// utils/nvfp4/quant/kernels/ms_eden/amax.rs:23-64.  rowwise: one global scale per row;
// packed: the scale bytes are in the packed tile layout.
__global__ void __launch_bounds__(256) nvfp4_amax_kernel(const uint8_t* __restrict__ bytes,
                                                          const uint8_t* __restrict__ scales,
                                                          const float* __restrict__ gscales, uint64_t n, uint32_t cols,
                                                          int rowwise, int packed, float* __restrict__ chunk_amax,
                                                          float* __restrict__ out, float* __restrict__ partials) {
  wait_for_prior_then_allow_next();
  bytes = after_prior(bytes);
  scales = after_prior(scales);
  gscales = after_prior(gscales);
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * 8;
  const uint64_t chunks = (n + 1023) / 1024;
  float running = 0.0f;
  for (uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); chunk < chunks; chunk += warps) {
    const uint64_t base = chunk * 1024;
    float m = 0.0f;
    const uint64_t end = min(n, base + 1024);
    // one 16-group (8 bytes, 1 scale) per lane per step
    for (uint64_t g0 = base + lane * 16ull; g0 < end; g0 += 512) {
      const uint32_t srow = static_cast<uint32_t>(g0 / cols);
      const uint32_t skg = static_cast<uint32_t>(g0 - static_cast<uint64_t>(srow) * cols) >> 4;
      const float gs = rowwise ? gscales[srow] : gscales[0];
      const float sc = e4m3_value(packed ? scales[packed_scale_offset(srow, skg, cols >> 6)] : scales[g0 >> 4]);
      const uint2 raw = __ldg(reinterpret_cast<const uint2*>(bytes + (g0 >> 1)));
      // |e2m1| grows with its 3-bit magnitude code and (q * sc) * gs is monotonic in q >= 0, so
      // the group's largest decoded magnitude is that of its largest code: one decode per group
      uint32_t mx = __vmaxu4(__vmaxu4(raw.x & 0x07070707u, (raw.x >> 4) & 0x07070707u),
                             __vmaxu4(raw.y & 0x07070707u, (raw.y >> 4) & 0x07070707u));
      mx = __vmaxu4(mx, mx >> 16);
      mx = __vmaxu4(mx, mx >> 8) & 0x7u;
      m = max_f32(m, fabsf(e2m1_value(mx) * sc * gs));
    }
    m = warp_max(m);
    if (lane == 0 && chunk_amax) chunk_amax[chunk] = m;
    running = max_f32(running, m);
  }
  cta_publish_max(running, out, partials);
}

// max over chunk values -> out[0] (transform 0) or the MS-EDEN global scale (transform 1).
// utils/nvfp4/quant/kernels/row_amax.rs:86-101, ms_eden/amax.rs:67-104, utils/quartet.rs:6-12.
__global__ void __launch_bounds__(256) amax_from_chunks_kernel(const float* __restrict__ chunk_amax,
                                                                float* __restrict__ out, uint32_t chunk_count,
                                                                int transform) {
  wait_for_prior_then_allow_next();
  chunk_amax = after_prior(chunk_amax);
  __shared__ float partial[8];
  float m = 0.0f;
  for (uint32_t i = threadIdx.x; i < chunk_count; i += 256) m = max_f32(m, chunk_amax[i]);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) r = max_f32(r, partial[i]);
    if (transform == 1) {
      const float so = (17.0f / 16.0f) * 0.93f;
      r = (r == 0.0f) ? 1.0f : r * so / (256.0f * 6.0f);
    }
    out[0] = r;
  }
}

// out[0] = MS-EDEN global scale of amax[0] (single thread).
__global__ void ms_eden_scale_from_amax_kernel(const float* __restrict__ amax, float* __restrict__ out) {
  wait_for_prior_then_allow_next();
  amax = after_prior(amax);
  out[0] = ms_eden_scale_of_amax(amax[0]);
}

// ============================================================================
// four-six
// ============================================================================
//
// Bound by instruction dispatch like the MS-EDEN kernels (ms_eden_tile.cu has the measured costs): per 16-group two
// candidate scales, two sets of nibbles and two error sums.  Only which error is the smaller leaves the group, so the sums
// are taken the cheap way first (differences in scaled units, fused multiply-adds) and in the reference's order and
// roundings only where the two lie closer together than both ways can differ.  Code for rare cases stands out of line, returns
// by value and keeps nothing in local memory.  The scalar side of a group -- two quotients by the global scale, two reciprocals,
// two E4M3 conversions -- is straight-line code for global scales inside [2^-80, 2^80]; other global scales, NaN included, take
// the generic code per group.  One branch decides between cheap and exact errors, one more takes the latter (24.5 -> 23.0
// instructions an element, 65536 x 768 bf16 rowwise 46.4 -> 43.2 us in four_six_rowwise_kernel, of zeros 73 -> 44).
//
// Both candidates of the scalar side stand in the lanes of packed operations (kPacked) where warps have other groups to go on with:
// fewer instructions, 4096 x 8192 bf16 with given maxima 20.3 -> 20.1 us, 20000 x 2048 with its own 27.3 -> 26.9.  Where a thread
// has one group and little beside it, a group's chain counts, and a packed operation takes longer than a scalar one (with packs and
// unpacks around it): scalar in four_six_kernel, the schedule-free weight of 3072 x 768 9.52 -> 9.39 us with its amax, 256 x 256
// 5.22 -> 5.12, a tensor of 256 x 256 f32 2.01 -> 1.83, 300 x 768 f32 with given maxima 1.98 -> 1.88 (8192 x 768 5.99 -> 6.08).

__device__ __forceinline__ float four_six_global_scale(float amax) {
  // utils/nvfp4/quant/kernels/four_six/helpers.rs:33-39 with scale_override = 1.0
  return nz(amax == 0.0f ? 1.0f : amax * 1.0f / (256.0f * 6.0f));
}

// What the groups of one global scale share.
__device__ __noinline__ float four_six_global_scale_any(float amax) { return four_six_global_scale(amax); }
template <bool kPacked>
struct FourSixScale {
  float gs;       // global scale
  f32x2_t d, y;   // 6 gs + eps and 4 gs + eps, and their reciprocals
  float limit;    // groups with a larger amax (the caller's was not theirs, or gs is outside the straight-line code's range) take
                  // the generic code; up to 2^60, where the reference's squares do not overflow
  FourSixScale() = default;
  __device__ __forceinline__ explicit FourSixScale(float amax) {
    // amax / 1536 correctly rounded (the remainder form, exact for every amax the straight-line code accepts); one for zero
    gs = amax == 0.0f ? 1.0f : div_by_rcp(amax, 1536.0f, 1.0f / 1536.0f);
    const bool plain = gs >= 0x1p-80f && gs <= 0x1p80f;
    if (!plain) gs = four_six_global_scale_any(amax);
    if (kPacked) {
      d = add2(mul2_rounded(pack2(gs, gs), pack2(6.0f, 4.0f)), pack2(kDenomEps, kDenomEps));
      y = rcp_in_range2(d);
    } else {
      const float d6 = 6.0f * gs + kDenomEps, d4 = 4.0f * gs + kDenomEps;
      d = pack2(d6, d4);
      y = pack2(rcp_in_range(d6), rcp_in_range(d4));
    }
    limit = plain ? fminf(gs * 0x1p20f, 0x1p60f) : -1.0f;
  }
};

// V[i] = (v[2 i], v[2 i + 1]) of a group
struct Group16 {
  f32x2_t V[8];
};

// V * inv and its nibble bytes
__device__ __forceinline__ uint2 trial16(const f32x2_t (&V)[8], float inv, float (&x)[16]) {
  const f32x2_t inv2 = pack2(inv, inv);
#pragma unroll
  for (int i = 0; i < 8; ++i) unpack2(mul2(V[i], inv2), x[2 * i], x[2 * i + 1]);
  return make_uint2(cvt_e2m1x8(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]),
                    cvt_e2m1x8(x[8], x[9], x[10], x[11], x[12], x[13], x[14], x[15]));
}

// One candidate scale: the nibble bytes q(v * inv) (the winner's are the output) and the squared error in units of the
// candidate's step, sum of (q - v * inv)^2, in four partial sums.
__device__ __forceinline__ float candidate16(const Group16& g, float inv, uint32_t opaque_zero, uint2& nib) {
  float x[16];
  nib = trial16(g.V, inv, x);
  f32x2_t sum[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float t[8] = {x[8 * h], x[8 * h + 1], x[8 * h + 2], x[8 * h + 3], x[8 * h + 4], x[8 * h + 5], x[8 * h + 6], x[8 * h + 7]};
    float d[8];
    e2m1x8_minus(h ? nib.y : nib.x, opaque_zero, t, d);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const f32x2_t e = pack2(d[2 * i], d[2 * i + 1]);
      sum[h] = i == 0 ? mul2(e, e) : fma2(e, e, sum[h]);
    }
  }
  float a, b;
  unpack2(add2(sum[0], sum[1]), a, b);
  return a + b;
}

// Squared quantization error of the group for one candidate as the reference rounds it: sum of (v - q * dq)^2 in butterfly
// order (utils/nvfp4/quant/kernels/convert.rs:27-35).
__device__ __forceinline__ float exact_error16(const f32x2_t (&V)[8], float inv, float dq, uint32_t opaque_zero, uint2& nib) {
  const f32x2_t dq2 = pack2(dq, dq);
  float x[16], qa[8], qb[8];
  nib = trial16(V, inv, x);
  e2m1x8_unpacked(nib.x, opaque_zero, qa);
  e2m1x8_unpacked(nib.y, opaque_zero, qb);
  f32x2_t e[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const f32x2_t q = i < 4 ? pack2(qa[2 * i], qa[2 * i + 1]) : pack2(qb[2 * i - 8], qb[2 * i - 7]);
    const f32x2_t d = sub2(V[i], mul2_rounded(q, dq2));
    e[i] = mul2_rounded(d, d);
  }
  float a, b;  // e[i] + e[i + 8], then + 4, + 2, + 1: even places in one lane, odd ones in the other
  unpack2(add2(add2(add2(e[0], e[4]), add2(e[2], e[6])), add2(add2(e[1], e[5]), add2(e[3], e[7]))), a, b);
  return a + b;
}

__device__ __forceinline__ float2 e4m3x2_values(uint32_t codes) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(codes)));
  return __half22float2(*reinterpret_cast<__half2*>(&h2));
}

// Largest decoded magnitude of a group, (q * scale) * gs as the stand-alone NVFP4 amax kernel evaluates it
// (utils/nvfp4/quant/kernels/ms_eden/amax.rs:23-64): rounding to E2M1 is monotonic in |x|, so the largest nibble is the one of
// the element with the largest magnitude, ga.
__device__ __forceinline__ float decoded_max(float ga, float inv, float scale, float gs) {
  const float q = e2m1x2_values(cvt_e2m1x2(0.0f, ga * inv)).x;
  return fabsf(q * scale * gs);
}

// A group by the exact errors.  Not inlined: its registers would be the kernel's.
struct FourSixChoice {
  uint2 nib;
  uint32_t code;
  float inv, scale;
};
// codes: the two scale bytes (six in bits 0..7, four in bits 8..15) with their reciprocals
__device__ __noinline__ FourSixChoice exact_choice(const Group16 g, float gs, uint32_t codes, float inv6, float inv4, uint32_t opaque_zero) {
  const float2 s = e4m3x2_values(codes);
  uint2 nib6, nib4;
  const bool six = exact_error16(g.V, inv6, s.x * gs, opaque_zero, nib6) <= exact_error16(g.V, inv4, s.y * gs, opaque_zero, nib4);
  return {six ? nib6 : nib4, six ? codes & 0xffu : codes >> 8, six ? inv6 : inv4, six ? s.x : s.y};
}
// The same with the scale bytes, any values.
__device__ __noinline__ FourSixChoice exact_choice_any(const Group16 g, float ga, float gs, uint32_t opaque_zero) {
  const uint32_t b6 = cvt_e4m3(ga * 1.0f / (6.0f * gs + kDenomEps));
  const uint32_t b4 = cvt_e4m3(ga * 1.0f / (4.0f * gs + kDenomEps));
  return exact_choice(g, gs, b6 | (b4 << 8), inv_scale(e4m3_value(b6), gs), inv_scale(e4m3_value(b4), gs), opaque_zero);
}

// v: one 16-group, ga its amax.  Returns the scale byte and writes the 8 nibble bytes into `packed`.
// helpers.rs:42-76 and four_six.rs:309-344 of utils/nvfp4/quant/kernels.  The output nibbles are cvt(v * inv) with the
// chosen candidate's inv, i.e. exactly that candidate's trial bytes.
template <bool kPacked>
__device__ __forceinline__ uint32_t four_six_group(const float (&v)[16], float ga, const FourSixScale<kPacked>& sc, uint32_t opaque_zero,
                                                   uint2& packed, float* decoded_amax = nullptr) {
  uint32_t codes;
  {
    float q6, q4;
    if (kPacked) {
      unpack2(div_by_rcp2(pack2(ga, ga), sc.d, sc.y), q6, q4);
    } else {
      float d6, d4, y6, y4;
      unpack2(sc.d, d6, d4);
      unpack2(sc.y, y6, y4);
      q6 = div_by_rcp(ga, d6, y6);
      q4 = div_by_rcp(ga, d4, y4);
    }
    uint16_t c;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(c) : "f"(q4), "f"(q6));
    codes = c;
  }
  // a zero scale byte counts as one
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(static_cast<uint16_t>(codes)));
  const __half2 raw = *reinterpret_cast<const __half2*>(&h2);
  const float2 s = __half22float2(__hadd2(raw, __heq2(raw, __floats2half2_rn(0.0f, 0.0f))));
  float step6, step4, inv6, inv4;
  if (kPacked) {
    const f32x2_t step = mul2_rounded(pack2(s.x, s.y), pack2(sc.gs, sc.gs));
    unpack2(step, step6, step4);
    unpack2(rcp_in_range2(add2(step, pack2(kDenomEps, kDenomEps))), inv6, inv4);
  } else {
    step6 = s.x * sc.gs;
    step4 = s.y * sc.gs;
    inv6 = rcp_in_range(step6 + kDenomEps);
    inv4 = rcp_in_range(step4 + kDenomEps);
  }
  Group16 g;
#pragma unroll
  for (int i = 0; i < 8; ++i) g.V[i] = pack2(v[2 * i], v[2 * i + 1]);
  // How far the cheap errors can be off, with u = 2^-24, D the exact differences v - q dq and |q dq| <= |v| + |D| <= 2 |v|
  // (2-norms over the group; rounding to the grid never takes a value further than its own size), all in steps of "six":
  //   cheap: v * inv is v / dq within 4.6 u (1e-20 is below 1.5 u of a step of 2^-43 and more), then the difference, the
  //          products, the sums, and for "four" the ratio of the steps, its square and a product:
  //                                                      | sqrt(e) - |D| |   <= 4.6 u |v| + 7 u |D|
  //   exact: q dq, the difference, square and sums:      | sqrt(err) - |D| | <= 2 u |v| + 3.5 u |D|
  // A scale byte of zero stands for the step gs in v * inv and for dq = 0: all q are 0 then, D = v, and with gs as the step
  // the same bounds hold.  With |D| <= |v| <= 4 ga both candidates together shift sqrt(e6) - sqrt(e4) by less than 2 (4.6 + 7 + 2
  // + 3.5) 4 u ga < 137 u ga, and ga is at most 9 steps of "six" (the largest quotient that rounds to the smallest scale byte is 1.5
  // times it) unless both scale bytes saturate.  Multiplied by sqrt(e6) + sqrt(e4) <= sqrt(2 (e6 + e4)) and squared: the order is
  // certain where (e6 - e4)^2 exceeds 2 (1233 u)^2 < 2^-26.4 times e6 + e4, and is taken for certain beyond 2^-26.  Where the byte of
  // "six" alone is zero, the step of "four" is down to 2^-9 of it, 2^-52, and 1e-20 is below 757 u of that; but then ga is at most
  // 6 * 2^-10 steps of "six", and (137 + 4 * 757) u ga below 19 u.  Two candidates of one scale byte (zero groups, saturated ones) are
  // the same candidate: "six", where the error is a number, and the same bytes either way.  Otherwise -- NaN, scales and values
  // outside the range of the bounds -- the exact errors decide.
  bool certain = false;
  uint32_t code;
  float inv, scale;
  if (ga <= sc.limit && step6 >= 0x1p-43f) {
    uint2 nib6, nib4;
    const float e6 = candidate16(g, inv6, opaque_zero, nib6), e4 = candidate16(g, inv4, opaque_zero, nib4);
    const float ratio = step4 * inv6, e4_in_six = e4 * (ratio * ratio);
    const float gap = e6 - e4_in_six;
    const bool six = e6 <= e4_in_six;
    packed = six ? nib6 : nib4;
    code = six ? codes & 0xffu : codes >> 8;
    inv = six ? inv6 : inv4;
    scale = six ? s.x : s.y;
    certain = gap * gap > 0x1p-26f * (e6 + e4_in_six);
    if (!certain) certain = (codes & 0xffu) == codes >> 8 && e6 == e4;
  }
  if (!certain) {
    const FourSixChoice exact = ga <= sc.limit ? exact_choice(g, sc.gs, codes, inv6, inv4, opaque_zero)
                                               : exact_choice_any(g, ga, sc.gs, opaque_zero);
    packed = exact.nib;
    code = exact.code;
    inv = exact.inv;
    scale = exact.scale;
  }
  if (decoded_amax) *decoded_amax = decoded_max(ga, inv, scale, sc.gs);
  return code;
}

__device__ __forceinline__ float group_amax16(const float (&v)[16]) {
  float ga = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; i += 2) ga = max3_abs(ga, v[i], v[i + 1]);
  return ga;
}

// The stored words of a 16-group, widened as they are or as relu(x)^2 (max(x, 0) drops NaN like the reference's max_f32, the
// square is one rounded multiply); bf16 pairs meet the zero before they are widened.
template <typename T>
struct RawGroup;
template <>
struct RawGroup<float> {
  uint4 w[4];
  __device__ __forceinline__ void load(const float* p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
  }
  template <bool kRelu2>
  __device__ __forceinline__ void widen(float (&v)[16]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[4 * i] = __uint_as_float(w[i].x);
      v[4 * i + 1] = __uint_as_float(w[i].y);
      v[4 * i + 2] = __uint_as_float(w[i].z);
      v[4 * i + 3] = __uint_as_float(w[i].w);
    }
    if (kRelu2) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = max_f32(v[i], 0.0f);
      square_all(v);
    }
  }
  __device__ __forceinline__ static void square_all(float (&v)[16]) {
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const f32x2_t t = pack2(v[i], v[i + 1]);
      unpack2(mul2(t, t), v[i], v[i + 1]);
    }
  }
  template <bool kRelu2>
  __device__ __forceinline__ float amax() const {  // of the widened values
    float v[16];
    widen<kRelu2>(v);
    return group_amax16(v);
  }
};
template <>
struct RawGroup<__nv_bfloat16> {
  uint4 w[2];
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
#pragma unroll
    for (int i = 0; i < 2; ++i) w[i] = __ldg(reinterpret_cast<const uint4*>(p) + i);
  }
  template <bool kRelu2>
  __device__ __forceinline__ void widen(float (&v)[16]) const {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      uint32_t t[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (kRelu2) {
          const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&t[j]), __floats2bfloat162_rn(0.0f, 0.0f));
          t[j] = *reinterpret_cast<const uint32_t*>(&r);
        }
        v[8 * i + 2 * j] = widen_bf16_lo(t[j]);
        v[8 * i + 2 * j + 1] = widen_bf16_hi(t[j]);
      }
    }
    if (kRelu2) RawGroup<float>::square_all(v);
  }
  // Of the widened values, on packed pairs (a maximum rounds nothing and drops NaN; the largest square is that of the largest).
  template <bool kRelu2>
  __device__ __forceinline__ float amax() const {
    __nv_bfloat162 m = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t t[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&t[j]);
        m = __hmax2(m, kRelu2 ? b : __habs2(b));
      }
    }
    const float a = max_f32(__low2float(m), __high2float(m));
    return kRelu2 ? a * a : a;
  }
};

// What a quantizer reads: a group of 16 values of a stored tensor, relu(x)^2 of it (the MLP activation computed on load
// from the stored pre-activation: max(x, 0) drops NaN like the reference's max_f32, the square is one rounded multiply),
// or the schedule-free weight y = z + beta (x - z) of two f32 masters, which is never written out in f32
// (gpt/optimizer/schedule_free/{value,amax,four_six}.rs).
template <typename T, bool kRelu2>
struct TensorSource {
  const T* x;
  __device__ __forceinline__ void pin_loads() { x = after_prior(x); }
  struct Words {
    RawGroup<T> raw;
    __device__ __forceinline__ float amax() const { return raw.template amax<kRelu2>(); }
    __device__ __forceinline__ void widen(float (&v)[16]) const { raw.template widen<kRelu2>(v); }
  };
  __device__ __forceinline__ void load(size_t group, Words& w) const { w.raw.load(x + group * 16); }
  __device__ __forceinline__ void load16(size_t group, float (&v)[16]) const {
    Words w;
    load(group, w);
    w.widen(v);
  }
};
__device__ __forceinline__ float schedule_free_value(float z, float x, float beta) { return z + beta * (x - z); }
struct ScheduleFreeSource {
  const float* z;
  const float* x;
  float beta;
  __device__ __forceinline__ void pin_loads() {
    z = after_prior(z);
    x = after_prior(x);
  }
  __device__ __forceinline__ void load16(size_t group, float (&v)[16]) const {
    float zv[16], xv[16];
    Load16<float>::run(z + group * 16, zv);
    Load16<float>::run(x + group * 16, xv);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = schedule_free_value(zv[i], xv[i], beta);
  }
  struct Words {
    float value[16];
    __device__ __forceinline__ float amax() const { return group_amax16(value); }
    __device__ __forceinline__ void widen(float (&v)[16]) const {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = value[i];
    }
  };
  __device__ __forceinline__ void load(size_t group, Words& w) const { load16(group, w.value); }
};

// Scale bytes of four neighbouring lanes (one k-atom of a row) as one 32-bit store; every lane of the warp calls it.
__device__ __forceinline__ void store_scale_quad(uint8_t* dst, uint32_t byte, bool first_of_four) {
  uint32_t word = byte | (__shfl_down_sync(0xffffffffu, byte, 1) << 8);
  word |= __shfl_down_sync(0xffffffffu, word, 2) << 16;
  if (first_of_four) *reinterpret_cast<uint32_t*>(dst) = word;
}

// Max over `count` non-negative partial maxima, by the whole CTA (256 threads).
__device__ __forceinline__ float cta_max_of(const float* partials, uint32_t count) {
  if (count == 1) return partials[0];
  __shared__ uint32_t bits;
  if (threadIdx.x == 0) bits = 0u;
  __syncthreads();
  float m = 0.0f;
  for (uint32_t i = threadIdx.x; i < count; i += 256) m = max_f32(m, partials[i]);
  const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31u) == 0) atomicMax(&bits, w);
  __syncthreads();
  return __uint_as_float(bits);
}

// Rowwise four-six of rows that whole warps cover.  A warp takes 32 kGroups groups at a time, a lane kGroups of them: kRows = 2
// whole rows, a row, or, where the rows' maxima are given (kOwn = false), a part of one.  All of them are loaded before the first
// is quantized, the row maximum is a reduction of the warp, so that nothing ties the warps of a CTA together, and what depends
// on the row alone -- its maximum, its scale, the place of its scale bytes -- is computed once.  Bound by issue slots like its
// neighbours (16 instructions an element in place of 24, and four groups of a lane give the schedulers independent chains): bf16
// with own maxima 65536 x 768 46.4 -> 35.8 us, 8192 x 768 7.6 -> 5.9, 16384 x 2048 29.5 -> 20.7 (against a CTA per row block
// with a barrier, four_six_rowwise_kernel, which takes the other widths and few rows); relu^2 with given maxima
// 65536 x 3072 166 -> 146, 8192 x 4096 29.3 -> 25.3.  With 80 registers and three CTAs an SM 8192 x 768 took 8.1 us.
template <typename Source, bool kOwn, int kGroups, int kRows>
__global__ void __launch_bounds__(256, 2)
    four_six_rows_kernel(Source src, const float* __restrict__ amax, uint8_t* __restrict__ out_fp4, uint8_t* __restrict__ out_scales,
                         float* __restrict__ out_gs, float* __restrict__ out_amax, float* __restrict__ decoded_amax, uint32_t rows,
                         uint32_t plane_rows, uint32_t units, uint32_t groups_per_row, const FastDiv units_per_row,
                         int packed_scales, uint32_t opaque_zero) {
  static_assert(kOwn || kRows == 1, "parts of a row only where its maximum is given");
  wait_for_prior_then_allow_next();
  src.pin_loads();
  amax = after_prior(amax);
  constexpr uint32_t kRowGroups = 32 / kRows * kGroups;  // of a row in a unit
  const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * 8u;
  // this lane's groups inside a unit: row, scale byte
  bool in_second[kGroups];
  uint32_t scale_at[kGroups];
#pragma unroll
  for (int i = 0; i < kGroups; ++i) {
    const uint32_t g = lane + 32u * i;
    in_second[i] = kRows == 2 && g >= kRowGroups;
    const uint32_t kg = in_second[i] ? g - kRowGroups : g;
    scale_at[i] = packed_scales ? (kg >> 2) * 512u + (kg & 3u) + (in_second[i] ? 16u : 0u) : g;
  }
  float dec = 0.0f;
  for (uint32_t u = blockIdx.x * 8u + (threadIdx.x >> 5); u < units; u += warps) {
    const uint32_t row = kOwn ? u * kRows : units_per_row.div(u), kg0 = kOwn ? 0u : (u - row * units_per_row.d) * kRowGroups;
    const bool first = row < rows, second = kRows == 2 && row + 1 < rows;
    const size_t group = static_cast<size_t>(u) * (32u * kGroups) + lane;
    typename Source::Words words[kGroups] = {};
    float ga[kGroups], row_amax[kRows] = {};
    if (!kOwn && first) row_amax[0] = amax[row];
#pragma unroll
    for (int i = 0; i < kGroups; ++i)
      if (in_second[i] ? second : first) src.load(group + 32u * i, words[i]);
#pragma unroll
    for (int i = 0; i < kGroups; ++i) {
      ga[i] = words[i].amax();
      if (!kOwn) {
        continue;
      } else if (kRows == 1 || 32u * (i + 1) <= kRowGroups) {
        row_amax[0] = max_f32(row_amax[0], ga[i]);
      } else if (32u * i >= kRowGroups) {
        row_amax[kRows - 1] = max_f32(row_amax[kRows - 1], ga[i]);
      } else {
        row_amax[0] = max_f32(row_amax[0], in_second[i] ? 0.0f : ga[i]);
        row_amax[kRows - 1] = max_f32(row_amax[kRows - 1], in_second[i] ? ga[i] : 0.0f);
      }
    }
    FourSixScale<true> sc[kRows];
#pragma unroll
    for (int h = 0; h < kRows; ++h) {  // non-negative floats order like their bit patterns
      if (kOwn) row_amax[h] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(row_amax[h])));
      sc[h] = FourSixScale<true>(row_amax[h]);
    }
    if (kg0 == 0 && lane < kRows && row + lane < rows) {
      out_gs[row + lane] = lane ? sc[kRows - 1].gs : sc[0].gs;
      if (kOwn && out_amax) out_amax[row + lane] = lane ? row_amax[kRows - 1] : row_amax[0];
    }
    uint8_t* const scales = out_scales + (packed_scales ? packed_scale_offset(row, kg0, groups_per_row >> 2)
                                                             : static_cast<size_t>(row) * groups_per_row + kg0);
#pragma unroll
    for (int i = 0; i < kGroups; ++i) {
      float v[16], d;
      words[i].widen(v);
      FourSixScale<true> mine = sc[0];
      if (in_second[i]) mine = sc[kRows - 1];
      uint2 nibbles;
      uint32_t b = four_six_group(v, ga[i], mine, opaque_zero, nibbles, decoded_amax ? &d : nullptr);
      const bool inside = in_second[i] ? second : first;
      if (inside) *reinterpret_cast<uint2*>(out_fp4 + (group + 32u * i) * 8) = nibbles;
      if (inside && decoded_amax) dec = max_f32(dec, d);
      if (!inside) b = 0x38u;  // pad rows of a packed plane hold 1.0
      if (row + (in_second[i] ? 1u : 0u) < plane_rows) scales[scale_at[i]] = static_cast<uint8_t>(b);
    }
  }
  if (decoded_amax) cta_atomic_max(warp_max(dec), decoded_amax);  // uniform across the CTA
}

// One thread per 16-group and step over a [rows][cols] tensor; `groups` counts those of the pad rows too where the
// scales are packed (pad rows of the plane hold 1.0, the nibbles have none).  Rowwise: amax holds one value per row;
// otherwise `amax_count` partial maxima whose maximum is the tensor's, published in out_amax when asked for.
// decoded_amax (optional, zeroed by the launcher): max |decoded value| of the quantized tensor.
template <typename Source, bool kRowwise, bool kPacked, bool kQuads>
__global__ void __launch_bounds__(256, 4)
    four_six_kernel(Source src, const float* __restrict__ amax, uint32_t amax_count, float* __restrict__ out_amax,
                    uint8_t* __restrict__ out_fp4, uint8_t* __restrict__ out_scales, float* __restrict__ out_gs,
                    float* __restrict__ decoded_amax, uint32_t rows, uint32_t groups, const FastDiv groups_per_row,
                    uint32_t opaque_zero) {
  wait_for_prior_then_allow_next();
  src.pin_loads();
  amax = after_prior(amax);
  float dec = 0.0f;
  float tensor_amax = 0.0f;
  if (!kRowwise) {
    tensor_amax = cta_max_of(amax, amax_count);
    if (out_amax && blockIdx.x == 0 && threadIdx.x == 0) out_amax[0] = tensor_amax;
  }
  const FourSixScale<false> tensor_scale(tensor_amax);
  const uint32_t step = gridDim.x * 256u;
  // whole warps walk together: the scale bytes of neighbouring lanes leave in one store
  for (uint32_t g0 = blockIdx.x * 256u + (threadIdx.x & ~31u); g0 < groups; g0 += step) {
    const uint32_t g = g0 + (threadIdx.x & 31u);
    const uint32_t row = groups_per_row.div(g), kg = g - row * groups_per_row.d;
    const bool in_plane = g < groups;
    uint32_t b = 0x38u;
    if (in_plane && row < rows) {
      float v[16];
      src.load16(g, v);
      const FourSixScale<false> sc = kRowwise ? FourSixScale<false>(amax[row]) : tensor_scale;
      uint2 packed;
      float d;
      b = four_six_group(v, group_amax16(v), sc, opaque_zero, packed, decoded_amax ? &d : nullptr);
      if (decoded_amax) dec = max_f32(dec, d);
      *reinterpret_cast<uint2*>(out_fp4 + static_cast<size_t>(g) * 8) = packed;
      if (kRowwise ? (kg == 0) : (g == 0)) out_gs[kRowwise ? row : 0] = sc.gs;
    }
    uint8_t* const dst = out_scales + (kPacked ? packed_scale_offset(row, kg, groups_per_row.d >> 2) : static_cast<size_t>(g));
    if (kQuads)
      store_scale_quad(dst, b, in_plane && (kg & 3u) == 0);
    else if (in_plane)
      *dst = static_cast<uint8_t>(b);
    if (g0 + step < g0) break;  // the index space ends below 2^32
  }
  if (decoded_amax) cta_atomic_max(warp_max(dec), decoded_amax);  // uniform across the CTA
}

// Row amax and rowwise four-six in ONE pass over the input: a CTA owns whole rows (one thread per 16-group), the row
// amax is the shared-memory max of the group amaxes the quantizer needs anyway, and the groups are quantized from
// registers.  Same bytes as row_amax followed by the rowwise kernel
// (crates/gpt2-nvfp4/src/types/nvfp4_scratch/scratch.rs:35-52 issues those two).  CTAs walk row blocks blockIdx.x,
// blockIdx.x + gridDim.x, ... with the raw words of the next block in flight while the current one is quantized: one
// CTA-wide barrier per row block, the per-row maxima rotate through three shared-memory buffers so that clearing a
// buffer is always separated from its next use by a barrier.  Row blocks run on to the pad rows of a packed scale
// plane, which are written with 1.0.
// decoded_amax (optional, zeroed by the launcher): max |decoded value| of the whole quantized tensor, i.e. what
// utils/nvfp4/quant/kernels/ms_eden/amax.rs:23-64 computes from the stored tensor before the backward transposer --
// handed over so that pass can be skipped.
constexpr int kStreamMaxRowsPerCta = 256;
template <typename T, bool kPacked, bool kRelu2>
__global__ void __launch_bounds__(256, 3)
    four_six_rowwise_kernel(const T* __restrict__ x, uint8_t* __restrict__ out_fp4, uint8_t* __restrict__ out_scales,
                            float* __restrict__ out_gs, float* __restrict__ out_amax, float* __restrict__ decoded_amax,
                            uint32_t rows, uint32_t padded_rows, uint32_t groups_per_row, uint32_t rows_per_cta,
                            uint32_t row_blocks, uint32_t opaque_zero) {
  // What needs no memory of the kernel before this one comes ahead of the wait for it, and the first rows are in flight while
  // the shared memory is cleared: at the smallest sizes a launch is such latencies and little else (back to back, against all
  // of it behind the wait: bf16 16 x 768 1.90 -> 1.66 us, 1000 x 768 2.58 -> 2.48, 1000 x 3072 4.36 -> 4.06, f32 16 x 768
  // 2.07 -> 1.78, 500 x 3072 3.36 -> 3.21).
  __shared__ unsigned int row_amax_bits[3][kStreamMaxRowsPerCta];
  const uint32_t t = threadIdx.x, lane_id = t & 31u;
  const uint32_t local_row = t / groups_per_row;
  const uint32_t kg = t - local_row * groups_per_row;
  const bool in_use = local_row < rows_per_cta;
  // four neighbouring lanes hold four neighbouring scale bytes of one aligned word
  const bool quads = (groups_per_row & 3u) == 0 && (reinterpret_cast<uintptr_t>(out_scales) & 3u) == 0;
  const bool first_of_quad = (kg & 3u) == 0;
  // Row max: non-negative floats order like their bit patterns.  With at least 32 groups per row a warp touches at most two
  // rows: two warp-wide integer maxima, of the lanes in its first row and of the others, and an atomic max of one lane each.
  const bool two_rows = groups_per_row >= 32;
  const bool in_first = !two_rows || local_row == __shfl_sync(0xffffffffu, local_row, 0);
  const uint32_t other_lanes = __ballot_sync(0xffffffffu, !in_first && in_use);
  const bool leads_row = two_rows ? in_use && (lane_id == 0 || (other_lanes != 0u && lane_id + 1u == __ffs(other_lanes))) : in_use;

  uint32_t row = blockIdx.x * rows_per_cta + local_row;
  const uint32_t row_step = gridDim.x * rows_per_cta;
  size_t group = static_cast<size_t>(row) * groups_per_row + kg;
  const size_t group_step = static_cast<size_t>(row_step) * groups_per_row;
  wait_for_prior_then_allow_next();
  x = after_prior(x);
  RawGroup<T> raw = {};
  if (in_use && row < rows) raw.load(x + group * 16);
  for (uint32_t i = t; i < kStreamMaxRowsPerCta; i += blockDim.x) row_amax_bits[0][i] = row_amax_bits[1][i] = row_amax_bits[2][i] = 0u;
  __syncthreads();
  float dec_running = 0.0f;
  unsigned int *here = row_amax_bits[0], *next = row_amax_bits[1], *stale = row_amax_bits[2];
  for (uint32_t blk = blockIdx.x; blk < row_blocks; blk += gridDim.x, row += row_step, group += group_step) {
    const bool active = in_use && row < rows;
    float v[16];
    raw.template widen<kRelu2>(v);
    const float ga = group_amax16(v);
    // the next row block's words: in flight across the barrier and the whole quantization below (row numbers end below 2^32)
    if (in_use && row < rows - min(rows, row_step)) raw.load(x + (group + group_step) * 16);
    const uint32_t ga_bits = active ? __float_as_uint(ga) : 0u;
    uint32_t row_bits = ga_bits;
    if (two_rows) {
      row_bits = __reduce_max_sync(0xffffffffu, in_first ? ga_bits : 0u);
      if (other_lanes != 0u) {
        const uint32_t m_other = __reduce_max_sync(0xffffffffu, in_first ? 0u : ga_bits);
        if (!in_first) row_bits = m_other;
      }
    }
    if (leads_row) atomicMax(&here[local_row], row_bits);
    __syncthreads();
    // every thread is past its reads of the buffer of the previous row block: clear it for the block after next
    if (t < rows_per_cta) stale[t] = 0u;
    uint32_t b = 0x38u;
    if (active) {
      const float amax = __uint_as_float(here[local_row]);
      const FourSixScale<true> sc(amax);
      uint2 packed;
      float dec;
      b = four_six_group(v, ga, sc, opaque_zero, packed, decoded_amax ? &dec : nullptr);
      *reinterpret_cast<uint2*>(out_fp4 + group * 8) = packed;
      if (kg == 0) {
        out_gs[row] = sc.gs;
        if (out_amax) out_amax[row] = amax;
      }
      if (decoded_amax) dec_running = max_f32(dec_running, dec);
    }
    const bool in_plane = in_use && row < (kPacked ? padded_rows : rows);
    uint8_t* const dst = out_scales + (kPacked ? packed_scale_offset(row, kg, groups_per_row >> 2) : group);
    if (quads)
      store_scale_quad(dst, b, in_plane && first_of_quad);
    else if (in_plane)
      *dst = static_cast<uint8_t>(b);
    unsigned int* const done = here;
    here = next;
    next = stale;
    stale = done;
  }
  if (decoded_amax) {  // uniform across the CTA; the CTA may have fewer than eight warps
    __shared__ unsigned int dec_bits;
    if (t == 0) dec_bits = 0u;
    __syncthreads();
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(dec_running));
    if (lane_id == 0) atomicMax(&dec_bits, m);
    __syncthreads();
    if (t == 0) atomicMax(reinterpret_cast<unsigned int*>(decoded_amax), dec_bits);
  }
}

// Tensor amax of the schedule-free weight, 1024-value chunks per warp.
__global__ void __launch_bounds__(256) schedule_free_amax_kernel(const float* __restrict__ z,
                                                                  const float* __restrict__ x,
                                                                  float* __restrict__ chunk_amax, float* __restrict__ out,
                                                                  float* __restrict__ partials, float beta, uint64_t n) {
  wait_for_prior_then_allow_next();
  z = after_prior(z);
  x = after_prior(x);
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * 8;
  const uint64_t chunks = (n + 1023) / 1024;
  float running = 0.0f;
  for (uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); chunk < chunks; chunk += warps) {
    const uint64_t base = chunk * 1024;
    float m = 0.0f;
    if (base + 1024 <= n && ((reinterpret_cast<uintptr_t>(z + base) | reinterpret_cast<uintptr_t>(x + base)) & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(z + base) + i * 32 + lane);
        const float4 b = __ldg(reinterpret_cast<const float4*>(x + base) + i * 32 + lane);
        m = max3_abs(m, schedule_free_value(a.x, b.x, beta), schedule_free_value(a.y, b.y, beta));
        m = max3_abs(m, schedule_free_value(a.z, b.z, beta), schedule_free_value(a.w, b.w, beta));
      }
    } else {
      const uint32_t count = static_cast<uint32_t>(min(static_cast<uint64_t>(1024), n - base));
      for (uint32_t i = lane; i < count; i += 32)
        m = max_f32(m, fabsf(schedule_free_value(__ldg(z + base + i), __ldg(x + base + i), beta)));
    }
    m = warp_max(m);
    if (lane == 0 && chunk_amax) chunk_amax[chunk] = m;
    running = max_f32(running, m);
  }
  cta_publish_max(running, out, partials);
}

// Padded / transposed-padded variants: generic gather, zero outside the source extent.
// utils/nvfp4/quant/kernels/four_six.rs:110-142,173-211,346-395.
template <bool kTransposed>
__global__ void __launch_bounds__(256)
    four_six_padded_kernel(const float* __restrict__ x, const float* __restrict__ amax, uint8_t* __restrict__ out_fp4,
                           uint8_t* __restrict__ out_scales, float* __restrict__ out_gs, uint32_t rows, uint32_t cols,
                           uint32_t padded_cols, uint64_t group_count, uint32_t opaque_zero) {
  const uint64_t g = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (g >= group_count) return;
  const FourSixScale<false> sc(amax[0]);
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const uint64_t idx = g * 16 + i;
    const uint32_t r = static_cast<uint32_t>(idx / padded_cols);
    const uint32_t c = static_cast<uint32_t>(idx - static_cast<uint64_t>(r) * padded_cols);
    if (!kTransposed)
      v[i] = (r < rows && c < cols) ? x[static_cast<size_t>(r) * cols + c] : 0.0f;
    else
      v[i] = (r < cols && c < rows) ? x[static_cast<size_t>(c) * cols + r] : 0.0f;
  }
  uint2 packed;
  const uint32_t b = four_six_group(v, group_amax16(v), sc, opaque_zero, packed);
  *reinterpret_cast<uint2*>(out_fp4 + g * 8) = packed;
  out_scales[g] = static_cast<uint8_t>(b);
  if (g == 0) out_gs[0] = sc.gs;
}

// Fills the pad rows [rows, padded_rows) of a packed scale plane with 0x38 (= 1.0).
__global__ void __launch_bounds__(256) packed_scale_pad_kernel(uint8_t* __restrict__ packed, uint32_t rows,
                                                                uint32_t padded_rows, uint32_t k_groups) {
  const uint64_t total = static_cast<uint64_t>(padded_rows - rows) * k_groups;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * 256) {
    const uint32_t r = rows + static_cast<uint32_t>(i / k_groups);
    const uint32_t kg = static_cast<uint32_t>(i % k_groups);
    packed[packed_scale_offset(r, kg, k_groups >> 2)] = 0x38;
  }
}

// ============================================================================
// MS-EDEN
// ============================================================================

// Generic one-thread-per-chunk kernel (row sources, and the fallback for odd transposed
// shapes).  Input gathers follow utils/nvfp4/quant/kernels/ms_eden/input/padded.rs:9-96.
template <int kKind, typename T>
__global__ void __launch_bounds__(128) ms_eden_kernel(const MsEdenParams p) {
  const uint32_t chunks_per_row = p.out.dst_row_len >> 5;
  const uint64_t chunk_count = static_cast<uint64_t>(p.out.rows) * chunks_per_row;
  const uint64_t chunk = static_cast<uint64_t>(blockIdx.x) * 128 + threadIdx.x;
  if (chunk >= chunk_count) return;
  const uint32_t row = static_cast<uint32_t>(chunk / chunks_per_row);
  const uint32_t chunk_in_row = static_cast<uint32_t>(chunk - static_cast<uint64_t>(row) * chunks_per_row);
  const uint32_t col0 = chunk_in_row * 32;
  const float gs = p.use_host_scale ? p.global_scale_host : p.global_scale_dev[0];
  float u[32];
  if (kKind == 0) {
    const T* x = static_cast<const T*>(p.x) + static_cast<size_t>(row) * p.a;
    const bool full = col0 + 32 <= p.a && ((reinterpret_cast<uintptr_t>(x + col0) & 15u) == 0);
    if (full) {
      float lo[16], hi[16];
      Load16<T>::run(x + col0, lo);
      Load16<T>::run(x + col0 + 16, hi);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        u[j] = lo[j];
        u[16 + j] = hi[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) u[j] = (col0 + j < p.a) ? load_as_f32<T>(x, col0 + j) : 0.0f;
    }
  } else if (kKind == 1) {
    const T* x = static_cast<const T*>(p.x);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const uint32_t c = col0 + j;
      u[j] = (c < p.a) ? load_as_f32<T>(x, static_cast<size_t>(c) * p.b + row) : 0.0f;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const uint32_t c = col0 + j;
      if (c < p.a) {
        const float sg = (kKind == 2) ? p.src_global[0] : p.src_global[c];
        const size_t index = static_cast<size_t>(c) * p.b + row;
        const uint32_t byte = p.src_bytes[index >> 1];
        const uint32_t nib = (index & 1) ? (byte >> 4) : (byte & 0xfu);
        const size_t sidx = p.src_packed ? packed_scale_offset(c, row >> 4, p.b >> 6) : (index >> 4);
        u[j] = e2m1_value(nib) * e4m3_value(p.src_scales[sidx]) * sg;
      } else {
        u[j] = 0.0f;
      }
    }
  }
  uint32_t neg_mask = 0;  // x * (-1) == -x exactly: the random signs are applied as sign-bit flips
#pragma unroll
  for (int j = 0; j < 32; ++j)
    neg_mask |= (random_sign_negative(p.sign_seed, col0 + j + p.out.sign_offset) ? 1u : 0u) << j;
  f32x2_t P[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) P[i] = signed_pair(u[i], u[i + 16], neg_mask, i);
  ms_eden_emit_chunk(P, p.out, gs, p.scale_override, row, chunk_in_row);
}

// Tiled kernel for the transposed operands.  A CTA stages a [128 source rows x 64 source
// columns] tile in shared memory with coalesced 128-bit loads (decoding NVFP4 sources on the
// way), then each thread takes one 32-chunk DOWN a column (the transposed operand, K = source
// row) and, in pair mode, one 32-chunk ALONG a row (the row operand, K = source column): the
// source is read from memory once for both orientations, where the reference reads it twice
// and gathers the transposed half with a row-pitch stride
// (utils/nvfp4/quant/kernels/ms_eden/fp32_pair/dispatch.rs:13-43, input/padded.rs:9-96).
constexpr int kTileRows = 128, kTileCols = 64, kTileLd = kTileCols + 1;

template <int kSrc, typename T, bool kPair>
__global__ void __launch_bounds__(256) ms_eden_tile_kernel(const MsEdenTileParams p) {
  wait_for_prior_then_allow_next();
  __shared__ float tile[kTileRows * kTileLd];
  __shared__ uint32_t neg_r[kTileRows / 32];  // sign bits of the tile's rows (K of the transposed operand)
  __shared__ uint32_t neg_c[kTileCols / 32];  // sign bits of the tile's columns (K of the row operand)
  const uint32_t tid = threadIdx.x;
  const uint32_t c0 = blockIdx.x * kTileCols, r0 = blockIdx.y * kTileRows;
  if (tid < kTileRows) {
    const uint32_t bits = __ballot_sync(0xffffffffu, random_sign_negative(p.sign_seed, r0 + tid + p.t.sign_offset));
    if ((tid & 31) == 0) neg_r[tid >> 5] = bits;
  } else if (kPair && tid < kTileRows + kTileCols) {
    const uint32_t bits =
        __ballot_sync(0xffffffffu, random_sign_negative(p.sign_seed, c0 + (tid - kTileRows) + p.r.sign_offset));
    if ((tid & 31) == 0) neg_c[(tid - kTileRows) >> 5] = bits;
  }

  if (kSrc == 0) {
    const T* x = static_cast<const T*>(p.x);
    constexpr int V = VecTraits<T>::kPerVec;
    constexpr int kVecPerRow = kTileCols / V;
    const bool vec_ok = (p.src_cols % V == 0) && ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) &&
                        (c0 + kTileCols <= p.src_cols);
    for (uint32_t i = tid; i < kTileRows * kVecPerRow; i += 256) {
      const uint32_t row = i / kVecPerRow, v = i % kVecPerRow;
      const uint32_t r = r0 + row;
      float vals[V];
#pragma unroll
      for (int k = 0; k < V; ++k) vals[k] = 0.0f;
      if (r < p.src_rows) {
        const T* src = x + static_cast<size_t>(r) * p.src_cols + c0 + v * V;
        if (vec_ok) {
          if (V == 4) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(src));
            vals[0] = t.x, vals[1] = t.y, vals[2] = t.z, vals[3] = t.w;
          } else {
            const uint4 t = __ldg(reinterpret_cast<const uint4*>(src));
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              vals[(2 * k) % V] = __uint_as_float(w[k] << 16);
              vals[(2 * k + 1) % V] = __uint_as_float(w[k] & 0xffff0000u);
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < V; ++k)
            if (c0 + v * V + k < p.src_cols) vals[k] = load_as_f32<T>(src, k);
        }
      }
#pragma unroll
      for (int k = 0; k < V; ++k) tile[row * kTileLd + v * V + k] = vals[k];
    }
  } else {
    // NVFP4 source: per row of the tile 32 nibble bytes and 4 scale bytes; two threads per row
    const uint32_t row = tid >> 1, half = tid & 1;
    const uint32_t r = r0 + row, c = c0 + half * 32;
    float vals[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) vals[k] = 0.0f;
    if (r < p.src_rows) {
      const float sg = kSrc == 2 ? p.src_global[0] : p.src_global[r];
      const size_t index = static_cast<size_t>(r) * p.src_cols + c;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (c + 16 * g < p.src_cols) {
          const uint2 raw = __ldg(reinterpret_cast<const uint2*>(p.src_bytes + ((index + 16 * g) >> 1)));
          const size_t sidx = p.src_packed ? packed_scale_offset(r, (c >> 4) + g, p.src_cols >> 6) : (index >> 4) + g;
          const float sc = e4m3_value(p.src_scales[sidx]);
          const uint32_t w[2] = {raw.x, raw.y};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float2 q = e2m1x2_values((w[j >> 2] >> (8 * (j & 3))) & 0xffu);
            vals[16 * g + 2 * j] = q.x * sc * sg;
            vals[16 * g + 2 * j + 1] = q.y * sc * sg;
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) tile[row * kTileLd + half * 32 + k] = vals[k];
  }
  __syncthreads();

  if (kPair && p.col_sum_partials) {
    // Column sums of this tile (the bias gradient's partial sums), in a fixed order: four
    // sequential 32-row sums per column, then ((q0 + q1) + q2) + q3.
    __shared__ float quarter_sum[4][kTileCols];
    const uint32_t c = tid & 63, quarter = tid >> 6;
    float acc = 0.0f;
#pragma unroll 8
    for (int j = 0; j < 32; ++j) acc += tile[(quarter * 32 + j) * kTileLd + c];
    quarter_sum[quarter][c] = acc;
    __syncthreads();
    if (tid < kTileCols && c0 + tid < p.src_cols)
      p.col_sum_partials[static_cast<size_t>(blockIdx.y) * p.src_cols + c0 + tid] =
          ((quarter_sum[0][tid] + quarter_sum[1][tid]) + quarter_sum[2][tid]) + quarter_sum[3][tid];
  }

  const float gs = p.use_host_scale ? p.global_scale_host : p.global_scale_dev[0];
  {
    const uint32_t c = tid & 63, chunk = tid >> 6;
    const uint32_t out_row = c0 + c, k0 = r0 + chunk * 32;
    if (out_row < p.t.rows && k0 < p.t.dst_row_len) {
      const uint32_t mask = neg_r[chunk];
      f32x2_t P[16];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        P[i] = signed_pair(tile[(chunk * 32 + i) * kTileLd + c], tile[(chunk * 32 + i + 16) * kTileLd + c], mask, i);
      ms_eden_emit_chunk(P, p.t, gs, p.scale_override, out_row, k0 >> 5);
    }
  }
  if (kPair) {
    const uint32_t row = tid >> 1, chunk = tid & 1;
    const uint32_t out_row = r0 + row, k0 = c0 + chunk * 32;
    if (out_row < p.r.rows && k0 < p.r.dst_row_len) {
      const uint32_t mask = neg_c[chunk];
      f32x2_t P[16];
#pragma unroll
      for (int i = 0; i < 16; ++i)
        P[i] = signed_pair(tile[row * kTileLd + chunk * 32 + i], tile[row * kTileLd + chunk * 32 + i + 16], mask, i);
      ms_eden_emit_chunk(P, p.r, gs, p.scale_override, out_row, k0 >> 5);
    }
  }
}

// ReLU^2 backward between the two MLP linears (gpt/mlp/kernels.rs:72-104):
// d_pre = (d_out * 2) * max(pre, 0).  Element types: pre f32 / f16 / bf16, d_out and d_pre f32 / bf16
// (the reference has pre f32 | f16 with f32 gradients).  Eight elements per thread and step.
enum { kPreF32 = 0, kPreBf16 = 1, kPreF16 = 2 };

template <int kPre>
__device__ __forceinline__ void load8_pre(const void* p, size_t i, float (&v)[8]) {
  if (kPre == kPreF32) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p) + i));
    const float4 b = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p) + i) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
    const uint4 t = __ldg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p) + i));
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (kPre == kPreBf16) {
        v[2 * k] = __uint_as_float(w[k] << 16);
        v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
        v[2 * k] = f.x;
        v[2 * k + 1] = f.y;
      }
    }
  }
}
template <int kPre>
__device__ __forceinline__ float load1_pre(const void* p, size_t i) {
  if (kPre == kPreF32) return __ldg(static_cast<const float*>(p) + i);
  const uint16_t h = __ldg(static_cast<const uint16_t*>(p) + i);
  if (kPre == kPreBf16) return __uint_as_float(static_cast<uint32_t>(h) << 16);
  return __half2float(__ushort_as_half(h));
}
template <bool kBf16>
__device__ __forceinline__ void store8_grad(void* p, size_t i, const float (&v)[8]) {
  if (!kBf16) {
    float4* q = reinterpret_cast<float4*>(static_cast<float*>(p) + i);
    q[0] = make_float4(v[0], v[1], v[2], v[3]);
    q[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
      w[k] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p) + i) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// With chunk_amax set the kernel also emits, per CTA, the amax of the values it stored (after their rounding to
// the gradient type): the chunk list nvfp4_linear_backward_ms_eden accepts in place of its own amax pass over dY
// (the hand-over gpt/loss/kernels.rs:67-88 -> backward/final_head/run.rs:34,54 makes for the loss gradient).
template <int kPre, bool kGradBf16, bool kAmax>
__global__ void __launch_bounds__(256) relu2_backward_kernel(const void* __restrict__ pre, const void* __restrict__ d_out,
                                                              void* __restrict__ d_pre, uint64_t n, int vectorized,
                                                              float* __restrict__ chunk_amax) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * 256;
  const uint64_t tid = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
  const uint64_t vec_n = vectorized ? n / 8 : 0;
  float m = 0.0f;
  for (uint64_t i = tid; i < vec_n; i += stride) {
    float p[8], d[8], r[8];
    load8_pre<kPre>(pre, i * 8, p);
    load8_pre<kGradBf16 ? kPreBf16 : kPreF32>(d_out, i * 8, d);
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = (d[k] * 2.0f) * max_f32(p[k], 0.0f);
    store8_grad<kGradBf16>(d_pre, i * 8, r);
    if (kAmax) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float stored = kGradBf16 ? __bfloat162float(__float2bfloat16_rn(r[k])) : r[k];
        m = max_f32(m, fabsf(stored));
      }
    }
  }
  for (uint64_t i = vec_n * 8 + tid; i < n; i += stride) {
    const float p = load1_pre<kPre>(pre, i);
    const float d = load1_pre<kGradBf16 ? kPreBf16 : kPreF32>(d_out, i);
    const float r = (d * 2.0f) * max_f32(p, 0.0f);
    float stored = r;
    if (kGradBf16) {
      const __nv_bfloat16 h = __float2bfloat16_rn(r);
      static_cast<__nv_bfloat16*>(d_pre)[i] = h;
      stored = __bfloat162float(h);
    } else {
      static_cast<float*>(d_pre)[i] = r;
    }
    if (kAmax) m = max_f32(m, fabsf(stored));
  }
  if (kAmax) {
    __shared__ float partial[8];
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      float r = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) r = max_f32(r, partial[i]);
      chunk_amax[blockIdx.x] = r;
    }
  }
}

// ============================================================================
// decode, scale pack, padding, post-ops, bias gradient
// ============================================================================

// utils/nvfp4/decode/kernels.rs:11-57
__global__ void __launch_bounds__(256) decode_kernel(const uint8_t* __restrict__ bytes,
                                                      const uint8_t* __restrict__ scales,
                                                      const float* __restrict__ gscales, float* __restrict__ out,
                                                      uint32_t rows, uint32_t cols, int rowwise, int transpose) {
  const uint64_t idx = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (idx >= n) return;
  const uint32_t r = static_cast<uint32_t>(idx / cols), c = static_cast<uint32_t>(idx % cols);
  const float v = nvfp4_value(bytes, scales, rowwise ? gscales[r] : gscales[0], idx);
  out[transpose ? static_cast<size_t>(c) * rows + r : idx] = v;
}

// Row-major decode, eight elements (one 32-byte store) per thread and step, four steps in flight: one element per thread
// spent its time on index arithmetic and four-byte accesses (8192 x 768: 23 us; this form 5.5 us, HBM allows 4.4).
__global__ void __launch_bounds__(256) decode_rows_kernel(const uint8_t* __restrict__ bytes, const uint8_t* __restrict__ scales,
                                                           const float* __restrict__ gscales, float* __restrict__ out,
                                                           uint32_t octets, const FastDiv octets_per_row, int rowwise) {
  wait_for_prior_then_allow_next();
  bytes = after_prior(bytes);
  scales = after_prior(scales);
  gscales = after_prior(gscales);
  const float tensor_gs = rowwise ? 0.0f : gscales[0];
  for (uint32_t i0 = blockIdx.x * 1024u + threadIdx.x; i0 < octets; i0 += gridDim.x * 1024u) {
    uint32_t word[4], sc[4];
    float gs[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t i = i0 + 256u * k;
      if (i < octets && i >= i0) {
        word[k] = __ldg(reinterpret_cast<const uint32_t*>(bytes) + i);
        sc[k] = __ldg(scales + (i >> 1));
        gs[k] = rowwise ? __ldg(gscales + octets_per_row.div(i)) : tensor_gs;
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint32_t i = i0 + 256u * k;
      if (i < octets && i >= i0) {
        float q[8];
        e2m1x8_values(word[k], q);
        const float s = e4m3_value(sc[k]);
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __float_as_uint(q[j] * s * gs[k]);
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + static_cast<size_t>(i) * 8),
                     "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
      }
    }
    if (i0 + gridDim.x * 1024u < i0) break;
  }
}

// One [128 rows x 16 k-atoms] block of a logical scale plane into its sixteen packed 512-byte tiles, through shared
// memory: 64-byte row segments in, whole tiles out (a byte per thread gathered one byte per 4-byte access and wrote
// single bytes 16 apart: 8192 x 8192 8.9 us; this form 3.1 us).
// The row blocks of a second plane may follow those of the first in the same launch: a GEMM whose two operands carry
// logical scales packs both in 6.5 us instead of twice that (planes of 0.5 to 2 MB cost their latency, not their bytes).
struct ScalePlane {
  const uint8_t* logical;
  uint8_t* packed;
  uint32_t mn, row_blocks;
};
__global__ void __launch_bounds__(256) scale_pack_tiles_kernel(const ScalePlane first, const ScalePlane second, uint32_t k_atoms) {
  wait_for_prior_then_allow_next();
  __shared__ uint32_t words[128][17];
  const bool is_first = blockIdx.y < first.row_blocks;
  const uint8_t* const logical = after_prior(is_first ? first.logical : second.logical);
  uint8_t* const packed = is_first ? first.packed : second.packed;
  const uint32_t mn = is_first ? first.mn : second.mn, row_block = is_first ? blockIdx.y : blockIdx.y - first.row_blocks;
  const uint32_t atom0 = blockIdx.x * 16u, row0 = row_block * 128u;
  const uint32_t atoms = min(16u, k_atoms - atom0);
  const uint32_t w = threadIdx.x & 15u;
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k) {
    const uint32_t r = (threadIdx.x >> 4) + 16u * k;
    if (w < atoms)
      words[r][w] = row0 + r < mn ? __ldg(reinterpret_cast<const uint32_t*>(logical) + static_cast<size_t>(row0 + r) * k_atoms + atom0 + w)
                                  : 0x38383838u;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < 2; ++k) {
    const uint32_t i = threadIdx.x + 256u * k, atom = i >> 5, l = i & 31u;
    if (atom < atoms)
      reinterpret_cast<uint4*>(packed)[(static_cast<size_t>(row_block) * k_atoms + atom0 + atom) * 32u + l] =
          make_uint4(words[l][atom], words[l + 32][atom], words[l + 64][atom], words[l + 96][atom]);
  }
}

// utils/nvfp4_tma_matmul/scale_pack.rs:14-40
__global__ void __launch_bounds__(256) scale_pack_kernel(const uint8_t* __restrict__ logical,
                                                          uint8_t* __restrict__ packed, uint32_t mn, uint32_t padded_mn,
                                                          uint32_t k_groups) {
  const uint64_t total = static_cast<uint64_t>(padded_mn) * k_groups;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * 256) {
    const uint32_t r = static_cast<uint32_t>(i / k_groups), kg = static_cast<uint32_t>(i % k_groups);
    packed[packed_scale_offset(r, kg, k_groups >> 2)] = r < mn ? logical[i] : 0x38;
  }
}

// utils/nvfp4_tma_matmul/pad.rs:115-210
__global__ void __launch_bounds__(256) pad_u4_rows_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst,
                                                           uint64_t src_bytes, uint64_t dst_bytes) {
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < dst_bytes;
       i += static_cast<uint64_t>(gridDim.x) * 256)
    dst[i] = i < src_bytes ? src[i] : 0;
}
template <bool kTranspose>
__global__ void __launch_bounds__(256) pad_f32_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                       uint32_t rows, uint32_t cols, uint32_t padded_rows,
                                                       uint32_t padded_cols) {
  const uint64_t total = static_cast<uint64_t>(padded_rows) * padded_cols;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * 256) {
    const uint32_t r = static_cast<uint32_t>(i / padded_cols), c = static_cast<uint32_t>(i % padded_cols);
    float v = 0.0f;
    if (!kTranspose) {
      if (r < rows && c < cols) v = src[static_cast<size_t>(r) * cols + c];
    } else {
      if (r < cols && c < rows) v = src[static_cast<size_t>(c) * cols + r];
    }
    dst[i] = v;
  }
}
__global__ void __launch_bounds__(256) crop_f32_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                        uint32_t rows, uint32_t src_cols, uint32_t dst_cols) {
  const uint64_t total = static_cast<uint64_t>(rows) * dst_cols;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * 256) {
    const uint32_t r = static_cast<uint32_t>(i / dst_cols), c = static_cast<uint32_t>(i % dst_cols);
    dst[i] = src[static_cast<size_t>(r) * src_cols + c];
  }
}

// gpt/projection_postop.rs:97-162.  mode 0: raw += bias; 1: residual = fma(1, raw + bias, residual);
// 2: pre = raw + bias (in place), out = max(pre, 0)^2.
__global__ void __launch_bounds__(256) postop_kernel(float* __restrict__ raw, float* __restrict__ other,
                                                      const uint8_t* __restrict__ bias_bytes,
                                                      const uint8_t* __restrict__ bias_scales,
                                                      const float* __restrict__ bias_gs, uint64_t n, uint32_t cols,
                                                      int mode) {
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < n;
       i += static_cast<uint64_t>(gridDim.x) * 256) {
    const uint32_t col = static_cast<uint32_t>(i % cols);
    const float bias = nvfp4_value(bias_bytes, bias_scales, bias_gs[0], col);
    if (mode == 0) {
      raw[i] = raw[i] + bias;
    } else if (mode == 1) {
      other[i] = __fmaf_rn(1.0f, raw[i] + bias, other[i]);
    } else {
      const float pre = raw[i] + bias;
      const float r = max_f32(pre, 0.0f);
      raw[i] = pre;
      other[i] = r * r;
    }
  }
}

// gpt/linear_backward/bias.rs:18-69: 8 row lanes x 32 columns per CTA; each row lane sums
// rows lane, lane+8, ... in order; the 8 lane sums are then added left to right.
template <typename T>
__global__ void __launch_bounds__(256) bias_grad_kernel(const T* __restrict__ e, float* __restrict__ dbias,
                                                         uint32_t tokens, uint32_t n) {
  __shared__ float sums[256];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t col = blockIdx.x * 32 + lane;
  float local = 0.0f;
  if (col < n) {
    uint32_t row = w;
    for (; row + 8 * 7 < tokens; row += 64) {
      float t[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) t[i] = load_as_f32<T>(e, static_cast<size_t>(row + 8 * i) * n + col);
#pragma unroll
      for (int i = 0; i < 8; ++i) local += t[i];
    }
    for (; row < tokens; row += 8) local += load_as_f32<T>(e, static_cast<size_t>(row) * n + col);
  }
  sums[threadIdx.x] = local;
  __syncthreads();
  if (w == 0 && col < n) {
    float s = sums[lane];
#pragma unroll
    for (int i = 1; i < 8; ++i) s = s + sums[lane + 32 * i];
    dbias[col] = s;
  }
}

// dbias[c] = sum over row tiles of the tile column sums in a fixed order: eight lanes per
// column each add tiles lane, lane+8, ... in sequence, then the lane sums are added 0..7.
__global__ void __launch_bounds__(256) col_sum_reduce_kernel(const float* __restrict__ partials,
                                                              float* __restrict__ dbias, uint32_t tiles, uint32_t n) {
  wait_for_prior_then_allow_next();
  partials = after_prior(partials);
  __shared__ float sums[256];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * 32 + lane;
  float acc = 0.0f;
  if (c < n) {
    // sixteen loads in flight per thread, added in tile order (the loads dominate: few CTAs, long latency)
    uint32_t t = w;
    for (; t + 8 * 15 < tiles; t += 8 * 16) {
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __ldg(partials + static_cast<size_t>(t + 8 * j) * n + c);
#pragma unroll
      for (int j = 0; j < 16; ++j) acc += v[j];
    }
    for (; t < tiles; t += 8) acc += __ldg(partials + static_cast<size_t>(t) * n + c);
  }
  sums[threadIdx.x] = acc;
  __syncthreads();
  if (w == 0 && c < n) {
    float r = sums[lane];
#pragma unroll
    for (int i = 1; i < 8; ++i) r = r + sums[lane + 32 * i];
    dbias[c] = r;
  }
}

// ============================================================================
// launchers
// ============================================================================

static inline uint32_t blocks_for(uint64_t n, uint32_t per_block, uint32_t cap = 0x7fffffffu) {
  uint64_t b = (n + per_block - 1) / per_block;
  if (b == 0) b = 1;
  return static_cast<uint32_t>(b > cap ? cap : b);
}

#define NVFP4_RETURN_LAST() \
  do {                       \
    count_launch();          \
    return static_cast<int>(cudaGetLastError()); \
  } while (0)

int launch_row_amax(cudaStream_t s, const void* x, int dtype, float* out, uint32_t rows, uint32_t row_len) {
  if (rows == 0) return 0;
  if (dtype == 0)
    return launch_chained(row_amax_kernel<float>, blocks_for(rows, 8), 256, 0, s, static_cast<const float*>(x), out, rows, row_len);
  return launch_chained(row_amax_kernel<__nv_bfloat16>, blocks_for(rows, 8), 256, 0, s, static_cast<const __nv_bfloat16*>(x), out,
                        rows, row_len);
}

uint32_t tensor_amax_partials(uint64_t n, uint32_t max_partials) { return blocks_for((n + 1023) / 1024, 8, max_partials); }

int launch_tensor_amax(cudaStream_t s, const void* x, int dtype, float* chunk_amax, float* out, uint64_t n, float* partials,
                       uint32_t max_partials) {
  if (!partials) {
    const cudaError_t err = cudaMemsetAsync(out, 0, sizeof(float), s);
    if (err != cudaSuccess) return static_cast<int>(err);
    if (n == 0) return 0;
  }
  const uint32_t grid = partials ? tensor_amax_partials(n, max_partials) : blocks_for((n + 1023) / 1024, 8, 148 * 8);
  if (dtype == 0)
    return launch_chained(tensor_amax_kernel<float>, grid, 256, 0, s, static_cast<const float*>(x), chunk_amax, out, partials, n);
  return launch_chained(tensor_amax_kernel<__nv_bfloat16>, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(x), chunk_amax, out,
                        partials, n);
}

int launch_nvfp4_amax(cudaStream_t s, const uint8_t* bytes, const uint8_t* scales, const float* gscales, uint32_t rows,
                      uint32_t cols, int rowwise, int packed, float* chunk_amax, float* out, float* partials,
                      bool out_cleared) {
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (!partials) {
    if (!out_cleared) {
      const cudaError_t err = cudaMemsetAsync(out, 0, sizeof(float), s);
      if (err != cudaSuccess) return static_cast<int>(err);
    }
    if (n == 0) return 0;
  }
  return launch_chained(nvfp4_amax_kernel, tensor_amax_partials(n, kAmaxScratchPartials), 256, 0, s, bytes, scales, gscales, n, cols,
                        rowwise, packed, chunk_amax, out, partials);
}

int launch_amax_from_chunks(cudaStream_t s, const float* chunk_amax, float* out, uint32_t chunk_count, int transform) {
  return launch_chained(amax_from_chunks_kernel, 1, 256, 0, s, chunk_amax, out, chunk_count, transform);
}

int launch_ms_eden_scale_from_amax(cudaStream_t s, const float* amax, float* out) {
  return launch_chained(ms_eden_scale_from_amax_kernel, 1, 1, 0, s, amax, out);
}

// Groups of one launch stay below 2^32 (32-bit index space): larger tensors go in slabs of whole 128-row blocks.
template <typename Source>
static Source advance(const Source& s, size_t elements);
template <>
TensorSource<float, false> advance(const TensorSource<float, false>& s, size_t n) { return {s.x + n}; }
template <>
TensorSource<float, true> advance(const TensorSource<float, true>& s, size_t n) { return {s.x + n}; }
template <>
TensorSource<__nv_bfloat16, false> advance(const TensorSource<__nv_bfloat16, false>& s, size_t n) { return {s.x + n}; }
template <>
TensorSource<__nv_bfloat16, true> advance(const TensorSource<__nv_bfloat16, true>& s, size_t n) { return {s.x + n}; }
template <>
ScheduleFreeSource advance(const ScheduleFreeSource& s, size_t n) { return {s.z + n, s.x + n, s.beta}; }

template <typename Source, bool kOwn, int kGroups, int kRows>
static int launch_four_six_rows(cudaStream_t s, const Source& src, const float* amax, uint32_t rows, uint32_t plane_rows, uint32_t gpr,
                                uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs, float* out_amax, float* decoded_amax) {
  const uint32_t per_row = kRows == 2 ? 1u : gpr / (32 * kGroups);
  const uint32_t units = kRows == 2 ? (plane_rows + 1) / 2 : plane_rows * per_row;
  // Every resident CTA of eight warps: an SM's units are what counts.  Fewer CTAs, each with the same number of units, put two of
  // them on some SMs and one on the others: 2368 x 2048 bf16 6.5 -> 5.0 us, 1184 x 8192 with given maxima 9.2 -> 7.6.
  const uint32_t grid = min((units + 7u) / 8u, 148u * 2u);
  return launch_chained(four_six_rows_kernel<Source, kOwn, kGroups, kRows>, grid, 256, 0, s, src, amax, out_fp4, out_scales, out_gs,
                        out_amax, decoded_amax, rows, plane_rows, units, gpr, FastDiv(per_row), packed, 0u);
}
// -1: no form of the kernel takes such rows
template <typename Source>
static int launch_four_six_own_rows(cudaStream_t s, const Source& src, uint32_t rows, uint32_t plane_rows, uint32_t gpr, uint8_t* out_fp4,
                                    uint8_t* out_scales, int packed, float* out_gs, float* out_amax, float* decoded_amax) {
  // Fewer than four warps an SM leave most of it idle while a lane quantizes its groups one after the other.  With three groups of
  // two rows or four of one, whose chains are the longest, four_six_rowwise_kernel is the faster one as long as its CTAs are all
  // resident (444 of five and two rows), and from 1185 to 1776 rows of 128 groups, where it needs its second turn and this kernel a
  // second CTA on the SMs; us there and here, bf16: 1000 x 768 2.61, 2.85; 2048 x 768 2.74, 2.83; 2368 x 768 4.08, 3.48; 640 x 2048
  // 2.69, 2.91; 1000 x 2048 4.05, 3.00; 1300 x 2048 4.09, 4.07 (f32 4.64, 5.05); 1776 x 2048 5.36, 4.17.
  if (plane_rows / (gpr == 16 || gpr == 48 ? 2u : 1u) < 148u * 4u) return -1;
  if (gpr == 48 && plane_rows <= 444u * 5u) return -1;
  if (gpr == 128 && (plane_rows <= 444u * 2u || (plane_rows > 148u * 8u && plane_rows <= 444u * 4u))) return -1;
#define NVFP4_ROWS(G, R)                                                                                                    \
  return launch_four_six_rows<Source, true, G, R>(s, src, nullptr, rows, plane_rows, gpr, out_fp4, out_scales, packed, out_gs, \
                                                  out_amax, decoded_amax)
  switch (gpr) {
    case 16: NVFP4_ROWS(1, 2);
    case 32: NVFP4_ROWS(1, 1);
    case 48: NVFP4_ROWS(3, 2);
    case 64: NVFP4_ROWS(2, 1);
    case 96: NVFP4_ROWS(3, 1);
    case 128: NVFP4_ROWS(4, 1);
    default: return -1;
  }
#undef NVFP4_ROWS
}
// Sources whose rows with given maxima go to four_six_rows_kernel.
template <typename Source>
struct TakesGivenRows {
  static constexpr bool value = false;
};
template <bool kRelu2>
struct TakesGivenRows<TensorSource<__nv_bfloat16, kRelu2>> {
  static constexpr bool value = true;
};

template <typename Source>
static int launch_four_six_source(cudaStream_t s, const Source& src, const float* amax, uint32_t amax_count, float* out_amax,
                                  int rowwise, uint32_t rows, uint32_t cols, uint8_t* out_fp4, uint8_t* out_scales, int packed,
                                  float* out_gs, float* decoded_amax) {
  const uint32_t gpr = cols / 16;
  const uint64_t limit = 0xfff00000ull;
  const uint64_t slab_rows = limit / gpr >= 128 ? limit / gpr / 128 * 128 : limit / gpr;
  if (rows > slab_rows) {
    if (packed && slab_rows < 128) return static_cast<int>(cudaErrorInvalidValue);  // 2^36 elements: beyond the memory
    for (uint64_t r = 0; r < rows; r += slab_rows) {
      const uint32_t n = static_cast<uint32_t>(rows - r < slab_rows ? rows - r : slab_rows);
      const size_t g = static_cast<size_t>(r) * gpr;
      const int rc = launch_four_six_source(s, advance(src, g * 16), rowwise ? amax + r : amax, amax_count, out_amax, rowwise, n,
                                            cols, out_fp4 + g * 8, out_scales + g, packed, rowwise ? out_gs + r : out_gs, decoded_amax);
      if (rc) return rc;
    }
    return 0;
  }
  // few but very long rows: the plane's pad rows alone would leave the index space, they get their own launch
  const uint64_t plane_rows = packed ? (rows + 127u) / 128u * 128u : rows;
  const bool pad_apart = plane_rows * gpr > limit;
  const uint32_t groups = static_cast<uint32_t>((pad_apart ? rows : plane_rows) * gpr);
  if constexpr (TakesGivenRows<Source>::value) {
    // bf16 sources; f32 ones are bound by HBM and L2 as they are (4096 x 8192 26.5 us one group at a time, 26.8 and more by
    // rows).  A warp takes several groups of every lane at a time, so this pays where most warps have work in each turn, or there
    // are many turns: plain and relu^2 us one group at a time and by rows, 888 x 6144 5.1, 6.1 and 5.4, 6.7; 1100 x 3072 4.3, 5.1 and
    // 3.4, 4.3; 3000 x 4096 9.4, 11.3 and 9.3, 11.6; 8192 x 3072 17.6, 21.1 and 15.3, 18.9.  Two groups a lane gain less: 8192 x 1024
    // 6.8, 8.2 and 7.0, 8.7; 16384 x 1024 12.3, 14.8 and 11.4, 13.9.
    const uint64_t warps = 148u * 16u, form = gpr % 128 == 0 ? 4u : gpr % 96 == 0 ? 3u : 2u, units = plane_rows * (gpr / (32u * form));
    const uint64_t turns = (units + warps - 1) / warps;
    const bool by_rows = turns > (form == 2u ? 4u : 3u) || units * 10u >= turns * warps * (form > 2u && turns == 1 ? 8u : 9u);
    if (rowwise && (gpr % 64 == 0 || gpr % 96 == 0) && by_rows) {
      const uint32_t launched_rows = static_cast<uint32_t>(pad_apart ? rows : plane_rows);
      const auto launch = form == 4u   ? launch_four_six_rows<Source, false, 4, 1>
                          : form == 3u ? launch_four_six_rows<Source, false, 3, 1>
                                       : launch_four_six_rows<Source, false, 2, 1>;
      const int rc = launch(s, src, amax, rows, launched_rows, gpr, out_fp4, out_scales, packed, out_gs, nullptr, decoded_amax);
      return rc == 0 && pad_apart ? launch_packed_scale_pad(s, out_scales, rows, cols) : rc;
    }
  }
  // one wave of resident CTAs where the prologue reduces partial maxima or the tensor is large; each thread then walks
  const uint32_t grid = blocks_for(groups, 256, 148u * 4u);
  const bool quads = gpr % 4 == 0 && (reinterpret_cast<uintptr_t>(out_scales) & 3u) == 0;
  const FastDiv div(gpr);
  int rc;
#define NVFP4_LAUNCH_FS(R, P, Q)                                                                                          \
  rc = launch_chained(four_six_kernel<Source, R, P, Q>, grid, 256, 0, s, src, amax, amax_count, out_amax, out_fp4,         \
                      out_scales, out_gs, decoded_amax, rows, groups, div, 0u)
  if (rowwise) {
    if (packed) { if (quads) NVFP4_LAUNCH_FS(true, true, true); else NVFP4_LAUNCH_FS(true, true, false); }
    else { if (quads) NVFP4_LAUNCH_FS(true, false, true); else NVFP4_LAUNCH_FS(true, false, false); }
  } else {
    if (packed) { if (quads) NVFP4_LAUNCH_FS(false, true, true); else NVFP4_LAUNCH_FS(false, true, false); }
    else { if (quads) NVFP4_LAUNCH_FS(false, false, true); else NVFP4_LAUNCH_FS(false, false, false); }
  }
#undef NVFP4_LAUNCH_FS
  return rc == 0 && pad_apart ? launch_packed_scale_pad(s, out_scales, rows, cols) : rc;
}

int launch_four_six(cudaStream_t s, const void* x, int dtype, const float* amax, int rowwise, uint32_t rows,
                    uint32_t cols, uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs, int relu2,
                    float* decoded_amax, uint32_t amax_count, bool decoded_cleared) {
  if (decoded_amax && !decoded_cleared) {
    const cudaError_t err = cudaMemsetAsync(decoded_amax, 0, sizeof(float), s);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  if (rows == 0 || cols == 0) return 0;
#define NVFP4_FS_SOURCE(T, R)                                                                                              \
  launch_four_six_source(s, TensorSource<T, R>{static_cast<const T*>(x)}, amax, amax_count, nullptr, rowwise, rows, cols,   \
                         out_fp4, out_scales, packed, out_gs, decoded_amax)
  if (dtype == NVFP4_DTYPE_F32) return relu2 ? NVFP4_FS_SOURCE(float, true) : NVFP4_FS_SOURCE(float, false);
  return relu2 ? NVFP4_FS_SOURCE(__nv_bfloat16, true) : NVFP4_FS_SOURCE(__nv_bfloat16, false);
#undef NVFP4_FS_SOURCE
}

// Fused row amax + rowwise four-six.  Returns -1 when the row is too long for one CTA (the
// caller then runs the two-kernel path).
int launch_four_six_rowwise_fused(cudaStream_t s, const void* x, int dtype, uint32_t rows, uint32_t cols,
                                  uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs, float* out_amax,
                                  float* decoded_amax, int relu2, bool decoded_cleared) {
  const uint32_t gpr = cols / 16;
  if (gpr == 0 || gpr > 256) return -1;
  if (decoded_amax && !decoded_cleared) {
    const cudaError_t err = cudaMemsetAsync(decoded_amax, 0, sizeof(float), s);
    if (err != cudaSuccess) return static_cast<int>(err);
  }
  if (rows == 0) return 0;
  const uint64_t plane_rows = packed ? (static_cast<uint64_t>(rows) + 127u) / 128u * 128u : rows;
  if (plane_rows * gpr <= 0xfff00000ull) {
    const uint32_t plane = static_cast<uint32_t>(plane_rows);
#define NVFP4_OWN_ROWS(T, R)                                                                                          \
  launch_four_six_own_rows(s, TensorSource<T, R>{static_cast<const T*>(x)}, rows, plane, gpr, out_fp4, out_scales, packed, \
                           out_gs, out_amax, decoded_amax)
    const int rc = dtype == NVFP4_DTYPE_F32 ? (relu2 ? NVFP4_OWN_ROWS(float, true) : NVFP4_OWN_ROWS(float, false))
                                            : (relu2 ? NVFP4_OWN_ROWS(__nv_bfloat16, true) : NVFP4_OWN_ROWS(__nv_bfloat16, false));
#undef NVFP4_OWN_ROWS
    if (rc >= 0) return rc;
  }
  const uint32_t rpc = 256 / gpr;
  const uint32_t threads = (rpc * gpr + 31) / 32 * 32;
  const uint32_t padded_rows = packed ? (rows + 127u) / 128u * 128u : rows;
  const uint32_t row_blocks = (padded_rows + rpc - 1) / rpc;
  // one wave of resident CTAs (80 registers: 768 threads per SM), every one with the same number of row blocks
  const uint32_t resident = 148u * (768u / threads);
  const uint32_t per_cta = (row_blocks + resident - 1) / resident;
  const uint32_t grid = (row_blocks + per_cta - 1) / per_cta;
#define NVFP4_LAUNCH_FUSED(T, P, R)                                                                                   \
  return launch_chained(four_six_rowwise_kernel<T, P, R>, grid, threads, 0, s, static_cast<const T*>(x), out_fp4,      \
                        out_scales, out_gs, out_amax, decoded_amax, rows, padded_rows, gpr, rpc, row_blocks, 0u)
#define NVFP4_LAUNCH_FUSED_R(T, P)       \
  do {                                   \
    if (relu2) NVFP4_LAUNCH_FUSED(T, P, true); \
    else NVFP4_LAUNCH_FUSED(T, P, false);      \
  } while (0)
  if (dtype == NVFP4_DTYPE_F32) {
    if (packed) NVFP4_LAUNCH_FUSED_R(float, true);
    else NVFP4_LAUNCH_FUSED_R(float, false);
  } else {
    if (packed) NVFP4_LAUNCH_FUSED_R(__nv_bfloat16, true);
    else NVFP4_LAUNCH_FUSED_R(__nv_bfloat16, false);
  }
#undef NVFP4_LAUNCH_FUSED_R
#undef NVFP4_LAUNCH_FUSED
}

int launch_schedule_free_materialize(cudaStream_t s, const float* z, const float* x, float beta, float* chunk_amax,
                                     float* amax, uint8_t* out_fp4, uint8_t* out_scales, int packed, float* out_gs,
                                     uint32_t rows, uint32_t cols, float* partials) {
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (!partials || n == 0) {
    const cudaError_t err = cudaMemsetAsync(amax, 0, sizeof(float), s);
    if (err != cudaSuccess) return static_cast<int>(err);
    if (n == 0) return 0;
  }
  const uint32_t grid = partials ? tensor_amax_partials(n) : blocks_for((n + 1023) / 1024, 8, 148 * 8);
  const int rc = launch_chained(schedule_free_amax_kernel, grid, 256, 0, s, z, x, chunk_amax, amax, partials, beta, n);
  if (rc) return rc;
  return launch_four_six_source(s, ScheduleFreeSource{z, x, beta}, partials ? partials : amax, partials ? grid : 1u,
                                partials ? amax : nullptr, 0, rows, cols, out_fp4, out_scales, packed, out_gs, nullptr);
}

int launch_packed_scale_pad(cudaStream_t s, uint8_t* packed, uint32_t rows, uint32_t k_dim) {
  const uint32_t padded = (rows + 127u) / 128u * 128u;
  if (padded == rows) return 0;
  const uint32_t kg = k_dim / 16;
  packed_scale_pad_kernel<<<blocks_for(static_cast<uint64_t>(padded - rows) * kg, 256, 1024), 256, 0, s>>>(packed, rows,
                                                                                                         padded, kg);
  NVFP4_RETURN_LAST();
}

int launch_four_six_padded(cudaStream_t s, const float* x, const float* amax, uint8_t* out_fp4, uint8_t* out_scales,
                           float* out_gs, uint32_t rows, uint32_t cols, uint32_t padded_rows, uint32_t padded_cols,
                           int transposed) {
  const uint64_t groups = static_cast<uint64_t>(padded_rows) * padded_cols / 16;
  if (groups == 0) return 0;
  if (transposed)
    four_six_padded_kernel<true>
        <<<blocks_for(groups, 256), 256, 0, s>>>(x, amax, out_fp4, out_scales, out_gs, rows, cols, padded_cols, groups, 0u);
  else
    four_six_padded_kernel<false>
        <<<blocks_for(groups, 256), 256, 0, s>>>(x, amax, out_fp4, out_scales, out_gs, rows, cols, padded_cols, groups, 0u);
  NVFP4_RETURN_LAST();
}

static MsEdenOut make_out(const nvfp4_ms_eden_args& a, uint32_t out_rows) {
  MsEdenOut o;
  o.fp4 = a.out_fp4;
  o.scales = a.out_scales;
  o.global_scales = a.out_global_scales;
  o.chunk_amax = a.out_chunk_amax;
  o.rows = out_rows;
  o.dst_row_len = a.dst_row_len;
  o.scale_seed = a.scale_seed;
  o.group_offset = a.group_offset;
  o.group_row_stride = a.group_row_stride ? a.group_row_stride : a.dst_row_len / 16u;
  o.sign_offset = a.col_offset;
  o.packed = a.scale_layout == NVFP4_SCALES_PACKED;
  return o;
}

template <int kSrc, typename T, bool kPair>
static void launch_tile(cudaStream_t s, const MsEdenTileParams& p) {
  dim3 grid((p.src_cols + kTileCols - 1) / kTileCols, (p.src_rows + kTileRows - 1) / kTileRows);
  ms_eden_tile_kernel<kSrc, T, kPair><<<grid, 256, 0, s>>>(p);
}

// The tile kernel covers K positions [0, ceil(rows/128)*128) of the transposed operand and
// [0, ceil(cols/64)*64) of the row operand; longer destinations use the generic kernel.
static bool tile_covers(uint32_t src_rows, uint32_t dst_row_len) {
  return dst_row_len <= (src_rows + kTileRows - 1) / kTileRows * kTileRows;
}

bool ms_eden_takes_amax(const nvfp4_ms_eden_args& a) {
  const bool nv_kind = a.src_kind == NVFP4_SRC_NVFP4_TRANSPOSED || a.src_kind == NVFP4_SRC_ROWWISE_NVFP4_TRANSPOSED;
  return nv_kind && a.rows != 0 && a.cols != 0 && a.dst_row_len >= 32 && tile_covers(a.rows, a.dst_row_len) &&
         ms_eden_nvfp4_has_tile_form(a.src_bytes, a.src_scales, a.cols);
}

int launch_ms_eden(cudaStream_t s, const nvfp4_ms_eden_args& a_in, const float* amax_in, float* gs_out, uint32_t amax_count) {
  nvfp4_ms_eden_args a = a_in;
  const bool nv_tiles = ms_eden_takes_amax(a);
  if (amax_count > 0 && !nv_tiles) return static_cast<int>(cudaErrorInvalidValue);
  if (amax_in) {
    // the tiled NVFP4 transposer derives the scale from the amax itself; every other kernel gets it from a
    // one-thread kernel first
    if (!nv_tiles) {
      const int rc = launch_ms_eden_scale_from_amax(s, amax_in, gs_out);
      if (rc) return rc;
      amax_in = nullptr;
    }
    a.global_scale = gs_out;
    a.host_global_scale_valid = 0;
  }
  const bool rows_kind = a.src_kind == NVFP4_SRC_F32_ROWS;
  const uint32_t out_rows = rows_kind ? a.rows : a.cols;
  const uint64_t chunks = static_cast<uint64_t>(out_rows) * (a.dst_row_len / 32);
  if (chunks == 0) return 0;
  const bool bf16 = a.src_dtype == NVFP4_DTYPE_BF16;
  const int packed = a.scale_layout == NVFP4_SCALES_PACKED;
  if (!rows_kind && tile_covers(a.rows, a.dst_row_len)) {
    MsEdenTileParams p;
    p.x = a.x;
    p.src_bytes = a.src_bytes;
    p.src_scales = a.src_scales;
    p.src_global = a.src_global;
    p.src_packed = a.src_scale_layout == NVFP4_SCALES_PACKED;
    p.src_rows = a.rows;
    p.src_cols = a.cols;
    p.global_scale_dev = a.global_scale;
    p.global_scale_host = a.host_global_scale;
    p.use_host_scale = a.host_global_scale_valid;
    p.scale_override = a.scale_override;
    p.sign_seed = a.sign_seed;
    p.t = make_out(a, out_rows);
    p.r = p.t;
    p.col_sum_partials = nullptr;
    p.amax_in = amax_in;
    p.gs_out = gs_out;
    p.amax_count = amax_count;
    if (nv_tiles) return launch_ms_eden_nvfp4_tiles(s, p, a.src_kind == NVFP4_SRC_ROWWISE_NVFP4_TRANSPOSED);
    switch (a.src_kind) {
      case NVFP4_SRC_F32_TRANSPOSED:
        if (bf16) launch_tile<0, __nv_bfloat16, false>(s, p);
        else launch_tile<0, float, false>(s, p);
        break;
      case NVFP4_SRC_NVFP4_TRANSPOSED:
        launch_tile<2, float, false>(s, p);
        break;
      case NVFP4_SRC_ROWWISE_NVFP4_TRANSPOSED:
        launch_tile<3, float, false>(s, p);
        break;
      default:
        return 1;
    }
  } else {
    MsEdenParams p;
    p.x = a.x;
    p.src_bytes = a.src_bytes;
    p.src_scales = a.src_scales;
    p.src_global = a.src_global;
    p.src_packed = a.src_scale_layout == NVFP4_SCALES_PACKED;
    p.a = rows_kind ? a.cols : a.rows;
    p.b = a.cols;
    p.global_scale_dev = a.global_scale;
    p.global_scale_host = a.host_global_scale;
    p.use_host_scale = a.host_global_scale_valid;
    p.scale_override = a.scale_override;
    p.sign_seed = a.sign_seed;
    p.out = make_out(a, out_rows);
    const uint32_t grid = blocks_for(chunks, 128);
    switch (a.src_kind) {
      case NVFP4_SRC_F32_ROWS:
        if (bf16) ms_eden_kernel<0, __nv_bfloat16><<<grid, 128, 0, s>>>(p);
        else ms_eden_kernel<0, float><<<grid, 128, 0, s>>>(p);
        break;
      case NVFP4_SRC_F32_TRANSPOSED:
        if (bf16) ms_eden_kernel<1, __nv_bfloat16><<<grid, 128, 0, s>>>(p);
        else ms_eden_kernel<1, float><<<grid, 128, 0, s>>>(p);
        break;
      case NVFP4_SRC_NVFP4_TRANSPOSED:
        ms_eden_kernel<2, float><<<grid, 128, 0, s>>>(p);
        break;
      case NVFP4_SRC_ROWWISE_NVFP4_TRANSPOSED:
        ms_eden_kernel<3, float><<<grid, 128, 0, s>>>(p);
        break;
      default:
        return 1;
    }
  }
  count_launch();
  int rc = static_cast<int>(cudaGetLastError());
  if (rc) return rc;
  if (packed) return launch_packed_scale_pad(s, a.out_scales, out_rows, a.dst_row_len);
  return 0;
}

// Row operand and transposed operand of one f32 / bf16 matrix in a single pass over it.
// `rows_args` describes the row operand (src_kind F32_ROWS), `t_args` the transposed one
// (src_kind F32_TRANSPOSED) of the same matrix; both use the same global scale and sign seed.
uint32_t ms_eden_pair_row_tiles(uint32_t rows) { return (rows + kTileRows - 1) / kTileRows; }

bool ms_eden_pair_is_tiled(const nvfp4_ms_eden_args& r, const nvfp4_ms_eden_args& t) {
  return r.rows != 0 && r.cols != 0 && tile_covers(r.rows, t.dst_row_len) &&
         r.dst_row_len <= (r.cols + kTileCols - 1) / kTileCols * kTileCols;
}

int launch_col_sum_reduce(cudaStream_t s, const float* partials, float* dbias, uint32_t tiles, uint32_t n) {
  if (n == 0) return 0;
  return launch_chained(col_sum_reduce_kernel, blocks_for(n, 32), 256, 0, s, partials, dbias, tiles, n);
}

bool ms_eden_pair_takes_amax(const nvfp4_ms_eden_args& r, const nvfp4_ms_eden_args& t) {
  return ms_eden_pair_is_tiled(r, t) && ms_eden_pair_has_tile_form(r.x, r.src_dtype, r.cols);
}

int launch_ms_eden_pair(cudaStream_t s, const nvfp4_ms_eden_args& r, const nvfp4_ms_eden_args& t,
                        float* col_sum_partials, const float* amax_in, float* gs_out, uint32_t amax_count, void* zero,
                        uint64_t zero_words, bool beside_others) {
  const uint32_t rows = r.rows, cols = r.cols;
  if ((amax_in || zero_words) && !ms_eden_pair_takes_amax(r, t)) return static_cast<int>(cudaErrorInvalidValue);
  if (!ms_eden_pair_is_tiled(r, t)) {
    int rc = launch_ms_eden(s, r);
    return rc ? rc : launch_ms_eden(s, t);
  }
  MsEdenTileParams p;
  p.x = r.x;
  p.src_bytes = nullptr;
  p.src_scales = nullptr;
  p.src_global = nullptr;
  p.src_packed = 0;
  p.src_rows = rows;
  p.src_cols = cols;
  p.global_scale_dev = r.global_scale;
  p.global_scale_host = r.host_global_scale;
  p.use_host_scale = r.host_global_scale_valid;
  p.scale_override = r.scale_override;
  p.sign_seed = r.sign_seed;
  p.t = make_out(t, cols);
  p.r = make_out(r, rows);
  p.col_sum_partials = col_sum_partials;
  p.amax_in = amax_in;
  p.gs_out = gs_out;
  p.amax_count = amax_count;
  p.zero = static_cast<uint4*>(zero);
  p.zero_words = zero_words;
  if (ms_eden_pair_has_tile_form(r.x, r.src_dtype, cols)) return launch_ms_eden_pair_tiles(s, p, r.src_dtype, beside_others);
  if (r.src_dtype == NVFP4_DTYPE_BF16) {
    launch_tile<0, __nv_bfloat16, true>(s, p);
  } else {
    launch_tile<0, float, true>(s, p);
  }
  count_launch();
  int rc = static_cast<int>(cudaGetLastError());
  if (rc) return rc;
  if (p.r.packed) rc = launch_packed_scale_pad(s, r.out_scales, rows, r.dst_row_len);
  if (rc) return rc;
  if (p.t.packed) rc = launch_packed_scale_pad(s, t.out_scales, cols, t.dst_row_len);
  return rc;
}

uint32_t relu2_backward_grid(uint64_t n) { return blocks_for((n + 7) / 8, 256, 148 * 8); }

int launch_relu2_backward(cudaStream_t s, const void* pre, int pre_kind, const void* d_out, void* d_pre, int grad_bf16,
                          uint64_t n, float* chunk_amax) {
  if (n == 0) return 0;
  const int vectorized = ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(d_out) |
                           reinterpret_cast<uintptr_t>(d_pre)) & 15u) == 0;
  const uint32_t grid = relu2_backward_grid(n);
#define NVFP4_RELU2_BWD_A(K, G, A) \
  relu2_backward_kernel<K, G, A><<<grid, 256, 0, s>>>(pre, d_out, d_pre, n, vectorized, chunk_amax)
#define NVFP4_RELU2_BWD(K, G)                     \
  do {                                            \
    if (chunk_amax) NVFP4_RELU2_BWD_A(K, G, true); \
    else NVFP4_RELU2_BWD_A(K, G, false);          \
  } while (0)
  if (grad_bf16) {
    if (pre_kind == kPreF32) NVFP4_RELU2_BWD(kPreF32, true);
    else if (pre_kind == kPreBf16) NVFP4_RELU2_BWD(kPreBf16, true);
    else NVFP4_RELU2_BWD(kPreF16, true);
  } else {
    if (pre_kind == kPreF32) NVFP4_RELU2_BWD(kPreF32, false);
    else if (pre_kind == kPreBf16) NVFP4_RELU2_BWD(kPreBf16, false);
    else NVFP4_RELU2_BWD(kPreF16, false);
  }
#undef NVFP4_RELU2_BWD
#undef NVFP4_RELU2_BWD_A
  NVFP4_RETURN_LAST();
}

int launch_decode(cudaStream_t s, const uint8_t* bytes, const uint8_t* scales, const float* gscales, int rowwise,
                  int transpose, float* out, uint32_t rows, uint32_t cols) {
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (n == 0) return 0;
  // the wide form needs whole 16-groups per row, aligned words and a 32-bit index space
  if (!transpose && cols % 16 == 0 && n / 8 < 0xff000000ull && (reinterpret_cast<uintptr_t>(bytes) & 3u) == 0 &&
      (reinterpret_cast<uintptr_t>(out) & 31u) == 0) {
    const uint32_t octets = static_cast<uint32_t>(n / 8);
    return launch_chained(decode_rows_kernel, blocks_for(octets, 1024, 148u * 8u), 256, 0, s, bytes, scales, gscales, out, octets,
                          FastDiv(cols / 8), rowwise);
  }
  decode_kernel<<<blocks_for(n, 256), 256, 0, s>>>(bytes, scales, gscales, out, rows, cols, rowwise, transpose);
  NVFP4_RETURN_LAST();
}

static ScalePlane scale_plane(const uint8_t* logical, uint8_t* packed, uint32_t mn) {
  return ScalePlane{logical, packed, mn, (mn + 127u) / 128u};
}
// the tiled kernel reads 32-bit words and writes 16 bytes at a time
static bool scale_pack_tiled(const ScalePlane& p) {
  return (reinterpret_cast<uintptr_t>(p.logical) & 3u) == 0 && (reinterpret_cast<uintptr_t>(p.packed) & 15u) == 0 &&
         p.row_blocks <= 65535u;
}

int launch_scale_pack(cudaStream_t s, const uint8_t* logical, uint8_t* packed, uint32_t mn, uint32_t k_dim) {
  const uint32_t padded = (mn + 127u) / 128u * 128u, kg = k_dim / 16;
  const uint64_t total = static_cast<uint64_t>(padded) * kg;
  if (total == 0) return 0;
  const uint32_t k_atoms = kg / 4u;
  const ScalePlane plane = scale_plane(logical, packed, mn);
  if (scale_pack_tiled(plane))
    return launch_chained(scale_pack_tiles_kernel, dim3((k_atoms + 15u) / 16u, plane.row_blocks), 256, 0, s, plane, ScalePlane{},
                          k_atoms);
  scale_pack_kernel<<<blocks_for(total, 256, 148 * 16), 256, 0, s>>>(logical, packed, mn, padded, kg);
  NVFP4_RETURN_LAST();
}

int launch_scale_pack_pair(cudaStream_t s, const uint8_t* const (&logical)[2], uint8_t* const (&packed)[2],
                           const uint32_t (&mn)[2], uint32_t k_dim) {
  const ScalePlane a = scale_plane(logical[0], packed[0], mn[0]), b = scale_plane(logical[1], packed[1], mn[1]);
  const uint32_t k_atoms = k_dim / 64u;
  if (!scale_pack_tiled(a) || !scale_pack_tiled(b) || a.row_blocks + b.row_blocks > 65535u || k_dim % 64u != 0 || k_atoms == 0 ||
      a.row_blocks == 0 || b.row_blocks == 0) {
    const int rc = launch_scale_pack(s, logical[0], packed[0], mn[0], k_dim);
    return rc ? rc : launch_scale_pack(s, logical[1], packed[1], mn[1], k_dim);
  }
  return launch_chained(scale_pack_tiles_kernel, dim3((k_atoms + 15u) / 16u, a.row_blocks + b.row_blocks), 256, 0, s, a, b,
                        k_atoms);
}

int launch_pad_u4_rows(cudaStream_t s, const uint8_t* src, uint8_t* dst, uint32_t rows, uint32_t padded_rows,
                       uint32_t cols) {
  const uint64_t sb = static_cast<uint64_t>(rows) * cols / 2, db = static_cast<uint64_t>(padded_rows) * cols / 2;
  if (db == 0) return 0;
  pad_u4_rows_kernel<<<blocks_for(db, 256, 148 * 16), 256, 0, s>>>(src, dst, sb, db);
  NVFP4_RETURN_LAST();
}

int launch_pad_f32(cudaStream_t s, const float* src, float* dst, uint32_t rows, uint32_t cols, uint32_t padded_rows,
                   uint32_t padded_cols, int transpose) {
  const uint64_t total = static_cast<uint64_t>(padded_rows) * padded_cols;
  if (total == 0) return 0;
  if (transpose)
    pad_f32_kernel<true><<<blocks_for(total, 256, 148 * 16), 256, 0, s>>>(src, dst, rows, cols, padded_rows, padded_cols);
  else
    pad_f32_kernel<false><<<blocks_for(total, 256, 148 * 16), 256, 0, s>>>(src, dst, rows, cols, padded_rows, padded_cols);
  NVFP4_RETURN_LAST();
}

int launch_crop_f32(cudaStream_t s, const float* src, float* dst, uint32_t rows, uint32_t src_cols, uint32_t dst_cols) {
  const uint64_t total = static_cast<uint64_t>(rows) * dst_cols;
  if (total == 0) return 0;
  crop_f32_kernel<<<blocks_for(total, 256, 148 * 16), 256, 0, s>>>(src, dst, rows, src_cols, dst_cols);
  NVFP4_RETURN_LAST();
}

int launch_postop(cudaStream_t s, float* raw, float* other, const uint8_t* bias_bytes, const uint8_t* bias_scales,
                  const float* bias_gs, uint32_t rows, uint32_t cols, int mode) {
  const uint64_t n = static_cast<uint64_t>(rows) * cols;
  if (n == 0) return 0;
  postop_kernel<<<blocks_for(n, 256, 148 * 16), 256, 0, s>>>(raw, other, bias_bytes, bias_scales, bias_gs, n, cols, mode);
  NVFP4_RETURN_LAST();
}

int launch_bias_grad(cudaStream_t s, const void* e, int dtype, float* dbias, uint32_t tokens, uint32_t n) {
  if (n == 0) return 0;
  if (dtype == NVFP4_DTYPE_F32)
    bias_grad_kernel<float><<<blocks_for(n, 32), 256, 0, s>>>(static_cast<const float*>(e), dbias, tokens, n);
  else
    bias_grad_kernel<__nv_bfloat16>
        <<<blocks_for(n, 32), 256, 0, s>>>(static_cast<const __nv_bfloat16*>(e), dbias, tokens, n);
  NVFP4_RETURN_LAST();
}

}  // namespace nvfp4
