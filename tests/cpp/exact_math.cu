// The quantizers' divisions against the division operators: rcp_in_range, div_by_rcp, their packed forms and FastDiv of
// csrc/common.cuh over the operands their callers give them.  Prints one "<what> <operands> <mismatches>" line each;
// exits with 1 if there is a mismatch, with 2 on a CUDA error.
#include <cstdio>
#include <cstdlib>

#include "common.cuh"

using namespace nvfp4;

namespace {

using Count = unsigned long long;

__device__ void report(Count bad, Count* total) {
  if (bad) atomicAdd(total, bad);
}
__device__ uint32_t mix(uint64_t v) {  // splitmix64's finaliser
  v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ull;
  v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
  return static_cast<uint32_t>((v ^ (v >> 31)) >> 16);
}
__device__ float power_of_two(int e) { return __uint_as_float(static_cast<uint32_t>(e + 127) << 23); }

// 1 / b for every float in [2^first, 2^last)
__global__ void reciprocals(int first, int last, Count* mismatches) {
  const uint32_t lo = static_cast<uint32_t>(first + 127) << 23, hi = static_cast<uint32_t>(last + 127) << 23;
  Count bad = 0;
  for (uint32_t bits = lo + blockIdx.x * blockDim.x + threadIdx.x; bits < hi; bits += gridDim.x * blockDim.x) {
    const float b = __uint_as_float(bits);
    bad += __float_as_uint(rcp_in_range(b)) != __float_as_uint(__frcp_rn(b));
  }
  report(bad, mismatches);
}

// the same two at a time, each lane over every float, one of them backwards
__global__ void packed_reciprocals(int first, int last, Count* mismatches) {
  const uint32_t lo = static_cast<uint32_t>(first + 127) << 23, hi = static_cast<uint32_t>(last + 127) << 23;
  Count bad = 0;
  for (uint32_t bits = lo + blockIdx.x * blockDim.x + threadIdx.x; bits < hi; bits += gridDim.x * blockDim.x) {
    const float b0 = __uint_as_float(bits), b1 = __uint_as_float(hi - 1u - (bits - lo));
    float y0, y1;
    unpack2(rcp_in_range2(pack2(b0, b1)), y0, y1);
    bad += __float_as_uint(y0) != __float_as_uint(__frcp_rn(b0)) || __float_as_uint(y1) != __float_as_uint(__frcp_rn(b1));
  }
  report(bad, mismatches);
}

// a / b, mantissas at random, b in [2^first, 2^last), the quotient between 2^-21 and 2^21
__device__ void operands(Count i, int first, int last, float& a, float& b) {
  const uint32_t r = mix(3 * i + 1), eb = r % static_cast<uint32_t>(last - first), eq = (r >> 16) % 41u;
  b = __uint_as_float(0x3f800000u | (mix(3 * i + 2) & 0x7fffffu)) * power_of_two(first + static_cast<int>(eb));
  a = __uint_as_float(0x3f800000u | (mix(3 * i + 3) & 0x7fffffu)) * power_of_two(first + static_cast<int>(eb) + static_cast<int>(eq) - 20);
}
__global__ void quotients(int first, int last, Count pairs, Count* mismatches) {
  Count bad = 0;
  for (Count i = static_cast<Count>(blockIdx.x) * blockDim.x + threadIdx.x; i < pairs; i += static_cast<Count>(gridDim.x) * blockDim.x) {
    float a, b;
    operands(i, first, last, a, b);
    bad += __float_as_uint(div_by_rcp(a, b, __frcp_rn(b))) != __float_as_uint(__fdiv_rn(a, b));
  }
  report(bad, mismatches);
}
// other operands in either lane
__global__ void packed_quotients(int first, int last, Count pairs, Count* mismatches) {
  Count bad = 0;
  for (Count i = static_cast<Count>(blockIdx.x) * blockDim.x + threadIdx.x; i < pairs / 2; i += static_cast<Count>(gridDim.x) * blockDim.x) {
    float a0, b0, a1, b1, q0, q1;
    operands(pairs + 2 * i, first, last, a0, b0);
    operands(pairs + 2 * i + 1, first, last, a1, b1);
    unpack2(div_by_rcp2(pack2(a0, a1), pack2(b0, b1), pack2(__frcp_rn(b0), __frcp_rn(b1))), q0, q1);
    bad += __float_as_uint(q0) != __float_as_uint(__fdiv_rn(a0, b0));
    bad += __float_as_uint(q1) != __float_as_uint(__fdiv_rn(a1, b1));
  }
  report(bad, mismatches);
}

// a / 1536 for every a whose quotient lies in [2^-80, 2^80]
__global__ void amax_quotients(Count* operands, Count* mismatches) {
  const uint32_t lo = __float_as_uint(1536.0f * 0x1p-80f), hi = __float_as_uint(1536.0f * 0x1p80f);
  Count bad = 0;
  for (uint32_t bits = lo + blockIdx.x * blockDim.x + threadIdx.x; bits <= hi; bits += gridDim.x * blockDim.x) {
    const float a = __uint_as_float(bits);
    bad += __float_as_uint(div_by_rcp(a, 1536.0f, 1.0f / 1536.0f)) != __float_as_uint(__fdiv_rn(a, 1536.0f));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *operands = hi - lo + 1;
  report(bad, mismatches);
}

// n / d around multiples of d, at the ends of the index space and at random
__global__ void index_quotients(const FastDiv div, Count* mismatches) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, r = mix((static_cast<uint64_t>(div.d) << 32) + i);
  const uint32_t multiple = r / div.d * div.d;
  const uint32_t n[6] = {r, multiple, multiple - 1u, multiple + div.d - 1u, i, 0xffffffffu - i};
  Count bad = 0;
#pragma unroll
  for (int k = 0; k < 6; ++k) bad += div.div(n[k]) != n[k] / div.d;
  report(bad, mismatches);
}

void check(cudaError_t e) {
  if (e == cudaSuccess) return;
  std::fprintf(stderr, "%s\n", cudaGetErrorString(e));
  std::exit(2);
}

}  // namespace

int main() {
  Count* counts;
  check(cudaMallocManaged(&counts, 7 * sizeof(Count)));
  for (int i = 0; i < 7; ++i) counts[i] = 0;
  // divisors of the four-six scales: 4 gs + eps and above, with gs from 2^-80 (eps is 1e-20) to 2^80 and a block scale of up
  // to 448; sums of the MS-EDEN correction: 2^-3 to 2^71
  const int first = -67, last = 90;
  const Count pairs = 1ull << 35;
  reciprocals<<<148 * 8, 256>>>(first, last, counts);
  check(cudaGetLastError());
  quotients<<<148 * 8, 256>>>(first, last, pairs, counts + 1);
  check(cudaGetLastError());
  packed_reciprocals<<<148 * 8, 256>>>(first, last, counts + 5);
  check(cudaGetLastError());
  packed_quotients<<<148 * 8, 256>>>(first, last, pairs, counts + 6);
  check(cudaGetLastError());
  amax_quotients<<<148 * 8, 256>>>(counts + 2, counts + 3);
  check(cudaGetLastError());
  Count divisors = 0;
  auto divide_by = [&](uint32_t d) {
    index_quotients<<<64, 256>>>(FastDiv(d), counts + 4);
    check(cudaGetLastError());
    ++divisors;
  };
  for (uint32_t d = 1; d <= 2048; ++d) divide_by(d);
  for (uint32_t e = 11; e < 32; ++e)
    for (uint32_t d : {(1u << e) - 1u, 1u << e, (1u << e) + 1u, 3u << (e - 2)}) divide_by(d);
  divide_by(0xffffffffu);
  check(cudaDeviceSynchronize());
  std::printf("reciprocals %llu %llu\n", static_cast<Count>(last - first) << 23, counts[0]);
  std::printf("quotients %llu %llu\n", pairs, counts[1]);
  std::printf("packed_reciprocals %llu %llu\n", static_cast<Count>(last - first) << 23, counts[5]);
  std::printf("packed_quotients %llu %llu\n", pairs, counts[6]);
  std::printf("amax_quotients %llu %llu\n", counts[2], counts[3]);
  std::printf("index_quotients %llu %llu\n", divisors * 64 * 256 * 6, counts[4]);
  return counts[0] || counts[1] || counts[3] || counts[4] || counts[5] || counts[6] ? 1 : 0;
}
