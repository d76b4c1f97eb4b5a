// NVFP4 block-scaled projection GEMM for sm_100a.
//
//   out[m][n] = epilogue( (sum_k A[m][k]*sa[m][k/16] * B[n][k]*sb[n][k/16]) * weight * ga * gb )
//
// Semantics follow the reference's TMA GEMM and its post-op kernels
// (crates/cuda-kernels/src/utils/nvfp4_tma_matmul/kernels.rs:310-351,538-568 and
// gpt/projection_postop.rs:97-162); the engine is new: a persistent, warp-specialised
// kernel in which
//   warp 0      streams A / B nibble tiles with TMA (128-byte swizzle) and the packed
//               scale-factor tiles with bulk copies into a shared-memory ring,
//   warp 1      issues tcgen05.mma.kind::mxf4nvf4.block_scale (128 x BLOCK_N x 64 per
//               instruction), FP32 accumulators in tensor memory,
//   warps 2, 3  issue the TMA stores of the two epilogue groups; warp 2 owns the tensor-memory allocation,
//   warps 4..7 and 12..15  two epilogue groups: drain accumulators (tcgen05.ld), apply global
//               scales / bias / ReLU^2 / residual, cast and store; the groups take alternate
//               128-byte column sub-tiles of a tile (a warp reaches the tensor-memory lanes of
//               its index modulo four, so warps w and w + 8 share a lane quadrant),
//   warps 8..11 move the scale factors shared -> tensor memory (tcgen05.st).
// Three tile widths.  BLOCK_N = 128 and 192 double buffer the accumulator (2 x 192 accumulator
// columns + 3 x 40 scale-factor columns fill the 512 columns of tensor memory), so the epilogue of
// one tile overlaps the main loop of the next; the 256-column accumulators of consecutive tiles share
// 128 columns, which the epilogue takes first, so that half of it overlaps as well.  Every mbarrier
// wait is bounded: on expiry the kernel records a status word, drains, frees its tensor memory and returns.
//
// Clusters only as CTA pairs for long main loops (cta_group::2), no multicast loads: every load reads this GPU's own memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "kernels.h"

namespace nvfp4 {

__device__ uint32_t g_device_status = 0;

namespace {

constexpr int kRowBlock = 128;                    // rows of one MMA, one scale-factor block, one epilogue sub-tile
constexpr int kBlockKBytes = 128;                 // 256 nibbles = one 128-byte swizzle row
constexpr int kKAtomsPerStage = 4;                // 64-element k-atoms (one MMA each per row block) per stage
constexpr int kAHalfBytes = kRowBlock * kBlockKBytes;  // A rows of one MMA in a stage
constexpr int kSfTileBytes = 512;                 // 128 rows x 4 scale bytes
constexpr int kSfBlockStageBytes = kKAtomsPerStage * kSfTileBytes;  // one 128-row scale block of a stage
constexpr int kStoreStageBytes = kRowBlock * 128;  // one epilogue sub-tile: 128 rows x 128 bytes
constexpr int kTmemCols = 512;
constexpr int kMaxStages = 8;
constexpr int kSmemBudget = 227 * 1024;
constexpr int kThreads = 512;
constexpr uint32_t kMaxFinal = 10;  // staging buffers of a CTA's last tile beside the ring's
constexpr uint64_t kDefaultWaitTimeoutNs = 2000000000ull;  // 2 s

constexpr uint32_t kStatusProducerTimeout = 1u, kStatusMmaTimeout = 2u, kStatusEpilogueTimeout = 4u;
constexpr uint32_t kDebugSkipFirstLoad = 1u, kDebugRefuseOutputMaps = 2u;

// Tile shapes: 128 x {128, 192, 256} and the tall 256 x 192.  The tall tile issues two MMAs per k-atom (rows
// 0..127 and 128..255 of the A stage against the same B stage), so a stage's B bytes feed twice the flops:
// streaming GEMMs are bound by the operand bytes an SM can pull from L2, and the tall tile moves 21 % fewer of
// them per flop than 128 x 256.  Its two 192-column accumulators and two scale-factor column sets fill tensor
// memory (2 x 192 + 2 x 56 = 496 of 512 columns), so the accumulator is single buffered.
// kPanel: 0 streaming, else resident with a B panel of up to so many k-tiles.  kPair: two CTAs of a cluster on neighbouring SMs
// (cta_group::2) work on 256 x 256; each loads its 128 rows of A and half of B, a third fewer operand bytes per flop.
template <int kBlockM, int kBlockN, int kPanel, bool kPair>
struct Cfg {
  static constexpr bool kResident = kPanel != 0;
  static_assert(!kPair || (kPanel == 0 && kBlockM == 128 && kBlockN == 256), "a pair streams 128 x 256 tiles");
  static constexpr int kMHalves = kBlockM / kRowBlock;
  static_assert(kBlockM == 128 || (kBlockM == 256 && kBlockN == 192 && !kResident), "unsupported tile shape");
  static constexpr int kAStageBytes = kMHalves * kAHalfBytes;
  static constexpr int kSfaStageBytes = kMHalves * kSfBlockStageBytes;
  // 128-row scale-factor blocks of B a tile can touch: a 192-column tile starts either on a block
  // boundary or in the middle of a block, and spans two blocks either way
  static constexpr int kSfBlocks = (kBlockN + 127) / 128;
  static constexpr int kBRows = kPair ? kBlockN / 2 : kBlockN;  // rows of B a CTA loads
  static constexpr int kBStageBytes = kBRows * kBlockKBytes;
  static constexpr int kSfbStageBytes = kSfBlocks * kSfBlockStageBytes;
  static constexpr int kAccStages = (kBlockN == 256 || kMHalves == 2) ? 1 : 2;
  static constexpr int kAccCols = kMHalves * kBlockN;  // columns of one accumulator buffer (row halves side by side)
  // The 256-column accumulator lies at columns 0 and 128 in turn: a tile's MMAs wait for the half of the tile before it that
  // they overwrite, which the epilogue takes first, and run beside its other half.  With one fixed accumulator they waited
  // 1900 cycles of a tile's 4700.  Together with the panel's scale factors kept in tensor memory, two staging buffers a group
  // and A prefetched: 65536 x 2304 x K 768 bf16 76 -> 65 us, x 3072 99 -> 86, 8192 x 3072 17.5 -> 15.3; streaming, where only
  // the accumulator changed: 4096 x 1024 x K 8192 f32 19.5 -> 18.2.
  static constexpr bool kRotate = kBlockN == 256;
  static constexpr int kAccRegion = kRotate ? 384 : kAccStages * kAccCols;
  // Scale factors behind the accumulators.  Streaming: a ring of column sets (one per k-tile, A and B), so the copies for
  // the next k-tile never overwrite columns an MMA in flight reads.  Resident: those of the whole B panel, and a ring for A.
  static constexpr int kSfaSetCols = kMHalves * 4 * kKAtomsPerStage;
  static constexpr int kSfbColsPerAtom = kBlockN / 32;
  static constexpr int kSfbTileCols = kSfbColsPerAtom * kKAtomsPerStage;
  static constexpr int kTmemPanel = kAccRegion;           // resident: B scale factors of the panel
  static constexpr int kTmemSfa = kAccRegion + kPanel * kSfbTileCols;  // set 0: A, streaming B behind it
  static constexpr int kSfSetCols = kSfaSetCols + (kResident ? 0 : kSfbTileCols);
  static constexpr int kSfSets = (kTmemCols - kTmemSfa) / kSfSetCols < 4 ? (kTmemCols - kTmemSfa) / kSfSetCols : 4;
  static constexpr int kStageBytes = kAStageBytes + kSfaStageBytes;                    // of the ring, A side
  static constexpr int kSlotBytes = kBStageBytes + (kResident ? 0 : kSfbStageBytes);  // of the panel or the ring, B side
  // epilogue staging ring: deep for the narrow tile and for short K, which are epilogue bound, shallow where the shared memory
  // goes to pipeline stages (streaming wide tiles) or the panel (four k-tiles of 192 columns: with two more buffers three A
  // stages are left instead of five, 8192 x 32000 x K 1024 193 us against 154)
  static constexpr int kStoreBufs = kBlockN == 128 || kPanel == 3 ? 4 : 2;
  static constexpr int kBiasSlots = (kBlockN + 127) / 128;  // bias values a thread of an epilogue group fetches
  static constexpr int kFixedBytes =
      1024 /*alignment slack*/ + kStoreBufs * kStoreStageBytes + 512 /*barriers*/ +
      2 * kBlockN * 4 /*bias of the tile, one copy per epilogue group*/;
  static_assert(kSfSets >= 2, "tensor memory overflow");
};

// How a sub-tile leaves: registers to memory (outputs a tensor map cannot describe, a bf16 residual), staging buffer and
// TMA store, or the same added to the f32 residual stream.
enum class StorePath { kDirect, kTma, kTmaResidual };

struct GemmParams {
  const uint8_t* sfa;
  const uint8_t* sfb;
  const float* a_global;
  const float* b_global;
  const float* bias;
  // NVFP4-encoded bias [n] (bytes, logical scale bytes, f32[1] global scale): used when bias == nullptr
  const uint8_t* bias_bytes;
  const uint8_t* bias_scales;
  const float* bias_global;
  float* row_amax;  // optional f32[m]: max over the row of relu(stored value)^2 (red.max, zeroed by the launcher)
  void* out;
  void* aux;
  uint32_t m, n, k, ldo;
  uint32_t num_m_blocks, num_n_blocks, k_atoms, sfa_blocks128, sfb_blocks128;
  uint32_t k_splits, k_tiles_per_split, num_k_tiles;
  uint32_t stages;  // depth of the A (and, when streaming, B) ring
  uint32_t resident_cpn;  // resident mode: CTAs per column block (0 = contiguous tile ranges instead)
  int mode, epilogue, vec_store, tma_store, stream_out;
  float weight;
  uint64_t wait_timeout_ns;  // limit of every mbarrier wait
  uint32_t debug_flags;      // bit 0: CTA 0 never loads its first k-tile (exercises the bounded waits)
  uint32_t lets_next_beside;  // GemmNeighbour::kLetsNextBeside
#ifdef NVFP4_GEMM_TRACE
  unsigned long long* trace;  // measurement builds only: [5 roles][1024] (clock << 8 | tag) records of CTA 0
#endif
};

// Measurement builds (-DNVFP4_GEMM_TRACE) record a time line of CTA 0: one (SM clock, tag) word per event and
// role (0 producer, 1 MMA issuer, 2 first scale-factor warp, 3 / 4 epilogue groups).  Product builds compile
// the macro away.
#ifdef NVFP4_GEMM_TRACE
#define GEMM_TRACE(role, tag, leader)                                                                      \
  do {                                                                                                     \
    if (p.trace && blockIdx.x == 0 && (leader)) {                                                          \
      const uint32_t trace_i = trace_n++;                                                                  \
      if (trace_i < 1024u) p.trace[(role) * 1024u + trace_i] = (static_cast<unsigned long long>(clock64()) << 8) | (tag); \
    }                                                                                                      \
  } while (0)
#else
#define GEMM_TRACE(role, tag, leader) do { } while (0)
#endif

// ---- PTX wrappers ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t clock32() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%clock;" : "=r"(t));
  return t;
}

// Bounded wait.  Returns false when the CTA is aborting (this waiter timed out, or another
// role already did); the caller then leaves its loop and goes to the common teardown.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag,
                                          uint32_t status_bit, uint64_t timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  uint32_t polls = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++polls & 255u) == 0) {
      if (*abort_flag) return false;
      if (global_timer_ns() - t0 > timeout_ns) {
        *abort_flag = 1;
        atomicOr(&g_device_status, status_bit);
        return false;
      }
    }
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_prefetch(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<uint64_t>(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int32_t x, int32_t y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_2d_streaming(const CUtensorMap* map, uint32_t src, int32_t x, int32_t y) {
  uint64_t policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group.L2::cache_hint [%0, {%2, %3}], [%1], %4;" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y), "l"(policy)
               : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, uint32_t src, int32_t x, int32_t y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kPending) : "memory");
}
__device__ __forceinline__ void bulk_wait_group0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// one named barrier per epilogue warp group (ids 1 and 2), 128 threads each
__device__ __forceinline__ void epilogue_barrier(uint32_t group) {
  asm volatile("bar.sync %0, 128;" ::"r"(group + 1u) : "memory");
}

__device__ __forceinline__ void wait_for_prior_kernels() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next_kernel() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A GEMM beside its predecessor does not wait for it: that one let it start only behind its own wait, so that everything before
// it is complete.
template <bool kBeside>
__device__ __forceinline__ void wait_for_inputs() {
  if (!kBeside) wait_for_prior_kernels();
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcgen05_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// The forms of a CTA pair (two CTAs of a cluster on neighbouring SMs, cta_group::2).  `kBothCtas`: the signal goes to the
// barrier at this offset in both.
constexpr uint16_t kBothCtas = 3;
template <bool kPair>
__device__ __forceinline__ void commit(uint32_t bar) {
  if constexpr (kPair)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(kBothCtas)
                 : "memory");
  else
    tcgen05_commit(bar);
}
__device__ __forceinline__ uint32_t leader_address(uint32_t addr) {  // of the same variable in the pair's first CTA
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
// At CTA scope: what the other CTA's MMAs read has been ordered by the tcgen05 fences, and a release at cluster scope in this
// place waited 1200 cycles for the thread's other memory operations.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// An operand load of either CTA of a pair, counted by the barrier `bar` of one of them.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tcgen05_mma_nvf4_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                      uint32_t accumulate, uint32_t tmem_sfa, uint32_t tmem_sfb) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}
__device__ __forceinline__ void tcgen05_mma_nvf4(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t tmem_sfa, uint32_t tmem_sfb) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}
__device__ __forceinline__ void tcgen05_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// Packed FP32 pairs for the epilogue arithmetic: one instruction per two accumulator columns, each lane
// rounded exactly like the scalar operation.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void fma_f32x2(float& lo, float& hi, uint32_t a_lo, uint32_t a_hi, uint64_t b, uint64_t c) {
  asm("{\n\t.reg .b64 a, d;\n\tmov.b64 a, {%2, %3};\n\tfma.rn.f32x2 d, a, %4, %5;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "r"(a_lo), "r"(a_hi), "l"(b), "l"(c));
}
__device__ __forceinline__ void mul_f32x2(float& lo, float& hi, float a_lo, float a_hi, uint64_t b) {
  asm("{\n\t.reg .b64 a, d;\n\tmov.b64 a, {%2, %3};\n\tmul.rn.f32x2 d, a, %4;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "f"(a_lo), "f"(a_hi), "l"(b));
}
__device__ __forceinline__ void square_f32x2(float& lo, float& hi) {
  asm("{\n\t.reg .b64 a;\n\tmov.b64 a, {%0, %1};\n\tmul.rn.f32x2 a, a, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(lo), "+f"(hi));
}
__device__ __forceinline__ void tcgen05_st_x4(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tcgen05_st_x2(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(r[0]), "r"(r[1]) : "memory");
}
__device__ __forceinline__ void tcgen05_st_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tcgen05_st_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tcgen05_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptors (sm_100 format: version 1 in bits 46..47).
// A / B tiles: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart; the K offset of a
// 64-element MMA inside the swizzle row (32 bytes) is added to the start address.
__device__ __forceinline__ uint64_t make_ab_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1024u >> 4) << 32;  // stride byte offset
  d |= 1ull << 46;                               // descriptor version
  d |= 2ull << 61;                               // SWIZZLE_128B
  return d;
}
// Instruction descriptor of kind::mxf4nvf4: E2M1 x E2M1, UE4M3 scales, K-major A and B,
// M = 128 (256 of a pair), N = kBlockN, K = 64.
template <int kBlockN, bool kPair>
__device__ __forceinline__ constexpr uint32_t make_idesc() {
  return (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kBlockN >> 3) << 17) | (0u << 23) |
         (static_cast<uint32_t>(((kPair ? 2 : 1) * kRowBlock) >> 4) << 24);
}

// Loads of values that the kernel before this one may have written.  Volatile and through the coherent path: a read-only
// load counts as movable, and must not move above the wait for that kernel.
__device__ __forceinline__ float load_prior(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void load_prior(const uint8_t* p, uint32_t* r) {  // 16 bytes
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(p) : "memory");
}
__device__ __forceinline__ void lds_128(uint32_t addr, uint32_t* r) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t load_prior(const uint8_t* p) {
  uint32_t v;
  asm volatile("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Bias of one output column: an f32 vector, or an NVFP4-encoded one decoded as the reference's post-op
// kernels decode it, (e2m1 * e4m3) * global_scale (utils/nvfp4/tensor.rs:48-57, gpt/projection_postop.rs:97-115).
__device__ __forceinline__ float bias_value(const GemmParams& p, uint32_t col) {
  if (p.bias) return load_prior(p.bias + col);
  const uint32_t byte = load_prior(p.bias_bytes + (col >> 1));
  const uint32_t nib = (col & 1u) ? (byte >> 4) : (byte & 0xfu);
  uint32_t h2;
  asm("{ .reg .b8 t; cvt.u8.u32 t, %1; cvt.rn.f16x2.e2m1x2 %0, t; }" : "=r"(h2) : "r"(nib));
  const float q = __low2float(*reinterpret_cast<__half2*>(&h2));
  uint32_t s2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(s2) : "h"(static_cast<uint16_t>(load_prior(p.bias_scales + (col >> 4)))));
  const float sc = __low2float(*reinterpret_cast<__half2*>(&s2));
  return __fmul_rn(__fmul_rn(q, sc), load_prior(p.bias_global));
}

// ---- epilogue stores ------------------------------------------------------------------------

template <typename OutT>
__device__ __forceinline__ void store_row32(OutT* dst, const float (&v)[32], uint32_t valid, bool vec);

template <>
__device__ __forceinline__ void store_row32<float>(float* dst, const float (&v)[32], uint32_t valid, bool vec) {
  if (vec && valid == 32) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (static_cast<uint32_t>(i) < valid) dst[i] = v[i];
  }
}
template <>
__device__ __forceinline__ void store_row32<__nv_bfloat16>(__nv_bfloat16* dst, const float (&v)[32], uint32_t valid,
                                                           bool vec) {
  if (vec && valid == 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * i + 2 * j], v[8 * i + 2 * j + 1]);
        w[j] = *reinterpret_cast<uint32_t*>(&h);
      }
      reinterpret_cast<uint4*>(dst)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (static_cast<uint32_t>(i) < valid) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

template <typename OutT>
__device__ __forceinline__ float load_out(const OutT* p);
template <>
__device__ __forceinline__ float load_out<float>(const float* p) {
  return *p;
}
template <>
__device__ __forceinline__ float load_out<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}

// One row (128 bytes) of an epilogue sub-tile into the staging buffer, 16-byte chunks XOR-swizzled
// with the row index exactly as the SWIZZLE_128B tensor map of the output expects.
template <typename OutT>
struct SubTile;
template <>
struct SubTile<float> {
  static constexpr int kCols = 32;
  __device__ __forceinline__ static void stage(uint32_t row_addr, uint32_t row, const float* v) {
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      const uint32_t dst = row_addr + ((c ^ (row & 7u)) << 4);
      asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "f"(v[4 * c]), "f"(v[4 * c + 1]),
                   "f"(v[4 * c + 2]), "f"(v[4 * c + 3])
                   : "memory");
    }
  }
};
// v += the row of an f32 sub-tile that a TMA load has left in the staging buffer, laid out as `stage` writes it
__device__ __forceinline__ void add_staged_row(uint32_t row_addr, uint32_t row, float* v) {
#pragma unroll
  for (uint32_t c = 0; c < 8; ++c) {
    float r[4];
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3])
                 : "r"(row_addr + ((c ^ (row & 7u)) << 4))
                 : "memory");
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) v[4 * c + j] = __fadd_rn(v[4 * c + j], r[j]);
  }
}
template <>
struct SubTile<__nv_bfloat16> {
  static constexpr int kCols = 64;
  __device__ __forceinline__ static void stage(uint32_t row_addr, uint32_t row, const float* v) {
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * c + 2 * j], v[8 * c + 2 * j + 1]);
        w[j] = *reinterpret_cast<uint32_t*>(&h);
      }
      const uint32_t dst = row_addr + ((c ^ (row & 7u)) << 4);
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3])
                   : "memory");
    }
  }
};

// ---- the kernel -----------------------------------------------------------------------------

// Shared-memory plan of one launch, chosen on the host (all offsets from the 1024-byte aligned
// base): A stages, B slots, SFA stages, SFB stages, kStoreBufs epilogue staging buffers, barriers.
// Streaming mode: one B slot and one SFB stage per pipeline stage.  Resident mode (short K): the whole
// [kBlockN x K] B panel of the current column block stays in shared memory -- one slot per
// k-tile, its scale factors in tensor memory only -- while a CTA walks down the row blocks, so only A
// tiles stream through the ring.  A CTA's last tile is staged over the A stages and B slots.
// kBeside: launched with GemmNeighbour::kBesidePrior.  A form of its own, because a test at run time in the five roles' waits cost
// every launch 2 % (24 shapes up to 9 us: 7136 x 448 x K 1344 f32 7.8 -> 8.4 us, 1000 x 1024 x K 4096 bf16 7.2 -> 7.5).
template <int kBlockM, int kBlockN, typename OutT, StorePath kStore, int kPanel, bool kPair, bool kBeside>
__global__ void __launch_bounds__(kThreads, 1)
    nvfp4_gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                              const __grid_constant__ CUtensorMap tmap_out,
                              const __grid_constant__ CUtensorMap tmap_aux, const GemmParams p) {
  using C = Cfg<kBlockM, kBlockN, kPanel, kPair>;
  constexpr bool kResident = C::kResident;
  constexpr bool kTmaStore = kStore != StorePath::kDirect, kResidual = kStore == StorePath::kTmaResidual;
  static_assert(!kResidual || sizeof(OutT) == 4, "the residual stream of the TMA path is f32");
  constexpr int kMHalves = C::kMHalves;
  constexpr int kAStageBytes = C::kAStageBytes;
  constexpr int kSfaStageBytes = C::kSfaStageBytes;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

  const uint32_t stages = p.stages;
  const uint32_t b_slots = kResident ? p.num_k_tiles : stages;
  // No more column sets than stages: a scale-factor warp that has a free set for a k-tile, whose predecessor there has been
  // issued, then knows that the `full` barrier it is going to arrive on is in that k-tile's phase.
  const uint32_t sf_sets = min(static_cast<uint32_t>(C::kSfSets), stages);
  const uint32_t smem_a = smem_base;
  const uint32_t smem_b = smem_a + stages * kAStageBytes;
  const uint32_t smem_sfa = smem_b + b_slots * C::kBStageBytes;
  const uint32_t smem_sfb = smem_sfa + stages * kSfaStageBytes;
  const uint32_t smem_store = smem_sfb + (kResident ? 0 : stages * C::kSfbStageBytes);  // staging ring, 16 KB buffers, 1024-byte aligned
  const uint32_t smem_bar = smem_store + C::kStoreBufs * kStoreStageBytes;
  // barrier block: full[8], empty[8], scales_full[8], tmem_full[2], tmem_empty[2], b_full, b_empty, mma_drain,
  // staged[4], stored[4], final[10], tmem base, abort flag
  const uint32_t smem_bias = smem_bar + 512;  // kBlockN floats per epilogue group
  const uint32_t bar_full = smem_bar;
  const uint32_t bar_empty = bar_full + 8 * kMaxStages;
  const uint32_t bar_scales_full = bar_empty + 8 * kMaxStages;  // the scale tiles of a stage, ahead of its operands
  const uint32_t bar_tmem_full = bar_scales_full + 8 * kMaxStages;
  const uint32_t bar_tmem_empty = bar_tmem_full + 16;
  const uint32_t bar_b_full = bar_tmem_empty + 16;
  const uint32_t bar_b_empty = bar_b_full + 8;
  const uint32_t bar_mma_drain = bar_b_empty + 8;  // abort path only: issued MMAs have retired
  const uint32_t bar_staged = bar_mma_drain + 8;               // one per staging buffer: a sub-tile is in it
  const uint32_t bar_stored = bar_staged + 8 * C::kStoreBufs;  // one per staging buffer: its TMA store has read it
  const uint32_t bar_final = bar_stored + 8 * C::kStoreBufs;   // one per buffer of a CTA's last tile: a sub-tile is in it
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(
      smem_gen + (smem_bar - smem_base) + 8 * (3 * kMaxStages + 7 + 2 * C::kStoreBufs + kMaxFinal));
  volatile uint32_t* abort_flag = tmem_base_ptr + 1;

  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
#ifdef NVFP4_GEMM_TRACE
  uint32_t trace_n = 0;
#endif

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_b)) : "memory");
    if (kTmaStore) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_out)) : "memory");
      if (p.aux) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_aux)) : "memory");
    }
    *abort_flag = 0;
  }
  // In a pair, a tile is two CTAs' blocks of rows beside one block of columns, of which each loads a half; the first issues the
  // MMAs of both.  Its `full` and `tmem_empty` barriers count both CTAs.
  uint32_t rank = 0;
  if (kPair) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  rank = __shfl_sync(0xffffffffu, rank, 0);
  if (warp == 1) {  // a barrier per lane and pass, in the order of the barrier block
    constexpr uint32_t kTmemEmpty = 3 * kMaxStages + 2, kStaged = kTmemEmpty + 5, kStored = kStaged + C::kStoreBufs,
                       kFinal = kStored + C::kStoreBufs;
    for (uint32_t b = lane; b < kFinal + kMaxFinal; b += 32) {
      // full: the operands, and the scale factors of the four warps; a released accumulator: both groups' warps; a staged
      // sub-tile: the group's warps
      const uint32_t count = b < kMaxStages                                        ? (kPair ? 9 : 5)
                             : b == kTmemEmpty || b == kTmemEmpty + 1              ? (kPair ? 16 : 8)
                             : (b >= kStaged && b < kStored) || b >= kFinal ? 4
                                                                                   : 1;
      mbar_init(smem_bar + 8 * b, count);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    if constexpr (kPair) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_ptr)),
                   "r"(static_cast<uint32_t>(kTmemCols))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_ptr)),
                   "r"(static_cast<uint32_t>(kTmemCols))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
  }
  // Programmatic dependent launch: the CTA touches only its own SM up to the roles' waits for what runs before it in the stream,
  // each of which stands ahead of the role's first access to memory, behind the fetch of its code and of its first tile.  The
  // GEMM itself does not allow the next kernel to start early: its CTAs end at different times, and the first SMs that come
  // free would take all of a small grid's CTAs.  Another GEMM that needs nothing of it is the exception (GemmNeighbour).
  if (kPair)
    cluster_sync();
  else
    __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_base_ptr, 0);  // warp uniform also to the compiler

  // Work list, identical in every role.  Streaming: work items (tile, k-split) strided over the
  // grid, column block fastest (neighbouring CTAs share A rows in L2).  Resident: each CTA owns a
  // contiguous range of tiles ordered column block major, so its B panel changes at most a
  // couple of times.
  const uint32_t tiles_mn = p.num_m_blocks * p.num_n_blocks;
  uint32_t w_begin, w_end, w_step, band_n = 0;
  if (kResident && p.resident_cpn) {
    // Column block c / cpn, row blocks j, j + cpn, j + 2 cpn, ...: at any moment the CTAs of all
    // column blocks work on the same band of cpn row blocks, so whole output rows are written at
    // about the same time (full DRAM pages when L2 writes them back).
    const bool has_work = blockIdx.x < p.resident_cpn * p.num_n_blocks;
    band_n = blockIdx.x / p.resident_cpn;
    w_begin = blockIdx.x - band_n * p.resident_cpn;
    w_end = has_work ? p.num_m_blocks : 0;
    w_step = p.resident_cpn;
  } else if (kResident) {
    w_begin = static_cast<uint32_t>(static_cast<uint64_t>(tiles_mn) * blockIdx.x / gridDim.x);
    w_end = static_cast<uint32_t>(static_cast<uint64_t>(tiles_mn) * (blockIdx.x + 1) / gridDim.x);
    w_step = 1;
  } else {
    w_begin = kPair ? blockIdx.x / 2 : blockIdx.x;
    w_end = tiles_mn * p.k_splits;
    w_step = kPair ? gridDim.x / 2 : gridDim.x;
  }
  auto decode = [&](uint32_t w, uint32_t& m_blk, uint32_t& n_blk, uint32_t& split) {
    if (kResident && p.resident_cpn) {
      n_blk = band_n;
      m_blk = w;
      split = 0;
    } else if (kResident) {
      n_blk = w / p.num_m_blocks;
      m_blk = w - n_blk * p.num_m_blocks;
      split = 0;
    } else {
      const uint32_t tile = w % tiles_mn;
      split = w / tiles_mn;
      m_blk = tile / p.num_n_blocks;
      n_blk = tile - m_blk * p.num_n_blocks;
      if (kPair) m_blk = 2 * m_blk + rank;  // may lie below the matrix
    }
  };

  // Sub-tiles of 128 rows x 128 bytes leave through shared memory with TMA stores.  The items of a tile -- (row half,
  // column sub-tile) -- alternate between the two epilogue groups; with an odd number of items per tile (192 bf16
  // columns = 3) the group that takes two alternates from tile to tile, which the double-buffered accumulator evens out.
  constexpr int kSub = SubTile<OutT>::kCols;
  constexpr int kNumSub = kBlockN / kSub;
  constexpr int kItems = kMHalves * kNumSub;
  constexpr uint32_t kRing = C::kStoreBufs / 2;  // staging buffers per group
  // The rotating accumulator is taken from the half the next tile overwrites: columns 128.. of the tiles at column 0, 0.. of
  // those at column 128.
  constexpr int kTurns = (kItems + 1) / 2;               // items of a group and tile, at most
  constexpr int kFirstTurns = C::kRotate ? kTurns / 2 : kTurns;  // of them, those the next tile's MMAs wait for
  auto item_of = [&](uint32_t group, uint32_t tile_iter, int turn) {  // kItems: none
    if (C::kRotate) return static_cast<int>(group) + 2 * ((tile_iter & 1u) ? turn : (turn + kFirstTurns) % kTurns);
    return min(static_cast<int>((kItems & 1) ? (group ^ (tile_iter & 1u)) : group) + 2 * turn, kItems);
  };
  // The last tile of a CTA has the shared memory of the operands to itself: what the ring does not hold of it is staged there,
  // every sub-tile in a buffer of its own, and no sub-tile waits for a store: 2304 x 768 x K 8192 f32 17.4 -> 16.0 us, 1024 x
  // 1024 x K 8192 13.4 -> 12.0, 8192 x 768 x K 2304 bf16 11.2 -> 10.8.  (Not for 192 columns and four k-tiles: it spills.)
  constexpr int kOperandBytes = 3 * (kAStageBytes + (kResident ? 0 : C::kBStageBytes)) + kPanel * C::kBStageBytes / 2;  // at least
  constexpr int kBeyondRing = kTurns - static_cast<int>(kRing), kSpare = kOperandBytes / (2 * kStoreStageBytes);
  constexpr int kFinalTurns =
      kResidual || (kPanel == 4 && kBlockN == 192) || kBeyondRing < 0 ? 0 : kBeyondRing < kSpare ? kBeyondRing : kSpare;
  static_assert(2 * kFinalTurns <= static_cast<int>(kMaxFinal), "buffers of the last tile");
  auto in_final = [&](int turn) { return turn >= static_cast<int>(kRing) && turn < static_cast<int>(kRing) + kFinalTurns; };
  auto final_index = [&](uint32_t group, int turn) { return static_cast<uint32_t>(turn - static_cast<int>(kRing)) * 2u + group; };
  auto item_valid = [&](int item, uint32_t m_blk, uint32_t n_blk) {  // there is one, and not wholly outside the matrix
    if (item >= kItems) return false;
    const uint32_t h = static_cast<uint32_t>(item / kNumSub), sub = static_cast<uint32_t>(item % kNumSub);
    return n_blk * kBlockN + sub * kSub < p.n && m_blk * kBlockM + h * kRowBlock < p.m;
  };
  // epilogue and store warps wait on what the MMA warp feeds them: their limit is the longer one, so that the status
  // word names the role whose input failed to come
  const uint64_t downstream_timeout_ns = 2 * p.wait_timeout_ns;
  // a ReLU^2 with its pre-activation kept stores every item twice: the pre-activation, then the activation
  const int item_passes = (!kResidual && p.epilogue == NVFP4_EPI_RELU2 && p.aux) ? 2 : 1;
  // kResidual, the f32 residual stream: an item's old values arrive in the staging buffer the item will leave from,
  // `stored` of a buffer then means that they are there, and the epilogue adds to them in place.

  if (warp == 0) {
    // ===================== TMA producer =====================
    // Warp uniform like the MMA issuer: from inside a single-lane branch every copy took about 140 cycles to issue, and the six of
    // a streamed k-tile 840 of the 1170 to 1300 the k-tile had (480 now).  8192 x 768 x K 3072 bf16 14.7 -> 13.2 us, 8192 x
    // 32000 x K 768 142 -> 118, 16 x 2304 x K 768 5.7 -> 4.8, 65536 x 3072 x K 768 111 -> 101.
    uint32_t stage = 0, phase = 0, issued = 0, runs = 0, prev_n = 0xffffffffu;
    [[maybe_unused]] uint32_t tile_iter = 0;
    bool ok = true;
    for (uint32_t w = w_begin; w < w_end && ok; w += w_step) {
      uint32_t m_blk, n_blk, split;
      decode(w, m_blk, n_blk, split);
      const uint32_t kt_begin = split * p.k_tiles_per_split;
      const uint32_t kt_end = min(p.num_k_tiles, kt_begin + p.k_tiles_per_split);
      const uint32_t first_blk128 = n_blk * kBlockN / 128u;
      const uint32_t blks128 = min(static_cast<uint32_t>(C::kSfBlocks), p.sfb_blocks128 - first_blk128);
      if (kResident && n_blk != prev_n) {
        // new column block: wait until the MMAs of the previous run have retired, then load the panel
        const bool free = runs == 0 || mbar_wait(bar_b_empty, (runs - 1) & 1u, abort_flag, kStatusProducerTimeout, p.wait_timeout_ns);
        if (!__all_sync(0xffffffffu, free)) {
          ok = false;
          break;
        }
        wait_for_inputs<kBeside>();
        if (elect_one()) {
          mbar_expect_tx(bar_b_full, p.num_k_tiles * C::kBStageBytes);
          for (uint32_t kt = 0; kt < p.num_k_tiles; ++kt)
            tma_load_2d(smem_b + kt * C::kBStageBytes, &tmap_b, bar_b_full, static_cast<int32_t>(kt * kBlockKBytes),
                        static_cast<int32_t>(n_blk * kBlockN));
        }
        __syncwarp();
        prev_n = n_blk;
        ++runs;
      }
      // scale blocks of A inside the matrix (the second row half of a tall tile may lie below it)
      const uint32_t a_blks = min(static_cast<uint32_t>(kMHalves), p.sfa_blocks128 - min(m_blk * kMHalves, p.sfa_blocks128));
      if (kResident) {
        // A goes to L2 two tiles ahead: from HBM, beside the output's writes, a k-tile takes 1900 cycles and more, longer than
        // the ring covers (65536 x 2304 x K 768 80 us without).  In a banded schedule the column blocks' CTAs read the same A
        // at about the same time and take turns.
        const uint32_t ahead = w + 2 * w_step;
        if (ahead < w_end && (p.resident_cpn == 0 || (tile_iter + band_n) % p.num_n_blocks == 0) && elect_one()) {
          uint32_t m_ahead, n_ahead, none;
          decode(ahead, m_ahead, n_ahead, none);
          for (uint32_t kt = 0; kt < p.num_k_tiles; ++kt)
            tma_prefetch_2d(&tmap_a, static_cast<int32_t>(kt * kBlockKBytes), static_cast<int32_t>(m_ahead * kBlockM));
          bulk_prefetch(p.sfa + static_cast<size_t>(m_ahead) * p.k_atoms * kSfTileBytes, p.k_atoms * kSfTileBytes);
        }
        __syncwarp();
        ++tile_iter;
      }
      for (uint32_t kt = kt_begin; kt < kt_end; ++kt) {
        const bool free = mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_flag, kStatusProducerTimeout, p.wait_timeout_ns);
        if (!__all_sync(0xffffffffu, free)) {
          ok = false;
          break;
        }
        if (issued == 0) wait_for_inputs<kBeside>();
        GEMM_TRACE(0, 1, lane == 0);
        // test hook: this stage is never armed nor loaded, so its consumers' waits run out
        const bool skip = (p.debug_flags & kDebugSkipFirstLoad) && blockIdx.x == 0 && issued == 0;
        if (!skip && elect_one()) {
          const uint32_t atoms = min(static_cast<uint32_t>(kKAtomsPerStage), p.k_atoms - kt * kKAtomsPerStage);
          const uint32_t sf_bytes = atoms * kSfTileBytes;
          // The scale tiles first and on a barrier of their own: they are in tensor memory when the operands land.  On one
          // barrier with them a stage was occupied 460 cycles longer.
          const uint32_t scales = bar_scales_full + 8 * stage, full = bar_full + 8 * stage;
          mbar_expect_tx(scales, sf_bytes * (a_blks + (kResident ? 0u : blks128)));
#pragma unroll
          for (uint32_t h = 0; h < static_cast<uint32_t>(kMHalves); ++h)
            if (h < a_blks)
              bulk_load(smem_sfa + stage * kSfaStageBytes + h * kSfBlockStageBytes,
                        p.sfa + (static_cast<size_t>(m_blk * kMHalves + h) * p.k_atoms + kt * kKAtomsPerStage) * kSfTileBytes,
                        sf_bytes, scales);
          if (!kResident) {
#pragma unroll
            for (uint32_t i = 0; i < static_cast<uint32_t>(C::kSfBlocks); ++i)
              if (i < blks128)
                bulk_load(smem_sfb + stage * C::kSfbStageBytes + i * kSfBlockStageBytes,
                          p.sfb + (static_cast<size_t>(first_blk128 + i) * p.k_atoms + kt * kKAtomsPerStage) * kSfTileBytes,
                          sf_bytes, scales);
          }
          const int32_t x = static_cast<int32_t>(kt * kBlockKBytes);
          if constexpr (kPair) {
            const uint32_t both = leader_address(full);
            if (rank == 0) mbar_expect_tx(full, 2 * (kAStageBytes + C::kBStageBytes));
            tma_load_2d_pair(smem_a + stage * kAStageBytes, &tmap_a, both, x, static_cast<int32_t>(m_blk * kBlockM));
            tma_load_2d_pair(smem_b + stage * C::kBStageBytes, &tmap_b, both, x,
                             static_cast<int32_t>(n_blk * kBlockN + rank * C::kBRows));
          } else {
            mbar_expect_tx(full, kAStageBytes + (kResident ? 0 : C::kBStageBytes));
            tma_load_2d(smem_a + stage * kAStageBytes, &tmap_a, full, x, static_cast<int32_t>(m_blk * kBlockM));
            if (!kResident) tma_load_2d(smem_b + stage * C::kBStageBytes, &tmap_b, full, x, static_cast<int32_t>(n_blk * kBlockN));
          }
        }
        __syncwarp();
        GEMM_TRACE(0, 2, lane == 0);
        ++issued;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (kPair) {
      // the commits that hand the last stages back come from the other CTA: they arrive before this one ends
      for (uint32_t i = 0; i < stages && ok; ++i) {  // (a stage never used is free at once)
        ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * stage, phase ^ 1u, abort_flag, kStatusProducerTimeout, p.wait_timeout_ns));
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok) {
      // aborting: give copies already in flight a bounded chance to land before the CTA exits
      const uint32_t pending = min(issued, stages);
      for (uint32_t i = 0; i < pending; ++i) {
        const uint32_t s = (stage + stages - 1 - i) % stages;
        const uint32_t ph = (s < stage) ? phase : (phase ^ 1u);
        for (int spin = 0; spin < 4096 && !(mbar_try_wait(bar_scales_full + 8 * s, ph) && mbar_try_wait(bar_full + 8 * s, ph)); ++spin) {
        }
      }
    }
    // This grid is not complete before the one beside it.  One CTA waits, so that the SMs of the others go to the CTAs still to start
    // (all of them: backward of 1000 x 3072 f32 39.4 -> 41.6 us).
    if (kBeside && blockIdx.x == 0) wait_for_prior_kernels();
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    // The whole warp walks the loops so that tile / stage bookkeeping and the descriptors stay warp
    // uniform (uniform registers); one elected lane issues the tensor-core instructions.  Issuing
    // from inside a single-lane branch instead costs ~140 cycles per tcgen05.mma.
    {
      constexpr uint32_t idesc = make_idesc<kBlockN, kPair>();
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0, runs = 0, prev_n = 0xffffffffu, sf_set = 0, tile_iter = 0;
      bool ok = true;
      for (uint32_t w = rank == 0 ? w_begin : w_end; w < w_end && ok; w += w_step, ++tile_iter) {
        uint32_t m_blk, n_blk, split;
        decode(w, m_blk, n_blk, split);
        const uint32_t kt_begin = split * p.k_tiles_per_split;
        const uint32_t kt_end = min(p.num_k_tiles, kt_begin + p.k_tiles_per_split);
        if (kResident && n_blk != prev_n) {
          if (!__all_sync(0xffffffffu, mbar_wait(bar_b_full, runs & 1u, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns))) {
            ok = false;
            break;
          }
          prev_n = n_blk;
          ++runs;
        }
        GEMM_TRACE(1, 10, lane == 0);
        if (!__all_sync(0xffffffffu, mbar_wait(bar_tmem_empty + 8 * acc, acc_phase ^ 1u, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns))) {
          ok = false;
          break;
        }
        GEMM_TRACE(1, 11, lane == 0);
        tcgen05_fence_after();
        const uint32_t tmem_acc = tmem_base + (C::kRotate ? (tile_iter & 1u) * 128u : acc * C::kAccCols);
        for (uint32_t kt = kt_begin; kt < kt_end; ++kt) {
          // operands in shared memory, scale factors in column set `sf_set`
          const bool ready = mbar_wait(bar_full + 8 * stage, phase, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns);
          if (!__all_sync(0xffffffffu, ready)) {
            ok = false;
            break;
          }
          GEMM_TRACE(1, 12, lane == 0);
          tcgen05_fence_after();
          const uint32_t atoms = min(static_cast<uint32_t>(kKAtomsPerStage), p.k_atoms - kt * kKAtomsPerStage);
          const uint32_t b_slot = kResident ? kt : stage;
          const uint32_t tsfa = tmem_base + C::kTmemSfa + sf_set * C::kSfSetCols;
          const uint32_t tsfb = kResident ? tmem_base + C::kTmemPanel + kt * C::kSfbTileCols : tsfa + C::kSfaSetCols;
          const uint64_t desc_a = make_ab_desc(smem_a + stage * kAStageBytes);
          const uint64_t desc_b = make_ab_desc(smem_b + b_slot * C::kBStageBytes);
          if (elect_one()) {
#pragma unroll
            for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
              // 64 nibbles = 32 bytes further along the swizzled row: +2 in the 16-byte start field; the
              // second row half of a tall tile sits 16 KB further in the A stage and has its own accumulator
              // and A scale columns
              if (kb < atoms) {
#pragma unroll
                for (uint32_t h = 0; h < static_cast<uint32_t>(kMHalves); ++h)
                  (kPair ? tcgen05_mma_nvf4_pair : tcgen05_mma_nvf4)(tmem_acc + h * kBlockN, desc_a + h * (kAHalfBytes >> 4) + kb * 2, desc_b + kb * 2, idesc,
                                   (kt > kt_begin || kb > 0) ? 1u : 0u, tsfa + h * 4 * kKAtomsPerStage + kb * 4,
                                   tsfb + kb * C::kSfbColsPerAtom);
              }
            }
            commit<kPair>(bar_empty + 8 * stage);  // frees the stage and the scale-factor column set once these MMAs retire
          }
          __syncwarp();
          GEMM_TRACE(1, 13, lane == 0);
          if (++sf_set == sf_sets) sf_set = 0;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        // last tile of this column block: the resident panel may be replaced once everything issued so far has retired (a
        // banded schedule keeps one column block)
        const bool release_panel = kResident && p.resident_cpn == 0 && w + 1 == (n_blk + 1) * p.num_m_blocks;
        if (elect_one()) {
          commit<kPair>(bar_tmem_full + 8 * acc);  // accumulator complete
          if (release_panel) tcgen05_commit(bar_b_empty);
        }
        __syncwarp();
        GEMM_TRACE(1, 14, lane == 0);
        if (++acc == C::kAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
      if (!ok) {
        // aborting: give the MMAs already issued a bounded chance to retire before tensor memory is freed
        if (elect_one()) commit<kPair>(bar_mma_drain);
        __syncwarp();
        for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(bar_mma_drain, 0); ++spin) {
        }
      }
    }
  } else if (warp >= 8 && warp < 12) {
    // ===================== scale-factor warps =====================
    // Four warps (one per 32-lane quadrant of tensor memory) read the 512-byte scale tiles of each
    // k-tile from shared memory -- lane l takes the 16 bytes of rows l, l+32, l+64, l+96 -- and write
    // them with tcgen05.st into the four columns per k-atom the MMA expects, replicated in every
    // quadrant.  This keeps scale-factor transport off the tensor pipe (tcgen05.cp runs in order
    // with the MMAs and costs about a third of a wide-tile main loop).
    const uint32_t quad = warp & 3u;
    uint32_t stage = 0, phase = 0, sf_set = 0, runs = 0, prev_n = 0xffffffffu;
    // The commit that frees a k-tile's stage says that its column set is free as well: the set is written again for the k-tile
    // `sf_sets` further on, no more than a ring of stages, so that stage's barrier cannot have gone a second phase on.  With a
    // commit of the set's own the issuing warp had one more each k-tile: 16384 x 768 x K 768 bf16 10.8 -> 10.6 us, 4096 x 3072
    // 10.5 -> 10.4, 2048 x 4096 x K 1024 ReLU^2 f32 15.9 -> 15.7; nothing slower.
    uint32_t fresh_sets = sf_sets, prior_stage = 0, prior_phase = 0;
    bool ok = true;
    for (uint32_t w = w_begin; w < w_end && ok; w += w_step) {
      uint32_t m_blk, n_blk, split;
      decode(w, m_blk, n_blk, split);
      const uint32_t kt_begin = split * p.k_tiles_per_split;
      const uint32_t kt_end = min(p.num_k_tiles, kt_begin + p.k_tiles_per_split);
      if (kResident && n_blk != prev_n) {
        // The panel's B scale factors, once per column block and from memory: its tiles then leave only those of A to move
        // (500 to 600 cycles a k-tile with B, more than its MMAs take).  The MMAs of the column block before have retired.
        if (runs > 0 && !mbar_wait(bar_b_empty, (runs - 1) & 1u, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns)) break;
        __syncwarp();
        tcgen05_fence_after();
        wait_for_inputs<kBeside>();
        const uint32_t first_blk128 = n_blk * kBlockN / 128u;
        const uint8_t* src = p.sfb + static_cast<size_t>(first_blk128) * p.k_atoms * kSfTileBytes + lane * 16;
        const size_t block_bytes = static_cast<size_t>(p.k_atoms) * kSfTileBytes;
#pragma unroll 1
        for (uint32_t kt = 0; kt < p.num_k_tiles; ++kt) {
          const uint32_t atoms = min(static_cast<uint32_t>(kKAtomsPerStage), p.k_atoms - kt * kKAtomsPerStage);
          const uint32_t dst = tmem_base + C::kTmemPanel + kt * C::kSfbTileCols + ((quad * 32u) << 16);
          uint32_t r[kKAtomsPerStage][C::kSfBlocks * 4] = {};  // blocks outside the matrix: zeros
#pragma unroll
          for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb)
#pragma unroll
            for (uint32_t i = 0; i < static_cast<uint32_t>(C::kSfBlocks); ++i)
              if (kb < atoms && first_blk128 + i < p.sfb_blocks128)
                load_prior(src + i * block_bytes + (kt * kKAtomsPerStage + kb) * kSfTileBytes, &r[kb][4 * i]);
#pragma unroll
          for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
            if (kb < atoms) {
              if constexpr (kBlockN == 192) {
                const bool odd = (n_blk & 1u) != 0;  // the tile starts in the middle of its first block
                uint32_t sel[6];
#pragma unroll
                for (int j = 0; j < 6; ++j) sel[j] = odd ? r[kb][j + 2] : r[kb][j];
                tcgen05_st_x4(dst + kb * 6, sel);
                tcgen05_st_x2(dst + kb * 6 + 4, sel + 4);
              } else {
#pragma unroll
                for (int i = 0; i < C::kSfBlocks; ++i) tcgen05_st_x4(dst + kb * C::kSfbColsPerAtom + i * 4, &r[kb][4 * i]);
              }
            }
          }
        }
        prev_n = n_blk;
        ++runs;
      }
      for (uint32_t kt = kt_begin; kt < kt_end; ++kt) {
        if (!mbar_wait(bar_scales_full + 8 * stage, phase, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns)) {
          ok = false;
          break;
        }
        GEMM_TRACE(2, 20, warp == 8 && lane == 0);
        const uint32_t atoms = min(static_cast<uint32_t>(kKAtomsPerStage), p.k_atoms - kt * kKAtomsPerStage);
        const uint32_t sfa_s = smem_sfa + stage * kSfaStageBytes + lane * 16;
        const uint32_t tsfa = tmem_base + C::kTmemSfa + sf_set * C::kSfSetCols + ((quad * 32u) << 16);
        // all shared-memory reads first (independent, pipelined), then the tensor-memory stores
        uint32_t ra[kMHalves][kKAtomsPerStage][4];
#pragma unroll
        for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
          if (kb < atoms) {
#pragma unroll
            for (int h = 0; h < kMHalves; ++h) lds_128(sfa_s + h * kSfBlockStageBytes + kb * kSfTileBytes, ra[h][kb]);
          }
        }
        [[maybe_unused]] uint32_t rb[kKAtomsPerStage][C::kSfBlocks * 4];
        if constexpr (!kResident) {
          const uint32_t sfb_s = smem_sfb + stage * C::kSfbStageBytes + lane * 16;
#pragma unroll
          for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
            if (kb < atoms) {
#pragma unroll
              for (int i = 0; i < C::kSfBlocks; ++i) lds_128(sfb_s + i * kSfBlockStageBytes + kb * kSfTileBytes, &rb[kb][4 * i]);
            }
          }
        }
        if (fresh_sets) {
          --fresh_sets;
        } else {
          if (!mbar_wait(bar_empty + 8 * prior_stage, prior_phase, abort_flag, kStatusMmaTimeout, p.wait_timeout_ns)) {
            ok = false;
            break;
          }
          if (++prior_stage == stages) {
            prior_stage = 0;
            prior_phase ^= 1u;
          }
        }
        tcgen05_fence_after();
        __syncwarp();
        if (atoms == kKAtomsPerStage) {
#pragma unroll
          for (int h = 0; h < kMHalves; ++h) tcgen05_st_x16(tsfa + h * 4 * kKAtomsPerStage, &ra[h][0][0]);
        } else {
#pragma unroll
          for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
            if (kb < atoms) {
#pragma unroll
              for (int h = 0; h < kMHalves; ++h) tcgen05_st_x4(tsfa + h * 4 * kKAtomsPerStage + kb * 4, ra[h][kb]);
            }
          }
        }
        if constexpr (!kResident) {
          const uint32_t tsfb = tsfa + C::kSfaSetCols;
          if constexpr (kBlockN == 192) {
            // Six scale words (192 rows of B) per k-atom out of the eight loaded: words 0..5 when the tile
            // starts on a 128-row block boundary (even column block), words 2..7 when it starts in the
            // middle of the first block (odd column block).
            const bool odd = (n_blk & 1u) != 0;
            uint32_t sel[kKAtomsPerStage][6];
#pragma unroll
            for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb)
#pragma unroll
              for (int j = 0; j < 6; ++j) sel[kb][j] = odd ? rb[kb][j + 2] : rb[kb][j];
            if (atoms == kKAtomsPerStage) {
              tcgen05_st_x16(tsfb, &sel[0][0]);
              tcgen05_st_x8(tsfb + 16, &sel[0][0] + 16);
            } else {
#pragma unroll
              for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
                if (kb < atoms) {
                  tcgen05_st_x4(tsfb + kb * 6, sel[kb]);
                  tcgen05_st_x2(tsfb + kb * 6 + 4, sel[kb] + 4);
                }
              }
            }
          } else if (atoms == kKAtomsPerStage) {
            tcgen05_st_x16(tsfb, &rb[0][0]);
            if constexpr (C::kSfBlocks == 2) tcgen05_st_x16(tsfb + 16, &rb[2][0]);
          } else {
#pragma unroll
            for (uint32_t kb = 0; kb < kKAtomsPerStage; ++kb) {
              if (kb < atoms) {
#pragma unroll
                for (int i = 0; i < C::kSfBlocks; ++i) tcgen05_st_x4(tsfb + kb * C::kSfbColsPerAtom + i * 4, &rb[kb][4 * i]);
              }
            }
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tcgen05_fence_before();
        __syncwarp();
        // scale factors visible to the MMA issuer; that the slot has been read follows from the MMAs that need them
        if (lane == 0) {
          if (kPair)
            mbar_arrive_cluster(leader_address(bar_full + 8 * stage));
          else
            mbar_arrive(bar_full + 8 * stage);
        }
        GEMM_TRACE(2, 21, warp == 8 && lane == 0);
        if (++sf_set == sf_sets) sf_set = 0;
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  } else if (warp == 2 || warp == 3) {
    // ===================== store warps (one per epilogue group) =====================
    // Issuing a TMA store takes about 250 cycles and its read of the staging buffer up to 1000.  This warp waits for both, so
    // that between two sub-tiles the epilogue warps have only the next sub-tile to do.  Measured against one epilogue thread
    // issuing the stores between two barriers of its group: 65536 x 2304 and x 3072 bf16 at K = 768, 87.3 -> 83.0 us and
    // 116.9 -> 111.3 us.
    if (kTmaStore) {
      wait_for_inputs<kBeside>();
      const uint32_t eg = warp - 2u;
      uint32_t buf = 0, phase = 0, tile_iter = 0, issued = 0;
      bool ok = true;
      auto item_x = [&](int item, uint32_t n_blk) { return static_cast<int32_t>(n_blk * kBlockN + (item % kNumSub) * kSub); };
      auto item_y = [&](int item, uint32_t m_blk) { return static_cast<int32_t>(m_blk * kBlockM + (item / kNumSub) * kRowBlock); };
      // residual stream: a second walk over the group's items, one ring ahead, loads what they will be added to
      uint32_t load_w = w_begin, load_tile = 0, load_m = 0, load_n = 0, load_split = 0, loads = 0;
      int load_turn = kTurns;  // next turn in the tile (load_m, load_n); kTurns: on to the tile of load_w
      auto load_next = [&](uint32_t slot) {
        while (true) {
          if (load_turn >= kTurns) {
            if (load_w >= w_end) return;
            decode(load_w, load_m, load_n, load_split);
            ++load_tile;
            load_turn = 0;
            load_w += w_step;
          }
          const int item = item_of(eg, load_tile - 1, load_turn++);
          if (!item_valid(item, load_m, load_n)) continue;
          if (elect_one()) {
            mbar_expect_tx(bar_stored + 8 * slot, kStoreStageBytes);  // parts outside the matrix arrive as zeros
            tma_load_2d(smem_store + slot * kStoreStageBytes, &tmap_out, bar_stored + 8 * slot, item_x(item, load_n),
                        item_y(item, load_m));
          }
          __syncwarp();
          ++loads;
          return;
        }
      };
      if (kResidual)
        for (uint32_t b = 0; b < kRing; ++b) load_next(eg * kRing + b);
      for (uint32_t w = w_begin; w < w_end && ok; w += w_step, ++tile_iter) {
        uint32_t m_blk, n_blk, split;
        decode(w, m_blk, n_blk, split);
        if (kResidual) {
          // The items of this tile that no buffer is free for yet go to L2 during its main loop, spread over it: all at
          // once they would stand before the operands in the queue to HBM.  8192 x 768 x K 3072 from HBM: 27.2 us without,
          // 27.5 all at once, 23.4 spread; from L2 20.2.
          const uint32_t t0 = clock32(), pace = p.num_k_tiles * 700u / (kItems / 2);
          uint32_t due = 0;
          for (int turn = kRing; turn < kTurns; ++turn) {
            const int item = item_of(eg, tile_iter, turn);
            if (!item_valid(item, m_blk, n_blk)) continue;
            due += pace;
            bool staged = false;
            while (!staged && __any_sync(0xffffffffu, clock32() - t0 < due))
              staged = __any_sync(0xffffffffu, mbar_try_wait(bar_staged + 8 * (eg * kRing + buf), phase));
            if (staged) break;
            if (elect_one()) tma_prefetch_2d(&tmap_out, item_x(item, n_blk), item_y(item, m_blk));
            __syncwarp();
          }
        }
        const bool final_tile = kFinalTurns > 0 && item_passes == 1 && w + w_step >= w_end;
        for (int turn = 0; turn < kTurns && ok; ++turn) {
          const int item = item_of(eg, tile_iter, turn);
          if (!item_valid(item, m_blk, n_blk)) continue;
          const int32_t x = item_x(item, n_blk), y = item_y(item, m_blk);
          if (final_tile && in_final(turn)) {
            const uint32_t f = final_index(eg, turn);
            ok = __all_sync(0xffffffffu, mbar_wait(bar_final + 8 * f, 0, abort_flag, kStatusEpilogueTimeout, downstream_timeout_ns));
            if (ok && elect_one()) {
              if (p.k_splits > 1)
                tma_reduce_add_2d(&tmap_out, smem_base + f * kStoreStageBytes, x, y);
              else if (kResident && p.stream_out)
                tma_store_2d_streaming(&tmap_out, smem_base + f * kStoreStageBytes, x, y);
              else
                tma_store_2d(&tmap_out, smem_base + f * kStoreStageBytes, x, y);
              bulk_commit_group();
            }
            __syncwarp();
            continue;
          }
          for (int pass = 0; pass < item_passes; ++pass) {
            const uint32_t slot = eg * kRing + buf;
            const bool staged = mbar_wait(bar_staged + 8 * slot, phase, abort_flag, kStatusEpilogueTimeout, downstream_timeout_ns);
            if (!__all_sync(0xffffffffu, staged)) {
              ok = false;
              break;
            }
            // the same lane is elected every time: it is the one whose bulk groups these are
            if (elect_one()) {
              const CUtensorMap* map = item_passes == 2 && pass == 0 ? &tmap_aux : &tmap_out;
              if (!kResidual && p.k_splits > 1)
                tma_reduce_add_2d(map, smem_store + slot * kStoreStageBytes, x, y);
              else if (kResident && p.stream_out)
                tma_store_2d_streaming(map, smem_store + slot * kStoreStageBytes, x, y);
              else
                tma_store_2d(map, smem_store + slot * kStoreStageBytes, x, y);
              bulk_commit_group();
              // the buffer the epilogue needs next is handed back as soon as its store has read it: this one with a
              // single buffer, the previous one with two; with a load to come into it, this one at once
              if (kResidual) {
                bulk_wait_group_read<0>();
              } else {
                bulk_wait_group_read<static_cast<int>(kRing) - 1>();
                if (kRing == 1)
                  mbar_arrive(bar_stored + 8 * slot);
                else if (issued > 0)
                  mbar_arrive(bar_stored + 8 * (eg * kRing + (buf ^ 1u)));
              }
            }
            __syncwarp();
            if (kResidual) load_next(slot);
            ++issued;
            if (++buf == kRing) {
              buf = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (elect_one()) bulk_wait_group0();  // stores complete before the CTA exits
      __syncwarp();
      if (kResidual && !ok) {
        // aborting: give loads already in flight a bounded chance to land; load j is phase j / kRing of its buffer
        for (uint32_t j = loads > kRing ? loads - kRing : 0; j < loads; ++j)
          for (int spin = 0; spin < 4096 && !mbar_try_wait(bar_stored + 8 * (eg * kRing + j % kRing), (j / kRing) & 1u); ++spin) {
          }
      }
    }
  } else if (warp >= 4) {
    // ===================== epilogue (two groups of four warps) =====================
    const uint32_t ew = warp & 3u;               // lane quadrant of tensor memory this warp reaches
    const uint32_t eg = warp >= 12 ? 1u : 0u;    // epilogue group
    const uint32_t gtid = ew * 32 + lane;        // thread index inside the group, also the tile row
    [[maybe_unused]] const bool elected = gtid == 0;
    OutT* out = static_cast<OutT*>(p.out);
    OutT* aux = static_cast<OutT*>(p.aux);
    uint32_t acc = 0, acc_phase = 0, store_buf = 0, store_phase = kResidual ? 0u : 1u, tile_iter = 0;
    bool ok = true;  // warp uniform; false: some wait ran out, the rest of the list is walked without work
    const uint32_t my_bias = smem_bias + eg * kBlockN * 4;
    const float* my_bias_gen = reinterpret_cast<const float*>(smem_gen + (my_bias - smem_base));
    wait_for_inputs<kBeside>();
    if (gtid == 0 && eg == 0 && p.lets_next_beside) allow_next_kernel();
    const float gb = p.mode == NVFP4_GS_NONE ? 1.0f : load_prior(p.b_global);
    const float ga_scalar = p.mode == NVFP4_GS_TENSOR ? load_prior(p.a_global) : 1.0f;
    // the rows' global scales of a tile are fetched one tile ahead: their load latency would
    // otherwise sit between the accumulator becoming ready and the first store
    auto row_scale = [&](uint32_t mb, uint32_t h) {
      const uint32_t r = mb * kBlockM + h * kRowBlock + gtid;
      return (p.mode == NVFP4_GS_ROWWISE_A && r < p.m) ? load_prior(p.a_global + r) : 0.0f;
    };
    // The bias slice of a tile travels the same way: its values are fetched into registers one tile ahead
    // and reach shared memory only when the column block changes (a banded schedule keeps a CTA on one
    // column block for many tiles).
    float bias_next[C::kBiasSlots];
    uint32_t staged_bias_blk = 0xffffffffu;
    auto fetch_bias = [&](uint32_t nb) {
#pragma unroll
      for (int j = 0; j < C::kBiasSlots; ++j) {
        const uint32_t in_tile = gtid + 128 * j;
        const uint32_t col = nb * kBlockN + in_tile;
        bias_next[j] = (kTmaStore && p.epilogue != NVFP4_EPI_NONE && in_tile < static_cast<uint32_t>(kBlockN) && col < p.n)
                           ? bias_value(p, col)
                           : 0.0f;
      }
    };
    float ga_next[kMHalves] = {};
    uint32_t m_next = 0, n_next = 0, split_next = 0;
    if (w_begin < w_end) {
      decode(w_begin, m_next, n_next, split_next);
      fetch_bias(n_next);
#pragma unroll
      for (int h = 0; h < kMHalves; ++h) ga_next[h] = row_scale(m_next, h);
    }
    for (uint32_t w = w_begin; w < w_end; w += w_step, ++tile_iter) {
      const uint32_t m_blk = m_next, n_blk = n_next, split = split_next;
      float ga_row[kMHalves];
#pragma unroll
      for (int h = 0; h < kMHalves; ++h) ga_row[h] = ga_next[h];
      if (w + w_step < w_end) {
        decode(w + w_step, m_next, n_next, split_next);
#pragma unroll
        for (int h = 0; h < kMHalves; ++h) ga_next[h] = row_scale(m_next, h);
      }
      // the tile's bias slice goes through shared memory once (every row then reads it broadcast), staged before the
      // wait for the accumulator so that this hides behind the main loop
      const bool add_bias = kTmaStore && p.epilogue != NVFP4_EPI_NONE && (p.k_splits == 1 || split == 0);
      if (add_bias && n_blk != staged_bias_blk) {  // uniform across the group
        epilogue_barrier(eg);  // every warp has read the slice staged before
#pragma unroll
        for (int j = 0; j < C::kBiasSlots; ++j)
          if (gtid + 128 * j < static_cast<uint32_t>(kBlockN))
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(my_bias + (gtid + 128 * j) * 4), "f"(bias_next[j]) : "memory");
        epilogue_barrier(eg);
        staged_bias_blk = n_blk;
      }
      if (n_next != n_blk) fetch_bias(n_next);
      // Once a wait has run out a warp walks the rest of its tiles without work instead of leaving: the group's
      // barriers (a bias slice per change of column block) then always see all four warps.
      GEMM_TRACE(3 + eg, 30, elected);
      ok = ok && mbar_wait(bar_tmem_full + 8 * acc, acc_phase, abort_flag, kStatusEpilogueTimeout, downstream_timeout_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) continue;
      GEMM_TRACE(3 + eg, 31, elected);
      tcgen05_fence_after();
      // reference order: (weight * a_scale) * b_scale, then acc * scale
      float scale_h[kMHalves];
#pragma unroll
      for (int h = 0; h < kMHalves; ++h)
        scale_h[h] = __fmul_rn(__fmul_rn(p.weight, p.mode == NVFP4_GS_ROWWISE_A ? ga_row[h] : ga_scalar), gb);
      const uint32_t taddr_row = tmem_base + (C::kRotate ? (tile_iter & 1u) * 128u : acc * C::kAccCols) + ((ew * 32u) << 16);
      // The accumulator buffer goes back to the MMA warp as soon as this warp's last tcgen05.ld of the
      // tile has landed in registers: scaling, staging and the stores of that last sub-tile then run
      // beside the next tile's main loop.
      auto release_accumulator = [&]() {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (kPair)
            mbar_arrive_cluster(leader_address(bar_tmem_empty + 8 * acc));
          else
            mbar_arrive(bar_tmem_empty + 8 * acc);
        }
      };
      if (kTmaStore) {
        // the group's sub-tiles go through its shared-memory ring to the store warp; rows / columns outside the matrix
        // are clipped by the tensor map
        const bool final_tile = kFinalTurns > 0 && item_passes == 1 && w + w_step >= w_end;
        int last_turn = -1;  // behind which the accumulator, or the half of it that the next tile needs, is in registers
#pragma unroll
        for (int turn = 0; turn < kFirstTurns; ++turn)
          if (item_valid(item_of(eg, tile_iter, turn), m_blk, n_blk)) last_turn = turn;
        if (last_turn < 0) release_accumulator();  // nothing of it is for this group to read
        float row_max = -INFINITY;  // largest value this thread stores for its row in the current row half
        uint32_t max_h = 0;
        auto flush_row_max = [&]() {
          const uint32_t r = m_blk * kBlockM + max_h * kRowBlock + gtid;
          if (p.row_amax && r < p.m && row_max > 0.0f) {
            // max over the row of relu(stored value)^2: rounding to the stored type and relu^2 are both
            // monotonic, so they apply to the maximum instead of to every element; a reduction without a
            // return value, so the thread does not wait for it
            const float stored = sizeof(OutT) == 2 ? __bfloat162float(__float2bfloat16_rn(row_max)) : row_max;
            const uint32_t bits = __float_as_uint(__fmul_rn(stored, stored));
            asm volatile("red.global.max.u32 [%0], %1;" ::"l"(reinterpret_cast<unsigned int*>(p.row_amax) + r), "r"(bits)
                         : "memory");
          }
          row_max = -INFINITY;
        };
#pragma unroll 1
        for (int turn = 0; turn < kTurns; ++turn) {
          const int item = item_of(eg, tile_iter, turn);
          if (!item_valid(item, m_blk, n_blk)) continue;
          const uint32_t h = static_cast<uint32_t>(item / kNumSub);
          const int c = (item % kNumSub) * kSub;
          const uint32_t col0 = n_blk * kBlockN + c;
          if (h != max_h) {
            flush_row_max();
            max_h = h;
          }
          const float scale = kMHalves == 1 ? scale_h[0] : (h == 0 ? scale_h[0] : scale_h[kMHalves - 1]);
          const uint64_t scale2 = pack_f32x2(scale, scale);
          float v[kSub];
          {
            uint32_t r[kSub / 32][32];
#pragma unroll
            for (int q = 0; q < kSub / 32; ++q) tcgen05_ld_32x32b_x32(taddr_row + h * kBlockN + c + 32 * q, r[q]);
            tcgen05_wait_ld();
            GEMM_TRACE(3 + eg, 32, elected);
            if (turn == last_turn) release_accumulator();
            if (kResidual) {
              // the roundings of the direct path: the product, the sum with the bias, then the one with the stream
#pragma unroll
              for (int i = 0; i < kSub; i += 4) {
                const float4 b = *reinterpret_cast<const float4*>(my_bias_gen + c + i);
                mul_f32x2(v[i], v[i + 1], __uint_as_float(r[i / 32][i % 32]), __uint_as_float(r[i / 32][i % 32 + 1]), scale2);
                mul_f32x2(v[i + 2], v[i + 3], __uint_as_float(r[i / 32][i % 32 + 2]), __uint_as_float(r[i / 32][i % 32 + 3]), scale2);
                v[i] = __fadd_rn(v[i], b.x), v[i + 1] = __fadd_rn(v[i + 1], b.y);
                v[i + 2] = __fadd_rn(v[i + 2], b.z), v[i + 3] = __fadd_rn(v[i + 3], b.w);
              }
            } else if (add_bias) {
              // acc * scale + bias in one rounding (the reference rounds the product first; the
              // difference is below the f32 ulp and far inside the GEMM tolerance)
#pragma unroll
              for (int i = 0; i < kSub; i += 4) {
                const float4 b = *reinterpret_cast<const float4*>(my_bias_gen + c + i);
                fma_f32x2(v[i], v[i + 1], r[i / 32][i % 32], r[i / 32][i % 32 + 1], scale2, pack_f32x2(b.x, b.y));
                fma_f32x2(v[i + 2], v[i + 3], r[i / 32][i % 32 + 2], r[i / 32][i % 32 + 3], scale2, pack_f32x2(b.z, b.w));
              }
            } else {
#pragma unroll
              for (int i = 0; i < kSub; i += 2)
                mul_f32x2(v[i], v[i + 1], __uint_as_float(r[i / 32][i % 32]), __uint_as_float(r[i / 32][i % 32 + 1]),
                          scale2);
            }
          }
          if (p.row_amax) {
            // columns past n hold zero-filled operands (acc = 0): only real columns count
            const uint32_t valid = min(static_cast<uint32_t>(kSub), p.n - col0);
            if (valid == static_cast<uint32_t>(kSub)) {
              // four independent chains instead of one of kSub dependent maxima
              float m0 = v[0], m1 = v[1], m2 = v[2], m3 = v[3];
#pragma unroll
              for (int i = 4; i < kSub; i += 4) {
                m0 = fmaxf(m0, v[i]);
                m1 = fmaxf(m1, v[i + 1]);
                m2 = fmaxf(m2, v[i + 2]);
                m3 = fmaxf(m3, v[i + 3]);
              }
              row_max = fmaxf(row_max, fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)));
            } else {
#pragma unroll
              for (int i = 0; i < kSub; ++i)
                if (static_cast<uint32_t>(i) < valid) row_max = fmaxf(row_max, v[i]);
            }
          }
          for (int pass = 0; pass < item_passes; ++pass) {
            const bool is_pre = item_passes == 2 && pass == 0;
            if (p.epilogue == NVFP4_EPI_RELU2 && !is_pre) {
#pragma unroll
              for (int i = 0; i < kSub; i += 2) {
                v[i] = fmaxf(v[i], 0.0f);
                v[i + 1] = fmaxf(v[i + 1], 0.0f);
                square_f32x2(v[i], v[i + 1]);
              }
            }
            if (final_tile && in_final(turn)) {
              const uint32_t f = final_index(eg, turn);
              if (ok) {
                SubTile<OutT>::stage(smem_base + f * kStoreStageBytes + gtid * 128, gtid, v);
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_final + 8 * f);
              }
              continue;
            }
            const uint32_t slot = eg * kRing + store_buf;
            ok = ok && mbar_wait(bar_stored + 8 * slot, store_phase, abort_flag, kStatusEpilogueTimeout, downstream_timeout_ns);
            ok = __all_sync(0xffffffffu, ok);
            GEMM_TRACE(3 + eg, 36, elected);
            if (ok) {
              if constexpr (kResidual) add_staged_row(smem_store + slot * kStoreStageBytes + gtid * 128, gtid, v);
              SubTile<OutT>::stage(smem_store + slot * kStoreStageBytes + gtid * 128, gtid, v);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_staged + 8 * slot);
            }
            GEMM_TRACE(3 + eg, 33, elected);
            if (++store_buf == kRing) {
              store_buf = 0;
              store_phase ^= 1u;
            }
          }
        }
        flush_row_max();
      } else {
#pragma unroll 1
        for (uint32_t h = 0; h < static_cast<uint32_t>(kMHalves); ++h) {
          const uint32_t row = m_blk * kBlockM + h * kRowBlock + gtid;
          const bool row_ok = row < p.m;
          const float scale = kMHalves == 1 ? scale_h[0] : (h == 0 ? scale_h[0] : scale_h[kMHalves - 1]);
#pragma unroll 1
          for (int step = 0; step < kBlockN / 64; ++step) {
            // 32 columns; a rotating accumulator's second half first where the tile lies at column 0
            const int c = (C::kRotate && (tile_iter & 1u) == 0 ? (step + 2) % 4 : step) * 64 + eg * 32;
            uint32_t r[32];
            tcgen05_ld_32x32b_x32(taddr_row + h * kBlockN + c, r);
            tcgen05_wait_ld();
            if (h + 1 == static_cast<uint32_t>(kMHalves) && step + 1 == (C::kRotate ? 2 : kBlockN / 64)) release_accumulator();
            const uint32_t col0 = n_blk * kBlockN + c;
            if (row_ok && col0 < p.n) {
              const uint32_t valid = min(32u, p.n - col0);
              float v[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = __fmul_rn(__uint_as_float(r[i]), scale);
              const size_t off = static_cast<size_t>(row) * p.ldo + col0;
              if (p.k_splits > 1) {
                // split-K partial sums: f32 reduction into a zero-initialised output; bias joins once
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (static_cast<uint32_t>(i) < valid) {
                    float t = v[i];
                    if (p.epilogue == NVFP4_EPI_BIAS && split == 0) t = __fadd_rn(t, bias_value(p, col0 + i));
                    atomicAdd(reinterpret_cast<float*>(p.out) + off + i, t);
                  }
              } else {
                if (p.epilogue != NVFP4_EPI_NONE) {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    if (static_cast<uint32_t>(i) < valid) v[i] = __fadd_rn(v[i], bias_value(p, col0 + i));
                }
                if (p.epilogue == NVFP4_EPI_RELU2) {
                  if (aux) store_row32<OutT>(aux + off, v, valid, p.vec_store != 0);
#pragma unroll
                  for (int i = 0; i < 32; ++i) {
                    const float t = fmaxf(v[i], 0.0f);
                    v[i] = __fmul_rn(t, t);
                  }
                } else if (p.epilogue == NVFP4_EPI_RESIDUAL) {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    if (static_cast<uint32_t>(i) < valid) v[i] = __fmaf_rn(1.0f, v[i], load_out<OutT>(out + off + i));
                }
                store_row32<OutT>(out + off, v, valid, p.vec_store != 0);
              }
            }
          }
        }
      }  // direct-store path
      if (++acc == C::kAccStages) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }

  // ===================== teardown =====================
  tcgen05_fence_before();
  if (kPair) {
    __syncwarp();
    cluster_sync();  // neither CTA ends while the other may still signal it
  } else {
    __syncthreads();
  }
  if (warp == 2) {
    tcgen05_fence_after();
    if constexpr (kPair)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<uint32_t>(kTmemCols))
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(static_cast<uint32_t>(kTmemCols))
                   : "memory");
  }
}

// ---- host side ------------------------------------------------------------------------------

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// Tensor maps are pure functions of (address, extents, pitch, box): they say nothing about the bytes in
// memory.  Buffers of a training step never move, so every host thread keeps the maps it has encoded
// (the reference encodes four maps and copies them to the device before every GEMM,
// utils/nvfp4_tma_matmul/launcher.rs:106-166).
struct MapKey {
  uint64_t base;
  uint32_t kind, rows, cols, ld_or_box;
  bool operator==(const MapKey& o) const {
    return base == o.base && kind == o.kind && rows == o.rows && cols == o.cols && ld_or_box == o.ld_or_box;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    uint64_t h = k.base * 0x9E3779B97F4A7C15ull;
    h ^= (static_cast<uint64_t>(k.kind) << 56) ^ (static_cast<uint64_t>(k.rows) << 24) ^ k.cols;
    h = (h ^ (h >> 29)) * 0xBF58476D1CE4E5B9ull;
    h ^= k.ld_or_box;
    return static_cast<size_t>(h ^ (h >> 32));
  }
};
struct MapCache {
  std::unordered_map<MapKey, CUtensorMap, MapKeyHash> maps;
  uint64_t hits = 0, misses = 0;
};
MapCache& map_cache() {
  static thread_local MapCache cache;
  return cache;
}
constexpr size_t kMapCacheLimit = 8192;  // entries per host thread; the cache starts over when it is full

// Nibble matrix [rows][k] seen as bytes [rows][k/2]; box = 128 bytes x box_rows, 128-byte swizzle.
int encode_operand_map(CUtensorMap* map, const uint8_t* base, uint32_t rows, uint32_t k, uint32_t box_rows) {
  MapCache& cache = map_cache();
  const MapKey key{reinterpret_cast<uint64_t>(base), 0u, rows, k, box_rows};
  auto it = cache.maps.find(key);
  if (it != cache.maps.end()) {
    ++cache.hits;
    *map = it->second;
    return 0;
  }
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) {
    set_last_error("cuTensorMapEncodeTiled is not available from the CUDA driver");
    return static_cast<int>(cudaErrorNotSupported);
  }
  const cuuint64_t dims[2] = {k / 2, rows};
  const cuuint64_t strides[1] = {k / 2};
  const cuuint32_t box[2] = {kBlockKBytes, box_rows};
  const cuuint32_t elem_strides[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(base), dims, strides, box, elem_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled rejected the operand (base must be 16-byte aligned, k % 32 == 0)");
    return static_cast<int>(cudaErrorInvalidValue);
  }
  ++cache.misses;
  if (cache.maps.size() >= kMapCacheLimit) cache.maps.clear();
  cache.maps.emplace(key, *map);
  return 0;
}

// Output matrix [rows][ld] of f32 / bf16; box = 128 bytes x 128 rows, 128-byte swizzle.
int encode_output_map(CUtensorMap* map, void* base, int dtype, uint32_t rows, uint32_t cols, uint32_t ld) {
  MapCache& cache = map_cache();
  const MapKey key{reinterpret_cast<uint64_t>(base), dtype == NVFP4_DTYPE_F32 ? 1u : 2u, rows, cols, ld};
  auto it = cache.maps.find(key);
  if (it != cache.maps.end()) {
    ++cache.hits;
    *map = it->second;
    return 0;
  }
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return static_cast<int>(cudaErrorNotSupported);
  const size_t esz = dtype == NVFP4_DTYPE_F32 ? 4 : 2;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * esz};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / esz), kRowBlock};
  const cuuint32_t elem_strides[2] = {1, 1};
  CUresult r = fn(map, dtype == NVFP4_DTYPE_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  base, dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return static_cast<int>(cudaErrorInvalidValue);
  ++cache.misses;
  if (cache.maps.size() >= kMapCacheLimit) cache.maps.clear();
  cache.maps.emplace(key, *map);
  return 0;
}

constexpr int kMaxDevices = 64;

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -1;
  return dev;
}

// SM count of the current device (cached per device ordinal).
int sm_count() {
  static std::atomic<int> counts[kMaxDevices];
  const int dev = current_device();
  if (dev < 0) return 148;
  int c = counts[dev].load(std::memory_order_relaxed);
  if (c == 0) {
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0) c = 148;
    counts[dev].store(c, std::memory_order_relaxed);
  }
  return c;
}

// Optional event timing of GEMM launches (off by default; a measurement aid for benchmarks).
struct GemmTimingRecord {
  cudaEvent_t start, stop;
  double flops;
};
struct GemmTiming {
  std::mutex mu;
  bool enabled = false;
  std::vector<GemmTimingRecord> pool;  // events created once by timing_begin
  size_t used = 0;
} g_timing;

// Everything the host decides about one launch.
struct GemmPlan {
  uint32_t block_m = 128, block_n = 128, num_n_blocks = 0, k_splits = 1, k_tiles_per_split = 0;
  uint32_t stages = 0, grid = 0, b_resident = 0, panel = 0, resident_cpn = 0, tma_store = 0, vec_store = 0, pair = 0;
  size_t smem_bytes = 0;
  bool beside = false;  // GemmNeighbour::kBesidePrior
};

struct TileBytes {
  int fixed, stage, slot;  // see Cfg
};
template <int kBlockM, int kBlockN, int kPanel, bool kPair = false>
constexpr TileBytes tile_bytes_of() {
  using C = Cfg<kBlockM, kBlockN, kPanel, kPair>;
  return {C::kFixedBytes, C::kStageBytes, C::kSlotBytes};
}
// The resident form of a tile for so many k-tiles.
constexpr uint32_t panel_of(uint32_t block_n, uint32_t num_k_tiles) { return block_n == 128 || num_k_tiles > 3 ? 4 : 3; }
TileBytes tile_bytes(uint32_t block_m, uint32_t block_n, uint32_t panel, bool pair) {
  if (pair) return tile_bytes_of<128, 256, 0, true>();
  if (block_m == 256) return tile_bytes_of<256, 192, 0>();
  if (block_n == 256) return panel ? tile_bytes_of<128, 256, 3>() : tile_bytes_of<128, 256, 0>();
  if (block_n == 192)
    return panel == 0 ? tile_bytes_of<128, 192, 0>() : panel == 3 ? tile_bytes_of<128, 192, 3>() : tile_bytes_of<128, 192, 4>();
  return panel ? tile_bytes_of<128, 128, 4>() : tile_bytes_of<128, 128, 0>();
}

template <int kBlockM, int kBlockN, typename OutT, StorePath kStore, int kPanel, bool kPair = false, bool kBeside = false>
int launch_schedule_variant(cudaStream_t s, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo,
                         const CUtensorMap& mx, const GemmParams& p, const GemmPlan& pl) {
  if constexpr (kStore == StorePath::kTma && !kBeside) {
    if (pl.beside) return launch_schedule_variant<kBlockM, kBlockN, OutT, kStore, kPanel, kPair, true>(s, ma, mb, mo, mx, p, pl);
  }
  // the opt-in to more than 48 KB of dynamic shared memory is a per-device attribute of the kernel
  static std::atomic<int> attr_state[kMaxDevices];  // 0 = not set, 1 = set, -(error) = failed
  const int dev = current_device();
  if (dev < 0) return static_cast<int>(cudaErrorInvalidDevice);
  int st = attr_state[dev].load(std::memory_order_acquire);
  if (st == 0) {
    const cudaError_t e = cudaFuncSetAttribute(nvfp4_gemm_tcgen05_kernel<kBlockM, kBlockN, OutT, kStore, kPanel, kPair, kBeside>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
    st = e == cudaSuccess ? 1 : -static_cast<int>(e);
    attr_state[dev].store(st, std::memory_order_release);
  }
  if (st < 0) return -st;
  GemmTimingRecord* rec = nullptr;
  if (g_timing.enabled) {
    std::lock_guard<std::mutex> lock(g_timing.mu);
    if (g_timing.enabled && g_timing.used < g_timing.pool.size()) rec = &g_timing.pool[g_timing.used++];
  }
  if (rec) {
    rec->flops = 2.0 * p.m * p.n * p.k;
    cudaEventRecord(rec->start, s);
  }
  // The kernel may be set up while the one before it in the stream drains (the quantizers allow it from their start).
  // Every allocation, barrier and tensor-map fetch of the prologue and the launch itself then cost nothing behind a
  // quantizer: 16 tokens x 768 -> 2304 with its quantizer 12.3 -> 10.5 us, 8192 tokens 30.8 -> 28.5 us.
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = 2;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem_bytes;
  cfg.stream = s;
  cfg.attrs = attrs;
  cfg.numAttrs = kPair ? 2 : 1;
  int rc = static_cast<int>(
      cudaLaunchKernelEx(&cfg, nvfp4_gemm_tcgen05_kernel<kBlockM, kBlockN, OutT, kStore, kPanel, kPair, kBeside>, ma, mb, mo, mx, p));
  count_launch();
  if (rc == 0) rc = static_cast<int>(cudaGetLastError());
  if (rec) cudaEventRecord(rec->stop, s);
  return rc;
}

template <int kBlockM, int kBlockN, typename OutT, StorePath kStore>
int launch_store_variant(cudaStream_t s, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo,
                         const CUtensorMap& mx, const GemmParams& p, const GemmPlan& pl) {
  if constexpr (kBlockM == 128) {
    if constexpr (kBlockN != 128) {
      if (pl.panel == 3) return launch_schedule_variant<kBlockM, kBlockN, OutT, kStore, 3>(s, ma, mb, mo, mx, p, pl);
    }
    if constexpr (kBlockN != 256) {
      if (pl.panel == 4) return launch_schedule_variant<kBlockM, kBlockN, OutT, kStore, 4>(s, ma, mb, mo, mx, p, pl);
    }
  }
  if constexpr (kStore != StorePath::kDirect && kBlockN == 256) {
    if (pl.pair) return launch_schedule_variant<kBlockM, kBlockN, OutT, kStore, 0, true>(s, ma, mb, mo, mx, p, pl);
  }
  return launch_schedule_variant<kBlockM, kBlockN, OutT, kStore, 0>(s, ma, mb, mo, mx, p, pl);
}

// The store path is a compile-time property of the kernel: each variant carries only its own epilogue code.  Deciding for
// the residual stream at run time inside the f32 TMA variant cost the others their registers: 1000 tokens x 768 -> 32000,
// f32 out, 41.0 -> 42.7 us.
template <int kBlockM, int kBlockN, typename OutT>
int launch_variant(cudaStream_t s, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo,
                   const CUtensorMap& mx, const GemmParams& p, const GemmPlan& pl) {
  if (!p.tma_store) return launch_store_variant<kBlockM, kBlockN, OutT, StorePath::kDirect>(s, ma, mb, mo, mx, p, pl);
  if constexpr (sizeof(OutT) == 4) {
    if (p.epilogue == NVFP4_EPI_RESIDUAL)
      return launch_store_variant<kBlockM, kBlockN, OutT, StorePath::kTmaResidual>(s, ma, mb, mo, mx, p, pl);
  }
  return launch_store_variant<kBlockM, kBlockN, OutT, StorePath::kTma>(s, ma, mb, mo, mx, p, pl);
}

std::atomic<int> g_tile_override{-1};  // -1 = read NVFP4_GEMM_TILE once, 0 = automatic, else (block_m << 16) | block_n
std::atomic<bool> g_allow_tall{true};  // the automatic choice may take the 256 x 192 tile
std::atomic<uint64_t> g_wait_timeout_ns{kDefaultWaitTimeoutNs};
std::atomic<uint32_t> g_debug_flags{0};
#ifdef NVFP4_GEMM_TRACE
std::atomic<unsigned long long*> g_trace_buffer{nullptr};
#endif
bool tile_shape_ok(int bm, int bn) {
  return (bm == 128 && (bn == 128 || bn == 192 || bn == 256)) || (bm == 256 && bn == 192);
}

int tile_override() {
  int v = g_tile_override.load(std::memory_order_relaxed);
  if (v < 0) {
    // NVFP4_GEMM_TILE = "<width>" (128-row tile) or "<height>x<width>"
    const char* env = std::getenv("NVFP4_GEMM_TILE");
    int bm = 128, bn = 0;
    if (env) {
      const char* x = std::strchr(env, 'x');
      if (x) {
        bm = std::atoi(env);
        bn = std::atoi(x + 1);
      } else {
        bn = std::atoi(env);
      }
    }
    v = tile_shape_ok(bm, bn) ? ((bm << 16) | bn) : 0;
    g_tile_override.store(v, std::memory_order_relaxed);
  }
  return v;
}

int validate_gemm(const nvfp4_gemm_args& a) {
  if (a.k == 0 || a.k % 64 != 0 || a.ldo < a.n) {
    set_last_error("nvfp4_gemm: k must be a non-zero multiple of 64 and ldo >= n");
    return static_cast<int>(cudaErrorInvalidValue);
  }
  if ((reinterpret_cast<uintptr_t>(a.a_bytes) | reinterpret_cast<uintptr_t>(a.b_bytes) |
       reinterpret_cast<uintptr_t>(a.a_scales) | reinterpret_cast<uintptr_t>(a.b_scales)) & 15u) {
    set_last_error("nvfp4_gemm: operand and scale pointers must be 16-byte aligned");
    return static_cast<int>(cudaErrorInvalidValue);
  }
  const bool has_bias = a.bias || (a.bias_nvfp4_bytes && a.bias_nvfp4_scales && a.bias_nvfp4_global);
  if (a.epilogue < NVFP4_EPI_NONE || a.epilogue > NVFP4_EPI_RESIDUAL || (a.epilogue != NVFP4_EPI_NONE && !has_bias) ||
      a.global_scale_mode < NVFP4_GS_NONE || a.global_scale_mode > NVFP4_GS_ROWWISE_A ||
      (a.global_scale_mode != NVFP4_GS_NONE && (!a.a_global || !a.b_global)) ||
      (a.out_dtype != NVFP4_DTYPE_F32 && a.out_dtype != NVFP4_DTYPE_BF16) || !a.out) {
    set_last_error("nvfp4_gemm: inconsistent epilogue / scale mode / dtype arguments");
    return static_cast<int>(cudaErrorInvalidValue);
  }
  return 0;
}

// Tile width, split-K count, shared-memory plan and grid of one GEMM on `sms` SMs.
// maps_refused: the output's tensor maps could not be encoded, direct stores it is.
void plan_gemm(const nvfp4_gemm_args& a, int sms, GemmPlan& pl, bool maps_refused = false) {
  const uint32_t k_atoms = a.k / 64;
  const uint32_t num_k_tiles = (k_atoms + kKAtomsPerStage - 1) / kKAtomsPerStage;
  const uint32_t usms = static_cast<uint32_t>(sms);
  const size_t esz = a.out_dtype == NVFP4_DTYPE_F32 ? 4 : 2;
  const uint32_t vec_elems = 16 / static_cast<uint32_t>(esz);
  pl.vec_store = ((reinterpret_cast<uintptr_t>(a.out) & 15u) == 0 && a.ldo % vec_elems == 0 &&
                  (!a.aux || (reinterpret_cast<uintptr_t>(a.aux) & 15u) == 0))
                     ? 1
                     : 0;
  // TMA-store epilogue whenever the output satisfies the tensor-map rules (16-byte aligned base
  // and row pitch); odd layouts use direct stores.  The f32 residual stream goes through the staging buffers as well, where
  // its lanes would read and write a row each: 4096 x 2048 x K 8192 100 us with direct stores, 54 us (36 on CTA pairs).  A TMA
  // reduction into the stream took 48 us where this took 54, but every f32 reduction in global memory takes subnormals for
  // zero.  A bf16 residual stays on the direct path, which adds in f32 and rounds once.
  pl.tma_store = (pl.vec_store && !maps_refused && (a.epilogue != NVFP4_EPI_RESIDUAL || a.out_dtype == NVFP4_DTYPE_F32)) ? 1 : 0;
  const bool can_split = a.out_dtype == NVFP4_DTYPE_F32 &&
                         (a.epilogue == NVFP4_EPI_NONE || a.epilogue == NVFP4_EPI_BIAS) && num_k_tiles >= 16;
  // The f32 residual stream is loaded into the staging buffers its sums leave from.  Two buffers per group (128 x 128)
  // keep a load in flight beside a store; one (the wider streaming tiles) has them take turns, which a main loop of up to eight
  // k-tiles does not hide: 65536 x 768 x K 1536 81 us at 128 x 128, 113 to 120 at the others; K 768, where the panels of up to
  // three k-tiles have two buffers as well, 79 against 77 to 80 (tall 111).  Beyond, the estimate carries what the turns add to
  // a tile (8192 x 768 x K 3072 20 us at 128 x 128, 21 at 128 x 192).
  const bool f32_residual = a.epilogue == NVFP4_EPI_RESIDUAL && a.out_dtype == NVFP4_DTYPE_F32;
  // CTA pairs for the main loops that are long enough, at 64 operand bytes per cycle and SM, to earn back what setting up and
  // tearing down a pair and the signals between its CTAs cost (about 1.5 us): 8192 x 1024 x K 32000 bf16 127 -> 102 us, 32000 x
  // 1024 x K 8192 f32 125 -> 110, 4096 x 2048 x K 8192 f32 residual 41 -> 36.4; 8192 x 1024 x K 4096 bf16 18.2 either way, 1024 x
  // 1024 x K 2048 (a split of 8192) f32 12.9 -> 14.2.  Not the tall tile: its two column sets for scale factors leave no slack
  // for those signals (8192 x 768 x K 32000 81 -> 85).  A pair per two SMs must need no more waves.
  auto pairs_of = [&](uint32_t splits) { return (a.m + 255u) / 256u * ((a.n + 255u) / 256u) * splits; };
  auto tiles_of = [&](uint32_t bm, uint32_t bn) { return ((a.m + bm - 1) / bm) * ((a.n + bn - 1) / bn); };
  auto pair_fits = [&](uint32_t bm, uint32_t bn, uint32_t splits, uint32_t k_tiles_per_split) {
    if (!pl.tma_store || bm != 128 || bn != 256 || k_tiles_per_split < 32 || usms % 2 != 0) return false;
    return (pairs_of(splits) + usms / 2 - 1) / (usms / 2) <= (tiles_of(bm, bn) * splits + usms - 1) / usms;
  };
  // Short K and many row blocks: keep the B panel resident and stream only A (halves the
  // operand traffic per tile; these shapes are otherwise bound by L2 -> SM bandwidth).
  // Four tiles a CTA, or three where the banded schedule leaves no CTA more than a tenth of its time without one: 8192 x 2304 x K
  // 768 bf16 (64 row blocks on 16 CTAs a column block) 12.6 -> 11.9 us, f32 18.3 -> 17.1, 4096 x 2304 8.8 -> 8.4.  Three anywhere:
  // 16384 x 768 10.9 -> 11.3.
  auto resident_shape = [&](uint32_t bm, uint32_t bn, uint32_t splits, uint32_t tiles) {
    if (bm != 128 || splits != 1 || num_k_tiles > (bn == 256 ? 3u : 4u) || tiles < 3 * usms) return false;
    if (tiles >= 4 * usms) return true;
    const uint32_t n_blocks = (a.n + bn - 1) / bn, m_blocks = (a.m + bm - 1) / bm, cpn = usms / n_blocks;
    return cpn * n_blocks * 20 >= usms * 19 && m_blocks >= 4 * cpn && (m_blocks + cpn - 1) / cpn * cpn * 10 <= m_blocks * 11;
  };
  // Waves and an estimated duration (SM cycles) of a candidate shape: per wave the k-tiles, at what their operand bytes or
  // MMAs take, and the part of the epilogue that no main loop hides; a split adds the clearing of the output and the
  // reduction.  The constants are a fit, in round figures, to the four tiles measured on 58 shapes (16 to 65536 rows, 512 to
  // 32000 columns, K 320 to 65536).  On 47 of them the tile taken was 8 % slower than the fastest one on average with the
  // constants from before tiles overlapped their epilogues (k-tiles 700, 980, 1150, 1360; epilogues 1500, 2000, 3500, 5000),
  // and is 2 % slower with these: 3072 x 768 x K 8192 f32 17.2 -> 14.2 us (128 x 128 in one wave, not three splits of 256 x
  // 192), 3072 x 1024 x K 8192 f32 26.3 -> 17.7, 4096 x 8192 x K 2048 f32 ReLU^2 with its second output 80 -> 61, 4096 x 4096 x
  // K 2048 bf16 24.5 -> 20.9, 2048 x 2304 x K 768 bf16 7.4 -> 6.0.  A pair's setting up and tearing down count once, not per
  // wave: 32000 x 768 x K 8192 f32 99 -> 93, where a split of 768 x 768 x K 65536 over pairs stays with the tall tile.  Direct
  // stores (odd pitches) take an SM 24 us for every 128 x 128 elements of bf16, 15 of f32, and half of that again for a second
  // output or the stream they add to, more in the tall tile, where no main loop runs beside them.  Weighed like the TMA stores' epilogue they put 696 x 3101 x K 8320 bf16 on the
  // tall tile (87 us, 49 at 128 x 128), 1024 x 2979 x K 1536 too (71 us, 52) and split 768 x 1685 x K 12736 f32 five ways (47
  // us, 31 unsplit).
  // Two outputs at 128 x 128 cost less than their first fit, at 4096 x 8192 x K 2048 alone, said (its buffers come in pairs): 8192 x
  // 4096 x K 1024 f32 62 -> 51 us, bf16 38.7 -> 31.7, 1000 x 4096 14.2 -> 9.6, 4096 x 3072 x K 768 bf16 16.9 -> 13.3.  The other
  // tiles' second outputs by the four tiles timed on 574 shapes (256 to 32768 rows, 256 to 16384 columns, K 256 to 8192, both types):
  // the tile taken is 0.7 % slower than the fastest on average, 1.1 % with 3500 and 7000, which put 8192 x 12288 x K 4096 f32 (349 us,
  // 289), 1024 x 12288 x K 8192 bf16 (60, 50) and 8192 x 16384 x K 3072 f32 (420, 351) on the tall tile; where it is the faster one by
  // less, 1371 x 13768 x K 3648 bf16 (46, 50 at 128 x 192), they lose.
  struct Candidate {
    uint32_t splits;
    uint64_t cost;
  };
  auto evaluate = [&](uint32_t bm, uint32_t bn) {
    const uint32_t tiles = tiles_of(bm, bn);
    const int shape = bm == 256 ? 3 : bn == 256 ? 2 : bn == 192 ? 1 : 0;
    constexpr uint64_t kTileCycles[4] = {550, 700, 850, 1050}, kResidentTileCycles = 300;
    constexpr uint64_t kPairTileCycles = 710, kPairF32Epilogue = 2000, kPairSetup = 6000;
    constexpr uint64_t kEpilogue[4] = {2000, 3000, 2500, 4000}, kF32Epilogue[4] = {4000, 3000, 6000, 6000};
    constexpr uint64_t kSecondOutput[4] = {0, 500, 3000, 9000}, kResidualTurns[4] = {0, 1000, 6000, 11000};
    constexpr uint64_t kDirectBf16[4] = {46000, 68000, 90000, 125000}, kDirectSecondBf16[4] = {26000, 42000, 57000, 92000};
    constexpr uint64_t kDirectF32[4] = {29000, 42000, 56000, 76000}, kDirectSecondF32[4] = {14000, 22000, 28000, 75000};
    constexpr uint64_t kDirectResidual[4] = {42000, 63000, 84000, 145000};
    constexpr uint64_t kSplitCycles = 4000;
    const bool f32_out = a.out_dtype == NVFP4_DTYPE_F32, second = a.epilogue == NVFP4_EPI_RELU2 && a.aux;
    const uint64_t direct = (f32_residual ? kDirectResidual : f32_out ? kDirectF32 : kDirectBf16)[shape] +
                            (second ? (f32_out ? kDirectSecondF32 : kDirectSecondBf16)[shape] : 0);
    const uint64_t staged = kEpilogue[shape] + (second ? kSecondOutput[shape] : 0) + (f32_residual ? kResidualTurns[shape] : 0);
    const uint64_t ce = pl.tma_store ? staged : direct;
    const bool two_outputs = second && pl.tma_store;
    Candidate best{1, ~0ull};
    uint32_t max_splits = 1;
    if (can_split && tiles < 2 * usms) {
      max_splits = num_k_tiles / 8;
      if (max_splits > 32) max_splits = 32;
      if (max_splits > 2 && gemm_get_deterministic()) max_splits = 2;
      if (max_splits < 1) max_splits = 1;
    }
    for (uint32_t sp = 1; sp <= max_splits; ++sp) {
      const uint32_t per = (num_k_tiles + sp - 1) / sp;
      const uint32_t real = (num_k_tiles + per - 1) / per;
      const bool pair = pair_fits(bm, bn, real, per);
      const uint32_t waves = pair ? (pairs_of(real) + usms / 2 - 1) / (usms / 2) : (tiles * real + usms - 1) / usms;
      const uint64_t ck = resident_shape(bm, bn, real, tiles) ? kResidentTileCycles : pair ? kPairTileCycles : kTileCycles[shape];
      const uint64_t cf = !f32_out || !pl.tma_store ? 0 : pair ? kPairF32Epilogue : two_outputs && shape == 0 ? 3000 : kF32Epilogue[shape];
      // however short the main loop is: two outputs of a 128 x 192 tile take turns with its stores (one staging buffer a group), those
      // of a 128 x 128 tile take their time to memory
      const uint64_t least = !two_outputs || shape > 1 ? 0 : shape == 1 ? (f32_out ? 11500 : 7300) : (f32_out ? 6500 : 4000);
      const uint64_t wave = per * ck + ce + cf;
      const uint64_t cost = waves * (wave > least ? wave : least) + (real > 1 ? kSplitCycles : 0) + (pair ? kPairSetup : 0);
      if (cost < best.cost) best = Candidate{real, cost};  // ties go to fewer splits
    }
    return best;
  };
  uint32_t block_m = 128, block_n = 128;
  Candidate best{1, ~0ull};
  const int forced = tile_override();
  if (forced) {
    block_m = static_cast<uint32_t>(forced) >> 16;
    block_n = static_cast<uint32_t>(forced) & 0xffffu;
  } else if (!f32_residual || num_k_tiles > 8) {
    const uint32_t tiles192 = tiles_of(128, 192), tiles256 = tiles_of(128, 256);
    // columns of the last 192-wide block that lie outside the matrix, as a share of all columns computed
    const uint32_t cols192 = (a.n + 191) / 192 * 192;
    const bool fits192 = (cols192 - a.n) * 16u <= cols192 && a.n >= 192;  // at most 1/16 wasted
    const bool ok192 = fits192 && (tiles192 >= usms || can_split);
    const bool wide_shape = a.n % 256 == 0 || a.n > 1024;
    const bool ok256 = wide_shape && ((num_k_tiles >= 4 && (tiles256 >= usms || can_split)) ||
                                      (a.n % 256 == 0 && resident_shape(128, 256, 1, tiles256)));
    auto consider = [&](uint32_t bm, uint32_t bn) {
      const Candidate c = evaluate(bm, bn);
      if (c.cost >= best.cost) return;
      best = c;
      block_m = bm;
      block_n = bn;
    };
    // Short K with a resident B panel is bound by writing the output, which the estimate does not see: the widest tile.
    const bool wide_resident = num_k_tiles <= 3 && ok192 && (ok256 || resident_shape(128, 192, 1, tiles192));
    if (wide_resident) {
      consider(128, ok256 ? 256 : 192);
    } else {
      if (ok192) consider(128, 192);
      if (ok256) consider(128, 256);
      // The narrow tile where its finer waves pay: six k-tiles and more that cannot be split go to the wide ones.
      if (can_split || num_k_tiles < 6 || (!ok192 && !ok256)) consider(128, 128);
    }
    // the tall tile: streamed long-K GEMMs only (its A stages leave no room for a resident panel, and short-K
    // GEMMs are bound by writing their output)
    if (fits192 && num_k_tiles >= 6 && g_allow_tall.load(std::memory_order_relaxed)) consider(256, 192);
  }
  pl.block_m = block_m;
  pl.block_n = block_n;
  pl.num_n_blocks = (a.n + block_n - 1) / block_n;
  const uint32_t num_m_blocks = (a.m + block_m - 1) / block_m;
  const uint32_t tiles = num_m_blocks * pl.num_n_blocks;

  // split-K for long GEMMs with few tiles (dW = dY^T.X): f32 output, linear epilogue only; the split count is
  // the one that minimises waves x (main loop + exposed epilogue) of one work item
  if (best.cost == ~0ull) best = evaluate(block_m, block_n);  // a tile that was not chosen by its cost
  pl.k_splits = best.splits;
  pl.k_tiles_per_split = (num_k_tiles + pl.k_splits - 1) / pl.k_splits;
  pl.k_splits = (num_k_tiles + pl.k_tiles_per_split - 1) / pl.k_tiles_per_split;

  const uint32_t work = tiles * pl.k_splits;
  pl.grid = work < usms ? work : usms;
  pl.b_resident = pl.panel = pl.resident_cpn = 0;
  auto stages_beside = [&](const TileBytes& tb, uint32_t slots) {
    return (kSmemBudget - tb.fixed - static_cast<int>(slots) * tb.slot) / tb.stage;
  };
  if (resident_shape(block_m, block_n, pl.k_splits, tiles)) {
    const uint32_t panel = panel_of(block_n, num_k_tiles);
    const int st = stages_beside(tile_bytes(block_m, block_n, panel, false), num_k_tiles);
    if (st >= 3) {
      pl.b_resident = 1;
      pl.panel = panel;
      pl.stages = static_cast<uint32_t>(st > kMaxStages ? kMaxStages : st);
      // banded schedule when the column blocks divide the grid almost evenly, or, for many row blocks, fill four fifths of it:
      // one A tile for all CTAs at a time and whole output rows are worth that many idle SMs (65536 x 32000 x K 768 on
      // 125 SMs 1003 us, contiguous on 148 1187; 8192 rows 112 and 114).  Direct stores of bf16 take an SM's time and not the
      // memory's: 28928 x 5695 x K 448 1774 us on all, 2193 on 132; 27392 x 6272 x K 960 residual 1177 and 1337; those of f32 gain
      // like TMA stores (31744 x 3759 x K 448 918 and 817)
      const uint32_t cpn = pl.grid / pl.num_n_blocks, used = cpn * pl.num_n_blocks;
      const bool most = (pl.tma_store || a.out_dtype == NVFP4_DTYPE_F32) && used * 5 >= pl.grid * 4 && num_m_blocks >= 16 * cpn;
      if (cpn >= 1 && ((used * 20 >= pl.grid * 19 && num_m_blocks >= 4 * cpn) || most)) pl.resident_cpn = cpn;
    }
  }
  pl.pair = !pl.b_resident && pair_fits(block_m, block_n, pl.k_splits, pl.k_tiles_per_split) ? 1 : 0;
  if (pl.pair) pl.grid = 2 * (pairs_of(pl.k_splits) < usms / 2 ? pairs_of(pl.k_splits) : usms / 2);
  const TileBytes tb = tile_bytes(block_m, block_n, pl.panel, pl.pair != 0);
  if (!pl.b_resident) {
    const int st = (kSmemBudget - tb.fixed) / (tb.stage + tb.slot);
    pl.stages = static_cast<uint32_t>(st > kMaxStages ? kMaxStages : st);
  }
  const uint32_t slots = pl.b_resident ? num_k_tiles : pl.stages;
  pl.smem_bytes = tb.fixed + static_cast<size_t>(pl.stages) * tb.stage + static_cast<size_t>(slots) * tb.slot;
}

}  // namespace

// Split-K sums its partial tiles with TMA reduce-add in arrival order: with two splits the sum is
// order-free (0 + a + b), with more it can differ in the last bits from run to run.  The switch below
// caps the split count at two for callers that need run-to-run identical dW.
static std::atomic<int> g_deterministic_splits{0};
void gemm_set_deterministic(int on) { g_deterministic_splits.store(on ? 1 : 0, std::memory_order_relaxed); }
int gemm_get_deterministic() { return g_deterministic_splits.load(std::memory_order_relaxed); }

#ifdef NVFP4_GEMM_TRACE
extern "C" void nvfp4_gemm_set_trace_buffer(unsigned long long* device_words) {
  g_trace_buffer.store(device_words, std::memory_order_relaxed);
}
#endif

int gemm_timing_begin(uint32_t max_records) {
  std::lock_guard<std::mutex> lock(g_timing.mu);
  while (g_timing.pool.size() < max_records) {
    GemmTimingRecord r;
    r.flops = 0;
    cudaError_t e = cudaEventCreate(&r.start);
    if (e == cudaSuccess) e = cudaEventCreate(&r.stop);
    if (e != cudaSuccess) return static_cast<int>(e);
    g_timing.pool.push_back(r);
  }
  g_timing.used = 0;
  g_timing.enabled = true;
  return 0;
}

int gemm_timing_end(uint32_t* count, double* total_ms, double* total_flops, float* per_launch_ms,
                    double* per_launch_flops, uint32_t capacity) {
  std::lock_guard<std::mutex> lock(g_timing.mu);
  g_timing.enabled = false;
  double ms_sum = 0, fl_sum = 0;
  for (size_t i = 0; i < g_timing.used; ++i) {
    float ms = 0;
    cudaError_t e = cudaEventSynchronize(g_timing.pool[i].stop);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, g_timing.pool[i].start, g_timing.pool[i].stop);
    if (e != cudaSuccess) return static_cast<int>(e);
    ms_sum += ms;
    fl_sum += g_timing.pool[i].flops;
    if (per_launch_ms && i < capacity) per_launch_ms[i] = ms;
    if (per_launch_flops && i < capacity) per_launch_flops[i] = g_timing.pool[i].flops;
  }
  if (count) *count = static_cast<uint32_t>(g_timing.used);
  if (total_ms) *total_ms = ms_sum;
  if (total_flops) *total_flops = fl_sum;
  g_timing.used = 0;
  return 0;
}

uint32_t* device_status_word() {
  uint32_t* ptr = nullptr;
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_device_status) != cudaSuccess) return nullptr;
  return ptr;
}

int gemm_plan_query(const nvfp4_gemm_args& a, nvfp4_gemm_plan* out, uint32_t* pair) {
  std::memset(out, 0, sizeof(*out));
  *pair = 0;
  if (a.m == 0 || a.n == 0) return 0;
  const int rc = validate_gemm(a);
  if (rc) return rc;
  GemmPlan pl;
  plan_gemm(a, sm_count(), pl);
  // launch_gemm plans again when an output map cannot be encoded; that has not been seen for outputs that pass the plan's
  // alignment test, so the query reports the test's verdict
  out->block_m = pl.block_m;
  out->block_n = pl.block_n;
  out->acc_stages = (pl.block_n == 256 || pl.block_m == 256) ? 1 : 2;
  out->k_splits = pl.k_splits;
  out->b_resident = pl.b_resident;
  out->resident_cpn = pl.resident_cpn;
  out->stages = pl.stages;
  out->grid = pl.grid;
  out->tma_store = pl.tma_store;
  out->smem_bytes = static_cast<uint32_t>(pl.smem_bytes);
  *pair = pl.pair;
  return 0;
}

void gemm_set_tile_override(int block_m, int block_n) {
  g_tile_override.store(tile_shape_ok(block_m, block_n) ? ((block_m << 16) | block_n) : 0, std::memory_order_relaxed);
}
void gemm_set_wait_timeout_ns(uint64_t ns) { g_wait_timeout_ns.store(ns ? ns : kDefaultWaitTimeoutNs, std::memory_order_relaxed); }
void gemm_set_debug_flags(uint32_t flags) { g_debug_flags.store(flags, std::memory_order_relaxed); }
void gemm_map_cache_stats(uint64_t* hits, uint64_t* misses) {
  if (hits) *hits = map_cache().hits;
  if (misses) *misses = map_cache().misses;
}

int gemm_prepare_operand_maps(const uint8_t* a_bytes, const uint8_t* b_bytes, uint32_t m, uint32_t k, uint32_t n) {
  if (k == 0 || k % 64 != 0) {
    set_last_error("prepare_tma: input_dim must be a non-zero multiple of 64");
    return static_cast<int>(cudaErrorInvalidValue);
  }
  CUtensorMap tmp;
  // operands are read with boxes as tall as the tile the launch will choose: encode every candidate
  int rc = 0;
  for (uint32_t box : {128u, 256u})
    if (!rc) rc = encode_operand_map(&tmp, a_bytes, m, k, box);
  for (uint32_t box : {128u, 192u, 256u})
    if (!rc) rc = encode_operand_map(&tmp, b_bytes, n, k, box);
  return rc;
}

bool gemm_adds_into_output(const nvfp4_gemm_args& a) {
  if (a.m == 0 || a.n == 0 || a.k == 0 || a.k % 64 != 0) return false;
  GemmPlan pl;
  plan_gemm(a, sm_count(), pl);
  return pl.k_splits > 1;
}

int launch_gemm(cudaStream_t s, const nvfp4_gemm_args& a, bool out_is_zero, bool row_amax_cleared, GemmNeighbour neighbour,
                GemmNeighbour* launched_as) {
  if (a.m == 0 || a.n == 0) return 0;
  int rc = validate_gemm(a);
  if (rc) return rc;
  const uint32_t debug_flags = g_debug_flags.load(std::memory_order_relaxed);
  GemmPlan pl;
  plan_gemm(a, sm_count(), pl);
  CUtensorMap ma, mb, mo, mx;
  // An output that passes the plan's test of its alignment has not been seen refused.  Should it be, the whole plan is made again:
  // pairs, for one, have no direct stores.
  if (pl.tma_store &&
      ((debug_flags & kDebugRefuseOutputMaps) || encode_output_map(&mo, a.out, a.out_dtype, a.m, a.n, a.ldo) != 0 ||
       (a.aux && encode_output_map(&mx, a.aux, a.out_dtype, a.m, a.n, a.ldo) != 0)))
    plan_gemm(a, sm_count(), pl, true);
  if (a.relu2_row_amax && (!pl.tma_store || a.epilogue == NVFP4_EPI_RESIDUAL)) {
    set_last_error("nvfp4_gemm: relu2_row_amax needs a 16-byte aligned output and row pitch and no residual epilogue");
    return static_cast<int>(cudaErrorInvalidValue);
  }

  GemmParams p;
  p.sfa = a.a_scales;
  p.sfb = a.b_scales;
  p.a_global = a.a_global;
  p.b_global = a.b_global;
  p.bias = a.bias;
  p.bias_bytes = a.bias_nvfp4_bytes;
  p.bias_scales = a.bias_nvfp4_scales;
  p.bias_global = a.bias_nvfp4_global;
  p.row_amax = a.relu2_row_amax;
  p.out = a.out;
  p.aux = a.aux;
  p.m = a.m;
  p.n = a.n;
  p.k = a.k;
  p.ldo = a.ldo;
  p.mode = a.global_scale_mode;
  p.epilogue = a.epilogue;
  p.weight = a.weight_global_scale;
  p.k_atoms = a.k / 64;
  p.num_k_tiles = (p.k_atoms + kKAtomsPerStage - 1) / kKAtomsPerStage;
  const uint32_t tile_rows = pl.pair ? 2 * pl.block_m : pl.block_m;
  p.num_m_blocks = (a.m + tile_rows - 1) / tile_rows;
  p.num_n_blocks = pl.num_n_blocks;
  p.sfa_blocks128 = (a.m + 127) / 128;
  p.sfb_blocks128 = (a.n + 127) / 128;
  p.k_splits = pl.k_splits;
  p.k_tiles_per_split = pl.k_tiles_per_split;
  p.stages = pl.stages;
  p.resident_cpn = pl.resident_cpn;
  p.vec_store = static_cast<int>(pl.vec_store);
  p.tma_store = static_cast<int>(pl.tma_store);
  // An output that L2 (126 MB) does not hold leaves it first, so that the operands stay: the contiguous schedule, whose CTAs
  // are all over the matrix, 1000 x 32000 x K 768 f32 36 -> 30 us, 8192 x 32000 x K 1024 bf16 150 -> 145.  Not the banded
  // one: its rows are completed by several CTAs before they should leave (65536 x 2304 x K 768 65 -> 77 us).
  p.stream_out = pl.b_resident && pl.resident_cpn == 0 &&
                 static_cast<uint64_t>(a.m) * a.ldo * (a.out_dtype == NVFP4_DTYPE_F32 ? 4 : 2) > (96ull << 20);
  p.wait_timeout_ns = g_wait_timeout_ns.load(std::memory_order_relaxed);
  p.debug_flags = debug_flags;
#ifdef NVFP4_GEMM_TRACE
  p.trace = g_trace_buffer.load(std::memory_order_relaxed);
#endif

  rc = encode_operand_map(&ma, a.a_bytes, a.m, a.k, pl.block_m);
  if (rc) return rc;
  rc = encode_operand_map(&mb, a.b_bytes, a.n, a.k, pl.pair ? pl.block_n / 2 : pl.block_n);
  if (rc) return rc;
  if (!pl.tma_store) mo = ma;
  if (!pl.tma_store || !a.aux) mx = ma;

  const size_t esz = a.out_dtype == NVFP4_DTYPE_F32 ? 4 : 2;
  if (p.k_splits > 1 && !out_is_zero) {
    cudaError_t e = cudaMemset2DAsync(a.out, static_cast<size_t>(a.ldo) * esz, 0, static_cast<size_t>(a.n) * esz, a.m, s);
    if (e != cudaSuccess) return static_cast<int>(e);
    // not directly behind the other GEMM; one that lets its follower start has waited for the clearing by then
    if (neighbour == GemmNeighbour::kBesidePrior) neighbour = GemmNeighbour::kNone;
  }
  if (neighbour == GemmNeighbour::kBesidePrior && !pl.tma_store) neighbour = GemmNeighbour::kNone;  // no such form
  if (g_timing.enabled) neighbour = GemmNeighbour::kNone;  // events between the launches
  p.lets_next_beside = neighbour == GemmNeighbour::kLetsNextBeside ? 1u : 0u;
  pl.beside = neighbour == GemmNeighbour::kBesidePrior;
  if (launched_as) *launched_as = neighbour;
  if (a.relu2_row_amax && !row_amax_cleared) {
    cudaError_t e = cudaMemsetAsync(a.relu2_row_amax, 0, static_cast<size_t>(a.m) * sizeof(float), s);
    if (e != cudaSuccess) return static_cast<int>(e);
  }

  const bool f32 = a.out_dtype == NVFP4_DTYPE_F32;
  if (pl.block_m == 256)
    return f32 ? launch_variant<256, 192, float>(s, ma, mb, mo, mx, p, pl)
               : launch_variant<256, 192, __nv_bfloat16>(s, ma, mb, mo, mx, p, pl);
  switch (pl.block_n) {
    case 256:
      return f32 ? launch_variant<128, 256, float>(s, ma, mb, mo, mx, p, pl)
                 : launch_variant<128, 256, __nv_bfloat16>(s, ma, mb, mo, mx, p, pl);
    case 192:
      return f32 ? launch_variant<128, 192, float>(s, ma, mb, mo, mx, p, pl)
                 : launch_variant<128, 192, __nv_bfloat16>(s, ma, mb, mo, mx, p, pl);
    default:
      return f32 ? launch_variant<128, 128, float>(s, ma, mb, mo, mx, p, pl)
                 : launch_variant<128, 128, __nv_bfloat16>(s, ma, mb, mo, mx, p, pl);
  }
}

}  // namespace nvfp4
