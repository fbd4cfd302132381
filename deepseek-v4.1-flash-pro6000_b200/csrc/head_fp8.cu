// FP8 LM head for sm_100a: logits[m, n] = sum over 128-wide K blocks of a_scale[m, kb] * w_scale[n/128, kb] *
// dot(a_e4m3[m, kb], w_e4m3[n, kb]).
//
// The reference's head is a BF16 GEMV (components/fuse-head/src/head_half_tune.cu:7-21) and its only FP8 GEMM is
// ds41_dense_fp8 for the dense projections (components/dense/src/dense.cu:25-91, UE8M0 scales per 32x32 block).
// This operator is new: e4m3 weights with one fp32 scale per 128x128 block, activations quantised per (row, 128-K
// group) by the reference's power-of-two rule (dense.cu:8-16) widened to the weight block.  It keeps the plugin
// conventions of fuse_head.h:8 (caller-owned buffers, stream-ordered, no allocation, no synchronisation).
//
// Three kernels, all persistent: a warp streams W and A tiles with TMA (128-byte swizzle) into a ring of shared-memory stages, one
// issues four K=32 tcgen05.mma per 128-wide K block, the others pull each finished K block out of TMEM (tcgen05.ld), hand its
// accumulator back at once, scale and add in fp32 registers.
// * head_fp8_decode_kernel, up to 64 rows: 128 vocabulary ids are the M dimension (TMEM lanes), the 16, 32 or 64 batch rows N.  M is
//   always 128, so this way an MMA reads and multiplies no row that is not there, and a K block takes the tensor core 160 to 192
//   cycles instead of 256 (and beside the copies' writes to the same shared memory about 450, which made it the bound: weights
//   arrive every 700).  A hand-over costs the issuing warp another 100, so that one covers a whole stage of two or four K blocks.
//   A lane holds one id for all batch rows: a store writes 128 consecutive bytes of a row as it is.  The activation scale is another
//   one for each column; its product with the weight scale is exact (a power of two), the sums are those of the other kernels.
//   Eight epilogue warps: sixteen leave 96 registers, too few to have all columns of a stage in flight.
// * head_fp8_kernel, 65 to 128 rows: the batch rows are the M dimension, 128 ids N: the combined scale
//   a_scale[m,kb] * w_scale[n/128,kb] of a K block is ONE number per epilogue thread.  (The decode kernel with N = 128 takes 127 to 139
//   us here instead of 106 to 120: eight warps with 64 columns each, or sixteen without the registers.)
// * head_fp8_pair_kernel, more rows: the same with a pair of SMs on 256 batch rows x 256 ids (cta_group::2).  Each CTA fetches its own
//   128 rows of A and half of the ids' rows, 32 KB a K block instead of the 48 KB of a 128 x 256 tile alone, which alone took 404 of
//   652 us at 1024 rows.  Both CTAs' copies count on the leading CTA's barriers, its one warp issues, and the epilogues of both
//   hand accumulators back to it.
// What bounds it (129280 x 4096, us with quantisation and launch; before: with head_fp8_kernel for every size, 128 x 256 tiles from 129
// rows on): up to 64 rows the weights' 530 MB and the logits (81 to 86 at the measured copy rate): 1 row 78 (88 before), 16 rows
// 80 (92), 32 rows 83 (95), 64 rows 90 (102); with the row records 79, 81, 84 and 98 (90, 95, 97, 105).  From 65 rows on the epilogue
// (106 at 65 rows, 120 at 128): beside the MMAs' operands and the copies, which fill the shared memory's bandwidth, every access of the
// epilogue to it, waits and scales included, takes 100 to 230 cycles.  Run without pause, as in a decode loop, the power cap (about
// 1.6 GHz) counts as much: 256 rows 168 to 200 (198 to 222 before), 512 rows 342 to 361 (403), 1024 rows 689 to 707 (764 to 778); with the
// row records 713 to 735 (801 to 810).  The issuing warp waits as a whole and elects the lane that issues (108 to 104 at 64 rows
// against one lane on its own path).
// Every wait is bounded; on expiry the kernel raises *error_flag, frees its TMEM and returns.
#include "ds41_b200.h"
#include "cluster.cuh"
#include "flat.cuh"
#include "host_error.h"
#include "launch.h"
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdlib.h>

namespace ds41 {
namespace {

constexpr int kTmemColumns = 512;  // all of an SM's tensor memory: 4 accumulators of 128 columns or 2 of 256
constexpr int kTileK = 128;   // K elements per block = one 128-byte swizzle row of e4m3
constexpr int kEpiWarps = 16, kHeadThreads = 64 + 32 * kEpiWarps, kPairThreads = 128 + 32 * kEpiWarps;
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return shared_addr(p); }

struct Abort {  // shared flag: once set every later wait returns immediately
  volatile int *flag;
  __device__ __forceinline__ bool set() const { return *flag != 0; }
};

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Bounded wait on a phase parity.  Returns false (and raises the abort flag) if the phase never completed.  The first
// probe carries no other work: the single threads that issue the copies and the MMAs call this once or twice per K
// block, and every instruction on their path delays the tensor pipe.
// kCluster: what completes the phase are relaxed arrivals of another CTA (mbar_arrive_leader), so the wait has the cluster for its scope as
// they have; as there, the order of the tensor memory's accesses comes from the tcgen05 fences on both sides.
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_try(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  if constexpr (kCluster)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
  return done != 0;
}
// (In line: around a call the 64 sums of an epilogue thread would be spilled.)
template <bool kCluster = false>
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, const Abort &ab) {
  if (mbar_try<kCluster>(bar, parity)) return true;
#pragma unroll 1
  for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
    if (mbar_try<kCluster>(bar, parity)) return true;
    if ((spin & 255u) == 255u && ab.set()) return false;
  }
  *ab.flag = 1;
  return false;
}

// Box {128 bytes, rows, K blocks} of the operand seen as [K/128][rows][128 bytes] (see make_map).
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int row, int kb) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
          "r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(row), "r"(kb)
      : "memory");
}

// The same with an L2 eviction policy.
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int row, int kb, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], "
      "[%2], %6;" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(x), "r"(row), "r"(kb), "l"(policy)
      : "memory");
}

// The same box into the L2 only.
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap *map, int x, int row, int kb, uint64_t policy) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile.L2::cache_hint [%0, {%1, %2, %3}], %4;" ::
                   "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(row), "r"(kb), "l"(policy)
               : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: rows are 128 bytes apart, groups of 8 rows 1024 bytes
// apart (stride byte offset), leading byte offset unused (1), descriptor version 1 for sm_100.
constexpr uint64_t kDescFixed = (uint64_t(1) << 16)              // leading byte offset (>>4), bits [16,30)
                                | (uint64_t(1024 >> 4) << 32)    // stride byte offset (>>4), bits [32,46)
                                | (uint64_t(1) << 46)            // version, bits [46,48)
                                | (uint64_t(2) << 61);           // layout type SWIZZLE_128B, bits [61,64)
// addr16 = shared-memory byte address >> 4 (start address field, bits [0,14); shared memory ends below 2^18 bytes)
__device__ __forceinline__ uint64_t umma_desc16(uint32_t addr16) { return kDescFixed | uint64_t(addr16); }
// Instruction descriptor for kind::f8f6f4, E4M3 x E4M3 -> F32, both operands K-major, M=128, N=n_cols.
__host__ __device__ constexpr uint32_t umma_idesc(int n_cols) {
  return (1u << 4) | (uint32_t(n_cols >> 3) << 17) | (uint32_t(128 >> 4) << 24);
}
template <bool kAccumulate>
__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
// true in one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(one));
  return one != 0;
}
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Four bytes from global to shared memory without a register; copies_done() waits for all of the thread's.
__device__ __forceinline__ void copy4_async(float *to, const float *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(to)), "l"(__cvta_generic_to_global(from)) : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

// Two fp32 fused multiply-adds in one instruction (fma.rn.f32x2: each half is the same correctly rounded FMA as
// fmaf): the promotion of a K block is 32 or 64 of them per thread, and the epilogue warps' issue slots are what the
// tensor pipe ends up waiting for.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void fma2_acc(float &s0, float &s1, uint32_t d0, uint32_t d1, unsigned long long scale2) {
  unsigned long long d, c, out;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(d0), "r"(d1));
  asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(s0), "f"(s1));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out) : "l"(d), "l"(scale2), "l"(c));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(s0), "=f"(s1) : "l"(out));
}

__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}

// ---- a pair of CTAs (a cluster of two) on one tile
// An accumulator is handed back to the leading CTA.  Relaxed is enough because nothing is published: the arrival only keeps the next MMA from
// overwriting what has been read, and it is issued once tcgen05.wait::ld has returned the values in every lane (__syncwarp), with a
// tcgen05 fence on either side.  So nothing else may be handed over by this barrier.
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Into this CTA's shared memory; the bytes are counted by a barrier of the leading CTA.
__device__ __forceinline__ void tma_load_pair(void *dst, const CUtensorMap *map, uint32_t leader_bar, int x, int row, int kb, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint [%0], "
      "[%1, {%3, %4, %5}], [%2], %6;" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(x), "r"(row), "r"(kb), "l"(policy)
      : "memory");
}
// Instruction descriptor as umma_idesc, M = 256: 128 rows of A from each CTA, 128 of the 256 rows of B from each.
constexpr uint32_t kPairIdesc = (1u << 4) | (uint32_t(256 >> 3) << 17) | (uint32_t(256 >> 4) << 24);
template <bool kAccumulate>
__device__ __forceinline__ void umma_f8_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(a_desc), "l"(b_desc), "r"(kPairIdesc), "n"(kAccumulate ? 1 : 0)
      : "memory");
}
// Arrives at both CTAs' copies of the barrier.
__device__ __forceinline__ void umma_commit_pair(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_addr(bar)),
               "h"(uint16_t(3))
               : "memory");
}

// 128 batch rows of each CTA of a pair x 256 vocabulary ids.  A stage is one K block: 128 rows of activations and 128 of the ids' rows.
struct PairSmem {
  static constexpr int kAccBufs = 2;
  static constexpr int kStageBytes = 2 * 128 * kTileK, kStages = 5;
  static constexpr int kOutFloats = 32 * 16;   // an epilogue warp's 32 rows x 16 ids on their way out
  // bytes beside the stages: alignment slack, output blocks, statistics, scale tables [K/128][128] and [warps][2][K/128], barriers and flags
  static constexpr size_t fixed_bytes(int kblocks) {
    return 1024 + kEpiWarps * (kOutFloats * 4 + 32 * 16) + size_t(kblocks) * (128 + 2 * kEpiWarps) * 4 + (2 * kStages + 2 * kAccBufs) * 8 + 16;
  }
  static constexpr int stages(int kblocks) {
    const long long room = 227 * 1024 - (long long)fixed_bytes(kblocks);
    const int n = room < 0 ? 0 : int(room / kStageBytes);
    return n > kStages ? kStages : n;
  }
};

// 128 batch rows x 128 vocabulary ids
struct HeadSmem {
  static constexpr int kAccBufs = kTmemColumns / 128;
  static constexpr int kStageBytes = 2 * 128 * kTileK;
  static constexpr int kMaxStages = 12;
  // bytes beside the stages: alignment slack, scale tables [K/128][128] and [warps][K/128], barriers and flags
  static constexpr size_t fixed_bytes(int kblocks) {
    return 1024 + size_t(kblocks) * (128 + kEpiWarps) * 4 + (2 * kMaxStages + 2 * kAccBufs) * 8 + 16;
  }
  // a stage holds `group` consecutive K blocks (one TMA box per operand)
  static constexpr int stages(int kblocks, int group) {
    const long long room = 227 * 1024 - (long long)fixed_bytes(kblocks);
    const int n = room < 0 ? 0 : int(room / (kStageBytes * group));
    return n > kMaxStages ? kMaxStages : n;
  }
};

constexpr int kMaxOwners = 8;
struct HeadArgs {
  const float *a_scale;  // [M, K/128]
  const float *w_scale;  // [ceil(N/128), K/128]
  float *logits;         // [M, ldl]
  long long ldl;
  int M, N, K;
  int *error_flag;       // device word, raised on a wait timeout (may be null)
  // Row-scattered output (vocabulary-sharded head): batch row m, the call's row g = first_row + m, goes to owner g / rows_per_owner, into
  // owner_base[owner] + (g % rows_per_owner) * ldl + col_offset + n.  The bases may be peer GPUs' memory; the epilogue
  // writes them with plain stores, so the vocabulary-to-row transposition rides on the GEMM.  rows_per_owner == 0: off.
  float *owner_base[kMaxOwners];
  int rows_per_owner, col_offset;
  int first_row;         // rows of the call in front of this launch's (a call may take two, see run_head)
  // Optional per-row statistics for the sampler (zero-initialised by the host): every epilogue thread keeps the first
  // maximum, the minimum and a finiteness flag of the logits it produces for its batch row and merges them with atomic
  // maxima when it leaves the row, so the sampler's own pass over the logits for these three numbers can be skipped.
  HeadRowStats *row_stats;
  // The same records in the row-scattered variant: row m's record lies owner_stats_offset bytes behind owner_base[owner]
  // at index (first_row + m) % rows_per_owner (0: none).  Several GPUs merge into one record, so those atomics have system scope.
  long long owner_stats_offset;
  int stages;            // shared-memory stages of the TMA ring (host: stages() of the kernel's own layout)
  int group;             // K blocks per stage: every row of a weight tile is fetched as group*128 contiguous bytes
};

// Merges a thread's statistics of batch row m into the row's record.  id 0x7fffffff: no maximum (only NaN and -inf seen).
__device__ __forceinline__ void merge_stats(const HeadArgs &p, int m, float best, int id, float low, bool bad) {
  auto ordered = [](float v) {
    const uint32_t bits = __float_as_uint(v == 0.f ? 0.f : v);  // -0 and +0 are the same logit
    return bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u);
  };
  const unsigned long long key = (unsigned long long)(ordered(best)) << 32 | (0xffffffffu - uint32_t(id + p.col_offset));
  const bool any = id != 0x7fffffff;
  if (p.owner_stats_offset) {
    const int g = p.first_row + m, owner = g / p.rows_per_owner;
    HeadRowStats *rs = reinterpret_cast<HeadRowStats *>(reinterpret_cast<unsigned char *>(p.owner_base[owner]) +
                                                        p.owner_stats_offset) + (g - owner * p.rows_per_owner);
    if (any) {
      atomicMax_system(&rs->max_key, key);
      atomicMax_system(&rs->min_key, ~ordered(low));
    }
    if (bad) atomicOr_system(&rs->flags, 1u);
  } else {
    HeadRowStats *rs = p.row_stats + m;
    if (any) {
      atomicMax(&rs->max_key, key);
      atomicMax(&rs->min_key, ~ordered(low));
    }
    if (bad) atomicOr(&rs->flags, 1u);
  }
}

// 65 to 128 rows: 128 batch rows x 128 vocabulary ids a tile.
__global__ void __launch_bounds__(kHeadThreads, 1)
head_fp8_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ HeadArgs p) {
  using Smem = HeadSmem;
  constexpr int kRows = 128, kTileN = 128, kAccBufs = Smem::kAccBufs;
  constexpr int kStageBytes = Smem::kStageBytes;
  constexpr int kMaxStages = Smem::kMaxStages;
  const int kStages = p.stages, group = p.group;
  const int stage_bytes = kStageBytes * group, a_bytes = kRows * kTileK * group;  // [A g0..][W g0..]
  constexpr int kMyCols = 32, kEpiThreads = 32 * kEpiWarps;   // epilogue warp = (lane quadrant, group of 32 columns)
  extern __shared__ __align__(1024) unsigned char smem[];
  // carve: [stages][A tiles 16 KB | W tiles 16 KB], then the scale tables, then barriers
  unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
  float *sa = reinterpret_cast<float *>(tiles + size_t(kStages) * stage_bytes);  // [K/128][kRows]
  const int kblocks = p.K / kTileK;
  float *sw = sa + size_t(kblocks) * kRows;                                                              // [epilogue warp][K/128]
  uint64_t *bars = reinterpret_cast<uint64_t *>(sw + size_t(kblocks) * kEpiWarps);
  uint64_t *full = bars, *empty = bars + kMaxStages, *acc_full = bars + 2 * kMaxStages, *acc_empty = acc_full + kAccBufs;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + kAccBufs);
  int *abort_word = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_tiles = (p.N + kTileN - 1) / kTileN;
  Abort ab{abort_word};

  if (threadIdx.x == 0) {
    *abort_word = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < kAccBufs; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], kEpiWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // TMEM allocation by one full warp; the address lands in shared memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(uint32_t(kTmemColumns)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      // every weight is read once per step, and 530 MB of them would push everything else out of the L2 -- the logits, the
      // activations, the code of the kernels around this one
      uint64_t policy;
      asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
      // the ring's first weights are on their way to the L2 while the kernel in front of this one (the quantiser) finishes
      const int early = kblocks / group < kStages ? kblocks / group : kStages;
      for (int s = 0; s < early; ++s) tma_prefetch_3d(&map_w, 0, int(blockIdx.x) * kTileN, s * group, policy);
      cudaGridDependencySynchronize();
      cudaTriggerProgrammaticLaunchCompletion();
      for (int tile = blockIdx.x; tile < total_tiles && !ab.set(); tile += gridDim.x) {
        for (int kb = 0; kb < kblocks; kb += group) {
          if (!mbar_wait(&empty[stage], phase ^ 1, ab)) break;
          unsigned char *a_dst = tiles + size_t(stage) * stage_bytes, *w_dst = a_dst + a_bytes;
          mbar_expect_tx(&full[stage], uint32_t(stage_bytes));
          tma_load_3d(w_dst, &map_w, &full[stage], 0, tile * kTileN, kb, policy);
          tma_load_3d(a_dst, &map_a, &full[stage], 0, 0, kb);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer: the warp waits together, one lane issues
    cudaGridDependencySynchronize();
    constexpr uint32_t idesc = umma_idesc(kTileN);
    const uint32_t tiles16 = smem_addr(tiles) >> 4, stage16 = uint32_t(stage_bytes) >> 4;
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
    for (int tile = blockIdx.x; tile < total_tiles && !__any_sync(0xffffffffu, ab.set()); tile += gridDim.x) {
      bool ok = true;
      for (int kb = 0; kb < kblocks && ok; kb += group) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, ab))) break;
        uint32_t a16 = tiles16 + stage * stage16, w16 = a16 + (a_bytes >> 4);  // addresses >> 4
        for (int g = 0; g < group; ++g) {
          ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[acc], acc_phase ^ 1, ab));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t d_addr = tmem_base + acc * kTileN;
          if (leader) {
            // D[batch row, vocabulary id] (+)= A[batch row, k] * W[vocabulary id, k], K = 32 bytes per instruction
            umma_f8<false>(d_addr, umma_desc16(a16), umma_desc16(w16), idesc);
            umma_f8<true>(d_addr, umma_desc16(a16 + 2), umma_desc16(w16 + 2), idesc);
            umma_f8<true>(d_addr, umma_desc16(a16 + 4), umma_desc16(w16 + 4), idesc);
            umma_f8<true>(d_addr, umma_desc16(a16 + 6), umma_desc16(w16 + 6), idesc);
            umma_commit(&acc_full[acc]);   // accumulator of this K block is complete
            if (g + 1 == group) umma_commit(&empty[stage]);  // the stage may be refilled once these MMAs have read it
          }
          __syncwarp();
          if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
          w16 += (kTileN * kTileK) >> 4; a16 += (kRows * kTileK) >> 4;
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue: warp = (lane quadrant, column group)
    cudaGridDependencySynchronize();
    const int quad = warp & 3;          // TMEM lanes [32*quad, 32*quad+32) are readable by this warp: batch rows
    const int group = (warp - 2) >> 2;  // vocabulary ids [32*group, 32*group+32) of the tile
    const int row = quad * 32 + lane;   // batch row inside the tile
    const int et = threadIdx.x - 64;
    const uint32_t lane_base = tmem_base + group * kMyCols + (uint32_t(quad * 32) << 16);
    float *my_sw = sw + size_t(warp - 2) * kblocks;
    uint32_t acc = 0, acc_phase = 0;
    bool alive = true;  // warp-uniform
    // running statistics of this thread's batch row over its tiles (vocabulary tiles come in ascending
    // order, so a strict comparison keeps the first maximum).  The column is looked for only in a tile
    // that raises the maximum of one of the warp's rows.  (Looking it up in the logits when the row is left took 10 us at 128
    // rows and 28 at 256: the reads stand behind everything that the GPU has just written.)
    float st_best = -CUDART_INF_F, st_low = CUDART_INF_F, st_bad = 0.f, st_bad1 = 0.f;
    int st_id = 0x7fffffff;
    const bool stats_on = p.row_stats != nullptr || p.owner_stats_offset != 0;
    auto row_of = [&](int m) {   // batch row m of the output
      if (p.rows_per_owner == 0) return p.logits + size_t(m) * p.ldl;
      const int g = p.first_row + m, owner = g / p.rows_per_owner;
      return p.owner_base[owner] + size_t(g - owner * p.rows_per_owner) * p.ldl + p.col_offset;
    };
    for (int i = et; i < kblocks * kRows; i += kEpiThreads) {   // activation scales: sa[kb][row]
      const int r = i / kblocks, kb = i % kblocks;
      sa[kb * kRows + r] = r < p.M ? load_input(p.a_scale + size_t(r) * kblocks + kb) : 0.f;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
    for (int tile = blockIdx.x; tile < total_tiles && alive; tile += gridDim.x) {
      // fp32 scales of the tile's weight block, copied once per tile: a global load in the loop below, even one that hits, delays the
      // hand-over of each accumulator.  (Fetched a tile ahead, as the other two kernels do: 107.5 us at 65 rows instead of 106.5.)
      for (int i = lane; i < kblocks; i += 32) my_sw[i] = load_input(p.w_scale + size_t(tile) * kblocks + i);
      __syncwarp();
      float sum[kMyCols];
#pragma unroll
      for (int c = 0; c < kMyCols; ++c) sum[c] = 0.f;
      for (int kb = 0; kb < kblocks && alive; ++kb) {
        alive = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_phase, ab));
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const float scale = sa[kb * kRows + row] * my_sw[kb];
        const unsigned long long scale2 = pack2(scale, scale);
        uint32_t r[32];
        tmem_ld32(lane_base + acc * kTileN, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // the values are in registers: the accumulator can be refilled while they are scaled and added
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
#pragma unroll
        for (int c = 0; c < 32; c += 2) fma2_acc(sum[c], sum[c + 1], r[c], r[c + 1], scale2);
        if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
      }
      // Output, while the tensor cores wait: as few instructions as it takes.
      const int n0 = tile * kTileN + group * kMyCols;
      const bool whole = n0 + kMyCols <= p.N;
      if (alive && stats_on) {
        if (whole) {
          const unsigned long long zero2 = pack2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < kMyCols; c += 2)   // NaN once any logit is NaN or infinite
            fma2_acc(st_bad, st_bad1, __float_as_uint(sum[c]), __float_as_uint(sum[c + 1]), zero2);
          float hi = sum[0], low = sum[0];
#pragma unroll
          for (int c = 1; c < kMyCols; ++c) { hi = fmaxf(hi, sum[c]); low = fminf(low, sum[c]); }
          if (__any_sync(0xffffffffu, hi > st_best)) {
            int at = 0;
#pragma unroll
            for (int c = kMyCols - 1; c > 0; --c) at = sum[c] == hi ? c : at;
            if (sum[0] == hi) at = 0;
            if (hi > st_best) { st_best = hi; st_id = n0 + at; }
          }
          st_low = fminf(st_low, low);
        } else {
#pragma unroll
          for (int c = 0; c < kMyCols; ++c) {
            const float v = sum[c];
            if (n0 + c < p.N) {
              st_bad = fmaf(v, 0.f, st_bad);
              if (v > st_best) { st_best = v; st_id = n0 + c; }
              st_low = fminf(st_low, v);
            }
          }
        }
      }
      // Lane l holds row l of the warp's 32 x 32 block.  Written as it is, one store instruction would touch 32 rows with 16
      // bytes each; butterflies of the 16-byte column groups at lane distances 8, 16 and 4 turn that into 4 rows with 128
      // contiguous bytes, which the local L2 and a peer GPU's memory both want (without the third one, 8 rows of 64 bytes:
      // 122 us against 119 at 128 rows).
      if (alive) {
        const bool scattered = p.rows_per_owner != 0;
        const bool plain = !scattered && whole && p.ldl % 4 == 0 && (reinterpret_cast<uintptr_t>(p.logits) & 15u) == 0;
        float4 x[8];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          x[c] = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
        auto exchange = [&](int bit, int dist) {   // column group bit of the index <-> the lane bit of that distance
          const bool upper = (lane & dist) != 0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if ((c >> bit) & 1) continue;
            const int c2 = c | (1 << bit);
            const float4 give = upper ? x[c] : x[c2];
            float4 take;
            take.x = __shfl_xor_sync(0xffffffffu, give.x, dist);
            take.y = __shfl_xor_sync(0xffffffffu, give.y, dist);
            take.z = __shfl_xor_sync(0xffffffffu, give.z, dist);
            take.w = __shfl_xor_sync(0xffffffffu, give.w, dist);
            if (upper) x[c] = take; else x[c2] = take;
          }
        };
        exchange(0, 8);
        exchange(1, 16);
        exchange(2, 4);
        // x[c] = columns [4 * (lane / 8) + 16 * (lane / 4 % 2), +4) of block row 8 * (c % 4) + 4 * (c / 4) + lane % 4
        if (plain) {
          const int r = quad * 32 + (lane & 3), rows = p.M - r;
          float *dst = p.logits + size_t(r) * p.ldl + n0 + 4 * (lane >> 3) + 16 * ((lane >> 2) & 1);
          const long long step = 4 * p.ldl;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            if (4 * c < rows) *reinterpret_cast<float4 *>(dst) = x[(c >> 1) | ((c & 1) << 2)];
            dst += step;
          }
        } else {
          const int n = n0 + 4 * (lane >> 3) + 16 * ((lane >> 2) & 1);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int m = quad * 32 + 8 * (c & 3) + 4 * (c >> 2) + (lane & 3);
            if (m >= p.M || n >= p.N) continue;
            float *dst = row_of(m) + n;
            if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
              *reinterpret_cast<float4 *>(dst) = x[c];
            } else {
              const float v[4] = {x[c].x, x[c].y, x[c].z, x[c].w};
#pragma unroll
              for (int k = 0; k < 4; ++k)
                if (n + k < p.N) dst[k] = v[k];
            }
          }
        }
      }
    }
    if (alive && stats_on && row < p.M) merge_stats(p, row, st_best, st_id, st_low, st_bad + st_bad1 != 0.f);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemColumns)));
  }
  if (threadIdx.x == 0 && *abort_word && p.error_flag) atomicExch(p.error_flag, 1);
}

// Larger batches: pairs of CTAs, 256 batch rows x 256 vocabulary ids a tile.  An epilogue thread keeps 64 sums, so every register
// counts: 112 each (the warps beside them give theirs up), statistics in shared memory between the tiles (737 -> 713 us with the
// records at 1024 rows), waits in line (around a call all sums would be spilled).  The hand-back to the leading CTA is a relaxed
// arrival: with release semantics at cluster scope a K block took 1870 cycles instead of 840.  Tried without gain: 128 ids a tile, four
// accumulators, 32 sums and boxes stored by TMA (829 us: 24 KB a K block of half the size); the next K block's scales, its wait or its
// first load ahead (721 to 850: spills); sixteen columns a load (740).  Every batch tile has rows for both CTAs (run_head).
__global__ void __launch_bounds__(kPairThreads, 1)
head_fp8_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ HeadArgs p) {
  using Smem = PairSmem;
  constexpr int kAccBufs = Smem::kAccBufs, kStageBytes = Smem::kStageBytes, kMaxStages = Smem::kStages;
  constexpr int kCols = 64;             // ids of an epilogue warp: warp = (lane quadrant, group of 64 ids)
  const int kStages = p.stages;
  extern __shared__ __align__(1024) unsigned char smem[];
  // carve: [stages][A 16 KB | W 16 KB], then output blocks, scale tables, barriers; the same places in both CTAs
  unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
  float *out = reinterpret_cast<float *>(tiles + size_t(kStages) * kStageBytes);   // [epilogue warp][32][16], the 16-byte pieces of a row in an order of its own
  float4 *stats = reinterpret_cast<float4 *>(out + kEpiWarps * Smem::kOutFloats);  // [epilogue thread] maximum, minimum, its id, not finite
  float *sa = reinterpret_cast<float *>(stats + kEpiWarps * 32);                   // [K/128][128]
  const int kblocks = p.K / kTileK;
  float *sw = sa + size_t(kblocks) * 128;                                          // [epilogue warp][2][K/128]
  uint64_t *bars = reinterpret_cast<uint64_t *>(sw + size_t(kblocks) * 2 * kEpiWarps);
  uint64_t *full = bars, *empty = bars + kMaxStages, *acc_full = bars + 2 * kMaxStages, *acc_empty = acc_full + kAccBufs;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + kAccBufs);
  int *abort_word = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(cluster_rank()), pair = int(blockIdx.x) >> 1, pairs = int(gridDim.x) >> 1;
  const int b_tiles = (p.M + 255) / 256, total_tiles = (p.N + 255) / 256 * b_tiles;
  // tile t = (vocabulary tile t / b_tiles, batch tile t % b_tiles)
  Abort ab{abort_word};

  if (threadIdx.x == 0) {
    *abort_word = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < kAccBufs; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * kEpiWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // TMEM allocation by one full warp of each CTA; the address lands in shared memory
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(uint32_t(kTmemColumns)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();   // both CTAs have started and set up their barriers
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer, one in each CTA
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      // one batch tile: every weight is read once per step, and 530 MB of them would push everything else out of the L2 --
      // the logits, the activations, the code of the kernels around this one
      uint64_t policy, keep;
      if (b_tiles == 1) asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
      else asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
      asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(keep));
      // the ring's first weights are on their way to the L2 while the kernel in front of this one (the quantiser) finishes
      const int early = kblocks < kStages ? kblocks : kStages;
      for (int s = 0; s < early; ++s) tma_prefetch_3d(&map_w, 0, pair / b_tiles * 256 + 128 * rank, s, policy);
      cudaGridDependencySynchronize();
      cudaTriggerProgrammaticLaunchCompletion();
      const uint32_t leader_full = peer_addr(full, 0);
      for (int tile = pair; tile < total_tiles && !ab.set(); tile += pairs) {
        const int id = tile / b_tiles * 256 + 128 * rank, mine = tile % b_tiles * 256 + 128 * rank;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, ab)) break;
          unsigned char *a_dst = tiles + size_t(stage) * kStageBytes, *w_dst = a_dst + 128 * kTileK;
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * kStageBytes);   // of both CTAs
          tma_load_pair(w_dst, &map_w, leader_full + 8 * stage, 0, id, kb, policy);
          tma_load_pair(a_dst, &map_a, leader_full + 8 * stage, 0, mine, kb, keep);
          if (++stage == uint32_t(kStages)) { stage = 0; phase ^= 1; }
        }
      }
      // every release has arrived before this CTA's shared memory goes away
      for (int s = 0; s < kStages && !ab.set(); ++s) {
        mbar_wait(&empty[stage], phase ^ 1, ab);
        if (++stage == uint32_t(kStages)) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of the leading CTA: the warp waits together, one lane issues
    cudaGridDependencySynchronize();
    if (rank == 0) {
      const uint32_t tiles16 = smem_addr(tiles) >> 4;
      const bool leader = elect_one();
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      for (int tile = pair; tile < total_tiles && !__any_sync(0xffffffffu, ab.set()); tile += pairs) {
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, ab))) break;
          if (!__all_sync(0xffffffffu, mbar_wait<true>(&acc_empty[acc], acc_phase ^ 1, ab))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a16 = tiles16 + stage * (kStageBytes >> 4), w16 = a16 + ((128 * kTileK) >> 4);  // addresses >> 4
          const uint32_t d_addr = tmem_base + acc * 256;
          if (leader) {
            // D[batch row, vocabulary id] (+)= A[batch row, k] * W[vocabulary id, k], K = 32 bytes per instruction
            umma_f8_pair<false>(d_addr, umma_desc16(a16), umma_desc16(w16));
            umma_f8_pair<true>(d_addr, umma_desc16(a16 + 2), umma_desc16(w16 + 2));
            umma_f8_pair<true>(d_addr, umma_desc16(a16 + 4), umma_desc16(w16 + 4));
            umma_f8_pair<true>(d_addr, umma_desc16(a16 + 6), umma_desc16(w16 + 6));
            umma_commit_pair(&acc_full[acc]);   // accumulator of this K block is complete
            umma_commit_pair(&empty[stage]);    // the stage may be refilled: these MMAs have read it
          }
          __syncwarp();
          if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
          if (++stage == uint32_t(kStages)) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else {
    cudaGridDependencySynchronize();
  }
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // ------------------------------------------------------------------ epilogue: warp = (lane quadrant, column group)
    cudaGridDependencySynchronize();
    const int quad = warp & 3;          // TMEM lanes [32*quad, 32*quad+32) are readable by this warp: batch rows
    const int group = (warp - 4) >> 2;  // vocabulary ids [64*group, 64*group+64) of the tile
    const int row = quad * 32 + lane;   // batch row inside the CTA's 128
    const int et = threadIdx.x - 128;
    const uint32_t lane_base = tmem_base + group * kCols + (uint32_t(quad * 32) << 16);
    const uint32_t leader_empty = peer_addr(acc_empty, 0);
    float *my_sw = sw + size_t(warp - 4) * 2 * kblocks;
    float *my_out = out + (warp - 4) * Smem::kOutFloats;
    // fp32 scales of the 128-row weight block this warp's columns belong to, on their way into shared memory
    auto fetch_scales = [&](int tile, float *to) {
      if (tile < total_tiles) {
        const int w_block = min(tile / b_tiles * 2 + (group >> 1), (p.N + 127) / 128 - 1);
        for (int i = lane; i < kblocks; i += 32) copy4_async(to + i, p.w_scale + size_t(w_block) * kblocks + i);
      }
    };
    fetch_scales(pair, my_sw);
    int which = 0;
    uint32_t acc = 0, acc_phase = 0;
    int table_bt = -1;
    bool alive = true;  // warp-uniform; once false the remaining tiles are walked without waiting or computing,
                        // so that all epilogue threads still meet at every named barrier
    // running statistics of this thread's batch row over the tiles of one batch tile (vocabulary tiles come in ascending
    // order, so a strict comparison keeps the first maximum)
    const float4 nothing = make_float4(-CUDART_INF_F, CUDART_INF_F, __int_as_float(0x7fffffff), 0.f);
    stats[et] = nothing;   // (in shared memory: the registers are the sums')
    const bool stats_on = p.row_stats != nullptr || p.owner_stats_offset != 0;
    auto row_of = [&](int m) {   // batch row m of the output
      if (p.rows_per_owner == 0) return p.logits + size_t(m) * p.ldl;
      const int g = p.first_row + m, owner = g / p.rows_per_owner;
      return p.owner_base[owner] + size_t(g - owner * p.rows_per_owner) * p.ldl + p.col_offset;
    };
    auto flush_stats = [&](int bt_of) {
      const int m = bt_of * 256 + 128 * rank + row;
      const float4 st = stats[et];
      if (stats_on && m < p.M) merge_stats(p, m, st.x, __float_as_int(st.z), st.y, st.w != 0.f);
      stats[et] = nothing;
    };
    for (int tile = pair; tile < total_tiles; tile += pairs) {
      const int nt = tile / b_tiles, bt = tile % b_tiles, m0 = bt * 256 + 128 * rank;
      if (bt != table_bt) {  // activation scales of this CTA's rows: sa[kb][row] (a number of pairs that is a multiple of b_tiles
                             // keeps bt fixed per CTA, so this normally happens once)
        if (table_bt >= 0) flush_stats(table_bt);
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");  // readers of the previous table are done
        for (int i = et; i < kblocks * 128; i += 32 * kEpiWarps) {
          const int r = i / kblocks, kb = i % kblocks, m = m0 + r;
          sa[kb * 128 + r] = m < p.M ? load_input(p.a_scale + size_t(m) * kblocks + kb) : 0.f;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
        table_bt = bt;
      }
      // The next tile's scales are fetched a tile ahead: they come from DRAM, and a load of them between two tiles would keep the
      // accumulators waiting.
      const float *tile_sw = my_sw + which * kblocks;
      copies_done();
      __syncwarp();
      which ^= 1;
      fetch_scales(tile + pairs, my_sw + which * kblocks);
      float sum[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) sum[c] = 0.f;
      for (int kb = 0; kb < kblocks && alive; ++kb) {
        const float scale = sa[kb * 128 + row] * tile_sw[kb];
        const unsigned long long scale2 = pack2(scale, scale);
        alive = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_phase, ab));
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[2][8];
        tmem_ld8(lane_base + acc * 256, r[0]);
#pragma unroll
        for (int q = 0; q < kCols / 8; ++q) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (q + 1 < kCols / 8) {
            tmem_ld8(lane_base + acc * 256 + 8 * (q + 1), r[(q + 1) & 1]);
          } else {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(leader_empty + 8 * acc);
          }
#pragma unroll
          for (int c = 0; c < 8; c += 2) fma2_acc(sum[8 * q + c], sum[8 * q + c + 1], r[q & 1][c], r[q & 1][c + 1], scale2);
        }
        if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
      }
      // Output, while the tensor cores wait: as few instructions as it takes.
      const int n0 = nt * 256 + group * kCols;
      const bool whole = n0 + kCols <= p.N;
      if (alive && stats_on) {
        const float4 st = stats[et];
        float st_best = st.x, st_low = st.y, st_bad = st.w, st_bad1 = 0.f;
        int st_id = __float_as_int(st.z);
        if (whole) {
          const unsigned long long zero2 = pack2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < kCols; c += 2)   // NaN once any logit is NaN or infinite
            fma2_acc(st_bad, st_bad1, __float_as_uint(sum[c]), __float_as_uint(sum[c + 1]), zero2);
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            if (sum[c] > st_best) { st_best = sum[c]; st_id = n0 + c; }
            st_low = fminf(st_low, sum[c]);
          }
        } else {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            const float v = sum[c];
            if (n0 + c < p.N) {
              st_bad = fmaf(v, 0.f, st_bad);
              if (v > st_best) { st_best = v; st_id = n0 + c; }
              st_low = fminf(st_low, v);
            }
          }
        }
        stats[et] = make_float4(st_best, st_low, __int_as_float(st_id), st_bad + st_bad1);
      }
      // Lane l holds row l of the warp's 32 x 64 block.  Sixteen ids at a time go through shared memory, so that a store instruction
      // writes 64 contiguous bytes of eight rows.  (A row of the block is 64 bytes; its four pieces are swapped by bits 1 and 2 of the row's
      // number, so that neither side has a bank conflict.)
      if (alive) {
        const bool plain = p.rows_per_owner == 0 && whole && p.ldl % 4 == 0 && (reinterpret_cast<uintptr_t>(p.logits) & 15u) == 0;
        const int r0 = quad * 32 + (lane >> 2), col = 4 * (lane & 3);
#pragma unroll
        for (int q = 0; q < kCols / 16; ++q) {
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 16; c += 4)
            *reinterpret_cast<float4 *>(my_out + lane * 16 + (c ^ (4 * ((lane >> 1) & 3)))) =
                make_float4(sum[16 * q + c], sum[16 * q + c + 1], sum[16 * q + c + 2], sum[16 * q + c + 3]);
          __syncwarp();
          if (plain) {
            float *dst = p.logits + size_t(m0 + r0) * p.ldl + n0 + 16 * q + col;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 v = *reinterpret_cast<const float4 *>(my_out + ((lane >> 2) + 8 * i) * 16 + (col ^ (4 * ((lane >> 3) & 3))));
              if (m0 + r0 + 8 * i < p.M) *reinterpret_cast<float4 *>(dst) = v;
              dst += 8 * p.ldl;
            }
          } else {
            const int n = n0 + 16 * q + col;
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
              const int m = m0 + r0 + 8 * i;
              const float *v = my_out + ((lane >> 2) + 8 * i) * 16 + (col ^ (4 * ((lane >> 3) & 3)));
              if (m >= p.M || n >= p.N) continue;
              float *dst = row_of(m) + n;
              if (n + 4 <= p.N && (reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
                *reinterpret_cast<float4 *>(dst) = *reinterpret_cast<const float4 *>(v);
              } else {
                for (int k = 0; k < 4; ++k)
                  if (n + k < p.N) dst[k] = v[k];
              }
            }
          }
        }
      }
    }
    if (alive && table_bt >= 0) flush_stats(table_bt);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();   // no CTA leaves, or gives its tensor memory back, while the other's MMAs and arrivals can still reach it
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemColumns)));
  }
  if (threadIdx.x == 0 && *abort_word && p.error_flag) atomicExch(p.error_flag, 1);
  cluster_barrier();
}

// ---------------------------------------------------------------------------------------------------------------
// Batches of up to 64 rows: the weights are the M dimension of the MMA, the batch its N.
constexpr int kDecodeWarps = 8, kDecodeThreads = 64 + 32 * kDecodeWarps;   // epilogue warps; with TMA and MMA warp
template <int kRows>
struct DecodeSmem {
  static constexpr int kStageBytes = (128 + kRows) * kTileK;
  static constexpr int kMaxAccs = 16;
  static constexpr int kMaxGroup = kRows <= 32 ? 4 : 2;                      // K blocks of a stage
  static constexpr int kMaxStages = 12;
  // for the statistics an epilogue warp turns its logits, kTurn batch rows at a time, in a block of shared memory (with four batch
  // rows at a time the 16-row tile's ring still has its third stage)
  static constexpr int kTurn = kRows == 16 ? 4 : 16, kTurnFloats = 36 * kTurn;
  // bytes beside the stages: alignment slack, blocks, scale tables [K/128][kRows] and [warps][2][K/128], barriers and flags
  static constexpr size_t fixed_bytes(int kblocks) {
    return 1024 + kDecodeWarps * kTurnFloats * 4 + size_t(kblocks) * (kRows + 2 * kDecodeWarps) * 4 +
           (2 * kMaxStages + 2 * kMaxAccs) * 8 + 16;
  }
  static constexpr int stages(int kblocks, int group) {
    const long long room = 227 * 1024 - (long long)fixed_bytes(kblocks);
    const int n = room < 0 ? 0 : int(room / (kStageBytes * group));
    return n > kMaxStages ? kMaxStages : n;
  }
};

template <int kN>
struct Blocks { static constexpr int value = kN; };
template <int kCols>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t *r) {
  if constexpr (kCols == 8) {
    tmem_ld8(taddr, r);
  } else if constexpr (kCols == 16) {
    tmem_ld16(taddr, r);
  } else {
    static_assert(kCols == 32, "8, 16 or 32 columns");
    tmem_ld32(taddr, r);
  }
}
template <int kRows>
__global__ void __launch_bounds__(kDecodeThreads, 1)
head_fp8_decode_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ HeadArgs p) {
  using Smem = DecodeSmem<kRows>;
  constexpr int kMaxAccs = Smem::kMaxAccs, kMaxStages = Smem::kMaxStages, kStageBytes = Smem::kStageBytes;
  constexpr int kCols = kRows / 2;   // batch rows of an epilogue warp: warp = (lane quadrant, half of the batch rows)
  const int kStages = p.stages, group = p.group;
  const int accs = min(kMaxAccs, kTmemColumns / (kRows * group));   // sets of accumulators: one per K block of a stage, kRows columns each
  const int stage_bytes = kStageBytes * group, w_bytes = 128 * kTileK * group;   // [W g0..][A g0..]
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
  float *turn = reinterpret_cast<float *>(tiles + size_t(kStages) * stage_bytes);   // [epilogue warp][kTurn][36]
  float *sa = turn + kDecodeWarps * Smem::kTurnFloats;                              // [K/128][kRows]
  const int kblocks = p.K / kTileK;
  float *sw = sa + size_t(kblocks) * kRows;                                         // [epilogue warp][2][K/128]
  uint64_t *bars = reinterpret_cast<uint64_t *>(sw + size_t(kblocks) * 2 * kDecodeWarps);
  uint64_t *full = bars, *empty = bars + kMaxStages, *acc_full = bars + 2 * kMaxStages, *acc_empty = acc_full + kMaxAccs;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + kMaxAccs);
  int *abort_word = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total_tiles = (p.N + 127) / 128;
  const int active = p.M > kCols ? 2 : 1;   // halves with a batch row in them
  Abort ab{abort_word};

  if (threadIdx.x == 0) {
    *abort_word = 0;
    for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < accs; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4 * active); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // TMEM allocation by one full warp; the address lands in shared memory
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(uint32_t(kTmemColumns)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      // every weight is read once per step, and 530 MB of them would push everything else out of the L2 -- the logits, the
      // activations, the code of the kernels around this one
      uint64_t policy;
      asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
      // the ring's first weights are on their way to the L2 while the kernel in front of this one (the quantiser) finishes
      const int early = kblocks / group < kStages ? kblocks / group : kStages;
      for (int s = 0; s < early; ++s) tma_prefetch_3d(&map_w, 0, int(blockIdx.x) * 128, s * group, policy);
      cudaGridDependencySynchronize();
      cudaTriggerProgrammaticLaunchCompletion();
      for (int tile = blockIdx.x; tile < total_tiles && !ab.set(); tile += gridDim.x) {
        for (int kb = 0; kb < kblocks; kb += group) {
          if (!mbar_wait(&empty[stage], phase ^ 1, ab)) break;
          unsigned char *w_dst = tiles + size_t(stage) * stage_bytes, *a_dst = w_dst + w_bytes;
          mbar_expect_tx(&full[stage], uint32_t(stage_bytes));
          tma_load_3d(w_dst, &map_w, &full[stage], 0, tile * 128, kb, policy);
          tma_load_3d(a_dst, &map_a, &full[stage], 0, 0, kb);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer: the warp waits together, one lane issues
    cudaGridDependencySynchronize();
    constexpr uint32_t idesc = umma_idesc(kRows);
    const uint32_t tiles16 = smem_addr(tiles) >> 4, stage16 = uint32_t(stage_bytes) >> 4;
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
    for (int tile = blockIdx.x; tile < total_tiles && !__any_sync(0xffffffffu, ab.set()); tile += gridDim.x) {
      bool ok = true;
      for (int kb = 0; kb < kblocks && ok; kb += group) {
        if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase, ab))) break;
        uint32_t w16 = tiles16 + stage * stage16, a16 = w16 + (uint32_t(w_bytes) >> 4);  // addresses >> 4
        ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[acc], acc_phase ^ 1, ab));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
          uint32_t d_addr = tmem_base + acc * group * kRows;
          for (int g = 0; g < group; ++g) {
            // D[vocabulary id, batch row] (+)= W[vocabulary id, k] * A[batch row, k], K = 32 bytes per instruction
            umma_f8<false>(d_addr, umma_desc16(w16), umma_desc16(a16), idesc);
            umma_f8<true>(d_addr, umma_desc16(w16 + 2), umma_desc16(a16 + 2), idesc);
            umma_f8<true>(d_addr, umma_desc16(w16 + 4), umma_desc16(a16 + 4), idesc);
            umma_f8<true>(d_addr, umma_desc16(w16 + 6), umma_desc16(a16 + 6), idesc);
            d_addr += kRows; w16 += (128 * kTileK) >> 4; a16 += (kRows * kTileK) >> 4;
          }
          umma_commit(&acc_full[acc]);   // the accumulators of these K blocks are complete
          umma_commit(&empty[stage]);    // the stage may be refilled: these MMAs have read it
        }
        __syncwarp();
        if (++acc == uint32_t(accs)) { acc = 0; acc_phase ^= 1; }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (((warp - 2) >> 2) < active) {
    // ------------------------------------------------------------------ epilogue: warp = (lane quadrant, half of the batch rows)
    cudaGridDependencySynchronize();
    const int quad = warp & 3;            // TMEM lanes [32*quad, 32*quad+32) are readable by this warp: vocabulary ids
    const int first = ((warp - 2) >> 2) * kCols, et = threadIdx.x - 64;   // batch rows [first, first + kCols)
    const int epi_threads = 128 * active;
    const uint32_t lane_base = tmem_base + first + (uint32_t(quad * 32) << 16);
    float *my_sw = sw + size_t(warp - 2) * 2 * kblocks;
    auto fetch_scales = [&](int tile, float *to) {   // the tile's weight scales on their way into shared memory
      if (tile < total_tiles)
        for (int i = lane; i < kblocks; i += 32) copy4_async(to + i, p.w_scale + size_t(tile) * kblocks + i);
    };
    fetch_scales(blockIdx.x, my_sw);
    int which = 0;
    for (int i = et; i < kblocks * kRows; i += epi_threads) {   // activation scales: sa[kb][row]
      const int r = i / kblocks, kb = i % kblocks;
      sa[kb * kRows + r] = r < p.M ? load_input(p.a_scale + size_t(r) * kblocks + kb) : 0.f;
    }
    asm volatile("bar.sync 1, %0;" ::"r"(epi_threads) : "memory");
    uint32_t acc = 0, acc_phase = 0;
    bool alive = true;  // warp-uniform
    // Statistics: in each turn a lane looks at kTurn consecutive ids of one of kTurn batch rows (tiles come in ascending order, so
    // a strict comparison keeps the first maximum).
    constexpr int kTurn = Smem::kTurn, kTurns = kCols / kTurn;
    float st_best[kTurns], st_low[kTurns], st_bad[kTurns];   // (st_bad: NaN once a logit is NaN or infinite)
    int st_id[kTurns];
#pragma unroll
    for (int h = 0; h < kTurns; ++h) { st_best[h] = -CUDART_INF_F; st_low[h] = CUDART_INF_F; st_id[h] = 0x7fffffff; st_bad[h] = 0.f; }
    float *my_turn = turn + (warp - 2) * Smem::kTurnFloats;
    const bool stats_on = p.row_stats != nullptr || p.owner_stats_offset != 0;
    for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
      // The next tile's scales are fetched a tile ahead: they come from DRAM.
      const float *tile_sw = my_sw + which * kblocks;
      copies_done();
      __syncwarp();
      which ^= 1;
      fetch_scales(tile + gridDim.x, my_sw + which * kblocks);
      float sum[kCols];
#pragma unroll
      for (int c = 0; c < kCols; ++c) sum[c] = 0.f;
      for (int kb = 0; kb < kblocks;) {
        alive = __all_sync(0xffffffffu, mbar_wait(&acc_full[acc], acc_phase, ab));
        if (!alive) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        auto consume = [&](auto blocks) {   // that many K blocks: all loads in flight together, one wait
          constexpr int kBlocks = decltype(blocks)::value;
          const uint32_t taddr = lane_base + acc * kBlocks * kRows;
          uint32_t r[kBlocks * kCols];
#pragma unroll
          for (int u = 0; u < kBlocks; ++u) tmem_ld<kCols>(taddr + u * kRows, r + u * kCols);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          // the values are in registers: the accumulators can be refilled while they are scaled and added
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[acc]);
#pragma unroll
          for (int u = 0; u < kBlocks; ++u, ++kb) {
            const unsigned long long w_scale = pack2(tile_sw[kb], tile_sw[kb]);
            const ulonglong2 *row_scale = reinterpret_cast<const ulonglong2 *>(sa + kb * kRows + first);
#pragma unroll
            for (int c = 0; c < kCols; c += 4) {
              const ulonglong2 s = row_scale[c >> 2];
              const uint32_t *d = r + u * kCols + c;
              fma2_acc(sum[c], sum[c + 1], d[0], d[1], mul2(s.x, w_scale));
              fma2_acc(sum[c + 2], sum[c + 3], d[2], d[3], mul2(s.y, w_scale));
            }
          }
        };
        if (Smem::kMaxGroup >= 4 && group == 4) consume(Blocks<Smem::kMaxGroup >= 4 ? 4 : 1>{});
        else if (group == 2) consume(Blocks<2>{});
        else consume(Blocks<1>{});
        if (++acc == uint32_t(accs)) { acc = 0; acc_phase ^= 1; }
      }
      if (!alive) break;
      const int n0 = tile * 128 + 32 * quad, n = n0 + lane;
      const bool in = n < p.N;
      // a store instruction writes 128 contiguous bytes of a row
      const int g = p.first_row + first;
      int owner = p.rows_per_owner ? g / p.rows_per_owner : 0, left = p.rows_per_owner ? (owner + 1) * p.rows_per_owner - g : kRows;
      float *dst = p.rows_per_owner ? p.owner_base[owner] + size_t(p.rows_per_owner - left) * p.ldl + p.col_offset + n
                                    : p.logits + size_t(first) * p.ldl + n;
#pragma unroll
      for (int c = 0; c < kCols; ++c, dst += p.ldl) {
        if (left-- == 0) {              // the next owner's rows (a batch row's buffer exists)
          if (first + c < p.M) dst = p.owner_base[++owner] + p.col_offset + n;
          left = p.rows_per_owner - 1;
        }
        if (in && first + c < p.M) *dst = sum[c];
      }
      if (stats_on) {
        const int turn_row = lane % kTurn, turn_id = lane / kTurn * kTurn, ids = min(kTurn, p.N - n0 - turn_id);
#pragma unroll
        for (int h = 0; h < kTurns; ++h) {
          __syncwarp();
#pragma unroll
          for (int c = 0; c < kTurn; ++c) my_turn[36 * c + lane] = sum[h * kTurn + c];
          __syncwarp();
          float v[kTurn];
#pragma unroll
          for (int c = 0; c < kTurn; c += 4)
            *reinterpret_cast<float4 *>(v + c) = *reinterpret_cast<const float4 *>(my_turn + 36 * turn_row + turn_id + c);
          if (ids < kTurn)             // the last ids of the vocabulary: those beyond it repeat the last one (or are left out)
#pragma unroll
            for (int c = 1; c < kTurn; ++c) v[c] = c < ids ? v[c] : v[c - 1];
          float hi = v[0], low = v[0], bad = st_bad[h];
#pragma unroll
          for (int c = 0; c < kTurn; ++c) { hi = fmaxf(hi, v[c]); low = fminf(low, v[c]); bad = fmaf(v[c], 0.f, bad); }
          if (ids <= 0) { hi = -CUDART_INF_F; low = CUDART_INF_F; bad = st_bad[h]; }
          st_bad[h] = bad;
          st_low[h] = fminf(st_low[h], low);
          if (__any_sync(0xffffffffu, hi > st_best[h])) {
            int at = 0;
#pragma unroll
            for (int c = kTurn - 1; c > 0; --c) at = v[c] == hi ? c : at;
            if (v[0] == hi) at = 0;
            if (hi > st_best[h]) { st_best[h] = hi; st_id[h] = n0 + turn_id + at; }
          }
        }
      }
    }
    if (stats_on) {
      // The four lane quadrants' records of a batch row are merged here: all CTAs raise the same few lines at the end.  (The ring is
      // free: the last accumulators have been waited for.)
      struct Record { float best, low; int id, bad; };
      Record *records = reinterpret_cast<Record *>(tiles);   // [quadrant][kRows]
#pragma unroll
      for (int h = 0; h < kTurns; ++h) {
        int bad = st_bad[h] == 0.f ? 0 : 1;
        for (int o = kTurn; o < 32; o <<= 1) {
          const float best = __shfl_xor_sync(0xffffffffu, st_best[h], o);
          const int id = __shfl_xor_sync(0xffffffffu, st_id[h], o);
          if (best > st_best[h] || (best == st_best[h] && id < st_id[h])) { st_best[h] = best; st_id[h] = id; }
          st_low[h] = fminf(st_low[h], __shfl_xor_sync(0xffffffffu, st_low[h], o));
          bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        }
        if (alive && lane < kTurn) records[quad * kRows + first + h * kTurn + lane] = Record{st_best[h], st_low[h], st_id[h], bad};
      }
      asm volatile("bar.sync 1, %0;" ::"r"(epi_threads) : "memory");
      if (alive && et < p.M) {
        Record all = records[et];
#pragma unroll
        for (int q = 1; q < 4; ++q) {
          const Record r = records[q * kRows + et];
          if (r.best > all.best || (r.best == all.best && r.id < all.id)) { all.best = r.best; all.id = r.id; }
          all.low = fminf(all.low, r.low);
          all.bad |= r.bad;
        }
        merge_stats(p, et, all.best, all.id, all.low, all.bad != 0);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemColumns)));
  }
  if (threadIdx.x == 0 && *abort_word && p.error_flag) atomicExch(p.error_flag, 1);
}

// ---------------------------------------------------------------------------------------------------------------
// Activation quantisation: per (row, 128-wide K group) scale = 2^ceil(log2(max(amax,1e-4)/448)), e4m3 round to
// nearest even with saturation (components/dense/src/dense.cu:8-16 with the group widened from 32 to 128).
__global__ void quantize_kernel(const __nv_bfloat16 *x, uint8_t *a, float *scale, int groups) {
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= groups) return;
  const uint2 raw = *reinterpret_cast<const uint2 *>(x + size_t(g) * 128 + lane * 4);
  const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162 *>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162 *>(&raw.y);
  float v[4] = {__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi)};
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const uint32_t bits = __float_as_uint(__fmul_rn(fmaxf(amax, 1e-4f), 1.f / 448.f));
  const uint32_t exponent = (bits >> 23) + ((bits & 0x7fffffu) != 0);
  const float s = __uint_as_float(exponent << 23);
  uint32_t packed = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float q = fminf(448.f, fmaxf(-448.f, __fdiv_rn(v[i], s)));
    packed |= uint32_t(__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3)) << (8 * i);
  }
  *reinterpret_cast<uint32_t *>(a + size_t(g) * 128 + lane * 4) = packed;
  if (lane == 0) scale[g] = s;
}

// Clears the row records before the head raises them.  (A memset would stand between two programmatic launches and wait for
// the first.  This kernel lets the head be set up at once, ahead of its own wait: the head touches nothing before this kernel
// has finished, which it only does after the kernel in front of it.  With the wait first a decode step takes 126.6 us instead
// of 126.0 at 8 rows, 170.9 instead of 169.9 at 64.)
__global__ void clear_stats_kernel(HeadRowStats *stats, int rows) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  for (int i = threadIdx.x; i < rows; i += blockDim.x) stats[i] = HeadRowStats{0ull, 0u, 0u};
}

// ---------------------------------------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn encoder() {
  static EncodeFn fn = [] {
    void *sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      sym = nullptr;
    return reinterpret_cast<EncodeFn>(sym);
  }();
  return fn;
}
// uint8 matrix [rows, cols] row-major seen as a 3-D tensor [cols/128][rows][128 bytes] (strides 128 and cols bytes),
// box {128 bytes, box_rows, group}: one copy brings `group` consecutive K blocks of box_rows rows, laid out in shared
// memory as `group` K-major tiles of box_rows x 128 bytes with the 128-byte swizzle, and reads every row of the matrix
// in runs of group*128 contiguous bytes.  Zero fill outside.
bool make_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t group) {
  EncodeFn enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {uint64_t(kTileK), rows, cols / kTileK};
  const cuuint64_t strides[2] = {cols, uint64_t(kTileK)};
  const cuuint32_t box[3] = {uint32_t(kTileK), box_rows, group};
  const cuuint32_t elem[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_head(const CUtensorMap &mw, const CUtensorMap &ma, const HeadArgs &p, int sms, cudaStream_t stream) {
  HeadArgs q = p;
  q.stages = HeadSmem::stages(p.K / kTileK, p.group);
  if (q.stages < 2) return cudaErrorInvalidValue;
  const size_t smem = HeadSmem::fixed_bytes(p.K / kTileK) + size_t(q.stages) * HeadSmem::kStageBytes * p.group;
  static thread_local int configured = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (configured != dev) {
    e = cudaFuncSetAttribute(head_fp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int tiles = (p.N + 127) / 128;   // one batch tile
  return launch_early(head_fp8_kernel, tiles < sms ? tiles : sms, kHeadThreads, smem, stream, mw, ma, q);
}

cudaError_t launch_pairs(const CUtensorMap &mw, const CUtensorMap &ma, const HeadArgs &p, int sms, cudaStream_t stream) {
  HeadArgs q = p;
  q.stages = PairSmem::stages(p.K / kTileK);
  if (q.stages < 2) return cudaErrorInvalidValue;
  static thread_local int configured = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (configured != dev) {
    e = cudaFuncSetAttribute(head_fp8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int b_tiles = (p.M + 255) / 256, tiles = ((p.N + 255) / 256) * b_tiles;
  int pairs = tiles < sms / 2 ? tiles : sms / 2;
  if (b_tiles <= pairs) pairs -= pairs % b_tiles;  // every CTA then keeps one batch tile (and its scale table) for good
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(2 * pairs));
  cfg.blockDim = dim3(kPairThreads);
  cfg.dynamicSmemBytes = PairSmem::fixed_bytes(p.K / kTileK) + size_t(q.stages) * PairSmem::kStageBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1] = programmatic_launch();
  cfg.attrs = attr; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, head_fp8_pair_kernel, mw, ma, q);
}

template <int kRows>
cudaError_t launch_decode(const CUtensorMap &mw, const CUtensorMap &ma, const HeadArgs &p, int sms, cudaStream_t stream) {
  using Smem = DecodeSmem<kRows>;
  HeadArgs q = p;
  q.stages = Smem::stages(p.K / kTileK, p.group);
  if (q.stages < 2) return cudaErrorInvalidValue;
  const size_t smem = Smem::fixed_bytes(p.K / kTileK) + size_t(q.stages) * Smem::kStageBytes * p.group;
  static thread_local int configured = -1;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (configured != dev) {
    e = cudaFuncSetAttribute(head_fp8_decode_kernel<kRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    configured = dev;
  }
  const int tiles = (p.N + 127) / 128;
  return launch_early(head_fp8_decode_kernel<kRows>, tiles < sms ? tiles : sms, kDecodeThreads, smem, stream, mw, ma, q);
}

}  // namespace
}  // namespace ds41

using namespace ds41;

extern "C" int ds41_b200_quantize_activations(const void *x_bf16, void *a_e4m3, float *a_scale, int M, int K,
                                              cudaStream_t stream) {
  if (!x_bf16 || !a_e4m3 || !a_scale || M < 1 || K < 128 || K % 128) return invalid("quantize arguments");
  const int groups = M * (K / 128);
  return int(launch_early(quantize_kernel, (groups * 32 + 255) / 256, 256, 0, stream, static_cast<const __nv_bfloat16 *>(x_bf16),
                          static_cast<uint8_t *>(a_e4m3), a_scale, groups));
}

namespace {
int run_head(const void *a_e4m3, const float *a_scale, const void *w_e4m3, const float *w_scale, HeadArgs p,
             cudaStream_t stream);
}

extern "C" int ds41_b200_head_fp8(const void *a_e4m3, const float *a_scale, const void *w_e4m3, const float *w_scale,
                                  float *logits, int64_t logits_stride, int M, int N, int K, int *error_flag,
                                  cudaStream_t stream) {
  if (!a_e4m3 || !a_scale || !w_e4m3 || !w_scale || !logits || M < 1 || N < 1 || K < 128 || K % 128 || K > 16384 ||
      logits_stride < N)
    return invalid("head arguments");
  HeadArgs p{};
  p.a_scale = a_scale; p.w_scale = w_scale; p.logits = logits; p.ldl = logits_stride;
  p.M = M; p.N = N; p.K = K; p.error_flag = error_flag;
  return run_head(a_e4m3, a_scale, w_e4m3, w_scale, p, stream);
}

extern "C" int ds41_b200_head_fp8_stats(const void *a_e4m3, const float *a_scale, const void *w_e4m3, const float *w_scale,
                                        float *logits, int64_t logits_stride, int M, int N, int K, void *row_extremes,
                                        int *error_flag, cudaStream_t stream) {
  if (!a_e4m3 || !a_scale || !w_e4m3 || !w_scale || !logits || M < 1 || N < 1 || K < 128 || K % 128 || K > 16384 ||
      logits_stride < N || !row_extremes || (reinterpret_cast<uintptr_t>(row_extremes) & 15u))
    return invalid("head arguments");
  static_assert(sizeof(HeadRowStats) == DS41_B200_ROW_EXTREMES_BYTES, "row record size");
  const cudaError_t e = launch_early(clear_stats_kernel, 1, 512, 0, stream, static_cast<HeadRowStats *>(row_extremes), M);
  if (e != cudaSuccess) return int(e);
  HeadArgs p{};
  p.a_scale = a_scale; p.w_scale = w_scale; p.logits = logits; p.ldl = logits_stride;
  p.M = M; p.N = N; p.K = K; p.error_flag = error_flag;
  p.row_stats = static_cast<HeadRowStats *>(row_extremes);
  return run_head(a_e4m3, a_scale, w_e4m3, w_scale, p, stream);
}

extern "C" int ds41_b200_head_fp8_scatter_stats(const void *a_e4m3, const float *a_scale, const void *w_e4m3,
                                                const float *w_scale, float *const *owner_logits, int owners,
                                                int rows_per_owner, int64_t logits_stride, int vocab_offset, int M,
                                                int N, int K, int64_t stats_offset_bytes, int *error_flag,
                                                cudaStream_t stream);

extern "C" int ds41_b200_head_fp8_scatter(const void *a_e4m3, const float *a_scale, const void *w_e4m3,
                                          const float *w_scale, float *const *owner_logits, int owners,
                                          int rows_per_owner, int64_t logits_stride, int vocab_offset, int M, int N,
                                          int K, int *error_flag, cudaStream_t stream) {
  return ds41_b200_head_fp8_scatter_stats(a_e4m3, a_scale, w_e4m3, w_scale, owner_logits, owners, rows_per_owner,
                                          logits_stride, vocab_offset, M, N, K, 0, error_flag, stream);
}

extern "C" int ds41_b200_head_fp8_scatter_stats(const void *a_e4m3, const float *a_scale, const void *w_e4m3,
                                                const float *w_scale, float *const *owner_logits, int owners,
                                                int rows_per_owner, int64_t logits_stride, int vocab_offset, int M,
                                                int N, int K, int64_t stats_offset_bytes, int *error_flag,
                                                cudaStream_t stream) {
  if (stats_offset_bytes < 0 || (stats_offset_bytes & 15) ||
      (stats_offset_bytes && stats_offset_bytes < int64_t(rows_per_owner) * logits_stride * 4))
    return invalid("scattered head: the row records must lie behind the owner's logits, 16-byte aligned");
  if (!a_e4m3 || !a_scale || !w_e4m3 || !w_scale || !owner_logits || M < 1 || N < 1 || K < 128 || K % 128 ||
      K > 16384 || owners < 1 || owners > kMaxOwners || rows_per_owner < 1 || vocab_offset < 0 ||
      logits_stride < int64_t(vocab_offset) + N || int64_t(owners) * rows_per_owner < M)
    return invalid("scattered head arguments");
  HeadArgs p{};
  p.a_scale = a_scale; p.w_scale = w_scale; p.logits = nullptr; p.ldl = logits_stride;
  p.M = M; p.N = N; p.K = K; p.error_flag = error_flag;
  p.rows_per_owner = rows_per_owner; p.col_offset = vocab_offset;
  p.owner_stats_offset = stats_offset_bytes;
  for (int r = 0; r < owners; ++r) {
    if (!owner_logits[r] && int64_t(r) * rows_per_owner < M) return invalid("scattered head: null owner buffer");
    p.owner_base[r] = owner_logits[r];
  }
  return run_head(a_e4m3, a_scale, w_e4m3, w_scale, p, stream);
}

namespace {
int run_head(const void *a_e4m3, const float *a_scale, const void *w_e4m3, const float *w_scale, HeadArgs p,
             cudaStream_t stream) {
  (void)a_scale; (void)w_scale;
  const int M = p.M, N = p.N, K = p.K;
  if ((reinterpret_cast<uintptr_t>(a_e4m3) & 15u) || (reinterpret_cast<uintptr_t>(w_e4m3) & 15u))
    return invalid("head operands must be 16-byte aligned");
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return int(e);
  const int kblocks = K / kTileK;
  CUtensorMap mw, ma;
  // Three, five ... times 128 rows: what is behind the last whole pair tile would take half of one for its own, and goes to a launch
  // by itself instead, by the kernel of its size.  One launch / two, us with the quantiser (short runs at full clocks; in brackets the
  // 128 x 256 tiles before the pairs): 257 rows 275 / 234 (253), 300 rows 273 / 247 (253), 340 rows 277 / 266 (261), 384 rows 280 / 274
  // (268), 513 rows 416 / 360 (396), 640 rows 423 / 409 (420), 770 rows 555 / 507 (543), 880 rows 557 / 548 (565).  The rows of several
  // owners are cut the same way (eight owners, with the row records): 257 rows 294 / 244 (280), 384 rows 299 / 290 (289), 513 rows 452 /
  // 384 (432), 640 rows 455 / 434 (451), 770 rows 597 / 544 (587).
  if (M > 256 && ((M + 127) / 128 & 1)) {
    const int whole = M & ~255;
    HeadArgs rest = p;
    p.M = whole; rest.M = M - whole;
    rest.a_scale += size_t(whole) * (K / kTileK);
    if (p.rows_per_owner) rest.first_row = whole;   // (a row's owner follows from its place in the call)
    else rest.logits += size_t(whole) * p.ldl;
    if (rest.row_stats) rest.row_stats += whole;
    const int rc = run_head(a_e4m3, a_scale, w_e4m3, w_scale, p, stream);
    return rc ? rc : run_head(static_cast<const uint8_t *>(a_e4m3) + size_t(whole) * K, rest.a_scale, w_e4m3, w_scale, rest, stream);
  }
  if (M > 128) {
    if (!make_map(&mw, w_e4m3, uint64_t(N), uint64_t(K), 128, 1) || !make_map(&ma, a_e4m3, uint64_t(M), uint64_t(K), 128, 1))
      return invalid("cuTensorMapEncodeTiled failed");
    return int(launch_pairs(mw, ma, p, sms, stream));
  }
  const int rows = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  // K blocks per stage: the largest number that divides K/128 and still leaves a ring of at least 2 stages (longer contiguous
  // runs per weight row and fewer hand-overs beat a deeper ring of shorter stages; 64 rows take at most two, whose columns an epilogue
  // thread has the registers for)
  auto ring = [&](int g) {
    return rows == 16 ? DecodeSmem<16>::stages(kblocks, g) : rows == 32 ? DecodeSmem<32>::stages(kblocks, g)
         : rows == 64 ? DecodeSmem<64>::stages(kblocks, g) : HeadSmem::stages(kblocks, g);
  };
  int group = 1;
  const int most = rows == 64 ? DecodeSmem<64>::kMaxGroup : 4;
  for (int g = most; g > 1; g >>= 1)
    if (kblocks % g == 0 && ring(g) >= 2) { group = g; break; }
  p.group = group;
  if (!make_map(&mw, w_e4m3, uint64_t(N), uint64_t(K), 128, uint32_t(group)) ||
      !make_map(&ma, a_e4m3, uint64_t(M), uint64_t(K), uint32_t(rows), uint32_t(group)))
    return invalid("cuTensorMapEncodeTiled failed");
  switch (rows) {
    case 16: e = launch_decode<16>(mw, ma, p, sms, stream); break;
    case 32: e = launch_decode<32>(mw, ma, p, sms, stream); break;
    case 64: e = launch_decode<64>(mw, ma, p, sms, stream); break;
    default: e = launch_head(mw, ma, p, sms, stream); break;
  }
  return int(e);
}
}  // namespace

extern "C" size_t ds41_fuse_head_fp8_workspace_bytes(int M, int K) {
  if (M < 1 || K < 128 || K % 128) return 0;
  return ((size_t(M) * K + 255) & ~size_t(255)) + size_t(M) * (K / 128) * sizeof(float);
}

extern "C" int ds41_fuse_head_fp8(const void *x_bf16, const void *w_e4m3, const float *w_scale, float *logits, int M,
                                  int N, int K, void *workspace, size_t workspace_bytes, int *error_flag,
                                  cudaStream_t stream) {
  const size_t need = ds41_fuse_head_fp8_workspace_bytes(M, K);
  if (!need || !workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 255u))
    return invalid("head workspace too small or misaligned");
  uint8_t *a = static_cast<uint8_t *>(workspace);
  float *a_scale = reinterpret_cast<float *>(a + ((size_t(M) * K + 255) & ~size_t(255)));
  int rc = ds41_b200_quantize_activations(x_bf16, a, a_scale, M, K, stream);
  if (rc) return rc;
  return ds41_b200_head_fp8(a, a_scale, w_e4m3, w_scale, logits, N, M, N, K, error_flag, stream);
}
