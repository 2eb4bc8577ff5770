// Contraction on the 5th-generation tensor cores (tcgen05) for 16-bit floats with f32 accumulation in tensor memory:
//   out[m, n] = sum_k lhs[m, k] * rhs[k, n]        lhs k-contiguous; rhs n-contiguous ([k, n]) or k-contiguous ([n, k])
//
// The product is computed transposed, D^T[n, m] = W^T[n, k] . x^T[k, m]: the 128-row side of the MMA is the weight's
// n axis and the cheap N side (16..256) is m. One decode row, a batch of 32 rows or a 256-row prefill tile all use
// the same kernel; a small m costs a narrow MMA instead of a padded 128-row one, and no CUDA-core FMA work is left on
// the SM, so for small m the kernel is a pure HBM stream: TMA in, tensor core, a tiny epilogue.
//
// Work decomposition: a thread-block cluster of `ksplit` CTAs (1..8, one or two CTAs per SM) owns a tile of 128 columns x m_tile
// rows and walks tiles c, c + clusters, ...; each of its CTAs contracts 1/ksplit of k. The partial accumulators are
// summed through distributed shared memory: every CTA sends the rows that CTA r finishes to CTA r, counts itself in on
// r's mbarrier, and sums what it received itself in rank order (run-to-run identical results). Nothing goes through
// global memory and no CTA waits for another cluster. The host chooses m_tile and ksplit with a model of the HBM time,
// the per-SM rate and the number of waves (umma_choose in dot.cu).
// This replaced equal shares of 64-deep units per CTA with f32 partials in global memory and a fold by the CTA that
// arrived last: there every launch paid its HBM time plus 14 to 21 us, 7 us of them the tail (partials out, arrival
// counter, two dependent rounds of loads through one SM). Measured per launch, before and now (events around a graph
// node, the events' own time taken off): 32 rows, bf16, 4096 x 6144 22.5 / 18 us, 4096 x 4096 22.2 / 15.6 us, 14336 x 4096
// 34.4 / 28 us, 4096 x 28672 49 / 42 us, 4096 x 128256 170 / 163 us; 16 rows, int8, 4096 x 28672 49.2 / 40 us, 4096 x 128256
// 180 / 122 us. What is left at these sizes is the launch itself (set-up, first copies, sum, exit: 8 to 10 us) and, above it,
// HBM.
//
// Roles of a CTA:
//   producer lane   per unit (one [128 n x 64*SUB k] weight block + the matching [m_tile x 64*SUB] activation block),
//                   tiled TMA copies with the 128-byte swizzle into a ring of shared-memory stages; completion is
//                   counted on the stage's `full` mbarrier
//   MMA lane        4*SUB tcgen05.mma.cta_group::1.kind::f16 (M=128, N=m_tile, K=16) per stage, operands read through
//                   shared-memory descriptors, accumulator in TMEM (two accumulators, so the epilogue of one tile
//                   overlaps the MMAs of the next); tcgen05.commit releases the stage (`empty`) and, after a
//                   tile's last MMA, publishes the accumulator (`acc_full`)
//   epilogue warps  tcgen05.ld of the 128 x m_tile accumulator (TMEM lane = n, one per thread), the cluster's sum, the
//                   converted output
//   converter warps (sources other than kTile) write the weight operand straight into TMEM, from where tcgen05.mma
//                   takes its A side as well: the 16-bit values never occupy shared memory
//
// Weight sources (template parameter SRC):
//   kTile    16-bit weights whose rows TMA can copy (16-byte pitch): swizzled tiles in shared memory
//   kBytes   int8 weights with a 16-byte pitch and one f16 scale per column, the program's convert(s8 -> f16) * scale
//            [-> bf16] feeding the contraction. The weights stay one byte wide in HBM; a stage receives the raw bytes
//            and eight converter warps turn them into the integers (exact in either 16-bit type) in TMEM; the epilogue
//            multiplies each accumulator by its column's scale in f32. That is the contraction the program wrote with
//            the scale moved out of the sum: sum_k x[k] * (w[k,n] * s[n]) = s[n] * sum_k x[k] * w[k,n]. The op-by-op
//            program rounds every w * s to the element type first; this form skips that rounding (one relative 2^-9 per
//            weight at bf16), so the two agree to rounding, not bit for bit, and a product w * s that overflows f16 in
//            the written program stays finite here.
//            Converting into shared memory instead moved 110 KB through it per 128-deep stage (1630 cycles on the
//            4096 x 128256 LM head, where HBM needs 715); through TMEM it is 36 KB.
//   kLoose   16-bit weights of any pitch and alignment (an odd vocabulary, say): converter warps read them with plain
//            loads, one column per thread, and write them to TMEM. TMA cannot describe such rows. 5 x 2048 x 32001 f16: 85 us
//            (one thread per output before: 739), 1.6 TB/s; the converters' ALU is 65 % busy and waits for 2-byte loads.
//
// Programmatic dependent launch: weights are never written by earlier work of the stream (`early_rhs`), so their
// copies for the first ring of stages are issued before griddepcontrol.wait; activation copies and all stores wait.
// Dependents are released only after the tensor-memory allocation: a successor's CTA that moved in first could
// otherwise take the tensor memory this one is about to ask for and then wait for this grid.
//
// Every mbarrier wait is bounded by time (`timeout_ns` per launch, two seconds by default; the thread that sees the deadline pass sets a CTA-wide
// abort word and every other wait gives up at its next check); the kernel then sets *error_flag, every role falls
// through to the common exit, the allocating warp frees its tensor memory, and the kernel returns. CTAs of a cluster
// leave together, so nobody writes into the shared memory of a CTA that is gone. Cluster barriers have no limit of their own:
// like __syncthreads they end because every way to them is bounded.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace pjrtx {
namespace umma {

constexpr int kGroupMax = 4;
constexpr int kTileN = 128;          // weight columns per tile (MMA M)
constexpr int kSubK = 64;            // k elements per swizzle row (128 bytes of 16-bit data)
constexpr int kSplitMax = 8;         // CTAs of a cluster (the portable limit)
constexpr int kBaseThreads = 192;    // warps 0-3 epilogue, warp 4 TMA producer, warp 5 MMA issuer

enum Source { kTile = 0, kBytes = 1, kLoose = 2 };
// Converter warps (from warp 6 on): four per quarter of the 128 columns where the loads come from global memory (the
// bytes in flight are theirs), two where TMA brings the bytes.
__host__ __device__ constexpr int converter_warps(int src) { return src == kTile ? 0 : src == kBytes ? 8 : 16; }
__host__ __device__ constexpr int threads_of(int src) { return kBaseThreads + 32 * converter_warps(src); }
// Weight operand tiles in TMEM (sources other than kTile), 32 * SUB columns each.
constexpr int kOperandSlots = 3;

struct Params {
  int m, k;
  int m_tile;            // MMA N: multiple of 16, 16..256 (at most 128 when the weight operand lives in TMEM)
  int m_tiles;           // ceil(m / m_tile)
  int count;             // contractions sharing lhs
  int tile_begin[kGroupMax + 1];  // prefix sums of (n tiles * m tiles) over the group
  void* out[kGroupMax];
  long long n[kGroupMax];
  long long ldo[kGroupMax];       // out row stride in elements
  int kblocks;           // ceil(k / (64 * SUB))
  int tiles;             // all tiles of the launch
  int ksplit;            // CTAs per cluster; CTA r of a cluster contracts k blocks [r*kblocks/ksplit, (r+1)*kblocks/ksplit)
  int rows_per_rank;     // m_tile / ksplit, rounded up to a multiple of 4: rows of a tile that one CTA of the cluster finishes
  int sum_buffers;       // 1 or 2 (a cluster with several tiles): receive buffers for the cluster's sum
  int* error_flag;
  unsigned long long timeout_ns;  // budget of the launch for all of its waits
  int stages;
  int is_bf16;
  int rhs_k_major;       // 1: rhs is [n, k] with k contiguous
  int rhs_3d;            // rhs [k, n] with n % 64 == 0: one copy per stage through a 3-d view {64 n, k, n / 64}
  int early_rhs;         // rhs copies may start before the preceding kernel of the stream has finished
  const void* scale[kGroupMax];  // int8: f16 scale per weight column
  const void* rhs[kGroupMax];    // kLoose
  long long rhs_pitch[kGroupMax];
};

struct Maps {
  // kTile [k, n]: dims {n, k}, box {64, 64*SUB}, or (rhs_3d) dims {64, k, n/64}, box {64, 64*SUB, 2};
  // kTile [n, k]: dims {k, n}, box {64, 128}; kBytes: dims {n, k}, box {128, 64*SUB}
  CUtensorMap rhs[kGroupMax];
  CUtensorMap lhs;             // dims {k, m}, box {64, m_tile}
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Deadline of the launch (every thread reads the timer when it starts) and the CTA's abort word in shared memory.
struct WaitBudget {
  unsigned long long deadline;
  volatile int* abort;
};
// Bounded by time: gives up when the launch's deadline has passed or another thread of the CTA already gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, const WaitBudget& w) {
  for (unsigned spin = 0;; spin++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 15) == 15) {
      if (*w.abort) return false;
      if (global_timer_ns() > w.deadline) {
        *w.abort = 1;
        return false;
      }
    }
  }
}
// x = innermost coordinate (always a multiple of 64 elements here, i.e. 128 bytes), y = outer coordinate.
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   smem_dst),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
// The same with an L2 eviction policy.
__device__ __forceinline__ void tma_load_2d_hint(uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(
          smem_dst),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_hint(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(
          smem_dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// AND of a predicate over the 128 epilogue threads (named barrier 1), so that all four warps take the same branch
// around the warp-collective TMEM loads and the named barriers that follow.
__device__ __forceinline__ bool epilogue_all(bool ok) {
  unsigned out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(out)
      : "r"((unsigned)ok)
      : "memory");
  return out != 0;
}

// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte offsets in 16-byte units,
// descriptor version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t smem_addr, uint32_t leading_bytes, uint32_t stride_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fff);
  d |= (uint64_t)((leading_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((stride_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;  // version
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16: f32 accumulate, B (activations) K-major.
__host__ __device__ inline uint32_t instr_desc(int is_bf16, int mma_n, int a_mn_major) {
  uint32_t d = 0;
  d |= 1u << 4;                                // D format f32
  d |= (uint32_t)(is_bf16 ? 1 : 0) << 7;       // A format
  d |= (uint32_t)(is_bf16 ? 1 : 0) << 10;      // B format
  d |= (uint32_t)(a_mn_major ? 1 : 0) << 15;   // A major: MN (weights [k, n]) or K (weights [n, k], operand in TMEM)
  d |= (uint32_t)(mma_n >> 3) << 17;
  d |= (uint32_t)(kTileN >> 4) << 24;
  return d;
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// The same with the A operand (128 rows x 16 k: eight 32-bit columns, one row per lane) in tensor memory.
__device__ __forceinline__ void mma_f16_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Thread-block cluster: shared-memory address of the same variable in CTA `rank`, remote arrive, and a wait that sees
// what the arriving CTAs wrote before.
__device__ __forceinline__ uint32_t cluster_address(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_arrive(uint32_t remote_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
}
__device__ __forceinline__ bool cluster_wait(uint64_t* bar, unsigned parity, const WaitBudget& w) {
  for (unsigned spin = 0;; spin++) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((spin & 15) == 15) {
      if (*w.abort) return false;
      if (global_timer_ns() > w.deadline) {
        *w.abort = 1;
        return false;
      }
    }
  }
}

// A stage of the ring: the weight tile (16-bit and swizzled, or raw bytes, or nothing) and the activation tile behind it.
__host__ __device__ constexpr uint32_t weight_stage_bytes(int src, int sub) {
  return src == kTile ? (uint32_t)sub * 16384u : src == kBytes ? (uint32_t)sub * 8192u : 0u;
}
__host__ __device__ inline size_t stage_bytes(int m_tile, int sub, int src) {
  return (size_t)sub * m_tile * 128 + weight_stage_bytes(src, sub);
}
// Receive buffers of the cluster's sum: [buffer][source CTA][four rows][128 columns][4 rows] f32 (rows_per_rank is a
// multiple of four).
__host__ __device__ inline size_t sum_bytes(int ksplit, int rows_per_rank, int buffers) {
  return ksplit > 1 ? (size_t)buffers * ksplit * rows_per_rank * kTileN * 4 : 0;
}
constexpr size_t kBarrierBytes = 512;
// Two accumulators of m_tile f32 columns, then the operand slots; an allocation is a power of two >= 32 columns.
__host__ __device__ inline uint32_t tmem_columns(int m_tile, int sub, int src) {
  uint32_t cols = 32;
  while (cols < 2u * m_tile + (src == kTile ? 0u : kOperandSlots * 32u * sub)) cols <<= 1;
  return cols;
}
// An SM's tensor memory (512 columns) must hold the allocations of all CTAs that fit its shared memory (228 KiB, 1 KiB of
// it per CTA reserved), whichever kernels they belong to: a CTA whose allocation blocks could keep its cluster waiting. A
// CTA of at most 256 columns asks for at least 80 KiB (two fit, three do not; kSharedSmem is the most two can have), one of
// more columns for at least 150 KiB (nothing else that allocates tensor memory fits beside it).
constexpr size_t kSharedSmem = 113 * 1024;
__host__ __device__ constexpr size_t least_smem(uint32_t tmem_cols) { return (tmem_cols <= 256 ? 80 : 150) * 1024; }
inline size_t smem_bytes(int stages, int m_tile, int sub, int src, size_t sum) {
  // stages (every block 1024-byte aligned: m_tile is a multiple of 16, so m_tile * 128 is a multiple of 2048) +
  // receive buffers + barriers and flags + slack for aligning the dynamic segment to 1024 bytes.
  const size_t bytes = (size_t)stages * stage_bytes(m_tile, sub, src) + sum + kBarrierBytes + 1024;
  const size_t least = least_smem(tmem_columns(m_tile, sub, src));
  return bytes < least ? least : bytes;
}

struct Tile {
  int group, n_tile, m_idx;
};
__device__ __forceinline__ Tile locate_tile(const Params& p, int tile) {
  int g = 0;
#pragma unroll
  for (int q = 1; q < kGroupMax; q++)
    if (q < p.count && tile >= p.tile_begin[q]) g = q;
  const int t = tile - p.tile_begin[g];
  const int n_tile = t / p.m_tiles;
  return Tile{g, n_tile, t - n_tile * p.m_tiles};
}

// Four signed bytes -> four integers in the 16-bit type, two per word, exactly.
__device__ __forceinline__ void widen_bytes(uint32_t word, int is_bf16, uint32_t* packed) {
  if (is_bf16) {
    // b = low7 - 128 * sign. {0x43, low7} is the bf16 128 + low7 and {0x43, sign << 7} is 128 or 256: their difference
    // is b, exactly.
    const uint32_t low7 = word & 0x7f7f7f7fu, sign = word & 0x80808080u;
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const uint32_t sel = e ? 0x4342 : 0x4140;
      const uint32_t x = __byte_perm(low7, 0x43434343u, sel), y = __byte_perm(sign, 0x43434343u, sel);
      const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
      packed[e] = *reinterpret_cast<const uint32_t*>(&v);
    }
  } else {
    // {0x64, b + 128} is the f16 1024 + 128 + b.
    const uint32_t flipped = word ^ 0x80808080u;
    const __half2 bias = __float2half2_rn(1152.0f);
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const uint32_t x = __byte_perm(flipped, 0x64646464u, e ? 0x4342 : 0x4140);
      const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&x), bias);
      packed[e] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
}

// Sixteen registers per thread: 32 lanes (one per thread) x 16 columns.
__device__ __forceinline__ void tmem_store_rows(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Four 16-lane x 8-column blocks next to each other: of every four registers, 0 and 1 go to lane t/4, columns 2*(t%4) and
// + 1; 2 and 3 to lane t/4 + 8.
__device__ __forceinline__ void tmem_store_blocks(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// SUB: 64-deep k sub-blocks per stage (1 or 2; the sources other than kTile use 2).
// The converters' bounds spill: 68 bytes at 72 registers for kBytes, the price of two CTAs of 448 threads per SM (one cannot
// keep the chain of copy, conversion and MMA full); 136 bytes at 80 for kLoose, whose 704 threads leave no more. Neither was
// timed without its spills. kTile has none.
template <int SUB, int SRC>
__global__ void __launch_bounds__(threads_of(SRC), SRC == kLoose ? 1 : 2) umma_stream_kernel(const Params p, const __grid_constant__ Maps maps) {
  extern __shared__ unsigned char smem_dyn[];
  // 128-byte swizzled tiles need 1024-byte aligned bases.
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  constexpr uint32_t w_bytes = weight_stage_bytes(SRC, SUB);  // a stage is [weight tile][activation tile]
  constexpr bool kTmemA = SRC != kTile;
  constexpr int kDepth = kSubK * SUB;  // k elements per unit
  const uint32_t per_stage = (uint32_t)stage_bytes(p.m_tile, SUB, SRC);
  float* sums = reinterpret_cast<float*>(base_ptr + (size_t)p.stages * per_stage);
  uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(sums) + sum_bytes(p.ksplit, p.rows_per_rank, p.sum_buffers));
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;   // [2]
  uint64_t* acc_empty = acc_full + 2;      // [2]
  uint64_t* sum_full = acc_empty + 2;      // [2] every CTA of the cluster has delivered its part of this CTA's rows
  uint64_t* ready = sum_full + 2;          // [kOperandSlots] the converters have written the slot's operand
  uint64_t* slot_empty = ready + kOperandSlots;  // [kOperandSlots] the MMAs that read the slot have completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(slot_empty + kOperandSlots);
  int* flags = reinterpret_cast<int*>(tmem_slot + 1);  // [0] abort
  const WaitBudget budget{global_timer_ns() + p.timeout_ns, flags};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ksplit = p.ksplit;
  const int cluster = (int)blockIdx.x / ksplit, rank = (int)blockIdx.x - cluster * ksplit, clusters = (int)gridDim.x / ksplit;
  const int kb_begin = (int)((long long)rank * p.kblocks / ksplit), kb_end = (int)((long long)(rank + 1) * p.kblocks / ksplit);
  const int my_tiles = cluster < p.tiles ? (p.tiles - 1 - cluster) / clusters + 1 : 0;
  const int count = my_tiles * (kb_end - kb_begin);  // units of this CTA
  const uint32_t tmem_cols = tmem_columns(p.m_tile, SUB, SRC);

  if (threadIdx.x == 4 * 32) {
    for (int g = 0; g < p.count && (SRC == kTile || SRC == kBytes); g++) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.rhs[g]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.lhs) : "memory");
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < kOperandSlots; s++) {
      mbar_init(&ready[s], kTmemA ? converter_warps(SRC) : 1);
      mbar_init(&slot_empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
      mbar_init(&sum_full[b], 4u * ksplit);
    }
    flags[0] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Weights are read once per tile row: evict-first, so that they do not push activations and caches out of L2.
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  auto load_rhs = [&](const Tile& t, int kb, int stage) {
    const uint32_t st = base + (uint32_t)stage * per_stage;
    const int k0 = kb * kDepth, n0 = t.n_tile * kTileN;
    if (SRC == kBytes) {
      tma_load_2d_hint(st, &maps.rhs[t.group], n0, k0, &full[stage], policy);  // [64 * SUB k rows][128 bytes], swizzled
    } else if (SRC == kTile) {
      if (p.rhs_3d) {
        // Blocks of 64 columns are the outer coordinate: the box lands as [column block][k row][128 bytes], which
        // is the layout the two-box form produces, in one copy of 16 * SUB KiB.
        tma_load_3d_hint(st, &maps.rhs[t.group], 0, k0, n0 / 64, &full[stage], policy);
      } else if (p.rhs_k_major) {
#pragma unroll
        for (int s = 0; s < SUB; s++) tma_load_2d_hint(st + s * 16384u, &maps.rhs[t.group], k0 + s * kSubK, n0, &full[stage], policy);
      } else {
        tma_load_2d_hint(st, &maps.rhs[t.group], n0, k0, &full[stage], policy);
        tma_load_2d_hint(st + SUB * 8192u, &maps.rhs[t.group], n0 + 64, k0, &full[stage], policy);
      }
    }
  };
  // The weights of the first ring are requested before anything else: they depend on nothing.
  const int first = p.early_rhs ? min(count, p.stages) : 0;
  if (threadIdx.x == 4 * 32) {
    int tile = cluster, kb = kb_begin;
    for (int i = 0; i < first; i++) {
      const Tile t = locate_tile(p, tile);
      mbar_expect_tx(&full[i], per_stage);
      load_rhs(t, kb, i);
      if (++kb == kb_end) {
        kb = kb_begin;
        tile += clusters;
      }
    }
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t operand_base = tmem_base + 2u * p.m_tile;
  // The cluster's CTAs have initialised their barriers: waited for only before the first remote access and at the exit.
  if (ksplit > 1) asm volatile("barrier.cluster.arrive.release;" ::: "memory");

  if (warp == 4) {
    // ---- TMA producer ------------------------------------------------------------------------------------------
    if (lane == 0 && count > 0) {
      auto load_lhs = [&](const Tile& t, int kb, int stage) {
        const uint32_t st = base + (uint32_t)stage * per_stage + w_bytes;
#pragma unroll
        for (int s = 0; s < SUB; s++)
          tma_load_2d(st + (uint32_t)s * p.m_tile * 128u, &maps.lhs, kb * kDepth + s * kSubK, t.m_idx * p.m_tile, &full[stage]);
      };
      asm volatile("griddepcontrol.wait;" ::: "memory");
      int tile = cluster, kb = kb_begin, stage = 0;
      unsigned phase = 0;
      Tile t = locate_tile(p, tile);
      for (int i = 0; i < count; i++) {
        if (i >= first) {
          if (i >= p.stages && !mbar_wait(&empty[stage], phase ^ 1, budget)) {
            atomicExch(p.error_flag, 11);
            // Nothing more is requested; the copies in flight get a bounded time to land before the CTA leaves.
            for (int b = 1; b <= p.stages; b++) {
              const int j = i - b;  // the last unit requested into each stage
              for (unsigned spin = 0; spin < (1u << 16) && !mbar_try_wait(&full[j % p.stages], (unsigned)(j / p.stages) & 1u); spin++) {
              }
            }
            break;
          }
          mbar_expect_tx(&full[stage], per_stage);
          load_rhs(t, kb, stage);
        }
        load_lhs(t, kb, stage);
        if (++kb == kb_end) {
          kb = kb_begin;
          tile += clusters;
          if (tile < p.tiles) t = locate_tile(p, tile);
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 5) {
    // ---- MMA issuer ----------------------------------------------------------------------------------------------
    if (lane == 0 && count > 0) {
      const uint32_t idesc = instr_desc(p.is_bf16, p.m_tile, !kTmemA && !p.rhs_k_major);
      int stage = 0, slot = 0;
      unsigned phase = 0, slot_phase = 0;
      bool ok = true;
      for (int seg = 0; seg < my_tiles && ok; seg++) {
        // Take the next accumulator once the epilogue has drained its previous use.
        const int buf = seg & 1;
        if (seg >= 2 && !mbar_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, budget)) {
          atomicExch(p.error_flag, 14);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + (uint32_t)(buf * p.m_tile);
        for (int kb = kb_begin; kb < kb_end; kb++) {
          // The copies of the stage have landed; the converters have also filled the slot.
          if (!mbar_wait(&full[stage], phase, budget) || (kTmemA && !mbar_wait(&ready[slot], slot_phase, budget))) {
            atomicExch(p.error_flag, 12);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t st = base + (uint32_t)stage * per_stage;
#pragma unroll
          for (int kk = 0; kk < 4 * SUB; kk++) {
            const uint64_t b_desc = smem_desc(st + w_bytes + (uint32_t)(kk >> 2) * p.m_tile * 128u + (kk & 3) * 32u, 16, 1024);
            const uint32_t accumulate = (kb == kb_begin && kk == 0) ? 0u : 1u;
            if (kTmemA) {
              mma_f16_tmem_a(acc, operand_base + (uint32_t)(slot * 32 * SUB + kk * 8), b_desc, idesc, accumulate);
            } else if (p.rhs_k_major) {
              // A K-major like B: 64-k sub-blocks 16 KiB apart, 32 bytes per 16-k step inside the swizzled row.
              mma_f16(acc, smem_desc(st + (kk >> 2) * 16384u + (kk & 3) * 32u, 16, 1024), b_desc, idesc, accumulate);
            } else {
              // A MN-major: 16 k rows = two 1024-byte swizzle atoms further down; the two 64-column boxes are
              // SUB * 8192 bytes apart (leading offset), 8-row groups 1024 bytes apart (stride offset).
              mma_f16(acc, smem_desc(st + kk * 2048u, SUB * 8192u, 1024), b_desc, idesc, accumulate);
            }
          }
          mma_commit(&empty[stage]);  // the stage is free once these MMAs have read it
          if (kTmemA) {
            mma_commit(&slot_empty[slot]);  // and so is the operand slot
            if (++slot == kOperandSlots) {
              slot = 0;
              slot_phase ^= 1;
            }
          }
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) mma_commit(&acc_full[buf]);
      }
    }
  } else if (kTmemA && warp >= 6) {
    // ---- converters: weights -> 16-bit operand in TMEM (lane = weight column, 32-bit column = two consecutive k) ----
    // A warp can reach the 32 TMEM lanes of its quarter (warp % 4) only.
    const int quarter = warp & 3, part = (warp - 6) >> 2;
    const uint32_t quarter_addr = (uint32_t)(quarter * 32) << 16;
    int stage = 0, slot = 0;
    unsigned phase = 0, slot_phase = 0;
    auto slot_free = [&](int i) { return i < kOperandSlots || mbar_wait(&slot_empty[slot], slot_phase ^ 1, budget); };
    auto publish = [&]() {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[slot]);
      if (++slot == kOperandSlots) {
        slot = 0;
        slot_phase ^= 1;
      }
    };
    if constexpr (SRC == kBytes) {
      // A thread owns the 4 adjacent columns 4 * (lane / 4) .. + 3 of its warp's 32 and, of every 16-row step, the rows
      // 4 * (lane % 4) .. + 3: four 32-bit reads; byte permutes pair up the bytes of rows 0 and 1, 2 and 3 of a column,
      // and each column's four k values are the two words the 16-lane store wants from this thread. Column 4 * c + j of the
      // warp lands in TMEM lane 8 * j + c. (The bytes are in the 128-byte swizzle, 16-byte chunk ^= row % 8: lanes of
      // rows 8 apart share a bank, two reads per request. Reading those rows in another order avoids that, but the selects it
      // takes cost more than the reads: the ALU, 28 permutes and masks per 16 bytes, is what limits the converters.)
      const int c = lane >> 2, q = lane & 3;
      const int word = quarter * 8 + c;  // of the 32 words of a row
      const uint32_t chunk = (uint32_t)(word >> 2), in_chunk = (uint32_t)(word & 3) * 4u;
      for (int i = 0; i < count; i++) {
        const bool ok = mbar_wait(&full[stage], phase, budget) && slot_free(i);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) atomicExch(p.error_flag, 15);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned char* raw = base_ptr + (size_t)stage * per_stage;
        const uint32_t dst = operand_base + quarter_addr + (uint32_t)(slot * 32 * SUB);
        uint32_t w[2 * SUB][4];  // every word of this thread is requested before the first is converted
#pragma unroll
        for (int s = 0; s < 2 * SUB; s++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int row = (part * 2 * SUB + s) * 16 + 4 * q + e;
            w[s][e] = *reinterpret_cast<const uint32_t*>(raw + row * 128 + ((chunk ^ (uint32_t)(row & 7)) << 4) + in_chunk);
          }
        static_assert(SRC != kBytes || SUB == 2, "four 16-row steps per warp and unit");
        const uint32_t at = dst + (uint32_t)(part * 16 * SUB);
#pragma unroll
        for (int half = 0; half < 2; half++) {  // lanes 0-15 and 16-31 of the quarter
          uint32_t v[16];
#pragma unroll
          for (int s = 0; s < 2 * SUB; s++) {
            uint32_t lo[2], hi[2];  // rows 0, 1 and rows 2, 3 of two columns
            widen_bytes(__byte_perm(w[s][0], w[s][1], half ? 0x7362 : 0x5140), p.is_bf16, lo);
            widen_bytes(__byte_perm(w[s][2], w[s][3], half ? 0x7362 : 0x5140), p.is_bf16, hi);
            v[4 * s] = lo[0];
            v[4 * s + 1] = hi[0];
            v[4 * s + 2] = lo[1];
            v[4 * s + 3] = hi[1];
          }
          tmem_store_blocks(at + (half ? 16u << 16 : 0u), v);
        }
        publish();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    } else if constexpr (SRC == kLoose) {
      // One column per thread, 16 * SUB rows per unit; the next unit's loads are in flight while this one is converted.
      constexpr int R = 16 * SUB;
      if (!p.early_rhs) asm volatile("griddepcontrol.wait;" ::: "memory");  // (returns at once: these launches are ordered)
      int tile = cluster, kb = kb_begin;
      Tile t = locate_tile(p, min(tile, p.tiles - 1));
      unsigned short next[R];
      auto request = [&]() {
        const long long n = (long long)t.n_tile * kTileN + quarter * 32 + lane;
        const int k0 = kb * kDepth + part * R;
        const long long pitch = p.rhs_pitch[t.group];
        const unsigned short* src = static_cast<const unsigned short*>(p.rhs[t.group]) + (long long)k0 * pitch + n;
        const bool in = n < p.n[t.group];
        const int rows = p.k - k0;
#pragma unroll
        for (int r = 0; r < R; r++) {
          next[r] = (in && r < rows) ? __ldg(src) : (unsigned short)0;
          src += pitch;
        }
        if (++kb == kb_end) {
          kb = kb_begin;
          tile += clusters;
          if (tile < p.tiles) t = locate_tile(p, tile);
        }
      };
      if (count > 0) request();
      for (int i = 0; i < count; i++) {
        uint32_t packed[R / 2];
#pragma unroll
        for (int r = 0; r < R / 2; r++) packed[r] = (uint32_t)next[2 * r] | (uint32_t)next[2 * r + 1] << 16;
        if (i + 1 < count) request();
        const bool ok = slot_free(i);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) atomicExch(p.error_flag, 15);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_store_rows(operand_base + quarter_addr + (uint32_t)(slot * 32 * SUB + part * (R / 2)), packed);
        publish();
      }
    }
  } else if (warp < 4) {
    // ---- epilogue warps 0..3: TMEM lane quarter = warp index ------------------------------------------------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (ksplit > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    // The tile column whose values are in this thread's TMEM lane (kBytes writes its operand in that order).
    const int n_local = warp * 32 + (SRC == kBytes ? 4 * (lane & 7) + (lane >> 3) : lane);
    for (int seg = 0; seg < my_tiles; seg++) {
      const Tile t = locate_tile(p, cluster + seg * clusters);
      const int buf = seg & 1;
      // One decision for all four warps: tcgen05.ld is warp-collective.
      if (!epilogue_all(mbar_wait(&acc_full[buf], (seg >> 1) & 1, budget))) {
        if (threadIdx.x == 0) atomicExch(p.error_flag, 13);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const long long n = (long long)t.n_tile * kTileN + n_local;
      const bool in = n < p.n[t.group];
      const int m0 = t.m_idx * p.m_tile;
      const int m_rows = min(p.m_tile, p.m - m0);  // rows of this tile that exist
      const long long ldo = p.ldo[t.group];
      constexpr bool int8 = SRC == kBytes;
      // Int8 weights: the tensor core contracted the integers; this thread's column scale finishes the product.
      const float scale = int8 && in ? __half2float(static_cast<const __half*>(p.scale[t.group])[n]) : 1.f;
      auto store = [&](int row, float v) {
        if (int8) v *= scale;
        const long long at = (long long)(m0 + row) * ldo + n;
        if (p.is_bf16) static_cast<__nv_bfloat16*>(p.out[t.group])[at] = __float2bfloat16_rn(v);
        else static_cast<__half*>(p.out[t.group])[at] = __float2half_rn(v);
      };
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * p.m_tile);
      const int sum_buf = p.sum_buffers == 2 ? buf : 0;
      float* received = sums + (size_t)sum_buf * ksplit * p.rows_per_rank * kTileN;
      for (int c0 = 0; c0 < m_rows; c0 += 16) {
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (ksplit > 1) {
          // Rows go to the CTA that sums them, four of a column in one 16-byte store (512 contiguous bytes per warp).
          // Rows past m up to the tile's height are delivered too and not used.
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            const int owner = (c0 + j) / p.rows_per_rank, row = c0 + j - owner * p.rows_per_rank;
            const uint32_t at = cluster_address(smem_u32(received + ((size_t)rank * p.rows_per_rank + row) * kTileN + threadIdx.x * 4), (uint32_t)owner);
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3])
                         : "memory");
          }
        } else if (in) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (c0 + j < m_rows) store(c0 + j, __uint_as_float(r[j]));
        }
      }
      // The accumulator is in registers / memory now: hand it back to the MMA lane.
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      if (ksplit > 1) {
        // A receive buffer is written again two tiles later, after its writer has seen this CTA's arrivals for the tile
        // in between, which follow the reads below.
        if (lane == 0)
          for (int q = 0; q < ksplit; q++) cluster_arrive(cluster_address(smem_u32(&sum_full[buf]), (uint32_t)q));
        if (!epilogue_all(cluster_wait(&sum_full[buf], (seg >> 1) & 1, budget))) {
          if (threadIdx.x == 0) atomicExch(p.error_flag, 16);
          break;
        }
        const int row0 = rank * p.rows_per_rank;
        const int rows = min(p.rows_per_rank, m_rows - row0);
        const float4* src = reinterpret_cast<const float4*>(received) + threadIdx.x;
        const int source_stride = p.rows_per_rank / 4 * kTileN;
        for (int j = 0; j < rows; j += 4) {
          float4 v[kSplitMax];
#pragma unroll
          for (int q = 0; q < kSplitMax; q++)
            if (q < ksplit) v[q] = src[q * source_stride + j / 4 * kTileN];
#pragma unroll
          for (int q = 1; q < kSplitMax; q++)
            if (q < ksplit) {
              v[0].x += v[q].x;
              v[0].y += v[q].y;
              v[0].z += v[q].z;
              v[0].w += v[q].w;
            }
          if (in) {
            store(row0 + j, v[0].x);
            if (j + 1 < rows) store(row0 + j + 1, v[0].y);
            if (j + 2 < rows) store(row0 + j + 2, v[0].z);
            if (j + 3 < rows) store(row0 + j + 3, v[0].w);
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  if (ksplit > 1) {
    // First the barrier everyone arrived at in the beginning (the epilogue warps have waited for it), then the exit.
    if (warp >= 4) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

}  // namespace umma
}  // namespace pjrtx
