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
// What bounds it at the decode sizes is the launch itself (set-up, first copies, sum, exit: 7 to 9 us) and, above it, HBM.
//
// Who issues: the copy warp and the MMA warp run their loops converged and let one elected thread issue (elect_one; the copy
// warp of kLoose is the exception). With a single thread in those loops every operand of an issued instruction went through
// a vector register: the MMA lane needed 1380 cycles per 128-deep unit beside busy converters, of which the products take 370,
// and 570 per 64-deep unit without them. Launches one after the other, us, before and now: 32 rows bf16 4096 x 4096 16.5 / 14.8, 4096 x 6144 18.6 /
// 16.9, 14336 x 4096 30.2 / 27.4, 2048 x 14336 20.5 / 18.5, 7168 x 2048 16.8 / 14.7, 4096 x 28672 43.3 / 42.8 (HBM).
//
// Roles of a CTA:
//   copy warp       per unit (one [128 n x 64*SUB k] weight block + the matching [m_tile x 64*SUB] activation block),
//                   tiled TMA copies with the 128-byte swizzle into a ring of shared-memory stages; completion is
//                   counted on the stage's `full` mbarrier
//   MMA warp        4*SUB tcgen05.mma.cta_group::1.kind::f16 (M=128, N=m_tile, K=16) per stage, operands read through
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
//            4096 x 128256 LM head, where HBM needs 715); through TMEM it is 36 KB. The warps of a quarter take units in
//            turn, read them transposed (ldmatrix) and share the arithmetic out between the ALU and the packed units
//            (widen_byte_pair). 16 rows, us, before these and the issue above, and now: 4096 x 28672 40.9 / 33.3, 14336 x
//            4096 30.8 / 26.1, 8192 x 57344 114 / 94.5, 4096 x 128256 119.5 / 102 (5.2 TB/s).
//   kLoose   16-bit weights of any pitch and alignment (an odd vocabulary, say): converter warps read them with plain
//            loads, one column per thread, and write them to TMEM, at 1.7 TB/s: the converters' ALU is 65 % busy and waits for
//            2-byte loads. Few rows of large weights go by residues instead (umma_shift.cuh).
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
// Weight operand tiles in TMEM (sources other than kTile), 32 * SUB columns each. kBytes: a warp converts every second unit only
// and therefore sees every second phase of the barriers that the units in between share with its own, where a parity that is
// one phase behind counts as complete. What keeps it from that: unit i's slot is free once the products of unit i - kOperandSlots
// are done, so all units up to there have landed, and those are all earlier users of its stage that the warp has not waited
// for itself (a ring of two stages has its own units only). So a warp waits for the slot first, then for the stage.
constexpr int kOperandSlots = 3;
static_assert(kOperandSlots <= 3, "a ring of three stages relies on it");

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
// x = innermost coordinate (a multiple of 64 elements here, of 8 in umma_shift.cuh: 16 bytes), y = outer coordinate.
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

// Advanced by a number of bytes (a multiple of 16) inside shared memory: the start address is the descriptor's lowest field
// and does not run over into the next one.
__device__ __forceinline__ uint64_t desc_advance(uint64_t desc, uint32_t bytes) {
  return (desc & 0xffffffff00000000ull) | (uint32_t)((uint32_t)desc + (bytes >> 4));
}
// One thread of a converged warp. The MMA warps run their loops as a whole and let this thread issue: addresses and
// descriptors are then the same for the whole warp and sit in uniform registers, which the tcgen05 instructions want.
// With one thread of the warp in the loop an instruction took 120 cycles to issue and a 128-deep unit 1380 (its products
// take 370).
__device__ __forceinline__ bool elect_one() {
  unsigned one;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(one));
  return one != 0;
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
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with the A operand (128 rows x 16 k: eight 32-bit columns, one row per lane) in tensor memory.
__device__ __forceinline__ void mma_f16_tmem_a(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
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

// Bytes J and J + 2 of a word of signed bytes -> the two integers in the 16-bit type, exactly, byte J in the low half.
// f16: with its top bit flipped a byte is u = b + 128, and {0x64, u} is 1024 + u: one three-input logic operation masks,
// flips and adds the exponent (behind a shift for J = 1), one packed subtraction takes the constant away.
// bf16 has seven fraction bits, and two ways that load the ALU and the packed multiply-add units differently (both issue every
// second cycle): J = 0 takes one logic operation and three packed, J = 1 a shift, two and one, which balances the two (16 x
// 4096 x 128256: 103 us; the first way for both 120, the second 117; f16 101).
//   J = 0: {0x43, u} is v = 128 + u below 128 and 2 * u from there on; with r = v / 2 - 128, b is r where r >= 0 and 2 * r
//          below: r - max(-r, 0). Every step is exact in eight significant bits.
//   J = 1: {0x43, low seven bits} is 128 + low and {0x43, top bit} is 128 or 256: their difference is b.
template <int J, bool BF16>
__device__ __forceinline__ uint32_t widen_byte_pair(uint32_t word) {
  if (!BF16) {
    const uint32_t x = ((J ? word >> 8 : word) & 0x00ff00ffu) ^ 0x64806480u;
    const __half2 b = __hsub2(*reinterpret_cast<const __half2*>(&x), __float2half2_rn(1152.0f));
    return *reinterpret_cast<const uint32_t*>(&b);
  }
  __nv_bfloat162 b;
  if (J == 0) {
    const uint32_t x = (word & 0x00ff00ffu) ^ 0x43804380u;
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&x);
    const __nv_bfloat162 half = __float2bfloat162_rn(0.5f), bias = __float2bfloat162_rn(128.0f);
    b = __hsub2(__hfma2(v, half, __hneg2(bias)), __hfma2_relu(v, __hneg2(half), bias));
  } else {
    const uint32_t high = word >> 8, x = (high & 0x007f007fu) | 0x43004300u, y = (high & 0x00800080u) | 0x43004300u;
    b = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
  }
  return *reinterpret_cast<const uint32_t*>(&b);
}

// Sixteen registers per thread: 32 lanes (one per thread) x 16 columns.
__device__ __forceinline__ void tmem_store_rows(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Eight 16-lane x 4-column blocks next to each other: registers 2 * i and 2 * i + 1 of thread t go to lanes t / 4 and
// t / 4 + 8, column 4 * i + t % 4.
__device__ __forceinline__ void tmem_store_blocks(uint32_t addr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Four 8 x 8 blocks of 16-bit units, transposed: thread t gets units [2 * (t % 4)][t / 4] and [2 * (t % 4) + 1][t / 4] of each
// block, whose rows start at the addresses of threads 8 * block .. + 7.
__device__ __forceinline__ void load_blocks_transposed(uint32_t (&w)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
               : "r"(addr)
               : "memory");
}

// One warp's share of a unit of 128 k x 128 columns of signed bytes: the 32 columns of its quarter. `row`: shared-memory
// address of the lane's row among the first 32.
template <bool BF16>
__device__ __forceinline__ void convert_unit(uint32_t row, int quarter, int lane, uint32_t dst) {
  uint32_t w[8][4];  // 32 rows each; the first four are of lanes 0-15 of the quarter, the others of 16-31
#pragma unroll
  for (int i = 0; i < 8; i++)
    load_blocks_transposed(w[i], row + (((uint32_t)(quarter * 2 + (i >> 2)) ^ (uint32_t)(lane & 7)) << 4) + (uint32_t)(i & 3) * 4096u);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t v[16];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      v[2 * i] = widen_byte_pair<0, BF16>(w[2 * q + (i >> 2)][i & 3]);
      v[2 * i + 1] = widen_byte_pair<1, BF16>(w[2 * q + (i >> 2)][i & 3]);
    }
    tmem_store_blocks(dst + (uint32_t)((q & 1) * 32) + (q >> 1 ? 16u << 16 : 0u), v);
  }
}

// SUB: 64-deep k sub-blocks per stage (1 or 2; the sources other than kTile use 2).
// The bounds make the epilogue spill: 52 bytes at 72 registers for kBytes, the price of two CTAs of 448 threads per SM (one cannot
// keep the chain of copy, conversion and MMA full); 102 bytes at 80 for kLoose, whose 704 threads leave no more. Neither was
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

  const bool leader = elect_one();  // of every warp; the copy and the MMA warp issue through theirs
  if (warp == 4 && leader) {
    for (int g = 0; g < p.count && (SRC == kTile || SRC == kBytes); g++) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.rhs[g]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.lhs) : "memory");
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < kOperandSlots; s++) {
      mbar_init(&ready[s], SRC == kBytes ? 4 : kTmemA ? converter_warps(SRC) : 1);  // the warps of a unit
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
  if (warp == 4) {
    int tile = cluster, kb = kb_begin;
    Tile t = locate_tile(p, min(tile, p.tiles - 1));
    for (int i = 0; i < first; i++) {
      if (leader) {
        mbar_expect_tx(&full[i], per_stage);
        load_rhs(t, kb, i);
      }
      if (++kb == kb_end) {
        kb = kb_begin;
        tile += clusters;
        t = locate_tile(p, min(tile, p.tiles - 1));
      }
    }
    __syncwarp();
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
    auto load_lhs = [&](const Tile& t, int kb, int stage) {
      const uint32_t st = base + (uint32_t)stage * per_stage + w_bytes;
#pragma unroll
      for (int s = 0; s < SUB; s++)
        tma_load_2d(st + (uint32_t)s * p.m_tile * 128u, &maps.lhs, kb * kDepth + s * kSubK, t.m_idx * p.m_tile, &full[stage]);
    };
    auto gave_up = [&](int i) {
      atomicExch(p.error_flag, 11);
      // Nothing more is requested; the copies in flight get a bounded time to land before the CTA leaves.
      for (int b = 1; b <= p.stages; b++) {
        const int j = i - b;  // the last unit requested into each stage
        for (unsigned spin = 0; spin < (1u << 16) && !mbar_try_wait(&full[j % p.stages], (unsigned)(j / p.stages) & 1u); spin++) {
        }
      }
    };
    int tile = cluster, kb = kb_begin, stage = 0;
    unsigned phase = 0;
    if constexpr (SRC == kLoose) {
      // Activations only, by one lane: beside sixteen converter warps the converged form of this loop costs the launch 4 to 8 %
      // (us, converged and so: 5 x 65536 x 3001 260 / 237, 33 x 8192 x 32001 330 / 305, 64 x 2048 x 32001 95 / 88; 64 x 2048 x 1001
      // 14.5 either way). Which part of it does was not found: waiting by one lane alone did not help.
      if (lane == 0 && count > 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        Tile t = locate_tile(p, tile);
        for (int i = 0; i < count; i++) {
          if (i >= first) {
            if (i >= p.stages && !mbar_wait(&empty[stage], phase ^ 1, budget)) {
              gave_up(i);
              break;
            }
            mbar_expect_tx(&full[stage], per_stage);
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
    } else {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      Tile t = locate_tile(p, min(tile, p.tiles - 1));
      for (int i = 0; i < count; i++) {
        if (i >= p.stages && !__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, budget))) {
          if (leader) gave_up(i);
          break;
        }
        if (leader) {
          if (i >= first) {
            mbar_expect_tx(&full[stage], per_stage);
            load_rhs(t, kb, stage);
          }
          load_lhs(t, kb, stage);
        }
        __syncwarp();
        if (++kb == kb_end) {
          kb = kb_begin;
          tile += clusters;
          t = locate_tile(p, min(tile, p.tiles - 1));
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ---- MMA issuer ----------------------------------------------------------------------------------------------
    const uint32_t idesc = instr_desc(p.is_bf16, p.m_tile, !kTmemA && !p.rhs_k_major);
    // Operands of stage 0. Weights K-major like the activations: 64-k sub-blocks 16 KiB apart, 32 bytes per 16-k step inside
    // the swizzled row. MN-major: 16 k rows = two 1024-byte swizzle atoms further down; the two 64-column boxes are
    // SUB * 8192 bytes apart (leading offset), 8-row groups 1024 bytes apart (stride offset).
    const uint64_t a_first = p.rhs_k_major ? smem_desc(base, 16, 1024) : smem_desc(base, SUB * 8192u, 1024);
    const uint64_t b_first = smem_desc(base + w_bytes, 16, 1024);
    int stage = 0, slot = 0;
    unsigned phase = 0, slot_phase = 0;
    bool ok = true;
    for (int seg = 0; seg < my_tiles && ok; seg++) {
      // Take the next accumulator once the epilogue has drained its previous use.
      const int buf = seg & 1;
      ok = seg < 2 || __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, budget));
      if (!ok) {
        if (leader) atomicExch(p.error_flag, 14);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem_base + (uint32_t)(buf * p.m_tile);
      for (int kb = kb_begin; kb < kb_end; kb++) {
        // The copies of the stage have landed; the converters have also filled the slot.
        ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, budget) && (!kTmemA || mbar_wait(&ready[slot], slot_phase, budget)));
        if (!ok) {
          if (leader) atomicExch(p.error_flag, 12);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t a = desc_advance(a_first, (uint32_t)stage * per_stage), b = desc_advance(b_first, (uint32_t)stage * per_stage);
        const uint32_t operand = operand_base + (uint32_t)(slot * 32 * SUB);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 4 * SUB; kk++) {
            const uint64_t b_desc = desc_advance(b, (uint32_t)(kk >> 2) * p.m_tile * 128u + (kk & 3) * 32u);
            const uint32_t accumulate = (kb == kb_begin && kk == 0) ? 0u : 1u;
            if (kTmemA) mma_f16_tmem_a(acc, operand + (uint32_t)(kk * 8), b_desc, idesc, accumulate);
            else mma_f16(acc, desc_advance(a, p.rhs_k_major ? (kk >> 2) * 16384u + (kk & 3) * 32u : kk * 2048u), b_desc, idesc, accumulate);
          }
          mma_commit(&empty[stage]);  // the stage is free once these MMAs have read it
          if (kTmemA) mma_commit(&slot_empty[slot]);  // and so is the operand slot
          if (kb + 1 == kb_end) mma_commit(&acc_full[buf]);
        }
        __syncwarp();
        if (kTmemA && ++slot == kOperandSlots) {
          slot = 0;
          slot_phase ^= 1;
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
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
      // 16 columns of 8 rows are a block of 8 x 8 16-bit units: read transposed, a thread gets columns 2 * c and 2 * c + 1
      // (c = lane / 4) of rows 2 * (lane % 4) and + 1 in one word, which is two k values of each column, and those are the
      // 32-bit columns that the 16-lane store wants from this thread for lanes c and c + 8. (The 128-byte swizzle spreads
      // the block's eight rows over all banks.) The two warps of a quarter take units in turn: one waits, reads and stores
      // while the other converts.
      static_assert(SRC != kBytes || SUB == 2, "128 rows per unit");
      auto next_unit = [&]() {
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      };
      auto next_slot = [&]() {
        if (++slot == kOperandSlots) {
          slot = 0;
          slot_phase ^= 1;
        }
      };
      if (part) {
        next_unit();
        next_slot();
      }
      for (int i = part; i < count; i += 2) {
        const bool ok = slot_free(i) && mbar_wait(&full[stage], phase, budget);  // in this order (kOperandSlots)
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) atomicExch(p.error_flag, 15);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t dst = operand_base + quarter_addr + (uint32_t)(slot * 32 * SUB);
        const uint32_t row = base + (uint32_t)stage * per_stage + (uint32_t)lane * 128u;
        if (p.is_bf16) convert_unit<true>(row, quarter, lane, dst);
        else convert_unit<false>(row, quarter, lane, dst);
        publish();
        next_slot();
        next_unit();
        next_unit();
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
    const int n_local = warp * 32 + (SRC == kBytes ? (lane & 16) + 2 * (lane & 7) + ((lane >> 3) & 1) : lane);
    for (int seg = 0; seg < my_tiles; seg++) {
      const Tile t = locate_tile(p, cluster + seg * clusters);
      const int buf = seg & 1;
      const long long n = (long long)t.n_tile * kTileN + n_local;
      const bool in = n < p.n[t.group];
      const int m0 = t.m_idx * p.m_tile;
      const int m_rows = min(p.m_tile, p.m - m0);  // rows of this tile that exist
      const long long ldo = p.ldo[t.group];
      constexpr bool int8 = SRC == kBytes;
      // Int8 weights: the tensor core contracted the integers; this thread's column scale finishes the product.
      const float scale = int8 && in ? __half2float(static_cast<const __half*>(p.scale[t.group])[n]) : 1.f;
      // One decision for all four warps: tcgen05.ld is warp-collective.
      if (!epilogue_all(mbar_wait(&acc_full[buf], (seg >> 1) & 1, budget))) {
        if (threadIdx.x == 0) atomicExch(p.error_flag, 13);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      auto store = [&](int row, float v) {
        if (int8) v *= scale;
        const long long at = (long long)(m0 + row) * ldo + n;
        if (p.is_bf16) static_cast<__nv_bfloat16*>(p.out[t.group])[at] = __float2bfloat16_rn(v);
        else static_cast<__half*>(p.out[t.group])[at] = __float2half_rn(v);
      };
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * p.m_tile);
      const int sum_buf = p.sum_buffers == 2 ? buf : 0;
      float* received = sums + (size_t)sum_buf * ksplit * p.rows_per_rank * kTileN;
      int owner = 0, owner_row = 0;  // the CTA that finishes the next four rows, and their place among its rows
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
            const uint32_t at =
                cluster_address(smem_u32(received + ((size_t)rank * p.rows_per_rank + owner_row) * kTileN + threadIdx.x * 4), (uint32_t)owner);
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3])
                         : "memory");
            if ((owner_row += 4) == p.rows_per_rank) {
              owner_row = 0;
              owner++;
            }
          }
        } else if (in) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (c0 + j < m_rows) store(c0 + j, __uint_as_float(r[j]));
        }
      }
      // The accumulator is in registers / memory now: hand it back to the MMA warp.
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      if (ksplit > 1) {
        // A receive buffer is written again two tiles later, after its writer has seen this CTA's arrivals for the tile
        // in between, which follow the reads below.
        if (lane < ksplit) cluster_arrive(cluster_address(smem_u32(&sum_full[buf]), (uint32_t)lane));
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
