// Large contractions of 16-bit floats on paired SMs (tcgen05, cta_group::2), f32 accumulation in tensor memory:
//   out[m, n] = sum_k lhs[m, k] * rhs[k, n]        lhs k-contiguous; rhs n-contiguous ([k, n]) or k-contiguous ([n, k])
// The prefill side of umma_gemm.cuh, with the same transposed product D^T[n, m] = W^T . x^T and the same operand layouts.
//
// What bounds it: shared memory. One SM's tensor core finishes 128 x 256 x 16 in 128 cycles and reads 12 KiB of operands
// for it, while the copies write 12 KiB more: 192 bytes per cycle where shared memory moves 128. A pair of SMs works on
// one 256 (n) x m_tile tile instead: each CTA holds 128 weight columns and HALF of the tile's activation rows, and the
// tensor cores read the other half from the peer, so an SM moves 8 KiB in and 8 KiB out per 128 cycles.
//
// One persistent cluster of two CTAs per pair of SMs. Both CTAs run the same roles, CTA 0 leads:
//   copy warp       (each CTA) copies its 128 weight columns and its m_tile / 2 activation rows into its own ring; the
//                   bytes of both CTAs are counted on the leader's `full` mbarrier
//   MMA warp        (leader) issues tcgen05.mma.cta_group::2 (M = 256, N = m_tile, K = 16); the commits release the stage
//                   (`empty`) and publish the accumulator (`acc_full`) in both CTAs
//   epilogue warps  (each CTA) drain the CTA's own 128 rows of the accumulator (two accumulators: the next tile's MMAs
//                   run meanwhile) and tell the leader (`acc_empty`)
// Tiles are dealt out in bands of kBand weight tiles, activations fastest inside a band, so that the tiles in flight on the
// chip form a compact block and share both operands through L2.
//
// Both warps run converged and let an elected thread issue (elect_one in umma_gemm.cuh); by a single thread a 64-deep unit took
// 300 ns and 0.5 ns per row, now 195 and 0.57. Measured, bf16, us, one SM per tile, pairs issued by a single thread, pairs now:
// 517 rows, 14336 x 4096 - / 85 / 71.5, 4096 x 28672 - / 120 / 109, 4096 x 4096 40 / 35.5 / 31; 2048 rows, 4096 x 28672 - / 332 / 315
// (1527 TFLOP/s); 8192 rows inside a full-depth prefill, under the power cap and ordered after the predecessor, 4096 x 28672 2030 /
// 1382 / 1307, 14336 x 4096 880 / 675 / 662, 4096 x 6144 429 / 325 / 311, 4096 x 4096 291 / 220 / 212 (the first of each four alone).
//
// No copy is multicast. Waits are bounded by time as in umma_gemm.cuh. The launch is ordered after its predecessor; its
// dependents are released after the tensor-memory allocation.
#pragma once

#include "umma_gemm.cuh"

namespace pjrtx {
namespace umma {

constexpr int kPairN = 256;   // weight columns of a tile (128 per CTA)
constexpr int kBand = 8;      // weight tiles of a band

struct PairParams {
  int m;
  int m_tile;                      // multiple of 32, 32..256
  int m_tiles, n_tiles;            // n_tiles over the whole group
  int count;
  int n_tile_begin[kGroupMax + 1];  // prefix sums of weight tiles over the group
  void* out[kGroupMax];
  long long n[kGroupMax];
  long long ldo[kGroupMax];
  int kblocks;                     // ceil(k / 64)
  int stages;
  int is_bf16;
  int rhs_k_major, rhs_3d;
  int* error_flag;
  unsigned long long timeout_ns;
};

__host__ __device__ inline size_t pair_stage_bytes(int m_tile) { return 16384 + (size_t)m_tile * 64; }
inline size_t pair_smem_bytes(int stages, int m_tile) {
  const size_t bytes = stages * pair_stage_bytes(m_tile) + kBarrierBytes + 1024;
  return bytes < least_smem(512) ? least_smem(512) : bytes;
}

// Copies of a CTA pair: the data lands in the executing CTA, `bar` may be the peer's mbarrier (a shared::cluster address).
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void pair_mma_f16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the mbarrier at this offset in both CTAs once the MMAs issued so far have completed.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((unsigned short)3)
               : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

struct PairTile {
  int group, n0, m_idx;  // n0: first column of the tile inside its contraction
};
__device__ __forceinline__ PairTile locate_pair_tile(const PairParams& p, int tile) {
  const int per_band = kBand * p.m_tiles;
  const int band = tile / per_band, in_band = tile - band * per_band;
  const int width = min(kBand, p.n_tiles - band * kBand);
  const int m_idx = in_band / width, n_tile = band * kBand + in_band - m_idx * width;
  int g = 0;
#pragma unroll
  for (int q = 1; q < kGroupMax; q++)
    if (q < p.count && n_tile >= p.n_tile_begin[q]) g = q;
  return PairTile{g, (n_tile - p.n_tile_begin[g]) * kPairN, m_idx};
}

__global__ void __launch_bounds__(kBaseThreads, 1) umma_pair_kernel(const PairParams p, const __grid_constant__ Maps maps) {
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  const uint32_t per_stage = (uint32_t)pair_stage_bytes(p.m_tile);
  uint64_t* full = reinterpret_cast<uint64_t*>(base_ptr + (size_t)p.stages * per_stage);
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;  // [2]
  uint64_t* acc_empty = acc_full + 2;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* flags = reinterpret_cast<int*>(tmem_slot + 1);  // [0] abort
  const WaitBudget budget{global_timer_ns() + p.timeout_ns, flags};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)blockIdx.x & 1, pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  const int tiles = p.m_tiles * p.n_tiles;
  const int my_tiles = pair < tiles ? (tiles - 1 - pair) / pairs + 1 : 0;
  const int count = my_tiles * p.kblocks;
  const uint32_t tmem_cols = tmem_columns(p.m_tile, 1, kTile);  // two accumulators, as there
  const bool leader = elect_one();  // of the warp: the copy and the MMA warp issue through theirs

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);  // four epilogue warps of each CTA
    }
    flags[0] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The paired allocation is collective: its warp may issue it only once the peer CTA is known to have launched, and the
  // peer has to stay until the paired free has completed (the last barrier of the kernel). CTAs of a cluster are scheduled
  // together, but nothing else says that the peer already runs. The same barrier publishes the mbarriers.
  cluster_sync();
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // This CTA has its tensor memory: the MMA warp waits for the peer's word before the first MMA, which writes both CTAs'
  // columns, everybody else at the exit.
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    // ---- TMA producer (each CTA its own half of both operands) -----------------------------------------------------
    const int lhs_rows = p.m_tile / 2;
    PairTile t = locate_pair_tile(p, min(pair, tiles - 1));
    int seg = 0, kb = 0, stage = 0;
    unsigned phase = 0;
    for (int i = 0; i < count; i++) {
      if (i >= p.stages && !__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, budget))) {
        if (leader) {
          atomicExch(p.error_flag, 17);
          // The copies in flight get time to land before the pair leaves.
          const unsigned long long until = global_timer_ns() + 50000;
          while (global_timer_ns() < until) {
          }
        }
        break;
      }
      if (leader) {
        const uint32_t st = base + (uint32_t)stage * per_stage;
        const uint32_t bar = cluster_address(smem_u32(&full[stage]), 0);
        const int k0 = kb * kSubK, n0 = t.n0 + rank * 128;
        if (rank == 0) mbar_expect_tx(&full[stage], 2 * per_stage);
        if (p.rhs_3d) {
          pair_load_3d(st, &maps.rhs[t.group], 0, k0, n0 / 64, bar);
        } else if (p.rhs_k_major) {
          pair_load_2d(st, &maps.rhs[t.group], k0, n0, bar);
        } else {
          pair_load_2d(st, &maps.rhs[t.group], n0, k0, bar);
          pair_load_2d(st + 8192u, &maps.rhs[t.group], n0 + 64, k0, bar);
        }
        pair_load_2d(st + 16384u, &maps.lhs, k0, t.m_idx * p.m_tile + rank * lhs_rows, bar);
      }
      __syncwarp();
      if (++kb == p.kblocks) {
        kb = 0;
        if (++seg < my_tiles) t = locate_pair_tile(p, pair + seg * pairs);
      }
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ---- MMA issuer (leader) -----------------------------------------------------------------------------------------
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    __syncwarp();
    if (rank == 0) {
      // M = 256: twice the single-CTA instruction's.
      const uint32_t idesc = instr_desc(p.is_bf16, p.m_tile, !p.rhs_k_major) + ((uint32_t)(kTileN >> 4) << 24);
      const uint64_t a_first = p.rhs_k_major ? smem_desc(base, 16, 1024) : smem_desc(base, 8192u, 1024);
      const uint64_t b_first = smem_desc(base + 16384u, 16, 1024);
      const uint32_t a_step = p.rhs_k_major ? 32u : 2048u;
      int stage = 0;
      unsigned phase = 0;
      bool ok = true;
      for (int seg = 0; seg < my_tiles && ok; seg++) {
        const int buf = seg & 1;
        ok = seg < 2 || __all_sync(0xffffffffu, cluster_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, budget));
        if (!ok) {
          if (leader) atomicExch(p.error_flag, 20);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + (uint32_t)(buf * p.m_tile);
        for (int kb = 0; kb < p.kblocks; kb++) {
          ok = __all_sync(0xffffffffu, cluster_wait(&full[stage], phase, budget));
          if (!ok) {
            if (leader) atomicExch(p.error_flag, 18);
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t a = desc_advance(a_first, (uint32_t)stage * per_stage), b = desc_advance(b_first, (uint32_t)stage * per_stage);
          if (leader) {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              pair_mma_f16(acc, desc_advance(a, kk * a_step), desc_advance(b, kk * 32u), idesc, (kb == 0 && kk == 0) ? 0u : 1u);
            pair_commit(&empty[stage]);
            if (kb + 1 == p.kblocks) pair_commit(&acc_full[buf]);
          }
          __syncwarp();
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue warps 0..3 of each CTA: TMEM lane = weight column ------------------------------------------------------
    for (int seg = 0; seg < my_tiles; seg++) {
      const PairTile t = locate_pair_tile(p, pair + seg * pairs);
      const int buf = seg & 1;
      if (!epilogue_all(mbar_wait(&acc_full[buf], (seg >> 1) & 1, budget))) {
        if (threadIdx.x == 0) atomicExch(p.error_flag, 19);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const long long n = t.n0 + rank * 128 + warp * 32 + lane;
      const bool in = n < p.n[t.group];
      const int m0 = t.m_idx * p.m_tile;
      const int m_rows = min(p.m_tile, p.m - m0);
      const long long ldo = p.ldo[t.group];
      unsigned short* out = static_cast<unsigned short*>(p.out[t.group]) + (long long)m0 * ldo + n;
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * p.m_tile);
      for (int c0 = 0; c0 < m_rows; c0 += 32) {
        uint32_t r[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
              "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
              "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
              "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr + (uint32_t)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (in) {
#pragma unroll
          for (int j = 0; j < 32; j++)
            if (c0 + j < m_rows) {
              const float v = __uint_as_float(r[j]);
              out[(long long)(c0 + j) * ldo] = p.is_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
            }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) cluster_arrive(cluster_address(smem_u32(&acc_empty[buf]), 0));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncwarp();
  if (warp != 5) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  cluster_sync();  // nobody frees or leaves while the peer may still write here
  if (warp == 5) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    __syncwarp();
  }
  // The paired free is collective too: neither CTA leaves before both have issued it.
  cluster_sync();
}

}  // namespace umma
}  // namespace pjrtx
