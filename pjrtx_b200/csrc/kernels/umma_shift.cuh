// Contraction of few rows with 16-bit weights [k, n] whose row pitch p is not a multiple of 16 bytes (an odd vocabulary), on
// the tensor cores (tcgen05) with tiled tensor-map copies all the same:
//   out[m, n] = sum_k lhs[m, k] * rhs[k, n]        m <= 32, lhs k-contiguous
//
// A tensor map cannot describe such rows, but it can describe every R-th of them (R = 2, 4 or 8, the least for which R * p is
// a multiple of 8 elements): the rows k = R * q + j of one residue j are a matrix of pitch R * p whose first row starts
// delta_j = j * p mod 8 elements behind a 16-byte boundary. Copied from that boundary on, its columns lie delta_j places further
// right. So the product is computed as in umma_gemm.cuh, D^T[n, m] = W^T . x^T with the weight's columns on the 128-row side,
// once for every residue with an accumulator of its own, on columns as they lie:
//   P_j[c, m] = sum_q raw_j[q, c] * x[m, R * q + j]         out[n, m] = sum_j P_j[n + delta_j, m]
// and the epilogue, which sums the residues in f32 in the order of j, moves each by its delta. A tile of 128 raw columns finishes
// 120 results; the 8 it shares with the next tile come from L2. x is rearranged by residue first (residue_rows_kernel, a few
// hundred KB), zeros where a residue has fewer rows.
//
// What bounds it: HBM, and above it 12 us for two launches, the first copies and the residues' sum. Before it, one 2-byte load
// per weight through the converter warps of umma_stream_kernel<2, kLoose>, 1.6 TB/s, which remains for more rows and for small
// weights (shift_pays in dot.cu). 5 rows of f16, launches one after the
// other, us, before and now: 2048 x 32001 83 / 31.6, 4096 x 32001 156 / 54, 8192 x 32001 300 / 101 (5.2 TB/s); 32 rows 85 / 36,
// 158 / 62.5, 302 / 106. Errors against 64 bits are equal to three digits (the rounding of the output), the fourth is smaller.
//
// Roles and waits as in umma_gemm.cuh: copy warp, MMA warp, four epilogue warps, two sets of accumulators, every mbarrier wait
// bounded by time. The launch is ordered after the rearrangement, whose own launch may start early.
#pragma once

#include "umma_gemm.cuh"

namespace pjrtx {
namespace umma {

constexpr int kShiftMax = 8;           // residues
constexpr int kShiftOut = kTileN - 8;  // results of a tile
constexpr int kShiftPad = kTileN + 8;  // columns of the epilogue's exchange buffer (a thread reads up to delta behind its own)

struct ShiftParams {
  int m, residues;
  int kblocks;  // blocks of 64 rows of a residue
  int tiles;
  long long n, ldo;
  void* out;
  int delta[kShiftMax];
  int stages;
  int is_bf16;
  int early_rhs;
  int* error_flag;
  unsigned long long timeout_ns;
};
struct ShiftMaps {
  CUtensorMap rhs[kShiftMax];  // dims {n + delta_j, rows of the residue}, box {64, 64}
  CUtensorMap lhs;             // dims {residues * kblocks * 64, m}, box {64, m_tile}
};

__host__ __device__ constexpr uint32_t shift_stage_bytes(int m_tile) { return 16384u + (uint32_t)m_tile * 128u; }
__host__ __device__ constexpr uint32_t shift_exchange_bytes(int m_tile) { return (uint32_t)m_tile * kShiftPad * 4u; }
__host__ __device__ inline uint32_t shift_tmem_columns(int m_tile, int residues) {
  uint32_t cols = 32;
  while (cols < 2u * m_tile * residues) cols <<= 1;
  return cols;
}
inline size_t shift_smem_bytes(int stages, int m_tile, int residues) {
  const size_t bytes = (size_t)stages * shift_stage_bytes(m_tile) + shift_exchange_bytes(m_tile) + kBarrierBytes + 1024;
  const size_t least = least_smem(shift_tmem_columns(m_tile, residues));
  return bytes < least ? least : bytes;
}

// x[m, R * q + j] -> out[m, j * depth + q], zeros behind a residue's rows.
__global__ void __launch_bounds__(256) residue_rows_kernel(const unsigned short* __restrict__ x, long long pitch, int m, int k, int residues,
                                                           int depth, unsigned short* __restrict__ out) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const long long width = (long long)residues * depth, total = m * width;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long row = i / width, c = i - row * width, j = c / depth, at = (c - j * depth) * residues + j;
    out[i] = at < k ? x[row * pitch + at] : (unsigned short)0;
  }
}

template <int MT>
__global__ void __launch_bounds__(kBaseThreads, MT == 16 ? 2 : 1) umma_shift_kernel(const __grid_constant__ ShiftParams p, const __grid_constant__ ShiftMaps maps) {
  static_assert(MT == 16 || MT == 32, "");
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  constexpr uint32_t per_stage = shift_stage_bytes(MT);
  float4* exchange = reinterpret_cast<float4*>(base_ptr + (size_t)p.stages * per_stage);  // [MT / 4][kShiftPad]
  uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(exchange) + shift_exchange_bytes(MT));
  uint64_t* empty = full + p.stages;
  uint64_t* acc_full = empty + p.stages;  // [2]
  uint64_t* acc_empty = acc_full + 2;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  int* flags = reinterpret_cast<int*>(tmem_slot + 1);  // [0] abort
  const WaitBudget budget{global_timer_ns() + p.timeout_ns, flags};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();
  const int my_tiles = (int)blockIdx.x < p.tiles ? (p.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int per_tile = p.residues * p.kblocks;  // units: 64 rows of a residue
  const int count = my_tiles * per_tile;
  const uint32_t tmem_cols = shift_tmem_columns(MT, p.residues);

  if (warp == 4 && leader) {
    for (int j = 0; j < p.residues; j++) asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.rhs[j]) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.lhs) : "memory");
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    flags[0] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  struct Unit {
    int tile, residue, kb;
  };
  auto advance = [&](Unit* u) {
    if (++u->kb == p.kblocks) {
      u->kb = 0;
      if (++u->residue == p.residues) {
        u->residue = 0;
        u->tile += (int)gridDim.x;
      }
    }
  };
  auto load_rhs = [&](const Unit& u, int stage) {
    const uint32_t st = base + (uint32_t)stage * per_stage;
    const int n0 = u.tile * kShiftOut;  // a multiple of 8 elements
    tma_load_2d_hint(st, &maps.rhs[u.residue], n0, u.kb * 64, &full[stage], policy);
    tma_load_2d_hint(st + 8192u, &maps.rhs[u.residue], n0 + 64, u.kb * 64, &full[stage], policy);
  };
  // The weights of the first ring depend on nothing.
  const int first = p.early_rhs ? min(count, p.stages) : 0;
  if (warp == 4) {
    Unit u{(int)blockIdx.x, 0, 0};
    for (int i = 0; i < first; i++) {
      if (leader) {
        mbar_expect_tx(&full[i], per_stage);
        load_rhs(u, i);
      }
      advance(&u);
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

  if (warp == 4) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    Unit u{(int)blockIdx.x, 0, 0};
    int stage = 0;
    unsigned phase = 0;
    for (int i = 0; i < count; i++) {
      if (i >= p.stages && !__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, budget))) {
        if (leader) {
          atomicExch(p.error_flag, 23);
          // Nothing more is requested; the copies in flight get a bounded time to land before the CTA leaves.
          for (int b = 1; b <= p.stages; b++) {
            const int j = i - b;
            for (unsigned spin = 0; spin < (1u << 16) && !mbar_try_wait(&full[j % p.stages], (unsigned)(j / p.stages) & 1u); spin++) {
            }
          }
        }
        break;
      }
      if (leader) {
        if (i >= first) {
          mbar_expect_tx(&full[stage], per_stage);
          load_rhs(u, stage);
        }
        tma_load_2d(base + (uint32_t)stage * per_stage + 16384u, &maps.lhs, (u.residue * p.kblocks + u.kb) * 64, 0, &full[stage]);
      }
      __syncwarp();
      advance(&u);
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    const uint32_t idesc = instr_desc(p.is_bf16, MT, 1);
    const uint64_t a_first = smem_desc(base, 8192u, 1024), b_first = smem_desc(base + 16384u, 16, 1024);
    int stage = 0;
    unsigned phase = 0;
    bool ok = true;
    for (int seg = 0; seg < my_tiles && ok; seg++) {
      const int buf = seg & 1;
      ok = seg < 2 || __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, budget));
      if (!ok) {
        if (leader) atomicExch(p.error_flag, 24);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t acc = tmem_base + (uint32_t)(buf * p.residues * MT);
      int kb = 0;
      for (int i = 0; i < per_tile; i++) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, budget));
        if (!ok) {
          if (leader) atomicExch(p.error_flag, 25);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t a = desc_advance(a_first, (uint32_t)stage * per_stage), b = desc_advance(b_first, (uint32_t)stage * per_stage);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 4; kk++)
            mma_f16(acc, desc_advance(a, kk * 2048u), desc_advance(b, kk * 32u), idesc, (kb == 0 && kk == 0) ? 0u : 1u);
          mma_commit(&empty[stage]);
          if (i + 1 == per_tile) mma_commit(&acc_full[buf]);
        }
        __syncwarp();
        if (++kb == p.kblocks) {
          kb = 0;
          acc += MT;
        }
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    __syncwarp();
  } else {
    // ---- epilogue warps 0..3: TMEM lane = raw column of the tile ----------------------------------------------------
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = (int)threadIdx.x;
    for (int seg = 0; seg < my_tiles; seg++) {
      const int buf = seg & 1;
      if (!epilogue_all(mbar_wait(&acc_full[buf], (seg >> 1) & 1, budget))) {
        if (t == 0) atomicExch(p.error_flag, 26);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t taddr = tmem_base + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * p.residues * MT);
      float4 sum[MT / 4];
#pragma unroll
      for (int q = 0; q < MT / 4; q++) sum[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int j = 0; j < p.residues; j++) {
#pragma unroll
        for (int c = 0; c < MT; c += 16) {
          uint32_t r[16];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
              : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
              : "r"(taddr + (uint32_t)(j * MT + c)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int q = 0; q < 4; q++)
            exchange[(c / 4 + q) * kShiftPad + t] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                                                 __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        // The last threads read past the tile's columns; they finish no result.
        const float4* from = exchange + t + p.delta[j];
#pragma unroll
        for (int q = 0; q < MT / 4; q++) {
          const float4 v = from[q * kShiftPad];
          sum[q].x += v.x;
          sum[q].y += v.y;
          sum[q].z += v.z;
          sum[q].w += v.w;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      const long long n = (long long)((int)blockIdx.x + seg * (int)gridDim.x) * kShiftOut + t;
      if (t < kShiftOut && n < p.n) {
        unsigned short* out = static_cast<unsigned short*>(p.out) + n;
#pragma unroll
        for (int q = 0; q < MT / 4; q++) {
          const float v[4] = {sum[q].x, sum[q].y, sum[q].z, sum[q].w};
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (4 * q + e < p.m)
              out[(4 * q + e) * p.ldo] =
                  p.is_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v[e])) : __half_as_ushort(__float2half_rn(v[e]));
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 5) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
}

}  // namespace umma
}  // namespace pjrtx
