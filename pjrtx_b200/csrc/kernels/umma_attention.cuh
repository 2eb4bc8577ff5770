// Causal self-attention over whole sequences (prefill) on the 5th-generation tensor cores (tcgen05), scores, probabilities
// and outputs in tensor memory:
//   out[b, g, s, r, :] = softmax_j( q[b, g, s, r, :] . k[b, j, g, :] * scale  for j <= s ) . v[b, j, g, :]
//
// q is [batch, kv_heads, seq, rep, head_dim] (the operand layout of the recognised dot_general -> masked softmax ->
// dot_general form), so the `seq * rep` query rows that share one KV head are one contiguous row-major matrix; row `x`
// belongs to position x / rep. out has that layout too, or [batch, seq, kv_heads, rep, head_dim] where the program only reads
// it transposed so (a launch of its own before: 26 us for 4 x 2048 positions of 32 heads, 4 us for 517). Scores and
// probabilities never leave the SM.
//
// A CTA owns TILES (1 or 2) tiles of 128 query rows and walks the keys 0..(its last position) in blocks of 128:
//   copy warp      q once, then K and V blocks into a ring of shared-memory slots (tiled tensor-map copies, 128-byte
//                  swizzle)
//   MMA warp       S_t = Q_t . K^T (M = 128 rows, N = 128 keys) and O_t += P_t . V (A operand P_t in tensor memory) for the
//                  tiles in turn: while the softmax warps of one tile work, the tensor core runs the other tile's products
//   softmax warps  four per tile, one query row per thread (TMEM lane = row): the block's row maximum needs no shuffle;
//                  probabilities go back to tensor memory, over the scores they came from, in the element type
// Tensor memory: S_t (128 columns, its first 64 reused for P_t) and O_t (head_dim columns) per tile.
//
// O is rescaled only when a row's maximum has grown by more than 2^8 since the scale in use was chosen (the conditional
// rescaling published with FlashAttention-4): until then the probabilities are relative to the older maximum (at most 256, in
// range for every type involved; the common factor cancels in the division by the row sum), and the round trip of O through
// registers is saved. The row sum is kept in f32 and is taken of the probabilities as the second product reads them, rounded
// to the element type, so that their rounding cancels where few keys carry a row: with equal values under all keys the result
// is that value.
// A block's S is complete only after the product O += P . V issued before it (one commit covers both), so a softmax thread
// that has seen S may touch O.
//
// What bounds it: per block and tile 1024 cycles of tensor core and 1024 cycles of exponentials (128 x 128 at 16 per
// cycle), which overlap between the two tiles. Measured for 4 x 2048 positions, 32 query heads of 128 over 8 KV heads: the
// warp-level kernel before this one (mma.sync, 64 rows per CTA) 627 us, this one 260 us inside a full-depth prefill (the
// transposed store included) and 204 us alone; 1 x 517 positions 24 and 13.5 us.
// Two tiles per CTA (320 threads) get 168 registers and spill 56 to 60 bytes, one tile of 64 elements a row with two CTAs per
// SM the same and 68 bytes; one of 128 has 180 and none. Reading the scores
// twice in 32-column chunks to hold fewer of them was slower (248 / 275 us).
//
// Row tiles are scheduled longest first. Waits are bounded by time (code 8 is reported). The launch is ordered after its predecessor; dependents are released after the
// tensor-memory allocation. The allocations of CTAs that share an SM fit its tensor memory (least_smem).
#pragma once

#include "umma_gemm.cuh"

namespace pjrtx {
namespace umma {

constexpr int kAttnRows = 128, kAttnKeys = 128;
constexpr int kAttnSlots = 5;

struct AttnParams {
  long long rows;  // seq * rep query rows per (sequence, KV head)
  int rep, kv_heads;
  long long out_batch, out_head, out_pos;  // element strides of the result; a position's `rep` heads are contiguous
  float scale_log2;  // |scale| * log2(e) (1 where scale is zero)
  float sign;        // 1, -1 or 0: what the scores are multiplied by first, so that the largest score has the largest exponent
  int* error_flag;
  unsigned long long timeout_ns;
};

__host__ __device__ constexpr int attn_slot_bytes(int hd) { return kAttnKeys * hd * 2; }
// CTAs an SM holds: two of one tile of 64 elements a row (98 KiB and 256 tensor-memory columns each), else one.
__host__ __device__ constexpr int attn_per_sm(int hd, int tiles) { return hd == 64 && tiles == 1 ? 2 : 1; }
__host__ __device__ constexpr size_t attn_smem_bytes(int hd, int tiles) {
  const size_t bytes = (size_t)tiles * kAttnRows * hd * 2 + (size_t)kAttnSlots * attn_slot_bytes(hd) + 512 + 1024;
  const size_t least = least_smem(attn_per_sm(hd, tiles) == 2 ? 256 : 512);
  return bytes < least ? least : bytes;
}

__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, int w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tmem_load_32(uint32_t addr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_store_32(uint32_t addr, const float* v) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <bool BF16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if (BF16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Adds the two elements of a packed pair to two f32 sums (mixed-precision additions, exact in the 16-bit operand).
// 4 x 2048 positions, 32 heads of 128 over 8: 201 us in bf16 and f16; widening first 201 and 208; sums of the unrounded
// probabilities 199 and 199.
template <bool BF16>
__device__ __forceinline__ void add_pair(uint32_t pair, float& lo, float& hi) {
  unsigned short l, h;
  asm("mov.b32 {%0, %1}, %2;" : "=h"(l), "=h"(h) : "r"(pair));
  if (BF16) {
    asm("add.rn.f32.bf16 %0, %1, %0;" : "+f"(lo) : "h"(l));
    asm("add.rn.f32.bf16 %0, %1, %0;" : "+f"(hi) : "h"(h));
  } else {
    asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(lo) : "h"(l));
    asm("add.rn.f32.f16 %0, %1, %0;" : "+f"(hi) : "h"(h));
  }
}

template <bool BF16, int HD, int TILES>
__global__ void __launch_bounds__(128 * TILES + 64, attn_per_sm(HD, TILES))
umma_attention_kernel(const AttnParams p, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                      const __grid_constant__ CUtensorMap vmap, void* __restrict__ out) {
  static_assert(HD == 64 || HD == 128, "");
  constexpr int kHalves = HD / 64;
  constexpr uint32_t kTileBytes = kAttnRows * HD * 2, kSlotBytes = attn_slot_bytes(HD);
  constexpr uint32_t kBlock = 128 * 128;  // bytes of one 64-element column block of 128 rows
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  const uint32_t ring = base + TILES * kTileBytes;
  uint64_t* q_full = reinterpret_cast<uint64_t*>(base_ptr + TILES * kTileBytes + kAttnSlots * kSlotBytes);
  uint64_t* slot_full = q_full + 1;               // [kAttnSlots]
  uint64_t* slot_empty = slot_full + kAttnSlots;  // [kAttnSlots]
  uint64_t* s_full = slot_empty + kAttnSlots;     // [TILES] scores of the next block are in tensor memory
  uint64_t* p_ready = s_full + TILES;             // [TILES] probabilities are in tensor memory, O may be accumulated
  uint64_t* o_full = p_ready + TILES;             // [TILES] the last product has completed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + TILES);
  int* flags = reinterpret_cast<int*>(tmem_slot + 1);  // [0] abort
  const WaitBudget budget{global_timer_ns() + p.timeout_ns, flags};
  constexpr uint32_t kTmemCols = TILES == 2 ? 512 : 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kMmaWarp = 4 * TILES, kCopyWarp = 4 * TILES + 1;
  const bool leader = elect_one();  // of the warp: the copy and the MMA warp issue through theirs
  const int g = blockIdx.y, b = blockIdx.z;
  const long long row0 = (long long)(gridDim.x - 1 - blockIdx.x) * (kAttnRows * TILES);  // longest first
  const long long last_row = min(row0 + kAttnRows * TILES, p.rows) - 1;
  const int blocks = (int)(last_row / p.rep) / kAttnKeys + 1;  // blocks of keys up to the last position
  const long long matrix_row = ((long long)b * p.kv_heads + g) * p.rows + row0;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < kAttnSlots; s++) {
      mbar_init(&slot_full[s], 1);
      mbar_init(&slot_empty[s], 1);
    }
    for (int t = 0; t < TILES; t++) {
      mbar_init(&s_full[t], 1);
      mbar_init(&p_ready[t], 4);
      mbar_init(&o_full[t], 1);
    }
    flags[0] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // Columns: S of every tile, then O of every tile.
  auto s_col = [&](int t) { return tmem_base + (uint32_t)(t * kAttnKeys); };
  auto o_col = [&](int t) { return tmem_base + (uint32_t)(TILES * kAttnKeys + t * HD); };

  if (warp == kCopyWarp) {
    if (leader) {
      mbar_expect_tx(q_full, TILES * kTileBytes);
      for (int t = 0; t < TILES; t++)
        for (int c = 0; c < kHalves; c++)
          tma_load_2d(base + t * kTileBytes + c * kBlock, &qmap, c * 64, (int)(matrix_row + t * kAttnRows), q_full);
    }
    __syncwarp();
    // K0 V0 K1 V1 ...; a block is two boxes of 64 keys per 64 elements. Keys past a row's position are masked, keys past
    // the sequence arrive as zeros.
    int slot = 0;
    unsigned phase = 0;
    for (int i = 0; i < 2 * blocks; i++) {
      if (i >= kAttnSlots && !__all_sync(0xffffffffu, mbar_wait(&slot_empty[slot], phase ^ 1, budget))) {
        // The copies in flight get a bounded time to land before the CTA leaves.
        for (int r = 1; r <= kAttnSlots && leader; r++) {
          const int j = i - r;
          for (unsigned spin = 0; spin < (1u << 16) && !mbar_try_wait(&slot_full[j % kAttnSlots], (unsigned)(j / kAttnSlots) & 1u); spin++) {
          }
        }
        break;
      }
      if (leader) {
        const CUtensorMap* map = (i & 1) ? &vmap : &kmap;
        const uint32_t dst = ring + (uint32_t)slot * kSlotBytes;
        const int key0 = (i >> 1) * kAttnKeys;
        mbar_expect_tx(&slot_full[slot], kSlotBytes);
        for (int c = 0; c < kHalves; c++)
          for (int h = 0; h < 2; h++) tma_load_4d(dst + c * kBlock + h * (kBlock / 2), map, c * 64, key0 + h * 64, g, b, &slot_full[slot]);
      }
      __syncwarp();
      if (++slot == kAttnSlots) {
        slot = 0;
        phase ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // N = 128 keys with K as a K-major B operand; N = head_dim with V as an MN-major one (bit 16).
    const uint32_t idesc_s = instr_desc(BF16, kAttnKeys, 0);
    const uint32_t idesc_o = instr_desc(BF16, HD, 0) | 1u << 16;
    const uint64_t q_first = smem_desc(base, 16, 1024), k_first = smem_desc(ring, 16, 1024), v_first = smem_desc(ring, kBlock, 1024);
    int slot = 0;
    unsigned phase = 0;
    auto next_slot = [&]() {
      const int s = slot;
      if (++slot == kAttnSlots) {
        slot = 0;
        phase ^= 1;
      }
      return s;
    };
    auto wait = [&](uint64_t* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, budget)) != 0; };
    // Issued by the elected thread.
    auto scores = [&](int t, int k_slot) {
      const uint64_t q = desc_advance(q_first, t * kTileBytes), k = desc_advance(k_first, (uint32_t)k_slot * kSlotBytes);
#pragma unroll
      for (int kk = 0; kk < HD / 16; kk++) {
        const uint32_t at = (uint32_t)(kk >> 2) * kBlock + (uint32_t)(kk & 3) * 32u;
        mma_f16(s_col(t), desc_advance(q, at), desc_advance(k, at), idesc_s, kk ? 1u : 0u);
      }
      mma_commit(&s_full[t]);
    };
    auto values = [&](int t, int v_slot, bool accumulate) {
      const uint64_t v = desc_advance(v_first, (uint32_t)v_slot * kSlotBytes);
#pragma unroll
      for (int kk = 0; kk < kAttnKeys / 16; kk++)
        mma_f16_tmem_a(o_col(t), s_col(t) + (uint32_t)kk * 8u, desc_advance(v, (uint32_t)kk * 2048u), idesc_o, (accumulate || kk) ? 1u : 0u);
    };
    bool ok = wait(q_full, 0) && wait(&slot_full[0], 0);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        for (int t = 0; t < TILES; t++) scores(t, 0);
        mma_commit(&slot_empty[0]);
      }
      __syncwarp();
      next_slot();
    }
    for (int j = 0; j < blocks && ok; j++) {
      const unsigned v_phase = phase;
      const int v_slot = next_slot();
      const unsigned k_phase = phase;
      const bool more = j + 1 < blocks;
      const int k_slot = more ? next_slot() : 0;
      ok = wait(&slot_full[v_slot], v_phase);
#pragma unroll
      for (int t = 0; t < TILES; t++) {
        ok = ok && wait(&p_ready[t], (unsigned)j & 1u) && (!more || t > 0 || wait(&slot_full[k_slot], k_phase));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
          values(t, v_slot, j > 0);
          if (more) scores(t, k_slot);
          else mma_commit(&o_full[t]);
          if (t + 1 == TILES) {
            mma_commit(&slot_empty[v_slot]);
            if (more) mma_commit(&slot_empty[k_slot]);
          }
        }
        __syncwarp();
      }
    }
    if (!ok && leader && p.error_flag) atomicExch(p.error_flag, 8);
    __syncwarp();
  } else {
    const int t = warp >> 2;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_addr = s_col(t) + lanes, o_addr = o_col(t) + lanes;
    const long long row = row0 + t * kAttnRows + (warp & 3) * 32 + lane;
    // Rows past the matrix end have position -1: every key is masked and nothing is stored.
    const int pos = row < p.rows ? (int)(row / p.rep) : -1;
    const int first_pos = (int)((row0 + t * kAttnRows + (warp & 3) * 32) / p.rep);  // of the warp
    float m_used = -INFINITY, sum = 0.f;
    bool ok = true;
    for (int j = 0; j < blocks; j++) {
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[t], (unsigned)j & 1u, budget));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[kAttnKeys];
#pragma unroll
      for (int c = 0; c < 4; c++) tmem_load_32(s_addr + c * 32, s + c * 32);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (p.sign != 1.f) {
#pragma unroll
        for (int e = 0; e < kAttnKeys; e++) s[e] *= p.sign;
      }
      const int key0 = j * kAttnKeys;
      if (key0 + kAttnKeys - 1 > first_pos) {
#pragma unroll
        for (int e = 0; e < kAttnKeys; e++)
          if (key0 + e > pos) s[e] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int e = 4; e < kAttnKeys; e++) mx[e & 3] = fmaxf(mx[e & 3], s[e]);
      const float m_block = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2;
      float corr = 1.f;
      if (m_block > m_used + 8.f) {
        corr = exp2_approx(m_used - m_block);  // 0 the first time
        m_used = m_block;
        sum *= corr;
      }
      if (j > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll 1
        for (int c = 0; c < HD; c += 32) {
          float o[32];
          tmem_load_32(o_addr + c, o);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 32; e++) o[e] *= corr;
          tmem_store_32(o_addr + c, o);
        }
      }
      const float shift = m_used == -INFINITY ? 0.f : -m_used;
      float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 2; c++) {
        float packed[32];
#pragma unroll
        for (int e = 0; e < 32; e++) {
          const float x = exp2_approx(fmaf(s[c * 64 + 2 * e], p.scale_log2, shift));
          const float y = exp2_approx(fmaf(s[c * 64 + 2 * e + 1], p.scale_log2, shift));
          const uint32_t pair = pack_pair<BF16>(x, y);
          add_pair<BF16>(pair, part[(2 * e) & 3], part[(2 * e + 1) & 3]);
          packed[e] = __uint_as_float(pair);
        }
        tmem_store_32(s_addr + c * 32, packed);
      }
      sum += (part[0] + part[1]) + (part[2] + part[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
    }
    ok = ok && __all_sync(0xffffffffu, mbar_wait(&o_full[t], 0, budget));
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float inv = sum > 0.f ? 1.f / sum : sum != sum ? sum : 0.f;
      const long long at = b * p.out_batch + g * p.out_head + row / p.rep * p.out_pos + row % p.rep * HD;
      uint4* dst = reinterpret_cast<uint4*>(static_cast<unsigned short*>(out) + at);
#pragma unroll
      for (int c = 0; c < HD; c += 32) {
        float o[32];
        tmem_load_32(o_addr + c, o);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row < p.rows) {
#pragma unroll
          for (int e = 0; e < 32; e += 8)
            dst[(c + e) / 8] = make_uint4(pack_pair<BF16>(o[e] * inv, o[e + 1] * inv), pack_pair<BF16>(o[e + 2] * inv, o[e + 3] * inv),
                                          pack_pair<BF16>(o[e + 4] * inv, o[e + 5] * inv), pack_pair<BF16>(o[e + 6] * inv, o[e + 7] * inv));
        }
      }
    } else if (lane == 0 && p.error_flag) {
      atomicExch(p.error_flag, 8);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == kMmaWarp) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

}  // namespace umma
}  // namespace pjrtx
