// dot_general kernels for sm_100a.
//
// The kernels behind one canonical contraction out[b0,b1,m,n] = sum_k lhs*rhs
// (the reference reaches MLX matmul/tensordot for the same op,
// src/backend/mlx_metal/api.cc:3349-3498; its generated kernels are the
// one-thread-per-output and 256-thread tiled dots of
// src/backend/mlx_metal/metal_graph_dot.zig:46-64 and :199-256):
//   1  stream_kn : m <= 8, rhs[K,N] with N contiguous. Bandwidth-bound GEMV /
//                  skinny GEMM: 16-byte loads of rhs rows, f32 accumulators in
//                  registers, K split over warps and CTAs, deterministic
//                  last-CTA fold of the f32 partials. Without batch axes: the
//                  TMA-fed persistent kernel (stream_tma.cuh), or small_dot_kernel
//                  for a k that one round of loads covers.
//   2  stream_nk : m <= 8, rhs[N,K] with K contiguous (attention scores, tied
//                  heads): lane groups own output columns and shuffle-reduce.
//   3  tile      : shared-memory tiled FFMA contraction with f32 accumulate
//                  (f32 matmul at 1e-5 needs real FFMA, not TF32): 128 x 64
//                  tiles, 64 x 64 tiles with k split over a cluster, or 64 x 64
//                  tiles for any strides.
//   0  generic   : one thread per output element, any strides, any m.
// 16-bit floats without batch axes whose operands a TMA tensor map can describe run on the tensor cores instead
// (umma_gemm.cuh, CTA pairs: umma_pair.cuh): rhs[K,N] as a variant of path 1 (so that q/k/v and gate/up still share one
// launch), rhs[N,K] as path 4, rhs[K,N] rows that a tensor map cannot describe as path 5. PJRTX_B200_UMMA=0 turns that off.
// Paths 1 and 4 start at three rows (one row takes the same on either side; two are 7 % faster on the tensor cores over 8
// layers of 8B widths, but f16 errors against 64 bits grow in the fourth digit there), large int8 weights, unless narrow or flat, at one;
// PJRTX_B200_UMMA_MIN_M, where it is set, is the least m for both.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "../common.h"
#include "kernels.h"
#include "stream_tma.cuh"
#include "umma_gemm.cuh"
#include "umma_pair.cuh"
#include "umma_shift.cuh"

namespace pjrtx {

namespace {

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Sixteen bytes of T held in registers; get(i) unpacks without taking an address
// so the value never leaves the register file.
__device__ __forceinline__ unsigned word_of(const uint4& r, int i) { return i == 0 ? r.x : i == 1 ? r.y : i == 2 ? r.z : r.w; }
template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int N = 4;
  uint4 raw;
  __device__ __forceinline__ float get(int i) const { return __uint_as_float(word_of(raw, i)); }
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  uint4 raw;
  __device__ __forceinline__ float get(int i) const {
    const unsigned u = word_of(raw, i >> 1);
    return __uint_as_float((i & 1) ? (u & 0xffff0000u) : (u << 16));
  }
};
template <> struct Vec16<__half> {
  static constexpr int N = 8;
  uint4 raw;
  __device__ __forceinline__ float get(int i) const {
    const unsigned u = word_of(raw, i >> 1);
    return __half2float(__ushort_as_half((unsigned short)((i & 1) ? (u >> 16) : (u & 0xffffu))));
  }
};

// Streaming 16-byte load that does not pollute L1 (weights are read once).
__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// ---------------------------------------------------------------- generic
template <typename T>
__global__ void dot_generic_kernel(DotShape s, const T* __restrict__ lhs, const T* __restrict__ rhs, T* __restrict__ out) {
  PJRTX_PDL_PROLOGUE();
  const int64_t total = s.b0 * s.b1 * s.m * s.n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i % s.n, m = (i / s.n) % s.m, b1 = (i / (s.n * s.m)) % s.b1, b0 = i / (s.n * s.m * s.b1);
    const T* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1 + m * s.lhs_m;
    const T* b = rhs + b0 * s.rhs_b0 + b1 * s.rhs_b1 + n * s.rhs_n;
    float acc = 0.f;
    for (int64_t k = 0; k < s.k; k++) acc = fmaf(to_f(a[k * s.lhs_k]), to_f(b[k * s.rhs_k]), acc);
    out[b0 * s.out_b0 + b1 * s.out_b1 + m * s.out_m + n] = from_f<T>(acc);
  }
}

// ---------------------------------------------------------------- stream_kn
constexpr int kKnUnroll = 8;
constexpr int kKnChunk = 512;  // lhs elements staged in shared memory per pass

// Up to four contractions that share lhs, m and k run as one launch: the column
// tiles of all of them form one grid (q/k/v or gate/up projections; the reference
// groups dots that share an lhs the same way, src/backend/mlx_metal/metal_graph_dot.zig:70-152).
struct KnGroup {
  int count;
  int tile_begin[kDotGroupMax + 1];
  const void* rhs[kDotGroupMax];
  void* out[kDotGroupMax];
  long long n[kDotGroupMax];
  long long rhs_k[kDotGroupMax];
  long long partial_offset[kDotGroupMax];  // in floats
};

template <typename T, int M, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
stream_kn_kernel(DotShape s, KnGroup grp, const T* __restrict__ lhs, float* __restrict__ partials,
                 unsigned* __restrict__ counters, int ksplit, int kslice) {
  PJRTX_PDL_PROLOGUE();
  constexpr int V = Vec16<T>::N;
  constexpr int TILE = 32 * V;
  constexpr int THREADS = WARPS * 32;
  __shared__ float red[WARPS - 1][M][TILE];
  __shared__ T xs[M][kKnChunk];
  __shared__ int is_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int g = 0;
#pragma unroll
  for (int q = 1; q < kDotGroupMax; q++)
    if (q < grp.count && (int)blockIdx.x >= grp.tile_begin[q]) g = q;
  const int64_t n_cols = grp.n[g], ldb = grp.rhs_k[g];
  const int64_t batch = blockIdx.z, b0 = batch / s.b1, b1 = batch % s.b1;
  const int64_t col = (int64_t)((int)blockIdx.x - grp.tile_begin[g]) * TILE + lane * V;
  const int64_t k_begin = (int64_t)blockIdx.y * kslice;
  const int64_t k_end = min(k_begin + (int64_t)kslice, s.k);
  const T* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1;
  const T* b = static_cast<const T*>(grp.rhs[g]) + b0 * s.rhs_b0 + b1 * s.rhs_b1;
  T* out = static_cast<T*>(grp.out[g]);
  const int rows = (int)min((int64_t)M, s.m);

  float acc[M][V];
#pragma unroll
  for (int m = 0; m < M; m++)
#pragma unroll
    for (int v = 0; v < V; v++) acc[m][v] = 0.f;

  const bool col_ok = col < n_cols;
  for (int64_t kc = k_begin; kc < k_end; kc += kKnChunk) {
    const int chunk = (int)min((int64_t)kKnChunk, k_end - kc);
    __syncthreads();
    for (int idx = threadIdx.x; idx < rows * chunk; idx += THREADS) {
      const int m = idx / chunk, kk = idx % chunk;
      xs[m][kk] = a[m * s.lhs_m + (kc + kk) * s.lhs_k];
    }
    __syncthreads();
    if (col_ok) {
      const T* bp = b + (kc + warp) * ldb + col;
      int kk = warp;
      for (; kk + (kKnUnroll - 1) * WARPS < chunk; kk += kKnUnroll * WARPS) {
        Vec16<T> w[kKnUnroll];
#pragma unroll
        for (int u = 0; u < kKnUnroll; u++) w[u].raw = ld_stream(bp + (int64_t)u * WARPS * ldb);
        bp += (int64_t)kKnUnroll * WARPS * ldb;
#pragma unroll
        for (int u = 0; u < kKnUnroll; u++)
#pragma unroll
          for (int m = 0; m < M; m++) {
            const float x = to_f(xs[m][kk + u * WARPS]);
#pragma unroll
            for (int v = 0; v < V; v++) acc[m][v] = fmaf(x, w[u].get(v), acc[m][v]);
          }
      }
      for (; kk < chunk; kk += WARPS) {
        Vec16<T> w;
        w.raw = ld_stream(bp);
        bp += (int64_t)WARPS * ldb;
#pragma unroll
        for (int m = 0; m < M; m++) {
          const float x = to_f(xs[m][kk]);
#pragma unroll
          for (int v = 0; v < V; v++) acc[m][v] = fmaf(x, w.get(v), acc[m][v]);
        }
      }
    }
  }
  // Fold the warps of this CTA in a fixed order.
  if (warp > 0) {
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
      for (int v = 0; v < V; v++) red[warp - 1][m][lane * V + v] = acc[m][v];
  }
  __syncthreads();
  float* part = partials + grp.partial_offset[g];
  if (warp == 0 && col_ok) {
#pragma unroll
    for (int m = 0; m < M; m++)
#pragma unroll
      for (int v = 0; v < V; v++) {
        float t = acc[m][v];
#pragma unroll
        for (int w = 0; w < WARPS - 1; w++) t += red[w][m][lane * V + v];
        acc[m][v] = t;
      }
    if (ksplit == 1) {
#pragma unroll
      for (int m = 0; m < M; m++) {
        if (m < rows) {
          T* o = out + b0 * s.out_b0 + b1 * s.out_b1 + m * n_cols + col;
#pragma unroll
          for (int v = 0; v < V; v++) o[v] = from_f<T>(acc[m][v]);
        }
      }
    } else {
      float* p = part + ((batch * ksplit + blockIdx.y) * (int64_t)M) * n_cols + col;
#pragma unroll
      for (int m = 0; m < M; m++)
        if (m < rows) {
#pragma unroll
          for (int v = 0; v < V; v++) p[(int64_t)m * n_cols + v] = acc[m][v];
        }
    }
  }
  if (ksplit == 1) return;
  // The CTA that arrives last for this column tile folds the partials in slice order.
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned prev = atomicAdd(&counters[batch * gridDim.x + blockIdx.x], 1u);
    is_last = prev == (unsigned)ksplit - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  const int64_t slice_stride = (int64_t)M * n_cols;
  for (int idx = threadIdx.x; idx < rows * TILE; idx += THREADS) {
    const int m = idx / TILE;
    const int64_t c = (int64_t)((int)blockIdx.x - grp.tile_begin[g]) * TILE + idx % TILE;
    if (c >= n_cols) continue;
    const float* p = part + (batch * ksplit * (int64_t)M + m) * n_cols + c;
    float t = 0.f;
    int ks = 0;
    for (; ks + 8 <= ksplit; ks += 8) {  // loads first, then the adds in slice order
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = __ldcg(p + (int64_t)(ks + u) * slice_stride);
#pragma unroll
      for (int u = 0; u < 8; u++) t += v[u];
    }
    for (; ks < ksplit; ks++) t += __ldcg(p + (int64_t)ks * slice_stride);
    out[b0 * s.out_b0 + b1 * s.out_b1 + m * n_cols + c] = from_f<T>(t);
  }
  if (threadIdx.x == 0) counters[batch * gridDim.x + blockIdx.x] = 0;  // ready for the next launch
}

// ---------------------------------------------------------------- stream_nk
template <typename T, int M>
__global__ void __launch_bounds__(256)
stream_nk_kernel(DotShape s, const T* __restrict__ lhs, const T* __restrict__ rhs, T* __restrict__ out, int group) {
  PJRTX_PDL_PROLOGUE();
  constexpr int V = Vec16<T>::N;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows_per_warp = 32 / group;
  const int64_t batch = blockIdx.y, b0 = batch / s.b1, b1 = batch % s.b1;
  const int64_t n = ((int64_t)blockIdx.x * 8 + warp) * rows_per_warp + lane / group;
  const int gl = lane % group;
  const T* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1;
  const T* b = rhs + b0 * s.rhs_b0 + b1 * s.rhs_b1 + n * s.rhs_n;
  const int rows = (int)min((int64_t)M, s.m);
  float acc[M];
#pragma unroll
  for (int m = 0; m < M; m++) acc[m] = 0.f;
  if (n < s.n) {
    for (int64_t k = (int64_t)gl * V; k < s.k; k += (int64_t)group * V) {
      Vec16<T> w;
      w.raw = ld_stream(b + k);
#pragma unroll
      for (int m = 0; m < M; m++) {
        if (m < rows) {
          Vec16<T> x;
          x.raw = __ldg(reinterpret_cast<const uint4*>(a + m * s.lhs_m + k));
#pragma unroll
          for (int v = 0; v < V; v++) acc[m] = fmaf(x.get(v), w.get(v), acc[m]);
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < M; m++)
    for (int o = group >> 1; o > 0; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
  if (n < s.n && gl == 0) {
#pragma unroll
    for (int m = 0; m < M; m++)
      if (m < rows) out[b0 * s.out_b0 + b1 * s.out_b1 + m * s.out_m + n] = from_f<T>(acc[m]);
  }
}

// ---------------------------------------------------------------- tile
constexpr int kTile = 64, kTileK = 16;

template <typename T>
__global__ void __launch_bounds__(256)
tile_kernel(DotShape s, const T* __restrict__ lhs, const T* __restrict__ rhs, T* __restrict__ out) {
  PJRTX_PDL_PROLOGUE();
  __shared__ float As[kTileK][kTile + 4];
  __shared__ float Bs[kTileK][kTile + 4];
  const int64_t batch = blockIdx.z, b0 = batch / s.b1, b1 = batch % s.b1;
  const T* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1;
  const T* b = rhs + b0 * s.rhs_b0 + b1 * s.rhs_b1;
  const int64_t m0 = (int64_t)blockIdx.y * kTile, n0 = (int64_t)blockIdx.x * kTile;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4] = {};
  for (int64_t k0 = 0; k0 < s.k; k0 += kTileK) {
    for (int idx = threadIdx.x; idx < kTile * kTileK; idx += 256) {
      // Walk the contiguous axis fastest for both operands.
      int mm, kk;
      if (s.lhs_k == 1) { kk = idx % kTileK; mm = idx / kTileK; } else { mm = idx % kTile; kk = idx / kTile; }
      const int64_t gm = m0 + mm, gk = k0 + kk;
      As[kk][mm] = (gm < s.m && gk < s.k) ? to_f(a[gm * s.lhs_m + gk * s.lhs_k]) : 0.f;
      int nn;
      if (s.rhs_n == 1) { nn = idx % kTile; kk = idx / kTile; } else { kk = idx % kTileK; nn = idx / kTileK; }
      const int64_t gn = n0 + nn, gk2 = k0 + kk;
      Bs[kk][nn] = (gn < s.n && gk2 < s.k) ? to_f(b[gk2 * s.rhs_k + gn * s.rhs_n]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kTileK; kk++) {
      float av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int64_t gm = m0 + ty * 4 + i;
    if (gm >= s.m) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t gn = n0 + tx * 4 + j;
      if (gn < s.n) out[b0 * s.out_b0 + b1 * s.out_b1 + gm * s.out_m + gn] = from_f<T>(acc[i][j]);
    }
  }
}

// ---------------------------------------------------------------- f32 tile, register-blocked
// out[m, n] = sum_k lhs[m, k] * rhs[k, n] in true f32 (the parity bar for f32 contractions is rel 1e-5, which TF32
// products miss at k = 1024), for dense operands: lhs k-contiguous, rhs n-contiguous, 16-byte aligned rows.
// 128 x 64 output tile per CTA of 256 threads, 8 x 4 outputs per thread, k in slabs of 16: the next slab travels
// global -> registers while the current one is multiplied out of shared memory (two buffers, one barrier per slab).
// Per k step a thread issues three 16-byte shared loads (two broadcast, one conflict-free) for 32 FFMAs, so the FMA pipe
// is the limit. A 1024^3 product is 128 tiles: one wave of one CTA per SM.
constexpr int kSgBM = 128, kSgBN = 64, kSgBK = 16;

__global__ void __launch_bounds__(256, 2)
sgemm_kernel(DotShape s, const float* __restrict__ lhs, const float* __restrict__ rhs, float* __restrict__ out) {
  PJRTX_PDL_PROLOGUE();
  __shared__ __align__(16) float As[2][kSgBK][kSgBM + 4];
  __shared__ __align__(16) float Bs[2][kSgBK][kSgBN + 4];
  const int tid = threadIdx.x;
  const int64_t batch = blockIdx.z, b0 = batch / s.b1, b1 = batch % s.b1;
  const float* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1;
  const float* b = rhs + b0 * s.rhs_b0 + b1 * s.rhs_b1;
  float* o = out + b0 * s.out_b0 + b1 * s.out_b1;
  const int64_t m0 = (int64_t)blockIdx.y * kSgBM, n0 = (int64_t)blockIdx.x * kSgBN;
  // Global -> register mapping: A slab = 128 rows x 4 chunks of 4 k (two chunks per thread), B slab = 16 rows x 16
  // chunks of 4 n (one per thread).
  const int a_row[2] = {tid >> 2, (tid + 256) >> 2}, a_kc = tid & 3;
  const int b_row = tid >> 4, b_nc = tid & 15;
  float4 ra[2], rb;
  auto gload = [&](int64_t k0) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int64_t gm = m0 + a_row[i], gk = k0 + a_kc * 4;
      if (gm < s.m && gk + 3 < s.k) {
        ra[i] = *reinterpret_cast<const float4*>(a + gm * s.lhs_m + gk);
      } else {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = (gm < s.m && gk + j < s.k) ? a[gm * s.lhs_m + gk + j] : 0.f;
        ra[i] = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
    const int64_t gk = k0 + b_row, gn = n0 + b_nc * 4;
    if (gk < s.k && gn + 3 < s.n) {
      rb = *reinterpret_cast<const float4*>(b + gk * s.rhs_k + gn);
    } else {
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) v[j] = (gk < s.k && gn + j < s.n) ? b[gk * s.rhs_k + gn + j] : 0.f;
      rb = make_float4(v[0], v[1], v[2], v[3]);
    }
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      As[buf][a_kc * 4 + 0][a_row[i]] = ra[i].x;
      As[buf][a_kc * 4 + 1][a_row[i]] = ra[i].y;
      As[buf][a_kc * 4 + 2][a_row[i]] = ra[i].z;
      As[buf][a_kc * 4 + 3][a_row[i]] = ra[i].w;
    }
    *reinterpret_cast<float4*>(&Bs[buf][b_row][b_nc * 4]) = rb;
  };
  const int tx = tid & 15, ty = tid >> 4;  // outputs: rows ty * 8 .. + 7, columns tx * 4 .. + 3
  float acc[8][4] = {};
  const int64_t slabs = (s.k + kSgBK - 1) / kSgBK;
  gload(0);
  sstore(0);
  __syncthreads();
  for (int64_t t = 0; t < slabs; t++) {
    const int buf = (int)(t & 1);
    if (t + 1 < slabs) gload((t + 1) * kSgBK);
#pragma unroll
    for (int kk = 0; kk < kSgBK; kk++) {
      const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8]);
      const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8 + 4]);
      const float4 bv = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bw[j], acc[i][j]);
    }
    if (t + 1 < slabs) sstore(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int64_t gm = m0 + ty * 8 + i, gn = n0 + tx * 4;
    if (gm >= s.m) continue;
    float* dst = o + gm * s.out_m + gn;
    if (gn + 3 < s.n && (s.out_m & 3) == 0) {
      *reinterpret_cast<float4*>(dst) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (gn + j < s.n) dst[j] = acc[i][j];
    }
  }
}

// True when the register-blocked f32 kernel can take the contraction as it lies in memory.
inline bool sgemm_ok(const DotShape& s, const void* lhs, const void* rhs, const void* out) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return s.dtype == kF32 && s.lhs_k == 1 && s.rhs_n == 1 && (s.lhs_m & 3) == 0 && (s.rhs_k & 3) == 0 && (s.lhs_b0 & 3) == 0 &&
         (s.lhs_b1 & 3) == 0 && (s.rhs_b0 & 3) == 0 && (s.rhs_b1 & 3) == 0 && (s.out_b0 & 3) == 0 && (s.out_b1 & 3) == 0 &&
         al16(lhs) && al16(rhs) && al16(out) && (s.m + kSgBM - 1) / kSgBM <= 65535;
}

// ---------------------------------------------------------------- 64 x 64 tiles, k split over a cluster
// out[m, n] = sum_k lhs[m, k] * rhs[k, n] in true f32, lhs k-contiguous, rhs n-contiguous, any pitch: f32 contractions that
// do not fill the chip with the tiles of the kernel above or do not have its 16-byte rows, and 16-bit ones of pitches the
// tensor cores cannot take, widened on the way in. Those ran one or a few CTAs through all of k with a load, a barrier and
// a latency per slab of 16.
// 64 x 64 outputs per CTA of 64 threads, 8 x 8 per thread, k in slabs of 16 through two shared-memory buffers; the next slab
// travels (cp.async for f32) while the current one is multiplied. `split` CTAs of a cluster contract a slice of k each and
// sum their tiles through distributed shared memory in rank order.
// Measured: a call with a small ragged product 112 -> 49 us; 333 x 1777 x 777 f32 74 us, issue slots 57 % busy, one
// scalar cp.async per element of its odd rows. The 16-bit form spills 94 bytes at its bound of 168 registers (six CTAs per SM;
// its slab waits in registers), the f32 forms none. Where 128 x 64 tiles fill the chip the kernel above is ahead
// (1024^3 70 us against 75 here: both are bound by shared-memory reads beside the FMAs, and this one also sums four parts).
constexpr int kSplitTile = 64, kSplitBK = 16, kSplitThreads = 64, kSplitPad = 4;

__device__ __forceinline__ void cp_async(void* dst, const void* src, int bytes, bool vec) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (vec) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kSplitThreads, sizeof(T) == 4 ? 8 : 6)
split_tile_kernel(DotShape s, const T* __restrict__ lhs, const T* __restrict__ rhs, T* __restrict__ out, int split) {
  constexpr bool F32 = sizeof(T) == 4;
  __shared__ __align__(16) float smem[2 * kSplitTile * (kSplitBK + kSplitPad) + 2 * kSplitBK * kSplitTile];
  float (*As)[kSplitTile][kSplitBK + kSplitPad] = reinterpret_cast<float (*)[kSplitTile][kSplitBK + kSplitPad]>(smem);
  float (*Bs)[kSplitBK][kSplitTile] = reinterpret_cast<float (*)[kSplitBK][kSplitTile]>(smem + 2 * kSplitTile * (kSplitBK + kSplitPad));
  PJRTX_PDL_PROLOGUE();
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int rank = (int)blockIdx.x % split;
  const int64_t batch = blockIdx.z, b0 = batch / s.b1, b1 = batch % s.b1;
  const T* a = lhs + b0 * s.lhs_b0 + b1 * s.lhs_b1;
  const T* b = rhs + b0 * s.rhs_b0 + b1 * s.rhs_b1;
  T* o = out + b0 * s.out_b0 + b1 * s.out_b1;
  const int64_t m0 = (int64_t)blockIdx.y * kSplitTile, n0 = (int64_t)(blockIdx.x / split) * kSplitTile;
  const int64_t slabs = (s.k + kSplitBK - 1) / kSplitBK;
  const int64_t first = rank * slabs / split, last = (rank + 1) * slabs / split;

  T ra[F32 ? 1 : 16], rb[F32 ? 1 : 16];  // 16-bit operands pass through registers
  auto request = [&](int64_t slab, int buf) {
    const int64_t k0 = slab * kSplitBK;
    if constexpr (F32) {
      if (VEC) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = (tid >> 2) + 16 * i, kc = (tid & 3) * 4;  // lhs: 64 rows x 4 chunks
          const int64_t left = m0 + row < s.m ? s.k - k0 - kc : 0;
          cp_async(&As[buf][row][kc], left > 0 ? a + (m0 + row) * s.lhs_m + k0 + kc : a, (int)(left <= 0 ? 0 : left < 4 ? left : 4) * 4, true);
          const int kr = (tid >> 4) + 4 * i, nc = (tid & 15) * 4;  // rhs: 16 rows x 16 chunks
          const int64_t wide = k0 + kr < s.k ? s.n - n0 - nc : 0;
          cp_async(&Bs[buf][kr][nc], wide > 0 ? b + (k0 + kr) * s.rhs_k + n0 + nc : b, (int)(wide <= 0 ? 0 : wide < 4 ? wide : 4) * 4, true);
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < 16; i++) {
          const int row = (tid >> 4) + 4 * i, kc = tid & 15;
          const bool in = m0 + row < s.m && k0 + kc < s.k;
          cp_async(&As[buf][row][kc], in ? a + (m0 + row) * s.lhs_m + k0 + kc : a, in ? 4 : 0, false);
          const bool inb = k0 + i < s.k && n0 + tid < s.n;
          cp_async(&Bs[buf][i][tid], inb ? b + (k0 + i) * s.rhs_k + n0 + tid : b, inb ? 4 : 0, false);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    } else {
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const int row = (tid >> 4) + 4 * i, kc = tid & 15;
        ra[i] = m0 + row < s.m && k0 + kc < s.k ? a[(m0 + row) * s.lhs_m + k0 + kc] : from_f<T>(0.f);
        rb[i] = k0 + i < s.k && n0 + tid < s.n ? b[(k0 + i) * s.rhs_k + n0 + tid] : from_f<T>(0.f);
      }
    }
  };
  auto deposit = [&](int buf) {
    if constexpr (!F32) {
#pragma unroll
      for (int i = 0; i < 16; i++) {
        As[buf][(tid >> 4) + 4 * i][tid & 15] = to_f(ra[i]);
        Bs[buf][i][tid] = to_f(rb[i]);
      }
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
  };
  float acc[8][8] = {};  // rows ty + 8 i, columns 32 h + 4 tx + j
  if (first < last) {
    request(first, 0);
    deposit(0);
  }
  __syncthreads();
  for (int64_t t = first; t < last; t++) {
    const int buf = (int)((t - first) & 1);
    if (t + 1 < last) request(t + 1, buf ^ 1);
#pragma unroll
    for (int k4 = 0; k4 < kSplitBK; k4 += 4) {
      float4 av[8];
#pragma unroll
      for (int i = 0; i < 8; i++) av[i] = *reinterpret_cast<const float4*>(&As[buf][ty + 8 * i][k4]);
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        const float4 blo = *reinterpret_cast<const float4*>(&Bs[buf][k4 + kk][4 * tx]);
        const float4 bhi = *reinterpret_cast<const float4*>(&Bs[buf][k4 + kk][32 + 4 * tx]);
        const float bw[8] = {blo.x, blo.y, blo.z, blo.w, bhi.x, bhi.y, bhi.z, bhi.w};
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float ai = kk == 0 ? av[i].x : kk == 1 ? av[i].y : kk == 2 ? av[i].z : av[i].w;
#pragma unroll
          for (int j = 0; j < 8; j++) acc[i][j] = fmaf(ai, bw[j], acc[i][j]);
        }
      }
    }
    if (t + 1 < last) deposit(buf ^ 1);
    __syncthreads();
  }
  auto store = [&](int i, int h, float4 v) {
    const int64_t gm = m0 + ty + 8 * i, gn = n0 + 32 * h + 4 * tx;
    if (gm >= s.m) return;
    T* dst = o + gm * s.out_m + gn;
    if (VEC && F32 && gn + 3 < s.n) {
      *reinterpret_cast<float4*>(dst) = v;
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (gn + j < s.n) dst[j] = from_f<T>(e[j]);
    }
  };
  if (split == 1) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int h = 0; h < 2; h++) store(i, h, make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]));
    return;
  }
  // The slabs' memory receives the cluster's tiles: [source CTA][rows i of this CTA][h][thread], once every CTA is done.
  const int rows = 8 / split;
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  const unsigned base = (unsigned)__cvta_generic_to_shared(smem) + (unsigned)tid * 16u;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    unsigned remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(base), "r"(i / rows));
#pragma unroll
    for (int h = 0; h < 2; h++)
      asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote + (unsigned)(((rank * rows + i % rows) * 2 + h) * kSplitThreads * 16)),
                   "f"(acc[i][4 * h]), "f"(acc[i][4 * h + 1]), "f"(acc[i][4 * h + 2]), "f"(acc[i][4 * h + 3])
                   : "memory");
  }
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  const float4* got = reinterpret_cast<const float4*>(smem) + tid;
  for (int r = 0; r < rows; r++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      float4 v = got[(r * 2 + h) * kSplitThreads];
      for (int q = 1; q < split; q++) {
        const float4 w = got[((q * rows + r) * 2 + h) * kSplitThreads];
        v.x += w.x;
        v.y += w.y;
        v.z += w.z;
        v.w += w.w;
      }
      store(rank * rows + r, h, v);
    }
}

// True when the split-tile kernel can take the contraction as it lies in memory.
inline bool split_tile_ok(const DotShape& s) {
  return s.lhs_k == 1 && s.rhs_n == 1 && (s.m + kSplitTile - 1) / kSplitTile <= 65535 && (s.n + kSplitTile - 1) / kSplitTile <= (1ll << 27);
}
// CTAs per tile: pieces of at least 64 k, doubled until there are four CTAs for every SM (four to seven then).
inline int split_tile_parts(const DotShape& s, int64_t batch, int sm_count) {
  const int64_t tiles = (s.m + kSplitTile - 1) / kSplitTile * ((s.n + kSplitTile - 1) / kSplitTile) * batch;
  int split = 1;
  while (split < 8 && tiles * split < (int64_t)sm_count * 4 && s.k / (2 * split) >= 64) split *= 2;
  return split;
}
// 128 x 64 tiles (sgemm_kernel, where its 16-byte rows apply): for a k of up to 128, where a split buys nothing (64 x 64
// x 64 and 200 x 64 x 1024 10.8 us, split tiles 12.8; 500 x 128 x 1024 15.1 / 16.8, 500 x 256 x 1024 23 / 19), and where they give more than three
// quarters of the SMs a CTA (1024^3 70 us, split tiles 75; 500 x 1024 x 1024, 64 CTAs, 70 / 44).
inline bool wide_tiles_pay(const DotShape& s, int64_t batch, int sm_count) {
  return s.k <= 128 || (s.n + kSgBN - 1) / kSgBN * ((s.m + kSgBM - 1) / kSgBM) * batch > sm_count * 3 / 4;
}
// Whether split tiles pay against what runs otherwise: one thread per output (up to eight rows) or tile_kernel (16-bit, more
// rows; f32 always splits there: 9 x 77 x 96 of cold weights 17 us against 23, 500 x 4099 x 256 60 / 70, both near equal at k = 16).
// A tile costs its 64 rows whatever m is, so few rows of many tiles belong to the threads, whose time hardly depends on n up
// to 64000 outputs. Measured, threads / split tiles, us, weights in L2 and cold where that differs: f32 1 x 257 x 8001 33 / 25,
// x 16001 33 / 40 and 83 / 40, x 32001 34 / 64, x 64001 35 / 109; 1 x 2049 x 32001 594 / 400, x 40001 596 / 592, x 64001 592 /
// 777; 4 x 513 x 32001 76 / 113, 4 x 1025 x 64001 549 / 394, 8 x 2049 x 64001 1589 / 776. 16-bit, where a slab waits in
// registers: 5 x 65 x 1001 17 / 21, 4 x 129 x 8001 27 / 25, 4 x 257 x 16001 50 / 56, 4 x 513 x 16001 92 / 89, 2 x 129 x 32001
// 29 / 56, 2 x 2049 x 64001 848 / 1392, 8 x 513 x 32001 167 / 154; tile_kernel / split tiles 64 x 97 x 1001 21 / 29, 64 x 193
// x 1001 34 / 31, 1000 x 257 x 1001 52 / 58, 1000 x 513 x 1001 95 / 93, 500 x 513 x 4001 141 / 158, 1000 x 2049 x 4001 868 / 1078.
inline bool split_tiles_pay(const DotShape& s, int64_t batch, int sm_count) {
  const int64_t tiles = (s.m + kSplitTile - 1) / kSplitTile * ((s.n + kSplitTile - 1) / kSplitTile) * batch;
  if (dtype_size(s.dtype) == 2)
    return s.k >= 128 && (tiles <= sm_count || (tiles <= 2 * sm_count && s.k >= 512) || (s.m > 6 && s.m <= 8 && s.k >= 512));
  if (s.m > 8) return true;
  if (s.k < 64) return false;
  return tiles <= 2 * sm_count || s.m > 6 || (s.m > 3 && s.k >= 768) || (s.k >= 1024 && 2 * tiles <= 7 * sm_count);
}

template <typename T>
int launch_split_tile(const DotShape& s, const T* a, const T* b, T* o, int64_t batch, int split, bool pdl, cudaStream_t stream) {
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const bool vec = sizeof(T) == 4 && (s.lhs_m & 3) == 0 && (s.rhs_k & 3) == 0 && (s.out_m & 3) == 0 && (s.lhs_b0 & 3) == 0 &&
                   (s.lhs_b1 & 3) == 0 && (s.rhs_b0 & 3) == 0 && (s.rhs_b1 & 3) == 0 && (s.out_b0 & 3) == 0 && (s.out_b1 & 3) == 0 &&
                   al16(a) && al16(b) && al16(o);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((s.n + kSplitTile - 1) / kSplitTile * split), (unsigned)((s.m + kSplitTile - 1) / kSplitTile), (unsigned)batch);
  cfg.blockDim = dim3(kSplitThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  cfg.attrs = attr;
  cfg.numAttrs = fill_launch_attributes(attr, pdl);
  if (split > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)split;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    cfg.numAttrs++;
  }
  if (vec) return cudaLaunchKernelEx(&cfg, split_tile_kernel<T, sizeof(T) == 4>, s, a, b, o, split) == cudaSuccess ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, split_tile_kernel<T, false>, s, a, b, o, split) == cudaSuccess ? 1 : 0;
}

// ---------------------------------------------------------------- small streaming contractions
// out[m, n] = sum_k lhs[m, k] * rhs[k, n] for m <= 8, n contiguous and k so small (small_max_k) that a CTA can hold its
// whole share of the rhs in registers: toy decoders, closed-over blocks. What bounds such a contraction is the chain of
// dependent latencies, not bytes. The persistent kernel's chain is tensor map -> copy -> mbarrier -> partial sums in global
// memory -> arrival counter -> fold; here a CTA owns 64 columns for all of k, requests every 16-byte piece of its weights
// at once (before the preceding kernel has finished, where nothing writes them), then the lhs, multiplies, and folds the
// eight warps through shared memory in a fixed order. (16-bit at eight rows would spill 72 bytes; 16-bit operands come
// here with one and two rows only, from three up the tensor cores take them wherever rows are aligned.)
constexpr int kSmallCols = 64, kSmallThreads = 256, kSmallPasses = 16;
// Rows a CTA covers in one round of loads: 8 warps x 32 lanes x 16 bytes over 64 columns.
__host__ __device__ constexpr int small_rows_per_pass(int esize) { return kSmallThreads * 16 / (kSmallCols * esize); }
__host__ __device__ constexpr int small_max_k(int esize) { return kSmallPasses * small_rows_per_pass(esize); }

struct SmallGroup {
  int count;
  int tile_begin[kDotGroupMax + 1];
  const void* rhs[kDotGroupMax];
  void* out[kDotGroupMax];
  long long n[kDotGroupMax], rhs_k[kDotGroupMax], out_m[kDotGroupMax];
  int m, k;
  long long lhs_m, lhs_k;
  int early_rhs;
};

template <typename T, int M>
__global__ void __launch_bounds__(kSmallThreads) small_dot_kernel(SmallGroup grp, const T* __restrict__ lhs) {
  constexpr int V = 16 / sizeof(T), LANES = kSmallCols / V, RP = small_rows_per_pass(sizeof(T));
  __shared__ float fold[kSmallThreads / 32][M][kSmallCols];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  int g = 0;
#pragma unroll
  for (int q = 1; q < kDotGroupMax; q++)
    if (q < grp.count && (int)blockIdx.x >= grp.tile_begin[q]) g = q;
  const long long n0 = (long long)((int)blockIdx.x - grp.tile_begin[g]) * kSmallCols;
  const int chunk = threadIdx.x % LANES, row0 = threadIdx.x / LANES;  // this thread: V columns of rows row0, row0 + RP, ...
  const long long n = n0 + chunk * V;
  const bool in = n < grp.n[g];  // (n is a multiple of V)
  const T* rhs = static_cast<const T*>(grp.rhs[g]) + n;
  uint4 w[kSmallPasses];
  auto load_rhs = [&]() {
#pragma unroll
    for (int i = 0; i < kSmallPasses; i++) {
      const int k = row0 + i * RP;
      w[i] = in && k < grp.k ? ld_stream(rhs + (long long)k * grp.rhs_k[g]) : make_uint4(0, 0, 0, 0);
    }
  };
  if (grp.early_rhs) load_rhs();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!grp.early_rhs) load_rhs();
  float acc[M][V];
#pragma unroll
  for (int m = 0; m < M; m++)
#pragma unroll
    for (int j = 0; j < V; j++) acc[m][j] = 0.f;
  float x[M][kSmallPasses];
#pragma unroll
  for (int m = 0; m < M; m++)
#pragma unroll
    for (int i = 0; i < kSmallPasses; i++) {
      const int k = row0 + i * RP;
      x[m][i] = m < grp.m && k < grp.k ? to_f(__ldcg(lhs + m * grp.lhs_m + k * grp.lhs_k)) : 0.f;
    }
#pragma unroll
  for (int i = 0; i < kSmallPasses; i++) {
    const T* e = reinterpret_cast<const T*>(&w[i]);
#pragma unroll
    for (int j = 0; j < V; j++) {
      const float v = to_f(e[j]);
#pragma unroll
      for (int m = 0; m < M; m++) acc[m][j] = fmaf(x[m][i], v, acc[m][j]);
    }
  }
  // Lanes of a warp that hold the same columns, then the eight warps.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int m = 0; m < M; m++)
#pragma unroll
    for (int j = 0; j < V; j++) {
#pragma unroll
      for (int o = LANES; o < 32; o <<= 1) acc[m][j] += __shfl_xor_sync(0xffffffffu, acc[m][j], o);
      if (lane < LANES) fold[warp][m][lane * V + j] = acc[m][j];
    }
  __syncthreads();
  for (int o = threadIdx.x; o < M * kSmallCols; o += kSmallThreads) {
    const int m = o / kSmallCols, c = o % kSmallCols;
    float v = fold[0][m][c];
#pragma unroll
    for (int q = 1; q < kSmallThreads / 32; q++) v += fold[q][m][c];
    if (m < grp.m && n0 + c < grp.n[g]) static_cast<T*>(grp.out[g])[m * grp.out_m[g] + n0 + c] = from_f<T>(v);
  }
}

template <typename T>
int launch_small(const DotShape* shapes, int count, const void* lhs, const void* const* rhs, void* const* out, bool early_rhs, bool pdl,
                 cudaStream_t stream) {
  const DotShape& s = shapes[0];
  SmallGroup grp{};
  grp.count = count;
  int tiles = 0;
  for (int g = 0; g < count; g++) {
    if ((reinterpret_cast<uintptr_t>(rhs[g]) & 15) != 0) return 0;
    grp.tile_begin[g] = tiles;
    tiles += (int)((shapes[g].n + kSmallCols - 1) / kSmallCols);
    grp.rhs[g] = rhs[g];
    grp.out[g] = out[g];
    grp.n[g] = shapes[g].n;
    grp.rhs_k[g] = shapes[g].rhs_k;
    grp.out_m[g] = shapes[g].out_m;
  }
  for (int g = count; g <= kDotGroupMax; g++) grp.tile_begin[g] = tiles;
  grp.m = (int)s.m;
  grp.k = (int)s.k;
  grp.lhs_m = s.lhs_m;
  grp.lhs_k = s.lhs_k;
  grp.early_rhs = early_rhs ? 1 : 0;
  const T* a = static_cast<const T*>(lhs);
  cudaError_t e;
#define SMALL(MM) e = launch_kernel(small_dot_kernel<T, MM>, dim3((unsigned)tiles), dim3(kSmallThreads), 0, stream, pdl, grp, a)
  if (s.m <= 1) SMALL(1); else if (s.m <= 2) SMALL(2); else if (s.m <= 4) SMALL(4); else SMALL(8);
#undef SMALL
  return e == cudaSuccess ? 1 : 0;
}

template <typename T>
int launch_group_typed(const DotShape* shapes, int count, const DotScratch& plan, const void* lhs, const void* const* rhs,
                       void* const* out, void* partials, void* counters, bool pdl, cudaStream_t stream) {
  constexpr int V = 16 / sizeof(T);
  const int tile = 32 * V;
  const DotShape& s = shapes[0];
  const int M = s.m <= 1 ? 1 : s.m <= 2 ? 2 : s.m <= 4 ? 4 : 8;
  KnGroup grp{};
  grp.count = count;
  int tiles = 0;
  long long poff = 0;
  for (int g = 0; g < count; g++) {
    grp.tile_begin[g] = tiles;
    tiles += (int)((shapes[g].n + tile - 1) / tile);
    grp.rhs[g] = rhs[g];
    grp.out[g] = out[g];
    grp.n[g] = shapes[g].n;
    grp.rhs_k[g] = shapes[g].rhs_k;
    grp.partial_offset[g] = poff;
    poff += (long long)s.b0 * s.b1 * plan.ksplit * M * shapes[g].n;
  }
  for (int g = count; g <= kDotGroupMax; g++) grp.tile_begin[g] = tiles;
  dim3 grid((unsigned)tiles, (unsigned)plan.ksplit, (unsigned)(s.b0 * s.b1));
  const int kslice = (int)((s.k + plan.ksplit - 1) / plan.ksplit);
  const T* a = static_cast<const T*>(lhs);
  float* p = static_cast<float*>(partials);
  unsigned* c = static_cast<unsigned*>(counters);
  cudaError_t e;
#define KN(MM, WW) e = launch_kernel(stream_kn_kernel<T, MM, WW>, grid, dim3(WW * 32), 0, stream, pdl, s, grp, a, p, c, plan.ksplit, kslice)
  if (M == 1) KN(1, 8); else if (M == 2) KN(2, 8); else if (M == 4) KN(4, 8); else KN(8, 4);
#undef KN
  return e == cudaSuccess ? 1 : 0;
}

template <typename T>
int launch_typed(const DotShape& s, const DotScratch& plan, const void* lhs, const void* rhs, void* out, void* partials,
                 void* counters, bool pdl, cudaStream_t stream) {
  const T* a = static_cast<const T*>(lhs);
  const T* b = static_cast<const T*>(rhs);
  T* o = static_cast<T*>(out);
  constexpr int V = 16 / sizeof(T);
  const int64_t batch = s.b0 * s.b1;
  if (plan.path == 1) {
    const DotShape* one = &s;
    const void* rhs_list[1] = {rhs};
    void* out_list[1] = {out};
    return launch_group_typed<T>(one, 1, plan, lhs, rhs_list, out_list, partials, counters, pdl, stream);
  }
  if (plan.path == 2) {
    int group = 32;
    while (group > 1 && (int64_t)group * V > s.k) group >>= 1;
    const int rows_per_cta = 8 * (32 / group);
    dim3 grid((unsigned)((s.n + rows_per_cta - 1) / rows_per_cta), (unsigned)batch);
    cudaError_t e;
#define NK(MM) e = launch_kernel(stream_nk_kernel<T, MM>, grid, dim3(256), 0, stream, pdl, s, a, b, o, group)
    if (s.m <= 1) NK(1); else if (s.m <= 2) NK(2); else if (s.m <= 4) NK(4); else NK(8);
#undef NK
    return e == cudaSuccess ? 1 : 0;
  }
  if (plan.path == 3) {
    if (plan.wide && sgemm_ok(s, lhs, rhs, out)) {
      dim3 grid((unsigned)((s.n + kSgBN - 1) / kSgBN), (unsigned)((s.m + kSgBM - 1) / kSgBM), (unsigned)batch);
      return launch_kernel(sgemm_kernel, grid, dim3(256), 0, stream, pdl, s, (const float*)lhs, (const float*)rhs, (float*)out) == cudaSuccess ? 1 : 0;
    }
    if (plan.ksplit > 0 && split_tile_ok(s)) return launch_split_tile<T>(s, a, b, o, batch, plan.ksplit, pdl, stream);
    dim3 grid((unsigned)((s.n + kTile - 1) / kTile), (unsigned)((s.m + kTile - 1) / kTile), (unsigned)batch);
    return launch_kernel(tile_kernel<T>, grid, dim3(256), 0, stream, pdl, s, a, b, o) == cudaSuccess ? 1 : 0;
  }
  const int64_t total = batch * s.m * s.n;
  const unsigned blocks = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 32);
  return launch_kernel(dot_generic_kernel<T>, dim3(blocks ? blocks : 1), dim3(256), 0, stream, pdl, s, a, b, o) == cudaSuccess ? 1 : 0;
}

}  // namespace

namespace {
int umma_eligible(const DotShape& s);
DotScratch umma_plan(const DotShape* shapes, int count, int sm_count, int kind);
}  // namespace

namespace {
int env_int(const char* name, int fallback) {
  const char* v = getenv(name);
  return v && *v ? atoi(v) : fallback;
}
}  // namespace

unsigned long long wait_timeout_ns() {
  static const unsigned long long ns = [] {
    const int ms = env_int("PJRTX_B200_WAIT_TIMEOUT_MS", 2000);
    return (unsigned long long)(ms < 1 ? 1 : ms) * 1000000ull;
  }();
  return ns;
}

namespace {
// Ring depth and CTAs per SM of the TMA streaming kernel: two CTAs per SM with three 32 KiB stages each while the
// cross-warp fold buffer is small (m <= 2 for 16-bit types), one CTA with a deeper ring otherwise.
void tma_ring(int M, int V, int* stages, int* per_sm) {
  const size_t red = (size_t)tma::kConsumerWarps * M * 32 * V * sizeof(float);
  const bool two = red <= 16 * 1024;
  *per_sm = two ? 2 : 1;
  *stages = two ? 3 : (M <= 4 ? 5 : 4);
  static const int env_stages = env_int("PJRTX_B200_TMA_STAGES", 0);
  if (env_stages >= 2 && env_stages <= 6) *stages = env_stages;
}
}  // namespace

DotScratch dot_group_plan(const DotShape* shapes, int count, int sm_count, bool allow_tensor) {
  DotScratch p;
  p.path = 1;
  const DotShape& s = shapes[0];
  const int esize = (int)dtype_size(s.dtype);
  const int V = 16 / esize;
  const int64_t batch = s.b0 * s.b1;
  int64_t tiles = 0, n_total = 0;
  for (int g = 0; g < count; g++) {
    tiles += (shapes[g].n + 32 * V - 1) / (32 * V);
    n_total += shapes[g].n;
  }
  const int M = s.m <= 1 ? 1 : s.m <= 2 ? 2 : s.m <= 4 ? 4 : 8;
  if (batch == 1 && allow_tensor) {
    bool all_umma = true;
    for (int g = 0; g < count; g++) all_umma &= umma_eligible(shapes[g]) == 1;
    if (all_umma) return umma_plan(shapes, count, sm_count, 1);
  }
  if (batch == 1) {
    // A k that one round of loads covers and few CTAs: the kernel without rings and folds, and without
    // scratch. Measured: eight steps of a toy decoder (72 such launches) 1290 us on the persistent kernel and 1233 on this
    // one, together with the generated kernels' vector reads; a toy f32 block (seven such launches) 55 us on either.
    int64_t small_tiles = 0;
    for (int g = 0; g < count; g++) small_tiles += (shapes[g].n + kSmallCols - 1) / kSmallCols;
    // Persistent TMA kernel: equal shares of (column tile, row chunk) units per CTA, two CTAs per SM with a ring of
    // 32 KiB stages each. Measured on the 8B-shape decode step (ms per step): two CTAs x 3 stages 3.50; one CTA x 5
    // stages 3.67; two CTAs x 6 stages of 16 KiB 3.94; one CTA x 6 stages of 16 KiB 4.95.
    p.tma = 1;
    // Where the persistent kernel's launch is as short, it stays: five to eight rows of a k up to 64 (8 x 64 x 1024 f32 8.9
    // us, 10.9 here) or of many tiles (8 x 256 x 4736 11 / 13 of cold weights), three and four rows of a wave (4 x 256 x 9472
    // 10.8 / 12.9).
    const int64_t most = s.m > 4 ? sm_count / 8 : s.m > 2 ? sm_count * 3 / 4 : sm_count;
    if (allow_tensor && s.k <= small_max_k(esize) && small_tiles <= most && (s.m <= 4 || s.k > 64)) {
      p.small = 1;
      p.grid = (int)small_tiles;
      return p;
    }
    const int chunks = (int)((s.k + tma::kUnitRows - 1) / tma::kUnitRows);
    const int64_t units = tiles * chunks;
    int per_sm = 1;
    tma_ring(M, V, &p.stages, &per_sm);
    // A fixed grid of one (or two) CTAs per SM; units are dealt out evenly (shares differ by at most one unit).
    const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>(units, (int64_t)sm_count * per_sm));
    p.grid = (int)ctas;
    p.per_cta = units / ctas;
    p.max_contrib = (int)((chunks + p.per_cta - 1) / p.per_cta) + 1;
    p.smem = tma::smem_bytes(p.stages, M, 32 * V);
    p.ksplit = p.max_contrib;
    p.partial_bytes = (uint64_t)tiles * p.max_contrib * M * 32 * V * sizeof(float);
    p.counter_bytes = (uint64_t)tiles * sizeof(unsigned);
    return p;
  }
  // About two CTAs per SM, every CTA streaming at least 256 rows of its tile.
  const int64_t want = ((int64_t)sm_count * 2 + tiles * batch - 1) / (tiles * batch);
  const int64_t max_split = std::max<int64_t>(1, s.k / 256);
  p.ksplit = (int)std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(want, max_split), 32));
  if (p.ksplit > 1) {
    p.partial_bytes = (uint64_t)batch * p.ksplit * M * n_total * sizeof(float);
    p.counter_bytes = (uint64_t)batch * tiles * sizeof(unsigned);
  }
  return p;
}

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
    return (EncodeTiledFn)p;
  }();
  return fn;
}

template <typename T, int M, bool EXTRAS>
int launch_tma_m(const tma::Params& prm, const tma::Maps& maps, int grid, size_t smem, bool pdl, cudaStream_t stream) {
  if (!raise_smem_limit((const void*)tma::stream_tma_kernel<T, M, EXTRAS>, 200 * 1024)) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(tma::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = fill_launch_attributes(attr, pdl);
  return cudaLaunchKernelEx(&cfg, tma::stream_tma_kernel<T, M, EXTRAS>, prm, maps) == cudaSuccess ? 1 : 0;
}

// Fills one segment of the kernel parameters (and its tensor maps) from a group of contractions sharing an lhs.
template <typename T>
bool fill_segment(const DotShape* shapes, int count, const DotLhs& lhs_desc, const void* lhs, const void* lhs2,
                  const void* const* rhs, void* const* out, const void* const* residual, int max_contrib, float* partials,
                  unsigned* counters, tma::Segment* sg, CUtensorMap* maps) {
  constexpr int V = 16 / sizeof(T);
  constexpr int COLS = 32 * V;
  const DotShape& s = shapes[0];
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  sg->lhs = lhs;
  sg->lhs2 = lhs2;
  sg->lhs_m = s.lhs_m;
  sg->lhs_k = s.lhs_k;
  sg->lhs_kind = lhs_desc.kind;
  sg->norm_scale = lhs_desc.norm_scale;
  sg->norm_eps = lhs_desc.norm_eps;
  sg->m = (int)s.m;
  sg->k = (int)s.k;
  sg->count = count;
  int tiles = 0;
  const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  for (int g = 0; g < count; g++) {
    sg->tile_begin[g] = tiles;
    tiles += (int)((shapes[g].n + COLS - 1) / COLS);
    sg->out[g] = out[g];
    sg->residual[g] = residual ? residual[g] : nullptr;
    sg->n[g] = shapes[g].n;
    cuuint64_t gdim[2] = {(cuuint64_t)shapes[g].n, (cuuint64_t)s.k};
    cuuint64_t gstride[1] = {(cuuint64_t)shapes[g].rhs_k * sizeof(T)};
    cuuint32_t box[2] = {(cuuint32_t)COLS, (cuuint32_t)tma::kUnitRows};
    cuuint32_t estr[2] = {1, 1};
    if (enc(&maps[g], dt, 2, const_cast<void*>(rhs[g]), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  for (int g = count; g <= tma::kGroupMax; g++) sg->tile_begin[g] = tiles;
  for (int g = count; g < tma::kGroupMax; g++) maps[g] = maps[0];
  sg->chunks = (int)((s.k + tma::kUnitRows - 1) / tma::kUnitRows);
  sg->units = (long long)tiles * sg->chunks;
  sg->max_contrib = max_contrib;
  sg->partials = partials;
  sg->counters = counters;
  sg->ssq_out = nullptr;
  sg->ssq_in = nullptr;
  sg->ssq_tiles = 0;
  return true;
}

template <typename T>
int launch_tma_params(tma::Params& p, const tma::Maps& maps, int m, int grid, int stages, size_t smem, int* error_flag,
                      bool early_rhs, bool pdl, cudaStream_t stream) {
  p.error_flag = error_flag;
  p.timeout_ns = wait_timeout_ns();
  p.stages = stages;
  p.early_rhs = early_rhs ? 1 : 0;
  static const int env_evict = env_int("PJRTX_B200_TMA_EVICT_FIRST", 1);
  p.evict_first = env_evict;
  const int M = m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : 8;
  // The plain contraction (one segment, untransformed lhs, no residual) runs the kernel without the segment machinery.
  bool extras = p.segments > 1 || p.seg[0].lhs_kind != tma::kLhsPlain;
  for (int g = 0; g < p.seg[0].count; g++) extras |= p.seg[0].residual[g] != nullptr;
#define GO(MM) (extras ? launch_tma_m<T, MM, true>(p, maps, grid, smem, pdl, stream) : launch_tma_m<T, MM, false>(p, maps, grid, smem, pdl, stream))
  switch (M) {
    case 1: return GO(1);
    case 2: return GO(2);
    case 4: return GO(4);
    default: return GO(8);
  }
#undef GO
}

template <typename T>
int launch_tma(const DotShape* shapes, int count, const DotScratch& plan, const void* lhs, const void* const* rhs, void* const* out,
               void* partials, void* counters, int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream) {
  tma::Params p{};
  tma::Maps maps{};
  p.segments = 1;
  p.barrier = nullptr;
  if (!fill_segment<T>(shapes, count, DotLhs{}, lhs, nullptr, rhs, out, nullptr, plan.max_contrib, static_cast<float*>(partials),
                       static_cast<unsigned*>(counters), &p.seg[0], maps.map[0]))
    return 0;
  return launch_tma_params<T>(p, maps, (int)shapes[0].m, plan.grid, plan.stages, plan.smem, error_flag, early_rhs, pdl, stream);
}

template <typename T>
int launch_chain(const DotChainSegment* segs, const DotChainArgs* args, int n, const DotChainPlan& plan, void* partials,
                 void* counters, int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream) {
  tma::Params p{};
  tma::Maps maps{};
  p.segments = n;
  unsigned* words = static_cast<unsigned*>(counters);
  p.barrier = words;  // the barrier words come first, then every segment's tile counters
  for (int s = 0; s < n; s++) {
    if (!fill_segment<T>(segs[s].shapes, segs[s].count, segs[s].lhs, args[s].lhs, args[s].lhs2, args[s].rhs, args[s].out,
                         args[s].residual, plan.max_contrib[s], static_cast<float*>(partials),
                         words + plan.counter_offset[s] / sizeof(unsigned), &p.seg[s], maps.map[s]))
      return 0;
  }
  for (int s = 0; s + 1 < n; s++)
    if (plan.ssq_offset[s]) {
      float* ssq = reinterpret_cast<float*>(static_cast<unsigned char*>(counters) + plan.ssq_offset[s]);
      p.seg[s].ssq_out = ssq;
      p.seg[s + 1].ssq_in = ssq;
      p.seg[s + 1].ssq_tiles = plan.tiles[s];
    }
  for (int s = n; s < tma::kSegmentMax; s++)
    for (int g = 0; g < tma::kGroupMax; g++) maps.map[s][g] = maps.map[0][0];
  return launch_tma_params<T>(p, maps, (int)segs[0].shapes[0].m, plan.grid, plan.stages, plan.smem, error_flag, early_rhs, pdl, stream);
}


// ---- tensor-core stream (umma_gemm.cuh) ---------------------------------------------------------------------------

int least_rows_asked_for() {
  static const int m = env_int("PJRTX_B200_UMMA_MIN_M", -1);
  return m;
}

// 0: not eligible, 1: rhs[K,N] with N contiguous, 2: rhs[N,K] with K contiguous, 3: rhs[K,N] with N contiguous whose rows
// the tensor maps cannot describe. Tensor maps need 16-byte multiples for every row stride; lhs must be k-contiguous.
// Int8 weights can start at one row (dot_s8_pays says where they do) unless the environment sets a least number.
// Case 3 (odd vocabularies) has no lower bound on m: the alternative is one thread per output (path 0) or 64 x 64 tiles on
// the CUDA cores (path 3). Measured, 5 x 2048 x 32001 f16: 739 us on path 0. Below 64 columns or a k of 64 a tile would be
// mostly padding and the other paths stay.
int umma_eligible(const DotShape& s) {
  static const int enabled = env_int("PJRTX_B200_UMMA", 1);
  const int set_min_m = least_rows_asked_for(), min_m = set_min_m < 0 ? 3 : set_min_m;
  if (!enabled || (s.dtype != kF16 && s.dtype != kBF16)) return 0;
  if (s.b0 * s.b1 != 1 || s.m < 1 || s.k < 1 || s.n < 1) return 0;
  if (s.lhs_k != 1 || (s.m > 1 && s.lhs_m % 8 != 0)) return 0;
  if (s.m > (1 << 20) || s.n > (1ll << 30) || s.k > (1ll << 30)) return 0;
  const bool pitch_ok = s.rhs_s8 ? s.rhs_k % 16 == 0 : s.rhs_k % 8 == 0;
  if (s.rhs_n == 1 && s.rhs_k >= s.n) {
    if (pitch_ok) return s.m >= min_m || (s.rhs_s8 && set_min_m < 0) ? 1 : 0;
    return s.n >= 64 && s.k >= 64 && !s.rhs_s8 ? 3 : 0;
  }
  if (s.rhs_s8 || s.m < min_m) return 0;
  if (s.rhs_k == 1 && s.rhs_n % 8 == 0 && s.rhs_n >= s.k) return 2;
  return 0;
}

int umma_source(const DotShape& s, bool loose) {
  return s.rhs_s8 ? umma::kBytes : loose ? umma::kLoose : umma::kTile;
}

// Clusters of `size` CTAs, `per_sm` CTAs on an SM, that fit the chip at once. A cluster stays inside a GPC, so SMs are left
// over; the table is what cudaOccupancyMaxActiveClusters answers for one CTA per SM on a B200 (148 SMs).
int64_t clusters_that_fit(int sm_count, int size, int per_sm) {
  static const int on_b200[umma::kSplitMax + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  return std::max<int64_t>(1, (int64_t)on_b200[size] * per_sm * sm_count / 148);
}

// Whether the receive buffers of the cluster's sum and a ring worth running fit a CTA's shared memory: all of it, where two
// stages have to fit (tall int8 tiles split over three CTAs and more leave less than that: 128 rows over three 135 KiB of
// receive buffers beside stages of 48 KiB), or half of it where the tensor memory of two CTAs fits, with four stages.
bool umma_fits(int m_tile, int ksplit, bool several_tiles, int src, bool half) {
  const int sub = src == umma::kTile ? 1 : 2, rows = (m_tile + 4 * ksplit - 1) / (4 * ksplit) * 4;
  if (half && (src == umma::kLoose || umma::tmem_columns(m_tile, sub, src) > 256)) return false;
  return umma::sum_bytes(ksplit, rows, several_tiles ? 2 : 1) + (half ? 4 : 2) * umma::stage_bytes(m_tile, sub, src) + umma::kBarrierBytes + 1024 <=
         (half ? umma::kSharedSmem : 227 * 1024);
}

// Tile height, split of k, CTAs per SM and ring size with the least modelled time, in nanoseconds. The constants and the
// points below were taken while a single thread issued copies and products; converged issue took 1.5 to 3 us off a decode launch and
// more off int8 (umma_gemm.cuh), and they were kept for the choices they make: refitted to single launches of int8 they put one CTA
// on an SM at small widths (14336 x 4096 alone 26.6 -> 22.6 us), and a whole step of 32 layers went from 4522 to 5530 us; refitted
// above 64 rows (regret 2.6 -> 1.2 % over 1600 launches) they left pairs out at 708 x 512..1792, which that sweep did not cover.
// The weights arrive at the
// HBM rate or at the rate of the CTAs, 16 KiB per 250 ns with the whole ring, per 305 ns with half of it and per 400 ns where
// two CTAs of the launch share an SM (32 x 14336 x 4096 by 32 CTAs: 64 us with the whole ring, 79 with half, the same for 16
// to 128 rows); near the crossing the two add up softly. Tall tiles are bound by shared memory, the copies in and the tensor
// core's reads out at about 88 bytes per cycle. One CTA per SM with half of the shared memory lets the next launch's CTA move
// in, set up and request its first weights meanwhile, which is worth 1 to 1.5 us against two CTAs and the whole ring. The
// cluster's sum costs about 0.6 us and the exchange of its rows. Int8 weights run two CTAs per SM wherever they fit: a unit
// is a chain of copy, conversion and MMA that one CTA cannot keep full.
// Measured, us per launch in a chain at 32 rows, best against the others: 4096 x 4096 4 CTAs per tile, half ring 15.4 (whole
// 17.6; two per SM 16.5; 1 CTA per tile 24); 14336 x 4096 4, whole 28.6 (half 30.8); 4096 x 28672 1, two per SM 44.4 (whole
// 49.3, half 53.5); 8192 x 57344 1, two per SM 150 (3 CTAs per tile 153); 28672 x 8192 4, two per SM 75.8 (2, whole 77).
struct UmmaChoice {
  double ns = 0;
  int m_tile = 0, ksplit = 1, per_sm = 1;
  bool half = false;
};
UmmaChoice umma_choose(const DotShape* shapes, int count, int sm_count, int src) {
  const DotShape& s = shapes[0];
  const double weight_unit = umma::weight_stage_bytes(src == umma::kLoose ? umma::kTile : src, 1);
  const int64_t kblocks = (s.k + 127) / 128 * 2;
  UmmaChoice best;
  int64_t n_tiles = 0;
  for (int g = 0; g < count; g++) n_tiles += (shapes[g].n + 127) / 128;
  static const int64_t caps[] = {256, 192, 128, 96, 64};
  for (int64_t cap : caps) {
    if (src != umma::kTile && cap > 128) continue;
    const int64_t m_tiles = (s.m + cap - 1) / cap;
    const int64_t mt = ((s.m + m_tiles - 1) / m_tiles + 15) / 16 * 16;
    const int64_t tiles = n_tiles * m_tiles;
    for (int split = 1; split <= umma::kSplitMax; split++) {
      if (split > 1 && (mt > 128 || split > kblocks / 2)) break;
      bool shared = false;  // two CTAs per SM are possible
      for (int mode = 2; mode >= 0; mode--) {  // 2: two CTAs per SM, 1: half of the shared memory, 0: all of it
        const int per_sm = mode == 2 ? 2 : 1;
        const int64_t clusters = std::min<int64_t>(tiles, clusters_that_fit(sm_count, split, per_sm));
        if (!umma_fits((int)mt, split, tiles > clusters, src, mode > 0)) continue;
        if (mode == 2) shared = true;
        else if (shared && src == umma::kBytes) continue;
        const double smem_ns = 2.9 * ((src == umma::kTile ? 16384 : weight_unit) + mt * 128) / 128 / 1.85;
        const double unit_ns = std::max(smem_ns, src != umma::kTile ? 305.0 : mode == 0 ? 250.0 : mode == 1 ? 305.0 : 400.0);
        const double cta_ns = (double)((tiles + clusters - 1) / clusters) * (double)((kblocks + split - 1) / split) * unit_ns;
        const double hbm_ns = (double)n_tiles * kblocks * weight_unit / 6500.0;
        const double ns = std::pow(std::pow(cta_ns, 4) + std::pow(hbm_ns, 4), 0.25) + (mode == 0 ? 1500 : mode == 2 ? 1000 : 0) +
                          (split > 1 ? 600 + 8.0 * mt : 0);
        if (best.ns == 0 || ns < best.ns * 0.99) best = UmmaChoice{ns, (int)mt, split, per_sm, mode > 0};
      }
    }
  }
  return best;
}

// The same model for CTA pairs (umma_pair.cuh), whose units took 300 ns and half a nanosecond per row by a single thread (now
// 195 and 0.57, see above). Measured then, us, one SM per tile and pairs: 128 x 4096 x 4096 20 / 31, 128 x 4096 x 28672 87 / 59,
// 256 x 14336 x 4096 52 / 81, 256 x 4096 x 28672 84 / 68, 517 x 4096 x 4096 40 / 34 (now 31).
double umma_pair_choose(const DotShape* shapes, int count, int sm_count, int* m_tile) {
  const DotShape& s = shapes[0];
  const int64_t kblocks = (s.k + 63) / 64;
  int64_t n_tiles = 0;
  for (int g = 0; g < count; g++) n_tiles += (shapes[g].n + umma::kPairN - 1) / umma::kPairN;
  double best = 0;
  for (int64_t cap = 256; cap >= 64; cap -= 32) {
    const int64_t m_tiles = (s.m + cap - 1) / cap;
    const int64_t mt = ((s.m + m_tiles - 1) / m_tiles + 31) / 32 * 32;
    const int64_t pairs = std::min<int64_t>(n_tiles * m_tiles, sm_count / 2);
    const double unit_ns = 300 + 0.5 * mt;
    const double cta_ns = (double)((n_tiles * m_tiles + pairs - 1) / pairs) * kblocks * unit_ns;
    const double t = std::max(cta_ns, (double)n_tiles * umma::kPairN * s.k * 2 / 6500.0);
    if (best == 0 || t < best * 0.98) {
      best = t;
      *m_tile = (int)mt;
    }
  }
  return best;
}

// Rows without a 16-byte pitch by residue (umma_shift.cuh) or through converters (kLoose). By residue costs a launch and a
// longer epilogue, 4 us, and does not split k, but streams three times as fast. Measured at 16 rows, us, residues and
// converters: 2048 x 1001 18.7 / 14.3, x 2001 18.7 / 17.6, x 3001 18.7 / 20.1, x 4001 18.8 / 20.4, x 8001 19 / 29; 8192 x 2001
// 43 / 35, x 4001 43 / 48, x 8001 45 / 87; 256 x 16001 16.3 / 14.3. Up to 26 tiles of 128 columns the converters' clusters of five
// are one wave: 16384 x 3201 74.0 / 71.8, x 3401 73.8 / 85.2, 65536 x 3001 262 / 242, x 3401 263 / 298. Beyond 16 rows the 64 rows
// that a short k's residues are padded to weigh more: 17 rows 64 x 93801 28.8 / 24.8, 96 x 200001 47.2 / 45.1, 128 x 46901 20.6 / 20.3,
// 32 rows 64 x 93801 30.8 / 28.5, 128 x 46901 20.6 / 22.3 (16 rows 64 x 93801 18.6 / 22.4).
bool shift_pays(const DotShape& s) {
  return s.m <= 32 && s.n > (s.k <= 2048 ? 3000 : 26 * umma::kTileN) && s.n * s.k >= 6000000 && (s.m <= 16 || s.k >= 128);
}

DotScratch shift_plan(const DotShape& s, int sm_count) {
  DotScratch p;
  p.path = 5;
  p.umma = 1;
  p.shift = 8;
  while (p.shift > 2 && (p.shift / 2) * s.rhs_k % 8 == 0) p.shift /= 2;
  p.m_tile = s.m <= 16 ? 16 : 32;
  p.tmem = (int)umma::shift_tmem_columns(p.m_tile, p.shift);
  p.ordered = 1;  // like the converters' launches
  const int per_sm = p.m_tile == 16 ? 2 : 1;
  p.grid = (int)std::min<int64_t>((s.n + umma::kShiftOut - 1) / umma::kShiftOut, (int64_t)per_sm * sm_count);
  const size_t budget = (per_sm == 2 ? umma::kSharedSmem : 227 * 1024) - 1024 - umma::kBarrierBytes - umma::shift_exchange_bytes(p.m_tile);
  p.stages = (int)std::min<size_t>(12, budget / umma::shift_stage_bytes(p.m_tile));
  p.smem = umma::shift_smem_bytes(p.stages, p.m_tile, p.shift);
  const int64_t depth = ((s.k + p.shift - 1) / p.shift + 63) / 64 * 64;
  p.partial_bytes = (uint64_t)(s.m * p.shift * depth) * 2;
  return p;
}

DotScratch umma_plan(const DotShape* shapes, int count, int sm_count, int kind) {
  DotScratch p;
  const DotShape& s = shapes[0];
  if (kind == 3 && count == 1 && shift_pays(s)) return shift_plan(s, sm_count);
  const int src = umma_source(s, kind == 3);
  p.path = kind == 1 ? 1 : kind == 2 ? 4 : 5;
  p.umma = 1;
  const UmmaChoice choice = umma_choose(shapes, count, sm_count, src);
  p.m_tile = choice.m_tile;
  p.ksplit = choice.ksplit;
  int pair_tile = 0;
  if (src == umma::kTile && s.m > 64 && umma_pair_choose(shapes, count, sm_count, &pair_tile) < choice.ns) {
    int64_t tiles = 0;
    for (int g = 0; g < count; g++) tiles += (shapes[g].n + umma::kPairN - 1) / umma::kPairN * ((s.m + pair_tile - 1) / pair_tile);
    p.pair = 1;
    p.m_tile = pair_tile;
    p.ksplit = 1;
    p.grid = 2 * (int)std::min<int64_t>(tiles, sm_count / 2);
    p.stages = (int)std::min<size_t>(12, (227 * 1024 - 1024 - umma::kBarrierBytes) / umma::pair_stage_bytes(pair_tile));
    p.smem = umma::pair_smem_bytes(p.stages, pair_tile);
    p.tmem = (int)umma::tmem_columns(pair_tile, 1, umma::kTile);
    p.ordered = 1;
    return p;
  }
  const int64_t m_tiles = (s.m + p.m_tile - 1) / p.m_tile;
  int64_t tiles = 0;
  for (int g = 0; g < count; g++) tiles += (shapes[g].n + umma::kTileN - 1) / umma::kTileN * m_tiles;
  const int64_t clusters = std::min<int64_t>(tiles, clusters_that_fit(sm_count, p.ksplit, choice.per_sm));
  p.grid = (int)(clusters * p.ksplit);
  const int rows_per_rank = (p.m_tile + 4 * p.ksplit - 1) / (4 * p.ksplit) * 4;
  const size_t sum = umma::sum_bytes(p.ksplit, rows_per_rank, tiles > clusters ? 2 : 1);
  const size_t ring_budget = (choice.half ? umma::kSharedSmem : 227 * 1024) - 1024 - umma::kBarrierBytes - sum;
  // 128-deep stages once every CTA gets a long run of them (fewer hand-overs); 64-deep otherwise, and whenever the ring
  // would hold fewer than four of the deep ones. Converted weights always come 128 deep: 64-deep stages double the
  // hand-overs between copies, converters and the MMA warp (int8, 8B-width layers at 32 rows: 1.54 against 1.25 ms).
  const int64_t deep_units = (tiles + clusters - 1) / clusters * ((s.k + 127) / 128) / p.ksplit;
  p.sub = src != umma::kTile || (deep_units >= 16 && ring_budget / umma::stage_bytes(p.m_tile, 2, src) >= 4) ? 2 : 1;
  p.stages = (int)std::min<size_t>(12, ring_budget / umma::stage_bytes(p.m_tile, p.sub, src));  // two or more (umma_fits)
  p.smem = umma::smem_bytes(p.stages, p.m_tile, p.sub, src, sum);
  p.tmem = (int)umma::tmem_columns(p.m_tile, p.sub, src);
  // Launches that take more than half of an SM's tensor memory start after their predecessor has completed, like pairs and
  // the prefill attention: one prefill that had such kernels start beside leaving ones did not finish, and what stopped it
  // was not observed. Unaligned rows took part in it and are ordered at any size.
  p.ordered = p.tmem > 256 || src == umma::kLoose ? 1 : 0;
  return p;
}

template <int SUB, int SRC>
int launch_umma_sub(const umma::Params& prm, const umma::Maps& maps, const DotScratch& plan, bool pdl, cudaStream_t stream) {
  if (!raise_smem_limit((const void*)umma::umma_stream_kernel<SUB, SRC>, 227 * 1024)) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)plan.grid);
  cfg.blockDim = dim3(umma::threads_of(SRC));
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  cfg.attrs = attr;
  cfg.numAttrs = fill_launch_attributes(attr, pdl && !plan.ordered);
  if (plan.ksplit > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)plan.ksplit;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs].val.clusterDim.z = 1;
    cfg.numAttrs++;
  }
  return cudaLaunchKernelEx(&cfg, umma::umma_stream_kernel<SUB, SRC>, prm, maps) == cudaSuccess ? 1 : 0;
}

int launch_umma_pair(const umma::PairParams& prm, const umma::Maps& maps, const DotScratch& plan, cudaStream_t stream) {
  if (!raise_smem_limit((const void*)umma::umma_pair_kernel, 227 * 1024)) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)plan.grid);
  cfg.blockDim = dim3(umma::kBaseThreads);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[3];
  cfg.attrs = attr;
  cfg.numAttrs = fill_launch_attributes(attr, false);  // (plan.ordered)
  attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
  attr[cfg.numAttrs].val.clusterDim.x = 2;
  attr[cfg.numAttrs].val.clusterDim.y = 1;
  attr[cfg.numAttrs].val.clusterDim.z = 1;
  cfg.numAttrs++;
  return cudaLaunchKernelEx(&cfg, umma::umma_pair_kernel, prm, maps) == cudaSuccess ? 1 : 0;
}

int launch_umma_shift(const DotShape& s, const DotScratch& plan, const void* lhs, const void* rhs, void* out, void* rearranged,
                      int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream) {
  EncodeTiledFn enc = encode_tiled();
  // The residues' maps start at most 14 bytes before their first row: on a 16-byte boundary if the weights do.
  if (!enc || !rearranged || (reinterpret_cast<uintptr_t>(rhs) & 15) != 0) return 0;
  const int residues = plan.shift;
  const int64_t depth = ((s.k + residues - 1) / residues + 63) / 64 * 64;
  umma::ShiftParams p{};
  umma::ShiftMaps maps{};
  p.m = (int)s.m;
  p.residues = residues;
  p.kblocks = (int)(depth / 64);
  p.tiles = (int)((s.n + umma::kShiftOut - 1) / umma::kShiftOut);
  p.n = s.n;
  p.ldo = s.out_m;
  p.out = out;
  p.stages = plan.stages;
  p.is_bf16 = s.dtype == kBF16;
  p.early_rhs = early_rhs ? 1 : 0;
  p.error_flag = error_flag;
  p.timeout_ns = wait_timeout_ns();
  const CUtensorMapDataType dt = p.is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const cuuint32_t estr[2] = {1, 1};
  auto encode = [&](CUtensorMap* map, const void* base, cuuint64_t inner, cuuint64_t rows, cuuint64_t pitch, cuuint32_t box_rows) {
    const cuuint64_t gdim[2] = {inner, rows}, gstride[1] = {pitch * 2};
    const cuuint32_t box[2] = {64, box_rows};
    return enc(map, dt, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  for (int j = 0; j < residues; j++) {
    p.delta[j] = (int)(j * s.rhs_k % 8);
    // From the 16-byte boundary at or before the residue's first row (for j > 0 inside the row before it) to its last column.
    const unsigned short* base = static_cast<const unsigned short*>(rhs) + j * s.rhs_k - p.delta[j];
    if (!encode(&maps.rhs[j], base, (cuuint64_t)(s.n + p.delta[j]), (cuuint64_t)((s.k - j + residues - 1) / residues),
                (cuuint64_t)(residues * s.rhs_k), 64))
      return 0;
  }
  const cuuint64_t width = (cuuint64_t)(residues * depth);
  if (!encode(&maps.lhs, rearranged, width, (cuuint64_t)s.m, width, (cuuint32_t)plan.m_tile)) return 0;
  const unsigned blocks = (unsigned)std::min<int64_t>((s.m * (int64_t)width + 255) / 256, 1024);
  if (launch_kernel(umma::residue_rows_kernel, dim3(blocks), dim3(256), 0, stream, pdl, static_cast<const unsigned short*>(lhs), (long long)s.lhs_m,
                    p.m, (int)s.k, residues, (int)depth, static_cast<unsigned short*>(rearranged)) != cudaSuccess)
    return 0;
  auto launch = [&](auto* kernel) {
    return raise_smem_limit((const void*)kernel, 227 * 1024) &&
           launch_kernel(kernel, dim3((unsigned)plan.grid), dim3(umma::kBaseThreads), plan.smem, stream, pdl && !plan.ordered, p, maps) == cudaSuccess;
  };
  return (plan.m_tile == 16 ? launch(umma::umma_shift_kernel<16>) : launch(umma::umma_shift_kernel<32>)) ? 2 : 0;
}

int launch_umma(const DotShape* shapes, int count, const DotScratch& plan, const void* lhs, const void* const* rhs, void* const* out,
                int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream, const void* const* scales) {
  const DotShape& s = shapes[0];
  const bool w8 = s.rhs_s8 != 0, loose = plan.path == 5;
  if (w8 && (!scales || plan.path == 4)) return 0;
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return 0;
  const bool k_major = plan.path == 4;
  const int tw = umma::kTileN;
  umma::Params p{};
  umma::Maps maps{};
  p.m = (int)s.m;
  p.k = (int)s.k;
  p.m_tile = plan.m_tile;
  p.m_tiles = (int)((s.m + plan.m_tile - 1) / plan.m_tile);
  p.count = count;
  const CUtensorMapDataType dt = s.dtype == kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const cuuint32_t estr[2] = {1, 1};
  // One 3-d copy per stage when every rhs is made of whole 64-column blocks (a ragged last block would make the
  // view read past the end of the last row).
  bool use_3d = !k_major && !w8 && !loose;
  for (int g = 0; g < count; g++) use_3d &= shapes[g].n % 64 == 0;
  int tiles = 0;
  for (int g = 0; g < count; g++) {
    if (!loose && (reinterpret_cast<uintptr_t>(rhs[g]) & 15) != 0) return 0;
    p.rhs[g] = rhs[g];
    p.rhs_pitch[g] = shapes[g].rhs_k;
    p.tile_begin[g] = tiles;
    tiles += (int)((shapes[g].n + tw - 1) / tw) * p.m_tiles;
    p.out[g] = out[g];
    p.n[g] = shapes[g].n;
    p.ldo[g] = shapes[g].out_m;
    p.scale[g] = w8 ? scales[g] : nullptr;
  }
  auto encode_rhs = [&](bool three_d) {
    for (int g = 0; g < count; g++) {
      cuuint64_t gdim[3], gstride[2];
      cuuint32_t box[3];
      const cuuint32_t estr3[3] = {1, 1, 1};
      int rank = 2;
      if (w8) {
        // raw bytes: one box of 128 columns x 64 * SUB rows per stage, swizzled so that the converters' reads of four
        // columns x one row per thread spread over all banks
        gdim[0] = (cuuint64_t)shapes[g].n; gdim[1] = (cuuint64_t)s.k;
        gstride[0] = (cuuint64_t)shapes[g].rhs_k;
        box[0] = 128; box[1] = (cuuint32_t)(64 * plan.sub);
        // A row of the box is 128 bytes: with 256-byte promotion L2 would fetch the neighbouring tile's 128 bytes with
        // every row and usually lose them again before that tile's turn (measured on the 4096 x 128256 LM head:
        // 742 MB read for 525 MB of weights).
        if (enc(&maps.rhs[g], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(rhs[g]), gdim, gstride, box, estr3,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
          return false;
        continue;
      }
      if (three_d) {
        rank = 3;
        gdim[0] = 64; gdim[1] = (cuuint64_t)s.k; gdim[2] = (cuuint64_t)shapes[g].n / 64;
        gstride[0] = (cuuint64_t)shapes[g].rhs_k * 2; gstride[1] = 128;
        box[0] = 64; box[1] = (cuuint32_t)(64 * plan.sub); box[2] = 2;
      } else if (k_major) {
        gdim[0] = (cuuint64_t)s.k; gdim[1] = (cuuint64_t)shapes[g].n;
        gstride[0] = (cuuint64_t)shapes[g].rhs_n * 2;
        box[0] = 64; box[1] = 128;
      } else {
        gdim[0] = (cuuint64_t)shapes[g].n; gdim[1] = (cuuint64_t)s.k;
        gstride[0] = (cuuint64_t)shapes[g].rhs_k * 2;
        box[0] = 64; box[1] = (cuuint32_t)(64 * plan.sub);
      }
      if (enc(&maps.rhs[g], dt, rank, const_cast<void*>(rhs[g]), gdim, gstride, box, estr3, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    }
    return true;
  };
  if (use_3d && !encode_rhs(true)) use_3d = false;  // the driver refused the view: fall back to two boxes per half
  if (!use_3d && !loose && !encode_rhs(false)) return 0;
  p.rhs_3d = use_3d ? 1 : 0;
  for (int g = count; g <= umma::kGroupMax; g++) p.tile_begin[g] = tiles;
  for (int g = count; g < umma::kGroupMax; g++) maps.rhs[g] = maps.rhs[0];
  {
    if ((reinterpret_cast<uintptr_t>(lhs) & 15) != 0) return 0;
    cuuint64_t gdim[2] = {(cuuint64_t)s.k, (cuuint64_t)s.m};
    // A single row has no stride to honour; any 16-byte multiple that covers the row will do.
    cuuint64_t gstride[1] = {(cuuint64_t)(s.m > 1 ? s.lhs_m : (s.k + 7) / 8 * 8) * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)(plan.pair ? plan.m_tile / 2 : plan.m_tile)};
    if (enc(&maps.lhs, dt, 2, const_cast<void*>(lhs), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return 0;
  }
  p.kblocks = (int)((s.k + 64 * plan.sub - 1) / (64 * plan.sub));
  if (plan.pair) {
    umma::PairParams q{};
    q.m = p.m;
    q.m_tile = p.m_tile;
    q.m_tiles = p.m_tiles;
    q.count = count;
    for (int g = 0; g < count; g++) {
      q.n_tile_begin[g] = q.n_tiles;
      q.n_tiles += (int)((shapes[g].n + umma::kPairN - 1) / umma::kPairN);
      q.out[g] = p.out[g];
      q.n[g] = p.n[g];
      q.ldo[g] = p.ldo[g];
    }
    for (int g = count; g <= umma::kGroupMax; g++) q.n_tile_begin[g] = q.n_tiles;
    q.kblocks = p.kblocks;
    q.stages = plan.stages;
    q.is_bf16 = s.dtype == kBF16;
    q.rhs_k_major = k_major ? 1 : 0;
    q.rhs_3d = p.rhs_3d;
    q.error_flag = error_flag;
    q.timeout_ns = wait_timeout_ns();
    return launch_umma_pair(q, maps, plan, stream);
  }
  p.tiles = tiles;
  p.ksplit = plan.ksplit;
  p.rows_per_rank = (plan.m_tile + 4 * plan.ksplit - 1) / (4 * plan.ksplit) * 4;
  p.sum_buffers = tiles > plan.grid / plan.ksplit ? 2 : 1;
  p.error_flag = error_flag;
  p.timeout_ns = wait_timeout_ns();
  p.stages = plan.stages;
  p.is_bf16 = s.dtype == kBF16;
  p.rhs_k_major = k_major ? 1 : 0;
  p.early_rhs = early_rhs ? 1 : 0;
  switch (umma_source(s, loose)) {
    case umma::kBytes: return launch_umma_sub<2, umma::kBytes>(p, maps, plan, pdl, stream);
    case umma::kLoose: return launch_umma_sub<2, umma::kLoose>(p, maps, plan, pdl, stream);
    default:
      return plan.sub == 2 ? launch_umma_sub<2, umma::kTile>(p, maps, plan, pdl, stream) : launch_umma_sub<1, umma::kTile>(p, maps, plan, pdl, stream);
  }
}

}  // namespace

bool dot_chain_eligible(const DotShape& s, int sm_count) {
  if (s.b0 * s.b1 != 1) return false;
  const DotScratch p = dot_plan(s, sm_count);
  return p.path == 1 && p.tma == 1 && p.umma == 0;
}

DotChainPlan dot_chain_plan(const DotChainSegment* segs, int n, int sm_count) {
  DotChainPlan p;
  if (n < 1 || n > kDotChainMax) return p;
  const DotShape& first = segs[0].shapes[0];
  const int esize = (int)dtype_size(first.dtype);
  const int V = 16 / esize;
  const int M = first.m <= 1 ? 1 : first.m <= 2 ? 2 : first.m <= 4 ? 4 : 8;
  int per_sm = 1;
  tma_ring(M, V, &p.stages, &per_sm);
  const bool two_per_sm = per_sm == 2;
  p.smem = tma::smem_bytes(p.stages, M, 32 * V);
  // Every CTA takes part in the barriers between segments, so the grid must be wholly resident, and every CTA must own
  // at least one unit of every segment (the tile bookkeeping assumes consecutive, non-empty shares).
  int64_t grid = (int64_t)sm_count * (two_per_sm ? 2 : 1);
  int64_t tiles_all[kDotChainMax], chunks_all[kDotChainMax];
  for (int s = 0; s < n; s++) {
    int64_t tiles = 0;
    for (int g = 0; g < segs[s].count; g++) tiles += (segs[s].shapes[g].n + 32 * V - 1) / (32 * V);
    const int64_t chunks = (segs[s].shapes[0].k + tma::kUnitRows - 1) / tma::kUnitRows;
    tiles_all[s] = tiles;
    chunks_all[s] = chunks;
    grid = std::min(grid, std::max<int64_t>(1, tiles * chunks));
  }
  p.grid = (int)grid;
  p.segments = n;
  uint64_t counters = (uint64_t)2 * kDotChainMax * sizeof(unsigned);  // barrier words
  counters = (counters + 255) / 256 * 256;
  for (int s = 0; s < n; s++) {
    const int64_t per_cta = std::max<int64_t>(1, tiles_all[s] * chunks_all[s] / grid);
    p.max_contrib[s] = (int)std::min<int64_t>(chunks_all[s], (chunks_all[s] + per_cta - 1) / per_cta + 1);
    p.counter_offset[s] = counters;
    p.tiles[s] = (int)tiles_all[s];
    counters += ((uint64_t)tiles_all[s] * sizeof(unsigned) + 255) / 256 * 256;
    if (s + 1 < n && segs[s + 1].norm_of_previous && segs[s + 1].lhs.kind == kDotLhsRmsNorm && segs[s].count == 1) {
      p.ssq_offset[s] = counters;
      counters += ((uint64_t)tiles_all[s] * M * sizeof(float) + 255) / 256 * 256;
    }
    p.partial_bytes = std::max<uint64_t>(p.partial_bytes, (uint64_t)tiles_all[s] * p.max_contrib[s] * M * 32 * V * sizeof(float));
  }
  p.counter_bytes = counters;
  return p;
}

int dot_chain_launch(const DotChainSegment* segs, const DotChainArgs* args, int n, const DotChainPlan& plan, void* partials,
                     void* counters, int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream) {
  if (n < 1 || n > kDotChainMax || plan.segments != n) return 0;
  switch (segs[0].shapes[0].dtype) {
    case kF32: return launch_chain<float>(segs, args, n, plan, partials, counters, error_flag, early_rhs, pdl, stream);
    case kF16: return launch_chain<__half>(segs, args, n, plan, partials, counters, error_flag, early_rhs, pdl, stream);
    case kBF16: return launch_chain<__nv_bfloat16>(segs, args, n, plan, partials, counters, error_flag, early_rhs, pdl, stream);
    default: return 0;
  }
}

namespace {
// One CTA waits, with the streaming kernel's own bounded wait, on an mbarrier that nothing ever completes.
__global__ void bounded_wait_probe_kernel(unsigned long long timeout_ns, int* error_flag) {
  __shared__ uint64_t bar;
  __shared__ int abort_word;
  if (threadIdx.x == 0) {
    abort_word = 0;
    tma::mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const tma::WaitBudget budget{tma::global_timer_ns() + timeout_ns, &abort_word};
  if (!tma::mbar_wait(&bar, 0, budget) && threadIdx.x == 0) atomicExch(error_flag, 31);
}
}  // namespace

int bounded_wait_probe_launch(unsigned timeout_ms, int* error_flag, cudaStream_t stream) {
  if (!error_flag || timeout_ms < 1 || timeout_ms > 1000) return 0;
  bounded_wait_probe_kernel<<<1, 64, 0, stream>>>((unsigned long long)timeout_ms * 1000000ull, error_flag);
  return cudaGetLastError() == cudaSuccess ? 1 : 0;
}

bool dot_s8_supported(const DotShape& s) {
  DotShape probe = s;
  probe.rhs_s8 = 1;
  return umma_eligible(probe) == 1;
}

// Under one or two rows the alternative writes the scaled weights out and reads them again, five bytes per weight, while the
// bytes' own way is a chain per 128 rows of k that at most eight CTAs share. Measured, us, written form and bytes, one row / two
// rows: 1024 x 1024 10.9 10.2 / 11.1 10.3, 4096 x 4096 22.6 16.1 / 24.7 16.2, 14336 x 4096 56 25 and 4096 x 32000 122 33 at one; k
// long against n: 4096 x 256 10.8 10.3 / 12.4 10.3, 16384 x 256 18.5 16.4 / 26.7 16.5, 32768 x 512 25.2 22.6 / 32.5 22.6, 24576 x 384
// 18.5 18.8 / 25.1 18.9, 65536 x 256 28.8 34.9 / 39.2 34.9, 8192 x 192 12.0 12.5 / 16.3 12.4, 8192 x 128 11.7 12.4 / 16.3 12.4, 32768 x
// 32 16.5 22.5 / 25.9 22.6, 65536 x 16 18.4 34.2 / 28.6 34.2; k short: 128 x 8192 9.4 8.7 / 9.6 8.6, 96 x 65536 16.5 12.4 / 18.5 12.4,
// 64 x 65536 11.1 12.4 / 12.1 12.4, 16 x 65536 11.0 12.4 / 10.8 12.4. Below a million weights neither side was measured against
// the other and the written rounding stays.
bool dot_s8_pays(const DotShape& s, bool shared) {
  if (s.m > 2 || least_rows_asked_for() >= 0) return true;  // (dot_s8_supported has looked at what was asked for)
  if (s.k * s.n < (1 << 20)) return false;
  return shared || (s.k >= 96 && (s.m == 1 ? s.n >= 256 && s.k <= 64 * s.n : s.k <= 1024 * s.n));
}

int dot_group_launch(const DotShape* shapes, int count, const DotScratch& plan, const void* lhs, const void* const* rhs,
                     void* const* out, void* partials, void* counters, int* error_flag, bool early_rhs, bool pdl,
                     cudaStream_t stream, const void* const* scales) {
  if (count < 1 || count > kDotGroupMax) return 0;
  if (plan.shift) return launch_umma_shift(shapes[0], plan, lhs, rhs[0], out[0], partials, error_flag, early_rhs, pdl, stream);
  if (plan.umma) return launch_umma(shapes, count, plan, lhs, rhs, out, error_flag, early_rhs, pdl, stream, scales);
  if (shapes[0].rhs_s8) return 0;  // int8 weights run on the tensor-core stream only
  if (plan.small) {
    switch (shapes[0].dtype) {
      case kF32: return launch_small<float>(shapes, count, lhs, rhs, out, early_rhs, pdl, stream);
      case kF16: return launch_small<__half>(shapes, count, lhs, rhs, out, early_rhs, pdl, stream);
      case kBF16: return launch_small<__nv_bfloat16>(shapes, count, lhs, rhs, out, early_rhs, pdl, stream);
      default: return 0;
    }
  }
  if (plan.tma) {
    switch (shapes[0].dtype) {
      case kF32: return launch_tma<float>(shapes, count, plan, lhs, rhs, out, partials, counters, error_flag, early_rhs, pdl, stream);
      case kF16: return launch_tma<__half>(shapes, count, plan, lhs, rhs, out, partials, counters, error_flag, early_rhs, pdl, stream);
      case kBF16: return launch_tma<__nv_bfloat16>(shapes, count, plan, lhs, rhs, out, partials, counters, error_flag, early_rhs, pdl, stream);
      default: return 0;
    }
  }
  switch (shapes[0].dtype) {
    case kF32: return launch_group_typed<float>(shapes, count, plan, lhs, rhs, out, partials, counters, pdl, stream);
    case kF16: return launch_group_typed<__half>(shapes, count, plan, lhs, rhs, out, partials, counters, pdl, stream);
    case kBF16: return launch_group_typed<__nv_bfloat16>(shapes, count, plan, lhs, rhs, out, partials, counters, pdl, stream);
    default: return 0;
  }
}

DotScratch dot_plan(const DotShape& s, int sm_count) {
  DotScratch p;
  const int esize = (int)dtype_size(s.dtype);
  if (esize == 0 || !dtype_is_float(s.dtype)) return p;
  const int V = 16 / esize;
  const int64_t batch = s.b0 * s.b1;
  auto aligned = [&](int64_t stride) { return stride % V == 0; };
  const bool batches_fit = batch <= 65535;
  const int tensor = umma_eligible(s);
  if (tensor) return umma_plan(&s, 1, sm_count, tensor);
  if (s.m <= 8 && s.rhs_n == 1 && s.n % V == 0 && aligned(s.rhs_k) && aligned(s.rhs_b0) && aligned(s.rhs_b1) &&
      batches_fit && s.k >= 1) {
    p.path = 1;
    const DotShape one = s;
    return dot_group_plan(&one, 1, sm_count);
  }
  if (s.m <= 8 && s.rhs_k == 1 && s.lhs_k == 1 && s.k % V == 0 && aligned(s.rhs_n) && aligned(s.rhs_b0) &&
      aligned(s.rhs_b1) && aligned(s.lhs_m) && aligned(s.lhs_b0) && aligned(s.lhs_b1) && batches_fit) {
    p.path = 2;
    return p;
  }
  const bool split = s.k >= 1 && s.n >= 1 && split_tile_ok(s) && split_tiles_pay(s, batch, sm_count);
  const bool few = split && s.n >= 64;  // few rows of pitches the streaming kernels cannot take
  if ((s.m > 8 || few) && batches_fit && (s.m + kTile - 1) / kTile <= 65535) {
    p.path = 3;
    p.wide = wide_tiles_pay(s, batch, sm_count) ? 1 : 0;
    p.ksplit = split ? split_tile_parts(s, batch, sm_count) : 0;
    return p;
  }
  p.path = 0;
  return p;
}

int dot_launch(const DotShape& s, const DotScratch& plan, const void* lhs, const void* rhs, void* out, void* partials,
               void* counters, int* error_flag, bool early_rhs, bool pdl, cudaStream_t stream, const void* scale) {
  if (s.b0 * s.b1 * s.m * s.n == 0) return 1;
  if (plan.umma || (plan.path == 1 && plan.tma)) {
    const void* rhs_list[1] = {rhs};
    void* out_list[1] = {out};
    const void* scale_list[1] = {scale};
    return dot_group_launch(&s, 1, plan, lhs, rhs_list, out_list, partials, counters, error_flag, early_rhs, pdl, stream, scale_list);
  }
  if (s.rhs_s8) return 0;
  switch (s.dtype) {
    case kF32: return launch_typed<float>(s, plan, lhs, rhs, out, partials, counters, pdl, stream);
    case kF16: return launch_typed<__half>(s, plan, lhs, rhs, out, partials, counters, pdl, stream);
    case kBF16: return launch_typed<__nv_bfloat16>(s, plan, lhs, rhs, out, partials, counters, pdl, stream);
    default: return 0;
  }
}

}  // namespace pjrtx
