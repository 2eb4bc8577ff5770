// dynamic_update_slice and split-KV attention kernels for sm_100a.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../common.h"
#include "kernels.h"

namespace pjrtx {

namespace {

__device__ __forceinline__ int64_t load_index(const void* p, int dtype) {
  switch (dtype) {
    case kS32: return *static_cast<const int32_t*>(p);
    case kU32: return *static_cast<const uint32_t*>(p);
    case kS64: return *static_cast<const int64_t*>(p);
    case kU64: return (int64_t)*static_cast<const uint64_t*>(p);
    case kS8: return *static_cast<const int8_t*>(p);
    case kU8: return *static_cast<const uint8_t*>(p);
    case kS16: return *static_cast<const int16_t*>(p);
    case kU16: return *static_cast<const uint16_t*>(p);
    default: return 0;
  }
}

struct DusArgs {
  int rank;
  int unit;             // bytes moved per thread step
  int64_t upd_units[8];  // update dims, innermost in units
  int64_t dst_units[8];
  int64_t dst_dims[8];   // element dims for clamping
  int64_t upd_dims[8];
  int start_dtype[8];
  const void* start[8];
  int64_t last_scale;    // units per index step along the innermost kept axis
  int64_t total_units;
};

// Start indices are clamped to [0, dst_dim - upd_dim] as StableHLO specifies
// (the reference passes them to MLX slice_update, src/backend/mlx_metal/api.cc:2552-2635).
template <typename U>
__global__ void dus_kernel(DusArgs a, U* __restrict__ dst, const U* __restrict__ upd) {
  PJRTX_PDL_PROLOGUE();
  __shared__ int64_t start[8];
  if (threadIdx.x < a.rank) {
    const int d = threadIdx.x;
    int64_t s = a.start[d] ? load_index(a.start[d], a.start_dtype[d]) : 0;
    const int64_t hi = a.dst_dims[d] - a.upd_dims[d];
    s = s < 0 ? 0 : (s > hi ? hi : s);
    start[d] = (d == a.rank - 1) ? s * a.last_scale : s;
  }
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.total_units; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t rem = i, off = 0, stride = 1;
    for (int d = a.rank - 1; d >= 0; d--) {
      const int64_t c = rem % a.upd_units[d];
      rem /= a.upd_units[d];
      off += (c + start[d]) * stride;
      stride *= a.dst_units[d];
    }
    dst[off] = upd[i];
  }
}

// ------------------------------------------------------------------ copies around a replayed graph
// A call of a captured program has its small arguments brought into their fixed slots before the graph and its results
// copied out of the arena behind it. One copy command each cost 2 to 4 us of the stream and of the host: a 32-layer int8
// decode step has 66 small arguments (the column scales of the narrow projections among them), a toy decoder nine. Whole
// calls, a command each against this: that decode step 5344 -> 5154 us, toy decoder (eight tokens) 1205 -> 1073 us, 8 layers
// 2048 wide 748 -> 691 us, a prefill of 517 positions that hands 16 caches of 1 MB out 3364 -> 3275 us.
// A block moves one piece of one entry: 256 threads x 8 loads of 16 bytes, all requested before the first is stored.
constexpr int kCopyThreads = 256, kCopyUnroll = 8;
constexpr uint64_t kCopyPiece = (uint64_t)kCopyThreads * kCopyUnroll * 16;

template <int N>
struct CopyBatch {
  CopyEntry entry[N];
  unsigned end[N];  // blocks of entries 0..i
  int count;
};
static_assert(sizeof(CopyBatch<kCopyBatchMax>) <= 4096, "kernel parameters");

template <int N>
__global__ void __launch_bounds__(kCopyThreads) copy_batch_kernel(const __grid_constant__ CopyBatch<N> b) {
  int lo = 0, hi = b.count - 1;  // the first entry whose blocks end behind this one
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x < b.end[mid]) hi = mid;
    else lo = mid + 1;
  }
  const CopyEntry& e = b.entry[lo];
  const uint64_t piece = blockIdx.x - (lo ? b.end[lo - 1] : 0u);
  const uint64_t begin = piece * kCopyPiece, end = min(e.bytes, begin + kCopyPiece);
  const unsigned char* src = static_cast<const unsigned char*>(e.src);
  unsigned char* dst = static_cast<unsigned char*>(e.dst);
  const uint4* s = reinterpret_cast<const uint4*>(src + begin);
  uint4* d = reinterpret_cast<uint4*>(dst + begin);
  const int vectors = (int)((end - begin) / 16);
  uint4 v[kCopyUnroll];
#pragma unroll
  for (int i = 0; i < kCopyUnroll; i++) {
    const int at = i * kCopyThreads + (int)threadIdx.x;
    if (at < vectors) v[i] = s[at];
  }
#pragma unroll
  for (int i = 0; i < kCopyUnroll; i++) {
    const int at = i * kCopyThreads + (int)threadIdx.x;
    if (at < vectors) d[at] = v[i];
  }
  // The last piece of an entry may end between two boundaries.
  const uint64_t at = begin + (uint64_t)vectors * 16 + threadIdx.x;
  if (at < end) dst[at] = src[at];
}

// ------------------------------------------------------------------ attention
template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

struct AttnArgs {
  int64_t batch, q_len, heads, kv_len, kv_heads, head_dim;
  int token_dtype;
  float scale;
};

// One thread per (batch, query, head): two passes over the keys, scores held
// only as running max / sum. Correctness path for any head_dim and dtype
// (the reference's generated attention kernel has the same shape:
// src/backend/mlx_metal/executable_metal_graph_custom_call.zig:126-219).
template <typename T>
__global__ void sdpa_simple_kernel(AttnArgs a, const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                                   const void* __restrict__ token, T* __restrict__ out) {
  PJRTX_PDL_PROLOGUE();
  const int64_t total = a.batch * a.q_len * a.heads;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int64_t h = t % a.heads, qi = (t / a.heads) % a.q_len, b = t / (a.heads * a.q_len);
  const int64_t g = h / (a.heads / a.kv_heads);
  int64_t limit = load_index(token, a.token_dtype) + qi;  // keys 0..limit are visible
  if (limit >= a.kv_len) limit = a.kv_len - 1;
  const T* qp = q + ((b * a.q_len + qi) * a.heads + h) * a.head_dim;
  T* op = out + ((b * a.q_len + qi) * a.heads + h) * a.head_dim;
  const T* kb = k + (b * a.kv_len * a.kv_heads + g) * a.head_dim;
  const T* vb = v + (b * a.kv_len * a.kv_heads + g) * a.head_dim;
  const int64_t row = a.kv_heads * a.head_dim;
  float m = -INFINITY;
  for (int64_t j = 0; j <= limit; j++) {
    float s = 0.f;
    for (int64_t d = 0; d < a.head_dim; d++) s = fmaf(to_f(qp[d]), to_f(kb[j * row + d]), s);
    m = fmaxf(m, s * a.scale);
  }
  float l = 0.f;
  for (int64_t j = 0; j <= limit; j++) {
    float s = 0.f;
    for (int64_t d = 0; d < a.head_dim; d++) s = fmaf(to_f(qp[d]), to_f(kb[j * row + d]), s);
    l += expf(s * a.scale - m);
  }
  for (int64_t d = 0; d < a.head_dim; d++) {
    float acc = 0.f;
    for (int64_t j = 0; j <= limit; j++) {
      float s = 0.f;
      for (int64_t e = 0; e < a.head_dim; e++) s = fmaf(to_f(qp[e]), to_f(kb[j * row + e]), s);
      acc = fmaf(expf(s * a.scale - m), to_f(vb[j * row + d]), acc);
    }
    op[d] = from_f<T>(limit < 0 ? 0.f : acc / l);
  }
}

}  // namespace

template <int N>
static bool copy_batches(const CopyEntry* entries, size_t count, cudaStream_t stream) {
  CopyBatch<N> b;
  for (size_t at = 0; at < count;) {
    b.count = 0;
    uint64_t blocks = 0;
    for (; at < count && b.count < N; at++) {
      const uint64_t pieces = (entries[at].bytes + kCopyPiece - 1) / kCopyPiece;
      if (blocks && blocks + pieces > 0x7fffffffull) break;  // a grid's limit
      if (pieces == 0) continue;
      if (((reinterpret_cast<uintptr_t>(entries[at].src) | reinterpret_cast<uintptr_t>(entries[at].dst)) & 15) != 0) return false;
      blocks += pieces;
      b.entry[b.count] = entries[at];
      b.end[b.count++] = (unsigned)blocks;
    }
    if (b.count == 0) continue;
    if (launch_kernel(copy_batch_kernel<N>, dim3((unsigned)blocks), dim3(kCopyThreads), 0, stream, false, b) != cudaSuccess) return false;
  }
  return true;
}

bool copy_batch_launch(const CopyEntry* entries, size_t count, cudaStream_t stream) {
  // The parameters travel with the launch: most calls have few copies.
  return count <= 16 ? copy_batches<16>(entries, count, stream) : copy_batches<kCopyBatchMax>(entries, count, stream);
}

int dus_launch(const SliceUpdateShape& s, void* dst, const void* update, const void* const* start_ptrs, bool pdl,
               cudaStream_t stream) {
  if (s.rank < 0 || s.rank > 8 || s.elem_size <= 0) return 0;
  int64_t upd[8] = {1}, dstd[8] = {1};
  const int rank = s.rank == 0 ? 1 : s.rank;
  int64_t total = 1;
  for (int d = 0; d < s.rank; d++) {
    upd[d] = s.upd_dims[d];
    dstd[d] = s.dst_dims[d];
    total *= upd[d];
  }
  if (total == 0) return 1;
  // Trailing axes the update covers completely have start 0; fold them into
  // the last axis that can move so each thread copies one contiguous unit.
  int t = rank - 1;
  int64_t covered = 1;
  while (t > 0 && upd[t] == dstd[t]) {
    covered *= upd[t];
    t--;
  }
  int unit = s.elem_size;
  if ((covered * s.elem_size) % 16 == 0) unit = 16;
  else if (upd[t] == dstd[t] && (upd[t] * covered * s.elem_size) % 16 == 0) unit = 16;
  DusArgs k{};
  k.rank = t + 1;
  k.unit = unit;
  for (int d = 0; d <= t; d++) {
    k.upd_dims[d] = upd[d];
    k.dst_dims[d] = dstd[d];
    k.upd_units[d] = upd[d];
    k.dst_units[d] = dstd[d];
    k.start_dtype[d] = s.rank == 0 ? 0 : s.start_dtype[d];
    k.start[d] = s.rank == 0 ? nullptr : start_ptrs[d];
  }
  k.upd_units[t] = upd[t] * covered * s.elem_size / unit;
  k.dst_units[t] = dstd[t] * covered * s.elem_size / unit;
  // Units per step of the start index along axis t (0 when that axis is fully covered).
  k.last_scale = upd[t] == dstd[t] ? 0 : covered * s.elem_size / unit;
  k.total_units = 1;
  for (int d = 0; d <= t; d++) k.total_units *= k.upd_units[d];
  const unsigned blocks = (unsigned)std::min<int64_t>((k.total_units + 255) / 256, 148 * 16);
  switch (unit) {
    case 16: launch_kernel(dus_kernel<uint4>, dim3(blocks), dim3(256), 0, stream, pdl, k, (uint4*)dst, (const uint4*)update); break;
    case 8: launch_kernel(dus_kernel<uint2>, dim3(blocks), dim3(256), 0, stream, pdl, k, (uint2*)dst, (const uint2*)update); break;
    case 4: launch_kernel(dus_kernel<uint32_t>, dim3(blocks), dim3(256), 0, stream, pdl, k, (uint32_t*)dst, (const uint32_t*)update); break;
    case 2: launch_kernel(dus_kernel<uint16_t>, dim3(blocks), dim3(256), 0, stream, pdl, k, (uint16_t*)dst, (const uint16_t*)update); break;
    case 1: launch_kernel(dus_kernel<uint8_t>, dim3(blocks), dim3(256), 0, stream, pdl, k, (uint8_t*)dst, (const uint8_t*)update); break;
    default: return 0;
  }
  return 1;
}

int sdpa_launch(const SdpaShape& s, const void* q, const void* k, const void* v, const void* token_index, void* out,
                bool pdl, cudaStream_t stream) {
  AttnArgs a{s.batch, s.q_len, s.heads, s.kv_len, s.kv_heads, s.head_dim, s.token_dtype,
             1.0f / sqrtf((float)s.head_dim)};
  const int64_t total = s.batch * s.q_len * s.heads;
  if (total == 0) return 1;
  const unsigned blocks = (unsigned)((total + 63) / 64);
  switch (s.dtype) {
    case kF32: launch_kernel(sdpa_simple_kernel<float>, dim3(blocks), dim3(64), 0, stream, pdl, a, (const float*)q, (const float*)k, (const float*)v, token_index, (float*)out); break;
    case kF16: launch_kernel(sdpa_simple_kernel<__half>, dim3(blocks), dim3(64), 0, stream, pdl, a, (const __half*)q, (const __half*)k, (const __half*)v, token_index, (__half*)out); break;
    case kBF16: launch_kernel(sdpa_simple_kernel<__nv_bfloat16>, dim3(blocks), dim3(64), 0, stream, pdl, a, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, token_index, (__nv_bfloat16*)out); break;
    default: return 0;
  }
  return 1;
}

}  // namespace pjrtx
