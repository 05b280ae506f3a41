// Small kernels of the attention module around the attention itself.
//
//  * lengths_kernel   valid lengths of a right-padded batch from its mask, and the check that the mask is one: a CTA per
//                     sequence.  As tensor operators this was nine launches of a few hundred bytes each.
//  * column_sums      bias gradients: sums over the rows of one or two bf16 matrices side by side, fp32 inside.  Bound by
//                     reading them; the row ranges of a column are summed in a fixed order by a second launch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"
#include "sm100_ptx.cuh"

namespace fdb {
namespace {

constexpr int kThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kThreads) lengths_kernel(const T* __restrict__ mask, int seqlen, int64_t batch_stride, int64_t token_stride,
                                                           T value_bits, int32_t* __restrict__ lens, int32_t* __restrict__ status) {
  __shared__ int s_count[kThreads / 32], s_last[kThreads / 32];
  const T* row = mask + blockIdx.x * batch_stride;
  int count = 0, last = 0;  // valid tokens; one past the last of them
  for (int t = threadIdx.x; t < seqlen; t += kThreads)
    if ((row[t * token_stride] & value_bits) != 0) { ++count; last = t + 1; }
  count = __reduce_add_sync(0xffffffffu, count);
  last = __reduce_max_sync(0xffffffffu, last);
  if ((threadIdx.x & 31) == 0) { s_count[threadIdx.x >> 5] = count; s_last[threadIdx.x >> 5] = last; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; ++w) { count += s_count[w]; last = max(last, s_last[w]); }
    lens[blockIdx.x] = count;
    if (last != count && status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(status), FDB_DEV_BAD_MASK);
  }
}

// 32 x 8 threads: eight columns per thread, 256 columns and a range of rows per CTA
struct SumPart { const __nv_bfloat16* x; int64_t row_stride; int rows, cols, splits; };

__global__ void __launch_bounds__(kThreads) column_partials_kernel(SumPart a, SumPart b, int cols, float* __restrict__ partial) {
  __shared__ float s[8][32][9];
  const bool first = (int)blockIdx.y < a.splits;
  const SumPart p = first ? a : b;
  const int split = first ? blockIdx.y : blockIdx.y - a.splits;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 256 + tx * 8;
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < p.cols) {
    const int r1 = (int)((int64_t)p.rows * (split + 1) / p.splits);
#pragma unroll 4
    for (int r = (int)((int64_t)p.rows * split / p.splits) + ty; r < r1; r += 8) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(p.x + r * p.row_stride + c));
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sum[2 * i] += __uint_as_float(w[i] << 16);
        sum[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s[ty][tx][i] = sum[i];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < cols) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) t += s[y][threadIdx.x >> 3][threadIdx.x & 7];
    partial[(int64_t)blockIdx.y * cols + col] = t;
  }
}

__global__ void __launch_bounds__(kThreads) column_finish_kernel(const float* __restrict__ partial, int splits, int cols, __nv_bfloat16* __restrict__ out) {
  const int c = blockIdx.x * kThreads + threadIdx.x;
  if (c >= cols) return;
  float t = 0.f;
#pragma unroll 8
  for (int s = 0; s < splits; ++s) t += partial[(int64_t)s * cols + c];
  out[c] = __float2bfloat16_rn(t);
}

int splits_of(int64_t rows) { return (int)std::max<int64_t>(1, std::min<int64_t>(64, rows / 64)); }

template <typename T>
void lengths(const void* mask, int batch, int seqlen, int64_t bs, int64_t ts, T bits, int32_t* lens, int32_t* status, cudaStream_t s) {
  lengths_kernel<T><<<batch, kThreads, 0, s>>>(static_cast<const T*>(mask), seqlen, bs, ts, bits, lens, status);
}

}  // namespace
}  // namespace fdb

using namespace fdb;

extern "C" FDB_API int fdb_lengths_from_mask(const void* mask, int32_t mask_type, int32_t batch, int32_t seqlen, int64_t batch_stride,
                                             int64_t token_stride, int32_t* lens, int32_t* status, void* stream) {
  clear_error();
  if (batch < 0 || seqlen < 0) return fail(FDB_ERR_INVALID_ARGUMENT, "lengths_from_mask: batch %d, seqlen %d", batch, seqlen);
  if (batch == 0) return FDB_OK;
  if ((mask == nullptr && seqlen > 0) || lens == nullptr) return fail(FDB_ERR_INVALID_ARGUMENT, "lengths_from_mask: NULL pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (mask_type) {  // a float is zero when no bit but the sign is set
    case kMaskF32: lengths<uint32_t>(mask, batch, seqlen, batch_stride, token_stride, 0x7fffffffu, lens, status, s); break;
    case kMaskI64: lengths<uint64_t>(mask, batch, seqlen, batch_stride, token_stride, ~uint64_t(0), lens, status, s); break;
    case kMaskI32: lengths<uint32_t>(mask, batch, seqlen, batch_stride, token_stride, ~0u, lens, status, s); break;
    case kMaskU8: lengths<uint8_t>(mask, batch, seqlen, batch_stride, token_stride, 0xff, lens, status, s); break;
    case kMaskBf16: lengths<uint16_t>(mask, batch, seqlen, batch_stride, token_stride, 0x7fff, lens, status, s); break;
    default: return fail(FDB_ERR_INVALID_ARGUMENT, "lengths_from_mask: mask type %d", mask_type);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "lengths_from_mask launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

extern "C" FDB_API uint64_t fdb_column_sums_workspace_bytes(int64_t rows, int64_t more_rows, int32_t cols) {
  return uint64_t(splits_of(rows) + (more_rows > 0 ? splits_of(more_rows) : 0)) * uint64_t(cols) * sizeof(float);
}

extern "C" FDB_API int fdb_column_sums(const void* x, int64_t rows, int32_t cols, const void* more, int64_t more_rows, int32_t more_cols,
                                       void* out, void* workspace, uint64_t workspace_bytes, void* stream) {
  clear_error();
  if (x == nullptr || out == nullptr || rows < 0 || cols <= 0 || rows > 2147483647LL || more_rows < 0 || more_rows > 2147483647LL ||
      more_cols > cols || (more_rows > 0 && (more == nullptr || more_cols <= 0)))
    return fail(FDB_ERR_INVALID_ARGUMENT, "column_sums: bad pointer or size");
  if (cols % 8 != 0 || more_cols % 8 != 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(more)) & 15u) != 0)
    return fail(FDB_ERR_ALIGNMENT, "column_sums: columns must be a multiple of 8, pointers 16-byte aligned");
  if (workspace == nullptr || workspace_bytes < fdb_column_sums_workspace_bytes(rows, more_rows, cols))
    return fail(FDB_ERR_WORKSPACE, "column_sums: workspace too small");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const SumPart a = {static_cast<const __nv_bfloat16*>(x), cols, (int)rows, cols, splits_of(rows)};
  const SumPart b = {static_cast<const __nv_bfloat16*>(more), more_cols, (int)more_rows, more_cols, more_rows > 0 ? splits_of(more_rows) : 0};
  float* partial = static_cast<float*>(workspace);
  column_partials_kernel<<<dim3((unsigned)((cols + 255) / 256), (unsigned)(a.splits + b.splits)), kThreads, 0, s>>>(a, b, cols, partial);
  column_finish_kernel<<<(cols + kThreads - 1) / kThreads, kThreads, 0, s>>>(partial, a.splits + b.splits, cols, static_cast<__nv_bfloat16*>(out));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "column_sums launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}
