// Small kernels of the attention module around the attention itself.
//
//  * lengths_kernel   valid lengths of a right-padded batch from its mask, and the check that the mask is one: a CTA per
//                     sequence.  As tensor operators this was nine launches of a few hundred bytes each.
//  * fdb_projected_forward  the module's forward in training: two launches of the linear kernel, then the attention.  Operator by
//                     operator (two concatenations, two GEMMs, a transposition, the attention call) it was 110 us of host time.
//  * column_sums      bias gradients: sums over the rows of one or two bf16 matrices side by side, fp32 inside.  Bound by
//                     reading them; the row ranges of a column are summed in a fixed order by a second launch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"
#include "linear.h"
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
  const unsigned mask_bytes[] = {4, 8, 4, 1, 2};  // of FDB_MASK_*
  if (mask_type >= FDB_MASK_F32 && mask_type <= FDB_MASK_BF16 && (!aligned_to(mask_bytes[mask_type], mask) || !aligned_to(4, lens, status)))
    return fail(FDB_ERR_ALIGNMENT, "lengths_from_mask: mask, lens and status must be aligned to their elements");
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
  if (cols % 8 != 0 || more_cols % 8 != 0 || !aligned_to(16, x, more) || !aligned_to(4, workspace) || !aligned_to(2, out))
    return fail(FDB_ERR_ALIGNMENT, "column_sums: columns must be a multiple of 8, matrices 16-byte aligned, the others to their elements");
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

extern "C" FDB_API int fdb_projected_forward(const fdb_projected_params* c, void* stream) {
  clear_error();
  if (c == nullptr || c->struct_bytes != sizeof(fdb_projected_params))
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_projected_params: NULL or struct_bytes %u != %zu", c ? c->struct_bytes : 0u, sizeof(fdb_projected_params));
  int rc = validate(c->attn, true);
  if (rc != FDB_OK) return rc;
  const fdb_attn_params& p = *c->attn;
  const int inner = p.heads * kHeadDim, table_rows = 2 * (p.position_buckets > 0 ? p.position_buckets : p.max_relative_positions);
  if (p.dtype != FDB_BF16 || c->in_features <= 0 || c->in_features % 64 != 0)
    return fail(FDB_ERR_UNSUPPORTED, "fdb_projected_forward takes bf16 and in_features a multiple of 64");
  if (!p.pos_key || !p.pos_query || !c->x || !c->rel || !c->wq || !c->bq || !c->wk || !c->bk || !c->wv || !c->bv)
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_projected_forward: NULL pointer");
  const uintptr_t all = (uintptr_t)c->x | (uintptr_t)c->rel | (uintptr_t)c->wq | (uintptr_t)c->bq | (uintptr_t)c->wk | (uintptr_t)c->bk |
                        (uintptr_t)c->wv | (uintptr_t)c->bv;
  if ((all & 15u) != 0 || p.q_row_stride != p.k_row_stride || p.q_row_stride != p.v_row_stride || p.q_head_stride != kHeadDim ||
      p.k_head_stride != kHeadDim || p.v_head_stride != kHeadDim || c->table_head_stride != kHeadDim || c->table_row_stride < inner ||
      c->table_row_stride % 8 != 0)
    return fail(FDB_ERR_ALIGNMENT, "fdb_projected_forward: pointers must be 16-byte aligned, q, k and v rows of one stride, heads 64 apart");
  if (p.batch == 0 || p.total_rows == 0) return FDB_OK;
  const ExpandGeometry g = expand_geometry(p.lut_d_min, p.lut_len);
  const WorkspaceLayout w = workspace_layout(p, g);
  if (p.workspace == nullptr || p.workspace_bytes < w.total || (reinterpret_cast<uintptr_t>(p.workspace) & 255u) != 0)
    return fail(FDB_ERR_WORKSPACE, "workspace of %llu bytes needed (256-byte aligned), %llu given", (unsigned long long)w.total, (unsigned long long)p.workspace_bytes);
  CUtensorMap map_x, map_rel;
  LinearWeight wq, wk, wv;
  if ((rc = make_linear_input_map(&map_x, c->x, p.total_rows, c->in_features)) != FDB_OK) return rc;
  if ((rc = make_linear_input_map(&map_rel, c->rel, table_rows, c->in_features)) != FDB_OK) return rc;
  if ((rc = make_linear_maps(&wq, c->wq, inner, c->in_features)) != FDB_OK || (rc = make_linear_maps(&wk, c->wk, inner, c->in_features)) != FDB_OK ||
      (rc = make_linear_maps(&wv, c->wv, inner, c->in_features)) != FDB_OK) return rc;
  LinearCall lin = {};
  lin.x_map = &map_x; lin.rows = p.total_rows; lin.out_stride = p.q_row_stride;
  lin.k = c->in_features; lin.n = inner; lin.groups = 3; lin.status = p.status;
  lin.weight[0] = &wq; lin.weight[1] = &wk; lin.weight[2] = &wv;
  lin.bias[0] = c->bq; lin.bias[1] = c->bk; lin.bias[2] = c->bv;
  lin.out[0] = const_cast<void*>(p.q); lin.out[1] = const_cast<void*>(p.k); lin.out[2] = const_cast<void*>(p.v);
  if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
  lin.x_map = &map_rel; lin.rows = table_rows; lin.out_stride = c->table_row_stride; lin.groups = 2;
  lin.out[0] = const_cast<void*>(p.pos_query); lin.out[1] = const_cast<void*>(p.pos_key);
  if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
  fdb_attn_params q = p;
  q.prepared = 0;
  const AttnBuffers b = attn_buffers(q, w);
  bool prepared;
  if ((rc = launch_prepare(q, g, b, stream, &prepared, {c->table_row_stride, c->table_head_stride})) != FDB_OK) return rc;
  return launch_attn_fwd_sm100(q, g, b, stream, prepared);
}
