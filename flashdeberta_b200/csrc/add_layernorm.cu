// out = LayerNorm(x + residual) over the last dimension, bf16 in and out, fp32 statistics: the tail of both output blocks of
// a DeBERTa layer (transformers' DebertaV2SelfOutput / DebertaV2Output, which the reference's FlashDebertaV2Attention and
// FlashDebertaV2Layer keep as they are, src/flashdeberta/model.py:259-272): dense -> dropout -> LayerNorm(hidden + input).
// In eager mode that is an elementwise add (3 passes over HBM) followed by torch's layer-norm kernel (2 passes, measured
// at 1.2 TB/s on this shape); here it is one kernel with 3 passes at streaming speed.  The sum is rounded to bf16 before
// the statistics, as the eager expression `self.LayerNorm(hidden_states + input_tensor)` does.
//
// One warp per row, 16-byte loads, the row stays in registers (hidden = VEC * 256 elements, VEC <= 8).  HBM-bound:
// 3 * hidden * 2 bytes per row (2 when there is no residual).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"

namespace fdb {
namespace {

constexpr int kRowsPerBlock = 4;

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float round_bf16(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The attention mask of a token as the eager expression multiplies by it: cast to the activation type first.
__device__ __forceinline__ float mask_value(const void* mask, int type, int64_t i) {
  switch (type) {
    case kMaskF32Exact: return static_cast<const float*>(mask)[i];
    case kMaskF32: return round_bf16(static_cast<const float*>(mask)[i]);
    case kMaskI64: return round_bf16((float)static_cast<const int64_t*>(mask)[i]);
    case kMaskI32: return round_bf16((float)static_cast<const int32_t*>(mask)[i]);
    case kMaskU8: return (float)static_cast<const uint8_t*>(mask)[i];
    default: return __bfloat162float(static_cast<const __nv_bfloat16*>(mask)[i]);
  }
}

template <int VEC>
__global__ void __launch_bounds__(32 * kRowsPerBlock) add_layernorm_kernel(const LayerNormCall c) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kRowsPerBlock + (threadIdx.x >> 5);
  ptx::grid_launch();
  ptx::grid_wait();
  constexpr int kVecPerRow = VEC * 32;
  const int64_t rows = c.rows_dev != nullptr ? (int64_t)*c.rows_dev : c.rows;
  if (row >= rows) {
    if (c.zero_tail != nullptr && row < c.rows && row < rows + kTileN) {
      uint4* z = static_cast<uint4*>(c.zero_tail) + row * kVecPerRow;
#pragma unroll
      for (int i = 0; i < VEC; ++i) z[i * 32 + lane] = make_uint4(0, 0, 0, 0);
    }
    return;
  }
  int64_t src = row;
  float scale = 1.f;
  if (c.ids != nullptr) {  // embedding form: x is a table, this row is table[ids[token]]
    const int64_t token = c.token_index != nullptr ? c.token_index[row] : row;
    if (c.mask != nullptr) scale = mask_value(c.mask, c.mask_type, token);
    src = c.ids[token];
    if (src < 0 || src >= c.table_rows) {
      if (lane == 0 && c.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(c.status), FDB_DEV_BAD_INDEX);
      src = src < 0 ? 0 : c.table_rows - 1;
    }
  }
  const uint4* xr = static_cast<const uint4*>(c.x) + src * kVecPerRow;
  const uint4* rr = c.residual != nullptr ? static_cast<const uint4*>(c.residual) + row * kVecPerRow : nullptr;
  float v[VEC * 8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const uint4 a = __ldg(xr + i * 32 + lane);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
    if (rr != nullptr) {
      const uint4 b = __ldg(rr + i * 32 + lane);
      const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[i * 8 + 2 * k] = round_bf16(bf16_lo(aw[k]) + bf16_lo(bw[k]));
        v[i * 8 + 2 * k + 1] = round_bf16(bf16_hi(aw[k]) + bf16_hi(bw[k]));
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[i * 8 + 2 * k] = bf16_lo(aw[k]);
        v[i * 8 + 2 * k + 1] = bf16_hi(aw[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += v[i * 8 + k];
  }
  constexpr float kInv = 1.f / float(VEC * 256);
  const float mean = warp_sum(sum) * kInv;
  float sq = 0.f;
#pragma unroll
  for (int k = 0; k < VEC * 8; ++k) {
    const float d = v[k] - mean;
    sq = fmaf(d, d, sq);
  }
  const float rstd = rsqrtf(warp_sum(sq) * kInv + c.eps);
  uint4* orow = static_cast<uint4*>(c.out) + (c.out_index != nullptr ? (int64_t)c.out_index[row] : row) * kVecPerRow;
  const uint4* gamma = static_cast<const uint4*>(c.gamma);
  const uint4* beta = static_cast<const uint4*>(c.beta);
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    const uint4 g = __ldg(gamma + i * 32 + lane), b = __ldg(beta + i * 32 + lane);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, bw[4] = {b.x, b.y, b.z, b.w};
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float lo = fmaf((v[i * 8 + 2 * k] - mean) * rstd, bf16_lo(gw[k]), bf16_lo(bw[k]));
      float hi = fmaf((v[i * 8 + 2 * k + 1] - mean) * rstd, bf16_hi(gw[k]), bf16_hi(bw[k]));
      if (c.mask != nullptr) {  // the normalised row is rounded before it is scaled, as two separate kernels would
        lo = round_bf16(lo) * scale;
        hi = round_bf16(hi) * scale;
      }
      o[k] = pack2(lo, hi);
    }
    orow[i * 32 + lane] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int VEC>
int launch(const LayerNormCall& c, cudaStream_t s) {
  const dim3 grid((unsigned)((c.rows + kRowsPerBlock - 1) / kRowsPerBlock));
  const cudaError_t e = launch_kernel<LayerNormCall>(add_layernorm_kernel<VEC>, c, grid, 32 * kRowsPerBlock, 0, c.chained, s);
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "add_layernorm launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace

int launch_layernorm(const LayerNormCall& c, void* stream) {
  if (c.rows < 0 || c.rows > (int64_t(1) << 31) * kRowsPerBlock - 1) return fail(FDB_ERR_LIMIT, "rows = %lld", (long long)c.rows);
  if (c.hidden <= 0 || c.hidden % 256 != 0 || c.hidden > 2048)
    return fail(FDB_ERR_UNSUPPORTED, "hidden = %d: the kernel handles multiples of 256 up to 2048", c.hidden);
  const uintptr_t all = reinterpret_cast<uintptr_t>(c.x) | reinterpret_cast<uintptr_t>(c.residual) |
                        reinterpret_cast<uintptr_t>(c.gamma) | reinterpret_cast<uintptr_t>(c.beta) | reinterpret_cast<uintptr_t>(c.out);
  if ((all & 15u) != 0) return fail(FDB_ERR_ALIGNMENT, "pointers must be 16-byte aligned");
  if (c.rows == 0) return FDB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (c.hidden / 256) {
    case 1: return launch<1>(c, s);
    case 2: return launch<2>(c, s);
    case 3: return launch<3>(c, s);
    case 4: return launch<4>(c, s);
    case 5: return launch<5>(c, s);
    case 6: return launch<6>(c, s);
    case 7: return launch<7>(c, s);
    default: return launch<8>(c, s);
  }
}

}  // namespace fdb

using namespace fdb;

extern "C" FDB_API int fdb_add_layernorm(const void* x, const void* residual, const void* gamma, const void* beta, void* out,
                                         int64_t rows, int32_t hidden, float eps, void* stream) {
  clear_error();
  if (x == nullptr || gamma == nullptr || beta == nullptr || out == nullptr)
    return fail(FDB_ERR_INVALID_ARGUMENT, "x, gamma, beta and out must not be NULL");
  LayerNormCall c = {};
  c.x = x; c.residual = residual; c.gamma = gamma; c.beta = beta; c.out = out;
  c.rows = rows; c.hidden = hidden; c.eps = eps;
  return launch_layernorm(c, stream);
}

extern "C" FDB_API int fdb_embed_layernorm(const int64_t* ids, const void* table, int64_t table_rows, const void* gamma,
                                           const void* beta, const float* row_scale, void* out, int64_t rows,
                                           int32_t hidden, float eps, int32_t* status, void* stream) {
  clear_error();
  if (ids == nullptr || table == nullptr || gamma == nullptr || beta == nullptr || out == nullptr)
    return fail(FDB_ERR_INVALID_ARGUMENT, "ids, table, gamma, beta and out must not be NULL");
  if (table_rows <= 0) return fail(FDB_ERR_INVALID_ARGUMENT, "table_rows = %lld", (long long)table_rows);
  LayerNormCall c = {};
  c.x = table; c.gamma = gamma; c.beta = beta; c.out = out;
  c.rows = rows; c.hidden = hidden; c.eps = eps;
  c.ids = ids; c.table_rows = table_rows; c.mask = row_scale; c.mask_type = kMaskF32Exact; c.status = status;
  return launch_layernorm(c, stream);
}
