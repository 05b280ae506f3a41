// Per-slab amax scaling of bf16 rows to float8 e4m3 (the FP8 option; the reference has no FP8 code).
//
// A slab is a run of rows [slab_start[s], slab_start[s+1]) — one sequence, or one head's position table — and every
// (slab, head) gets its own scale = amax/448, so the stored value times the scale gives the input back.
// Two kernels over up to five tensors at once, each with enough CTAs to fill the GPU whatever the number of slabs:
//   amax_kernel      a CTA takes 32-row chunks of one slab; eight lanes share a row of one head and keep that head, so the maximum
//                    stays in a register until the end, then goes through shared memory into the amax array (bit pattern of a
//                    non-negative float, so an unsigned atomicMax orders it)
//   quantize_kernel  the same walk, x * 448/amax -> e4m3; the slab's first CTA writes its scales
// What bounds them is reading the tensors, the second time mostly from L2.  q, k, v (2 x 4096 x 16 heads) and two tables: tensor by
// tensor, with a memset in front and a kernel for the scales behind, 20 launches and 150 us; all at once 27 + 26 us; with a thread's
// head fixed (no division, shuffles and atomics once at the end instead of per row) 13 + 12 us.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"

namespace fdb {
namespace {

constexpr int kQuantThreads = 256;
constexpr int kChunkRows = 32;

constexpr int kQuantTensors = 5;
constexpr int kUnroll = 4;  // 16-byte loads in flight per thread

// One tensor.  CTAs [first_cta, first_cta + per_slab * n_slabs) work on it.
struct Job {
  const __nv_bfloat16* x;
  uint8_t* y;
  const int32_t* slab_start;  // NULL: every slab has slab_rows rows
  unsigned int* amax_bits;    // (n_slabs, heads)
  float* scale;               // (n_slabs, heads)
  int64_t row_stride, head_stride;
  int rows, slab_rows, n_slabs, heads, per_slab, first_cta;
};
struct Jobs { Job job[kQuantTensors]; int n; };

__device__ __forceinline__ const Job& job_of(const Jobs& jobs, int& slab, int& part) {
  int j = 0;
  while (j + 1 < jobs.n && (int)blockIdx.x >= jobs.job[j + 1].first_cta) ++j;
  const int at = blockIdx.x - jobs.job[j].first_cta;
  slab = at / jobs.job[j].per_slab;
  part = at % jobs.job[j].per_slab;
  return jobs.job[j];
}

// Walks this CTA's 32-row chunks of its slab: the CTA's 32 groups of eight lanes (16 bytes each) are dealt to 32 / heads rows of up
// to 32 heads.  `head(h)` before the rows of a head, `body(r, v)` for each row, kUnroll rows loaded at a time, `done(h)` behind
// them (whole warps get there, whatever their lanes' rows).
template <typename H, typename F, typename D>
__device__ __forceinline__ void walk_slab(const Job& job, int slab, int part, H&& head, F&& body, D&& done) {
  // slab bounds clamped to the rows that exist
  const int s0 = job.slab_start != nullptr ? job.slab_start[slab] : slab * job.slab_rows;
  const int s1 = job.slab_start != nullptr ? job.slab_start[slab + 1] : s0 + job.slab_rows;
  const int r0 = min(max(s0, 0), job.rows);
  const int len = max(min(s1, job.rows) - r0, 0);
  const int sub = threadIdx.x & 7, group = threadIdx.x >> 3;
  for (int h0 = 0; h0 < job.heads; h0 += kQuantThreads / 8) {
    const int n = min(job.heads - h0, kQuantThreads / 8), step = kQuantThreads / 8 / n;  // heads and rows per pass
    const int h = h0 + group % n, first = group < step * n ? group / n : kChunkRows;
    head(h);
    const __nv_bfloat16* x = job.x + h * job.head_stride + sub * 8;
    for (int chunk = part; chunk * kChunkRows < len; chunk += job.per_slab) {
      const int base = r0 + chunk * kChunkRows, rows = min(kChunkRows, len - chunk * kChunkRows);
      for (int i = first; i < rows; i += step * kUnroll) {
        uint4 v[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          v[u] = make_uint4(0, 0, 0, 0);
          if (i + u * step < rows) v[u] = *reinterpret_cast<const uint4*>(x + (int64_t)(base + i + u * step) * job.row_stride);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (i + u * step < rows) body(base + i + u * step, v[u]);
      }
    }
    __syncwarp();
    done(h);
  }
}

__global__ void __launch_bounds__(kQuantThreads) amax_kernel(const __grid_constant__ Jobs jobs) {
  extern __shared__ unsigned int s_amax[];
  int slab, part;
  const Job& job = job_of(jobs, slab, part);
  for (int h = threadIdx.x; h < job.heads; h += kQuantThreads) s_amax[h] = 0u;
  __syncthreads();
  const int sub = threadIdx.x & 7;
  float a = 0.f;
  walk_slab(job, slab, part, [&](int) { a = 0.f; },
            [&](int, const uint4& v) {
              const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(b[k]);
                a = fmaxf(a, fmaxf(fabsf(f.x), fabsf(f.y)));
              }
            },
            [&](int h) {
              a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
              a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 2));
              a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 4));
              if (sub == 0 && a > 0.f) atomicMax(&s_amax[h], __float_as_uint(a));
            });
  __syncthreads();
  for (int h = threadIdx.x; h < job.heads; h += kQuantThreads)
    if (s_amax[h] != 0u) atomicMax(&job.amax_bits[(int64_t)slab * job.heads + h], s_amax[h]);
}

__device__ __forceinline__ float scale_of(unsigned int amax_bits) { return fmaxf(__uint_as_float(amax_bits), 1e-12f) / 448.f; }

__global__ void __launch_bounds__(kQuantThreads) quantize_kernel(const __grid_constant__ Jobs jobs) {
  extern __shared__ unsigned int s_amax[];
  int slab, part;
  const Job& job = job_of(jobs, slab, part);
  float* s_inv = reinterpret_cast<float*>(s_amax);
  for (int h = threadIdx.x; h < job.heads; h += kQuantThreads) {
    const float scale = scale_of(job.amax_bits[(int64_t)slab * job.heads + h]);
    s_inv[h] = 1.f / scale;
    if (part == 0 && job.scale != nullptr) job.scale[(int64_t)slab * job.heads + h] = scale;
  }
  __syncthreads();
  const int sub = threadIdx.x & 7;
  float inv = 0.f;
  uint8_t* y = nullptr;
  walk_slab(job, slab, part, [&](int h) { inv = s_inv[h]; y = job.y + h * 64 + sub * 8; },
            [&](int r, const uint4& v) {
              const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
              uint16_t o[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(b[k]);
                o[k] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
              }
              *reinterpret_cast<uint2*>(y + (int64_t)r * job.heads * 64) =
                  make_uint2((uint32_t)o[0] | ((uint32_t)o[1] << 16), (uint32_t)o[2] | ((uint32_t)o[3] << 16));
            },
            [](int) {});
}

__global__ void scale_kernel(float* __restrict__ scale, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) scale[i] = scale_of(__float_as_uint(scale[i]));
}

int run(Jobs& jobs, void* bits, size_t bits_bytes, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(bits, 0, bits_bytes, s);
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "quantize_e4m3 memset: %s", cudaGetErrorString(e));
  int ctas = 0, heads = 0;
  for (int j = 0; j < jobs.n; ++j) {
    Job& job = jobs.job[j];
    // the slab lengths are on the device: a fixed number of CTAs per slab walks its 32-row chunks (about 1200 CTAs for a tensor, and no
    // more than a slab of that many rows can use)
    const int chunks = (job.slab_start != nullptr ? job.rows : job.slab_rows) / kChunkRows + 1;
    job.per_slab = std::max(1, std::min({(1184 + job.n_slabs - 1) / job.n_slabs, 256, chunks}));
    job.first_cta = ctas;
    ctas += job.per_slab * job.n_slabs;
    heads = std::max(heads, job.heads);
  }
  const size_t smem = sizeof(unsigned int) * heads;
  amax_kernel<<<ctas, kQuantThreads, smem, s>>>(jobs);
  quantize_kernel<<<ctas, kQuantThreads, smem, s>>>(jobs);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "quantize_e4m3 launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace

int launch_quantize_e4m3(const void* x, int64_t rows, int64_t row_stride, int64_t head_stride, const int32_t* slab_start,
                         int32_t n_slabs, int32_t heads, int32_t head_dim, void* y, float* scale, void* stream) {
  if (head_dim != 64) return fail(FDB_ERR_UNSUPPORTED, "quantize_e4m3 is built for head_dim 64, got %d", head_dim);
  if (n_slabs <= 0 || heads <= 0) return FDB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int n = n_slabs * heads;
  Jobs jobs;
  jobs.n = 1;
  jobs.job[0] = {static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(y), slab_start, reinterpret_cast<unsigned int*>(scale), nullptr,
                 row_stride, head_stride, (int)rows, 0, n_slabs, heads, 0, 0};
  const int rc = run(jobs, scale, sizeof(float) * n, s);
  if (rc != FDB_OK) return rc;
  scale_kernel<<<(n + 255) / 256, 256, 0, s>>>(scale, n);  // amax -> scale in place
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "quantize_e4m3 launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace fdb

using namespace fdb;

extern "C" FDB_API int fdb_quantize_attn(const fdb_quantize_attn_params* q, void* stream) {
  clear_error();
  if (q == nullptr || q->struct_bytes != sizeof(fdb_quantize_attn_params))
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_quantize_attn_params: NULL or struct_bytes %u != %zu", q ? q->struct_bytes : 0u, sizeof(fdb_quantize_attn_params));
  const int rc = validate(q->in, true);
  if (rc != FDB_OK) return rc;
  const fdb_attn_params& p = *q->in;
  if (p.dtype != FDB_BF16) return fail(FDB_ERR_UNSUPPORTED, "fdb_quantize_attn takes bf16 tensors");
  if (p.batch == 0 || p.total_rows == 0) return FDB_OK;
  const int table_rows = 2 * (p.position_buckets > 0 ? p.position_buckets : p.max_relative_positions);
  const int table_slabs = (p.pos_key ? p.heads : 0) + (p.pos_query ? p.heads : 0);
  const uint64_t need = (3 * uint64_t(p.batch) * p.heads + table_slabs) * sizeof(float);
  if (q->amax == nullptr || q->amax_bytes < need) return fail(FDB_ERR_WORKSPACE, "amax buffer of %llu bytes needed", (unsigned long long)need);
  unsigned int* bits = static_cast<unsigned int*>(q->amax);
  Jobs jobs;
  jobs.n = 0;
  auto add = [&](const void* x, void* y, float* scale, int64_t rs, int64_t hs, int rows, const int32_t* starts, int slab_rows, int slabs, int heads) {
    jobs.job[jobs.n++] = {static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(y), starts, bits, scale, rs, hs, rows, slab_rows, slabs, heads, 0, 0};
    bits += (int64_t)slabs * heads;
  };
  add(p.q, q->q, q->q_scale, p.q_row_stride, p.q_head_stride, p.total_rows, p.cu_seqlens, p.max_seqlen, p.batch, p.heads);
  add(p.k, q->k, q->k_scale, p.k_row_stride, p.k_head_stride, p.total_rows, p.cu_seqlens, p.max_seqlen, p.batch, p.heads);
  add(p.v, q->v, q->v_scale, p.v_row_stride, p.v_head_stride, p.total_rows, p.cu_seqlens, p.max_seqlen, p.batch, p.heads);
  // a table is one slab of table_rows rows per head
  if (p.pos_key) add(p.pos_key, q->pos_key, q->pos_key_scale, 64, 64, p.heads * table_rows, nullptr, table_rows, p.heads, 1);
  if (p.pos_query) add(p.pos_query, q->pos_query, q->pos_query_scale, 64, 64, p.heads * table_rows, nullptr, table_rows, p.heads, 1);
  if (!aligned_to(8, q->q, q->k, q->v, q->pos_key, q->pos_query) ||
      !aligned_to(4, q->amax, q->q_scale, q->k_scale, q->v_scale, q->pos_key_scale, q->pos_query_scale))
    return fail(FDB_ERR_ALIGNMENT, "fdb_quantize_attn: e4m3 outputs must be 8-byte aligned, scales and amax to their elements");
  for (int j = 0; j < jobs.n; ++j)
    if (jobs.job[j].y == nullptr || jobs.job[j].scale == nullptr) return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_quantize_attn: NULL output");
  return run(jobs, q->amax, need, static_cast<cudaStream_t>(stream));
}
