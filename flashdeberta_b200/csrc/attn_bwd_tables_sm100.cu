// The two products of the attention backward that use the bucket sums of one side, in one pass over them (sm_100a):
//   d[rows, 64]         = core + sums . table                          (dQ with pos_key, dK with pos_query)
//   dtable[W, 64]       = sum over the rows of sums^T . operand        (dpos_key with Q, dpos_query with K)
// for every head; sums is (heads, rows, W) bf16, core fp32, the results bf16.
//
// The sums are by far the largest thing read (1 KB per row and head at W = 512, against 128 to 256 bytes for the others), so a
// 128 x 128 piece of them is brought to shared memory once and read by both products: as it lies (K-major) for the first one,
// transposed by the operand descriptor (MN-major) for the second.  One CTA per SM walks a share of one head's row tiles:
//   warps 0-3  core + product -> d      warp 4  issues the tcgen05.mma      warp 5  issues the TMA loads
// Tensor memory: two row products (128 x 64, alternating) and up to four 128 x 64 pieces of dtable, which stay there until the
// CTA's last tile; the CTAs' parts of dtable then go to memory in fp32 and bwd_table_reduce_kernel adds them in a fixed order.
//
// What bounds it: reading the sums.  8192 rows x 12 heads x 512: 36 us and 5 for the reduction, where two library products, the
// addition and its fp32 round trip took 79 (and 18 for a memset of the sums that went with them).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "attn_bwd.h"
#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"
#include "tensor_map.cuh"

namespace fdb {
namespace {

using namespace ptx;

constexpr int kThreads = 192, kMmaWarp = 4, kTmaWarp = 5;
constexpr int kPieces = 4;                       // 128 table rows each: what tensor memory holds of dtable
constexpr int kStages = 4;
constexpr uint32_t kPieceBytes = 128 * 128 * 2;  // sums: two panels of 64 table rows
constexpr uint32_t kSmemTable = 0;               // kPieces x (128 x 128 B)
constexpr uint32_t kSmemOperand = kPieces * 16384;
constexpr uint32_t kSmemSums = kSmemOperand + 2 * 16384;
constexpr uint32_t kSmemBars = kSmemSums + kStages * kPieceBytes;
constexpr uint32_t kSmemBytes = kSmemBars + 256 + 1024;
constexpr uint32_t kTmemCols = 512, kColRow = 0, kColTable = 128;
static_assert(kSmemBytes <= 232448, "shared memory");

enum Bar : uint32_t {
  kBarTable = 0,                     // table landed
  kBarOp = 1, kBarOpFree = 3,        // operand tile landed / read, two of each
  kBarSums = 5, kBarSumsFree = 9,    // piece of the sums landed / read, kStages of each
  kBarRow = 13, kBarRowFree = 15,    // row product finished / read (4 warps), two of each
  kBarLast = 17,                     // every product finished
  kNumBars = 18
};

struct alignas(64) TableArgs {
  CUtensorMap tm_sums, tm_table, tm_operand;
  float* core;               // (heads, 64) per row: read; written unless this is the last group of table rows
  int64_t core_row_stride;
  __nv_bfloat16* out;        // last group: rows of row_stride elements, heads of head_stride
  int64_t row_stride, head_stride;
  float* partial;            // (heads, parts, group rows, 64)
  int32_t* status;
  int rows, heads, w0, w_rows;  // this launch's group of table rows
  bool last;
};

__global__ void __launch_bounds__(kThreads, 1) bwd_tables_kernel(const __grid_constant__ TableArgs args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = (int)uniform(uint32_t(tid) >> 5), lane = tid & 31;
  const int head = blockIdx.y, part = blockIdx.x, parts = gridDim.x;
  const int all_tiles = (args.rows + 127) / 128;
  const int t0 = (int)((int64_t)all_tiles * part / parts), t1 = (int)((int64_t)all_tiles * (part + 1) / parts);  // at least one
  const int pieces = (args.w_rows + 127) / 128;

  auto bar = [&](uint32_t i) -> uint32_t { return smem + kSmemBars + 8u * i; };
  const uint32_t tmem_slot = bar(kNumBars);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBars + 8u * kNumBars + 8u);
  if (tid == 0) {
    *abort_flag = 0u;
    for (uint32_t i = 0; i < kNumBars; ++i) mbar_init(bar(i), i == kBarRowFree || i == kBarRowFree + 1 ? 4u : 1u);
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBars + 8u * kNumBars));

  bool ok = true;
  auto wait = [&](uint32_t b, uint32_t parity) {
    if (ok) ok = mbar_wait_warp(b, parity, abort_flag);
  };

  if (warp == kTmaWarp) {
    if (elect_one()) {
      mbar_expect_tx(bar(kBarTable), uint32_t(pieces) * 16384u);
      for (int p = 0; p < pieces; ++p)
        tma_load_3d(smem + kSmemTable + uint32_t(p) * 16384u, &args.tm_table, bar(kBarTable), 0, head, args.w0 + p * 128);
    }
    uint32_t n = 0;  // pieces so far
#pragma unroll 1
    for (int t = t0; t < t1 && ok; ++t) {
      const uint32_t i = uint32_t(t - t0), o = i & 1u;
      if (i >= 2) wait(bar(kBarOpFree + o), ((i >> 1) - 1u) & 1u);
      if (ok && elect_one()) {
        mbar_expect_tx(bar(kBarOp + o), 16384u);
        tma_load_3d(smem + kSmemOperand + o * 16384u, &args.tm_operand, bar(kBarOp + o), 0, head, t * 128);
      }
#pragma unroll 1
      for (int p = 0; p < pieces && ok; ++p, ++n) {
        const uint32_t s = n % kStages;
        if (n >= kStages) wait(bar(kBarSumsFree + s), (n / kStages - 1u) & 1u);
        if (ok && elect_one()) {
          const uint32_t dst = smem + kSmemSums + s * kPieceBytes;
          mbar_expect_tx(bar(kBarSums + s), kPieceBytes);
          tma_load_3d(dst, &args.tm_sums, bar(kBarSums + s), args.w0 + p * 128, t * 128, head);
          tma_load_3d(dst + 16384u, &args.tm_sums, bar(kBarSums + s), args.w0 + p * 128 + 64, t * 128, head);
        }
      }
    }
  } else if (warp == kMmaWarp) {
    const uint32_t idesc_row = instr_desc(128, 64, 1, 0, 1), idesc_table = instr_desc(128, 64, 1, 1, 1);
    const uint64_t dtable = smem_desc_sw128(smem + kSmemTable, 1024, 16);
    wait(bar(kBarTable), 0);
    uint32_t n = 0;
#pragma unroll 1
    for (int t = t0; t < t1 && ok; ++t) {
      const uint32_t i = uint32_t(t - t0), o = i & 1u;
      if (i >= 2) wait(bar(kBarRowFree + o), ((i >> 1) - 1u) & 1u);
      wait(bar(kBarOp + o), (i >> 1) & 1u);
      const uint64_t dop = smem_desc_sw128(smem + kSmemOperand + o * 16384u, 1024, 16);
#pragma unroll 1
      for (int p = 0; p < pieces && ok; ++p, ++n) {
        const uint32_t s = n % kStages;
        wait(bar(kBarSums + s), (n / kStages) & 1u);
        tc_fence_after();
        if (ok && elect_one()) {
          const uint32_t at = smem + kSmemSums + s * kPieceBytes;
          const uint64_t d_k = smem_desc_sw128(at, 1024, 16);       // rows of the sums as M
          const uint64_t d_mn = smem_desc_sw128(at, 1024, 16384);   // table rows as M: panels of 64 lie 16 KB apart
#pragma unroll
          for (int k = 0; k < 8; ++k)
            mma_bf16(tmem_base + kColRow + 64u * o, d_k + uint64_t(((k >> 2) * 16384 + (k & 3) * 32) >> 4),
                     dtable + uint64_t((p * 16384 + k * 2048) >> 4), idesc_row, uint32_t(p > 0 || k > 0));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            mma_bf16(tmem_base + kColTable + 64u * uint32_t(p), d_mn + uint64_t((k * 2048) >> 4), dop + uint64_t((k * 2048) >> 4),
                     idesc_table, uint32_t(i > 0 || k > 0));
          mma_commit(bar(kBarSumsFree + s));
          if (p == pieces - 1) {
            mma_commit(bar(kBarOpFree + o));
            mma_commit(bar(kBarRow + o));
            if (t == t1 - 1) mma_commit(bar(kBarLast));
          }
        }
      }
    }
  } else {
    const int r = warp * 32 + lane;
    const uint32_t tmem_lane = tmem_base + (uint32_t(warp * 32) << 16);
#pragma unroll 1
    for (int t = t0; t < t1; ++t) {
      const uint32_t i = uint32_t(t - t0), o = i & 1u;
      const int row = t * 128 + r;
      const bool valid = row < args.rows;
      float4* core = reinterpret_cast<float4*>(args.core + (int64_t)(valid ? row : args.rows - 1) * args.core_row_stride + head * 64);
      float4 c[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) c[q] = core[q];
      wait(bar(kBarRow + o), (i >> 1) & 1u);
      tc_fence_after();
      uint32_t x[64];
      tmem_ld32(tmem_lane + kColRow + 64u * o, reinterpret_cast<uint32_t(&)[32]>(x[0]));
      tmem_ld32(tmem_lane + kColRow + 64u * o + 32u, reinterpret_cast<uint32_t(&)[32]>(x[32]));
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(bar(kBarRowFree + o));
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        c[q].x += __uint_as_float(x[4 * q]);
        c[q].y += __uint_as_float(x[4 * q + 1]);
        c[q].z += __uint_as_float(x[4 * q + 2]);
        c[q].w += __uint_as_float(x[4 * q + 3]);
      }
      if (valid && !args.last) {
#pragma unroll
        for (int q = 0; q < 16; ++q) core[q] = c[q];
      } else if (valid) {
        uint4* out = reinterpret_cast<uint4*>(args.out + (int64_t)row * args.row_stride + (int64_t)head * args.head_stride);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          out[q] = make_uint4(pack_bf16x2(c[2 * q].x, c[2 * q].y), pack_bf16x2(c[2 * q].z, c[2 * q].w),
                              pack_bf16x2(c[2 * q + 1].x, c[2 * q + 1].y), pack_bf16x2(c[2 * q + 1].z, c[2 * q + 1].w));
      }
      __syncwarp();
    }
    wait(bar(kBarLast), 0);
    tc_fence_after();
#pragma unroll 1
    for (int p = 0; p < pieces; ++p) {
      uint32_t x[64];
      tmem_ld32(tmem_lane + kColTable + 64u * uint32_t(p), reinterpret_cast<uint32_t(&)[32]>(x[0]));
      tmem_ld32(tmem_lane + kColTable + 64u * uint32_t(p) + 32u, reinterpret_cast<uint32_t(&)[32]>(x[32]));
      tmem_wait_ld();
      const int w = p * 128 + r;
      float4* dst = reinterpret_cast<float4*>(args.partial + (((int64_t)head * parts + part) * args.w_rows + w) * 64);
      if (w < args.w_rows) {
#pragma unroll
        for (int q = 0; q < 16; ++q)
          dst[q] = make_float4(__uint_as_float(x[4 * q]), __uint_as_float(x[4 * q + 1]), __uint_as_float(x[4 * q + 2]), __uint_as_float(x[4 * q + 3]));
      }
      __syncwarp();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (tid == 0 && args.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(args.status), FDB_DEV_TIMEOUT);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // copies and MMAs in flight get a bounded time to land
    __syncthreads();
  }
  if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
}

// dtable = sum of the CTAs' parts, in bf16
__global__ void __launch_bounds__(256) bwd_table_reduce_kernel(const float4* __restrict__ partial, int parts, int w_rows, int w0, int heads,
                                                               int64_t row_stride, int64_t head_stride, __nv_bfloat16* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;  // (head, w, 4 columns)
  const int64_t per_head = (int64_t)w_rows * 16;
  if (i >= per_head * heads) return;
  const int64_t h = i / per_head, at = i % per_head;
  const float4* src = partial + h * parts * per_head + at;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int p = 0; p < parts; ++p) {
    const float4 v = src[p * per_head];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  *reinterpret_cast<uint2*>(out + h * head_stride + (w0 + at / 16) * row_stride + at % 16 * 4) = make_uint2(pack_bf16x2(s.x, s.y), pack_bf16x2(s.z, s.w));
}

// (heads, rows, width) bf16, contiguous -> box of 64 x 128 x 1 elements, 128-byte swizzle
int make_map_sums(CUtensorMap* m, const void* base, int width, int64_t rows, int heads) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return fail(FDB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[3] = {(cuuint64_t)width, (cuuint64_t)rows, (cuuint64_t)heads};
  const cuuint64_t strides[2] = {(cuuint64_t)width * 2, (cuuint64_t)width * 2 * (cuuint64_t)rows};
  const cuuint32_t box[3] = {64, 128, 1}, estr[3] = {1, 1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FDB_ERR_CUDA, "cuTensorMapEncodeTiled(bucket sums) failed with CUresult %d", (int)r);
  return FDB_OK;
}

// One CTA per SM: a head's row tiles are shared by as many CTAs as that gives, by at most one CTA per tile.
int parts_of(int64_t rows, int heads) {
  const int sms = sm_count() > 0 ? sm_count() : 148;
  return (int)std::max<int64_t>(1, std::min<int64_t>(sms / heads, (rows + 127) / 128));
}

}  // namespace

int launch_zero_table(void* dtable, int64_t row_stride, int64_t head_stride, int heads, int table_rows, cudaStream_t stream) {
  const int64_t n = (int64_t)heads * table_rows * 16;  // a sum of no parts
  bwd_table_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(nullptr, 0, table_rows, 0, heads, row_stride, head_stride,
                                                                          static_cast<__nv_bfloat16*>(dtable));
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "attn_bwd tables launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

uint64_t bwd_tables_partial_bytes(int64_t rows, int heads, int table_rows) {
  return uint64_t(heads) * parts_of(rows, heads) * std::min(table_rows, 128 * kPieces) * 64 * sizeof(float);
}

int launch_bwd_tables(const BwdTablesCall& c, cudaStream_t stream) {
  TableArgs a;
  int rc;
  if ((rc = make_map_sums(&a.tm_sums, c.sums, c.table_rows, c.rows, c.heads))) return rc;
  if ((rc = make_map_rows(&a.tm_table, c.table, c.table_rows, c.heads, c.table_row_stride, c.table_head_stride, 128, false, "position table"))) return rc;
  if ((rc = make_map_rows(&a.tm_operand, c.operand, c.rows, c.heads, c.operand_row_stride, c.operand_head_stride, 128, false, "backward operand"))) return rc;
  a.core = c.core; a.core_row_stride = c.core_row_stride;
  a.out = static_cast<__nv_bfloat16*>(c.out);
  a.row_stride = c.out_row_stride; a.head_stride = c.out_head_stride;
  a.partial = c.partial;
  a.status = c.status;
  a.rows = (int)c.rows; a.heads = c.heads;
  const int parts = parts_of(c.rows, c.heads);
  static std::atomic<uint64_t> smem_done{0};
  cudaError_t e = allow_smem(smem_done, reinterpret_cast<const void*>(bwd_tables_kernel), (int)kSmemBytes);
  // 512 table rows at a time: what tensor memory holds of dtable (256 buckets, as in every DeBERTa-v3 model, are one launch)
  for (int w0 = 0; w0 < c.table_rows && e == cudaSuccess; w0 += 128 * kPieces) {
    a.w0 = w0;
    a.w_rows = std::min(c.table_rows - w0, 128 * kPieces);
    a.last = w0 + a.w_rows == c.table_rows;
    e = launch_kernel<TableArgs>(bwd_tables_kernel, a, dim3((unsigned)parts, (unsigned)c.heads), kThreads, kSmemBytes, false, stream);
    if (e != cudaSuccess) break;
    const int64_t n = (int64_t)c.heads * a.w_rows * 16;
    bwd_table_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(reinterpret_cast<const float4*>(c.partial), parts, a.w_rows, w0, c.heads,
                                                                            c.table_row_stride, c.table_head_stride, static_cast<__nv_bfloat16*>(c.dtable));
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "attn_bwd tables launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace fdb
