// Set-up kernels that run in front of the fused attention kernel, on the same stream.
//
//  * seq_info_kernel   turns cu_seqlens / seq_lens into (first row, length) per sequence and an exclusive prefix of
//                      query tiles per sequence, so the fused kernel's CTAs can find their tile without any host
//                      involvement.  The reference builds the same map in a Python loop with one device->host read per
//                      sequence (src/flashdeberta/ops/flash_attention_varlen.py:71-83) and re-uploads it every layer.
//  * expand_tables_kernel  gathers rows of the projected position tables through the bucket table:
//                      expanded[h][u] = table[h][ idx(d_first + u) ].  After this the relative index of
//                      (query m, key n) is just the row (m - n) - d_first: every tile pair needs a contiguous window
//                      of rows and the fused kernel never evaluates the bucket function.
#include <cuda_runtime.h>

#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"

namespace fdb {

ExpandGeometry expand_geometry(int32_t lut_d_min, int32_t lut_len) {
  ExpandGeometry g;
  g.sat_lo = lut_d_min;
  g.sat_hi = lut_d_min + lut_len - 1;
  // A tile pair that is not saturated has distances [d0, d0+254] with sat_lo-253 <= d0 <= sat_hi-1 and loads the
  // kWindow rows starting at d0.
  g.d_first = g.sat_lo - 254;
  g.rows = (g.sat_hi + 254) - g.d_first + 1;
  return g;
}

static inline uint64_t align256(uint64_t x) { return (x + 255) & ~uint64_t(255); }

// Two launches pay off once a query tile has key tiles with saturated position terms on both sides of the band.
bool want_split(const fdb_attn_params& p) {
  if (p.dtype == FDB_E4M3 || (p.pos_key == nullptr && p.pos_query == nullptr)) return false;
  if (p.tune & FDB_TUNE_ONE_LAUNCH) return false;
  if (p.tune & FDB_TUNE_TWO_LAUNCHES) return true;
  return p.max_seqlen >= kSplitSeqlen;
}

int64_t tile_slots(const fdb_attn_params& p) {
  const int64_t dense_tiles = (int64_t)p.batch * ((p.max_seqlen + kTileM - 1) / kTileM);
  if (p.cu_seqlens == nullptr) return dense_tiles;
  const int64_t bound = (int64_t)(p.total_rows + kTileM - 1) / kTileM + p.batch;
  return dense_tiles < bound ? dense_tiles : bound;
}

WorkspaceLayout workspace_layout(const fdb_attn_params& p, const ExpandGeometry& g, bool allow_split) {
  WorkspaceLayout w;
  const uint64_t esz = p.dtype == FDB_E4M3 ? 1 : 2;
  uint64_t off = 0;
  w.seq_info = off;   off = align256(off + uint64_t(p.batch) * 2 * sizeof(int32_t));
  w.tile_first = off; off = align256(off + uint64_t(p.batch + 1) * sizeof(int32_t));
  w.slot_info = off;  off = align256(off + uint64_t(tile_slots(p)) * 4 * sizeof(int32_t));
  const uint64_t table = uint64_t(p.heads) * g.rows * kHeadDim * esz;
  w.exp_key = off;    off = align256(off + (p.pos_key ? table : 0));
  w.exp_query = off;  off = align256(off + (p.pos_query ? table : 0));
  w.split = allow_split && want_split(p);
  const uint64_t cells = w.split ? uint64_t(p.total_rows) * p.heads : 0;
  w.part_o = off;     off = align256(off + cells * kHeadDim * sizeof(float));
  w.part_ml = off;    off = align256(off + cells * 2 * sizeof(float));
  w.total = off;
  return w;
}

namespace {

constexpr int kScanThreads = 1024;

// inclusive scan over the CTA; `total` of all threads
__device__ __forceinline__ int32_t block_scan(int32_t v, int32_t* s_warp, int32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t up = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += up;
  }
  __syncthreads();  // s_warp may still be read from the scan before
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  int32_t w = s_warp[lane];  // every warp scans the 32 warp sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int32_t up = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += up;
  }
  total = __shfl_sync(0xffffffffu, w, 31);
  return v + (warp > 0 ? __shfl_sync(0xffffffffu, w, warp - 1) : 0);
}

// The pos-th query tile of a sequence of n tiles.  The tiles away from both ends come first: they have the most band key tiles
// (the expensive kind), so the CTAs that run last are the cheaper ones.  4 .. n-5, then the pairs (k, n-1-k) for k = 3 .. 0.
__device__ __forceinline__ int tile_at(int pos, int n) {
  const int inner = n > 8 ? n - 8 : 0;
  if (pos < inner) return pos + 4;
  int r = pos - inner, k = n >= 8 ? 3 : (n - 1) / 2;
  if (n < 8 && (n & 1)) {  // the middle tile is its own pair
    if (r == 0) return k;
    --r;
    --k;
  }
  k -= r >> 1;
  return (r & 1) ? n - 1 - k : k;
}

// One CTA.  Its latency stands in front of every call, so it takes two scans by shuffles, works in shared memory and fills the
// slot table with all threads (one thread wrote the slots of a sequence and the
// lengths were ranked out of global memory: 4.5 -> 3.2 us for two sequences).
__global__ void __launch_bounds__(kScanThreads) seq_info_kernel(const int32_t* __restrict__ cu_seqlens,
                                                                const int32_t* __restrict__ seq_lens, int batch,
                                                                int max_seqlen, int total_rows,
                                                                int32_t* __restrict__ seq_info,
                                                                int32_t* __restrict__ tile_first,
                                                                int4* __restrict__ slot_info, int slots,
                                                                int32_t* __restrict__ status) {
  __shared__ int32_t s_warp[32], s_len[kScanThreads], s_start[kScanThreads], s_first[kScanThreads + 1], s_seq[kScanThreads];
  ptx::grid_launch();
  const int t = threadIdx.x;
  const int per = (batch + kScanThreads - 1) / kScanThreads;
  const int b0 = t * per, b1 = min(batch, b0 + per);
  const bool packed = cu_seqlens != nullptr;
  const int dense_tiles = (max_seqlen + kTileM - 1) / kTileM;
  bool bad = false;
  int32_t sum = 0;
  int start = 0, len = 0;
  for (int b = b0; b < b1; ++b) {
    if (packed) {
      start = cu_seqlens[b];
      len = cu_seqlens[b + 1] - start;
      if (start < 0 || len < 0 || len > max_seqlen || start + len > total_rows) { bad = true; len = 0; start = 0; }
    } else {
      start = b * max_seqlen;
      len = seq_lens != nullptr ? seq_lens[b] : max_seqlen;
      if (len < 0 || len > max_seqlen) { bad = true; len = len < 0 ? 0 : max_seqlen; }
    }
    seq_info[2 * b] = start;
    seq_info[2 * b + 1] = len;
    // dense: every tile of the padded row range is visited so padding rows get their zeros
    sum += packed ? (len + kTileM - 1) / kTileM : dense_tiles;
  }
  s_len[t] = len;
  s_start[t] = start;
  int32_t total_tiles;
  const int32_t first = block_scan(sum, s_warp, total_tiles) - sum;
  int32_t run = first;
  for (int b = b0; b < b1; ++b) {
    tile_first[b] = run;
    run += per == 1 ? sum : (packed ? (seq_info[2 * b + 1] + kTileM - 1) / kTileM : dense_tiles);
  }
  if (t == kScanThreads - 1) tile_first[batch] = total_tiles;

  // Slot table: the order in which the fused kernels' CTAs take the query tiles.  A query tile costs in proportion to its
  // sequence's length, so the sequences go longest first (ties by index): the last CTAs of a ragged batch are then the
  // cheap ones.  With more sequences than threads the order stays that of the batch.
  if (batch <= kScanThreads) {
    int rank = 0;
    if (t < batch)
      for (int o = 0; o < batch; ++o) {
        const int lo = s_len[o];
        rank += (lo > len || (lo == len && o < t)) ? 1 : 0;
      }
    if (t < batch) s_seq[rank] = t;
    __syncthreads();
    const int seq = t < batch ? s_seq[t] : 0;  // from here on thread t stands for the sequence of rank t
    const int32_t tiles = t < batch ? (packed ? (s_len[seq] + kTileM - 1) / kTileM : dense_tiles) : 0;
    int32_t all;
    s_first[t + 1] = block_scan(tiles, s_warp, all);
    if (t == 0) s_first[0] = 0;
    __syncthreads();
    for (int i = t; i < min(total_tiles, slots); i += kScanThreads) {
      int lo = 0, hi = batch - 1;  // the last rank whose first slot is at or before i and that has tiles
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_first[mid] <= i) lo = mid; else hi = mid - 1;
      }
      const int b = s_seq[lo];
      slot_info[i] = make_int4(b, tile_at(i - s_first[lo], s_first[lo + 1] - s_first[lo]) * kTileM, s_start[b], s_len[b]);
    }
  } else {
    int at = first;
    for (int b = b0; b < b1; ++b) {
      const int start = seq_info[2 * b], len = seq_info[2 * b + 1];
      const int tiles = packed ? (len + kTileM - 1) / kTileM : dense_tiles;
      for (int i = 0; i < tiles && at + i < slots; ++i) slot_info[at + i] = make_int4(b, i * kTileM, start, len);
      at += tiles;
    }
  }
  for (int i = total_tiles + t; i < slots; i += kScanThreads) slot_info[i] = make_int4(-1, 0, 0, 0);
  if (bad && status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(status), FDB_DEV_BAD_SEQLEN);
}

// One thread copies 16 bytes.  row_bytes is 128 (bf16) or 64 (e4m3).  Runs beside seq_info_kernel when launched behind it: neither
// reads what the other writes.
struct ExpandArgs {
  const uint4 *pos_key, *pos_query;
  uint4 *exp_key, *exp_query;
  const int16_t* lut;
  int lut_d_min, lut_len, d_first, rows, heads, vec_per_row;
  int64_t row_stride, head_stride;  // of the tables, in 16-byte units
};

__global__ void __launch_bounds__(256) expand_tables_kernel(ExpandArgs a) {
  ptx::grid_launch();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t total = (int64_t)a.heads * a.rows * a.vec_per_row;
  if (i < total) {
    const int c = (int)(i % a.vec_per_row);
    const int u = (int)((i / a.vec_per_row) % a.rows);
    const int h = (int)(i / ((int64_t)a.vec_per_row * a.rows));
    int li = a.d_first + u - a.lut_d_min;
    li = li < 0 ? 0 : (li >= a.lut_len ? a.lut_len - 1 : li);
    const int src = a.lut[li];
    const int64_t s = h * a.head_stride + src * a.row_stride + c;
    if (a.pos_key != nullptr) a.exp_key[i] = a.pos_key[s];
    if (a.pos_query != nullptr) a.exp_query[i] = a.pos_query[s];
  }
  ptx::grid_wait();  // behind seq_info_kernel: a kernel chained to this one may then rely on both
}

}  // namespace

AttnBuffers attn_buffers(const fdb_attn_params& p, const WorkspaceLayout& w) {
  char* ws = static_cast<char*>(p.workspace);
  AttnBuffers b;
  b.seq_info = reinterpret_cast<int32_t*>(ws + w.seq_info);
  b.tile_first = reinterpret_cast<int32_t*>(ws + w.tile_first);
  b.slot_info = reinterpret_cast<int32_t*>(ws + w.slot_info);
  b.exp_key = p.pos_key != nullptr ? ws + w.exp_key : nullptr;
  b.exp_query = p.pos_query != nullptr ? ws + w.exp_query : nullptr;
  b.part_o = w.split ? reinterpret_cast<float*>(ws + w.part_o) : nullptr;
  b.part_ml = w.split ? reinterpret_cast<float*>(ws + w.part_ml) : nullptr;
  b.split = w.split;
  return b;
}

int launch_seq_info(const fdb_attn_params& p, const AttnBuffers& b, void* stream) {
  seq_info_kernel<<<1, kScanThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      p.cu_seqlens, p.seq_lens, p.batch, p.max_seqlen, p.total_rows, b.seq_info, b.tile_first,
      reinterpret_cast<int4*>(b.slot_info), (int)tile_slots(p), p.status);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "seq_info launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

int launch_expand_tables(const fdb_attn_params& p, const ExpandGeometry& g, const AttnBuffers& b, void* stream, bool chained, TableStrides strides) {
  const int esz = p.dtype == FDB_E4M3 ? 1 : 2;
  ExpandArgs a;
  a.pos_key = static_cast<const uint4*>(p.pos_key);
  a.pos_query = static_cast<const uint4*>(p.pos_query);
  a.exp_key = static_cast<uint4*>(b.exp_key);
  a.exp_query = static_cast<uint4*>(b.exp_query);
  a.lut = p.bucket_lut; a.lut_d_min = p.lut_d_min; a.lut_len = p.lut_len;
  a.d_first = g.d_first; a.rows = g.rows; a.heads = p.heads;
  a.vec_per_row = kHeadDim * esz / 16;
  const int table_rows = 2 * (p.position_buckets > 0 ? p.position_buckets : p.max_relative_positions);
  a.row_stride = strides.row > 0 ? strides.row * esz / 16 : a.vec_per_row;
  a.head_stride = strides.row > 0 ? strides.head * esz / 16 : (int64_t)table_rows * a.vec_per_row;
  const int64_t total = (int64_t)p.heads * g.rows * a.vec_per_row;
  const cudaError_t e = launch_kernel<ExpandArgs>(expand_tables_kernel, a, dim3((unsigned)((total + 255) / 256)), 256, 0, chained,
                                                  static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "expand_tables launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

int launch_prepare(const fdb_attn_params& p, const ExpandGeometry& g, const AttnBuffers& b, void* stream, bool* launched, TableStrides strides) {
  int rc = FDB_OK;
  const bool schedule = (p.prepared & FDB_PREPARED_SCHEDULE) == 0;
  const bool tables = (p.pos_key != nullptr || p.pos_query != nullptr) && (p.prepared & FDB_PREPARED_TABLES) == 0;
  if (schedule) rc = launch_seq_info(p, b, stream);
  if (rc == FDB_OK && tables) rc = launch_expand_tables(p, g, b, stream, schedule, strides);
  *launched = schedule || tables;
  return rc;
}

}  // namespace fdb
