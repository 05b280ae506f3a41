// The encoder as one launch sequence (fdb_encoder_forward): mask analysis and packing on the device, embedding stage, and
// per layer the kernels of linear_sm100.cu, attn_fwd_sm100.cu and add_layernorm.cu on one stream.
//
// Module by module from Python a layer costs the host about 300 us (a dozen torch operators and this library's calls behind
// as many nn.Module calls), which is what bounds a forward of up to some 4000 tokens; from here a layer is seven launches.
// The number of valid tokens of a masked batch is not read back: the packing kernel leaves it in device memory, grids are
// sized for the padded batch and the kernels look the number up.
// Replaces the module walk of src/flashdeberta/model.py:275-310 and :418-496 of the reference (and its per-layer
// unpadding, :216-231).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <new>
#include <vector>

#include "encoder_small.h"
#include "internal.h"
#include "linear.h"
#include "sm100_ptx.cuh"

namespace fdb {
namespace {

struct LayerPlan {
  fdb_encoder_layer d;
  LinearWeight wq, wk, wv, wo, wi, wd;
};
constexpr int kMaxLayers = 4096;  // (a layer's plan is some 3 KB)
struct EncoderPlan {
  int hidden, heads, ffn;
  std::vector<LayerPlan> layers;
};

// ---------------------------------------------------------------------------------------------------------------------
// Mask -> packed rows.  A CTA takes 1024 tokens of one sequence; the valid tokens in front of it are counted by the same
// walk over the whole mask (small batches: one launch less) or come from pack_count_kernel.  Writes the token of every
// packed row, cu_seqlens and the number of rows, and zeros the output rows of invalid tokens.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kPackThreads = 256, kPackPer = 4, kPackChunk = kPackThreads * kPackPer;
constexpr int64_t kRecountTokens = 8192;  // up to here every CTA counts the tokens in front of it itself

__device__ __forceinline__ bool mask_valid(const void* mask, int type, int64_t i) {
  switch (type) {
    case kMaskF32: return static_cast<const float*>(mask)[i] != 0.f;
    case kMaskI64: return static_cast<const int64_t*>(mask)[i] != 0;
    case kMaskI32: return static_cast<const int32_t*>(mask)[i] != 0;
    case kMaskU8: return static_cast<const uint8_t*>(mask)[i] != 0;
    default: return (static_cast<const uint16_t*>(mask)[i] & 0x7fffu) != 0;
  }
}

__device__ __forceinline__ int block_sum(int v, int* s_warp) {  // every thread gets the sum over the CTA
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
  __syncthreads();
  int sum = 0;
#pragma unroll
  for (int w = 0; w < kPackThreads / 32; ++w) sum += s_warp[w];
  return sum;
}

__global__ void __launch_bounds__(kPackThreads) pack_count_kernel(const void* mask, int type, int seqlen, int chunks, int32_t* counts) {
  __shared__ int s_warp[kPackThreads / 32];
  ptx::grid_launch();
  ptx::grid_wait();
  const int b = blockIdx.x / chunks, c = blockIdx.x % chunks;
  int n = 0;
#pragma unroll
  for (int i = 0; i < kPackPer; ++i) {
    const int t = c * kPackChunk + i * kPackThreads + threadIdx.x;
    if (t < seqlen) n += mask_valid(mask, type, (int64_t)b * seqlen + t) ? 1 : 0;
  }
  n = block_sum(n, s_warp);
  if (threadIdx.x == 0) counts[blockIdx.x] = n;
}

__global__ void __launch_bounds__(kPackThreads) pack_kernel(const void* mask, int type, int batch, int seqlen, int chunks,
                                                            const int32_t* __restrict__ counts, int32_t* __restrict__ index,
                                                            int32_t* __restrict__ cu, int32_t* __restrict__ rows,
                                                            uint4* __restrict__ out, int vec_per_row) {
  __shared__ int s_warp[kPackThreads / 32];
  __shared__ int s_invalid[kPackChunk];
  __shared__ int s_n_invalid;
  ptx::grid_launch();
  ptx::grid_wait();
  const int b = blockIdx.x / chunks, c = blockIdx.x % chunks;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_n_invalid = 0;
  int n = 0;
  if (counts != nullptr) {
    for (int i = threadIdx.x; i < (int)blockIdx.x; i += kPackThreads) n += counts[i];
  } else {
    const int64_t before = (int64_t)b * seqlen + c * kPackChunk;
    for (int64_t i = threadIdx.x; i < before; i += kPackThreads) n += mask_valid(mask, type, i) ? 1 : 0;
  }
  const int base = block_sum(n, s_warp);
  // four consecutive tokens per thread, so that rows keep the tokens' order
  const int t0 = c * kPackChunk + threadIdx.x * kPackPer;
  bool valid[kPackPer];
  int mine = 0;
#pragma unroll
  for (int i = 0; i < kPackPer; ++i) {
    valid[i] = t0 + i < seqlen && mask_valid(mask, type, (int64_t)b * seqlen + t0 + i);
    mine += valid[i] ? 1 : 0;
    if (t0 + i < seqlen && !valid[i]) s_invalid[atomicAdd(&s_n_invalid, 1)] = t0 + i;
  }
  int inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += up;
  }
  __syncthreads();  // s_warp is free again
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  int at = base + inc - mine, total = 0;
#pragma unroll
  for (int w = 0; w < kPackThreads / 32; ++w) {
    if (w < warp) at += s_warp[w];
    total += s_warp[w];
  }
#pragma unroll
  for (int i = 0; i < kPackPer; ++i)
    if (valid[i]) index[at++] = b * seqlen + t0 + i;
  if (threadIdx.x == 0) {
    if (c == 0) cu[b] = base;
    if ((int)blockIdx.x == batch * chunks - 1) { cu[batch] = base + total; *rows = base + total; }
  }
  const int invalid = s_n_invalid;
  for (int i = warp; i < invalid; i += kPackThreads / 32) {
    uint4* o = out + ((int64_t)b * seqlen + s_invalid[i]) * vec_per_row;
    for (int v = lane; v < vec_per_row; v += 32) o[v] = make_uint4(0, 0, 0, 0);
  }
}

struct Layout {  // byte offsets into the workspace
  uint64_t counts, index, cu, rows, barrier, attn, x, h, qkv, ctx, proj, mid, total;
  WorkspaceLayout attn_layout;
};

uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }

fdb_attn_params attn_params(const fdb_encoder_call& c, const EncoderPlan& plan) {
  fdb_attn_params p = {};
  p.struct_bytes = sizeof(p);
  p.dtype = FDB_BF16;
  p.q_row_stride = p.k_row_stride = p.v_row_stride = p.out_row_stride = plan.hidden;
  p.q_head_stride = p.k_head_stride = p.v_head_stride = p.out_head_stride = kHeadDim;
  const fdb_encoder_layer& l0 = plan.layers[0].d;
  p.pos_key = l0.exp_key;      // only whether they are there counts: the gathered tables come with every layer
  p.pos_query = l0.exp_query;
  p.batch = c.batch;
  p.max_seqlen = c.max_seqlen;
  p.total_rows = c.total_rows;
  p.heads = plan.heads;
  p.head_dim = kHeadDim;
  p.position_buckets = c.position_buckets;
  p.max_relative_positions = c.max_relative_positions;
  p.bucket_lut = c.lut;
  p.lut_d_min = c.lut_d_min;
  p.lut_len = c.lut_len;
  p.sm_scale = c.sm_scale;
  p.status = c.status;
  return p;
}

SmallLayer small_layer(const fdb_encoder_layer& d) {
  auto p = [](const void* x) { return static_cast<const __nv_bfloat16*>(x); };
  return {p(d.wq), p(d.bq), p(d.wk), p(d.bk), p(d.wv), p(d.bv), p(d.wo), p(d.bo), p(d.ln1_gamma), p(d.ln1_beta), p(d.wi), p(d.bi),
          p(d.wd), p(d.bd), p(d.ln2_gamma), p(d.ln2_beta), p(d.exp_key), p(d.exp_query), d.ln1_eps, d.ln2_eps};
}

Layout layout_of(const fdb_encoder_call& c, const EncoderPlan& plan, const fdb_attn_params& p) {
  Layout l;
  const uint64_t rows = (uint64_t)c.total_rows, h = (uint64_t)plan.hidden * 2;
  const uint64_t chunks = (uint64_t)((c.max_seqlen + kPackChunk - 1) / kPackChunk) * c.batch;
  uint64_t off = 0;
  l.counts = off; off = align256(off + chunks * 4);
  l.index = off;  off = align256(off + (c.mask ? rows * 4 : 0));
  l.cu = off;     off = align256(off + (uint64_t)(c.batch + 1) * 4);
  l.rows = off;   off = align256(off + 4);
  l.barrier = off; off = align256(off + 8);
  fdb_attn_params q = p;
  q.pos_key = q.pos_query = nullptr;  // no room for gathered tables: they are the plan's
  ExpandGeometry none = {0, 0, 0, 0};
  l.attn_layout = workspace_layout(q, none, false);
  // the partial results of a call in two launches
  l.attn_layout.split = want_split(p);
  const uint64_t cells = l.attn_layout.split ? rows * plan.heads : 0;
  l.attn_layout.part_o = l.attn_layout.total;
  l.attn_layout.part_ml = align256(l.attn_layout.part_o + cells * kHeadDim * sizeof(float));
  l.attn = off;
  off = align256(off + l.attn_layout.part_ml + cells * 2 * sizeof(float));
  l.x = off;    off = align256(off + rows * h);
  l.h = off;    off = align256(off + rows * h);
  l.qkv = off;  off = align256(off + 3 * rows * h);
  l.ctx = off;  off = align256(off + rows * h);
  l.proj = off; off = align256(off + rows * h);
  l.mid = off;  off = align256(off + rows * (uint64_t)plan.ffn * 2);
  l.total = off;
  return l;
}

int check_call(const fdb_encoder_call* c) {
  if (c == nullptr || c->struct_bytes != sizeof(fdb_encoder_call))
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: NULL or struct_bytes %u != %zu", c ? c->struct_bytes : 0u, sizeof(fdb_encoder_call));
  if (c->plan == nullptr || c->ids == nullptr || c->emb_table == nullptr || c->emb_gamma == nullptr || c->emb_beta == nullptr || c->out == nullptr)
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: plan, ids, embedding stage and out are required");
  if (c->batch < 0 || c->max_seqlen < 0 || c->total_rows < 0 || c->emb_rows <= 0)
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: negative size");
  if (c->cu_seqlens != nullptr && c->mask != nullptr) return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: give a mask or cu_seqlens, not both");
  if (c->cu_seqlens == nullptr && (int64_t)c->batch * c->max_seqlen != c->total_rows)
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: dense ids need total_rows == batch * max_seqlen");
  if (c->mask_type < FDB_MASK_F32 || c->mask_type > FDB_MASK_BF16) return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_call: unknown mask_type %d", c->mask_type);
  const unsigned mask_bytes[] = {4, 8, 4, 1, 2};  // of FDB_MASK_*
  if (!aligned_to(16, c->out, c->emb_table, c->emb_gamma, c->emb_beta) || !aligned_to(8, c->ids) || !aligned_to(4, c->cu_seqlens, c->status) ||
      !aligned_to(2, c->lut) || !aligned_to(mask_bytes[c->mask_type], c->mask))
    return fail(FDB_ERR_ALIGNMENT, "fdb_encoder_call: out and the embedding stage must be 16-byte aligned, the others to their elements");
  if ((int64_t)c->total_rows > (int64_t(1) << 31) - 256) return fail(FDB_ERR_LIMIT, "fdb_encoder_call: total_rows");
  return FDB_OK;
}

}  // namespace
}  // namespace fdb

using namespace fdb;

extern "C" FDB_API int32_t fdb_expanded_rows(int32_t lut_d_min, int32_t lut_len) { return expand_geometry(lut_d_min, lut_len).rows; }

extern "C" FDB_API int fdb_expand_tables(const void* pos_key, const void* pos_query, void* exp_key, void* exp_query, int32_t heads,
                                         int32_t table_rows, const int16_t* lut, int32_t lut_d_min, int32_t lut_len, void* stream) {
  clear_error();
  if ((pos_key != nullptr) != (exp_key != nullptr) || (pos_query != nullptr) != (exp_query != nullptr) || lut == nullptr || lut_len < 2 ||
      heads <= 0 || table_rows <= 0 || table_rows % 2 != 0)
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_expand_tables: bad argument");
  if (!aligned_to(16, pos_key, pos_query, exp_key, exp_query) || !aligned_to(2, lut))
    return fail(FDB_ERR_ALIGNMENT, "fdb_expand_tables: tables must be 16-byte aligned");
  if (pos_key == nullptr && pos_query == nullptr) return FDB_OK;
  fdb_attn_params p = {};
  p.dtype = FDB_BF16;
  p.pos_key = pos_key; p.pos_query = pos_query;
  p.heads = heads; p.position_buckets = table_rows / 2;
  p.bucket_lut = lut; p.lut_d_min = lut_d_min; p.lut_len = lut_len;
  AttnBuffers b = {};
  b.exp_key = exp_key; b.exp_query = exp_query;
  return launch_expand_tables(p, expand_geometry(lut_d_min, lut_len), b, stream);
}

extern "C" FDB_API int fdb_encoder_create(const fdb_encoder_layer* layers, int32_t n_layers, int32_t hidden, int32_t heads,
                                          int32_t ffn, void** plan) {
  clear_error();
  if (layers == nullptr || plan == nullptr || n_layers <= 0) return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_create: bad argument");
  if (heads <= 0 || hidden != heads * kHeadDim || hidden % 256 != 0 || hidden > 2048 || ffn <= 0 || ffn % 64 != 0)
    return fail(FDB_ERR_UNSUPPORTED, "fdb_encoder_create: hidden %d, heads %d, ffn %d", hidden, heads, ffn);
  if (n_layers > kMaxLayers) return fail(FDB_ERR_LIMIT, "fdb_encoder_create: %d layers (at most %d)", n_layers, kMaxLayers);
  EncoderPlan* e = new (std::nothrow) EncoderPlan;
  if (e == nullptr) return fail(FDB_ERR_LIMIT, "fdb_encoder_create: out of host memory");
  e->hidden = hidden; e->heads = heads; e->ffn = ffn;
  try {  // (no exception leaves a C entry)
    e->layers.resize(n_layers);
  } catch (const std::bad_alloc&) {
    delete e;
    return fail(FDB_ERR_LIMIT, "fdb_encoder_create: out of host memory");
  }
  int rc = FDB_OK;
  for (int i = 0; i < n_layers && rc == FDB_OK; ++i) {
    LayerPlan& l = e->layers[i];
    l.d = layers[i];
    const fdb_encoder_layer& d = l.d;
    if (!d.wq || !d.wk || !d.wv || !d.wo || !d.wi || !d.wd || !d.ln1_gamma || !d.ln1_beta || !d.ln2_gamma || !d.ln2_beta) {
      rc = fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_create: layer %d has a NULL weight", i);
      break;
    }
    const uintptr_t all = (uintptr_t)d.wq | (uintptr_t)d.bq | (uintptr_t)d.wk | (uintptr_t)d.bk | (uintptr_t)d.wv | (uintptr_t)d.bv |
                          (uintptr_t)d.wo | (uintptr_t)d.bo | (uintptr_t)d.wi | (uintptr_t)d.bi | (uintptr_t)d.wd | (uintptr_t)d.bd |
                          (uintptr_t)d.exp_key | (uintptr_t)d.exp_query | (uintptr_t)d.ln1_gamma | (uintptr_t)d.ln1_beta |
                          (uintptr_t)d.ln2_gamma | (uintptr_t)d.ln2_beta;
    if ((all & 15u) != 0) { rc = fail(FDB_ERR_ALIGNMENT, "fdb_encoder_create: layer %d has a pointer that is not 16-byte aligned", i); break; }
    struct { LinearWeight* w; const void* p; int n, k; } maps[6] = {
        {&l.wq, d.wq, hidden, hidden}, {&l.wk, d.wk, hidden, hidden}, {&l.wv, d.wv, hidden, hidden},
        {&l.wo, d.wo, hidden, hidden}, {&l.wi, d.wi, ffn, hidden}, {&l.wd, d.wd, hidden, ffn}};
    for (auto& m : maps)
      if ((rc = make_linear_maps(m.w, m.p, m.n, m.k)) != FDB_OK) break;
  }
  if (rc != FDB_OK) { delete e; return rc; }
  *plan = e;
  return FDB_OK;
}

extern "C" FDB_API void fdb_encoder_destroy(void* plan) { delete static_cast<EncoderPlan*>(plan); }

extern "C" FDB_API uint64_t fdb_encoder_workspace_bytes(const fdb_encoder_call* c) {
  clear_error();
  if (check_call(c) != FDB_OK) return 0;
  const EncoderPlan& plan = *static_cast<const EncoderPlan*>(c->plan);
  return layout_of(*c, plan, attn_params(*c, plan)).total;
}

extern "C" FDB_API int fdb_encoder_forward(fdb_encoder_call* c, void* stream) {
  clear_error();
  int rc = check_call(c);
  if (rc != FDB_OK) return rc;
  c->launches = 0;
  if (c->batch == 0 || c->total_rows == 0) return FDB_OK;
  const EncoderPlan& plan = *static_cast<const EncoderPlan*>(c->plan);
  ExpandGeometry g = {0, 0, 0, 0};
  const bool pos = plan.layers[0].d.exp_key != nullptr || plan.layers[0].d.exp_query != nullptr;
  if (pos && (c->lut == nullptr || c->lut_len < 2)) return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_encoder_forward: position tables without a bucket table");
  if (pos) g = expand_geometry(c->lut_d_min, c->lut_len);
  fdb_attn_params p = attn_params(*c, plan);
  const Layout l = layout_of(*c, plan, p);
  if (c->workspace == nullptr || c->workspace_bytes < l.total)
    return fail(FDB_ERR_WORKSPACE, "workspace of %llu bytes needed, %llu given", (unsigned long long)l.total, (unsigned long long)c->workspace_bytes);
  if ((reinterpret_cast<uintptr_t>(c->workspace) & 255u) != 0) return fail(FDB_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(c->workspace);
  const int64_t rows = c->total_rows;
  int launches = 0;
  // A handful of rows: the layers are one kernel.  (Timing events around the attention of every layer need launches of their own.)
  const bool small = c->attn_events == nullptr && small_encoder_covers(rows, plan.hidden, plan.ffn, (int)plan.layers.size());
  if (small) {
    const cudaError_t e = cudaMemsetAsync(ws + l.barrier, 0, 8, s);
    if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "encoder memset: %s", cudaGetErrorString(e));
  }

  // ---- which rows there are -------------------------------------------------------------------------------------------
  const int32_t *index = nullptr, *rows_dev = nullptr;
  p.cu_seqlens = c->cu_seqlens;
  if (c->mask != nullptr) {
    const int chunks = (c->max_seqlen + kPackChunk - 1) / kPackChunk;
    int32_t* counts = rows > kRecountTokens ? reinterpret_cast<int32_t*>(ws + l.counts) : nullptr;
    if (counts != nullptr) {
      pack_count_kernel<<<(unsigned)(c->batch * chunks), kPackThreads, 0, s>>>(c->mask, c->mask_type, c->max_seqlen, chunks, counts);
      ++launches;
    }
    pack_kernel<<<(unsigned)(c->batch * chunks), kPackThreads, 0, s>>>(
        c->mask, c->mask_type, c->batch, c->max_seqlen, chunks, counts, reinterpret_cast<int32_t*>(ws + l.index),
        reinterpret_cast<int32_t*>(ws + l.cu), reinterpret_cast<int32_t*>(ws + l.rows), static_cast<uint4*>(c->out), plan.hidden / 8);
    ++launches;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "pack launch: %s", cudaGetErrorString(e));
    index = reinterpret_cast<const int32_t*>(ws + l.index);
    rows_dev = reinterpret_cast<const int32_t*>(ws + l.rows);
    p.cu_seqlens = reinterpret_cast<const int32_t*>(ws + l.cu);
  }
  p.workspace = ws + l.attn;
  AttnBuffers b = attn_buffers(p, l.attn_layout);
  if (!small) {
    if ((rc = launch_seq_info(p, b, stream)) != FDB_OK) return rc;
    ++launches;
  }

  // ---- embedding stage --------------------------------------------------------------------------------------------------
  LayerNormCall ln = {};
  ln.x = c->emb_table; ln.gamma = c->emb_gamma; ln.beta = c->emb_beta; ln.out = ws + l.x;
  ln.rows = rows; ln.rows_dev = rows_dev; ln.hidden = plan.hidden; ln.eps = c->emb_eps;
  ln.ids = c->ids; ln.table_rows = c->emb_rows; ln.token_index = index;
  ln.mask = c->mask; ln.mask_type = c->mask_type; ln.status = c->status; ln.chained = true;
  // the last key tile of the last sequence reads values behind the valid rows, which have to be finite
  if (rows_dev != nullptr) ln.zero_tail = ws + l.qkv + 2 * (uint64_t)rows * plan.hidden * 2;
  if ((rc = launch_layernorm(ln, stream)) != FDB_OK) return rc;
  ++launches;

  if (small) {
    SmallEncoderArgs a;
    a.n_layers = (int)plan.layers.size();
    for (int i = 0; i < a.n_layers; ++i) a.layer[i] = small_layer(plan.layers[i].d);
    a.hidden = plan.hidden; a.ffn = plan.ffn;
    a.row_bound = (int)rows; a.rows_dev = rows_dev;
    a.cu_seqlens = p.cu_seqlens; a.batch = c->batch; a.max_seqlen = c->max_seqlen;
    a.xrows = g.rows; a.d_first = g.d_first;
    a.sm_scale = c->sm_scale;
    auto at = [&](uint64_t offset) { return reinterpret_cast<__nv_bfloat16*>(ws + offset); };
    a.x = at(l.x); a.qkv = at(l.qkv); a.ctx = at(l.ctx); a.y = at(l.proj); a.mid = at(l.mid);
    a.out = static_cast<__nv_bfloat16*>(c->out); a.out_index = index;
    a.barrier = reinterpret_cast<uint32_t*>(ws + l.barrier);
    a.status = c->status;
    if ((rc = launch_small_encoder(a, stream)) != FDB_OK) return rc;
    c->launches = launches + 1;
    return FDB_OK;
  }

  // ---- layers -------------------------------------------------------------------------------------------------------------
  CUtensorMap map_x, map_ctx, map_h, map_mid;
  if ((rc = make_linear_input_map(&map_x, ws + l.x, rows, plan.hidden)) != FDB_OK) return rc;
  if ((rc = make_linear_input_map(&map_ctx, ws + l.ctx, rows, plan.hidden)) != FDB_OK) return rc;
  if ((rc = make_linear_input_map(&map_h, ws + l.h, rows, plan.hidden)) != FDB_OK) return rc;
  if ((rc = make_linear_input_map(&map_mid, ws + l.mid, rows, plan.ffn)) != FDB_OK) return rc;
  char* qkv[3];
  for (int i = 0; i < 3; ++i) qkv[i] = ws + l.qkv + (uint64_t)i * rows * plan.hidden * 2;
  p.q = qkv[0]; p.k = qkv[1]; p.v = qkv[2]; p.out = ws + l.ctx;
  const int n_layers = (int)plan.layers.size();
  for (int i = 0; i < n_layers; ++i) {
    const LayerPlan& lp = plan.layers[i];
    LinearCall lin = {};
    lin.rows = rows; lin.rows_dev = rows_dev; lin.chained = true; lin.status = c->status;
    // query, key and value projections
    lin.x_map = &map_x; lin.k = plan.hidden; lin.n = plan.hidden; lin.out_stride = plan.hidden; lin.groups = 3;
    lin.weight[0] = &lp.wq; lin.weight[1] = &lp.wk; lin.weight[2] = &lp.wv;
    lin.bias[0] = lp.d.bq; lin.bias[1] = lp.d.bk; lin.bias[2] = lp.d.bv;
    for (int k = 0; k < 3; ++k) lin.out[k] = qkv[k];
    if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
    // attention
    b.exp_key = const_cast<void*>(lp.d.exp_key);
    b.exp_query = const_cast<void*>(lp.d.exp_query);
    if (c->attn_events != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(c->attn_events[2 * i]), s);
    if ((rc = launch_attn_fwd_sm100(p, g, b, stream, true)) != FDB_OK) return rc;
    if (c->attn_events != nullptr) cudaEventRecord(static_cast<cudaEvent_t>(c->attn_events[2 * i + 1]), s);
    // output block
    lin.groups = 1;
    lin.x_map = &map_ctx; lin.weight[0] = &lp.wo; lin.bias[0] = lp.d.bo; lin.out[0] = ws + l.proj;
    if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
    LayerNormCall n1 = {};
    n1.x = ws + l.proj; n1.residual = ws + l.x; n1.gamma = lp.d.ln1_gamma; n1.beta = lp.d.ln1_beta; n1.out = ws + l.h;
    n1.rows = rows; n1.rows_dev = rows_dev; n1.hidden = plan.hidden; n1.eps = lp.d.ln1_eps; n1.chained = true;
    if ((rc = launch_layernorm(n1, stream)) != FDB_OK) return rc;
    // feed-forward block
    lin.x_map = &map_h; lin.n = plan.ffn; lin.out_stride = plan.ffn; lin.gelu = true;
    lin.weight[0] = &lp.wi; lin.bias[0] = lp.d.bi; lin.out[0] = ws + l.mid;
    if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
    lin.x_map = &map_mid; lin.k = plan.ffn; lin.n = plan.hidden; lin.out_stride = plan.hidden; lin.gelu = false;
    lin.weight[0] = &lp.wd; lin.bias[0] = lp.d.bd; lin.out[0] = ws + l.proj;
    if ((rc = launch_linear(lin, stream)) != FDB_OK) return rc;
    LayerNormCall n2 = n1;
    n2.residual = ws + l.h; n2.gamma = lp.d.ln2_gamma; n2.beta = lp.d.ln2_beta; n2.eps = lp.d.ln2_eps;
    n2.out = ws + l.x;
    if (i == n_layers - 1) { n2.out = c->out; n2.out_index = index; }
    if ((rc = launch_layernorm(n2, stream)) != FDB_OK) return rc;
    launches += 7 + (b.split ? 1 : 0);
  }
  c->launches = launches;
  return FDB_OK;
}
