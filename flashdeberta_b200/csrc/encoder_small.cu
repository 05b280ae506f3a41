// The whole encoder stack in one kernel for a handful of tokens (a query, a short sentence): at most 64 rows.
//
// At that size a layer's seven launches are all latency: 4 to 10 us each for a microsecond of work, one behind the other.  Here one
// CTA per SM stays for the whole forward and the steps of a layer are separated by grid barriers:
//   1  LayerNorm of the layer before -> shared memory; query, key and value projections
//   2  attention, four warps per (row, head), on the CUDA cores
//   3  output projection, + residual
//   4  LayerNorm -> shared memory; first feed-forward product, GELU
//   5  second feed-forward product, + residual
// Every CTA normalises all rows for itself (the next product needs them all) and keeps them, so the residuals of steps 3 and 5 come from
// shared memory too.  A product's columns are dealt over the CTAs in tiles of 8, its K over the warps; the warps' partial sums
// meet in shared memory.  What bounds a step is latency (barrier, one trip to L2 for the rows, one for the weights, which are
// fetched to L2 ahead of the barrier): with 16 to 64 rows there is nothing to fill tcgen05 tiles of 128 rows with, and fragments
// that go from memory to registers save the trip through shared memory and tensor memory, so the products are warp MMAs.  Both
// operands are read 32 bytes per thread: K is permuted the same way in both, which a sum over K does not see.
//
// 12 layers of 768, 29 tokens: 610 us a call as 84 launches, 320 in one kernel.  Of a layer (45 000 clocks): five barriers 13 700, the
// two LayerNorms 8000, the four products 3800 to 7600 each, attention 4000.  It was 391 us (55 300) with a warp for a (row, head) in the
// attention (6500 clocks), LayerNorms that asked at run time how long a row is (6000 each), integer divisions in the products' last
// step and loads of the fifth step that came a half block at a time (8750).  Weights ahead of the barrier by a bulk prefetch or not at
// all made no difference; scale and shift prefetched to the first-level cache cost 130 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "encoder_small.h"
#include "gelu.cuh"
#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"

namespace fdb {
namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kMaxTiles = 4;  // 8-column tiles of one product per CTA

struct Ctx {
  const SmallEncoderArgs* a;
  uint8_t* s_x;        // rows of hidden bf16 + 16 bytes: with 32 bytes per thread, eight threads read all banks
  float* s_red;
  int rows, pitch, tid, warp, lane;
};

__device__ __forceinline__ float lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// All CTAs' writes before it are visible after it.  Bounded: after about two seconds of SM clock, or once another CTA has given up,
// every CTA returns.
__device__ __forceinline__ bool grid_barrier(const SmallEncoderArgs& a, uint32_t* s_ok, uint32_t target) {
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t ok = 1;
    __threadfence();
    atomicAdd(a.barrier, 1u);
    const long long t0 = clock64();
    uint32_t seen = 0;
    for (uint32_t i = 0; i < (1u << 30); ++i) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.barrier) : "memory");
      if (seen >= target) break;
      if ((i & 63u) == 63u && (clock64() - t0 > 4000000000LL || *reinterpret_cast<volatile uint32_t*>(a.barrier + 1) != 0u)) break;
    }
    if (seen < target) {
      ok = 0;
      atomicExch(a.barrier + 1, 1u);
      if (a.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(a.status), FDB_DEV_TIMEOUT);
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// One product out[rows][n] = x . w^T over K = k; this CTA's tiles of 8 columns are [tile0, tile0 + tiles).
struct Product {
  const __nv_bfloat16 *w0, *w1, *w2;   // (group columns, k) each; group g holds columns g * group_cols ...
  const __nv_bfloat16 *b0, *b1, *b2;
  int group_cols, k, tile0, tiles;
};

__device__ __forceinline__ Product make_product(const Ctx& c, const __nv_bfloat16* w0, const __nv_bfloat16* w1, const __nv_bfloat16* w2,
                                                const __nv_bfloat16* b0, const __nv_bfloat16* b1, const __nv_bfloat16* b2, int group_cols,
                                                int groups, int k) {
  Product p = {w0, w1, w2, b0, b1, b2, group_cols, k, 0, 0};
  const int all = group_cols * groups / 8, per = (all + (int)gridDim.x - 1) / (int)gridDim.x;
  p.tile0 = blockIdx.x * per;
  p.tiles = max(0, min(per, all - p.tile0));
  return p;
}
__device__ __forceinline__ int group_of(const Product& p, int col) { return (col >= p.group_cols ? 1 : 0) + (col >= 2 * p.group_cols ? 1 : 0); }
__device__ __forceinline__ const __nv_bfloat16* weight_row(const Product& p, int tile, int r) {
  const int col = tile * 8, g = group_of(p, col);
  return (g == 0 ? p.w0 : (g == 1 ? p.w1 : p.w2)) + (int64_t)(col - g * p.group_cols + r) * p.k;
}
// the CTA's weights of a coming product to L2
__device__ __forceinline__ void prefetch(const Ctx& c, const Product& p) {
  const int lines = p.k / 64;
  for (int i = c.tid; i < p.tiles * 8 * lines; i += kThreads) {
    const int row = i / lines;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(weight_row(p, p.tile0 + (row >> 3), row & 7) + (i - row * lines) * 64));
  }
}

// Partial sums of the warps over their share of K, then `store(row, column, v0, v1)` for pairs of columns with the bias added.  The
// rows come from shared memory, or (kInMemory) from `src`.
template <int MT, int NT, int kSplit, bool kInMemory, typename Store>
__device__ __forceinline__ void product_tiles(const Ctx& c, const Product& p, const __nv_bfloat16* src, Store&& store) {
  const int g = c.lane >> 2, t = c.lane & 3;
  constexpr int kgs = kWarps / kSplit, cols = NT * kSplit * 8;  // kSplit: the tiles are dealt to this many sets of warps
  const int kg = c.warp % kgs, tile = (c.warp / kgs) * NT;
  const int blocks = p.k / 64;
  // the bias of the pair of columns that this thread finishes first, on its way while the product is made
  auto bias_of = [&](int cp) -> uint32_t {
    const int col = p.tile0 * 8 + cp, grp = group_of(p, col);
    const __nv_bfloat16* bias = grp == 0 ? p.b0 : (grp == 1 ? p.b1 : p.b2);
    return bias != nullptr ? __ldg(reinterpret_cast<const uint32_t*>(bias + col - grp * p.group_cols)) : 0u;
  };
  const uint32_t first_bias = bias_of(c.tid % (cols / 2) * 2);
  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
  // of each 64 of K, thread t of a fragment's row has the 16 values from 16 t on: four steps of the MMA
  const __nv_bfloat16* w[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) w[n] = weight_row(p, p.tile0 + min(tile + n, p.tiles - 1), g) + t * 16;
  // A batch of steps (half a block each) at a time: all its loads, then its MMAs.  With the rows in memory the batch is what the
  // registers hold, for it is a trip to L2 each; in shared memory, a warp's one block of the weights.
  constexpr int kBatch = kInMemory ? (MT == 1 ? 4 : (MT == 2 ? 3 : 1)) : 2;
  const int steps = kg < blocks ? 2 * ((blocks - kg - 1) / kgs + 1) : 0;
#pragma unroll 1
  for (int s0 = 0; s0 < steps; s0 += kBatch) {
    uint4 x[kBatch][MT][2], y[kBatch][NT];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int at = (kg + ((s0 + j) >> 1) * kgs) * 64 + ((s0 + j) & 1) * 8;
      const bool live = kBatch <= 2 || s0 + j < steps;  // (the number of steps is even)
#pragma unroll
      for (int n = 0; n < NT; ++n) y[j][n] = live ? __ldg(reinterpret_cast<const uint4*>(w[n] + at)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = m * 16 + h * 8 + g;
          if constexpr (kInMemory) x[j][m][h] = live && row < c.rows ? __ldcg(reinterpret_cast<const uint4*>(src + (int64_t)row * p.k + at + t * 16)) : make_uint4(0, 0, 0, 0);
          else x[j][m][h] = *reinterpret_cast<const uint4*>(c.s_x + row * c.pitch + (at + t * 16) * 2);
        }
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          mma16816(acc[m][n], x[j][m][0].x, x[j][m][1].x, x[j][m][0].y, x[j][m][1].y, y[j][n].x, y[j][n].y);
          mma16816(acc[m][n], x[j][m][0].z, x[j][m][1].z, x[j][m][0].w, x[j][m][1].w, y[j][n].z, y[j][n].w);
        }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
      if (tile + n < p.tiles) {
        float* at = c.s_red + ((int64_t)(kg * MT * 16 + m * 16 + g)) * cols + (tile + n) * 8 + 2 * t;
        *reinterpret_cast<float2*>(at) = make_float2(acc[m][n][0], acc[m][n][1]);
        *reinterpret_cast<float2*>(at + 8 * cols) = make_float2(acc[m][n][2], acc[m][n][3]);
      }
  __syncthreads();
  for (int i = c.tid; i < c.rows * (cols / 2); i += kThreads) {
    const int row = i / (cols / 2), cp = (i - row * (cols / 2)) * 2;
    float2 s = make_float2(0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < kgs; ++k) {
      const float2 v = *reinterpret_cast<const float2*>(c.s_red + (int64_t)(k * MT * 16 + row) * cols + cp);
      s.x += v.x;
      s.y += v.y;
    }
    const uint32_t bias = i < kThreads ? first_bias : bias_of(cp);
    const int col = p.tile0 * 8 + cp, grp = group_of(p, col), in = col - grp * p.group_cols;
    store(row, grp, in, round_bf16(s.x + lo(bias)), round_bf16(s.y + hi(bias)));
  }
}

template <int MT, bool kInMemory, typename Store>
__device__ __forceinline__ void product(const Ctx& c, const Product& p, const __nv_bfloat16* src, Store&& store) {
  if (p.tiles == 0) return;  // (uniform over the CTA)
  if (p.tiles == 1) product_tiles<MT, 1, 1, kInMemory>(c, p, src, store);
  else if (p.tiles == 2) product_tiles<MT, 2, 1, kInMemory>(c, p, src, store);
  else if (p.tiles == 3) product_tiles<MT, 3, 1, kInMemory>(c, p, src, store);
  else product_tiles<MT, 2, 2, kInMemory>(c, p, src, store);  // (four: the partial sums of 16 warps would not fit)
}

// a bf16 pair as two floats
__device__ __forceinline__ uint64_t wide(uint32_t w) { return ptx::pack_f32x2(lo(w), hi(w)); }
__device__ __forceinline__ uint64_t both(float v) { return ptx::pack_f32x2(v, v); }
__device__ __forceinline__ float across(uint64_t v) {
  float a, b;
  ptx::unpack_f32x2(v, a, b);
  return a + b;
}

// LayerNorm of the rows of `y` (the sums of add_layernorm.cu, two at a time), two rows of a warp together; gamma == NULL: the rows as
// they are.  With all rows on every CTA this is bound by instructions, not by memory.
template <int kVec, typename Out>
__device__ __forceinline__ void normalise_rows(const Ctx& c, const __nv_bfloat16* y, const __nv_bfloat16* gamma, const __nv_bfloat16* beta, float eps,
                                          int first, int step, Out&& out) {
  const float inv = 1.f / (float)c.a->hidden;
#pragma unroll 1
  for (int row = first; row < c.rows; row += 2 * step) {
    uint4 raw[2][kVec];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < kVec; ++i)
        raw[r][i] = __ldcg(reinterpret_cast<const uint4*>(y + (int64_t)min(row + r * step, c.rows - 1) * c.a->hidden) + i * 32 + c.lane);
    if (gamma != nullptr) {
      uint64_t d[2][4 * kVec];
      float mean[2], rstd[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint64_t sum = both(0.f);
#pragma unroll
        for (int i = 0; i < kVec; ++i) {
          const uint32_t w[4] = {raw[r][i].x, raw[r][i].y, raw[r][i].z, raw[r][i].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) sum = ptx::add_f32x2(sum, d[r][i * 4 + k] = wide(w[k]));
        }
        mean[r] = across(sum);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 2; ++r) mean[r] += __shfl_xor_sync(0xffffffffu, mean[r], o);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint64_t m = both(-mean[r] * inv);
        uint64_t sq = both(0.f);
#pragma unroll
        for (int i = 0; i < 4 * kVec; ++i) {
          d[r][i] = ptx::add_f32x2(d[r][i], m);
          sq = ptx::fma_f32x2(d[r][i], d[r][i], sq);
        }
        rstd[r] = across(sq);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 2; ++r) rstd[r] += __shfl_xor_sync(0xffffffffu, rstd[r], o);
#pragma unroll
      for (int r = 0; r < 2; ++r) rstd[r] = rsqrtf(rstd[r] * inv + eps);
#pragma unroll
      for (int i = 0; i < kVec; ++i) {
        const uint4 gv = __ldg(reinterpret_cast<const uint4*>(gamma) + i * 32 + c.lane), bv = __ldg(reinterpret_cast<const uint4*>(beta) + i * 32 + c.lane);
        const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w}, bw[4] = {bv.x, bv.y, bv.z, bv.w};
        uint32_t o[2][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float v0, v1;
            ptx::unpack_f32x2(ptx::fma_f32x2(ptx::mul_f32x2(d[r][i * 4 + k], both(rstd[r])), wide(gw[k]), wide(bw[k])), v0, v1);
            o[r][k] = ptx::pack_bf16x2(v0, v1);
          }
#pragma unroll
        for (int r = 0; r < 2; ++r) raw[r][i] = make_uint4(o[r][0], o[r][1], o[r][2], o[r][3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int i = 0; i < kVec; ++i)
        if (row + r * step < c.rows) out(row + r * step, i * 32 + c.lane, raw[r][i]);
  }
}
// (with the length of a row known at compile time: a branch per 16 bytes kept the rows' arithmetic apart, 6000 against 4000 clocks for 29 rows)
template <typename Out>
__device__ __forceinline__ void normalise(const Ctx& c, const __nv_bfloat16* y, const __nv_bfloat16* gamma, const __nv_bfloat16* beta, float eps,
                                          int first, int step, Out&& out) {
  switch (c.a->hidden / 256) {
    case 1: normalise_rows<1>(c, y, gamma, beta, eps, first, step, out); break;
    case 2: normalise_rows<2>(c, y, gamma, beta, eps, first, step, out); break;
    case 3: normalise_rows<3>(c, y, gamma, beta, eps, first, step, out); break;
    default: normalise_rows<4>(c, y, gamma, beta, eps, first, step, out); break;
  }
}

// softmax((q.k + c2p + p2c) * scale) v of one row and head by four warps (a head of 29 rows leaves a CTA two or three of these to do, and
// one warp alone is a chain of latencies: 6500 clocks against 4000).  Scores: warp w has keys 8w .. 8w+7 (and 32 more), four lanes a
// key, 16 features each.  Output: warp w has features 16w .. 16w+15, a lane a pair of them over every fourth key.  `scores`: 64
// floats that the last row but one of these warps used.
__device__ __forceinline__ void attention_row(const Ctx& c, const SmallLayer& l, int row, int head, int start, int len, float* scores) {
  const SmallEncoderArgs& a = *c.a;
  const int w = c.warp & 3;
  const int64_t hd = (int64_t)head * 64;
  uint32_t* out = reinterpret_cast<uint32_t*>(a.ctx + (int64_t)row * a.hidden + hd) + w * 8 + (c.lane & 7);
  if (len == 0) {  // a row of no sequence
    if (c.lane < 8) *out = 0u;
    return;
  }
  const int64_t plane = (int64_t)a.row_bound * a.hidden;
  const __nv_bfloat16 *q = a.qkv, *k = a.qkv + plane, *v = a.qkv + 2 * plane;
  const int sub = c.lane >> 3;
  const uint32_t* vr = reinterpret_cast<const uint32_t*>(v + (int64_t)start * a.hidden + hd) + w * 8 + (c.lane & 7);
  uint32_t vw[8];  // keys sub, sub + 4, .. of the first 32, on their way beside the scores
#pragma unroll
  for (int i = 0; i < 8; ++i) vw[i] = sub + 4 * i < len ? __ldcg(vr + (int64_t)(sub + 4 * i) * (a.hidden / 2)) : 0u;
  const int m = row - start, part = (c.lane & 3) * 2;  // 16-byte pieces of the row
  const uint4* qr = reinterpret_cast<const uint4*>(q + (int64_t)row * a.hidden + hd) + part;
#pragma unroll 1
  for (int n = w * 8 + (c.lane >> 2); n - (c.lane >> 2) < 64 && (n & 32 ? len > 32 : true); n += 32) {
    const int key = min(n, len - 1);
    const uint4* kr = reinterpret_cast<const uint4*>(k + (int64_t)(start + key) * a.hidden + hd) + part;
    const int64_t at = ((int64_t)head * a.xrows + (m - key - a.d_first)) * 64;
    const uint4* xk = reinterpret_cast<const uint4*>(l.exp_key + at) + part;
    const uint4* xq = reinterpret_cast<const uint4*>(l.exp_query + at) + part;
    uint4 qv[2], kv[2], kp[2], qp[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      qv[i] = __ldcg(qr + i);
      kv[i] = __ldcg(kr + i);
      kp[i] = l.exp_key != nullptr ? __ldg(xk + i) : make_uint4(0, 0, 0, 0);
      qp[i] = l.exp_query != nullptr ? __ldg(xq + i) : make_uint4(0, 0, 0, 0);
    }
    uint64_t sum_q = both(0.f), sum_k = both(0.f);  // q . (k + pos_key), k . pos_query
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t qw[4] = {qv[i].x, qv[i].y, qv[i].z, qv[i].w}, kw[4] = {kv[i].x, kv[i].y, kv[i].z, kv[i].w};
      const uint32_t pw[4] = {kp[i].x, kp[i].y, kp[i].z, kp[i].w}, rw[4] = {qp[i].x, qp[i].y, qp[i].z, qp[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint64_t kk = wide(kw[e]);
        sum_q = ptx::fma_f32x2(wide(qw[e]), ptx::add_f32x2(kk, wide(pw[e])), sum_q);
        sum_k = ptx::fma_f32x2(kk, wide(rw[e]), sum_k);
      }
    }
    float s = across(ptx::add_f32x2(sum_q, sum_k));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((c.lane & 3) == 0) scores[n] = n < len ? s * (a.sm_scale * 1.4426950408889634f) : -INFINITY;
  }
  ptx::bar_sync(1u + uint32_t(c.warp >> 2), 128);
  const float s0 = scores[c.lane], s1 = len > 32 ? scores[32 + c.lane] : -INFINITY;
  float top = fmaxf(s0, s1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  const float p0 = ptx::ex2(s0 - top), p1 = ptx::ex2(s1 - top);
  const float inv = 1.f / warp_sum(p0 + p1);
  uint64_t o = both(0.f);
#pragma unroll
  for (int i = 0; i < 8; ++i) o = ptx::fma_f32x2(both(__shfl_sync(0xffffffffu, p0, sub + 4 * i)), wide(vw[i]), o);  // (probability zero behind the sequence)
  if (len > 32) {
#pragma unroll
    for (int i = 0; i < 8; ++i) vw[i] = 32 + sub + 4 * i < len ? __ldcg(vr + (int64_t)(32 + sub + 4 * i) * (a.hidden / 2)) : 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) o = ptx::fma_f32x2(both(__shfl_sync(0xffffffffu, p1, sub + 4 * i)), wide(vw[i]), o);
  }
  float o0, o1;
  ptx::unpack_f32x2(o, o0, o1);
#pragma unroll
  for (int d = 8; d < 32; d <<= 1) {
    o0 += __shfl_xor_sync(0xffffffffu, o0, d);
    o1 += __shfl_xor_sync(0xffffffffu, o1, d);
  }
  if (c.lane < 8) *out = ptx::pack_bf16x2(o0 * inv, o1 * inv);
}

template <int MT>
__global__ void __launch_bounds__(kThreads, 1) encoder_small_kernel(const __grid_constant__ SmallEncoderArgs args) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ int s_start[kSmallRows], s_len[kSmallRows];
  __shared__ uint32_t s_ok;
  Ctx c;
  c.a = &args;
  c.tid = threadIdx.x; c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31;
  c.rows = args.rows_dev != nullptr ? min(*args.rows_dev, args.row_bound) : args.row_bound;
  c.pitch = args.hidden * 2 + 16;
  c.s_x = smem;
  c.s_red = reinterpret_cast<float*>(smem + MT * 16 * c.pitch);

  // the sequence of every row
  for (int i = c.tid; i < kSmallRows; i += kThreads) s_start[i] = s_len[i] = 0;
  for (int i = c.tid; i < (MT * 16 - c.rows) * (c.pitch / 16); i += kThreads)  // rows of the tiles behind the last one
    reinterpret_cast<uint4*>(c.s_x + c.rows * c.pitch)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int b = c.tid; b < args.batch; b += kThreads) {
    int start = b * args.max_seqlen, end = start + args.max_seqlen;
    if (args.cu_seqlens != nullptr) {
      start = args.cu_seqlens[b];
      end = args.cu_seqlens[b + 1];
      if (start < 0 || end < start || end - start > args.max_seqlen || end > args.row_bound) {
        if (blockIdx.x == 0 && args.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(args.status), FDB_DEV_BAD_SEQLEN);
        continue;
      }
    }
    for (int r = start; r < min(end, c.rows); ++r) { s_start[r] = start; s_len[r] = end - start; }
  }
  __syncthreads();

  const int hidden = args.hidden, heads = hidden / 64;
  uint32_t barriers = 0;
  auto sync_grid = [&]() -> bool { return grid_barrier(args, &s_ok, ++barriers * gridDim.x); };
  auto keep = [&](int row, int i, uint4 v) { *reinterpret_cast<uint4*>(c.s_x + row * c.pitch + i * 16) = v; };
  auto residual = [&](int row, int col) -> uint32_t { return *reinterpret_cast<const uint32_t*>(c.s_x + row * c.pitch + col * 2); };
  auto add_to = [&](__nv_bfloat16* y) {
    return [=](int row, int, int col, float v0, float v1) {
      const uint32_t r = residual(row, col);
      *reinterpret_cast<uint32_t*>(y + (int64_t)row * hidden + col) = ptx::pack_bf16x2(v0 + lo(r), v1 + hi(r));
    };
  };

  for (int i = 0; i < args.n_layers; ++i) {
    const SmallLayer& l = args.layer[i];
    const Product qkv = make_product(c, l.wq, l.wk, l.wv, l.bq, l.bk, l.bv, hidden, 3, hidden);
    const Product proj = make_product(c, l.wo, nullptr, nullptr, l.bo, nullptr, nullptr, hidden, 1, hidden);
    const Product up = make_product(c, l.wi, nullptr, nullptr, l.bi, nullptr, nullptr, args.ffn, 1, hidden);
    const Product down = make_product(c, l.wd, nullptr, nullptr, l.bd, nullptr, nullptr, hidden, 1, args.ffn);
    // 1
    if (i == 0) normalise(c, args.x, nullptr, nullptr, 0.f, c.warp, kWarps, keep);
    else normalise(c, args.y, args.layer[i - 1].ln2_gamma, args.layer[i - 1].ln2_beta, args.layer[i - 1].ln2_eps, c.warp, kWarps, keep);
    __syncthreads();
    product<MT, false>(c, qkv, nullptr, [&](int row, int grp, int col, float v0, float v1) {
      *reinterpret_cast<uint32_t*>(args.qkv + ((int64_t)grp * args.row_bound + row) * hidden + col) = ptx::pack_bf16x2(v0, v1);
    });
    prefetch(c, proj);
    if (!sync_grid()) return;
    // 2
    float* scores = c.s_red + (c.warp >> 2) * 128;  // (the products' partial sums have been read)
    int turn = 0;
    for (int item = blockIdx.x + gridDim.x * (c.warp >> 2); item < c.rows * heads; item += gridDim.x * (kWarps / 4)) {
      const int row = item / heads, len = s_len[row];
      attention_row(c, l, row, item - row * heads, s_start[row], len, scores + turn * 64);
      if (len > 0) turn ^= 1;  // (a row of no sequence passes no barrier: the scores of the row before may still be read)
    }
    prefetch(c, up);
    if (!sync_grid()) return;
    // 3
    product<MT, true>(c, proj, args.ctx, add_to(args.y));
    prefetch(c, down);
    if (!sync_grid()) return;
    // 4
    normalise(c, args.y, l.ln1_gamma, l.ln1_beta, l.ln1_eps, c.warp, kWarps, keep);
    __syncthreads();
    product<MT, false>(c, up, nullptr, [&](int row, int, int col, float v0, float v1) {
      float g0, g1;
      ptx::unpack_f32x2(gelu_erf2(ptx::pack_f32x2(v0, v1)), g0, g1);
      *reinterpret_cast<uint32_t*>(args.mid + (int64_t)row * args.ffn + col) = ptx::pack_bf16x2(g0, g1);
    });
    if (i + 1 < args.n_layers) {
      const SmallLayer& n = args.layer[i + 1];
      prefetch(c, make_product(c, n.wq, n.wk, n.wv, nullptr, nullptr, nullptr, hidden, 3, hidden));
    }
    if (!sync_grid()) return;
    // 5
    product<MT, true>(c, down, args.mid, add_to(args.y));
    if (!sync_grid()) return;
  }
  const SmallLayer& l = args.layer[args.n_layers - 1];
  normalise(c, args.y, l.ln2_gamma, l.ln2_beta, l.ln2_eps, blockIdx.x + gridDim.x * c.warp, gridDim.x * kWarps, [&](int row, int i, uint4 v) {
    reinterpret_cast<uint4*>(args.out + (int64_t)(args.out_index != nullptr ? args.out_index[row] : row) * hidden)[i] = v;
  });
}

size_t smem_bytes(int mt, int hidden, int ffn, int sms) {
  int tiles = 0;  // per CTA; with four of them half as many partial sums (the last CTA may have three)
  for (int n : {3 * hidden, hidden, ffn}) tiles = std::max(tiles, (n / 8 + sms - 1) / sms);
  return size_t(mt) * 16 * (hidden * 2 + 16) + size_t(mt) * 16 * 4 * std::min(tiles, 3) * 8 * kWarps;
}

}  // namespace

bool small_encoder_covers(int64_t row_bound, int hidden, int ffn, int n_layers) {
  const int sms = sm_count();
  if (sms <= 0 || row_bound > kSmallRows || hidden > 1024 || n_layers > kSmallLayers) return false;
  // Where it is the faster form.  16 / 32 / 48 / 64 rows, us against the separate launches: 12 layers of 768 298 / 326 / 443 / 471
  // against 610; 24 layers of 1024 649 / 751 / 1148 against 1390.  The line between 48 and 64 rows of 1024 was drawn when 64 took 1480
  // here; they take 1196 against 1380 by now, so it lies too low for the row counts in between.
  if (row_bound * hidden > 48 * 1024) return false;
  const int most = std::max(3 * hidden, ffn);
  return (most / 8 + sms - 1) / sms <= kMaxTiles && smem_bytes(row_bound <= 16 ? 1 : (row_bound <= 32 ? 2 : 4), hidden, ffn, sms) <= 227 * 1024 - 1024;
}

int launch_small_encoder(const SmallEncoderArgs& a, void* stream) {
  const int sms = sm_count(), mt = a.row_bound <= 16 ? 1 : (a.row_bound <= 32 ? 2 : 4);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto kernel = mt == 1 ? encoder_small_kernel<1> : (mt == 2 ? encoder_small_kernel<2> : encoder_small_kernel<4>);
  static std::atomic<uint64_t> smem_done[3];
  cudaError_t e = allow_smem(smem_done[mt >> 1], reinterpret_cast<const void*>(kernel), 227 * 1024 - 1024);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sms);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem_bytes(mt, a.hidden, a.ffn, sms);
  cfg.stream = s;
  cudaLaunchAttribute at;  // the CTAs wait for one another: all of them have to be resident
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  void* ptr = const_cast<SmallEncoderArgs*>(&a);
  if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), &ptr);
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "small encoder launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace fdb
