// Fused backward of the disentangled attention for sm_100a: tcgen05 tiles, probabilities rebuilt in tensor memory, nothing
// quadratic in the sequence length in global memory.
//
// Replaces the reference's two Triton backward kernels (src/flashdeberta/ops/flash_attention.py:616-797 dK/dV with the
// position-bias gradients scattered by atomics :770-786, :799-940 dQ).  Like them it is one kernel per stationary side:
//   <false>  rows = queries, columns = keys:   S = Q.K^T, dP = dO.V^T, G = scale * P * (dP - delta);  dQ += G.K
//   <true>   rows = keys, columns = queries:   S^T, dP^T;                                              dV += P^T.dO, dK += G^T.Q
// The second is the first with the roles of queries and keys, of the two position tables and of the sign of the distance
// exchanged, so one template serves both: "row term" is the position term of the row's own operand (c2p of a query row, p2c
// of a key row), "column term" the other one.
//
// One CTA = 128 rows of one (sequence, head), columns in tiles of 64, two CTAs per SM (256 tensor-memory columns, 111 KB of
// shared memory, 32768 registers each): what is serial inside a tile runs beside the other CTA.
//   warps 0-7    thread r of a half owns row r and 32 of the 64 columns     warps 8-11  run sums of the rows (position gradients)
//   warp 12      issues every tcgen05.mma                                   warp 13     issues every TMA load
// Tensor memory: R0 64 | R1 64 | accumulators 64 + 64.  Everything passes through R0 and R1:
//   row term     the products row . X[window]^T of the tile's 192 window positions, 64 at a time.  Row r needs the 64 positions
//                r .. r+63, so a thread needs 32 consecutive ones that start at its lane: it shifts 64 registers down by its lane;
//   column term  the products X[window] . column^T arranged so that the value a thread needs lies in its own 32-lane quarter:
//                one select and one warp shuffle per element (as in the forward kernel);
//   S, dP        then P and G go back over S as bf16 pairs, the A operand of the accumulating products.
// Tiles whose distances are all saturated have one value per row (a dot product) and one per column (accumulated into S from
// eight identical rows of the table).
//
// Position gradients: along a row the distance falls by one per column and the table row never rises, so the elements that
// share a table row are one run.  Warps 8-11 carry the running sum of each row's run, park it in shared memory when the table
// row changes, and write finished groups of eight to global memory: (heads, rows, table rows) in bf16, every entry written
// once, no atomics (attn_bwd_tables_sm100.cu does the rest: dQ += sums . pos_key, dpos_key = sums^T . Q, the same for the keys).
// They clear their rows of the sums themselves while the first tile is on its way: a memset in front cost 18 us a side.
//
// What bounds it: the chain row term -> column term -> S -> P -> G inside a tile, about 10.5 thousand clocks of which the
// row-term shift takes 2.4 and the wait for its products 2.2 or more; the run sums (5) lie beside it.  4 x 2048 rows x 12 heads,
// both terms, us per kernel (<false> / <true>): one warpgroup for the whole tile, row term through shared memory 1345 / 1494; two
// column halves and run sums of their own warps 570 / 628; the register shift and a second window buffer 558 / 592; run sums from
// registers, sixteen columns at a time 451 / 468.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "attn_bwd.h"
#include "attn_fwd_common.cuh"
#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"
#include "tensor_map.cuh"

namespace fdb {
namespace {

using namespace ptx;
using namespace fwd;

constexpr int kCols = 64;       // columns of a tile
constexpr int kWin = 192;       // window positions of a tile: 128 + 64 - 1
constexpr int kThreads = 512;   // two column halves, run sums, issuing warps: a warpgroup each
constexpr int kSumWarp0 = 8, kMmaWarp = 12, kTmaWarp = 13;
constexpr int kMathRegs = 88, kSumRegs = 56, kAuxRegs = 24;  // 2 CTAs per SM: 32768 = 88 * 256 + 56 * 128 + 24 * 128
constexpr uint32_t kTmemCols = 256;
constexpr uint32_t kColR = 0, kColAcc = 128;
constexpr int kMaxRows = 4096;  // rows of an expanded table (one bit each in shared memory)

constexpr uint32_t kSmemRow = 0;                        // two operands of 128 x 128 B
constexpr uint32_t kSmemCol = 32768;                    // two operands of 64 x 128 B
constexpr uint32_t kSmemWin = 49152;                    // 192 x 128 B window of the row table, the same of the column table
constexpr uint32_t kSmemSat = kSmemWin + 2 * kWin * 128;  // 2 x (8 x 128 B) saturated rows of the column table (hi, lo)
constexpr uint32_t kEmitPitch = 80;                     // per row: finished run sums (bf16), three groups of eight, and padding
constexpr uint32_t kSmemEmit = kSmemSat + 2048;
constexpr uint32_t kSmemCols = kSmemEmit + 128 * kEmitPitch;  // float [2][2][64]: LSE and delta of the columns (<true>)
constexpr uint32_t kSmemBits = kSmemCols + 1024;        // one bit per expanded row: its table row differs from the row before
constexpr uint32_t kSmemBars = kSmemBits + kMaxRows / 8;
constexpr uint32_t kSmemBytes = kSmemBars + 128 + 1024;
static_assert(2 * (kSmemBytes + 1024) <= 232448, "two CTAs per SM");

enum Bar : uint32_t {
  kBarRow = 0,    // 1  row operands landed
  kBarCol = 1,    // 1  column operands landed
  kBarAcc = 2,    // 1  the accumulating products of a tile finished (the column operands are free)
  kBarWin = 3,    // 1  window of the row / column table landed
  kBarWinFree = 5,// 1  the products that read it finished
  kBarU = 7,      // 1  R0 / R1 filled
  kBarUFree = 9,  // 8  R0 / R1 read by both halves
  kBarG = 11,     // 8  P and G are in R0
  kBarGRead = 12, // 4  the run sums have read G
  kNumBars = 13
};

struct alignas(64) BwdArgs {
  CUtensorMap tm_row[2], tm_col[2];       // <false>: Q, dO; K, V.  <true>: K, V; Q, dO
  CUtensorMap tm_xrow, tm_xcol, tm_xcol_sat;
  const int4* slot_info;
  const __nv_bfloat16* xrow;              // expanded table of the row term (heads, xrows, 64), NULL without the term
  const __nv_bfloat16* xcol;              // of the column term
  const float *lse, *delta;               // (rows, heads)
  float* core;                            // with the row term: (rows, heads, 64), dQ or dK without its part
  __nv_bfloat16* grad;                    // without it: dQ or dK
  __nv_bfloat16* dv;                      // <true>
  int64_t grad_rs, grad_hs;               // strides of dQ, dK, dV
  __nv_bfloat16* sums;                    // (heads of this launch, rows, table_rows); every pointer starts at the launch's first head
  const int16_t* lut;
  int32_t* status;
  int lut_d_min, lut_len, table_rows;
  int heads, packed, max_seqlen, total_rows;
  int sum_heads;                          // heads that `sums` has room for
  int sat_lo, sat_hi, d_first, xrows;     // in distances row - column
  float sm_scale;
};

// table row of distance d = row - column
template <bool DKV>
__device__ __forceinline__ int table_row(const BwdArgs& a, int d) {
  int i = (DKV ? -d : d) - a.lut_d_min;
  i = i < 0 ? 0 : (i >= a.lut_len ? a.lut_len - 1 : i);
  return a.lut[i];
}

// `n` threads, this one the `lane`th, clear what this kernel writes of a row outside every sequence
template <bool DKV>
__device__ __forceinline__ void zero_row(const BwdArgs& a, int64_t row, int head, int lane, int n) {
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  for (int i = lane; i < 16; i += n) {
    const int64_t at = row * a.grad_rs + head * a.grad_hs + (i & 7) * 8;
    if (a.xrow != nullptr) *reinterpret_cast<uint4*>(a.core + (row * a.heads + head) * 64 + i * 4) = z;
    else if (i < 8) *reinterpret_cast<uint4*>(a.grad + at) = z;
    if (DKV && i < 8) *reinterpret_cast<uint4*>(a.dv + at) = z;
  }
  if (a.xrow != nullptr && head < a.sum_heads)
    for (int i = lane; i < a.table_rows / 8; i += n)
      *reinterpret_cast<uint4*>(a.sums + ((int64_t)head * a.total_rows + row) * a.table_rows + i * 8) = z;
}

template <bool DKV>
__global__ void __launch_bounds__(kThreads, 2) bwd_kernel(const __grid_constant__ BwdArgs args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = (int)uniform(uint32_t(tid) >> 5), lane = tid & 31;
  const int head = blockIdx.y;

  const int4 slot = __ldg(args.slot_info + blockIdx.x);  // (sequence, first row of the tile in it, its first row, its length)
  if (slot.x < 0) return;
  const int r0 = (int)uniform(slot.y), seq_row0 = (int)uniform(slot.z), len = (int)uniform(slot.w);
  const int row_limit = args.packed ? len : args.max_seqlen;  // rows of the padded batch that this sequence owns

  const bool row_term = args.xrow != nullptr, col_term = args.xcol != nullptr;
  if (r0 >= len) {  // dense padding: zero gradients
    for (int row = r0 + warp; row < min(r0 + 128, row_limit); row += kThreads / 32) zero_row<DKV>(args, seq_row0 + row, head, lane, 32);
    return;
  }

  const int n_tiles = (len + kCols - 1) / kCols;
  // tiles [jb, jb + nb) have distances inside the bucketed range; saturated high in front of them, low behind
  int jb = 0, je = 0;
  if (row_term || col_term) {
    // (one distance of slack: the column behind a saturated tile must still share the tile's table row, so that no run ends there)
    const int lo = r0 - (kCols - 1) - args.sat_hi - 1;
    jb = min(lo < 0 ? 0 : lo / kCols + 1, n_tiles);
    je = min((r0 + 127 - args.sat_lo - 1) / kCols + 1, n_tiles);
    je = max(je, jb);
  }
  auto kind_of = [&](int j) -> int {
    if (!row_term && !col_term) return kPlain;
    return j < jb ? kSatHi : (j < je ? kBand : kSatLo);
  };

  auto bar = [&](uint32_t i) -> uint32_t { return smem + kSmemBars + 8u * i; };
  const uint32_t tmem_slot = smem + kSmemBars + 8u * kNumBars;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBars + 8u * kNumBars + 8u);
  if (tid == 0) {
    *abort_flag = 0u;
    for (uint32_t i = 0; i < kNumBars; ++i) mbar_init(bar(i), i == kBarGRead ? 4u : (i >= kBarUFree ? 8u : 1u));
    fence_barrier_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  if (row_term) {
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem_gen + kSmemBits);
    for (int i = tid; i < ((args.xrows + 31) & ~31); i += kThreads) {
      const int d = args.d_first + i;
      const uint32_t w = __ballot_sync(0xffffffffu, table_row<DKV>(args, d) != table_row<DKV>(args, d - 1));
      if (lane == 0) bits[i >> 5] = w;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBars + 8u * kNumBars));

  bool ok = true;
  auto wait = [&](uint32_t b, uint32_t parity) {  // whole warps wait, the result is warp-uniform
    if (ok) ok = mbar_wait_warp(b, parity, abort_flag);
  };
  auto arrive = [&](uint32_t b) {  // one arrival per warp
    __syncwarp();
    if (elect_one()) mbar_arrive(b);
  };

  if (warp >= kMmaWarp) {
    reg_dealloc<kAuxRegs>();
    if (warp == kTmaWarp) {
      // ================================================= TMA producer ===================================================
      if (elect_one()) {
        mbar_expect_tx(bar(kBarRow), 32768u + (col_term ? 2048u : 0u));
        tma_load_3d(smem + kSmemRow, &args.tm_row[0], bar(kBarRow), 0, head, seq_row0 + r0);
        tma_load_3d(smem + kSmemRow + 16384, &args.tm_row[1], bar(kBarRow), 0, head, seq_row0 + r0);
        if (col_term) {
          tma_load_3d(smem + kSmemSat, &args.tm_xcol_sat, bar(kBarRow), 0, args.xrows - 8, head);
          tma_load_3d(smem + kSmemSat + 1024, &args.tm_xcol_sat, bar(kBarRow), 0, 0, head);
        }
      }
      uint32_t n_band = 0;  // band tiles so far
      auto load_window = [&](uint32_t w, const CUtensorMap* map, int j) {
        if (n_band > 0) wait(bar(kBarWinFree + w), (n_band - 1u) & 1u);
        if (ok && elect_one()) {
          mbar_expect_tx(bar(kBarWin + w), uint32_t(kWin) * 128u);
          tma_load_3d(smem + kSmemWin + w * uint32_t(kWin * 128), map, bar(kBarWin + w), 0, r0 - j * kCols - (kCols - 1) - args.d_first, head);
        }
      };
#pragma unroll 1
      for (int j = 0; j < n_tiles && ok; ++j) {
        if (kind_of(j) == kBand) {
          if (row_term) load_window(0, &args.tm_xrow, j);
          if (col_term) load_window(1, &args.tm_xcol, j);
          ++n_band;
        }
        if (j > 0) wait(bar(kBarAcc), uint32_t(j - 1) & 1u);
        if (ok && elect_one()) {
          mbar_expect_tx(bar(kBarCol), 16384u);
          tma_load_3d(smem + kSmemCol, &args.tm_col[0], bar(kBarCol), 0, head, seq_row0 + j * kCols);
          tma_load_3d(smem + kSmemCol + 8192, &args.tm_col[1], bar(kBarCol), 0, head, seq_row0 + j * kCols);
        }
      }
    } else if (warp == kMmaWarp) {
      // ================================================= MMA issuer =====================================================
      const uint32_t idesc_64 = instr_desc(128, 64, 1, 0, 0), idesc_32 = instr_desc(128, 32, 1, 0, 0);
      const uint32_t idesc_acc = instr_desc(128, 64, 1, 0, 1);
      const uint64_t drow = smem_desc_sw128(smem + kSmemRow, 1024, 16), dcol = smem_desc_sw128(smem + kSmemCol, 1024, 16);
      const uint64_t dwin_r = smem_desc_sw128(smem + kSmemWin, 1024, 16), dwin_c = smem_desc_sw128(smem + kSmemWin + kWin * 128, 1024, 16), dsat = smem_desc_sw128(smem + kSmemSat, 0, 16);
      constexpr uint64_t blk32 = (32u * 128u) >> 4;
      uint32_t n_band = 0, used[2] = {0, 0};
      auto next_use = [&](uint32_t i) {  // R_i may be written again
        if (used[i] > 0) wait(bar(kBarUFree + i), (used[i] - 1u) & 1u);
        ++used[i];
        tc_fence_after();
      };
      auto product = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) mma_bf16(d, a + uint64_t((ks * 32) >> 4), b + uint64_t((ks * 32) >> 4), idesc, add | uint32_t(ks > 0));
      };
      wait(bar(kBarRow), 0);
#pragma unroll 1
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int kind = kind_of(j);
        if (j > 0) {  // P and G of the tile before have been read out of R0
          wait(bar(kBarAcc), uint32_t(j - 1) & 1u);
          if (row_term) wait(bar(kBarGRead), uint32_t(j - 1) & 1u);
        }
        if (kind == kBand && row_term) {
          wait(bar(kBarWin), n_band & 1u);
#pragma unroll
          for (uint32_t k = 0; k < 3; ++k) {
            next_use(k & 1u);
            if (ok && elect_one()) {
              product(tmem_base + kColR + 64u * (k & 1u), drow, dwin_r + uint64_t(k) * 2u * blk32, idesc_64, 0);
              mma_commit(bar(kBarU + (k & 1u)));
              if (k == 2) mma_commit(bar(kBarWinFree));
            }
          }
        }
        wait(bar(kBarCol), uint32_t(j) & 1u);
        if (kind == kBand && col_term) {
          // 32-column block b needs the window rows starting at 32(1-b) (t = 0) and 32(2-b) (t = 1); unit u has start row
          // 64 - 32u: block u-1 (t = 0) in its first 32 columns, block u (t = 1) in the last 32
          wait(bar(kBarWin + 1), n_band & 1u);
#pragma unroll
          for (uint32_t u = 0; u < 3; ++u) {
            const uint32_t i = (u & 1u) ^ 1u;
            next_use(i);
            if (ok && elect_one()) {
              product(tmem_base + kColR + 64u * i + (u == 0 ? 32u : 0u), dwin_c + uint64_t(2u - u) * blk32,
                      dcol + uint64_t(u == 2 ? 1u : 0u) * blk32, u == 1 ? idesc_64 : idesc_32, 0);
              mma_commit(bar(kBarU + i));
              if (u == 2) mma_commit(bar(kBarWinFree + 1));
            }
          }
        }
        n_band += kind == kBand ? 1u : 0u;
        next_use(0);
        if (ok && elect_one()) {
          product(tmem_base + kColR, drow, dcol, idesc_64, 0);
          if (col_term && (kind == kSatHi || kind == kSatLo))
            product(tmem_base + kColR, dsat + uint64_t(kind == kSatHi ? 0u : (1024u >> 4)), dcol, idesc_64, 1);
          mma_commit(bar(kBarU));
        }
        next_use(1);
        if (ok && elect_one()) {
          product(tmem_base + kColR + 64u, drow + (16384u >> 4), dcol + (8192u >> 4), idesc_64, 0);
          mma_commit(bar(kBarU + 1));
        }
        wait(bar(kBarG), uint32_t(j) & 1u);
        tc_fence_after();
        if (ok && elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {  // 16 columns of the tile per step = 2048 bytes of the column operand
            const uint32_t more = j > 0 || ks > 0 ? 1u : 0u;
            const uint32_t op = tmem_base + kColR + 32u * uint32_t(ks >> 1) + 8u * uint32_t(ks & 1);  // P; G 16 columns on
            mma_bf16_ts(tmem_base + kColAcc, op + 16u, dcol + uint64_t((ks * 2048) >> 4), idesc_acc, more);
            if (DKV) mma_bf16_ts(tmem_base + kColAcc + 64u, op, dcol + ((8192u + ks * 2048u) >> 4), idesc_acc, more);
          }
          mma_commit(bar(kBarAcc));
        }
      }
    }
  } else if (warp >= kSumWarp0) {
    // ================================================= run sums =========================================================
    // Thread r follows row r through the columns: sums of G (as rounded for the products) over the columns that share a table row.
    reg_dealloc<kSumRegs>();
    const int quad = warp & 3;
    const int my_row = r0 + quad * 32 + lane;
    const bool valid_row = my_row < len;
    const uint32_t tmem_lane = tmem_base + (uint32_t(quad * 32) << 16);
    if (row_term) {
      for (int i = 0; i < 32; ++i) {  // a row at a time: whole lines (a packed row behind the sequence is another one's)
        const int row = r0 + quad * 32 + i;
        if (row >= len && (args.packed || row >= row_limit)) break;
        uint4* z = reinterpret_cast<uint4*>(args.sums + ((int64_t)head * args.total_rows + seq_row0 + row) * args.table_rows);
        for (int c = lane; c < args.table_rows / 8; c += 32) z[c] = make_uint4(0u, 0u, 0u, 0u);
      }
      __syncwarp();
      float run = 0.f;                            // sum of the current run
      int b = table_row<DKV>(args, my_row);       // and its table row: falls by one per run (<true>: rises)
      // Finished sums wait in a row of three aligned groups of eight table rows: the current group lies in the last one (<true>:
      // the first), the next ones go towards the other end.  Sixteen columns complete at most two groups.
      const uint32_t mine = smem + kSmemEmit + uint32_t(quad * 32 + lane) * kEmitPitch;
      constexpr uint32_t kHome = DKV ? 0u : 32u;  // byte offset of the current group
      sts_v4(mine + kHome, 0u, 0u, 0u, 0u);
      uint4* sums = reinterpret_cast<uint4*>(args.sums + ((int64_t)head * args.total_rows + seq_row0 + (valid_row ? my_row : len - 1)) * args.table_rows);
      const uint32_t* bits = reinterpret_cast<const uint32_t*>(smem_gen + kSmemBits);
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) {
        wait(bar(kBarG), uint32_t(j) & 1u);
        tc_fence_after();
        uint32_t g[2][16];
        tmem_ld16(tmem_lane + kColR + 16u, g[0]);
        tmem_ld16(tmem_lane + kColR + 48u, g[1]);
        tmem_wait_ld();
        tc_fence_before();
        arrive(bar(kBarGRead));
        if (kind_of(j) != kBand) {
          float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            a[i & 1] += __uint_as_float(g[i >> 4][i & 15] << 16);
            a[2 + (i & 1)] += __uint_as_float(g[i >> 4][i & 15] & 0xffff0000u);
          }
          run += (a[0] + a[1]) + (a[2] + a[3]);
          continue;
        }
        // bit n: a run ends with column n, i.e. the distance after it (one less) has another table row
        const int c0 = j * kCols;
        const int top = my_row - c0 - args.d_first;  // expanded row of column 0; column n is n rows below
        const int w = top >> 5, sh = top & 31;
        const uint32_t b2 = bits[w], b1 = w > 0 ? bits[w - 1] : 0u, b0 = w > 1 ? bits[w - 2] : 0u;
        // rows top-31 .. top and top-63 .. top-32, lowest row in the lowest bit; reversed: bit n is column n, n + 32
        uint32_t ends[2] = {__brev(__funnelshift_rc(b1, b2, sh + 1)), __brev(__funnelshift_rc(b0, b1, sh + 1))};
        const int last = len - c0 - 1;  // the last column of the sequence ends no run here: that is done behind the loop
        if (last < 64) {
          ends[0] &= last <= 0 ? 0u : (last >= 32 ? 0xffffffffu : (1u << last) - 1u);
          ends[1] &= last <= 32 ? 0u : (1u << (last - 32)) - 1u;
        }
        if (!valid_row) ends[0] = ends[1] = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int group = b >> 3;
          uint32_t at = mine + kHome + 2u * uint32_t(b & 7);
#pragma unroll
          for (int n = 0; n < 16; ++n) {
            const uint32_t w = g[q >> 1][(8 * q + (n >> 1)) & 15];
            run += __uint_as_float((n & 1) ? (w & 0xffff0000u) : (w << 16));
            const uint32_t end = ends[q >> 1] & (1u << ((16 * q + n) & 31));
            // predicated, not branched around: with 32 rows one distance apart some lane ends a run at nearly every column
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.u16 [%1], %2;\n\t}" ::"r"(end), "r"(at),
                         "h"(__bfloat16_as_ushort(__float2bfloat16_rn(run))) : "memory");
            at = end ? (DKV ? at + 2u : at - 2u) : at;
            b = end ? (DKV ? b + 1 : b - 1) : b;
            run = end ? 0.f : run;
          }
          const int full = DKV ? (b >> 3) - group : group - (b >> 3);  // groups completed: 0, 1 or 2
          if (__any_sync(0xffffffffu, full > 0)) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
              if (full > i) sums[DKV ? group + i : group - i] = lds_v4(mine + (DKV ? 16u * i : 32u - 16u * i));
            if (full > 0) {  // what is left of the last group goes home
              const uint4 v = lds_v4(mine + (DKV ? 16u * uint32_t(full) : 32u - 16u * uint32_t(full)));
              sts_v4(mine + kHome, v.x, v.y, v.z, v.w);
            }
          }
        }
      }
      if (valid_row) {  // the last run, then zeros up to the end of its group
        uint32_t at = mine + kHome + 2u * uint32_t(b & 7);
        sts_u16(at, uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(run))));
        for (int i = b & 7; i != (DKV ? 7 : 0); i += DKV ? 1 : -1) {
          at = DKV ? at + 2u : at - 2u;
          sts_u16(at, 0u);
        }
        sums[b >> 3] = lds_v4(mine + kHome);
      }
    }
  } else {
    // =================================================== P and G ========================================================
    reg_alloc<kMathRegs>();
    const int h = warp >> 2;                 // column half: columns 32h .. 32h+31 of every tile
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t tmem_lane = tmem_base + (uint32_t(quad * 32) << 16);
    const int my_row = r0 + r;
    const bool valid_row = my_row < len;
    const float c_eff = args.sm_scale * 1.4426950408889634f;
    const int64_t rh = (int64_t)(seq_row0 + (valid_row ? my_row : len - 1)) * args.heads + head;
    float row_lse = 0.f, row_delta = 0.f;  // LSE in log2 units
    if (!DKV) {
      row_lse = __ldg(args.lse + rh) * 1.4426950408889634f;
      row_delta = __ldg(args.delta + rh);
    }
    // <true>: LSE and delta belong to the columns; of the first half, thread r < 64 brings the LSE of column r, thread r >= 64 the
    // delta of column r - 64
    auto column_value = [&](int j) -> float {
      const int c = j * kCols + (r & 63);
      const int64_t at = (int64_t)(seq_row0 + (c < len ? c : len - 1)) * args.heads + head;
      return r < 64 ? __ldg(args.lse + at) * 1.4426950408889634f : __ldg(args.delta + at);
    };
    float next_col = 0.f;
    if (DKV && h == 0) next_col = column_value(0);

    wait(bar(kBarRow), 0);
    float rc_lo = 0.f, rc_hi = 0.f;  // saturated row terms
    if (row_term && ok) {
      const uint32_t row_addr = smem + kSmemRow + uint32_t(r) * 128u;
      const __nv_bfloat16* x = args.xrow + (int64_t)head * args.xrows * kHeadDim;
      rc_lo = dot_q_row(row_addr, r, x);
      rc_hi = dot_q_row(row_addr, r, x + (int64_t)(args.xrows - 1) * kHeadDim);
    }

    uint32_t seen = 0;               // phase bits of R0, R1
    auto wait_u = [&](uint32_t i) {
      wait(bar(kBarU + i), (seen >> i) & 1u);
      seen ^= 1u << i;
      tc_fence_after();
    };
    auto free_u = [&](uint32_t i) {
      tc_fence_before();
      arrive(bar(kBarUFree + i));
    };

#pragma unroll 1
    for (int j = 0; j < n_tiles; ++j) {
      const int kind = kind_of(j);
      const int c0 = j * kCols;
      if (DKV) {
        if (h == 0) {
          sts_f32(smem + kSmemCols + (uint32_t(j) & 1u) * 512u + uint32_t(r) * 4u, next_col);
          if (j + 1 < n_tiles) next_col = column_value(j + 1);
        }
        bar_sync(1, 256);  // (a thread two tiles ahead cannot be: the tile after this one syncs too)
      }
      float s[32];
      int lane_i = lane;  // opaque: what is computed from it per column stays inside the loop instead of in registers around it
      asm volatile("" : "+r"(lane_i));
      if (kind == kBand && row_term) {
        // position p = r + 63 - column of the window, 32-position blocks, unit k = blocks 2k and 2k+1 in R0, R1, R0.  With
        // B = quad + 1 - half the thread's 32 positions start at entry `lane` of block B: it takes blocks B and B + 1 and
        // shifts them down by its lane, one bit of it at a time (186 selects; through a shared-memory row of its own the
        // same took 64 predicated stores, 32 loads and twice the time).
        const int B = quad + 1 - h;
        wait_u(0);  // unit 0
        if (B >= 2) free_u(0);
        wait_u(1);  // unit 1
        if (B >= 3) wait_u(0);  // unit 2
        uint32_t x[64];
        tmem_ld32(tmem_lane + kColR + uint32_t(((B >> 1) & 1) * 64 + (B & 1) * 32), reinterpret_cast<uint32_t(&)[32]>(x[0]));
        tmem_ld32(tmem_lane + kColR + uint32_t((((B + 1) >> 1) & 1) * 64 + ((B + 1) & 1) * 32), reinterpret_cast<uint32_t(&)[32]>(x[32]));
        tmem_wait_ld();
        if (B < 2) free_u(0);
        free_u(1);
        if (B < 3) wait_u(0);  // unit 2 holds nothing for this warp
        free_u(0);
#pragma unroll
        for (int i = 0; i < 47; ++i) x[i] = (lane_i & 16) ? x[i + 16] : x[i];
#pragma unroll
        for (int i = 0; i < 39; ++i) x[i] = (lane_i & 8) ? x[i + 8] : x[i];
#pragma unroll
        for (int i = 0; i < 35; ++i) x[i] = (lane_i & 4) ? x[i + 4] : x[i];
#pragma unroll
        for (int i = 0; i < 33; ++i) x[i] = (lane_i & 2) ? x[i + 2] : x[i];
#pragma unroll
        for (int n = 0; n < 32; ++n) s[n] = __uint_as_float((lane_i & 1) ? x[32 - n] : x[31 - n]);
      } else {
        const float row_const = kind == kSatHi ? rc_hi : (kind == kSatLo ? rc_lo : 0.f);
#pragma unroll
        for (int n = 0; n < 32; ++n) s[n] = row_const;
      }
      if (kind == kBand && col_term) {
        // this half's 32-column block: t = 1 from unit h, t = 0 from unit h + 1 (units 0, 1, 2 in R1, R0, R1)
        wait_u(1);
        wait_u(0);
        uint32_t t1[16], t0[16];
        const uint32_t col1 = tmem_lane + kColR + (h == 0 ? 64u : 0u) + 32u, col0 = tmem_lane + kColR + (h == 0 ? 0u : 64u);
        if (h == 1) {
          free_u(1);
          wait_u(1);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          {
            tmem_ld16(col1 + 16u * q, t1);
            tmem_ld16(col0 + 16u * q, t0);
            tmem_wait_ld();
          }
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int cc = 16 * q + c;
            const uint32_t x = (lane_i + cc <= 30) ? t1[c] : t0[c];
            s[cc] += __uint_as_float(__shfl_sync(0xffffffffu, x, lane_i + 31 - cc));  // the source lane is taken modulo 32
          }
        }
        free_u(1);
        free_u(0);
        if (h == 0) {
          wait_u(1);
          free_u(1);
        }
      }
      wait_u(0);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t t[16];
        {
          tmem_ld16(tmem_lane + kColR + 32u * h + 16u * q, t);
          tmem_wait_ld();
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) s[16 * q + c] += __uint_as_float(t[c]);
      }
      free_u(0);

      // ---- P ----
      const int valid = len - c0 - 32 * h;  // columns of this half inside the sequence
      const uint32_t cols = smem + kSmemCols + (uint32_t(j) & 1u) * 512u + 128u * uint32_t(h);
#pragma unroll
      for (int n = 0; n < 32; n += 4) {
        float l4[4] = {row_lse, row_lse, row_lse, row_lse};
        if (DKV) {
          const uint4 v = lds_v4(cols + 4u * uint32_t(n));
          l4[0] = __uint_as_float(v.x); l4[1] = __uint_as_float(v.y); l4[2] = __uint_as_float(v.z); l4[3] = __uint_as_float(v.w);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n + e] = ex2(fmaf(s[n + e], c_eff, -l4[e]));
      }
      if (valid < 32 || !valid_row) {
#pragma unroll
        for (int n = 0; n < 32; ++n) s[n] = valid_row && n < valid ? s[n] : 0.f;
      }
      // P and G go over this half's own scores: P in the first 16 columns, G in the last 16
      const uint32_t col_p = tmem_lane + kColR + 32u * uint32_t(h);
      if (DKV) {
        uint32_t p[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) p[i] = pack_bf16x2(s[2 * i], s[2 * i + 1]);
        tmem_st16(col_p, p);
      }
      // ---- G = scale * P * (dP - delta) ----
      wait_u(1);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t t[16];
        {
          tmem_ld16(tmem_lane + kColR + 64u + 32u * h + 16u * q, t);
          tmem_wait_ld();
        }
        if (q == 1) free_u(1);
#pragma unroll
        for (int n = 0; n < 16; n += 4) {
          float d4[4] = {row_delta, row_delta, row_delta, row_delta};
          if (DKV) {
            const uint4 v = lds_v4(cols + 256u + 4u * uint32_t(16 * q + n));
            d4[0] = __uint_as_float(v.x); d4[1] = __uint_as_float(v.y); d4[2] = __uint_as_float(v.z); d4[3] = __uint_as_float(v.w);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) s[16 * q + n + e] *= args.sm_scale * (__uint_as_float(t[n + e]) - d4[e]);
        }
      }
      uint32_t p[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) p[i] = pack_bf16x2(s[2 * i], s[2 * i + 1]);
      tmem_st16(col_p + 16u, p);
      tmem_wait_st();
      tc_fence_before();
      arrive(bar(kBarG));
    }

    // ---- output: 32 columns per half ----
    wait(bar(kBarAcc), uint32_t(n_tiles - 1) & 1u);
    tc_fence_after();
    const bool store = my_row < row_limit;
    const int64_t row = seq_row0 + my_row, at = row * args.grad_rs + (int64_t)head * args.grad_hs + 32 * h;
    uint32_t o[32];
    auto store_bf16 = [&](__nv_bfloat16* to) {
      uint4* d = reinterpret_cast<uint4*>(to);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        d[q] = !valid_row ? make_uint4(0u, 0u, 0u, 0u)
                          : make_uint4(pack_bf16x2(__uint_as_float(o[8 * q + 0]), __uint_as_float(o[8 * q + 1])),
                                       pack_bf16x2(__uint_as_float(o[8 * q + 2]), __uint_as_float(o[8 * q + 3])),
                                       pack_bf16x2(__uint_as_float(o[8 * q + 4]), __uint_as_float(o[8 * q + 5])),
                                       pack_bf16x2(__uint_as_float(o[8 * q + 6]), __uint_as_float(o[8 * q + 7])));
    };
    tmem_ld32(tmem_lane + kColAcc + 32 * h, o);  // whole warps execute this, whatever their rows
    tmem_wait_ld();
    if (store && row_term) {
      float4* d = reinterpret_cast<float4*>(args.core + (row * args.heads + head) * 64 + 32 * h);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        d[q] = valid_row ? make_float4(__uint_as_float(o[4 * q]), __uint_as_float(o[4 * q + 1]), __uint_as_float(o[4 * q + 2]), __uint_as_float(o[4 * q + 3]))
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    } else if (store) {
      store_bf16(args.grad + at);
    }
    __syncwarp();
    if (DKV) {
      tmem_ld32(tmem_lane + kColAcc + 64 + 32 * h, o);
      tmem_wait_ld();
      if (store) store_bf16(args.dv + at);
    }
  }

  // ---- teardown ----
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (tid == 0 && args.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(args.status), FDB_DEV_TIMEOUT);
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // copies and MMAs in flight get a bounded time to land
    __syncthreads();
  }
  if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
}

// delta = sum over the head dimension of dO * O, fp32, (rows, heads); eight lanes per (row, head).  Packed rows in front of the
// first and behind the last sequence, which the tile kernels do not visit, are cleared here (`dq` and `dkv` name the outputs).
__global__ void __launch_bounds__(256) bwd_delta_kernel(const __nv_bfloat16* __restrict__ dout, int64_t d_rs, int64_t d_hs,
                                                        const __nv_bfloat16* __restrict__ out, int64_t o_rs, int64_t o_hs,
                                                        int64_t cells, int heads, float* __restrict__ delta,
                                                        const int32_t* __restrict__ cu_seqlens, int batch,
                                                        const __grid_constant__ BwdArgs dq, const __grid_constant__ BwdArgs dkv) {
  const int64_t cell = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 3;
  const int sub = threadIdx.x & 7;
  float sum = 0.f;
  if (cell < cells) {
    const int64_t row = cell / heads, h = cell % heads;
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(dout + row * d_rs + h * d_hs) + sub);
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(out + row * o_rs + h * o_hs) + sub);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sum = fmaf(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), sum);
      sum = fmaf(__uint_as_float(aw[i] & 0xffff0000u), __uint_as_float(bw[i] & 0xffff0000u), sum);
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (sub == 0 && cell < cells) delta[cell] = sum;
  if (cu_seqlens != nullptr && cell < cells) {
    const int64_t row = cell / heads;
    if (row < cu_seqlens[0] || row >= cu_seqlens[batch]) {
      zero_row<false>(dq, row, (int)(cell % heads), sub, 8);
      zero_row<true>(dkv, row, (int)(cell % heads), sub, 8);
    }
  }
}

// The four expanded tables: by distance query - key (as in the forward) and by distance key - query (the same rows backwards).
__global__ void __launch_bounds__(256) bwd_expand_kernel(const uint4* __restrict__ pos_key, const uint4* __restrict__ pos_query,
                                                         uint4* __restrict__ key, uint4* __restrict__ query,
                                                         uint4* __restrict__ key_rev, uint4* __restrict__ query_rev,
                                                         const int16_t* __restrict__ lut, int lut_len, int rows, int heads, int64_t row_stride, int64_t head_stride) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= (int64_t)heads * rows * 8) return;
  const int c = (int)(i & 7);
  const int u = (int)((i >> 3) % rows), h = (int)((i >> 3) / rows);
  int li = u - 254;  // expanded row 0 is 254 distances below the table
  li = li < 0 ? 0 : (li >= lut_len ? lut_len - 1 : li);
  const int64_t src = h * head_stride + lut[li] * row_stride + c;
  const int64_t rev = ((int64_t)h * rows + (rows - 1 - u)) * 8 + c;
  if (pos_key != nullptr) { const uint4 v = pos_key[src]; key[i] = v; key_rev[rev] = v; }
  if (pos_query != nullptr) { const uint4 v = pos_query[src]; query[i] = v; query_rev[rev] = v; }
}

int table_rows_of(const fdb_attn_params& p) { return 2 * (p.position_buckets > 0 ? p.position_buckets : p.max_relative_positions); }

TableStrides table_strides(const fdb_attn_bwd_params& b) {
  if (b.table_row_stride > 0) return {b.table_row_stride, b.table_head_stride};
  return {kHeadDim, (int64_t)table_rows_of(*b.fwd) * kHeadDim};
}

uint64_t align256(uint64_t x) { return (x + 255) & ~uint64_t(255); }

// Heads whose bucket sums are in memory at a time.  The sums are 2 bytes per row, head and table row, by far the largest thing in the
// workspace; heads are independent, so the largest calls go through them in groups of at most this many bytes (131072 rows of 16
// heads and 512 table rows are one group), and the workspace grows with the rows only by what every row needs once.
constexpr uint64_t kSumBytes = uint64_t(1) << 31;
int sum_heads_of(const fdb_attn_params& p) {
  if (p.pos_key == nullptr && p.pos_query == nullptr) return p.heads;  // no sums
  const uint64_t head = uint64_t(p.total_rows) * table_rows_of(p) * 2;
  const uint64_t most = head == 0 ? p.heads : std::max<uint64_t>(1, std::min<uint64_t>(p.heads, kSumBytes / head));
  const int groups = (int)((p.heads + most - 1) / most);
  return (p.heads + groups - 1) / groups;  // groups of about the same size
}

struct Layout { uint64_t seq_info, tile_first, slot_info, delta, table[4], core, sums, partial, total; };

Layout layout_of(const fdb_attn_params& p, const ExpandGeometry& g) {
  Layout l;
  uint64_t off = 0;
  l.seq_info = off;   off = align256(off + uint64_t(p.batch) * 8);
  l.tile_first = off; off = align256(off + uint64_t(p.batch + 1) * 4);
  l.slot_info = off;  off = align256(off + uint64_t(tile_slots(p)) * 16);
  l.delta = off;      off = align256(off + uint64_t(p.total_rows) * p.heads * 4);
  const uint64_t table = uint64_t(p.heads) * g.rows * kHeadDim * 2;
  for (int i = 0; i < 4; ++i) { l.table[i] = off; off = align256(off + ((i & 1) ? (p.pos_query ? table : 0) : (p.pos_key ? table : 0))); }
  // the two sides run one after the other and share these
  const bool terms = p.pos_key != nullptr || p.pos_query != nullptr;
  const int table_rows = table_rows_of(p), group = sum_heads_of(p), rest = p.heads % group;
  l.core = off;    off = align256(off + (terms ? uint64_t(p.total_rows) * p.heads * kHeadDim * 4 : 0));
  l.sums = off;    off = align256(off + (terms ? uint64_t(p.total_rows) * group * table_rows * 2 : 0));
  const uint64_t partial = std::max(bwd_tables_partial_bytes(p.total_rows, group, table_rows),
                                    rest > 0 ? bwd_tables_partial_bytes(p.total_rows, rest, table_rows) : 0);
  l.partial = off; off = align256(off + (terms ? partial : 0));
  l.total = off;
  return l;
}

// Arguments for heads [head0, head0 + heads) of the call.
template <bool DKV>
int make_args(BwdArgs& a, const fdb_attn_bwd_params& b, const ExpandGeometry& g, const Layout& l, char* ws, int head0, int heads) {
  const fdb_attn_params& p = *b.fwd;
  auto at = [&](const void* base, int64_t head_stride) { return static_cast<const __nv_bfloat16*>(base) + head0 * head_stride; };
  auto operand = [&](CUtensorMap* m, const void* base, int64_t rs, int64_t hs, int box) {
    return make_map_rows(m, at(base, hs), p.total_rows, heads, rs, hs, box, false, "backward operand");
  };
  int rc;
  const int row = 128, col = kCols;
  if ((rc = operand(&a.tm_row[0], DKV ? p.k : p.q, DKV ? p.k_row_stride : p.q_row_stride, DKV ? p.k_head_stride : p.q_head_stride, row))) return rc;
  if ((rc = operand(&a.tm_row[1], DKV ? p.v : b.dout, DKV ? p.v_row_stride : b.dout_row_stride, DKV ? p.v_head_stride : b.dout_head_stride, row))) return rc;
  if ((rc = operand(&a.tm_col[0], DKV ? p.q : p.k, DKV ? p.q_row_stride : p.k_row_stride, DKV ? p.q_head_stride : p.k_head_stride, col))) return rc;
  if ((rc = operand(&a.tm_col[1], DKV ? b.dout : p.v, DKV ? b.dout_row_stride : p.v_row_stride, DKV ? b.dout_head_stride : p.v_head_stride, col))) return rc;
  // <true>: the row term is p2c, distances are key - query
  const bool has_row = DKV ? p.pos_query != nullptr : p.pos_key != nullptr, has_col = DKV ? p.pos_key != nullptr : p.pos_query != nullptr;
  a.xrow = has_row ? at(ws + l.table[DKV ? 3 : 0], (int64_t)g.rows * kHeadDim) : nullptr;
  a.xcol = has_col ? at(ws + l.table[DKV ? 2 : 1], (int64_t)g.rows * kHeadDim) : nullptr;
  a.tm_xrow = a.tm_xcol = a.tm_xcol_sat = a.tm_row[0];
  if (has_row && (rc = make_map_table(&a.tm_xrow, a.xrow, g.rows, heads, false, "row table", kWin))) return rc;
  if (has_col && (rc = make_map_table(&a.tm_xcol, a.xcol, g.rows, heads, false, "column table", kWin))) return rc;
  if (has_col && (rc = make_map_table(&a.tm_xcol_sat, a.xcol, g.rows, heads, false, "saturated rows", 8))) return rc;
  a.slot_info = reinterpret_cast<const int4*>(ws + l.slot_info);
  a.lse = p.lse + head0;
  a.delta = reinterpret_cast<const float*>(ws + l.delta) + head0;
  a.core = reinterpret_cast<float*>(ws + l.core) + (int64_t)head0 * kHeadDim;
  a.grad = const_cast<__nv_bfloat16*>(at(DKV ? b.dk : b.dq, b.grad_head_stride));
  a.dv = DKV ? const_cast<__nv_bfloat16*>(at(b.dv, b.grad_head_stride)) : nullptr;
  a.grad_rs = b.grad_row_stride; a.grad_hs = b.grad_head_stride;
  a.sums = reinterpret_cast<__nv_bfloat16*>(ws + l.sums);
  a.lut = p.bucket_lut; a.lut_d_min = p.lut_d_min; a.lut_len = p.lut_len;
  a.table_rows = table_rows_of(p);
  a.status = p.status;
  a.sum_heads = sum_heads_of(p);
  a.heads = p.heads; a.packed = p.cu_seqlens != nullptr; a.max_seqlen = p.max_seqlen; a.total_rows = p.total_rows;
  a.sat_lo = DKV ? -g.sat_hi : g.sat_lo;
  a.sat_hi = DKV ? -g.sat_lo : g.sat_hi;
  a.d_first = a.sat_lo - 254;
  a.xrows = g.rows;
  a.sm_scale = p.sm_scale;
  return FDB_OK;
}

// One side for all heads, from the arguments of the first group of them.
template <bool DKV>
int launch_bwd(BwdArgs a, const fdb_attn_bwd_params& b, const ExpandGeometry& g, const Layout& l, char* ws, int64_t slots, cudaStream_t stream) {
  const fdb_attn_params& p = *b.fwd;
  static std::atomic<uint64_t> smem_done{0};
  auto kernel = bwd_kernel<DKV>;
  cudaError_t e = allow_smem(smem_done, reinterpret_cast<const void*>(kernel), (int)kSmemBytes);
  int rc = FDB_OK;
  for (int head0 = 0, heads; head0 < p.heads; head0 += heads) {
    heads = std::min(a.sum_heads, p.heads - head0);
    if (head0 > 0 && (rc = make_args<DKV>(a, b, g, l, ws, head0, heads)) != FDB_OK) return rc;
    if (e == cudaSuccess && slots > 0) e = launch_kernel<BwdArgs>(kernel, a, dim3((unsigned)slots, heads), kThreads, kSmemBytes, false, stream);
    if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "attn_bwd launch: %s", cudaGetErrorString(e));
    if (a.xrow == nullptr) continue;
    auto at = [&](const void* base, int64_t head_stride) { return static_cast<const __nv_bfloat16*>(base) + head0 * head_stride; };
    BwdTablesCall c;
    c.sums = a.sums;
    const TableStrides strides = table_strides(b);
    c.table = at(DKV ? p.pos_query : p.pos_key, strides.head);
    c.table_row_stride = strides.row; c.table_head_stride = strides.head;
    c.operand_row_stride = DKV ? p.k_row_stride : p.q_row_stride;
    c.operand_head_stride = DKV ? p.k_head_stride : p.q_head_stride;
    c.operand = at(DKV ? p.k : p.q, c.operand_head_stride);
    c.core = a.core;
    c.core_row_stride = (int64_t)p.heads * kHeadDim;
    c.out = a.grad;
    c.out_row_stride = a.grad_rs; c.out_head_stride = a.grad_hs;
    c.dtable = const_cast<__nv_bfloat16*>(at(DKV ? b.dpos_query : b.dpos_key, strides.head));
    c.partial = reinterpret_cast<float*>(ws + l.partial);
    c.rows = p.total_rows; c.heads = heads; c.table_rows = a.table_rows;
    c.status = p.status;
    if ((rc = launch_bwd_tables(c, stream)) != FDB_OK) return rc;
  }
  return FDB_OK;
}

int check_bwd(const fdb_attn_bwd_params* b, ExpandGeometry* g) {
  if (b == nullptr || b->struct_bytes != sizeof(fdb_attn_bwd_params))
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_attn_bwd_params: NULL or struct_bytes %u != %zu", b ? b->struct_bytes : 0u, sizeof(fdb_attn_bwd_params));
  const int rc = validate(b->fwd, true);
  if (rc != FDB_OK) return rc;
  const fdb_attn_params& p = *b->fwd;
  if (p.dtype != FDB_BF16) return fail(FDB_ERR_UNSUPPORTED, "fdb_attn_bwd takes bf16 tensors");
  *g = {0, 0, 0, 0};
  if (p.pos_key != nullptr || p.pos_query != nullptr) {
    *g = expand_geometry(p.lut_d_min, p.lut_len);
    const int span = p.position_buckets > 0 ? p.position_buckets : p.max_relative_positions;
    if (span % 4 != 0) return fail(FDB_ERR_UNSUPPORTED, "fdb_attn_bwd: att_span %d is not a multiple of 4", span);
    if (g->rows > kMaxRows) return fail(FDB_ERR_LIMIT, "fdb_attn_bwd: bucket table of %d entries (at most %d)", p.lut_len, kMaxRows - 508);
  }
  return FDB_OK;
}

}  // namespace
}  // namespace fdb

using namespace fdb;

extern "C" FDB_API uint64_t fdb_attn_bwd_workspace_bytes(const fdb_attn_bwd_params* b) {
  clear_error();
  ExpandGeometry g;
  if (check_bwd(b, &g) != FDB_OK) return 0;
  return layout_of(*b->fwd, g).total;
}

extern "C" FDB_API int fdb_attn_bwd(const fdb_attn_bwd_params* b, void* stream) {
  clear_error();
  ExpandGeometry g;
  int rc = check_bwd(b, &g);
  if (rc != FDB_OK) return rc;
  const fdb_attn_params& p = *b->fwd;
  if (p.total_rows == 0) {  // nothing but the tables' gradients to write
    const TableStrides strides = table_strides(*b);
    for (void* d : {b->dpos_key, b->dpos_query})
      if (d != nullptr && (rc = launch_zero_table(d, strides.row, strides.head, p.heads, table_rows_of(p), static_cast<cudaStream_t>(stream))) != FDB_OK) return rc;
    return FDB_OK;
  }
  if (b->dout == nullptr || p.lse == nullptr || b->dq == nullptr || b->dk == nullptr || b->dv == nullptr ||
      (p.pos_key != nullptr) != (b->dpos_key != nullptr) || (p.pos_query != nullptr) != (b->dpos_query != nullptr))
    return fail(FDB_ERR_INVALID_ARGUMENT, "fdb_attn_bwd: dout, lse, dq, dk, dv and the gradient of every position table are required");
  const uintptr_t all = (uintptr_t)b->dout | (uintptr_t)b->dq | (uintptr_t)b->dk | (uintptr_t)b->dv | (uintptr_t)b->dpos_key | (uintptr_t)b->dpos_query;
  const int64_t strides[4] = {b->dout_row_stride, b->dout_head_stride, b->grad_row_stride, b->grad_head_stride};
  bool aligned = (all & 15u) == 0;
  for (int64_t s : strides) aligned = aligned && s > 0 && s % 8 == 0;
  aligned = aligned && b->table_row_stride >= 0 && b->table_row_stride % 8 == 0 && (b->table_row_stride == 0 || b->table_head_stride > 0) && b->table_head_stride % 8 == 0;
  if (!aligned) return fail(FDB_ERR_ALIGNMENT, "fdb_attn_bwd: pointers must be 16-byte aligned, strides positive multiples of 8 elements");
  const Layout l = layout_of(p, g);
  if (b->workspace == nullptr || b->workspace_bytes < l.total)
    return fail(FDB_ERR_WORKSPACE, "workspace of %llu bytes needed, %llu given", (unsigned long long)l.total, (unsigned long long)b->workspace_bytes);
  if ((reinterpret_cast<uintptr_t>(b->workspace) & 255u) != 0) return fail(FDB_ERR_ALIGNMENT, "workspace must be 256-byte aligned");
  const int64_t slots = tile_slots(p);  // none when no sequence is given: every row is outside then
  if (slots > 2147483647LL || p.heads > 65535) return fail(FDB_ERR_LIMIT, "grid too large");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  char* ws = static_cast<char*>(b->workspace);
  AttnBuffers buf = {};
  buf.seq_info = reinterpret_cast<int32_t*>(ws + l.seq_info);
  buf.tile_first = reinterpret_cast<int32_t*>(ws + l.tile_first);
  buf.slot_info = reinterpret_cast<int32_t*>(ws + l.slot_info);
  if (slots > 0 && (rc = launch_seq_info(p, buf, stream)) != FDB_OK) return rc;
  BwdArgs dq, dkv;
  const int first = sum_heads_of(p);  // (the heads of a group; all of them but in the largest calls)
  if ((rc = make_args<false>(dq, *b, g, l, ws, 0, first)) != FDB_OK || (rc = make_args<true>(dkv, *b, g, l, ws, 0, first)) != FDB_OK) return rc;
  if (p.pos_key != nullptr || p.pos_query != nullptr) {
    const int64_t n = (int64_t)p.heads * g.rows * 8;
    const TableStrides strides = table_strides(*b);
    auto table = [&](int i) { return reinterpret_cast<uint4*>(ws + l.table[i]); };
    bwd_expand_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(static_cast<const uint4*>(p.pos_key), static_cast<const uint4*>(p.pos_query),
                                                                 table(0), table(1), table(2), table(3), p.bucket_lut, p.lut_len, g.rows, p.heads,
                                                                 strides.row / 8, strides.head / 8);
  }
  const int64_t cells = (int64_t)p.total_rows * p.heads;
  bwd_delta_kernel<<<(unsigned)((cells * 8 + 255) / 256), 256, 0, s>>>(
      static_cast<const __nv_bfloat16*>(b->dout), b->dout_row_stride, b->dout_head_stride, static_cast<const __nv_bfloat16*>(p.out),
      p.out_row_stride, p.out_head_stride, cells, p.heads, reinterpret_cast<float*>(ws + l.delta), p.cu_seqlens, p.batch, dq, dkv);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "attn_bwd set-up: %s", cudaGetErrorString(e));
  if ((rc = launch_bwd<false>(dq, *b, g, l, ws, slots, s)) != FDB_OK) return rc;
  return launch_bwd<true>(dkv, *b, g, l, ws, slots, s);
}
