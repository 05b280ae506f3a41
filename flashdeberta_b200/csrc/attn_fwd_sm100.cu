// Fused DeBERTa disentangled-attention forward for sm_100a — warp-specialised kernel.
//
// Replaces the reference's Triton forward kernels (src/flashdeberta/ops/flash_attention.py:146-300 and
// src/flashdeberta/ops/flash_attention_varlen.py:85-225) and the two bias GEMMs in front of them
// (src/flashdeberta/model.py:189-192, :210-214).
//
// Work item = one 128-row query tile of one (sequence, head) = one block of the grid; a CTA (one per SM) does its own and then takes
// blocks over that have not started (cluster launch control), in the grid's order, heaviest tiles first.  16 warps in four
// warpgroups (registers move from the producer and drain groups to the softmax groups with setmaxnreg):
//   warps 0-3   softmax group 0: thread r owns row r of the tile, keys   0..63  of every 128-key tile
//   warps 4-7   softmax group 1: thread r owns row r of the tile, keys  64..127
//   warp  8     score-side tcgen05.mma: S = Q.K^T and the position products (the warp allocates TMEM)
//   warp  9     every TMA load: Q once, K/V double-buffered, position-table windows; asks for further work items
//   warp  10    O += P.V
//   warp  11    saturated c2p terms (one dot product per row and side)
//               (8-10 stay converged and issue through an elected lane: see elect_one)
//   warps 12-15 drain group: moves the c2p product of a band tile from tensor memory to shared memory (bf16)
// Tensor memory (512 columns): O 64 | P 64 | S 128 | R 256 (position products of a band tile).
//
// Per key tile j:  S = Q.K^T (tensor core, fp32 in TMEM)  ->  both softmax groups pull their half of S (and of the p2c
// product) into registers and release S and R at once, so the tensor core computes the scores of tile j+1 while the
// softmax of tile j runs  ->  the groups agree on the row maximum through shared memory, write P = exp2(...) as bf16 pairs
// into the P columns  ->  O += P.V with P read from tensor memory and V from shared memory.  O stays in TMEM and is
// rescaled only when the running maximum moved by more than 2^8.
//
// Position terms (tables arrive expanded through the bucket function, see attn_prepare.cu; row of (m, n) is (m-n)-d_first):
//   * saturated tile pair (all distances beyond a saturation point): c2p is one dot product per query row, folded into the
//     row's exponent offset; p2c is one dot product per key, accumulated into S on the tensor core as R.K^T where all rows
//     of R equal the saturated pos_query row (R is 8 rows of shared memory read with a zero group stride);
//   * band tile pair: p2c comes from products X_q[32(3-b+t) .. +128).K[32b .. +32)^T, b = key block, t = 0/1 (issued as three
//     128x64 and two 128x32 MMAs groups), arranged so that the value thread (quadrant w, lane l) needs for key 32b+c sits in
//     its own quadrant at lane (l+31-c)&31 of product t = (l > c): one select on the source side and one warp shuffle per
//     score element, fp32, no shared memory;
//     c2p needs a shift by the row: Q.X_k[window]^T goes through tensor memory to the drain group while the softmax of the previous
//     tile is still running; the group writes row m of it to shared memory as bf16, rotated by m, and thread m reads its 64 values
//     as one aligned run.
// No (rows x 2*span) bias tensor is ever written to global memory.
//
// What a band tile costs, 8 x 2048 x 12 heads, clocks of 4500: the two products of p2c pulled and shuffled 1200, c2p added and the
// maximum 810, its exchange and the decision 350, 64 exponentials per thread 1300, hops between the roles the rest; beside it the
// products of the next tile (20 narrow p2c MMAs 900, drain 1250).  Neither side hides the other wholly: of this kernel with one part
// left out, the exponentials were worth 10 % of a call, selects and shuffles 7 %, c2p 3 %, the drain's stores 2 to 3 %, the p2c MMAs
// and the windows' loads nothing.  Hence shuffle sources in registers, c2p added by the mixed-precision add (no unpacking), stores of
// the drain at fixed distances from two bases, a stage pitch with fewer bank conflicts, and waits that are over by then in front
// of the ones that are not: 364 -> 353 us a call at this shape, 168 -> 164 at 32 x 512, packed 48 x <= 4099 x 16 heads 1431 -> 1393.
//
// Every mbarrier wait is bounded and gives up early once another role has raised the abort flag; the CTA then sets
// FDB_DEV_TIMEOUT in the status word, waits a millisecond for copies in flight, releases its TMEM and returns.
// No TMA load uses multicast.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "internal.h"
#include "launch.h"
#include "sm100_ptx.cuh"
#include "tensor_map.cuh"
#include "attn_fwd_common.cuh"

namespace fdb {
namespace {

using namespace ptx;
using namespace fwd;

constexpr int kSoftmaxThreads = 256;
constexpr int kDrainThreads = 128;
constexpr int kThreads = 512;            // four warpgroups: softmax 0, softmax 1, warps 8-11 (issue and saturated terms), drain
constexpr int kMmaWarp = 8, kTmaWarp = 9, kPvWarp = 10, kSatWarp = 11, kDrainWarp0 = 12;
// 128 registers per thread at launch; after setmaxnreg: 48 * 128 + 64 * 128 + 200 * 256 = 65536
constexpr int kProducerRegs = 48, kDrainRegs = 64, kSoftmaxRegs = 200;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColO = 0;     // 64 columns: output accumulator
constexpr uint32_t kColP = 64;    // 64 columns: P as bf16 pairs (keys 0..63 in the first 32, keys 64..127 in the last 32)
constexpr uint32_t kColS = 128;   // 128 columns: scores
constexpr uint32_t kColR = 256;   // 256 columns: position products of a band tile

// shared memory map (bytes from a 1024-aligned base)
constexpr uint32_t kSmemQ = 0;                      // 128 x 128 B
constexpr uint32_t kSmemK = 16384;                  // 2 stages
constexpr uint32_t kSmemV = 49152;                  // 2 stages
constexpr uint32_t kSmemWinK = 81920;               // 256 x 128 B window of expanded pos_key
constexpr uint32_t kSmemWinQ = 114688;              // 256 x 128 B window of expanded pos_query
// c2p stage: bf16 [128 query rows][256 window positions], rows padded by 48 B.  Row m is rotated by m: position p of the
// window sits in column (p - m) & 255, so the 64 values a softmax thread needs are one aligned 128-byte run whose place does
// not depend on m.
// A pitch of 140 words: 16-byte loads of eight rows meet in no bank.  The drain group's 4-byte stores (row r of a warp in bank
// 12 r - ceil(r / 2)) do in three pairs of the 32 rows, a second wavefront each; at 132 words it was eleven pairs.
constexpr uint32_t kStageCPitch = 560;
constexpr uint32_t kSmemStageC = 147456;
constexpr uint32_t kSmemSat = kSmemStageC + 71680;  // 2 x (8 x 128 B) saturated pos_query rows (hi, lo)
static_assert(128 * kStageCPitch <= 71680, "c2p stage");
constexpr uint32_t kSmemXchg = kSmemSat + 2048;     // float [2 parities][2 groups][128 rows] row maxima
constexpr uint32_t kSmemLsum = kSmemXchg + 2048;    // float [2 groups][128 rows] row sums at the end
constexpr uint32_t kSmemRc = kSmemLsum + 1024;      // float [2 items][hi, lo][128 rows] saturated c2p terms
constexpr uint32_t kSmemItem = kSmemRc + 2048;      // 16 B answer to a request for another block; 2 x 32 B work items
constexpr uint32_t kSmemBars = kSmemItem + 96;
constexpr uint32_t kSmemBytes = kSmemBars + 256 + 1024;  // + alignment slack
static_assert(kSmemSat % 1024 == 0, "shared memory map");
static_assert(kSmemBytes <= 232448, "exceeds 227 KB");

// mbarriers.  "count" = arrivals per phase.
enum Bar : uint32_t {
  kBarQ = 0,         // 1   Q (and the saturated pos_query rows of the head) landed (TMA)
  kBarK = 1,         // 1   K stage s landed (TMA), 2 stages
  kBarV = 3,         // 1   V stage s landed (TMA), 2 stages
  kBarKFree = 5,     // 1   the MMAs that read K stage s finished (tcgen05.commit)
  kBarVFree = 7,     // 1   the P.V that read V stage s finished
  kBarWin = 9,       // 1   position windows landed (TMA)
  kBarWinFree = 10,  // 1   the MMAs that read the windows finished
  kBarS = 11,        // 1   S (and the p2c product) of a tile are in tensor memory
  kBarSFree = 12,    // 8   both softmax groups hold their scores in registers: S and R may be overwritten
  kBarP = 13,        // 8   P of a tile is in tensor memory
  kBarO = 14,        // 1   P.V of a tile finished
  kBarC2p = 15,      // 1   the c2p product of a band tile is in R
  kBarStage = 16,    // 4   the drain group has written the c2p stage (R may be overwritten, the stage may be read)
  kBarGather = 17,   // 8   both softmax groups are done reading the c2p stage
  kBarQFree = 18,    // 1   the MMAs that read Q (and the saturated rows) of an item finished
  kBarRc = 19,       // 1   the saturated c2p terms of an item are in buffer s (Q has been read for them), 2 buffers: with items of one
                     //     tile the next item's are there before the softmax groups look for these
  kBarAnswer = 21,   // 1   the answer to a request for another block is there
  kBarItem = 22,     // 1   work item in slot s, 2 slots
  kBarItemFree = 24, // 15  every other role has read it
  kNumBars = 26
};
constexpr uint32_t kItemReaders = 15;  // softmax 8, drain 4, score, P.V, saturated terms

// One work item: a query tile of one (sequence, head) and the key tiles that this launch gives it.
struct Item {
  int seq, m0, row0, len, head;
  int j_first, n_proc;  // key tiles j_first .. j_first + n_proc - 1; none: an empty slot or a padding tile
  bool resume;          // the far kernel has left a partial result for this tile
};
__device__ __forceinline__ Item make_item(const FwdArgs& args, int4 slot, uint32_t head) {
  Item it;
  it.seq = (int)uniform(slot.x); it.m0 = (int)uniform(slot.y); it.row0 = (int)uniform(slot.z); it.len = (int)uniform(slot.w);
  it.head = (int)uniform(head);
  it.j_first = it.n_proc = 0;
  it.resume = false;
  if (it.seq < 0 || it.m0 >= it.len) return it;  // a slot behind the last sequence, a dense padding tile
  // key tiles this launch works on: all of them, or (split launch) the contiguous run of band tiles
  const int num_kt = (it.len + kTileN - 1) / kTileN;
  it.n_proc = num_kt;
  if (args.band_only && it.len >= args.split_len) band_run(it.m0, num_kt, args.sat_lo, args.sat_hi, it.j_first, it.n_proc);
  it.resume = args.band_only && it.n_proc < num_kt;
  return it;
}

template <bool F8>
__global__ void __launch_bounds__(kThreads, 1) attn_fwd_kernel(const __grid_constant__ FwdArgs args) {
  using G = Geo<F8>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = (int)uniform(uint32_t(tid) >> 5), lane = tid & 31;
  grid_launch();
  grid_wait();
  const bool has_c2p = args.xk != nullptr, has_p2c = args.xq != nullptr;
  const bool has_pos = has_c2p || has_p2c;
  auto tile_kind = [&](const Item& it, int j) -> int {
    if (!has_pos) return kPlain;
    const int d0 = it.m0 - j * kTileN - (kTileN - 1);  // smallest distance of the pair; the largest is d0 + 254
    return d0 >= args.sat_hi ? kSatHi : (d0 + 254 <= args.sat_lo ? kSatLo : kBand);
  };

  auto bar = [&](uint32_t i) -> uint32_t { return smem + kSmemBars + 8u * i; };
  const uint32_t tmem_slot = smem + kSmemBars + 8u * kNumBars;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + kSmemBars + 8u * kNumBars + 8u);
  volatile uint32_t* handed_out = abort_flag + 1;  // items handed from role to role, plus one; 0 until the last one was

  // ---- set-up ---------------------------------------------------------------------------------------------------------
  if (tid == 0) {
    *abort_flag = *handed_out = 0u;
    for (uint32_t i = 0; i < kNumBars; ++i) {
      uint32_t count = 1u;
      if (i == kBarSFree || i == kBarP || i == kBarGather) count = kSoftmaxThreads / 32;  // one arrival per warp
      if (i == kBarItemFree || i == kBarItemFree + 1) count = kItemReaders;
      if (i == kBarStage) count = kDrainThreads / 32;
      mbar_init(bar(i), count);
    }
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
  auto wait = [&](uint32_t b, uint32_t parity) {  // whole warps wait, the result is warp-uniform
    if (ok) ok = mbar_wait_warp(b, parity, abort_flag);
  };
  auto arrive = [&](uint32_t b) {  // one arrival per warp
    __syncwarp();
    if (elect_one()) mbar_arrive(b);
  };

  auto has_saturated = [&](const Item& it) -> bool {  // (the band tiles are one run)
    return tile_kind(it, it.j_first) != kBand || tile_kind(it, it.j_first + it.n_proc - 1) != kBand;
  };

  // ---- work items ------------------------------------------------------------------------------------------------------
  // The CTA stays on its SM and takes further blocks of the grid over (cluster launch control): the roles run ahead of one another
  // across the border between two items, so the set-up, the first loads, the first c2p blocks and their drain of an item lie
  // under the last tile and the output of the item before.  As blocks of their own, one behind the other because an SM's tensor memory
  // and shared memory hold one, those took 11 700 clocks an item beside 4500 per band tile; what is left between two items is 3000.
  // 353 -> 336 us a call at 8 x 2048 x 12 heads, 164 -> 132 at 32 x 512, padded 24 x <= 779 124 -> 110, packed 48 x <= 4099 x 16
  // 1393 -> 1310.  Every count below that a barrier's phase depends on runs on from item to item.
  // The TMA warp asks and hands the items on, worked out: what the other roles execute between two items is code that the
  // tiles' loops have pushed out of the instruction cache, so there is little of it.
  uint32_t taken = 0;
  auto wait_item = [&]() { wait(bar(kBarItem + (taken & 1u)), (taken >> 1) & 1u); };
  auto read_item = [&](Item& it) -> bool {
    const uint32_t slot = taken & 1u, at = smem + kSmemItem + 32u + 32u * slot;
    ++taken;
    const uint4 what = lds_v4(at);
    const uint4 rest = lds_v4(at + 16u);
    arrive(bar(kBarItemFree + slot));
    it.seq = (int)uniform(what.x); it.m0 = (int)uniform(what.y); it.row0 = (int)uniform(what.z); it.len = (int)uniform(what.w);
    it.head = (int)uniform(rest.x); it.j_first = (int)uniform(rest.y); it.n_proc = (int)uniform(rest.z);
    const uint32_t flags = uniform(rest.w);
    it.resume = (flags & 2u) != 0u;
    return (flags & 1u) != 0u;
  };
  auto next_item = [&](Item& it) -> bool {
    wait_item();
    return ok && read_item(it);
  };
  // The softmax warps meet at named barriers, which have no limit of their own and count on every warp.  So they work on the same items,
  // whichever of them gave up on a wait: such a warp goes on without waiting and without results and takes every item that was handed out.
  // How many those are is known once the TMA warp has left its loop, which it does at the first wait that it gives up itself.  (A vote
  // of the eight warps between two items does the same for 2 % of a call with items of one tile.)
  auto next_item_of_all = [&](Item& it) -> bool {
    wait_item();
    if (!ok) {
      uint32_t n = 0;
#pragma unroll 1
      for (uint32_t i = 0; i < (1u << 28) && n == 0u; ++i) n = uniform(*handed_out);
      __threadfence_block();
      if (taken + 1u >= n) return false;
    }
    return read_item(it);
  };
  // (sequence, first row of the tile in it, its first row, its length)
  Item it = make_item(args, __ldg(args.slot_info + blockIdx.x), blockIdx.y);

  if (warp >= kDrainWarp0) {
    // =================================================== drain group ====================================================
    reg_dealloc<kDrainRegs>();
    const int quad = warp & 3;
    const int r = quad * 32 + lane;  // TMEM lane = position row inside a 128-position block
    const uint32_t tmem_lane = tmem_base + (uint32_t(quad * 32) << 16);
    uint32_t bands = 0;  // band tiles of all items so far
    bool first_item = true;
    do {
    uint32_t band_idx = 0;
    for (int jj = 0; jj < it.n_proc; ++jj) {
      const int j = it.j_first + jj;
      if (tile_kind(it, j) != kBand) continue;
      if (bands > 0) wait(bar(kBarGather), (bands - 1u) & 1u);   // nobody reads the previous stage any more
      wait(bar(kBarC2p), bands & 1u);                            // the product is there
      const bool c2p_outside_r = first_item && jj == 0 && !it.resume;
      tc_fence_after();
      if (has_c2p && ok) {
        // The product has query rows in the lanes and window positions in the columns, so this thread holds row r.  The
        // windows of consecutive band tiles overlap by half: only the first tile of the run brings 256 positions, every
        // later one the 128 new ones (block 0), written over the half of the stage the new window no longer covers:
        // position p of the current window is "physical" position p ^ flip, stored in column (physical - r) & 255.
        const int nblk = band_idx == 0 ? 2 : 1;
        const uint32_t flip = (band_idx & 1u) ? 128u : 0u;
        const uint32_t row_addr = smem + kSmemStageC + uint32_t(r) * kStageCPitch;
#pragma unroll 1
        for (int blk = 0; blk < nblk; ++blk) {
          // where the score-issuing warp put the block (see there)
          const uint32_t col = tmem_lane + (band_idx > 0 ? kColS : (c2p_outside_r ? (blk == 0 ? kColS : kColO) : kColR + blk * 128));
          const uint32_t start = ((uint32_t(blk) * 128u) ^ flip) - uint32_t(r);  // column of the block's first position (mod 256)
          // an odd start puts value 2k-1 and 2k into one 32-bit word: funnel shift over consecutive pairs by 16 bits;
          // an even start keeps the pairs (shift "32" = take the upper word)
          const uint32_t sh = (start & 1u) ? 16u : 32u;
          const int w0 = int((start & 255u) >> 1);  // word of the block's first value; the row wraps behind word 127
          uint32_t prev = 0;
          uint32_t t[32];
          tmem_ld32(col, t);
          tmem_wait_ld();
#pragma unroll 1  // kept rolled: this loop runs beside the softmax warps, whose unrolled code already fills the instruction cache
          for (int c4 = 0; c4 < 4; ++c4) {
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(__uint_as_float(t[2 * i]), __uint_as_float(t[2 * i + 1]));
            if (c4 < 3) tmem_ld32(col + (c4 + 1) * 32, t);  // the next 32 columns are in flight while these are stored
            // 16 words at a fixed distance from one of two bases: in front of the wrap and behind it
            const int front = 128 - (w0 + 16 * c4);
            const uint32_t to = row_addr + 4u * uint32_t(w0 + 16 * c4), to_wrapped = to - 512u;
            if (c4 == 0 && (start & 1u)) {
              // the low half of the first word belongs to the other block's last position: write the upper half only
              sts_u16(to + 2u, pk[0] & 0xffffu);
            } else {
              sts_u32(front > 0 ? to : to_wrapped, __funnelshift_rc(prev, pk[0], sh));
            }
#pragma unroll
            for (int k = 1; k < 16; ++k) sts_u32((k < front ? to : to_wrapped) + 4u * uint32_t(k), __funnelshift_rc(pk[k - 1], pk[k], sh));
            prev = pk[15];
            if (c4 < 3) tmem_wait_ld();
          }
          if (start & 1u) sts_u16(row_addr + 4u * (((start + 128u) >> 1) & 127u), prev >> 16);  // the block's last value
        }
      }
      tc_fence_before();
      arrive(bar(kBarStage));
      ++band_idx;
      ++bands;
    }
    if (it.n_proc > 0) first_item = false;
    } while (next_item(it));
  } else if (warp >= kMmaWarp) {
    reg_dealloc<kProducerRegs>();
    if (warp == kTmaWarp) {
      // ================================================= TMA producer ===================================================
      if (elect_one()) { tma_prefetch_desc(&args.tm_q); tma_prefetch_desc(&args.tm_k); tma_prefetch_desc(&args.tm_v); }
      uint32_t items = 0, tiles = 0, bands = 0, asked = 0;
      bool more = false;
      do {
      if (it.n_proc > 0) {
        if (items > 0) {
          wait(bar(kBarQFree), (items - 1u) & 1u);
          wait(bar(kBarRc + ((items - 1u) & 1u)), ((items - 1u) >> 1) & 1u);
        }
        ++items;
      }
      if (ok && it.n_proc > 0 && elect_one()) {
        mbar_expect_tx(bar(kBarQ), G::kTile + (has_p2c ? 16u * G::kRow : 0u));
        tma_load_3d(smem + kSmemQ, &args.tm_q, bar(kBarQ), 0, it.head, it.row0 + it.m0);
        if (has_p2c) {
          // Saturated pos_query rows as MMA operands: the last (first) eight rows of an expanded table are all the row of
          // distances beyond sat_hi (sat_lo), so an 8-row box is the 8 identical rows in the swizzled layout.
          tma_load_3d(smem + kSmemSat, &args.tm_xq_sat, bar(kBarQ), 0, args.xrows - 8, it.head);
          tma_load_3d(smem + kSmemSat + 1024, &args.tm_xq_sat, bar(kBarQ), 0, 0, it.head);
        }
      }
      uint32_t band_idx = 0;
#pragma unroll 1
      for (int jj = 0; jj < it.n_proc && ok; ++jj) {
        const int j = it.j_first + jj;
        const uint32_t s = tiles & 1u, use = tiles >> 1;  // how often this stage was used before
        FDB_STAMP(asked, 3, j, 0);
        if (use > 0) wait(bar(kBarKFree + s), (use - 1u) & 1u);
        if (!ok) break;
        FDB_STAMP(asked, 3, j, 1);
        if (elect_one()) {
          mbar_expect_tx(bar(kBarK + s), G::kTile);
          tma_load_3d(smem + kSmemK + s * 16384, &args.tm_k, bar(kBarK + s), 0, it.head, it.row0 + j * kTileN);
        }
        if (tile_kind(it, j) == kBand) {
          if (bands > 0) wait(bar(kBarWinFree), (bands - 1u) & 1u);
          if (!ok) break;
          const int u0 = it.m0 - j * kTileN - (kTileN - 1) - args.d_first;
          if (elect_one()) {
            // (of pos_key the first tile of the run takes the whole window, the others its 128 new rows)
            mbar_expect_tx(bar(kBarWin), (has_c2p ? (band_idx == 0 ? G::kWin : G::kTile) : 0u) + (has_p2c ? G::kWin : 0u));
            if (has_c2p) tma_load_3d(smem + kSmemWinK, &args.tm_xk, bar(kBarWin), 0, u0, it.head);
            if (has_c2p && band_idx == 0) tma_load_3d(smem + kSmemWinK + G::kTile, &args.tm_xk, bar(kBarWin), 0, u0 + 128, it.head);
            if (has_p2c) tma_load_3d(smem + kSmemWinQ, &args.tm_xq, bar(kBarWin), 0, u0, it.head);
          }
          ++band_idx;
          ++bands;
        }
        if (use > 0) wait(bar(kBarVFree + s), (use - 1u) & 1u);
        if (!ok) break;
        FDB_STAMP(asked, 3, j, 2);
        if (elect_one()) {
          mbar_expect_tx(bar(kBarV + s), G::kTile);
          tma_load_3d(smem + kSmemV + s * 16384, &args.tm_v, bar(kBarV + s), 0, it.head, it.row0 + j * kTileN);
        }
        ++tiles;
      }
        // another item: asked for when this one is on its way (asked for at its start, the items at the end of a launch would go to
        // whoever started early, not to whoever is done first)
        if (ok && elect_one()) {
          mbar_expect_tx(bar(kBarAnswer), 16u);
          launch_take_over(smem + kSmemItem, bar(kBarAnswer));
        }
        wait(bar(kBarAnswer), asked & 1u);
        if (!ok) break;
        uint32_t x, y;
        more = launch_taken_over(smem + kSmemItem, x, y);
        fence_proxy_async();  // (the answer is written through the asynchronous proxy again)
        const uint32_t slot = asked & 1u, at = smem + kSmemItem + 32u + 32u * slot;
        it = make_item(args, __ldg(args.slot_info + (more ? x : 0u)), y);
        if (asked >= 2) wait(bar(kBarItemFree + slot), ((asked >> 1) - 1u) & 1u);
        if (!ok) break;  // (somebody may still be reading it)
        if (elect_one()) {
          sts_v4(at, (uint32_t)it.seq, (uint32_t)it.m0, (uint32_t)it.row0, (uint32_t)it.len);
          sts_v4(at + 16u, (uint32_t)it.head, (uint32_t)it.j_first, (uint32_t)it.n_proc, (more ? 1u : 0u) | (it.resume ? 2u : 0u));
          mbar_arrive(bar(kBarItem + slot));
        }
        ++asked;
      } while (more);
      __syncwarp();
      __threadfence_block();
      if (elect_one()) *handed_out = asked + 1u;
    } else if (warp == kSatWarp) {
      // ============================================= saturated c2p terms ================================================
      // Q[m].X_k[first row] and Q[m].X_k[last row] of the item's rows, for its saturated tiles.  (The buffer of the item before the last
      // is free: Q of this one is loaded once the scores of the last one's last tile exist.)
      uint32_t items = 0;
      do {
        if (it.n_proc == 0) continue;
        wait(bar(kBarQ), items & 1u);
        if (has_c2p && ok && has_saturated(it)) {
          const uint32_t rc = smem + kSmemRc + 1024u * (items & 1u);
          const uint8_t* x = static_cast<const uint8_t*>(args.xk) + (int64_t)it.head * args.xrows * G::kRow;
          float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
          auto chunk = [&](int c, const uint8_t* row) { return __ldg(reinterpret_cast<const uint4*>(row) + c); };
          const uint8_t* x_last = x + (int64_t)(args.xrows - 1) * G::kRow;
          uint4 first = chunk(0, x), last = chunk(0, x_last);
#pragma unroll 1
          for (int c = 0; c < (int)G::kRow / 16; ++c) {
            const int next = min(c + 1, (int)G::kRow / 16 - 1);
            const uint4 first_n = chunk(next, x), last_n = chunk(next, x_last);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int r = 32 * i + lane;
              const uint4 a = lds_v4(smem + kSmemQ + uint32_t(r) * G::kRow + (uint32_t(F8 ? c ^ ((r >> 1) & 3) : c ^ (r & 7)) << 4));
              lo[i] = F8 ? dot_f8(a, first, lo[i]) : dot_bf16(a, first, lo[i]);
              hi[i] = F8 ? dot_f8(a, last, hi[i]) : dot_bf16(a, last, hi[i]);
            }
            first = first_n;
            last = last_n;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sts_f32(rc + 4u * uint32_t(32 * i + lane), hi[i]);
            sts_f32(rc + 512u + 4u * uint32_t(32 * i + lane), lo[i]);
          }
        }
        arrive(bar(kBarRc + (items & 1u)));
        ++items;
      } while (next_item(it));
    } else if (warp == kMmaWarp) {
      // ================================================= score MMA issuer ===============================================
      // S = Q.K^T (+ saturated p2c) and the position products of band tiles.  Descriptors are built once; per MMA only the
      // start-address field moves (a 64-bit add), which keeps the single issuing thread short of instructions.
      const uint32_t idesc_s = instr_desc(128, 128, G::kFmt, 0, 0);
      const uint32_t idesc_p2c = instr_desc(128, 32, G::kFmt, 0, 0);
      const uint32_t idesc_p2c64 = instr_desc(128, 64, G::kFmt, 0, 0);
      const uint64_t dq = G::desc(smem + kSmemQ, G::kGroup);
      const uint64_t dk0 = G::desc(smem + kSmemK, G::kGroup);
      const uint64_t dwk = G::desc(smem + kSmemWinK, G::kGroup);
      const uint64_t dwq = G::desc(smem + kSmemWinQ, G::kGroup);
      const uint64_t dsat = G::desc(smem + kSmemSat, 0);  // group stride 0: every 8-row group is the same rows
      uint32_t items = 0, tiles = 0, bands = 0;
      do {
      int band_idx = 0;
      // When the CTA's very first key tile is a band tile, the output and P columns are still unused: the two c2p blocks of
      // that tile go to the S columns and to O|P instead of R, so its p2c products need not wait for the drain group.
      const bool c2p_outside_r = items == 0 && !it.resume && it.n_proc > 0 && tile_kind(it, it.j_first) == kBand;
      if (it.n_proc > 0) {
        wait(bar(kBarQ), items & 1u);
        ++items;
      }
#pragma unroll 1
      for (int jj = 0; jj < it.n_proc; ++jj) {
        const int j = it.j_first + jj;
        const int kind = tile_kind(it, j);
        const uint32_t s = tiles & 1u;
        const uint64_t dk = dk0 + uint64_t(s) * (16384u >> 4);  // stages are 16 KB apart in either build
        wait(bar(kBarK + s), (tiles >> 1) & 1u);
        if (kind == kBand) wait(bar(kBarWin), bands & 1u);
        // both softmax groups hold the tile before in registers: S and R are free
        if (tiles > 0) wait(bar(kBarSFree), (tiles - 1u) & 1u);
        if (kind == kBand) {
          tc_fence_after();
          // Order of issue.  First band tile of the run: c2p (two 128-position blocks) -> R, scores -> S, and once the
          // drain group has emptied R, the p2c products -> R.  Later tiles bring one c2p block, and it goes to the S
          // columns (free until this tile's scores are computed), so the p2c products can be issued into R at once and
          // run while the drain group works; only the four score MMAs wait for the drain.  The same holds for a first
          // band tile that is the CTA's first tile at all (c2p_outside_r).
          const bool first = band_idx == 0;
          if (ok && has_c2p && elect_one()) {
            // c2p[m][p] = Q[m].X_k[p] in 128-position blocks (later tiles reuse the lower half of the previous window
            // from the stage)
            const int nblk = first ? 2 : 1;
#pragma unroll 1
            for (int blk = 0; blk < nblk; ++blk)
#pragma unroll
              for (int ks = 0; ks < G::kSteps; ++ks)
                G::mma(tmem_base + (!first ? kColS : (c2p_outside_r ? (blk == 0 ? kColS : kColO) : kColR + blk * 128)),
                       dq + uint64_t((ks * 32) >> 4), dwk + uint64_t((blk * G::kTile + ks * 32) >> 4), idesc_s, ks > 0);
          }
          if (elect_one()) mma_commit(bar(kBarC2p));
          const bool scores_last = !first || c2p_outside_r;  // a c2p block sits in the S columns until it is drained
          if (ok && !scores_last && elect_one()) {
#pragma unroll
            for (int ks = 0; ks < G::kSteps; ++ks)
              G::mma(tmem_base + kColS, dq + uint64_t((ks * 32) >> 4), dk + uint64_t((ks * 32) >> 4), idesc_s, ks > 0);
          }
          if (!scores_last) {
            wait(bar(kBarStage), bands & 1u);  // the drain group has moved the c2p product out of R
            tc_fence_after();
          }
          if (ok && has_p2c && elect_one()) {
            // p2c products.  Key block b (32 keys) needs X_q rows starting at 32(3-b) (t = 0) and 32(4-b) (t = 1); blocks
            // b and b+1 share the start row 32(3-b), so three 128x64 products cover six of the eight (b, t) pairs and
            // two 128x32 products the rest (a narrow MMA costs the tensor pipe about as much as a 64-wide one):
            //   start row 96: keys   0..63  -> R +   0 (b=0,t=0 | b=1,t=1)     start row 128: keys  0..31  -> R + 192 (b=0,t=1)
            //   start row 64: keys  32..95  -> R +  64 (b=1,t=0 | b=2,t=1)     start row   0: keys 96..127 -> R + 224 (b=3,t=0)
            //   start row 32: keys  64..127 -> R + 128 (b=2,t=0 | b=3,t=1)
            const uint64_t blk32 = (32u * G::kRow) >> 4;  // 32 rows of an operand, in descriptor address units
#pragma unroll 1
            for (int q = 0; q < 3; ++q) {
              const uint64_t da = dwq + uint64_t(3 - q) * blk32, db = dk + uint64_t(q) * blk32;
#pragma unroll
              for (int ks = 0; ks < G::kSteps; ++ks)
                G::mma(tmem_base + kColR + 64 * q, da + uint64_t((ks * 32) >> 4), db + uint64_t((ks * 32) >> 4),
                       idesc_p2c64, ks > 0);
            }
#pragma unroll
            for (int ks = 0; ks < G::kSteps; ++ks)
              G::mma(tmem_base + kColR + 192, dwq + 4 * blk32 + uint64_t((ks * 32) >> 4),
                     dk + uint64_t((ks * 32) >> 4), idesc_p2c, ks > 0);
#pragma unroll
            for (int ks = 0; ks < G::kSteps; ++ks)
              G::mma(tmem_base + kColR + 224, dwq + uint64_t((ks * 32) >> 4),
                     dk + 3 * blk32 + uint64_t((ks * 32) >> 4), idesc_p2c, ks > 0);
          }
          if (scores_last) {
            wait(bar(kBarStage), bands & 1u);  // the drain group has moved the c2p product out of S
            tc_fence_after();
            if (ok && elect_one()) {
#pragma unroll
              for (int ks = 0; ks < G::kSteps; ++ks)
                G::mma(tmem_base + kColS, dq + uint64_t((ks * 32) >> 4), dk + uint64_t((ks * 32) >> 4), idesc_s, ks > 0);
            }
          }
          ++band_idx;
          ++bands;
        } else {
          tc_fence_after();
        }
        if (ok && kind != kBand && elect_one()) {
#pragma unroll
          for (int ks = 0; ks < G::kSteps; ++ks)
            G::mma(tmem_base + kColS, dq + uint64_t((ks * 32) >> 4), dk + uint64_t((ks * 32) >> 4), idesc_s, ks > 0);
          if (has_p2c && (kind == kSatHi || kind == kSatLo)) {
            // bf16: accumulated straight into S.  e4m3: the term has its own scale, so it goes to the (idle) product
            // area and the softmax threads add it with the ratio of the scales.
            const uint64_t ds = dsat + uint64_t(kind == kSatHi ? 0u : (1024u >> 4));
#pragma unroll
            for (int ks = 0; ks < G::kSteps; ++ks)
              G::mma(tmem_base + (F8 ? kColR : kColS), ds + uint64_t((ks * 32) >> 4), dk + uint64_t((ks * 32) >> 4),
                     idesc_s, (F8 ? ks > 0 : 1));
          }
        }
        if (elect_one()) {
          mma_commit(bar(kBarS));
          mma_commit(bar(kBarKFree + s));
          if (kind == kBand) mma_commit(bar(kBarWinFree));
          if (jj == it.n_proc - 1) mma_commit(bar(kBarQFree));
        }
        ++tiles;
        FDB_STAMP(taken, 2, j, 0);
      }
      } while (next_item(it));
    } else if (warp == kPvWarp) {
      // ================================================= P.V MMA issuer =================================================
      const uint32_t idesc_pv = instr_desc(128, 64, G::kFmt, 0, 1);
      const uint64_t dv0 = G::desc(smem + kSmemV, G::kGroup);  // V is the MN-major operand: keys run along K
      uint32_t tiles = 0;
      do {
#pragma unroll 1
      for (int jj = 0; jj < it.n_proc; ++jj) {
        const uint32_t s = tiles & 1u;
        const uint64_t dv = dv0 + uint64_t(s) * (16384u >> 4);
        wait(bar(kBarV + s), (tiles >> 1) & 1u);
        wait(bar(kBarP), tiles & 1u);  // both groups have written P (and read the output of the item before)
        tc_fence_after();
        FDB_STAMP(taken, 2, it.j_first + jj, 3);
        if (ok && elect_one()) {
#pragma unroll
          for (int ks = 0; ks < G::kPvSteps; ++ks)  // one step = 2048 bytes of V in either build (16 x 128 B, 32 x 64 B)
            G::mma_ts(tmem_base + kColO, tmem_base + kColP + G::kPColsPerStep * ks, dv + uint64_t((ks * 2048) >> 4),
                      idesc_pv, (jj > 0 || ks > 0 || it.resume) ? 1u : 0u);
        }
        if (elect_one()) {
          mma_commit(bar(kBarO));
          mma_commit(bar(kBarVFree + s));
        }
        ++tiles;
        FDB_STAMP(taken, 2, it.j_first + jj, 5);
      }
      } while (next_item(it));
    }
  } else {
    // =================================================== softmax groups =================================================
    reg_alloc<kSoftmaxRegs>();
    const int g = warp >> 2;                 // key half
    const int quad = warp & 3;
    const int r = quad * 32 + lane;          // row of the tile
    const uint32_t tmem_lane = tmem_base + (uint32_t(quad * 32) << 16);
    // lane that holds the p2c value of key c of a 32-key block; kept in registers (an addition per shuffle otherwise)
    [[maybe_unused]] int from[32];
    if constexpr (!F8) {
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        from[c] = lane + 31 - c;  // (taken modulo 32)
        asm volatile("" : "+r"(from[c]));
      }
    }
    uint32_t items = 0, tiles = 0, bands = 0;
    do {
    const int m0 = it.m0, len = it.len, seq_row0 = it.row0, head = it.head, j_first = it.j_first, n_proc = it.n_proc;
    const bool resume = it.resume;
    const int my_row = m0 + r;
    // rows of this tile that may be written: packed -> the sequence's own rows; dense -> the padded row range
    const int row_limit = args.packed ? len : args.max_seqlen;
    if (n_proc == 0) {  // dense padding tile: zeros, nothing else (src/flashdeberta/padding.py:30-44)
      if (it.seq >= 0 && g == 0 && my_row < row_limit) {
        uint4* o4 = reinterpret_cast<uint4*>(args.out + (int64_t)(seq_row0 + my_row) * args.o_rs + (int64_t)head * args.o_hs);
#pragma unroll
        for (int c = 0; c < 8; ++c) o4[c] = make_uint4(0, 0, 0, 0);
        if (args.lse != nullptr) args.lse[(int64_t)(seq_row0 + my_row) * args.heads + head] = 0.f;
      }
      __syncwarp();
      continue;
    }
    // e4m3: value = stored * scale.  The three score terms carry different scale products; they are brought to the one of
    // Q.K^T (ratio_c, ratio_p) when they are added, and that product goes into the softmax scale.
    float c_eff = args.scale_log2, ratio_c = 1.f, ratio_p = 1.f, v_scale = 1.f;
    if constexpr (F8) {
      const int64_t at = (int64_t)it.seq * args.heads + head;
      const float sq = __ldg(args.q_scale + at), sk = __ldg(args.k_scale + at);
      v_scale = __ldg(args.v_scale + at);
      c_eff = args.scale_log2 * sq * sk;
      if (has_c2p) ratio_c = __ldg(args.xk_scale + head) / sk;
      if (has_p2c) ratio_p = __ldg(args.xq_scale + head) / sq;
    }

    float rc_lo = 0.f, rc_hi = 0.f;  // saturated c2p terms of this row
    bool rc_read = !has_c2p;

    uint32_t band_idx = 0;
    // Rows behind the sequence (padding, the next sequence, unused memory) never ask for a rescale, which the rows of their warp take
    // part in: a sequence's rounding is its own.
    float m_used = my_row < len ? -INFINITY : INFINITY, l_run = 0.f;
    if (resume && ok) {
      // continue from what the far kernel accumulated over the plain and saturated tiles of this row: O goes back into
      // tensor memory (this group's 32 columns), the reference maximum and the row sum into registers
      const int64_t rh = (int64_t)(seq_row0 + (my_row < len ? my_row : len - 1)) * args.heads + head;
      const float4* po = reinterpret_cast<const float4*>(args.part_o + rh * 64 + 32 * g);
      uint32_t o[32];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 v4 = __ldg(po + q);
        o[4 * q + 0] = __float_as_uint(v4.x); o[4 * q + 1] = __float_as_uint(v4.y);
        o[4 * q + 2] = __float_as_uint(v4.z); o[4 * q + 3] = __float_as_uint(v4.w);
      }
      tmem_st32(tmem_lane + kColO + 32 * g, o);
      tmem_wait_st();
      const float2 ml = __ldg(reinterpret_cast<const float2*>(args.part_ml + rh * 2));
      if (my_row < len) m_used = ml.x;
      l_run = g == 0 ? ml.y : 0.f;
    }

#pragma unroll 1
    for (int jj = 0; jj < n_proc; ++jj) {
      const int j = j_first + jj;
      const int n0 = j * kTileN;
      const int kind = tile_kind(it, j);

      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 0);
      if (!rc_read && kind != kBand) {
        // (in front of this tile's scores: until they are read nothing of the item after the next one is loaded, which shares the buffer)
        wait(bar(kBarRc + (items & 1u)), (items >> 1) & 1u);
        const uint32_t rc = smem + kSmemRc + 1024u * (items & 1u) + 4u * uint32_t(r);
        rc_hi = ratio_c * lds_f32(rc);
        rc_lo = ratio_c * lds_f32(rc + 512u);
        rc_read = true;
      }
      wait(bar(kBarS), tiles & 1u);
      tc_fence_after();
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 1);

      // ---- this thread's 64 scores (+ p2c through the quadrant shuffle) into registers, then S and R are released ----
      float s[64];
      if (kind == kBand && has_p2c) {
        if constexpr (F8) {
          // 16 keys at a time, the loads of the next 16 in flight while these are combined (two sets of three 16-register runs; in the
          // other form, which needs its registers for the scale ratios too, 438 against 431 us a call of 2 x 4096 x 16 heads)
          uint32_t a[2][16], t0[2][16], t1[2][16];
          auto pull = [&](int q) {
            // key block b = 2g + (q >> 1): columns of its two products (see the score-issuing warp)
            const int b = 2 * g + (q >> 1);
            const uint32_t c0 = b == 3 ? 224u : 64u * uint32_t(b);
            const uint32_t c1 = b == 0 ? 192u : 64u * uint32_t(b) - 32u;
            const uint32_t hf = 16u * uint32_t(q & 1);
            tmem_ld16(tmem_lane + kColS + 64 * g + 16 * q, a[q & 1]);
            tmem_ld16(tmem_lane + kColR + c0 + hf, t0[q & 1]);
            tmem_ld16(tmem_lane + kColR + c1 + hf, t1[q & 1]);
          };
          pull(0);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 16; ++c)  // nothing below uses them in front of the wait
              asm volatile("" : "+r"(a[q & 1][c]), "+r"(t0[q & 1][c]), "+r"(t1[q & 1][c]));
            if (q < 3) pull(q + 1);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const int cc = 16 * (q & 1) + c;
              const uint32_t x = (lane + cc <= 30) ? t1[q & 1][c] : t0[q & 1][c];
              const uint32_t y = __shfl_sync(0xffffffffu, x, lane + 31 - cc);  // the source lane is taken modulo 32
              s[16 * q + c] = fmaf(__uint_as_float(y), ratio_p, __uint_as_float(a[q & 1][c]));
            }
          }
        } else {
          // the scores, then 16 keys at a time the two products: the loads of the next 16 are in flight while these are shuffled
          uint32_t a0[32], a1[32], t0[16], t1[16], x[16];
          auto pull = [&](int q) {
            // key block b = 2g + (q >> 1): columns of its two products (see the score-issuing warp)
            const int b = 2 * g + (q >> 1);
            const uint32_t hf = 16u * uint32_t(q & 1);
            tmem_ld16(tmem_lane + kColR + (b == 3 ? 224u : 64u * uint32_t(b)) + hf, t0);
            tmem_ld16(tmem_lane + kColR + (b == 0 ? 192u : 64u * uint32_t(b) - 32u) + hf, t1);
          };
          tmem_ld32(tmem_lane + kColS + 64 * g, a0);
          tmem_ld32(tmem_lane + kColS + 64 * g + 32, a1);
          pull(0);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            tmem_wait_ld();
            if (q == 0) {
#pragma unroll
              for (int c = 0; c < 32; ++c) asm volatile("" : "+r"(a0[c]), "+r"(a1[c]));  // nothing below uses them in front of the wait
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) asm volatile("" : "+r"(t0[c]), "+r"(t1[c]));
#pragma unroll
            for (int c = 0; c < 16; ++c) x[c] = (lane + 16 * (q & 1) + c <= 30) ? t1[c] : t0[c];
            if (q < 3) {
#pragma unroll
              for (int c = 0; c < 16; ++c) asm volatile("" : "+r"(x[c]));
              pull(q + 1);
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              const uint32_t y = __shfl_sync(0xffffffffu, x[c], from[16 * (q & 1) + c]);
              s[16 * q + c] = fmaf(__uint_as_float(y), ratio_p, __uint_as_float(q < 2 ? a0[16 * q + c] : a1[16 * q + c - 32]));
            }
          }
        }
      } else {
        uint32_t a0[32], a1[32];
        tmem_ld32(tmem_lane + kColS + 64 * g, a0);
        tmem_ld32(tmem_lane + kColS + 64 * g + 32, a1);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          s[c] = __uint_as_float(a0[c]);
          s[32 + c] = __uint_as_float(a1[c]);
        }
        if (F8 && has_p2c && kind != kPlain) {
          // e4m3: the saturated p2c term of these keys sits in the product area (same value in every row)
#pragma unroll
          for (int ch = 0; ch < 2; ++ch) {
            uint32_t t0[32];
            tmem_ld32(tmem_lane + kColR + 64 * g + 32 * ch, t0);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; ++c) s[32 * ch + c] = fmaf(__uint_as_float(t0[c]), ratio_p, s[32 * ch + c]);
          }
        }
      }
      tc_fence_before();
      arrive(bar(kBarSFree));
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 2);

      float row_const = 0.f;
      if (kind == kBand) {
        wait(bar(kBarStage), bands & 1u);  // the c2p stage of this tile is complete
        if (has_c2p) {
          // c2p[m][i] is position p = m + 127 - i of the window, stored in column ((p ^ flip) - m) & 255 of row m (see the
          // drain group): for this thread's keys i = 64g .. 64g+63 that is the aligned run of 64 columns ending at
          // 127 - 64g (+ 128 when flipped), read with eight 16-byte loads, key i in column (run start) + 63 - (i - 64g).
          const uint32_t run = smem + kSmemStageC + uint32_t(r) * kStageCPitch +
                               2u * (uint32_t(64 * (1 - g)) + ((band_idx & 1u) ? 128u : 0u));
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint4 w4 = lds_v4(run + 16u * uint32_t(q));
            const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {  // column 8q + e of the run -> key 63 - (8q + e)
              float& to = s[63 - (8 * q + e)];
              if constexpr (F8) to = fmaf(__uint_as_float((e & 1) ? (w[e >> 1] & 0xffff0000u) : (w[e >> 1] << 16)), ratio_c, to);
              else to = (e & 1) ? add_bf16_hi(to, w[e >> 1]) : add_bf16_lo(to, w[e >> 1]);
            }
          }
        }
        arrive(bar(kBarGather));
        ++band_idx;
        ++bands;
      } else if (kind == kSatHi) {
        row_const = rc_hi;
      } else if (kind == kSatLo) {
        row_const = rc_lo;
      }
      if (n0 + kTileN > len) {  // keys past the end of the sequence
        const int valid = len - n0 - 64 * g;
#pragma unroll
        for (int i = 0; i < 64; ++i) s[i] = i < valid ? s[i] : -INFINITY;
      }
      float mx4[4] = {max3(s[0], s[4], s[8]), max3(s[1], s[5], s[9]), max3(s[2], s[6], s[10]), max3(s[3], s[7], s[11])};
#pragma unroll
      for (int i = 12; i < 60; i += 8)
#pragma unroll
        for (int q = 0; q < 4; ++q) mx4[q] = max3(mx4[q], s[i + q], s[i + 4 + q]);
#pragma unroll
      for (int q = 0; q < 4; ++q) mx4[q] = fmaxf(mx4[q], s[60 + q]);
      float mx = max3(mx4[0], mx4[1], fmaxf(mx4[2], mx4[3]));
      // the two threads of a row agree on the row maximum
      const uint32_t xch = smem + kSmemXchg + (tiles & 1u) * 1024u;
      sts_f32(xch + uint32_t(g) * 512u + uint32_t(r) * 4u, mx);
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 3);
      bar_sync(1, kSoftmaxThreads);
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 4);
      mx = fmaxf(mx, lds_f32(xch + uint32_t(g ^ 1) * 512u + uint32_t(r) * 4u));

      const float t_max = (mx + row_const) * c_eff;
      if (jj == 0 && !resume) {
        m_used = fmaxf(m_used, t_max);
      } else {
        // The previous P.V has finished: O may be rescaled and the P columns overwritten.  Observed on every tile (it is
        // long done by now) so that this thread never falls two phases behind the barrier, which a parity wait could
        // not tell apart.
        if (jj > 0) wait(bar(kBarO), (tiles - 1u) & 1u);
        tc_fence_after();
        // bf16: O is rescaled only when the maximum moved by more than 2^8 (P <= 256 is harmless in bf16).
        // e4m3: P is stored as 2^8 * exp2(.), so it has to stay <= 1: rescale whenever the maximum moves.
        const bool need = t_max > m_used + (F8 ? 0.f : 8.f);
        if (__any_sync(0xffffffffu, need)) {  // warp-uniform, and the same in both groups: rescale O of these 32 rows
          const float m_new = fmaxf(m_used, t_max);
          const float alpha = ex2(m_used - m_new);
          l_run *= alpha;
          m_used = m_new;
          {
            uint32_t o[32];
            tmem_ld32(tmem_lane + kColO + 32 * g, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st32(tmem_lane + kColO + 32 * g, o);
            tmem_wait_st();
          }
        }
      }
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 5);
      const float off = row_const * c_eff - m_used + (F8 ? 8.f : 0.f);
      if constexpr (F8) {
        float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          s[i] = ex2(fmaf(s[i], c_eff, off));
          l4[i & 3] += s[i];
        }
        l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
        if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 6);
        {  // 16 columns of e4m3 quadruples
          uint32_t p[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) p[i] = pack_e4m3x4(s[4 * i], s[4 * i + 1], s[4 * i + 2], s[4 * i + 3]);
          tmem_st16(tmem_lane + kColP + 16 * g, p);
          tmem_wait_st();
        }
      } else {
        // p = 2^(s * scale + off) with the two-wide fp32 forms; the bf16 pairs of the first 32 keys are on their way to
        // tensor memory while the other 32 are computed
        const uint64_t scale2 = pack_f32x2(c_eff, c_eff), off2 = pack_f32x2(off, off);
        uint64_t l2[2] = {0ull, 0ull};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t p[16];
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            float e0, e1, e2, e3;
            unpack_f32x2(fma_f32x2(pack_f32x2(s[32 * h + i], s[32 * h + i + 1]), scale2, off2), e0, e1);
            unpack_f32x2(fma_f32x2(pack_f32x2(s[32 * h + i + 2], s[32 * h + i + 3]), scale2, off2), e2, e3);
            e0 = ex2(e0); e1 = ex2(e1); e2 = ex2(e2); e3 = ex2(e3);
            l2[0] = add_f32x2(l2[0], pack_f32x2(e0, e1));
            l2[1] = add_f32x2(l2[1], pack_f32x2(e2, e3));
            p[i >> 1] = pack_bf16x2(e0, e1);
            p[(i >> 1) + 1] = pack_bf16x2(e2, e3);
          }
          tmem_st16(tmem_lane + kColP + 32 * g + 16 * h, p);
        }
        float s0, s1, s2, s3;
        unpack_f32x2(l2[0], s0, s1);
        unpack_f32x2(l2[1], s2, s3);
        l_run += (s0 + s1) + (s2 + s3);
        if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 6);
        tmem_wait_st();
      }
      tc_fence_before();
      arrive(bar(kBarP));
      ++tiles;
      if (lane == 0 && quad == 0) FDB_STAMP(taken, g, j, 7);
    }

    // ---- epilogue: combine the two row sums, O / l, write this group's 32 output columns ----
    sts_f32(smem + kSmemLsum + uint32_t(g) * 512u + uint32_t(r) * 4u, l_run);
    bar_sync(1, kSoftmaxThreads);
    const float l_tot = l_run + lds_f32(smem + kSmemLsum + uint32_t(g ^ 1) * 512u + uint32_t(r) * 4u);
    wait(bar(kBarO), (tiles - 1u) & 1u);
    tc_fence_after();
    if (ok) {
      const bool valid = my_row < len;
      const bool pad = !valid && my_row < row_limit;  // dense padding rows inside a partly valid tile get zeros
      const float inv = valid ? v_scale / l_tot : 0.f;
      uint32_t o[32];
      tmem_ld32(tmem_lane + kColO + 32 * g, o);  // whole warps execute this, whatever their rows
      tmem_wait_ld();
      if (valid || pad) {
        uint4* o4 = reinterpret_cast<uint4*>(args.out + (int64_t)(seq_row0 + my_row) * args.o_rs +
                                             (int64_t)head * args.o_hs + 32 * g);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (valid)
            v = make_uint4(pack_bf16x2(__uint_as_float(o[q4 * 8 + 0]) * inv, __uint_as_float(o[q4 * 8 + 1]) * inv),
                           pack_bf16x2(__uint_as_float(o[q4 * 8 + 2]) * inv, __uint_as_float(o[q4 * 8 + 3]) * inv),
                           pack_bf16x2(__uint_as_float(o[q4 * 8 + 4]) * inv, __uint_as_float(o[q4 * 8 + 5]) * inv),
                           pack_bf16x2(__uint_as_float(o[q4 * 8 + 6]) * inv, __uint_as_float(o[q4 * 8 + 7]) * inv));
          o4[q4] = v;
        }
        if (g == 0 && args.lse != nullptr)
          args.lse[(int64_t)(seq_row0 + my_row) * args.heads + head] =
              valid ? (m_used + log2f(l_tot) - (F8 ? 8.f : 0.f)) * 0.6931471805599453f : 0.f;
      }
    }
    tc_fence_before();
    __syncwarp();
    ++items;
    } while (next_item_of_all(it));
  }

  // ---- teardown -------------------------------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (tid == 0 && args.status != nullptr) atomicOr(reinterpret_cast<unsigned int*>(args.status), FDB_DEV_TIMEOUT);
    // give copies and MMAs that may still be in flight a bounded time to land before TMEM and shared memory go away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
}

}  // namespace

int launch_attn_fwd_sm100(const fdb_attn_params& p, const ExpandGeometry& g, const AttnBuffers& b, void* stream, bool chained) {
  const bool f8 = p.dtype == FDB_E4M3;
  FwdArgs a;
  int rc;
  if ((rc = make_map_rows(&a.tm_q, p.q, p.total_rows, p.heads, p.q_row_stride, p.q_head_stride, kTileM, f8, "q"))) return rc;
  if ((rc = make_map_rows(&a.tm_k, p.k, p.total_rows, p.heads, p.k_row_stride, p.k_head_stride, kTileN, f8, "k"))) return rc;
  if ((rc = make_map_rows(&a.tm_v, p.v, p.total_rows, p.heads, p.v_row_stride, p.v_head_stride, kTileN, f8, "v"))) return rc;
  a.xk = b.exp_key;
  a.xq = b.exp_query;
  a.q_scale = p.q_scale; a.k_scale = p.k_scale; a.v_scale = p.v_scale;
  a.xk_scale = p.pos_key_scale; a.xq_scale = p.pos_query_scale;
  // a map is always encoded so the kernel argument is well formed; an unused one points at q
  if (a.xk) { if ((rc = make_map_table(&a.tm_xk, a.xk, g.rows, p.heads, f8, "expanded pos_key", 128))) return rc; } else a.tm_xk = a.tm_q;
  if (a.xq) { if ((rc = make_map_table(&a.tm_xq, a.xq, g.rows, p.heads, f8, "expanded pos_query"))) return rc; } else a.tm_xq = a.tm_q;
  if (a.xq) { if ((rc = make_map_table(&a.tm_xq_sat, a.xq, g.rows, p.heads, f8, "saturated pos_query rows", 8))) return rc; } else a.tm_xq_sat = a.tm_q;
  a.out = static_cast<__nv_bfloat16*>(p.out);
  a.o_rs = p.out_row_stride; a.o_hs = p.out_head_stride;
  a.seq_info = b.seq_info;
  a.tile_first = b.tile_first;
  a.slot_info = reinterpret_cast<const int4*>(b.slot_info);
  a.lse = p.lse; a.status = p.status;
  a.batch = p.batch; a.heads = p.heads; a.packed = p.cu_seqlens != nullptr; a.max_seqlen = p.max_seqlen;
  a.sat_lo = g.sat_lo; a.sat_hi = g.sat_hi; a.d_first = g.d_first; a.xrows = g.rows;
  a.scale_log2 = p.sm_scale * 1.4426950408889634f;
  a.part_o = b.part_o;
  a.part_ml = b.part_ml;
  a.band_only = b.split ? 1 : 0;
  a.split_len = (p.tune & FDB_TUNE_TWO_LAUNCHES) ? 0 : kSplitSeqlen;  // forced two launches: every sequence is split
#ifdef FDB_TRACE
  a.trace = reinterpret_cast<long long*>(trace_from_env("FDB_TRACE_PTR"));
  a.trace_item = (uint32_t)trace_from_env("FDB_TRACE_ITEM");
#endif

  const int64_t slots = tile_slots(p);
  a.slots = (int)slots;
  if (slots <= 0) return FDB_OK;
  if (slots > 2147483647LL || p.heads > 65535) return fail(FDB_ERR_LIMIT, "grid too large");

  // bf16: key tiles with saturated (or no) position terms go to the far kernel (half an SM per CTA, two CTAs per SM); with
  // position terms the band tiles follow in attn_fwd_kernel, which picks up the partial result on the same stream.
  const bool no_pos = a.xk == nullptr && a.xq == nullptr;
  if (!f8 && (b.split || (no_pos && !(p.tune & FDB_TUNE_ONE_LAUNCH)))) {
    rc = launch_attn_fwd_far1(&a, slots, p.heads, stream, chained);
    if (rc != FDB_OK) return rc;
    if (no_pos) return FDB_OK;
  }

  auto kernel = f8 ? attn_fwd_kernel<true> : attn_fwd_kernel<false>;
  static std::atomic<uint64_t> smem_done[2];
  cudaError_t e = allow_smem(smem_done[f8 ? 1 : 0], reinterpret_cast<const void*>(kernel), (int)kSmemBytes);
  if (e == cudaSuccess)
    e = launch_kernel<FwdArgs>(kernel, a, dim3((unsigned)slots, p.heads), kThreads, kSmemBytes, chained, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "attn_fwd launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

}  // namespace fdb
