// out = act(x . W^T + bias) for sm_100a, act = identity or erf GELU: the linear layers of an encoder layer.
//
// The reference inherits them from transformers (the projections of DisentangledSelfAttention, DebertaV2SelfOutput,
// DebertaV2Intermediate, DebertaV2Output behind FlashDebertaV2Layer, src/flashdeberta/model.py:259-272): cuBLAS GEMMs with a
// bias epilogue and, in the intermediate block, an elementwise kernel that reads and rewrites the (rows, 4 * hidden)
// activation.  Here bias and GELU are applied on the way out of tensor memory, and up to three weights over the same input
// (query, key, value) are one launch.
//
// Persistent grid; a tile is 128 rows (CG = 1) or 256 rows (CG = 2, a pair of CTAs on two SMs) x BN output features, K in
// steps of 64 through a ring of stages:
//   warp 0  TMA, the CTA's 128 x 64 tile of x and its BN / CG rows of W
//   warp 1  (of the pair's even CTA) tcgen05.mma, four per stage; two accumulators in tensor memory, so the epilogue
//           of one tile runs beside the main loop of the next (both warps stay converged and issue through an elected lane)
//   warps 2-9: epilogue, two warps per 32-lane quarter of tensor memory: + bias, rounded to bf16 as the separate GEMM would
//           leave it, GELU in fp32, bf16 out with 32-byte stores
// What bounds a tile is shared memory, not the tensor pipe: a stage is written once by TMA and read once by the MMAs, at
// 128 bytes per clock.  Per 64 of K a 128 x 256 tile moves 96 KB (750 clocks for 512 clocks of MMA); the pair of CTAs halves
// the W traffic of each SM and brings 256 x 256 to 64 KB (512 for 512).  `kConfigs` holds these costs, and the launcher takes
// the tile whose waves over the SMs cost least.
// Every wait is bounded; on a timeout the CTA raises FDB_DEV_TIMEOUT in the status word, frees its tensor memory and
// returns.  No TMA multicast.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gelu.cuh"
#include "internal.h"
#include "launch.h"
#include "linear.h"
#include "sm100_ptx.cuh"
#include "tensor_map.cuh"

namespace fdb {
namespace {

using namespace ptx;

constexpr int kBM = 128, kBK = 64;
constexpr int kThreads = 320;
constexpr int kTmaWarp = 0, kMmaWarp = 1, kEpiWarp0 = 2, kEpiWarps = 8;

struct LinearArgs {
  CUtensorMap tm_x, tm_w[3];
  const __nv_bfloat16* bias[3];  // entries may be NULL
  __nv_bfloat16* out[3];
  const int32_t* rows_dev;       // the number of rows, when only the device knows it (at most `rows`)
  int32_t* status;
  int64_t rows, out_stride;
  int k, groups, tiles_n;        // groups = weights over the same x; tiles_n = feature tiles of one weight
  bool sectors;                  // every row of every output starts on a 32-byte boundary
};

// 32 bytes per thread in one store (whole sectors)
__device__ __forceinline__ void st_global_32B(void* p, const uint32_t (&o)[16], int at) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(o[at]), "r"(o[at + 1]), "r"(o[at + 2]),
               "r"(o[at + 3]), "r"(o[at + 4]), "r"(o[at + 5]), "r"(o[at + 6]), "r"(o[at + 7])
               : "memory");
}

template <int CG, int BN> struct Tile {
  static constexpr uint32_t kBytesA = kBM * kBK * 2, kBytesW = BN / CG * kBK * 2, kStageBytes = kBytesA + kBytesW;
  // 190 KB of stages; the narrowest tile keeps to half an SM so that two kernels of a chain can share it
  static constexpr int kStages = BN == 64 ? 4 : (BN == 256 ? 6 : (BN == 192 ? 6 : (CG == 2 ? 8 : 6)));
  static constexpr uint32_t kSmemBars = kStages * kStageBytes;
  enum : uint32_t { kBarFull = 0, kBarEmpty = kStages, kBarAccFull = 2 * kStages, kBarAccEmpty = 2 * kStages + 2, kNumBars = 2 * kStages + 4 };
  static constexpr uint32_t kSmemBytes = kSmemBars + 8 * kNumBars + 16 + 1024;  // + tensor-memory slot, abort flag, alignment slack
  static constexpr uint32_t kAccStride = BN == 192 ? 256 : BN, kTmemCols = 2 * kAccStride;
};

template <int CG, int BN, bool GELU>
__global__ void __launch_bounds__(kThreads, 1) linear_kernel(const __grid_constant__ LinearArgs args) {
  using T = Tile<CG, BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem - smem_u32(smem_raw));
  const int tid = threadIdx.x, warp = (int)uniform(uint32_t(tid) >> 5), lane = tid & 31;
  const uint32_t rank = CG == 2 ? cluster_rank() : 0u;

  auto bar = [&](uint32_t i) -> uint32_t { return smem + T::kSmemBars + 8u * i; };
  const uint32_t tmem_slot = smem + T::kSmemBars + 8u * T::kNumBars;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem_gen + T::kSmemBars + 8u * T::kNumBars + 8u);

  if (tid == 0) {
    *abort_flag = 0u;
    for (uint32_t i = 0; i < T::kNumBars; ++i) mbar_init(bar(i), (i >= T::kBarAccEmpty) ? uint32_t(kEpiWarps * CG) : 1u);
    fence_barrier_init();
    tma_prefetch_desc(&args.tm_x);
    tma_prefetch_desc(&args.tm_w[0]);
  }
  if (warp == kMmaWarp) {
    if constexpr (CG == 2) { tmem_alloc_pair(tmem_slot, T::kTmemCols); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, T::kTmemCols); tmem_relinquish(); }
  }
  tc_fence_before();
  if constexpr (CG == 2) cluster_sync(); else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(*reinterpret_cast<volatile uint32_t*>(smem_gen + T::kSmemBars + 8u * T::kNumBars));

  grid_launch();
  const int tiles_n = args.tiles_n * args.groups;
  const int first = blockIdx.x / CG, step = gridDim.x / CG;
  const int kblocks = args.k / kBK;
  auto load_w = [&](uint32_t st, int kb, const CUtensorMap* tm_w, int n0) {
    const uint32_t w = smem + st * T::kStageBytes + T::kBytesA;
    if constexpr (CG == 2) {
      if (rank == 0) mbar_expect_tx(bar(T::kBarFull + st), 2 * T::kStageBytes);
      tma_load_3d_pair(w, tm_w, bar(T::kBarFull + st), 0, kb, n0);
    } else {
      mbar_expect_tx(bar(T::kBarFull + st), T::kStageBytes);
      tma_load_3d(w, tm_w, bar(T::kBarFull + st), 0, kb, n0);
    }
  };
  // The weights are nobody's output: the first stages of W are on their way before the kernel in front has finished.
  const int early = kblocks < T::kStages ? kblocks : T::kStages;
  if (warp == kTmaWarp) {
    const int tn = first % tiles_n, group = tn / args.tiles_n;
    const int n0 = (tn - group * args.tiles_n) * BN + int(rank) * (BN / CG);
#pragma unroll 1
    for (int kb = 0; kb < early; ++kb)
      if (elect_one()) load_w(uint32_t(kb), kb, &args.tm_w[group], n0);
  }
  grid_wait();
  const int64_t rows = args.rows_dev != nullptr ? (int64_t)*args.rows_dev : args.rows;
  const int tiles_m = (int)((rows + kBM * CG - 1) / (kBM * CG));
  // every CTA has loads in flight for its first tile, so it works through that one even when there are no rows for it
  const int num_tiles = max(tiles_m * tiles_n, first + 1);
  bool ok = true;
  auto wait = [&](uint32_t b, uint32_t parity) {
    if (ok) ok = mbar_wait_warp(b, parity, abort_flag);
  };

  if (warp == kTmaWarp) {
    uint32_t st = 0, phase = 0;
    int skip = early;  // stages whose W is already on its way
#pragma unroll 1
    for (int tile = first; tile < num_tiles && ok; tile += step) {
      const int m0 = (tile / tiles_n) * (kBM * CG) + int(rank) * kBM;
      const int tn = tile % tiles_n, group = tn / args.tiles_n;
      const int n0 = (tn - group * args.tiles_n) * BN + int(rank) * (BN / CG);
      const CUtensorMap* tm_w = &args.tm_w[group];
#pragma unroll 1
      for (int kb = 0; kb < kblocks; ++kb) {
        if (skip == 0) wait(bar(T::kBarEmpty + st), phase ^ 1u);  // (the first round passes at once)
        if (!ok) break;
        if (elect_one()) {
          if (skip == 0) load_w(st, kb, tm_w, n0);
          if constexpr (CG == 2) tma_load_3d_pair(smem + st * T::kStageBytes, &args.tm_x, bar(T::kBarFull + st), 0, kb, m0);
          else tma_load_3d(smem + st * T::kStageBytes, &args.tm_x, bar(T::kBarFull + st), 0, kb, m0);
        }
        skip -= skip > 0 ? 1 : 0;
        if (++st == T::kStages) { st = 0; phase ^= 1u; }
      }
    }
  } else if (warp == kMmaWarp) {
    if (rank == 0) {
      const uint32_t idesc = instr_desc(kBM * CG, BN, 1, 0, 0);
      const uint64_t da0 = smem_desc_sw128(smem, 1024, 16), dw0 = smem_desc_sw128(smem + T::kBytesA, 1024, 16);
      uint32_t st = 0, phase = 0, local = 0;
#pragma unroll 1
      for (int tile = first; tile < num_tiles && ok; tile += step, ++local) {
        const uint32_t acc = local & 1u, d = tmem_base + acc * T::kAccStride;
        wait(bar(T::kBarAccEmpty + acc), ((local >> 1) & 1u) ^ 1u);  // the epilogue has read this accumulator
        tc_fence_after();
#pragma unroll 1
        for (int kb = 0; kb < kblocks; ++kb) {
          wait(bar(T::kBarFull + st), phase);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = da0 + uint64_t(st * (T::kStageBytes >> 4)), dw = dw0 + uint64_t(st * (T::kStageBytes >> 4));
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint32_t more = (kb > 0 || ks > 0) ? 1u : 0u;
              if constexpr (CG == 2) mma_bf16_pair(d, da + uint64_t((ks * 32) >> 4), dw + uint64_t((ks * 32) >> 4), idesc, more);
              else mma_bf16(d, da + uint64_t((ks * 32) >> 4), dw + uint64_t((ks * 32) >> 4), idesc, more);
            }
            if constexpr (CG == 2) mma_commit_pair(bar(T::kBarEmpty + st)); else mma_commit(bar(T::kBarEmpty + st));
            if (kb == kblocks - 1) { if constexpr (CG == 2) mma_commit_pair(bar(T::kBarAccFull + acc)); else mma_commit(bar(T::kBarAccFull + acc)); }
          }
          if (++st == T::kStages) { st = 0; phase ^= 1u; }
        }
      }
    }
  } else {
    const int quarter = warp & 3;                // the 32 tensor-memory lanes this warp may read
    const int half = (warp - kEpiWarp0) >> 2;    // which half of the tile's columns
    constexpr int kChunks = BN / 64;             // 32 columns at a time
    const uint32_t tmem_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    uint32_t acc_empty[2] = {bar(T::kBarAccEmpty), bar(T::kBarAccEmpty + 1)};
    if constexpr (CG == 2) { acc_empty[0] = map_to_rank(acc_empty[0], 0); acc_empty[1] = map_to_rank(acc_empty[1], 0); }
    uint32_t local = 0;
#pragma unroll 1
    for (int tile = first; tile < num_tiles; tile += step, ++local) {
      const int m0 = (tile / tiles_n) * (kBM * CG) + int(rank) * kBM;
      const int tn = tile % tiles_n, group = tn / args.tiles_n;
      const int n0 = (tn - group * args.tiles_n) * BN + half * (BN / 2);
      const uint32_t acc = local & 1u;
      wait(bar(T::kBarAccFull + acc), (local >> 1) & 1u);
      tc_fence_after();
      const int64_t row = (int64_t)m0 + quarter * 32 + lane;
      const bool live = row < rows;
      __nv_bfloat16* orow = args.out[group] + row * args.out_stride + n0;
      const __nv_bfloat16* bias = args.bias[group];
#pragma unroll 1
      for (int ch = 0; ch < kChunks; ++ch) {
        uint32_t a[32];
        if (ok) {  // whole warps execute the load, whatever their rows
          tmem_ld32(tmem_lane + acc * T::kAccStride + uint32_t(half * (BN / 2) + ch * 32), a);
          tmem_wait_ld();
        }
        if (ch == kChunks - 1) {  // the accumulator is in registers: the next tile but one may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) { if constexpr (CG == 2) mbar_arrive_cluster(acc_empty[acc]); else mbar_arrive(acc_empty[acc]); }
        }
        uint32_t o[16];
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
          uint4 bw = make_uint4(0, 0, 0, 0);
          if (bias != nullptr) bw = __ldg(reinterpret_cast<const uint4*>(bias + n0 + ch * 32 + c));
          const uint32_t b4[4] = {bw.x, bw.y, bw.z, bw.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // the sum as the separate GEMM would leave it: rounded to bf16
            float s0, s1;
            unpack_f32x2(add_f32x2(pack_f32x2(__uint_as_float(a[c + 2 * e]), __uint_as_float(a[c + 2 * e + 1])),
                                   pack_f32x2(__uint_as_float(b4[e] << 16), __uint_as_float(b4[e] & 0xffff0000u))), s0, s1);
            const uint32_t r = pack_bf16x2(s0, s1);
            if constexpr (GELU) {
              unpack_f32x2(gelu_erf2(pack_f32x2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u))), s0, s1);
              o[(c >> 1) + e] = pack_bf16x2(s0, s1);
            } else {
              o[(c >> 1) + e] = r;
            }
          }
        }
        if (live && ok) {
          if (args.sectors) {
            st_global_32B(orow + ch * 32, o, 0);
            st_global_32B(orow + ch * 32 + 16, o, 8);
          } else {
#pragma unroll
            for (int c = 0; c < 16; c += 4) *reinterpret_cast<uint4*>(orow + ch * 32 + 2 * c) = make_uint4(o[c], o[c + 1], o[c + 2], o[c + 3]);
          }
        }
      }
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
  if constexpr (CG == 2) {
    cluster_sync();  // the pair's arrivals on this CTA's barriers have landed, and both are done with tensor memory
    if (warp == kMmaWarp) tmem_dealloc_pair(tmem_base, T::kTmemCols);
  } else {
    if (warp == kMmaWarp) tmem_dealloc(tmem_base, T::kTmemCols);
  }
}

template <int CG, int BN, bool GELU>
int launch(const LinearArgs& a, int grid, bool chained, cudaStream_t stream) {
  static std::atomic<uint64_t> smem_done{0};
  auto kernel = linear_kernel<CG, BN, GELU>;
  cudaError_t e = allow_smem(smem_done, reinterpret_cast<const void*>(kernel), (int)Tile<CG, BN>::kSmemBytes);
  if (e == cudaSuccess) e = launch_kernel<LinearArgs>(kernel, a, dim3((unsigned)grid), kThreads, Tile<CG, BN>::kSmemBytes, chained, stream, CG);
  if (e != cudaSuccess) return fail(FDB_ERR_CUDA, "linear launch: %s", cudaGetErrorString(e));
  return FDB_OK;
}

// Tile shapes: clocks per 64 of K as measured over whole waves (16384 x 3072 -> 768: 59.3, 61.0, 65.2, 74.7, 141 us; what
// bounds each is at the head of the file) and clocks a launch adds on top (first loads, last epilogue).
struct Config { int cg, bn, clocks, extra; };
constexpr Config kConfigs[] = {{2, 256, 540, 2600}, {2, 192, 420, 2000}, {2, 128, 300, 1600}, {1, 128, 340, 1500}, {1, 64, 350, 600}};

}  // namespace

int make_linear_maps(LinearWeight* w, const void* weight, int n, int k) {
  for (int i = 0; i < 3; ++i) {
    const int rc = make_map_rows(&w->map[i], weight, n, k / kBK, k, kBK, kLinearBoxRows[i], false, "weight");
    if (rc != FDB_OK) return rc;
  }
  return FDB_OK;
}

int make_linear_input_map(CUtensorMap* m, const void* x, int64_t rows, int k) {
  return make_map_rows(m, x, rows, k / kBK, k, kBK, kBM, false, "x");
}

int launch_linear(const LinearCall& c, void* stream) {
  const int sms = sm_count();
  if (sms <= 0) return fail(FDB_ERR_CUDA, "linear set-up: no device");
  const Config* best = nullptr;
  int64_t best_cost = 0, best_tiles = 0;
  for (const Config& f : kConfigs) {
    if (c.n % f.bn != 0) continue;
    const int64_t tiles = (c.rows + kBM * f.cg - 1) / (kBM * f.cg) * (int64_t)(c.n / f.bn) * c.groups;
    const int64_t units = sms / f.cg, waves = (tiles + units - 1) / units;
    const int64_t cost = waves * ((int64_t)(c.k / kBK) * f.clocks) + f.extra;
    if (best == nullptr || cost < best_cost) { best = &f; best_cost = cost; best_tiles = tiles; }
  }
  if (best == nullptr || best_tiles * 2 > 2147483647LL) return fail(FDB_ERR_LIMIT, "linear: %lld rows x %d features", (long long)c.rows, c.n);
  // The epilogue stores 32 bytes per thread where it may, else 16, which callers' buffers have to allow.
  uintptr_t outs = (uintptr_t)c.out_stride * 2;
  for (int g = 0; g < c.groups; ++g) outs |= reinterpret_cast<uintptr_t>(c.out[g]);
  if ((outs & 15u) != 0) return fail(FDB_ERR_ALIGNMENT, "linear: output rows must be 16-byte aligned");
  LinearArgs a;
  a.sectors = (outs & 31u) == 0;
  a.tm_x = *c.x_map;
  const int box = best->bn / best->cg;
  for (int g = 0; g < 3; ++g) {
    const int s = g < c.groups ? g : 0;
    a.tm_w[g] = c.weight[s]->map[box == 128 ? 2 : (box == 96 ? 1 : 0)];
    a.bias[g] = static_cast<const __nv_bfloat16*>(c.bias[s]);
    a.out[g] = static_cast<__nv_bfloat16*>(c.out[s]);
  }
  a.rows_dev = c.rows_dev;
  a.status = c.status;
  a.rows = c.rows;
  a.out_stride = c.out_stride;
  a.k = c.k;
  a.groups = c.groups;
  a.tiles_n = c.n / best->bn;
  const int units = sms / best->cg;
  const int grid = (int)(best_tiles < units ? best_tiles : units) * best->cg;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
#define FDB_LINEAR(CG, BN) (c.gelu ? launch<CG, BN, true>(a, grid, c.chained, s) : launch<CG, BN, false>(a, grid, c.chained, s))
  if (best->cg == 2) return best->bn == 256 ? FDB_LINEAR(2, 256) : (best->bn == 192 ? FDB_LINEAR(2, 192) : FDB_LINEAR(2, 128));
  return best->bn == 128 ? FDB_LINEAR(1, 128) : FDB_LINEAR(1, 64);
#undef FDB_LINEAR
}

}  // namespace fdb

using namespace fdb;

extern "C" FDB_API int fdb_linear_gelu(const void* x, const void* weight, const void* bias, void* out, int64_t rows,
                                       int32_t in_features, int32_t out_features, int32_t* status, void* stream) {
  clear_error();
  if (x == nullptr || weight == nullptr || out == nullptr)
    return fail(FDB_ERR_INVALID_ARGUMENT, "x, weight and out must not be NULL");
  if (rows < 0 || rows > (int64_t(1) << 31) - 2 * kBM) return fail(FDB_ERR_LIMIT, "rows = %lld", (long long)rows);
  if (in_features <= 0 || in_features % kBK != 0)
    return fail(FDB_ERR_UNSUPPORTED, "in_features = %d: the kernel handles multiples of %d", in_features, kBK);
  if (out_features <= 0 || out_features % 256 != 0)
    return fail(FDB_ERR_UNSUPPORTED, "out_features = %d: the kernel handles multiples of %d", out_features, 256);
  const uintptr_t all = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) |
                        reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(out);
  if ((all & 15u) != 0) return fail(FDB_ERR_ALIGNMENT, "pointers must be 16-byte aligned");
  if (rows == 0) return FDB_OK;

  CUtensorMap xm;
  LinearWeight w;
  int rc = make_linear_input_map(&xm, x, rows, in_features);
  if (rc == FDB_OK) rc = make_linear_maps(&w, weight, out_features, in_features);
  if (rc != FDB_OK) return rc;
  LinearCall c = {};
  c.x_map = &xm;
  c.weight[0] = &w;
  c.bias[0] = bias;
  c.out[0] = out;
  c.rows = rows;
  c.out_stride = out_features;
  c.k = in_features;
  c.n = out_features;
  c.groups = 1;
  c.gelu = true;
  c.status = status;
  return launch_linear(c, stream);
}
