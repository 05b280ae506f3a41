// Host interface of the linear-layer kernels (linear_sm100.cu) for the other translation units.
#pragma once

#include <cuda.h>

#include <cstdint>

namespace fdb {

// Tensor maps of one (n, k) weight, one per number of weight rows a CTA loads at a time.
constexpr int kLinearBoxRows[3] = {64, 96, 128};
struct LinearWeight { CUtensorMap map[3]; };

struct LinearCall {
  const CUtensorMap* x_map;      // make_linear_input_map over at least `rows` rows
  const LinearWeight* weight[3]; // `groups` weights of the same shape over the same x
  const void* bias[3];           // bf16 (n) or NULL
  void* out[3];                  // bf16 rows of n, out_stride elements apart
  int64_t rows, out_stride;
  const int32_t* rows_dev;       // device: the actual number of rows (at most `rows`), or NULL
  int k, n, groups;              // k a multiple of 64, n of 64
  bool gelu;
  bool chained;                  // launch with programmatic stream serialisation (the kernel before allows it)
  int32_t* status;
};

int make_linear_maps(LinearWeight* w, const void* weight, int n, int k);
int make_linear_input_map(CUtensorMap* m, const void* x, int64_t rows, int k);
int launch_linear(const LinearCall& c, void* stream);

}  // namespace fdb
