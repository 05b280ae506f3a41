// Host interface of the one-kernel encoder for at most kSmallRows rows (encoder_small.cu).
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace fdb {

constexpr int kSmallRows = 64, kSmallLayers = 32;

struct SmallLayer {
  const __nv_bfloat16 *wq, *bq, *wk, *bk, *wv, *bv, *wo, *bo, *ln1_gamma, *ln1_beta, *wi, *bi, *wd, *bd, *ln2_gamma, *ln2_beta;
  const __nv_bfloat16 *exp_key, *exp_query;  // NULL without the term
  float ln1_eps, ln2_eps;
};

struct SmallEncoderArgs {
  SmallLayer layer[kSmallLayers];
  int n_layers, hidden, ffn;
  int row_bound;               // rows of the buffers
  const int32_t* rows_dev;     // actual rows, or NULL: row_bound
  const int32_t* cu_seqlens;   // or NULL: `batch` sequences of max_seqlen rows
  int batch, max_seqlen;
  int xrows, d_first;          // of the expanded tables
  float sm_scale;
  const __nv_bfloat16* x;      // (row_bound, hidden): result of the embedding stage
  __nv_bfloat16 *qkv, *ctx, *y, *mid;  // (3, row_bound, hidden), (row_bound, hidden) twice, (row_bound, ffn)
  __nv_bfloat16* out;
  const int32_t* out_index;    // row -> row of out, or NULL
  uint32_t* barrier;           // two words, zero
  int32_t* status;
};

bool small_encoder_covers(int64_t row_bound, int hidden, int ffn, int n_layers);
int launch_small_encoder(const SmallEncoderArgs& a, void* stream);

}  // namespace fdb
