// What the files of the fused attention backward share (attn_bwd_sm100.cu, attn_bwd_tables_sm100.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace fdb {

// out = core + sums . table, dtable = sums^T . operand, for every head.
struct BwdTablesCall {
  const void* sums;     // bf16 (heads, rows, table_rows)
  const void* table;    // bf16 (heads, table_rows, 64) with the strides below
  int64_t table_row_stride, table_head_stride;
  const void* operand;  // bf16, rows of operand_row_stride elements
  int64_t operand_row_stride, operand_head_stride;
  float* core;          // (heads, 64) per row, rows core_row_stride elements apart; overwritten when table_rows is above 512
  int64_t core_row_stride;
  void* out;            // bf16
  int64_t out_row_stride, out_head_stride;
  void* dtable;         // bf16, laid out like the table
  float* partial;       // bwd_tables_partial_bytes()
  int64_t rows;
  int heads, table_rows;
  int32_t* status;
};
uint64_t bwd_tables_partial_bytes(int64_t rows, int heads, int table_rows);
int launch_bwd_tables(const BwdTablesCall& c, cudaStream_t stream);
// Zeros for the gradient of a table of a call without rows.
int launch_zero_table(void* dtable, int64_t row_stride, int64_t head_stride, int heads, int table_rows, cudaStream_t stream);

}  // namespace fdb
