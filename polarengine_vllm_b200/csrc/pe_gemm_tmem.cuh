// Arguments and launcher of the tensor-core matmul for some hundred activation rows and for grouped launches
// (pe_gemm_tmem.cu).
#pragma once
#include "pe_gemm.cuh"

namespace pe {

struct TmemGemmArgs {
  const __half* norms; int64_t ld_norms;
  const float* ct; int n_levels;
  void* y; int y_dtype; int64_t ld_y;
  const __half* bias;
  int M, N, nb;          // rows, output columns, 128-blocks of K
  int tiles_m, tiles_n;  // dense launch: tiles of `tok` activation rows x 128 * halves weight rows
  int tok, halves, ksplit;
  float* part;           // [ksplit][M][N] fp32 when ksplit > 1
  int xbox;              // activation rows per TMA copy
  int x_stage, nx;       // bytes and number of the activation stages
  const int4* gtiles;    // grouped launch: per tile (first activation row, rows, first weight row inside the expert, expert)
  const int* n_gtiles;
  int64_t expert_norms;  // halves between the norms of consecutive experts
  int expert_codes;      // code rows between consecutive experts
  int up_row;            // > 0: the second half of a tile is weight row n + up_row, and y = silu(first) * second
  int* status;
};

int launch_gemm_tmem(TmemGemmArgs& a, const void* codes, int packed, int64_t ld_codes, int64_t code_rows, const void* xq, int64_t x_total, int units,
                     int sms, cudaStream_t st);

}  // namespace pe
