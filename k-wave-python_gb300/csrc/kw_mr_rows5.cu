// Mixed-radix row stages: ST_INIT ST_UREC ST_P0FFT ST_P0BACK (kw_mr_rows.cuh).
#include "kw_mr_rows.cuh"

cudaError_t kw_mr_rows_go_5(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st, const MrRowsParams* W,
                            const MrRowsParams* Ps, const int2* map, bool pdl) {
  (void)dim;
#define KW_GO(STAGE, DIM) kw_mr_rows_go<STAGE, DIM>(odd, blocks, threads, smem, st, W, Ps, map, pdl)
  switch (stage) {
    case ST_INIT: return KW_GO(ST_INIT, 0);
    case ST_UREC: return KW_GO(ST_UREC, 0);
    case ST_P0FFT: return KW_GO(ST_P0FFT, 0);
    case ST_P0BACK: return KW_GO(ST_P0BACK, 0);
    default: return cudaErrorInvalidValue;
  }
#undef KW_GO
}
