// Mixed-radix row stages: ST_ADJ_A ST_ADJ_B ST_ADJ_C ST_ADJ_D ST_ADJ_E (kw_mr_rows.cuh).
#include "kw_mr_rows.cuh"

cudaError_t kw_mr_rows_go_4(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st, const MrRowsParams* W,
                            const MrRowsParams* Ps, const int2* map, bool pdl) {
  (void)dim;
#define KW_GO(STAGE, DIM) kw_mr_rows_go<STAGE, DIM>(odd, blocks, threads, smem, st, W, Ps, map, pdl)
  switch (stage) {
    case ST_ADJ_A: return KW_GO(ST_ADJ_A, 0);
    case ST_ADJ_B: return KW_GO(ST_ADJ_B, 0);
    case ST_ADJ_C: return KW_GO(ST_ADJ_C, 0);
    case ST_ADJ_D: return KW_GO(ST_ADJ_D, 0);
    case ST_ADJ_E: return KW_GO(ST_ADJ_E, 0);
    default: return cudaErrorInvalidValue;
  }
#undef KW_GO
}
