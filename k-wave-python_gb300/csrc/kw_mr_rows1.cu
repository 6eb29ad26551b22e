// Mixed-radix row stages: ST_U (kw_mr_rows.cuh).
#include "kw_mr_rows.cuh"

cudaError_t kw_mr_rows_go_1(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st, const MrRowsParams* W,
                            const MrRowsParams* Ps, const int2* map, bool pdl) {
#define KW_GO(STAGE, DIM) kw_mr_rows_go<STAGE, DIM>(odd, blocks, threads, smem, st, W, Ps, map, pdl)
  switch (stage) {
    case ST_U: return dim == 3 ? KW_GO(ST_U, 3) : KW_GO(ST_U, 2);
    default: return cudaErrorInvalidValue;
  }
#undef KW_GO
}
