// Mixed-radix row stages: ST_EOS ST_SRC (kw_mr_rows.cuh).
#include "kw_mr_rows.cuh"

cudaError_t kw_mr_rows_go_3(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st, const MrRowsParams* W,
                            const MrRowsParams* Ps, const int2* map, bool pdl) {
  (void)dim;
#define KW_GO(STAGE, DIM) kw_mr_rows_go<STAGE, DIM>(odd, blocks, threads, smem, st, W, Ps, map, pdl)
  switch (stage) {
    case ST_EOS: return KW_GO(ST_EOS, 0);
    case ST_SRC: return KW_GO(ST_SRC, 0);
    default: return cudaErrorInvalidValue;
  }
#undef KW_GO
}
