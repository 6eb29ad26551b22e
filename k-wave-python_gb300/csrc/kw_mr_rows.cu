// Host side of the mixed-radix row stages: block geometry and launch.
#include "kw_mr_launch.cuh"

#include <algorithm>

#define KW_MR_ROWS_DECL(i)                                                                                        \
  cudaError_t kw_mr_rows_go_##i(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st, \
                                const MrRowsParams* W, const MrRowsParams* Ps, const int2* map, bool pdl);
KW_MR_ROWS_DECL(1)
KW_MR_ROWS_DECL(2)
KW_MR_ROWS_DECL(3)
KW_MR_ROWS_DECL(4)
KW_MR_ROWS_DECL(5)

// Launch shape of one row stage for nsm SMs to fill.  X.W holds Q, L, tw and
// pos; the block geometry is set here: P threads per sequence, so that a thread
// has 8 points of each component (the largest radices then occupy every thread
// of a pass), blocks of about 128 threads, fewer rows per block and fewer
// points per thread while the grid would leave SMs without work.
void kw_mr_rows_plan(int stage, int nsm, KwMrRowsLaunch& X) {
  MrRowsParams& W = X.W;
  const RowsParams& Q = W.Q;
  const int D = Q.ndim, M = W.L.n, odd = !Q.even;
  const bool ku = Q.srcu_on[0] || Q.srcu_on[1] || Q.srcu_on[2];
  bool sparse = false;
  for (int a = 0; a < D; ++a) sparse |= Q.src[a].active != 0;
  // components at once, and regions of shared memory (kw_mr_rows.cuh)
  const int nq = stage == ST_U || stage == ST_RHO || stage >= ST_ADJ_A ? D : stage == ST_EOS ? 2 : 1;
  const int regions = nq + (stage == ST_RHO && (Q.srcp_on || sparse) ? 1 : stage == ST_U && ku ? D : 0);
  const int nseq = odd ? (Q.nrows + 1) / 2 : Q.nrows;
  int P = std::min((M + 7) / 8, KW_MR_THREADS / nq);
  int SB = std::max(1, 128 / (nq * P));
  while (SB > 1 && nseq < 4 * nsm * SB) SB = (SB + 1) / 2;
  while (2 * P * SB * nq <= 64 && P < M) P *= 2;
  W.pdl = 0;
  W.SB = SB;
  W.rpb = odd ? 2 * SB : SB;
  W.P = P;
  W.PT = nq * P;
  W.G = SB * nq;
  W.region = SB * W.L.slots;
  W.ncp = (M + 1) / 2;
  W.half = !odd && M % 2 == 0 ? M / 2 : 0;
  W.dP = kw_divu_make((uint32_t)P);
  W.dPT = kw_divu_make((uint32_t)W.PT);
  W.dSB = kw_divu_make((uint32_t)SB);
  W.dN1 = kw_divu_make((uint32_t)(D == 3 ? Q.N1 : 1));
  X.stage = stage;
  X.odd = odd;
  X.dim = D;
  X.blocks = (Q.nrows + W.rpb - 1) / W.rpb;
  X.threads = SB * nq * P;
  X.smem = sizeof(float2) * (size_t)regions * W.region;
}

static cudaError_t rows_go(int stage, int odd, int dim, int blocks, int threads, size_t smem, cudaStream_t st,
                           const MrRowsParams* W, const MrRowsParams* Ps, const int2* map, bool pdl) {
  if (stage == ST_U) return kw_mr_rows_go_1(stage, odd, dim, blocks, threads, smem, st, W, Ps, map, pdl);
  if (stage == ST_RHO) return kw_mr_rows_go_2(stage, odd, dim, blocks, threads, smem, st, W, Ps, map, pdl);
  if (stage == ST_EOS || stage == ST_SRC) return kw_mr_rows_go_3(stage, odd, dim, blocks, threads, smem, st, W, Ps, map, pdl);
  if (stage >= ST_ADJ_A) return kw_mr_rows_go_4(stage, odd, dim, blocks, threads, smem, st, W, Ps, map, pdl);
  return kw_mr_rows_go_5(stage, odd, dim, blocks, threads, smem, st, W, Ps, map, pdl);
}

cudaError_t kw_mr_rows_launch(const KwMrRowsLaunch& X, cudaStream_t st) {
  return rows_go(X.stage, X.odd, X.dim, X.blocks, X.threads, X.smem, st, &X.W, nullptr, nullptr, false);
}

cudaError_t kw_mr_rows_group_launch(int stage, int dim, int blocks, int threads, size_t smem, cudaStream_t st,
                                    const MrRowsParams* Ps, const int2* map, bool pdl) {
  return rows_go(stage, 0, dim, blocks, threads, smem, st, nullptr, Ps, map, pdl);
}
