// Host side of the mixed-radix axis passes: pass kind, tile width, launch.
#include "kw_mr_launch.cuh"

#define KW_MR_AXIS_DECL(name)                                                                                    \
  cudaError_t kw_mr_axis_go_##name(dim3 grid, int threads, size_t smem, cudaStream_t st, const MrAxisParams* W,  \
                                   const MrAxisParams* Ps, const int2* map, bool pdl);
KW_MR_AXIS_DECL(fwd)
KW_MR_AXIS_DECL(inv)
KW_MR_AXIS_DECL(grad)
KW_MR_AXIS_DECL(div)
KW_MR_AXIS_DECL(nab)
KW_MR_AXIS_DECL(gen)

namespace {
// Columns per block (a power of two) for `nbuf` column buffers of length L:
// 16 (a row of a tile is then one 128-byte line) as long as three blocks of
// plain passes fit an SM, fewer for long axes; halved down to 4 (one 32-byte
// sector) while the grid would leave SMs without a block.
int mr_tile_log2(const KwMrLen& L, int nbuf, long long ncoltot, int nitems, int nsm) {
  int lg = 4;
  while (lg > 0 && ((size_t)L.slots * sizeof(float2) << lg) * nbuf > 72 * 1024) --lg;
  while (lg > 2 && ((ncoltot + (1 << lg) - 1) >> lg) * nitems < 2LL * nsm) --lg;
  return lg;
}
}  // namespace

// Parameters and launch shape of one pass along an axis: A in plain mode over
// `nb` buffers, or its job list; nouter outer blocks of A.ncols columns; nsm
// SMs to fill.
cudaError_t kw_mr_axis_plan(const AxisParams& A, const KwMrLen& L, const float2* tw, int nouter, int nb, int nsm,
                            KwMrAxisLaunch& X) {
  MrAxisParams& W = X.W;
  W.A = A;
  W.L = L;
  W.tw = tw;
  W.dcols = kw_divu_make((uint32_t)A.ncols);
  W.ncoltot = (uint32_t)A.ncols * (uint32_t)nouter;
  W.gate = nullptr;
  W.gate_end = 0;
  W.pdl = 0;
  int nitems = nb, nbuf = 1;
  if (A.mode < 2) {
    X.kind = A.mode == 0 ? MK_FWD : MK_INV;
  } else {
    const int D = A.ndim;
    bool grad = A.njobs == D, div = A.njobs == D && (A.jobs[0].op == OP_DIV || A.jobs[0].op == OP_GRAD);
    bool nab = A.njobs >= 1 && A.njobs <= 2;
    int ni = 0;
    for (int j = 0; j < A.njobs; ++j) {
      const AxisJob& J = A.jobs[j];
      grad &= J.in == B_P && J.out == j && J.op == OP_GRAD && J.axis == j;
      div &= J.in == j && J.out == j && J.op == A.jobs[0].op && J.axis == j;
      nab &= J.in == j && J.out == j && J.op == (j == 0 ? OP_NAB1 : OP_NAB2);
      bool seen = false;
      for (int i = 0; i < ni; ++i) seen |= W.inp[i] == J.in;
      if (!seen) W.inp[ni++] = J.in;
    }
    // the inputs run in blocks of their own: no job may write another one's input
    for (int j = 0; j < A.njobs; ++j)
      for (int i = 0; i < ni; ++i)
        if (A.jobs[j].out == W.inp[i] && A.jobs[j].in != W.inp[i]) return cudaErrorInvalidValue;
    X.kind = grad ? MK_GRAD : div ? MK_DIV : nab ? MK_NAB : MK_GEN;
    W.der = A.jobs[0].op;
    nitems = grad ? 1 : div ? D : nab ? A.njobs : ni;
    nbuf = (X.kind == MK_GRAD || X.kind == MK_GEN) ? 2 : 1;
  }
  W.lgT = mr_tile_log2(L, nbuf, W.ncoltot, nitems, nsm);
  const int T = 1 << W.lgT;
  int per = 0;
  for (int l = 0; l < L.np; ++l) per = L.per[l] > per ? L.per[l] : per;
  X.threads = (per * T + 31) / 32 * 32;
  if (X.threads > 256) X.threads = 256;
  X.smem = ((size_t)L.slots * sizeof(float2) << W.lgT) * nbuf;
  if (X.smem > KW_MR_AXIS_SMEM) return cudaErrorInvalidValue;
  W.gx = X.gx = (int)((W.ncoltot + T - 1) / T);
  X.gy = nitems;
  return cudaSuccess;
}

static cudaError_t axis_go(int kind, dim3 grid, int threads, size_t smem, cudaStream_t st, const MrAxisParams* W,
                           const MrAxisParams* Ps, const int2* map, bool pdl) {
  switch (kind) {
    case MK_FWD: return kw_mr_axis_go_fwd(grid, threads, smem, st, W, Ps, map, pdl);
    case MK_INV: return kw_mr_axis_go_inv(grid, threads, smem, st, W, Ps, map, pdl);
    case MK_GRAD: return kw_mr_axis_go_grad(grid, threads, smem, st, W, Ps, map, pdl);
    case MK_DIV: return kw_mr_axis_go_div(grid, threads, smem, st, W, Ps, map, pdl);
    case MK_NAB: return kw_mr_axis_go_nab(grid, threads, smem, st, W, Ps, map, pdl);
    default: return kw_mr_axis_go_gen(grid, threads, smem, st, W, Ps, map, pdl);
  }
}

cudaError_t kw_mr_axis_launch(const KwMrAxisLaunch& X, cudaStream_t st) {
  return axis_go(X.kind, dim3(X.gx, X.gy), X.threads, X.smem, st, &X.W, nullptr, nullptr, false);
}

cudaError_t kw_mr_axis_group_launch(int kind, int blocks, int threads, size_t smem, cudaStream_t st,
                                    const MrAxisParams* Ps, const int2* map, bool pdl) {
  return axis_go(kind, dim3(blocks), threads, smem, st, nullptr, Ps, map, pdl);
}
