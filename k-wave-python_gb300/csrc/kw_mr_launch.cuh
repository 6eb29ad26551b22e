// Host interface of the mixed-radix passes: parameters and launch shape of one
// axis pass or row stage, launched alone or with those of other plans.
#pragma once
#include "kw_mr_axis.cuh"
#include "kw_mr_rows.cuh"

struct KwMrAxisLaunch {
  MrAxisParams W;
  int kind, gx, gy, threads;  // KwMrKind; column tiles and items
  size_t smem;
};

struct KwMrRowsLaunch {
  MrRowsParams W;
  int stage, odd, dim, blocks, threads;
  size_t smem;
};

// cudaErrorInvalidValue when a job of A writes another job's input
cudaError_t kw_mr_axis_plan(const AxisParams& A, const KwMrLen& L, const float2* tw, int nouter, int nb, int nsm,
                            KwMrAxisLaunch& X);
cudaError_t kw_mr_axis_launch(const KwMrAxisLaunch& X, cudaStream_t st);
void kw_mr_rows_plan(int stage, int nsm, KwMrRowsLaunch& X);
cudaError_t kw_mr_rows_launch(const KwMrRowsLaunch& X, cudaStream_t st);
// Grouped: Ps[m] the members' parameters, map[i] = (member, its block) of block i.
cudaError_t kw_mr_axis_group_launch(int kind, int blocks, int threads, size_t smem, cudaStream_t st,
                                    const MrAxisParams* Ps, const int2* map, bool pdl);
cudaError_t kw_mr_rows_group_launch(int stage, int dim, int blocks, int threads, size_t smem, cudaStream_t st,
                                    const MrRowsParams* Ps, const int2* map, bool pdl);
