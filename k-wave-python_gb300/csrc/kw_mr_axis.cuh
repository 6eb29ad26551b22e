// Strided-axis transforms on the mixed-radix register passes (kw_mr.cuh).
//
// A block of up to 256 threads owns T columns.  The first pass reads its
// points straight from global memory into registers (one row of T columns is
// one contiguous segment) and the last pass writes its points straight back,
// so a column crosses shared memory np - 1 times per transform.  In operator
// passes the last forward pass, the spectral operator and the first inverse
// pass work on the same registers.
//
//   KIND as in the TMA-fed pass: MK_FWD / MK_INV plain transforms (block
//   row blockIdx.y = buffer), MK_GRAD one input and D outputs (kappa / N folded
//   in once; the y and z gradients share one inverse transform), MK_DIV (the
//   derivative of input a along axis a) and MK_NAB one input per blockIdx.y,
//   its operator in place, MK_GEN any job
//   list (blockIdx.y = distinct input, its jobs one after another).
//
// The columns of all outer blocks are one sequence (column q: outer block
// q / ncols, position q % ncols), so no tile is cut at a plane's edge.
#pragma once
#include "kw_kernels.cuh"
#include "kw_mr.cuh"
#include "kw_regfft.cuh"
#include "kw_tma.cuh"

#define KW_MR_AXIS_SMEM (160 * 1024)  // most dynamic shared memory of a block

enum KwMrKind { MK_FWD = 0, MK_INV = 1, MK_GRAD = 2, MK_DIV = 3, MK_NAB = 4, MK_GEN = 5 };

struct MrAxisParams {
  AxisParams A;
  KwMrLen L;
  const float2* tw;     // pass twiddles of the axis
  KwDivU dcols;         // division by A.ncols
  uint32_t ncoltot;     // A.ncols x outer blocks
  int lgT;
  int inp[KW_MAX_JOBS];  // distinct inputs (MK_GEN)
  int der;               // MK_DIV: OP_DIV or OP_GRAD
  const int* gate;       // grouped source passes: device step counter; the pass is idle from step
  int gate_end;          // gate_end on (null: always on)
  int gx;                // column tiles (grouped launches)
  int pdl;               // launched as a programmatic dependent (host)
};

namespace kwmr {

// One pass over shared memory in place (the middle passes).
template <int R, bool INV>
__device__ __forceinline__ void axis_mid(float2* A, const KwMrLen& L, int l, const float2* tw, int it0, int nit, int cc,
                                         int lgT) {
  const int per = L.per[l], m = L.m[l], ms = L.ms[l] << lgT;
  const float2* w = tw + L.off[l];
  for (int i = it0; i < per; i += nit) {
    const int b = kw_divu(i, L.dm[l]), t = i - b * m;
    float2* a = A + (slot_of(L, l, b, t) << lgT) + cc;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = a[j * ms];
    if (INV) twiddle<R>(v, w + t, m);
    dft<R>(v);
    if (!INV) twiddle<R>(v, w + t, m);
#pragma unroll
    for (int j = 0; j < R; ++j) a[j * ms] = v[j];
  }
}

template <bool INV>
__device__ __forceinline__ void axis_mids(float2* A, const KwMrLen& L, const float2* tw, int it0, int nit, int cc, int lgT) {
  if (L.np == 2) return;
  for (int i = 1; i < L.np - 1; ++i) {
    const int l = INV ? L.np - 1 - i : i;
    switch (L.r[l]) {
#define KW_MR_CASE(R) \
  case R: axis_mid<R, INV>(A, L, l, tw, it0, nit, cc, lgT); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
    __syncthreads();
  }
}

// First forward pass: global rows -> shared memory.
template <int R>
__device__ __forceinline__ void axis_first_fwd(float2* A, const MrAxisParams& W, const float2* in, bool act, int it0,
                                               int nit, int cc) {
  const KwMrLen& L = W.L;
  const int m = L.m[0], ms = L.ms[0] << W.lgT;
  const uint32_t xs = (uint32_t)W.A.xs;
  for (int t = it0; t < m; t += nit) {
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = act ? in[(uint32_t)(t + j * m) * xs] : make_float2(0.f, 0.f);
    dft<R>(v);
    twiddle<R>(v, W.tw + t, m);
    float2* a = A + (slot_of(L, 0, 0, t) << W.lgT) + cc;
#pragma unroll
    for (int j = 0; j < R; ++j) a[j * ms] = v[j];
  }
}

// Last forward pass to global rows.
template <int R>
__device__ __forceinline__ void axis_last_fwd(const float2* A, const MrAxisParams& W, float2* out, bool act, int it0,
                                              int nit, int cc) {
  const KwMrLen& L = W.L;
  const uint32_t xs = (uint32_t)W.A.xs;
  for (int b = it0; b < L.q; b += nit) {
    const float2* a = A + ((b * L.mp) << W.lgT) + cc;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = a[j << W.lgT];
    dft<R>(v);
    const int f = kw_mr_freq(L, b);
    if (act) {
#pragma unroll
      for (int j = 0; j < R; ++j) out[(uint32_t)(f + j * L.q) * xs] = v[j];
    }
  }
}

// First inverse pass: global rows (frequencies) -> shared memory, parts exchanged.
template <int R>
__device__ __forceinline__ void axis_first_inv(float2* A, const MrAxisParams& W, const float2* in, bool act, int it0,
                                               int nit, int cc) {
  const KwMrLen& L = W.L;
  const uint32_t xs = (uint32_t)W.A.xs;
  for (int b = it0; b < L.q; b += nit) {
    const int f = kw_mr_freq(L, b);
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = act ? swp(in[(uint32_t)(f + j * L.q) * xs]) : make_float2(0.f, 0.f);
    dft<R>(v);
    float2* a = A + ((b * L.mp) << W.lgT) + cc;
#pragma unroll
    for (int j = 0; j < R; ++j) a[j << W.lgT] = v[j];
  }
}

// Last inverse pass to global rows (parts exchanged back); store(row, value).
template <int R, class ST>
__device__ __forceinline__ void axis_last_inv(const float2* A, const MrAxisParams& W, int it0, int nit, int cc, ST store) {
  const KwMrLen& L = W.L;
  const int m = L.m[0], ms = L.ms[0] << W.lgT;
  for (int t = it0; t < m; t += nit) {
    const float2* a = A + (slot_of(L, 0, 0, t) << W.lgT) + cc;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = a[j * ms];
    twiddle<R>(v, W.tw + t, m);
    dft<R>(v);
#pragma unroll
    for (int j = 0; j < R; ++j) store(t + j * m, swp(v[j]));
  }
}

__device__ __forceinline__ float mr_kk(const AxisParams& A, int x, const ColK& g) {
  const float kx = __ldg(A.k[0] + x);
  float kk = __fadd_rn(__fmul_rn(kx, kx), g.ky2);
  if (A.ndim == 3) kk = __fadd_rn(kk, g.kz2);
  return kk;
}

__device__ __forceinline__ float mr_kappa(const AxisParams& A, float kk) {
  if (!A.use_kspace) return 1.f;
  const float y = (A.kcoef * A.kcoef) * kk;
  if (!(y < 9.0f)) {
    const float x = sqrtf(y);
    return sinf(x) / x;
  }
  return kwreg::sinc_taylor_sq(y);
}

// |k|^p from |k|^2 (0 at k = 0), p the exponent of fractional Laplacian q: with the
// centre c of the eighth of an octave that |k|^2 lies in, c^(p/2) (1 + z)^(p/2), z =
// |k|^2 / c - 1, |z| <= 1/17.  c^(p/2) comes from a table in two parts, the rest is the
// binomial series to z^6 (its next term is below 2e-9), so that nothing but the last
// addition rounds to float: errors of 2.5e-8 rms and 6.2e-8 at most for p -1.4 to 0.9,
// against 2.0e-8..4.5e-8 and 1.5e-7 for powf(|k|, p) behind a square root and
// 4.1e-8..7.9e-8 and 6e-7, with a mean of up to 6e-8, for exp2f(p/2 log2f(|k|^2)).
__device__ __forceinline__ float mr_kpow(const AxisParams& A, int q, float kk) {
  const uint32_t i = min((uint32_t)(__float_as_int(kk) >> 20) - A.kpow_first, A.kpow_n - 1u);
  const float4 e = __ldg(A.kpow[q] + i);  // 1 / c, c^(p/2) in two parts
  const float* b = A.kpow_b[q];
  const float z = fmaf(kk, e.x, -1.f);
  float s = fmaf(b[5], z, b[4]);
#pragma unroll
  for (int j = 3; j >= 0; --j) s = fmaf(s, z, b[j]);
  return kk == 0.f ? 0.f : e.y + fmaf(s * z, e.y, e.z);
}

// x / (N_total gain) at x frequency kx: scaled() with axis 0's own gain.
__device__ __forceinline__ float mr_scaled(const AxisParams& A, float x, float lo, int kx) {
  return scaled(A, x, lo + __ldg(A.eps[0] + kx));
}

// Column-constant 1-D factor of an operator along axis 1 or 2.
__device__ __forceinline__ float2 mr_col_factor(const AxisParams& A, int op, int axis, const ColK& g) {
  if (axis == 0 || !g.valid) return make_float2(0.f, 0.f);
  const int ai = (axis == 1) ? g.a1 : g.a2;
  switch (op) {
    case OP_GRAD: return __ldg(A.fg[axis] + ai);
    case OP_DIV: return __ldg(A.fd[axis] + ai);
    case OP_UNSTAG: return __ldg(A.us[axis] + ai);
    default: return make_float2(0.f, 0.f);
  }
}

// Operator of job J at x frequency x (any operator).
__device__ __forceinline__ float2 mr_op(const AxisParams& A, const AxisJob& J, int x, const ColK& g, float2 fcol, float lo) {
  switch (J.op) {
    case OP_GRAD:
    case OP_DIV: {
      const float kp = mr_scaled(A, mr_kappa(A, mr_kk(A, x, g)), lo, x);
      const float2 f = J.axis == 0 ? __ldg((J.op == OP_GRAD ? A.fg[0] : A.fd[0]) + x) : fcol;
      return make_float2(f.x * kp, f.y * kp);
    }
    case OP_NAB1:
    case OP_NAB2: {
      return make_float2(mr_scaled(A, mr_kpow(A, J.op == OP_NAB1 ? 0 : 1, mr_kk(A, x, g)), lo, x), 0.f);
    }
    case OP_SKAPPA:
      return make_float2(mr_scaled(A, A.use_kspace ? cosf(A.kcoef * sqrtf(mr_kk(A, x, g))) : 1.f, lo, x), 0.f);
    case OP_WIN: {
      float r2 = A.wc[0][x] + A.wc[1][g.a1];
      if (A.ndim == 3) r2 += A.wc[2][g.a2];
      return make_float2(mr_scaled(A, window_at(A.wtab, A.wlen, A.wrad, r2), lo, x), 0.f);
    }
    default: {
      const float2 f = J.axis == 0 ? __ldg(A.us[0] + x) : fcol;
      return make_float2(mr_scaled(A, f.x, lo, x), mr_scaled(A, f.y, lo, x));
    }
  }
}

// Last forward pass, operator, first inverse pass on the same registers.
template <int R, int KIND>
__device__ __forceinline__ void axis_turn(float2* A, float2* B, const MrAxisParams& W, const ColK& g, bool on, int item,
                                          float2 fcol, float lo, int it0, int nit, int cc) {
  const KwMrLen& L = W.L;
  const AxisParams& P = W.A;
  for (int b = it0; b < L.q; b += nit) {
    const int s0 = ((b * L.mp) << W.lgT) + cc;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = A[s0 + (j << W.lgT)];
    dft<R>(v);
    const int f = kw_mr_freq(L, b);
    if constexpr (KIND == MK_GRAD) {
      float2 y[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int x = f + j * L.q;
        const float kp = on ? mr_scaled(P, mr_kappa(P, mr_kk(P, x, g)), lo, x) : 0.f;
        v[j] = make_float2(v[j].x * kp, v[j].y * kp);
        y[j] = swp(cmulf(__ldg(P.fg[0] + x), v[j]));
        v[j] = swp(v[j]);
      }
      dft<R>(y);
#pragma unroll
      for (int j = 0; j < R; ++j) B[s0 + (j << W.lgT)] = y[j];
    } else if constexpr (KIND == MK_DIV) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int x = f + j * L.q;
        const float kp = on ? mr_scaled(P, mr_kappa(P, mr_kk(P, x, g)), lo, x) : 0.f;
        const float2 d = item == 0 ? __ldg((W.der == OP_GRAD ? P.fg[0] : P.fd[0]) + x) : fcol;
        v[j] = swp(cmulf(make_float2(d.x * kp, d.y * kp), v[j]));
      }
    } else if constexpr (KIND == MK_NAB) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int x = f + j * L.q;
        const float a = on ? mr_scaled(P, mr_kpow(P, item, mr_kk(P, x, g)), lo, x) : 0.f;
        v[j] = make_float2(v[j].y * a, v[j].x * a);
      }
    }
    dft<R>(v);
#pragma unroll
    for (int j = 0; j < R; ++j) A[s0 + (j << W.lgT)] = v[j];
  }
}

// One pass over the last radix's points in place, without twiddles (MK_GEN).
template <int R>
__device__ __forceinline__ void axis_block_dft(float2* A, const KwMrLen& L, int it0, int nit, int cc, int lgT) {
  for (int b = it0; b < L.q; b += nit) {
    float2* a = A + ((b * L.mp) << lgT) + cc;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = a[j << lgT];
    dft<R>(v);
#pragma unroll
    for (int j = 0; j < R; ++j) a[j << lgT] = v[j];
  }
}

__device__ __forceinline__ void axis_blocks(float2* A, const KwMrLen& L, int it0, int nit, int cc, int lgT) {
  switch (L.rl) {
#define KW_MR_CASE(R) \
  case R: axis_block_dft<R>(A, L, it0, nit, cc, lgT); break;
    KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
    default: break;
  }
  __syncthreads();
}

}  // namespace kwmr

template <int KIND>
__device__ __forceinline__ void mr_axis_body(const MrAxisParams& W, int tile, int item) {
  using namespace kwmr;
  extern __shared__ float4 smem_f4[];
  const KwMrLen& L = W.L;
  const AxisParams& P = W.A;
  const int T = 1 << W.lgT;
  float2* A = reinterpret_cast<float2*>(smem_f4);
  float2* B = A + ((size_t)L.slots << W.lgT);  // MK_GRAD, MK_GEN
  const int cc = threadIdx.x & (T - 1), it0 = threadIdx.x >> W.lgT, nit = blockDim.x >> W.lgT;
  const uint32_t q = ((uint32_t)tile << W.lgT) + cc;
  const bool act = q < W.ncoltot;
  const uint32_t outer = act ? (uint32_t)kw_divu((int)q, W.dcols) : 0u;
  const uint32_t c = act ? q - outer * (uint32_t)P.ncols : 0u;
  const uint32_t base = outer * (uint32_t)P.os + c;
  const uint32_t xs = (uint32_t)P.xs;
  // up to here and in the column's factors only the parameters and the plan's tables are read
  if constexpr (KIND == MK_FWD || KIND == MK_INV) kwtma::grid_dep_wait();

  if constexpr (KIND == MK_FWD) {
    float2* buf = P.bufs[P.plain[item]] + base;
    switch (L.r[0]) {
#define KW_MR_CASE(R) \
  case R: axis_first_fwd<R>(A, W, buf, act, it0, nit, cc); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
    __syncthreads();
    axis_mids<false>(A, L, W.tw, it0, nit, cc, W.lgT);
    kwtma::grid_dep_launch();
    switch (L.rl) {
#define KW_MR_CASE(R) \
  case R: axis_last_fwd<R>(A, W, buf, act, it0, nit, cc); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
  } else if constexpr (KIND == MK_INV) {
    float2* buf = P.bufs[P.plain[item]] + base;
    switch (L.rl) {
#define KW_MR_CASE(R) \
  case R: axis_first_inv<R>(A, W, buf, act, it0, nit, cc); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
    __syncthreads();
    axis_mids<true>(A, L, W.tw, it0, nit, cc, W.lgT);
    kwtma::grid_dep_launch();
    auto store = [&](int row, float2 v) {
      if (act) buf[(uint32_t)row * xs] = v;
    };
    switch (L.r[0]) {
#define KW_MR_CASE(R) \
  case R: axis_last_inv<R>(A, W, it0, nit, cc, store); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
  } else {
    const int ib = KIND == MK_GRAD ? (int)B_P : KIND == MK_GEN ? W.inp[item] : item;
    const float2* in = P.bufs[ib] + base;
    const ColK g = col_geometry(P, (int)c);
    const bool on = act && g.valid;
    const float lo = col_scale_lo(P, g.a1, g.a2, g.valid);
    kwtma::grid_dep_wait();
    switch (L.r[0]) {
#define KW_MR_CASE(R) \
  case R: axis_first_fwd<R>(A, W, in, act, it0, nit, cc); break;
      KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
      default: break;
    }
    __syncthreads();
    axis_mids<false>(A, L, W.tw, it0, nit, cc, W.lgT);
    if constexpr (KIND != MK_GEN) {
      const float2 fcol = KIND == MK_DIV ? mr_col_factor(P, W.der, item, g) : make_float2(0.f, 0.f);
      switch (L.rl) {
#define KW_MR_CASE(R) \
  case R: axis_turn<R, KIND>(A, B, W, g, on, item, fcol, lo, it0, nit, cc); break;
        KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
        default: break;
      }
      __syncthreads();
      axis_mids<true>(A, L, W.tw, it0, nit, cc, W.lgT);
      if constexpr (KIND == MK_GRAD) {
        axis_mids<true>(B, L, W.tw, it0, nit, cc, W.lgT);
        kwtma::grid_dep_launch();
        const float2 f1 = mr_col_factor(P, OP_GRAD, 1, g);
        const float2 f2 = P.ndim == 3 ? mr_col_factor(P, OP_GRAD, 2, g) : make_float2(0.f, 0.f);
        float2* o0 = P.bufs[0] + base;
        float2* o1 = P.bufs[1] + base;
        float2* o2 = P.ndim == 3 ? P.bufs[2] + base : nullptr;
        auto st_x = [&](int row, float2 v) {
          if (act) o0[(uint32_t)row * xs] = v;
        };
        auto st_yz = [&](int row, float2 v) {
          if (!act) return;
          const uint32_t o = (uint32_t)row * xs;
          o1[o] = cmulf(f1, v);
          if (o2) o2[o] = cmulf(f2, v);
        };
        switch (L.r[0]) {
#define KW_MR_CASE(R)                             \
  case R:                                         \
    axis_last_inv<R>(B, W, it0, nit, cc, st_x);   \
    axis_last_inv<R>(A, W, it0, nit, cc, st_yz);  \
    break;
          KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
          default: break;
        }
      } else {
        kwtma::grid_dep_launch();
        float2* out = P.bufs[ib] + base;
        auto store = [&](int row, float2 v) {
          if (act) out[(uint32_t)row * xs] = v;
        };
        switch (L.r[0]) {
#define KW_MR_CASE(R) \
  case R: axis_last_inv<R>(A, W, it0, nit, cc, store); break;
          KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
          default: break;
        }
      }
    } else {
      axis_blocks(A, L, it0, nit, cc, W.lgT);
      for (int jj = 0; jj < P.njobs; ++jj) {
        const AxisJob J = P.jobs[jj];
        if (J.in != ib) continue;
        const float2 fcol = mr_col_factor(P, J.op, J.axis, g);
        // the spectrum stays in A; operator times spectrum, parts exchanged, goes to B
        for (int e = it0; e < L.n; e += nit) {
          const int b = kw_divu(e, L.drl), j = e - b * L.rl;
          const int s = ((b * L.mp + j) << W.lgT) + cc;
          B[s] = on ? swp(cmulf(mr_op(P, J, kw_mr_freq(L, b) + j * L.q, g, fcol, lo), A[s])) : make_float2(0.f, 0.f);
        }
        __syncthreads();
        axis_blocks(B, L, it0, nit, cc, W.lgT);
        axis_mids<true>(B, L, W.tw, it0, nit, cc, W.lgT);
        float2* out = P.bufs[J.out] + base;
        auto store = [&](int row, float2 v) {
          if (act) out[(uint32_t)row * xs] = v;
        };
        switch (L.r[0]) {
#define KW_MR_CASE(R) \
  case R: axis_last_inv<R>(B, W, it0, nit, cc, store); break;
          KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
          default: break;
        }
        __syncthreads();
      }
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(256, (KIND == MK_GRAD || KIND == MK_GEN) ? 2 : 3)
    k_mr_axis(const __grid_constant__ MrAxisParams W) {
  mr_axis_body<KIND>(W, blockIdx.x, blockIdx.y);
}

// One pass of several plans: block i works on member map[i].x, its block
// map[i].y (item x tiles + tile).
template <int KIND>
__global__ void __launch_bounds__(256, (KIND == MK_GRAD || KIND == MK_GEN) ? 2 : 3)
    k_mr_axis_group(const MrAxisParams* __restrict__ Ps, const int2* __restrict__ map) {
  __shared__ __align__(16) MrAxisParams sp;
  const int2 me = map[blockIdx.x];
  const int* src = reinterpret_cast<const int*>(Ps + me.x);
  for (int w = threadIdx.x; w < (int)(sizeof(MrAxisParams) / 4); w += blockDim.x) reinterpret_cast<int*>(&sp)[w] = src[w];
  __syncthreads();
  kwtma::grid_dep_wait();
  if (sp.gate && *sp.gate >= sp.gate_end) return;
  const int item = me.y / sp.gx;
  mr_axis_body<KIND>(sp, me.y - item * sp.gx, item);
}

// One plan's pass, or (Ps set) the grouped pass over `grid.x` blocks.  Only a launch
// that needs it asks for more shared memory (one constant, so that plans of several
// threads never lower it): the call loads the kernel.  When set-up asked for every
// kernel of a length, used or not, the first 128^2 run of a process took 91 ms, so 39.
template <int KIND>
static cudaError_t kw_mr_axis_go(dim3 grid, int threads, size_t smem, cudaStream_t st, const MrAxisParams* W,
                                 const MrAxisParams* Ps, const int2* map, bool pdl) {
  if (smem > 40 * 1024) {
    const cudaError_t e =
        Ps ? cudaFuncSetAttribute(k_mr_axis_group<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, KW_MR_AXIS_SMEM)
           : cudaFuncSetAttribute(k_mr_axis<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, KW_MR_AXIS_SMEM);
    if (e != cudaSuccess) return e;
  }
  if (Ps) return kwtma::launch_k(k_mr_axis_group<KIND>, grid, dim3(threads), smem, st, pdl, Ps, map);
  return kwtma::launch_k(k_mr_axis<KIND>, grid, dim3(threads), smem, st, W->pdl != 0, *W);
}

#define KW_MR_AXIS_DEFINE(name, KIND)                                                                              \
  cudaError_t kw_mr_axis_go_##name(dim3 grid, int threads, size_t smem, cudaStream_t st, const MrAxisParams* W,    \
                                   const MrAxisParams* Ps, const int2* map, bool pdl) {                            \
    return kw_mr_axis_go<KIND>(grid, threads, smem, st, W, Ps, map, pdl);                                          \
  }
