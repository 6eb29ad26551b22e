// Row stages of the time step on the mixed-radix register passes (kw_mr.cuh),
// for any row length whose transform factors there.
//
// A block works on SB row sequences in shared memory.  A sequence is one
// complex transform of M points: an even row of L = 2 M reals (points 2n,
// 2n+1), or a pair of odd rows of L = M reals (row 2s real part, row 2s + 1
// imaginary part), so that odd lengths cost no more per cell than even ones.
// All components of a stage are in the block at once, each in its own region
// of SB sequences:
//
//   c2r   half spectra from global memory, two frequencies k and M - k at a
//         time, into frequency order, parts exchanged; inverse passes
//   stage physics: a thread takes a point of a row with all its components, so
//         sums over components stay in registers
//   r2c   forward passes, then frequencies k and M - k to global memory
//
// One set of passes (and of barriers) thus serves all components, and a
// butterfly pass has enough work for every thread of a small block; five or
// six blocks on an SM hide the latency of one block's loads and barriers.
// Each block asks for its rows of every array in L2 when it starts.  Each
// direction's passes are expanded once per kernel.
// The arithmetic of the physics and its order follow kwave/solvers/
// kspace_solver.py (Simulation.step, :691-747) as the generic row kernel does.
#pragma once
#include "kw_kernels.cuh"
#include "kw_mr.cuh"
#include "kw_tma.cuh"

#define KW_MR_THREADS 192  // most threads of a row block
#define KW_MR_MAXM 1024    // most points of a sequence
// Most dynamic shared memory of a row block: one sequence of 1024 points in each
// of up to six regions, slots of up to 3 / 2 of the points (a last radix of 2 is
// padded to 3): 72 KB.
#define KW_MR_ROWS_SMEM (96 * 1024)

struct MrRowsParams {
  RowsParams Q;
  KwMrLen L;
  const float2* tw;       // pass twiddles of the row transform
  const uint32_t* pos;    // slots of frequencies k (low half) and M - k (high half), k < M
  int pdl;                // launched as a programmatic dependent (host)
  int SB, rpb;            // sequences per region and rows per block
  int P, PT, G;           // threads per sequence (c2r, r2c), per row (physics), sequences at a time: threads / P
  int region;             // slots of a region: SB x L.slots
  int ncp;                // (k, M - k) couples of a sequence: ceil(M / 2)
  int half;               // even rows with even M: M / 2, the frequency that is its own mirror (else 0)
  KwDivU dP, dPT, dSB, dN1;  // division by P, PT, SB and N1
};

namespace kwmr {

// Pass l over the block's sequences.  WHERE: 0 the first pass (one block of
// butterflies a sequence), 2 the last (neighbouring points, no twiddles), 1 between.
template <int R, bool INV, int WHERE>
__device__ __forceinline__ void row_pass(float2* A, const KwMrLen& L, int l, int nseq, const float2* tw) {
  const int per = L.per[l], m = L.m[l], total = nseq * per;
  const int ms = WHERE == 2 ? 1 : L.ms[l];
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int s = kw_divu(i, L.dper[l]), rem = i - s * per;
    int slot, t = 0;
    if (WHERE == 2) {
      slot = rem * L.mp;
    } else if (WHERE == 0) {
      t = rem;
      slot = slot_of(L, 0, 0, t);
    } else {
      const int b = kw_divu(rem, L.dm[l]);
      t = rem - b * m;
      slot = slot_of(L, l, b, t);
    }
    float2* a = A + s * L.slots + slot;
    float2 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = a[j * ms];
    if (INV && WHERE != 2) twiddle<R>(v, tw + L.off[l] + t, m);
    dft<R>(v);
    if (!INV && WHERE != 2) twiddle<R>(v, tw + L.off[l] + t, m);
#pragma unroll
    for (int j = 0; j < R; ++j) a[j * ms] = v[j];
  }
}

template <bool INV, int WHERE>
__device__ __forceinline__ void row_pass_any(float2* A, const KwMrLen& L, int l, int r, int nseq, const float2* tw) {
  switch (r) {
#define KW_MR_CASE(R) \
  case R: row_pass<R, INV, WHERE>(A, L, l, nseq, tw); break;
    KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
    default: break;
  }
  __syncthreads();
}

// All passes over the block's nseq sequences; starts and ends with a barrier.
template <bool INV>
__device__ __forceinline__ void row_passes(float2* A, const KwMrLen& L, int nseq, const float2* tw) {
  __syncthreads();
  if (INV) row_pass_any<INV, 2>(A, L, L.np - 1, L.rl, nseq, tw);
  if (!INV) row_pass_any<INV, 0>(A, L, 0, L.r[0], nseq, tw);
#pragma unroll 1
  for (int i = 1; i < L.np - 1; ++i) {
    const int l = INV ? L.np - 1 - i : i;
    row_pass_any<INV, 1>(A, L, l, L.r[l], nseq, tw);
  }
  if (INV) row_pass_any<INV, 0>(A, L, 0, L.r[0], nseq, tw);
  if (!INV) row_pass_any<INV, 2>(A, L, L.np - 1, L.rl, nseq, tw);
}

__device__ __forceinline__ float2 mul(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ float2 mul(float a, float2 b) { return make_float2(__fmul_rn(a, b.x), __fmul_rn(a, b.y)); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)); }
__device__ __forceinline__ float2 dvd(float2 a, float2 b) { return make_float2(__fdiv_rn(a.x, b.x), __fdiv_rn(a.y, b.y)); }

template <bool ODD>
struct Rows {
  const MrRowsParams& W;
  const RowsParams& Q;
  float2* A;         // the regions
  int r0, nr, nseq;  // first row, rows and sequences of this block
  int s, t;          // physics: this thread's sequence and place in it
  int M;             // points of the sequence, 0 for a thread without one
  bool two;          // odd rows: the sequence has a second row
  uint32_t fb;       // first field element of the sequence: float2 (even) or float (odd) index

  __device__ __forceinline__ Rows(const MrRowsParams& w, int bx, float2* smem) : W(w), Q(w.Q), A(smem) {
    r0 = bx * W.rpb;
    nr = min(W.rpb, Q.nrows - r0);
    nseq = ODD ? (nr + 1) >> 1 : nr;
    s = kw_divu(threadIdx.x, W.dPT);
    t = threadIdx.x - s * W.PT;
    M = s < nseq ? W.L.n : 0;
    two = 2 * s + 1 < nr;
    fb = (uint32_t)(r0 + (ODD ? 2 * s : s)) * (uint32_t)(ODD ? Q.L : W.L.n);
  }

  // half spectra -> points of regions 0 .. nq - 1 (unnormalised: L x), parts
  // exchanged; spec(q) is region q's spectrum
  template <class SPEC>
  __device__ __forceinline__ void c2r(int nq, SPEC spec) const {
    const int N = W.L.n, P = W.P;
    const int g = kw_divu(threadIdx.x, W.dP), k1 = threadIdx.x - g * P;
#pragma unroll 1
    for (int qs = g < W.G ? g : nq * W.SB; qs < nq * W.SB; qs += W.G) {
      const int q = kw_divu(qs, W.dSB), sq = qs - q * W.SB;
      if (sq >= nseq) continue;
      const bool both = 2 * sq + 1 < nr;
      float2* a = A + qs * W.L.slots;
      const float2* sr = spec(q) + (uint32_t)(r0 + (ODD ? 2 * sq : sq)) * (uint32_t)Q.Hp;
#pragma unroll 1
      for (int k0 = k1; k0 < W.ncp; k0 += 4 * P) {
        float2 xa[4], xb[4], xh = make_float2(0.f, 0.f);
        uint32_t pk[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = k0 + i * P;
          const bool in = k < W.ncp;
          xa[i] = in ? sr[k] : make_float2(0.f, 0.f);
          if constexpr (ODD)
            xb[i] = in && both ? sr[Q.Hp + k] : make_float2(0.f, 0.f);
          else
            xb[i] = in ? sr[N - k] : make_float2(0.f, 0.f);
          pk[i] = in ? __ldg(W.pos + k) : 0u;
        }
        if (k0 == 0) {
          if (!ODD && W.half) xh = sr[W.half];
          xa[0].y = xb[0].y = 0.f;  // frequency 0 (and N) of a real row is real
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = k0 + i * P;
          if (k >= W.ncp) continue;
          float2 z, zm;
          if constexpr (!ODD) {
            const float2 e = make_float2(xa[i].x + xb[i].x, xa[i].y - xb[i].y);
            const float2 o = cmulf(make_float2(xa[i].x - xb[i].x, xa[i].y + xb[i].y), cconj(__ldg(Q.twpost + k)));
            z = make_float2(e.y + o.x, e.x - o.y);
            zm = make_float2(o.x - e.y, e.x + o.y);
          } else {
            z = make_float2(xa[i].y + xb[i].x, xa[i].x - xb[i].y);
            zm = make_float2(xb[i].x - xa[i].y, xa[i].x + xb[i].y);
          }
          // k = 0: its mirror slot is the slot of frequency `half` (or its own)
          if (i == 0 && k == 0) zm = !ODD && W.half ? make_float2(-2.f * xh.y, 2.f * xh.x) : z;
          a[pk[i] & 0xffffu] = z;
          a[pk[i] >> 16] = zm;
        }
      }
    }
    row_passes<true>(A, W.L, nq * W.SB, W.tw);
  }

  // points of regions 0 .. nq - 1 -> half spectra
  template <class SPEC>
  __device__ __forceinline__ void r2c(int nq, SPEC spec) const {
    row_passes<false>(A, W.L, nq * W.SB, W.tw);
    kwtma::grid_dep_launch();
    const int N = W.L.n, P = W.P;
    const int g = kw_divu(threadIdx.x, W.dP), k1 = threadIdx.x - g * P;
#pragma unroll 1
    for (int qs = g < W.G ? g : nq * W.SB; qs < nq * W.SB; qs += W.G) {
      const int q = kw_divu(qs, W.dSB), sq = qs - q * W.SB;
      if (sq >= nseq) continue;
      const bool both = 2 * sq + 1 < nr;
      const float2* a = A + qs * W.L.slots;
      float2* sr = spec(q) + (uint32_t)(r0 + (ODD ? 2 * sq : sq)) * (uint32_t)Q.Hp;
#pragma unroll 4
      for (int k = k1; k < W.ncp; k += P) {
        const uint32_t pk = __ldg(W.pos + k);
        const float2 zk = a[pk & 0xffffu];
        float2 zm = a[pk >> 16];
        if (k == 0) {
          if (!ODD && W.half) sr[W.half] = cconj(zm);
          zm = zk;
        }
        const float2 e = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        const float2 o = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
        if constexpr (!ODD) {
          const float2 tt = cmulf(__ldg(Q.twpost + k), o);
          sr[k] = make_float2(e.x + tt.x, e.y + tt.y);
          sr[N - k] = make_float2(e.x - tt.x, tt.y - e.y);
        } else {
          sr[k] = e;
          if (both) sr[Q.Hp + k] = o;
        }
      }
    }
    __syncthreads();
  }

  // ---- points ---------------------------------------------------------------
  // shared-memory slot of point n in region 0
  __device__ __forceinline__ int slot(int n) const {
    return s * W.L.slots + n + (W.L.mp != W.L.rl ? kw_divu(n, W.L.drl) : 0);
  }
  // field values of point n: reals 2n and 2n + 1 of a row, or real n of two rows
  __device__ __forceinline__ float2 ld(const float* __restrict__ f, int n) const {
    if constexpr (!ODD) {
      return reinterpret_cast<const float2*>(f)[fb + (uint32_t)n];
    } else {
      const float a = f[fb + (uint32_t)n];
      return make_float2(a, two ? f[fb + (uint32_t)Q.L + (uint32_t)n] : a);
    }
  }
  __device__ __forceinline__ float2 ld(const float* __restrict__ f, float sc, int n) const {
    return f ? ld(f, n) : make_float2(sc, sc);
  }
  __device__ __forceinline__ void st(float* __restrict__ f, int n, float2 v) const {
    if constexpr (!ODD) {
      reinterpret_cast<float2*>(f)[fb + (uint32_t)n] = v;
    } else {
      f[fb + (uint32_t)n] = v.x;
      if (two) f[fb + (uint32_t)Q.L + (uint32_t)n] = v.y;
    }
  }
  // PML factors of the sequence's rows along an axis other than the last
  __device__ __forceinline__ float2 pml_row(const float* __restrict__ tab, int axis) const {
    if (axis == Q.ndim - 1 || M == 0) return make_float2(1.f, 1.f);
    const int row = r0 + (ODD ? 2 * s : s);
    const float a = __ldg(tab + row_index(axis, row));
    return make_float2(a, ODD ? (two ? __ldg(tab + row_index(axis, row + 1)) : 1.f) : a);
  }
  __device__ __forceinline__ int row_index(int axis, int row) const {
    if (Q.ndim == 2) return row;
    const int x = kw_divu(row, W.dN1);
    return axis == 0 ? x : row - x * Q.N1;
  }
  // PML factors of point n along the last axis
  __device__ __forceinline__ float2 pml_last(const float* __restrict__ tab, int n) const {
    if constexpr (!ODD) return __ldg(reinterpret_cast<const float2*>(tab) + n);
    const float v = __ldg(tab + n);
    return make_float2(v, v);
  }
  // region q at a slot; an absent second row goes in as zero, whatever was computed for it
  __device__ __forceinline__ void put(int q, int sl, float2 v) const {
    if (ODD && !two) v.y = 0.f;
    A[q * W.region + sl] = v;
  }
  __device__ __forceinline__ float2 get(int q, int sl) const { return swp(A[q * W.region + sl]); }  // after c2r
  __device__ __forceinline__ float2 raw(int q, int sl) const { return A[q * W.region + sl]; }

  // the real of region q that a sparse entry (row, position) addresses
  __device__ __forceinline__ float& real_at(int q, int row, int position, bool swapped) const {
    const int d = row - r0;
    const int sq = ODD ? d >> 1 : d, n = ODD ? position : position >> 1;
    const int prt = (ODD ? d : position) & 1;
    float2& v = A[q * W.region + sq * W.L.slots + n + kw_divu(n, W.L.drl) * (W.L.mp - W.L.rl)];
    return (prt != 0) != swapped ? v.y : v.x;
  }
  // sparse source on region q (kspace_solver.py:86-109), between the caller's barriers
  __device__ __forceinline__ void source(int q, const KwSrcDev& S, int ts) const {
    const int e0 = S.row_ptr[r0], e1 = S.row_ptr[r0 + nr];
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
      const int4 en = S.ent[e];
      const float val = S.sig[(long long)ts * S.nsig + (S.nsig == 1 ? 0 : en.z)];
      float& f = real_at(q, en.x, en.y, false);
      f = S.mode == SRC_DIRICHLET ? val : __fadd_rn(f, val);
    }
  }
  __device__ __forceinline__ bool source_on(const KwSrcDev& S, int ts) const { return S.active && ts < S.len; }
  // k-space corrected sources: on in this launch and not over at step ts (a
  // grouped launch serves members whose sources end at different steps)
  __device__ __forceinline__ bool srcp_on(int ts) const { return Q.srcp_on && ts < Q.src[0].len; }
  __device__ __forceinline__ bool srcu_on(int a, int ts) const { return Q.srcu_on[a] && ts < Q.src[3 + a].len; }
  // the source's values on a zeroed region
  __device__ __forceinline__ void scatter(const KwSrcDev& S, int ts) const {
    for (int i = threadIdx.x; i < W.region; i += blockDim.x) A[i] = make_float2(0.f, 0.f);
    __syncthreads();
    const int e0 = S.row_ptr[r0], e1 = S.row_ptr[r0 + nr];
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
      const int4 en = S.ent[e];
      real_at(0, en.x, en.y, false) = S.sig[(long long)ts * S.nsig + (S.nsig == 1 ? 0 : en.z)];
    }
  }
  __device__ __forceinline__ bool recording(const float* rec) const {
    return rec != nullptr && kw_rec_row(Q) >= 0 && Q.sens_row_ptr != nullptr;
  }
  // sensor samples from region q, which the caller has completed with a barrier
  __device__ __forceinline__ void record(int q, float* rec, bool swapped) const {
    const int e0 = Q.sens_row_ptr[r0], e1 = Q.sens_row_ptr[r0 + nr];
    float* out = rec + (long long)kw_rec_row(Q) * Q.nslots;
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
      const int4 en = Q.sens_ent[e];
      out[en.z] = real_at(q, en.x, en.y, swapped);
    }
  }
  // lp += S^T r at the block's sensor points of region 0; barriers on both sides
  __device__ __forceinline__ void add_residual() const {
    __syncthreads();
    if (recording(Q.rec[0])) {
      const int e0 = Q.sens_row_ptr[r0], e1 = Q.sens_row_ptr[r0 + nr];
      const float* res = Q.rec[0] + (long long)kw_rec_row(Q) * Q.nslots;
      for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
        const int4 en = Q.sens_ent[e];
        float& f = real_at(0, en.x, en.y, false);
        f = __fadd_rn(f, res[en.z]);
      }
    }
    __syncthreads();
  }

  // ask for the block's rows of an array in L2 (the first line is rounded
  // down to its 128-byte boundary, which stays inside the allocation)
  __device__ __forceinline__ void prefetch(const void* base, uint32_t row_bytes) const {
    if (base == nullptr) return;
    const uintptr_t a = (uintptr_t)base + (uintptr_t)r0 * row_bytes;
    const uintptr_t e = a + (uintptr_t)nr * row_bytes;
    for (uintptr_t l = (a & ~(uintptr_t)127) + (uintptr_t)threadIdx.x * 128; l < e; l += (uintptr_t)blockDim.x * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(l));
  }
  __device__ __forceinline__ void prefetch_spec(const float2* S) const { prefetch(S, (uint32_t)Q.Hp * 8u); }
  __device__ __forceinline__ void prefetch_field(const float* f) const { prefetch(f, (uint32_t)Q.L * 4u); }
};

}  // namespace kwmr

// Blocks on an SM each stage is compiled for.
constexpr int kw_mr_blocks(int stage) { return stage == ST_RHO ? 3 : 4; }

// A thread's points, C at a time: LOAD fills registers (index i), then BODY
// computes and stores; n is the point's place in the sequence, sl its slot.
#define KW_MR_POINTS(C, LOAD, BODY)                                        \
  _Pragma("unroll 1") for (int n0 = c.t; n0 < c.M; n0 += (C) * W.PT) {     \
    _Pragma("unroll") for (int i = 0; i < (C); ++i) {                      \
      const int n = n0 + i * W.PT;                                         \
      if (n < c.M) {                                                       \
        LOAD                                                               \
      }                                                                    \
    }                                                                      \
    _Pragma("unroll") for (int i = 0; i < (C); ++i) {                      \
      const int n = n0 + i * W.PT;                                         \
      if (n < c.M) {                                                       \
        const int sl = c.slot(n);                                          \
        (void)sl;                                                          \
        BODY                                                               \
      }                                                                    \
    }                                                                      \
  }

// One block of a stage.  DIM: dimensions, 0 for stages that read them at run time.
template <int STAGE, bool ODD, int DIM>
__device__ __forceinline__ void mr_rows_body(const MrRowsParams& W, int bx) {
  using namespace kwmr;
  extern __shared__ float4 smem_f4[];
  const RowsParams& Q = W.Q;
  const Rows<ODD> c(W, bx, reinterpret_cast<float2*>(smem_f4));
  const int D = DIM ? DIM : Q.ndim;
  constexpr int MD = DIM ? DIM : 3;
  kwtma::grid_dep_wait();
  const int t = kw_step_t(Q);

  if constexpr (STAGE == ST_INIT) {
    // t = 0 with p0: p = p0, rho_i = p0 / (c0^2 D) (kspace_solver.py:729-733)
    const float sc = Q.p0_scale ? *Q.p0_scale : 1.f;
    float2 p0[4], cc[4];
    KW_MR_POINTS(4, {
      p0[i] = c.ld(Q.p0, n);
      cc[i] = c.ld(Q.c0, Q.c0_s, n);
    }, {
      float2 pv = p0[i];
      if (Q.p0_scale) pv = mul(sc, pv);
      const float2 r = dvd(pv, mul((float)D, mul(cc[i], cc[i])));
      float2 rs = r;
      for (int a = 0; a < D; ++a) {
        c.st(Q.rho[a], n, r);
        if (a > 0) rs = add(rs, r);
      }
      if (Q.rho_sum) c.st(Q.rho_sum, n, rs);
      if (Q.write_p) c.st(Q.p, n, pv);
      c.put(0, sl, pv);
    })
    if (c.recording(Q.rec[0])) {
      __syncthreads();
      c.record(0, Q.rec[0], false);
    }
    c.r2c(1, [&](int) { return Q.S[3]; });
  } else if constexpr (STAGE == ST_U) {
    // u_i = pml_sg (pml_sg u_i - dt/rho_sg_i g_i) (kspace_solver.py:703-707).
    // Regions: the components, then the k-space corrected sources (kspace_solver.py:91-98)
    for (int a = 0; a < D; ++a) {
      c.prefetch_spec(Q.S[a]);
      if (!Q.init) c.prefetch_field(Q.u[a]);
      c.prefetch_field(Q.dtrsg[a]);
    }
    bool ks = false, src = false, rec = false;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      if (!Q.init && c.srcu_on(a, t))
        ks = true;
      else if (!Q.init && c.source_on(Q.src[3 + a], t))
        src = true;
      rec |= c.recording(Q.rec[1 + a]);
    }
    c.c2r(ks ? 2 * D : D, [&](int q) {
      const float2* s = Q.S[q < D ? q : B_SRCU0 + q - D];
      return s ? s : Q.S[0];  // a component without a source: transformed, not used
    });
    float2 row[MD];
#pragma unroll
    for (int a = 0; a < D; ++a) row[a] = c.pml_row(Q.pmlsg[a], a);
    constexpr int C = DIM == 3 ? 3 : 4;
    float2 dtr[C][MD], u[C][MD];
    KW_MR_POINTS(C, {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        dtr[i][a] = c.ld(Q.dtrsg[a], Q.dtrsg_s[a], n);
        if (!Q.init) u[i][a] = c.ld(Q.u[a], n);
      }
    }, {
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const float2 g = c.get(a, sl);
        float2 v;
        if (Q.init) {
          v = mul(mul(0.5f, dtr[i][a]), g);
        } else {
          const float2 sg = a == D - 1 ? c.pml_last(Q.pmlsg[a], n) : row[a];
          v = mul(sg, sub(mul(sg, u[i][a]), mul(dtr[i][a], g)));
          if (ks && c.srcu_on(a, t)) v = add(v, c.get(D + a, sl));
        }
        c.put(a, sl, v);
        if (!src) c.st(Q.u[a], n, v);
      }
    })
    if (src) {
      __syncthreads();
      for (int a = 0; a < D; ++a)
        if (!c.srcu_on(a, t) && c.source_on(Q.src[3 + a], t)) c.source(a, Q.src[3 + a], t);
      __syncthreads();
      KW_MR_POINTS(1, {}, {
        for (int a = 0; a < D; ++a) c.st(Q.u[a], n, c.raw(a, sl));
      })
    }
    if (rec) {
      if (!src) __syncthreads();
      for (int a = 0; a < D; ++a)
        if (c.recording(Q.rec[1 + a])) c.record(a, Q.rec[1 + a], false);
    }
    if (!Q.init || Q.init_r2c) c.r2c(D, [&](int q) { return Q.S[q]; });
  } else if constexpr (STAGE == ST_RHO) {
    // mass conservation with split density (kspace_solver.py:709-717).
    // Regions: the components, then the k-space corrected source
    // (kspace_solver.py:91-98, scale :619-624) or, with a sparse source, the divergence
    const bool powerlaw = Q.absorb == 1;
    for (int a = 0; a < D; ++a) {
      c.prefetch_spec(Q.S[a]);
      c.prefetch_field(Q.rho[a]);
    }
    c.prefetch_field(Q.rho0);
    if (powerlaw && Q.nonlin) c.prefetch_field(Q.rho_sum);
    const int ks = c.srcp_on(t) ? 1 : 0;
    bool src = false;
    if (!ks)
      for (int a = 0; a < D; ++a) src |= c.source_on(Q.src[a], t);
    // second round: the recorded velocities on the pressure grid (kspace_solver.py:740-743)
#pragma unroll 1
    for (int round = 0; round < (Q.rec_us ? 2 : 1); ++round) {
      c.c2r(round ? D : D + ks, [&](int q) {
        const float2* s = Q.S[round ? B_US0 + q : q < D ? q : (int)B_SRCP];
        return s ? s : Q.S[0];
      });
      if (round) {
        for (int a = 0; a < D; ++a)
          if ((Q.rec_us & (1 << a)) && c.recording(Q.rec[4 + a])) c.record(a, Q.rec[4 + a], true);
        break;
      }
      float2 row[MD];
#pragma unroll
      for (int a = 0; a < D; ++a) row[a] = c.pml_row(Q.pml[a], a);
      // the result of a point: density sum rs, divergence dv
      auto finish = [&](int n, int sl, float2 rs, float2 dv, float2 r0v) {
        if (powerlaw) {
          c.st(Q.rho_sum, n, rs);
          c.put(0, sl, mul(r0v, dv));
          if (Q.disp) c.put(1, sl, rs);
        } else {
          // equation of state without fractional Laplacians (kspace_solver.py:719-723)
          const float2 cc = c.ld(Q.c0, Q.c0_s, n);
          float2 acc = rs;
          if (Q.absorb == 2) acc = add(acc, mul(mul(c.ld(Q.tau, Q.tau_s, n), r0v), dv));
          if (Q.nonlin) acc = add(acc, dvd(mul(c.ld(Q.bona, Q.bona_s, n), mul(rs, rs)), mul(2.f, r0v)));
          const float2 pv = mul(mul(cc, cc), acc);
          if (Q.write_p) c.st(Q.p, n, pv);
          c.put(0, sl, pv);
        }
      };
      constexpr int C = DIM == 3 ? 3 : 4;
      float2 ro[C][MD], r0v[C], sr[C];
      KW_MR_POINTS(C, {
        r0v[i] = c.ld(Q.rho0, Q.rho0_s, n);
#pragma unroll
        for (int a = 0; a < D; ++a) ro[i][a] = c.ld(Q.rho[a], n);
        if (powerlaw && Q.nonlin) sr[i] = c.ld(Q.rho_sum, n);  // written by the previous step
      }, {
        float2 w = mul(Q.dt, r0v[i]);
        if (Q.nonlin) {
          if (!powerlaw) {
            sr[i] = ro[i][0];
#pragma unroll
            for (int a = 1; a < D; ++a) sr[i] = add(sr[i], ro[i][a]);
          }
          w = mul(w, dvd(add(mul(2.f, sr[i]), r0v[i]), r0v[i]));
        }
        float2 dv = make_float2(0.f, 0.f);
        float2 rs = make_float2(0.f, 0.f);
        const float2 kv = ks ? c.get(D, sl) : make_float2(0.f, 0.f);
#pragma unroll
        for (int a = 0; a < D; ++a) {
          const float2 du = c.get(a, sl);
          dv = a == 0 ? du : add(dv, du);
          const float2 pm = a == D - 1 ? c.pml_last(Q.pml[a], n) : row[a];
          float2 v = mul(pm, sub(mul(pm, ro[i][a]), mul(w, du)));
          if (ks) v = add(v, mul(Q.inv_d[a], kv));
          if (src)
            c.put(a, sl, v);
          else
            c.st(Q.rho[a], n, v);
          rs = a == 0 ? v : add(rs, v);
        }
        if (src)
          c.put(D, sl, dv);
        else
          finish(n, sl, rs, dv, r0v[i]);
      })
      if (src) {
        __syncthreads();
        for (int a = 0; a < D; ++a)
          if (c.source_on(Q.src[a], t)) c.source(a, Q.src[a], t);
        __syncthreads();
        KW_MR_POINTS(1, {}, {
          float2 rs = make_float2(0.f, 0.f);
          for (int a = 0; a < D; ++a) {
            const float2 v = c.raw(a, sl);
            c.st(Q.rho[a], n, v);
            rs = a == 0 ? v : add(rs, v);
          }
          finish(n, sl, rs, c.raw(D, sl), c.ld(Q.rho0, Q.rho0_s, n));
        })
      }
      if (!powerlaw && c.recording(Q.rec[0])) {
        __syncthreads();
        c.record(0, Q.rec[0], false);
      }
      c.r2c(powerlaw && Q.disp ? 2 : 1, [&](int q) { return Q.S[powerlaw ? q : 3]; });
    }
  } else if constexpr (STAGE == ST_EOS) {
    // p = c0^2 (rho + tau F^-1[nabla1 F[rho0 div]] - eta F^-1[nabla2 F[rho]] + B/A rho^2 / (2 rho0))
    c.prefetch_spec(Q.S[0]);
    if (Q.disp) c.prefetch_spec(Q.S[1]);
    c.prefetch_field(Q.rho_sum);
    c.prefetch_field(Q.tau);
    if (Q.disp) c.prefetch_field(Q.eta);
    c.prefetch_field(Q.c0);
    if (Q.nonlin) {
      c.prefetch_field(Q.rho0);
      c.prefetch_field(Q.bona);
    }
    c.c2r(Q.disp ? 2 : 1, [&](int q) { return Q.S[q]; });
    float2 rs[4], ta[4], et[4], cc[4], bo[4], r0v[4];
    KW_MR_POINTS(4, {
      rs[i] = c.ld(Q.rho_sum, n);
      ta[i] = c.ld(Q.tau, Q.tau_s, n);
      if (Q.disp) et[i] = c.ld(Q.eta, Q.eta_s, n);
      cc[i] = c.ld(Q.c0, Q.c0_s, n);
      if (Q.nonlin) {
        bo[i] = c.ld(Q.bona, Q.bona_s, n);
        r0v[i] = c.ld(Q.rho0, Q.rho0_s, n);
      }
    }, {
      float2 v = add(rs[i], mul(ta[i], c.get(0, sl)));
      if (Q.disp) v = sub(v, mul(et[i], c.get(1, sl)));
      if (Q.nonlin) v = add(v, dvd(mul(bo[i], mul(rs[i], rs[i])), mul(2.f, r0v[i])));
      v = mul(mul(cc[i], cc[i]), v);
      if (Q.write_p) c.st(Q.p, n, v);
      c.put(0, sl, v);
    })
    if (c.recording(Q.rec[0])) {
      __syncthreads();
      c.record(0, Q.rec[0], false);
    }
    c.r2c(1, [&](int) { return Q.S[3]; });
  } else if constexpr (STAGE == ST_SRC) {
    // scattered source fields of this step, transformed for the source-kappa pass
#pragma unroll 1
    for (int q = 0; q < 1 + D; ++q) {
      if (!(q == 0 ? c.srcp_on(t) : c.srcu_on(q - 1, t))) continue;
      c.scatter(Q.src[q == 0 ? 0 : 2 + q], t);
      c.r2c(1, [&](int) { return Q.S[q == 0 ? (int)B_SRCP : B_SRCU0 + q - 1]; });
    }
  } else if constexpr (STAGE == ST_UREC) {
#pragma unroll 1
    for (int a = 0; a < D; ++a) {
      if (!(Q.rec_us & (1 << a))) continue;
      c.c2r(1, [&](int) { return Q.S[B_US0 + a]; });
      if (c.recording(Q.rec[4 + a])) c.record(0, Q.rec[4 + a], true);
      __syncthreads();
    }
  } else if constexpr (STAGE == ST_P0FFT) {
    // spectrum of p0 for the smoothing window
    KW_MR_POINTS(1, {}, { c.put(0, sl, c.ld(Q.p0w, n)); })
    c.r2c(1, [&](int) { return Q.S[B_P]; });
  } else if constexpr (STAGE == ST_P0BACK) {
    c.c2r(1, [&](int) { return Q.S[B_P]; });
    KW_MR_POINTS(1, {}, { c.st(Q.p0w, n, c.get(0, sl)); })
  } else if constexpr (STAGE == ST_ADJ_A || STAGE == ST_ADJ_D) {
    // the transposed step (see adjoint_body in kw_generic.cuh); region 0 holds lp first
    {
      float2 v[4];
      KW_MR_POINTS(4, { v[i] = c.ld(Q.p, n); }, { c.put(0, sl, v[i]); })
    }
    c.add_residual();
    float2 row[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) row[a] = STAGE == ST_ADJ_A && a < D ? c.pml_row(Q.pml[a], a) : make_float2(1.f, 1.f);
    const bool acc = STAGE == ST_ADJ_A && Q.gacc;
    float2 f[2], g[2], cc[2], b[2], lr[2][3];
    KW_MR_POINTS(2, {
      if (acc) {
        f[i] = c.ld(Q.fsum, n);
        g[i] = c.ld(Q.gacc, n);
      }
      if (STAGE == ST_ADJ_A) {
        cc[i] = c.ld(Q.c0, Q.c0_s, n);
        b[i] = c.ld(Q.rho0, Q.rho0_s, n);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (a < D) lr[i][a] = c.ld(STAGE == ST_ADJ_A ? Q.rho[a] : Q.u[a], n);
    }, {
      const float2 v = c.raw(0, sl);
      if (STAGE == ST_ADJ_D) c.st(Q.p, n, v);
      if (acc) c.st(Q.gacc, n, make_float2(__fmaf_rn(f[i].x, v.x, g[i].x), __fmaf_rn(f[i].y, v.y, g[i].y)));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (a >= D) continue;
        if (STAGE == ST_ADJ_A) {
          const float2 pm = a == D - 1 ? c.pml_last(Q.pml[a], n) : row[a];
          const float2 l = add(lr[i][a], mul(mul(cc[i], cc[i]), v));
          c.st(Q.rho[a], n, mul(mul(pm, pm), l));
          c.put(a, sl, mul(mul(mul(Q.dt, b[i]), pm), l));
        } else {
          c.put(a, sl, mul(mul(0.5f, c.ld(Q.dtrsg[a], Q.dtrsg_s[a], n)), lr[i][a]));
        }
      }
    })
    c.r2c(D, [&](int q) { return Q.S[q]; });
  } else if constexpr (STAGE == ST_ADJ_B) {
    for (int a = 0; a < D; ++a) {
      c.prefetch_spec(Q.S[a]);
      c.prefetch_field(Q.u[a]);
    }
    c.c2r(D, [&](int q) { return Q.S[q]; });
    float2 row[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) row[a] = a < D ? c.pml_row(Q.pmlsg[a], a) : make_float2(1.f, 1.f);
    float2 dtr[2][3], u[2][3];
    KW_MR_POINTS(2, {
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (a < D) {
          dtr[i][a] = c.ld(Q.dtrsg[a], Q.dtrsg_s[a], n);
          u[i][a] = c.ld(Q.u[a], n);
        }
    }, {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (a >= D) continue;
        const float2 sg = a == D - 1 ? c.pml_last(Q.pmlsg[a], n) : row[a];
        const float2 lu = add(u[i][a], c.get(a, sl));
        c.st(Q.u[a], n, mul(mul(sg, sg), lu));
        c.put(a, sl, mul(mul(dtr[i][a], sg), lu));
      }
    })
    c.r2c(D, [&](int q) { return Q.S[q]; });
  } else {
    // ST_ADJ_C / ST_ADJ_E
    c.c2r(D, [&](int q) { return Q.S[q]; });
    KW_MR_POINTS(2, {}, {
      float2 v = c.get(0, sl);
      for (int a = 1; a < D; ++a) v = add(v, c.get(a, sl));
      if (STAGE == ST_ADJ_C) {
        c.st(Q.p, n, v);
      } else {
        const float2 cc = c.ld(Q.c0, Q.c0_s, n);
        const float2 den = mul((float)D, mul(cc, cc));
        float2 acc = c.ld(Q.p, n);
        float2 lr = make_float2(0.f, 0.f);
        for (int a = 0; a < D; ++a) {
          const float2 r = c.ld(Q.rho[a], n);
          acc = add(acc, dvd(r, den));
          lr = a == 0 ? r : add(lr, r);
        }
        c.st(Q.p, n, sub(acc, v));
        if (Q.gacc) {
          const float2 ov = dvd(mul(c.ld(Q.p0, n), lr), mul(den, mul(cc, cc)));
          c.st(Q.gacc, n, mul(mul(2.f, cc), sub(c.ld(Q.gacc, n), ov)));
        }
      }
    })
  }
}

template <int STAGE, bool ODD, int DIM>
__global__ void __launch_bounds__(KW_MR_THREADS, kw_mr_blocks(STAGE)) k_mr_rows(const __grid_constant__ MrRowsParams W) {
  mr_rows_body<STAGE, ODD, DIM>(W, blockIdx.x);
}

// One stage of several plans: block i works on member map[i].x, its block map[i].y.
template <int STAGE, int DIM>
__global__ void __launch_bounds__(KW_MR_THREADS, kw_mr_blocks(STAGE))
    k_mr_rows_group(const MrRowsParams* __restrict__ Ps, const int2* __restrict__ map) {
  __shared__ __align__(16) MrRowsParams sp;
  const int2 me = map[blockIdx.x];
  const int* src = reinterpret_cast<const int*>(Ps + me.x);
  for (int w = threadIdx.x; w < (int)(sizeof(MrRowsParams) / 4); w += blockDim.x) reinterpret_cast<int*>(&sp)[w] = src[w];
  __syncthreads();
  if (sp.Q.even)
    mr_rows_body<STAGE, false, DIM>(sp, me.y);
  else
    mr_rows_body<STAGE, true, DIM>(sp, me.y);
}

// One plan's stage, or (Ps set) the grouped stage over `blocks` blocks.
template <int STAGE, int DIM>
static cudaError_t kw_mr_rows_go(int odd, int blocks, int threads, size_t smem, cudaStream_t st, const MrRowsParams* W,
                                 const MrRowsParams* Ps, const int2* map, bool pdl) {
  // one constant, so that plans of several threads never lower it under one another
  if (smem > 40 * 1024) {
    if (smem > KW_MR_ROWS_SMEM) return cudaErrorInvalidValue;
    cudaError_t e =
        cudaFuncSetAttribute(k_mr_rows<STAGE, true, DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, KW_MR_ROWS_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_mr_rows<STAGE, false, DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, KW_MR_ROWS_SMEM);
    if (e != cudaSuccess) return e;
  }
  if (Ps) {
    // the stages of a step that batches repeat
    if constexpr (STAGE == ST_U || STAGE == ST_RHO || STAGE == ST_EOS || STAGE == ST_SRC) {
      if (smem > 40 * 1024) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_mr_rows_group<STAGE, DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, KW_MR_ROWS_SMEM);
        if (e != cudaSuccess) return e;
      }
      return kwtma::launch_k(k_mr_rows_group<STAGE, DIM>, dim3(blocks), dim3(threads), smem, st, pdl, Ps, map);
    } else {
      return cudaErrorInvalidValue;
    }
  }
  if (odd) return kwtma::launch_k(k_mr_rows<STAGE, true, DIM>, dim3(blocks), dim3(threads), smem, st, W->pdl != 0, *W);
  return kwtma::launch_k(k_mr_rows<STAGE, false, DIM>, dim3(blocks), dim3(threads), smem, st, W->pdl != 0, *W);
}
