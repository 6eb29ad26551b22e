// Mixed-radix register-pass transforms for any composite 2,3,5,7-smooth
// length n = r_0 r_1 ... (two to six factors of at most 16).
//
// A transform is np passes.  In pass l every thread takes whole butterflies:
// r_l points spaced m_l = n / (r_0 .. r_l) apart go to registers, one unrolled
// r_l-point DFT with constant twiddles, one table twiddle per point, and back
// to the same slots (decimation in frequency, in place).  Slot
// k_0 m_0 + k_1 m_1 + ... then holds frequency k_0 + r_0 k_1 + r_0 r_1 k_2 ...;
// the inverse runs the passes backwards (twiddle before the DFT), from that
// order to natural order.  The inverse works on values with real and imaginary
// part exchanged, which turns its DFTs into the forward ones.
//
// Against the radix-2..7 Stockham stages of kw_fft.cuh (one shared-memory
// round trip and one set of index divisions per radix) this takes two or three
// round trips, and one or two divisions per 8..16 points: 55 instead of 273
// executed instructions per point and transform at n = 180, where the Stockham
// pass was bound by instruction issue (80 % busy, DRAM at a quarter of its
// rate): y passes of 216 x 180 x 150 over three spectra 80 -> 34 us (142 MB),
// the x gradient pass 142 -> 54 us, whole tissue steps 1450 -> 710 us.
//
// Slots of the last pass's r = r_{np-1} consecutive points are padded to an odd
// count (mp = r | 1): consecutive threads then read distinct shared-memory banks.
#pragma once
#include "kw_fft.cuh"

#define KW_MR_MAXP 6
#define KW_MR_SIZES(X) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(15) X(16)

struct KwMrLen {
  int n, np;            // np = 0: no factorisation (length not supported)
  int rl, mp, q;        // last radix, its padded block, n / rl
  int slots;            // padded slots of one sequence: q mp
  int r[KW_MR_MAXP];    // radix of pass l
  int m[KW_MR_MAXP];    // point spacing of pass l
  int ms[KW_MR_MAXP];   // the same in padded slots
  int per[KW_MR_MAXP];  // butterflies of pass l: n / r_l
  int off[KW_MR_MAXP];  // pass l's twiddles w_{r_l m_l}^{t k} start here, at [k m_l + t]
  KwDivU dper[KW_MR_MAXP], dm[KW_MR_MAXP], dr[KW_MR_MAXP], drl;
};

inline bool kw_mr_size_ok(int r) {
  switch (r) {
#define KW_MR_CASE(R) case R:
    KW_MR_SIZES(KW_MR_CASE)
#undef KW_MR_CASE
    return true;
    default:
      return false;
  }
}

// Non-increasing factor lists of n with sizes at most `most`: the best by
// passes then sum, or (brief) by the cost of kw_mr_factor.
inline void kw_mr_search(int n, int most, int* f, int np, bool brief, int* best, int& bnp, int& bcost) {
  if (n == 1) {
    if (np < 2) return;
    int cost = brief ? 8 * np : 0;
    for (int i = 0; i < np; ++i) cost += brief ? (f[i] > 10 ? 3 : 2) * f[i] : f[i];
    if (bnp && (brief ? cost >= bcost : np > bnp || (np == bnp && cost >= bcost))) return;
    bnp = np;
    bcost = cost;
    for (int i = 0; i < np; ++i) best[i] = f[i];
    return;
  }
  if (np == KW_MR_MAXP) return;
  for (int r = most; r >= 2; --r) {
    if (!kw_mr_size_ok(r) || n % r) continue;
    f[np] = r;
    kw_mr_search(n / r, r, f, np + 1, brief, best, bnp, bcost);
  }
}

// Factor n into radices, largest first.  Grids with work for every SM take the
// fewest passes (fewest shared-memory round trips), balanced: 180 = 15 12.
// Small grids (brief) take smaller radices: there a pass is a few butterflies
// per SM and lasts as long as one thread takes through its straight-line code,
// most of it instruction fetch.  Cost of a pass: its radix (half as much again
// above 10) and 4.  Measured, us of the gradient pass: 128 as 16 8 12.4, 8 4 4
// 9.1, 4 4 4 2 8.4; 300 as 10 6 5 11.0, 5 5 4 3 11.9; 375 as 15 5 5 14.0,
// 5 5 5 3 12.2; whole steps of 1024^2: 16 8 8 125, 8 8 4 4 120, 4 4 4 4 4 148.
// False when n is not a product of two to six sizes (n < 4, a prime, not smooth).
inline bool kw_mr_factor(int n, KwMrLen& L, bool brief) {
  L = KwMrLen{};
  L.n = n;
  int best[KW_MR_MAXP] = {0}, f[KW_MR_MAXP], bnp = 0, bcost = 0;
  kw_mr_search(n, 16, f, 0, brief, best, bnp, bcost);
  if (!bnp) return false;
  L.np = bnp;
  L.rl = best[bnp - 1];
  L.mp = L.rl | 1;
  L.q = n / L.rl;
  L.slots = L.q * L.mp;
  L.drl = kw_divu_make((uint32_t)L.rl);
  int m = n, off = 0;
  for (int l = 0; l < KW_MR_MAXP; ++l) {
    const int r = l < bnp ? best[l] : 1;
    m /= r;
    L.r[l] = r;
    L.m[l] = m;
    L.ms[l] = l < bnp - 1 ? m / L.rl * L.mp : 1;
    L.per[l] = n / r;
    L.off[l] = off;
    if (l < bnp - 1) off += r * m;
    L.dper[l] = kw_divu_make((uint32_t)L.per[l]);
    L.dm[l] = kw_divu_make((uint32_t)m);
    L.dr[l] = kw_divu_make((uint32_t)r);
  }
  return true;
}

// Gain of a forward and inverse transform pair at each frequency, minus 1.
// The constant twiddles of a register DFT are few, so their rounding to float
// does not average out: it scales every pair by up to 1 +- 8e-8 (162 = 9 6 3),
// the same at each time step, and the phase of a wave drifts by that share of
// the distance travelled.  The spectral operators divide by it (the low part
// of their 1 / N).  To first order the passes add: a DFT F with rounded
// constants gains mean_j Re F[k][j] conj(F[j][k]) at its output k, a twiddle
// table the mean of |w|^2 over the butterflies of its output k.
inline void kw_mr_dft_host(int N, const double* xr, const double* xi, int st, double* yr, double* yi) {
  auto cs = [&](int k, int n) { return (double)(float)kw_ct_trig(k, n, false); };
  auto sn = [&](int k, int n) { return (double)(float)kw_ct_trig(k, n, true); };
  if (N == 1) {
    yr[0] = xr[0];
    yi[0] = xi[0];
    return;
  }
  if (N == 2 || N == 3 || N == 4 || N == 5 || N == 7) {  // exact but for the cosines and sines of 2 pi j / N
    for (int k = 0; k < N; ++k) {
      yr[k] = yi[k] = 0.0;
      for (int n = 0; n < N; ++n) {
        const int j = (k * n) % N;
        const double c = cs(j, N), s = sn(j, N), a = xr[n * st], b = xi[n * st];
        yr[k] += a * c + b * s;
        yi[k] += b * c - a * s;
      }
    }
    return;
  }
  const int R = (N % 4 == 0) ? 4 : (N % 2 == 0) ? 2 : (N % 3 == 0) ? 3 : 5, M = N / R;
  double sr[16], si[16], tr[5], ti[5], ur[5], ui[5];
  for (int j = 0; j < R; ++j) {
    kw_mr_dft_host(M, xr + j * st, xi + j * st, R * st, sr + j * M, si + j * M);
    for (int k = 0; k < M; ++k) {
      const double c = cs(j * k, N), s = sn(j * k, N), a = sr[j * M + k], b = si[j * M + k];
      sr[j * M + k] = a * c + b * s;
      si[j * M + k] = b * c - a * s;
    }
  }
  for (int k = 0; k < M; ++k) {
    for (int j = 0; j < R; ++j) {
      tr[j] = sr[j * M + k];
      ti[j] = si[j * M + k];
    }
    kw_mr_dft_host(R, tr, ti, 1, ur, ui);
    for (int q = 0; q < R; ++q) {
      yr[k + M * q] = ur[q];
      yi[k + M * q] = ui[q];
    }
  }
}

// Frequency of the j = 0 point of butterfly b of the last pass; point j holds
// frequency kw_mr_freq(L, b) + j L.q.
// (Block digits b = (.. (k_0 r_1 + k_1) r_2 ..) + k_{np-2}.)
__host__ __device__ __forceinline__ int kw_mr_freq(const KwMrLen& L, int b) {
  if (L.np == 2) return b;
  int f = 0;
  for (int l = L.np - 2; l >= 1; --l) {
#ifdef __CUDA_ARCH__
    const int up = kw_divu(b, L.dr[l]);
#else
    const int up = b / L.r[l];
#endif
    f = (f + b - up * L.r[l]) * L.r[l - 1];
    b = up;
  }
  return f + b;
}

// Gains of the r-point register DFT at its outputs (worked out once per size).
inline const double* kw_mr_dft_gain(int r) {
  struct Table {
    double g[17][16];
    Table() {
      for (int n = 2; n <= 16; ++n) {
        if (!kw_mr_size_ok(n)) continue;
        double Fr[16][16], Fi[16][16];  // F[k][j]
        for (int j = 0; j < n; ++j) {
          double xr[16] = {0.0}, xi[16] = {0.0}, yr[16], yi[16];
          xr[j] = 1.0;
          kw_mr_dft_host(n, xr, xi, 1, yr, yi);
          for (int k = 0; k < n; ++k) {
            Fr[k][j] = yr[k];
            Fi[k][j] = yi[k];
          }
        }
        for (int k = 0; k < n; ++k) {
          double sum = 0.0;
          for (int j = 0; j < n; ++j) sum += Fr[k][j] * Fr[j][k] + Fi[k][j] * Fi[j][k];
          g[n][k] = sum / n - 1.0;
        }
      }
    }
  };
  static const Table table;
  return table.g[r];
}

// eps[k] of the n frequencies (see above); w: the pass twiddles in float.
inline void kw_mr_gain(const KwMrLen& L, const float2* w, double* eps) {
  double part[KW_MR_MAXP][16];
  for (int l = 0; l < L.np; ++l) {
    const double* g = kw_mr_dft_gain(L.r[l]);
    for (int k = 0; k < L.r[l]; ++k) {
      double w2 = 0.0;
      if (l < L.np - 1)
        for (int t = 0; t < L.m[l]; ++t) {
          const double c = w[L.off[l] + k * L.m[l] + t].x, s = w[L.off[l] + k * L.m[l] + t].y;
          w2 += (c * c + s * s - 1.0) / L.m[l];
        }
      part[l][k] = g[k] + w2;
    }
  }
  for (int b = 0; b < L.q; ++b)
    for (int j = 0; j < L.rl; ++j) {
      int rest = b;
      double e = part[L.np - 1][j];
      for (int l = L.np - 2; l >= 0; --l) {
        e += part[l][rest % L.r[l]];
        rest /= L.r[l];
      }
      eps[kw_mr_freq(L, b) + j * L.q] = e;
    }
}

// Gains of the two-level power-of-two passes (kw_regfft.cuh, n = E P), which share
// grids with mixed-radix ones: E-point DFTs, the table twiddle w_n^{t k1}, P-point
// DFTs; w: that table.  Entry (k, j) of their N-point DFT: N = N1 N2 with constant
// twiddles rounded to float.
inline void kw_reg_dft_entry(int N, int k, int j, double* re, double* im) {
  if (N <= 4) {  // exact
    const int q = (k * j) % N * (4 / N);
    *re = q == 0 ? 1.0 : q == 2 ? -1.0 : 0.0;
    *im = q == 1 ? -1.0 : q == 3 ? 1.0 : 0.0;
    return;
  }
  const int N1 = N == 32 ? 8 : 4, N2 = N / N1, k1 = k % N1, k2 = k / N1, n1 = j / N2, n2 = j % N2;
  double ar, ai, br, bi;
  kw_reg_dft_entry(N1, k1, n1, &ar, &ai);
  kw_reg_dft_entry(N2, k2, n2, &br, &bi);
  const double c = (double)(float)kw_ct_trig(n2 * k1, N, false), s = -(double)(float)kw_ct_trig(n2 * k1, N, true);
  const double tr = br * c - bi * s, ti = br * s + bi * c;
  *re = tr * ar - ti * ai;
  *im = tr * ai + ti * ar;
}

// Gains of the N-point DFT at its outputs (N a power of two up to 32, worked out once).
inline const double* kw_reg_dft_gain(int N) {
  struct Table {
    double g[33][32];
    Table() {
      for (int n = 2; n <= 32; n *= 2)
        for (int k = 0; k < n; ++k) {
          double sum = 0.0;
          for (int j = 0; j < n; ++j) {
            double ar, ai, br, bi;
            kw_reg_dft_entry(n, k, j, &ar, &ai);
            kw_reg_dft_entry(n, j, k, &br, &bi);
            sum += ar * br + ai * bi;
          }
          g[n][k] = sum / n - 1.0;
        }
    }
  };
  static const Table table;
  return table.g[N];
}

inline void kw_reg_gain(int E, int P, const float2* w, double* eps) {
  const double *ge = kw_reg_dft_gain(E), *gp = kw_reg_dft_gain(P);
  for (int k1 = 0; k1 < E; ++k1) {
    double g = ge[k1];
    for (int t = 0; t < P; ++t) {
      const double c = w[t * k1].x, s = w[t * k1].y;
      g += (c * c + s * s - 1.0) / P;
    }
    for (int k2 = 0; k2 < P; ++k2) eps[k1 + E * k2] = g + gp[k2];
  }
}

// ---------------------------------------------------------------------------
// register DFTs on packed two-lane adds (FADD2 / FFMA2)
// ---------------------------------------------------------------------------
namespace kwmr {

__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 pfma(float c, float2 a, float2 b) { return __ffma2_rn(make_float2(c, c), a, b); }
__device__ __forceinline__ float2 pmul(float c, float2 a) { return __fmul2_rn(make_float2(c, c), a); }
__device__ __forceinline__ float2 swp(float2 a) { return make_float2(a.y, a.x); }
// a -/+ i b
__device__ __forceinline__ float2 sub_i(float2 a, float2 b) { return make_float2(a.x + b.y, a.y - b.x); }
__device__ __forceinline__ float2 add_i(float2 a, float2 b) { return make_float2(a.x - b.y, a.y + b.x); }
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

template <int N>
__device__ __forceinline__ void dft(float2 (&v)[N]);

template <>
__device__ __forceinline__ void dft<1>(float2 (&)[1]) {}
template <>
__device__ __forceinline__ void dft<2>(float2 (&v)[2]) {
  const float2 a = v[0], b = v[1];
  v[0] = padd(a, b);
  v[1] = psub(a, b);
}
template <>
__device__ __forceinline__ void dft<3>(float2 (&v)[3]) {
  constexpr float s1 = (float)kw_ct_trig(1, 3, true);
  const float2 s = padd(v[1], v[2]), d = pmul(s1, psub(v[1], v[2]));
  const float2 m = pfma(-0.5f, s, v[0]);
  v[0] = padd(v[0], s);
  v[1] = sub_i(m, d);
  v[2] = add_i(m, d);
}
template <>
__device__ __forceinline__ void dft<4>(float2 (&v)[4]) {
  const float2 a0 = padd(v[0], v[2]), a1 = psub(v[0], v[2]);
  const float2 b0 = padd(v[1], v[3]), d = psub(v[1], v[3]);
  v[0] = padd(a0, b0);
  v[2] = psub(a0, b0);
  v[1] = sub_i(a1, d);
  v[3] = add_i(a1, d);
}
template <>
__device__ __forceinline__ void dft<5>(float2 (&v)[5]) {
  constexpr float c1 = (float)kw_ct_trig(1, 5, false), c2 = (float)kw_ct_trig(2, 5, false);
  constexpr float s1 = (float)kw_ct_trig(1, 5, true), s2 = (float)kw_ct_trig(2, 5, true);
  const float2 a1 = padd(v[1], v[4]), b1 = psub(v[1], v[4]);
  const float2 a2 = padd(v[2], v[3]), b2 = psub(v[2], v[3]);
  const float2 m1 = pfma(c2, a2, pfma(c1, a1, v[0]));
  const float2 m2 = pfma(c1, a2, pfma(c2, a1, v[0]));
  const float2 n1 = pfma(s2, b2, pmul(s1, b1));
  const float2 n2 = pfma(-s1, b2, pmul(s2, b1));
  v[0] = padd(v[0], padd(a1, a2));
  v[1] = sub_i(m1, n1);
  v[4] = add_i(m1, n1);
  v[2] = sub_i(m2, n2);
  v[3] = add_i(m2, n2);
}
template <>
__device__ __forceinline__ void dft<7>(float2 (&v)[7]) {
  constexpr float c1 = (float)kw_ct_trig(1, 7, false), c2 = (float)kw_ct_trig(2, 7, false),
                  c3 = (float)kw_ct_trig(3, 7, false);
  constexpr float s1 = (float)kw_ct_trig(1, 7, true), s2 = (float)kw_ct_trig(2, 7, true),
                  s3 = (float)kw_ct_trig(3, 7, true);
  const float2 a1 = padd(v[1], v[6]), b1 = psub(v[1], v[6]);
  const float2 a2 = padd(v[2], v[5]), b2 = psub(v[2], v[5]);
  const float2 a3 = padd(v[3], v[4]), b3 = psub(v[3], v[4]);
  const float2 m1 = pfma(c3, a3, pfma(c2, a2, pfma(c1, a1, v[0])));
  const float2 m2 = pfma(c1, a3, pfma(c3, a2, pfma(c2, a1, v[0])));
  const float2 m3 = pfma(c2, a3, pfma(c1, a2, pfma(c3, a1, v[0])));
  const float2 n1 = pfma(s3, b3, pfma(s2, b2, pmul(s1, b1)));
  const float2 n2 = pfma(-s1, b3, pfma(-s3, b2, pmul(s2, b1)));
  const float2 n3 = pfma(s2, b3, pfma(-s1, b2, pmul(s3, b1)));
  v[0] = padd(v[0], padd(a1, padd(a2, a3)));
  v[1] = sub_i(m1, n1);
  v[6] = add_i(m1, n1);
  v[2] = sub_i(m2, n2);
  v[5] = add_i(m2, n2);
  v[3] = sub_i(m3, n3);
  v[4] = add_i(m3, n3);
}

template <int N, int R, int M, int... E>
__device__ __forceinline__ void twiddle_block(float2 (&sub)[R][M], std::integer_sequence<int, E...>) {
  ((sub[E / M][E % M] = kw_twc<(E / M) * (E % M), N>(sub[E / M][E % M])), ...);
}

// N = R M: R sub-DFTs of M points (j, j + R, ...), constant twiddles, radix-R butterflies.
template <int N>
__device__ __forceinline__ void dft(float2 (&v)[N]) {
  constexpr int R = (N % 4 == 0) ? 4 : (N % 2 == 0) ? 2 : (N % 3 == 0) ? 3 : 5;
  constexpr int M = N / R;
  float2 sub[R][M];
#pragma unroll
  for (int j = 0; j < R; ++j)
#pragma unroll
    for (int i = 0; i < M; ++i) sub[j][i] = v[j + R * i];
#pragma unroll
  for (int j = 0; j < R; ++j) dft<M>(sub[j]);
  twiddle_block<N, R, M>(sub, std::make_integer_sequence<int, R * M>{});
#pragma unroll
  for (int k = 0; k < M; ++k) {
    float2 t[R];
#pragma unroll
    for (int j = 0; j < R; ++j) t[j] = sub[j][k];
    dft<R>(t);
#pragma unroll
    for (int q = 0; q < R; ++q) v[k + M * q] = t[q];
  }
}

// Table twiddles of one butterfly: v[k] *= w^{t k}; w points at the pass's
// table + t, m entries per k.
template <int R>
__device__ __forceinline__ void twiddle(float2 (&v)[R], const float2* __restrict__ w, int m) {
#pragma unroll
  for (int k = 1; k < R; ++k) v[k] = cmulf(v[k], __ldg(w + k * m));
}

// Padded slot of butterfly (block b, offset t) of pass l < np - 1.
__device__ __forceinline__ int slot_of(const KwMrLen& L, int l, int b, int t) {
  int s = b * L.r[l] * L.ms[l] + t;
  if (l + 2 < L.np) s += kw_divu(t, L.drl) * (L.mp - L.rl);
  return s;
}

}  // namespace kwmr
