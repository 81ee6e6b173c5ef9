// One line of a pass by the G threads of its LineFft (fft_reg.cuh): FFT, phase factors, inverse
// FFT, in place in the line's own N slots of a shared-memory tile.  Between a row's forward and
// inverse DFT its points get the phase factors, so the spectrum never leaves the registers.
//
// The line chirp exp(i C (n - (n >= N/2 ? N : 0))) at n = k + R1 r wraps where r >= G/2, so it is
// T[r] e_k: the line's T[r], one evaluated by each of its threads into shared memory with the
// scale folded in, times the thread's own e_k.
#pragma once
#include "fft_reg.cuh"
#include "phase.cuh"

namespace me {

constexpr int kTileLines = 16;  // per CTA

// Chirp of one line; T is the line's G table entries in shared memory.
template <int N>
struct LineChirp {
  static constexpr int G = LineFft<N>::G, R1 = LineFft<N>::R1, NI = LineFft<N>::NI;
  const float2* T;
  float2 e, sg;    // exp(i C k) of the current item, exp(i C G)
  float dmr, tdr;  // multipliers per unit of n - (wrap): dm r_o 2 pi / N and 2 pi / N
  bool deriv, tderiv, conj;
  // every thread of the line calls this; the table is complete after a __syncwarp
  __device__ __forceinline__ void init(const Phase& P, const PhaseCoef& Cf, double r_o, int j,
                                       float scale, float scale_lo, float2* table) {
    const double d = kTwoPi / N;
    const double C = (P.conj ? -1.0 : 1.0) * (Cf.a * r_o + Cf.b) * d;
    table[j] = cscale2(expi_reduced(C * (double)(j * R1 - (j >= G / 2 ? N : 0))), scale, scale_lo);
    T = table;
    e = expi_reduced(C * (double)j);
    if (NI > 1) sg = expi_reduced(C * G);
    dmr = (float)(Cf.dm * r_o * d);
    tdr = (float)d;
    deriv = P.deriv != 0;
    tderiv = P.trans_deriv != 0;
    conj = P.conj != 0;
  }
  __device__ __forceinline__ void apply(float2 (&X)[G], int k) const {
    if (deriv || tderiv) {
#pragma unroll
      for (int r = 0; r < G; r++) {
        const float mm = (float)(k + R1 * r - (r >= G / 2 ? N : 0));
        float2 f = cmul(e, T[r]);
        if (deriv) f = cscale(conj ? mul_mi(f) : mul_i(f), dmr * mm);
        if (tderiv) f = cscale(conj ? mul_i(f) : mul_mi(f), tdr * mm);
        X[r] = cmul(X[r], f);
      }
    } else {
#pragma unroll
      for (int r = 0; r < G; r++) X[r] = cmul(X[r], cmul(e, T[r]));
    }
  }
  __device__ __forceinline__ void next() {
    if (NI > 1) e = cmul(e, sg);
  }
};

// The whole of one line (u, v along axes au and av) of pass A in mode MODE by thread j of its
// G, with the volume's coefficients in coef: s0 and s1 are the line's slots in the first and
// the second tile (the other input or output of the dual modes), table the line's 2 G chirp
// table entries.  midway() is called by every thread after the first stage.
template <int N, int MODE, class S, class Hook>
__device__ __forceinline__ void pass_line(const PassArgs& A, const PhaseCoef* coef, int u, int v,
                                          int j, const S& s0, const S& s1, float2* table,
                                          Hook midway) {
  using L = LineFft<N>;
  constexpr int G = L::G, R1 = L::R1, NI = L::NI;
  constexpr bool kDual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  const bool id0 = phase_is_identity(A.ph[0]), id1 = phase_is_identity(A.ph[1]);
  const bool sep0 = !id0 && A.ph[0].sep, sep1 = kDual && !id1 && A.ph[1].sep;
  LineChirp<N> ch0, ch1;
  auto r_o = [&](const Phase& P) { return P.rvec ? P.rvec[P.oaxis == A.au ? u : v] : 0.0; };
  // (the tables' readers of the previous line are past that line's last __syncwarp)
  if (sep0) ch0.init(A.ph[0], coef[0], r_o(A.ph[0]), j, A.scale, A.scale_lo, table);
  if (sep1) ch1.init(A.ph[1], coef[1], r_o(A.ph[1]), j, A.scale, A.scale_lo, table + G);
  auto load0 = [&](int r, int) { return s0.tab(r, 0); };
  auto load1 = [&](int r, int) { return s1.tab(r, 0); };
  auto store0 = [&](int r, int, float2 x) { s0.tab(r, 0) = x; };
  auto store1 = [&](int r, int, float2 x) { s1.tab(r, 0) = x; };
  if (MODE != PM_INV) L::template first<true>(s0, j, load0);
  if (MODE == PM_DUAL_IN) L::template first<true>(s1, j, load1);
  midway();
  // X (index k + R1 r) times the factors of phase 0 or 1, the form decided once per line
  auto factor = [&](const bool id, const bool sep, const LineChirp<N>& ch, const int q, int k,
                    float2 (&X)[G]) {
    if (id) {
#pragma unroll
      for (int r = 0; r < G; r++) X[r] = cscale2(X[r], A.scale, A.scale_lo);
    } else if (sep) {
      ch.apply(X, k);
    } else {
#pragma unroll
      for (int r = 0; r < G; r++)
        X[r] = cmul(X[r], phase_value_call(A, q, coef[q], k + R1 * r, u, v));
    }
  };
  if (MODE == PM_FWD || MODE == PM_INV) {
    // the spectrum's natural slots belong to other items: all rows are read before any is written
    float2 X[NI][G];
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int k = j + G * i;
      if (k < R1) {
        if (MODE == PM_FWD) {
          L::row_forward(s0, k, X[i]);
        } else {
#pragma unroll
          for (int r = 0; r < G; r++) X[i][r] = s0.at(k + R1 * r);
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int k = j + G * i;
      if (k < R1) {
        factor(id0, sep0, ch0, 0, k, X[i]);
        if (MODE == PM_FWD) {
#pragma unroll
          for (int r = 0; r < G; r++) s0.at(k + R1 * r) = X[i][r];
        } else {
          L::row_inverse(s0, k, X[i]);
        }
      }
      if (sep0) ch0.next();
    }
    __syncwarp();
    if (MODE == PM_INV) L::template last<true>(s0, j, store0);
    return;
  }
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int k = j + G * i;
    if (R1 % G == 0 || k < R1) {
      float2 X[G];
      L::row_forward(s0, k, X);
      if (MODE == PM_DUAL_IN) {
        float2 Y[G];
        factor(id0, sep0, ch0, 0, k, X);
        L::row_forward(s1, k, Y);
        factor(id1, sep1, ch1, 1, k, Y);
#pragma unroll
        for (int r = 0; r < G; r++) X[r] = cadd(X[r], Y[r]);
        L::row_inverse(s0, k, X);
      } else if (MODE == PM_DUAL_OUT) {
        float2 Y[G];
#pragma unroll
        for (int r = 0; r < G; r++) Y[r] = X[r];
        factor(id0, sep0, ch0, 0, k, X);
        L::row_inverse(s0, k, X);
        factor(id1, sep1, ch1, 1, k, Y);
        L::row_inverse(s1, k, Y);
      } else {
        factor(id0, sep0, ch0, 0, k, X);
        L::row_inverse(s0, k, X);
      }
    }
    if (NI > 1 && sep0) ch0.next();
    if (NI > 1 && sep1) ch1.next();
  }
  __syncwarp();
  L::template last<true>(s0, j, store0);
  if (MODE == PM_DUAL_OUT) L::template last<true>(s1, j, store1);
}

}  // namespace me
