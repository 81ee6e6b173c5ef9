// One line of a pass, N = G R1 points by G threads (G = 8 up to 128 points, 16 above): FFT, phase
// factors, inverse FFT, in place in the line's own N slots of a shared-memory tile.
//
//   stage 1: thread j < G transforms x[j + G r], r < R1, in registers and puts output k into slot
//            G k + (j + k) mod G;
//   stage 2: item k (thread k mod G, up to two items each) reads row k, multiplies by W_N^{r k},
//            transforms its G points into X[k + R1 r], multiplies by the phase factors, and runs
//            the same steps back into the same slots;
//   stage 3: thread j takes its R1 slots back and writes x[j + G r].
//
// Why the second radix is the number of threads: no lane idles in the first stage and few do in
// the second (R1 of G ceil(R1/G) items).  With plans that led with a 16-point stage, 9 of 16 lanes
// idled in it at 112 = 16 x 7 points (133 instructions per voxel and pass; 128 = 16 x 8: 119).
// The lanes are dealt so that a half warp holds eight threads of each of two neighbouring lines:
// with a row's start turned by k these touch 16 distinct 8-byte banks in every access, in a tile
// that interleaves the two lines or keeps them 64 bytes apart modulo 128, and the transposes need
// no scratch beside the tile.  Only __syncwarp separates the stages.
//
// The line chirp exp(i C (n - (n >= N/2 ? N : 0))) at n = k + R1 r wraps where r >= G/2, so it is
// T[r] e_k: the line's T[r], one evaluated by each of its threads into shared memory with the
// scale folded in, times the thread's own e_k.
#pragma once
#include "fft_reg.cuh"
#include "phase.cuh"

namespace me {

constexpr int kTileLines = 16;  // per CTA

__host__ __device__ constexpr int line_threads(int n) { return n <= 128 ? 8 : 16; }

template <int N> __device__ __forceinline__ const float2* tp_table();
#define ME_TP_TABLE(N, R1, R2) \
  template <> __device__ __forceinline__ const float2* tp_table<N>() { return tp_##N; }
ME_FAST_LENGTHS(ME_TP_TABLE)
#undef ME_TP_TABLE

// This thread's line g of the CTA's 16 and its place j < G in it.
template <int G>
__device__ __forceinline__ void line_place(int& g, int& j) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (G == 8) {
    g = warp * 4 + (lane >> 3);
    j = lane & 7;
  } else {
    g = warp * 2 + ((lane >> 3) & 1);
    j = (lane & 7) | ((lane >> 4) << 3);
  }
}

// A line's slots in a tile, as thread j of the line sees them.  A row of G slots is ROW bytes from
// the next; slot (j + q) mod G of a row lies at F[q mod 8], the other half of 16 slots at XOR HALF.
//   STRIDED: tile [n][16 lines] with the tensor map's 128-byte swizzle (the 16-byte chunk of
//     line pair g / 2 at index n is g / 2 XOR n mod 8);
//   else: the line's N slots in a row, neighbouring lines 64 bytes apart modulo 128.
template <int G, bool STRIDED>
struct Slots {
  static constexpr int ROW = STRIDED ? 128 * G : 8 * G;
  static constexpr int HALF = STRIDED ? 1024 : 64;
  unsigned char* line;
  int F[8];
  int g;
  __device__ __forceinline__ int in_row(int m) const {
    return STRIDED ? m * 128 + ((((g >> 1) ^ m) & 7) << 4) + ((g & 1) << 3) : m * 8;
  }
  __device__ __forceinline__ void init(int g_, int j) {
    g = g_;
#pragma unroll
    for (int q = 0; q < 8; q++) F[q] = in_row((j + q) & (G - 1));
  }
  // row `row`, slot (j + q) mod G
  __device__ __forceinline__ float2& tab(int row, int q) const {
    const int f = F[q & 7] ^ ((G == 16 && (q & 8)) ? HALF : 0);
    return *reinterpret_cast<float2*>(line + f + row * ROW);
  }
  __device__ __forceinline__ float2& at(int n) const {
    return *reinterpret_cast<float2*>(line + (n / G) * ROW + in_row(n & (G - 1)));
  }
};

template <int N>
struct PassLine {
  static constexpr int G = line_threads(N);
  static constexpr int R1 = N / G;
  static constexpr int NI = (R1 + G - 1) / G;  // stage 2 items per thread
  static constexpr int THREADS = kTileLines * G;

  // stages 1 and 3
  template <class S>
  static __device__ __forceinline__ void first(const S& s) {
    float2 u[R1];
#pragma unroll
    for (int r = 0; r < R1; r++) u[r] = s.tab(r, 0);
    RDft<R1, false>::run(u);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < R1; k++) s.tab(k, k) = u[k];
    __syncwarp();
  }
  template <class S>
  static __device__ __forceinline__ void last(const S& s) {
    float2 u[R1];
#pragma unroll
    for (int k = 0; k < R1; k++) u[k] = s.tab(k, k);
    RDft<R1, true>::run(u);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < R1; r++) s.tab(r, 0) = u[r];
  }
  // row k = j + G i to its spectrum X[k + R1 r] and back
  template <class S>
  static __device__ __forceinline__ void row_forward(const S& s, int k, float2 (&X)[G]) {
#pragma unroll
    for (int r = 0; r < G; r++) {
      const float2 y = s.tab(k, r);
      X[r] = (r == 0) ? y : cmul(y, __ldg(tp_table<N>() + r * R1 + k));
    }
    RDft<G, false>::run(X);
  }
  template <class S>
  static __device__ __forceinline__ void row_inverse(const S& s, int k, float2 (&X)[G]) {
    RDft<G, true>::run(X);
#pragma unroll
    for (int r = 0; r < G; r++)
      s.tab(k, r) = (r == 0) ? X[r] : cmulc(X[r], __ldg(tp_table<N>() + r * R1 + k));
  }
};

// Chirp of one line; T is the line's G table entries in shared memory.
template <int N>
struct LineChirp {
  static constexpr int G = PassLine<N>::G, R1 = PassLine<N>::R1, NI = PassLine<N>::NI;
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
// table entries.
template <int N, int MODE, class S>
__device__ __forceinline__ void pass_line(const PassArgs& A, const PhaseCoef* coef, int u, int v,
                                          int j, const S& s0, const S& s1, float2* table) {
  using L = PassLine<N>;
  constexpr int G = L::G, R1 = L::R1, NI = L::NI;
  constexpr bool kDual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  const bool id0 = phase_is_identity(A.ph[0]), id1 = phase_is_identity(A.ph[1]);
  const bool sep0 = !id0 && A.ph[0].sep, sep1 = kDual && !id1 && A.ph[1].sep;
  LineChirp<N> ch0, ch1;
  auto r_o = [&](const Phase& P) { return P.rvec ? P.rvec[P.oaxis == A.au ? u : v] : 0.0; };
  // (the tables' readers of the previous line are past that line's last __syncwarp)
  if (sep0) ch0.init(A.ph[0], coef[0], r_o(A.ph[0]), j, A.scale, A.scale_lo, table);
  if (sep1) ch1.init(A.ph[1], coef[1], r_o(A.ph[1]), j, A.scale, A.scale_lo, table + G);
  if (MODE != PM_INV) L::first(s0);
  if (MODE == PM_DUAL_IN) L::first(s1);
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
    if (MODE == PM_INV) L::last(s0);
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
  L::last(s0);
  if (MODE == PM_DUAL_OUT) L::last(s1);
}

}  // namespace me
