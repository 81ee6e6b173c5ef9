// Register-resident small DFTs and the two-stage line FFT used by the compile-time kernels.
//
// A line of N = G R1 points belongs to G threads (G = 8 up to 128 points, 16 above) and N slots of
// shared memory:
//   stage 1: thread j < G transforms x[j + G r], r < R1, in registers and puts output k into slot
//            G k + (j + k) mod G;
//   stage 2: item k (thread k mod G, up to two items each) reads row k, multiplies by W_N^{r k}
//            and transforms its G points into X[k + R1 r].
// The inverse runs the same steps backwards.
//
// Why the second radix is the number of threads: no lane idles in the first stage and few do in
// the second (R1 of G ceil(R1/G) items).  With plans that led with a 16-point stage, 9 of 16 lanes
// idled in it at 112 = 16 x 7 points (133 instructions per voxel of a line pass; 128 = 16 x 8: 119).
// The lanes are dealt so that a half warp holds eight threads of each of two neighbouring lines:
// with a row's start turned by k these touch 16 distinct 8-byte banks in every access, in a tile
// that interleaves the two lines or keeps them 64 bytes apart modulo 128, and the transposes need
// no scratch beside the line.  Only __syncwarp separates the stages, and all index arithmetic but
// the turns is compile-time.
#pragma once
#include "common.cuh"
#include "dft_consts.cuh"

namespace me {

template <int R, bool INV>
__device__ __forceinline__ float2 wr(int m) {
  // W_R^m = exp(-2 pi i m / R) (forward) or its conjugate (inverse); m is a compile-time
  // constant after unrolling, so this folds to immediates.
  const int mm = ((m % R) + R) % R;
  return make_float2(RadixConst<R>::c(mm), INV ? RadixConst<R>::s(mm) : -RadixConst<R>::s(mm));
}

template <int R, bool INV>
struct RDft;

template <bool INV>
struct RDft<1, INV> {
  static __device__ __forceinline__ void run(float2* v) {}
};

template <bool INV>
struct RDft<2, INV> {
  static __device__ __forceinline__ void run(float2* v) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <bool INV>
struct RDft<4, INV> {
  static __device__ __forceinline__ void run(float2* v) {
    const float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    const float2 t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
    const float2 t3r = INV ? mul_i(t3) : mul_mi(t3);
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3r);
    v[3] = csub(t1, t3r);
  }
};

// Odd prime R: pair x_p with x_{R-p} (X[k] and X[R-k] share the cos / sin sums).
template <int R, bool INV>
struct RDftPrime {
  static __device__ __forceinline__ void run(float2* v) {
    constexpr int H = (R - 1) / 2;
    float2 a[H], b[H];
#pragma unroll
    for (int p = 1; p <= H; p++) {
      a[p - 1] = cadd(v[p], v[R - p]);
      b[p - 1] = csub(v[p], v[R - p]);
    }
    const float2 x0 = v[0];
    float2 s0 = x0;
#pragma unroll
    for (int p = 0; p < H; p++) s0 = cadd(s0, a[p]);
    float2 out[R];
    out[0] = s0;
#pragma unroll
    for (int k = 1; k <= H; k++) {
      float2 re = x0, im = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 1; p <= H; p++) {
        const float c = RadixConst<R>::c((p * k) % R);
        const float s = RadixConst<R>::s((p * k) % R);
        re.x = fmaf(c, a[p - 1].x, re.x);
        re.y = fmaf(c, a[p - 1].y, re.y);
        im.x = fmaf(s, b[p - 1].x, im.x);
        im.y = fmaf(s, b[p - 1].y, im.y);
      }
      // forward: X[k] = re - i im, X[R-k] = re + i im ; inverse: signs swapped
      const float2 iim = mul_i(im);
      out[k] = INV ? cadd(re, iim) : csub(re, iim);
      out[R - k] = INV ? csub(re, iim) : cadd(re, iim);
    }
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = out[k];
  }
};

template <bool INV> struct RDft<3, INV> : RDftPrime<3, INV> {};
template <bool INV> struct RDft<5, INV> : RDftPrime<5, INV> {};
template <bool INV> struct RDft<7, INV> : RDftPrime<7, INV> {};
template <bool INV> struct RDft<11, INV> : RDftPrime<11, INV> {};
template <bool INV> struct RDft<13, INV> : RDftPrime<13, INV> {};

// t *= W_R^m for a compile-time m, quarter turns without a multiplication.
template <int R, bool INV>
__device__ __forceinline__ float2 mul_wr(float2 t, int m) {
  if (m == 0) return t;
  if (4 * m == R) return INV ? mul_i(t) : mul_mi(t);
  return cmul(t, wr<R, INV>(m));
}

// Composite R = A * B: n = B n1 + n2, k = k1 + A k2,
// X[k1 + A k2] = sum_{n2} W_R^{n2 k1} W_B^{n2 k2} sum_{n1} x[B n1 + n2] W_A^{n1 k1}.
template <int A, int B, bool INV>
struct RDftComp {
  static __device__ __forceinline__ void run(float2* v) {
    constexpr int R = A * B;
    float2 t[R];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) {
      float2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; n1++) u[n1] = v[B * n1 + n2];
      RDft<A, INV>::run(u);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) t[n2 * A + k1] = mul_wr<R, INV>(u[k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      float2 w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; n2++) w[n2] = t[n2 * A + k1];
      RDft<B, INV>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = w[k2];
    }
  }
};

// Coprime R = A * B by the prime-factor map (Good, 1958): n = B n1 + A n2 and k = k1 mod A,
// k2 mod B turn the DFT into A- and B-point DFTs with no twiddles between (14 points: 156
// floating-point instructions instead of 184).
template <int A, int B, bool INV>
struct RDftPfa {
  // the multiple of B that is 1 mod A (E1) and the multiple of A that is 1 mod B (E2)
  static constexpr int unit(int mult, int mod) {
    int e = mult;
    while (e % mod != 1) e += mult;
    return e;
  }
  static __device__ __forceinline__ void run(float2* v) {
    constexpr int R = A * B, E1 = unit(B, A), E2 = unit(A, B);
    float2 t[R];
#pragma unroll
    for (int n2 = 0; n2 < B; n2++) {
      float2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; n1++) u[n1] = v[(B * n1 + A * n2) % R];
      RDft<A, INV>::run(u);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) t[n2 * A + k1] = u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      float2 w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; n2++) w[n2] = t[n2 * A + k1];
      RDft<B, INV>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[(E1 * k1 + E2 * k2) % R] = w[k2];
    }
  }
};

template <bool INV> struct RDft<6, INV> : RDftPfa<2, 3, INV> {};
template <bool INV> struct RDft<10, INV> : RDftPfa<2, 5, INV> {};
template <bool INV> struct RDft<12, INV> : RDftPfa<4, 3, INV> {};
template <bool INV> struct RDft<14, INV> : RDftPfa<2, 7, INV> {};
template <bool INV> struct RDft<15, INV> : RDftPfa<3, 5, INV> {};
template <bool INV> struct RDft<18, INV> : RDftPfa<2, 9, INV> {};
template <bool INV> struct RDft<20, INV> : RDftPfa<4, 5, INV> {};
template <bool INV> struct RDft<21, INV> : RDftPfa<3, 7, INV> {};
template <bool INV> struct RDft<22, INV> : RDftPfa<2, 11, INV> {};
template <bool INV> struct RDft<24, INV> : RDftPfa<8, 3, INV> {};
template <bool INV> struct RDft<26, INV> : RDftPfa<2, 13, INV> {};
template <bool INV> struct RDft<28, INV> : RDftPfa<4, 7, INV> {};
template <bool INV> struct RDft<30, INV> : RDftPfa<2, 15, INV> {};
template <bool INV> struct RDft<8, INV> : RDftComp<2, 4, INV> {};
template <bool INV> struct RDft<9, INV> : RDftComp<3, 3, INV> {};
template <bool INV> struct RDft<16, INV> : RDftComp<4, 4, INV> {};
template <bool INV> struct RDft<25, INV> : RDftComp<5, 5, INV> {};
template <bool INV> struct RDft<27, INV> : RDftComp<3, 9, INV> {};
template <bool INV> struct RDft<32, INV> : RDftComp<4, 8, INV> {};

// Second-stage twiddles W_N^{r k} in the order r R1 + k.
template <int N> __device__ __forceinline__ const float2* twp_table();
#define ME_TWP_TABLE(N) \
  template <> __device__ __forceinline__ const float2* twp_table<N>() { return twp##N; }
ME_FAST_LENGTHS(ME_TWP_TABLE)
#undef ME_TWP_TABLE

__host__ __device__ constexpr int line_threads(int n) { return n <= 128 ? 8 : 16; }

// Bytes between the lines of a linear tile: a multiple of 16, 64 modulo 128.
__host__ __device__ constexpr int line_pitch(int n) { return n * 8 + (n % 16 == 0 ? 64 : 0); }

// This thread's line g of the CTA's and its place j < G in it.
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
  __device__ __forceinline__ float2& put(int k) const { return tab(k, k); }
  __device__ __forceinline__ float2& row(int k, int r) const { return tab(k, r); }
};

// Slots of a line that has a region of its own beside the data (line_region elements): rows by
// thread with an odd stride, so that all offsets but the thread's own are compile-time.  Free of
// bank conflicts with sixteen threads of one line to a half warp, and with eight of two lines
// whose regions lie 8 elements apart modulo 16.
__host__ __device__ constexpr int line_region(int n) {
  const int g = line_threads(n), r1 = n / g, need = g * (r1 | 1) > n ? g * (r1 | 1) : n;
  return (need + 7) / 16 * 16 + 8;
}
template <int N>
struct PaddedSlots {
  static constexpr int S1 = (N / line_threads(N)) | 1;
  float2* line;
  float2* mine;  // line + j S1
  __device__ __forceinline__ void init(float2* l, int j) {
    line = l;
    mine = l + j * S1;
  }
  __device__ __forceinline__ float2& at(int n) const { return line[n]; }
  __device__ __forceinline__ float2& put(int k) const { return mine[k]; }
  __device__ __forceinline__ float2& row(int k, int r) const { return line[r * S1 + k]; }
};

template <int N>
struct LineFft {
  static constexpr int G = line_threads(N);
  static constexpr int R1 = N / G;
  static constexpr int NI = (R1 + G - 1) / G;  // stage 2 items per thread

  // Stage 1 of x[n] = load(r, n) (n = j + G r, read once) into the turned slots.  IN_PLACE: load
  // reads the slots themselves, which other threads are about to overwrite.
  template <bool IN_PLACE, class S, class Load>
  static __device__ __forceinline__ void first(const S& s, int j, Load load) {
    float2 u[R1];
#pragma unroll
    for (int r = 0; r < R1; r++) u[r] = load(r, j + G * r);
    RDft<R1, false>::run(u);
    if (IN_PLACE) __syncwarp();
#pragma unroll
    for (int k = 0; k < R1; k++) s.put(k) = u[k];
    __syncwarp();
  }
  // Stage 3: the turned slots to store(r, n, x[n]).
  template <bool IN_PLACE, class S, class Store>
  static __device__ __forceinline__ void last(const S& s, int j, Store store) {
    float2 u[R1];
#pragma unroll
    for (int k = 0; k < R1; k++) u[k] = s.put(k);
    RDft<R1, true>::run(u);
    if (IN_PLACE) __syncwarp();
#pragma unroll
    for (int r = 0; r < R1; r++) store(r, j + G * r, u[r]);
  }
  // Row k = j + G i to its spectrum X[k + R1 r] and back.
  template <class S>
  static __device__ __forceinline__ void row_forward(const S& s, int k, float2 (&X)[G]) {
#pragma unroll
    for (int r = 0; r < G; r++) {
      const float2 y = s.row(k, r);
      X[r] = (r == 0) ? y : cmul(y, __ldg(twp_table<N>() + r * R1 + k));
    }
    RDft<G, false>::run(X);
  }
  template <class S>
  static __device__ __forceinline__ void row_inverse(const S& s, int k, float2 (&X)[G]) {
    RDft<G, true>::run(X);
#pragma unroll
    for (int r = 0; r < G; r++)
      s.row(k, r) = (r == 0) ? X[r] : cmulc(X[r], __ldg(twp_table<N>() + r * R1 + k));
  }
  // Forward transform of load(r, n) to the natural-order spectrum in the line's slots, and the
  // inverse of that spectrum to store(r, n, x[n]).  The natural slots of one row's results belong
  // to other rows, so a thread holds all its rows before any is written.
  template <class S, class Load>
  static __device__ __forceinline__ void forward(const S& s, int j, Load load) {
    first<false>(s, j, load);
    float2 X[NI][G];
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (R1 % G == 0 || j + G * i < R1) row_forward(s, j + G * i, X[i]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (R1 % G == 0 || j + G * i < R1) {
#pragma unroll
        for (int r = 0; r < G; r++) s.at(j + G * i + R1 * r) = X[i][r];
      }
  }
  template <class S, class Store>
  static __device__ __forceinline__ void inverse(const S& s, int j, Store store) {
    float2 X[NI][G];
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (R1 % G == 0 || j + G * i < R1) {
#pragma unroll
        for (int r = 0; r < G; r++) X[i][r] = s.at(j + G * i + R1 * r);
      }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NI; i++)
      if (R1 % G == 0 || j + G * i < R1) row_inverse(s, j + G * i, X[i]);
    __syncwarp();
    last<false>(s, j, store);
  }
};

}  // namespace me
