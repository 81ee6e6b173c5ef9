// Two-stage line FFT N = R1 * R2 with radices chosen at run time, for the lengths that have no
// compile-time plan (fft_reg.cuh): any N whose plan finds R1 <= 16 and R2 <= 32 among the
// register DFTs below, which is every length up to 256 with prime factors up to 13 but 245, and
// most up to 512.
//
// A stage is one register DFT per work item, its radix picked by a switch that the whole CTA
// takes the same way, so the DFTs stay unrolled while a kernel serves every length.  A kernel's
// registers are those of its largest radix: R2 above 16 has kernels of its own, of 128 registers;
// the stack frames are 80 bytes at most there and 48 bytes elsewhere.  Items are dealt to threads over all of a tile's lines (thread i has the one item i
// of a stage), so a radix that is no power of two leaves whole warps idle at the end of the
// CTA rather than lanes in every warp:
//   stage 1: item (line b, j < R2) transforms x[j + r R2], r < R1, into row j of the line's
//            [R2][S1] table (S1 = R1 rounded up to odd);
//   stage 2: item (line b, k < R1) reads column k, multiplies by W_N^{r k}, transforms over
//            r < R2 and holds X[k + r R1].
// The inverse runs the same steps backwards.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fft_reg.cuh"

namespace me {

#define ME_RT_SMALL(X) \
  X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)
#define ME_RT_LARGE(X) \
  X(18) X(20) X(21) X(22) X(24) X(25) X(26) X(27) X(28) X(30) X(32)

constexpr int kRtMaxR1 = 16;

struct RtPlan {
  int n = 0;
  int r1 = 0, r2 = 0;
  int s1 = 0;          // R1 | 1
  FastDiv d1, d2;      // division by R1 and R2 (item -> line and position)
  int rmax() const { return r1 > r2 ? r1 : r2; }
  bool large() const { return r2 > 16; }
};

// Approximate cost per point of a register DFT (FP32 instructions), to compare plans.
inline double rt_radix_cost(int r) {
  if (r == 1) return 0.0;
  const int p[6] = {4, 2, 3, 5, 7, 11};
  for (int i = 0; i < 6; i++) {
    if (r == p[i]) break;
    if (r % p[i] == 0) {
      const int a = p[i], b = r / p[i];
      const bool coprime = (a % 2 || b % 2) && (a % 3 || b % 3) && (a % 5 || b % 5);
      return rt_radix_cost(a) + rt_radix_cost(b) + (coprime ? 0.0 : 4.0 * (a - 1) * (b - 1) / r);
    }
  }
  if (r == 2) return 2.0;
  if (r == 4) return 4.0;
  const double h = 0.5 * (r - 1);
  return (4.0 * h * h + 8.0 * h) / r;
}

// The plan of length n: the cheapest pair, with a lead for radices up to 16 (twice the lines
// per CTA and more of them resident).  False when no pair fits.
inline bool rt_plan(int n, RtPlan* p) {
  static const bool ok2[33] = {0, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1,
                               0, 1, 0, 1, 1, 1, 0, 1, 1, 1, 1, 1, 0, 1, 0, 1};
  double best = 1e30;
  for (int r1 = 1; r1 <= kRtMaxR1; r1++) {
    if (n % r1) continue;
    const int r2 = n / r1;
    if (r2 > 32 || !ok2[r2]) continue;
    const double c = rt_radix_cost(r1) + rt_radix_cost(r2) + (r2 > 16 ? 12.0 : 0.0) +
                     0.05 * (r1 > r2 ? r1 - r2 : r2 - r1);
    if (c < best) {
      best = c;
      p->r1 = r1;
      p->r2 = r2;
    }
  }
  if (best > 1e29) return false;
  p->n = n;
  p->s1 = p->r1 | 1;
  p->d1.set(p->r1);
  p->d2.set(p->r2);
  return true;
}

// The second stage's twiddles W_N^{r k} (forward) in the order r R1 + k, cooperatively.
__device__ __forceinline__ void rt_init_twiddles(float2* tw, const RtPlan& P) {
  for (int i = threadIdx.x; i < P.n; i += blockDim.x) {
    const int r = P.d1.div(i), k = i - r * P.r1;
    double s, c;
    sincospi(-2.0 * (double)(r * k) / (double)P.n, &s, &c);
    tw[i] = make_float2((float)c, (float)s);
  }
}

// v, hidden from the compiler's knowledge of how it came about.  The multiples r * step of a stride
// that does not change between tiles would otherwise be kept in registers across the tile loop, a
// set for every radix of the switches, and spilled: the line passes had stack frames of 0.5 to
// 4.9 KB, which also size the local memory that the device sets aside for all threads.
__device__ __forceinline__ int fresh(int v) {
  asm volatile("" : "+r"(v));
  return v;
}
__device__ __forceinline__ i64 fresh(i64 v) {
  asm volatile("" : "+l"(v));
  return v;
}

// Calls f(std::integral_constant<int, R>) with the radix of a stage.
template <class F>
__device__ __forceinline__ void rt_switch1(int r, F&& f) {
  switch (r) {
#define ME_RT_CASE(R) \
  case R: f(std::integral_constant<int, R>{}); break;
    ME_RT_SMALL(ME_RT_CASE)
    default: break;
  }
}
template <bool LARGE, class F>
__device__ __forceinline__ void rt_switch2(int r, F&& f) {
  if constexpr (LARGE) {
    switch (r) {
      ME_RT_LARGE(ME_RT_CASE)
      default: break;
    }
  } else {
    rt_switch1(r, f);
  }
}
#undef ME_RT_CASE

}  // namespace me
