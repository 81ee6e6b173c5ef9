// Dispatch of the run-time passes (rt_pass.cuh); each mode is compiled in a file of its own.
#include <atomic>
#include <cmath>

#include "fft_rt.cuh"
#include "line_pass.cuh"

namespace me {

template <int MODE>
int launch_rt_mode(PassArgs& A, const RtPlan& P, cudaStream_t stream);

// Mean of |w|^2 over the twiddles exp(-2 pi i a b / n), a < na, b < nb, rounded to float: what a
// transform and its inverse multiply an element by at that level, on average.
static double twiddle_gain(int n, int na, int nb) {
  double sum = 0.0;
  for (int a = 0; a < na; a++)
    for (int b = 0; b < nb; b++) {
      const double ang = kTwoPi * (double)((a * b) % n) / n;
      const double c = (float)std::cos(ang), s = (float)std::sin(ang);
      sum += (a * b == 0) ? 1.0 : c * c + s * s;
    }
  return sum / ((double)na * nb);
}

// The same for a register DFT (RDft, fft_reg.cuh): radices 2 and 4 are exact, a prime's
// coefficients are its twiddles, a composite is two DFTs with twiddles between where its
// factors are not coprime.
static double radix_gain(int r) {
  if (r <= 2 || r == 4) return 1.0;
  static const int first[33] = {0, 0, 0, 0, 0, 0, 2, 0, 2, 3, 2, 0, 4, 0, 2, 3, 4,
                                0, 2, 0, 4, 3, 2, 0, 8, 5, 2, 3, 4, 0, 2, 0, 4};
  const int a = first[r];
  if (a == 0) return twiddle_gain(r, r, r);
  const int b = r / a;
  const bool coprime = (a % 2 || b % 2) && (a % 3 || b % 3) && (a % 5 || b % 5);
  return radix_gain(a) * radix_gain(b) * (coprime ? 1.0 : twiddle_gain(r, a, b));
}

double fft_pair_gain(int n) {
  static std::atomic<double> known[ME_MAX_LINE + 1];
  if (n < 1 || n > ME_MAX_LINE) return 1.0;
  double g = known[n].load(std::memory_order_relaxed);
  if (g != 0.0) return g;
  int r1 = 0, r2 = 0;
  switch (n) {
#define ME_GAIN_CASE(N)       \
  case N:                     \
    r1 = LineFft<N>::R1;      \
    r2 = LineFft<N>::G;       \
    break;
    ME_FAST_LENGTHS(ME_GAIN_CASE)
#undef ME_GAIN_CASE
    default: {
      RtPlan P;
      if (rt_plan(n, &P)) {
        r1 = P.r1;
        r2 = P.r2;
      }
    }
  }
  g = r1 ? radix_gain(r1) * radix_gain(r2) * twiddle_gain(n, r1, r2) : 1.0;
  known[n].store(g, std::memory_order_relaxed);
  return g;
}

int try_rt_pass(int mode, PassArgs& A, cudaStream_t stream) {
  RtPlan P;
  if (!rt_plan(A.plan.n, &P)) return -1;
  switch (mode) {
    case PM_SHEAR: return launch_rt_mode<PM_SHEAR>(A, P, stream);
    case PM_DUAL_OUT: return launch_rt_mode<PM_DUAL_OUT>(A, P, stream);
    case PM_DUAL_IN: return launch_rt_mode<PM_DUAL_IN>(A, P, stream);
    case PM_FWD: return launch_rt_mode<PM_FWD>(A, P, stream);
    default: return launch_rt_mode<PM_INV>(A, P, stream);
  }
}

}  // namespace me
