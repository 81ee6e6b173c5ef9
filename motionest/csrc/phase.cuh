// Device evaluation of a line pass's phase factors (struct Phase, line_pass.cuh).
#pragma once
#include "line_pass.cuh"

namespace me {

struct PhaseCoef {
  double a, b, dm;
};

__device__ __forceinline__ PhaseCoef phase_coef(const Phase& P, const double* prm, int ax) {
  PhaseCoef c{0.0, 0.0, 0.0};
  if (P.kind != PH_NONE) {
    const double th = prm[3 + P.rot];
    if (P.kind == PH_TAN) {
      const double t = tan(th * 0.5);
      c.a = t;
      c.dm = 0.5 * (1.0 + t * t);
    } else {
      c.a = -sin(th);
      c.dm = -cos(th);
    }
  }
  if (P.trans) c.b = -prm[ax];
  return c;
}

__device__ __forceinline__ bool phase_is_identity(const Phase& P) {
  return P.kind == PH_NONE && !P.trans && !P.trans_deriv && !P.deriv;
}

// Phase factor for frequency index n along the pass axis at spatial coordinates c[0..2]
// (c[ax] is ignored by the planes, which are constant or broadcast along the pass axis in
// frequency; c[ax] carries n itself).
__device__ __forceinline__ float2 phase_value(const Phase& P, const PhaseCoef& C, int n,
                                              const int c[3], float scale, float scale_lo) {
  double rk = 0.0, kn = 0.0;
  if (P.plane) rk = P.plane[c[0] * P.ps[0] + c[1] * P.ps[1] + c[2] * P.ps[2]];
  if (P.kv) kn = P.kv[n];
  float2 e = expi_reduced(C.a * rk + C.b * kn);
  if (P.deriv) e = cscale(mul_i(e), (float)(C.dm * rk));
  if (P.trans_deriv) e = cscale(mul_mi(e), (float)kn);
  if (P.conj) e = cconj(e);
  return cscale2(e, scale, scale_lo);
}

// Phase q of pass A at (u, v) along axes au and av, as a call: for the rare grids whose phases
// are no line chirps.
__device__ __noinline__ static float2 phase_value_call(const PassArgs& A, int q, PhaseCoef C,
                                                       int n, int u, int v) {
  int c[3];
  c[A.au] = u;
  c[A.av] = v;
  c[A.ax] = n;
  return phase_value(A.ph[q], C, n, c, A.scale, A.scale_lo);
}

}  // namespace me
