// Line passes of the lengths without a compile-time plan, on the run-time two-stage FFT
// (fft_rt.cuh).  Same contract as line_pass_kernel (line_pass.cu).
//
// One CTA owns a tile of B lines (16, or 8 when R2 > 16) of one volume and takes tiles in turn.
// The first stage reads its elements straight from global memory into registers and the last
// one writes them straight back, coalesced over the lines of the tile where the pass axis is
// strided and along the line where it is contiguous, so a line crosses shared memory twice in
// each direction instead of four times and no alignment is asked of the volume.  What bounds it:
// the latency of those loads, which three CTAs per SM (two for R2 > 16 and the dual modes) cover,
// and instruction issue.  Strides are taken through `fresh` (fft_rt.cuh) and the dual modes hold one
// spectrum at a time, so that next to nothing is spilled; with all their multiples kept and both
// spectra held, one partial derivative (12 passes, three of them dual) of a 27x125x216 image took
// 1,146 us instead of 234 (on the Stockham engine of line_pass_kernel 911), of 60x63x50 210 instead
// of 113, of 180x150x126 682 instead of 456 (Stockham 3,154), and the device set 1.2 GB aside for
// local memory.  Not used where a compile-time plan exists: at 256x224x176, 64 volumes, ten
// passes took 37.0 ms here and 26.1 ms on the TMA tiles of tma_pass_kernel (both measured before
// the spills were gone).
#pragma once
#include <algorithm>
#include <atomic>

#include "fft_rt.cuh"
#include "line_pass.cuh"
#include "phase.cuh"

namespace me {

// Table position of (line b, row j, column k): line-fastest for strided lines (the lanes of a
// warp hold neighbouring lines), else one odd-strided region per line.
struct RtIndex {
  int sb, sj, sk;
  __device__ __forceinline__ int at(int b, int j, int k) const { return b * sb + j * sj + k * sk; }
};

template <int MODE, bool LARGE>
__global__ void __launch_bounds__(256, (LARGE || MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT) ? 2 : 3)
    rt_pass_kernel(const __grid_constant__ PassArgs A, const __grid_constant__ RtPlan P) {
  constexpr int B = LARGE ? 8 : 16;
  constexpr bool kDual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  constexpr int NPH = kDual ? 2 : 1;
  constexpr int R2MAX = LARGE ? 32 : 16;
  extern __shared__ __align__(16) float2 smem[];
  __shared__ PhaseCoef coef_s[2];
  // scale * exp(i C (r R1 - N where r R1 >= N/2)), r < R2, and in row R2 the wrapped form of the
  // one row in which some k pass N/2
  __shared__ float2 step_s[NPH][R2MAX + 1][B];
  const int N = P.n, R1 = P.r1, R2 = P.r2, S1 = P.s1;
  const bool bfast = (A.st[A.av] == 1);
  RtIndex ix;
  int region;
  if (bfast) {
    ix.sb = 1;
    ix.sj = S1 * B;
    ix.sk = B;
    region = R2 * S1 * B;
  } else {
    ix.sb = (R2 * S1) | 1;
    ix.sj = S1;
    ix.sk = 1;
    region = ix.sb * B;
  }
  float2* tw = smem;
  float2* reg0 = tw + N;
  float2* reg1 = reg0 + region;  // dual modes
  rt_init_twiddles(tw, P);

  // this thread's item of the stages over j < R2 (1 and 3) and of the one over k < R1 (2)
  const int tid = threadIdx.x;
  int b1, j1, b2, k2;
  if (bfast) {
    b1 = b2 = tid % B;
    j1 = k2 = tid / B;
  } else {
    b1 = P.d2.div(tid);
    j1 = tid - b1 * R2;
    b2 = P.d1.div(tid);
    k2 = tid - b2 * R1;
  }
  const bool has1 = tid < B * R2, has2 = tid < B * R1;

  const int tiles_per_vol = (A.nlines + B - 1) / B;
  const int total = tiles_per_vol * A.nvol;
  const i64 sa = A.st[A.ax];
  const int dv = A.dims[A.av];
  const bool id0 = phase_is_identity(A.ph[0]);
  const bool id1 = phase_is_identity(A.ph[1]);
  const bool sep0 = !id0 && A.ph[0].sep, sep1 = kDual && !id1 && A.ph[1].sep;
  const int half = N / 2;
  const int rwrap = half > 0 ? (half - 1) / R1 : 0;  // the last row that starts below N/2
  const double odd_h = (N & 1) ? 0.5 : 0.0;

  chain_next();
  chain_wait();
  int coef_vol = -1;
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    const int vol = A.div_tiles.div(t);
    const int l0 = (t - vol * tiles_per_vol) * B;
    const int nl = min(B, A.nlines - l0);
    // the shear coefficients depend on the volume only; their last readers are past the barrier
    // that the previous tile's third stage follows
    if (vol != coef_vol) {
      if (tid < NPH) {
        PhaseCoef cf{0, 0, 0};
        if (A.params) cf = phase_coef(A.ph[tid], A.params + (i64)vol * A.pstride, A.ax);
        coef_s[tid] = cf;
      }
      coef_vol = vol;
      __syncthreads();
    }
    // base offset of a line, and its coordinates
    auto line = [&](int b, int& u, int& v) {
      const int l = l0 + min(b, nl - 1);
      u = A.div_av.div(l);
      v = l - u * dv;
      return (i64)u * A.st[A.au] + (i64)v * A.st[A.av];
    };
    // C = (a r_o + b) 2 pi / N of a line: its factor at index n is
    // exp(i C (n + h - (n >= N/2 ? N : 0))), h = 1/2 for odd N
    auto chirp_c = [&](const Phase& ph, const PhaseCoef& cf, int u, int v) {
      const int o = (ph.oaxis == A.au) ? u : v;
      const double r_o = ph.rvec ? ph.rvec[o] : 0.0;
      return (ph.conj ? -1.0 : 1.0) * (cf.a * r_o + cf.b) * (kTwoPi / N);
    };

    if (MODE != PM_INV && has1) {
      int u, v;
      const i64 base = line(b1, u, v) + (i64)j1 * sa;
      const i64 step = fresh((i64)R2 * sa);
      const int sk = fresh(ix.sk);
      const bool live = b1 < nl;
      rt_switch1(R1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
#pragma unroll
        for (int q = 0; q < (MODE == PM_DUAL_IN ? 2 : 1); q++) {
          const float2* src = (q == 0 ? A.in0 : A.in1) + (i64)vol * A.in_vs + base;
          float2 x[R];
#pragma unroll
          for (int r = 0; r < R; r++, src += step) x[r] = live ? *src : make_float2(0.f, 0.f);
          RDft<R, false>::run(x);
          float2* dst = (q == 0 ? reg0 : reg1) + ix.at(b1, j1, 0);
#pragma unroll
          for (int r = 0; r < R; r++, dst += sk) *dst = x[r];
        }
      });
    }
    // chirp tables: row r of a line by the thread of item (line, j = r)
    if ((sep0 || sep1) && has1) {
      int u, v;
      line(b1, u, v);
#pragma unroll
      for (int q = 0; q < NPH; q++) {
        if (!(q == 0 ? sep0 : sep1)) continue;
        const double C = chirp_c(A.ph[q], coef_s[q], u, v);
        const int n0 = j1 * R1;
        step_s[q][j1][b1] = cscale2(expi_reduced(C * (double)(n0 >= half ? n0 - N : n0)), A.scale,
                                    A.scale_lo);
        if (j1 == rwrap)
          step_s[q][R2][b1] = cscale2(expi_reduced(C * (double)(n0 - N)), A.scale, A.scale_lo);
      }
    }
    __syncthreads();

    if (has2) {
      int u, v;
      const i64 base = line(b2, u, v) + (i64)k2 * sa;
      const i64 step = fresh((i64)R1 * sa);
      const bool live = b2 < nl;
      int c[3];
      c[A.au] = u;
      c[A.av] = v;
      c[A.ax] = 0;
      float2* col0 = reg0 + ix.at(b2, 0, k2);
      float2* col1 = reg1 + ix.at(b2, 0, k2);
      // the thread's own exp(i C (k + h)), and the row whose table entry it takes wrapped
      float2 e[NPH];
      const int rsel = (k2 + rwrap * R1 >= half && rwrap * R1 < half) ? rwrap : -1;
#pragma unroll
      for (int q = 0; q < NPH; q++) {
        e[q] = make_float2(0.f, 0.f);
        if (q == 0 ? sep0 : sep1)
          e[q] = expi_reduced(chirp_c(A.ph[q], coef_s[q], u, v) * ((double)k2 + odd_h));
      }
      // a phase that is no line chirp: its factors one by one into a column that this thread
      // has already read
      auto general = [&](const int q, float2* col) {
        if ((q == 0 ? id0 || sep0 : id1 || sep1)) return;
#pragma unroll 1
        for (int r = 0; r < R2; r++) {
          c[A.ax] = k2 + r * R1;
          col[r * ix.sj] = phase_value(A.ph[q], coef_s[q], k2 + r * R1, c, A.scale, A.scale_lo);
        }
      };
      rt_switch2<LARGE>(R2, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        auto forward = [&](const float2* col, float2 (&X)[R]) {
          const int sj = fresh(ix.sj), st = fresh(R1);
          const float2* w = tw + k2;
#pragma unroll
          for (int r = 0; r < R; r++, col += sj, w += st) X[r] = (r == 0) ? *col : cmul(*col, *w);
          RDft<R, false>::run(X);
        };
        auto inverse = [&](float2* col, float2 (&X)[R]) {
          RDft<R, true>::run(X);
          const int sj = fresh(ix.sj), st = fresh(R1);
          const float2* w = tw + k2;
#pragma unroll
          for (int r = 0; r < R; r++, col += sj, w += st) *col = (r == 0) ? X[r] : cmulc(X[r], *w);
        };
        // X[r] (index k + r R1) times the factors of phase q: the line's table entry times the
        // thread's own, one rounding each
        auto factor = [&](const int q, float2* col, float2 (&X)[R]) {
          const Phase& ph = A.ph[q];
          if (q == 0 ? id0 : id1) {
#pragma unroll
            for (int r = 0; r < R; r++) X[r] = cscale2(X[r], A.scale, A.scale_lo);
          } else if (q == 0 ? sep0 : sep1) {
            const float2* st = &step_s[q][0][b2];
            if (ph.deriv || ph.trans_deriv) {
              const int o = (ph.oaxis == A.au) ? u : v;
              const double r_o = ph.rvec ? ph.rvec[o] : 0.0;
              const float dmr = (float)(coef_s[q].dm * r_o * (kTwoPi / N));
              const float tdr = (float)(kTwoPi / N);
              int n = fresh(k2);
              const int dn = fresh(R1);
#pragma unroll
              for (int r = 0; r < R; r++, n += dn) {
                const float mm = (float)(n - (n >= half ? N : 0)) + (float)odd_h;
                float2 f = cmul(e[q], st[(r == rsel ? R2 : r) * B]);
                if (ph.deriv) f = cscale(ph.conj ? mul_mi(f) : mul_i(f), dmr * mm);
                if (ph.trans_deriv) f = cscale(ph.conj ? mul_i(f) : mul_mi(f), tdr * mm);
                X[r] = cmul(X[r], f);
              }
            } else {
#pragma unroll
              for (int r = 0; r < R; r++)
                X[r] = cmul(X[r], cmul(e[q], st[(r == rsel ? R2 : r) * B]));
            }
          } else {
            general(q, col);
            const int sj = fresh(ix.sj);
#pragma unroll
            for (int r = 0; r < R; r++, col += sj) X[r] = cmul(X[r], *col);
          }
        };
        float2 X[R];
        if (MODE == PM_INV) {
          const float2* src = A.in0 + (i64)vol * A.in_vs + base;
#pragma unroll
          for (int r = 0; r < R; r++, src += step) X[r] = live ? *src : make_float2(0.f, 0.f);
        } else {
          forward(col0, X);
        }
        // The dual modes park a spectrum in a column that this thread alone reads and writes, so
        // that one of them is in registers at a time.
        auto park = [&](float2* col) {
          const int sj = fresh(ix.sj);
#pragma unroll
          for (int r = 0; r < R; r++, col += sj) *col = X[r];
        };
        if (MODE == PM_DUAL_IN) {
          factor(0, col0, X);
          park(col0);
          forward(col1, X);
          factor(1, col1, X);
          const float2* first = col0;
          const int sj = fresh(ix.sj);
#pragma unroll
          for (int r = 0; r < R; r++, first += sj) X[r] = cadd(*first, X[r]);
          inverse(col0, X);
        } else if (MODE == PM_DUAL_OUT) {
          park(col1);
          factor(0, col0, X);
          inverse(col0, X);
          const float2* parked = col1;
          const int sj = fresh(ix.sj);
#pragma unroll
          for (int r = 0; r < R; r++, parked += sj) X[r] = *parked;
          factor(1, col1, X);
          inverse(col1, X);
        } else if (MODE == PM_FWD) {
          factor(0, col0, X);
          if (live) {
            float2* dst = A.out0 + (i64)vol * A.out_vs + base;
#pragma unroll
            for (int r = 0; r < R; r++, dst += step) *dst = X[r];
          }
        } else {
          factor(0, col0, X);
          inverse(col0, X);
        }
      });
    }
    __syncthreads();

    if (MODE != PM_FWD && has1 && b1 < nl) {
      // an item of this stage reads the table entries that the same thread writes in the next
      // tile's first stage, so no barrier separates the two
      int u, v;
      const i64 base = line(b1, u, v) + (i64)j1 * sa;
      const i64 step = fresh((i64)R2 * sa);
      const int sk = fresh(ix.sk);
      rt_switch1(R1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
#pragma unroll
        for (int q = 0; q < (MODE == PM_DUAL_OUT ? 2 : 1); q++) {
          const float2* src = (q == 0 ? reg0 : reg1) + ix.at(b1, j1, 0);
          float2 x[R];
#pragma unroll
          for (int r = 0; r < R; r++, src += sk) x[r] = *src;
          RDft<R, true>::run(x);
          float2* dst = (q == 0 ? A.out0 : A.out1) + (i64)vol * A.out_vs + base;
          if (q == 0 && A.accum) {
#pragma unroll
            for (int r = 0; r < R; r++, dst += step) *dst = cadd(x[r], *dst);
          } else {
#pragma unroll
            for (int r = 0; r < R; r++, dst += step) *dst = x[r];
          }
        }
      });
    }
  }
}

template <int MODE, bool LARGE>
static int launch_rt_t(PassArgs& A, const RtPlan& P, cudaStream_t stream) {
  constexpr int B = LARGE ? 8 : 16;
  constexpr bool kDual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  const bool bfast = (A.st[A.av] == 1);
  const size_t region = (size_t)B * (bfast ? P.r2 * P.s1 : ((P.r2 * P.s1) | 1));
  const size_t smem = sizeof(float2) * (P.n + (kDual ? 2 : 1) * region);
  const int threads = (B * P.rmax() + 31) & ~31;
  auto kern = rt_pass_kernel<MODE, LARGE>;
  const int rc = check_cuda(allow_smem(kern, smem), "run-time pass smem");
  if (rc != ME_OK) return rc;
  A.div_tiles.set((A.nlines + B - 1) / B);
  // resident CTAs on the device for this length and layout (a property of the kernel)
  static std::atomic<int> occ[8][2][ME_MAX_LINE + 1];
  int dev = 0;
  cudaGetDevice(&dev);
  int res = (dev < 8) ? occ[dev][bfast][P.n].load(std::memory_order_relaxed) : 0;
  if (res == 0) {
    int nb = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, threads, smem);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    res = std::max(1, nb) * std::max(1, sms);
    if (dev < 8) occ[dev][bfast][P.n].store(res, std::memory_order_relaxed);
  }
  const long long tiles = (long long)((A.nlines + B - 1) / B) * A.nvol;
  count_launch();
  return check_cuda(launch_chained(tiles <= res, kern, (int)std::min<long long>(tiles, res), threads,
                                   smem, stream, A, P),
                    "run-time pass launch");
}

template <int MODE>
int launch_rt_mode(PassArgs& A, const RtPlan& P, cudaStream_t stream) {
  return P.large() ? launch_rt_t<MODE, true>(A, P, stream)
                   : launch_rt_t<MODE, false>(A, P, stream);
}

}  // namespace me
