// SENSE operators on the sampled k-space of each shot (image_estimation.py:89-129,
// transform_estimation.py:39-68, joint_recon.py:108-115).
//
// Every mask is constant along z, so F^H M_s F = F_xy^H M_s F_xy: nothing is transformed along
// z per iteration, and the data are kept in hybrid space (orthonormal IFFT_z of k-space, done
// once at set-up).  For one readout plane z the forward model of coil c is
//     K_s[j] = (1/sqrt(XY)) sum_x exp(-2 pi i kx_j x / X) FFT_y(mps_c . u)[x, ky_j]
// i.e. a full FFT along y of every x row followed by a sparse DFT along x evaluated only at the
// shot's samples (a few hundred points instead of the X*Y plane).  The adjoint scatters the
// samples back along x for each ky, inverse-FFTs along y, multiplies by conj(mps_c) and sums
// over coils.
//
//   sense_fwd_kernel  CTA = (plane z, coil c, shot): streams the plane's x rows through shared
//                     memory, FFT_y, accumulates its samples in registers; epilogue writes K,
//                     or the residual energy, or the 28 Gauss-Newton statistics (LM).
//   sense_adj_kernel  CTA = (plane z, x-block, shot): loops over coils, builds the H rows from
//                     K, IFFT_y, accumulates conj(mps) . h in registers, writes one image block.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "fft_reg.cuh"
#include "line_pass.cuh"
#include "rigid.cuh"
#include "sense.cuh"

namespace me {

#define ME_TRY(x)                 \
  do {                            \
    int _rc = (x);                \
    if (_rc != ME_OK) return _rc; \
  } while (0)

// Resident CTAs per SM that the compile-time forward is built for.  Lines of eight threads leave room
// for three unless a thread holds eight samples, whose accumulators and indices then spill (24 to
// 112 points, 32 planes, 8 coils, 8 shots of 1,500 samples, 80 and 128 registers: 143 and 130 us at
// 24, 165 and 150 at 56, 227 and 196 at 112; 128 points 202 and 206).  Four samples a thread hold
// three (1,000 samples at 56 and 112 points, three and two CTAs: 111 and 119 us, 156 and 158).
__host__ __device__ constexpr int sense_min_ctas(int y, int mpt) {
  return line_threads(y) == 8 && mpt <= 4 ? 3 : 2;
}

// Gauss-Newton sums of one sample: |r|^2, Re(conj(r) J_p) and Re(conj(J_p) J_q) for q >= p.
__device__ __forceinline__ void lm_accumulate(double (&st)[kLmStats], float2 r, const float2 (&J)[6]) {
  st[0] += (double)r.x * r.x + (double)r.y * r.y;
#pragma unroll
  for (int p = 0; p < 6; p++) st[1 + p] += (double)r.x * J[p].x + (double)r.y * J[p].y;
  int k = 7;
#pragma unroll
  for (int p = 0; p < 6; p++)
#pragma unroll
    for (int q = p; q < 6; q++) {
      st[k] += (double)J[p].x * J[q].x + (double)J[p].y * J[q].y;
      k++;
    }
}

template <int MPT, int V, int MODE>
__global__ void __launch_bounds__(kThreads) sense_fwd_kernel(const FwdArgs A) {
  extern __shared__ float2 sm[];
  const int z = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
  const int s = A.shot0 + b;
  const int X = A.X, Y = A.Y;
  float2* twY = sm;
  float2* twX = twY + pad2(Y);
  float2* buf0 = twX + pad2(X);
  float2* buf1 = buf0 + (i64)Y * A.es;
  const int L = V * A.XR;

  init_twiddles(twY, Y);
  init_twiddles(twX, X);

  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  int mkx[MPT], mky[MPT];
  float2 acc[V][MPT];
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    const int j = threadIdx.x + m * kThreads;
    mkx[m] = -1;
    mky[m] = 0;
    if (j < ns) {
      mkx[m] = A.kx[soff + j];
      mky[m] = A.ky[soff + j];
    }
#pragma unroll
    for (int v = 0; v < V; v++) acc[v][m] = make_float2(0.f, 0.f);
  }

  const i64 plane = (i64)X * Y;
  const float2* mrow = A.mps + ((i64)z * A.C + c) * plane;
  const float2* vbase = A.vols + (i64)b * V * A.vol_stride + (i64)z * plane;

  for (int x0 = 0; x0 < X; x0 += A.XR) {
    const int nr = min(A.XR, X - x0);
    __syncthreads();
    for (int t = threadIdx.x; t < A.XR * Y; t += kThreads) {
      const int xr = t / Y, y = t - xr * Y;
      if (xr < nr) {
        const float2 m = mrow[(i64)(x0 + xr) * Y + y];
#pragma unroll
        for (int v = 0; v < V; v++) {
          const float2 u = vbase[(i64)v * A.vol_stride + (i64)(x0 + xr) * Y + y];
          buf0[y * A.es + v * A.XR + xr] = cmul(m, u);
        }
      } else {
#pragma unroll
        for (int v = 0; v < V; v++) buf0[y * A.es + v * A.XR + xr] = make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
    const float2* G = fft_lines<false>(buf0, buf1, A.plan, L, A.es, twY);
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      if (mkx[m] < 0) continue;
      int idx = (int)(((long long)mkx[m] * x0) % X);
      const float2* grow = G + mky[m] * A.es;
      for (int xr = 0; xr < nr; xr++) {
        const float2 w = twX[idx];
#pragma unroll
        for (int v = 0; v < V; v++) acc[v][m] = cadd(acc[v][m], cmul(grow[v * A.XR + xr], w));
        idx += mkx[m];
        if (idx >= X) idx -= X;
      }
    }
  }

  const i64 zc = (i64)z * A.C + c;
  if constexpr (MODE == FWD_K) {
    const i64 rel = A.kout_abs ? (i64)soff : (i64)(soff - A.shot_off[A.shot0]);
    const i64 base = rel * A.C * A.Z + zc * ns;
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      const int j = threadIdx.x + m * kThreads;
      if (j < ns) A.kout[base + j] = cscale(acc[0][m], A.scale);
    }
  } else if constexpr (MODE == FWD_RESID) {
    const i64 base = (i64)soff * A.C * A.Z + zc * ns;
    double e[1] = {0.0};
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      const int j = threadIdx.x + m * kThreads;
      if (j < ns) {
        const float2 r = csub(cscale(acc[0][m], A.scale), A.ydat[base + j]);
        e[0] += (double)r.x * r.x + (double)r.y * r.y;
      }
    }
    block_reduce_store<1>(e, A.partial + ((i64)b * A.Z * A.C + zc));
  } else {
    const i64 base = (i64)soff * A.C * A.Z + zc * ns;
    double st[kLmStats];
#pragma unroll
    for (int k = 0; k < kLmStats; k++) st[k] = 0.0;
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      const int j = threadIdx.x + m * kThreads;
      if (j >= ns) continue;
      const float2 r = csub(cscale(acc[0][m], A.scale), A.ydat[base + j]);
      float2 J[6];
#pragma unroll
      for (int p = 0; p < 6; p++) J[p] = cscale(acc[(p + 1) % V][m], A.scale);
      lm_accumulate(st, r, J);
    }
    block_reduce_store<kLmStats>(st, A.partial + ((i64)b * A.Z * A.C + zc) * kLmStats);
  }
}

template <int EPT>
__global__ void __launch_bounds__(kThreads) sense_adj_kernel(const AdjArgs A) {
  extern __shared__ float2 sm[];
  const int z = blockIdx.x, x0 = blockIdx.y * A.XB, b = blockIdx.z;
  const int s = A.shot0 + b;
  const int X = A.X, Y = A.Y;
  const int nr = min(A.XB, X - x0);
  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  float2* twY = sm;
  float2* twX = twY + pad2(Y);
  float2* Ks = twX + pad2(X);
  float2* buf0 = Ks + pad2(ns);
  float2* buf1 = buf0 + (i64)Y * A.es;
  init_twiddles(twY, Y);
  init_twiddles(twX, X);

  const int* kyo = A.ky_off + (i64)s * (Y + 1);
  const int* kxs = A.kx + soff;
  const i64 kbase0 = (A.kin_rel ? (i64)(soff - A.shot_off[A.shot0]) : (i64)soff) * A.C * A.Z;
  const i64 plane = (i64)X * Y;

  float2 w[EPT];
#pragma unroll
  for (int m = 0; m < EPT; m++) w[m] = make_float2(0.f, 0.f);

  for (int c = 0; c < A.C; c++) {
    __syncthreads();
    const float2* kc = A.kin + kbase0 + ((i64)z * A.C + c) * ns;
    for (int j = threadIdx.x; j < ns; j += kThreads) Ks[j] = kc[j];
    __syncthreads();
    for (int t = threadIdx.x; t < A.XB * Y; t += kThreads) {
      const int xr = t % A.XB, ky = t / A.XB;
      float2 acc = make_float2(0.f, 0.f);
      if (xr < nr) {
        const int x = x0 + xr;
        for (int j = kyo[ky]; j < kyo[ky + 1]; j++) {
          const int idx = (kxs[j] * x) % X;
          acc = cadd(acc, cmulc(Ks[j], twX[idx]));
        }
      }
      buf0[ky * A.es + xr] = acc;
    }
    __syncthreads();
    const float2* R = fft_lines<true>(buf0, buf1, A.plan, A.XB, A.es, twY);
    const float2* mrow = A.mps + ((i64)z * A.C + c) * plane + (i64)x0 * Y;
#pragma unroll
    for (int m = 0; m < EPT; m++) {
      const int e = threadIdx.x + m * kThreads;
      if (e < nr * Y) {
        const int xr = e / Y, y = e - xr * Y;
        w[m] = cadd(w[m], cmulc(R[y * A.es + xr], mrow[e]));
      }
    }
  }
  float2* o = A.out + (i64)b * A.vol_stride + (i64)z * plane + (i64)x0 * Y;
#pragma unroll
  for (int m = 0; m < EPT; m++) {
    const int e = threadIdx.x + m * kThreads;
    if (e < nr * Y) o[e] = cscale(w[m], A.scale);
  }
}

// ---------------------------------------------------------------- compile-time plane widths
// Fast variants of the two kernels above for line lengths Y with a register FFT plan
// (fft_reg.cuh).  Same arguments, layouts and results.

__device__ __forceinline__ void init_twiddles_any(float2* tw, int n) {
  const float2* g = nullptr;
  switch (n) {
#define ME_TW_CASE(N) \
  case N: g = tw##N; break;
    ME_FAST_LENGTHS(ME_TW_CASE)
#undef ME_TW_CASE
    default: break;
  }
  if (g) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) tw[k] = __ldg(g + k);
  } else {
    init_twiddles(tw, n);
  }
}

// Map and image rows go from L2 straight into the registers of the DFT that uses them (16 or 14
// loads in flight per thread); staging them in shared memory first, by bulk copies, cost more in
// shared-memory traffic than it hid: without it, and with the plans of LineFft, the forward went
// from 55.8 to 53.5 ms and the adjoint from 63.6 to 60.8 ms at 256x224x176, 32 coils, 64 shots,
// and from 2.50 to 1.68 and 3.47 to 2.10 ms at 128x112x88, 16 coils, 32 shots (three CTAs per SM
// instead of two for the forward up to 128 points and four samples a thread).  What bounds both: instruction issue and the
// shared-memory pipe together (transposes, columns of the sample sums, H rows).

// This thread's row group g and its place j < G in it: sixteen threads of one row to a half warp,
// or eight of two.  (With half warps of two rows of 224 points the forward took 62.1 ms instead
// of 56.8 ms.)
template <int G>
__device__ __forceinline__ void row_place(int& g, int& j) {
  g = threadIdx.x / G;
  j = threadIdx.x % G;
}

// Rows per chunk of the forward kernel (one row per thread group) and its shared-memory plan.
template <int Y>
struct FwdPlan {
  using F = LineFft<Y>;
  static constexpr int G = F::G;
  static constexpr int NG = kThreads / G;
  static constexpr int RC = NG;
  static constexpr int LS = line_region(Y);
  static constexpr int LINES = NG * LS;
};

// sum_row L[row] W^(kx row) over a chunk's RC rows of one spectrum column (rows LS apart) by
// Horner's rule in interleaved chains of eight rows: two stepping by W^2kx, or four by W^4kx where
// a chunk has 32 rows.  A chain carries the rounding of its step up to its length.  At 128 points, 128
// rows, against 64 bits: two chains of sixteen 2.53e-7, four of eight 1.77e-7 (two chains over
// chunks of 16 rows: 1.72e-7); 32 planes, 8 coils, 8 shots of 400 samples 101.9 and 102.8 us, of 1,000
// samples 147.9 and 155.2 us.  (Two sums of 16 rows a chunk, each with a table twiddle of its own:
// 1.72e-7, 106.6 and 159.5 us.)
constexpr int fwd_chains(int rc) { return rc >= 32 ? 4 : 2; }
template <int RC, int LS>
__device__ __forceinline__ float2 sample_sum(const float2* Lk, float2 st, float2 st2, float2 st4) {
  constexpr int NC = fwd_chains(RC);
  static_assert(RC % NC == 0, "the chains take rows in turn");
  const float2 step = NC == 4 ? st4 : st2;
  float2 h[NC];
#pragma unroll
  for (int q = 0; q < NC; q++) h[q] = Lk[(RC - NC + q) * LS];
#pragma unroll
  for (int i = RC - 2 * NC; i >= 0; i -= NC) {
#pragma unroll
    for (int q = 0; q < NC; q++) h[q] = cfma(h[q], step, Lk[(i + q) * LS]);
  }
  const float2 lo = cfma(h[1], st, h[0]);
  if (NC == 2) return lo;
  return cfma(cfma(h[NC - 1], st, h[NC - 2]), st2, lo);
}

// The steps W^kx, W^2kx and W^4kx of a sample (the last one where there are four chains).
struct SampleSteps {
  float2 st, st2, st4;
  template <int RC>
  __device__ __forceinline__ void set(const float2* twX, int kx, int X) {
    int k = 2 * kx;
    if (k >= X) k -= X;
    st = twX[kx];
    st2 = twX[k];
    k *= 2;
    if (k >= X) k -= X;
    st4 = fwd_chains(RC) == 4 ? twX[k] : st2;
  }
};

template <int Y, int MPT, int MODE>
__global__ void __launch_bounds__(kThreads, sense_min_ctas(Y, MPT)) fast_fwd_kernel(const FwdArgs A) {
  static_assert(MODE == FWD_K || MODE == FWD_RESID, "one volume per CTA");
  using P = FwdPlan<Y>;
  using F = typename P::F;
  constexpr int G = P::G, RC = P::RC, LS = P::LS;
  extern __shared__ __align__(16) float2 sm[];
  // shots vary fastest, so the CTAs of all shots of one (z, coil) run together and share the
  // map plane (and each shot's image plane across coils) through L2
  const int bx = blockIdx.x, c = blockIdx.y, z = blockIdx.z;
  const int b = bx / A.vps, vk = bx - b * A.vps;  // shot in the batch, volume of the shot
  const int s = A.shot0 + b;
  const int X = A.X;
  float2* lines = sm;  // one line region per thread group
  float2* twX = lines + P::LINES;
  init_twiddles_any(twX, X);
  chain_next();
  chain_wait();

  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  // per sample: kx, ky, the twiddle index kx x0 mod X of the current chunk and its step kx RC
  int mkx[MPT], mky[MPT], idx[MPT], dix[MPT];
  float2 acc[MPT];
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    const int jj = threadIdx.x + m * kThreads;
    mkx[m] = -1;
    mky[m] = 0;
    idx[m] = 0;
    dix[m] = 0;
    if (jj < ns) {
      mkx[m] = A.kx[soff + jj];
      mky[m] = A.ky[soff + jj];
      dix[m] = mulmod(mkx[m], RC % X, X, 1.0f / (float)X);
    }
    acc[m] = make_float2(0.f, 0.f);
  }
  int g, j;
  row_place<G>(g, j);
  const i64 plane = (i64)X * Y;
  const float2* mrow = A.mps + ((i64)z * A.C + c) * plane;
  const float2* vbase = A.vols + (i64)bx * A.vol_stride + (i64)z * plane;
  PaddedSlots<Y> slots;
  slots.init(lines + g * LS, j);

  // The Horner steps do not change between chunks: with few samples per thread they stay in
  // registers, else in shared memory in sample order, where a warp's reads are free of the bank
  // conflicts of reading them out of twX in every chunk (128 rows, 32 planes, 8 coils, 8 shots of
  // 1,000 samples: 56 points 111 -> 103 us, 112 155 -> 150, 224 233 -> 223; of 1,500: 150 -> 140,
  // 196 -> 189, 298 -> 278).
  constexpr bool kHoist = MPT <= 2;
  SampleSteps hst[kHoist ? MPT : 1];
  float2* steps = twX + pad2(X);  // [3][MPT * kThreads]
  __syncthreads();  // twX is written above by all threads
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    SampleSteps t;
    t.set<RC>(twX, mkx[m] < 0 ? 0 : mkx[m], X);
    if (kHoist) {
      hst[m] = t;
    } else if (mkx[m] >= 0) {
      float2* p = steps + threadIdx.x + m * kThreads;
      p[0] = t.st;
      p[MPT * kThreads] = t.st2;
      if (fwd_chains(RC) == 4) p[2 * MPT * kThreads] = t.st4;
    }
  }
  for (int x0 = 0; x0 < X; x0 += RC) {
    const int nr = min(RC, X - x0);
    if (x0 > 0) __syncthreads();
    {
      // FFT of map row x image row, read and multiplied as the first stage needs them; rows past
      // nr transform zeros
      const float2* ms = mrow + (i64)(x0 + g) * Y;
      const float2* us = vbase + (i64)(x0 + g) * Y;
      const bool live = g < nr;
      F::forward(slots, j, [&](int, int n) {
        return live ? cmul(ms[n], us[n]) : make_float2(0.f, 0.f);
      });
    }
    __syncthreads();
    // Sample sums over the chunk's rows, then one table twiddle W^(kx x0) per chunk.  Rows past nr
    // hold zeros (zero lines transform to zero), so every chunk runs all RC rows.
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      if (mkx[m] < 0) continue;
      SampleSteps t;
      if (kHoist) {
        t = hst[m];
      } else {
        const float2* p = steps + threadIdx.x + m * kThreads;
        t.st = p[0];
        t.st2 = p[MPT * kThreads];
        t.st4 = fwd_chains(RC) == 4 ? p[2 * MPT * kThreads] : t.st2;
      }
      acc[m] = cfma(sample_sum<RC, LS>(lines + mky[m], t.st, t.st2, t.st4), twX[idx[m]], acc[m]);
      idx[m] += dix[m];
      if (idx[m] >= X) idx[m] -= X;
    }
  }

  const i64 zc = (i64)z * A.C + c;
  if constexpr (MODE == FWD_K) {
    const i64 rel = A.kout_abs ? (i64)soff : (i64)(soff - A.shot_off[A.shot0]);
    const i64 base = rel * A.C * A.Z + zc * ns;
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      const int jj = threadIdx.x + m * kThreads;
      if (jj < ns) A.kout[(i64)vk * A.kout_vs + base + jj] = cscale2(acc[m], A.scale, A.scale_lo);
    }
  } else {
    const i64 base = (i64)soff * A.C * A.Z + zc * ns;
    double e[1] = {0.0};
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      const int jj = threadIdx.x + m * kThreads;
      if (jj < ns) {
        const float2 r = csub(cscale2(acc[m], A.scale, A.scale_lo), A.ydat[base + jj]);
        e[0] += (double)r.x * r.x + (double)r.y * r.y;
      }
    }
    block_reduce_store<1>(e, A.partial + ((i64)b * A.Z * A.C + zc));
  }
}

// Gauss-Newton statistics of the LM step straight from the seven volumes of each shot (T x and
// its six partials, [shot][7] in A.vols): the forward model of all seven runs in one CTA per
// (shot, coil, plane), each chunk's map rows read seven times in turn (from L1), and the sampled
// values J_v = M_s F C U_v are contracted in registers into e0 = |J_0 - y|^2, g_p = Re<J_0 - y,
// J_p> and H_pq = Re<J_p, J_q> (transform_estimation.py:39-68) instead of being written out.
// The sums per sample and their block reduction are those of lm_stats_kernel, in the same order,
// so the statistics are bit-identical to the two-kernel path.
template <int Y, int MPT>
__global__ void __launch_bounds__(kThreads, 2) fast_lm_kernel(const FwdArgs A) {
  using P = FwdPlan<Y>;
  using F = typename P::F;
  constexpr int G = P::G, RC = P::RC, LS = P::LS;
  constexpr int NV = 7;
  extern __shared__ __align__(16) float2 sm[];
  const int b = blockIdx.x, c = blockIdx.y, z = blockIdx.z;
  const int s = A.shot0 + b;
  const int X = A.X;
  float2* lines = sm;  // one line region per thread group
  float2* twX = lines + P::LINES;
  init_twiddles_any(twX, X);

  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  int mkx[MPT], mky[MPT], idx[MPT], dix[MPT];
  float2 acc[NV][MPT];
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    const int jj = threadIdx.x + m * kThreads;
    mkx[m] = -1;
    mky[m] = 0;
    idx[m] = 0;
    dix[m] = 0;
    if (jj < ns) {
      mkx[m] = A.kx[soff + jj];
      mky[m] = A.ky[soff + jj];
      dix[m] = mulmod(mkx[m], RC % X, X, 1.0f / (float)X);
    }
#pragma unroll
    for (int v = 0; v < NV; v++) acc[v][m] = make_float2(0.f, 0.f);
  }
  int g, j;
  row_place<G>(g, j);
  const i64 plane = (i64)X * Y;
  const float2* mrow = A.mps + ((i64)z * A.C + c) * plane;
  const float2* vbase = A.vols + (i64)b * NV * A.vol_stride + (i64)z * plane;
  PaddedSlots<Y> slots;
  slots.init(lines + g * LS, j);

  constexpr bool kHoist = MPT <= 2;
  SampleSteps hst[kHoist ? MPT : 1];
  __syncthreads();  // twX is written above by all threads
  if constexpr (kHoist) {
#pragma unroll
    for (int m = 0; m < MPT; m++) hst[m].set<RC>(twX, mkx[m] < 0 ? 0 : mkx[m], X);
  }
  for (int x0 = 0; x0 < X; x0 += RC) {
    const int nr = min(RC, X - x0);
#pragma unroll 1
    for (int v = 0; v < NV; v++) {
      __syncthreads();
      {
        const float2* ms = mrow + (i64)(x0 + g) * Y;
        const float2* us = vbase + (i64)v * A.vol_stride + (i64)(x0 + g) * Y;
        const bool live = g < nr;
        F::forward(slots, j, [&](int, int n) {
          return live ? cmul(ms[n], us[n]) : make_float2(0.f, 0.f);
        });
      }
      __syncthreads();
      // sample sums of volume v over the chunk's rows (as fast_fwd_kernel)
#pragma unroll
      for (int m = 0; m < MPT; m++) {
        if (mkx[m] < 0) continue;
        SampleSteps t;
        if (kHoist) t = hst[m];
        else t.set<RC>(twX, mkx[m], X);
        const float2 sum = sample_sum<RC, LS>(lines + mky[m], t.st, t.st2, t.st4);
        // the accumulators rotate as a queue, so that volume v's is always acc[0] (v is not a
        // compile-time index); after the seven volumes of a chunk acc[u] is volume u's again
        const float2 nv = cfma(sum, twX[idx[m]], acc[0][m]);
#pragma unroll
        for (int u = 0; u < NV - 1; u++) acc[u][m] = acc[u + 1][m];
        acc[NV - 1][m] = nv;
      }
    }
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      if (mkx[m] < 0) continue;
      idx[m] += dix[m];
      if (idx[m] >= X) idx[m] -= X;
    }
  }

  const i64 zc = (i64)z * A.C + c;
  const i64 yb = (i64)soff * A.C * A.Z + zc * ns;
  double st[kLmStats];
#pragma unroll
  for (int k = 0; k < kLmStats; k++) st[k] = 0.0;
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    const int jj = threadIdx.x + m * kThreads;
    if (jj < ns) {
      // K rounded to float before the difference, as the two-kernel path stores it
      const float2 k0 = cscale2(acc[0][m], A.scale, A.scale_lo);
      const float2 r = csub(k0, A.ydat[yb + jj]);
      float2 J[6];
#pragma unroll
      for (int p = 0; p < 6; p++) J[p] = cscale2(acc[1 + p][m], A.scale, A.scale_lo);
      lm_accumulate(st, r, J);
    }
  }
  block_reduce_store<kLmStats>(st, A.partial + ((i64)b * A.Z * A.C + zc) * kLmStats);
}

// Adjoint plan: one image row per thread group; the H rows are built by one thread per ky bin
// (and part of the rows), walking its samples with a twiddle recurrence along x.
template <int Y>
struct AdjPlan {
  using F = LineFft<Y>;
  static constexpr int G = F::G;
  static constexpr int NG = kThreads / G;
  static constexpr int LS = line_region(Y);
  static constexpr int NP0 = (kThreads / Y) < 1 ? 1 : (kThreads / Y);
  static constexpr int NPARTS = NP0 >= 16 ? 16 : NP0 >= 8 ? 8 : NP0 >= 4 ? 4 : NP0 >= 2 ? 2 : 1;
  static constexpr int RP = NG / NPARTS;  // rows per H-building thread
  // When one thread per bin leaves threads idle (Y < 256, all rows per thread), each idle
  // thread takes the second half of the rows of one of the heaviest bins (bins come sorted by
  // sample count), halving the longest walk; both halves write their own rows.
  static constexpr int NSPLIT = (NPARTS == 1 && Y < kThreads) ? (kThreads - Y < Y ? kThreads - Y : Y) : 0;
  static constexpr int RH = RP > 1 ? RP / 2 : 1;  // rows of each half of a shared bin
  // middle rows of the threads' row ranges (whole ranges, or the whole and the two halves of a
  // shared bin); their sample twiddles are tabulated as factors when they are few
  static constexpr int STARTS = NSPLIT > 0 ? 3 : NPARTS;
  static constexpr bool TABULATE = STARTS <= 3;
  // W^3kx is tabulated too (h_rows) where threads walk all their rows in step
  static constexpr bool CUBE = TABULATE && NSPLIT == 0 && RP >= 8;
  // With that table in the place of the second sample buffer, the next coil's samples arrive under
  // the FFT alone.
  static constexpr int NK = CUBE ? 1 : 2;
  static constexpr int TABLES = 1 + STARTS + (CUBE ? 1 : 0);
  static __host__ __device__ constexpr int start_row(int q) {
    return NSPLIT > 0 ? (q == 0 ? RH : q == 1 ? RH / 2 : RH + RH / 2) : q * RP + RP / 2;
  }
};

template <int Y>
__global__ void __launch_bounds__(kThreads, Y <= 64 ? 3 : 2) fast_adj_kernel(const AdjArgs A) {
  using P = AdjPlan<Y>;
  using F = typename P::F;
  constexpr int G = P::G, NG = P::NG, LS = P::LS, RP = P::RP, NSPLIT = P::NSPLIT;
  extern __shared__ __align__(16) float2 sm[];
  chain_next();
  chain_wait();
  // shots vary fastest: the CTAs of all shots of one (z, row block) share the map rows in L2
  const int b = blockIdx.x, x0 = blockIdx.y * NG, z = blockIdx.z;
  const int s = A.shot0 + b;
  const int X = A.X;
  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  const int kcap = (A.XB + 1) & ~1;   // max samples per shot, padded
  float2* Kb = sm;                    // NK x kcap samples
  float2* lines = Kb + P::NK * kcap;  // NG x LS
  float2* twX = lines + NG * LS;
  // per sample, shared by all coils: conj W^kx and, at the middle row of each of the P::STARTS row
  // ranges that threads build, conj W^(kx x) -- as factors (and conj W^3kx where P::CUBE), or
  // (short lines, many ranges) as indices into twX
  float2* tw_s = twX + pad2(X);
  float2* tw_0 = tw_s + kcap;
  float2* tw_3 = tw_0 + P::STARTS * kcap;
  unsigned short* ix_s = reinterpret_cast<unsigned short*>(tw_s);
  unsigned short* ix_0 = ix_s + kcap;
  init_twiddles_any(twX, X);

  int g, j;
  row_place<G>(g, j);
  const int x = x0 + g;
  const bool live = x < X;
  const float inv_x = 1.0f / (float)X;
  const int* kyo = A.ky_off + (i64)s * (Y + 1);
  const i64 kbase0 = (A.kin_rel ? (i64)(soff - A.shot_off[A.shot0]) : (i64)soff) * A.C * A.Z;
  const i64 plane = (i64)X * Y;
  __syncthreads();
  for (int i = threadIdx.x; i < ns; i += kThreads) {
    const int kx = A.kx[soff + i];
    if (P::TABULATE) tw_s[i] = cconj(twX[kx]);
    else ix_s[i] = (unsigned short)kx;
    if (P::CUBE) tw_3[i] = cconj(twX[3 * kx % X]);
    for (int q = 0; q < P::STARTS; q++) {
      const int xi = mulmod(kx, (x0 + P::start_row(q)) % X, X, inv_x);
      if (P::TABULATE) tw_0[q * kcap + i] = cconj(twX[xi]);
      else ix_0[q * kcap + i] = (unsigned short)xi;
    }
  }

  // H-building role: bin hb, rows [hr0, hr0 + RP), or [hr0, hr0 + RH) for a shared bin
  const bool split = (NSPLIT > 0) && (A.ky_order != nullptr);
  int hb = 0, hr0 = 0;
  bool hbuild = false, half = false;
  if ((int)threadIdx.x < Y * P::NPARTS) {
    const int slot = threadIdx.x % Y;
    hb = A.ky_order ? A.ky_order[(i64)s * Y + slot] : slot;
    hr0 = (threadIdx.x / Y) * RP;
    hbuild = true;
    half = split && slot < NSPLIT;
  } else if (split && (int)threadIdx.x - Y < NSPLIT) {
    hb = A.ky_order[(i64)s * Y + (threadIdx.x - Y)];
    hr0 = P::RH;
    hbuild = true;
    half = true;
  }
  const int hlo = hbuild ? kyo[hb] : 0, hhi = hbuild ? kyo[hb + 1] : 0;
  const int start = kcap * (NSPLIT == 0 ? hr0 / RP : half ? 1 + hr0 / P::RH : 0);

  // coil c's samples into buffer c mod NK
  auto issue = [&](int c) {
    const float2* kc = A.kin + kbase0 + ((i64)z * A.C + c) * ns;
    float2* kd = Kb + (c % P::NK) * kcap;
    for (int i = threadIdx.x; i < ns; i += kThreads) cp_async8(kd + i, kc + i);
    cp_async_commit();
  };

  // image row accumulators in the inverse FFT's output layout: thread j owns y = j + G q
  float2 w[F::R1];
#pragma unroll
  for (int m = 0; m < F::R1; m++) w[m] = make_float2(0.f, 0.f);
  PaddedSlots<Y> slots;
  slots.init(lines + g * LS, j);

  issue(0);
  for (int c = 0; c < A.C; c++) {
    cp_async_wait_all();
    __syncthreads();
    if (P::NK == 2 && c + 1 < A.C) issue(c + 1);
    const float2* K = Kb + (c % P::NK) * kcap;
    const float2* ms = A.mps + ((i64)z * A.C + c) * plane + (i64)x * Y + j;
    if (hbuild) {
      // H[x][ky] += K exp(+2 pi i kx x / X)
      auto walk = [&](auto rows) {
        h_rows<decltype(rows)::value, P::CUBE>(
            hlo, hhi,
            [&](int i, float2& v, float2& st, float2& st3) {
              st = P::TABULATE ? tw_s[i] : cconj(twX[ix_s[i]]);
              if (P::CUBE) st3 = tw_3[i];
              v = cmul(K[i], P::TABULATE ? tw_0[start + i] : cconj(twX[ix_0[start + i]]));
            },
            [&](int r, float2 h) { lines[(hr0 + r) * LS + hb] = h; });
      };
      if constexpr (NSPLIT > 0) {
        if (half) walk(std::integral_constant<int, P::RH>{});
        else walk(std::integral_constant<int, RP>{});
      } else {
        walk(std::integral_constant<int, RP>{});
      }
    }
    __syncthreads();
    if (P::NK == 1 && c + 1 < A.C) issue(c + 1);
    // Added to the sum over the coils as one term, the product rounds it once; fused into it, twice
    // (128 points, 32 coils: 1.6e-7 from 64 bits and, fused, 2.1e-7).  144 to 224 points keep the
    // fused form: the other one spills at 192 and 224 (1.5 to 5% there).
    F::inverse(slots, j, [&](int q, int, float2 v) {
      if (!live) return;
      const float2 m = __ldg(ms + q * G);
      w[q] = NSPLIT == 0 ? cadd(w[q], cmulc(v, m)) : cfmac(v, m, w[q]);
    });
  }
  if (live) {
    float2* o = A.out + (i64)b * A.vol_stride + (i64)z * plane + (i64)x * Y + j;
#pragma unroll
    for (int q = 0; q < F::R1; q++) o[q * G] = cscale2(w[q], A.scale, A.scale_lo);
  }
}

// Gauss-Newton sums from the sampled T x and its six partials, written by the forward kernel
// into seven K regions kvs apart (offsets relative to the batch's first shot); one CTA per
// (z, coil) plane and shot, FP64 sums reduced in a fixed order.
__global__ void __launch_bounds__(kThreads) lm_stats_kernel(const float2* __restrict__ K, i64 kvs,
                                                            const float2* __restrict__ ydat,
                                                            const int* __restrict__ shot_off,
                                                            int shot0, int ZC,
                                                            double* __restrict__ partial) {
  const i64 zc = blockIdx.x;
  const int b = blockIdx.y;
  const int s = shot0 + b;
  const int soff = shot_off[s], ns = shot_off[s + 1] - soff;
  const i64 kb = (i64)(soff - shot_off[shot0]) * ZC + zc * ns;
  const i64 yb = (i64)soff * ZC + zc * ns;
  double st[kLmStats];
#pragma unroll
  for (int k = 0; k < kLmStats; k++) st[k] = 0.0;
  for (int j = threadIdx.x; j < ns; j += kThreads) {
    const float2 r = csub(K[kb + j], ydat[yb + j]);
    float2 J[6];
#pragma unroll
    for (int p = 0; p < 6; p++) J[p] = K[(p + 1) * kvs + kb + j];
    lm_accumulate(st, r, J);
  }
  block_reduce_store<kLmStats>(st, partial + ((i64)b * ZC + zc) * kLmStats);
}

// Geodesic-acceleration direction volumes.  For each shot b of the batch, with its six partial
// volumes U_b[1 + p] (a Jacobian sweep, shot block of `bs` elements) and its step v_b:
//   first pass  (first = 1): D_b = sum_p v_bp U_b[1 + p]          (ga_mode 1, intended), or
//                            D_b = (1 + v_b5) U_b[6]               (ga_mode 0, as the reference
//                            computes it: its accumulator is overwritten by each partial, so only
//                            the last one, scaled by 1 + v_5, survives)
//   second pass (first = 0): D_b = (D_b - sum_p v_bp U_b[1 + p]) / eps
// D_b lives at U_b[7].
__global__ void ga_combine_kernel(float2* __restrict__ U, i64 bs, i64 vox, int nb,
                                  const double* __restrict__ v, int ga_mode, int first,
                                  double eps) {
  const i64 n = (i64)nb * vox;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const int b = (int)(i / vox);
    const i64 e = i - (i64)b * vox;
    float2* u = U + (i64)b * bs + e;
    const double* vb = v + (i64)b * 6;
    float2 d;
    if (first && ga_mode == 0) {
      d = cscale(u[6 * vox], (float)(1.0 + vb[5]));
    } else {
      d = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 0; p < 6; p++) d = cadd(d, cscale(u[(1 + p) * vox], (float)vb[p]));
      if (!first) d = cscale(csub(u[7 * vox], d), (float)(1.0 / eps));
    }
    u[7 * vox] = d;
  }
}

// rhs partials: -Re<K_D, K_p> for p = 0..5 over one (z, coil) plane of a shot, with the six
// partials' K in regions 0..5 and the direction's in region 6 (kvs apart).
__global__ void __launch_bounds__(kThreads) ga_dots_kernel(const float2* __restrict__ K, i64 kvs,
                                                           const int* __restrict__ shot_off,
                                                           int shot0, int ZC,
                                                           double* __restrict__ partial) {
  const i64 zc = blockIdx.x;
  const int b = blockIdx.y;
  const int s = shot0 + b;
  const int soff = shot_off[s], ns = shot_off[s + 1] - soff;
  const i64 kb = (i64)(soff - shot_off[shot0]) * ZC + zc * ns;
  double st[6];
#pragma unroll
  for (int p = 0; p < 6; p++) st[p] = 0.0;
  for (int j = threadIdx.x; j < ns; j += kThreads) {
    const float2 d = K[6 * kvs + kb + j];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const float2 jp = K[p * kvs + kb + j];
      st[p] -= (double)d.x * jp.x + (double)d.y * jp.y;
    }
  }
  block_reduce_store<6>(st, partial + ((i64)b * ZC + zc) * 6);
}

// Residual in place over one (z, coil) plane of a shot, and its energy partial: r = K - y for
// the gradient-only statistics (me_lm_gradient), r = y - K (YMK) for the CG's initial residual
// (me_sense_residual).  |r|^2 is the same either way.
template <bool YMK>
__global__ void __launch_bounds__(kThreads) resid_inplace_kernel(float2* __restrict__ K,
                                                                 const float2* __restrict__ ydat,
                                                                 const int* __restrict__ shot_off,
                                                                 int shot0, int ZC,
                                                                 double* __restrict__ partial) {
  const i64 zc = blockIdx.x;
  const int b = blockIdx.y;
  const int s = shot0 + b;
  const int soff = shot_off[s], ns = shot_off[s + 1] - soff;
  const i64 kb = (i64)(soff - shot_off[shot0]) * ZC + zc * ns;
  const i64 yb = (i64)soff * ZC + zc * ns;
  double e[1] = {0.0};
  for (int j = threadIdx.x; j < ns; j += kThreads) {
    const float2 r = YMK ? csub(ydat[yb + j], K[kb + j]) : csub(K[kb + j], ydat[yb + j]);
    K[kb + j] = r;
    e[0] += (double)r.x * r.x + (double)r.y * r.y;
  }
  block_reduce_store<1>(e, partial + ((i64)b * ZC + zc));
}

// Re<W_b, U_b[1 + p]> partials, p = 0..5, over a grid-stride share of the volume of shot b
// (W_b = U_b[7], shot block of bs elements).
__global__ void __launch_bounds__(kThreads) grad_dots_kernel(const float2* __restrict__ U, i64 bs,
                                                             i64 vox, double* __restrict__ partial) {
  const int b = blockIdx.y;
  const float2* u = U + (i64)b * bs;
  double st[6];
#pragma unroll
  for (int p = 0; p < 6; p++) st[p] = 0.0;
  for (i64 i = blockIdx.x * (i64)kThreads + threadIdx.x; i < vox; i += (i64)gridDim.x * kThreads) {
    const float2 w = u[7 * vox + i];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const float2 d = u[(1 + p) * vox + i];
      st[p] += (double)w.x * d.x + (double)w.y * d.y;
    }
  }
  block_reduce_store<6>(st, partial + ((i64)b * gridDim.x + blockIdx.x) * 6);
}

// grad[shot0 + b] = {sum of the ZC energy partials, sums of the nblk dot partials}, in order.
__global__ void grad_finish_kernel(const double* __restrict__ epart, int ZC,
                                   const double* __restrict__ dpart, int nblk,
                                   double* __restrict__ grad, int shot0) {
  const int b = blockIdx.x;
  if (threadIdx.x > 6) return;
  double a = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ZC; i++) a += epart[(i64)b * ZC + i];
  } else {
    const int p = threadIdx.x - 1;
    for (int i = 0; i < nblk; i++) a += dpart[((i64)b * nblk + i) * 6 + p];
  }
  grad[(i64)(shot0 + b) * 7 + threadIdx.x] = a;
}

// out[i] = M[i] * ((out[i] if accumulate) + sum_b vols[b][i])
__global__ void sum_volumes_kernel(const float2* __restrict__ vols, i64 vs, int nb,
                                   const unsigned char* __restrict__ M, float2* __restrict__ out,
                                   i64 n, int accumulate) {
  // The running sum starts from out and adds the batch's shots in order, so the sum over all
  // shots is the same sequence of additions whatever the shots-per-launch batch.
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    float2 a = accumulate ? out[i] : make_float2(0.f, 0.f);
    for (int b = 0; b < nb; b++) a = cadd(a, vols[(i64)b * vs + i]);
    if (M && !M[i]) a = make_float2(0.f, 0.f);
    out[i] = a;
  }
}

// stats[shot0 + b][k] = sum over the Z*C partials of batch entry b
__global__ void reduce_partials_kernel(const double* __restrict__ partial, int nparts, int nstat,
                                       double* __restrict__ out, int shot0) {
  const int b = blockIdx.x;
  for (int k = 0; k < nstat; k++) {
    double a = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) a += partial[((i64)b * nparts + i) * nstat + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
      out[(i64)(shot0 + b) * nstat + k] = t;
    }
    __syncthreads();
  }
}

__global__ void precond_kernel(const float2* __restrict__ mps, int C, i64 plane, int Z, float* P,
                               unsigned char* M) {
  const i64 n = plane * Z;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
    const i64 z = i / plane, r = i - z * plane;
    float a = 0.f;
    for (int c = 0; c < C; c++) {
      const float2 m = mps[(z * C + c) * plane + r];
      a += m.x * m.x + m.y * m.y;
    }
    P[i] = 1.0f / (a + 1e-3f);
    M[i] = a > 0.1f ? 1 : 0;
  }
}

// ydat[shot s][z][c][j] = ksp_h[c][kx_j][ky_j][z]
__global__ void gather_kernel(const float2* __restrict__ ksp, int X, int Y, int Z, int C,
                              const int* shot_off, const int* kx, const int* ky, int nshots,
                              float2* __restrict__ ydat) {
  const i64 total = (i64)shot_off[nshots] * C * Z;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < total; i += (i64)gridDim.x * blockDim.x) {
    const int z = (int)(i % Z);
    const i64 rest = i / Z;
    const int c = (int)(rest % C);
    const int g = (int)(rest / C);  // global sample index
    // find the shot of sample g (binary search on shot_off)
    int lo = 0, hi = nshots;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (shot_off[mid] <= g) lo = mid; else hi = mid;
    }
    const int s = lo, ns = shot_off[s + 1] - shot_off[s], j = g - shot_off[s];
    const float2 v = ksp[(((i64)c * X + kx[g]) * Y + ky[g]) * Z + z];
    ydat[(i64)shot_off[s] * C * Z + ((i64)z * C + c) * ns + j] = v;
  }
}

// ksp_h[c][kx][ky][z] += K[s][z][c][j] for the samples of shot s (no duplicates within a shot)
__global__ void scatter_kernel(const float2* __restrict__ K, int X, int Y, int Z, int C,
                               const int* shot_off, const int* kx, const int* ky, int s,
                               float2* __restrict__ ksp) {
  const int soff = shot_off[s], ns = shot_off[s + 1] - soff;
  const i64 total = (i64)ns * C * Z;
  for (i64 i = blockIdx.x * (i64)blockDim.x + threadIdx.x; i < total; i += (i64)gridDim.x * blockDim.x) {
    const int z = (int)(i % Z);
    const i64 rest = i / Z;
    const int c = (int)(rest % C);
    const int j = (int)(rest / C);
    const int g = soff + j;
    const float2 v = K[(i64)soff * C * Z + ((i64)z * C + c) * ns + j];
    float2* d = ksp + (((i64)c * X + kx[g]) * Y + ky[g]) * Z + z;
    *d = cadd(*d, v);
  }
}

// ------------------------------------------------------------------------------ launchers
static int grid_1d(i64 n) {
  i64 b = (n + kThreads - 1) / kThreads;
  return (int)std::min<i64>(b, 148LL * 16);
}

static int check_problem(const me_sense* pb) {
  if (!pb) return fail("problem is NULL");
  if (pb->nx < 1 || pb->ny < 1 || pb->nz < 1 || pb->ncoils < 1 || pb->nshots < 1)
    return fail("problem dims must be positive");
  if (!pb->mps || !pb->samples.shot_off || !pb->samples.kx || !pb->samples.ky ||
      !pb->samples.ky_off || !pb->grid || !pb->transforms)
    return fail("problem has a NULL pointer");
  if (pb->samples.nshots != pb->nshots || pb->samples.nx != pb->nx || pb->samples.ny != pb->ny)
    return fail("samples do not match the problem dims");
  if (pb->grid->nx != pb->nx || pb->grid->ny != pb->ny || pb->grid->nz != pb->nz)
    return fail("grid does not match the problem dims");
  if (pb->samples.max_per_shot > 8 * kThreads)
    return fail("a shot has more than 2048 samples per plane; unsupported");
  if (pb->nx > ME_MAX_LINE || pb->ny > ME_MAX_LINE) return fail("plane too large");
  return ME_OK;
}

static me_layout zxy_layout(const me_sense* pb) {
  me_layout l;
  l.sx = pb->ny;
  l.sy = 1;
  l.sz = (i64)pb->nx * pb->ny;
  return l;
}

static i64 vox_of(const me_sense* pb) { return (i64)pb->nx * pb->ny * pb->nz; }

static bool fast_sense_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ME_GENERIC_FFT");
    v = (e && e[0] == '1') ? 0 : 1;
  }
  return v == 1;
}

// 1/sqrt(XY), with the gain of the FFT along y taken out
static double sense_scale(const me_sense* pb) {
  return 1.0 / sqrt((double)pb->nx * pb->ny * (fast_sense_enabled() ? fft_pair_gain(pb->ny) : 1.0));
}

static int fwd_rows(int V, int Y) {
  int xr = (V == 1) ? 16 : 4;
  while (xr > 1 && 2 * (i64)Y * (V * xr + 1) * 8 > 160 * 1024) xr /= 2;
  return xr;
}

template <int MPT, int V, int MODE>
static int launch_fwd_t(FwdArgs& A, int nb, cudaStream_t st) {
  A.es = V * A.XR + 1;
  const size_t smem = sizeof(float2) * (pad2(A.Y) + pad2(A.X) + 2 * (size_t)A.Y * A.es);
  ME_TRY(check_cuda(allow_smem(sense_fwd_kernel<MPT, V, MODE>, smem), "sense_fwd smem"));
  dim3 grid(A.Z, A.C, nb);
  count_launch();
  sense_fwd_kernel<MPT, V, MODE><<<grid, kThreads, smem, st>>>(A);
  return check_cuda(cudaGetLastError(), "sense_fwd launch");
}

template <int V, int MODE>
static int launch_fwd_v(FwdArgs& A, int maxps, int nb, cudaStream_t st) {
  if (maxps <= kThreads) return launch_fwd_t<1, V, MODE>(A, nb, st);
  if (maxps <= 2 * kThreads) return launch_fwd_t<2, V, MODE>(A, nb, st);
  if (maxps <= 4 * kThreads) return launch_fwd_t<4, V, MODE>(A, nb, st);
  return launch_fwd_t<8, V, MODE>(A, nb, st);
}

// The LM statistics from the fused seven-volume kernel unless ME_LM_TWO_PASS=1 (the forward
// kernel writing seven K regions, then lm_stats_kernel; bit-identical, kept for comparison).
static bool fused_lm_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ME_LM_TWO_PASS");
    v = (e && e[0] == '1') ? 0 : 1;
  }
  return v == 1;
}

template <int Y, int MPT, int MODE>
static int launch_fast_fwd_t(FwdArgs& A, int nb, cudaStream_t st) {
  using P = FwdPlan<Y>;
  const size_t smem = sizeof(float2) * ((size_t)P::LINES + pad2(A.X) +
                                        (MPT > 2 ? fwd_chains(P::RC) == 4 ? 3 : 2 : 0) * MPT * kThreads);
  ME_TRY(check_cuda(allow_smem(fast_fwd_kernel<Y, MPT, MODE>, smem), "fwd smem"));
  dim3 grid(nb * A.vps, A.C, A.Z);
  count_launch();
  return check_cuda(launch_chained(true, fast_fwd_kernel<Y, MPT, MODE>, grid, kThreads, smem, st, A),
                    "fast sense_fwd launch");
}

template <int Y, int MODE>
static int launch_fast_fwd_m(FwdArgs& A, int maxps, int nb, cudaStream_t st) {
  if (maxps <= kThreads) return launch_fast_fwd_t<Y, 1, MODE>(A, nb, st);
  if (maxps <= 2 * kThreads) return launch_fast_fwd_t<Y, 2, MODE>(A, nb, st);
  if (maxps <= 4 * kThreads) return launch_fast_fwd_t<Y, 4, MODE>(A, nb, st);
  return launch_fast_fwd_t<Y, 8, MODE>(A, nb, st);
}

template <int Y, int MPT>
static int launch_fast_lm_t(FwdArgs& A, int nb, cudaStream_t st) {
  using P = FwdPlan<Y>;
  const size_t smem = sizeof(float2) * ((size_t)P::LINES + pad2(A.X));
  ME_TRY(check_cuda(allow_smem(fast_lm_kernel<Y, MPT>, smem), "lm smem"));
  dim3 grid(nb, A.C, A.Z);
  count_launch();
  fast_lm_kernel<Y, MPT><<<grid, kThreads, smem, st>>>(A);
  return check_cuda(cudaGetLastError(), "fast lm launch");
}

// The fused statistics kernel keeps seven accumulators per sample in registers: up to two
// samples per thread (512 per shot).  It serves widths up to 128 points (64x64x48, 8 coils, 16
// shots: 1.64 ms a statistics call against 1.72 in two kernels; 128x128x96, 16 coils, 32 shots:
// 28.3 against 29.1).  Above, the forward kernel, which has the registers to keep its sample
// twiddles, is faster seven times over than the fused kernel (256x224x32, 32 coils, 64 shots:
// 102.3 ms against 103.9).
template <int Y>
static int launch_fast_lm_y(FwdArgs& A, int maxps, int nb, cudaStream_t st) {
  if constexpr (line_threads(Y) == 8) {
    if (maxps <= kThreads) return launch_fast_lm_t<Y, 1>(A, nb, st);
    if (maxps <= 2 * kThreads) return launch_fast_lm_t<Y, 2>(A, nb, st);
  }
  return -1;
}

static int try_fast_lm(FwdArgs& A, int maxps, int nb, cudaStream_t st) {
  switch (A.Y) {
#define ME_LM_CASE(N) \
  case N: return launch_fast_lm_y<N>(A, maxps, nb, st);
    ME_FAST_LENGTHS(ME_LM_CASE)
#undef ME_LM_CASE
    default: return -1;
  }
}

// The compile-time kernels take one volume per CTA (FWD_K, FWD_RESID); the seven-volume LM
// statistics use FWD_K over seven volumes per shot and lm_stats_kernel instead of FWD_LM.
template <int Y>
static int launch_fast_fwd_y(FwdArgs& A, int mode, int maxps, int nb, cudaStream_t st) {
  if (mode == FWD_K) return launch_fast_fwd_m<Y, FWD_K>(A, maxps, nb, st);
  if (mode == FWD_RESID) return launch_fast_fwd_m<Y, FWD_RESID>(A, maxps, nb, st);
  return -1;
}

static int try_fast_fwd(FwdArgs& A, int mode, int maxps, int nb, cudaStream_t st) {
  switch (A.Y) {
#define ME_FWD_CASE(N) \
  case N: return launch_fast_fwd_y<N>(A, mode, maxps, nb, st);
    ME_FAST_LENGTHS(ME_FWD_CASE)
#undef ME_FWD_CASE
    default: return -1;
  }
}

template <int Y>
static int launch_fast_adj_y(AdjArgs& A, int maxps, int nb, cudaStream_t st) {
  using P = AdjPlan<Y>;
  constexpr int NG = P::NG;
  A.XB = maxps;
  const size_t kcap = pad2(maxps);
  const size_t smem = sizeof(float2) * (P::NK * kcap + (size_t)NG * P::LS + pad2(A.X)) +
                      P::TABLES * kcap * (P::TABULATE ? sizeof(float2) : sizeof(short));
  ME_TRY(check_cuda(allow_smem(fast_adj_kernel<Y>, smem), "adj smem"));
  dim3 grid(nb, (A.X + NG - 1) / NG, A.Z);
  count_launch();
  return check_cuda(launch_chained(true, fast_adj_kernel<Y>, grid, kThreads, smem, st, A),
                    "fast sense_adj launch");
}

static int try_fast_adj(AdjArgs& A, int maxps, int nb, cudaStream_t st) {
  switch (A.Y) {
#define ME_ADJ_CASE(N) \
  case N: return launch_fast_adj_y<N>(A, maxps, nb, st);
    ME_FAST_LENGTHS(ME_ADJ_CASE)
#undef ME_ADJ_CASE
    default: return -1;
  }
}

static bool has_fast_length(int n) {
  switch (n) {
#define ME_HAS_CASE(N) \
  case N: return true;
    ME_FAST_LENGTHS(ME_HAS_CASE)
#undef ME_HAS_CASE
    default: return false;
  }
}

// Whether the compile-time or run-time SENSE kernels serve this problem (they take the K of
// several volumes per shot in one launch, which the LM statistics use).
static bool fast_sense_for(const me_sense* pb) {
  return fast_sense_enabled() && pb->nx <= 512 &&
         (has_fast_length(pb->ny) || has_rt_sense(pb->ny));
}

static int launch_fwd(const me_sense* pb, int mode, const float2* vols, i64 vol_stride, int shot0,
                      int nb, float2* kout, double* partial, cudaStream_t st, int kout_abs = 0,
                      int vps = 1, i64 kout_vs = 0) {
  FwdArgs A{};
  A.kout_abs = kout_abs;
  A.vps = vps;
  A.kout_vs = kout_vs;
  A.X = pb->nx;
  A.Y = pb->ny;
  A.Z = pb->nz;
  A.C = pb->ncoils;
  A.mps = (const float2*)pb->mps;
  A.vols = vols;
  A.vol_stride = vol_stride;
  A.shot0 = shot0;
  A.shot_off = pb->samples.shot_off;
  A.kx = pb->samples.kx;
  A.ky = pb->samples.ky;
  A.ydat = (const float2*)pb->ydat;
  A.kout = kout;
  A.partial = partial;
  const double scale = sense_scale(pb);
  A.scale = (float)scale;
  A.scale_lo = (float)(scale - (double)A.scale);
  if (!make_plan(pb->ny, &A.plan)) {
    set_error("ny has a prime factor > 13");
    return ME_ERR_UNSUPPORTED;
  }
  const int maxps = pb->samples.max_per_shot;
  if (fast_sense_enabled() && pb->nx <= 512) {
    // FWD_LM over the seven volumes of each shot: the fused statistics kernel, or -1 (not
    // handled) for the caller's two-kernel path
    if (mode == FWD_LM && vps == 7) return fused_lm_enabled() ? try_fast_lm(A, maxps, nb, st) : -1;
    int rc = try_fast_fwd(A, mode, maxps, nb, st);
    if (rc < 0) rc = try_rt_fwd(A, mode, maxps, nb, st);
    if (rc >= 0) return rc;
  }
  if (vps != 1) {
    set_error("several volumes per shot need the compile-time or run-time SENSE kernels");
    return ME_ERR_UNSUPPORTED;
  }
  if (mode == FWD_LM) {
    A.XR = fwd_rows(7, pb->ny);
    return launch_fwd_v<7, FWD_LM>(A, maxps, nb, st);
  }
  A.XR = fwd_rows(1, pb->ny);
  if (mode == FWD_K) return launch_fwd_v<1, FWD_K>(A, maxps, nb, st);
  return launch_fwd_v<1, FWD_RESID>(A, maxps, nb, st);
}

static int launch_fwd_abs(const me_sense* pb, const float2* vols, i64 vol_stride, int shot0,
                          int nb, float2* kout, cudaStream_t st) {
  return launch_fwd(pb, FWD_K, vols, vol_stride, shot0, nb, kout, nullptr, st, 1);
}

template <int EPT>
static int launch_adj_t(AdjArgs& A, int maxps, int nb, cudaStream_t st) {
  A.es = A.XB + 1;
  const size_t smem =
      sizeof(float2) * (pad2(A.Y) + pad2(A.X) + pad2(maxps) + 2 * (size_t)A.Y * A.es);
  ME_TRY(check_cuda(allow_smem(sense_adj_kernel<EPT>, smem), "sense_adj smem"));
  dim3 grid(A.Z, (A.X + A.XB - 1) / A.XB, nb);
  count_launch();
  sense_adj_kernel<EPT><<<grid, kThreads, smem, st>>>(A);
  return check_cuda(cudaGetLastError(), "sense_adj launch");
}

static int launch_adj(const me_sense* pb, const float2* kin, int kin_rel, float2* out, i64 vs,
                      int shot0, int nb, cudaStream_t st) {
  AdjArgs A{};
  A.X = pb->nx;
  A.Y = pb->ny;
  A.Z = pb->nz;
  A.C = pb->ncoils;
  A.mps = (const float2*)pb->mps;
  A.kin = kin;
  A.kin_rel = kin_rel;
  A.out = out;
  A.vol_stride = vs;
  A.shot0 = shot0;
  A.shot_off = pb->samples.shot_off;
  A.kx = pb->samples.kx;
  A.ky_off = pb->samples.ky_off;
  A.ky_order = pb->samples.ky_order;
  const double scale = sense_scale(pb);
  A.scale = (float)scale;
  A.scale_lo = (float)(scale - (double)A.scale);
  if (!make_plan(pb->ny, &A.plan)) {
    set_error("ny has a prime factor > 13");
    return ME_ERR_UNSUPPORTED;
  }
  if (fast_sense_enabled() && pb->nx <= 512) {
    int rc = try_fast_adj(A, pb->samples.max_per_shot, nb, st);
    if (rc < 0) rc = try_rt_adj(A, pb->samples.max_per_shot, nb, st);
    if (rc >= 0) return rc;
  }
  A.XB = std::max(1, std::min(std::min(pb->nx, 32), 4096 / pb->ny));
  const int ept = (A.XB * pb->ny + kThreads - 1) / kThreads;
  const int maxps = pb->samples.max_per_shot;
  if (ept <= 4) return launch_adj_t<4>(A, maxps, nb, st);
  if (ept <= 8) return launch_adj_t<8>(A, maxps, nb, st);
  return launch_adj_t<16>(A, maxps, nb, st);
}

// Blocks per shot of the gradient's image-space dot products, and the partial sums it keeps
// per shot: one energy partial per (z, coil) plane, then six per block.
constexpr int kGradBlocks = 296;
static i64 grad_partials(const me_sense* pb) {
  return (i64)pb->nz * pb->ncoils + 6LL * kGradBlocks;
}

struct Ws {
  float2* U;
  float2* K;
  double* partial;
  i64 kvs;  // elements per K region (one region per volume of a shot)
};

static i64 align256(i64 n) { return (n + 255) & ~255LL; }

static i64 ws_layout(const me_sense* pb, int batch, int vols_per_shot, int extra_vols, Ws* w,
                     void* base, int kvols = 1, i64 min_partials_per_shot = 0) {
  const i64 vox = vox_of(pb);
  const i64 nU = (i64)batch * vols_per_shot * vox + (i64)extra_vols * vox;
  const i64 nK1 = (i64)batch * pb->samples.max_per_shot * pb->ncoils * pb->nz;
  const i64 nK = nK1 * kvols;
  const i64 nP = (i64)batch * std::max<i64>((i64)pb->nz * pb->ncoils * kLmStats,
                                            min_partials_per_shot);
  const i64 bU = align256(nU * 8), bK = align256(nK * 8), bP = align256(nP * 8);
  if (w && base) {
    char* p = (char*)base;
    w->U = (float2*)p;
    w->K = (float2*)(p + bU);
    w->partial = (double*)(p + bU + bK);
    w->kvs = nK1;
  }
  return bU + bK + bP;
}

}  // namespace me

using namespace me;

extern "C" {

long long me_sense_workspace_bytes(const me_sense* pb, int batch) {
  if (check_problem(pb) != ME_OK || batch < 1) return -1;
  batch = std::min(batch, pb->nshots);
  return ws_layout(pb, batch, 1, 0, nullptr, nullptr);
}

long long me_lm_ga_workspace_bytes(const me_sense* pb, int batch) {
  if (check_problem(pb) != ME_OK || batch < 1) return -1;
  batch = std::min(batch, pb->nshots);
  return ws_layout(pb, batch, 13, 0, nullptr, nullptr, 7);
}

long long me_lm_gradient_workspace_bytes(const me_sense* pb, int batch) {
  if (check_problem(pb) != ME_OK || batch < 1) return -1;
  batch = std::min(batch, pb->nshots);
  return ws_layout(pb, batch, 13, 0, nullptr, nullptr, 1, grad_partials(pb));
}

long long me_lm_workspace_bytes(const me_sense* pb, int batch) {
  if (check_problem(pb) != ME_OK || batch < 1) return -1;
  batch = std::min(batch, pb->nshots);
  return ws_layout(pb, batch, 12, 0, nullptr, nullptr, fast_sense_for(pb) ? 7 : 1);
}

int me_sense_precond(const me_c64* mps, int nx, int ny, int nz, int ncoils, float* P,
                     unsigned char* M, void* stream) {
  if (!mps || !P || !M) return fail("me_sense_precond: NULL pointer");
  const i64 plane = (i64)nx * ny;
  count_launch();
  precond_kernel<<<grid_1d(plane * nz), kThreads, 0, (cudaStream_t)stream>>>(
      (const float2*)mps, ncoils, plane, nz, P, M);
  return check_cuda(cudaGetLastError(), "precond launch");
}

int me_sense_gather(const me_sense* pb, const me_c64* ksp_h, me_c64* ydat, void* stream) {
  ME_TRY(check_problem(pb));
  if (!ksp_h || !ydat) return fail("me_sense_gather: NULL pointer");
  const i64 approx = (i64)pb->nshots * pb->samples.max_per_shot * pb->ncoils * pb->nz;
  count_launch();
  gather_kernel<<<grid_1d(approx), kThreads, 0, (cudaStream_t)stream>>>(
      (const float2*)ksp_h, pb->nx, pb->ny, pb->nz, pb->ncoils, pb->samples.shot_off,
      pb->samples.kx, pb->samples.ky, pb->nshots, (float2*)ydat);
  return check_cuda(cudaGetLastError(), "gather launch");
}

int me_sense_normal(const me_sense* pb, const me_c64* p, me_c64* out, int batch, void* work,
                    void* stream) {
  ME_TRY(check_problem(pb));
  if (!p || !out || !work) return fail("me_sense_normal: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 1, 0, &w, work);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, pb->transforms + 6 * (i64)s0, 6, st);
    ME_TRY(R.apply((const float2*)p, 0, w.U, vox, nb, false));
    ME_TRY(launch_fwd(pb, FWD_K, w.U, vox, s0, nb, w.K, nullptr, st));
    ME_TRY(launch_adj(pb, w.K, 1, w.U, vox, s0, nb, st));
    ME_TRY(R.adjoint(w.U, vox, w.U, vox, nb, false));
    count_launch();
    sum_volumes_kernel<<<grid_1d(vox), kThreads, 0, st>>>(w.U, vox, nb, pb->M, (float2*)out, vox,
                                                          s0 > 0);
    ME_TRY(check_cuda(cudaGetLastError(), "sum_volumes launch"));
  }
  return ME_OK;
}

int me_sense_rhs(const me_sense* pb, me_c64* b, int batch, void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!b || !work || !pb->ydat) return fail("me_sense_rhs: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 1, 0, &w, work);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, pb->transforms + 6 * (i64)s0, 6, st);
    ME_TRY(launch_adj(pb, (const float2*)pb->ydat, 0, w.U, vox, s0, nb, st));
    ME_TRY(R.adjoint(w.U, vox, w.U, vox, nb, false));
    count_launch();
    sum_volumes_kernel<<<grid_1d(vox), kThreads, 0, st>>>(w.U, vox, nb, pb->M, (float2*)b, vox,
                                                          s0 > 0);
    ME_TRY(check_cuda(cudaGetLastError(), "sum_volumes launch"));
  }
  return ME_OK;
}

int me_sense_residual(const me_sense* pb, const me_c64* x, me_c64* r, double* e, int batch,
                      void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !r || !work || !pb->ydat) return fail("me_sense_residual: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 1, 0, &w, work);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  const int zc = pb->nz * pb->ncoils;
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, pb->transforms + 6 * (i64)s0, 6, st);
    ME_TRY(R.apply((const float2*)x, 0, w.U, vox, nb, false));
    ME_TRY(launch_fwd(pb, FWD_K, w.U, vox, s0, nb, w.K, nullptr, st));
    // y - K at the shot's samples, in place, with the energy partials of each (z, coil)
    count_launch();
    resid_inplace_kernel<true><<<dim3(zc, nb), kThreads, 0, st>>>(
        w.K, (const float2*)pb->ydat, pb->samples.shot_off, s0, zc, w.partial);
    ME_TRY(check_cuda(cudaGetLastError(), "residual launch"));
    if (e) {
      count_launch();
      reduce_partials_kernel<<<nb, kThreads, 0, st>>>(w.partial, zc, 1, e, s0);
      ME_TRY(check_cuda(cudaGetLastError(), "reduce launch"));
    }
    ME_TRY(launch_adj(pb, w.K, 1, w.U, vox, s0, nb, st));
    ME_TRY(R.adjoint(w.U, vox, w.U, vox, nb, false));
    count_launch();
    sum_volumes_kernel<<<grid_1d(vox), kThreads, 0, st>>>(w.U, vox, nb, pb->M, (float2*)r, vox,
                                                          s0 > 0);
    ME_TRY(check_cuda(cudaGetLastError(), "sum_volumes launch"));
  }
  return ME_OK;
}

int me_sense_residual_norms(const me_sense* pb, const me_c64* x, const double* transforms,
                            double* e, int batch, void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !transforms || !e || !work || !pb->ydat)
    return fail("me_sense_residual_norms: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 1, 0, &w, work);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, transforms + 6 * (i64)s0, 6, st);
    ME_TRY(R.apply((const float2*)x, 0, w.U, vox, nb, false));
    ME_TRY(launch_fwd(pb, FWD_RESID, w.U, vox, s0, nb, nullptr, w.partial, st));
    count_launch();
    reduce_partials_kernel<<<nb, kThreads, 0, st>>>(w.partial, pb->nz * pb->ncoils, 1, e, s0);
    ME_TRY(check_cuda(cudaGetLastError(), "reduce launch"));
  }
  return ME_OK;
}

int me_sense_forward(const me_sense* pb, const me_c64* x, const double* transforms, me_c64* K,
                     int batch, void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !transforms || !K || !work) return fail("me_sense_forward: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 1, 0, &w, work);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, transforms + 6 * (i64)s0, 6, st);
    ME_TRY(R.apply((const float2*)x, 0, w.U, vox, nb, false));
    // K is written with offsets relative to shot_off[s0]; shift the base to the batch's block
    ME_TRY(launch_fwd_abs(pb, w.U, vox, s0, nb, (float2*)K, st));
  }
  return ME_OK;
}

int me_sense_forward_volumes(const me_sense* pb, const me_c64* vols, long long vol_stride,
                             int shot0, int nshots, me_c64* K, void* stream) {
  ME_TRY(check_problem(pb));
  if (!vols || !K) return fail("me_sense_forward_volumes: NULL pointer");
  if (shot0 < 0 || nshots < 1 || shot0 + nshots > pb->nshots)
    return fail("me_sense_forward_volumes: shot range outside the problem");
  if (vol_stride != 0 && vol_stride < vox_of(pb))
    return fail("me_sense_forward_volumes: volume stride must be 0 or at least one volume");
  return launch_fwd(pb, FWD_K, (const float2*)vols, vol_stride, shot0, nshots, (float2*)K,
                    nullptr, (cudaStream_t)stream);
}

int me_sense_adjoint_volumes(const me_sense* pb, const me_c64* K, int shot0, int nshots,
                             me_c64* vols, long long vol_stride, void* stream) {
  ME_TRY(check_problem(pb));
  if (!vols || !K) return fail("me_sense_adjoint_volumes: NULL pointer");
  if (shot0 < 0 || nshots < 1 || shot0 + nshots > pb->nshots)
    return fail("me_sense_adjoint_volumes: shot range outside the problem");
  if (vol_stride < vox_of(pb))
    return fail("me_sense_adjoint_volumes: volume stride must be at least one volume");
  return launch_adj(pb, (const float2*)K, 1, (float2*)vols, vol_stride, shot0, nshots,
                    (cudaStream_t)stream);
}

int me_sense_scatter(const me_sense* pb, const me_c64* K, me_c64* ksp_h, void* stream) {
  ME_TRY(check_problem(pb));
  if (!K || !ksp_h) return fail("me_sense_scatter: NULL pointer");
  const i64 per = (i64)pb->samples.max_per_shot * pb->ncoils * pb->nz;
  for (int s = 0; s < pb->nshots; s++) {
    count_launch();
    scatter_kernel<<<grid_1d(per), kThreads, 0, (cudaStream_t)stream>>>(
        (const float2*)K, pb->nx, pb->ny, pb->nz, pb->ncoils, pb->samples.shot_off,
        pb->samples.kx, pb->samples.ky, s, (float2*)ksp_h);
    ME_TRY(check_cuda(cudaGetLastError(), "scatter launch"));
  }
  return ME_OK;
}

int me_lm_normal_equations(const me_sense* pb, const me_c64* x, int jac_mode, double* stats,
                           int batch, void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !stats || !work || !pb->ydat) return fail("me_lm_normal_equations: NULL pointer");
  if (jac_mode != ME_JAC_REFERENCE && jac_mode != ME_JAC_EXACT) return fail("bad jacobian mode");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  const bool fast = fast_sense_for(pb);
  ws_layout(pb, batch, 12, 0, &w, work, fast ? 7 : 1);
  const i64 vox = vox_of(pb);
  const me_layout lay = zxy_layout(pb);
  float2* jwork = w.U + (i64)batch * 7 * vox;
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    {
      // T x and its six partials for the batch's shots at once: [shot][7] volumes in U, five
      // work volumes per shot after them
      Rigid R(pb->grid, lay, pb->transforms + 6 * (i64)s0, 6, st);
      ME_TRY(R.jacobian((const float2*)x, 0, w.U, vox, 7 * vox, nb, jac_mode, jwork, 5 * vox));
    }
    const int rcf = fast ? launch_fwd(pb, FWD_LM, w.U, vox, s0, nb, nullptr, w.partial, st, 0, 7)
                         : -1;
    if (rcf >= 0) {
      // fused: the statistics of the seven volumes contracted in registers
      ME_TRY(rcf);
    } else if (fast) {
      // the seven volumes of every shot through the one-volume forward kernel, then the sums
      ME_TRY(launch_fwd(pb, FWD_K, w.U, vox, s0, nb, w.K, nullptr, st, 0, 7, w.kvs));
      const int zc = pb->nz * pb->ncoils;
      count_launch();
      lm_stats_kernel<<<dim3(zc, nb), kThreads, 0, st>>>(w.K, w.kvs, (const float2*)pb->ydat,
                                                          pb->samples.shot_off, s0, zc, w.partial);
      ME_TRY(check_cuda(cudaGetLastError(), "lm stats launch"));
    } else {
      ME_TRY(launch_fwd(pb, FWD_LM, w.U, vox, s0, nb, nullptr, w.partial, st));
    }
    count_launch();
    reduce_partials_kernel<<<nb, kThreads, 0, st>>>(w.partial, pb->nz * pb->ncoils, kLmStats,
                                                     stats, s0);
    ME_TRY(check_cuda(cudaGetLastError(), "reduce launch"));
  }
  return ME_OK;
}

int me_lm_gradient(const me_sense* pb, const me_c64* x, int jac_mode, double* grad, int batch,
                   void* work, void* stream) {
  return me_lm_gradient_image(pb, x, jac_mode, grad, nullptr, batch, work, stream);
}

int me_lm_gradient_image(const me_sense* pb, const me_c64* x, int jac_mode, double* grad,
                         me_c64* gx, int batch, void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !grad || !work || !pb->ydat) return fail("me_lm_gradient: NULL pointer");
  if ((const void*)gx == (const void*)x) return fail("me_lm_gradient_image: gx must not be x");
  if (jac_mode != ME_JAC_REFERENCE && jac_mode != ME_JAC_EXACT) return fail("bad jacobian mode");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 13, 0, &w, work, 1, grad_partials(pb));
  const i64 vox = vox_of(pb);
  const i64 bs = 8 * vox;  // per shot: T x, six partials, W = C^H F^H M_s r
  const me_layout lay = zxy_layout(pb);
  float2* jwork = w.U + (i64)batch * bs;
  const int zc = pb->nz * pb->ncoils;
  const int nblk = kGradBlocks;
  double* dpart = w.partial + (i64)batch * zc;  // after the energy partials of the batch
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    Rigid R(pb->grid, lay, pb->transforms + 6 * (i64)s0, 6, st);
    ME_TRY(R.jacobian((const float2*)x, 0, w.U, vox, bs, nb, jac_mode, jwork, 5 * vox));
    // r = M_s F C T x - y at the shot's samples, then W = C^H F^H M_s r in image space
    ME_TRY(launch_fwd(pb, FWD_K, w.U, bs, s0, nb, w.K, nullptr, st));
    count_launch();
    resid_inplace_kernel<false><<<dim3(zc, nb), kThreads, 0, st>>>(
        w.K, (const float2*)pb->ydat, pb->samples.shot_off, s0, zc, w.partial);
    ME_TRY(check_cuda(cudaGetLastError(), "residual launch"));
    ME_TRY(launch_adj(pb, w.K, 1, w.U + 7 * vox, bs, s0, nb, st));
    // g_p = Re<r, M_s F C dT/dp x> = Re<W, dT/dp x>
    count_launch();
    grad_dots_kernel<<<dim3(nblk, nb), kThreads, 0, st>>>(w.U, bs, vox, dpart);
    ME_TRY(check_cuda(cudaGetLastError(), "gradient dots launch"));
    count_launch();
    grad_finish_kernel<<<nb, 32, 0, st>>>(w.partial, zc, dpart, nblk, grad, s0);
    ME_TRY(check_cuda(cudaGetLastError(), "gradient finish launch"));
    if (gx) {
      // the image's gradient is one adjoint transform away: sum_s T_s^H W_s
      ME_TRY(R.adjoint(w.U + 7 * vox, bs, w.U + 7 * vox, bs, nb, false));
      count_launch();
      sum_volumes_kernel<<<grid_1d(vox), kThreads, 0, st>>>(w.U + 7 * vox, bs, nb, nullptr,
                                                            (float2*)gx, vox, s0 > 0);
      ME_TRY(check_cuda(cudaGetLastError(), "sum_volumes launch"));
    }
  }
  return ME_OK;
}

int me_lm_ga_rhs(const me_sense* pb, const me_c64* x, int jac_mode, int ga_mode,
                 const double* t_eps, const double* v, double eps, double* rhs, int batch,
                 void* work, void* stream) {
  ME_TRY(check_problem(pb));
  if (!x || !t_eps || !v || !rhs || !work || !pb->ydat) return fail("me_lm_ga_rhs: NULL pointer");
  if (jac_mode != ME_JAC_REFERENCE && jac_mode != ME_JAC_EXACT) return fail("bad jacobian mode");
  if (ga_mode != ME_GA_REFERENCE && ga_mode != ME_GA_INTENDED) return fail("bad GA mode");
  if (!(eps > 0.0)) return fail("me_lm_ga_rhs: eps must be positive");
  cudaStream_t st = (cudaStream_t)stream;
  batch = std::max(1, std::min(batch, pb->nshots));
  Ws w;
  ws_layout(pb, batch, 13, 0, &w, work, 7);
  const i64 vox = vox_of(pb);
  const i64 bs = 8 * vox;  // per shot: T x, six partials, the direction D
  const me_layout lay = zxy_layout(pb);
  float2* jwork = w.U + (i64)batch * bs;
  const int zc = pb->nz * pb->ncoils;
  for (int s0 = 0; s0 < pb->nshots; s0 += batch) {
    const int nb = std::min(batch, pb->nshots - s0);
    const double* vb = v + 6 * (i64)s0;
    for (int pass = 0; pass < 2; pass++) {
      // partials at theta + eps v first, then at theta
      const double* prm = (pass == 0 ? t_eps : pb->transforms) + 6 * (i64)s0;
      Rigid R(pb->grid, lay, prm, 6, st);
      ME_TRY(R.jacobian((const float2*)x, 0, w.U, vox, bs, nb, jac_mode, jwork, 5 * vox));
      count_launch();
      ga_combine_kernel<<<grid_1d((i64)nb * vox), kThreads, 0, st>>>(w.U, bs, vox, nb, vb, ga_mode,
                                                                      pass == 0, eps);
      ME_TRY(check_cuda(cudaGetLastError(), "ga combine launch"));
    }
    // M_s F C of the six partials at theta and of D, one volume at a time per shot
    for (int k = 0; k < 7; k++)
      ME_TRY(launch_fwd(pb, FWD_K, w.U + (k < 6 ? 1 + k : 7) * vox, bs, s0, nb, w.K + k * w.kvs,
                        nullptr, st));
    count_launch();
    ga_dots_kernel<<<dim3(zc, nb), kThreads, 0, st>>>(w.K, w.kvs, pb->samples.shot_off, s0, zc,
                                                       w.partial);
    ME_TRY(check_cuda(cudaGetLastError(), "ga dots launch"));
    count_launch();
    reduce_partials_kernel<<<nb, kThreads, 0, st>>>(w.partial, zc, 6, rhs, s0);
    ME_TRY(check_cuda(cudaGetLastError(), "reduce launch"));
  }
  return ME_OK;
}

}  // extern "C"
