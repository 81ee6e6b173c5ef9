// SENSE forward and adjoint for plane widths Y without a compile-time plan, on the run-time
// two-stage FFT (fft_rt.cuh).  Same arguments, layouts and meaning as the kernels of sense.cu.
//
// Both give one CTA NR rows of a plane (32, 24, 16 or 8: as many as 256 threads hold at one DFT
// per thread and stage), read map and image rows from global memory straight into the DFTs that
// use them (they sit in L2: shots are fastest in the grid), and take a coil at a time, the
// sample twiddles set up once for all of the CTA's coils.
//
// Measured at 160x150x126, 16 coils, 20 shots of 1,200 samples: forward 6.3 ms and adjoint 6.6 ms
// where the Stockham kernels of sense.cu took about 96 ms together; the whole normal operator
// 163.7 -> 21.4 ms.  Reading the sample steps in sample order rather than out of twX took 0.3 and
// 0.5 ms of that.  Widths with a compile-time plan keep their kernels: at 256x224x176, 32 coils,
// 64 shots these took 67.8 and 90.7 ms when those took 55.8 and 63.6 ms.
#include <algorithm>

#include "fft_rt.cuh"
#include "sense.cuh"

namespace me {

// Planes of a launch: more (only calls on caller-transformed volumes can have them, whose z axis
// is no line) go to the kernels of sense.cu, which count them along x.
constexpr int kMaxGridZ = 65535;

constexpr int kOctet = 8;  // rows per H-building item; NR is a multiple

// Rows per CTA for a plan.
static int rt_rows(const RtPlan& P) {
  return std::min(32, kThreads / P.rmax() / kOctet * kOctet);
}

struct RtSense {
  RtPlan P;
  int NR;       // rows per chunk (forward) or per CTA (adjoint)
  int ls, ys;   // odd strides of a line's transpose table and of its spectrum
  int cg;       // coils per CTA (forward)
};

template <int MPT, int MODE, bool LARGE>
__global__ void __launch_bounds__(kThreads, (MPT > 4 || LARGE) ? 2 : 3)
    rt_fwd_kernel(const __grid_constant__ FwdArgs A, const __grid_constant__ RtSense T) {
  extern __shared__ __align__(16) float2 sm[];
  const RtPlan& P = T.P;
  const int bx = blockIdx.x, z = blockIdx.z;
  const int b = bx / A.vps, vk = bx - b * A.vps;
  const int s = A.shot0 + b;
  const int X = A.X, Y = A.Y, NR = T.NR, R1 = P.r1, R2 = P.r2, S1 = P.s1;
  const int tid = threadIdx.x;
  float2* tw = sm;
  float2* twX = tw + Y;
  float2* tab = twX + X;
  float2* spec = tab + NR * T.ls;
  // W^kx, W^2kx and W^4kx of each sample: in sample order, where a warp's reads are free of the bank
  // conflicts of reading them out of twX in every chunk
  float2* hst = spec + NR * T.ys;
  float2* hst2 = hst + MPT * kThreads;
  float2* hst4 = hst2 + MPT * kThreads;
  rt_init_twiddles(tw, P);
  init_twiddles(twX, X);
  chain_next();
  chain_wait();

  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  __syncthreads();
  // per sample: ky, and the step kx NR mod X of its chunk twiddle's index
  int mky[MPT], dix[MPT];
#pragma unroll
  for (int m = 0; m < MPT; m++) {
    const int jj = tid + m * kThreads;
    mky[m] = dix[m] = 0;
    if (jj < ns) {
      const int kx = A.kx[soff + jj];
      mky[m] = A.ky[soff + jj];
      dix[m] = mulmod(kx, NR % X, X, 1.0f / (float)X);
      hst[jj] = twX[kx];
      hst2[jj] = twX[2 * kx % X];
      hst4[jj] = twX[4 * kx % X];
    }
  }
  const int g1 = P.d2.div(tid), j1 = tid - g1 * R2;
  const int g2 = P.d1.div(tid), k2 = tid - g2 * R1;
  const bool has1 = g1 < NR, has2 = g2 < NR;
  const i64 plane = (i64)X * Y;
  const float2* vbase = A.vols + (i64)bx * A.vol_stride + (i64)z * plane;

  const int c1 = min(A.C, ((int)blockIdx.y + 1) * T.cg);
  for (int c = blockIdx.y * T.cg; c < c1; c++) {
    const float2* mrow = A.mps + ((i64)z * A.C + c) * plane;
    float2 acc[MPT];
    int idx[MPT];
#pragma unroll
    for (int m = 0; m < MPT; m++) {
      acc[m] = make_float2(0.f, 0.f);
      idx[m] = 0;
    }
    for (int x0 = 0; x0 < X; x0 += NR) {
      if (has1) {
        const bool live = x0 + g1 < X;
        const int off = (x0 + g1) * Y + j1;
        rt_switch1(R1, [&](auto rc) {
          constexpr int R = decltype(rc)::value;
          float2 u[R];
#pragma unroll
          for (int r = 0; r < R; r++)
            u[r] = live ? cmul(mrow[off + r * R2], vbase[off + r * R2]) : make_float2(0.f, 0.f);
          RDft<R, false>::run(u);
          float2* dst = tab + g1 * T.ls + j1 * S1;
#pragma unroll
          for (int r = 0; r < R; r++) dst[r] = u[r];
        });
      }
      __syncthreads();
      if (has2) {
        rt_switch2<LARGE>(R2, [&](auto rc) {
          constexpr int R = decltype(rc)::value;
          const float2* src = tab + g2 * T.ls + k2;
          float2 v[R];
#pragma unroll
          for (int r = 0; r < R; r++)
            v[r] = (r == 0) ? src[0] : cmul(src[r * S1], tw[r * R1 + k2]);
          RDft<R, false>::run(v);
          float2* dst = spec + g2 * T.ys + k2;
#pragma unroll
          for (int r = 0; r < R; r++) dst[r * R1] = v[r];
        });
      }
      __syncthreads();
      // sample sums over the chunk's rows by Horner's rule in four chains, each stepping by W^4kx
      // (rows past X hold zeros): of 32 rows, a chain carries the rounding of its step up to the
      // 7th power; two chains would to the 15th
#pragma unroll
      for (int m = 0; m < MPT; m++) {
        const int jj = tid + m * kThreads;
        if (jj >= ns) continue;
        const float2 st = hst[jj], st2 = hst2[jj], st4 = hst4[jj];
        const float2 w0 = twX[idx[m]];
        const float2* Lk = spec + mky[m];
        float2 h[4];
#pragma unroll
        for (int q = 0; q < 4; q++) h[q] = Lk[(NR - 4 + q) * T.ys];
#pragma unroll 2
        for (int i = NR - 8; i >= 0; i -= 4) {
#pragma unroll
          for (int q = 0; q < 4; q++) h[q] = cfma(h[q], st4, Lk[(i + q) * T.ys]);
        }
        const float2 lo = cfma(h[1], st, h[0]), hi = cfma(h[3], st, h[2]);
        acc[m] = cfma(cfma(hi, st2, lo), w0, acc[m]);
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
        const int jj = tid + m * kThreads;
        if (jj < ns)
          A.kout[(i64)vk * A.kout_vs + base + jj] = cscale2(acc[m], A.scale, A.scale_lo);
      }
    } else {
      const i64 base = (i64)soff * A.C * A.Z + zc * ns;
      double e[1] = {0.0};
#pragma unroll
      for (int m = 0; m < MPT; m++) {
        const int jj = tid + m * kThreads;
        if (jj < ns) {
          const float2 r = csub(cscale2(acc[m], A.scale, A.scale_lo), A.ydat[base + jj]);
          e[0] += (double)r.x * r.x + (double)r.y * r.y;
        }
      }
      block_reduce_store<1>(e, A.partial + ((i64)b * A.Z * A.C + zc));
    }
  }
}

template <bool LARGE>
__global__ void __launch_bounds__(kThreads, 2)
    rt_adj_kernel(const __grid_constant__ AdjArgs A, const __grid_constant__ RtSense T) {
  extern __shared__ __align__(16) float2 sm[];
  const RtPlan& P = T.P;
  const int X = A.X, Y = A.Y, NR = T.NR, R1 = P.r1, R2 = P.r2, S1 = P.s1;
  const int b = blockIdx.x, x0 = blockIdx.y * NR, z = blockIdx.z;
  const int s = A.shot0 + b;
  const int tid = threadIdx.x;
  chain_next();
  chain_wait();
  const int soff = A.shot_off[s];
  const int ns = A.shot_off[s + 1] - soff;
  const int kcap = A.XB;      // max samples per shot, rounded up to even
  const int no = NR / kOctet;
  float2* tw = sm;
  float2* twX = tw + Y;
  float2* K = twX + X;        // kcap samples of a coil
  float2* H = K + kcap;       // [NR][ys]
  float2* tab = H + NR * T.ys;
  float2* tw_s = tab + NR * T.ls;  // conj W^kx and conj W^3kx of a sample,
  float2* tw_3 = tw_s + kcap;
  float2* tw_0 = tw_3 + kcap;      // and conj W^(kx x) at each octet's middle
  rt_init_twiddles(tw, P);
  init_twiddles(twX, X);
  const float inv_x = 1.0f / (float)X;
  __syncthreads();
  for (int i = tid; i < ns; i += kThreads) {
    const int kx = A.kx[soff + i];
    tw_s[i] = cconj(twX[kx]);
    tw_3[i] = cconj(twX[3 * kx % X]);
    for (int o = 0; o < no; o++)
      tw_0[o * kcap + i] =
          cconj(twX[mulmod(kx, (x0 + o * kOctet + kOctet / 2) % X, X, inv_x)]);
  }
  const int* kyo = A.ky_off + (i64)s * (Y + 1);
  const int* order = A.ky_order ? A.ky_order + (i64)s * Y : nullptr;
  const i64 kbase0 = (A.kin_rel ? (i64)(soff - A.shot_off[A.shot0]) : (i64)soff) * A.C * A.Z;
  const i64 plane = (i64)X * Y;
  const int g1 = P.d2.div(tid), j1 = tid - g1 * R2;
  const int g2 = P.d1.div(tid), k2 = tid - g2 * R1;
  const bool has2 = g2 < NR, live = g1 < NR && x0 + g1 < X;
  const i64 off = (i64)(x0 + g1) * Y + j1;

  auto issue = [&](int c) {
    const float2* kc = A.kin + kbase0 + ((i64)z * A.C + c) * ns;
    for (int i = tid; i < ns; i += kThreads) cp_async8(K + i, kc + i);
    cp_async_commit();
  };
  float2 w[kRtMaxR1];
#pragma unroll
  for (int q = 0; q < kRtMaxR1; q++) w[q] = make_float2(0.f, 0.f);

  issue(0);
  for (int c = 0; c < A.C; c++) {
    cp_async_wait_all();
    __syncthreads();
    // H[x][ky] += K exp(+2 pi i kx x / X), eight rows of one bin per item, heaviest bins first
    for (int q = tid; q < Y * no; q += kThreads) {
      const int slot = q / no, o = q - slot * no;
      const int bin = order ? order[slot] : slot;
      h_rows<kOctet, true>(
          kyo[bin], kyo[bin + 1],
          [&](int i, float2& v, float2& st, float2& st3) {
            st = tw_s[i];
            st3 = tw_3[i];
            v = cmul(K[i], tw_0[o * kcap + i]);
          },
          [&](int r, float2 h) { H[(o * kOctet + r) * T.ys + bin] = h; });
    }
    __syncthreads();
    if (c + 1 < A.C) issue(c + 1);  // arrives under the FFT
    if (has2) {
      rt_switch2<LARGE>(R2, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const float2 *src = H + g2 * T.ys + k2, *w2 = tw + k2;
        const int step = fresh(R1), row = fresh(S1);
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++, src += step) v[r] = *src;
        RDft<R, true>::run(v);
        float2* dst = tab + g2 * T.ls + k2;
#pragma unroll
        for (int r = 0; r < R; r++, dst += row, w2 += step)
          *dst = (r == 0) ? v[0] : cmulc(v[r], *w2);
      });
    }
    __syncthreads();
    if (live) {
      const float2* ms = A.mps + ((i64)z * A.C + c) * plane + off;
      rt_switch1(R1, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const float2* src = tab + g1 * T.ls + j1 * S1;
        float2 u[R];
#pragma unroll
        for (int q = 0; q < R; q++) u[q] = src[q];
        RDft<R, true>::run(u);
#pragma unroll
        for (int q = 0; q < R; q++)  // (one rounding of the sum a coil; fused, two)
          w[q] = cadd(w[q], cmulc(u[q], ms[q * R2]));
      });
    }
  }
  if (live) {
    float2* o = A.out + (i64)b * A.vol_stride + (i64)z * plane + off;
#pragma unroll
    for (int q = 0; q < kRtMaxR1; q++)
      if (q < R1) o[q * R2] = cscale2(w[q], A.scale, A.scale_lo);
  }
}

static bool rt_sense_plan(int ny, RtSense* T) {
  if (!rt_plan(ny, &T->P)) return false;
  T->NR = rt_rows(T->P);
  T->ls = (T->P.r2 * T->P.s1) | 1;
  T->ys = ny | 1;
  T->cg = 1;
  return true;
}

bool has_rt_sense(int ny) {
  RtSense T;
  return rt_sense_plan(ny, &T);
}

template <int MPT, int MODE, bool LARGE>
static int launch_rt_fwd_t(FwdArgs& A, const RtSense& T, int nb, cudaStream_t st) {
  const size_t smem = sizeof(float2) * ((size_t)A.Y + A.X + (size_t)T.NR * (T.ls + T.ys) +
                                        3 * MPT * (size_t)kThreads);
  const int rc = check_cuda(allow_smem(rt_fwd_kernel<MPT, MODE, LARGE>, smem), "rt fwd smem");
  if (rc != ME_OK) return rc;
  dim3 grid(nb * A.vps, (A.C + T.cg - 1) / T.cg, A.Z);
  count_launch();
  return check_cuda(launch_chained(true, rt_fwd_kernel<MPT, MODE, LARGE>, grid, kThreads, smem, st, A, T),
                    "rt sense_fwd launch");
}

template <int MODE, bool LARGE>
static int launch_rt_fwd_m(FwdArgs& A, const RtSense& T, int maxps, int nb, cudaStream_t st) {
  if (maxps <= kThreads) return launch_rt_fwd_t<1, MODE, LARGE>(A, T, nb, st);
  if (maxps <= 2 * kThreads) return launch_rt_fwd_t<2, MODE, LARGE>(A, T, nb, st);
  if (maxps <= 4 * kThreads) return launch_rt_fwd_t<4, MODE, LARGE>(A, T, nb, st);
  return launch_rt_fwd_t<8, MODE, LARGE>(A, T, nb, st);
}

int try_rt_fwd(FwdArgs& A, int mode, int maxps, int nb, cudaStream_t st) {
  RtSense T;
  if ((mode != FWD_K && mode != FWD_RESID) || A.Z > kMaxGridZ || !rt_sense_plan(A.Y, &T))
    return -1;
  // several coils per CTA while that leaves some ten waves of CTAs
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const i64 ctas = (i64)nb * A.vps * A.C * A.Z, wave = 3LL * std::max(1, sms);
  T.cg = (int)std::max<i64>(1, std::min<i64>(std::min(A.C, 8), ctas / (10 * wave)));
  if (mode == FWD_K)
    return T.P.large() ? launch_rt_fwd_m<FWD_K, true>(A, T, maxps, nb, st)
                       : launch_rt_fwd_m<FWD_K, false>(A, T, maxps, nb, st);
  return T.P.large() ? launch_rt_fwd_m<FWD_RESID, true>(A, T, maxps, nb, st)
                     : launch_rt_fwd_m<FWD_RESID, false>(A, T, maxps, nb, st);
}

template <bool LARGE>
static int launch_rt_adj(AdjArgs& A, const RtSense& T, int nb, cudaStream_t st) {
  const size_t smem = sizeof(float2) * ((size_t)A.Y + A.X + (3 + T.NR / kOctet) * (size_t)A.XB +
                                        (size_t)T.NR * (T.ls + T.ys));
  const int rc = check_cuda(allow_smem(rt_adj_kernel<LARGE>, smem), "rt adj smem");
  if (rc != ME_OK) return rc;
  dim3 grid(nb, (A.X + T.NR - 1) / T.NR, A.Z);
  count_launch();
  return check_cuda(launch_chained(true, rt_adj_kernel<LARGE>, grid, kThreads, smem, st, A, T),
                    "rt sense_adj launch");
}

int try_rt_adj(AdjArgs& A, int maxps, int nb, cudaStream_t st) {
  RtSense T;
  if (A.Z > kMaxGridZ || !rt_sense_plan(A.Y, &T)) return -1;
  A.XB = (maxps + 1) & ~1;
  return T.P.large() ? launch_rt_adj<true>(A, T, nb, st) : launch_rt_adj<false>(A, T, nb, st);
}

}  // namespace me
