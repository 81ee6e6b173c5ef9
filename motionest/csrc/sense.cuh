// Arguments and helpers shared by the SENSE kernels (sense.cu, rt_sense.cu).
#pragma once
#include "fft_smem.cuh"

namespace me {

enum FwdMode { FWD_K = 0, FWD_RESID = 1, FWD_LM = 2 };

constexpr int kLmStats = 28;  // e0, g[6], H upper triangle[21]
constexpr int kThreads = 256;

__host__ __device__ inline int pad2(int n) { return (n + 1) & ~1; }

struct FwdArgs {
  int X, Y, Z, C;
  const float2* mps;
  const float2* vols;
  i64 vol_stride;
  int shot0;
  const int* shot_off;
  const int* kx;
  const int* ky;
  const float2* ydat;
  float2* kout;  // offsets relative to shot_off[shot0], or absolute when kout_abs
  int kout_abs;
  int vps;       // volumes per shot (compile-time kernels, V = 1): vols holds [shot][vps] volumes
  i64 kout_vs;   // distance between the K regions of a shot's volumes
  double* partial;
  int XR, es;
  float scale, scale_lo;  // 1/sqrt(XY) and what its rounding to float left
  FftPlan plan;
};

template <int NV>
__device__ __forceinline__ void block_reduce_store(double (&v)[NV], double* out) {
  __shared__ double red[kThreads / 32][NV > 1 ? NV : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; k++) {
    double a = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) red[warp][k] = a;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double a = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) a += red[w][threadIdx.x];
    out[threadIdx.x] = a;
  }
}

struct AdjArgs {
  int X, Y, Z, C;
  const float2* mps;
  const float2* kin;
  int kin_rel;  // kin offsets relative to shot_off[shot0] (K workspace) or absolute (ydat)
  float2* out;
  i64 vol_stride;
  int shot0;
  const int* shot_off;
  const int* kx;
  const int* ky_off;
  const int* ky_order;  // may be null
  int XB, es;
  float scale, scale_lo;
  FftPlan plan;
};

// (a * b) mod n for 0 <= a, b < n <= 512 (product < 2^18: exact in float).
__device__ __forceinline__ int mulmod(int a, int b, int n, float inv_n) {
  const int p = a * b;
  int q = __float2int_rd((float)p * inv_n);
  int r = p - q * n;
  if (r < 0) r += n;
  if (r >= n) r -= n;
  return r;
}

// The H values of ROWS consecutive rows of one ky bin, H[x] = sum_i v_i st_i^(x - c): sample i's
// value v at the middle row c = ROWS / 2, its step st per row and, where CUBE, st^3 come from
// sample(i, v, st, st3).  Rows c + d and c - d take v st^d and
// v conj(st^d), which share their four products, so these are accumulated as products and combined
// once at the end: with the powers of st 4 instructions a row and sample where stepping v itself
// row by row takes 6 (and half as many steps in the chain).
// put(r, h) receives row r.
// With CUBE st^3 comes from the table and the higher powers from it: products of st alone bring the
// rounding of st to row c - d d times over (float32 walks of three samples a bin against 64 bits:
// 8 rows 7.9e-8 and, with st^3, 6.4e-8; 16 rows 1.15e-7 and 7.7e-8).
template <int ROWS, bool CUBE, class Sample, class Put>
__device__ __forceinline__ void h_rows(int lo, int hi, Sample sample, Put put) {
  constexpr int M = ROWS / 2;
  static_assert(ROWS >= 2 && ROWS % 2 == 0, "rows pair up around the middle");
  float2 h0 = make_float2(0.f, 0.f), hm = make_float2(0.f, 0.f);
  float a[M + 1], b[M + 1], c[M + 1], d[M + 1];  // sums of v.x w.x, v.y w.y, v.x w.y, v.y w.x at distance 1 .. M - 1
#pragma unroll
  for (int k = 1; k < M; k++) a[k] = b[k] = c[k] = d[k] = 0.f;
  for (int i = lo; i < hi; i++) {
    float2 v, st, st3;
    sample(i, v, st, st3);
    h0 = cadd(h0, v);
    auto add = [&](int k, float2 w) {
      a[k] = fmaf(v.x, w.x, a[k]);
      b[k] = fmaf(v.y, w.y, b[k]);
      c[k] = fmaf(v.x, w.y, c[k]);
      d[k] = fmaf(v.y, w.x, d[k]);
    };
    float2 w = st;  // st^k
    if constexpr (CUBE) {
      float2 p[M + 1];
      p[1] = st;
#pragma unroll
      for (int k = 2; k <= M; k++)
        p[k] = k == 2 ? cmulc(st3, st) : k == 3 ? st3 : cmul(st3, p[k - 3]);
#pragma unroll
      for (int k = 1; k < M; k++) add(k, p[k]);
      w = p[M];
    } else {
#pragma unroll
      for (int k = 1; k < M; k++) {
        add(k, w);
        w = cmul(w, st);
      }
    }
    // fused, the product rounds the running sum twice: too often where this is every second row
    if (M == 1) hm = cadd(hm, cmulc(v, w));
    else hm = cfmac(v, w, hm);
  }
  put(0, hm);
  put(M, h0);
#pragma unroll
  for (int k = 1; k < M; k++) {
    put(M + k, make_float2(a[k] - b[k], c[k] + d[k]));
    put(M - k, make_float2(a[k] + b[k], d[k] - c[k]));
  }
}

// The kernels on the run-time two-stage FFT (rt_sense.cu); -1 when ny has no such plan or the
// mode is not theirs (FWD_LM).
int try_rt_fwd(FwdArgs& A, int mode, int maxps, int nb, cudaStream_t st);
int try_rt_adj(AdjArgs& A, int maxps, int nb, cudaStream_t st);
bool has_rt_sense(int ny);

}  // namespace me
