// Line-pass kernels (see line_pass.cuh).  One CTA owns a tile of B lines of one volume, loads
// it into shared memory with coalesced accesses (rows of B consecutive lines along the
// contiguous axis, or whole contiguous lines), runs the FFT, the phase and the inverse FFT
// there, and writes the tile back.  Tiles are disjoint, so in == out is safe.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>

#include "pass_line.cuh"

namespace me {

ME_WAIT_FAULT_ACCESSOR(line_pass_wait_fault)

// The compile-time kernels handle every length in ME_FAST_LENGTHS; ME_GENERIC_FFT=1 in the
// environment forces the runtime-plan kernel for all lengths (used by the tests to cover it).
static bool fast_passes_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ME_GENERIC_FFT");
    v = (e && e[0] == '1') ? 0 : 1;
  }
  return v == 1;
}

// Global element offset of (line l, index n) inside a volume.
__device__ __forceinline__ i64 elem_offset(const PassArgs& A, int l, int n) {
  const int u = l / A.dims[A.av];
  const int v = l - u * A.dims[A.av];
  return (i64)u * A.st[A.au] + (i64)v * A.st[A.av] + (i64)n * A.st[A.ax];
}

__device__ __forceinline__ void line_coords(const PassArgs& A, int l, int n, int c[3]) {
  const int u = l / A.dims[A.av];
  const int v = l - u * A.dims[A.av];
  c[A.au] = u;
  c[A.av] = v;
  c[A.ax] = n;
}

// Load B lines (starting at line l0) of volume `src` into buf lines [dst_line0, dst_line0+B).
__device__ __forceinline__ void load_tile(const PassArgs& A, const float2* __restrict__ src,
                                          int l0, int nl, float2* buf, int dst_line0) {
  const int N = A.plan.n;
  const int B = A.B;
  if (A.st[A.av] == 1) {
    for (int t = threadIdx.x; t < B * N; t += blockDim.x) {
      const int b = t % B, n = t / B;
      float2 v = make_float2(0.f, 0.f);
      if (b < nl) v = src[elem_offset(A, l0 + b, n)];
      buf[n * A.es + dst_line0 + b] = v;
    }
  } else {
    for (int t = threadIdx.x; t < B * N; t += blockDim.x) {
      const int n = t % N, b = t / N;
      float2 v = make_float2(0.f, 0.f);
      if (b < nl) v = src[elem_offset(A, l0 + b, n)];
      buf[n * A.es + dst_line0 + b] = v;
    }
  }
}

__device__ __forceinline__ void store_tile(const PassArgs& A, float2* __restrict__ dst, int l0,
                                           int nl, const float2* buf, int src_line0, bool accum) {
  const int N = A.plan.n;
  const int B = A.B;
  const bool bfast = (A.st[A.av] == 1);
  for (int t = threadIdx.x; t < B * N; t += blockDim.x) {
    int b, n;
    if (bfast) {
      b = t % B;
      n = t / B;
    } else {
      n = t % N;
      b = t / N;
    }
    if (b >= nl) continue;
    const i64 off = elem_offset(A, l0 + b, n);
    float2 v = buf[n * A.es + src_line0 + b];
    if (accum) v = cadd(v, dst[off]);
    dst[off] = v;
  }
}

template <int MODE>
__global__ void __launch_bounds__(256) line_pass_kernel(const PassArgs A) {
  extern __shared__ float2 smem[];
  const int N = A.plan.n;
  const int vol = blockIdx.y;
  const int l0 = blockIdx.x * A.B;
  const int nl = min(A.B, A.nlines - l0);
  const int B = A.B;

  float2* tw = smem;
  float2* b0 = smem + ((N + 1) & ~1);
  float2* b1 = b0 + (i64)N * A.es;

  const double* prm = A.params ? A.params + (i64)vol * A.pstride : nullptr;
  PhaseCoef c0{0, 0, 0}, c1{0, 0, 0};
  if (prm) {
    c0 = phase_coef(A.ph[0], prm, A.ax);
    if (MODE == PM_DUAL_OUT || MODE == PM_DUAL_IN) c1 = phase_coef(A.ph[1], prm, A.ax);
  }
  const bool id0 = phase_is_identity(A.ph[0]);
  const bool id1 = phase_is_identity(A.ph[1]);

  init_twiddles(tw, N);
  const float2* in0 = A.in0 + (i64)vol * A.in_vs;
  load_tile(A, in0, l0, nl, b0, 0);
  if (MODE == PM_DUAL_IN) {
    const float2* in1 = A.in1 + (i64)vol * A.in_vs;
    load_tile(A, in1, l0, nl, b0, B);
  }
  __syncthreads();

  float2* R = b0;
  float2* S = b1;
  if (MODE != PM_INV) {
    const int nlines = (MODE == PM_DUAL_IN) ? 2 * B : B;
    R = fft_lines<false>(b0, b1, A.plan, nlines, A.es, tw);
    S = (R == b0) ? b1 : b0;
  }

  // phase multiply (and combine / split for the dual modes)
  for (int t = threadIdx.x; t < B * N; t += blockDim.x) {
    const int b = t % B, n = t / B;
    int c[3];
    line_coords(A, l0 + min(b, max(nl - 1, 0)), n, c);
    const float2 v0 = R[n * A.es + b];
    const float2 f0 = id0 ? make_float2(A.scale, 0.f) : phase_value(A.ph[0], c0, n, c, A.scale, A.scale_lo);
    if (MODE == PM_DUAL_OUT) {
      const float2 f1 = id1 ? make_float2(A.scale, 0.f) : phase_value(A.ph[1], c1, n, c, A.scale, A.scale_lo);
      R[n * A.es + b] = cmul(v0, f0);
      R[n * A.es + B + b] = cmul(v0, f1);
    } else if (MODE == PM_DUAL_IN) {
      const float2 f1 = id1 ? make_float2(A.scale, 0.f) : phase_value(A.ph[1], c1, n, c, A.scale, A.scale_lo);
      const float2 v1 = R[n * A.es + B + b];
      R[n * A.es + b] = cadd(cmul(v0, f0), cmul(v1, f1));
    } else {
      R[n * A.es + b] = cmul(v0, f0);
    }
  }
  __syncthreads();

  if (MODE != PM_FWD) {
    const int nlines = (MODE == PM_DUAL_OUT) ? 2 * B : B;
    R = fft_lines<true>(R, S, A.plan, nlines, A.es, tw);
  }

  float2* out0 = A.out0 + (i64)vol * A.out_vs;
  store_tile(A, out0, l0, nl, R, 0, A.accum != 0);
  if (MODE == PM_DUAL_OUT) {
    float2* out1 = A.out1 + (i64)vol * A.out_vs;
    store_tile(A, out1, l0, nl, R, B, false);
  }
}

// ------------------------------------------------------------------ compile-time lengths
// The pass for the compile-time lengths (pass_line.cuh): tiles of 16 lines, eight or sixteen
// threads a line, CTAs that are persistent over (volume, tile) work items and load the next tile
// while the current one is transformed.  The dual modes keep one buffer of two tiles (the
// next tile is then loaded after the current one is stored, and the other CTAs of the SM cover
// the load).
//
// What bounds it: instruction issue (DFTs, chirp, slot accesses) and, from 200 points on, DRAM.
// CTAs per SM it is compiled for: 16 warps of 128 registers, 20 of 96 at the shortest lengths.
constexpr int pass_min_ctas(int n, bool dual) { return n > 128 ? 2 : (dual || n > 64) ? 4 : 5; }

constexpr int pass_threads(int n) { return kTileLines * line_threads(n); }

// Coefficients of volume `vol`'s phases into shared memory when the CTA moves to another volume
// (uniform over the CTA, so the barrier is too); their last readers are past a barrier.
template <bool kDual>
__device__ __forceinline__ void set_coefs(const PassArgs& A, int vol, int& coef_vol,
                                          PhaseCoef* coef_s) {
  if (vol == coef_vol) return;
  if (threadIdx.x < (kDual ? 2 : 1)) {
    PhaseCoef cf{0, 0, 0};
    if (A.params) cf = phase_coef(A.ph[threadIdx.x], A.params + (i64)vol * A.pstride, A.ax);
    coef_s[threadIdx.x] = cf;
  }
  coef_vol = vol;
  __syncthreads();
}

// Tile staging by cp.async: any strides and alignments, and the plain FFT modes.
template <int N, int MODE>
__global__ void __launch_bounds__(pass_threads(N),
                                  pass_min_ctas(N, MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT))
    fast_pass_kernel(const __grid_constant__ PassArgs A) {
  constexpr int G = LineFft<N>::G, B = kTileLines;
  constexpr bool kDual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  constexpr int NT = kDual ? 2 : 1;    // tiles per buffer
  constexpr int NBUF = kDual ? 1 : 2;
  constexpr int PITCH = line_pitch(N), TILE = B * PITCH;
  extern __shared__ __align__(128) unsigned char tiles[];
  __shared__ i64 lb_s[2][B];  // line base offsets of the tile in each buffer
  __shared__ PhaseCoef coef_s[2];

  const int tiles_per_vol = (A.nlines + B - 1) / B;
  const int total = tiles_per_vol * A.nvol;
  const i64 sa = A.st[A.ax];
  const bool bfast = (A.st[A.av] == 1);
  const int dv = A.dims[A.av];
  int g, j;
  line_place<G>(g, j);
  __shared__ float2 chirp_s[kTileLines][2 * G];
  // this thread's line and first index when it copies: over the lines where they are neighbours
  // in memory, else along its own line
  const int cb = bfast ? threadIdx.x % B : threadIdx.x / G;
  const int cn = bfast ? threadIdx.x / B : threadIdx.x % G;
  Slots<G, false> s0, s1;
  s0.init(g, j);
  s1 = s0;

  auto line_base = [&](int l) {
    const int u = A.div_av.div(l);
    return (i64)u * A.st[A.au] + (i64)(l - u * dv) * A.st[A.av];
  };
  // issue the loads of work item t into buffer `bufi` (the caller has synchronised)
  auto issue = [&](int t, int bufi) {
    const int vol = A.div_tiles.div(t);
    const int l0 = (t - vol * tiles_per_vol) * B;
    const int nl = min(B, A.nlines - l0);
    if (threadIdx.x < B) lb_s[bufi][threadIdx.x] = line_base(l0 + min((int)threadIdx.x, nl - 1));
    const i64 base = line_base(l0 + min(cb, nl - 1));
#pragma unroll
    for (int k = 0; k < (MODE == PM_DUAL_IN ? 2 : 1); k++) {
      const float2* src = (k == 0 ? A.in0 : A.in1) + (i64)vol * A.in_vs + base;
      float2* dst = reinterpret_cast<float2*>(tiles + (bufi * NT + k) * TILE + cb * PITCH);
      for (int n = cn; n < N; n += G) {
        if (cb < nl) cp_async8(dst + n, src + n * sa);
        else dst[n] = make_float2(0.f, 0.f);
      }
    }
    cp_async_commit();
  };

  chain_next();
  chain_wait();
  int cur = 0, coef_vol = -1;
  if ((int)blockIdx.x < total) issue(blockIdx.x, 0);
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    const int vol = A.div_tiles.div(t);
    const int l0 = (t - vol * tiles_per_vol) * B;
    const int nl = min(B, A.nlines - l0);
    cp_async_wait_all();
    __syncthreads();
    if (NBUF == 2 && t + (int)gridDim.x < total) issue(t + gridDim.x, cur ^ 1);
    set_coefs<kDual>(A, vol, coef_vol, coef_s);
    const int l = l0 + min(g, nl - 1);
    const int u = A.div_av.div(l);
    s0.line = tiles + cur * NT * TILE + g * PITCH;
    s1.line = s0.line + TILE;
    pass_line<N, MODE>(A, coef_s, u, l - u * dv, j, s0, s1, chirp_s[g], [] {});
    __syncthreads();
#pragma unroll
    for (int k = 0; k < (MODE == PM_DUAL_OUT ? 2 : 1); k++) {
      if (cb >= nl) continue;
      float2* dst = (k == 0 ? A.out0 : A.out1) + (i64)vol * A.out_vs + lb_s[cur][cb];
      const bool acc = (k == 0) && A.accum;
      const float2* src = reinterpret_cast<const float2*>(tiles + (cur * NT + k) * TILE + cb * PITCH);
      for (int n = cn; n < N; n += G) {
        float2 v = src[n];
        if (acc) v = cadd(v, dst[n * sa]);
        dst[n * sa] = v;
      }
    }
    if (NBUF == 1) {
      __syncthreads();  // the store above has read the buffer the next tile goes into
      if (t + (int)gridDim.x < total) issue(t + gridDim.x, 0);
    } else {
      cur ^= 1;
    }
  }
  cp_async_wait_all();
}

// ------------------------------------------------------------------ tiles on the TMA engine
// The same pass with the tiles moved by the TMA engine, so that no thread issues per-element
// global loads or stores (loads complete on an mbarrier):
//   STRIDED (st[av] == 1): one tensor copy per tile and operand of up to 16 neighbouring lines of
//     a row, [n][16 lines] with the tensor map's 128-byte swizzle; lines past the row's end read
//     as zeros and are not written.  Needs base and strides that are multiples of 16 bytes.
//   else (st[ax] == 1): each of a tile's lines is one bulk copy, issued by a lane of its own, into
//     rows of line_pitch bytes.  Needs 16-byte aligned lines.
struct PassTma {
  CUtensorMap in[2];
  CUtensorMap out[2];
  int in_rank[2];   // 3: one volume (or a broadcast input), 4: indexed by volume
  int out_rank[2];
  FastDiv div_row;  // tiles per row of lines (strided)
  int row_tiles;
};

// Tile position of work item tt of a volume: the first line's coordinates, and the lines in it.
template <bool STRIDED>
__device__ __forceinline__ void tile_coords(const PassArgs& A, const FastDiv& div_row,
                                            int row_tiles, int tt, int& u, int& v0, int& nl) {
  if (STRIDED) {
    u = div_row.div(tt);
    v0 = (tt - u * row_tiles) * kTileLines;
    nl = min(kTileLines, A.dims[A.av] - v0);
  } else {
    const int l0 = tt * kTileLines;
    u = A.div_av.div(l0);
    v0 = l0 - u * A.dims[A.av];
    nl = min(kTileLines, A.nlines - l0);
  }
}

// Element offset of line b of a tile that starts at (u, v0) (contiguous lines; a tile may run
// over into the next rows of lines).
__device__ __forceinline__ i64 tile_line(const PassArgs& A, int u, int v0, int b) {
  const int l = u * A.dims[A.av] + v0 + b;
  const int ul = A.div_av.div(l);
  return (i64)ul * A.st[A.au] + (i64)(l - ul * A.dims[A.av]) * A.st[A.av];
}

template <int N, bool STRIDED>
struct TileShape {
  static constexpr int PITCH = line_pitch(N);
  static constexpr int TILE = STRIDED ? kTileLines * N * 8 : kTileLines * PITCH;
};

template <int N, int MODE, bool STRIDED>
__global__ void __launch_bounds__(pass_threads(N), pass_min_ctas(N, MODE != PM_SHEAR))
    tma_pass_kernel(const __grid_constant__ PassArgs A, const __grid_constant__ PassTma T) {
  constexpr int G = LineFft<N>::G;
  constexpr bool kDual = (MODE != PM_SHEAR);
  constexpr int NT = kDual ? 2 : 1;  // tiles per buffer
  constexpr int NBUF = kDual ? 1 : 2;
  constexpr int NIN = (MODE == PM_DUAL_IN) ? 2 : 1;
  constexpr int NOUT = (MODE == PM_DUAL_OUT) ? 2 : 1;
  constexpr int PITCH = TileShape<N, STRIDED>::PITCH, TILE = TileShape<N, STRIDED>::TILE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // the swizzle pattern repeats every 1024 bytes of shared-memory address
  unsigned char* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full[NBUF];
  __shared__ int4 place_s[NBUF];  // volume, u, v0 and lines of the tile in each buffer
  __shared__ PhaseCoef coef_s[2];

  const int tiles_per_vol = STRIDED ? T.row_tiles * A.dims[A.au] : (A.nlines + kTileLines - 1) / kTileLines;
  const int total = tiles_per_vol * A.nvol;
  int g, j;
  line_place<G>(g, j);
  __shared__ float2 chirp_s[kTileLines][2 * G];
  Slots<G, STRIDED> s0, s1;
  s0.init(g, j);
  s1 = s0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < NBUF; i++) mbar_init(&full[i], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // warp 0: load work item t into buffer bufi, once the stores out of that buffer have read it
  auto issue = [&](int t, int bufi) {
    const int vol = A.div_tiles.div(t);
    int u, v0, nl;
    tile_coords<STRIDED>(A, T.div_row, T.row_tiles, t - vol * tiles_per_vol, u, v0, nl);
    bulk_wait_read_all();
    fence_proxy_async_smem();
    __syncwarp();
    if (threadIdx.x == 0) {
      place_s[bufi] = make_int4(vol, u, v0, nl);  // released with the arrival
      mbar_arrive_expect_tx(&full[bufi], NIN * (STRIDED ? TILE : nl * N * 8));
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NIN; k++) {
      unsigned char* dst = tiles + (bufi * NT + k) * TILE;
      if (STRIDED) {
        if (threadIdx.x == 0) {
          if (T.in_rank[k] == 3) tma_load_3d(dst, &T.in[k], v0, 0, u, &full[bufi]);
          else tma_load_4d(dst, &T.in[k], v0, 0, u, vol, &full[bufi]);
        }
      } else if ((int)threadIdx.x < nl) {
        bulk_g2s(dst + threadIdx.x * PITCH,
                 (k == 0 ? A.in0 : A.in1) + (i64)vol * A.in_vs + tile_line(A, u, v0, threadIdx.x),
                 N * 8, &full[bufi]);
      }
    }
  };

  const bool mover = threadIdx.x < 32;
  chain_next();
  chain_wait();
  if (mover && (int)blockIdx.x < total) issue(blockIdx.x, 0);
  __syncthreads();  // a wait that gives up must still find the tile's place
  int coef_vol = -1;
  int it = 0;
  for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
    const int cur = (NBUF == 2) ? (it & 1) : 0;
    const unsigned parity = (NBUF == 2) ? ((it >> 1) & 1) : (it & 1);
    mbar_wait_bounded(&full[cur], parity, WF_LINE_PASS);
    const int4 place = place_s[cur];
    const int vol = place.x, u = place.y, v0 = place.z, nl = place.w;
    // (the barrier before the previous tile's store separates every read of coef_s from a write)
    set_coefs<kDual>(A, vol, coef_vol, coef_s);
    int ul = u, vl = v0 + min(g, nl - 1);
    if (!STRIDED && v0 + kTileLines > A.dims[A.av]) {  // the tile runs over into the next rows
      const int l = u * A.dims[A.av] + vl;
      ul = A.div_av.div(l);
      vl = l - ul * A.dims[A.av];
    }
    s0.line = tiles + cur * NT * TILE + (STRIDED ? 0 : g * PITCH);
    s1.line = s0.line + TILE;
    // The next tile goes into the buffer that the previous tile is being stored from.  By the end
    // of the first stage the store has read it; asked for earlier, warp 0 waits for that while
    // the other warps come to wait for it at the tile's end.
    pass_line<N, MODE>(A, coef_s, ul, vl, j, s0, s1, chirp_s[g], [&] {
      if (NBUF == 2 && mover && t + (int)gridDim.x < total) issue(t + gridDim.x, cur ^ 1);
    });
    // the tile's generic-proxy writes are ordered before the async-proxy store
    fence_proxy_async_smem();
    __syncthreads();
    if (mover) {
#pragma unroll
      for (int k = 0; k < NOUT; k++) {
        const unsigned char* src = tiles + (cur * NT + k) * TILE;
        if (STRIDED) {
          if (threadIdx.x == 0) {
            if (T.out_rank[k] == 3) tma_store_3d(&T.out[k], src, v0, 0, u);
            else tma_store_4d(&T.out[k], src, v0, 0, u, vol);
          }
        } else if ((int)threadIdx.x < nl) {
          bulk_s2g((k == 0 ? A.out0 : A.out1) + (i64)vol * A.out_vs + tile_line(A, u, v0, threadIdx.x),
                   src + threadIdx.x * PITCH, N * 8);
        }
      }
      bulk_commit();
      if (NBUF == 1 && t + (int)gridDim.x < total) issue(t + gridDim.x, 0);
    }
  }
  if (mover) bulk_wait_all();
}

// ME_NO_TMA=1 in the environment keeps every pass on the cp.async kernel (for comparisons).
static bool tma_passes_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("ME_NO_TMA");
    v = (e && e[0] == '1') ? 0 : 1;
  }
  return v == 1;
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor map of one operand of a strided TMA pass (8-byte elements, boxes of 16 lines); rank 3
// when the operand is one volume, else rank 4 with the volume index outermost.
static bool encode_pass_map(CUtensorMap* m, const void* base, const PassArgs& A, i64 vs, int rank) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)A.dims[A.av], (cuuint64_t)A.dims[A.ax],
                              (cuuint64_t)A.dims[A.au], (cuuint64_t)A.nvol};
  const cuuint64_t strides[3] = {(cuuint64_t)A.st[A.ax] * 8, (cuuint64_t)A.st[A.au] * 8,
                                 (cuuint64_t)vs * 8};
  const cuuint32_t box[4] = {kTileLines, (cuuint32_t)A.dims[A.ax], 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT64, (cuuint32_t)rank,
                         const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Whether pass A can run on the TMA kernel, and then how: strided or contiguous lines, the
// tensor maps of the former.  All strides have to be even (16 bytes) and all bases aligned.
static bool tma_pass_setup(int mode, const PassArgs& A, bool* strided, PassTma* T) {
  if (!tma_passes_enabled()) return false;
  if (mode != PM_SHEAR && mode != PM_DUAL_OUT && mode != PM_DUAL_IN) return false;
  if (A.accum) return false;
  const bool s = (A.st[A.av] == 1);
  if (!s && A.st[A.ax] != 1) return false;
  const i64 other = s ? A.st[A.ax] : A.st[A.av];
  if (other % 2 != 0 || A.st[A.au] % 2 != 0) return false;
  const i64 lim = (i64)1 << 36;  // strides below 2^40 bytes
  if (other >= lim || A.st[A.au] >= lim || A.in_vs >= lim || A.out_vs >= lim) return false;
  // A row's last tile may hold a few lines only and the tensor copy is still the better one (ten passes
  // of 128 x Y x 96, cp.async and TMA: Y = 18 89 and 68 us, 24 97 and 76, 30 95 and 73; 16
  // volumes, Y = 18 349 and 337 us, 24 466 and 403, 30 488 and 371).  Rows shorter than a tile
  // would be padding in every tile.
  if (s && A.dims[A.av] < kTileLines) return false;
  const int nin = (mode == PM_DUAL_IN) ? 2 : 1, nout = (mode == PM_DUAL_OUT) ? 2 : 1;
  const float2* ins[2] = {A.in0, A.in1};
  float2* outs[2] = {A.out0, A.out1};
  for (int k = 0; k < nin; k++) {
    if ((uintptr_t)ins[k] % 16 != 0) return false;
    const bool one = (A.in_vs == 0 || A.nvol == 1);
    if (!one && A.in_vs % 2 != 0) return false;
    T->in_rank[k] = one ? 3 : 4;
    if (s && !encode_pass_map(&T->in[k], ins[k], A, A.in_vs, T->in_rank[k])) return false;
  }
  for (int k = 0; k < nout; k++) {
    if ((uintptr_t)outs[k] % 16 != 0) return false;
    const bool one = (A.nvol == 1);
    if (!one && A.out_vs % 2 != 0) return false;
    T->out_rank[k] = one ? 3 : 4;
    if (s && !encode_pass_map(&T->out[k], outs[k], A, A.out_vs, T->out_rank[k])) return false;
  }
  T->row_tiles = s ? (A.dims[A.av] + kTileLines - 1) / kTileLines : 1;
  T->div_row.set(T->row_tiles);
  *strided = s;
  return true;
}

// Work items of a volume.
static int tiles_of(const PassArgs& A, bool strided_tma) {
  return strided_tma ? (A.dims[A.av] + kTileLines - 1) / kTileLines * A.dims[A.au]
                     : (A.nlines + kTileLines - 1) / kTileLines;
}

// Persistent grid of a kernel: all resident CTAs, or fewer where there are fewer tiles.  `occ`
// keeps the device's resident CTAs for the kernel (one launch shape per instantiation).
template <typename K>
static int pass_grid(K kern, int threads, size_t smem, long long tiles, std::atomic<int> (&occ)[8]) {
  int dev = 0;
  cudaGetDevice(&dev);
  int res = dev < 8 ? occ[dev].load(std::memory_order_relaxed) : 0;
  if (res == 0) {
    int nb = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, threads, smem);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    res = std::max(1, nb) * std::max(1, sms);
    if (dev < 8) occ[dev].store(res, std::memory_order_relaxed);
  }
  return (int)std::min<long long>(tiles, res);
}

template <int N, int MODE, bool STRIDED>
static int launch_tma(PassArgs& A, const PassTma& T, cudaStream_t stream) {
  const size_t smem = 1024 + 2 * (size_t)TileShape<N, STRIDED>::TILE;
  const int tiles = tiles_of(A, STRIDED);
  A.div_tiles.set(tiles);
  auto kern = tma_pass_kernel<N, MODE, STRIDED>;
  const int rc = check_cuda(allow_smem(kern, smem), "tma pass smem");
  if (rc != ME_OK) return rc;
  static std::atomic<int> occ[8];
  const int grid = pass_grid(kern, pass_threads(N), smem, (long long)tiles * A.nvol, occ);
  count_launch();
  return check_cuda(launch_chained(grid == (long long)tiles * A.nvol, kern, grid, pass_threads(N),
                                   smem, stream, A, T),
                    "tma pass launch");
}

template <int N, int MODE>
static int launch_fast(PassArgs& A, cudaStream_t stream) {
  if constexpr (MODE == PM_SHEAR || MODE == PM_DUAL_OUT || MODE == PM_DUAL_IN) {
    PassTma T;
    bool strided = false;
    if (tma_pass_setup(MODE, A, &strided, &T))
      return strided ? launch_tma<N, MODE, true>(A, T, stream)
                     : launch_tma<N, MODE, false>(A, T, stream);
  }
  const size_t smem = 2 * (size_t)kTileLines * line_pitch(N);
  const int tiles = tiles_of(A, false);
  A.div_tiles.set(tiles);
  auto kern = fast_pass_kernel<N, MODE>;
  const int rc = check_cuda(allow_smem(kern, smem), "pass smem");
  if (rc != ME_OK) return rc;
  static std::atomic<int> occ[8];
  const int grid = pass_grid(kern, pass_threads(N), smem, (long long)tiles * A.nvol, occ);
  count_launch();
  return check_cuda(launch_chained(grid == (long long)tiles * A.nvol, kern, grid, pass_threads(N),
                                   smem, stream, A),
                    "fast pass launch");
}

template <int N>
static int launch_fast_mode(int mode, PassArgs& A, cudaStream_t stream) {
  switch (mode) {
    case PM_SHEAR: return launch_fast<N, PM_SHEAR>(A, stream);
    case PM_DUAL_OUT: return launch_fast<N, PM_DUAL_OUT>(A, stream);
    case PM_DUAL_IN: return launch_fast<N, PM_DUAL_IN>(A, stream);
    case PM_FWD: return launch_fast<N, PM_FWD>(A, stream);
    default: return launch_fast<N, PM_INV>(A, stream);
  }
}

// Returns ME_OK / error if handled by a compile-time kernel, -1 if N has no such kernel.
static int try_fast(int mode, PassArgs& A, cudaStream_t stream) {
  switch (A.plan.n) {
#define ME_FAST_CASE(N) \
  case N: return launch_fast_mode<N>(mode, A, stream);
    ME_FAST_LENGTHS(ME_FAST_CASE)
#undef ME_FAST_CASE
    default: return -1;
  }
}

static int pick_B(int N) {
  int B = 16;
  while (B > 4 && N * B > 4096) B /= 2;
  return B;
}

template <int MODE>
static int launch_mode(PassArgs& A, cudaStream_t stream) {
  const int N = A.plan.n;
  const bool dual = (MODE == PM_DUAL_IN || MODE == PM_DUAL_OUT);
  A.es = (dual ? 2 * A.B : A.B) + 1;
  const size_t smem = sizeof(float2) * (((N + 1) & ~1) + 2 * (size_t)N * A.es);
  {
    const int rc = check_cuda(allow_smem(line_pass_kernel<MODE>, smem), "line_pass smem");
    if (rc != ME_OK) return rc;
  }
  dim3 grid((A.nlines + A.B - 1) / A.B, A.nvol);
  count_launch();
  line_pass_kernel<MODE><<<grid, 256, smem, stream>>>(A);
  return check_cuda(cudaGetLastError(), "line_pass launch");
}

int make_pass_args(int mode, const float2* in0, const float2* in1, float2* out0, float2* out1,
                   i64 in_vs, i64 out_vs, int nvol, const int dims[3], const i64 st[3], int axis,
                   const Phase& f0, const Phase& f1, const double* params, int pstride, int accum,
                   PassArgs* out) {
  if (axis < 0 || axis > 2) return fail("line pass: axis must be 0, 1 or 2");
  PassArgs A{};
  A.in0 = in0;
  A.in1 = in1;
  A.out0 = out0;
  A.out1 = out1;
  A.in_vs = in_vs;
  A.out_vs = out_vs;
  A.nvol = nvol;
  for (int i = 0; i < 3; i++) {
    A.dims[i] = dims[i];
    A.st[i] = st[i];
  }
  A.ax = axis;
  int o1 = (axis + 1) % 3, o2 = (axis + 2) % 3;
  // av: the other axis with the smaller stride (the coalescing axis)
  if (st[o1] <= st[o2]) {
    A.av = o1;
    A.au = o2;
  } else {
    A.av = o2;
    A.au = o1;
  }
  A.nlines = dims[A.au] * dims[A.av];
  A.div_av.set(dims[A.av]);
  const int N = dims[axis];
  if (N > ME_MAX_LINE) return fail("line pass: line length exceeds ME_MAX_LINE");
  if (!make_plan(N, &A.plan)) {
    set_error("line pass: line length has a prime factor > 13");
    return ME_ERR_UNSUPPORTED;
  }
  A.B = pick_B(N);
  A.accum = accum;
  A.params = params;
  A.pstride = pstride;
  A.ph[0] = f0;
  A.ph[1] = f1;
  const double gain = N * (fast_passes_enabled() ? fft_pair_gain(N) : 1.0);
  const bool pair = mode == PM_SHEAR || mode == PM_DUAL_OUT || mode == PM_DUAL_IN;
  const double scale = pair ? 1.0 / gain : 1.0 / sqrt(gain);
  A.scale = (float)scale;
  A.scale_lo = (float)(scale - (double)A.scale);
  *out = A;
  return ME_OK;
}

int launch_line_pass(int mode, const float2* in0, const float2* in1, float2* out0, float2* out1,
                     i64 in_vs, i64 out_vs, int nvol, const int dims[3], const i64 st[3], int axis,
                     const Phase& f0, const Phase& f1, const double* params, int pstride,
                     int accum, cudaStream_t stream) {
  if (axis < 0 || axis > 2) return fail("line pass: axis must be 0, 1 or 2");
  if (nvol < 1) return ME_OK;
  PassArgs A;
  const int rc0 = make_pass_args(mode, in0, in1, out0, out1, in_vs, out_vs, nvol, dims, st, axis,
                                 f0, f1, params, pstride, accum, &A);
  if (rc0 != ME_OK) return rc0;
  if (A.nlines == 0) return ME_OK;
  if (fast_passes_enabled()) {
    int rc = try_fast(mode, A, stream);
    if (rc < 0) rc = try_rt_pass(mode, A, stream);
    if (rc >= 0) return rc;
  }
  switch (mode) {
    case PM_SHEAR: return launch_mode<PM_SHEAR>(A, stream);
    case PM_DUAL_OUT: return launch_mode<PM_DUAL_OUT>(A, stream);
    case PM_DUAL_IN: return launch_mode<PM_DUAL_IN>(A, stream);
    case PM_FWD: return launch_mode<PM_FWD>(A, stream);
    case PM_INV: return launch_mode<PM_INV>(A, stream);
    default: return fail("line pass: bad mode");
  }
}

// ------------------------------------------------------------------ several jobs in one launch
// One shear step (PM_SHEAR) of several independent jobs -- volumes of different
// reconstructions, of any sizes -- as one persistent launch per distinct line length along the
// step's axis.  Work items are (job, volume, tile of lines) over the jobs of that length; each
// CTA takes items in turn and runs them through the compile-time tile code of the length, the
// same arithmetic as fast_pass_kernel, so the results are bit-identical to separate launches.
// Two tile buffers per CTA: the next item, of whichever job, is loaded while the current one is
// transformed.  (A single launch that switched between the sixteen compiled lengths would carry
// all their register needs at once.)
struct MultiPassArgs {
  int njobs;
  int tile_off[kMaxMultiJobs + 1];  // prefix sums of the jobs' work items
  PassArgs job[kMaxMultiJobs];
};

template <int N>
__global__ void __launch_bounds__(pass_threads(N), pass_min_ctas(N, false))
    multi_shear_kernel(const __grid_constant__ MultiPassArgs M) {
  constexpr int G = LineFft<N>::G, B = kTileLines;
  constexpr int PITCH = line_pitch(N), TILE = B * PITCH;
  extern __shared__ __align__(128) unsigned char tiles[];
  __shared__ PhaseCoef coef_s[2];
  const int total = M.tile_off[M.njobs];
  int g, j;
  line_place<G>(g, j);
  __shared__ float2 chirp_s[kTileLines][2 * G];
  Slots<G, false> s0;
  s0.init(g, j);
  auto job_of = [&](int t) {
    int k = 0;
    while (k + 1 < M.njobs && t >= M.tile_off[k + 1]) k++;
    return k;
  };
  // a work item's volume, first line and lines, and this thread's place when it copies
  struct Item {
    int vol, l0, nl, cb, cn;
    i64 base;
  };
  auto item = [&](const PassArgs& A, int tt) {
    Item I;
    const int tiles_per_vol = (A.nlines + B - 1) / B;
    I.vol = A.div_tiles.div(tt);
    I.l0 = (tt - I.vol * tiles_per_vol) * B;
    I.nl = min(B, A.nlines - I.l0);
    const bool bfast = (A.st[A.av] == 1);
    I.cb = bfast ? threadIdx.x % B : threadIdx.x / G;
    I.cn = bfast ? threadIdx.x / B : threadIdx.x % G;
    const int l = I.l0 + min(I.cb, I.nl - 1);
    const int u = A.div_av.div(l);
    I.base = (i64)u * A.st[A.au] + (i64)(l - u * A.dims[A.av]) * A.st[A.av];
    return I;
  };
  // issue the loads of work item t into buffer `bufi` (the caller has synchronised)
  auto issue = [&](int t, int bufi) {
    const int k = job_of(t);
    const PassArgs& A = M.job[k];
    const Item I = item(A, t - M.tile_off[k]);
    const i64 sa = A.st[A.ax];
    const float2* src = A.in0 + (i64)I.vol * A.in_vs + I.base;
    float2* dst = reinterpret_cast<float2*>(tiles + bufi * TILE + I.cb * PITCH);
    for (int n = I.cn; n < N; n += G) {
      if (I.cb < I.nl) cp_async8(dst + n, src + n * sa);
      else dst[n] = make_float2(0.f, 0.f);
    }
    cp_async_commit();
  };

  int cur = 0, coef_job = -1, coef_vol = -1;
  if ((int)blockIdx.x < total) issue(blockIdx.x, 0);
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    const int k = job_of(t);
    const PassArgs& A = M.job[k];
    const Item I = item(A, t - M.tile_off[k]);
    cp_async_wait_all();
    __syncthreads();
    if (t + (int)gridDim.x < total) issue(t + gridDim.x, cur ^ 1);
    if (k != coef_job) coef_vol = -1;
    coef_job = k;
    set_coefs<false>(A, I.vol, coef_vol, coef_s);
    const int l = I.l0 + min(g, I.nl - 1);
    const int u = A.div_av.div(l);
    s0.line = tiles + cur * TILE + g * PITCH;
    pass_line<N, PM_SHEAR>(A, coef_s, u, l - u * A.dims[A.av], j, s0, s0, chirp_s[g], [] {});
    __syncthreads();
    if (I.cb < I.nl) {
      const i64 sa = A.st[A.ax];
      float2* dst = A.out0 + (i64)I.vol * A.out_vs + I.base;
      const float2* src = reinterpret_cast<const float2*>(tiles + cur * TILE + I.cb * PITCH);
      for (int n = I.cn; n < N; n += G) dst[n * sa] = src[n];
    }
    cur ^= 1;
  }
  cp_async_wait_all();
}

// The multi-job shear step on TMA tiles: the tiles of every job move as in tma_pass_kernel,
// through each job's own tensor maps.  Used when every job of the launch qualifies for
// tma_pass_kernel with the same tile layout (all strided or all contiguous, as the jobs of one
// shear step in the same volume layout are).
struct MultiTmaJob {
  CUtensorMap in;
  CUtensorMap out;
  int in_rank, out_rank;
  FastDiv div_row;
  int row_tiles;
};

struct MultiTmaArgs {
  int njobs;
  int tile_off[kMaxMultiJobs + 1];
  PassArgs job[kMaxMultiJobs];
  MultiTmaJob tm[kMaxMultiJobs];
};

template <int N, bool STRIDED>
__global__ void __launch_bounds__(pass_threads(N), pass_min_ctas(N, false))
    tma_multi_shear_kernel(const __grid_constant__ MultiTmaArgs M) {
  constexpr int G = LineFft<N>::G;
  constexpr int PITCH = TileShape<N, STRIDED>::PITCH, TILE = TileShape<N, STRIDED>::TILE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* tiles = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int4 place_s[2];  // volume, u, v0 and lines of the tile in each buffer
  __shared__ int job_s[2];
  __shared__ PhaseCoef coef_s[2];
  const int total = M.tile_off[M.njobs];
  int g, j;
  line_place<G>(g, j);
  __shared__ float2 chirp_s[kTileLines][2 * G];
  Slots<G, STRIDED> s0;
  s0.init(g, j);
  if (threadIdx.x == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto job_of = [&](int t) {
    int k = 0;
    while (k + 1 < M.njobs && t >= M.tile_off[k + 1]) k++;
    return k;
  };
  auto coords = [&](int k, int t, int& vol, int& u, int& v0, int& nl) {
    const PassArgs& A = M.job[k];
    const MultiTmaJob& J = M.tm[k];
    const int per_vol = STRIDED ? J.row_tiles * A.dims[A.au] : (A.nlines + kTileLines - 1) / kTileLines;
    const int tt = t - M.tile_off[k];
    vol = A.div_tiles.div(tt);
    tile_coords<STRIDED>(A, J.div_row, J.row_tiles, tt - vol * per_vol, u, v0, nl);
  };
  // warp 0: load work item t into buffer bufi, once the stores out of that buffer have read it
  auto issue = [&](int t, int bufi) {
    const int k = job_of(t);
    int vol, u, v0, nl;
    coords(k, t, vol, u, v0, nl);
    const PassArgs& A = M.job[k];
    const MultiTmaJob& J = M.tm[k];
    bulk_wait_read_all();
    fence_proxy_async_smem();
    __syncwarp();
    if (threadIdx.x == 0) {
      place_s[bufi] = make_int4(vol, u, v0, nl);  // released with the arrival
      job_s[bufi] = k;
      mbar_arrive_expect_tx(&full[bufi], STRIDED ? TILE : nl * N * 8);
    }
    __syncwarp();
    unsigned char* dst = tiles + bufi * TILE;
    if (STRIDED) {
      if (threadIdx.x == 0) {
        if (J.in_rank == 3) tma_load_3d(dst, &J.in, v0, 0, u, &full[bufi]);
        else tma_load_4d(dst, &J.in, v0, 0, u, vol, &full[bufi]);
      }
    } else if ((int)threadIdx.x < nl) {
      bulk_g2s(dst + threadIdx.x * PITCH,
               A.in0 + (i64)vol * A.in_vs + tile_line(A, u, v0, threadIdx.x), N * 8, &full[bufi]);
    }
  };

  const bool mover = threadIdx.x < 32;
  if (mover && (int)blockIdx.x < total) issue(blockIdx.x, 0);
  __syncthreads();  // a wait that gives up must still find the tile's place
  int coef_job = -1, coef_vol = -1;
  int it = 0;
  for (int t = blockIdx.x; t < total; t += gridDim.x, it++) {
    const int cur = it & 1;
    mbar_wait_bounded(&full[cur], (it >> 1) & 1, WF_LINE_PASS);
    const int4 place = place_s[cur];
    const int vol = place.x, u = place.y, v0 = place.z, nl = place.w;
    const int k = job_s[cur];
    const PassArgs& A = M.job[k];
    const MultiTmaJob& J = M.tm[k];
    if (k != coef_job) coef_vol = -1;
    coef_job = k;
    set_coefs<false>(A, vol, coef_vol, coef_s);
    int ul = u, vl = v0 + min(g, nl - 1);
    if (!STRIDED && v0 + kTileLines > A.dims[A.av]) {  // the tile runs over into the next rows
      const int l = u * A.dims[A.av] + vl;
      ul = A.div_av.div(l);
      vl = l - ul * A.dims[A.av];
    }
    unsigned char* tb = tiles + cur * TILE;
    s0.line = tb + (STRIDED ? 0 : g * PITCH);
    pass_line<N, PM_SHEAR>(A, coef_s, ul, vl, j, s0, s0, chirp_s[g], [&] {
      if (mover && t + (int)gridDim.x < total) issue(t + gridDim.x, cur ^ 1);
    });
    fence_proxy_async_smem();
    __syncthreads();
    if (mover) {
      if (STRIDED) {
        if (threadIdx.x == 0) {
          if (J.out_rank == 3) tma_store_3d(&J.out, tb, v0, 0, u);
          else tma_store_4d(&J.out, tb, v0, 0, u, vol);
        }
      } else if ((int)threadIdx.x < nl) {
        bulk_s2g(A.out0 + (i64)vol * A.out_vs + tile_line(A, u, v0, threadIdx.x),
                 tb + threadIdx.x * PITCH, N * 8);
      }
      bulk_commit();
    }
  }
  if (mover) bulk_wait_all();
}

template <typename K, typename M>
static int launch_multi_kernel(K kern, const M& args, int threads, size_t smem, cudaStream_t stream) {
  const int rc = check_cuda(allow_smem(kern, smem), "multi shear smem");
  if (rc != ME_OK) return rc;
  int dev = 0, sms = 148, nb = 2;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, threads, smem);
  const int total = args.tile_off[args.njobs];
  const int grid = (int)std::min<long long>(total, (long long)std::max(1, nb) * sms);
  count_launch();
  kern<<<grid, threads, smem, stream>>>(args);
  return check_cuda(cudaGetLastError(), "multi shear launch");
}

template <int N, bool STRIDED>
static int launch_tma_multi_n(const MultiTmaArgs& M, cudaStream_t stream) {
  return launch_multi_kernel(tma_multi_shear_kernel<N, STRIDED>, M, pass_threads(N),
                             1024 + 2 * (size_t)TileShape<N, STRIDED>::TILE, stream);
}

template <int N>
static int launch_multi_n(const MultiPassArgs& M, cudaStream_t stream) {
  return launch_multi_kernel(multi_shear_kernel<N>, M, pass_threads(N),
                             2 * (size_t)kTileLines * line_pitch(N), stream);
}

static bool fast_length(int n) {
  switch (n) {
#define ME_FAST_IS(N) \
  case N: return true;
    ME_FAST_LENGTHS(ME_FAST_IS)
#undef ME_FAST_IS
    default: return false;
  }
}

int launch_multi_shear(const PassArgs* jobs, int njobs, cudaStream_t stream) {
  if (njobs < 1) return ME_OK;
  if (njobs > kMaxMultiJobs) return fail("multi shear: too many jobs in one launch");
  for (int k = 0; k < njobs; k++)
    if (!fast_length(jobs[k].plan.n)) {
      set_error("multi shear: a job's line length has no compile-time FFT");
      return ME_ERR_UNSUPPORTED;
    }
  // one launch per distinct line length, over the jobs of that length in job order
  bool done[kMaxMultiJobs] = {false};
  for (int k0 = 0; k0 < njobs; k0++) {
    if (done[k0]) continue;
    const int n = jobs[k0].plan.n;
    MultiPassArgs M;
    MultiTmaArgs MT;
    M.njobs = 0;
    // on TMA tiles when every job of this length qualifies
    bool tma = true, strided = true;
    for (int k = k0; k < njobs; k++) {
      if (done[k] || jobs[k].plan.n != n) continue;
      done[k] = true;
      const int q = M.njobs++;
      M.job[q] = jobs[k];
      PassTma T;
      bool s = false;
      tma = tma && tma_pass_setup(PM_SHEAR, jobs[k], &s, &T);
      if (!tma) continue;
      if (q == 0) strided = s;
      tma = (s == strided);
      MT.tm[q].in = T.in[0];
      MT.tm[q].out = T.out[0];
      MT.tm[q].in_rank = T.in_rank[0];
      MT.tm[q].out_rank = T.out_rank[0];
      MT.tm[q].div_row = T.div_row;
      MT.tm[q].row_tiles = T.row_tiles;
    }
    long long total = 0;
    M.tile_off[0] = 0;
    for (int q = 0; q < M.njobs; q++) {
      const int tiles = tiles_of(M.job[q], tma && strided);
      total += (long long)tiles * M.job[q].nvol;
      if (total > 0x7fffffffLL) return fail("multi shear: too many work items");
      M.job[q].div_tiles.set(std::max(1, tiles));
      M.tile_off[q + 1] = (int)total;
    }
    if (total == 0) continue;
    if (tma) {
      MT.njobs = M.njobs;
      for (int q = 0; q < M.njobs; q++) MT.job[q] = M.job[q];
      for (int q = 0; q <= M.njobs; q++) MT.tile_off[q] = M.tile_off[q];
    }
    int rc = -1;
    switch (n) {
#define ME_MULTI_LAUNCH(N)                                             \
  case N:                                                                      \
    rc = !tma ? launch_multi_n<N>(M, stream)                               \
         : strided ? launch_tma_multi_n<N, true>(MT, stream)               \
                   : launch_tma_multi_n<N, false>(MT, stream);             \
    break;
      ME_FAST_LENGTHS(ME_MULTI_LAUNCH)
#undef ME_MULTI_LAUNCH
      default: break;
    }
    if (rc != ME_OK) return rc < 0 ? fail("multi shear: unsupported length") : rc;
  }
  return ME_OK;
}

}  // namespace me
