// Goldstein phase filter on sm_100a.
//
// Replaces goldstein_filter_cuda_host and its kernels (extract_patches,
// cuFFT forward, gaussian_filter, patchwise_normalize, spectrum_enhancement,
// cuFFT inverse, batched_overlap_add, normalize_output), reference
// csrc/src/goldstein.cu:87-408, with two kernels:
//   1. goldstein_run_kernel -- one warp per run of 1 to 8 vertically
//      neighbouring 32x32 patches.  Per patch: coalesced load, 2-D FFT as
//      32-point radix-2 FFTs held in registers (columns, then rows through a
//      padded shared tile), |F|, 7x7 circular smoothing, patch-mean
//      normalisation, S^alpha weighting, inverse 2-D FFT, triangular weight
//      and 1/n^2 scale; rows add up over the run in shared memory and leave
//      for the scratch once no later patch of the run reaches them.
//   2. goldstein_gather_kernel -- each output pixel sums the runs covering it
//      (4 columns by 1 or 2 runs where runs are long) in a fixed order and
//      divides by the summed weights.  No atomics: the result is
//      deterministic.
//
// 3217 x 1391 samples (68 400 patches): 318 us in kernel 1 and 62 us in kernel
// 2, against 405 and 184 with single patches as the unit.  Kernel 1 is bound
// by instruction issue and the FP32 pipe together (3000 instructions a patch,
// 58 % of the issue slots, packed FP32 instructions for two slots of the pipe
// each), kernel 2 by the latency of its loads from L2 and memory.  Against the
// former unit: the runs cut the scratch traffic from 8 KB a patch each way to
// 2.8 KB; columns first, so that loads, sums and stores are coalesced without a
// transpose (two per patch, not four); one copy of the FFT's code for the four
// transforms (unrolled four times, a fifth of the issue slots waited for the
// instruction cache); multiplications folded into the butterflies' additions;
// the patch mean from |F|, so that smoothed values are not kept.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "s1b.h"
#include "s1b_ctx_cache.h"
#include "s1b_device.cuh"
#include "s1b_frame.h"
#include "s1b_internal.h"

namespace {

constexpr int GN = 32;        // patch size (s1proc filter.window_size)
constexpr int GSTEP = GN / 4; // patch step, goldstein.cu:334
// One warp per CTA, so that the run's addresses are uniform: 394 us per
// 3217 x 1391 image against 405 with two.  12 CTAs per SM: 168 registers (the
// 32 complex values of a transform and the 32 magnitudes) and 17 KB of shared
// memory each.
constexpr int GCTAS_PER_SM = 12;
// Patches of the longest run, and how many runs an image has at least before
// its runs are made longer: a wave of one-warp CTAs.  Longer runs save scratch
// traffic, but a patch of a run waits for the one before it: 1217 x 391 samples
// (6850 patches) take 53 us in runs of 2 and 68 in runs of 8; 3217 x 1391 394
// in runs of 8 and 418 in runs of 16.
constexpr int GRUN_MAX = 8;
constexpr int GRUN_JOBS = 148 * GCTAS_PER_SM;
// Gathering: columns of a CTA, and output pixels from which a thread takes
// eight rows (columns and weights found once) instead of one (more loads in
// flight): 387 us against 394 at 3217 x 1391, 59 against 53 at 1217 x 391, 46
// against 33 at 430 x 470.
constexpr int GGATHER = 256;
constexpr int64_t kGatherRows8 = 1 << 20;

// cos(pi k / 16) and tan(pi k / 16), k = 0..4, evaluated in 50-digit decimal
// arithmetic: a rotation exp(-pi i k / 16) is taken as the larger of its
// cosine and sine times a shear by the tangent or cotangent (at most 1).
constexpr float kCos[5] = {1.0f, 0.9807852804032304f, 0.9238795325112867f, 0.8314696123025452f, 0.7071067811865476f};
constexpr float kTan[5] = {0.0f, 0.1989123673796580f, 0.4142135623730950f, 0.6681786379192989f, 1.0f};

// The reference project's 7x7 smoothing table, goldstein.cu:43-52: even in both
// offsets and symmetric, so the entries g[a][b], a, b = 0..3, in pairs (g[a][0],
// g[a][1]), (g[a][2], g[a][3]).  Kept as given: the filter output depends on
// these exact values.
__constant__ float2 c_gauss2[8] = {{0.221141f, 0.126584f}, {0.020584f, 0.000948f}, {0.126584f, 0.072410f},
                                   {0.011776f, 0.000543f}, {0.020584f, 0.011776f}, {0.001915f, 0.000088f},
                                   {0.000948f, 0.000543f}, {0.000088f, 0.000004f}};
// Sum of the table: g[0][0] + 4 sum_a g[a][0] + 4 sum_ab g[a][b], a, b = 1..3.
constexpr float kGaussSum =
    (float)(0.221141 + 4 * (0.126584 + 0.020584 + 0.000948) +
            4 * (0.072410 + 0.001915 + 0.000004 + 2 * (0.011776 + 0.000543 + 0.000088)));

__host__ __device__ constexpr int brev5(int i) {
  return ((i & 1) << 4) | ((i & 2) << 2) | (i & 4) | ((i & 8) >> 2) | ((i & 16) >> 4);
}

// Radix-2 butterfly with the twiddle exp(-2 pi i k / 32): u + w b into u, u -
// w b into b.  w b = c (shear of b), so the multiply by c rides on the two
// additions: two FFMA and two FFMA2, against two FMUL, an FFMA2 and two
// additions for the product formed first.
template <int k>
__device__ __forceinline__ void butterfly(float2 &u, float2 &b) {
  const float2 a = u;
  if constexpr (k == 0) {
    u = __fadd2_rn(a, b);
    b = __ffma2_rn(make_float2(-1.f, -1.f), b, a);
  } else if constexpr (k == 8) {  // -i b
    u = make_float2(a.x + b.y, a.y - b.x);
    b = make_float2(a.x - b.y, a.y + b.x);
  } else {
    // exp(-i t) b = cos t (b.x + tan t b.y, b.y - tan t b.x)
    //             = sin t (b.y + cot t b.x, -b.x + cot t b.y)
    constexpr int m = k < 8 ? k : 16 - k;  // mirrored at pi / 2
    constexpr bool by_cos = m <= 4;
    constexpr float tn = k < 8 ? kTan[by_cos ? m : 8 - m] : -kTan[by_cos ? m : 8 - m];
    constexpr float c = by_cos ? (k < 8 ? kCos[m] : -kCos[m]) : kCos[8 - m];
    const float2 t = by_cos ? make_float2(fmaf(tn, b.y, b.x), fmaf(-tn, b.x, b.y))
                            : make_float2(fmaf(tn, b.x, b.y), fmaf(tn, b.y, -b.x));
    u = __ffma2_rn(make_float2(c, c), t, a);
    b = __ffma2_rn(make_float2(-c, -c), t, a);
  }
}

template <int S, int J>
__device__ __forceinline__ void fft32_twiddle(float2 (&x)[GN]) {
  constexpr int m = 1 << S, half = m >> 1;
#pragma unroll
  for (int k = 0; k < GN; k += m) butterfly<J * (GN / m)>(x[k + J], x[k + J + half]);
  if constexpr (J + 1 < half) fft32_twiddle<S, J + 1>(x);
}

// 32-point forward DFT, exp(-2 pi i jk / 32), unnormalised: radix-2
// decimation in time, x[brev5(j)] = element j on entry, natural order on
// return.
__device__ __forceinline__ void fft32(float2 (&x)[GN]) {
  fft32_twiddle<1, 0>(x);
  fft32_twiddle<2, 0>(x);
  fft32_twiddle<3, 0>(x);
  fft32_twiddle<4, 0>(x);
  fft32_twiddle<5, 0>(x);
}

__device__ __forceinline__ float tri_weight(int t) {  // goldstein.cu:257-258
  return (float)(t < GN / 2 ? t : GN - 1 - t);
}

__device__ __forceinline__ int patch_origin(int p, int n) {  // goldstein.cu:308-313
  const int o = p * GSTEP;
  return o + GN > n ? n - GN : o;
}

__host__ __device__ inline void patch_grid(int nrow, int ncol, int &n_win_i, int &n_win_j) {  // goldstein.cu:335-340
  n_win_i = (int)ceilf((float)nrow / GSTEP) - 3;
  n_win_j = (int)ceilf((float)ncol / GSTEP) - 3;
  if (n_win_i <= 0) n_win_i = 1;
  if (n_win_j <= 0) n_win_j = 1;
}

// Patch rows that one warp takes in a run, for an image of ni x nj patches: a
// pure function of the image, so that a filter of many images sums in the
// order of the single one.
__host__ __device__ inline int run_patches(int ni, int nj) {
  int k = 1;
  while (k < GRUN_MAX && 2 * k <= ni && (int64_t)ni * nj >= (int64_t)(2 * k) * GRUN_JOBS) k *= 2;
  return k;
}

// Scratch rows of a run of k patches (32 columns each).  Runs x rows never
// exceed ni x 32: ceil(ni / k) (k + 3) / 4 <= ni for k <= ni.
__host__ __device__ inline int run_rows(int k) { return GSTEP * (k - 1) + GN; }

// Magnitude within one unit in the last place: the square root of the sum of
// squares, which is far from float overflow for interferogram samples.
__device__ __forceinline__ float magnitude(float2 v) {
  float m;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(m) : "f"(fmaf(v.x, v.x, v.y * v.y)));
  return m;
}

// The spectrum's weights, by the warp that holds it (lane = ky, x[kx]): F
// times S^alpha, S the smoothed |F| over its patch mean (goldstein.cu:105-176).
// Returns the conjugates in the order that fft32 reads, x[brev5(kx)].
__device__ __forceinline__ void goldstein_weigh(float2 (&x)[GN], float alpha) {
  const int lane = threadIdx.x & 31;
  float m[GN];
  float psum = 0.f;
#pragma unroll
  for (int c = 0; c < GN; ++c) {
    m[c] = magnitude(x[c]);
    psum += m[c];
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, off);
  // the smoothing is circular, so the mean of S is that of |F| times the sum
  // of the table
  const float mean = psum * (kGaussSum / (float)(GN * GN));
  const float inv = mean > 1e-8f ? 1.0f / mean : 0.0f;
  // 7x7 circular smoothing.  The table is even in both offsets and symmetric:
  //   S[kx] = W0[kx] + sum_{b=1..3} (Wb of the lanes ky - b and ky + b),
  //   Wb[kx] = sum_{a=0..3} g[a][b] (M[kx - a] + M[kx + a])  (a = 0 once):
  // the four filters Wb run along the lane's own spectrum, two at a time from
  // a sliding window of seven magnitudes, each kept twice; the offsets in ky
  // are lane shuffles (their wrap-around is the circular boundary).
  float2 win[7];
  float first[3];
#pragma unroll
  for (int i = 0; i < 6; ++i) win[i + 1] = make_float2(m[(i + GN - 3) & (GN - 1)], m[(i + GN - 3) & (GN - 1)]);
#pragma unroll
  for (int i = 0; i < 3; ++i) first[i] = m[i];
#pragma unroll
  for (int c = 0; c < GN; ++c) {
#pragma unroll
    for (int i = 0; i < 6; ++i) win[i] = win[i + 1];
    const float last = c + 3 < GN ? m[(c + 3) & (GN - 1)] : first[(c + 3) & (GN - 1) & 3];
    win[6] = make_float2(last, last);
    const float2 p1 = __fadd2_rn(win[2], win[4]), p2 = __fadd2_rn(win[1], win[5]), p3 = __fadd2_rn(win[0], win[6]);
    const float2 w01 = __ffma2_rn(c_gauss2[0], win[3], __ffma2_rn(c_gauss2[2], p1, __ffma2_rn(c_gauss2[4], p2, __fmul2_rn(c_gauss2[6], p3))));
    const float2 w23 = __ffma2_rn(c_gauss2[1], win[3], __ffma2_rn(c_gauss2[3], p1, __ffma2_rn(c_gauss2[5], p2, __fmul2_rn(c_gauss2[7], p3))));
    float s = w01.x;
    s += __shfl_sync(0xffffffffu, w01.y, (lane - 1) & (GN - 1)) + __shfl_sync(0xffffffffu, w01.y, (lane + 1) & (GN - 1));
    s += __shfl_sync(0xffffffffu, w23.x, (lane - 2) & (GN - 1)) + __shfl_sync(0xffffffffu, w23.x, (lane + 2) & (GN - 1));
    s += __shfl_sync(0xffffffffu, w23.y, (lane - 3) & (GN - 1)) + __shfl_sync(0xffffffffu, w23.y, (lane + 3) & (GN - 1));
    // S^alpha through the hardware exp2/log2 (relative error ~1e-6, far below
    // the filter's float tolerance); 0^alpha = 0 for alpha > 0, and a NaN
    // weight (0^0) leaves F unscaled, as a weight of 1 would
    float e;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(s * inv));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(alpha * e));
    m[c] = e > 0.0f ? e : 1.0f;
  }
#pragma unroll
  for (int c = 0; c < GN; ++c) {
    const int d = brev5(c);
    if (d < c) continue;
    const float2 t = __fmul2_rn(x[c], make_float2(m[c], -m[c]));
    if (d > c) x[c] = __fmul2_rn(x[d], make_float2(m[d], -m[d]));
    x[d] = t;
  }
}

struct GoldsteinTile {
  float2 T[GN][GN + 1];  // transposes
  float2 sums[GN][GN];   // of the rows that the next patch reaches too
};

// Run `job` (runs in row-major order over (run, patch column)) of an nrow x
// ncol image, by one warp.
__device__ __forceinline__ void goldstein_run(const float2 *__restrict__ in, float2 *__restrict__ runs, int nrow,
                                              int ncol, int ni, int nj, float alpha, int job, GoldsteinTile &tile) {
  float2(*T)[GN + 1] = tile.T;
  const int lane = threadIdx.x & 31;
  const int k = run_patches(ni, nj);
  const int p0 = job / nj * k, p1 = min(ni, p0 + k);
  const int j1 = patch_origin(job % nj, ncol);
  float2 *dst = runs + (size_t)job * run_rows(k) * GN + lane;
  const float wx = tri_weight(lane);
  // weighted sums so far of rows i1 .. i1 + 31 at column j1 + lane; the lane's
  // own, and the rows of i1 + 24 on stay zero (a patch keeps 32 - step < 32 - 7
  // rows, or fewer zeros above them after the shorter last step)
  float2 *sums = &tile.sums[0][lane];
#pragma unroll
  for (int r = 0; r < GN; ++r) sums[r * GN] = make_float2(0.f, 0.f);
  int i1 = patch_origin(p0, nrow);
#pragma unroll 1
  for (int p = p0; p < p1; ++p) {
    float2 x[GN];
    const float2 *src = in + (size_t)i1 * ncol + j1 + lane;
#pragma unroll
    for (int r = 0; r < GN; ++r) x[brev5(r)] = __ldg(src + (size_t)r * ncol);
    // forward transform along the lane's column, then, transposed, along the
    // lane's row; the inverse the same way from conjugate to conjugate.  One
    // copy of the transform's code serves the four.
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
      fft32(x);
      if (!(pass & 1)) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < GN; ++r) T[r][lane] = x[r];
        __syncwarp();
#pragma unroll
        for (int c = 0; c < GN; ++c) x[brev5(c)] = T[lane][c];
      } else if (pass == 1) {
        goldstein_weigh(x, alpha);
      }
    }
    // triangular weight and 1/n^2 (goldstein.cu:257-269); rows that the next
    // patch of the run does not reach are complete
    const int next = p + 1 < p1 ? patch_origin(p + 1, nrow) : i1 + GN;
    const int step = next - i1;
    float2 *keep = sums - step * GN;
#pragma unroll
    for (int r = 0; r < GN; ++r) {
      const float w = (wx + tri_weight(r)) * (1.0f / (float)(GN * GN));
      const float2 v = __ffma2_rn(x[r], make_float2(w, -w), sums[r * GN]);
      if (r < step)
        __stcg(dst + r * GN, v);
      else
        keep[r * GN] = v;
    }
    dst += step * GN;
    i1 = next;
  }
}

__global__ __launch_bounds__(32, GCTAS_PER_SM) void goldstein_run_kernel(
    const float2 *__restrict__ in, float2 *__restrict__ runs, int nrow, int ncol, int ni, int nj, float alpha) {
  __shared__ GoldsteinTile tile;
  goldstein_run(in, runs, nrow, ncol, ni, nj, alpha, blockIdx.x, tile);
}

// Output rows y0 .. y0 + R - 1 of column x, within a multiple of 8 and the
// next: each pixel the sum of the runs that
// cover it (run by run, columns ascending) over its weights.  The weights wx +
// wy of the covering patches are whole numbers: their sum over the ny x nx of
// them is exact as ny sum(wx) + nx sum(wy).
template <int R>
__device__ __forceinline__ void goldstein_gather(const float2 *__restrict__ runs, float2 *__restrict__ out, int nrow,
                                                 int ncol, int ni, int nj, int y0, int x) {
  const int k = run_patches(ni, nj), rows = run_rows(k);
  const int g = y0 / GSTEP, ny0 = min(R, nrow - y0);
  // the patch columns pj0 .. pj0 + 3 that lie before the last one, and the last
  const int pj0 = max(0, (x - (GN - 1) + GSTEP - 1) / GSTEP);
  bool cov[5];
  size_t off[5];  // of column x in the area of each
  float wx = 0.f, nx = 0.f;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int pj = j < 4 ? pj0 + j : nj - 1, tx = x - (j < 4 ? pj * GSTEP : patch_origin(pj, ncol));
    cov[j] = (j == 4 || pj < nj - 1) && tx >= 0;
    off[j] = (size_t)pj * (rows * GN) + tx;
    wx += cov[j] ? tri_weight(tx) : 0.f;
    nx += cov[j] ? 1.f : 0.f;
  }
  float2 acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = make_float2(0.f, 0.f);
  const int first = max(0, g - 3), last = patch_origin(ni - 1, nrow) < y0 + ny0 ? ni - 1 : g;
  for (int run = first / k; run <= last / k; ++run) {
    const int o = patch_origin(run * k, nrow), end = patch_origin(min(ni, run * k + k) - 1, nrow) + GN;
    const float2 *src = runs + (size_t)run * nj * rows * GN + (y0 - o) * GN;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r < ny0 && y0 + r >= o && y0 + r < end) {
        float2 v[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) v[j] = cov[j] ? __ldcg(src + r * GN + off[j]) : make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 5; ++j) acc[r] = __fadd2_rn(acc[r], v[j]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (r >= ny0) break;
    float wy = 0.f, ny = 0.f;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int pi = i < 4 ? first + i : ni - 1, ty = y0 + r - (i < 4 ? pi * GSTEP : patch_origin(pi, nrow));
      if ((i == 4 || pi < ni - 1) && ty >= 0 && ty < GN) {
        wy += tri_weight(ty);
        ny += 1.f;
      }
    }
    const float wsum = ny * wx + nx * wy;
    if (wsum > 0.f) {  // goldstein.cu:287-291
      acc[r].x /= wsum;
      acc[r].y /= wsum;
    }
    out[(size_t)(y0 + r) * ncol + x] = acc[r];
  }
}

template <int R>
__global__ __launch_bounds__(GGATHER) void goldstein_gather_kernel(const float2 *__restrict__ runs,
                                                                   float2 *__restrict__ out, int nrow, int ncol,
                                                                   int ni, int nj) {
  const int x = blockIdx.y * GGATHER + threadIdx.x;
  if (x >= ncol) return;
  goldstein_gather<R>(runs, out, nrow, ncol, ni, nj, blockIdx.x * R, x);
}

__host__ __device__ inline int run_jobs(int ni, int nj) {
  const int k = run_patches(ni, nj);
  return (ni + k - 1) / k * nj;
}



// ------------------------------------------------------------ frame stages
// Goldstein of every pair's interferogram: blockIdx.y = pair.  Pairs too
// small to filter get filt = ifg from the gather kernel.
__global__ __launch_bounds__(32, GCTAS_PER_SM) void frame_goldstein_run_kernel(const FrameDev d, const FrameIO io) {
  __shared__ GoldsteinTile tile;
  const int k = blockIdx.y;
  const s1b_frame_pair_t &r = io.pout[k];
  if (!r.ok || !r.filtered) return;
  int ni, nj;
  patch_grid(r.nrow_ml, r.ncol_ml, ni, nj);
  if ((int)blockIdx.x >= run_jobs(ni, nj)) return;
  const FramePair &pr = d.pairs[k];
  goldstein_run(io.ifg + pr.ml_off, io.work + pr.scratch_off, r.nrow_ml, r.ncol_ml, ni, nj, d.alpha, blockIdx.x,
                tile);
}

template <int R>
__global__ __launch_bounds__(GGATHER) void frame_goldstein_gather_kernel(const FrameDev d, const FrameIO io) {
  const int k = blockIdx.z;
  const s1b_frame_pair_t &r = io.pout[k];
  const int y0 = blockIdx.x * R, x = blockIdx.y * GGATHER + threadIdx.x;
  if (!r.ok || y0 >= r.nrow_ml || x >= r.ncol_ml) return;
  const FramePair &pr = d.pairs[k];
  if (r.filtered) {
    int ni, nj;
    patch_grid(r.nrow_ml, r.ncol_ml, ni, nj);
    goldstein_gather<R>(io.work + pr.scratch_off, io.filt + pr.ml_off, r.nrow_ml, r.ncol_ml, ni, nj, y0, x);
  } else {
    for (int y = y0; y < min(y0 + R, r.nrow_ml); ++y) {
      const size_t o = pr.ml_off + (size_t)y * r.ncol_ml + x;
      io.filt[o] = io.ifg[o];
    }
  }
}

int launch_goldstein(const void *in, void *out, int nrow, int ncol, int ni, int nj, float alpha, void *scratch,
                     cudaStream_t st) {
  goldstein_run_kernel<<<run_jobs(ni, nj), 32, 0, st>>>((const float2 *)in, (float2 *)scratch, nrow, ncol, ni, nj,
                                                        alpha);
  const int s = s1b_launch_status();
  if (s) return s;
  const dim3 grid(nrow, (ncol - 1) / GGATHER + 1);
  if ((int64_t)nrow * ncol >= kGatherRows8) {
    goldstein_gather_kernel<GSTEP><<<dim3((nrow - 1) / GSTEP + 1, grid.y), GGATHER, 0, st>>>(
        (const float2 *)scratch, (float2 *)out, nrow, ncol, ni, nj);
  } else {
    goldstein_gather_kernel<1><<<grid, GGATHER, 0, st>>>((const float2 *)scratch, (float2 *)out, nrow, ncol, ni, nj);
  }
  return s1b_launch_status();
}

}  // namespace

extern "C" size_t s1b_goldstein_scratch_bytes(int32_t nrow, int32_t ncol, int32_t n_win) {
  if (n_win != GN || nrow < GN || ncol < GN) return 0;
  int ni, nj;
  patch_grid(nrow, ncol, ni, nj);
  return (size_t)ni * nj * GN * GN * sizeof(float2);
}

extern "C" int s1b_goldstein(const void *in, void *out, int32_t nrow, int32_t ncol, int32_t n_win,
                             float alpha, void *scratch, size_t scratch_bytes, void *stream) {
  if (!in || !out) return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_goldstein: null argument");
  if (n_win != GN) return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_goldstein: only n_win = 32 is implemented");
  if (nrow < GN || ncol < GN)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_goldstein: image smaller than the window");
  const size_t need = s1b_goldstein_scratch_bytes(nrow, ncol, n_win);
  if (!scratch || scratch_bytes < need)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_goldstein: scratch buffer too small");
  int ni, nj;
  patch_grid(nrow, ncol, ni, nj);
  if ((int64_t)ni * nj > 0x7fffffff || (ncol + 255) / 256 > 65535)
    return s1b_fail(S1B_ERR_TOO_LARGE, "s1b_goldstein: image too large");
  return launch_goldstein(in, out, nrow, ncol, ni, nj, alpha, scratch, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Goldstein without any device allocation.
//
// Some callers cannot allocate device memory when they filter: a plugin
// running inside a host application whose own pool allocator has already
// reserved the GPU's memory (a raw cudaMalloc then fails although the pool
// has room), or a pipeline that forbids allocation after start-up to keep a
// fixed footprint.  For them the patch scratch lives in a file-scope device
// array of fixed size that every GPU loading this library holds until the
// process exits.
namespace {

constexpr size_t kNoAllocMaxPatches = S1B_GOLDSTEIN_NOALLOC_MAX_PATCHES;
__device__ __align__(256) float2 g_goldstein_scratch[kNoAllocMaxPatches * GN * GN];

// The array's device address, per CUDA context (see s1b_ctx_cache.h).
ContextKeyedCache<64> g_scratch_cache;

typedef CUresult (*CtxGetCurrentFn)(CUcontext *);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long *);

// The calling thread's current context and its unique id, through the
// driver entry points the runtime hands out (no link against libcuda).
// ctx is null when no context is current; cacheable is false when the
// driver cannot give the id, and then nothing is cached.
int current_context(const void **ctx, uint64_t *id, bool *cacheable) {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(p);
    p = nullptr;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(p);
    cudaGetLastError();
  });
  *ctx = nullptr;
  *id = 0;
  *cacheable = false;
  if (!get_current) return S1B_OK;
  CUcontext c = nullptr;
  if (get_current(&c) != CUDA_SUCCESS) return s1b_fail(S1B_ERR_CUDA, "s1b_goldstein_noalloc: cuCtxGetCurrent failed");
  *ctx = c;
  unsigned long long u = 0;
  if (c && get_id && get_id(c, &u) == CUDA_SUCCESS) {
    *id = u;
    *cacheable = true;
  }
  return S1B_OK;
}

// Device address of g_goldstein_scratch in the calling thread's current
// context.  The symbol name is only a host-side handle.  The address is
// looked up with cudaGetSymbolAddress the first time a context calls (which
// makes the device's primary context current when none is) and cached under
// that context's handle and id.
int noalloc_scratch(void **ptr) {
  const void *ctx;
  uint64_t id;
  bool cacheable;
  int s = current_context(&ctx, &id, &cacheable);
  if (s) return s;
  if (cacheable && g_scratch_cache.find(ctx, id, ptr)) return S1B_OK;
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_goldstein_scratch);
  if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  s = current_context(&ctx, &id, &cacheable);  // the context the lookup ran in
  if (s) return s;
  if (cacheable) g_scratch_cache.put(ctx, id, p);
  *ptr = p;
  return S1B_OK;
}

}  // namespace

extern "C" int s1b_goldstein_noalloc(const void *in, void *out, int32_t nrow, int32_t ncol,
                                     int32_t n_win, float alpha, void *stream) {
  if (!in || !out) return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_goldstein_noalloc: null argument");
  if (n_win != GN) return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_goldstein_noalloc: only n_win = 32 is implemented");
  if (nrow < GN || ncol < GN)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_goldstein_noalloc: image smaller than the window");
  int ni, nj;
  patch_grid(nrow, ncol, ni, nj);
  const int64_t npatch = (int64_t)ni * nj;
  if (npatch > (int64_t)kNoAllocMaxPatches)
    return s1b_fail(S1B_ERR_TOO_LARGE,
                    "s1b_goldstein_noalloc: image needs more than S1B_GOLDSTEIN_NOALLOC_MAX_PATCHES (4096) "
                    "patches of its fixed scratch (about 512 x 512 pixels); use s1b_goldstein");
  if ((ncol + 255) / 256 > 65535) return s1b_fail(S1B_ERR_TOO_LARGE, "s1b_goldstein_noalloc: image too wide");
  void *scratch = nullptr;
  int s = noalloc_scratch(&scratch);
  if (s) return s;
  // every scratch row that the gather reads is written by the kernel before
  // it, so nothing left by an earlier call needs clearing
  return launch_goldstein(in, out, nrow, ncol, ni, nj, alpha, scratch, (cudaStream_t)stream);
}

int frame_goldstein_patch_grid(int nrow, int ncol, int *ni, int *nj) {
  patch_grid(nrow, ncol, *ni, *nj);
  return S1B_OK;
}

int frame_launch_goldstein(const FrameDev &d, const FrameIO &io, cudaStream_t st) {
  if (d.max_nrow_ml <= 0 || d.max_ncol_ml <= 0) return S1B_OK;
  if (d.n_win != GN) return s1b_fail(S1B_ERR_UNSUPPORTED, "frame goldstein: only n_win = 32 is implemented");
  if (d.n_pairs > 65535 || (d.max_ncol_ml + 255) / 256 > 65535)
    return s1b_fail(S1B_ERR_TOO_LARGE, "frame goldstein: grid too large");
  if (d.max_patches > 0) {
    // CTAs beyond a pair's runs return.  Runs of ni x nj patches: at most 2 nj
    // (a run of more than ni / 2), or 2 GRUN_JOBS + nj, or ni nj / 8 + nj.
    const int64_t cols = (d.max_ncol_ml - 1) / GSTEP + 1;
    const int64_t jobs = std::max<int64_t>(2 * GRUN_JOBS, d.max_patches / GRUN_MAX) + 2 * cols;
    frame_goldstein_run_kernel<<<dim3((unsigned)std::min<int64_t>(d.max_patches, jobs), d.n_pairs), 32, 0, st>>>(d, io);
    int s = s1b_launch_status();
    if (s) return s;
  }
  const dim3 g2(d.max_nrow_ml, (d.max_ncol_ml - 1) / GGATHER + 1, d.n_pairs);
  if ((int64_t)d.max_nrow_ml * d.max_ncol_ml * d.n_pairs >= kGatherRows8)
    frame_goldstein_gather_kernel<GSTEP><<<dim3((d.max_nrow_ml - 1) / GSTEP + 1, g2.y, g2.z), GGATHER, 0, st>>>(d, io);
  else
    frame_goldstein_gather_kernel<1><<<g2, GGATHER, 0, st>>>(d, io);
  return s1b_launch_status();
}
