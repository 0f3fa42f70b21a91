// Coherence objective of radar-grid coregistration and its hand-written
// adjoint, fused: resample -> crossmul -> multilook windows -> coherence
// (-> gradient), for a stack of bursts of one size.  No reference
// counterpart (the reference has no differentiable path); the geometry and
// TOPS phase are the reference's (csrc/src/geo2rdr.cu:151-152, 210-219).
//
// Model, per burst b and pixel (row, col) of the reference grid:
//   az = row + az0 + p0 + p1 xa + p2 xr + daz_dh dh
//   rg = col + rg0 + p3 + p4 xa + p5 xr + drg_dh dh,
//   xa = (row - L/2) / L, xr = (col - S/2) / S,
//   s  = reramp(az, rg) * sum_ka sum_kr wa(fa)[ka] wr(fr)[kr] deramp(sec)[na + ka - 3, nr + kr - 3]
// (8-tap windowed sinc, zero where the support leaves the burst); over the
// rl x cl windows of the multilook grid I = sum conj(r) s, P1 = sum |r|^2,
// P2 = sum |s|^2, gamma = |I| / sqrt(P1 P2); J = -sum gamma / (windows).
// Gradient of gamma w.r.t. s (real/imaginary parts as one complex number):
//   g = gamma (I r / |I|^2 - s / P2),  d gamma / d theta = Re(conj(g) ds/dtheta),
//   ds/daz = rot (acc_a + i dPhi/daz acc),  ds/drg = rot (acc_r + i dPhi/drg acc),
// with acc_a, acc_r the interpolations with the weight derivatives dw/df.
// The backward recomputes the window sums instead of storing them.
#include <cuda_runtime.h>

#include <climits>
#include <cmath>
#include <mutex>

#include "s1b.h"
#include "s1b_device.cuh"
#include "s1b_internal.h"
#include "s1b_sinc.cuh"

struct s1b_adjoint {
  int device = 0;
  int n_bursts = 0, lines = 0, samples = 0, rowlook = 1, collook = 1;
  int tile_cols = 0, tiles_x = 0, tiles_y = 0;
  long long windows = 0;  // multilook windows over all bursts
  s1b_burst_plan_t *d_plans = nullptr;
};

namespace {

constexpr int A_TX = 64, A_TY = 4, A_RPT = 4, A_TH = A_TY * A_RPT;  // 16 rows x <= 64 columns
constexpr int A_WROWS = 32, A_WCOLS = 96;
constexpr int A_PARTS = 8;  // per-tile partials: 6 parameter sums, sum of gamma, windows

std::mutex g_tab_mu;
bool g_tab_ready[64] = {};

cudaError_t set_smem_attributes();  // after the kernels (dynamic shared memory of the current device)

// Normalised 8-tap windowed-sinc weights at A_BINS + 1 fractions (taps k =
// -3..4 at x = k - f: u = sinc(x) (0.5 + 0.5 cos(pi x / 4)), w = u / sum u),
// from the host in double precision, linear in between.  Taps 0-3 and 4-7 lie
// in arrays of their own: on terrain neighbouring pixels fall in neighbouring
// bins, whose entries are then neighbours too (a warp's 128-bit gather touches
// 4 lines instead of up to 32).
constexpr int A_BINS = 1024;
__device__ __align__(128) float4 g_w[2][A_BINS + 1];

int ensure_tables() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  if (dev < 0 || dev >= 64) return s1b_fail(S1B_ERR_UNSUPPORTED, "adjoint: device ordinal above 63");
  std::lock_guard<std::mutex> lock(g_tab_mu);
  if (g_tab_ready[dev]) return S1B_OK;
  static float4 w[2][A_BINS + 1];
  for (int b = 0; b <= A_BINS; ++b) {
    const double f = (double)b / A_BINS;
    double u[8], su = 0.0;
    for (int k = 0; k < 8; ++k) {
      const double x = (k - 3) - f;
      const double px = kPiD * x;
      u[k] = (x == 0.0 ? 1.0 : std::sin(px) / px) * (0.5 + 0.5 * std::cos(px / 4.0));
      su += u[k];
    }
    for (int h = 0; h < 2; ++h)
      w[h][b] = make_float4((float)(u[4 * h] / su), (float)(u[4 * h + 1] / su), (float)(u[4 * h + 2] / su),
                            (float)(u[4 * h + 3] / su));
  }
  e = cudaMemcpyToSymbol(g_w, w, sizeof(w));
  if (e == cudaSuccess) e = set_smem_attributes();
  if (e != cudaSuccess) return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  g_tab_ready[dev] = true;
  return S1B_OK;
}

__device__ __forceinline__ float2 fma2(float w, float2 v, float2 acc) {
  return __ffma2_rn(make_float2(w, w), v, acc);
}

// Weights at fraction f by linear interpolation of the table.
__device__ __forceinline__ void lut8(float f, float w[8]) {
  const float pos = f * A_BINS;
  const int b = min((int)pos, A_BINS - 1);
  const float t = pos - (float)b;
  const float2 tt = make_float2(t, t), m1 = make_float2(-1.f, -1.f);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 a = __ldg(&g_w[h][b]), n = __ldg(&g_w[h][b + 1]);
    const float2 lo = make_float2(a.x, a.y), hi = make_float2(a.z, a.w);
    const float2 l = __ffma2_rn(tt, __ffma2_rn(m1, lo, make_float2(n.x, n.y)), lo);
    const float2 u = __ffma2_rn(tt, __ffma2_rn(m1, hi, make_float2(n.z, n.w)), hi);
    w[4 * h] = l.x;
    w[4 * h + 1] = l.y;
    w[4 * h + 2] = u.x;
    w[4 * h + 3] = u.y;
  }
}

// Loads of the streamed rasters, which leave L1 to the weight table.
__device__ __forceinline__ float load_stream(const float *p) {
  float v;
  asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 load_stream(const float2 *p) {
  float2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}

// TOPS terms at a continuous range sample, phase in half-cycles: -kt and
// etaref (geo2rdr.cu:533-541 with the sample index fractional).
__device__ __forceinline__ void tops_range(const s1b_burst_plan_t &P, double rs, double &mkt, double &etaref) {
  const double tr = P.slant_range_time + rs / P.range_sampling_rate;
  double dt = tr - P.fm[0];
  const double ka = P.fm[1] + dt * (P.fm[2] + P.fm[3] * dt);
  dt = tr - P.dc[0];
  const double fnc = P.dc[1] + dt * (P.dc[2] + P.dc[3] * dt);
  const double kmk = ka - P.ks;
  const double inv = 1.0 / (ka * kmk);
  mkt = -(ka * P.ks * (ka * inv));
  etaref = -fnc * (kmk * inv) - P.etac0;
}

__device__ __forceinline__ float2 deramped_tap(const s1b_burst_plan_t &P, const float2 *sec, int r, int c) {
  const float2 v = __ldg(sec + (size_t)r * P.samples + c);
  double mkt, etaref;
  tops_range(P, (double)c, mkt, etaref);
  const double d = (-P.lines * P.ati / 2. + r * P.ati) - etaref;
  return cmul(v, phasor_pi(mkt * d * d));
}

struct AdjArgs {
  const s1b_burst_plan_t *plans;
  const float2 *ref, *sec;
  const float *az0, *rg0, *daz_dh, *drg_dh, *params, *dh;
  float *grad_dh;
  double *partials;  // [n_bursts * tiles][A_PARTS]
  int L, S, rl_log2, cl, tile_cols, tiles_x, tiles_per_burst;
  int nwr, nwc, wpr;       // multilook grid; windows across a tile
  float inv_cl, inv_wpr;
  float inv_windows;       // 1 / (windows over all bursts)
};

struct AdjSmem {
  float2 win[A_WROWS][A_WCOLS];         // deramped secondary window
  double mkt[A_WCOLS], eref[A_WCOLS];   // per window column
  double part[A_TX * A_TY / 32][A_PARTS];
  int red[4];
  float xa[A_TH];
  float2 s[A_TH][A_TX];  // per pixel: the fractions (azimuth, range) of its sample, then the resampled s
  int2 n[A_TH][A_TX];    // per pixel: the sample (row, column of the secondary), row INT_MIN outside it; then ds/daz
  float2 r[A_TH][A_TX];
  // kGrad: [A_TH][A_TX] ds/drg follow
};
// Once every pixel is interpolated the window's place holds the products
// Re I, Im I, P1, P2 of the pixels; a window's sums leave A I, B, gamma in its
// first pixel's entry.
static_assert(sizeof(float4[A_TH][A_TX]) <= sizeof(AdjSmem::win), "products fit the window's place");
constexpr size_t kAdjPix = sizeof(float2) * A_TH * A_TX;
constexpr size_t adjoint_smem(bool grad) { return sizeof(AdjSmem) + (grad ? kAdjPix : 0); }

// 8 x 8 taps of one pixel: value and, with kGrad, the range / azimuth
// derivative interpolations.  tap(ka, kr) returns the deramped sample.
template <bool kGrad, typename Tap>
__device__ __forceinline__ void interp_taps(const float wr[8], const float wa[8], const float dwr[8],
                                            const float dwa[8], Tap tap, float2 &acc, float2 &acc_a,
                                            float2 &acc_r) {
#pragma unroll
  for (int ka = 0; ka < 8; ++ka) {
    float2 rs = make_float2(0.f, 0.f), rsd = rs;
#pragma unroll
    for (int kr = 0; kr < 8; ++kr) {
      const float2 v = tap(ka, kr);
      rs = fma2(wr[kr], v, rs);
      if (kGrad) rsd = fma2(dwr[kr], v, rsd);
    }
    acc = fma2(wa[ka], rs, acc);
    if (kGrad) {
      acc_a = fma2(dwa[ka], rs, acc_a);
      acc_r = fma2(wa[ka], rsd, acc_r);
    }
  }
}

// The same with every sample read and deramped by itself, for a tile whose
// window exceeds the stage (rare: kept out of line, so that its registers do
// not burden the pixel loop).
template <bool kGrad>
__device__ __noinline__ void interp_direct(const s1b_burst_plan_t &P, const float2 *sec, int n0, int m0, float fr,
                                           float fa, float2 &acc, float2 &acc_a, float2 &acc_r) {
  float wr[8], wa[8], dwr[8] = {}, dwa[8] = {};
  lut8(fr, wr);
  lut8(fa, wa);
  if (kGrad) sinc8_slopes(fa, fr, dwa, dwr);
#pragma unroll 1
  for (int ka = 0; ka < 8; ++ka) {
    float2 rs = make_float2(0.f, 0.f), rsd = rs;
#pragma unroll 1
    for (int kr = 0; kr < 8; ++kr) {
      const float2 v = deramped_tap(P, sec, n0 + ka, m0 + kr);
      rs = fma2(wr[kr], v, rs);
      if (kGrad) rsd = fma2(dwr[kr], v, rsd);
    }
    acc = fma2(wa[ka], rs, acc);
    if (kGrad) {
      acc_a = fma2(dwa[ka], rs, acc_a);
      acc_r = fma2(wa[ka], rsd, acc_r);
    }
  }
}

// One tile of 16 rows x tile_cols columns (whole windows) per CTA; a thread
// owns 4 rows of a column.  What bounds it is instruction issue: the taps are
// 152 paired FP32 multiply-adds a pixel (forward 72) and 64 shared loads,
// about half of all 900.  So that three CTAs fit an SM (80 registers, 62 KB)
// the pixel loop stays rolled and carries a pixel's coordinates and results
// through shared memory, where the products take the window's place: two
// bursts of 1468 x 20968 pixels in 2.42 ms (61 % of issue slots; with two CTAs
// at 128 registers 2.78).  Before, with the weights and their derivatives in
// tables whose bins lay 32 bytes apart, coordinates in local memory and one
// thread per window summing its four products, 4.46 ms at 39 %, half of the
// L1 wavefronts for the tables.
template <bool kGrad>
__global__ __launch_bounds__(A_TX *A_TY, 3) void adjoint_kernel(const AdjArgs a) {
  extern __shared__ __align__(16) unsigned char adj_raw[];
  AdjSmem &sm = *reinterpret_cast<AdjSmem *>(adj_raw);
  float2(*s_dr)[A_TX] = reinterpret_cast<float2(*)[A_TX]>(adj_raw + sizeof(AdjSmem));
  float2(*s_da)[A_TX] = reinterpret_cast<float2(*)[A_TX]>(sm.n);
  float4(*pix)[A_TX] = reinterpret_cast<float4(*)[A_TX]>(sm.win);
  const int b = blockIdx.y, tile = blockIdx.x;
  const int tile_y = tile / a.tiles_x, tile_x = tile - tile_y * a.tiles_x;
  const s1b_burst_plan_t &P = a.plans[b];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * A_TX + tx, lane = tid & 31, warp = tid >> 5;
  const int L = a.L, S = a.S;
  const int col = tile_x * a.tile_cols + tx;
  const int row0 = tile_y * A_TH, rowb = row0 + ty * A_RPT;
  const int nwr = a.nwr, nwc = a.nwc;  // multilook grid
  const bool colin = tx < a.tile_cols && col < nwc * a.cl;
  const int rend = nwr << a.rl_log2;  // rows of the multilook grid
  const size_t boff = (size_t)b * L * S;
  if (tid == 0) {
    sm.red[0] = INT_MAX;
    sm.red[1] = INT_MIN;
    sm.red[2] = INT_MAX;
    sm.red[3] = INT_MIN;
  }
  const float xr = ((float)col - 0.5f * S) / S;
  const int lines = P.lines, samples = P.samples;
  {  // offsets of the thread's 4 pixels, and the tile's window
    const float *pr = a.params + 6 * b;
    if (tid < A_TH) sm.xa[tid] = ((float)(row0 + tid) - 0.5f * L) / L;
    __syncthreads();
    const float p0 = pr[0], p1 = pr[1], p2 = pr[2], p3 = pr[3], p4 = pr[4], p5 = pr[5];
    int mna = INT_MAX, xna = INT_MIN, mnr = INT_MAX, xnr = INT_MIN;
    float h[A_RPT], az[A_RPT], rg[A_RPT], da[A_RPT], dr[A_RPT];
#pragma unroll
    for (int q = 0; q < A_RPT; ++q) {
      h[q] = az[q] = rg[q] = da[q] = dr[q] = 0.f;
      if (colin && rowb + q < rend) {
        const size_t i = boff + (size_t)(rowb + q) * S + col;
        h[q] = load_stream(a.dh + i);
        az[q] = load_stream(a.az0 + i);
        rg[q] = load_stream(a.rg0 + i);
        da[q] = load_stream(a.daz_dh + i);
        dr[q] = load_stream(a.drg_dh + i);
      }
    }
#pragma unroll
    for (int q = 0; q < A_RPT; ++q) {
      const int row = rowb + q;
      const float xa = sm.xa[ty * A_RPT + q];
      bool ok = colin && row < rend;
      const float oa = az[q] + fmaf(p2, xr, fmaf(p1, xa, p0)) + da[q] * h[q];
      const float orr = rg[q] + fmaf(p5, xr, fmaf(p4, xa, p3)) + dr[q] * h[q];
      ok = ok && fabsf(oa) < 0x1p20f && fabsf(orr) < 0x1p20f;  // false for no number
      const float fla = ok ? floorf(oa) : 0.f, flr = ok ? floorf(orr) : 0.f;
      const int na = row + (int)fla, nr = col + (int)flr;
      ok = ok && na - 3 >= 0 && na + 4 < lines && nr - 3 >= 0 && nr + 4 < samples;
      sm.s[ty * A_RPT + q][tx] = make_float2(fminf(oa - fla, 0x1.fffffep-1f), fminf(orr - flr, 0x1.fffffep-1f));
      sm.n[ty * A_RPT + q][tx] = make_int2(ok ? na : INT_MIN, nr);
      if (ok) {
        mna = min(mna, na);
        xna = max(xna, na);
        mnr = min(mnr, nr);
        xnr = max(xnr, nr);
      }
    }
    mna = __reduce_min_sync(0xffffffffu, mna);
    xna = __reduce_max_sync(0xffffffffu, xna);
    mnr = __reduce_min_sync(0xffffffffu, mnr);
    xnr = __reduce_max_sync(0xffffffffu, xnr);
    if (lane == 0 && mna <= xna) {
      atomicMin(&sm.red[0], mna);
      atomicMax(&sm.red[1], xna);
      atomicMin(&sm.red[2], mnr);
      atomicMax(&sm.red[3], xnr);
    }
  }
  __syncthreads();
  const int wa0 = sm.red[0] - 3, wr0 = sm.red[2] - 3;
  const int wrows = sm.red[1] + 4 - wa0 + 1, wcols = sm.red[3] + 4 - wr0 + 1;
  const bool staged = sm.red[0] <= sm.red[1] && wrows <= A_WROWS && wcols <= A_WCOLS;
  const float2 *sec = a.sec + (size_t)b * lines * samples;
  const double eta0 = -lines * P.ati / 2.;  // line 0 from the burst centre
  if (staged) {
    // deramped window: column walks with the phasor recurrence (drift ~1e-6 rad)
    // quotients by a float reciprocal: (i + 0.5) / wcols with i <= 256 and
    // wcols <= 96 is >= 0.005 from an integer
    const float rn = __frcp_rn((float)wcols);
    const int groups = __float2int_rz((A_TX * A_TY + 0.5f) * rn);  // 2 or more
    const int seg = __float2int_rz((wrows + groups - 1 + 0.5f) * __frcp_rn((float)groups));
    const int g = __float2int_rz((tid + 0.5f) * rn), c = tid - g * wcols;
    if (g < groups) {
      const int r0 = g * seg, r1 = min(wrows, r0 + seg);
      double mkt, eref;
      tops_range(P, (double)(wr0 + c), mkt, eref);
      if (g == 0) {
        sm.mkt[c] = mkt;
        sm.eref[c] = eref;
      }
      if (r0 < r1) {
        const double u = fma((double)(wa0 + r0), P.ati, eta0) - eref;
        float2 ph = phasor_pi(mkt * u * u);
        float2 step = phasor_pi(mkt * P.ati * (2.0 * u + P.ati));
        const float2 dstep = phasor_pi(2.0 * mkt * P.ati * P.ati);
        // eight samples of the segment at a time are loaded first, so their
        // reads overlap
        const float2 *src = sec + (size_t)(wa0 + r0) * samples + (wr0 + c);
        float2 *dst = &sm.win[r0][c];
#pragma unroll 1
        for (int k0 = r1 - r0; k0 > 0; k0 -= 8) {
          float2 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < k0) v[k] = load_stream(src + (size_t)k * samples);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (k < k0) {
              dst[k * A_WCOLS] = cmul(v[k], ph);
              ph = cmul(ph, step);
              step = cmul(step, dstep);
            }
          }
          src += (size_t)8 * samples;
          dst += 8 * A_WCOLS;
        }
      }
    }
    __syncthreads();
  }
  // per pixel: resampled s, its derivatives, the products
#pragma unroll 1
  for (int q = 0; q < A_RPT; ++q) {
    const int lr = ty * A_RPT + q;
    const int row = row0 + lr;
    float2 s = make_float2(0.f, 0.f), sa = s, sr = s;
    float2 rv = make_float2(0.f, 0.f);
    if (colin && row < rend) rv = load_stream(a.ref + boff + (size_t)row * S + col);
    const int2 n = sm.n[lr][tx];
    const int na = n.x, nr = n.y;
    if (na != INT_MIN) {
      const float2 frac = sm.s[lr][tx];
      const float fa = frac.x, fr = frac.y;
      float2 acc = make_float2(0.f, 0.f), acc_a = acc, acc_r = acc;
      const int n0 = na - 3, m0 = nr - 3;
      if (staged) {
        float wr[8], wa[8], dwr[8] = {}, dwa[8] = {};
        lut8(fr, wr);
        lut8(fa, wa);
        if (kGrad) sinc8_slopes(fa, fr, dwa, dwr);
        const float2 *base = &sm.win[n0 - wa0][m0 - wr0];
        interp_taps<kGrad>(wr, wa, dwr, dwa, [&](int ka, int kr) { return base[ka * A_WCOLS + kr]; }, acc, acc_a,
                           acc_r);
      } else {
        interp_direct<kGrad>(P, sec, n0, m0, fr, fa, acc, acc_a, acc_r);
      }
      // reramp with the secondary's TOPS phase at (az, rg): Phi = -pi mkt d^2
      double k0, k1, e0, e1;
      if (staged) {
        const int c = nr - wr0;
        k0 = sm.mkt[c];
        k1 = sm.mkt[c + 1];
        e0 = sm.eref[c];
        e1 = sm.eref[c + 1];
      } else {
        tops_range(P, (double)nr, k0, e0);
        tops_range(P, (double)nr + 1.0, k1, e1);
      }
      const double dmkt = k1 - k0, deref = e1 - e0;
      const double t = fr;
      const double mkt = fma(t, dmkt, k0), eref = fma(t, deref, e0);
      const double d = fma(i32_to_f64(na) + (double)fa, P.ati, eta0) - eref;
      const double md = mkt * d;
      const float2 rot = phasor_pi(-(md * d));
      s = cmul(acc, rot);
      if (kGrad) {
        // dPhi/daz = -2 pi mkt d ati; dPhi/drg = pi (2 mkt d deref - dmkt d^2)
        const float pa = (float)(-2.0 * kPiD * P.ati * md);
        const float pg = (float)(kPiD * (2.0 * md * deref - dmkt * d * d));
        sa = cmul(make_float2(acc_a.x - pa * acc.y, acc_a.y + pa * acc.x), rot);
        sr = cmul(make_float2(acc_r.x - pg * acc.y, acc_r.y + pg * acc.x), rot);
      }
    }
    sm.s[lr][tx] = s;
    sm.r[lr][tx] = rv;
    if (kGrad) {
      s_da[lr][tx] = sa;
      s_dr[lr][tx] = sr;
    }
  }
  __syncthreads();  // the window has been read
#pragma unroll
  for (int q = 0; q < A_RPT; ++q) {  // conj(r) s, |r|^2, |s|^2
    const float2 rv = sm.r[ty * A_RPT + q][tx], s = sm.s[ty * A_RPT + q][tx];
    pix[ty * A_RPT + q][tx] = make_float4(rv.x * s.x + rv.y * s.y, rv.x * s.y - rv.y * s.x, rv.x * rv.x + rv.y * rv.y,
                                          s.x * s.x + s.y * s.y);
  }
  __syncthreads();
  // window sums, each in the order of its pixels: four lanes per window, one
  // for each of the four sums
  const int wpr = a.wpr, wtile = (A_TH >> a.rl_log2) * wpr;
  // quotients by float reciprocals: numerators below 2^11, so (i + 0.5) / n
  // stays 2^-11 / n or more from an integer
  auto first_pixel = [&](int wi, int &wy, int &wx) -> float4 * {
    wy = __float2int_rz((wi + 0.5f) * a.inv_wpr);
    wx = wi - wy * wpr;
    return &pix[wy << a.rl_log2][wx * a.cl];
  };
  for (int w0 = 0; w0 < wtile; w0 += A_TX * A_TY / 4) {
    const int wi = w0 + (tid >> 2), k = tid & 3;
    float sum = 0.f;
    float4 *entry = nullptr;
    if (wi < wtile) {
      int wy, wx;
      entry = first_pixel(wi, wy, wx);
      if (tile_y * (A_TH >> a.rl_log2) + wy < nwr && tile_x * wpr + wx < nwc) {
        const float *v = reinterpret_cast<const float *>(entry) + k;
        const int n = a.cl << a.rl_log2;
        int c = 0;  // column of the next value to load
        auto next = [&]() -> float {
          const float x = *v;
          v += 4;
          if (++c == a.cl) {
            c = 0;
            v += 4 * (A_TX - a.cl);
          }
          return x;
        };
        // one long chain of additions: the values of the next eight pixels
        // are loaded while the last eight are added
        float cur[8], nxt[8];
        int left = n - 8;
        if (left >= 0)
#pragma unroll
          for (int i = 0; i < 8; ++i) cur[i] = next();
        for (; left >= 8; left -= 8) {
#pragma unroll
          for (int i = 0; i < 8; ++i) nxt[i] = next();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            sum += cur[i];
            cur[i] = nxt[i];
          }
        }
        if (left >= 0)
#pragma unroll
          for (int i = 0; i < 8; ++i) sum += cur[i];
        for (left = left >= 0 ? left : n; left > 0; --left) sum += next();
      }
    }
    float4 acc;
    const int lane0 = lane & ~3;
    acc.x = __shfl_sync(0xffffffffu, sum, lane0);
    acc.y = __shfl_sync(0xffffffffu, sum, lane0 + 1);
    acc.z = __shfl_sync(0xffffffffu, sum, lane0 + 2);
    acc.w = __shfl_sync(0xffffffffu, sum, lane0 + 3);
    if (entry && k == 0) {
      const float den = acc.z * acc.w;
      const float i2 = fmaf(acc.y, acc.y, acc.x * acc.x);
      float gam = 0.f, A = 0.f, B = 0.f;
      if (den > 0.f && i2 > 0.f) {
        gam = sqrtf(i2) * rsqrtf(den);
        A = gam / i2;  // g = (A I) r - B s
        B = gam / acc.w;
      }
      // the window's own first entry: no other window reads it
      *entry = make_float4(A * acc.x, A * acc.y, B, gam);
    }
  }
  __syncthreads();
  float gsum = 0.f;
  for (int wi = tid; wi < wtile; wi += A_TX * A_TY) {
    int wy, wx;
    gsum += first_pixel(wi, wy, wx)->w;
  }
  double part[A_PARTS];
#pragma unroll
  for (int k = 0; k < A_PARTS; ++k) part[k] = 0.0;
  part[6] = gsum;
  if (kGrad) {
    // per pixel: g = A r - B s, dJ/daz, dJ/drg, height gradient, parameter sums
    float ga0 = 0.f, ga1 = 0.f, gr0 = 0.f, gr1 = 0.f;
    const int wc0 = __float2int_rz((tx + 0.5f) * a.inv_cl) * a.cl;
#pragma unroll
    for (int q = 0; q < A_RPT; ++q) {
      const int lr = ty * A_RPT + q;
      const int row = row0 + lr;
      if (tx >= a.tile_cols || col >= S || row >= L) continue;
      const size_t i = boff + (size_t)row * S + col;
      float gh = 0.f;  // pixels outside the multilook grid
      if (colin && row < rend) {
        const float4 w = pix[lr >> a.rl_log2 << a.rl_log2][wc0];
        const float2 rv = sm.r[lr][tx], s = sm.s[lr][tx], sa = s_da[lr][tx], sr = s_dr[lr][tx];
        // g = (Ar + i Ai) r - B s
        const float gx = w.x * rv.x - w.y * rv.y - w.z * s.x;
        const float gy = w.x * rv.y + w.y * rv.x - w.z * s.y;
        const float dja = -a.inv_windows * (gx * sa.x + gy * sa.y);  // -Re(conj(g) ds/daz) / windows
        const float djr = -a.inv_windows * (gx * sr.x + gy * sr.y);
        gh = fmaf(dja, load_stream(a.daz_dh + i), djr * load_stream(a.drg_dh + i));
        const float xa = sm.xa[lr];
        ga0 += dja;
        ga1 += dja * xa;
        gr0 += djr;
        gr1 += djr * xa;
      }
      __stcs(a.grad_dh + i, gh);
    }
    part[0] = ga0;
    part[1] = ga1;
    part[2] = ga0 * xr;
    part[3] = gr0;
    part[4] = gr1;
    part[5] = gr0 * xr;
  }
  // deterministic block reduction of the 8 sums: a butterfly that halves the
  // sums a lane carries, then the lanes, then the warps in order
#pragma unroll
  for (int half = A_PARTS / 2; half > 0; half >>= 1) {
    const bool up = lane & (half * 4);  // lane bits 4, 3, 2
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const double give = up ? part[k] : part[k + half], keep = up ? part[k + half] : part[k];
      part[k] = keep + __shfl_xor_sync(0xffffffffu, give, half * 4);
    }
  }
  double v = part[0];
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  if ((lane & 3) == 0) sm.part[warp][lane >> 2] = v;  // lane bits 4..2 name the sum
  __syncthreads();
  if (tid < A_PARTS) {
    double t = 0.0;
    for (int w = 0; w < A_TX * A_TY / 32; ++w) t += sm.part[w][tid];
    a.partials[((size_t)b * a.tiles_per_burst + tile) * A_PARTS + tid] = t;
  }
}

cudaError_t set_smem_attributes() {
  cudaError_t e = cudaFuncSetAttribute(adjoint_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)adjoint_smem(true));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(adjoint_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)adjoint_smem(false));
  return e;
}

// Tiles summed in a fixed order: A_RED blocks per burst (blockIdx.y) each sum
// a share of its tiles into [burst][block][7]; one block per burst took 95 us
// for 32,200 tiles.
constexpr int A_RED = 32;
__global__ __launch_bounds__(256) void adjoint_reduce_kernel(const double *__restrict__ partials, int tiles,
                                                             double *__restrict__ shares) {
  __shared__ double s[256];
  const int b = blockIdx.y, k = threadIdx.x & (A_PARTS - 1), t0 = threadIdx.x / A_PARTS;
  const int per = (tiles + A_RED - 1) / A_RED, first = blockIdx.x * per, last = min(tiles, first + per);
  double v = 0.0;
  for (int t = first + t0; t < last; t += 256 / A_PARTS) v += partials[((size_t)b * tiles + t) * A_PARTS + k];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = 128; w >= A_PARTS; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x < A_PARTS) shares[((size_t)b * A_RED + blockIdx.x) * A_PARTS + threadIdx.x] = s[threadIdx.x];
}

// The shares in order: parameter gradients per burst, and the objective J =
// -(sum over bursts of gamma) / windows, bursts in order.  One block.
__global__ __launch_bounds__(256) void adjoint_objective_kernel(const double *__restrict__ shares, int n_bursts,
                                                                double inv_windows, double *__restrict__ objective,
                                                                float *__restrict__ grad_params) {
  __shared__ double gam[256 / A_PARTS];
  const int k = threadIdx.x & (A_PARTS - 1), t0 = threadIdx.x / A_PARTS;
  double total = 0.0;
  for (int b0 = 0; b0 < n_bursts; b0 += 256 / A_PARTS) {
    const int b = b0 + t0;
    double v = 0.0;
    if (b < n_bursts) {
      const double *p = shares + (size_t)b * A_RED * A_PARTS + k;
#pragma unroll
      for (int i = 0; i < A_RED; ++i) v += p[i * A_PARTS];
      if (k < 6 && grad_params) grad_params[6 * b + k] = (float)v;
    }
    __syncthreads();
    if (k == 6) gam[t0] = v;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < min(256 / A_PARTS, n_bursts - b0); ++i) total += gam[i];
  }
  if (threadIdx.x == 0) objective[0] = -total * inv_windows;
}

}  // namespace

extern "C" int s1b_adjoint_create(const s1b_burst_plan_t *sec_plans, int32_t n_bursts, int32_t lines,
                                  int32_t samples, int32_t rowlook, int32_t collook, s1b_adjoint_t **out) {
  if (!out) return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_adjoint_create: null handle");
  *out = nullptr;
  if (!sec_plans || n_bursts < 1 || lines < 1 || samples < 1)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_adjoint_create: no bursts");
  if (rowlook < 1 || A_TH % rowlook != 0)
    return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_adjoint_create: rowlook must divide 16");
  if (collook < 1 || collook > A_TX) return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_adjoint_create: collook above 64");
  if (lines / rowlook < 1 || samples / collook < 1)
    return s1b_fail(S1B_ERR_EMPTY, "s1b_adjoint_create: no multilook window");
  for (int b = 1; b < n_bursts; ++b)
    if (sec_plans[b].lines != sec_plans[0].lines || sec_plans[b].samples != sec_plans[0].samples)
      return s1b_fail(S1B_ERR_UNSUPPORTED, "s1b_adjoint_create: secondary bursts must have one size");
  int s = ensure_tables();
  if (s) return s;
  s1b_adjoint *h = new s1b_adjoint();
  cudaGetDevice(&h->device);
  h->n_bursts = n_bursts;
  h->lines = lines;
  h->samples = samples;
  h->rowlook = rowlook;
  h->collook = collook;
  h->tile_cols = (A_TX / collook) * collook;
  h->tiles_x = (samples + h->tile_cols - 1) / h->tile_cols;
  h->tiles_y = (lines + A_TH - 1) / A_TH;
  h->windows = (long long)n_bursts * (lines / rowlook) * (samples / collook);
  cudaError_t e = cudaMalloc(&h->d_plans, n_bursts * sizeof(s1b_burst_plan_t));
  if (e == cudaSuccess)
    e = cudaMemcpy(h->d_plans, sec_plans, n_bursts * sizeof(s1b_burst_plan_t), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(h->d_plans);
    delete h;
    return s1b_fail(S1B_ERR_CUDA, cudaGetErrorString(e));
  }
  *out = h;
  return S1B_OK;
}

extern "C" void s1b_adjoint_destroy(s1b_adjoint_t *h) {
  if (!h) return;
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != h->device) cudaSetDevice(h->device);
  cudaFree(h->d_plans);
  if (prev >= 0 && prev != h->device) cudaSetDevice(prev);
  delete h;
}

extern "C" size_t s1b_adjoint_workspace_bytes(const s1b_adjoint_t *h) {
  if (!h) return 0;
  return ((size_t)h->n_bursts * h->tiles_x * h->tiles_y + (size_t)h->n_bursts * A_RED) * A_PARTS * sizeof(double);
}

extern "C" int s1b_adjoint_run(s1b_adjoint_t *h, const void *ref, const void *sec, const float *az0,
                               const float *rg0, const float *daz_dh, const float *drg_dh, const float *params,
                               const float *dh, double *objective, float *grad_params, float *grad_dh,
                               void *workspace, size_t workspace_bytes, void *stream) {
  if (!h || !ref || !sec || !az0 || !rg0 || !daz_dh || !drg_dh || !params || !dh || !objective || !workspace)
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_adjoint_run: null argument");
  const bool grad = grad_params || grad_dh;
  if (grad && (!grad_params || !grad_dh))
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_adjoint_run: give both gradient outputs or neither");
  if (workspace_bytes < s1b_adjoint_workspace_bytes(h))
    return s1b_fail(S1B_ERR_INVALID_ARGUMENT, "s1b_adjoint_run: workspace too small");
  const int tiles = h->tiles_x * h->tiles_y;
  if (h->n_bursts > 65535 || tiles < 1) return s1b_fail(S1B_ERR_TOO_LARGE, "s1b_adjoint_run: grid too large");
  cudaStream_t st = (cudaStream_t)stream;
  int s0 = ensure_tables();  // this device's table and shared-memory limits
  if (s0) return s0;
  AdjArgs a;
  a.plans = h->d_plans;
  a.ref = (const float2 *)ref;
  a.sec = (const float2 *)sec;
  a.az0 = az0;
  a.rg0 = rg0;
  a.daz_dh = daz_dh;
  a.drg_dh = drg_dh;
  a.params = params;
  a.dh = dh;
  a.grad_dh = grad_dh;
  a.partials = (double *)workspace;
  a.L = h->lines;
  a.S = h->samples;
  a.rl_log2 = 0;
  while ((1 << a.rl_log2) < h->rowlook) ++a.rl_log2;  // 1, 2, 4, 8 or 16
  a.cl = h->collook;
  a.nwr = h->lines / h->rowlook;
  a.nwc = h->samples / h->collook;
  a.wpr = h->tile_cols / h->collook;
  a.inv_cl = 1.0f / (float)h->collook;
  a.inv_wpr = 1.0f / (float)a.wpr;
  a.tile_cols = h->tile_cols;
  a.tiles_x = h->tiles_x;
  a.tiles_per_burst = tiles;
  a.inv_windows = (float)(1.0 / (double)h->windows);
  const dim3 grid(tiles, h->n_bursts);
  dim3 block(A_TX, A_TY);
  const size_t smem = adjoint_smem(grad);
  if (grad)
    adjoint_kernel<true><<<grid, block, smem, st>>>(a);
  else
    adjoint_kernel<false><<<grid, block, smem, st>>>(a);
  int s = s1b_launch_status();
  if (s) return s;
  double *shares = (double *)workspace + (size_t)h->n_bursts * tiles * A_PARTS;
  adjoint_reduce_kernel<<<dim3(A_RED, h->n_bursts), 256, 0, st>>>((const double *)workspace, tiles, shares);
  s = s1b_launch_status();
  if (s) return s;
  adjoint_objective_kernel<<<1, 256, 0, st>>>(shares, h->n_bursts, 1.0 / (double)h->windows, objective,
                                              grad ? grad_params : nullptr);
  return s1b_launch_status();
}
