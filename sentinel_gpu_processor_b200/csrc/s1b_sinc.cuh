// The 8-tap windowed-sinc weights and their derivatives as polynomials.
//
// At fraction f the taps k = -3..4 weigh w_k = u_k / sum u, u_k = sinc(k - f)
// (0.5 + 0.5 cos(pi (k - f) / 4)).  They are mirror images, w_k(f) =
// w_{1-k}(1 - f), so with t = f - 1/2 and v = t^2 the pair k = j + 1, -j (j =
// 0..3) is E_j(v) + t O_j(v) and E_j(v) - t O_j(v), and the derivatives d/df
// are A_j(v) + t B_j(v) and -A_j(v) + t B_j(v).
//
// E and O are of degree 4 in v and interpolate at the Chebyshev nodes of [0, 1/4]
// (in extended precision, rounded once).  Evaluated in FP32 as below the weights
// are within 1.9e-7; a table of 1024 bins with linear interpolation is within
// 4.9e-7 and takes four 128-bit gathers per axis.
//
// A and B are of degree 5 and belong to weights from such a table, which the
// adjoint keeps: linear interpolation adds h^2/12 times the second derivative (h =
// 1/1024) to what it interpolates, in the mean, so the slopes are fitted to w' +
// h^2/12 w''' (least squares, the coefficients rounded one after another, each
// fitted with the roundings before it: the slopes' mean over the fractions is
// within 1e-8 of a table's).  Without that term the parameter gradients, sums over
// all pixels, were 1.5 to 2.5 times as far from float64; with it they are as close
// as with a table of the slopes.  From w' itself they are within 7.6e-7 (a table
// within 1.1e-6).
#ifndef S1B_SINC_CUH
#define S1B_SINC_CUH

#include <cuda_runtime.h>

// (E, O) and (A, B), lowest power of v first, j = 0..3
[[maybe_unused]] static __constant__ float2 c_sinc8[4 * 5] = {
    {6.105329107e-01f, 1.316446621e+00f}, {-4.538659329e-01f, -1.385650424e+00f}, {3.016230370e-02f,
    4.766528965e-01f}, {7.631633308e-02f, 3.103252100e-02f}, {-3.687180599e-02f, -7.930388117e-02f},
    {-1.462624267e-01f, -1.742648246e-01f}, {6.141299856e-01f, 7.940191455e-01f}, {-9.641264395e-02f,
    -3.993102299e-01f}, {-9.226228625e-02f, 3.634804905e-02f}, {5.052040383e-02f, 3.815482832e-02f},
    {3.918042955e-02f, 6.172609592e-02f}, {-1.601065027e-01f, -2.948020942e-01f}, {-4.034295357e-03f,
    1.994073622e-01f}, {7.774411245e-02f, -2.761609895e-02f}, {-2.980353594e-02f, -1.460614983e-02f},
    {-3.450913596e-03f, -1.461180386e-02f}, {-1.575500278e-04f, 6.822906548e-02f}, {7.028463561e-02f,
    -3.939414541e-02f}, {-6.179815928e-02f, -2.851676288e-04f}, {1.615493810e-02f, 5.410020769e-03f},
};
[[maybe_unused]] static __constant__ float2 c_dsinc8[4 * 6] = {
    {1.316445947e+00f, -9.077257514e-01f}, {-4.156908512e+00f, 1.202650145e-01f}, {2.380939484e+00f,
    4.642541409e-01f}, {2.545031607e-01f, -3.322084546e-01f}, {-9.350069165e-01f, 6.493065506e-02f},
    {4.350179434e-01f, 2.819302864e-02f}, {-1.742644012e-01f, 1.228249550e+00f}, {2.382024527e+00f,
    -3.849985003e-01f}, {-1.994865060e+00f, -5.644497275e-01f}, {2.278422564e-01f, 4.691835940e-01f},
    {5.001379848e-01f, -1.219707802e-01f}, {-3.069335520e-01f, -2.386214584e-02f}, {6.172593310e-02f,
    -3.202104867e-01f}, {-8.843908906e-01f, -1.629424095e-02f}, {9.962563515e-01f, 4.689634144e-01f},
    {-1.810327768e-01f, -2.515847385e-01f}, {-2.037504315e-01f, 1.323884167e-02f}, {1.414684951e-01f,
    3.863516450e-02f}, {-1.461176574e-02f, -3.133237769e-04f}, {2.046836615e-01f, 2.810284197e-01f},
    {-1.967915148e-01f, -3.687810004e-01f}, {-4.810087383e-03f, 1.147192195e-01f}, {6.523892283e-02f,
    4.338708520e-02f}, {-3.236671165e-02f, -4.238435999e-02f},
};

// The 8 weights at the fraction f in [0, 1).
__device__ __forceinline__ void sinc8_weights(float f, float w[8]) {
  const float t = f - 0.5f, v = t * t;
  const float2 vv = make_float2(v, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 p = c_sinc8[j * 5 + 4];
#pragma unroll
    for (int k = 3; k >= 0; --k) p = __ffma2_rn(p, vv, c_sinc8[j * 5 + k]);
    w[4 + j] = fmaf(t, p.y, p.x);
    w[3 - j] = fmaf(-t, p.y, p.x);
  }
}

// The derivatives of the 8 weights at two fractions in [0, 1): both at once,
// so that each coefficient is fetched once.
__device__ __forceinline__ void sinc8_slopes(float fa, float fr, float da[8], float dr[8]) {
  const float ta = fa - 0.5f, tr = fr - 0.5f, va = ta * ta, vr = tr * tr;
  const float2 va2 = make_float2(va, va), vr2 = make_float2(vr, vr);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 a = c_dsinc8[j * 6 + 5], r = a;
#pragma unroll
    for (int k = 4; k >= 0; --k) {
      const float2 ck = c_dsinc8[j * 6 + k];
      a = __ffma2_rn(a, va2, ck);
      r = __ffma2_rn(r, vr2, ck);
    }
    da[4 + j] = fmaf(ta, a.y, a.x);
    dr[4 + j] = fmaf(tr, r.y, r.x);
    da[3 - j] = fmaf(ta, a.y, -a.x);
    dr[3 - j] = fmaf(tr, r.y, -r.x);
  }
}

#endif
