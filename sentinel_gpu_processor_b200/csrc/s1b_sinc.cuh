// The 8-tap windowed-sinc weights and their derivatives as polynomials.
//
// At fraction f the taps k = -3..4 weigh w_k = u_k / sum u, u_k = sinc(k - f)
// (0.5 + 0.5 cos(pi (k - f) / 4)).  They are mirror images, w_k(f) =
// w_{1-k}(1 - f), so with t = f - 1/2 and v = t^2 the pair k = j + 1, -j (j =
// 0..3) is E_j(v) + t O_j(v) and E_j(v) - t O_j(v), and the derivatives d/df
// are A_j(v) + t B_j(v) and -A_j(v) + t B_j(v).  E, O, A and B are of degree 4
// in v and interpolate at the Chebyshev nodes of [0, 1/4] (in extended
// precision, rounded once).  Evaluated in FP32 as below the weights are within
// 1.9e-7 and the derivatives within 1.01e-6 (1.01e-7 and 8.9e-7 of it from the
// rounded coefficients), where a table of 1024 bins with linear interpolation is
// within 4.9e-7 and 1.1e-6 and takes four 128-bit gathers per axis.
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
[[maybe_unused]] static __constant__ float2 c_dsinc8[4 * 5] = {
    {1.316447401e+00f, -9.077257542e-01f}, {-4.157075512e+00f, 1.202532931e-01f}, {2.386238463e+00f,
    4.646045500e-01f}, {1.950642090e-01f, -3.360972442e-01f}, {-6.631490782e-01f, 8.261869454e-02f},
    {-1.742653724e-01f, 1.228249694e+00f}, {2.382144502e+00f, -3.849884962e-01f}, {-1.998631491e+00f,
    -5.647455056e-01f}, {2.699200056e-01f, 4.724721402e-01f}, {3.080874626e-01f, -1.369410292e-01f},
    {6.172634864e-02f, -3.202104065e-01f}, {-8.844464100e-01f, -1.630983445e-02f}, {9.979949162e-01f,
    4.694392015e-01f}, {-2.004400475e-01f, -2.568907704e-01f}, {-1.152097402e-01f, 3.743479825e-02f},
    {-1.461186098e-02f, -3.135329796e-04f}, {2.046962935e-01f, 2.810450376e-01f}, {-1.971883674e-01f,
    -3.692982459e-01f}, {-3.748554609e-04f, 1.205158743e-01f}, {4.499077020e-02f, 1.688753637e-02f},
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
    float2 a = c_dsinc8[j * 5 + 4], r = a;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      const float2 ck = c_dsinc8[j * 5 + k];
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
