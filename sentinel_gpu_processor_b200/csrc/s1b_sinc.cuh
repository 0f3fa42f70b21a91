// The 8-tap windowed-sinc weights and their derivatives as polynomials.
//
// At fraction f the taps k = -3..4 weigh w_k = u_k / sum u, u_k = sinc(k - f)
// (0.5 + 0.5 cos(pi (k - f) / 4)).  They are mirror images, w_k(f) =
// w_{1-k}(1 - f), so with t = f - 1/2 and v = t^2 the pair k = j + 1, -j (j =
// 0..3) is E_j(v) + t O_j(v) and E_j(v) - t O_j(v), and the derivatives d/df
// are A_j(v) + t B_j(v) and -A_j(v) + t B_j(v).  E and O are of degree 4 in v, A
// and B of degree 5, and they interpolate at the Chebyshev nodes of [0, 1/4] (in
// extended precision, rounded once).  Evaluated in FP32 as below the weights are
// within 1.9e-7 and the derivatives within 2.0e-7 of them; a table of 1024 bins
// with linear interpolation is within 4.9e-7 and 1.1e-6 and takes four 128-bit
// gathers per axis (derivatives of degree 4: 1.01e-6, and 1.1 to 1.8 times the table's
// error in the mean square).
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
    {1.316446552e+00f, -9.077258134e-01f}, {-4.156906408e+00f, 1.202647961e-01f}, {2.380842802e+00f,
    4.642433924e-01f}, {2.553677144e-01f, -3.321071802e-01f}, {-9.383782774e-01f, 6.456524600e-02f},
    {4.398094776e-01f, 2.865423690e-02f}, {-1.742647798e-01f, 1.228249747e+00f}, {2.382026827e+00f,
    -3.849987145e-01f}, {-1.994884054e+00f, -5.644276188e-01f}, {2.280949945e-01f, 4.689836808e-01f},
    {4.987843807e-01f, -1.212380991e-01f}, {-3.044875765e-01f, -2.482252343e-02f}, {6.172607596e-02f,
    -3.202104851e-01f}, {-8.843923273e-01f, -1.629440105e-02f}, {9.962739779e-01f, 4.689513403e-01f},
    {-1.812433636e-01f, -2.514744057e-01f}, {-2.026988351e-01f, 1.283687023e-02f}, {1.396497900e-01f,
    3.915512843e-02f}, {-1.461179888e-02f, -3.134484851e-04f}, {2.046839378e-01f, 2.810283195e-01f},
    {-1.967943612e-01f, -3.687671139e-01f}, {-4.776554293e-03f, 1.145979051e-01f}, {6.507418728e-02f,
    4.383598285e-02f}, {-3.208509976e-02f, -4.298684190e-02f},
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
