// One refinement of a pose from Horn's problem with S and the centres as
// (hi, lo) pairs (sm_103a).
//
// The FP32 solve (horn_quaternion_fast) leaves the quaternion ~2e-7 off, and the
// pose it gives enters the next E-step times 1 / sigma: at sigma = 3e-3 that is
// the largest error of EM-ICP's rows and of its gradients. A Rayleigh residual
// r = N v - lambda v in pairs, one solve (sigma I - N) d = r in FP32 and R, t in
// pairs leave the rounding of R and t themselves: gradients at 10,007 x 9001
// 2.6e-6 / 7.3e-6 (two seeds) -> 1.4e-6 / 2.4e-6 relative to FP64. One thread,
// ~2 us of a step (by a warp 1.3 us, but the sweeps around it came out 8% slower).
#pragma once
#include "cesa_common.cuh"
#include "cesa_pose.h"

namespace cesa {

// S, Sl: cross-covariance (h_S layout); Xc, Xl, Yc, Yl: centres; q: the FP32
// solve's quaternion. Writes q, R and t = Xc - R Yc; leaves them as they are where
// the shifted matrix is not positive definite or the step is not small.
static __device__ __forceinline__ void horn_refine_dd(const float* S, const float* Sl, const float* Xc, const float* Xl,
                                                   const float* Yc, const float* Yl, float* q, float* R,
                                                   float* t) {
  // Horn's N entry by entry: hi and lo parts are both linear in S
  float Nh[4][4], Nl[4][4], scale = 0.f;
  {
    auto add = [](df a, float sb, df b) {
      df_add(a, df{sb * b.hi, sb * b.lo});
      return a;
    };
    auto s = [&](int k) { return dd_fast(S[k], Sl[k]); };
    auto put = [&](int i, int j, df v) {
      v = dd_fast(v.hi, v.lo);
      Nh[i][j] = Nh[j][i] = v.hi;
      Nl[i][j] = Nl[j][i] = v.lo;
      scale = fmaxf(scale, fabsf(v.hi));
    };
    const df xx = s(0), xy = s(1), xz = s(2), yx = s(3), yy = s(4), yz = s(5), zx = s(6), zy = s(7), zz = s(8);
    put(0, 0, add(add(xx, 1.f, yy), 1.f, zz));
    put(1, 1, add(add(xx, -1.f, yy), -1.f, zz));
    put(2, 2, add(add(yy, -1.f, xx), -1.f, zz));
    put(3, 3, add(add(zz, -1.f, xx), -1.f, yy));
    put(0, 1, add(yz, -1.f, zy));
    put(0, 2, add(zx, -1.f, xz));
    put(0, 3, add(xy, -1.f, yx));
    put(1, 2, add(xy, 1.f, yx));
    put(1, 3, add(zx, 1.f, xz));
    put(2, 3, add(yz, 1.f, zy));
  }
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = q[i];
  df nv[4], num = df_make(0.f), den = df_make(-1.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    nv[i] = df_make(0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      df_add_prod(nv[i], Nh[i][j], v[j]);
      nv[i].lo = __fmaf_rn(Nl[i][j], v[j], nv[i].lo);
    }
    nv[i] = dd_fast(nv[i].hi, nv[i].lo);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    df_add(num, dd_mul(nv[i], df_make(v[i])));
    df_add_prod(den, v[i], v[i]);
  }
  // lambda = num / |v|^2, |v|^2 = 1 + den with den ~ 1e-7
  const float dn = df_val(den);
  num = dd_fast(num.hi, num.lo);
  df lam = num;
  df_add(lam, -num.hi * dn);
  lam = dd_fast(lam.hi, lam.lo);
  float r[4], A[4][4], L[4][4], rd[4];
  const float sigma = lam.hi + 1e-3f * scale;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    df e = nv[i];
    const df lv = dd_mul(lam, df_make(v[i]));
    df_add(e, df{-lv.hi, -lv.lo});
    r[i] = df_val(e);
#pragma unroll
    for (int j = 0; j < 4; ++j) A[i][j] = (i == j ? sigma : 0.f) - Nh[i][j];
  }
  if (!chol4<float>(A, L, rd)) return;
  float y[4], d[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float x = r[i];
#pragma unroll
    for (int k = 0; k < i; ++k) x -= L[i][k] * y[k];
    y[i] = x * rd[i];
  }
#pragma unroll
  for (int i = 3; i >= 0; --i) {
    float x = y[i];
#pragma unroll
    for (int k = i + 1; k < 4; ++k) x -= L[k][i] * d[k];
    d[i] = x * rd[i];
  }
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) big = fmaxf(big, fabsf(d[i]));
  if (!(big < 1e-3f)) return;
  df w[4], n2 = df_make(-1.f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    w[i] = dd_sum(v[i], d[i]);
    df_add(n2, dd_mul(w[i], w[i]));
  }
  const float h = -0.5f * df_val(n2);  // 1/|w| = 1 + h to ~1e-12
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    df_add(w[i], w[i].hi * h);
    w[i] = dd_fast(w[i].hi, w[i].lo);
    q[i] = w[i].hi;
  }
  df p[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = i; j < 4; ++j) p[i][j] = dd_mul(w[i], w[j]);
  auto sum2 = [](df a, float sb, df b) {  // 2 (a + sb b)
    df_add(a, df{sb * b.hi, sb * b.lo});
    return df{2.f * a.hi, 2.f * a.lo};
  };
  auto diag = [](df a, df b, df c, df e) {  // a + b - c - e
    df_add(a, b);
    df_add(a, df{-c.hi, -c.lo});
    df_add(a, df{-e.hi, -e.lo});
    return a;
  };
  df M[9];
  M[0] = diag(p[0][0], p[1][1], p[2][2], p[3][3]);
  M[4] = diag(p[0][0], p[2][2], p[1][1], p[3][3]);
  M[8] = diag(p[0][0], p[3][3], p[1][1], p[2][2]);
  M[1] = sum2(p[1][2], -1.f, p[0][3]);
  M[2] = sum2(p[1][3], 1.f, p[0][2]);
  M[3] = sum2(p[1][2], 1.f, p[0][3]);
  M[5] = sum2(p[2][3], -1.f, p[0][1]);
  M[6] = sum2(p[1][3], -1.f, p[0][2]);
  M[7] = sum2(p[2][3], 1.f, p[0][1]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    df a = dd_fast(Xc[i], Xl[i]);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const df m = dd_fast(M[3 * i + j].hi, M[3 * i + j].lo);
      R[3 * i + j] = df_val(m);
      const df e = dd_mul(m, dd_fast(Yc[j], Yl[j]));
      df_add(a, df{-e.hi, -e.lo});
    }
    t[i] = df_val(a);
  }
}

}  // namespace cesa
