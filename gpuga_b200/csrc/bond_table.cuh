// An entry of the bond-order table of tersoff_ev.cu: b(s) = (1 + (beta s)^n)^(-1/2n) and b'(s) over an interval of
// s as one polynomial of degree 6, b = b0 + t (k0 + t (k1 + ...)), t = s - c, in eight 32-bit words.  b0 and k0 have the
// remainders of their rounding beside them: bonds that share few entries do not average it out.  The evaluation that
// uses k0's (FINE) takes three operations more.
//
// b' is what the polynomial is fitted to (degree 5 through six Chebyshev nodes), b its integral from the exact b(c):
// a polynomial through values of b has an error in b' that is 36 times its own at the ends of the interval.
// Which entries represent the function is decided where the error of such an interpolant has its extremes and no node
// lies, at both ends: even and odd terms of what is left out add up at one of them, so no single coefficient that
// happens to be zero can hide the rest.
//
// Bounds for an entry that is accepted (tests/test_bond_table_cpu.py; n from 0.3 to 50): b to 7e-8 of its size, b' to
// 2e-7 of the entry's largest (FINE: 1.3e-7), or of 1e-3 / s where that is larger.  Of that 4e-8 may be the interpolation's;
// the rest is the rounding of the FP32 coefficients and of their evaluation.  On eighths of octaves every entry is accepted
// for n up to 5 (interpolation: 4e-9 for n up to 3); of those with beta s between 0.05 and 8 all but 6 % at n = 8, 15 % at
// n = 12, 18 % at n = 18.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#include "exp_d.cuh"

#ifndef __CUDACC__
#define GPUGA_BT_HD inline
#else
#define GPUGA_BT_HD __host__ __device__ __forceinline__
#endif

namespace gpuga {

struct BondEntry {
  float b0, lo, k[6];  // lo: b0's remainder as a float, whose last 16 bits are k[0]'s (the upper half of a float)
  bool ok;
};

GPUGA_BT_HD uint32_t bt_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t i;
  std::memcpy(&i, &f, 4);
  return i;
#endif
}
GPUGA_BT_HD float bt_float(uint32_t i) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(i);
#else
  float f;
  std::memcpy(&f, &i, 4);
  return f;
#endif
}

// b and b' at s = c + t.
template <bool FINE>
GPUGA_BT_HD void bond_eval(float b0, float lo, float k0, float k1, float k2, float k3, float k4, float k5, float t, float& b,
                           float& db) {
  float p = fmaf(k5, t, k4), d = fmaf(k5, t, p);
  p = fmaf(p, t, k3);
  d = fmaf(d, t, p);
  p = fmaf(p, t, k2);
  d = fmaf(d, t, p);
  p = fmaf(p, t, k1);
  d = fmaf(d, t, p);
  if (FINE) {
    p = fmaf(p, t, bt_float(bt_bits(lo) << 16));
    db = k0 + fmaf(d, t, p);
    b = b0 + fmaf(p, t, fmaf(k0, t, lo));
  } else {
    p = fmaf(p, t, k0);
    db = fmaf(d, t, p);
    b = b0 + fmaf(p, t, lo);
  }
}

// b and db/ds in closed form at s = e^ls; mh = -1/(2n), lbeta = ln beta.  b = 1, b' = 0 below beta s = 1e-16
// (minimal_tersoff.cu:178-185).
GPUGA_BT_HD void bond_order(double n, double mh, double beta, double lbeta, double s, double ls, double& b, double& db) {
  const double z = n * (lbeta + ls);
  const bool big = z > 40.0, tiny = beta * s < 1e-16;  // big: 1 + e^z = e^z
  const double e = big ? 1.0 : exp_d_clamped(z);
  const double v = exp_d_clamped(mh * (big ? z : log(1.0 + e)));
  const double d = -0.5 * v * e / (big ? s : s * (1.0 + e));
  b = tiny ? 1.0 : v;
  db = tiny ? 0.0 : d;
}

// Where an entry is evaluated, in half widths from its center: six Chebyshev nodes, the center, both ends.
constexpr int kBondPoints = 9, kBondCenter = 6;
constexpr double kBondPoint[kBondPoints] = {0.96592582628906829,  0.70710678118654752,  0.25881904510252076, -0.25881904510252076,
                                            -0.70710678118654752, -0.96592582628906829, 0.0,                 -1.0, 1.0};

// The entry c - h .. c + h from h b' at those points (f) and b(c).
GPUGA_BT_HD BondEntry bond_fit(const double (&f)[kBondPoints], double bc, double c, double h) {
  constexpr double x[3] = {0.96592582628906829, 0.70710678118654752, 0.25881904510252076};
  double top = 0.0;
  for (int m = 0; m < 6; ++m) top = fmax(top, fabs(f[m]));
  // Chebyshev coefficients (T_k at the nodes: cos(k pi (2m + 1) / 12)), then powers of t / h
  const double e0 = f[0] + f[5], e1 = f[1] + f[4], e2 = f[2] + f[3];
  const double o0 = f[0] - f[5], o1 = f[1] - f[4], o2 = f[2] - f[3];
  const double a0 = (e0 + e1 + e2) / 6.0;
  const double a1 = (o0 * x[0] + o1 * x[1] + o2 * x[2]) / 3.0;
  const double a2 = (e0 - e2) * (0.86602540378443865 / 3.0);
  const double a3 = (o0 - o1 - o2) * (0.70710678118654752 / 3.0);
  const double a4 = (0.5 * e0 - e1 + 0.5 * e2) / 3.0;
  const double a5 = (o0 * x[2] - o1 * x[1] + o2 * x[0]) / 3.0;
  const double p[6] = {a0 - a2 + a4, a1 - 3.0 * a3 + 5.0 * a5, 2.0 * a2 - 8.0 * a4, 4.0 * a3 - 20.0 * a5, 8.0 * a4,
                       16.0 * a5};
  const double even = p[0] + p[2] + p[4], odd = p[1] + p[3] + p[5];
  const double left = fmax(fabs(even + odd - f[8]), fabs(even - odd - f[7]));
  BondEntry o;
  o.ok = left <= 4e-8 * fmax(top, 1e-3 * h / c);  // (a NaN is not)
  o.b0 = (float)bc;
  const double ih = 1.0 / h;
  double s = ih;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int j = 0; j < 6; ++j) {
    const double k = p[j] * s / (j + 1);
    o.k[j] = (float)k;
    o.ok = o.ok && fabs(k) <= 1e37;  // (intervals near s = 0: beyond FP32)
    s *= ih;
  }
  const float k0lo = (float)(p[0] * ih - (double)o.k[0]);
  o.lo = bt_float((bt_bits((float)(bc - (double)o.b0)) & 0xffff0000u) | (bt_bits(k0lo) >> 16));
  return o;
}

}  // namespace gpuga
