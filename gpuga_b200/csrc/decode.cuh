// Decoded parameters and derived constants of an individual, shared by the kernels that form them
// (batched.cu, spectral.cu).
#pragma once
#include "engine.hpp"

namespace gpuga {

// ----------------------------------------------------------------- per-individual constants
// Tersoff (minimal_tersoff.cu:39-75): per pair set s: lr = sqrt(2S)*A, la = sqrt(2/S)*A,
// cr = D0/(S-1), ca = S*D0/(S-1), r0; then n, beta, h, R1, R2, pi/(R2-R1), -1/(2n); then the
// FP64 remainders of lr, la, cr, ca and -1/(2n).  The FP32 rounding of these derived constants
// is the same for every bond of an individual, so it does not average out: cr, ca and lr, la
// enter fr' - b fa', which cancels near equilibrium, and -1/(2n) every bond order.  Without
// the remainders the fitness of a parameter set with S != 2 was off by up to 1e-5 relative.
enum { TC_LR = 0, TC_LA = 2, TC_CR = 4, TC_CA = 6, TC_R0 = 8, TC_EN = 10, TC_BETA, TC_H, TC_R1, TC_R2, TC_PF,
       TC_MHON, TC_LRL, TC_LAL = TC_LRL + 2, TC_CRL = TC_LAL + 2, TC_CAL = TC_CRL + 2, TC_MHONL = TC_CAL + 2,
       TC_COUNT };
static_assert(TC_COUNT <= kMaxConsts, "per-individual Tersoff constants");
// RI (ri.cu:36-110), pair-by-pair part in FP32: Buckingham A[3], b[3] = 1/rho and its FP64
// remainder (the exponent d/rho reaches ~20, where the FP32 rounding of b alone would move
// e^{-d/rho} by ~1e-6), the cation-anion Morse constants lr, la (with remainders), cr, ca (with
// remainders) and r0.  The linear part (damped shifted Coulomb and dispersion) takes FP64
// constants: qq[3] (K_C included), C[3], v_rc, dv_rc, rc and the self-energy coefficient.
enum { RC_A = 0, RC_B = 3, RC_BLO = 6, RC_LR = 9, RC_LA, RC_LRLO, RC_LALO, RC_CR, RC_CA, RC_CRLO, RC_CALO, RC_R0,
       RC_COUNT };
static_assert(RC_COUNT <= kMaxConsts, "per-individual RI constants");
enum { R64_QQ = 0, R64_C = 3, R64_VRC = 6, R64_DVRC, R64_RC, R64_SELF, R64_COUNT };

__device__ __forceinline__ float decode1(float mn, float mx, float x) {
  return __fadd_rn(mn, __fmul_rn(__fsub_rn(mx, mn), x));  // fitness.cu:320-324, no contraction
}

// Individual p by one thread: FP32 decode exactly like the reference, derived constants in FP64 rounded
// once to FP32.
__device__ __forceinline__ void decode_individual(const JobView& J, int p) {
  const int nv = J.num_vars, Pstride = J.Pstride, potential_type = J.potential_type;
  const int num_types = J.num_types;
  const float* __restrict__ pmin = J.pmin;
  const float* __restrict__ pmax = J.pmax;
  float* __restrict__ consts = J.consts;
  float* __restrict__ weights = J.weights;
  const float* x = J.pop + (size_t)p * nv;
  auto par = [&](int m) { return (double)decode1(pmin[m], pmax[m], x[m]); };
  auto put = [&](int k, double v) { consts[(size_t)k * Pstride + p] = (float)v; };
  auto put_lo = [&](int k, double v) { consts[(size_t)k * Pstride + p] = (float)(v - (double)(float)v); };
  if (potential_type == 1 || potential_type == 2) {
    const int off = num_types == 2 ? 4 : 0;
    for (int s = 0; s < 2; ++s) {
      const int q = (num_types == 2 && s == 1) ? 4 : 0;
      const double D0 = par(q + 0), A = par(q + 1), R0 = par(q + 2), S = par(q + 3);
      put(TC_LR + s, sqrt(2.0 * S) * A);
      put(TC_LA + s, sqrt(2.0 / S) * A);
      put(TC_CR + s, D0 / (S - 1.0));
      put(TC_CA + s, S * D0 / (S - 1.0));
      put(TC_R0 + s, R0);
      put_lo(TC_LRL + s, sqrt(2.0 * S) * A);
      put_lo(TC_LAL + s, sqrt(2.0 / S) * A);
      put_lo(TC_CRL + s, D0 / (S - 1.0));
      put_lo(TC_CAL + s, S * D0 / (S - 1.0));
    }
    const double en = par(4 + off), R1 = par(7 + off), R2 = par(8 + off);
    put(TC_EN, en);
    put(TC_BETA, par(5 + off));
    put(TC_H, par(6 + off));
    put(TC_R1, R1);
    put(TC_R2, R2);
    put(TC_PF, M_PI / (R2 - R1));
    put(TC_MHON, -0.5 / en);
    put_lo(TC_MHONL, -0.5 / en);
  } else if (is_ri_type(potential_type)) {
    double* __restrict__ c64 = J.consts64;
    auto put64 = [&](int k, double v) { c64[(size_t)k * Pstride + p] = v; };
    const double q0 = par(0), ratio = ri_charge_ratio(potential_type);
    const double kc = 14.399645;  // ri.cu:29
    put64(R64_QQ + 0, q0 * q0 * kc);
    put64(R64_QQ + 1, ratio * q0 * q0 * kc);
    put64(R64_QQ + 2, ratio * ratio * q0 * q0 * kc);
    for (int t = 0; t < 3; ++t) {
      put(RC_A + t, par(1 + 3 * t));
      put(RC_B + t, 1.0 / par(2 + 3 * t));
      put_lo(RC_BLO + t, 1.0 / par(2 + 3 * t));
      put64(R64_C + t, par(3 + 3 * t));
    }
    const double rc = par(10), alpha = 0.2, pif = 0.225675833419103;
    put64(R64_VRC, erfc(alpha * rc) / rc);
    put64(R64_DVRC, -erfc(alpha * rc) / (rc * rc) - pif * exp(-alpha * alpha * rc * rc) / rc);
    put64(R64_RC, rc);
    const double d0 = par(11), al = par(12), r0 = par(13), s = par(14);
    put(RC_LR, sqrt(2.0 * s) * al);
    put(RC_LA, sqrt(2.0 / s) * al);
    put_lo(RC_LRLO, sqrt(2.0 * s) * al);
    put_lo(RC_LALO, sqrt(2.0 / s) * al);
    put(RC_CR, d0 / (s - 1.0));
    put(RC_CA, s * d0 / (s - 1.0));
    put_lo(RC_CRLO, d0 / (s - 1.0));
    put_lo(RC_CALO, s * d0 / (s - 1.0));
    put(RC_R0, r0);
    // damped-Coulomb self energy per unit (q_i / q)^2 (develop/hfo2/find_E.m:10-13)
    put64(R64_SELF, J.ri_self ? q0 * q0 * kc *
                                    (alpha / sqrt(M_PI) + erfc(alpha * rc) / rc +
                                     0.5 * pif * exp(-alpha * alpha * rc * rc))
                              : 0.0);
  } else {
    for (int m = 0; m < nv; ++m) weights[(size_t)m * Pstride + p] = decode1(pmin[m], pmax[m], x[m]);
  }
}

struct Consts {
  const float* base;
  int stride;
  int p;
  __device__ __forceinline__ float operator[](int k) const { return __ldg(base + (size_t)k * stride + p); }
};

}  // namespace gpuga
