// Energy/virial items of the minimal Tersoff potential, pair by pair.
//
// With R1 and R2 fixed by their bounds (every potential.in of the reference) the cutoff is geometry, and a
// directed bond ij of an energy/virial configuration needs the individual's parameters in three places only:
//   s_ij = sum_k fc_ik (cos_jik - h)^2,     zeta = beta s,     b(s) = (1 + (beta s)^n)^(-1/2n),
//   E    = sum 1/2 fc (fr - b fa),
//   W    = -dE/d(strain) = sum [-1/2 A' d u (x) u + 1/2 fc fa b'(s) X(h)],   X = ds/d(strain),
// A' = fc' (fr - b fa) + fc (fr' - b fa') (minimal_tersoff.cu:122-405 sums the same tensor as -r_ij (x) f_ij;
// it is symmetric because a site energy does not change under rotation).  s and X are polynomials in
// dh = h - h0 (h0: the middle of the bounds of h), s = A + dh (B + dh C), X = X0 + dh (X1 + dh X2), whose
// coefficients are sums over k that are formed once per training set in FP64.  The two bonds of a pair share d, fc
// and the exponentials, and E and A' are linear in b, so they enter as b_ij + b_ji.  What remains per (individual,
// pair) is twice s, b and b', the pair terms once and 30 FMAs for W: no loop over triplets, and the same work for
// any number of neighbors.
//
// b and b' come from a table per individual, polynomials of degree 6 on eighths of octaves of s (bond_table.cuh):
// t = s - s_c is exact, so b is rounded once (5.9e-8 relative; powf_dd, which it replaces, 6.2e-8) and b' to 2e-7.  The FP64
// pair exponentials e^{-l t} come from a table on a 1/32 A grid and a polynomial of the rest, |l delta| <= l / 64, of
// degree m, which leaves out (l / 64)^(m + 1) / (m + 1)!: 3e-11 for m = 5 up to l = 3.38 A^-1 (alpha 1.5 with S 2.5) and for
// m = 9 up to 25.  Tables are per individual, lane-private in shared memory (no bank conflicts whatever a lane's index)
// and rebuilt each generation (tersoff_tables).  s outside the table, an individual whose n is too sharp for it (checked
// when it is built) or whose l is beyond the polynomial takes powf_dd and exp_d.
//
// Two forms of the items (TersoffEvView::wide).  The plain one has m = 5 and evaluates a batch that needs powf_dd a second
// time; the other m = 9, powf_dd bond by bond, and the fine evaluation of b'.  It is taken where
//   the bounds allow l above 3.38 (one that allows l above 25 leaves the set to the items by atom);
//   n may be above 5: 67 configurations of up to 1000 atoms at population 333 with n from 8 to 12 and beta s around 1, 394 us
//   a generation (530 in the plain form, 458 by atom), but 202 against 192 us for n below 0.8;
//   atoms have more than four bonds on average: the bonds of such crystals share few entries, and the rounding of an entry's
//   first coefficient does not average out (fitness error, geometric mean over 12 sets of 4 to 14 neighbors: plain 1.9e-8,
//   fine 1.0e-8, by atom 1.65e-8; sets of four neighbors: below that of the items by atom in either form).
#include <algorithm>
#include <cmath>
#include <cstring>

#include <cuda_pipeline.h>

#include "bond_table.cuh"
#include "decode.cuh"
#include "engine.hpp"
#include "exp_d.cuh"
#include "fold.cuh"
#include "powf_dd.cuh"

namespace gpuga {

namespace {

constexpr int kEvThreads = 384, kEvW = kEvThreads / 32;
constexpr int kEvBatch = 2;           // pairs that a warp takes at a time
constexpr int kEvConsts = 10;         // doubles per individual: la, ca, lr, cr of both pair sets, dh (and one unused)
constexpr int kSetBit = 1 << 16, kShellBit = 1 << 17;  // EvPair::code: pair set; a neighbor lies in R1 .. R2 (of any pair of the batch)
constexpr int kTabMax = 80, kExpMax = 96;
constexpr double kStep = 1.0 / 32.0;  // distance grid
constexpr double kExpFlat = 3.38, kExpSteep = 25.0;  // steepest exponential of the two polynomials, 1 / A

// bytes of an individual group's tables (32 lanes): b as two float4 per entry (the last entry, NaN, stands for
// every s outside the table), exponentials, constants
__host__ __device__ inline size_t tab_b_bytes(const TersoffEvView& v) { return (size_t)(v.tab_n + 1) * 32 * 32; }
__host__ __device__ inline size_t tab_bytes(const TersoffEvView& v) {
  return tab_b_bytes(v) + (size_t)v.n_exp * v.exp_n * 256 + kEvConsts * 256;
}

// centre and half width of entry i: eighths of octaves of s, by the top bits of its FP32 representation
__device__ __forceinline__ float entry_center(int i, int base) {
  return __int_as_float(((i + base) << 20) | 0x00080000);
}

// ------------------------------------------------------------------------------ set-up
// Per energy/virial atom: its pairs (neighbors of higher index) inside R2 and the range of d, and whether every bond
// has its reverse (count); then (fill) the coefficients of each of its bonds, into the pair's slot.
template <bool FILL>
__global__ void ev_bonds(int atom0, int n_atoms, const int* __restrict__ off, const int* __restrict__ nbr,
                         const int* __restrict__ rev, int* __restrict__ slot, const uint8_t* __restrict__ ptype,
                         const double4* __restrict__ g64, double r1, double r2, double h0, const int* __restrict__ start,
                         const int* __restrict__ place, int* __restrict__ count, EvPair* __restrict__ out,
                         float4* __restrict__ out2,
                         double2* __restrict__ range) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n_atoms) return;
  const int i = atom0 + a, b0 = off[i], be = off[i + 1];
  auto cutoff = [&](double d, double& fc, double& fcp) {
    fc = 1.0;
    fcp = 0.0;
    if (d >= r2) {
      fc = 0.0;
    } else if (d >= r1) {
      const double pf = M_PI / (r2 - r1);
      double s, c;
      sincos(pf * (d - r1), &s, &c);
      fc = 0.5 * c + 0.5;
      fcp = -0.5 * pf * s;
    }
  };
  int n = 0;
  double smin = 1e300, smax = 0.0;
  for (int b = b0; b < be; ++b) {
    const double4 v = g64[b];
    if (!(v.w < r2)) continue;
    const bool first = nbr[b] > i;  // the pair's first bond
    if (!FILL) {
      smin = fmin(smin, v.w);
      smax = fmax(smax, v.w);
      const int r = rev[b];
      if (nbr[r] != i || g64[r].w != v.w || nbr[b] == i) smax = 1e300;  // no such pair: the set is left to the items by atom
      if (first) slot[b] = n++;
      continue;
    }
    const double ij = 1.0 / v.w, uj[3] = {v.x * ij, v.y * ij, v.z * ij};
    double A = 0.0, B = 0.0, C = 0.0, X0[6] = {}, X1[6] = {}, X2[6] = {};
    bool shell = false;
    constexpr int ra[6] = {0, 1, 2, 0, 1, 2}, rb[6] = {0, 1, 2, 1, 2, 0};
    for (int k = b0; k < be; ++k) {
      if (k == b) continue;
      const double4 w = g64[k];
      if (!(w.w < r2)) continue;
      const double ik = 1.0 / w.w, uk[3] = {w.x * ik, w.y * ik, w.z * ik};
      double fc, fcp;
      cutoff(w.w, fc, fcp);
      shell |= fcp != 0.0;
      const double c = uj[0] * uk[0] + uj[1] * uk[1] + uj[2] * uk[2], y = c - h0;
      A += fc * y * y;
      B -= 2.0 * fc * y;
      C += fc;
      for (int t = 0; t < 6; ++t) {
        const double jk = uj[ra[t]] * uk[rb[t]] + uk[ra[t]] * uj[rb[t]];
        const double kk = uk[ra[t]] * uk[rb[t]];
        const double T = 2.0 * fc * (jk - c * (uj[ra[t]] * uj[rb[t]] + kk)), S = fcp * w.w * kk;
        X0[t] += S * y * y + y * T;
        X1[t] -= 2.0 * S * y + T;
        X2[t] += S;
      }
    }
    double fc, fcp;
    cutoff(v.w, fc, fcp);
    const int fb = first ? b : rev[b];  // the pair's first bond: its slot among its atom's pairs
    const int o = place[start[(first ? i : nbr[b]) - atom0] + slot[fb]], h = first ? 0 : 1;
    EvPair& q = out[o];
    q.A[h] = A;
    q.B[h] = B;
    q.C[h] = C;
    for (int t = 0; t < 6; ++t) {
      q.X[h][0][t] = (float)X0[t];
      q.X[h][1][t] = (float)X1[t];
    }
    out2[4 * (size_t)o + 2 * h] = make_float4((float)X2[0], (float)X2[1], (float)X2[2], (float)X2[3]);
    out2[4 * (size_t)o + 2 * h + 1] = make_float4((float)X2[4], (float)X2[5], shell ? 1.f : 0.f, 0.f);
    if (first) {
      const int grid = (int)rint(v.w * 32.0);
      q.delta = v.w - grid * kStep;
      q.hfc = 0.5 * fc;
      q.hfcp = 0.5 * fcp;
      q.hfc32 = (float)(0.5 * fc);
      q.code = grid | (ptype[b] ? kSetBit : 0);
      for (int t = 0; t < 6; ++t) q.D[t] = (float)(v.w * uj[ra[t]] * uj[rb[t]]);
      q.pad[0] = q.pad[1] = 0.f;
    }
    // least and largest s for h within its bounds (range[0].x, .y: the bounds less h0): ends and vertex
    const double lo = range[0].x, hi = range[0].y;
    const double e0 = A + lo * (B + lo * C), e1 = A + hi * (B + hi * C);
    smin = fmin(smin, fmin(e0, e1));
    smax = fmax(smax, fmax(e0, e1));
    if (C > 0.0) {
      const double x = -0.5 * B / C;
      if (x > lo && x < hi) smin = fmin(smin, A + x * (B + x * C));
    }
  }
  if (!FILL) count[a] = n;
  range[1 + a] = make_double2(smin, smax);
}

// Per batch: a slot beyond a segment's last pair repeats it with weight zero, and every pair's shell bit becomes the
// batch's.
__global__ void ev_batches(int n, const int* __restrict__ last, EvPair* __restrict__ pairs, float4* __restrict__ shell) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int b0 = t * kEvBatch, l = last[t];  // last real pair of the batch
  int bit = 0;
  for (int b = b0; b < b0 + kEvBatch; ++b) {
    if (b > l) {
      pairs[b] = pairs[l];
      pairs[b].hfc = pairs[b].hfcp = 0.0;
      pairs[b].hfc32 = 0.f;
      for (int k = 0; k < 4; ++k) shell[4 * (size_t)b + k] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else if (shell[4 * (size_t)b + 1].z != 0.f || shell[4 * (size_t)b + 3].z != 0.f) {
      bit = kShellBit;
    }
  }
  for (int b = b0; b < b0 + kEvBatch; ++b) pairs[b].code |= bit;
}

// ------------------------------------------------------------------------------ tables
// One CTA per (group of 32 individuals, entry of b): a warp per point of the entry (a chain of some 100 dependent FP64
// operations each), then the polynomials of b and b' (bond_table.cuh) by one of them, NaN where they are not exact enough.
// The last CTAs of a group hold its exponentials, one per warp, and the constants.
constexpr int kTabThreads = 32 * kBondPoints;
__host__ __device__ inline int tab_ctas(const TersoffEvView& v) {
  return v.tab_n + (v.n_exp * v.exp_n + kBondPoints) / kBondPoints;
}
__global__ void __launch_bounds__(kTabThreads) tersoff_tables(const JobView* __restrict__ jobs, const int2* __restrict__ groups) {
  const int2 jg = groups[blockIdx.x];
  const JobView& J = jobs[jg.x];
  const TersoffEvView& v = J.ev;
  if ((int)blockIdx.y >= tab_ctas(v)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = jg.y * 32 + lane < J.P ? jg.y * 32 + lane : J.P - 1;  // lanes without an individual repeat the last
  auto par = [&](int m) { return (double)decode1(J.pmin[m], J.pmax[m], J.pop[(size_t)p * J.num_vars + m]); };
  unsigned char* tab = v.tables + (size_t)jg.y * tab_bytes(v);
  float4* ta = reinterpret_cast<float4*>(tab);  // [entry][2][32]
  double* te = reinterpret_cast<double*>(tab + tab_b_bytes(v));
  double* tk = te + (size_t)v.n_exp * v.exp_n * 32;
  const int off = J.num_types == 2 ? 4 : 0;
  const float nan = __int_as_float(0x7fc00000);
  if ((int)blockIdx.y < v.tab_n) {
    __shared__ double at[kBondPoints + 1][32];
    const int i = blockIdx.y;
    const double n = par(4 + off), beta = par(5 + off);
    const double c = entry_center(i, v.tab_base), h = c - (double)__int_as_float((i + v.tab_base) << 20);
    const double2 x = v.points[(size_t)i * kBondPoints + warp];
    double b, db;
    bond_order(n, -0.5 / n, beta, log(beta), x.x, x.y, b, db);
    at[warp][lane] = h * db;
    if (warp == kBondCenter) at[kBondPoints][lane] = b;
    __syncthreads();
    if (warp > 0) return;
    double f[kBondPoints];
#pragma unroll
    for (int k = 0; k < kBondPoints; ++k) f[k] = at[k][lane];
    const BondEntry e = bond_fit(f, at[kBondPoints][lane], c, h);
    // not represented: taken as outside the table
    ta[i * 64 + lane] = make_float4(e.ok ? e.b0 : nan, e.lo, e.k[0], e.k[1]);
    ta[i * 64 + 32 + lane] = make_float4(e.k[2], e.k[3], e.k[4], e.k[5]);
    return;
  }
  const int k = (blockIdx.y - v.tab_n) * kBondPoints + warp;
  if (k < v.n_exp * v.exp_n) {
    const int which = k / v.exp_n, e = k - which * v.exp_n;
    // exponentials in the order la, lr (S not fixed at 2) of set 0, then of set 1
    const int per = v.n_exp / J.num_types, s = which / per, q = J.num_types == 2 && s == 1 ? 4 : 0;
    const double A = par(q + 1), R0 = par(q + 2), S = par(q + 3);
    const double l = which % per ? sqrt(2.0 * S) * A : sqrt(2.0 / S) * A;
    const double value = exp(-l * ((e + v.exp_base) * kStep - R0));
    te[(size_t)k * 32 + lane] = fabs(l) <= (v.wide ? kExpSteep : kExpFlat) ? value : (double)nan;  // NaN: the exact form
  } else if (k == v.n_exp * v.exp_n) {
    for (int s = 0; s < J.num_types; ++s) {
      const int q = 4 * s;
      const double D0 = par(q + 0), A = par(q + 1), S = par(q + 3);
      tk[(4 * s + 0) * 32 + lane] = sqrt(2.0 / S) * A;
      tk[(4 * s + 1) * 32 + lane] = S * D0 / (S - 1.0);
      tk[(4 * s + 2) * 32 + lane] = sqrt(2.0 * S) * A;
      tk[(4 * s + 3) * 32 + lane] = D0 / (S - 1.0);
    }
    // (R1's value is in the geometry, but an undefined one makes the results undefined)
    tk[8 * 32 + lane] = par(6 + off) - (double)v.h0 + 0.0 * par(7 + off);
    ta[v.tab_n * 64 + lane] = ta[v.tab_n * 64 + 32 + lane] = make_float4(nan, nan, nan, nan);
  }
}

// ------------------------------------------------------------------------------ items
// NT: atom types; LO: S is a fitted parameter (two exponentials per pair; else lr = 2 la and cr = ca / 2); WIDE: see
// above.
// One CTA: the segments of the item (up to kEvSegPairs pairs of one configuration each) for 32 individuals, a lane
// each; the warps take batches of 2 consecutive pairs in turn, whose coefficients come through a two-stage
// buffer per warp (cp.async), E summed in FP64, W in FP32 over a batch and in FP64 beyond.
// Bound by issue and by the shared-memory reads of the coefficients.  The 51 000 atoms x 1000 individuals of the
// 500-configuration Si set, alone: 1.78 ms atom by atom (batched.cu), 1.10 ms bond by bond with a test per bond for
// the table's range, the cutoff shell and the batch's end (170 instructions per bond), 0.91 ms without them (113),
// 0.72 ms by pairs with b' of degree 4 (180 instructions per pair, shared-memory wavefronts at 81 % of their peak), 0.75 with
// the present one of degree 5 (wavefronts 79 %, issue slots 72 %).  Error of the 64 near-optimum individuals of such sets
// against FP64: equal to a sixth of the atom items'.
template <int NT, bool LO>
struct EvLane {
  const float4* ta;   // this lane's tables
  const double* te;
  const double* tk;
  double la, ca, lr, cr, dh;
  float dhf;
  int tab_base, tab_n, exp_base, exp_n;
};

// b and b' by powf_dd (rare; out of line, so that its registers do not count).
__device__ __noinline__ float2 bond_exact(float s, float beta, float n, float mhon, float mhonl) {
  const float zeta = beta * s;
  if (zeta < 1.0e-16f) return make_float2(1.f, 0.f);
  const float zn = powf_dd(zeta, n), opz = 1.0f + zn;
  if (zn > 1.0e30f) {  // 1 + zeta^n = zeta^n, which may be beyond FP32
    const float b = powf_dd(zeta, -0.5f);
    return make_float2(b, -0.5f * b / s);
  }
  const float b = powf_dd(opz, mhon, mhonl);
  return make_float2(b, beta * __fdividef(-0.5f * b * zn, opz * zeta));
}

// The pairs of a batch.  WIDE: bonds outside the table take bond_exact one by one, before the pair terms; else EXACT, a
// second pass for all bonds of the batch.  EXACT: also exp_d where the exponentials lie outside the table.
template <int NT, bool LO, bool WIDE, bool EXACT>
__device__ __forceinline__ void ev_pairs_of(const EvLane<NT, LO>& L, const EvPair* q, const float4* x2, const Consts& kc,
                                            double& E, float (&w)[6]) {
  float Qh[kEvBatch][2];
  float bo[kEvBatch][2], db[kEvBatch][2];  // b(s), b'(s)
  auto exact = [&](int u, int h, float s) {
    const float2 r = bond_exact(s, kc[TC_BETA], kc[TC_EN], kc[TC_MHON], kc[TC_MHONL]);
    bo[u][h] = r.x;
    db[u][h] = r.y;
  };
  auto table = [&](int u, int h, float s) {
    const int bits = __float_as_int(s);
    const unsigned i = min((unsigned)((bits >> 20) - L.tab_base), (unsigned)L.tab_n);
    const float4 k0 = L.ta[i * 64], k1 = L.ta[i * 64 + 32];
    const float t = s - __int_as_float((bits & 0xfff00000) | 0x00080000);
    bond_eval<WIDE>(k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w, t, bo[u][h], db[u][h]);
  };
  if constexpr (WIDE) {
    auto s_of = [&](int u, int h) { return (float)fma(L.dh, fma(L.dh, q[u].C[h], q[u].B[h]), q[u].A[h]); };
    bool outside = false;
#pragma unroll
    for (int u = 0; u < kEvBatch; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        table(u, h, s_of(u, h));
        outside |= bo[u][h] != bo[u][h];
      }
    if (__any_sync(0xffffffffu, outside)) {
#pragma unroll
      for (int u = 0; u < kEvBatch; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (bo[u][h] != bo[u][h]) exact(u, h, s_of(u, h));  // its lanes alone: no result depends on the group
    }
  }
#pragma unroll
  for (int u = 0; u < kEvBatch; ++u) {
    const float4* f = reinterpret_cast<const float4*>(q + u);
    const double2 A = *reinterpret_cast<const double2*>(f), B = *reinterpret_cast<const double2*>(f + 1),
                  C = *reinterpret_cast<const double2*>(f + 2), f3 = *reinterpret_cast<const double2*>(f + 3);
    const float4 f4 = f[4];  // hfcp (double), hfc32, code
    if constexpr (!WIDE) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float s = h == 0 ? (float)fma(L.dh, fma(L.dh, C.x, B.x), A.x) : (float)fma(L.dh, fma(L.dh, C.y, B.y), A.y);
        if constexpr (EXACT) exact(u, h, s);
        else table(u, h, s);
      }
    }
    // pair terms: exponentials from the grid point and a polynomial of the rest
    const int code = __float_as_int(f4.w);
    const int e = (code & 0xffff) - L.exp_base;
    const int set = NT == 2 ? (code >> 16) & 1 : 0;
    const double la = NT == 2 ? L.tk[set * 128] : L.la, ca = NT == 2 ? L.tk[set * 128 + 32] : L.ca;
    const double* tx = L.te + (size_t)((NT == 2 ? set * (LO ? 2 : 1) * L.exp_n : 0) + e) * 32;
    auto ex = [&](double l, double base) {
      const double y = -l * f3.x;
      constexpr double inv_fact[10] = {1.0,         1.0,         0.5,          1.0 / 6.0,     1.0 / 24.0,
                                       1.0 / 120.0, 1.0 / 720.0, 1.0 / 5040.0, 1.0 / 40320.0, 1.0 / 362880.0};
      constexpr int deg = WIDE ? 9 : 5;
      double z = inv_fact[deg];
#pragma unroll
      for (int k = deg - 1; k >= 1; --k) z = fma(y, z, inv_fact[k]);
      double r = fma(base * y, z, base);
      // beyond the tables: of d - r0, d = grid point + delta exactly
      if (EXACT && r != r) r = exp_d_clamped(-l * ((code & 0xffff) * kStep + f3.x - (double)kc[TC_R0 + set]));
      return r;
    };
    const double ea = ex(la, tx[0]);
    const double fa = ca * ea, bs = (double)bo[u][0] + (double)bo[u][1];
    double en, dA;  // over both bonds: fr - b fa and fr' - b fa'
    if constexpr (LO) {
      const double lr = NT == 2 ? L.tk[set * 128 + 64] : L.lr, cr = NT == 2 ? L.tk[set * 128 + 96] : L.cr;
      const double fr2 = 2.0 * cr * ex(lr, tx[(size_t)L.exp_n * 32]);
      en = fma(-bs, fa, fr2);
      dA = fma(bs * la, fa, -lr * fr2);
    } else {
      // fr = fa ea / 2: en = fa (ea - bs), dA = -la (en + 2 fr) = -la fa (2 ea - bs)
      const double y = ea - bs;
      en = fa * y;
      dA = -la * fa * (y + ea);
    }
    E = fma(f3.y, en, E);
    const double hfcp = __hiloint2double(__float_as_int(f4.y), __float_as_int(f4.x));
    const float g = (float)-fma(hfcp, en, f3.y * dA);  // -A'/2
    const float fw = f4.z * (float)fa;
    const float Q0 = fw * db[u][0], Q1 = fw * db[u][1];
    Qh[u][0] = Q0 * L.dhf;
    Qh[u][1] = Q1 * L.dhf;
    // 24 + 6 floats from f5 on: D, then X0, X1 of the first and of the second bond
    const float4 f5 = f[5], f6 = f[6], f7 = f[7], f8 = f[8], f9 = f[9], fa4 = f[10], fb4 = f[11], fc4 = f[12];
    const float x[30] = {f5.x,  f5.y,  f5.z,  f5.w,  f6.x,  f6.y,  f6.z,  f6.w,  f7.x,  f7.y,  f7.z,  f7.w,  f8.x,  f8.y,  f8.z,
                         f8.w,  f9.x,  f9.y,  f9.z,  f9.w,  fa4.x, fa4.y, fa4.z, fa4.w, fb4.x, fb4.y, fb4.z, fb4.w, fc4.x, fc4.y};
#pragma unroll
    for (int k = 0; k < 6; ++k)
      w[k] = fmaf(g, x[k], fmaf(Q0, x[6 + k], fmaf(Qh[u][0], x[12 + k], fmaf(Q1, x[18 + k], fmaf(Qh[u][1], x[24 + k], w[k])))));
  }
  if (q->code & kShellBit) {
#pragma unroll
    for (int u = 0; u < kEvBatch; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 x = __ldg(x2 + 4 * u + 2 * h), y = __ldg(x2 + 4 * u + 2 * h + 1);
        const float z = Qh[u][h] * L.dhf;
        w[0] = fmaf(z, x.x, w[0]);
        w[1] = fmaf(z, x.y, w[1]);
        w[2] = fmaf(z, x.z, w[2]);
        w[3] = fmaf(z, x.w, w[3]);
        w[4] = fmaf(z, y.x, w[4]);
        w[5] = fmaf(z, y.y, w[5]);
      }
  }
}

// A batch again with exp_d (rare; out of line, so that its registers do not count).
template <int NT, bool LO, bool WIDE>
__device__ __noinline__ void ev_batch_exact(const EvLane<NT, LO>& L, const EvPair* q, const float4* x2, const Consts& kc,
                                            double& E, float (&w)[6]) {
  ev_pairs_of<NT, LO, WIDE, true>(L, q, x2, kc, E, w);
}

template <int NT, bool LO, bool WIDE>
__global__ void __launch_bounds__(kEvThreads, 2) tersoff_ev(const JobView* __restrict__ jobs,
                                                            const WorkItem* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char smem[];
  const WorkItem it = items[blockIdx.x];
  const JobView& J = jobs[it.job];
  const TersoffEvView v = J.ev;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = it.p0 + lane;
  const size_t bytes = tab_bytes(v);
  {
    const unsigned char* src = v.tables + (size_t)(it.p0 >> 5) * bytes;
    for (size_t k = threadIdx.x * 16; k < bytes; k += kEvThreads * 16) __pipeline_memcpy_async(smem + k, src + k, 16);
    __pipeline_commit();
  }
  EvLane<NT, LO> L;
  L.ta = reinterpret_cast<const float4*>(smem) + lane;
  L.te = reinterpret_cast<const double*>(smem + tab_b_bytes(v)) + lane;
  L.tk = L.te + (size_t)v.n_exp * v.exp_n * 32;
  L.tab_base = v.tab_base;
  L.tab_n = v.tab_n;
  L.exp_base = v.exp_base;
  L.exp_n = v.exp_n;
  double* red = reinterpret_cast<double*>(smem + bytes);  // [7][warps][32]
  EvPair* stage = reinterpret_cast<EvPair*>(red + 7 * kEvThreads) + warp * 2 * kEvBatch;
  __pipeline_wait_prior(0);
  __syncthreads();
  if constexpr (NT == 1) {
    L.la = L.tk[0];
    L.ca = L.tk[32];
    L.lr = LO ? L.tk[64] : 0.0;
    L.cr = LO ? L.tk[96] : 0.0;
  }
  L.dh = L.tk[8 * 32];
  L.dhf = (float)L.dh;
  const Consts kc{J.consts, J.Pstride, p < J.P ? p : J.P - 1};
  for (int sg = it.config; sg < it.config + it.gofs; ++sg) {
    const TersoffSegment seg = v.segs[sg];
    double E = 0.0, Wd[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    auto fetch = [&](int b, int st) {  // a batch is 26 x 16 bytes
      if (b < seg.n && lane < (int)sizeof(EvPair) * kEvBatch / 16)
        __pipeline_memcpy_async(reinterpret_cast<float4*>(stage + st * kEvBatch) + lane,
                                reinterpret_cast<const float4*>(v.pairs + seg.b0 + b) + lane, 16);
      __pipeline_commit();
    };
    fetch(warp * kEvBatch, 0);
    int st = 0;
    for (int b = warp * kEvBatch; b < seg.n; b += kEvW * kEvBatch, st ^= 1) {
      fetch(b + kEvW * kEvBatch, st ^ 1);
      __pipeline_wait_prior(1);
      __syncwarp();
      const EvPair* q = stage + st * kEvBatch;
      const float4* x2 = v.shell + 4 * (size_t)(seg.b0 + b);
      double Eb = 0.0;
      float w[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      ev_pairs_of<NT, LO, WIDE, false>(L, q, x2, kc, Eb, w);
      // the NaN of a bond order or an exponential outside the tables reaches the energy
      if (__any_sync(0xffffffffu, Eb != Eb)) {
        const EvLane<NT, LO> copy = L;  // (passed by address)
        double Ex = 0.0;
        float wx[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        ev_batch_exact<NT, LO, WIDE>(copy, q, x2, kc, Ex, wx);
        if (Eb != Eb) {  // only the lanes that need it: an individual's result does not depend on its group
          Eb = Ex;
#pragma unroll
          for (int k = 0; k < 6; ++k) w[k] = wx[k];
        }
      }
      E += Eb;
#pragma unroll
      for (int k = 0; k < 6; ++k) Wd[k] += (double)w[k];
      __syncwarp();  // every lane is done with this stage before it is refilled
    }
    __pipeline_wait_prior(0);
    red[threadIdx.x] = E;
#pragma unroll
    for (int k = 0; k < 6; ++k) red[(k + 1) * kEvThreads + threadIdx.x] = Wd[k];
    __syncthreads();
    // fixed order: the warps' sums of a lane, one component per warp
    if (warp < 7 && p < J.P) {
      double s = 0.0;
#pragma unroll
      for (int x = 0; x < kEvW; ++x) s += red[warp * kEvThreads + x * 32 + lane];
      if (seg.part < 0) J.res[((size_t)p * J.v.Nc + seg.config) * kResK + warp] = s;
      else v.part[((size_t)seg.part * 7 + warp) * J.Pstride + p] = s;
    }
    __syncthreads();
  }
  finish_item(jobs, it, 32);
}

}  // namespace

size_t tersoff_ev_smem(const TersoffEvView& v) {
  return tab_bytes(v) + sizeof(double) * 7 * kEvThreads + sizeof(EvPair) * kEvW * 2 * kEvBatch;
}
size_t tersoff_ev_plan_bytes(const TersoffEvView& v, int P) {
  const size_t groups = ((size_t)P + 31) / 32;
  return groups * tab_bytes(v) + sizeof(double) * 7 * std::max(v.n_part, 1) * groups * 32;
}
size_t tersoff_ev_group_bytes(int num_types) {
  TersoffEvView v{};
  v.tab_n = kTabMax;
  v.exp_n = kExpMax;
  v.n_exp = 2 * num_types;
  return tab_bytes(v);
}
size_t tersoff_ev_bytes(double pairs, int P) {
  const double segments = std::ceil(pairs / kEvSegPairs);
  return (size_t)((sizeof(EvPair) + 4 * sizeof(float4)) * (pairs + kEvBatch * segments) + sizeof(TersoffSegment) * segments +
                  (segments > 1 ? sizeof(double) * 7 * segments * ((P + 31) & ~31) : 0.0));
}

int tersoff_ev_build(Engine* e) {
  DevSet& d = e->d;
  const TrainingSet& ts = e->ts;
  const PotentialSpec& sp = e->spec;
  if (d.potential_type != 1 && d.potential_type != 2) return GPUGA_OK;
  const int Nev = ts.Nc - ts.Nc_force, na = ts.N - ts.N_force;
  const int off = d.num_types == 2 ? 4 : 0;
  if (Nev == 0 || na == 0 || (int)sp.pmin.size() < 9 + off) return GPUGA_OK;
  // R1 and R2 fixed, h bounded
  const float r1 = sp.pmin[7 + off], r2 = sp.pmin[8 + off], hlo = sp.pmin[6 + off], hhi = sp.pmax[6 + off];
  if (sp.pmax[7 + off] != r1 || sp.pmax[8 + off] != r2 || !(r1 < r2) || !std::isfinite(hlo) || !std::isfinite(hhi))
    return GPUGA_OK;
  bool exact = true;  // S fixed at 2: one exponential per bond (tersoff_consts_exact)
  for (int s = 0; s < d.num_types; ++s) exact &= sp.pmin[4 * s + 3] == 2.0f && sp.pmax[4 * s + 3] == 2.0f;
  // the steepest exponential within the bounds: sqrt(2 / S) alpha and sqrt(2 S) alpha
  double steepest = 0.0;
  for (int s = 0; s < d.num_types; ++s) {
    const double al = std::max(std::fabs(sp.pmin[4 * s + 1]), std::fabs(sp.pmax[4 * s + 1]));
    const double s0 = std::min(sp.pmin[4 * s + 3], sp.pmax[4 * s + 3]), s1 = std::max(sp.pmin[4 * s + 3], sp.pmax[4 * s + 3]);
    if (!(s0 > 0.0)) return GPUGA_OK;
    steepest = std::max(steepest, al * std::max(std::sqrt(2.0 / s0), exact ? 0.0 : std::sqrt(2.0 * s1)));
  }
  if (!(steepest <= kExpSteep)) return GPUGA_OK;
  cudaStream_t st = e->stream;
  TersoffEvView v{};
  v.h0 = 0.5f * hlo + 0.5f * hhi;
  int *d_count = nullptr, *d_start = nullptr, *d_place = nullptr, *d_last = nullptr, *d_slot = nullptr;
  double2* d_range = nullptr;
  std::vector<int> count(na), start(na + 1, 0);
  std::vector<double2> range(na + 1);
  auto run = [&]() -> int {
    GPUGA_CUDA(cudaMalloc(&d_count, sizeof(int) * na));
    GPUGA_CUDA(cudaMalloc(&d_start, sizeof(int) * (na + 1)));
    GPUGA_CUDA(cudaMalloc(&d_slot, sizeof(int) * (size_t)std::max(d.B, 1)));
    GPUGA_CUDA(cudaMalloc(&d_range, sizeof(double2) * (na + 1)));
    ev_bonds<false><<<(na + 127) / 128, 128, 0, st>>>(ts.N_force, na, d.off, d.nbr, d.rev, d_slot, d.ptype, d.g64, r1, r2, v.h0, nullptr, nullptr,
                                                      d_count, nullptr, nullptr, d_range);
    GPUGA_CUDA(cudaGetLastError());
    GPUGA_CUDA(cudaMemcpyAsync(count.data(), d_count, sizeof(int) * na, cudaMemcpyDeviceToHost, st));
    GPUGA_CUDA(cudaMemcpyAsync(range.data(), d_range, sizeof(double2) * (na + 1), cudaMemcpyDeviceToHost, st));
    GPUGA_CUDA(cudaStreamSynchronize(st));
    double dmin = 1e300, dmax = 0.0;
    for (int a = 0; a < na; ++a) {
      start[a + 1] = start[a] + count[a];
      // (every atom's, also of those without a pair of their own: a bond without its reverse sets the largest)
      dmin = std::min(dmin, range[1 + a].x);
      dmax = std::max(dmax, range[1 + a].y);
    }
    if (start[na] == 0 || !(dmax < 2000.0)) return GPUGA_OK;  // (EvPair::code has 16 bits for the grid point)
    // A configuration's fixed costs (two CTA barriers and the fold over the warps) outweigh its pairs below about 64:
    // sets of 8-atom cells (16 pairs) took 42-66 us by atom against 55-83 here, 64-atom cells (128 pairs)
    // 52-66 against 50-66, 216-atom ones 94-103 against 51-55.
    if (start[na] < 64LL * Nev) return GPUGA_OK;
    // the shorter polynomial's steepest exponential, n up to which every entry of the table is accepted, more than four bonds
    // per atom (and not a few beyond the second shell)
    v.wide = steepest > kExpFlat || !(std::max(sp.pmin[4 + off], sp.pmax[4 + off]) <= 5.0f) || 2.0 * start[na] > 4.5 * na;
    v.exp_base = (int)std::rint(dmin * 32.0);
    v.exp_n = (int)std::rint(dmax * 32.0) - v.exp_base + 1;
    if (v.exp_n > kExpMax) return GPUGA_OK;
    // segments of at most kEvSegPairs pairs of one configuration, each padded to whole batches
    std::vector<TersoffSegment> segs;
    std::vector<int> seg0(ts.Nc + 1, 0), place(start[na]), last;
    int parts = 0, slots = 0;
    for (int c = ts.Nc_force; c < ts.Nc; ++c) {
      const int b0 = start[ts.Na_sum[c] - ts.N_force], b1 = start[ts.Na_sum[c] + ts.Na[c] - ts.N_force];
      const int n = std::max(1, (b1 - b0 + kEvSegPairs - 1) / kEvSegPairs);
      const int size = ((b1 - b0 + n - 1) / n + kEvBatch - 1) / kEvBatch * kEvBatch;
      seg0[c] = parts;
      for (int k = 0; k < n; ++k) {
        const int a = std::min(b1, b0 + k * size), m = std::min(size, b1 - a);
        const int padded = (m + kEvBatch - 1) / kEvBatch * kEvBatch;
        for (int x = 0; x < m; ++x) place[a + x] = slots + x;
        for (int x = 0; x < padded; x += kEvBatch) last.push_back(slots + std::min(x + kEvBatch, m) - 1);
        segs.push_back({c, slots, padded, n > 1 ? parts++ : -1});
        slots += padded;
      }
    }
    seg0[ts.Nc] = parts;
    EvPair* pairs = nullptr;
    float4* shell = nullptr;
    GPUGA_TRY(e->alloc(&pairs, (size_t)slots));
    GPUGA_TRY(e->alloc(&shell, (size_t)slots * 4));
    GPUGA_CUDA(cudaMalloc(&d_place, sizeof(int) * place.size()));
    GPUGA_CUDA(cudaMalloc(&d_last, sizeof(int) * last.size()));
    GPUGA_CUDA(cudaMemcpyAsync(d_place, place.data(), sizeof(int) * place.size(), cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_last, last.data(), sizeof(int) * last.size(), cudaMemcpyHostToDevice, st));
    const double2 h = make_double2((double)std::min(hlo, hhi) - v.h0, (double)std::max(hlo, hhi) - v.h0);
    GPUGA_CUDA(cudaMemcpyAsync(d_range, &h, sizeof h, cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_start, start.data(), sizeof(int) * (na + 1), cudaMemcpyHostToDevice, st));
    ev_bonds<true><<<(na + 127) / 128, 128, 0, st>>>(ts.N_force, na, d.off, d.nbr, d.rev, d_slot, d.ptype, d.g64, r1, r2, v.h0, d_start, d_place,
                                                     d_count, pairs, shell, d_range);
    ev_batches<<<((int)last.size() + 127) / 128, 128, 0, st>>>((int)last.size(), d_last, pairs, shell);
    GPUGA_CUDA(cudaGetLastError());
    GPUGA_CUDA(cudaMemcpyAsync(range.data(), d_range, sizeof(double2) * (na + 1), cudaMemcpyDeviceToHost, st));
    GPUGA_CUDA(cudaStreamSynchronize(st));
    double smin = 1e300, smax = 0.0;
    for (int a = 0; a < na; ++a)
      if (count[a]) {
        smin = std::min(smin, range[1 + a].x);
        smax = std::max(smax, range[1 + a].y);
      }
    // entries from the least to the largest s (a little beyond, for the rounding), at most kTabMax from the top:
    // smaller s, rare, take powf_dd
    auto entry = [](double s) {
      const float f = (float)std::min(std::max(s, 1e-30), 1e30);
      int32_t i;
      memcpy(&i, &f, 4);
      return i >> 20;
    };
    const int top = entry(smax * 1.0001), low = std::max(entry(smin * 0.9999), top - kTabMax + 1);
    v.tab_base = low;
    v.tab_n = top - low + 1;
    std::vector<double2> points((size_t)v.tab_n * kBondPoints);
    for (int k = 0; k < v.tab_n; ++k) {
      const int32_t lo = (low + k) << 20, mid = lo | 0x00080000;
      float f, c;
      memcpy(&f, &lo, 4);
      memcpy(&c, &mid, 4);
      for (int x = 0; x < kBondPoints; ++x) {
        const double s = c + ((double)c - f) * kBondPoint[x];
        points[(size_t)k * kBondPoints + x] = make_double2(s, std::log(s));
      }
    }
    v.n_exp = d.num_types * (exact ? 1 : 2);
    if (tersoff_ev_smem(v) > 220 * 1024) return GPUGA_OK;
    TersoffSegment* d_segs = nullptr;
    int* d_seg0 = nullptr;
    double2* d_points = nullptr;
    GPUGA_TRY(e->alloc(&d_points, points.size()));
    GPUGA_CUDA(cudaMemcpyAsync(d_points, points.data(), sizeof(double2) * points.size(), cudaMemcpyHostToDevice, st));
    GPUGA_TRY(e->alloc(&d_segs, segs.size()));
    GPUGA_TRY(e->alloc(&d_seg0, seg0.size()));
    GPUGA_CUDA(cudaMemcpyAsync(d_segs, segs.data(), sizeof(TersoffSegment) * segs.size(), cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_seg0, seg0.data(), sizeof(int) * seg0.size(), cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaStreamSynchronize(st));
    // items: consecutive segments up to kEvSegPairs pairs
    e->h_ev_items.clear();
    for (int k = 0; k < (int)segs.size();) {
      int m = k, n = 0, atoms = 0;
      do {
        n += segs[m].n;
        atoms += segs[m].part < 0 ? ts.Na[segs[m].config] : 0;
        ++m;
      } while (m < (int)segs.size() && n + segs[m].n <= kEvSegPairs);
      e->h_ev_items.push_back({k, m - k, n, std::max(atoms, n / 2)});
      k = m;
    }
    v.pairs = pairs;
    v.shell = shell;
    v.segs = d_segs;
    v.points = d_points;
    v.seg0 = d_seg0;
    v.n_part = parts;
    v.n_items = (int)e->h_ev_items.size();
    d.ev = v;
    return GPUGA_OK;
  };
  const int s = run();
  cudaFree(d_count);
  cudaFree(d_start);
  cudaFree(d_place);
  cudaFree(d_last);
  cudaFree(d_slot);
  cudaFree(d_range);
  return s;
}

int tersoff_ev_plan(Engine* e, Plan* plan) {
  TersoffEvView v = e->d.ev;
  const size_t groups = (plan->P + 31) / 32;
  GPUGA_TRY(e->alloc(&v.tables, groups * tab_bytes(v)));
  GPUGA_TRY(e->alloc(&v.part, (size_t)std::max(v.n_part, 1) * 7 * plan->Pstride));
  plan->ev = v;
  return GPUGA_OK;
}

int tersoff_tables_launch(const LaunchSet* ls, cudaStream_t st) {
  int ctas = 0;  // of a group, of the job with most
  for (const JobView& j : ls->jobs)
    if (j.ev.pairs) ctas = std::max(ctas, tab_ctas(j.ev));
  tersoff_tables<<<dim3(ls->ev_groups, ctas), kTabThreads, 0, st>>>(ls->d_jobs, ls->d_evgroups);
  GPUGA_CUDA(cudaGetLastError());
  return GPUGA_OK;
}

template <int NT, bool LO, bool WIDE>
static int ev_launch(const JobView* jobs, const WorkItem* items, int count, size_t smem, bool configure, cudaStream_t st) {
  if (configure) {
    GPUGA_CUDA(cudaFuncSetAttribute(tersoff_ev<NT, LO, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    return GPUGA_OK;
  }
  tersoff_ev<NT, LO, WIDE><<<count, kEvThreads, smem, st>>>(jobs, items);
  GPUGA_CUDA(cudaGetLastError());
  return GPUGA_OK;
}

int tersoff_ev_items_launch(const JobView* jobs, const WorkItem* items, int count, size_t smem, int num_types, bool lo,
                            bool wide, bool configure, cudaStream_t st) {
  auto launch = num_types == 2 ? (lo ? (wide ? ev_launch<2, true, true> : ev_launch<2, true, false>)
                                     : (wide ? ev_launch<2, false, true> : ev_launch<2, false, false>))
                               : (lo ? (wide ? ev_launch<1, true, true> : ev_launch<1, true, false>)
                                     : (wide ? ev_launch<1, false, true> : ev_launch<1, false, false>));
  return launch(jobs, items, count, smem, configure, st);
}

}  // namespace gpuga
