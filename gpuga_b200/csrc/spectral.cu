// Pair expansion: fitness evaluation of the pair potentials (rigid ion, NN2B) without a pass over
// the pairs.
//
// The pair energy of an individual is a smooth function of the distance alone, U_t(d) per pair type
// t.  On a piece of the distance range, d = mid + half x, it is a Chebyshev series
//   U_t(d) = sum_k c_k T_k(x),    dU_t/dd = sum_k c_k T_k'(x) / half,
// so every result is linear in the coefficients: with the geometric sums (moments) formed once per
// training set in FP64,
//   F_i = sum_k c_k [sum_j (T_k'(x_ij) / half) u_ij],  E = sum_k c_k [sum_pairs T_k],
//   W = sum_k c_k [-sum_pairs d (T_k' / half) u (x) u]
// (NN2B: with its taper fc(d) in the sums, fd = U' fc + U g, g = fc fc' or, tapered consistently,
// fc').  A generation is then: the function's values at the Chebyshev nodes and its coefficients per
// individual (spectral_coefs), and one FP64 matrix product [individuals x columns] [columns x rows]
// (spectral_items).  The rigid ion's linear terms (Coulomb, dispersion; geometry.cu) and the reference
// force are columns as well, so the product of a force row is the force error itself, and its squared
// norm over a configuration is all that a generation needs of it: |X c|^2 = |R c|^2 with X = Q R, so
// each force configuration keeps the triangle R of at most as many rows as there are columns instead
// of its 3 rows per atom (spec_qr).  Energy/virial configurations keep their 7 rows.
// Per-atom forces (batched_forces) come from the direct items, in a launch set of their own.
//
// What it replaces: the direct items evaluate the pair function per (individual, pair) -- about 50
// instructions for an exponential pair, 2 000 for a 16-neuron network -- and were bound by instruction
// issue.  B200, one generation: 300 oxide configurations (28 000 force atoms, 146 pairs per atom) at
// population 400 4.75 -> 0.106 ms; 200 Si cells, 16 neurons, population 200 4.75 -> 0.138 ms; 13 oxide
// configurations at population 50 0.60 -> 0.052 ms.  The same product over all 3 rows per atom took
// 0.33 ms of the oxide set's generation (58 % of the FP64 tensor rate) against 0.066 ms for the triangles.
//
// Accuracy.  Coefficients and sums are FP64; a series is used for an individual only when its last 8
// coefficients are negligible (kTolRI, kTolNN below); an individual that does not meet that -- a
// network with a very sharp feature, parameters outside their bounds, NaN -- is left to the direct
// items (pair_batched), which evaluate its pairs one by one.  Coefficients beyond the last
// significant block of 8 are set to zero, so that a group of individuals may skip the blocks that
// none of them uses without changing a bit of any result.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "decode.cuh"
#include "engine.hpp"
#include "exp_d.cuh"
#include "fold.cuh"

namespace gpuga {

namespace {

constexpr int kMaxCtab = 3 * 4 * kSpecMaxK;
// NN2B: longest piece and terms per piece.  With weights drawn over the whole search range [-3, 3] and
// pieces of 0.85 A none of 1000 networks of 10 or 16 neurons needs more than 72 terms (the last 8 have
// to be negligible), 64 leave out 2 %; of 32 neurons 1.5 % do, and none at 0.6 A.  Shorter pieces need
// more columns in all (16 neurons: 89 on average at 0.85 A, 132 at 0.43 A).
constexpr int kNNTerms = 80;
double nn_piece_length(int n) { return 0.85 * std::min(1.0, 4.0 / std::sqrt((double)std::max(n, 1))); }
constexpr double kQrBatchBytes = 512e6;  // work space of the factorisation (one configuration may need more)
// A coefficient counts when |c_k| k^2 / half exceeds this share of the largest such value (the scale
// of dU/dd).  The rigid ion's exponentials converge faster than geometrically, so the strict bound
// costs a few terms; a tanh network converges geometrically, and 1e-9 lies two decades below the
// FP32 rounding of the direct form.
constexpr double kTolRI = 1e-12;
constexpr double kTolNN = 1e-9;
// A network whose last 8 coefficients still count is kept while they stay below this share: dU/dd is
// then as exact as the direct items' FP32 form (its rounding is above 1e-7 of the scale).  Of 32 000
// networks of 16 (10) neurons 14 (3) pass 1e-9 and none passes 5e-8; one of 32 000 does over a range
// of 6.5 A.
constexpr double kAcceptNN = 5e-8;

// Position of (row, col) within an 8 x 8 block: the MMA operand order, two k-steps of 4 side by side per lane.
__device__ __forceinline__ int in_block(int row, int col) {
  return (row & 7) * 8 + (col & 3) * 2 + ((col >> 2) & 1);
}
// (row, col) of set `set` in the moments, (individual, column) in the coefficients
__device__ __forceinline__ size_t moment_at(const SpecView& sp, int set, int row, int col) {
  return (size_t)sp.moff[set] + ((size_t)(col >> 3) * sp.mnb[set] + (row >> 3)) * 64 + in_block(row, col);
}
__device__ __forceinline__ size_t coef_at(const SpecView& sp, int p, int col) {
  return ((size_t)(p >> 5) * sp.ncb + (col >> 3)) * 256 + ((p >> 3) & 3) * 64 + in_block(p, col);
}
// set of an energy/virial configuration (the k-th one), its first row there
__device__ __forceinline__ int ev_set(int nc_force, int k) { return nc_force + k / kSpecEvBlocks; }
__device__ __forceinline__ int ev_row(int k) { return 8 * (k % kSpecEvBlocks); }
__device__ __forceinline__ int column_of(const SpecPiece& pc, int k) { return pc.cb[k >> 3] * 8 + (k & 7); }

// A force configuration's sums X before the factorisation, column-major at `off`: rows x columns.
struct QrTile {
  size_t off;
  int ld, rows;
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ int piece_of(const SpecPiece* pc, int n, int type, double d) {
  for (int q = 0; q < n; ++q)
    if (pc[q].type == type && d < pc[q].to) return q;
  return -1;
}

// FP64 taper of nn2b.cu:80-92
__device__ __forceinline__ void taper64(const NNTaper& tp, double d, double& fc, double& g) {
  fc = 1.0;
  double fcp = 0.0;
  if (d >= (double)tp.r2) {
    fc = 0.0;
  } else if (d >= (double)tp.r1) {
    const double pf = M_PI / ((double)tp.r2 - (double)tp.r1);
    double s, c;
    sincos(pf * (d - (double)tp.r1), &s, &c);
    fc = 0.5 * c + 0.5;
    fcp = -0.5 * pf * s;
  }
  g = tp.consistent ? fcp : fc * fcp;
}

// ------------------------------------------------------------------------------ set-up kernels
// Range of the evaluated distances per pair type: bits of the smallest and largest d (positive
// doubles order as their bits) and the number of bonds.
__global__ void spec_range(int B, const double4* __restrict__ g, const uint8_t* __restrict__ ptype, int active,
                           double dmax, unsigned long long* __restrict__ out) {
  __shared__ unsigned long long s[9];
  if (threadIdx.x < 9) s[threadIdx.x] = threadIdx.x % 3 == 0 ? ~0ull : 0ull;
  __syncthreads();
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < B; b += gridDim.x * blockDim.x) {
    const int t = ptype[b];
    const double d = g[b].w;
    if (t > 2 || !((active >> t) & 1) || !(d < dmax)) continue;
    const unsigned long long v = (unsigned long long)__double_as_longlong(d);
    if (v < s[3 * t]) atomicMin(&s[3 * t], v);
    if (v > s[3 * t + 1]) atomicMax(&s[3 * t + 1], v);
    atomicAdd(&s[3 * t + 2], 1ull);
  }
  __syncthreads();
  if (threadIdx.x < 9) {
    if (threadIdx.x % 3 == 0) atomicMin(&out[threadIdx.x], s[threadIdx.x]);
    else if (threadIdx.x % 3 == 1) atomicMax(&out[threadIdx.x], s[threadIdx.x]);
    else atomicAdd(&out[threadIdx.x], s[threadIdx.x]);
  }
}

// One bond's share of the sums, staged per lane: T_k(x) = cos(k theta), T_k'(x) = k sin(k theta) / sin(theta).
struct BondTerm {
  double t, inv_sin;  // theta / pi, 1 / sin(theta)
  double wT, wD;      // weights of T_k and of T_k' (1 / half included)
};

__device__ __forceinline__ void bond_term(const SpecPiece* pc, int q, double d, double fc, double g, BondTerm& o) {
  const double x = (d - pc[q].mid) / pc[q].half;  // |x| <= 0.99: pieces are wider than what they hold
  o.t = acos(x) * (1.0 / M_PI);
  o.inv_sin = rsqrt(1.0 - x * x);
  o.wT = g;
  o.wD = fc / pc[q].half;
}

// Force rows: one warp per atom, its lanes the terms k; bonds staged 32 at a time.
__global__ void spec_force_moments(int atom0, int n_atoms, SpecView sp, const QrTile* __restrict__ cfg,
                                   const int2* __restrict__ where, const int* __restrict__ off, const uint8_t* __restrict__ ptype,
                                   const double4* __restrict__ g64, NNTaper tp, int nn, int active,
                                   double* __restrict__ X) {
  __shared__ BondTerm term[8][32];
  __shared__ double u[8][32][3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = blockIdx.x * 8 + warp;
  if (a >= n_atoms) return;
  const int i = atom0 + a, be = off[i + 1];
  const int2 w0 = where[i];  // configuration of this batch, first row
  const int ld = cfg[w0.x].ld;
  double* x0 = X + cfg[w0.x].off + w0.y;
  for (int b0 = off[i]; b0 < be; b0 += 32) {
    int mine = -1;
    if (b0 + lane < be) {
      const double4 v = g64[b0 + lane];
      const int t = ptype[b0 + lane];
      double fc = 1.0, g = 0.0;
      if (nn) taper64(tp, v.w, fc, g);
      if (((active >> t) & 1) && (fc != 0.0 || g != 0.0)) mine = piece_of(sp.pieces, sp.n_pieces, t, v.w);
      if (mine >= 0) {
        bond_term(sp.pieces, mine, v.w, fc, g, term[warp][lane]);
        const double inv = 1.0 / v.w;
        u[warp][lane][0] = v.x * inv;
        u[warp][lane][1] = v.y * inv;
        u[warp][lane][2] = v.z * inv;
      }
    }
    __syncwarp();
    for (int q = 0; q < sp.n_pieces; ++q) {
      const unsigned in = __ballot_sync(0xffffffffu, mine == q);
      if (!in) continue;
      const int K = sp.pieces[q].K;
      for (int k = lane; k < K; k += 32) {
        double f[3] = {0.0, 0.0, 0.0};
        for (unsigned m = in; m; m &= m - 1) {
          const int l = __ffs(m) - 1;
          const BondTerm o = term[warp][l];
          double s, c;
          sincospi(k * o.t, &s, &c);
          const double w = o.wD * (k * s * o.inv_sin) + o.wT * c;
#pragma unroll
          for (int x = 0; x < 3; ++x) f[x] = fma(w, u[warp][l][x], f[x]);
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) x0[(size_t)column_of(sp.pieces[q], k) * ld + x] += f[x];
      }
    }
    __syncwarp();
  }
}

// Energy/virial rows: one CTA per (configuration, piece) over the unordered pairs.
constexpr int kEvWarps = 8;
__global__ void spec_ev_moments(int c0, SpecView sp, const int* __restrict__ Na, const int* __restrict__ Na_sum,
                                const int* __restrict__ off, const int* __restrict__ half_off,
                                const uint8_t* __restrict__ ptype, const double4* __restrict__ g64, NNTaper tp, int nn,
                                int active, double* __restrict__ M) {
  __shared__ BondTerm term[kEvWarps][32];
  __shared__ double u[kEvWarps][32][4];
  __shared__ double red[kEvWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = c0 + blockIdx.x, q = blockIdx.y;
  const int K = sp.pieces[q].K;
  constexpr int R = kSpecMaxK / 32;
  double acc[R][7];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int x = 0; x < 7; ++x) acc[r][x] = 0.0;
  for (int il = warp; il < Na[c]; il += kEvWarps) {
    const int i = Na_sum[c] + il, be = off[i + 1];
    for (int b0 = half_off[i]; b0 < be; b0 += 32) {
      bool mine = false;
      if (b0 + lane < be) {
        const double4 v = g64[b0 + lane];
        const int t = ptype[b0 + lane];
        double fc = 1.0, g = 0.0;
        if (nn) taper64(tp, v.w, fc, g);
        mine = ((active >> t) & 1) && (fc != 0.0 || g != 0.0) && piece_of(sp.pieces, sp.n_pieces, t, v.w) == q;
        if (mine) {
          bond_term(sp.pieces, q, v.w, fc, g, term[warp][lane]);
          const double inv = 1.0 / v.w;
          u[warp][lane][0] = v.x * inv;
          u[warp][lane][1] = v.y * inv;
          u[warp][lane][2] = v.z * inv;
          u[warp][lane][3] = v.w;
        }
      }
      __syncwarp();
      const unsigned in = __ballot_sync(0xffffffffu, mine);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = lane + 32 * r;
        if (k >= K) continue;
        for (unsigned m = in; m; m &= m - 1) {
          const int l = __ffs(m) - 1;
          const BondTerm o = term[warp][l];
          const double ux = u[warp][l][0], uy = u[warp][l][1], uz = u[warp][l][2], d = u[warp][l][3];
          double s, cs;
          sincospi(k * o.t, &s, &cs);
          const double fc = nn ? o.wD * sp.pieces[q].half : 1.0;
          acc[r][0] = fma(fc, cs, acc[r][0]);
          const double w = -d * (o.wD * (k * s * o.inv_sin) + o.wT * cs);
          acc[r][1] = fma(w * ux, ux, acc[r][1]);
          acc[r][2] = fma(w * uy, uy, acc[r][2]);
          acc[r][3] = fma(w * uz, uz, acc[r][3]);
          acc[r][4] = fma(w * ux, uy, acc[r][4]);
          acc[r][5] = fma(w * uy, uz, acc[r][5]);
          acc[r][6] = fma(w * uz, ux, acc[r][6]);
        }
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int x = 0; x < 7; ++x) {
      red[warp][lane] = acc[r][x];
      __syncthreads();
      if (warp == 0 && lane + 32 * r < K) {
        double s = 0.0;
        for (int w = 0; w < kEvWarps; ++w) s += red[w][lane];
        M[moment_at(sp, ev_set(c0, blockIdx.x), ev_row(blockIdx.x) + x, column_of(sp.pieces[q], lane + 32 * r))] = s;
      }
      __syncthreads();
    }
}

// Linear columns: the rigid ion's Coulomb and dispersion sums (geometry.cu), the self energy and the
// reference force.
__global__ void spec_linear_force(int atom0, int n_atoms, int N, SpecView sp, const QrTile* __restrict__ cfg,
                                  const int2* __restrict__ where, const double* __restrict__ lin,
                                  const float* __restrict__ force_ref, double* __restrict__ X) {
  const int a = atom0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= atom0 + n_atoms) return;
  const int ld = cfg[where[a].x].ld;
  double* x0 = X + cfg[where[a].x].off + where[a].y;
  for (int x = 0; x < 3; ++x) {
    if (lin) {
      const double* g = lin + (size_t)kRiAtomLin * a;
      for (int t = 0; t < 3; ++t) {
        x0[(size_t)(4 * t + 0) * ld + x] = -g[9 * t + x];
        x0[(size_t)(4 * t + 2) * ld + x] = -g[9 * t + 3 + x];
        x0[(size_t)(4 * t + 3) * ld + x] = 6.0 * g[9 * t + 6 + x];
      }
    }
    x0[(size_t)(sp.n_lin - 1) * ld + x] = -(double)force_ref[a + (size_t)x * N];
  }
}

__global__ void spec_linear_ev(int c0, int n, SpecView sp, const double* __restrict__ lin,
                               const double* __restrict__ qsum, double* __restrict__ M) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double* g = lin + (size_t)kRiCfgLin * (c0 + k);
  const int set = ev_set(c0, k), row = ev_row(k);
  for (int t = 0; t < 3; ++t, g += 22) {
    const int col = 4 * t;
    M[moment_at(sp, set, row, col + 0)] = g[0];
    M[moment_at(sp, set, row, col + 1)] = g[1];
    M[moment_at(sp, set, row, col + 2)] = -g[2];
    M[moment_at(sp, set, row, col + 3)] = -g[3];
    for (int w = 0; w < 6; ++w) {
      M[moment_at(sp, set, row + 1 + w, col + 0)] = g[4 + w];
      M[moment_at(sp, set, row + 1 + w, col + 2)] = g[10 + w];
      M[moment_at(sp, set, row + 1 + w, col + 3)] = -6.0 * g[16 + w];
    }
  }
  M[moment_at(sp, set, row, 12)] = -qsum[c0 + k];
}

// Householder QR of the tiles, in place: afterwards the upper trapezoid of a tile holds its R (what
// lies below is left over).  One CTA per tile of up to 1024 rows; panels of 16 columns are factored in
// shared memory, then applied to the columns behind them as a block, (I - V T' V') x, with FP64 tensor
// cores: 8 columns per warp, D = V' x over the rows, the triangular recurrence
// w_j = tau_j (d_j - sum_{i < j} (v_j . v_i) w_i) per column, x -= V w.  One column reflected at a time
// by a warp (x in registers, panels of 8) took 17 ms for a tile of 648 x 648, bound by the shared-memory
// reads of V.
constexpr int kQrThreads = 512, kQrRows = 1024, kQrPanel = 16, kQrLd = kQrRows + 4;  // + 4: other banks
static_assert(kSpecMaxCols <= kQrRows, "a level of the factorisation has fewer rows than the one before");
constexpr size_t kQrSmem = sizeof(double) * (kQrPanel * kQrLd + kQrThreads / 32 * kQrPanel * 8);
__global__ void __launch_bounds__(kQrThreads, 1) spec_qr(const QrTile* __restrict__ tiles, int n, double* __restrict__ X) {
  extern __shared__ double V[];  // [panel column][row], then [warp][panel column][8]
  __shared__ double part[kQrThreads / 32], tau[kQrPanel], diag[kQrPanel], G[kQrPanel][kQrPanel];
  const QrTile t = tiles[blockIdx.x];
  double* A = X + t.off;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = kQrThreads / 32;
  double* W = V + kQrPanel * kQrLd + warp * kQrPanel * 8;
  const int steps = min(t.rows, n);
  for (int p0 = 0; p0 < steps; p0 += kQrPanel) {
    const int m = t.rows - p0, pw = min(kQrPanel, n - p0), w = min(pw, steps - p0);
    const int mpad = min((m + 7) & ~7, kQrRows);  // zero rows up to a block of 8
    for (int c = warp; c < kQrPanel; c += nw)
      for (int r = lane; r < mpad; r += 32) V[c * kQrLd + r] = c < pw && r < m ? A[(size_t)(p0 + c) * t.ld + p0 + r] : 0.0;
    __syncthreads();
    for (int j = 0; j < w; ++j) {
      double* v = V + j * kQrLd;
      double s = 0.0;
      for (int r = j + 1 + tid; r < m; r += kQrThreads) s = fma(v[r], v[r], s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) part[warp] = s;
      __syncthreads();
      s = 0.0;
#pragma unroll
      for (int k = 0; k < nw; ++k) s += part[k];
      const double alpha = v[j];
      const double beta = s > 0.0 ? -copysign(sqrt(fma(alpha, alpha, s)), alpha) : alpha;
      const double tj = s > 0.0 ? (beta - alpha) / beta : 0.0;
      const double scale = s > 0.0 ? 1.0 / (alpha - beta) : 0.0;
      __syncthreads();  // alpha has been read
      for (int r = j + 1 + tid; r < m; r += kQrThreads) v[r] *= scale;
      if (tid == 0) {
        tau[j] = tj;
        diag[j] = beta;
        v[j] = 1.0;
      }
      __syncthreads();
      for (int c = j + 1 + warp; c < pw; c += nw) {
        double* x = V + c * kQrLd;
        double d = 0.0;
        for (int r = j + lane; r < m; r += 32) d = fma(v[r], x[r], d);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        d *= tj;
        for (int r = j + lane; r < m; r += 32) x[r] = fma(-d, v[r], x[r]);
      }
      __syncthreads();
    }
    // R of the panel, then the reflectors alone (zero above their unit, none where there is no step)
    for (int k = tid; k < kQrPanel * kQrPanel; k += kQrThreads) {
      const int c = k / kQrPanel, r = k % kQrPanel;
      if (c < pw && r < w && r <= c) A[(size_t)(p0 + c) * t.ld + p0 + r] = r == c ? diag[c] : V[c * kQrLd + r];
    }
    __syncthreads();
    if (p0 + pw >= n) break;
    for (int k = tid; k < kQrPanel * kQrPanel; k += kQrThreads) {
      const int c = k / kQrPanel, r = k % kQrPanel;
      if (r < c && r < mpad) V[c * kQrLd + r] = 0.0;
    }
    for (int c = w + warp; c < kQrPanel; c += nw)
      for (int r = lane; r < mpad; r += 32) V[c * kQrLd + r] = 0.0;
    if (tid >= w && tid < kQrPanel) tau[tid] = 0.0;
    __syncthreads();
    for (int k = warp; k < kQrPanel * kQrPanel; k += nw) {
      const int j = k / kQrPanel, i = k % kQrPanel;
      if (i >= j) continue;
      double d = 0.0;
      for (int r = j + lane; r < m; r += 32) d = fma(V[j * kQrLd + r], V[i * kQrLd + r], d);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if (lane == 0) G[j][i] = d;
    }
    __syncthreads();
    const int fr = lane >> 2, fk = lane & 3;
    for (int c0 = p0 + pw + 8 * warp; c0 < n; c0 += 8 * nw) {
      double* a = A + (size_t)c0 * t.ld + p0;
      double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      const double* xb = a + (size_t)fr * t.ld + fk;
#pragma unroll 8
      for (int r = 0; r < mpad; r += 4) {
        const double x = r + fk < m ? xb[r] : 0.0;
        dmma(d[0], V[fr * kQrLd + r + fk], x);
        dmma(d[1], V[(8 + fr) * kQrLd + r + fk], x);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        W[(8 * h + fr) * 8 + 2 * fk] = d[h][0];
        W[(8 * h + fr) * 8 + 2 * fk + 1] = d[h][1];
      }
      __syncwarp();
      if (lane < 8) {
        double wj[kQrPanel];
#pragma unroll
        for (int j = 0; j < kQrPanel; ++j) {
          double y = W[j * 8 + lane];
#pragma unroll
          for (int i = 0; i < j; ++i) y = fma(-G[j][i], wj[i], y);
          wj[j] = tau[j] * y;
          W[j * 8 + lane] = -wj[j];
        }
      }
      __syncwarp();
      double b[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) b[k] = W[(4 * k + fk) * 8 + fr];
      double* xc = a + (size_t)(2 * fk) * t.ld + fr;
#pragma unroll 4
      for (int r = 0; r < mpad; r += 8) {
        const bool in = r + fr < m;
        double x[2] = {in ? xc[r] : 0.0, in ? xc[t.ld + r] : 0.0};
#pragma unroll
        for (int k = 0; k < 4; ++k) dmma(x, V[(4 * k + fk) * kQrLd + r + fr], b[k]);
        if (in) {
          xc[r] = x[0];
          xc[t.ld + r] = x[1];
        }
      }
      __syncwarp();
    }
    __syncthreads();
  }
}

// R of tile `blockIdx.x` (rows above the diagonal of its first min(rows, n) rows) copied to `out`: the
// next level's stack of tiles.
__global__ void spec_stack(const QrTile* __restrict__ from, const QrTile* __restrict__ to, int n,
                           const double* __restrict__ X, double* __restrict__ Y) {
  const QrTile a = from[blockIdx.x], b = to[blockIdx.x];
  const int m = min(a.rows, n);
  for (int k = threadIdx.x; k < m * n; k += blockDim.x) {
    const int c = k / m, r = k - c * m;
    Y[b.off + (size_t)c * b.ld + r] = r <= c ? X[a.off + (size_t)c * a.ld + r] : 0.0;
  }
}

// R of each configuration into the blocked layout.
__global__ void spec_pack(const QrTile* __restrict__ cfg, SpecView sp, int c0, int n, const double* __restrict__ X,
                          double* __restrict__ M) {
  const QrTile a = cfg[blockIdx.x];
  const int m = min(a.rows, n), set = c0 + blockIdx.x;
  for (int k = threadIdx.x; k < m * n; k += blockDim.x) {
    const int r = k / n, c = k - r * n;
    if (r <= c) M[moment_at(sp, set, r, c)] = X[a.off + (size_t)c * a.ld + r];
  }
}

// ------------------------------------------------------------------------------ coefficients
__device__ __forceinline__ float param(const JobView& J, int p, int m) {
  return decode1(J.pmin[m], J.pmax[m], J.pop[(size_t)p * J.num_vars + m]);
}

// tanh(x) = 1 - 2 / (e^{2x} + 1) to an absolute 3e-16 (its values enter sums: those near 0 need no
// relative accuracy).  e^y as in exp_d.cuh (Cody-Waite reduction, Taylor series, here to r^12: 2e-16) for
// |y| <= 40, beyond which tanh rounds to 1; the reciprocal from the hardware's estimate by two Newton steps.
__device__ __forceinline__ double tanh_abs(double x) {
  const double y = fmin(fmax(2.0 * x, -40.0), 40.0);
  const double shifter = 0x1.8p52;
  const double ks = fma(y, 0x1.71547652b82fep+0, shifter), kd = ks - shifter;
  double r = fma(-kd, 0x1.62e42ff000000p-1, y);
  r = fma(kd, 0x1.718432a1b0e26p-35, r);
  constexpr double c[13] = {1.0,         1.0,          0.5,           1.0 / 6.0,      1.0 / 24.0,
                            1.0 / 120.0, 1.0 / 720.0,  1.0 / 5040.0,  1.0 / 40320.0,  1.0 / 362880.0,
                            1.0 / 3628800.0, 1.0 / 39916800.0, 1.0 / 479001600.0};
  double e = c[12];
#pragma unroll
  for (int i = 11; i >= 0; --i) e = fma(e, r, c[i]);
  const double d = __hiloint2double(__double2hiint(e) + (__double2loint(ks) << 20), __double2loint(e)) + 1.0;
  double q;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(d));
  q = fma(fma(-d, q, 1.0), q, q);
  q = fma(fma(-d, q, 1.0), q, q);
  return fma(-2.0, q, 1.0) + (x - x);
}

// NN2B energy before the taper (nn2b.cu:49-78) by two neighboring lanes, each every second neuron of both
// layers: the dependent FP64 chains (about 40 cycles a step) set the time, so lanes and the unrolled
// second layer keep several in flight.  Weights in shared memory: w0, b0, b1, w2, b2 and W1 with an odd row
// stride, so that the lanes of a pair read different banks.
constexpr int nn_stride(int n) { return n | 1; }
template <int NMAX>
__device__ __forceinline__ double nn_energy(const double* __restrict__ w, int n, double d) {
  const int odd = threadIdx.x & 1;
  double x1[NMAX];
#pragma unroll
  for (int m = 0; m < NMAX; m += 2) {
    const int mine = m + odd;
    const double own = mine < n ? tanh_abs(fma(w[mine], d, -w[n + mine])) : 0.0;
    const double other = __shfl_xor_sync(0xffffffffu, own, 1);
    x1[m] = odd ? other : own;
    x1[m + 1] = odd ? own : other;
  }
  const double* b1 = w + 2 * n;
  const double* w2 = w + 3 * n;
  const double* W1 = w + 4 * n + 1 + odd * nn_stride(n);
  double u = 0.0;
#pragma unroll 4
  for (int a = odd; a < n; a += 2) {
    double z0 = -b1[a], z1 = 0.0;
#pragma unroll
    for (int m = 0; m < NMAX; m += 2) {
      if (m < n) z0 = fma(W1[m], x1[m], z0);
      if (m + 1 < n) z1 = fma(W1[m + 1], x1[m + 1], z1);
    }
    u = fma(w2[a], tanh_abs(z0 + z1), u);
    W1 += 2 * nn_stride(n);
  }
  const double v = __shfl_xor_sync(0xffffffffu, u, 1);
  return (odd ? v + u : u + v) - w[4 * n];
}

// One CTA per individual: the pair energy at every piece's Chebyshev nodes, the coefficients
//   c_k = (2 - [k = 0]) / K sum_n U(d_n) cos(pi k (2n + 1) / (2K)),
// the number of column blocks of each piece that matter, and the linear columns' coefficients.
// NMAX: width class of the network (0: rigid ion); MAP's individuals are of that class.
constexpr int coef_threads(int nmax) { return nmax == 0 ? 128 : 512; }
template <int NMAX>
__global__ void __launch_bounds__(coef_threads(NMAX)) spectral_coefs(const JobView* __restrict__ jobs,
                                                               const int2* __restrict__ map) {
  constexpr bool ri = NMAX == 0;
  constexpr int kCoefThreads = coef_threads(NMAX);
  constexpr int kNodes = ri ? 3 * kSpecMaxK : kSpecMaxCols;
  __shared__ double val[kNodes], cf[kNodes];
  __shared__ double wts[ri ? 16 : 4 * NMAX + 1 + NMAX * nn_stride(NMAX)];
  __shared__ SpecPiece pieces[kSpecMaxPieces];
  __shared__ double ctab[ri ? kMaxCtab : 4 * kSpecMaxK];
  __shared__ double sD[kSpecMaxPieces], sU[kSpecMaxPieces], inv_half[kSpecMaxPieces];
  __shared__ int need[kSpecMaxPieces], left[kSpecMaxPieces], length[kSpecMaxPieces], again[kSpecMaxPieces], n_again, bad;
  __shared__ uint8_t owner[kNodes / 8];
  const int2 jp = map[blockIdx.x];
  const JobView& J = jobs[jp.x];
  const SpecView& sp = J.sp;
  const int p = jp.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) bad = 0;
  static_assert(sizeof(SpecPiece) % sizeof(int) == 0, "copied by words");
  for (int k = tid; k < sp.n_pieces * (int)(sizeof(SpecPiece) / sizeof(int)); k += kCoefThreads)
    reinterpret_cast<int*>(pieces)[k] = reinterpret_cast<const int*>(sp.pieces)[k];
  const int nn = J.num_neurons;
  for (int m = tid; m < (ri ? 15 : J.num_vars); m += kCoefThreads) {
    const float w = param(J, p, m);
    if (ri) {
      wts[m] = (double)w;
    } else {
      J.weights[(size_t)m * J.Pstride + p] = w;  // for the direct items
      // parameter order w0[n], b0[n], W1[n][n], b1[n], w2[n], b2
      const int k = m - 2 * nn;
      wts[k < 0 ? m : (k < nn * nn ? 4 * nn + 1 + k / nn * nn_stride(nn) + k % nn : m - nn * nn)] = (double)w;
    }
  }
  for (int j = tid; j < sp.n_ctab; j += kCoefThreads) ctab[j] = sp.ctab[j];
  __syncthreads();
  for (int q = warp; q < sp.n_pieces; q += kCoefThreads / 32) {
    for (int b = lane; b < pieces[q].K / 8; b += 32) owner[pieces[q].node0 / 8 + b] = (uint8_t)q;
    if (lane == 0) inv_half[q] = 1.0 / pieces[q].half;
  }
  // the rigid ion's constants (direct items and linear columns), beside the nodes of the other warps
  if (ri && tid == kCoefThreads - 1) decode_individual(J, p);
  // values at the nodes of a series of `len` terms for piece q, node n, and its coefficient k
  auto value = [&](int q, int n, int len) {
    const SpecPiece& pc = pieces[q];
    const double d = fma(pc.half, ctab[pc.ctab + (2 * n + 1) * (len == pc.K ? 1 : 2)], pc.mid);
    double U;
    if constexpr (ri) {
      const int t = pc.type;
      U = wts[1 + 3 * t] * exp(-d / wts[2 + 3 * t]);
      if (t == 1) {
        const double D0 = wts[11], al = wts[12], S = wts[14], x = d - wts[13];
        U += D0 / (S - 1.0) * exp(-sqrt(2.0 * S) * al * x) - S * D0 / (S - 1.0) * exp(-sqrt(2.0 / S) * al * x);
      }
    } else {
      U = nn_energy<NMAX>(wts, nn, d);
      if (tid & 1) return;
    }
    val[pc.node0 + n] = U;
    if (!(fabs(U) <= 1e30)) bad = 1;
  };
  auto coefficient = [&](int q, int k, int len) {
    const SpecPiece& pc = pieces[q];
    if (k >= len) {
      cf[pc.node0 + k] = 0.0;
      return;
    }
    const double* f = val + pc.node0;
    const double* ct = ctab + pc.ctab;
    const double sign = k & 1 ? -1.0 : 1.0;
    const int K4 = 4 * pc.K, step = 2 * k * (len == pc.K ? 1 : 2);
    double s0 = 0.0, s1 = 0.0;
    int j = step >> 1;  // k (2n + 1) K / len mod 4K
#pragma unroll 4
    for (int n = 0; n < len / 2; n += 2) {
      s0 = fma(fma(sign, f[len - 1 - n], f[n]), ct[j], s0);
      j += step;
      if (j >= K4) j -= K4;
      s1 = fma(fma(sign, f[len - 2 - n], f[n + 1]), ct[j], s1);
      j += step;
      if (j >= K4) j -= K4;
    }
    cf[pc.node0 + k] = (s0 + s1) * ((k ? 2.0 : 1.0) / len);
  };
  // the last significant block of each piece (one warp per piece); left: the last 8 terms still count
  auto judge = [&](double far) {
    for (int q = warp; q < sp.n_pieces; q += kCoefThreads / 32) {
      const SpecPiece& pc = pieces[q];
      double u = 0.0, dd = 0.0;
      for (int k = lane; k < pc.K; k += 32) {
        const double a = fabs(cf[pc.node0 + k]);
        u = fmax(u, a);
        dd = fmax(dd, a * ((double)k * k) * inv_half[q]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        u = fmax(u, __shfl_xor_sync(0xffffffffu, u, o));
        dd = fmax(dd, __shfl_xor_sync(0xffffffffu, dd, o));
      }
      if (lane == 0) {
        sU[q] = u;
        sD[q] = dd;
      }
    }
    __syncthreads();
    for (int q = warp; q < sp.n_pieces; q += kCoefThreads / 32) {
      const SpecPiece& pc = pieces[q];
      double u = 0.0, dd = 0.0;  // of the pieces of this type: the network's, or this exponential's
      for (int r = 0; r < sp.n_pieces; ++r)
        if (pieces[r].type == pc.type) {
          u = fmax(u, sU[r]);
          dd = fmax(dd, sD[r]);
        }
      // where dU/dd is small against U (a saturated network) the rounding of the coefficients, about
      // 1e-16 k^2 / half of U, would never meet the bound on the derivative: U sets it there
      const double tD = (ri ? kTolRI : kTolNN) * fmax(dd, (ri ? 1.0 : 0.05) * u), tU = (ri ? kTolRI : kTolNN) * u;
      int last = 0, l = 0;
      for (int k = lane; k < pc.K; k += 32) {
        const double a = fabs(cf[pc.node0 + k]), da = a * ((double)k * k) * inv_half[q];
        if (a > tU || da > tD) last = k / 8 + 1;
        l |= k < length[q] && k >= length[q] - 8 && (a > far * tU || da > far * tD);
      }
      last = __reduce_max_sync(0xffffffffu, last);
      l = __any_sync(0xffffffffu, l);
      if (lane == 0) {
        need[q] = last;
        left[q] = l;
      }
    }
    __syncthreads();
  };
  if constexpr (ri) {
    __syncthreads();
    for (int c = tid; c < sp.n_nodes; c += kCoefThreads) value(owner[c >> 3], c - pieces[owner[c >> 3]].node0, pieces[owner[c >> 3]].K);
    if (tid < sp.n_pieces) length[tid] = pieces[tid].K;
    __syncthreads();
    for (int c = tid; c < sp.n_nodes; c += kCoefThreads) coefficient(owner[c >> 3], c - pieces[owner[c >> 3]].node0, pieces[owner[c >> 3]].K);
    __syncthreads();
    judge(1.0);
  } else {
    // half the terms first: most pieces of most networks need no more
    constexpr int kHalf = kNNTerms / 2;
    // (whole warps: the lanes of a pair exchange values; nodes beyond the last repeat it)
    const int all = sp.n_pieces * kHalf;
    for (int c = tid; c < ((2 * all + 31) & ~31); c += kCoefThreads) {
      const int x = min(c >> 1, all - 1);
      value(x / kHalf, x % kHalf, kHalf);
    }
    if (tid < sp.n_pieces) length[tid] = kHalf;
    __syncthreads();
    for (int c = tid; c < sp.n_nodes; c += kCoefThreads) coefficient(c / kNNTerms, c % kNNTerms, kHalf);
    __syncthreads();
    judge(1.0);
    if (tid == 0) {
      int m = 0;
      for (int q = 0; q < sp.n_pieces; ++q)
        if (left[q]) again[m++] = q;
      n_again = m;
    }
    __syncthreads();
    const int m = n_again;  // uniform
    if (m > 0) {
      if (tid < m) length[again[tid]] = kNNTerms;
      for (int c = tid; c < 2 * m * kNNTerms; c += kCoefThreads)  // 160 m: whole warps
        value(again[(c >> 1) / kNNTerms], (c >> 1) % kNNTerms, kNNTerms);
      __syncthreads();
      for (int c = tid; c < m * kNNTerms; c += kCoefThreads) coefficient(again[c / kNNTerms], c % kNNTerms, kNNTerms);
      __syncthreads();
      judge(kAcceptNN / kTolNN);
    }
  }
  double v = 1.0;  // this thread's linear column; the last one: the reference force
  if (ri && tid < 13) {
    const double* c64 = J.consts64 + p;
    const size_t st = J.Pstride;
    // R64_* of batched.cu: qq[3], C[3], v_rc, dv_rc, rc, self
    const double vrc = c64[6 * st], dvrc = c64[7 * st], rc = c64[8 * st];
    const int t = tid >> 2;
    const double qq = tid < 12 ? c64[t * st] : 0.0;
    if (tid == 12) v = c64[9 * st];
    else v = (tid & 3) == 0 ? qq : ((tid & 3) == 1 ? qq * (dvrc * rc - vrc) : ((tid & 3) == 2 ? qq * dvrc : c64[(3 + t) * st]));
  }
  // an infinite constant times the zeros of a triangle would be NaN where the sum over pairs is infinite
  if ((tid < sp.n_pieces && left[tid]) || !(fabs(v) <= DBL_MAX)) bad = 1;
  __syncthreads();
  const bool out = bad;
  for (int c = tid; c < sp.n_nodes; c += kCoefThreads) {
    const int q = owner[c >> 3], k = c - pieces[q].node0;
    sp.coef[coef_at(sp, p, column_of(pieces[q], k))] = !out && k < 8 * need[q] ? cf[c] : 0.0;
  }
  if (tid < sp.n_lin) sp.coef[coef_at(sp, p, tid)] = out ? 0.0 : v;
  if (tid == 0) {
    sp.flagged[p] = out ? 1 : 0;
    unsigned long long w = 0;
    for (int q = 0; q < sp.n_pieces && !out; ++q) w |= (unsigned long long)need[q] << (4 * q);
    sp.need[p] = w;
    if (out) sp.list[atomicAdd(sp.count, 1)] = p;
  }
}

// ------------------------------------------------------------------------------ the product
// The products of NM x 8 individuals with NJ row blocks (blocks r0, r0 + W, ...) over the column blocks
// cols[t0 .. n): operands straight from L1/L2 in the fragments' order (16 bytes per lane), the moments D
// steps ahead.
template <int W, int NM, int NJ, int D>
__device__ __forceinline__ void products(const double2* __restrict__ A, const double2* __restrict__ B, int nb,
                                         const int* cols, int t0, int n, double (&acc)[4][2][2]) {
  double2 a[NM], an[NM], b[D][NJ];
#pragma unroll
  for (int s = 0; s < D; ++s) {
    const double2* x = B + (size_t)(cols[t0 + s] * nb) * 32;
#pragma unroll
    for (int j = 0; j < NJ; ++j) b[s][j] = __ldg(x + j * W * 32);
  }
#pragma unroll
  for (int m = 0; m < NM; ++m) a[m] = A[cols[t0] * 128 + m * 32];
  for (int t = t0; t < n; t += D) {
#pragma unroll
    for (int s = 0; s < D; ++s) {
      if (s > 0 && t + s >= n) break;
      const double2* y = A + cols[t + s + 1] * 128;
#pragma unroll
      for (int m = 0; m < NM; ++m) an[m] = y[m * 32];
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
#pragma unroll
        for (int m = 0; m < NM; ++m) dmma(acc[m][j], a[m].x, b[s][j].x);
#pragma unroll
        for (int m = 0; m < NM; ++m) dmma(acc[m][j], a[m].y, b[s][j].y);
      }
      const double2* x = B + (size_t)(cols[t + s + D] * nb) * 32;
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[s][j] = __ldg(x + j * W * 32);
#pragma unroll
      for (int m = 0; m < NM; ++m) a[m] = an[m];
    }
  }
}

// One CTA: 32 individuals x one force configuration (its triangle R) or up to kSpecEvBlocks
// energy/virial configurations (a row block each), row blocks dealt to the W warps in turn, two at a
// time, FP64 tensor-core products over the columns that some individual of the group uses.
//   force: the rows' squares are summed per individual (lanes of a fragment row, then the warps in
//   order); a row block r has no columns before its own, and none that count when r lies behind the
//   last used column: the columns are ordered by degree, so individuals with smooth functions skip
//   rows as well as columns;
//   energy/virial: (E, W[6], 0) of the results, and the sums of their squared errors.
// Operand addresses are one product per step and operand, the fragments of a step at fixed offsets: with
// an address and a guard per load, 10 instructions were issued per MMA and the 749 items of the 16-neuron set
// took 77 us (62 now; their MMAs alone 30).
template <int W, int D, int MINB>
__global__ void __launch_bounds__(W * 32, MINB) spectral_items(const JobView* __restrict__ jobs,
                                                               const WorkItem* __restrict__ items) {
  __shared__ int cols[kSpecMaxCols / 8 + 2 * D];
  __shared__ int s_n;
  __shared__ double red[2][8][32];
  const WorkItem it = items[blockIdx.x];
  const JobView& J = jobs[it.job];
  const SpecView& sp = J.sp;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int P = J.P, ncb = sp.ncb, nf = J.Nc_force;
  const bool force = (it.G >> 28) & 1;
  const int set = force ? it.config : ev_set(nf, it.config - nf);
  const int rows = sp.mnb[set];
  if (warp == 0) {
    // the used column blocks in ascending order: linear ones, then degree by degree
    const unsigned long long w = it.p0 + lane < P ? sp.need[it.p0 + lane] : 0;
    int n = (sp.n_lin + 7) >> 3;
    if (lane < n) cols[lane] = lane;
    int kb = 0, top = 0;  // kb: of piece `lane`
    for (int q = 0; q < sp.n_pieces; ++q) {
      const int m = __reduce_max_sync(0xffffffffu, (int)(w >> (4 * q)) & 15);
      if (lane == q) kb = m;
      top = max(top, m);
    }
    for (int b = 0; b < top; ++b) {
      const unsigned use = __ballot_sync(0xffffffffu, b < kb);
      if (b < kb) cols[n + __popc(use & ((1u << lane) - 1))] = sp.pieces[lane].cb[b];
      n += __popc(use);
    }
    if (lane == 0) s_n = n;
    if (lane < 2 * D) cols[n + lane] = 0;  // read ahead, not used
  }
  __syncthreads();
  const int n = s_n;
  const int nm = min(4, (P - it.p0 + 7) >> 3);
  // row blocks: the triangle's as far as a used column reaches, or one per energy/virial configuration
  const int nb = force ? min(rows, cols[n - 1] + 1) : rows;
  const double2* A = reinterpret_cast<const double2*>(sp.coef) + (size_t)(it.p0 >> 5) * ncb * 128 + lane;
  const double2* M = reinterpret_cast<const double2*>(sp.M + sp.moff[set]) + lane;
  // squared errors by row block modulo 8, whatever W: [class][individual block]
  constexpr int NC = 8 / W;
  double err[NC][4], errW[NC][4];
#pragma unroll
  for (int h = 0; h < NC; ++h)
#pragma unroll
    for (int m = 0; m < 4; ++m) err[h][m] = errW[h][m] = 0.0;
  for (int r0 = warp; r0 < nb; r0 += 2 * W) {
    double acc[4][2][2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[m][j][0] = acc[m][j][1] = 0.0;
    const double2* B = M + r0 * 32;
    int t = 0;
    if (force)
      while (cols[t] < r0) ++t;
    const bool two = r0 + W < nb;
    if (nm == 4) {
      if (two) products<W, 4, 2, D>(A, B, rows, cols, t, n, acc);
      else products<W, 4, 1, D>(A, B, rows, cols, t, n, acc);
    } else if (nm >= 2) {
      if (two) products<W, 3, 2, D>(A, B, rows, cols, t, n, acc);
      else products<W, 3, 1, D>(A, B, rows, cols, t, n, acc);
    } else {
      if (two) products<W, 1, 2, D>(A, B, rows, cols, t, n, acc);
      else products<W, 1, 1, D>(A, B, rows, cols, t, n, acc);
    }
    // lane: individual p0 + 8 m + lane / 4, rows 2 (lane % 4) and the next of every block
    if (force) {
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          err[j % NC][m] = __fma_rn(acc[m][j][0], acc[m][j][0], __fma_rn(acc[m][j][1], acc[m][j][1], err[j % NC][m]));
    } else {
      const int k = 2 * (lane & 3);  // result components k, k + 1 of (E, W[6], 0)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = it.config + r0 + j * W;
        if (r0 + j * W >= nb) continue;
        const double ref0 = k == 0 ? J.E_ref[c] : J.W_ref[c + (size_t)J.v.Nc * (k - 1)];
        const double ref1 = k == 6 ? 0.0 : J.W_ref[c + (size_t)J.v.Nc * k];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int p = it.p0 + 8 * m + (lane >> 2);
          if (p < P && !sp.flagged[p])
            *reinterpret_cast<double2*>(J.res + ((size_t)p * J.v.Nc + c) * kResK + k) = double2{acc[m][j][0], acc[m][j][1]};
          const double d0 = acc[m][j][0] - ref0, d1 = acc[m][j][1] - ref1;
          if (k == 0) err[j % NC][m] = __fma_rn(d0, d0, err[j % NC][m]);
          else errW[j % NC][m] = __fma_rn(d0, d0, errW[j % NC][m]);
          errW[j % NC][m] = __fma_rn(d1, d1, errW[j % NC][m]);
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < NC; ++h)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        err[h][m] += __shfl_xor_sync(0xffffffffu, err[h][m], o);
        errW[h][m] += __shfl_xor_sync(0xffffffffu, errW[h][m], o);
      }
      if ((lane & 3) == 0) {
        red[0][warp + h * W][8 * m + (lane >> 2)] = err[h][m];
        red[1][warp + h * W][8 * m + (lane >> 2)] = errW[h][m];
      }
    }
  __syncthreads();
  const int p = it.p0 + lane;
  if (warp < (force ? 1 : 2) && p < P) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += red[warp][w][lane];
    const int ne = (sp.n_part - nf) / 2;
    const int row = set + (force ? 0 : warp * ne);
    sp.part[(size_t)row * J.Pstride + p] = s;
    if (force && !sp.flagged[p]) J.res[((size_t)p * J.v.Nc + it.config) * kResK + 7] = s;
  }
  finish_item(jobs, it, 32);
}

// Terms that e^{-z x}, |x| <= 1, needs: the next 8 weigh less than kTolRI / 10 of the derivative's scale
// (the values fall faster than geometrically; far beyond, their rounding, times k^2, shows again).
int exp_terms(double z) {
  constexpr int N = 256;
  std::vector<double> f(N), c(4 * N), w(kSpecMaxK + 8);
  for (int j = 0; j < 4 * N; ++j) c[j] = std::cos(M_PI * j / (2.0 * N));
  for (int n = 0; n < N; ++n) f[n] = std::exp(-z * (c[2 * n + 1] + 1.0));
  double top = 0.0;
  for (int k = 0; k < (int)w.size(); ++k) {
    double s = 0.0;
    for (int n = 0; n < N; ++n) s += f[n] * c[k * (2 * n + 1) % (4 * N)];
    w[k] = std::fabs(s) * std::max(1.0, (double)k * k);
    top = std::max(top, w[k]);
  }
  int K = 1;
  for (int k = 0; k < (int)w.size() && k < K + 8; ++k)
    if (w[k] > 0.1 * kTolRI * top) K = k + 1;
  return K;
}

// Terms of the rigid ion's pair type t for distances lo .. hi (above kSpecMaxK: no series), from the steepest exponential
// that the bounds allow: Buckingham 1 / rho, Morse sqrt(2 S) alpha and sqrt(2 / S) alpha.
int ri_terms(const PotentialSpec& sp, int t, double lo, double hi) {
  const int a = 1 + 3 * t, rho = 2 + 3 * t;
  double k = 0.0;
  if (sp.pmin[a] != 0.0f || sp.pmax[a] != 0.0f) {
    if (!(sp.pmin[rho] > 0.0f) || !(sp.pmax[rho] > 0.0f)) return kSpecMaxK + 8;
    k = 1.0 / std::min(sp.pmin[rho], sp.pmax[rho]);
  }
  if (t == 1 && (sp.pmin[11] != 0.0f || sp.pmax[11] != 0.0f)) {
    const double al = std::max(std::fabs(sp.pmin[12]), std::fabs(sp.pmax[12]));
    const double s0 = std::min(sp.pmin[14], sp.pmax[14]), s1 = std::max(sp.pmin[14], sp.pmax[14]);
    if (!(s0 > 0.0)) return kSpecMaxK + 8;
    k = std::max(k, std::max(std::sqrt(2.0 * s1), std::sqrt(2.0 / s0)) * al);
  }
  const double z = k * (0.5 * (hi - lo) * 1.02 + 1e-3);
  return z < 200.0 ? ((exp_terms(z) + 7) & ~7) + 8 : kSpecMaxK + 8;  // one more block: it must be negligible
}

}  // namespace

// At most what the expansion takes for a training set and a population of P, with the work space of the factorisation: all
// pair types as present, distances up to the cutoff.
size_t spectral_bytes(const PotentialSpec& spec, const TrainingSet& ts, int P) {
  if (spec.type != 3 && !is_ri_type(spec.type)) return 0;
  double cols = 8.0;
  if (spec.type == 3) {
    cols += kNNTerms * (std::ceil(spec.cutoff / nn_piece_length(spec.num_neurons)) + 1);
  } else {
    cols += 8.0;
    if (spec.pmin.size() < 15 || spec.pmax.size() < 15) return 0;
    for (int t = 0; t < 3; ++t) cols += std::min(ri_terms(spec, t, 1.0, spec.cutoff), kSpecMaxK);
  }
  cols = std::min(cols, (double)kSpecMaxCols);
  double rows = 8.0 * (ts.Nc - ts.Nc_force), all = 0.0, largest = 0.0;
  for (int c = 0; c < ts.Nc_force; ++c) {
    rows += std::min(3.0 * ts.Na[c], cols) + 8.0;
    all += 24.0 * ts.Na[c] * cols;
    largest = std::max(largest, 24.0 * ts.Na[c] * cols);
  }
  const double moments = 8.0 * cols * rows, work = 2.0 * std::min(all, std::max(largest, kQrBatchBytes));
  const double plan = (double)((P + 31) & ~31) * 8.0 * (cols + ts.Nc_force + (ts.Nc - ts.Nc_force) / 8 + 4);
  return (size_t)(std::min(moments, (double)spec.expansion_bytes) + work + plan);
}

int spectral_class(const DevSet& d) {
  if (is_ri_type(d.potential_type)) return 0;
  return d.num_neurons <= 8 ? 1 : (d.num_neurons <= 12 ? 2 : (d.num_neurons <= 16 ? 3 : 4));
}

namespace {

// The triangles of the force configurations [c0, c1) into M: sums, QR (in levels of 1024-row tiles for
// large configurations), packing.
int factor_configs(Engine* e, const SpecView& v, int c0, int c1, const NNTaper& tp, int nn, int active, double* M) {
  const DevSet& d = e->d;
  const TrainingSet& ts = e->ts;
  cudaStream_t st = e->stream;
  const int n = 8 * v.ncb, nc = c1 - c0, a0 = ts.Na_sum[c0], a1 = ts.Na_sum[c1 - 1] + ts.Na[c1 - 1];
  std::vector<QrTile> cfg(nc);
  std::vector<int2> where(a1 - a0);
  size_t total = 0;
  for (int c = c0; c < c1; ++c) {
    cfg[c - c0] = {total, 3 * ts.Na[c], 3 * ts.Na[c]};
    total += (size_t)3 * ts.Na[c] * n;
    for (int k = 0; k < ts.Na[c]; ++k) where[ts.Na_sum[c] - a0 + k] = make_int2(c - c0, 3 * k);
  }
  std::vector<void*> tmp;
  // frees a level's work space; kernels that use it may still run (cudaFree waits for them)
  auto drop = [&](void* p) {
    const auto it = std::find(tmp.begin(), tmp.end(), p);
    if (it != tmp.end()) tmp.erase(it);
    cudaFree(p);
  };
  auto room = [&](size_t bytes) -> void* {
    void* p = nullptr;
    if (cudaMalloc(&p, std::max<size_t>(bytes, 16)) != cudaSuccess) return nullptr;
    tmp.push_back(p);
    return p;
  };
  auto put = [&](const auto& src) {
    using T = typename std::remove_reference<decltype(src)>::type::value_type;
    T* p = static_cast<T*>(room(sizeof(T) * src.size()));
    // (in the order of the kernels: the engine's stream does not wait for the legacy one)
    if (p && cudaMemcpyAsync(p, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice, st) != cudaSuccess) return (T*)nullptr;
    return p;
  };
  auto run = [&]() -> int {
    double* X = static_cast<double*>(room(sizeof(double) * total));
    QrTile* d_cfg = put(cfg);
    int2* d_where = put(where);
    if (!X || !d_cfg || !d_where) return GPUGA_ERR_OOM;
    GPUGA_CUDA(cudaMemsetAsync(X, 0, sizeof(double) * total, st));
    spec_force_moments<<<(a1 - a0 + 7) / 8, 256, 0, st>>>(a0, a1 - a0, v, d_cfg, d_where - a0, d.off, d.ptype, d.g64, tp, nn,
                                                          active, X);
    spec_linear_force<<<(a1 - a0 + 127) / 128, 128, 0, st>>>(a0, a1 - a0, ts.N, v, d_cfg, d_where - a0,
                                                             nn ? nullptr : d.ri_atom_lin, d.force_ref, X);
    GPUGA_CUDA(cudaGetLastError());
    GPUGA_CUDA(cudaFuncSetAttribute(spec_qr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQrSmem));
    for (;;) {
      std::vector<QrTile> tiles, stacked(nc), to;
      size_t next = 0;
      bool more = false;
      for (int c = 0; c < nc; ++c) {
        stacked[c] = {next, 0, 0};
        int rows = 0;
        const int nt0 = (int)tiles.size();
        for (int r = 0; r < cfg[c].rows; r += kQrRows) {
          tiles.push_back({cfg[c].off + r, cfg[c].ld, std::min(kQrRows, cfg[c].rows - r)});
          rows += std::min(tiles.back().rows, n);
        }
        more |= cfg[c].rows > kQrRows;
        stacked[c].ld = stacked[c].rows = rows;
        size_t o = next;
        for (int k = nt0; k < (int)tiles.size(); ++k) {
          to.push_back({o, rows, 0});
          o += std::min(tiles[k].rows, n);
        }
        next += (size_t)rows * n;
      }
      QrTile* d_tiles = put(tiles);
      if (!d_tiles) return GPUGA_ERR_OOM;
      spec_qr<<<(unsigned)tiles.size(), kQrThreads, kQrSmem, st>>>(d_tiles, n, X);
      GPUGA_CUDA(cudaGetLastError());
      if (!more) break;
      double* Y = static_cast<double*>(room(sizeof(double) * next));
      QrTile* d_to = put(to);
      if (!Y || !d_to) return GPUGA_ERR_OOM;
      spec_stack<<<(unsigned)tiles.size(), 256, 0, st>>>(d_tiles, d_to, n, X, Y);
      GPUGA_CUDA(cudaGetLastError());
      drop(X);  // (with 900 columns a level is 0.9 of the one before: a large cell has dozens)
      drop(d_tiles);
      drop(d_to);
      X = Y;
      cfg = stacked;
      d_cfg = put(cfg);
      if (!d_cfg) return GPUGA_ERR_OOM;
    }
    spec_pack<<<nc, 256, 0, st>>>(d_cfg, v, c0, n, X, M);
    GPUGA_CUDA(cudaGetLastError());
    GPUGA_CUDA(cudaStreamSynchronize(st));
    return GPUGA_OK;
  };
  const int s = run();
  if (s != GPUGA_OK) cudaStreamSynchronize(st);
  for (void* p : tmp) cudaFree(p);
  return s;
}

}  // namespace

int spectral_build(Engine* e) {
  DevSet& d = e->d;
  const TrainingSet& ts = e->ts;
  const PotentialSpec& sp = e->spec;
  const bool ri = is_ri_type(d.potential_type), nn = d.potential_type == 3;
  if ((!ri && !nn) || sp.expansion_bytes == 0 || d.B == 0) return GPUGA_OK;
  cudaStream_t st = e->stream;
  const NNTaper tp{sp.nn_r1, sp.nn_r2, 0.f, sp.nn_consistent};
  const int active = ri ? d.ri_active : 1;
  // distance ranges
  unsigned long long h[9], *d_h = nullptr;
  for (int k = 0; k < 9; ++k) h[k] = k % 3 == 0 ? ~0ull : 0ull;
  GPUGA_CUDA(cudaMalloc(&d_h, sizeof h));
  GPUGA_CUDA(cudaMemcpyAsync(d_h, h, sizeof h, cudaMemcpyHostToDevice, st));
  spec_range<<<std::min((d.B + 255) / 256, 1184), 256, 0, st>>>(d.B, d.g64, d.ptype, active, nn ? (double)sp.nn_r2 : DBL_MAX,
                                                                d_h);
  cudaError_t ce = cudaGetLastError();
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(h, d_h, sizeof h, cudaMemcpyDeviceToHost, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  cudaFree(d_h);
  GPUGA_CUDA(ce);
  std::vector<SpecPiece> pieces;
  std::vector<double> ctab;
  double bonds = 0.0;
  int cols = 0;
  auto add = [&](int type, double lo, double hi, double to, int K) {
    SpecPiece pc{};
    pc.mid = 0.5 * (lo + hi);
    pc.half = 0.5 * (hi - lo) * 1.02 + 1e-3;
    pc.to = to;
    pc.type = type;
    pc.K = K;
    pc.node0 = cols;
    pc.ctab = -1;
    for (const SpecPiece& o : pieces)
      if (o.K == K) pc.ctab = o.ctab;
    if (pc.ctab < 0) {
      pc.ctab = (int)ctab.size();
      for (int j = 0; j < 4 * K; ++j) ctab.push_back(std::cos(M_PI * j / (2.0 * K)));
    }
    cols += K;
    pieces.push_back(pc);
  };
  for (int t = 0; t < 3; ++t) {
    if (h[3 * t + 2] == 0) continue;
    double lo, hi;
    memcpy(&lo, &h[3 * t], 8);
    memcpy(&hi, &h[3 * t + 1], 8);
    bonds += (double)h[3 * t + 2];
    if (!(lo > 0.0) || !std::isfinite(hi)) return GPUGA_OK;
    if (nn) {
      const int S = std::max(1, (int)std::ceil((hi - lo) / nn_piece_length(d.num_neurons)));
      if (S > kSpecMaxPieces) return GPUGA_OK;
      for (int s = 0; s < S; ++s) {
        const double a = lo + (hi - lo) * s / S, b = lo + (hi - lo) * (s + 1) / S;
        add(t, a, b, s + 1 < S ? b : DBL_MAX, kNNTerms);
      }
    } else {
      const int K = ri_terms(sp, t, lo, hi);
      if (K > kSpecMaxK) return GPUGA_OK;
      add(t, lo, hi, DBL_MAX, K);
    }
  }
  SpecView v{};
  v.n_pieces = (int)pieces.size();
  v.n_nodes = cols;
  v.n_ctab = (int)ctab.size();
  v.n_lin = ri ? 14 : 1;
  v.ncb = (v.n_lin + 7) / 8;
  int top = 0;
  for (const SpecPiece& pc : pieces) top = std::max(top, pc.K / 8);
  for (int b = 0; b < top; ++b)
    for (SpecPiece& pc : pieces)
      if (b < pc.K / 8) pc.cb[b] = v.ncb++;
  if (v.n_pieces == 0 || 8 * v.ncb >= kSpecMaxCols) return GPUGA_OK;  // (fewer columns than a tile's rows: levels shrink)
  const int n = 8 * v.ncb, Nev = ts.Nc - ts.Nc_force;
  const int nev_items = (Nev + kSpecEvBlocks - 1) / kSpecEvBlocks;
  std::vector<long long> moff(ts.Nc_force + nev_items + 1);
  std::vector<int> mnb(ts.Nc_force + nev_items + 1, 0);
  e->h_spec_blocks.assign(std::max(ts.Nc_force, 1), 0);
  double products = (double)Nev * v.ncb;
  long long size = 0;
  for (int k = 0; k < ts.Nc_force + nev_items; ++k) {
    moff[k] = size;
    if (k < ts.Nc_force) {
      mnb[k] = (int)((std::min<long long>(3LL * ts.Na[k], n) + 7) / 8);
      for (int r = 0; r < mnb[k]; ++r) e->h_spec_blocks[k] += v.ncb - r;
      products += e->h_spec_blocks[k];
    } else {
      mnb[k] = std::min(kSpecEvBlocks, Nev - (k - ts.Nc_force) * kSpecEvBlocks);
    }
    size += 64LL * mnb[k] * v.ncb;
  }
  // The expansion pays when its products (64 FMAs at half the FP32 rate, hence the 2) and node values
  // cost less than the direct pairs (each unordered pair once, except the rigid ion's force items).
  const double w = d.num_neurons, share = (double)ts.N_force / ts.N;
  const double direct = ri ? bonds * (share + 0.5 * (1.0 - share)) * 50.0 : 0.5 * bonds * (2.0 * w * w + 40.0 * w);
  const double expanded = 128.0 * products + cols * (ri ? 200.0 : 2.0 * w * w + 240.0 * w) + 2.0 * cols * pieces[0].K;
  if (expanded > direct) return GPUGA_OK;
  // (the products' loads run up to a block past the last row block of a set)
  const size_t bytes = sizeof(double) * (size_t)(size + 64 * 32);
  if (bytes > sp.expansion_bytes) return GPUGA_OK;
  double* M = nullptr;
  GPUGA_TRY(e->alloc(&M, bytes / sizeof(double)));  // (no room: the direct path needs less)
  auto up = [&](auto** dst, const auto& src) -> int {
    using T = typename std::remove_reference<decltype(src[0])>::type;
    typename std::remove_const<T>::type* p = nullptr;
    GPUGA_TRY(e->alloc(&p, std::max<size_t>(src.size(), 1)));
    if (!src.empty()) GPUGA_CUDA(cudaMemcpyAsync(p, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice, st));
    *dst = p;
    return GPUGA_OK;
  };
  GPUGA_TRY(up(&v.pieces, pieces));
  GPUGA_TRY(up(&v.ctab, ctab));
  GPUGA_TRY(up(&v.moff, moff));
  GPUGA_TRY(up(&v.mnb, mnb));
  v.n_items = ts.Nc_force + nev_items;
  v.n_part = ts.Nc_force + 2 * nev_items;
  GPUGA_CUDA(cudaMemsetAsync(M, 0, bytes, st));
  for (int c0 = 0; c0 < ts.Nc_force;) {  // batches of bounded work space
    int c1 = c0;
    double size = 0.0;
    do size += 24.0 * ts.Na[c1++] * n;
    while (c1 < ts.Nc_force && size + 24.0 * ts.Na[c1] * n <= kQrBatchBytes);
    GPUGA_TRY(factor_configs(e, v, c0, c1, tp, nn, active, M));
    c0 = c1;
  }
  if (Nev > 0) {
    spec_ev_moments<<<dim3(Nev, v.n_pieces), kEvWarps * 32, 0, st>>>(ts.Nc_force, v, d.Na, d.Na_sum, d.off, d.half_off,
                                                                     d.ptype, d.g64, tp, nn, active, M);
    if (ri)
      spec_linear_ev<<<(Nev + 127) / 128, 128, 0, st>>>(ts.Nc_force, Nev, v, d.ri_cfg_lin, d.ri_qsum, M);
    GPUGA_CUDA(cudaGetLastError());
  }
  GPUGA_CUDA(cudaStreamSynchronize(st));
  v.M = M;
  d.sp = v;
  return GPUGA_OK;
}

int spectral_plan(Engine* e, Plan* plan) {
  SpecView v = e->d.sp;
  const int P = plan->P, groups = (P + 31) / 32 * 4;
  GPUGA_TRY(e->alloc(&v.coef, (size_t)groups * v.ncb * 64));
  GPUGA_TRY(e->alloc(&v.need, (size_t)P));
  GPUGA_TRY(e->alloc(&v.part, (size_t)v.n_part * plan->Pstride));
  GPUGA_TRY(e->alloc(&v.flagged, (size_t)P));
  GPUGA_TRY(e->alloc(&v.list, (size_t)P));
  GPUGA_TRY(e->alloc(&v.count, 2));
  GPUGA_CUDA(cudaMemset(v.coef, 0, sizeof(double) * (size_t)groups * v.ncb * 64));
  GPUGA_CUDA(cudaMemset(v.count, 0, 2 * sizeof(int)));
  plan->sp = v;
  return GPUGA_OK;
}

int spectral_coefficients(const LaunchSet* ls, cudaStream_t st) {
  const int2* map = ls->d_specmap;
  for (int k = 0; k < 5; ++k) {
    const int n = ls->spec_class[k];
    if (!n) continue;
    if (k == 0) spectral_coefs<0><<<n, coef_threads(0), 0, st>>>(ls->d_jobs, map);
    else if (k == 1) spectral_coefs<8><<<n, coef_threads(8), 0, st>>>(ls->d_jobs, map);
    else if (k == 2) spectral_coefs<12><<<n, coef_threads(12), 0, st>>>(ls->d_jobs, map);
    else if (k == 3) spectral_coefs<16><<<n, coef_threads(16), 0, st>>>(ls->d_jobs, map);
    else spectral_coefs<32><<<n, coef_threads(32), 0, st>>>(ls->d_jobs, map);
    GPUGA_CUDA(cudaGetLastError());
    map += n;
  }
  return GPUGA_OK;
}

int spectral_items_launch(const JobView* jobs, const WorkItem* items, int count, int sms, cudaStream_t st) {
  // Eight warps per CTA where there are fewer than four items per SM (each warp then has half the row blocks to walk),
  // four otherwise: 68 items of 31 configurations, 10 neurons at 8 A: 88 against 101 us per generation;
  // 2119 items of the 300-configuration oxide set: 117 against 103.  The sums do not depend on it.
  if (count < 4 * sms) spectral_items<8, 2, 2><<<count, 256, 0, st>>>(jobs, items);
  else spectral_items<4, 2, 4><<<count, 128, 0, st>>>(jobs, items);
  GPUGA_CUDA(cudaGetLastError());
  return GPUGA_OK;
}

}  // namespace gpuga
