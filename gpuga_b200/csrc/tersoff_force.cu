// Force items of the minimal Tersoff potential for configurations whose atoms have at most four bonds inside R2, R1 and
// R2 fixed by their bounds: two individuals per lane, in packed FP32 (fma.rn.f32x2 and its kin).
//
// A force item needs f_ij = dE_i / dr_ij of its whole configuration before F_i = sum_j (f_ij - f_ji) can be formed, so
// a CTA keeps them in shared memory.  With fc_k known, s_j = sum_k fc_k x_jk^2, x = cos - h, zeta = beta s and
//   S_j = beta b'(zeta_j) fa_j,   q_jk = x_jk fc_k (S_j + S_k),   V_j = sum_k q_jk u_k,
//   f_ij = (A'_j / 2 - fc'_j / 2 sum_k S_k fc_k x_jk^2) u_j + (fc_j / d_j) ((V_j . u_j) u_j - V_j)
// (minimal_tersoff.cu:122-316; V_j . u_j = sum_k q_jk cos_jk).  Atoms with four bonds inside R1 (fc = 1, fc' = 0) come
// first in each configuration and take a form without the cutoff terms; which form an atom takes is a property of the
// training set, so results do not depend on how atoms share a warp.
//
// What bounds it: issue, the FP32 pipe and the SFU in about equal parts (per two individuals and atom some 430
// instructions, 200 of them packed, and 40 SFU).  The scalar form in batched.cu issued about 516 per individual and
// atom: the packed operations halve the arithmetic, and geometry, addresses and cosines are shared by the two.  Bond
// orders and exponentials come from the SFU (lg2 / ex2 / rcp.approx.ftz) as there, 1 / d from the training set.
// It issues on about 40 % of cycles: 16 warps per SM (128 registers, the scratch) wait for the geometry from L2 and at the two
// barriers.  So CTAs are small: four of 128 threads whose phases overlap, 945 us at 1000 individuals x 250 configurations of
// 8 to 512 atoms, where two of 256 threads with twice the individuals took 1019 us (the scalar form: 1.58 ms).
#include <algorithm>
#include <cmath>

#include "decode.cuh"
#include "engine.hpp"
#include "fold.cuh"

namespace gpuga {

namespace {

constexpr int kFThreads = 128, kFThreadsLarge = 256;  // per CTA: scratch of up to kForceSmem, above

// ------------------------------------------------------------------------------ packed FP32
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup(float a) { return pack(a, a); }
__device__ __forceinline__ float2 unpack(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, dup(-1.0f), a); }
// the SFU's approximations, each half on its own (arguments and results are normal numbers or handled by the caller)
__device__ __forceinline__ f2 lg2_2(f2 v) {
  float2 x = unpack(v);
  asm("lg2.approx.ftz.f32 %0, %0;" : "+f"(x.x));
  asm("lg2.approx.ftz.f32 %0, %0;" : "+f"(x.y));
  return pack(x.x, x.y);
}
__device__ __forceinline__ f2 ex2_2(f2 v) {
  float2 x = unpack(v);
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.x));
  asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(x.y));
  return pack(x.x, x.y);
}
__device__ __forceinline__ f2 rcp_2(f2 v) {
  float2 x = unpack(v);
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(x.x));
  asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(x.y));
  return pack(x.x, x.y);
}

// ------------------------------------------------------------------------------ set-up
// Per force atom: the rank of each bond among those inside R2 (-1: beyond), their number, whether all four lie inside R1,
// and -1 where a bond has no reverse.
__global__ void force_ranks(int n_atoms, const int* __restrict__ off, const int* __restrict__ nbr, const int* __restrict__ rev,
                            const double4* __restrict__ g64, double r1, double r2, signed char* __restrict__ rank,
                            int* __restrict__ kind) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_atoms) return;
  int n = 0, inner = 1, ok = 1;
  for (int b = off[i]; b < off[i + 1]; ++b) {
    const double d = g64[b].w;
    if (!(d < r2)) {
      rank[b] = -1;
      continue;
    }
    inner &= d < r1;
    const int r = rev[b];
    ok &= nbr[r] == i && g64[r].w == d && nbr[b] != i;
    rank[b] = (signed char)min(n++, 100);
  }
  kind[i] = !ok || n > 4 ? -1 : (n == 4 && inner ? 1 : 0);
}

// Slot-major geometry: slot j of the atom at place il of its configuration at base + j Na + il.
__global__ void force_geometry(int n_atoms, const int* __restrict__ off, const int* __restrict__ nbr,
                               const int* __restrict__ rev, const uint8_t* __restrict__ ptype,
                               const double4* __restrict__ g64, double r1, double r2, const signed char* __restrict__ rank,
                               const int* __restrict__ place, const int2* __restrict__ where,
                               const float* __restrict__ force_ref, int N, float4* __restrict__ gu,
                               float4* __restrict__ gd, int* __restrict__ grev, double* __restrict__ ref) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_atoms) return;
  const int base = where[i].x, Na = where[i].y;  // base < 0: not one of these configurations
  if (base < 0) return;
  const int il = place[i];
  int n = 0;
  for (int b = off[i]; b < off[i + 1]; ++b) {
    const int r = rank[b];
    if (r < 0) continue;
    const double4 v = g64[b];
    double fc = 1.0, fcp = 0.0;
    if (v.w >= r1) {
      const double pf = M_PI / (r2 - r1);
      double s, c;
      sincos(pf * (v.w - r1), &s, &c);
      fc = 0.5 * c + 0.5;
      fcp = -0.5 * pf * s;
    }
    const int o = base + r * Na + il;
    gu[o] = make_float4((float)(v.x / v.w), (float)(v.y / v.w), (float)(v.z / v.w), (float)v.w);
    // 1 / d, its sign bit the pair set; d - (float)d; fc; fc'
    gd[o] = make_float4((float)(1.0 / v.w) * (ptype[b] ? -1.f : 1.f), (float)(v.w - (double)(float)v.w), (float)fc, (float)fcp);
    grev[o] = rank[rev[b]] * Na + place[nbr[b]];
    ++n;
  }
  for (int r = n; r < 4; ++r) {  // no bond: weight zero
    const int o = base + r * Na + il;
    gu[o] = make_float4(0.f, 0.f, 0.f, (float)r2);  // (a length at which the pair terms are ordinary numbers)
    gd[o] = make_float4(1.f, 0.f, 0.f, 0.f);
    grev[o] = r * Na + il;
  }
  for (int x = 0; x < 3; ++x) ref[(size_t)3 * (base / 4 + il) + x] = (double)force_ref[i + (size_t)x * N];
}

// ------------------------------------------------------------------------------ items
// Packed constants of a pair of individuals, in shared memory [constant][pair].
enum { FK_MH, FK_BETA, FK_EN, FK_MHON, FK_MHONL, FK_R0, FK_LA = FK_R0 + 2, FK_CA = FK_LA + 2, FK_LR = FK_CA + 2,
       FK_CR = FK_LR + 2, FK_LAL = FK_CR + 2, FK_CAL = FK_LAL + 2, FK_LRL = FK_CAL + 2, FK_CRL = FK_LRL + 2,
       FK_COUNT = FK_CRL + 2 };

template <int NT, bool LO>
struct ForceConsts {
  const f2* k;  // this lane's pair
  int H;
  __device__ __forceinline__ f2 operator[](int c) const { return k[c * H]; }
};

// b, beta b' and the pair terms of one bond: half of A' / fc (INNER: A' / 2), S = beta b' fa; e = fr - b fa (not INNER).
template <int NT, bool LO, bool INNER>
__device__ __forceinline__ void bond_terms(const ForceConsts<NT, LO>& K, f2 s, float d, float dlo, int set, f2& hdA, f2& S,
                                           f2& e) {
  const f2 zeta = mul2(K[FK_BETA], s);
  const f2 zn = ex2_2(mul2(K[FK_EN], lg2_2(zeta)));
  const f2 opz = add2(zn, dup(1.0f));
  const f2 lg = lg2_2(opz);
  f2 b = ex2_2(fma2(K[FK_MHON], lg, mul2(K[FK_MHONL], lg)));
  f2 db = mul2(mul2(mul2(b, dup(-0.5f)), zn), rcp_2(mul2(opz, s)));  // db / ds
  // b = 1, b' = 0 below zeta = 1e-16 (minimal_tersoff.cu:178-185; almost never met)
  const float2 z = unpack(zeta);
  if (fminf(z.x, z.y) < 1.0e-16f) {
    float2 bb = unpack(b), dd = unpack(db);
    if (z.x < 1.0e-16f) {
      bb.x = 1.f;
      dd.x = 0.f;
    }
    if (z.y < 1.0e-16f) {
      bb.y = 1.f;
      dd.y = 0.f;
    }
    b = pack(bb.x, bb.y);
    db = pack(dd.x, dd.y);
  }
  const f2 t = sub2(dup(d), K[FK_R0 + set]), la = K[FK_LA + set], ca = K[FK_CA + set];
  constexpr float kLog2e = 1.4426950408889634f;
  // e^{-l (t + d_lo)} = e^{-l t} (1 - l d_lo)
  const f2 nla = mul2(la, dup(-1.0f));
  f2 ea = ex2_2(mul2(mul2(nla, t), dup(kLog2e)));
  ea = fma2(mul2(nla, dup(dlo)), ea, ea);
  f2 fa = mul2(ca, ea);
  if constexpr (!LO) {
    // S = 2: fr = fa ea / 2, fr' - b fa' = la fa (b - ea)
    hdA = mul2(mul2(mul2(la, dup(0.5f)), fa), sub2(b, ea));
    if (!INNER) e = mul2(fa, sub2(mul2(ea, dup(0.5f)), b));
  } else {
    // two exponentials; the remainders of the constants to first order (batched.cu)
    const f2 lr = K[FK_LR + set], cr = K[FK_CR + set], lal = K[FK_LAL + set], lrl = K[FK_LRL + set];
    const f2 nlr = mul2(lr, dup(-1.0f));
    f2 er = ex2_2(mul2(mul2(nlr, t), dup(kLog2e)));
    er = fma2(mul2(nlr, dup(dlo)), er, er);
    f2 fr = mul2(cr, er);
    const f2 m1 = dup(-1.0f);
    fr = fma2(fma2(mul2(mul2(cr, m1), lrl), t, K[FK_CRL + set]), er, fr);
    fa = fma2(fma2(mul2(mul2(ca, m1), lal), t, K[FK_CAL + set]), ea, fa);
    const f2 frp = fma2(mul2(lrl, m1), fr, mul2(nlr, fr)), fap = fma2(mul2(lal, m1), fa, mul2(nla, fa));
    hdA = mul2(dup(0.5f), fma2(mul2(b, m1), fap, frp));
    if (!INNER) e = fma2(mul2(b, m1), fa, fr);
  }
  S = mul2(db, fa);
}

// f_ij of the atom at place il for the lane's two individuals, into the scratch (records of 3 x 8 bytes).
template <int NT, bool LO, bool INNER>
__device__ __forceinline__ void atom_forces(const ForceConsts<NT, LO>& K, const float4* __restrict__ gu,
                                            const float4* __restrict__ gd, int Na, int il, f2* __restrict__ rec, int lgH) {
  float4 u[4], w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    u[j] = __ldg(gu + j * Na + il);
    w[j] = __ldg(gd + j * Na + il);
  }
  // x_jk = cos_jk - h, both halves; index of the unordered pair
  auto at = [](int j, int k) { return j < k ? j * (7 - j) / 2 + k - j - 1 : k * (7 - k) / 2 + j - k - 1; };
  f2 x[6];
  const f2 mh = K[FK_MH];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = j + 1; k < 4; ++k)
      x[at(j, k)] = add2(dup(fmaf(u[j].z, u[k].z, fmaf(u[j].y, u[k].y, u[j].x * u[k].x))), mh);
  f2 hA[4], S[4], G[INNER ? 1 : 4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f2 s = 0;
    bool first = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == j) continue;
      const f2 a = x[at(j, k)];
      if constexpr (INNER) s = first ? mul2(a, a) : fma2(a, a, s);
      else s = first ? mul2(mul2(a, a), dup(w[k].z)) : fma2(mul2(a, a), dup(w[k].z), s);
      first = false;
    }
    f2 e;
    const int set = NT == 2 && w[j].x < 0.f ? 1 : 0;
    bond_terms<NT, LO, INNER>(K, s, u[j].w, w[j].y, set, hA[j], S[j], e);
    if constexpr (!INNER) {
      hA[j] = fma2(dup(0.5f * w[j].w), e, mul2(dup(w[j].z), hA[j]));
      // no bond, or one whose others all have weight zero: s = 0 gives b = 1, b' = 0 above; a slot without a bond has
      // weight zero throughout
    }
  }
  if constexpr (!INNER) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f2 g = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k == j) continue;
        const f2 a = x[at(j, k)];
        g = fma2(mul2(S[k], dup(w[k].z)), mul2(a, a), g);
      }
      G[j] = g;
    }
  }
  // x becomes x (S_j + S_k)
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = j + 1; k < 4; ++k) x[at(j, k)] = mul2(x[at(j, k)], add2(S[j], S[k]));
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f2 Vx = 0, Vy = 0, Vz = 0;
    bool first = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == j) continue;
      const f2 q = INNER ? x[at(j, k)] : mul2(x[at(j, k)], dup(w[k].z));
      Vx = first ? mul2(q, dup(u[k].x)) : fma2(q, dup(u[k].x), Vx);
      Vy = first ? mul2(q, dup(u[k].y)) : fma2(q, dup(u[k].y), Vy);
      Vz = first ? mul2(q, dup(u[k].z)) : fma2(q, dup(u[k].z), Vz);
      first = false;
    }
    const f2 acc = fma2(dup(u[j].z), Vz, fma2(dup(u[j].y), Vy, mul2(dup(u[j].x), Vx)));
    const float id = NT == 2 ? fabsf(w[j].x) : w[j].x;
    const float c = INNER ? id : id * w[j].z;
    f2 cu = fma2(dup(c), acc, hA[j]);
    if constexpr (!INNER) cu = fma2(dup(-0.5f * w[j].w), G[j], cu);
    f2* r = rec + 3 * ((size_t)(j * Na + il) << lgH);
    r[0] = fma2(cu, dup(u[j].x), mul2(dup(-c), Vx));
    r[1] = fma2(cu, dup(u[j].y), mul2(dup(-c), Vy));
    r[2] = fma2(cu, dup(u[j].z), mul2(dup(-c), Vz));
  }
}

// One CTA: one configuration x G = 2 H individuals, lane = pair of individuals x atom.  First every atom's f_ij into
// shared memory, then F_i and its squared error in FP64: per thread its atoms in step order, then the warps in order,
// then a butterfly over the atom slots of an individual (H is a property of the configuration, so is the order).
template <int NT, bool LO>
__global__ void __launch_bounds__(kFThreadsLarge, 2) tersoff_force(const JobView* __restrict__ jobs,
                                                              const WorkItem* __restrict__ items) {
  extern __shared__ __align__(16) unsigned char smem[];
  const WorkItem it = items[blockIdx.x];
  const JobView& J = jobs[it.job];
  const TersoffForceView& v = J.tf;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int c = it.config, Na = J.v.Na[c], P = J.P;
  const int lgH = v.lgH[c], H = 1 << lgH, A = 32 >> lgH;
  const int h = lane & (H - 1), aslot = lane >> lgH;
  const int base = v.base[c], n_inner = v.inner[c];
  f2* tab = reinterpret_cast<f2*>(smem);       // [FK_COUNT][H]
  f2* scratch = tab + FK_COUNT * 16;           // [slot][atom][H] records of 3
  for (int t = threadIdx.x; t < FK_COUNT * H; t += blockDim.x) {
    const int k = t >> lgH, hh = t & (H - 1);
    auto value = [&](int half) -> float {
      const int p = min(it.p0 + 2 * hh + half, P - 1);
      const Consts C{J.consts, J.Pstride, p};
      switch (k) {
        case FK_MH: return -C[TC_H] + 0.0f * C[TC_R1];  // (in the geometry; undefined if R1 is)
        case FK_BETA: return C[TC_BETA];
        case FK_EN: return C[TC_EN];
        case FK_MHON: return C[TC_MHON];
        case FK_MHONL: return C[TC_MHONL];
        default: {
          constexpr int from[8] = {TC_R0, TC_LA, TC_CA, TC_LR, TC_CR, TC_LAL, TC_CAL, TC_LRL};
          const int q = (k - FK_R0) >> 1, s = (k - FK_R0) & 1;
          return C[(q < 8 ? from[q] : TC_CRL) + s];
        }
      }
    };
    tab[t] = pack(value(0), value(1));
  }
  __syncthreads();
  const ForceConsts<NT, LO> K{tab + h, H};
  const float4* gu = v.gu + base;
  const float4* gd = v.gd + base;
  f2* rec = scratch + 3 * h;
  for (int il = warp * A + aslot; il < Na; il += warps * A) {
    if (il < n_inner) atom_forces<NT, LO, true>(K, gu, gd, Na, il, rec, lgH);
    else atom_forces<NT, LO, false>(K, gu, gd, Na, il, rec, lgH);
  }
  __syncthreads();
  const int* rev = v.rev + base;
  const double* ref = v.ref + (size_t)3 * (base / 4);
  double e0 = 0.0, e1 = 0.0;
  const f2 m1 = dup(-1.0f);
  for (int il = warp * A + aslot; il < Na; il += warps * A) {
    int rl[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) rl[j] = __ldg(rev + j * Na + il);
    f2 F[3] = {0, 0, 0};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const f2* a = rec + 3 * ((size_t)(j * Na + il) << lgH);
      const f2* b = rec + 3 * ((size_t)rl[j] << lgH);
#pragma unroll
      for (int k = 0; k < 3; ++k) F[k] = add2(F[k], fma2(b[k], m1, a[k]));
    }
    float2 f[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f[k] = unpack(F[k]);
      const double r = __ldg(ref + 3 * il + k), d0 = (double)f[k].x - r, d1 = (double)f[k].y - r;
      e0 = __fma_rn(d0, d0, e0);
      e1 = __fma_rn(d1, d1, e1);
    }
    if (J.fdump) {
      const int i = v.atom[base / 4 + il], Nf = J.v.N_force, p = it.p0 + 2 * h;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (p < P) J.fdump[((size_t)p * 3 + k) * Nf + i] = f[k].x;
        if (p + 1 < P) J.fdump[((size_t)(p + 1) * 3 + k) * Nf + i] = f[k].y;
      }
    }
  }
  __syncthreads();  // every f_ij has been read
  double* red = reinterpret_cast<double*>(smem);  // [half][thread]
  red[threadIdx.x] = e0;
  red[blockDim.x + threadIdx.x] = e1;
  __syncthreads();
  if (warp < 2) {
    double s = 0.0;
    for (int x = 0; x < warps; ++x) s += red[warp * blockDim.x + x * 32 + lane];
    for (int o = H; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const int p = it.p0 + 2 * lane + warp;
    if (lane < H && p < P) J.res[((size_t)p * J.v.Nc + c) * kResK + 7] = s;
  }
  finish_item(jobs, it, 2 * H);
}

constexpr size_t kForceSmem = 52 * 1024;      // four CTAs per SM
constexpr size_t kForceSmemMax = 200 * 1024;  // one: still better than 32 individuals with their scratch in global memory

size_t force_smem(int Na, int H) {
  return std::max((size_t)FK_COUNT * 16 * 8 + (size_t)4 * Na * H * 24, sizeof(double) * 2 * kFThreadsLarge);
}

}  // namespace

// log2 of the pairs of individuals per item for a configuration of Na atoms (-1: too large for shared memory): the
// largest of 16, 8, 4, 2, 1 whose scratch leaves room for four CTAs per SM, or one pair in a CTA of twice the threads (two
// CTAs per SM: 16 warps again).
int tersoff_force_lgH(int Na) {
  for (int l = 4; l >= 0; --l)
    if (force_smem(Na, 1 << l) <= kForceSmem) return l;
  return force_smem(Na, 1) <= kForceSmemMax ? 0 : -1;
}
bool tersoff_force_large(int Na) { return force_smem(Na, 1) > kForceSmem; }
size_t tersoff_force_smem(int Na) { return force_smem(Na, 1 << tersoff_force_lgH(Na)); }

int tersoff_force_build(Engine* e) {
  DevSet& d = e->d;
  const TrainingSet& ts = e->ts;
  const PotentialSpec& sp = e->spec;
  e->h_tf.assign(ts.Nc, 0);
  if ((d.potential_type != 1 && d.potential_type != 2) || ts.N_force == 0 || d.B == 0) return GPUGA_OK;
  const int off = d.num_types == 2 ? 4 : 0;
  if ((int)sp.pmin.size() < 9 + off) return GPUGA_OK;
  const float r1 = sp.pmin[7 + off], r2 = sp.pmin[8 + off];
  if (sp.pmax[7 + off] != r1 || sp.pmax[8 + off] != r2 || !(r1 < r2)) return GPUGA_OK;
  cudaStream_t st = e->stream;
  const int n = ts.N_force;
  signed char* d_rank = nullptr;
  int *d_kind = nullptr, *d_place = nullptr;
  int2* d_where = nullptr;
  auto run = [&]() -> int {
    GPUGA_CUDA(cudaMalloc(&d_rank, (size_t)d.B));
    GPUGA_CUDA(cudaMalloc(&d_kind, sizeof(int) * n));
    GPUGA_CUDA(cudaMalloc(&d_place, sizeof(int) * n));
    GPUGA_CUDA(cudaMalloc(&d_where, sizeof(int2) * n));
    force_ranks<<<(n + 127) / 128, 128, 0, st>>>(n, d.off, d.nbr, d.rev, d.g64, r1, r2, d_rank, d_kind);
    GPUGA_CUDA(cudaGetLastError());
    std::vector<int> kind(n), place(n), base(ts.Nc, 0), inner(ts.Nc, 0), lgH(ts.Nc, 0), atom;
    std::vector<int2> where(n, make_int2(-1, 0));
    GPUGA_CUDA(cudaMemcpyAsync(kind.data(), d_kind, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    GPUGA_CUDA(cudaStreamSynchronize(st));
    for (int c = 0; c < ts.Nc_force; ++c) {
      const int a0 = ts.Na_sum[c], Na = ts.Na[c], l = tersoff_force_lgH(Na);
      bool ok = l >= 0;
      for (int k = 0; k < Na; ++k) ok &= kind[a0 + k] >= 0;
      if (!ok) continue;
      base[c] = 4 * (int)atom.size();
      lgH[c] = l;
      for (int pass = 1; pass >= 0; --pass)
        for (int k = 0; k < Na; ++k)
          if (kind[a0 + k] == pass) {
            place[a0 + k] = (int)atom.size() - base[c] / 4;
            where[a0 + k] = make_int2(base[c], Na);
            atom.push_back(a0 + k);
            inner[c] += pass;
          }
      e->h_tf[c] = 1;
    }
    if (atom.empty()) return GPUGA_OK;
    const size_t slots = 4 * atom.size();
    TersoffForceView v{};
    float4 *gu = nullptr, *gd = nullptr;
    int *rev = nullptr, *d_base = nullptr, *d_inner = nullptr, *d_lgH = nullptr, *d_atom = nullptr;
    double* ref = nullptr;
    GPUGA_TRY(e->alloc(&gu, slots));
    GPUGA_TRY(e->alloc(&gd, slots));
    GPUGA_TRY(e->alloc(&rev, slots));
    GPUGA_TRY(e->alloc(&ref, 3 * atom.size()));
    GPUGA_TRY(e->alloc(&d_base, (size_t)ts.Nc));
    GPUGA_TRY(e->alloc(&d_inner, (size_t)ts.Nc));
    GPUGA_TRY(e->alloc(&d_lgH, (size_t)ts.Nc));
    GPUGA_TRY(e->alloc(&d_atom, atom.size()));
    GPUGA_CUDA(cudaMemcpyAsync(d_base, base.data(), sizeof(int) * ts.Nc, cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_inner, inner.data(), sizeof(int) * ts.Nc, cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_lgH, lgH.data(), sizeof(int) * ts.Nc, cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_atom, atom.data(), sizeof(int) * atom.size(), cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_place, place.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st));
    GPUGA_CUDA(cudaMemcpyAsync(d_where, where.data(), sizeof(int2) * n, cudaMemcpyHostToDevice, st));
    force_geometry<<<(n + 127) / 128, 128, 0, st>>>(n, d.off, d.nbr, d.rev, d.ptype, d.g64, r1, r2, d_rank, d_place, d_where,
                                                    d.force_ref, ts.N, gu, gd, rev, ref);
    GPUGA_CUDA(cudaGetLastError());
    GPUGA_CUDA(cudaStreamSynchronize(st));
    v.gu = gu;
    v.gd = gd;
    v.rev = rev;
    v.ref = ref;
    v.base = d_base;
    v.inner = d_inner;
    v.lgH = d_lgH;
    v.atom = d_atom;
    d.tf = v;
    return GPUGA_OK;
  };
  const int s = run();
  cudaFree(d_rank);
  cudaFree(d_kind);
  cudaFree(d_place);
  cudaFree(d_where);
  return s;
}

template <int NT, bool LO>
static int force_launch(const JobView* jobs, const WorkItem* items, int count, size_t smem, bool configure, cudaStream_t st) {
  if (configure) {
    GPUGA_CUDA(cudaFuncSetAttribute(tersoff_force<NT, LO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kForceSmemMax));
    return GPUGA_OK;
  }
  // items of the two kinds are in launches of their own
  tersoff_force<NT, LO><<<count, smem <= kForceSmem ? kFThreads : kFThreadsLarge, smem, st>>>(jobs, items);
  GPUGA_CUDA(cudaGetLastError());
  return GPUGA_OK;
}

int tersoff_force_launch(const JobView* jobs, const WorkItem* items, int count, size_t smem, int num_types, bool lo,
                         bool configure, cudaStream_t st) {
  if (num_types == 2)
    return lo ? force_launch<2, true>(jobs, items, count, smem, configure, st)
              : force_launch<2, false>(jobs, items, count, smem, configure, st);
  return lo ? force_launch<1, true>(jobs, items, count, smem, configure, st)
            : force_launch<1, false>(jobs, items, count, smem, configure, st);
}

}  // namespace gpuga
