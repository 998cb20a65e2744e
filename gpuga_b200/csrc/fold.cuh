// The fitness of an individual from its configurations' results, shared by the kernels that may
// finish an individual (batched.cu, spectral.cu).
#pragma once
#include "engine.hpp"

namespace gpuga {

// fitness.cu:329-331, 437-555 in FP64 for individual p, by 32 lanes: lane c sums configurations
// c, c + 32, ... in order (fold_sums), then a butterfly (fold_result, a warp); the same order whichever warp or
// launch folds, and the same operations: every product and sum is an explicit intrinsic, so that the compiler's
// choice of contracting a * b + c into an FMA cannot differ between the kernels this is inlined in.
// Reads go through L2 (ld.cg): other CTAs of the same launch wrote the results.
__device__ __forceinline__ void fold_sums(const JobView& J, int p, int lane, double& eE, double& eW, double& eF) {
  const int Nc = J.v.Nc, Nc_force = J.Nc_force;
  const double* res = J.res;
  // force errors of an individual that the pair expansion evaluated (spectral.cu)
  const bool expanded = J.sp.part && !__ldcg(J.sp.flagged + p);
  const double* __restrict__ E_ref = J.E_ref;
  const double* __restrict__ W_ref = J.W_ref;
  eE = eW = eF = 0;
  if (expanded) {
    // the items' sums: force configurations, then the energies and the virials per energy/virial item
    const double* part = J.sp.part + p;
    const int nf = Nc_force, ne = (J.sp.n_part - nf) / 2;
    for (int k = lane; k < nf; k += 32) eF += __ldcg(part + (size_t)k * J.Pstride);
    for (int k = lane; k < ne; k += 32) {
      eE += __ldcg(part + (size_t)(nf + k) * J.Pstride);
      eW += __ldcg(part + (size_t)(nf + ne + k) * J.Pstride);
    }
  }
  for (int c = expanded ? Nc : lane; c < Nc; c += 32) {
    const double* r = res + ((size_t)p * Nc + c) * kResK;
    if (c >= Nc_force && J.ev.pairs && J.ev.seg0[c + 1] > J.ev.seg0[c]) {
      // a configuration in several segments: their sums in order are its results
      double v[7];
#pragma unroll
      for (int k = 0; k < 7; ++k) v[k] = 0.0;
      for (int s = J.ev.seg0[c]; s < J.ev.seg0[c + 1]; ++s)
#pragma unroll
        for (int k = 0; k < 7; ++k) v[k] += __ldcg(J.ev.part + ((size_t)s * 7 + k) * J.Pstride + p);
      double* w = J.res + ((size_t)p * Nc + c) * kResK;
#pragma unroll
      for (int k = 0; k < 6; k += 2) *reinterpret_cast<double2*>(w + k) = double2{v[k], v[k + 1]};
      w[6] = v[6];
      const double de = v[0] - E_ref[c];
      eE = __fma_rn(de, de, eE);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double dw = v[1 + k] - W_ref[c + (size_t)Nc * k];
        eW = __fma_rn(dw, dw, eW);
      }
    } else if (c >= Nc_force) {
      const double de = __ldcg(r) - E_ref[c];
      eE = __fma_rn(de, de, eE);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const double dw = __ldcg(r + 1 + k) - W_ref[c + (size_t)Nc * k];
        eW = __fma_rn(dw, dw, eW);
      }
    } else {
      eF += __ldcg(r + 7);
    }
  }
}

// The fitness of individual p from its lanes' sums, by a warp.
__device__ __forceinline__ void fold_result(const JobView& J, int p, int lane, double eE, double eW, double eF) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    eE += __shfl_xor_sync(0xffffffffu, eE, o);
    eW += __shfl_xor_sync(0xffffffffu, eW, o);
    eF += __shfl_xor_sync(0xffffffffu, eF, o);
  }
  if (lane == 0) {
    const double rE = sqrt(eE / J.nE), rW = sqrt(eW / J.nW), rF = sqrt(eF / J.nF);
    J.fitness[p] = __dadd_rn(__dadd_rn(__dmul_rn((double)J.wE, rE), __dmul_rn((double)J.wW, rW)),
                             __dmul_rn((double)J.wF, rF));
    if (J.comps) {
      J.comps[3 * (size_t)p + 0] = rE;
      J.comps[3 * (size_t)p + 1] = rW;
      J.comps[3 * (size_t)p + 2] = rF;
    }
  }
}

__device__ __forceinline__ void fold_fitness(const JobView& J, int p, int lane) {
  double eE, eW, eF;
  fold_sums(J, p, lane, eE, eW, eF);
  fold_result(J, p, lane, eE, eW, eF);
}

// End of every work item: its results for individuals p0 .. p0 + G - 1 are written.  Each of those
// individuals' completion count goes up by one with a release-acquire atomic (the CTA barrier
// orders every thread's writes before it, and release is cumulative); the item that brings an individual to Nc
// configurations folds its fitness and resets the count for the next generation.  Nothing waits.
// Release-acquire increment at device scope: releases the CTA's writes ordered before it (by the
// preceding CTA barrier) and acquires the writes released by earlier increments.
__device__ __forceinline__ int atomic_add_acq_rel(int* a, int v) {
  int old;
  asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(a), "r"(v) : "memory");
  return old;
}

// p: the individual of this thread (threads 0 .. G - 1 of the CTA; -1: none).
__device__ __forceinline__ void finish_individuals(const JobView& J, int p, int G) {
  if (!J.fit_count) return;
  __shared__ int s_last[32];
  __syncthreads();
  if (threadIdx.x < 32) {
    int last = -1;
    if (threadIdx.x < G && p >= 0) {
      // items that count for p: one per configuration, or the expansion's items and, for an
      // individual that it handed to the direct items, theirs as well
      const int total = J.sp.part ? J.sp.n_items + (__ldcg(J.sp.flagged + p) ? J.v.Nc : 0)
                                  : (J.ev.pairs ? J.Nc_force + J.ev.n_items : J.v.Nc);
      if (atomic_add_acq_rel(&J.fit_count[p], 1) == total - 1) last = p;
    }
    s_last[threadIdx.x] = last;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int g = threadIdx.x >> 5; g < G; g += blockDim.x >> 5) {
    const int q = s_last[g];
    if (q < 0) continue;  // warp-uniform
    __threadfence();
    fold_fitness(J, q, lane);
    if (lane == 0) {
      J.fit_count[q] = 0;
      // the job's last individual: an empty list of direct individuals for the next generation
      if (J.sp.count && atomicAdd(J.sp.count + 1, 1) == J.P - 1) J.sp.count[0] = J.sp.count[1] = 0;
    }
  }
}

__device__ __forceinline__ void finish_item(const JobView* __restrict__ jobs, const WorkItem& it, int G) {
  const JobView& J = jobs[it.job];
  const int p = it.p0 + (int)threadIdx.x;
  finish_individuals(J, threadIdx.x < G && p < J.P ? p : -1, G);
}

}  // namespace gpuga
