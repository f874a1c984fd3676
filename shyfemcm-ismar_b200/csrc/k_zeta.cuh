// k_zeta.cuh -- the zeta system: system_init + the element scatter of system_assemble + system_add_rhs
// (simsys_spkaux.f90:137-154, 533-594, 687-705) as an atomic-free gather in
// element order (FP64 sums, as the reference's c2coo), then system_solve
// (sparskit_admin.f90:115-334): Krylov iterations in FP32 inside FP64
// residual refinement, stopped on the reference's test
// ||r|| <= rtol*||r0|| + atol (stopbis, spk_iters.f90:3304-3360), with r0 the
// residual of the reference's guess (the old water level).
//
// This file holds the helpers the solvers share; k_zeta_team.cuh keeps every
// basin resident on chip, k_zeta_grid.cuh streams basins too large for that,
// k_zeta_global.cuh works one cluster per basin with vectors in global memory.
// Included by step_zeta.cu.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "launch.h"
#include "physics.cuh"

namespace cg = cooperative_groups;

namespace shy {

// Sum of NV values over all threads of a cluster.  Fixed reduction order
// (warp shuffles, then warps, then cluster ranks in a shuffle tree), so every
// CTA obtains the same bits.  Uses one cluster barrier.
template <int NV>
__device__ __forceinline__ void cluster_sum(cg::cluster_group &cl, double (&v)[NV], double *wbuf,
                                            double *slots, double *bc, int &par, int CL) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; i++) {
    double x = v[i];
#pragma unroll
    for (int dd = 16; dd > 0; dd >>= 1) x += __shfl_xor_sync(0xffffffffu, x, dd);
    if (lane == 0) wbuf[i * 32 + warp] = x;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      double x = lane < nw ? wbuf[i * 32 + lane] : 0.;
#pragma unroll
      for (int dd = 16; dd > 0; dd >>= 1) x += __shfl_xor_sync(0xffffffffu, x, dd);
      if (lane == 0) slots[par * 4 + i] = x;
    }
  }
  cl.sync();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < NV; i++) {
      double x = lane < CL ? *cl.map_shared_rank(&slots[par * 4 + i], lane) : 0.;
#pragma unroll
      for (int dd = 16; dd > 0; dd >>= 1) x += __shfl_xor_sync(0xffffffffu, x, dd);
      if (lane == 0) bc[i] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; i++) v[i] = bc[i];
  par ^= 1;
}

// the fraction of the outer target the FP32 inner solve goes down to
__device__ __forceinline__ double tfrac(const ZetaArgs &za) {
  return za.tol_frac > 0.f ? (double)za.tol_frac : 0.25;
}

// one row of the assembly: FP64 gather of the element entries of every slot
// (element order), the rhs, the diagonal
__device__ __forceinline__ void assemble_row(const Dev &d, const ZetaArgs &za, int i, float dtf,
                                             double &diag, double &rhs, bool wd = false, bool w32 = true) {
  diag = 0.;
  for (int s = d.rowptr[i]; s < d.rowptr[i + 1]; s++) {
    double v = 0.;
    for (int t = d.slot_ptr[s]; t < d.slot_ptr[s + 1]; t++) {
      const int src = d.slot_src[t];
      const int e = src / 9, c = src - 9 * e;
      const float *ph = &za.hia[(size_t)c * za.cs + (size_t)e * za.es];
      v += (double)(wd ? __ldcg(ph) : *ph);      // dry systems are written in this launch
    }
    d.val64[s] = v;
    if (w32) d.val32[s] = (float)v;            // the FP32 copy the cluster solvers iterate on
    if (d.col[s] == i) diag = v;
  }
  rhs = 0.;
  for (int p = d.inc_ptr[i]; p < d.inc_ptr[i + 1]; p++) {
    const int q = d.inc[p];
    const int e = q / 3, ii = q - 3 * e;
    const float *pk = &za.hik[(size_t)ii * za.cs + (size_t)e * za.es];
    rhs += (double)(wd ? __ldcg(pk) : *pk);
  }
  // adjust_mass_flux (bnd_routines.f90:1185-1210): with wetting and drying
  // (wd) no flux enters a node out of the system
  if (!(wd && d.inod[i] == -2)) rhs += (double)(dtf * d.rqv[i]);
  d.rhs64[i] = rhs;
}

}  // namespace shy
