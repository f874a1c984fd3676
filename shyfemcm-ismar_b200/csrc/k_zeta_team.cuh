// k_zeta_team.cuh -- zeta assembly + solve with every basin resident on chip:
// the basin's rows are dealt to a team of CTAs that keep their share of the
// scaled matrix in registers and the Krylov vectors in registers and shared
// memory for the whole solve.  One cooperative launch works all basins of a
// model; a CTA takes its shares of several basins one after another.
//
// The solver is system_init + system_assemble + system_add_rhs + system_solve
// (simsys_spkaux.f90:137-154, 454-491, 533-594, 687-705; stop test
// ||r|| <= rtol*||r0|| + atol of spk_iters.f90:3304-3360): FP64 assembly in
// element order and FP64 residual refinement around Chronopoulos-Gear CG in
// FP32 on the Jacobi-scaled system S A S (S = D^-1/2), from the extrapolated
// level 2 z^n - z^(n-1).
//
// What bounds it.  An iteration of a streaming solver moves 88 bytes a row
// through L2 and HBM and ends in a grid barrier; with the rows resident only
// the product of a row at a share's border (its "ghost" copies in other
// CTAs) and three sums per CTA leave the chip, so an iteration costs the
// latency of one exchange through L2 plus the shared-memory gathers of the
// rows (8 per row).  Shares are compact patches of the mesh (the host
// bisects the nodes by coordinates), so a share of 1024 rows has about 140
// ghosts where a run of consecutive nodes would have twice the mesh's width.
//
// Exchange without barriers.  Each 8-byte word that crosses CTAs carries its
// value and the number of the exchange it belongs to; the reader polls the
// word itself until the number matches, so neither a flag nor a fence nor a
// barrier sits between a value and its use.  Ghost rows are replicated: the
// reader applies the vector updates to its copies and receives only the
// matrix product (w) of the owner.  A CTA can write exchange k+1 only after
// every member of its team has published exchange k, which each does after
// reading exchange k-1: two buffers in turn suffice (the first exchange
// uses three others).  Every wait is bounded; one that runs out sets the
// abort word, marks the basins SHY_ECUDA and all CTAs leave.  The number of
// an exchange is the launch's (16 bits) and its place in the launch (16
// bits).  A share's first exchange of a launch writes all its words, those
// that only later exchanges carry included, so an old word never has a
// number that is waited for: only 65536 launches in a row that were aborted
// before they reached the share would bring it back.
//
// Measured (a solve, CUDA events; before: shared-memory clusters up to 40k
// rows, the streaming solver above): 793 rows 52 iterations 268 -> 100 us,
// 7k rows 122 iterations 615 -> 293 us, 20k rows 636 -> 355 us, 90k rows
// 1156 -> 518 us, 250k rows 1139 -> 390 us, the 64-basin ensemble (2.1M rows)
// 5.05 -> 2.65 ms; BiCGStab, 12k rows with Coriolis, 55 iterations 2.65 ->
// 0.34 ms; the non-hydrostatic pressure (18k rows) 60 -> 7 us an iteration.  What is left of an iteration (2 to 4 us) is a chain of
// latencies: the gathers 0.5 us, the sums in the CTA and the FP64 scalars
// 0.6 us, one exchange through L2 0.5 us for a few members, 1 us for many.
//
// The shares and the order of every sum depend on the basin alone, so a
// basin gives the same bits alone and in any batch.
// Included by step_zeta.cu.
#pragma once
#include "k_zeta.cuh"

namespace shy {

typedef unsigned long long u64;

__device__ __forceinline__ u64 ld_relaxed_u64(const u64 *p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(u64 *p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned *p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// one word of an exchange: value in the low half, exchange number in the high
__device__ __forceinline__ void word_put(u64 *p, unsigned v, unsigned ep) {
  st_relaxed_u64(p, ((u64)ep << 32) | v);
}

// bounded wait for exchange ep of N words, all polled together; false when
// one did not come
template <int N>
__device__ __forceinline__ bool words_wait(const TeamPlan &tp, const u64 *const (&p)[N], unsigned ep, unsigned abortv,
                                           unsigned (&v)[N]) {
  long long spins = 0;
  for (;;) {
    bool all = true;
    u64 w[N];
#pragma unroll
    for (int k = 0; k < N; k++) w[k] = ld_relaxed_u64(p[k]);
#pragma unroll
    for (int k = 0; k < N; k++) {
      v[k] = (unsigned)w[k];
      all &= (unsigned)(w[k] >> 32) == ep;
    }
    if (all) return true;
    if ((++spins & 63) == 0 && (spins > tp.spin_limit || ld_relaxed_u32(tp.ctr) == abortv)) {
      atomicExch(tp.ctr, abortv);
      return false;
    }
  }
}

// shared memory of a CTA: NT threads, R rows and GR ghosts a thread
template <int NT, int R, int GR>
struct TeamShared {
  float u[NT * R + NT * GR];       // the product's input: own rows, from NT * R on the ghosts
  float sd[NT * R + NT * GR];      // Jacobi scale D^-1/2
  double x[NT * R + NT * GR];      // the FP64 iterate
  double wred[6][NT / 32];         // sums of the warps
  double tot[4];                   // sums of the team
  double tsum[6][NT / 32];         // its members', a warp's worth each
  double resid0, tol, rn, rn2, rs2;   // ||r0||, the target, ||r||, ||r||^2, ||S r||^2
  double itol2;                    // an FP32 sweep's target for ||S r||^2
  double rgamma, ralpha;           // 1 / gamma, 1 / alpha of the last update
  double rho, alpha;               // BiCGStab's (rh, r) and alpha
  float fa, fb, fo;                // alpha, beta, omega of the next update
  int stop, ok;
  TeamMember M;
};

// the sum of a over the warp in lanes 0-15, that of b in lanes 16-31
__device__ __forceinline__ double warp_sum2(double a, double b) {
  const bool lo = (threadIdx.x & 16) == 0;
  double x = (lo ? a : b) + __shfl_xor_sync(0xffffffffu, lo ? b : a, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// both sums in every lane, from warp_sum2's halves
__device__ __forceinline__ void both_sums(double x, double &a, double &b) {
  const bool lo = (threadIdx.x & 16) == 0;
  const double y = __shfl_xor_sync(0xffffffffu, x, 16);
  a = lo ? x : y;
  b = lo ? y : x;
}

// slot of a member's sums (down 0) or of the totals sent to it (down 1)
__device__ __forceinline__ u64 *team_slot(const TeamPlan &tp, unsigned xi, int down, int slot) {
  return tp.part + (((size_t)(xi & 1u) * 2 + down) * tp.nslot + slot) * kTeamSlotWords;
}

constexpr int kTeamSums = 12;        // words of the widest exchange (three pairs)
static_assert(kTeamSums <= kTeamSlotWords, "a slot holds them");

// word k of a slot that holds the 2 NP sums x (every lane has them all) as
// low and high halves.  The first exchange of a launch renews both buffers'
// words up to kTeamSums, whatever the exchanges that follow carry.
template <int NP>
__device__ __forceinline__ void sums_put(const TeamPlan &tp, unsigned xi, int down, int slot, const double (&x)[2 * NP],
                                         unsigned ep, int k) {
  double v = x[0];
#pragma unroll
  for (int c = 1; c < 2 * NP; c++) v = k >> 1 == c ? x[c] : v;
  const unsigned h = (k & 1) ? (unsigned)__double2hiint(v) : (unsigned)__double2loint(v);
  word_put(team_slot(tp, xi, down, slot) + k, h, ep);
  if (xi == 0u) word_put(team_slot(tp, 1u, down, slot) + k, h, ep);
}

template <int NP>
__device__ __forceinline__ bool sums_wait(const TeamPlan &tp, const u64 *p, unsigned ep, unsigned abortv,
                                          double (&x)[2 * NP]) {
  const u64 *pw[4 * NP];
  unsigned h[4 * NP];
#pragma unroll
  for (int k = 0; k < 4 * NP; k++) pw[k] = p + k;
  const bool ok = words_wait(tp, pw, ep, abortv, h);
#pragma unroll
  for (int c = 0; c < 2 * NP; c++) x[c] = __hiloint2double((int)h[2 * c + 1], (int)h[2 * c]);
  return ok;
}

// the sums of members t0 .. t0+31 of the team, added up, in every lane
template <int NP>
__device__ __forceinline__ bool poll_sums(const TeamPlan &tp, const TeamMember &M, int T, int t0, unsigned ep,
                                          unsigned xi, unsigned abortv, double (&tot)[2 * NP]) {
  const int t = t0 + (int)(threadIdx.x & 31);
  bool ok = true;
#pragma unroll
  for (int c = 0; c < 2 * NP; c++) tot[c] = 0.;
  if (t < T)                                       // the phantom's slot is never written
    ok = sums_wait<NP>(tp, team_slot(tp, xi, 0, t < M.T ? M.slot0 + t : tp.nslot - 1), ep, abortv, tot);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < NP; c++) both_sums(warp_sum2(tot[2 * c], tot[2 * c + 1]), tot[2 * c], tot[2 * c + 1]);
  return __all_sync(0xffffffffu, ok) != 0;
}

// The sums of an exchange, after a CTA barrier that follows the warps' sums
// in sh.wred; warp 0 receives the 2 NP totals in every lane.  Up to
// kTeamAllToAll members read each other's sums (one hop through L2, 0.5 us);
// in a wider team, whose T^2 reads would cost more than a second hop, member
// 0 reads them all and writes the totals to a slot of each member.  More
// than 32 slots are polled by several warps.  Words are read and written one
// by one: with 16-byte accesses an exchange took 0.5 to 1.5 us longer.
// Called by the whole CTA.
template <int NP, int NT, class SH>
__device__ __forceinline__ bool team_totals(SH &sh, const TeamPlan &tp, const TeamMember &M, unsigned ep, unsigned xi,
                                            unsigned abortv, double (&tot)[2 * NP]) {
  static_assert(NT <= 512, "a half warp sums the warps");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int T = M.T + tp.phantom;
  if (warp == 0) {                                 // the CTA's sums from its warps', in a fixed tree
#pragma unroll
    for (int c = 0; c < NP; c++) {
      double x = (lane & 15) < NT / 32 ? sh.wred[2 * c + (lane >> 4)][lane & 15] : 0.;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      both_sums(x, tot[2 * c], tot[2 * c + 1]);
    }
    if (T > 1 && lane < (xi == 0u ? kTeamSums : 4 * NP)) sums_put<NP>(tp, xi, 0, M.slot0 + M.rank, tot, ep, lane);
  }
  if (T == 1) return true;
  // nobody polls before warp 0 has published: the polls would queue ahead of its stores
  if (warp == 0) asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");
  else asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
  const bool all = T <= kTeamAllToAll;
  bool ok = true;
  if (all || M.rank == 0) {
    if (warp * 32 < T) {
      ok = poll_sums<NP>(tp, M, T, warp * 32, ep, xi, abortv, tot);
      if (T > 32 && lane == 0)
#pragma unroll
        for (int c = 0; c < 2 * NP; c++) sh.tsum[c][warp] = tot[c];
    }
    if (T > 32) {                                  // uniform in the CTA
      if (!ok) sh.ok = 0;
      __syncthreads();
      if (warp == 0) {
        const int nw = (T + 31) / 32;
        for (int w = 1; w < nw; w++)
#pragma unroll
          for (int c = 0; c < 2 * NP; c++) tot[c] += sh.tsum[c][w];
        if (!all && sh.ok) {                       // not the sums of a poll that ran out
          if (xi == 0u)
            for (int k = lane; k < kTeamSums * M.T; k += 32)
              sums_put<NP>(tp, xi, 1, M.slot0 + k / kTeamSums, tot, ep, k % kTeamSums);
          else
            for (int k = lane; k < 4 * NP * M.T; k += 32)
              sums_put<NP>(tp, xi, 1, M.slot0 + k / (4 * NP), tot, ep, k % (4 * NP));
        }
      }
    }
  } else if (warp == 0) {
    ok = sums_wait<NP>(tp, team_slot(tp, xi, 1, M.slot0 + M.rank), ep, abortv, tot);
  }
  return ok;
}

// entry k of a packed pair of columns, kept as byte offsets into a float array
__device__ __forceinline__ float at4(const float *a, unsigned pair, int k) {
  return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(a) + (k & 1 ? pair >> 16 : pair & 0xffffu));
}

// buffer of exchange number xi >= 1 (0 uses buffers 0, 2 and 3)
__device__ __forceinline__ u64 *team_buf(const TeamPlan &tp, unsigned xi) {
  return tp.word + (size_t)(xi & 1u) * tp.nrow;
}

// SYM: CG on the symmetrically scaled system S A S; else BiCGStab (van der
// Vorst 1992) on A D^-1 (right Jacobi preconditioning), for systems with
// Coriolis or dry elements, and the repeat loop of wetting and drying
// (hydrodynamic.f90:374-404).  Both scaled matrices have a unit diagonal.
// K: off-diagonal entries in a row's block.  CSR: not the zeta system but one
// given in CSR form (TeamPlan::csr), from a zero guess: the 3D pressure.
template <int NT, int R, int GR, int K, bool SYM, bool CSR>
__global__ void __launch_bounds__(NT, 1) k_zeta_team(Dev d, ZetaArgs za, TeamPlan tp) {
  static_assert(!(SYM && CSR), "the 3D system is not symmetric");
  typedef TeamShared<NT, R, GR> SH;
  __shared__ SH sh;
  const int tid = threadIdx.x;
  const int q0 = tp.cptr[blockIdx.x], q1 = tp.cptr[blockIdx.x + 1];
  // the launch's number, the same in every CTA: the high half of its exchange
  // numbers, and the abort word
  const unsigned launch = tp.cta_cnt[blockIdx.x] + 1u, abortv = launch;
  bool dead = false;
  if (tid == 0) sh.ok = 1;
  if (!CSR && blockIdx.x == 0 && tid == 0 && d.imax) { *d.imax = 0; *d.subj = 0; }

  for (int q = q0; q < q1; q++) {
    const int me = tp.clist[q];
    if (tid == 0) sh.M = tp.mem[me];
    __syncthreads();
    const TeamMember &M = sh.M;
    const BasinPar &P = d.par[M.basin];
    BasinOut &O = d.out[M.basin];
    unsigned xi = 0u;                            // exchanges of this solve
    auto number = [&] { return (launch << 16) | (xi & 0xffffu); };
    const int n = M.nrow, nr = (n + NT - 1) / NT;   // rows, rows a thread at most
    const int echunk = (P.ne + M.T - 1) / M.T;   // this member's elements (wetting and drying)
    const int ea = P.e0 + min(P.ne, M.rank * echunk), eb = min(P.e0 + P.ne, ea + echunk);
    if (!CSR && M.rank == 0 && tid < kMaxScal) O.stab[tid] = 0.f;   // reset for k_stab's max
    const float dtf = (float)P.dt;
    // wetting and drying: a domain that can change with the solution
    const bool wd = !SYM && !CSR && wd_basin(P);
    const bool extrap = !CSR && za.zprev != nullptr && O.steps > 0 && !wd;
    // a barrier of the team that also makes its global writes visible; sums
    // one value
    auto team_barrier = [&](double &v) -> bool {
      __threadfence();
      const double y = warp_sum2(v, 0.);
      if ((tid & 15) == 0) sh.wred[(tid >> 4) & 1][tid >> 5] = y;
      __syncthreads();
      double tot[2];
      const bool k = team_totals<1, NT>(sh, tp, M, number(), xi, abortv, tot);
      if (tid == 0) sh.tot[0] = tot[0];
      if (!k) sh.ok = 0;
      __syncthreads();
      __threadfence();
      xi++;
      v = sh.tot[0];
      return sh.ok != 0;
    };
    int iters = 0, outer = 0, refine = 0;
    for (int rep = 0;; rep++) {
    if (wd) {
      bool fine = true;
      double none = 0.;
      for (int j = tid; j < n; j += NT) fine &= wd_setnod(d, tp.rows[M.row0 + j] & 0x7fffffff);
      if (!fine) set_status(&O, SHY_EDEPTH);     // the open boundary dried (setnod :245)
      if (!team_barrier(none)) { dead = true; break; }
      for (int e = ea + tid; e < eb; e += NT)
        if (__ldcg(&d.iweg[e]) != 0) wd_dry_system(d, e);
      if (!team_barrier(none)) { dead = true; break; }
    }
    // the guess: the old level, in repeats the last solution
    const float *guess = rep == 0 ? za.zguess : d.zn;
    const int *rowptr = CSR ? tp.csr.rowptr : d.rowptr;
    double *val64 = CSR ? const_cast<double *>(tp.csr.val) : d.val64;
    const double *rhs64 = CSR ? tp.csr.rhs : d.rhs64;
    auto level = [&](int i) { return (double)(wd ? __ldcg(guess + i) : guess[i]); };

    // ---- assembly (FP64 sums in element order), Jacobi scale, and the
    // residuals of both starts, the old level's (the stop test's r0) and the
    // extrapolated one's ----
    auto elem = [&](const float *a, int c, int e) {   // dry systems are written in this launch
      const float *q = a + (size_t)c * za.cs + (size_t)e * za.es;
      return wd ? __ldcg(q) : *q;
    };
    int ri[R];                                   // global row, sign bit: published
    float rsA[R], rsB[R];
    double v4[4] = {0., 0., 0., 0.};
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int j = r * NT + tid;
      ri[r] = 0; rsA[r] = rsB[r] = 0.f;
      sh.sd[j] = 0.f;
      sh.u[j] = 0.f;
      if (j >= n) continue;
      ri[r] = tp.rows[M.row0 + j];
      const int i = ri[r] & 0x7fffffff;
      double diag = 0., tA, tB = 0.;
      if constexpr (CSR) {
        diag = val64[rowptr[i] + dpos_place(tp.dpos[M.row0 + j])];
        tA = rhs64[i];                           // the guess is zero
      } else {
        const int s0 = d.rowptr[i];
        const int dn = tp.dpos[M.row0 + j], dp = dpos_place(dn), nd = dpos_count(dn);   // diagonal's place, off-diagonal entries
        double rhs = 0.;
        const int p1 = d.inc_ptr[i + 1];
        for (int p0 = d.inc_ptr[i]; p0 < p1; p0 += 8) {   // eight elements at a time, their loads in flight together
          float ha[8], hb[8];
#pragma unroll
          for (int k = 0; k < 8; k++) {
            const bool in = p0 + k < p1;
            const int e3 = in ? d.inc[p0 + k] : 0, e = e3 / 3, ii = e3 - 3 * e;
            ha[k] = in ? elem(za.hia, 4 * ii, e) : 0.f;
            hb[k] = in ? elem(za.hik, ii, e) : 0.f;
          }
#pragma unroll
          for (int k = 0; k < 8; k++) { diag += (double)ha[k]; rhs += (double)hb[k]; }
        }
        // adjust_mass_flux (bnd_routines.f90:1185-1210): no flux enters a node
        // out of the system
        if (!(wd && d.inod[i] == -2)) rhs += (double)(dtf * d.rqv[i]);
        d.rhs64[i] = rhs;
        const double zg = level(i);
        d.val64[s0 + dp] = diag;
        tA = rhs - diag * zg;
        tB = extrap ? rhs - diag * (2. * zg - (double)za.zprev[i]) : 0.;
        // an off-diagonal entry: the elements on both sides of its edge (any
        // more in order after them)
        auto entry = [&](int k) {
          const int sl = s0 + k + (k >= dp);
          const int q0s = d.slot_ptr[sl], q1s = d.slot_ptr[sl + 1];
          const int srcA = d.slot_src[q0s], srcB = q1s - q0s > 1 ? d.slot_src[q0s + 1] : -1;
          const int eA = srcA / 9, eB = srcB < 0 ? 0 : srcB / 9;
          double a = (double)elem(za.hia, srcA - 9 * eA, eA);
          if (srcB >= 0) a += (double)elem(za.hia, srcB - 9 * eB, eB);
          for (int t = q0s + 2; t < q1s; t++) {
            const int e = d.slot_src[t] / 9;
            a += (double)elem(za.hia, d.slot_src[t] - 9 * e, e);
          }
          const int c = d.col[sl];
          d.val64[sl] = a;
          tA -= a * level(c);
          if (extrap) tB -= a * (2. * level(c) - (double)za.zprev[c]);
        };
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (k < nd) entry(k);
        for (int k = 8; k < nd; k++) entry(k);
      }
      const float sd = SYM ? (diag > 0. ? (float)(1. / sqrt(diag)) : 1.f) : (diag != 0. ? (float)(1. / diag) : 1.f);
      sh.sd[j] = sd;
      rsA[r] = (float)(SYM ? (double)sd * tA : tA);
      rsB[r] = (float)(SYM ? (double)sd * tB : tB);
      v4[0] += tA * tA;
      v4[1] += (double)rsA[r] * rsA[r];
      v4[2] += tB * tB;
      v4[3] += (double)rsB[r] * rsB[r];
    }
    unsigned ep = number();
#pragma unroll
    for (int r = 0; r < R; r++)
      if (ri[r] < 0) {
        const size_t i = (size_t)(ri[r] & 0x7fffffff);
        word_put(team_buf(tp, xi) + i, __float_as_uint(sh.sd[r * NT + tid]), ep);
        if (rep == 0) word_put(team_buf(tp, xi + 1u) + i, 0u, ep);   // every launch renews every word
        word_put(tp.word + 2 * (size_t)tp.nrow + i, __float_as_uint(rsA[r]), ep);
        word_put(tp.word + 3 * (size_t)tp.nrow + i, __float_as_uint(rsB[r]), ep);
      }
    {
      const double y0 = warp_sum2(v4[0], v4[1]), y1 = warp_sum2(v4[2], v4[3]);
      if ((tid & 15) == 0) {
        sh.wred[(tid >> 4) & 1][tid >> 5] = y0;
        sh.wred[2 + ((tid >> 4) & 1)][tid >> 5] = y1;
      }
    }
    __syncthreads();
    int gi[GR];                                  // the ghosts' global rows, -1: none
    float gr[GR], grB[GR];
    bool ok = true;
    const int gtid = NT - 1 - tid;               // ghosts from the last warps: warp 0 takes the sums
#pragma unroll
    for (int g = 0; g < GR; g++) {
      const int jg = g * NT + gtid;
      gi[g] = -1; gr[g] = 0.f; grB[g] = 0.f;
      float sd = 0.f;
      if (jg < M.nghost) {
        gi[g] = tp.ghost[M.ghost0 + jg];
        const u64 *p = tp.word + gi[g];
        const u64 *const pw[3] = {team_buf(tp, xi) + gi[g], p + 2 * (size_t)tp.nrow, p + 3 * (size_t)tp.nrow};
        unsigned h[3];
        ok = words_wait(tp, pw, ep, abortv, h) && ok;
        sd = __uint_as_float(h[0]);
        gr[g] = __uint_as_float(h[1]);
        grB[g] = __uint_as_float(h[2]);
      }
      sh.sd[NT * R + jg] = sd;
    }
    {
      double tot[4];
      ok = team_totals<2, NT>(sh, tp, M, ep, xi, abortv, tot) && ok;
      if (tid == 0) {
        const double rA = sqrt(tot[0]);
        if (rep == 0) sh.resid0 = rA;
        sh.tol = (double)P.rtol * rA + (double)P.atol;
        const bool useB = extrap && rA > sh.tol;
        sh.stop = useB;
        sh.rn2 = useB ? tot[2] : tot[0];
        sh.rs2 = useB ? tot[3] : tot[1];
        sh.rn = useB ? sqrt(tot[2]) : rA;
      }
    }
    if (!ok) sh.ok = 0;
    __syncthreads();
    if (!sh.ok) { dead = true; break; }
    xi++;

    // ---- the FP64 iterate and the scaled entries of the rows ----
    float rr[R];
    {
      const bool useB = sh.stop != 0;
      auto start = [&](int i) { return useB ? 2. * level(i) - (double)za.zprev[i] : level(i); };
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int j = r * NT + tid;
        rr[r] = useB ? rsB[r] : rsA[r];
        if (j < n) sh.x[j] = CSR ? 0. : start(ri[r] & 0x7fffffff);
      }
#pragma unroll
      for (int g = 0; g < GR; g++) {
        if (useB) gr[g] = grB[g];
        if (gi[g] >= 0) sh.x[NT * R + g * NT + gtid] = CSR ? 0. : start(gi[g]);
      }
    }
    float val[R][K];
    unsigned col[R][K / 2];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int j = r * NT + tid;
#pragma unroll
      for (int k = 0; k < K; k++) val[r][k] = 0.f;
#pragma unroll
      for (int k = 0; k < K / 2; k++) col[r][k] = 0u;
      if (j >= n) continue;
      if constexpr (K == 8) {
        const uint4 c4 = __ldg(reinterpret_cast<const uint4 *>(tp.lcol) + M.row0 + j);
        col[r][0] = c4.x; col[r][1] = c4.y; col[r][2] = c4.z; col[r][3] = c4.w;
      } else {
#pragma unroll
        for (int k = 0; k < K / 2; k++)
          col[r][k] = __ldg(reinterpret_cast<const unsigned *>(tp.lcol) + (size_t)(M.row0 + j) * (K / 2) + k);
      }
      const int i = ri[r] & 0x7fffffff;
      const int dn = tp.dpos[M.row0 + j], dp = dpos_place(dn), nd = dpos_count(dn);
      const double sdi = SYM ? (double)sh.sd[j] : 1.;
      const double *a = val64 + rowptr[i];
#pragma unroll
      for (int k = 0; k < K; k++)
        if (k < nd)
          val[r][k] = (float)(a[k + (k >= dp)] * sdi * (double)at4(sh.sd, col[r][k >> 1], k));
      if (tp.tptr)                               // a long row's tail
        for (int t = tp.tptr[M.row0 + j]; t < tp.tptr[M.row0 + j + 1]; t++)
          tp.tval[t] = (float)(val64[tp.tslot[t]] * sdi * (double)sh.sd[tp.tcol[t]]);
    }

    // the scaled matrix times u for the own rows: the unit diagonal times
    // their own input x, then slot order
    auto product = [&](const float (&x)[R], float (&w)[R]) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        w[r] = x[r];
        if (r >= nr) continue;
#pragma unroll
        for (int k = 0; k < K; k++)
          w[r] += val[r][k] * at4(sh.u, col[r][k >> 1], k);
        if (tp.tptr && r * NT + tid < n)
          for (int t = tp.tptr[M.row0 + r * NT + tid]; t < tp.tptr[M.row0 + r * NT + tid + 1]; t++)
            w[r] += tp.tval[t] * sh.u[tp.tcol[t]];
      }
    };
    // Publish a value per bordering row and the sums v, receive the ghosts' and
    // the totals, which thread 0 hands to `post`; the CTA barrier at the end
    // makes what it stores in sh visible.
    auto exchange = [&](const float (&w)[R], float (&gw)[GR], const auto &v, auto post) -> bool {
      constexpr int NP = sizeof(v) / (2 * sizeof(double));
      ep = number();
      u64 *buf = team_buf(tp, xi);
#pragma unroll
      for (int r = 0; r < R; r++)
        if (ri[r] < 0) word_put(buf + (ri[r] & 0x7fffffff), __float_as_uint(w[r]), ep);
#pragma unroll
      for (int c = 0; c < NP; c++) {
        const double y = warp_sum2(v[2 * c], v[2 * c + 1]);
        if ((tid & 15) == 0) sh.wred[2 * c + ((tid >> 4) & 1)][tid >> 5] = y;
      }
      __syncthreads();
      double tot[2 * NP];
      bool k = team_totals<NP, NT>(sh, tp, M, ep, xi, abortv, tot);
      if (tid == 0) post(tot);
#pragma unroll
      for (int g = 0; g < GR; g++) {
        unsigned h[1] = {0u};
        const u64 *const pw[1] = {buf + gi[g]};
        if (gi[g] >= 0) k = words_wait(tp, pw, ep, abortv, h) && k;
        gw[g] = __uint_as_float(h[0]);
      }
      if (!k) sh.ok = 0;
      __syncthreads();
      xi++;
      return sh.ok != 0;
    };

    for (outer = 0;;) {
      if (sh.rn <= sh.tol || outer >= za.max_outer || (CSR && iters >= P.maxit)) break;
      if (tid == 0) {
        // the FP32 sweep's target, moved into the norm of the residual it works on
        // (CG goes a tenth as far again: the iterations are the same in all, one
        // refinement of three falls away, 7k rows 331 -> 318 us, 250k rows 428
        // -> 405 us, and the level is closer to the exact one: the temperature
        // of the 20k-node basin after 240 steps is 8.0e-5 from the oracle's,
        // where rounding alone moved it between 7.7e-5 and 1.1e-4.  BiCGStab
        // gains nothing: 12k rows 352 -> 376 us.)
        const double it0 = fmax((SYM ? 0.1 : 1.) * (double)za.inner_rtol * sh.rn, tfrac(za) * sh.tol);
        sh.itol2 = sh.rn2 > 0. ? it0 * it0 * (sh.rs2 / sh.rn2) : 0.;
      }
      float e[R], ge[GR];                        // the correction
#pragma unroll
      for (int r = 0; r < R; r++) e[r] = 0.f;
#pragma unroll
      for (int g = 0; g < GR; g++) ge[g] = 0.f;
      if constexpr (SYM) {
        float p[R], s[R], w[R], gp[GR], gs[GR], gw[GR];
#pragma unroll
        for (int r = 0; r < R; r++) {
          p[r] = s[r] = 0.f;
          sh.u[r * NT + tid] = rr[r];
        }
#pragma unroll
        for (int g = 0; g < GR; g++) {
          gp[g] = gs[g] = 0.f;
          sh.u[NT * R + g * NT + gtid] = gr[g];
        }
        __syncthreads();
        product(rr, w);
        double v[2] = {0., 0.};
#pragma unroll
        for (int r = 0; r < R; r++) { v[0] += (double)rr[r] * rr[r]; v[1] += (double)w[r] * rr[r]; }
        // 1 / gamma and 1 / alpha are kept, so that beta = g / gamma and alpha
        // = g / (delta - beta g / alpha) wait for one reciprocal; a correctly
        // rounded one is shorter than a division (per solve: 7k rows 330 ->
        // 315 us, 793 rows 105.7 -> 102.6 us, 250k rows 428 -> 417 us)
        if (!exchange(w, gw, v, [&](const double (&t)[2]) {
              sh.fa = (float)(t[0] / t[1]);
              sh.fb = 0.f;
              sh.rgamma = __drcp_rn(t[0]);
              sh.ralpha = t[1] * sh.rgamma;
            })) { dead = true; break; }
        for (int inner = 1;; inner++) {
          // p = r + b p, s = w + b s, e += a p, r -= a s, then w = (S A S) r
          const float fa = sh.fa, fb = sh.fb;
#pragma unroll
          for (int r = 0; r < R; r++) {
            p[r] = rr[r] + fb * p[r];
            s[r] = w[r] + fb * s[r];
            e[r] += fa * p[r];
            rr[r] -= fa * s[r];
            sh.u[r * NT + tid] = rr[r];
          }
#pragma unroll
          for (int g = 0; g < GR; g++) {
            gp[g] = gr[g] + fb * gp[g];
            gs[g] = gw[g] + fb * gs[g];
            ge[g] += fa * gp[g];
            gr[g] -= fa * gs[g];
            sh.u[NT * R + g * NT + gtid] = gr[g];
          }
          __syncthreads();
          product(rr, w);
          v[0] = v[1] = 0.;
#pragma unroll
          for (int r = 0; r < R; r++) { v[0] += (double)rr[r] * rr[r]; v[1] += (double)w[r] * rr[r]; }
          if (!exchange(w, gw, v, [&](const double (&t)[2]) {
                const double beta = t[0] * sh.rgamma, den = t[1] - beta * t[0] * sh.ralpha;
                sh.fa = (float)(t[0] * __drcp_rn(den));
                sh.fb = (float)beta;
                sh.stop = !(t[0] > sh.itol2) || !(t[0] == t[0]) || inner >= P.maxit;
                sh.rgamma = __drcp_rn(t[0]);
                sh.ralpha = den * sh.rgamma;
              })) { dead = true; break; }
          iters++;
          if (sh.stop) break;
        }
      } else {
        // p = r + beta (p - omega v), v = A p, alpha = rho / (rh v),
        // s = r - alpha v, t = A s, omega = (t s) / (t t), r = s - omega t.
        // rho of the next turn and ||r||^2 follow from the sums of s and t, so
        // an iteration takes two exchanges.
        float rh[R], p[R], q[R], w[R], gp[GR], gv[GR], gw[GR];
#pragma unroll
        for (int r = 0; r < R; r++) { rh[r] = rr[r]; p[r] = q[r] = 0.f; }
#pragma unroll
        for (int g = 0; g < GR; g++) gp[g] = gv[g] = 0.f;
        if (tid == 0) {
          sh.rho = sh.rs2;                       // (rh, r)
          sh.fb = sh.fo = 0.f;
        }
        __syncthreads();
        for (int inner = 1;; inner++) {
          const float fb = sh.fb, fo = sh.fo;    // beta, omega
#pragma unroll
          for (int r = 0; r < R; r++) {
            p[r] = rr[r] + fb * (p[r] - fo * q[r]);
            sh.u[r * NT + tid] = p[r];
          }
#pragma unroll
          for (int g = 0; g < GR; g++) {
            gp[g] = gr[g] + fb * (gp[g] - fo * gv[g]);
            sh.u[NT * R + g * NT + gtid] = gp[g];
          }
          __syncthreads();
          product(p, q);
          double v1[2] = {0., 0.};
#pragma unroll
          for (int r = 0; r < R; r++) v1[0] += (double)rh[r] * q[r];
          if (!exchange(q, gv, v1, [&](const double (&t)[2]) {
                sh.alpha = t[0] != 0. ? sh.rho / t[0] : 0.;
                sh.fa = (float)sh.alpha;
              })) { dead = true; break; }
          const float fa = sh.fa;
#pragma unroll
          for (int r = 0; r < R; r++) {
            rr[r] -= fa * q[r];                  // s
            sh.u[r * NT + tid] = rr[r];
          }
#pragma unroll
          for (int g = 0; g < GR; g++) {
            gr[g] -= fa * gv[g];
            sh.u[NT * R + g * NT + gtid] = gr[g];
          }
          __syncthreads();
          product(rr, w);                        // t
          double v[6] = {0., 0., 0., 0., 0., 0.};
#pragma unroll
          for (int r = 0; r < R; r++) {
            const double sd = rr[r], td = w[r], hd = rh[r];
            v[0] += td * sd;
            v[1] += td * td;
            v[2] += sd * sd;
            v[3] += hd * sd;
            v[4] += hd * td;
          }
          if (!exchange(w, gw, v, [&](const double (&t)[6]) {
                const double om = t[1] > 0. ? t[0] / t[1] : 0.;
                const double rho = t[3] - om * t[4], r2 = t[2] - om * (2. * t[0] - om * t[1]);
                sh.fo = (float)om;
                sh.fb = (float)((rho / sh.rho) * (sh.alpha / om));
                sh.stop = !(r2 > sh.itol2) || !(r2 == r2) || om == 0. || sh.alpha == 0. || rho == 0. ||
                          (CSR ? iters + 1 : inner) >= P.maxit;
                sh.rho = rho;
              })) { dead = true; break; }
          const float fw = sh.fo;
#pragma unroll
          for (int r = 0; r < R; r++) {
            e[r] += fa * p[r] + fw * rr[r];
            rr[r] -= fw * w[r];
          }
#pragma unroll
          for (int g = 0; g < GR; g++) {
            ge[g] += fa * gp[g] + fw * gr[g];
            gr[g] -= fw * gw[g];
          }
          iters++;
          if (sh.stop) break;
        }
      }
      if (dead) break;
      // the correction in FP64, and the residual it leaves
#pragma unroll
      for (int r = 0; r < R; r++)
        if (r * NT + tid < n) sh.x[r * NT + tid] += (double)sh.sd[r * NT + tid] * (double)e[r];
#pragma unroll
      for (int g = 0; g < GR; g++)
        if (gi[g] >= 0) {
          const int j = NT * R + g * NT + gtid;
          sh.x[j] += (double)sh.sd[j] * (double)ge[g];
        }
      outer++;
      __syncthreads();
      double v[2] = {0., 0.};
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int j = r * NT + tid;
        rr[r] = 0.f;
        if (j >= n) continue;
        const int i = ri[r] & 0x7fffffff;
        const int dn = tp.dpos[M.row0 + j], dp = dpos_place(dn), nd = dpos_count(dn);
        const double *a = val64 + rowptr[i];
        double t = rhs64[i] - a[dp] * sh.x[j];
#pragma unroll
        for (int k = 0; k < K; k++)
          if (k < nd) t -= a[k + (k >= dp)] * sh.x[(k & 1 ? col[r][k >> 1] >> 16 : col[r][k >> 1] & 0xffffu) >> 2];
        if (tp.tptr)
          for (int q2 = tp.tptr[M.row0 + j]; q2 < tp.tptr[M.row0 + j + 1]; q2++)
            t -= val64[tp.tslot[q2]] * sh.x[tp.tcol[q2]];
        rr[r] = (float)(SYM ? (double)sh.sd[j] * t : t);
        v[0] += t * t;
        v[1] += (double)rr[r] * rr[r];
      }
      if (!exchange(rr, gr, v, [&](const double (&t)[2]) {
            sh.rn2 = t[0];
            sh.rs2 = t[1];
            sh.rn = sqrt(t[0]);
          })) { dead = true; break; }
    }
    if (dead) break;
    refine += outer;
#pragma unroll
    for (int r = 0; r < R; r++)
      if (r * NT + tid < n) {
        if constexpr (CSR) tp.csr.x[ri[r] & 0x7fffffff] = (float)sh.x[r * NT + tid];
        else d.zn[ri[r] & 0x7fffffff] = (float)sh.x[r * NT + tid];
      }
    if (!wd) break;
    // setweg(1): elements with a vertex below hzmin leave; then the step
    // counters, every element on the first pass of the step (a new time)
    double none = 0., chg = 0.;
    if (!team_barrier(none)) { dead = true; break; }   // the new levels of every row
    for (int e = ea + tid; e < eb; e += NT) {
      chg += wd_take_away(d, P, e) ? 1. : 0.;
      d.iwet[e] = wd_count(d.iweg[e], d.iwet[e], rep == 0);
    }
    if (!team_barrier(chg)) { dead = true; break; }
    if (chg == 0.) break;
    if (rep + 1 >= kWetDryRepeats) { if (M.rank == 0 && tid == 0) set_status(&O, SHY_ENOCONV); break; }
    }
    if (dead) break;
    if (tid == 0 && M.rank == 0) {
      if constexpr (CSR) {
        O.nh_iters = iters;
        O.nh_refinements = refine;
        O.nh_resid0 = sh.resid0;
        O.nh_resid = sh.rn;
      } else {
        O.iters = iters;
        O.refinements = refine;
        O.resid0 = sh.resid0;
        O.resid = sh.rn;
      }
      if (!(sh.rn <= sh.tol)) set_status(&O, SHY_ENOCONV);
    }
    __syncthreads();                             // sh is reused by the next basin
  }
  if (dead && tid == 0)                          // no solution: every basin this CTA has a share of
    for (int q = q0; q < q1; q++) set_status(&d.out[tp.mem[tp.clist[q]].basin], SHY_ECUDA);
  if (tid == 0) tp.cta_cnt[blockIdx.x] = abortv;
}

}  // namespace shy
