// step_zeta.cu -- launch wrappers and set-up of the zeta solvers (k_zeta,
// k_zeta_team, k_zeta_grid).  See step.cu.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "../../include/shygpu.h"
#include "common.cuh"
#include "launch.h"
#include "physics.cuh"
#include "k_wetdry.cuh"
#include "k_zeta.cuh"
#include "k_zeta_global.cuh"
#include "k_zeta_grid.cuh"
#include "k_zeta_team.cuh"

namespace shy {

static cudaLaunchConfig_t zeta_config(int CL, int threads, int nclusters, cudaStream_t st,
                                      cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nclusters * CL, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

cudaError_t launch_zeta(const Dev &d, const ZetaArgs &za, int CL, int threads, int nb, cudaStream_t st) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = zeta_config(CL, threads, nb, st, attr);
  return cudaLaunchKernelEx(&cfg, k_zeta, d, za, CL);
}

cudaError_t launch_zeta_grid(const Dev &d, const ZetaArgs &za, const GridPlan &gp, int G, bool staged,
                             size_t smem, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(gp.ctr, 0, 8 * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(G, 1, 1);
  cfg.blockDim = dim3(staged ? 1024 : 512, 1, 1);
  cfg.dynamicSmemBytes = staged ? smem : 0;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const bool c16 = gp.ecol16 != nullptr;
  if (staged) return c16 ? cudaLaunchKernelEx(&cfg, k_zeta_grid<1024, true, true>, d, za, gp)
                         : cudaLaunchKernelEx(&cfg, k_zeta_grid<1024, true, false>, d, za, gp);
  return c16 ? cudaLaunchKernelEx(&cfg, k_zeta_grid<512, false, true>, d, za, gp)
             : cudaLaunchKernelEx(&cfg, k_zeta_grid<512, false, false>, d, za, gp);
}

constexpr int kTeamNT = 512;
constexpr long long kTeamSpinLimit = 1LL << 22;   // polls of a word: seconds
// the zeta system (rows of up to eight neighbours in the block), and the 3D
// system (a row has its node's neighbours at the same layer and the two
// layers beside it, so most need 8 of the 26 places; longer ones have a tail)
constexpr auto kZetaSym = k_zeta_team<kTeamNT, 4, 1, 8, true, false>;
constexpr auto kZetaGen = k_zeta_team<kTeamNT, 4, 1, 8, false, false>;
constexpr auto kCsrGen = k_zeta_team<kTeamNT, 1, 2, 26, false, true>;

static cudaError_t launch_team(void (*kernel)(Dev, ZetaArgs, TeamPlan), const Dev &d, const ZetaArgs &za,
                               const TeamPlan &tp, int G, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(G, 1, 1);
  cfg.blockDim = dim3(kTeamNT, 1, 1);
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, d, za, tp);
}

cudaError_t launch_zeta_team(const Dev &d, const ZetaArgs &za, const TeamPlan &tp, int G, cudaStream_t st) {
  return launch_team(za.sym ? kZetaSym : kZetaGen, d, za, tp, G, st);
}

cudaError_t launch_csr_team(const Dev &d, const ZetaArgs &za, const TeamPlan &tp, int G, cudaStream_t st) {
  return launch_team(kCsrGen, d, za, tp, G, st);
}

static int team_capacity(void (*kernel)(Dev, ZetaArgs, TeamPlan)) {
  int dev = 0, nsm = 0, nb = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, kTeamNT, 0) != cudaSuccess) return 0;
  return std::min(nb * nsm, kTeamNT);      // one thread polls each member of a team
}
TeamShape zeta_team_shape() {
  return TeamShape{kTeamNT * 4, kTeamNT, 8, std::min(team_capacity(kZetaSym), team_capacity(kZetaGen))};
}
TeamShape csr_team_shape() { return TeamShape{kTeamNT, 2 * kTeamNT, 26, team_capacity(kCsrGen)}; }
// Rows a CTA gets.  Basins alone are faster in shares of 1024 rows than of
// 2048 (us a solve by CG: 3k rows 157 against 165, 7k 161/191, 12k 162/201,
// 20k 170/204, 36k 190/213, 60k 192/215, 90k 208/243; at 150k, 147 members,
// 271/258), many basins in one model in larger ones, whose teams take fewer
// turns on the CTAs (24 basins of 9000 rows 348 against 224, 24 of 20000
// 712/453, 16 members of the ensemble 1405/648, all 64 5100/2500).  A basin's
// bits may depend on the basin alone, so the rule cannot ask how many there
// are: small basins, which are run alone, get 1024 rows and pay 55% more
// where two dozen share a model; larger ones 2048, at 10 to 20% of their
// time alone.  The line between them lies at no knee of either curve.
int zeta_team_share(int nk) { return nk <= 12288 ? kTeamNT * 2 : kTeamNT * 4; }
long long zeta_team_spin_limit() { return kTeamSpinLimit; }

size_t zeta_grid_stage_smem(bool c16) { return 128 + 2 * (size_t)stage_layout(c16 ? 16 : 32).bytes; }

// resident CTAs of the device-wide solver; the fewer of its two column
// forms, so a plan holds whichever it launches
template <bool STAGED, bool C16>
static int grid_blocks(size_t smem) {
  constexpr int NT = STAGED ? 1024 : 512;
  int nb = 0;
  if (STAGED && cudaFuncSetAttribute(k_zeta_grid<NT, STAGED, C16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_zeta_grid<NT, STAGED, C16>, NT, STAGED ? smem : 0) !=
      cudaSuccess)
    return 0;
  return nb;
}

int zeta_grid_capacity(bool staged, size_t smem) {
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  const int nb = staged ? std::min(grid_blocks<true, true>(smem), grid_blocks<true, false>(smem))
                        : std::min(grid_blocks<false, true>(0), grid_blocks<false, false>(0));
  return nb * nsm;
}

int zeta_grid_max_slots() { return kGridMaxSlots; }
int zeta_grid_max_tiles() { return kGridMaxTiles; }
int zeta_grid_tile_rows() { return kGridTileRows; }
long long zeta_grid_spin_limit() { return kGridSpinLimit; }

cudaError_t zeta_kernel_setup(int CL) {
  return CL > 8 ? cudaFuncSetAttribute(k_zeta, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
}

int zeta_max_active_clusters(int CL, int threads) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = zeta_config(CL, threads, 1, nullptr, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, (const void *)k_zeta, &cfg) != cudaSuccess) return -1;
  return n;
}

}  // namespace shy
