// Solve kernel instances for one block size: STEEL_BLOCK threads per block, set by the build
// (solve.cu is compiled once per size into solve_<N>.o). One block per scene (body: solve_scene,
// solve.cuh); blocks take scenes in B.order (longest first), so the scenes with the longest serial
// chains start in the first wave.
#include "solve.cuh"

#ifndef STEEL_BLOCK
#error "compile with -DSTEEL_BLOCK=<threads per block>"
#endif
#define STEEL_CAT2(a, b) a##b
#define STEEL_CAT(a, b) STEEL_CAT2(a, b)
#define STEEL_NS STEEL_CAT(t, STEEL_BLOCK)

namespace steel {
namespace STEEL_NS {
// EXT: the batch has a scene with torsional/rolling friction of articulated contacts or the
// contact-then-internal row schedule; only that instance carries the 5-row angular block in its
// contact loop and the two-phase iteration. ROWS: which of the solve's bodies the instance has, by what
// the batch's scenes need (solve_scene).
template <bool EXT, uint32_t ROWS>
__global__ void __launch_bounds__(STEEL_BLOCK, blocks_per_sm_of(STEEL_BLOCK)) k_solve(BatchDev B) {
  const uint32_t sc = B.order[blockIdx.x];
  const unsigned long long t0 = B.trace_solve ? trace_clock() : 0ull;
  solve_scene<EXT, false, ROWS>(B, sc, Team<false>{});
  if (B.trace_solve) trace_block(B.trace_solve + 3ull * sc, t0);
}
#if STEEL_BLOCK == 512  // team launches run the 512-thread instances (one block per SM)
// A batch of one large scene: every block of this cooperative launch solves it together (team.cuh).
template <bool EXT, uint32_t ROWS>
__global__ void __launch_bounds__(STEEL_BLOCK, blocks_per_sm_of(STEEL_BLOCK)) k_solve_team(BatchDev B) {
  __shared__ uint32_t team_state[2];
  if (threadIdx.x == 0u) { team_state[0] = 0u; team_state[1] = 0u; }  // published by copy_scene's barrier
  const uint32_t sc = B.order[0];
  const unsigned long long t0 = B.trace_solve ? trace_clock() : 0ull;
  solve_scene<EXT, true, ROWS>(B, sc, Team<true>{B.team_bar, B.error, TEAM_WAIT_LIMIT, team_state});
  if (B.trace_solve && blockIdx.x == 0u) trace_block(B.trace_solve + 3ull * sc, t0);
}
#endif
}  // namespace STEEL_NS

typedef void (*SolveKernel)(BatchDev);
// The instance for a batch: [EXT][ROWS_*], and the team's (a batch of one scene is never mixed).
static SolveKernel solve_kernel(bool ext, uint32_t rows) {
  static const SolveKernel k[2][3] = {
      {STEEL_NS::k_solve<false, ROWS_PACKED>, STEEL_NS::k_solve<false, ROWS_RECORDS>, STEEL_NS::k_solve<false, ROWS_BOTH>},
      {STEEL_NS::k_solve<true, ROWS_PACKED>, STEEL_NS::k_solve<true, ROWS_RECORDS>, STEEL_NS::k_solve<true, ROWS_BOTH>}};
  return k[ext ? 1 : 0][rows - ROWS_PACKED];
}
#if STEEL_BLOCK == 512
static SolveKernel solve_team_kernel(bool ext, uint32_t rows) {
  if (rows == ROWS_PACKED) return ext ? STEEL_NS::k_solve_team<true, ROWS_PACKED> : STEEL_NS::k_solve_team<false, ROWS_PACKED>;
  return ext ? STEEL_NS::k_solve_team<true, ROWS_RECORDS> : STEEL_NS::k_solve_team<false, ROWS_RECORDS>;
}
#endif

template <>
cudaError_t configure_solve_t<STEEL_BLOCK>(size_t smem_bytes) {
  for (uint32_t ext = 0; ext < 2u; ext++)
    for (uint32_t rows = ROWS_PACKED; rows <= ROWS_BOTH; rows++) {
      cudaError_t e = cudaFuncSetAttribute((const void*)solve_kernel(ext != 0u, rows),
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
#if STEEL_BLOCK == 512
      if (e == cudaSuccess && rows != ROWS_BOTH)
        e = cudaFuncSetAttribute((const void*)solve_team_kernel(ext != 0u, rows),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
#endif
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}
template <>
void launch_solve_t<STEEL_BLOCK>(const BatchDev& b, cudaStream_t st) {
#if STEEL_BLOCK == 512
  if (b.team_blocks) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b.team_blocks);
    cfg.blockDim = dim3(STEEL_BLOCK);
    cfg.dynamicSmemBytes = b.team_smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;  // every block resident: the grid barrier's guarantee
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaMemsetAsync(b.team_bar, 0, sizeof(uint32_t), st);
    cudaLaunchKernelEx(&cfg, solve_team_kernel(b.solve_ext != 0u, b.solve_rows), b);
    return;
  }
#endif
  // The launch asks for the shared memory its resident blocks use and leaves the rest to L1, which
  // the articulated passes read through (without the hint the driver provides for as many blocks as
  // the registers allow).
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(b.nlaunch);
  cfg.blockDim = dim3(STEEL_BLOCK);
  cfg.dynamicSmemBytes = b.solve_smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  at[0].val.sharedMemCarveout = solve_carveout(b);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, solve_kernel(b.solve_ext != 0u, b.solve_rows), b);
}
template <>
int solve_team_blocks_per_sm_t<STEEL_BLOCK>(size_t smem_bytes) {
#if STEEL_BLOCK == 512
  int least = 0;
  for (uint32_t k = 0; k < 4u; k++) {
    int n = 0;
    const SolveKernel f = solve_team_kernel((k & 1u) != 0u, (k & 2u) != 0u ? ROWS_RECORDS : ROWS_PACKED);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, STEEL_BLOCK, smem_bytes) != cudaSuccess) return 0;
    if (k == 0u || n < least) least = n;
  }
  return least;
#else
  (void)smem_bytes;
  return 0;
#endif
}

}  // namespace steel
