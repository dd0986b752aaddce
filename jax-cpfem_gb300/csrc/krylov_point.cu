// Persistent BiCGSTAB with the point preconditioners (none, 1/diag, inverted 3x3 diagonal
// block) for systems whose Krylov vectors fit in shared memory (up to about 53^3 cells on one
// GB300): every mesh of the drop-in drivers and the RVEs of a batch.  Plans (the multigrid solve's
// too) and launches.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "krylov_team.cuh"

namespace cpfem {

static const void* point_kernel(bool transpose, int lanes) {
  if (transpose)
    return lanes == 8 ? (const void*)k_bicgstab_team<true, 8, void, NoMg> : lanes == 4 ? (const void*)k_bicgstab_team<true, 4, void, NoMg>
         : lanes == 2 ? (const void*)k_bicgstab_team<true, 2, void, NoMg> : (const void*)k_bicgstab_team<true, 1, void, NoMg>;
  return lanes == 8 ? (const void*)k_bicgstab_team<false, 8, void, NoMg> : lanes == 4 ? (const void*)k_bicgstab_team<false, 4, void, NoMg>
       : lanes == 2 ? (const void*)k_bicgstab_team<false, 2, void, NoMg> : (const void*)k_bicgstab_team<false, 1, void, NoMg>;
}

int point_max_blocks(int* blocks) {
  int dev = 0;
  CPFEM_CUDA_TRY(cudaGetDevice(&dev));
  CPFEM_CUDA_TRY(cudaDeviceGetAttribute(blocks, cudaDevAttrMultiProcessorCount, dev));
  *blocks = std::min(*blocks, kPointMaxBlocks);
  return CPFEM_OK;
}

// Shared memory of a block that owns up to `nodes` nodes: the vectors, and with the matrix
// rows.
static size_t point_smem(int64_t nodes, int precond, int lanes, bool matrix) {
  const size_t vec = sizeof(double) * (size_t)nodes * (24 + (precond == 2 ? 9 : precond == 1 ? 3 : 0));
  const size_t items = (size_t)ceil_div(nodes, 32 / lanes) * (size_t)ceil_div(kPtMaxWidth, lanes) * 32;
  return vec + (matrix ? items * (9 * sizeof(double) + sizeof(int)) : 0);
}

// Slot lanes per node: the split with the least FP64 work on the busiest sub-partition (a
// row's share of the slots, the adds of its lane sum, whole rounds), ties to fewer lanes.
static int point_lanes(int64_t nodes, int blocks) {
  int best = 1;
  double cost = 1e300;
  for (int ql = 1; ql <= 8; ql *= 2) {
    const int64_t units = ceil_div(ceil_div(nodes, 32 / ql), blocks);
    const double row = 3.0 * (double)ceil_div(kPtMaxWidth, ql) + 1.0 + std::log2((double)ql);
    const double c = row * (double)ceil_div(3 * units, 4);
    if (c < 0.97 * cost) { cost = c; best = ql; }
  }
  return best;
}

// The rest of a plan, the lanes given: rows staged in shared memory where they fit (16 warps), else
// read from L2 (24 warps, more loads in flight; what shared memory is left is L1's).
//
// Past some number of nodes a block the streaming kernel takes systems whose rows are not staged,
// where it is the faster one.  A transposed product gathers its blocks from the neighbours' rows: a
// block's range here is far from theirs, while the streaming kernel's blocks walk the mesh together
// and find them in L2.  us per iteration, here and there, nodes a block in brackets:
//   Jacobi transposed             40^3 cells (453) 115, 129     48^3 (774) 202, 182
//   FP64 V-cycle transposed       36^3 (333) 465, 504           40^3 631, 561
//   FP32 V-cycle transposed       44^3 (600) 529, 578           48^3 667, 661     52^3 (979) 990, 741
//   FP32 V-cycle                  44^3 441, 462                 48^3 558, 539     52^3 652, 598
//   FP64 V-cycle                  44^3 551, 633                 52^3 781, 911
// so the last stays here as long as its vectors fit.
static int64_t point_most(int precond, bool single, bool transpose) {
  if (precond == 3) return single ? 700 : transpose ? 400 : INT64_MAX;
  return transpose ? 512 : INT64_MAX;
}

static void point_fit(int64_t nodes, int blocks, int precond, bool single, bool transpose, bool teams, PointPlan* plan) {
  const int64_t npw = 32 / plan->lanes;
  const int64_t share = (ceil_div(ceil_div(nodes, npw), blocks) + (teams ? 1 : 0)) * npw;
  const size_t most = (size_t)kPtSmemBytes, vec = point_smem(share, precond, plan->lanes, false),
               all = point_smem(share, precond, plan->lanes, true);
  const bool staged = all <= most;
  plan->ok = vec <= most && (staged || share <= point_most(precond, single, transpose));
  plan->threads = precond == 3 ? kMgThreads : staged ? 512 : kPtMaxThreads;
  plan->smem_bytes = (int)std::max<size_t>(16, staged ? all : plan->ok ? vec : 0);
}

int point_plan(int64_t n, int precond, bool single, bool transpose, int grid_blocks, PointPlan* plan) {
  int sms = 0;
  const int rc = point_max_blocks(&sms);
  if (rc != CPFEM_OK) return rc;
  int64_t blocks = n <= 48 ? 1 : sms;
  if (grid_blocks > 0) blocks = std::min(grid_blocks, sms);
  blocks = std::max<int64_t>(1, std::min<int64_t>(blocks, ceil_div(n, 4)));
  plan->blocks = (int)blocks;
  plan->lanes = point_lanes(n, (int)blocks);
  if (precond == 3) plan->lanes = std::min(plan->lanes, 4);   // the V-cycle's kernels
  point_fit(n, (int)blocks, precond, single, transpose, false, plan);
  if (precond == 3 && plan->smem_bytes < (int)point_smem(ceil_div(n, blocks), precond, 1, true)) {
    // rows that stream: a unit of three rows per warp, as few lanes per node as keep most of
    // the eight warps at work
    plan->lanes = 1;
    while (plan->lanes < 4 && ceil_div(ceil_div(n, 32 / plan->lanes), blocks) < 6) plan->lanes *= 2;
    point_fit(n, (int)blocks, precond, single, transpose, false, plan);
  }
  return CPFEM_OK;
}

int point_plan_teams(int64_t max_nodes_per_block, int precond, int blocks, PointPlan* plan) {
  plan->blocks = blocks;
  plan->lanes = point_lanes(max_nodes_per_block, 1);
  point_fit(max_nodes_per_block, 1, precond, false, false, true, plan);
  return CPFEM_OK;
}

int point_launch(const PointPlan& plan, bool transpose, PointArgs args, cudaStream_t s) {
  const void* fn = point_kernel(transpose, plan.lanes);
  args.smem_bytes = plan.smem_bytes;
  CPFEM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtSmemBytes));
  NoMg none;
  void* pargs[] = {&args, &none};
  CPFEM_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3((unsigned)plan.blocks), dim3((unsigned)plan.threads), pargs,
                                             (size_t)plan.smem_bytes, s));
  return CPFEM_OK;
}

}  // namespace cpfem
