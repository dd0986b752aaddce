// Host interface of the persistent BiCGSTAB by teams of blocks (krylov_team.cuh): the point
// preconditioners for systems whose vectors fit in the SMs' shared memory (krylov_point.cu),
// and the multigrid V-cycle (krylov_mg.cu).
#pragma once

#include "cpfem_common.cuh"

namespace cpfem {

// One team of consecutive blocks and the node range it solves.
struct PointTeam {
  int first, nb;      // blocks first .. first + nb - 1
  int job, pad;       // where the team's report goes (info[2 job], info[2 job + 1])
  int64_t n0, n1;
};

constexpr int kPointMaxValues = 3;    // sums per reduction
constexpr int kPointMaxBlocks = 192;  // blocks of a launch, at most (one per SM)
// Two buffers of a team's partial sums, and a barrier counter (128 bytes apart) per team.
constexpr size_t kPointCellBytes = sizeof(double) * 2 * kPointMaxValues * kPointMaxBlocks;
constexpr size_t kPointCounterBytes = sizeof(unsigned int) * 32 * kPointMaxBlocks;

struct PointArgs {
  cpfem_sell_t L;
  const double* vals;
  const double* b;
  double* x;
  double *phat, *shat;          // 3 * num_nodes each: what the neighbours gather
  double* cells;                // kPointCellBytes
  unsigned int* counters;       // kPointCounterBytes, zeroed before the launch
  int* error;                   // set by a block that waited too long; zeroed before the launch (the report's
                                // own word for a single system)
  const PointTeam* teams;       // by team_of_block, or null: one team of all blocks
  const int* team_of_block;
  cpfem_solve_report_t* out;    // single system: the launch's report
  int32_t* info;                // teams: iterations and converged flag per job
  int precond;
  int maxiter, max_restarts;
  int true_res;                 // also form ||b - A x||^2 of the returned x
  double tol, atol;
  int smem_bytes;               // dynamic shared memory of a block
  int polls;                    // of a wait, at most
};

// How a solve is laid out: blocks, slot lanes per node; ok = false where the vectors do not
// fit and the streaming kernel has to run.
struct PointPlan {
  bool ok;
  int blocks;
  int lanes;
  int threads;
  int smem_bytes;
};

// Plan of one system of n nodes (grid_blocks > 0: that many blocks, at most one per SM; single: the
// V-cycle of precond 3 is FP32).
int point_plan(int64_t n, int precond, bool single, bool transpose, int grid_blocks, PointPlan* plan);
// Plan of teams whose largest share is max_nodes_per_block nodes.
int point_plan_teams(int64_t max_nodes_per_block, int precond, int blocks, PointPlan* plan);
// Blocks of a launch that can be resident together (one per SM).
int point_max_blocks(int* blocks);
int point_launch(const PointPlan& plan, bool transpose, PointArgs args, cudaStream_t s);

// The V-cycle-preconditioned solve (krylov_mg.cu).
int mg_launch(const PointPlan& plan, bool transpose, PointArgs args, const cpfem_mg_t& hierarchy, cudaStream_t s);
int mg_check(const cpfem_mg_t* mg, const cpfem_sell_t* sell);

inline bool sell_ok(const cpfem_sell_t* L) {
  return L && L->num_nodes >= 0 && L->group_off && L->group_width && L->cols && L->diag_slot &&
         L->num_groups == (L->num_nodes + 31) / 32;
}

}  // namespace cpfem
