// Multigrid hierarchy: Galerkin set-up, the coarse levels' dense operator, and the launches of
// the V-cycle-preconditioned BiCGSTAB.
#include <algorithm>

#include "krylov_mg.cuh"

namespace cpfem {

int mg_check(const cpfem_mg_t* mg, const cpfem_sell_t* sell) {
  CPFEM_REQUIRE(mg != nullptr, "precond 3 needs a multigrid hierarchy (opts.mg)");
  const int L = mg->num_levels;
  CPFEM_REQUIRE(L >= 2 && L <= CPFEM_MG_MAX_LEVELS, "multigrid num_levels must be 2..CPFEM_MG_MAX_LEVELS");
  CPFEM_REQUIRE(mg->pre_sweeps >= 1 && mg->post_sweeps >= 0 && mg->coarse_sweeps >= 1, "bad multigrid sweep counts");
  CPFEM_REQUIRE(mg->omega > 0.0 && mg->omega < 2.0, "multigrid omega must lie in (0, 2)");
  CPFEM_REQUIRE(sell == nullptr || mg->sell[0].num_nodes == sell->num_nodes, "level 0 must be the system's layout");
  CPFEM_REQUIRE(mg->precision == 0 || mg->precision == 1, "multigrid precision must be 0 (FP64) or 1 (FP32)");
  CPFEM_REQUIRE(mg->local_nodes >= 0, "multigrid local_nodes must be >= 0");
  const bool single = mg->precision == 1;
  for (int l = 0; l < L; ++l) {
    const int64_t n = (int64_t)mg->dims[l][0] * mg->dims[l][1] * mg->dims[l][2];
    CPFEM_REQUIRE(mg->dims[l][0] >= 1 && mg->dims[l][1] >= 1 && mg->dims[l][2] >= 1 && n == mg->sell[l].num_nodes,
                  "multigrid dims do not match the level's node count");
    CPFEM_REQUIRE(sell_ok(&mg->sell[l]) && mg->minv[l], "multigrid level arrays missing");
    CPFEM_REQUIRE(single ? ((l == 0 || mg->values32[l]) && mg->minv32[l] && mg->x32[l] && mg->t32[l])
                         : (mg->x[l] && mg->t[l]),
                  "multigrid work arrays missing");
    CPFEM_REQUIRE(mg->slot[l], "multigrid slot table missing");
    if (l + 1 < L) {
      CPFEM_REQUIRE(single ? mg->r32[l] != nullptr : mg->r[l] != nullptr, "multigrid residual array missing");
      const int64_t need = (int64_t)((mg->dims[l][0] - 1) / 2 + 1) * mg->dims[l][1] * mg->dims[l][2];
      CPFEM_REQUIRE(mg->scratch[0] && mg->scratch[1] && mg->scratch_nodes >= need,
                    "multigrid scratch missing or too small");
    }
    if (l >= 1) {
      CPFEM_REQUIRE(mg->values[l] && (single ? mg->b32[l] != nullptr : mg->b[l] != nullptr),
                    "multigrid coarse arrays missing");
      for (int d = 0; d < 3; ++d)
        CPFEM_REQUIRE((mg->dims[l - 1][d] - 1) % 2 == 0 && mg->dims[l][d] == (mg->dims[l - 1][d] - 1) / 2 + 1,
                      "each multigrid level must halve the cell counts of the finer one");
    }
  }
  return CPFEM_OK;
}

// Galerkin coarse operator P^T A P by three 1-D passes: P = P_z (x) P_y (x) P_x, so
// coarsening one direction at a time keeps a 27-point stencil and needs 7 (same coarse
// neighbour) or 3 (next one) fine pairs per output block instead of up to 343.  One thread
// per (output node, stencil offset); input and output stencils are [node][27][9]; the
// first pass reads the sliced-ELL fine operator through its slot table (Dirichlet dofs of
// level 0 left out on both sides), the last writes the coarse sliced-ELL operator.
// Fixed summation order: reproducible.
__global__ void __launch_bounds__(256) k_mg_rap_dir(int dir, int ix, int iy, int iz, int ox, int oy, int oz,
                                                    const cpfem_sell_t F, const double* __restrict__ vf,
                                                    const int8_t* __restrict__ slot_in,
                                                    const double* __restrict__ sin_,
                                                    const int8_t* __restrict__ free_dof, double* __restrict__ sout,
                                                    const cpfem_sell_t C, const int8_t* __restrict__ slot_out,
                                                    double* __restrict__ vc) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nout = (int64_t)ox * oy * oz;
  if (t >= 27 * nout) return;
  const int64_t o = t / 27;
  const int off = (int)(t % 27);
  int oc[3] = {(int)(o % ox), (int)((o / ox) % oy), (int)(o / ((int64_t)ox * oy))};
  int d[3] = {off % 3 - 1, (off / 3) % 3 - 1, off / 9 - 1};
  const int din[3] = {ix, iy, iz};
  const int del = d[dir];
  double acc[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.0;
  for (int a = -1; a <= 1; ++a)
    for (int b = -1; b <= 1; ++b) {
      const int e = 2 * del + b - a;      // input offset along dir
      if (e < -1 || e > 1) continue;
      int ic[3] = {oc[0], oc[1], oc[2]};
      ic[dir] = 2 * oc[dir] + a;
      int jc[3] = {ic[0] + d[0], ic[1] + d[1], ic[2] + d[2]};
      jc[dir] = ic[dir] + e;
      bool inside = true;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        inside = inside && ic[k] >= 0 && ic[k] < din[k] && jc[k] >= 0 && jc[k] < din[k];
      if (!inside) continue;
      const int64_t i = ic[0] + (int64_t)ix * (ic[1] + (int64_t)iy * ic[2]);
      int ed[3] = {d[0], d[1], d[2]};
      ed[dir] = e;
      const int code = (ed[2] + 1) * 9 + (ed[1] + 1) * 3 + (ed[0] + 1);
      const double w = (a ? 0.5 : 1.0) * (b ? 0.5 : 1.0);
      if (sin_ == nullptr) {
        const int sf = slot_in[27 * i + code];
        if (sf < 0) continue;
        const int64_t j = jc[0] + (int64_t)ix * (jc[1] + (int64_t)iy * jc[2]);
        const double* blk = vf + 9 * F.group_off[i >> 5] + (i & 31) + 288LL * sf;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (free_dof != nullptr && (free_dof[3 * i + r] == 0 || free_dof[3 * j + c] == 0)) continue;
            acc[3 * r + c] = fma(w, __ldg(&blk[32 * (3 * r + c)]), acc[3 * r + c]);
          }
      } else {
        const double* blk = sin_ + 9 * (27 * i + code);
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = fma(w, __ldg(&blk[k]), acc[k]);
      }
    }
  if (sout != nullptr) {
#pragma unroll
    for (int k = 0; k < 9; ++k) sout[9 * (27 * o + off) + k] = acc[k];
  } else {
    const int s = slot_out[27 * o + off];
    if (s < 0) return;
    double* blk = vc + 9 * C.group_off[o >> 5] + (o & 31) + 288LL * s;
#pragma unroll
    for (int k = 0; k < 9; ++k) blk[32 * k] = acc[k];
  }
}

// FP32 copy of n values, or of a sliced-ELL value array (9 * group_off[num_groups] values,
// read on the device) when slots != nullptr.
__global__ void __launch_bounds__(256) k_to_f32(const double* __restrict__ in, float* __restrict__ out, int64_t n,
                                                const int64_t* __restrict__ slots) {
  const int64_t m = slots != nullptr ? 9 * slots[0] : n;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (float)in[i];
}

// Columns of the dense operator of levels lb .. L-1 (mg_dense_level): a block runs the levels'
// cycle in its shared memory on one unit right-hand side after another.
template <typename R>
__global__ void __launch_bounds__(512, 1) k_mg_dense(const cpfem_mg_t mg, int lb) {
  const MgArrays<R> A{mg, nullptr};
  const MgShared lay = mg_shared_layout(mg, lb, sizeof(R));
  const bool staged = mg_stage<R>(mg, lb, A, lay);
  const int N = 3 * (int)mg.sell[lb].num_nodes;
  R* b = reinterpret_cast<R*>(mg_shared) + lay.vec[lb] + (size_t)3 * N;
  R* K = mg_dense<R>(mg);
  for (int c = blockIdx.x; c < N; c += gridDim.x) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) b[i] = i == c ? R(1) : R(0);
    __syncthreads();
    const R* X = staged ? mg_local_cycle<true>(mg, A, lay, lb) : mg_local_cycle<false>(mg, A, lay, lb);
    for (int i = threadIdx.x; i < N; i += blockDim.x) K[(size_t)i * N + c] = X[i];
    __syncthreads();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *mg_tag(mg) = mg_tag_of<R>(mg, A.minv(lb), lb);
}

template <typename R>
static int mg_dense_setup(const cpfem_mg_t& mg, cudaStream_t s) {
  const int lb = mg_dense_level(mg, sizeof(R));
  if (lb >= mg.num_levels) return CPFEM_OK;
  int sms = 0;
  if (const int rc = point_max_blocks(&sms); rc != CPFEM_OK) return rc;
  const size_t smem = mg_shared_layout(mg, lb, sizeof(R)).total;
  CPFEM_CUDA_TRY(cudaFuncSetAttribute((const void*)k_mg_dense<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMgStageBytes));
  k_mg_dense<R><<<(unsigned)std::min<int64_t>(sms, 3 * (int64_t)mg.sell[lb].num_nodes), 512, smem, s>>>(mg, lb);
  CPFEM_CUDA_TRY(cudaGetLastError());
  return CPFEM_OK;
}

template <typename R>
static const void* mg_kernel(bool transpose, int lanes) {
  if (transpose)
    return lanes >= 4 ? (const void*)k_bicgstab_team<true, 4, R, cpfem_mg_t>
         : lanes == 2 ? (const void*)k_bicgstab_team<true, 2, R, cpfem_mg_t> : (const void*)k_bicgstab_team<true, 1, R, cpfem_mg_t>;
  return lanes >= 4 ? (const void*)k_bicgstab_team<false, 4, R, cpfem_mg_t>
       : lanes == 2 ? (const void*)k_bicgstab_team<false, 2, R, cpfem_mg_t> : (const void*)k_bicgstab_team<false, 1, R, cpfem_mg_t>;
}

int mg_launch(const PointPlan& plan, bool transpose, PointArgs args, const cpfem_mg_t& hierarchy, cudaStream_t s) {
  cpfem_mg_t mg = hierarchy;
  const void* fn = mg.precision == 1 ? mg_kernel<float>(transpose, plan.lanes) : mg_kernel<double>(transpose, plan.lanes);
  args.smem_bytes = plan.smem_bytes;
  CPFEM_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtSmemBytes));
  void* pargs[] = {&args, &mg};
  CPFEM_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3((unsigned)plan.blocks), dim3((unsigned)plan.threads), pargs,
                                             (size_t)plan.smem_bytes, s));
  return CPFEM_OK;
}

}  // namespace cpfem

using namespace cpfem;

extern "C" int cpfem_mg_setup(const cpfem_mg_t* mg, const double* values0, void* stream) {
  CPFEM_REQUIRE(values0 != nullptr, "values0 is null");
  int rc = mg_check(mg, nullptr);
  if (rc != CPFEM_OK) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  k_precond_setup<false><<<(unsigned)ceil_div(mg->sell[0].num_nodes, 128), 128, 0, s>>>(mg->sell[0], values0, 2,
                                                                                         mg->minv[0]);
  CPFEM_CUDA_TRY(cudaGetLastError());
  for (int l = 0; l + 1 < mg->num_levels; ++l) {
    const double* vf = (l == 0) ? values0 : mg->values[l];
    const int32_t* fi = mg->dims[l];
    const int32_t* co = mg->dims[l + 1];
    const cpfem_sell_t& C = mg->sell[l + 1];
    // x pass: fine SELL -> scratch[0] (co.x, fi.y, fi.z); y pass -> scratch[1] (co.x, co.y,
    // fi.z); z pass -> the coarse SELL
    const int64_t n1 = (int64_t)co[0] * fi[1] * fi[2], n2 = (int64_t)co[0] * co[1] * fi[2];
    const int64_t n3 = (int64_t)co[0] * co[1] * co[2];
    k_mg_rap_dir<<<(unsigned)ceil_div(27 * n1, 256), 256, 0, s>>>(0, fi[0], fi[1], fi[2], co[0], fi[1], fi[2],
                                                                   mg->sell[l], vf, mg->slot[l], nullptr,
                                                                   (l == 0) ? mg->free_dof : nullptr,
                                                                   mg->scratch[0], C, nullptr, nullptr);
    CPFEM_CUDA_TRY(cudaGetLastError());
    k_mg_rap_dir<<<(unsigned)ceil_div(27 * n2, 256), 256, 0, s>>>(1, co[0], fi[1], fi[2], co[0], co[1], fi[2],
                                                                   mg->sell[l], nullptr, nullptr, mg->scratch[0],
                                                                   nullptr, mg->scratch[1], C, nullptr, nullptr);
    CPFEM_CUDA_TRY(cudaGetLastError());
    k_mg_rap_dir<<<(unsigned)ceil_div(27 * n3, 256), 256, 0, s>>>(2, co[0], co[1], fi[2], co[0], co[1], co[2],
                                                                   mg->sell[l], nullptr, nullptr, mg->scratch[1],
                                                                   nullptr, nullptr, C, mg->slot[l + 1],
                                                                   mg->values[l + 1]);
    CPFEM_CUDA_TRY(cudaGetLastError());
    k_precond_setup<false><<<(unsigned)ceil_div(C.num_nodes, 128), 128, 0, s>>>(C, mg->values[l + 1], 2,
                                                                                mg->minv[l + 1]);
    CPFEM_CUDA_TRY(cudaGetLastError());
  }
  if (mg->precision == 1) {
    // the FP32 V-cycle's coarse operators: rounded copies of the FP64 ones (level 0 reads
    // the system's values directly)
    for (int l = 0; l < mg->num_levels; ++l) {
      const cpfem_sell_t& S = mg->sell[l];
      if (l > 0) {
        k_to_f32<<<1216, 256, 0, s>>>(mg->values[l], mg->values32[l], 0, S.group_off + S.num_groups);
        CPFEM_CUDA_TRY(cudaGetLastError());
      }
      const int64_t nm = 9 * (int64_t)S.num_nodes;
      k_to_f32<<<(unsigned)std::min<int64_t>(ceil_div(nm, 256), 1216), 256, 0, s>>>(mg->minv[l], mg->minv32[l], nm,
                                                                                   nullptr);
      CPFEM_CUDA_TRY(cudaGetLastError());
    }
  }
  // the coarse levels' part of the cycle as a dense operator, one column per pass of a block
  if (mg->precision == 1) return mg_dense_setup<float>(*mg, s);
  return mg_dense_setup<double>(*mg, s);
}

