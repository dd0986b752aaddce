// Per-Gauss-point backward pass of one load step (the discrete adjoint of the load-step
// sequence; reference: ad_wrapper / implicit_vjp, crystal_plasticity_OR_design/solver.py:801-874,
// and jax.grad through newton_solver's custom_jvp, models_copper.py:251-259).
#include "cpfem_common.cuh"
#include "gp_adjoint.cuh"

namespace cpfem {

// Tangent directions per dual sweep: the six of s, and the nine of F, are whole sweeps of three.  The
// FP64 pipe bounds the kernel (64 cycles per warp instruction, some 8,000 a sweep).  ms for the two
// passes of two steps, 8,000 points, 12 systems: 5.8 (four directions: 6.4; the kernel before, slip
// systems unrolled, sweeps of four seeded through an index array: 6.0); 4,096 points of 24: 13.3
// (13.6; 17.7).
constexpr int kVjpK = 3;

template <int NS>
__global__ void __launch_bounds__(64) k_gp_vjp(const __grid_constant__ MatDev m, const cpfem_vjp_args_t a) {
  const int64_t gp = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t G = a.num_gp;
  if (gp >= G) return;
  const int64_t e = gp >> 3;
  const int32_t* cn = a.cells + e * 8;
  const double* sg = a.shape_grads + gp * 24;
  // every index gathered from the inputs is checked; a bad one is recorded, not read
  bool bad = false;
#pragma unroll
  for (int b = 0; b < 8; ++b) bad = bad || cn[b] < 0 || cn[b] >= a.num_nodes;
  const int64_t ri = a.rot_idx[gp];
  const int64_t pi = (a.param_idx != nullptr) ? a.param_idx[gp] : 0;
  bad = bad || ri < 0 || ri >= a.num_rot || pi < 0 || pi >= a.num_param;
  if (bad) {
    if (a.status != nullptr) atomicOr(a.status, CPFEM_GP_BOUNDS);
    return;
  }
  // kinematics at the checkpointed solution
  double F[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) F[k] = (k % 4 == 0) ? 1.0 : 0.0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int64_t nb = cn[b];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int J = 0; J < 3; ++J) F[3 * i + J] = fma(a.u[3 * nb + i], sg[3 * b + J], F[3 * i + J]);
  }
  double Fpi[9], R[9], th[5];
#pragma unroll
  for (int k = 0; k < 9; ++k) Fpi[k] = a.fpi[k * G + gp];
#pragma unroll
  for (int k = 0; k < 9; ++k) R[k] = a.rot_table[9 * ri + k];
#pragma unroll
  for (int k = 0; k < 5; ++k) th[k] = a.param_table[5 * pi + k];
  Cub cc{m.C11, m.C12, m.C44};
  if (a.elastic_table != nullptr) {
    cc.C11 = a.elastic_table[3 * pi];
    cc.C12 = a.elastic_table[3 * pi + 1];
    cc.C44 = a.elastic_table[3 * pi + 2];
  }
  auto g = [&](int s) { return a.g[s * G + gp]; };
  // recompute the converged local state from the checkpoint (u, Fp^-1, g and, if kept,
  // the converged S as the local Newton's start)
  const double cdt = m.ao * a.dt;
  double s[6], rn;
  {
    double A[9], AR[9], Ct[9];
    mm3(F, Fpi, A);
    mm3(A, R, AR);
    mm3_at(AR, AR, Ct);
    const bool warm = a.s_start != nullptr;
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k] = warm ? a.s_start[k * G + gp] : 0.0;
    rn = cp_root<NS>(m, cc, Ct, cdt, 1.0 / th[3], g, warm, s);
  }
  // output cotangents
  YBar ybar;
#pragma unroll
  for (int c = 0; c < 9; ++c) {
    ybar.P[c] = ybar.sig[c] = 0.0;
    ybar.Fp[c] = (a.fpi_bar != nullptr) ? a.fpi_bar[c * G + gp] : 0.0;
  }
  if (a.cell_sig_bar != nullptr) {
    double wsum = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) wsum += a.jxw[e * 8 + q];
    const double wq = a.jxw[gp] / wsum;
#pragma unroll
    for (int c = 0; c < 9; ++c) ybar.sig[c] = a.cell_sig_bar[e * 9 + c] * wq;
  }
  if (a.mode == 2 && a.mu != nullptr) {
    // P cotangent of the equilibrium term: -JxW * grad(mu)
    const double w = a.jxw[gp];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int64_t nb = cn[b];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int J = 0; J < 3; ++J) ybar.P[3 * i + J] = fma(-w * a.mu[3 * nb + i], sg[3 * b + J], ybar.P[3 * i + J]);
    }
  }
  auto gbar = [&](int s) { return (a.g_bar != nullptr) ? a.g_bar[s * G + gp] : 0.0; };
  // the cotangent of input idx goes to its place, where the caller wants it
  using X = XIn<NS>;
  auto out = [&](int idx, double v) {
    double* p = idx < X::kFp ? a.f_bar : idx < X::kG ? a.fpi_bar_old : idx < X::kTh ? a.g_bar_old : idx < X::kW ? a.theta_bar : a.rot_bar;
    const int at = idx - (idx < X::kFp ? X::kF : idx < X::kG ? X::kFp : idx < X::kTh ? X::kG : idx < X::kW ? X::kTh : X::kW);
    if (p != nullptr) p[at * G + gp] = v;
  };
  const bool ok = cp_vjp<NS, kVjpK>(m, cc, cdt, s, F, Fpi, R, th, g, ybar, gbar, a.mode == 1 ? X::kF : X::kFp,
                                    a.mode == 1 ? X::kFp : X::kN, out);
  if (a.status != nullptr) {
    int bits = 0;
    if (!(rn <= m.local_tol)) bits |= CPFEM_GP_MAXITER;
    if (!ok || !isfinite(rn)) bits |= CPFEM_GP_NONFINITE;
    if (bits) atomicOr(a.status, bits);
  }
}

}  // namespace cpfem

using namespace cpfem;

extern "C" int cpfem_gp_vjp(const cpfem_material_t* mat, const cpfem_vjp_args_t* args, void* stream) {
  CPFEM_REQUIRE(args != nullptr, "args is null");
  MatDev md;
  int rc = make_matdev(mat, &md);
  if (rc != CPFEM_OK) return rc;
  const cpfem_vjp_args_t& a = *args;
  if (a.num_gp == 0) return CPFEM_OK;
  CPFEM_REQUIRE(a.num_gp == (int64_t)a.num_cells * 8, "num_gp must be 8*num_cells");
  CPFEM_REQUIRE(a.mode == 1 || a.mode == 2, "mode must be 1 or 2");
  CPFEM_REQUIRE(a.u && a.cells && a.shape_grads && a.jxw && a.fpi && a.g && a.rot_table && a.rot_idx &&
                    a.param_table, "input pointer is null");
  CPFEM_REQUIRE(md.qmode == 0 || md.num_slip % 3 == 0, "qmode 1 needs num_slip % 3 == 0");
  CPFEM_REQUIRE(a.num_nodes > 0 && a.num_rot > 0 && a.num_param > 0, "table sizes must be given");
  const int threads = 64;
  const unsigned blocks = (unsigned)ceil_div(a.num_gp, threads);
  cudaStream_t s = (cudaStream_t)stream;
  const void* fn = (md.num_slip == 12) ? (const void*)k_gp_vjp<12> : (const void*)k_gp_vjp<24>;
  // the dual-number sweeps need a large per-thread stack: make sure the limit covers it
  cudaFuncAttributes attr;
  CPFEM_CUDA_TRY(cudaFuncGetAttributes(&attr, fn));
  // (the builds with another frame faulted, gp_adjoint.cuh)
  CPFEM_REQUIRE(attr.localSizeBytes % 32 == 0, "the backward kernel was built with a stack frame that is no multiple of 32");
  size_t limit = 0;
  CPFEM_CUDA_TRY(cudaDeviceGetLimit(&limit, cudaLimitStackSize));
  const size_t need = attr.localSizeBytes + 1024;
  if (limit < need) CPFEM_CUDA_TRY(cudaDeviceSetLimit(cudaLimitStackSize, need));
  if (md.num_slip == 12)
    k_gp_vjp<12><<<blocks, threads, 0, s>>>(md, a);
  else
    k_gp_vjp<24><<<blocks, threads, 0, s>>>(md, a);
  CPFEM_CUDA_TRY(cudaGetLastError());
  return CPFEM_OK;
}
