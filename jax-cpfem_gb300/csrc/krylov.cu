// Sliced-ELL SpMV and the persistent BiCGSTAB of the cpfem_gb300 C ABI.
//
// Values are stored per group of 32 consecutive nodes (one warp), slot-major, so the
// thread of node a reads its 3x3 blocks with fully coalesced loads and accumulates its
// three rows without any cross-lane reduction -- on GB300 the FP64 pipe, not HBM, is
// the SpMV's limit, and a shuffle reduction would cost as many FP64 adds as the FMAs.
//
// BiCGSTAB runs as one cooperative launch.  Systems whose vectors fit the blocks' shared
// memory use the kernel of krylov_team.cuh; the kernels here
// stream their vectors from memory, for larger systems and for batches of many.  In them
// every block owns a fixed set of nodes, the five global dependencies of an iteration (the halo of phat and shat, four dot
// products) are crossed with a grid barrier, and every block reduces the per-block
// partial sums in the same fixed order, so all blocks hold bitwise-identical scalars
// and take the same branch.  Barrier waits are bounded: a block that waits too long sets
// an error flag and the solve returns CPFEM_ERR_SOLVE.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>
#include <string>

#include "cpfem_common.cuh"
#include "krylov_mg.cuh"
#include "reduce.cuh"

namespace cpfem {

constexpr int kPThreads = 256;
constexpr int kMaxBlocks = 2048;
constexpr long long kSpinLimit = 1LL << 25;   // ~1-3 s of polling at ~50 ns per poll

struct GridSync {
  unsigned int count;   // arrivals so far (monotonic within a launch)
  unsigned int gen;     // unused (kept for the layout)
  int error;
  int polls;            // of a wait, at most (0: kSpinLimit)
};

// the launch's report, written by the kernel into the workspace (the public layout)
using SolveOut = cpfem_solve_report_t;
static_assert(sizeof(SolveOut) == 72 && offsetof(SolveOut, true_rs) == 56, "solve report layout");

// cpfem_krylov_opts_t.flags: also form the true residual of the returned x; report
// asynchronously instead of waiting for the solve
constexpr int kKrylovTrueResidual = 1;
constexpr int kKrylovDeferred = 2;
static_assert(kPointCounterBytes + kPointCellBytes <= sizeof(double) * 2 * 4 * kMaxBlocks,
              "the barrier counters and reduction cells fit in the partials");

static thread_local SolveOut g_last_solve = {0, 0, 0.0, 0.0, 0.0, 0.0, 0.0, 0, 0, -1.0, 0.0};

struct KWork {
  GridSync* sync;
  SolveOut* out;
  double* partials;   // 2 buffers x 4 values x kMaxBlocks
  double *r, *rhat, *p, *q, *s, *t, *phat, *shat, *minv;
};

static constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Bytes carve() lays out for n_nodes nodes, as a compile-time expression (the fixed scratch
// of the allocation-free entry point is checked against it when the library is built).
static constexpr size_t carve_bytes(int64_t n_nodes) {
  return align256(sizeof(GridSync)) + align256(sizeof(SolveOut)) + align256(sizeof(double) * 2 * 4 * kMaxBlocks) +
         8 * align256(sizeof(double) * 3 * (size_t)n_nodes) + align256(sizeof(double) * 9 * (size_t)n_nodes);
}

static size_t carve(void* base, int64_t n_nodes, KWork* w) {
  const int64_t n = 3 * n_nodes;
  char* p = (char*)base;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + off : nullptr;
    off += align256(bytes);
    return q;
  };
  KWork tmp;
  tmp.sync = (GridSync*)take(sizeof(GridSync));
  tmp.out = (SolveOut*)take(sizeof(SolveOut));
  tmp.partials = (double*)take(sizeof(double) * 2 * 4 * kMaxBlocks);
  double** vecs[] = {&tmp.r, &tmp.rhat, &tmp.p, &tmp.q, &tmp.s, &tmp.t, &tmp.phat, &tmp.shat};
  for (double** v : vecs) *v = (double*)take(sizeof(double) * n);
  tmp.minv = (double*)take(sizeof(double) * 9 * n_nodes);
  if (w) *w = tmp;
  return off;
}

// Three rows of node a of A x (or A^T x), in the precision R of the values and x (FP64 for
// the Krylov iteration, FP32 inside a single-precision V-cycle).  COHERENT selects L2
// loads for x, needed when x was written by other blocks earlier in the same launch.
template <bool TRANS, bool COHERENT, typename R, typename VT = R>
__device__ __forceinline__ void sell_rows(const cpfem_sell_t& L, const VT* __restrict__ vals,
                                          const R* x, int64_t a, R* acc) {
  const int64_t g = a >> 5;
  const int lane = (int)(a & 31);
  const int64_t c0 = L.group_off[g] + lane;
  const VT* v0 = vals + 9 * L.group_off[g] + lane;
  const int w = L.group_width[g];
  // two accumulators per row (even / odd slots): six independent FMA chains keep the FP64
  // pipe fed at one thread per node
  R e0 = R(0), e1 = R(0), e2 = R(0), o0 = R(0), o1 = R(0), o2 = R(0);
  auto slot = [&](int j, R& a0, R& a1, R& a2) {
    const int64_t b = __ldg(&L.cols[c0 + 32 * j]);
    R x0, x1, x2;
    if (COHERENT) {
      x0 = __ldcg(&x[3 * b]); x1 = __ldcg(&x[3 * b + 1]); x2 = __ldcg(&x[3 * b + 2]);
    } else {
      x0 = __ldg(&x[3 * b]); x1 = __ldg(&x[3 * b + 1]); x2 = __ldg(&x[3 * b + 2]);
    }
    if (!TRANS) {
      const VT* vj = v0 + 288 * j;
      a0 = mad(opval<R>(__ldg(&vj[0])), x0, mad(opval<R>(__ldg(&vj[32])), x1, mad(opval<R>(__ldg(&vj[64])), x2, a0)));
      a1 = mad(opval<R>(__ldg(&vj[96])), x0, mad(opval<R>(__ldg(&vj[128])), x1, mad(opval<R>(__ldg(&vj[160])), x2, a1)));
      a2 = mad(opval<R>(__ldg(&vj[192])), x0, mad(opval<R>(__ldg(&vj[224])), x1, mad(opval<R>(__ldg(&vj[256])), x2, a2)));
    } else {
      // A^T[3a+i][3b+k] = A[3b+k][3a+i]: node b, slot tpos, row k, column i
      const int64_t tp = __ldg(&L.tpos[c0 + 32 * j]);
      const VT* vb = vals + 9 * L.group_off[b >> 5] + (b & 31) + 288 * tp;
      a0 = mad(opval<R>(__ldg(&vb[0])), x0, mad(opval<R>(__ldg(&vb[96])), x1, mad(opval<R>(__ldg(&vb[192])), x2, a0)));
      a1 = mad(opval<R>(__ldg(&vb[32])), x0, mad(opval<R>(__ldg(&vb[128])), x1, mad(opval<R>(__ldg(&vb[224])), x2, a1)));
      a2 = mad(opval<R>(__ldg(&vb[64])), x0, mad(opval<R>(__ldg(&vb[160])), x1, mad(opval<R>(__ldg(&vb[256])), x2, a2)));
    }
  };
  int j = 0;
#pragma unroll 2
  for (; j + 1 < w; j += 2) {
    slot(j, e0, e1, e2);
    slot(j + 1, o0, o1, o2);
  }
  if (j < w) slot(j, e0, e1, e2);
  acc[0] = e0 + o0;
  acc[1] = e1 + o1;
  acc[2] = e2 + o2;
}

template <bool TRANS>
__global__ void __launch_bounds__(256) k_spmv(const cpfem_sell_t L, const double* __restrict__ vals,
                                              const double* __restrict__ x, double* __restrict__ y) {
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < L.num_nodes;
       a += (int64_t)gridDim.x * blockDim.x) {
    double acc[3];
    sell_rows<TRANS, false>(L, vals, x, a, acc);
    y[3 * a] = acc[0];
    y[3 * a + 1] = acc[1];
    y[3 * a + 2] = acc[2];
  }
}

__device__ __forceinline__ void apply_m(int precond, const double* __restrict__ minv, int64_t a,
                                        const double* v, double* out) {
  if (precond == 0) {
    out[0] = v[0]; out[1] = v[1]; out[2] = v[2];
  } else if (precond == 1) {
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = v[i] * minv[3 * a + i];
  } else {
    const double* bi = minv + 9 * a;
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = fma(bi[3 * i], v[0], fma(bi[3 * i + 1], v[1], bi[3 * i + 2] * v[2]));
  }
}

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add_u32(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Barrier over the nb blocks that share gs (the whole grid of a cooperative launch, or a
// team of it).  gs->count only grows (it is zeroed before the launch): the k-th barrier is
// complete when it reaches k*nb.  Thread 0 arrives with a release reduction, which
// publishes every write the block made before the __syncthreads, and waits with acquire
// loads; no reset is needed, so the last arrival costs no extra round trip.  The wait is
// bounded: after kSpinLimit polls (gs->polls, where that is set) the block records an error (also
// in *gerr) and returns false instead of hanging; on that error the others' waits and its own later
// ones end too.
__device__ __forceinline__ bool counted_barrier(GridSync* gs, unsigned int nb, unsigned int& gen, int* gerr) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int target = (gen + 1u) * nb;
    int ok = 1;
    red_release_add_u32(&gs->count, 1u);
    long long spins = 0;
    while (ld_acquire_u32(&gs->count) < target) {
      if ((++spins & 63) == 0 && (spins >= (gs->polls > 0 ? gs->polls : kSpinLimit) || *(volatile int*)&gs->error != 0)) {
        ok = 0;
        atomicExch(&gs->error, 1);
        if (gerr != nullptr) atomicExch(gerr, 1);
        break;
      }
      if (spins > 32) __nanosleep(32);
    }
    s_ok = ok && (*(volatile int*)&gs->error == 0);
  }
  __syncthreads();
  gen += 1u;
  return s_ok != 0;
}

__device__ __forceinline__ bool grid_barrier(GridSync* gs, unsigned int& gen) {
  return counted_barrier(gs, gridDim.x, gen, nullptr);
}

// Publish this block's NV partial sums, cross the grid barrier, and reduce all blocks'
// partials in a fixed order (the same in every block).  Returns false on barrier error.
template <int NV>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], double* partials, GridSync* gs, unsigned int& gen,
                                            double* smem, double* bcast) {
  block_sum<NV>(v, smem);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) partials[k * gridDim.x + blockIdx.x] = v[k];
  const bool ok = grid_barrier(gs, gen);
  if (threadIdx.x < 32) {
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) acc[k] = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 32)
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] += __ldcg(&partials[k * gridDim.x + b]);
    warp_sum<NV>(acc);
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) bcast[k] = acc[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = bcast[k];
  __syncthreads();
  return ok;
}

// One V-cycle out = M^-1 in of the streaming kernel, in precision R, level 0 a thread per node: node
// a is thread a's of the grid, as in the rest of the kernel, so `in` and `out` need no barrier of
// their own.  b: room for 3 kMgDenseNodes values in shared memory.
template <bool TRANS, typename R>
__device__ __forceinline__ void mg_vcycle_streaming(const cpfem_mg_t& mg, const double* vals, const double* in, double* out,
                                                    R* b, int lb, GridSync* gs, unsigned int& gen, bool& ok) {
  const MgArrays<R> A{mg, vals};
  const cpfem_sell_t& S = mg.sell[0];
  const R* Mi = A.minv(0);
  const R om = (R)mg.omega;
  const int64_t n = S.num_nodes, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto barrier = [&]() { ok = grid_barrier(gs, gen) && ok; };
  // X + om D^-1 (in - A X) at node a
  auto sweep = [&](const R* X, int64_t a, R* z) {
    R acc[3], r[3];
    sell_rows<TRANS, true, R, double>(S, vals, X, a, acc);
#pragma unroll
    for (int i = 0; i < 3; ++i) r[i] = to_prec<R>(in[3 * a + i]) - acc[i];
    mg_apply_minv<TRANS>(Mi, a, r, z);
#pragma unroll
    for (int i = 0; i < 3; ++i) z[i] = mad(om, z[i], __ldcg(&X[3 * a + i]));
  };
  R *X = A.x(0), *T = A.t(0);
  for (int64_t a = t0; a < n; a += stride) {
    R v[3], z[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = to_prec<R>(in[3 * a + i]);
    mg_apply_minv<TRANS>(Mi, a, v, z);
#pragma unroll
    for (int i = 0; i < 3; ++i) X[3 * a + i] = om * z[i];
  }
  for (int k = 1; k < mg.pre_sweeps; ++k) {
    barrier();
    for (int64_t a = t0; a < n; a += stride) {
      R z[3];
      sweep(X, a, z);
#pragma unroll
      for (int i = 0; i < 3; ++i) T[3 * a + i] = z[i];
    }
    R* tmp = X; X = T; T = tmp;
  }
  barrier();
  R* Res = A.r(0);
  for (int64_t a = t0; a < n; a += stride) {
    R acc[3];
    sell_rows<TRANS, true, R, double>(S, vals, X, a, acc);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const R rv = to_prec<R>(in[3 * a + i]) - acc[i];
      Res[3 * a + i] = (mg.free_dof != nullptr && mg.free_dof[3 * a + i] == 0) ? R(0) : rv;
    }
  }
  barrier();
  const R* X1 = mg_coarse_levels<TRANS, R>(mg, A, lb, t0 >> 2, stride >> 2, (int)(t0 & 3), blockIdx.x, gridDim.x, b, barrier);
  barrier();
  mg_prolong(mg, 0, X, X1, t0, stride, n);
  for (int k = 0; k < mg.post_sweeps; ++k) {
    barrier();
    for (int64_t a = t0; a < n; a += stride) {
      R z[3];
      sweep(X, a, z);
#pragma unroll
      for (int i = 0; i < 3; ++i) T[3 * a + i] = z[i];
    }
    R* tmp = X; X = T; T = tmp;
  }
  for (int64_t a = t0; a < n; a += stride)
#pragma unroll
    for (int i = 0; i < 3; ++i) out[3 * a + i] = to_f64(X[3 * a + i]);
}

// The streaming kernel, for systems too large for the shared-memory one (krylov_team.cuh): one
// thread per node, vectors in the workspace.  Three blocks a SM, six warps per sub-partition, hide
// the row products' loads; with the FP32 V-cycle one block of the whole register file does that
// better.  RESTARTS: max_restarts > 0; where the code that forms b - A x again is compiled in, an
// iteration at 56^3 cells takes 237 us instead of 226.  MR: void for a point preconditioner (precond), or the
// V-cycle's precision.
template <bool TRANS, bool RESTARTS, typename MR, typename MG>
__global__ void __launch_bounds__(kPThreads, std::is_same<MR, float>::value ? 1 : 3) k_bicgstab(
    const cpfem_sell_t L, const double* __restrict__ vals, const double* __restrict__ b, double* __restrict__ x,
    KWork w, int precond, double tol, double atol, int maxiter, int max_restarts, const __grid_constant__ MG mg) {
  constexpr bool kMg = !std::is_void<MR>::value;
  __shared__ double smem[4 * 32];
  __shared__ double bcast[4];
  const int64_t n = L.num_nodes;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned int gen = 0u;
  int buf = 0;
  auto parts = [&]() {
    double* p = w.partials + (size_t)buf * 4 * kMaxBlocks;
    buf ^= 1;
    return p;
  };
  bool ok = true;
  __shared__ double drift;     // ||b - A x||^2 where the last drift was seen
  if (threadIdx.x == 0) drift = INFINITY;
  // out = M v at this thread's nodes, by the V-cycle
  __shared__ double dense_b[kMg ? 3 * kMgDenseNodes : 1];
  __shared__ int lb;
  if constexpr (kMg) {
    if (threadIdx.x == 0) lb = mg_dense_from<MR>(mg);
    __syncthreads();
  }
  auto vcycle = [&](const double* v, double* out) {
    if constexpr (kMg)
      mg_vcycle_streaming<TRANS, MR>(mg, vals, v, out, reinterpret_cast<MR*>(dense_b), lb, w.sync, gen, ok);
  };

  // r = b - A x0 ; rhat = p = q = r
  double v2[2] = {0.0, 0.0};
  for (int64_t a = t0; a < n; a += stride) {
    double acc[3];
    sell_rows<TRANS, true>(L, vals, x, a, acc);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int64_t d = 3 * a + i;
      const double bv = b[d];
      const double rv = bv - acc[i];
      w.r[d] = rv; w.rhat[d] = rv; w.p[d] = rv; w.q[d] = rv;
      v2[0] = fma(bv, bv, v2[0]);
      v2[1] = fma(rv, rv, v2[1]);
    }
  }
  ok = grid_reduce<2>(v2, parts(), w.sync, gen, smem, bcast) && ok;
  const double atol2 = fmax(tol * tol * v2[0], atol * atol);
  if (blockIdx.x == 0 && threadIdx.x == 0) w.out->bb = v2[0];   // b.b, written now: nothing stays live
  double cap = 0.0;
  if constexpr (std::is_same<MR, float>::value) cap = 1e16 * fmax(v2[1], atol2);
  double rs = v2[1], rho_new = v2[1], rho = 1.0, alpha = 1.0, omega = 1.0;
  int k = 0, restarts = 0;

  while (ok && rs > atol2 && k < maxiter && k >= 0) {
    const double beta = rho_new / rho * alpha / omega;
    // p = r + beta (p - omega q); phat = M p
    for (int64_t a = t0; a < n; a += stride) {
      double pv[3], ph[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        pv[i] = w.r[d] + beta * (w.p[d] - omega * w.q[d]);
        w.p[d] = pv[i];
      }
      if constexpr (!kMg) {
        apply_m(precond, w.minv, a, pv, ph);
#pragma unroll
        for (int i = 0; i < 3; ++i) w.phat[3 * a + i] = ph[i];
      }
    }
    vcycle(w.p, w.phat);
    ok = grid_barrier(w.sync, gen) && ok;
    // q = A phat ; alpha = rho_new / (rhat . q)
    double v1[1] = {0.0};
    for (int64_t a = t0; a < n; a += stride) {
      double acc[3];
      sell_rows<TRANS, true>(L, vals, w.phat, a, acc);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        w.q[d] = acc[i];
        v1[0] = fma(w.rhat[d], acc[i], v1[0]);
      }
    }
    ok = grid_reduce<1>(v1, parts(), w.sync, gen, smem, bcast) && ok;
    alpha = rho_new / v1[0];
    // s = r - alpha q ; shat = M s ; exit_early = s.s < atol2
    double vs[1] = {0.0};
    for (int64_t a = t0; a < n; a += stride) {
      double sv[3], sh[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        sv[i] = w.r[d] - alpha * w.q[d];
        w.s[d] = sv[i];
        vs[0] = fma(sv[i], sv[i], vs[0]);
      }
      if constexpr (!kMg) {
        apply_m(precond, w.minv, a, sv, sh);
#pragma unroll
        for (int i = 0; i < 3; ++i) w.shat[3 * a + i] = sh[i];
      }
    }
    vcycle(w.s, w.shat);
    ok = grid_reduce<1>(vs, parts(), w.sync, gen, smem, bcast) && ok;   // also the shat halo barrier
    // t = A shat ; omega = (t.s)/(t.t)
    double vt[2] = {0.0, 0.0};
    for (int64_t a = t0; a < n; a += stride) {
      double acc[3];
      sell_rows<TRANS, true>(L, vals, w.shat, a, acc);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        w.t[d] = acc[i];
        vt[0] = fma(acc[i], w.s[d], vt[0]);
        vt[1] = fma(acc[i], acc[i], vt[1]);
      }
    }
    ok = grid_reduce<2>(vt, parts(), w.sync, gen, smem, bcast) && ok;
    const bool early = vs[0] < atol2;
    omega = vt[0] / vt[1];
    // x and r update
    double vr[2] = {0.0, 0.0};
    for (int64_t a = t0; a < n; a += stride) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        double rv;
        if (early) {
          x[d] = x[d] + alpha * w.phat[d];
          rv = w.s[d];
        } else {
          x[d] = x[d] + (alpha * w.phat[d] + omega * w.shat[d]);
          rv = w.s[d] - omega * w.t[d];
        }
        w.r[d] = rv;
        vr[0] = fma(rv, rv, vr[0]);
        vr[1] = fma(w.rhat[d], rv, vr[1]);
      }
    }
    ok = grid_reduce<2>(vr, parts(), w.sync, gen, smem, bcast) && ok;
    int kn = (omega == 0.0 || alpha == 0.0) ? -11 : k + 1;
    if (rho_new == 0.0) kn = -10;
    rho = rho_new;
    rho_new = vr[1];
    rs = vr[0];
    if (std::is_same<MR, float>::value && !(rs <= cap)) kn = -12;      // as in k_bicgstab_team
    // With restarts allowed: at a breakdown, and where the recursive residual met the stop rule but
    // the true one is ten times above it and half what it was there last, restart at the current x (rhat = p = q = r = b - A x; x is
    // complete: the last reduction crossed the grid barrier after every block wrote its part).
    if (RESTARTS && restarts < max_restarts && ok && (kn < 0 ? kn != -12 && rs > atol2 : rs <= atol2 && kn < maxiter)) {
      double v3[1] = {0.0};
      for (int64_t a = t0; a < n; a += stride) {
        double acc[3];
        sell_rows<TRANS, true>(L, vals, x, a, acc);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          const double rv = b[d] - acc[i];
          w.r[d] = rv; w.rhat[d] = rv; w.p[d] = rv; w.q[d] = rv;
          v3[0] = fma(rv, rv, v3[0]);
        }
      }
      ok = grid_reduce<1>(v3, parts(), w.sync, gen, smem, bcast) && ok;
      const bool again = kn < 0 || (v3[0] > 100.0 * atol2 && 4.0 * v3[0] < drift);
      __syncthreads();
      if (kn >= 0 && threadIdx.x == 0) drift = v3[0];
      if (again) {
        ++restarts;
        rs = v3[0];
        rho_new = v3[0];
        rho = alpha = omega = 1.0;
      }
      k = k + 1;
    } else {
      k = kn;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.out->true_rs = -1.0;
    w.out->restarts = restarts;
    w.out->k = k;
    w.out->error = ok ? 0 : 1;
    w.out->rs = rs;
    w.out->atol2 = atol2;
    w.out->rho = rho;
    w.out->alpha = alpha;
    w.out->omega = omega;
  }
}

// ||b - A x||^2 in block partials (fixed grid, fixed order inside a block).
template <bool TRANS>
__global__ void __launch_bounds__(kVecThreads) k_true_residual(const cpfem_sell_t L, const double* __restrict__ vals,
                                                               const double* __restrict__ b,
                                                               const double* __restrict__ x, double* partials) {
  __shared__ double smem[4 * 32];
  double v[1] = {0.0};
  for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < L.num_nodes;
       a += (int64_t)gridDim.x * blockDim.x) {
    double acc[3];
    sell_rows<TRANS, false>(L, vals, x, a, acc);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double r = b[3 * a + i] - acc[i];
      v[0] = fma(r, r, v[0]);
    }
  }
  block_sum<1>(v, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = v[0];
}

__global__ void k_sum_partials(const double* __restrict__ partials, int n, double* out) {
  double v[1] = {0.0};
  for (int i = threadIdx.x; i < n; i += 32) v[0] += partials[i];
  warp_sum<1>(v);
  if (threadIdx.x == 0) *out = v[0];
}

static int sm_count_and_blocks(const void* fn, int* blocks_per_sm, int* sms) {
  int dev = 0;
  CPFEM_CUDA_TRY(cudaGetDevice(&dev));
  CPFEM_CUDA_TRY(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
  CPFEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, kPThreads, 0));
  return CPFEM_OK;
}

// The launch's report: copied to the caller's pinned memory behind the solve (deferred: read
// after its next synchronisation of the stream), or waited for here.
static int finish_solve(const SolveOut* dev_out, int32_t* info, int flags, cpfem_solve_report_t* report,
                        cudaStream_t s) {
  if (flags & kKrylovDeferred) {
    CPFEM_CUDA_TRY(cudaMemcpyAsync(report, dev_out, sizeof(SolveOut), cudaMemcpyDeviceToHost, s));
    return CPFEM_OK;
  }
  SolveOut out;
  CPFEM_CUDA_TRY(cudaMemcpyAsync(&out, dev_out, sizeof(SolveOut), cudaMemcpyDeviceToHost, s));
  CPFEM_CUDA_TRY(cudaStreamSynchronize(s));
  info[0] = out.k;
  info[1] = (out.rs <= out.atol2) ? 1 : 0;
  g_last_solve = out;
  if (out.error) {
    set_error("BiCGSTAB grid barrier timed out");
    return CPFEM_ERR_SOLVE;
  }
  return CPFEM_OK;
}

template <bool TRANS>
static int run_bicgstab(const cpfem_sell_t& L, const double* vals, const double* b, double* x, int precond,
                        double tol, double atol, int32_t maxiter, void* workspace, int32_t* info, cudaStream_t s,
                        int max_restarts = 0, const cpfem_mg_t* mgp = nullptr, int grid_blocks = 0,
                        int flags = 0, cpfem_solve_report_t* report = nullptr, int lost_polls = 0) {
  KWork w;
  carve(workspace, L.num_nodes, &w);
  PointPlan plan{};
  if (const int rc = point_plan(L.num_nodes, precond, precond == 3 && mgp->precision == 1, TRANS, grid_blocks, &plan); rc != CPFEM_OK) return rc;
  if (plan.ok) {
    PointArgs a{};
    a.L = L; a.vals = vals; a.b = b; a.x = x;
    a.phat = w.phat; a.shat = w.shat;
    a.counters = (unsigned int*)w.partials;
    a.cells = w.partials + kPointCounterBytes / sizeof(double);
    a.error = &w.out->error;
    a.polls = lost_polls > 0 ? lost_polls : kPtSpinLimit;
    a.out = w.out;
    a.precond = precond; a.maxiter = maxiter; a.max_restarts = max_restarts;
    a.true_res = (flags & kKrylovTrueResidual) ? 1 : 0;
    a.tol = tol; a.atol = atol;
    // one memset over the report with its error word and the one team's counter (neighbours in
    // the workspace)
    CPFEM_CUDA_TRY(cudaMemsetAsync(w.sync, 0, (size_t)((char*)w.partials - (char*)w.sync) + 128, s));
    // the failure test: one arrival short (the count's first increment wraps it to 0)
    if (lost_polls > 0) CPFEM_CUDA_TRY(cudaMemsetAsync(a.counters, 0xFF, sizeof(unsigned int), s));
    const int rc = precond == 3 ? mg_launch(plan, TRANS, a, *mgp, s) : point_launch(plan, TRANS, a, s);
    if (rc != CPFEM_OK) return rc;
    return finish_solve(w.out, info, flags, report, s);
  }
  CPFEM_CUDA_TRY(cudaMemsetAsync(w.sync, 0, sizeof(GridSync), s));
  if (lost_polls > 0) {
    const GridSync short_one = {~0u, 0u, 0, lost_polls};
    CPFEM_CUDA_TRY(cudaMemcpyAsync(w.sync, &short_one, sizeof(short_one), cudaMemcpyHostToDevice, s));
  }
  if (precond == 1 || precond == 2) {
    k_precond_setup<TRANS><<<(unsigned)ceil_div(L.num_nodes, 128), 128, 0, s>>>(L, vals, precond, w.minv);
    CPFEM_CUDA_TRY(cudaGetLastError());
  }
  int per_sm = 0, sms = 0;
  const void* kfn = precond != 3 ? (max_restarts > 0 ? (const void*)k_bicgstab<TRANS, true, void, NoMg>
                                                     : (const void*)k_bicgstab<TRANS, false, void, NoMg>)
                    : mgp->precision == 1 ? (const void*)k_bicgstab<TRANS, true, float, cpfem_mg_t>
                                          : (const void*)k_bicgstab<TRANS, true, double, cpfem_mg_t>;
  int rc = sm_count_and_blocks(kfn, &per_sm, &sms);
  if (rc) return rc;
  if (per_sm < 1) {
    set_error("persistent BiCGSTAB kernel cannot be resident");
    return CPFEM_ERR_CUDA;
  }
  int64_t blocks = std::min<int64_t>((int64_t)per_sm * sms, ceil_div(L.num_nodes, kPThreads));
  if (grid_blocks > 0) blocks = std::min<int64_t>((int64_t)per_sm * sms, grid_blocks);
  blocks = std::max<int64_t>(1, std::min<int64_t>(blocks, kMaxBlocks));
  cpfem_sell_t Lc = L;
  const double* bb = b;
  double* xx = x;
  int pc = precond;
  double tl = tol, at = atol;
  int mi = maxiter, mr = max_restarts;
  cpfem_mg_t mg{};
  if (precond == 3) mg = *mgp;
  void* args[] = {&Lc, &vals, &bb, &xx, &w, &pc, &tl, &at, &mi, &mr, &mg};
  CPFEM_CUDA_TRY(cudaLaunchCooperativeKernel(kfn, dim3((unsigned)blocks), dim3(kPThreads), args, 0, s));
  if (flags & kKrylovTrueResidual) {
    // ||b - A x||^2 of the returned x: block partials, then one block sums them in order
    // (deterministic), into the SolveOut read below -- no extra synchronisation
    k_true_residual<TRANS><<<kVecBlocks, kVecThreads, 0, s>>>(L, vals, b, x, w.partials);
    CPFEM_CUDA_TRY(cudaGetLastError());
    k_sum_partials<<<1, 32, 0, s>>>(w.partials, kVecBlocks, &w.out->true_rs);
    CPFEM_CUDA_TRY(cudaGetLastError());
  }
  return finish_solve(w.out, info, flags, report, s);
}

}  // namespace cpfem

using namespace cpfem;

extern "C" {

int cpfem_spmv(const cpfem_sell_t* sell, const double* values, const double* x, double* y, int32_t transpose,
               void* stream) {
  CPFEM_REQUIRE(sell_ok(sell) && values && x && y, "bad spmv arguments");
  CPFEM_REQUIRE(!transpose || sell->tpos, "transpose needs tpos");
  if (sell->num_nodes == 0) return CPFEM_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(sell->num_nodes, 256), 8 * 152);
  if (transpose)
    k_spmv<true><<<blocks, 256, 0, (cudaStream_t)stream>>>(*sell, values, x, y);
  else
    k_spmv<false><<<blocks, 256, 0, (cudaStream_t)stream>>>(*sell, values, x, y);
  CPFEM_CUDA_TRY(cudaGetLastError());
  return CPFEM_OK;
}

size_t cpfem_bicgstab_workspace_bytes(int32_t num_nodes) { return carve(nullptr, num_nodes, nullptr); }

int cpfem_bicgstab_last_stats(double* out) {
  CPFEM_REQUIRE(out != nullptr, "out is null");
  out[0] = (double)g_last_solve.k;
  out[1] = g_last_solve.rs;
  out[2] = g_last_solve.atol2;
  out[3] = g_last_solve.rho;
  out[4] = g_last_solve.alpha;
  out[5] = g_last_solve.omega;
  out[6] = (double)g_last_solve.restarts;
  return CPFEM_OK;
}

int cpfem_bicgstab_last_stats_ex(double* out, int32_t n) {
  CPFEM_REQUIRE(out != nullptr && n >= 0, "bad stats arguments");
  const double v[9] = {(double)g_last_solve.k, g_last_solve.rs, g_last_solve.atol2, g_last_solve.rho,
                       g_last_solve.alpha, g_last_solve.omega, (double)g_last_solve.restarts,
                       g_last_solve.true_rs, g_last_solve.bb};
  for (int32_t i = 0; i < n && i < 9; ++i) out[i] = v[i];
  return CPFEM_OK;
}

static int solve_checked(const cpfem_sell_t* sell, const double* values, const double* b, double* x,
                         const cpfem_krylov_opts_t* opts, void* workspace, int32_t* info, void* stream,
                         int lost_polls) {
  CPFEM_REQUIRE(info != nullptr, "info is null");
  info[0] = 0;
  info[1] = 1;
  CPFEM_REQUIRE(opts != nullptr, "opts is null");
  CPFEM_REQUIRE(sell_ok(sell), "bad layout");
  if (sell->num_nodes == 0) return CPFEM_OK;
  CPFEM_REQUIRE(values && b && x && workspace, "bad bicgstab arguments");
  CPFEM_REQUIRE(((uintptr_t)workspace & 255) == 0, "workspace must be 256-byte aligned");
  CPFEM_REQUIRE(opts->precond >= 0 && opts->precond <= 3, "precond must be 0, 1, 2 or 3");
  if (opts->precond == 3) {
    CPFEM_REQUIRE(!opts->transpose || sell->tpos != nullptr, "a transposed multigrid solve needs tpos");
    const int rc = mg_check(opts->mg, sell);
    if (rc != CPFEM_OK) return rc;
  }
  CPFEM_REQUIRE(opts->maxiter >= 0, "maxiter must be >= 0");
  CPFEM_REQUIRE(opts->max_restarts >= 0, "max_restarts must be >= 0");
  CPFEM_REQUIRE(opts->grid_blocks >= 0, "grid_blocks must be >= 0");
  CPFEM_REQUIRE(!opts->transpose || sell->tpos != nullptr, "transpose needs tpos");
  CPFEM_REQUIRE(!(opts->flags & kKrylovDeferred) || opts->report != nullptr, "a deferred report needs opts.report");
  cudaStream_t s = (cudaStream_t)stream;
  if (opts->transpose)
    return run_bicgstab<true>(*sell, values, b, x, opts->precond, opts->tol, opts->atol, opts->maxiter, workspace,
                              info, s, opts->max_restarts, opts->mg, opts->grid_blocks, opts->flags, opts->report,
                              lost_polls);
  return run_bicgstab<false>(*sell, values, b, x, opts->precond, opts->tol, opts->atol, opts->maxiter, workspace,
                             info, s, opts->max_restarts, opts->mg, opts->grid_blocks, opts->flags, opts->report,
                             lost_polls);
}

int cpfem_bicgstab_ex(const cpfem_sell_t* sell, const double* values, const double* b, double* x,
                      const cpfem_krylov_opts_t* opts, void* workspace, int32_t* info, void* stream) {
  return solve_checked(sell, values, b, x, opts, workspace, info, stream, 0);
}

int cpfem_probe_lost_block(const cpfem_sell_t* sell, const double* values, const double* b, double* x,
                           const cpfem_krylov_opts_t* opts, int32_t polls, void* workspace, int32_t* info,
                           void* stream) {
  CPFEM_REQUIRE(info != nullptr, "info is null");
  CPFEM_REQUIRE(polls >= 1 && polls <= (1 << 20), "bad probe arguments");
  return solve_checked(sell, values, b, x, opts, workspace, info, stream, polls);
}

int cpfem_bicgstab(const cpfem_sell_t* sell, const double* values, const double* b, double* x, int32_t precond,
                   int32_t transpose, double tol, double atol, int32_t maxiter, void* workspace, int32_t* info,
                   void* stream) {
  CPFEM_REQUIRE(precond >= 0 && precond <= 2, "precond must be 0, 1 or 2 (multigrid: cpfem_bicgstab_ex)");
  const cpfem_krylov_opts_t o = {precond, transpose, maxiter, 0, tol, atol, nullptr, 0, 0, nullptr};
  return cpfem_bicgstab_ex(sell, values, b, x, &o, workspace, info, stream);
}

}  // extern "C"

// ---- ragged batch: teams of blocks, one instance per team --------------------------------
// A ragged batch (instances of very different sizes and iteration counts) is split over the
// co-resident blocks of one cooperative launch.  When the batch has no more instances than
// blocks, every instance gets a team of consecutive blocks sized by its estimated work
// (nodes x expected iterations), so a 24^3 RVE and an 8^3 RVE finish at about the same
// time; a team crosses its dependencies with its own bounded barrier and reduces its dot
// products in a fixed block order.  With more instances than blocks, every block is a team
// of one that pulls instances from a queue, largest first.
namespace cpfem {

constexpr int kMinNodesPerBlock = 256;

struct RTeam {
  int first;   // first block of the team
  int nb;      // blocks in the team
  int job;     // the team's job, or -1: pull jobs from the queue (nb == 1)
  int pad;
};

struct RJob {
  int inst;
  int pad;
  int64_t n0, n1;
};

struct RWork {
  double *r, *rhat, *p, *q, *s, *t, *phat, *shat, *minv;
  double* partials;      // 2 buffers x 4 values x kMaxBlocks, by block id
  int* team_of_block;    // kMaxBlocks
  RTeam* teams;          // kMaxBlocks
  GridSync* tsync;       // one barrier per team
  RJob* jobs;            // at most num_nodes (every listed instance owns a node)
  int32_t* info;         // 2 per job
  unsigned int* queue;
  int* error;
};

static size_t carve_ragged(void* base, int64_t n_nodes, RWork* w) {
  const int64_t n = 3 * n_nodes;
  const int64_t nj = std::max<int64_t>(n_nodes, 1);
  char* p = (char*)base;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = p ? p + off : nullptr;
    off += align256(bytes);
    return q;
  };
  RWork tmp;
  double** vecs[] = {&tmp.r, &tmp.rhat, &tmp.p, &tmp.q, &tmp.s, &tmp.t, &tmp.phat, &tmp.shat};
  for (double** v : vecs) *v = (double*)take(sizeof(double) * n);
  tmp.minv = (double*)take(sizeof(double) * 9 * n_nodes);
  tmp.partials = (double*)take(sizeof(double) * 2 * 4 * kMaxBlocks);
  tmp.team_of_block = (int*)take(sizeof(int) * kMaxBlocks);
  tmp.teams = (RTeam*)take(sizeof(RTeam) * kMaxBlocks);
  tmp.tsync = (GridSync*)take(sizeof(GridSync) * kMaxBlocks);
  tmp.jobs = (RJob*)take(sizeof(RJob) * nj);
  tmp.info = (int32_t*)take(sizeof(int32_t) * 2 * nj);
  tmp.queue = (unsigned int*)take(sizeof(unsigned int));
  tmp.error = (int*)take(sizeof(int));
  if (w) *w = tmp;
  return off;
}

__device__ __forceinline__ bool team_barrier(GridSync* gs, unsigned int nb, unsigned int& gen, int* gerr) {
  return counted_barrier(gs, nb, gen, gerr);
}

// Team-wide sums of NV values: block sum, then (teams of several blocks) publish, barrier
// and add the team's partials in block order.  Every block of the team gets the same bits.
template <int NV>
__device__ __forceinline__ bool team_reduce(double (&v)[NV], double* partials, int first, int nb, GridSync* gs,
                                            unsigned int& gen, int* gerr, double* smem, double* bcast) {
  block_sum<NV>(v, smem);
  bool ok = true;
  if (nb == 1) {
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) bcast[k] = v[k];
  } else {
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) partials[k * kMaxBlocks + blockIdx.x] = v[k];
    ok = team_barrier(gs, (unsigned)nb, gen, gerr);
    if (threadIdx.x < 32) {
      double acc[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) acc[k] = 0.0;
      for (int b = first + (int)threadIdx.x; b < first + nb; b += 32)
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k] += __ldcg(&partials[k * kMaxBlocks + b]);
      warp_sum<NV>(acc);
      if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) bcast[k] = acc[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = bcast[k];
  __syncthreads();
  return ok;
}

__global__ void __launch_bounds__(kPThreads, 4) k_bicgstab_ragged(
    const cpfem_sell_t L, const double* __restrict__ vals, const double* __restrict__ b, double* __restrict__ x,
    RWork w, int precond, double tol, double atol, int maxiter, int n_jobs) {
  __shared__ double smem[4 * 32];
  __shared__ double bcast[4];
  __shared__ int s_job;
  const int team = w.team_of_block[blockIdx.x];
  const RTeam tm = w.teams[team];
  GridSync* gs = w.tsync + team;
  const int nb = tm.nb, first = tm.first;
  const int64_t tid = (int64_t)(blockIdx.x - first) * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)nb * blockDim.x;
  unsigned int gen = 0u;
  int buf = 0;
  auto parts = [&]() {
    double* p = w.partials + (size_t)buf * 4 * kMaxBlocks;
    buf ^= 1;
    return p;
  };
  bool ok = true;
  for (int pass = 0; ok; ++pass) {
    int job;
    if (tm.job >= 0) {
      if (pass > 0) break;
      job = tm.job;
    } else {
      if (threadIdx.x == 0) s_job = (int)atomicAdd(w.queue, 1u);
      __syncthreads();
      job = s_job;
      __syncthreads();
    }
    if (job >= n_jobs) break;
    const RJob jb = w.jobs[job];
    const int64_t n0 = jb.n0, n1 = jb.n1;
    const int64_t a0 = ((n0 >> 5) << 5) + tid;   // group-aligned: a warp reads one sliced-ELL group

    double v2[2] = {0.0, 0.0};
    for (int64_t a = a0; a < n1; a += stride) {
      if (a < n0) continue;
      double acc[3];
      sell_rows<false, true>(L, vals, x, a, acc);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int64_t d = 3 * a + i;
        const double bv = b[d];
        const double rv = bv - acc[i];
        w.r[d] = rv; w.rhat[d] = rv; w.p[d] = rv; w.q[d] = rv;
        v2[0] = fma(bv, bv, v2[0]);
        v2[1] = fma(rv, rv, v2[1]);
      }
    }
    ok = team_reduce<2>(v2, parts(), first, nb, gs, gen, w.error, smem, bcast) && ok;
    const double atol2 = fmax(tol * tol * v2[0], atol * atol);
    double rs = v2[1], rho_new = v2[1], rho = 1.0, alpha = 1.0, omega = 1.0;
    int k = 0;
    while (ok && rs > atol2 && k < maxiter && k >= 0) {
      const double beta = rho_new / rho * alpha / omega;
      for (int64_t a = a0; a < n1; a += stride) {
        if (a < n0) continue;
        double pv[3], ph[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          pv[i] = w.r[d] + beta * (w.p[d] - omega * w.q[d]);
          w.p[d] = pv[i];
        }
        apply_m(precond, w.minv, a, pv, ph);
#pragma unroll
        for (int i = 0; i < 3; ++i) w.phat[3 * a + i] = ph[i];
      }
      if (nb > 1) ok = team_barrier(gs, (unsigned)nb, gen, w.error) && ok;
      else __syncthreads();
      double v1[1] = {0.0};
      for (int64_t a = a0; a < n1; a += stride) {
        if (a < n0) continue;
        double acc[3];
        sell_rows<false, true>(L, vals, w.phat, a, acc);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          w.q[d] = acc[i];
          v1[0] = fma(w.rhat[d], acc[i], v1[0]);
        }
      }
      ok = team_reduce<1>(v1, parts(), first, nb, gs, gen, w.error, smem, bcast) && ok;
      alpha = rho_new / v1[0];
      double vs[1] = {0.0};
      for (int64_t a = a0; a < n1; a += stride) {
        if (a < n0) continue;
        double sv[3], sh[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          sv[i] = w.r[d] - alpha * w.q[d];
          w.s[d] = sv[i];
          vs[0] = fma(sv[i], sv[i], vs[0]);
        }
        apply_m(precond, w.minv, a, sv, sh);
#pragma unroll
        for (int i = 0; i < 3; ++i) w.shat[3 * a + i] = sh[i];
      }
      ok = team_reduce<1>(vs, parts(), first, nb, gs, gen, w.error, smem, bcast) && ok;
      const bool early = vs[0] < atol2;
      double vt[2] = {0.0, 0.0};
      for (int64_t a = a0; a < n1; a += stride) {
        if (a < n0) continue;
        double acc[3];
        sell_rows<false, true>(L, vals, w.shat, a, acc);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          w.t[d] = acc[i];
          vt[0] = fma(acc[i], w.s[d], vt[0]);
          vt[1] = fma(acc[i], acc[i], vt[1]);
        }
      }
      ok = team_reduce<2>(vt, parts(), first, nb, gs, gen, w.error, smem, bcast) && ok;
      omega = vt[0] / vt[1];
      double vr[2] = {0.0, 0.0};
      for (int64_t a = a0; a < n1; a += stride) {
        if (a < n0) continue;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int64_t d = 3 * a + i;
          double rv;
          if (early) {
            x[d] = x[d] + alpha * w.phat[d];
            rv = w.s[d];
          } else {
            x[d] = x[d] + (alpha * w.phat[d] + omega * w.shat[d]);
            rv = w.s[d] - omega * w.t[d];
          }
          w.r[d] = rv;
          vr[0] = fma(rv, rv, vr[0]);
          vr[1] = fma(w.rhat[d], rv, vr[1]);
        }
      }
      ok = team_reduce<2>(vr, parts(), first, nb, gs, gen, w.error, smem, bcast) && ok;
      int kn = (omega == 0.0 || alpha == 0.0) ? -11 : k + 1;
      if (rho_new == 0.0) kn = -10;
      k = kn;
      rho = rho_new;
      rho_new = vr[1];
      rs = vr[0];
    }
    if ((int)blockIdx.x == first && threadIdx.x == 0) {
      w.info[2 * job] = k;
      w.info[2 * job + 1] = (rs <= atol2) ? 1 : 0;
    }
  }
}

// Teams of the shared-memory kernel, one per job: a block each, and then one after another to the
// team with the most work per block (at most one per kMinPointNodes nodes).  Not used (plan->ok =
// false) where that leaves a job's vectors too large for its blocks, or with more than half as many
// jobs as SMs: then the FP64 pipe is busy anyway and the streaming kernel's four blocks per
// SM hide more latency.
constexpr int64_t kMinPointNodes = 16;

static int ragged_point_plan(const std::vector<RJob>& jobs, const std::vector<double>& wts, int precond,
                             PointPlan* plan, std::vector<PointTeam>* teams, std::vector<int>* team_of_block) {
  plan->ok = false;
  int sms = 0;
  const int rc = point_max_blocks(&sms);
  if (rc != CPFEM_OK) return rc;
  const int nj = (int)jobs.size();
  if (2 * nj > sms) return CPFEM_OK;
  auto nodes = [&](int j) { return jobs[(size_t)j].n1 - jobs[(size_t)j].n0; };
  std::vector<int64_t> k((size_t)nj, 1);
  for (int left = sms - nj; left > 0; --left) {
    int best = -1;
    for (int j = 0; j < nj; ++j)
      if (k[(size_t)j] < ceil_div(nodes(j), kMinPointNodes) &&
          (best < 0 || wts[(size_t)j] / (double)k[(size_t)j] > wts[(size_t)best] / (double)k[(size_t)best]))
        best = j;
    if (best < 0) break;
    k[(size_t)best] += 1;
  }
  int next = 0;
  int64_t share = 0;
  for (int j = 0; j < nj; ++j) {
    const int nb = (int)k[(size_t)j];
    teams->push_back(PointTeam{next, nb, j, 0, jobs[(size_t)j].n0, jobs[(size_t)j].n1});
    team_of_block->insert(team_of_block->end(), (size_t)nb, j);
    next += nb;
    share = std::max(share, ceil_div(nodes(j), (int64_t)nb));
  }
  const int prc = point_plan_teams(share, precond, next, plan);
  if (prc != CPFEM_OK || !plan->ok) {
    teams->clear();
    team_of_block->clear();
  }
  return prc;
}

// The jobs' iteration counts and flags, waited for.
static int ragged_finish(const RWork& w, const std::vector<RJob>& jobs, int32_t* info, cudaStream_t s) {
  const int nj = (int)jobs.size();
  std::vector<int32_t> out((size_t)(2 * nj));
  int err = 0;
  CPFEM_CUDA_TRY(cudaMemcpyAsync(out.data(), w.info, sizeof(int32_t) * out.size(), cudaMemcpyDeviceToHost, s));
  CPFEM_CUDA_TRY(cudaMemcpyAsync(&err, w.error, sizeof(int), cudaMemcpyDeviceToHost, s));
  CPFEM_CUDA_TRY(cudaStreamSynchronize(s));
  for (int j = 0; j < nj; ++j) {
    info[2 * jobs[(size_t)j].inst] = out[(size_t)(2 * j)];
    info[2 * jobs[(size_t)j].inst + 1] = out[(size_t)(2 * j + 1)];
  }
  if (err) {
    set_error("ragged BiCGSTAB team barrier timed out");
    return CPFEM_ERR_SOLVE;
  }
  return CPFEM_OK;
}

}  // namespace cpfem

extern "C" {

size_t cpfem_bicgstab_batched_workspace_bytes(int32_t num_nodes) {
  return cpfem::carve_ragged(nullptr, num_nodes, nullptr);
}

int cpfem_bicgstab_batched(const cpfem_sell_t* sell, const double* values, const double* b, double* x,
                           int32_t precond, double tol, double atol, int32_t maxiter, int32_t num_instances,
                           const int32_t* node_off, int32_t num_active, const int32_t* active,
                           const double* weights, void* workspace, int32_t* info, void* stream) {
  using namespace cpfem;
  CPFEM_REQUIRE(sell_ok(sell), "bad layout");
  CPFEM_REQUIRE(num_instances >= 0 && num_active >= 0 && num_active <= num_instances, "bad instance counts");
  if (num_active == 0 || sell->num_nodes == 0) return CPFEM_OK;
  CPFEM_REQUIRE(values && b && x && active && node_off && workspace && info, "bad batched bicgstab arguments");
  CPFEM_REQUIRE(((uintptr_t)workspace & 255) == 0, "workspace must be 256-byte aligned");
  CPFEM_REQUIRE(precond >= 0 && precond <= 2 && maxiter >= 0, "bad solver settings");
  CPFEM_REQUIRE(node_off[0] >= 0 && node_off[num_instances] <= sell->num_nodes, "node_off outside the system");
  for (int32_t i = 0; i < num_instances; ++i)
    CPFEM_REQUIRE(node_off[i + 1] >= node_off[i], "node_off must be non-decreasing");
  // jobs: listed instances that own nodes, heaviest first
  std::vector<char> seen((size_t)num_instances, 0);
  std::vector<RJob> jobs;
  std::vector<double> wts;
  jobs.reserve((size_t)num_active);
  for (int32_t j = 0; j < num_active; ++j) {
    const int32_t inst = active[j];
    CPFEM_REQUIRE(inst >= 0 && inst < num_instances, "active instance out of range");
    CPFEM_REQUIRE(!seen[(size_t)inst], "an instance is listed twice");
    seen[(size_t)inst] = 1;
    const int64_t n0 = node_off[inst], n1 = node_off[inst + 1];
    if (n1 == n0) {
      info[2 * inst] = 0;
      info[2 * inst + 1] = 1;
      continue;
    }
    const double wt = weights ? weights[j] : std::pow((double)(n1 - n0), 4.0 / 3.0);
    CPFEM_REQUIRE(wt > 0.0 && std::isfinite(wt), "weights must be positive");
    jobs.push_back(RJob{inst, 0, n0, n1});
    wts.push_back(wt);
  }
  if (jobs.empty()) return CPFEM_OK;
  {
    std::vector<size_t> order(jobs.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t c) { return wts[a] > wts[c]; });
    std::vector<RJob> j2(jobs.size());
    std::vector<double> w2(jobs.size());
    for (size_t i = 0; i < order.size(); ++i) { j2[i] = jobs[order[i]]; w2[i] = wts[order[i]]; }
    jobs.swap(j2);
    wts.swap(w2);
  }
  const int nj = (int)jobs.size();
  cudaStream_t s = (cudaStream_t)stream;
  RWork w;
  carve_ragged(workspace, sell->num_nodes, &w);
  int dev = 0, sms = 0, per_sm = 0;
  CPFEM_CUDA_TRY(cudaGetDevice(&dev));
  CPFEM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  CPFEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)k_bicgstab_ragged, kPThreads, 0));
  if (per_sm < 1) {
    set_error("ragged BiCGSTAB kernel cannot be resident");
    return CPFEM_ERR_CUDA;
  }
  PointPlan plan{};
  std::vector<PointTeam> pteams;
  std::vector<int> team_of_block;
  if (const int prc = ragged_point_plan(jobs, wts, precond, &plan, &pteams, &team_of_block); prc != CPFEM_OK) return prc;
  if (plan.ok) {
    PointArgs a{};
    a.L = *sell; a.vals = values; a.b = b; a.x = x;
    a.phat = w.phat; a.shat = w.shat;
    a.counters = (unsigned int*)w.partials;
    a.cells = w.partials + kPointCounterBytes / sizeof(double);
    a.error = w.error;
    a.polls = kPtSpinLimit;
    a.teams = (PointTeam*)w.teams;
    a.team_of_block = w.team_of_block;
    a.info = w.info;
    a.precond = precond; a.maxiter = maxiter;
    a.tol = tol; a.atol = atol;
    CPFEM_CUDA_TRY(cudaMemcpyAsync(w.teams, pteams.data(), sizeof(PointTeam) * pteams.size(), cudaMemcpyHostToDevice, s));
    CPFEM_CUDA_TRY(cudaMemcpyAsync(w.team_of_block, team_of_block.data(), sizeof(int) * team_of_block.size(),
                                   cudaMemcpyHostToDevice, s));
    CPFEM_CUDA_TRY(cudaMemsetAsync(w.partials, 0, kPointCounterBytes, s));
    CPFEM_CUDA_TRY(cudaMemsetAsync(w.error, 0, sizeof(int), s));
    if (const int lrc = point_launch(plan, false, a, s); lrc != CPFEM_OK) return lrc;
    return ragged_finish(w, jobs, info, s);
  }
  const int bmax = (int)std::min<int64_t>((int64_t)per_sm * sms, kMaxBlocks);
  std::vector<RTeam> teams;
  if (nj <= bmax) {
    // static plan: one team per job, 1 block plus a share of the spare blocks by weight
    double wsum = 0.0;
    for (double v : wts) wsum += v;
    const int spare = bmax - nj;
    int next = 0;
    for (int j = 0; j < nj; ++j) {
      const int64_t cap = std::max<int64_t>(1, ceil_div(jobs[(size_t)j].n1 - jobs[(size_t)j].n0, kMinNodesPerBlock));
      int64_t k = 1 + (int64_t)std::floor((double)spare * wts[(size_t)j] / wsum);
      k = std::min<int64_t>(k, cap);
      teams.push_back(RTeam{next, (int)k, j, 0});
      for (int64_t c = 0; c < k; ++c) team_of_block.push_back(j);
      next += (int)k;
    }
  } else {
    for (int blk = 0; blk < bmax; ++blk) {
      teams.push_back(RTeam{blk, 1, -1, 0});
      team_of_block.push_back(blk);
    }
  }
  const int blocks = (int)team_of_block.size();
  CPFEM_CUDA_TRY(cudaMemcpyAsync(w.teams, teams.data(), sizeof(RTeam) * teams.size(), cudaMemcpyHostToDevice, s));
  CPFEM_CUDA_TRY(cudaMemcpyAsync(w.team_of_block, team_of_block.data(), sizeof(int) * (size_t)blocks,
                                 cudaMemcpyHostToDevice, s));
  CPFEM_CUDA_TRY(cudaMemcpyAsync(w.jobs, jobs.data(), sizeof(RJob) * (size_t)nj, cudaMemcpyHostToDevice, s));
  CPFEM_CUDA_TRY(cudaMemsetAsync(w.tsync, 0, sizeof(GridSync) * teams.size(), s));
  CPFEM_CUDA_TRY(cudaMemsetAsync(w.queue, 0, sizeof(unsigned int), s));
  CPFEM_CUDA_TRY(cudaMemsetAsync(w.error, 0, sizeof(int), s));
  if (precond != 0) {
    k_precond_setup<false><<<(unsigned)ceil_div(sell->num_nodes, 128), 128, 0, s>>>(*sell, values, precond, w.minv);
    CPFEM_CUDA_TRY(cudaGetLastError());
  }
  cpfem_sell_t Lc = *sell;
  const double* bb = b;
  double* xx = x;
  int pc = precond, mi = maxiter, njobs = nj;
  double tl = tol, at = atol;
  void* args[] = {&Lc, &values, &bb, &xx, &w, &pc, &tl, &at, &mi, &njobs};
  CPFEM_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_bicgstab_ragged, dim3((unsigned)blocks), dim3(kPThreads),
                                             args, 0, s));
  return ragged_finish(w, jobs, info, s);
}

}  // extern "C"

// ---- allocation-free variant ---------------------------------------------------------
// Some callers cannot allocate device memory at all: a host code that owns every device
// byte through its own pool, or a caller that must not grow its footprint inside a
// real-time loop.  cpfem_bicgstab_noalloc gives them the same solver with its scratch
// (Krylov vectors, preconditioner, reduction partials, barrier words) in a fixed
// file-scope device array, sized for CPFEM_NOALLOC_MAX_NODES nodes.  The array lives in
// every GPU that loads the library until the process exits.
#include <mutex>

namespace cpfem {

constexpr int64_t kNoAllocMaxNodes = CPFEM_NOALLOC_MAX_NODES;

static size_t noalloc_bytes_needed() { return carve(nullptr, kNoAllocMaxNodes, nullptr); }

// 256-byte aligned scratch; its size is fixed at compile time from the carve layout of
// kNoAllocMaxNodes nodes (checked again at run time).
static __device__ __align__(256) unsigned char g_noalloc_scratch[CPFEM_NOALLOC_SCRATCH_BYTES];
static_assert(carve_bytes(kNoAllocMaxNodes) <= CPFEM_NOALLOC_SCRATCH_BYTES,
              "the allocation-free scratch is smaller than the solver's layout for CPFEM_NOALLOC_MAX_NODES");

static std::mutex g_noalloc_mutex;
static void* g_noalloc_ptr[256] = {nullptr};

// Device address of the scratch on the current device.  Host code must not use the
// symbol's name as an address: it is a host-side stand-in.  Resolved once per device index
// and kept: the address belongs to that device's primary context (the runtime API's).
static int noalloc_scratch(void** out) {
  int dev = 0;
  CPFEM_CUDA_TRY(cudaGetDevice(&dev));
  CPFEM_REQUIRE(dev >= 0 && dev < 256, "device index out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    CPFEM_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    CPFEM_REQUIRE(ptr != nullptr && ((uintptr_t)ptr & 255) == 0, "scratch address is not 256-byte aligned");
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return CPFEM_OK;
}

}  // namespace cpfem

extern "C" int cpfem_bicgstab_noalloc(const cpfem_sell_t* sell, const double* values, const double* b, double* x,
                                      int32_t precond, int32_t transpose, double tol, double atol,
                                      int32_t maxiter, int32_t* info, void* stream) {
  using namespace cpfem;
  CPFEM_REQUIRE(info != nullptr, "info is null");
  info[0] = 0;
  info[1] = 1;
  CPFEM_REQUIRE(sell_ok(sell), "bad layout");
  if (sell->num_nodes > kNoAllocMaxNodes) {
    set_error("cpfem_bicgstab_noalloc: " + std::to_string(sell->num_nodes) + " nodes exceed the fixed scratch of " +
              std::to_string((long long)kNoAllocMaxNodes) + " nodes; use cpfem_bicgstab with a caller workspace");
    return CPFEM_ERR_SIZE;
  }
  CPFEM_REQUIRE(noalloc_bytes_needed() == carve_bytes(kNoAllocMaxNodes) &&
                    noalloc_bytes_needed() <= sizeof(g_noalloc_scratch),
                "scratch smaller than its layout");
  void* ws = nullptr;
  int rc = noalloc_scratch(&ws);
  if (rc != CPFEM_OK) return rc;
  // run_bicgstab clears the barrier words and writes every vector before reading it
  return cpfem_bicgstab(sell, values, b, x, precond, transpose, tol, atol, maxiter, ws, info, stream);
}
