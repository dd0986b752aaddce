// Per-Gauss-point Kalidindi update in FP64, one thread per GP.
//
// The reference (singlecrystal_copper/models_copper.py:155-259) solves for the second
// Piola-Kirchhoff stress S with 9 unknowns in the global frame:
//   r(S) = S - C'(R) : (Fe^T Fe - I)/2,   Fe = F Fp^-1_old (I - sum_a dg_a R P_a R^T),
//   dg_a = ao dt |tau_a/g_a|^(1/m) sign(tau_a),  tau_a = S : R P_a R^T.
// Here the same Newton iterates are computed in the lattice frame with the 6 symmetric
// unknowns s = R^T S R (11,22,33,23,13,12).  For an orthonormal R the residual norm, the
// Newton step, the line search and the converged S are the reference's (the map is an
// orthogonal change of variables, and from S0 = 0 the 9-unknown iterates stay
// symmetric because C' : E is symmetric).  This costs a 6x6 rather than a 9x9 solve and
// needs neither the rotated C' nor the rotated Schmid tensors.
//
// What bounds it: the FP64 pipe (64 cycles per warp instruction) and, before it, instruction
// fetch.  With the loops over slip systems, tangent directions and columns unrolled, a point
// ran through some 30,000 instructions of nearly straight code with 6.5 M spills per pass
// (32^3 cells), and with most iterations in FP32 two thirds of the stalled cycles were waits
// for an instruction (FP64 pipe 30 % active).  So those loops are rolled, each residual has one
// call site, and what the loops index -- the per-slip values and the stress derivatives -- lies
// in shared memory, one column per thread (GpSlab), where a dynamic index costs nothing.
// Unrolling by 2 measured best: by 1 +1 %, by 4 +7 to 17 %; three blocks per SM instead of
// two -1 to +2 %.  Tangent passes at 262,144 points, 12 systems: 7.0 ms before the FP32
// pre-solve and the rolling (first passes of a load step), 5.1 with the former alone, 3.2 now;
// later passes 2.2, 2.2 and 1.2 ms.
#pragma once

#include "cpfem_common.cuh"

namespace cpfem {

// x^e for x >= 0 and a non-negative integer e, by binary exponentiation.  The
// Kalidindi exponents 1/m - 1 and a are integers for every shipped material (1/m = 10,
// 20, 120; a = 2, 8), and this costs about 2 log2(e) FP64 multiplies against the ~100
// FP64 operations of a general pow.
template <typename T>
CPFEM_HD T ipow(T x, int e) {
  if (e == 0) return T(1);
  while (!(e & 1)) {       // the first factor without a multiplication by one
    x *= x;
    e >>= 1;
  }
  T r = x;
  while (e >>= 1) {
    x *= x;
    if (e & 1) r *= x;
  }
  return r;
}

// The integer exponent to use for x^p, or -1 when p is not a small non-negative integer.
CPFEM_HD int int_exponent(double p) {
  return (p >= 0.0 && p <= 1024.0 && p == floor(p)) ? (int)p : -1;
}

CPFEM_HD double powe(double x, double p, int ie) { return (ie >= 0) ? ipow(x, ie) : pow(x, p); }

// Per-thread columns in the block's dynamic shared memory (kDoubles doubles per thread):
// 1/g, the slip increments, d(dg)/d(tau) in FP64 and FP32; the 6 x 9 stress derivatives of the
// tangent take the place of the first two.
extern __shared__ __align__(16) double gp_slab[];

template <int NS, int THREADS>
struct GpSlab {
  static constexpr int kD = 54;                        // 2 NS <= 54
  static constexpr int kDoubles = kD + NS + NS / 2;
  static constexpr size_t kBytes = sizeof(double) * kDoubles * THREADS;
  static __device__ __forceinline__ double& ig(int a) { return gp_slab[a * THREADS + threadIdx.x]; }
  static __device__ __forceinline__ double& dg(int a) { return gp_slab[(NS + a) * THREADS + threadIdx.x]; }
  static __device__ __forceinline__ double& kk(int a) { return gp_slab[(kD + a) * THREADS + threadIdx.x]; }
  static __device__ __forceinline__ float& kf(int a) {
    return reinterpret_cast<float*>(gp_slab + (kD + NS) * THREADS)[a * THREADS + threadIdx.x];
  }
  // dP/ds_mm: nine values in the thread's own columns, two floats to a double
  static __device__ __forceinline__ void put9(int mm, const double* v) {
#pragma unroll
    for (int k = 0; k < 9; ++k) gp_slab[(9 * mm + k) * THREADS + threadIdx.x] = v[k];
  }
  static __device__ __forceinline__ void put9(int mm, const float* v) {
    float2* p = reinterpret_cast<float2*>(gp_slab);
#pragma unroll
    for (int k = 0; k < 5; ++k) p[(5 * mm + k) * THREADS + threadIdx.x] = make_float2(v[2 * k], k < 4 ? v[2 * k + 1] : 0.0f);
  }
  static __device__ __forceinline__ void get9(int mm, double* v) {
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = gp_slab[(9 * mm + k) * THREADS + threadIdx.x];
  }
  static __device__ __forceinline__ void get9(int mm, float* v) {
    const float2* p = reinterpret_cast<const float2*>(gp_slab);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float2 t = p[(5 * mm + k) * THREADS + threadIdx.x];
      v[2 * k] = t.x;
      if (k < 4) v[2 * k + 1] = t.y;
    }
  }
};

struct GPSolve {
  double s[6];      // converged lattice-frame S (tensor components)
  double B[9];      // I - L_p,lattice at s
  double M[9];      // Ct * B at s
  double rn;        // ||r|| at s
  int iters;
};

// Residual at s.  Ct = (F Fp^-1_old R)^T (F Fp^-1_old R) (symmetric, full 3x3).  Leaves the slip
// increments and their derivatives in the slab.
template <int NS, int TH>
__device__ __forceinline__ void cp_residual(const MatDev& m, const Cub& cc, const double* Ct, double cdt, double pexp,
                                            int ie1, const double* s, double* r, double& rn, double* B, double* M) {
  using Slab = GpSlab<NS, TH>;
  double L[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = 0.0;
#pragma unroll 2
  for (int a = 0; a < NS; ++a) {
    const double tau = fma(s[0], m.pv[a][0], fma(s[1], m.pv[a][1], fma(s[2], m.pv[a][2],
                       fma(s[3], m.pv[a][3], fma(s[4], m.pv[a][4], s[5] * m.pv[a][5])))));
    const double ig = Slab::ig(a);
    const double x = tau * ig;
    const double ax = fabs(x);
    // |x|^(p-1): dg = cdt |x|^(p-1) x = cdt |x|^p sign(tau) (g > 0), and the derivative
    // p cdt |x|^(p-1) / g uses the same power.
    const double pw1 = cp_greater(ax, 0.0) ? powe(ax, pexp - 1.0, ie1) : 0.0;
    const double d = cdt * pw1 * x;
    const double kk = cdt * pexp * pw1 * ig;
    Slab::dg(a) = d;
    Slab::kk(a) = kk;
    Slab::kf(a) = f32_of(kk);
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = fma(d, m.p9[a][k], L[k]);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) B[k] = ((k % 4) == 0 ? 1.0 : 0.0) - L[k];
  mm3(Ct, B, M);
  // E = (B^T M - I)/2 in 6-component form
  double e[6];
  e[0] = 0.5 * (fma(B[0], M[0], fma(B[3], M[3], B[6] * M[6])) - 1.0);
  e[1] = 0.5 * (fma(B[1], M[1], fma(B[4], M[4], B[7] * M[7])) - 1.0);
  e[2] = 0.5 * (fma(B[2], M[2], fma(B[5], M[5], B[8] * M[8])) - 1.0);
  e[3] = 0.5 * fma(B[1], M[2], fma(B[4], M[5], B[7] * M[8]));
  e[4] = 0.5 * fma(B[0], M[2], fma(B[3], M[5], B[6] * M[8]));
  e[5] = 0.5 * fma(B[0], M[1], fma(B[3], M[4], B[6] * M[7]));
  double t[6];
  cubic_apply(cc, e, t);
#pragma unroll
  for (int k = 0; k < 6; ++k) r[k] = s[k] - t[k];
  const double n2 = fma(r[0], r[0], fma(r[1], r[1], r[2] * r[2])) +
                    2.0 * fma(r[3], r[3], fma(r[4], r[4], r[5] * r[5]));
  rn = sqrt(n2);
}

// Slip tables and the slab's derivatives in the precision of a computation.
__device__ __forceinline__ double tab_d(const MatDev& m, double, int a, int i) { return m.d[a][i]; }
__device__ __forceinline__ float tab_d(const MatDev& m, float, int a, int i) { return m.d32[a][i]; }
__device__ __forceinline__ double tab_n(const MatDev& m, double, int a, int i) { return m.n[a][i]; }
__device__ __forceinline__ float tab_n(const MatDev& m, float, int a, int i) { return m.n32[a][i]; }
__device__ __forceinline__ double tab_pv(const MatDev& m, double, int a, int j) { return m.pv[a][j]; }
__device__ __forceinline__ float tab_pv(const MatDev& m, float, int a, int j) { return m.pv32[a][j]; }
__device__ __forceinline__ double tab_p9(const MatDev& m, double, int a, int k) { return m.p9[a][k]; }
__device__ __forceinline__ float tab_p9(const MatDev& m, float, int a, int k) { return m.d32[a][k / 3] * m.n32[a][k % 3]; }
template <int NS, int TH>
__device__ __forceinline__ double slab_kk(double, int a) { return GpSlab<NS, TH>::kk(a); }
template <int NS, int TH>
__device__ __forceinline__ float slab_kk(float, int a) { return GpSlab<NS, TH>::kf(a); }

// Cubic constants in the precision of a computation.
template <typename T>
struct CubT {
  T C11, C12, c44x2;
};
template <typename T>
__device__ __forceinline__ CubT<T> cub_of(const Cub& c) {
  return CubT<T>{to_prec<T>(c.C11), to_prec<T>(c.C12), to_prec<T>(2.0 * c.C44)};
}
template <typename T>
__device__ __forceinline__ void cubic_apply(const CubT<T>& m, const T* e, T* t) {
  const T d = m.C11 - m.C12, p = m.C12 * (e[0] + e[1] + e[2]);
  t[0] = cp_fma(d, e[0], p);
  t[1] = cp_fma(d, e[1], p);
  t[2] = cp_fma(d, e[2], p);
  t[3] = m.c44x2 * e[3];
  t[4] = m.c44x2 * e[4];
  t[5] = m.c44x2 * e[5];
}

// J = dr/ds = I + sum_a kk_a (C : sym(M^T d_a (x) n_a)) (x) pv_a
//           = I + C : Q,   Q = sum_a sym(M^T d_a (x) n_a) (x) (kk_a pv_a)
// (C is linear, so it is applied once to the six columns of Q instead of once per slip
// system; kk_a scales M^T d_a, and the 1/2 of sym's shear rows is in C's factor).  With the
// comparisons of the slip powers, the scale test and the pivot search taken off the FP64 pipe,
// that is 100 of some 1,400 FP64 instructions of an iteration: 5 % of the pass.  In FP64, or
// in FP32 for a Newton direction or a tangent that need not be exact.
template <int NS, int TH, typename T>
__device__ __forceinline__ void cp_jacobian(const MatDev& m, const CubT<T>& cc, const T* M, T* J) {
  T* Q = J;   // Q accumulates in J, then J = I + C : Q column by column in place
#pragma unroll
  for (int i = 0; i < 36; ++i) Q[i] = T(0);
#pragma unroll 2
  for (int a = 0; a < NS; ++a) {
    const T ka = slab_kk<NS, TH>(T(0), a);
    T d[3], n[3], w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      d[i] = tab_d(m, T(0), a, i);
      n[i] = tab_n(m, T(0), a, i);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = ka * cp_fma(M[i], d[0], cp_fma(M[3 + i], d[1], M[6 + i] * d[2]));
    T q[6];              // rows 3 to 5 without their factor 1/2
    q[0] = w[0] * n[0];
    q[1] = w[1] * n[1];
    q[2] = w[2] * n[2];
    q[3] = cp_fma(w[1], n[2], w[2] * n[1]);
    q[4] = cp_fma(w[0], n[2], w[2] * n[0]);
    q[5] = cp_fma(w[0], n[1], w[1] * n[0]);
    T c[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) c[j] = tab_pv(m, T(0), a, j);
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = 0; j < 6; ++j) Q[6 * i + j] = cp_fma(q[i], c[j], Q[6 * i + j]);
  }
  const CubT<T> ch{cc.C11, cc.C12, T(0.5) * cc.c44x2};
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    T col[6], t[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) col[i] = Q[6 * i + j];
    cubic_apply(ch, col, t);
#pragma unroll
    for (int i = 0; i < 6; ++i) J[6 * i + j] = (i == j ? T(1) : T(0)) + t[i];
  }
}

// FP32 is used for a direction or a tangent while the Jacobian's scale max_a kk_a C11 is at most
// kJ32Scale, where its rounding leaves them accurate to ~1e-4 or better.
constexpr double kJ32Scale = 1e4;

template <int NS, int TH>
__device__ __forceinline__ bool scale_f32_ok(const Cub& cc) {
  float kmax = 0.0f;
#pragma unroll 2
  for (int a = 0; a < NS; ++a) kmax = fmaxf(kmax, GpSlab<NS, TH>::kf(a));
  return kmax * f32_of(cc.C11) <= (float)kJ32Scale;
}

// A Newton direction ds = -J^-1 r at the slab's derivatives.  (Out of line it measured 1 %
// slower on few points and 1 % faster on the first passes of 262,144.)
template <typename T>
struct DirIn {
  T M[9], r[6];
  CubT<T> cc;
};
template <typename T>
struct Vec6 {
  T v[6];
};
template <int NS, int TH, typename T>
__device__ __forceinline__ Vec6<T> cp_direction(const MatDev& m, DirIn<T> in) {
  T J[36], dinv[6];
  int perm[6];
  cp_jacobian<NS, TH, T>(m, in.cc, in.M, J);
  lu_factor<6>(J, perm, dinv);
  Vec6<T> o;
#pragma unroll
  for (int k = 0; k < 6; ++k) o.v[k] = -in.r[k];
  lu_solve<6>(J, perm, dinv, o.v);
  return o;
}

// ---- FP32 pre-solve -----------------------------------------------------------------------
// A better start for the FP64 local Newton: the same residual equation solved in FP32 from the
// warm start, as far as FP32 resolves it.  GB300's FP64 pipe takes 64 cycles per warp
// instruction, its FP32 pipe 1, so the iterations that only bring the start near the root (five
// or six in the first passes of a load step, and all of a divergent warp's) cost next to
// nothing here, and one or two FP64 iterations remain.  The converged state is the root of the
// FP64 residual to its tolerance either way.  The strain is formed from E_trial = (Ct - I)/2,
//   (B^T Ct B - I)/2 = B^T E_trial B + (L^T L - L - L^T)/2,   B = I - L,
// so no term is larger than the strain and FP32's rounding is relative to it.
struct PreIn {
  float s[6];      // the start
  float e[6];      // E_trial (11,22,33,23,13,12)
  float cdt, pexp;
  CubT<float> cc;
  int ie1;
};

constexpr float kPreFar = 1e-4f;    // pre-solve where ||r|| exceeds this times the stress
constexpr float kPreNear = 2e-6f;   // and stop it below this
constexpr int kPreIters = 24, kPreTrials = 10;

template <int NS, int TH>
__device__ __forceinline__ float cp_residual_f32(const MatDev& m, const PreIn& in, const float* s, float* r, float* M) {
  using Slab = GpSlab<NS, TH>;
  float L[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = 0.0f;
#pragma unroll 2
  for (int a = 0; a < NS; ++a) {
    const float* pv = m.pv32[a];
    const float tau = fmaf(s[0], pv[0], fmaf(s[1], pv[1], fmaf(s[2], pv[2],
                      fmaf(s[3], pv[3], fmaf(s[4], pv[4], s[5] * pv[5])))));
    const float ig = f32_of(Slab::ig(a));
    const float x = tau * ig, ax = fabsf(x);
    const float pw = in.ie1 >= 0 ? ipow(ax, in.ie1) : (ax > 0.0f ? powf(ax, in.pexp - 1.0f) : 0.0f);
    const float t = in.cdt * pw;
    Slab::kf(a) = t * in.pexp * ig;
    const float d = t * x;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float v = d * m.d32[a][i];
#pragma unroll
      for (int j = 0; j < 3; ++j) L[3 * i + j] = fmaf(v, m.n32[a][j], L[3 * i + j]);
    }
  }
  float B[9], T[9];
  const float E[9] = {in.e[0], in.e[5], in.e[4], in.e[5], in.e[1], in.e[3], in.e[4], in.e[3], in.e[2]};
#pragma unroll
  for (int k = 0; k < 9; ++k) B[k] = ((k % 4) == 0 ? 1.0f : 0.0f) - L[k];
  mm3(E, B, T);
#pragma unroll
  for (int k = 0; k < 9; ++k) M[k] = fmaf(2.0f, T[k], B[k]);
  constexpr int I6[6] = {0, 1, 2, 1, 0, 0}, J6[6] = {0, 1, 2, 2, 2, 1};
  float e[6], t[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const int i = I6[c], j = J6[c];
    float v = 0.0f, q = -(L[3 * i + j] + L[3 * j + i]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v = fmaf(B[3 * k + i], T[3 * k + j], v);
      q = fmaf(L[3 * k + i], L[3 * k + j], q);
    }
    e[c] = fmaf(0.5f, q, v);
  }
  cubic_apply(in.cc, e, t);
#pragma unroll
  for (int c = 0; c < 6; ++c) r[c] = s[c] - t[c];
  return sqrtf(fmaf(r[0], r[0], fmaf(r[1], r[1], r[2] * r[2])) +
               2.0f * fmaf(r[3], r[3], fmaf(r[4], r[4], r[5] * r[5])));
}

// Damped Newton, `most` steps (at least 1) and kPreIters at most: a step is halved until the
// residual is finite and smaller.  Returns the start itself where that is near the root already, or
// where it or the equation is not finite in FP32; steps counts the steps taken.
template <int NS, int TH>
__device__ __noinline__ Vec6<float> cp_presolve(const MatDev& m, PreIn in, int most, int* steps) {
  Vec6<float> out;
  float s[6], st[6], ds[6], r[6], M[9];
  float rn = 0.0f, relax = 0.0f, size = 1.0f;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    out.v[k] = s[k] = st[k] = in.s[k];
    ds[k] = 0.0f;
    size = fmaxf(size, fabsf(s[k]));
  }
  // one residual evaluation per pass of the loop: the start's, or a trial's
  int it = -1, trial = 0;
  for (;;) {
    const float rt = cp_residual_f32<NS, TH>(m, in, st, r, M);
    bool last;
    if (it < 0) {
      last = !(rt > kPreFar * size);
    } else if (rt < rn) {
      size = 1.0f;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        s[k] = st[k];
        size = fmaxf(size, fabsf(s[k]));
      }
      last = !(rt > kPreNear * size) || it + 1 >= min(kPreIters, most) ||
             (rt > 0.3f * rn && rt < kPreFar * size);          // FP32's rounding has been reached
    } else {
      if (++trial >= kPreTrials) break;
      relax *= 0.5f;
#pragma unroll
      for (int k = 0; k < 6; ++k) st[k] = fmaf(relax, ds[k], s[k]);
      continue;
    }
    if (last) break;
    rn = rt;
    ++it;
    trial = 0;
    relax = 1.0f;
    DirIn<float> d;
#pragma unroll
    for (int k = 0; k < 9; ++k) d.M[k] = M[k];
#pragma unroll
    for (int k = 0; k < 6; ++k) d.r[k] = r[k];
    d.cc = in.cc;
    const Vec6<float> o = cp_direction<NS, TH, float>(m, d);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      ds[k] = o.v[k];
      st[k] = s[k] + ds[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) out.v[k] = s[k];
  *steps = it + 1;
  return out;
}

constexpr int kWarmStartIters = 8;   // a warm start still unconverged after this restarts from 0

// Local Newton with the cut-half line search of models_copper.py:218-245: trial
// residuals at s + relax ds, relax = 1, 1/2, ..., until the norm drops below the current
// one or max_sub_step trials were made; the last trial is taken.  It starts from s0 = 0,
// as the reference does, or -- given s_init, the same GP's last converged stress -- from
// there, which needs far fewer iterations once the global Newton iterates settle; with pre32 the
// FP32 pre-solve above moves that start to the root first, as far as FP32 resolves it.  A
// warm start that has not converged after kWarmStartIters iterations (or went
// non-finite) is abandoned: one step with a single trial evaluates the residual at
// s0 = 0 and the reference's iteration runs from there with its own max_iter.  Either way
// the result is the root of the same residual to the same tolerance.  st.iters counts every
// step, the restart and the pre-solve's included: max_iter from each start at most.  1/g is in
// the slab.
template <int NS, int TH>
__device__ __forceinline__ void cp_local_newton(const MatDev& m, const Cub& cc, const double* Ct, double cdt, double pexp,
                                                GPSolve& st, const double* s_init = nullptr, bool j32 = false,
                                                bool pre32 = false) {
  const int ie1 = int_exponent(pexp - 1.0);
  double r[6], st_s[6], ds[6];
  bool warm = s_init != nullptr;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    st_s[k] = warm ? s_init[k] : 0.0;
    ds[k] = 0.0;
  }
  int pre = 0;
  if (warm && pre32) {
    PreIn in;
    constexpr int I6[6] = {0, 4, 8, 5, 2, 1};
    bool fits = true;       // NaN or beyond FP32: left to the FP64 iteration
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      in.s[k] = f32_of(st_s[k]);
      in.e[k] = f32_of(0.5 * (k < 3 ? Ct[I6[k]] - 1.0 : Ct[I6[k]]));
      fits = fits && isfinite(in.s[k]);
    }
    in.cdt = f32_of(cdt); in.pexp = f32_of(pexp); in.ie1 = ie1;
    in.cc = cub_of<float>(cc);
    // the pre-solve's steps count toward max_iter, one of which is left for the restart from 0
    if (fits && m.max_iter > 1) {
      const Vec6<float> p = cp_presolve<NS, TH>(m, in, m.max_iter - 1, &pre);
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (p.v[k] != in.s[k]) st_s[k] = f64_of(p.v[k]);      // an unmoved start keeps its FP64 digits
    }
  }
  const int warm_iters = min(kWarmStartIters, m.max_iter - 1 - pre);
  // one residual evaluation per pass of the loop: the start's (it = -1), or a trial's of step it
  int it = -1, it0 = -pre;   // it0: the step the s0 = 0 iteration started at
  int sub = 0, sub_cap = 1;
  double relax = 1.0, rn0 = 0.0;
  for (;;) {
    cp_residual<NS, TH>(m, cc, Ct, cdt, pexp, ie1, st_s, r, st.rn, st.B, st.M);
    relax *= 0.5;
    ++sub;
    if (st.rn >= rn0 && sub < sub_cap) {
#pragma unroll
      for (int k = 0; k < 6; ++k) st_s[k] = fma(relax, ds[k], st.s[k]);
      continue;
    }
    // s + 2 relax ds with the halved relax is exactly the last trial point
#pragma unroll
    for (int k = 0; k < 6; ++k) st.s[k] = st_s[k];
    ++it;
    if (!((st.rn > m.local_tol || (warm && !(st.rn <= m.local_tol))) && it - it0 < m.max_iter)) break;
    sub_cap = m.max_sub_step;
    if (warm && (it >= warm_iters || !isfinite(st.rn))) {
      // abandon the warm start: the single trial below lands on s = 0 + 1 * 0
#pragma unroll
      for (int k = 0; k < 6; ++k) st.s[k] = ds[k] = 0.0;
      sub_cap = 1;
      warm = false;
      it0 = it + 1;
    } else {
      bool done = false;
      if (j32 && scale_f32_ok<NS, TH>(cc)) {
        DirIn<float> d;
#pragma unroll
        for (int k = 0; k < 9; ++k) d.M[k] = f32_of(st.M[k]);
#pragma unroll
        for (int k = 0; k < 6; ++k) d.r[k] = f32_of(r[k]);
        d.cc = cub_of<float>(cc);
        const Vec6<float> o = cp_direction<NS, TH, float>(m, d);
        done = true;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          ds[k] = f64_of(o.v[k]);
          done = done && isfinite(ds[k]);
        }
      }
      if (!done) {
        DirIn<double> d;
#pragma unroll
        for (int k = 0; k < 9; ++k) d.M[k] = st.M[k];
#pragma unroll
        for (int k = 0; k < 6; ++k) d.r[k] = r[k];
        d.cc = cub_of<double>(cc);
        const Vec6<double> o = cp_direction<NS, TH, double>(m, d);
#pragma unroll
        for (int k = 0; k < 6; ++k) ds[k] = o.v[k];
      }
    }
    rn0 = sub_cap == 1 ? 0.0 : st.rn;
    relax = 1.0;
    sub = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) st_s[k] = fma(relax, ds[k], st.s[k]);
  }
  st.iters = it + pre;
}

// Stress at the converged state.
//   H = Fp^-1_old R B,  Fe_l = F H,  P = F Y,  Y = H s H^T / det H
// (algebraically the reference's det(F) sigma F^-T with sigma = Fe S Fe^T / det Fe,
// models_copper.py:155-162).  W = s H^T and 1/det H are kept for the tangent.
CPFEM_HD void cp_stress(const double* F, const double* G /*Fp^-1_old R*/, const GPSolve& st, double* H,
                        double* W, double* Y, double& idet, double* P) {
  double S[9];
  mm3(G, st.B, H);
  S[0] = st.s[0]; S[4] = st.s[1]; S[8] = st.s[2];
  S[5] = S[7] = st.s[3];
  S[2] = S[6] = st.s[4];
  S[1] = S[3] = st.s[5];
  idet = 1.0 / det3(H);
  mm3_bt(S, H, W);           // W = s H^T
  mm3(H, W, Y);              // H s H^T
#pragma unroll
  for (int k = 0; k < 9; ++k) Y[k] *= idet;
  mm3(F, Y, P);
}

// Consistent tangent at the converged state:
// dP/dF = d_ik Y_lJ + (dP/ds)(ds/dF) with ds/dF = J^-1 C : sym(Fe_l[k,:] (x) H[l,:]),
// the implicit-function tangent of f_jvp (models_copper.py:251-259).
// The tangent column for F_kl is handed to store_col(kl, col[9], ds/dF_kl[6]), both in
// the precision T, as soon as it is known, so the 81 entries never need to be live at once.  Called after every other
// output of the Gauss point is written, so only what it needs is live.
// T is the precision of the computation: FP64, or FP32 for a tangent that only serves as
// the global Newton's Jacobian and the local solve's start prediction (the converged
// state and stress, and the residual that decides convergence, stay FP64 either way).
template <int NS, int TH, typename T, class StoreCol>
__device__ __forceinline__ void cp_tangent(const MatDev& m, const Cub& cc64, const double* F64, const double* G64,
                                           const GPSolve& st, const double* H64, const double* W64, const double* Y64,
                                           double idet64, StoreCol store_col) {
  using Slab = GpSlab<NS, TH>;
  T F[9], H[9], Y[9];
  // element i (0..2, not known at compile time) of a row or column of a 3x3 in registers
  auto pick = [](int i, T v0, T v1, T v2) { return i == 0 ? v0 : (i == 1 ? v1 : v2); };
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    F[k] = to_prec<T>(F64[k]); H[k] = to_prec<T>(H64[k]); Y[k] = to_prec<T>(Y64[k]);
  }
  const CubT<T> cc = cub_of<T>(cc64);
  {
    // dP/ds for the 6 symmetric basis directions, to the slab
    T G[9], W[9], B[9], Bi[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      G[k] = to_prec<T>(G64[k]); W[k] = to_prec<T>(W64[k]); B[k] = to_prec<T>(st.B[k]);
    }
    const T idet = to_prec<T>(idet64);
    inv3(B, Bi);
#pragma unroll 1
    for (int mm = 0; mm < 6; ++mm) {
      T dL[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) dL[k] = T(0);
#pragma unroll 2
      for (int a = 0; a < NS; ++a) {
        const T c = slab_kk<NS, TH>(T(0), a) * tab_pv(m, T(0), a, mm);
#pragma unroll
        for (int k = 0; k < 9; ++k) dL[k] = cp_fma(c, tab_p9(m, T(0), a, k), dL[k]);
      }
      T trace = T(0);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) trace = cp_fma(Bi[3 * i + j], dL[3 * j + i], trace);
      T dH[9], V[9], dY[9], dP[9];
      mm3(G, dL, dH);          // G dL  (= -dH)
      mm3(dH, W, V);           // V = (G dL) s H^T
      const int ei = (mm < 3) ? mm : ((mm == 3) ? 1 : 0);
      const int ej = (mm < 3) ? mm : ((mm == 5) ? 1 : 2);
      T Hi[3], Hj[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        Hi[i] = pick(ei, H[3 * i], H[3 * i + 1], H[3 * i + 2]);
        Hj[i] = pick(ej, H[3 * i], H[3 * i + 1], H[3 * i + 2]);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          T hh = Hi[i] * Hj[j];
          if (mm >= 3) hh = cp_fma(Hj[i], Hi[j], hh);
          dY[3 * i + j] = cp_fma(hh - V[3 * i + j] - V[3 * j + i], idet, Y[3 * i + j] * trace);
        }
      mm3(F, dY, dP);
      Slab::put9(mm, dP);
    }
  }

  // ds/dF column by column through the factorised Jacobian at the converged s
  T J[36];
  int perm[6];
  T dinv[6];
  {
    T M[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) M[k] = to_prec<T>(st.M[k]);
    cp_jacobian<NS, TH, T>(m, cc, M, J);
  }
  lu_factor<6>(J, perm, dinv);
  T Fe[9];
  mm3(F, H, Fe);
#pragma unroll 1
  for (int kl = 0; kl < 9; ++kl) {
    const int k = kl / 3, l = kl - 3 * k;
    T a[3], b[3], y[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      a[t] = pick(k, Fe[t], Fe[3 + t], Fe[6 + t]);
      b[t] = pick(l, H[t], H[3 + t], H[6 + t]);
      y[t] = pick(l, Y[t], Y[3 + t], Y[6 + t]);
    }
    T q[6], x[6];
    q[0] = a[0] * b[0];
    q[1] = a[1] * b[1];
    q[2] = a[2] * b[2];
    q[3] = T(0.5) * cp_fma(a[1], b[2], a[2] * b[1]);
    q[4] = T(0.5) * cp_fma(a[0], b[2], a[2] * b[0]);
    q[5] = T(0.5) * cp_fma(a[0], b[1], a[1] * b[0]);
    cubic_apply(cc, q, x);
    lu_solve<6>(J, perm, dinv, x);
    T col[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) col[3 * i + j] = (i == k) ? y[j] : T(0);
#pragma unroll
    for (int mm = 0; mm < 6; ++mm) {
      T dP[9];
      Slab::get9(mm, dP);
#pragma unroll
      for (int i = 0; i < 9; ++i) col[i] = cp_fma(dP[i], x[mm], col[i]);
    }
    store_col(kl, col, x);
  }
}

// Explicit hardening after the local solve (models_copper.py:176-187; per-GP parameters as in
// crystal_plasticity_OR_design/models_sens_rot.py:168-193): the increments h |dg_b| |1 - g_b/t|^a
// replace 1/g in the slab, then new_g(a, value) gets every slip resistance.
template <int NS, int TH, class Old, class New>
__device__ __forceinline__ void cp_hardening(const MatDev& m, double h, double t_sat, double gss_a, double rq, Old old_g,
                                             New new_g) {
  using Slab = GpSlab<NS, TH>;
  double total = 0.0;
  const int ia = int_exponent(gss_a);
#pragma unroll 1
  for (int b = 0; b < NS; ++b) {
    const double ratio = 1.0 - old_g(b) / t_sat;
    const double ar = fabs(ratio);
    const double pw = cp_greater(ar, 0.0) ? powe(ar, gss_a, ia) : 0.0;
    const double t = h * fabs(Slab::dg(b)) * copysign(pw, ratio);     // pw = 0 where ratio is 0 or NaN
    Slab::ig(b) = t;
    total += t;
  }
  if (m.qmode == 0) {
#pragma unroll 1
    for (int a = 0; a < NS; ++a) new_g(a, fma(rq, total, old_g(a)));
  } else {
#pragma unroll 1
    for (int a0 = 0; a0 < NS; a0 += 3) {
      const double blk = Slab::ig(a0) + Slab::ig(a0 + 1) + Slab::ig(a0 + 2);
      const double inc = fma(rq, total - blk, blk);
#pragma unroll
      for (int j = 0; j < 3; ++j) new_g(a0 + j, old_g(a0 + j) + inc);
    }
  }
}

}  // namespace cpfem
