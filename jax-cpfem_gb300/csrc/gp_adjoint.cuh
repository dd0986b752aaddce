// Backward of the converged local Newton (the implicit-function VJP of the reference's
// custom_jvp, singlecrystal_copper/models_copper.py:251-259, as jax.grad transposes it).
//
// y(s, x) evaluates, at a fixed lattice-frame stress s, the residual r and the outputs
// (P, sigma, Fp^-1_new, g_new) from the inputs x = (F, Fp^-1_old, g, rotation, params).
// At the converged s (r = 0) a cotangent ybar on the outputs pulls back to
//   xbar = (dy/dx)^T ybar - (dr/dx)^T nu,   nu = J^-T (dy/ds)^T ybar,   J = dr/ds.
// The partial derivatives are taken in forward mode with K-tangent dual numbers over the
// same formulas as the forward pass, K directions per sweep.
//
// No local array here is indexed by a run-time value, the slip systems are a loop, and one call site
// serves all sweeps.  With the systems unrolled and the directions in index arrays the kernel's
// results on the GPU were wrong for 24 systems (the same source on the host, and for 12 on the GPU,
// agreed with finite differences), and two of its builds, with stack frames of 2,832 and 7,312
// bytes, read illegal addresses, although run thread by thread on the host no index leaves its array.
#pragma once

#include "gp_update.cuh"

namespace cpfem {

template <int K>
struct Dual {
  double v;
  double d[K];
};

template <int K>
CPFEM_HD Dual<K> dconst(double v) {
  Dual<K> r;
  r.v = v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = 0.0;
  return r;
}

template <int K>
CPFEM_HD Dual<K> operator+(const Dual<K>& a, const Dual<K>& b) {
  Dual<K> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] + b.d[k];
  return r;
}

template <int K>
CPFEM_HD Dual<K> operator-(const Dual<K>& a, const Dual<K>& b) {
  Dual<K> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] - b.d[k];
  return r;
}

template <int K>
CPFEM_HD Dual<K> operator*(const Dual<K>& a, const Dual<K>& b) {
  Dual<K> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = fma(a.d[k], b.v, a.v * b.d[k]);
  return r;
}

template <int K>
CPFEM_HD Dual<K> operator*(double a, const Dual<K>& b) {
  Dual<K> r;
  r.v = a * b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a * b.d[k];
  return r;
}

template <int K>
CPFEM_HD Dual<K> recip(const Dual<K>& a) {
  Dual<K> r;
  r.v = 1.0 / a.v;
  const double c = -r.v * r.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = c * a.d[k];
  return r;
}

// a*b + c
template <int K>
CPFEM_HD Dual<K> dfma(const Dual<K>& a, const Dual<K>& b, const Dual<K>& c) {
  Dual<K> r;
  r.v = fma(a.v, b.v, c.v);
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = fma(a.d[k], b.v, fma(a.v, b.d[k], c.d[k]));
  return r;
}

// a*b + c with a plain a: half the FP64 instructions of a dual one
template <int K>
CPFEM_HD Dual<K> dfma(double a, const Dual<K>& b, const Dual<K>& c) {
  Dual<K> r;
  r.v = fma(a, b.v, c.v);
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = fma(a, b.d[k], c.d[k]);
  return r;
}

// a - b
template <int K>
CPFEM_HD Dual<K> rsub(double a, const Dual<K>& b) {
  Dual<K> r;
  r.v = a - b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = -b.d[k];
  return r;
}

// sign(v) * a, 0 for v = 0 (or NaN)
template <int K>
CPFEM_HD Dual<K> with_sign(double v, const Dual<K>& a) {
  Dual<K> r;
  const bool neg = v < 0.0, some = v > 0.0 || neg;
  r.v = some ? (neg ? -a.v : a.v) : 0.0;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = some ? (neg ? -a.d[k] : a.d[k]) : 0.0;
  return r;
}

// sign(a) * a, derivative sign(a) (0 at a = 0, as jnp.abs differentiates)
template <int K>
CPFEM_HD Dual<K> dabs(const Dual<K>& a) {
  return with_sign(a.v, a);
}

// x^q for x >= 0: value through powe, d = x^q (q dx/x + dq ln x); 0 at x = 0.  The logarithm only
// where q has a tangent (dq): it is a fifth of a slip system's FP64 instructions.
template <int K>
CPFEM_HD Dual<K> dpow(const Dual<K>& x, const Dual<K>& q, int iq, bool dq) {
  Dual<K> r;
  if (x.v > 0.0) {
    r.v = powe(x.v, q.v, iq);
    const double a = r.v * q.v / x.v;
#pragma unroll
    for (int k = 0; k < K; ++k) r.d[k] = a * x.d[k];
    if (dq) {
      const double b = r.v * log(x.v);
#pragma unroll
      for (int k = 0; k < K; ++k) r.d[k] = fma(b, q.d[k], r.d[k]);
    }
  } else {
    r = dconst<K>(0.0);
  }
  return r;
}

template <int K>
CPFEM_HD void dmm3(const Dual<K>* A, const Dual<K>* B, Dual<K>* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = dfma(A[3 * i], B[j], dfma(A[3 * i + 1], B[3 + j], A[3 * i + 2] * B[6 + j]));
}

template <int K>
CPFEM_HD void dmm3_bt(const Dual<K>* A, const Dual<K>* B, Dual<K>* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = dfma(A[3 * i], B[3 * j], dfma(A[3 * i + 1], B[3 * j + 1], A[3 * i + 2] * B[3 * j + 2]));
}

template <int K>
CPFEM_HD void dmm3_at(const Dual<K>* A, const Dual<K>* B, Dual<K>* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = dfma(A[i], B[j], dfma(A[3 + i], B[3 + j], A[6 + i] * B[6 + j]));
}

template <int K>
CPFEM_HD Dual<K> ddet3(const Dual<K>* A) {
  return A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
         A[2] * (A[3] * A[7] - A[4] * A[6]);
}

template <int K>
CPFEM_HD void dcubic(const Cub& m, const Dual<K>* e, Dual<K>* t) {
  t[0] = m.C11 * e[0] + m.C12 * (e[1] + e[2]);
  t[1] = m.C11 * e[1] + m.C12 * (e[0] + e[2]);
  t[2] = m.C11 * e[2] + m.C12 * (e[0] + e[1]);
  t[3] = (2.0 * m.C44) * e[3];
  t[4] = (2.0 * m.C44) * e[4];
  t[5] = (2.0 * m.C44) * e[5];
}

// Inputs of y(s, x), in the order of their tangent directions: s (6), F (9), Fp^-1_old (9), g (NS),
// theta = (gss_a, h, t_sat, xm, rq) (5), w (3) -- a spatial rotation increment, R -> (I + [w]x) R,
// the only rotation directions on which the lattice-frame formulas and the reference's global-frame
// ones agree.
template <int NS>
struct XIn {
  static constexpr int kS = 0, kF = 6, kFp = 15, kG = 24, kTh = 24 + NS, kW = 29 + NS, kN = 32 + NS;
};

// Input idx with its tangent seed: directions c0 .. c0 + K - 1 are in the K slots.
template <int K>
CPFEM_HD Dual<K> seeded(int c0, int idx, double v) {
  Dual<K> r;
  r.v = v;
#pragma unroll
  for (int j = 0; j < K; ++j) r.d[j] = (idx - c0 == j) ? 1.0 : 0.0;
  return r;
}

// Cotangents of the outputs P (9), sigma (9), Fp^-1_new (9); those of g_new come from a function.
struct YBar {
  double P[9], sig[9], Fp[9];
};

// y at the inputs, with tangents in the directions c0 .. c0 + K - 1: the residual r (6 duals), and
// yb = sum ybar . y over the outputs, so that the outputs never have to be live at once.  g(a) and
// gbar(a) give slip system a's resistance and the cotangent of its new one.
template <int NS, int K, class G, class GBar>
CPFEM_HD void cp_eval_dual(const MatDev& m, const Cub& cc, double cdt, const double* s0, const double* F0,
                           const double* Fp0, const double* R0, const double* th0, int c0, G g, const YBar& ybar,
                           GBar gbar, Dual<K>* r6, Dual<K>& yb) {
  Dual<K> s[6], F[9], Fp[9], R[9], th[5];
#pragma unroll
  for (int i = 0; i < 6; ++i) s[i] = seeded<K>(c0, XIn<NS>::kS + i, s0[i]);
#pragma unroll
  for (int i = 0; i < 9; ++i) F[i] = seeded<K>(c0, XIn<NS>::kF + i, F0[i]);
#pragma unroll
  for (int i = 0; i < 9; ++i) Fp[i] = seeded<K>(c0, XIn<NS>::kFp + i, Fp0[i]);
#pragma unroll
  for (int i = 0; i < 5; ++i) th[i] = seeded<K>(c0, XIn<NS>::kTh + i, th0[i]);
  {
    // R = (I + [w]x) R0 with w = 0 carrying the tangent
    Dual<K> w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = seeded<K>(c0, XIn<NS>::kW + i, 0.0);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double r0 = R0[j], r1 = R0[3 + j], r2 = R0[6 + j];
      // [w]x = [[0,-w2,w1],[w2,0,-w0],[-w1,w0,0]]
      R[j] = dfma(r2, w[1], dfma(-r1, w[2], dconst<K>(r0)));
      R[3 + j] = dfma(r0, w[2], dfma(-r2, w[0], dconst<K>(r1)));
      R[6 + j] = dfma(r1, w[0], dfma(-r0, w[1], dconst<K>(r2)));
    }
  }
  const Dual<K> pexp = recip(th[3]);
  Dual<K> pm1 = pexp;
  pm1.v -= 1.0;
  const int ie1 = int_exponent(pm1.v);
  const int ia = int_exponent(th[0].v);
  const bool dq = c0 < XIn<NS>::kW && c0 + K > XIn<NS>::kTh;     // a parameter is among the directions
  Dual<K> L[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) L[k] = dconst<K>(0.0);
  yb = dconst<K>(0.0);
  // the hardening terms t_a: their sum, and the coplanar blocks of three, each by its cotangents
  Dual<K> total = dconst<K>(0.0), blocks = dconst<K>(0.0);
  double y_all = 0.0;
  const Dual<K> it_sat = recip(th[2]);
  static_assert(NS % 3 == 0, "whole blocks of three");
  // a block of three at a time: three independent chains where few warps are at work
#pragma unroll 1
  for (int a0 = 0; a0 < NS; a0 += 3) {
    Dual<K> blk = dconst<K>(0.0);
    double y_blk = 0.0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int a = a0 + b;
      const Dual<K> gv = seeded<K>(c0, XIn<NS>::kG + a, g(a));
      Dual<K> tau = dconst<K>(0.0);
#pragma unroll
      for (int c = 0; c < 6; ++c) tau = dfma(m.pv[a][c], s[c], tau);
      const Dual<K> x = tau * recip(gv);
      const Dual<K> dg = cdt * (dpow(dabs(x), pm1, ie1, dq) * x);
#pragma unroll
      for (int k = 0; k < 9; ++k) L[k] = dfma(m.p9[a][k], dg, L[k]);
      const Dual<K> ratio = rsub(1.0, gv * it_sat);
      const Dual<K> t = with_sign(ratio.v, th[1] * dabs(dg) * dpow(dabs(ratio), th[0], ia, dq));
      const double y = gbar(a);
      yb = dfma(y, gv, yb);
      blk = blk + t;
      y_blk += y;
    }
    total = total + blk;
    y_all += y_blk;
    blocks = dfma(y_blk, blk, blocks);
  }
  // g_new_a = g_a + r total, or g_a + r (total - blk_a) + blk_a with blk_a the sum over a's block
  if (m.qmode == 0)
    yb = dfma(th[4], y_all * total, yb);
  else
    yb = yb + (th[4] * (y_all * total - blocks) + blocks);
  Dual<K> B[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) B[k] = rsub((k % 4 == 0) ? 1.0 : 0.0, L[k]);
  {
    Dual<K> A[9], AR[9], Ct[9], M[9], e[6], t[6];
    dmm3(F, Fp, A);
    dmm3(A, R, AR);
    dmm3_at(AR, AR, Ct);
    dmm3(Ct, B, M);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      e[i] = dfma(B[i], M[i], dfma(B[3 + i], M[3 + i], B[6 + i] * M[6 + i]));
      e[i].v -= 1.0;
      e[i] = 0.5 * e[i];
    }
    e[3] = 0.5 * dfma(B[1], M[2], dfma(B[4], M[5], B[7] * M[8]));
    e[4] = 0.5 * dfma(B[0], M[2], dfma(B[3], M[5], B[6] * M[8]));
    e[5] = 0.5 * dfma(B[0], M[1], dfma(B[3], M[4], B[6] * M[7]));
    dcubic<K>(cc, e, t);
#pragma unroll
    for (int i = 0; i < 6; ++i) r6[i] = s[i] - t[i];
  }
  // outputs
  Dual<K> GR[9], H[9], S[9], W[9], Y[9];
  dmm3(Fp, R, GR);
  dmm3(GR, B, H);
  dmm3_bt(H, R, W);      // Fp^-1_new
#pragma unroll
  for (int k = 0; k < 9; ++k) yb = dfma(ybar.Fp[k], W[k], yb);
  S[0] = s[0]; S[4] = s[1]; S[8] = s[2];
  S[5] = S[7] = s[3];
  S[2] = S[6] = s[4];
  S[1] = S[3] = s[5];
  const Dual<K> idet = recip(ddet3(H));
  dmm3_bt(S, H, W);
  dmm3(H, W, Y);
#pragma unroll
  for (int k = 0; k < 9; ++k) Y[k] = Y[k] * idet;
  Dual<K> P[9], sig[9];
  dmm3(F, Y, P);
  dmm3_bt(P, F, sig);
  Dual<K> ys = dconst<K>(0.0);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    yb = dfma(ybar.P[k], P[k], yb);
    ys = dfma(ybar.sig[k], sig[k], ys);
  }
  yb = dfma(ys, recip(ddet3(F)), yb);
}

// Implicit-function VJP at the converged s: out(idx, xbar) gets the cotangents of the inputs first ..
// last - 1 (XIn<NS>'s order).  Returns false if J is singular.
template <int NS, int K, class G, class GBar, class Out>
CPFEM_HD bool cp_vjp(const MatDev& m, const Cub& cc, double cdt, const double* s0, const double* F0, const double* Fp0,
                     const double* R0, const double* th0, G g, const YBar& ybar, GBar gbar, int first, int last, Out out) {
  // the directions of s, for J (6x6) and sbar = (dy/ds)^T ybar; then nu = J^-T sbar, kept in sbar;
  // then the inputs'.  One call site, and no array indexed by a loop variable.
  double JT[36], sbar[6], dinv[6];
  int perm[6];
  bool ok = true;
#pragma unroll 1
  for (int c0 = 0; c0 < last; c0 = (c0 + K >= 6 && c0 < 6) ? first : c0 + K) {
    Dual<K> r6[6], yb;
    cp_eval_dual<NS, K>(m, cc, cdt, s0, F0, Fp0, R0, th0, c0, g, ybar, gbar, r6, yb);
    if (c0 < 6) {
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < 6; ++j)
          if (c0 + k == j) {
#pragma unroll
            for (int i = 0; i < 6; ++i) JT[6 * j + i] = r6[i].d[k];
            sbar[j] = yb.d[k];
          }
      if (c0 + K >= 6) {
        lu_factor<6>(JT, perm, dinv);
#pragma unroll
        for (int i = 0; i < 6; ++i) ok = ok && isfinite(dinv[i]);
        lu_solve<6>(JT, perm, dinv, sbar);
      }
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        double acc = yb.d[k];
#pragma unroll
        for (int i = 0; i < 6; ++i) acc = fma(-sbar[i], r6[i].d[k], acc);
        if (c0 + k < last) out(c0 + k, acc);
      }
    }
  }
  return ok;
}

// The local Newton of gp_update.cuh (cp_local_newton) in FP64 alone, for a start that is as a rule
// the root: the slip loops rolled, the per-slip values formed again where they are needed.  Returns
// ||r|| at the s it leaves.
template <int NS, class G>
CPFEM_HD double cp_root(const MatDev& m, const Cub& cc, const double* Ct, double cdt, double pexp, G g, bool warm, double* s) {
  const int ie1 = int_exponent(pexp - 1.0);
  // |tau/g|^(p-1), tau/g and 1/g of slip system a
  auto slip = [&](const double* st, int a, double& x, double& ig) {
    const double* v = m.pv[a];
    const double tau = fma(st[0], v[0], fma(st[1], v[1], fma(st[2], v[2], fma(st[3], v[3], fma(st[4], v[4], st[5] * v[5])))));
    ig = 1.0 / g(a);
    x = tau * ig;
    const double ax = fabs(x);
    return (ax > 0.0) ? powe(ax, pexp - 1.0, ie1) : 0.0;
  };
  double r[6], B[9], M[9];
  auto residual = [&](const double* st) {
    double L[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) L[k] = 0.0;
#pragma unroll 1
    for (int a = 0; a < NS; ++a) {
      double x, ig;
      const double pw = slip(st, a, x, ig);
      const double d = cdt * pw * x;
#pragma unroll
      for (int k = 0; k < 9; ++k) L[k] = fma(d, m.p9[a][k], L[k]);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) B[k] = ((k % 4) == 0 ? 1.0 : 0.0) - L[k];
    mm3(Ct, B, M);
    double e[6], t[6];
    e[0] = 0.5 * (fma(B[0], M[0], fma(B[3], M[3], B[6] * M[6])) - 1.0);
    e[1] = 0.5 * (fma(B[1], M[1], fma(B[4], M[4], B[7] * M[7])) - 1.0);
    e[2] = 0.5 * (fma(B[2], M[2], fma(B[5], M[5], B[8] * M[8])) - 1.0);
    e[3] = 0.5 * fma(B[1], M[2], fma(B[4], M[5], B[7] * M[8]));
    e[4] = 0.5 * fma(B[0], M[2], fma(B[3], M[5], B[6] * M[8]));
    e[5] = 0.5 * fma(B[0], M[1], fma(B[3], M[4], B[6] * M[7]));
    cubic_apply(cc, e, t);
#pragma unroll
    for (int k = 0; k < 6; ++k) r[k] = st[k] - t[k];
    return sqrt(fma(r[0], r[0], fma(r[1], r[1], r[2] * r[2])) + 2.0 * fma(r[3], r[3], fma(r[4], r[4], r[5] * r[5])));
  };
  const int warm_iters = (kWarmStartIters < m.max_iter) ? kWarmStartIters : m.max_iter - 1;
  double st[6], ds[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (!warm) s[k] = 0.0;
    st[k] = s[k];
    ds[k] = 0.0;
  }
  // one residual evaluation per pass of the loop: the start's (it = -1), or a trial's of step it
  int it = -1, it0 = 0, sub = 0, sub_cap = 1;
  double relax = 1.0, rn0 = 0.0, rn;
  for (;;) {
    rn = residual(st);
    relax *= 0.5;
    ++sub;
    if (rn >= rn0 && sub < sub_cap) {
#pragma unroll
      for (int k = 0; k < 6; ++k) st[k] = fma(relax, ds[k], s[k]);
      continue;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k] = st[k];
    ++it;
    if (!((rn > m.local_tol || (warm && !(rn <= m.local_tol))) && it - it0 < m.max_iter)) return rn;
    sub_cap = m.max_sub_step;
    if (warm && (it >= warm_iters || !isfinite(rn))) {
      // abandon the warm start: the single trial below lands on s = 0
#pragma unroll
      for (int k = 0; k < 6; ++k) s[k] = ds[k] = 0.0;
      sub_cap = 1;
      warm = false;
      it0 = it + 1;
    } else {
      // ds = -J^-1 r, J = I + C : sum_a sym(M^T d_a (x) n_a) (x) (kk_a pv_a)
      double J[36], dinv[6];
      int perm[6];
#pragma unroll
      for (int i = 0; i < 36; ++i) J[i] = 0.0;
#pragma unroll 1
      for (int a = 0; a < NS; ++a) {
        double x, ig;
        const double kk = cdt * pexp * slip(s, a, x, ig) * ig;
        const double *d = m.d[a], *n = m.n[a];
        double w[3], q[6];
#pragma unroll
        for (int i = 0; i < 3; ++i) w[i] = kk * fma(M[i], d[0], fma(M[3 + i], d[1], M[6 + i] * d[2]));
        q[0] = w[0] * n[0];
        q[1] = w[1] * n[1];
        q[2] = w[2] * n[2];
        q[3] = 0.5 * fma(w[1], n[2], w[2] * n[1]);
        q[4] = 0.5 * fma(w[0], n[2], w[2] * n[0]);
        q[5] = 0.5 * fma(w[0], n[1], w[1] * n[0]);
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int j = 0; j < 6; ++j) J[6 * i + j] = fma(q[i], m.pv[a][j], J[6 * i + j]);
      }
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        double col[6], t[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) col[i] = J[6 * i + j];
        cubic_apply(cc, col, t);
#pragma unroll
        for (int i = 0; i < 6; ++i) J[6 * i + j] = (i == j ? 1.0 : 0.0) + t[i];
      }
      lu_factor<6>(J, perm, dinv);
#pragma unroll
      for (int k = 0; k < 6; ++k) ds[k] = -r[k];
      lu_solve<6>(J, perm, dinv, ds);
    }
    rn0 = sub_cap == 1 ? 0.0 : rn;
    relax = 1.0;
    sub = 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) st[k] = s[k] + ds[k];
  }
}

}  // namespace cpfem
