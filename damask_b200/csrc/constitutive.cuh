// Per-voxel constitutive update of the DAMASK grid hot path, FP64, one thread per
// material point, organised as passes over the voxels that still iterate.
//
// Restates, for one constituent with pass/isostrain homogenization (F_phase =
// F_cell, homogenization_mechanical.f90:94-123) and Hooke + phenopowerlaw slip:
//   phase_mechanical_constitutive   phase_mechanical.f90:1008-1090 (substep cutback)
//   mechanical_restore              phase_mechanical.f90:1096-1115
//   integrateStateFPI (+ damper)    phase_mechanical.f90:591-676
//   integrateStress (Lp Newton)     phase_mechanical.f90:379-584
//   plastic_LpAndItsTangents        phase_mechanical_plastic.f90:239-298
//   phenopowerlaw kinetics/dotState phase_mechanical_plastic_phenopowerlaw.f90:303-399,449-488
//
// Specialisation: no eigenstrain mechanism is active on this path, so the
// intermediate configuration stays Fi = I and Li = 0 (phase_mechanical_eigen.f90:133-165
// returns Li = 0; the Li loop of integrateStress then exits on its first pass).
// With Fi = I the Mandel stress is Mp = S and the Newton Jacobian
//   dR/dLp = I - dLp/dS : dS/dFe : dFe/dLp
// collapses to  J[kl][pb] = delta + dt * sum_s dgamma_s P_s(k,l) (A^T Fe Q_s)(p,b)
// with A = F Fp0^-1 and Q_s = C : P_nS_s precomputed per phase, so no 3x3x3x3
// temporaries are formed.
//
// Execution model.  The nested loops of the reference (substeps > state
// iterations > Newton iterations) are split at the state iteration: one pass
// performs, for every voxel still iterating, exactly one integrateStress (the Newton
// loop, in registers) followed by the state update and whatever substep control
// leads to the next integrateStress.  Between passes the per-voxel iteration state
// lives in HBM planes (PassWork), so the large per-system arrays of the state
// iteration are never live during the Newton loop; all indexing into register
// arrays is static, and the 9x9 Newton system, a rank-6 update of the identity, is
// solved through its 6x6 Woodbury form, five unknowns in phases without non-Schmid
// terms, by Householder QR (no data-dependent row exchange, so the matrix stays in
// registers).  Small grids run all of it in one launch (constitutive_fused_kernel).
#pragma once
#include "dmk_device.cuh"

namespace dmk {

__device__ __forceinline__ void load_ctl(const PassWork& w, int64_t N, int64_t v, VoxelCtl& c) {
  c.phase = w.ctl[v];
  c.status = w.ctl[N + v];
  c.it = w.ctl[2 * N + v];
  c.nsub = w.ctl[3 * N + v];
  c.nstate = w.ctl[4 * N + v];
  c.newton = w.ctl[5 * N + v];
  c.stepFrac = w.sub[v];
  c.step = w.sub[N + v];
  c.from_start = c.step < 0.0;
  c.step = fabs(c.step);
}
__device__ __forceinline__ void store_ctl(const PassWork& w, int64_t N, int64_t v, const VoxelCtl& c) {
  w.ctl[v] = c.phase;
  w.ctl[N + v] = c.status;
  w.ctl[2 * N + v] = c.it;
  w.ctl[3 * N + v] = c.nsub;
  w.ctl[4 * N + v] = c.nstate;
  w.ctl[5 * N + v] = c.newton;
  w.sub[v] = c.stepFrac;
  w.sub[N + v] = c.from_start ? -c.step : c.step;
}

// Solves A x = b for a row-major n x n A (overwritten with R) by Householder QR:
// column k is reflected onto alpha e_k with alpha = -sign(x0) |x|, v = x - alpha e_k,
// H y = y + v (v.y) / (alpha v0).  Returns true when a column of the remaining
// matrix is exactly zero (the matrix is singular; dgesv info > 0).  All indices are
// compile-time constants, so A stays in registers.
template <int n>
__device__ __forceinline__ bool qr_solve(double* A, double* b) {
  bool bad = false;
#pragma unroll
  for (int k = 0; k < n - 1; ++k) {
    double s2 = 0.0;
#pragma unroll
    for (int i = k; i < n; ++i) s2 = fma(A[i * n + k], A[i * n + k], s2);
    bad |= s2 == 0.0;
    const double sig = sqrt(s2);
    const double x0 = A[k * n + k];
    const double alpha = x0 >= 0.0 ? -sig : sig;
    const double v0 = x0 - alpha;
    const double rs = 1.0 / (alpha * v0);
#pragma unroll
    for (int c = k + 1; c < n; ++c) {
      double d = v0 * A[k * n + c];
#pragma unroll
      for (int i = k + 1; i < n; ++i) d = fma(A[i * n + k], A[i * n + c], d);
      d *= rs;
      A[k * n + c] = fma(d, v0, A[k * n + c]);
#pragma unroll
      for (int i = k + 1; i < n; ++i) A[i * n + c] = fma(d, A[i * n + k], A[i * n + c]);
    }
    {
      double d = v0 * b[k];
#pragma unroll
      for (int i = k + 1; i < n; ++i) d = fma(A[i * n + k], b[i], d);
      d *= rs;
      b[k] = fma(d, v0, b[k]);
#pragma unroll
      for (int i = k + 1; i < n; ++i) b[i] = fma(d, A[i * n + k], b[i]);
    }
    A[k * n + k] = alpha;
  }
  bad |= A[n * n - 1] == 0.0;
#pragma unroll
  for (int i = n - 1; i >= 0; --i) {
    double s = b[i];
#pragma unroll
    for (int k = i + 1; k < n; ++k) s = fma(-A[i * n + k], b[k], s);
    b[i] = s / A[i * n + i];
  }
  return bad;
}

// Threads and shared-memory slots of the stress kernels.  MINB: warps per scheduler that the registers
// are bounded for (2, 3 or 4: 255, 168 and 128 registers; 48 systems: three blocks of 64 threads).  A
// thread's slots (stride: the block's threads): 1/xi (NS), the Newton weights (NS; without non-Schmid
// terms also K, at least 30), A = F Fp0^-1 (9) and, where they fit, the last accepted Lp (9) and the
// Newton step (9), which stay in local memory otherwise: the L1 that the slots leave is too small for
// it, so every read of it goes to L2 (measured).
template <int NS, bool SCHMID, int MINB>
struct StressShape {
  static constexpr size_t consts = NS * sizeof(StressConst<SCHMID>) + 1024;   // with the system's 1 KB per block
  static constexpr int base = NS + (SCHMID && NS < 30 ? 30 : NS) + 9;
  static constexpr bool fits(int slots, int threads, int blocks) {
    return blocks * (consts + sizeof(double) * slots * threads) <= 228 * 1024;
  }
  static constexpr int threads = NS > 24 ? 64 : 128;
  static constexpr int blocks = NS > 24 ? 3 : MINB;
  static constexpr bool lo_shared = fits(base + 9, threads, blocks);
  static constexpr bool dl_shared = fits(base + 18, threads, blocks);
  static constexpr int slots = base + (lo_shared ? 9 : 0) + (dl_shared ? 9 : 0);
  static constexpr size_t smem = NS * sizeof(StressConst<SCHMID>) + sizeof(double) * slots * threads;
};

// nine values of a thread that are read rarely: in its shared-memory slots (stride T) or in local memory
template <bool SHARED, int T>
struct Rare9 {
  double* s;
  __device__ explicit Rare9(double* p) : s(p) {}
  __device__ double get(int k) const { return s[k * T]; }
  __device__ void set(int k, double x) { s[k * T] = x; }
};
template <int T>
struct Rare9<false, T> {
  volatile double a[9];
  __device__ explicit Rare9(double*) {}
  __device__ double get(int k) const { return a[k]; }
  __device__ void set(int k, double x) { a[k] = x; }
};

// A = F Fp0^-1 into the thread's slots; true if Fp0 is singular
template <int T>
__device__ __forceinline__ bool stress_begin(const double* F, const double* Fp0, double* sA) {
  double invFp0[9], A[9];
  if (inv33(Fp0, invFp0)) return true;
  mm33(F, invFp0, A);
#pragma unroll
  for (int k = 0; k < 9; ++k) sA[k * T] = A[k];
  return false;
}

// Fp = (Fp0^-1 B)^-1 / det^(1/3); P = F Fp^-1 S Fp^-T = Fe S Fp^-T (phase_mechanical.f90:571-581; Fe =
// F Fp0^-1 B is the last iterate's); Fp0 is read again, so that nothing of it stays in registers
// through the Newton loop.  Returns the status of the integration.
__device__ __forceinline__ int stress_end(const double* Fp0g, int64_t N, const double* B, const double* Fe,
                                          const double* s6, double* Fp, double* Pout) {
  double invFpn[9], Fpn[9];
  {
    double Fp0[9], invFp0[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) Fp0[k] = Fp0g[k * N];
    inv33(Fp0, invFp0);                                   // invertible: checked on entry
    mm33(invFp0, B, invFpn);
  }
  if (inv33(invFpn, Fpn)) return 5;
  const double cb = 1.0 / cbrt(det33(Fpn));
  const double Sm[9] = {s6[0], s6[5], s6[4], s6[5], s6[1], s6[3], s6[4], s6[3], s6[2]};
  double T1[9];
  mmt33(Sm, invFpn, T1);          // S Fp^-T
  mm33(Fe, T1, Pout);
#pragma unroll
  for (int k = 0; k < 9; ++k) Fp[k] = Fpn[k] * cb;
  return 0;
}

// integrateStress, phase_mechanical.f90:379-584 (Fi = I, Li = 0).
// F, Fp0: the values of voxel v; Fp0g: its Fp0 planes (stride N), read again for the final Fp / P.
// xs: this thread's shared-memory slots (see StressShape).  adg_g: the voxel's plane of |dot_gamma|
// (stride N), written in every residual evaluation for the state update after a converged integration.
// Lp (in/out) is the warm start and, on success, the result; S, Fp and P are written only on success; Fe is
// the last iterate's.
template <int NS, class Shape>
__device__ int integrate_stress(const PhaseConst<NS>& pc, const SysConst* __restrict__ sc, const Numerics& nm,
                                const double* F, const double* Fp0, const double* Fp0g, int64_t N, double* xs, double dt,
                                double* Lp, double* S, double* Fp, double* Pout, double* Fe, int& newton,
                                double* __restrict__ adg_g) {
  constexpr int T = Shape::threads;
  double* const sw = xs + NS * T;
  double* const sA = xs + (Shape::base - 9) * T;
  if (stress_begin<T>(F, Fp0, sA)) return 5;        // STATUS_FAIL_PHASE_MECHANICAL_STRESS

  Rare9<Shape::lo_shared, T> lo(xs + Shape::base * T);
  Rare9<Shape::dl_shared, T> dl(xs + (Shape::base + 9) * T);
  double Lg[9], B[9], s6[6];
#pragma unroll
  for (int k = 0; k < 9; ++k) { Lg[k] = Lp[k]; lo.set(k, Lp[k]); dl.set(k, 0.0); }
  double step = 1.0, res_old = 1.7976931348623157e308;
  int jaco = 0;
  for (int it = 1;; ++it) {
    if (it > nm.N_iter_Lp_max) return 6;                  // STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_MAXIT
    ++newton;
#pragma unroll
    for (int k = 0; k < 9; ++k) B[k] = fma(-dt, Lg[k], (k % 4 == 0) ? 1.0 : 0.0);
    {
      double A[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) A[k] = sA[k * T];
      mm33(A, B, Fe);
    }
    hooke_S<NS>(pc, Fe, s6);
    // Lp_c = sum_s dot_gamma_s P_s and the weights of its derivative
    double Lc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    static_assert(NS <= 64, "one sense bit per slip system");
    SenseMask<NS> neg = 0u;
#pragma unroll 2
    for (int s = 0; s < NS; ++s) {
      const SysConst& c = sc[s];
      double2 p[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) p[t] = c.p6[t];
      const double tp = fma(s6[5], p[5].x, fma(s6[4], p[4].x, fma(s6[3], p[3].x, dot3(s6[0], p[0].x, s6[1], p[1].x, s6[2], p[2].x))));
      const double tn = fma(s6[5], p[5].y, fma(s6[4], p[4].y, fma(s6[3], p[3].y, dot3(s6[0], p[0].y, s6[1], p[1].y, s6[2], p[2].y))));
      const bool pos = tp > tn;
      const double tmax = pos ? tp : tn;
      const double ixs = xs[s * T];
      const double r = tmax * ixs;
      const double2 kin = c.kin;
      const int ni = c.n_int;
      double g, dg;
      if (ni >= 1) {
        const double rn1 = powi_fixed<6>(r, ni - 1);
        const double sd = pos ? kin.x : -kin.x;
        g = sd * (rn1 * r);
        dg = (sd * kin.y) * rn1 * ixs;
      } else {
        g = (pos ? kin.x : -kin.x) * pow(r, kin.y);
        dg = g * kin.y / tmax;
      }
      if (!(fabs(g) > TINY10)) dg = 0.0;
      // P_nS sense of the derivative follows the sign of dot_gamma (phenopowerlaw.f90:327)
      if (!(g > 0.0)) neg |= SenseMask<NS>(1) << s;
      sw[s * T] = dt * dg;
      adg_g[s * N] = fabs(g);
      double2 P[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) P[k] = c.P[k];
      const double Ps[9] = {P[0].x, P[0].y, P[1].x, P[1].y, P[2].x, P[2].y, P[3].x, P[3].y, P[4].x};
#pragma unroll
      for (int k = 0; k < 9; ++k) Lc[k] = fma(g, Ps[k], Lc[k]);
    }
    double R[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) R[k] = Lg[k] - Lc[k];
    const double nR = norm9(R);
    const double atol = fmax(nm.eps_rel_Lp * fmax(norm9(Lg), norm9(Lc)), nm.eps_abs_Lp);
    if (isnan(nR)) return 7;                              // STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_NAN
    if (nR < atol) break;
    if (nR < res_old) {
      res_old = nR;
#pragma unroll
      for (int k = 0; k < 9; ++k) lo.set(k, Lg[k]);
      step = 1.0;
    } else {
      step = nm.r_linesearch_Lp * step;
#pragma unroll
      for (int k = 0; k < 9; ++k) Lg[k] = fma(dl.get(k), step, lo.get(k));
      continue;
    }
    double X[9];
    if (jaco % nm.f_update_jacobi_Lp == 0) {
      ++jaco;
      // Newton step J dLp = -R with J = I + K, K[kl][pb] = (M H^(kl))(p,b), M = A^T Fe,
      // H^(kl) = sum_s w_s P_s(k,l) Q_s.  Every row of K is M times a symmetric matrix,
      // so K = Hm L^T has rank 6 (Hm: 9x6 rows h^(kl); L: 9x6, L^T z = symfold(M^T Z)) and
      // by the Woodbury identity  J^-1 z = z - Hm (I6 + L^T Hm)^-1 L^T z.  With P_s = d_s (x) n_s,
      //   C6 = I6 + sum_s w_s symfold((M^T d_s) (x) n_s) (x) q_s,   y = C6^-1 symfold(M^T R),
      //   dLp = sum_s w_s (q_s . y) P_s - R,
      // the same solution as the 9x9 system without forming it.
      double M[9];
      {
        double A[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) A[k] = sA[k * T];
        mtm33(A, Fe, M);                                  // M = A^T Fe, M[p + 3q] = M(p,q)
      }
      double C6[36];
#pragma unroll
      for (int i = 0; i < 36; ++i) C6[i] = (i % 7 == 0) ? 1.0 : 0.0;
#pragma unroll 2
      for (int s = 0; s < NS; ++s) {
        const SysConst& c = sc[s];
        const double ws = sw[s * T];
        const bool ng = (neg >> s) & 1u;
        double q[6];
#pragma unroll
        for (int t = 0; t < 6; ++t) {
          const double2 qq = c.q6[t];
          q[t] = ng ? qq.y : qq.x;
        }
        const double2 dn0 = c.dn[0], dn1 = c.dn[1], dn2 = c.dn[2];
        const double d0 = dn0.x, d1 = dn0.y, d2 = dn1.x, n0 = dn1.y, n1 = dn2.x, n2 = dn2.y;
        // u = M^T d
        const double u0 = dot3(M[0], d0, M[1], d1, M[2], d2);
        const double u1 = dot3(M[3], d0, M[4], d1, M[5], d2);
        const double u2 = dot3(M[6], d0, M[7], d1, M[8], d2);
        const double a6[6] = {ws * (u0 * n0), ws * (u1 * n1), ws * (u2 * n2), ws * fma(u1, n2, u2 * n1),
                              ws * fma(u0, n2, u2 * n0), ws * fma(u0, n1, u1 * n0)};
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int j = 0; j < 6; ++j) C6[6 * i + j] = fma(a6[i], q[j], C6[6 * i + j]);
      }
      // y6 = symfold(M^T R)
      double y6[6];
      {
        double G[9];
        mtm33(M, R, G);                                   // G(a,b) = sum_p M(p,a) R(p,b)
        y6[0] = G[0]; y6[1] = G[4]; y6[2] = G[8];
        y6[3] = G[7] + G[5]; y6[4] = G[6] + G[2]; y6[5] = G[3] + G[1];
      }
      if (qr_solve<6>(C6, y6)) return 8;                 // singular: STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_DGESV
#pragma unroll
      for (int k = 0; k < 9; ++k) X[k] = -R[k];
#pragma unroll 2
      for (int s = 0; s < NS; ++s) {
        const SysConst& c = sc[s];
        const bool ng = (neg >> s) & 1u;
        double cq = 0.0;
#pragma unroll
        for (int t = 0; t < 6; ++t) {
          const double2 qq = c.q6[t];
          cq = fma(ng ? qq.y : qq.x, y6[t], cq);
        }
        cq *= sw[s * T];
        double2 P[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) P[k] = c.P[k];
        const double Ps[9] = {P[0].x, P[0].y, P[1].x, P[1].y, P[2].x, P[2].y, P[3].x, P[3].y, P[4].x};
#pragma unroll
        for (int k = 0; k < 9; ++k) X[k] = fma(cq, Ps[k], X[k]);
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) dl.set(k, X[k]);
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) X[k] = dl.get(k);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) Lg[k] = fma(X[k], step, Lg[k]);
  }
  if (stress_end(Fp0g, N, B, Fe, s6, Fp, Pout)) return 5;
#pragma unroll
  for (int k = 0; k < 9; ++k) Lp[k] = Lg[k];
#pragma unroll
  for (int k = 0; k < 6; ++k) S[k] = s6[k];
  return 0;
}

// The same for a phase without non-Schmid terms and cubic elasticity (every phase of this path has the
// latter).  Both senses of a system then share P_s, so tau = S : P_s with the sign of dot_gamma taken
// from it, and C : P_s is traceless.  With the coordinates (u, v) of P_s (SchmidConst) and
//   zeta(Y) = (CY11 - CY33, CY22 - CY33, 2 CY23, 2 CY13, 2 CY12), CY = C : sym(Y),
// the resolved shear of E is u . zeta(E) and the rank-6 system of the general form closes in five unknowns:
//   K_k = sum_s w_s P_s u_s,k,   z + sum_k zeta(M^T K_k) z_k = zeta(M^T R),   dLp = sum_k K_k z_k - R.
// The u-u part of K is symmetric, so a system adds 15 + 15 products to it instead of 36 to C6, and dLp needs
// no second pass over the systems.  What bounds the kernel is the FP64 instructions of this function and
// the latency of their chains at twelve warps per SM (more warps have no registers), then every memory
// round trip that they cannot hide: all of a voxel's loads are issued at once (stress_voxel), and of the
// loop only the Newton step, where it does not fit into the slots, lives in memory (spills and planes of
// it went to L2: the slots leave little of L1).  Stress kernels of one increment, general form with its
// loads one after the other -> this: 24 systems at 128^3 147 -> 94 ms, 48 systems at 40^3 17.5 -> 9.7 ms, 12
// systems at 64^3 9.5 -> 6.8 ms.  First full pass at 24 systems (64^3 -> 96x96x64): FP64 pipe 35 -> 46 %
// busy, long-scoreboard stalls per issue 2.0 -> 0.7.
template <int NS, class Shape>
__device__ int integrate_stress(const PhaseConst<NS>& pc, const SchmidConst* __restrict__ sc, const Numerics& nm,
                                const double* F, const double* Fp0, const double* Fp0g, int64_t N, double* xs, double dt,
                                double* Lp, double* S, double* Fp, double* Pout, double* Fe, int& newton,
                                double* __restrict__ adg_g) {
  constexpr int T = Shape::threads;
  double* const sw = xs + NS * T;                         // weights, then K (15 + 15 products)
  double* const sA = xs + (Shape::base - 9) * T;
  if (stress_begin<T>(F, Fp0, sA)) return 5;        // STATUS_FAIL_PHASE_MECHANICAL_STRESS
  const double c1 = pc.C66[0][0] - pc.C66[0][1], c4 = pc.C66[3][3];   // C11 - C12, 2 C44

  Rare9<Shape::lo_shared, T> lo(xs + Shape::base * T);
  Rare9<Shape::dl_shared, T> dl(xs + (Shape::base + 9) * T);
  double Lg[9], B[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) { Lg[k] = Lp[k]; lo.set(k, Lp[k]); dl.set(k, 0.0); }
  double step = 1.0, res_old = 1.7976931348623157e308;
  int jaco = 0;
  for (int it = 1;; ++it) {
    if (it > nm.N_iter_Lp_max) return 6;                  // STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_MAXIT
    ++newton;
#pragma unroll
    for (int k = 0; k < 9; ++k) B[k] = fma(-dt, Lg[k], (k % 4 == 0) ? 1.0 : 0.0);
    {
      double A[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) A[k] = sA[k * T];
      mm33(A, B, Fe);
    }
    double z[5];                                          // zeta(E), E = (Fe^T Fe - I)/2
    {
      const double f33 = dot3(Fe[6], Fe[6], Fe[7], Fe[7], Fe[8], Fe[8]);
      z[0] = (0.5 * c1) * (dot3(Fe[0], Fe[0], Fe[1], Fe[1], Fe[2], Fe[2]) - f33);
      z[1] = (0.5 * c1) * (dot3(Fe[3], Fe[3], Fe[4], Fe[4], Fe[5], Fe[5]) - f33);
      z[2] = c4 * dot3(Fe[3], Fe[6], Fe[4], Fe[7], Fe[5], Fe[8]);
      z[3] = c4 * dot3(Fe[0], Fe[6], Fe[1], Fe[7], Fe[2], Fe[8]);
      z[4] = c4 * dot3(Fe[0], Fe[3], Fe[1], Fe[4], Fe[2], Fe[5]);
    }
    // Lp_c = sum_s dot_gamma_s P_s and the weights of its derivative
    double R[9];
    {
      double l[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 2
      for (int s = 0; s < NS; ++s) {
        const double2 u01 = sc[s].u01, u23 = sc[s].u23, u4v0 = sc[s].u4v0, v12 = sc[s].v12, kin = sc[s].kin;
        const double tau = fma(u01.x, z[0], u01.y * z[1]) + fma(u23.x, z[2], fma(u23.y, z[3], u4v0.x * z[4]));
        const double ta = fabs(tau);
        const double ixs = xs[s * T];
        const double r = ta * ixs;
        const int ni = sc[s].n_int;
        double g, dg;                                      // |dot_gamma| and its derivative
        if (ni >= 1) {
          const double rn1 = powi_fixed<6>(r, ni - 1);
          g = (kin.x * rn1) * r;
          dg = (kin.x * kin.y) * rn1 * ixs;
        } else {
          g = kin.x * pow(r, kin.y);
          dg = g * kin.y / ta;
        }
        if (!(g > TINY10)) dg = 0.0;
        sw[s * T] = dt * dg;
        adg_g[s * N] = g;
        g = copysign(g, tau);
        l[0] = fma(g, u01.x, l[0]);
        l[1] = fma(g, u01.y, l[1]);
        l[2] = fma(g, u23.x, l[2]);
        l[3] = fma(g, u23.y, l[3]);
        l[4] = fma(g, u4v0.x, l[4]);
        l[5] = fma(g, u4v0.y, l[5]);
        l[6] = fma(g, v12.x, l[6]);
        l[7] = fma(g, v12.y, l[7]);
      }
      const double Lc[9] = {l[0], l[4] - l[7], l[3] - l[6], l[4] + l[7], l[1], l[2] - l[5], l[3] + l[6], l[2] + l[5],
                            -(l[0] + l[1])};
#pragma unroll
      for (int k = 0; k < 9; ++k) R[k] = Lg[k] - Lc[k];
      const double nR = norm9(R);
      const double atol = fmax(nm.eps_rel_Lp * fmax(norm9(Lg), norm9(Lc)), nm.eps_abs_Lp);
      if (isnan(nR)) return 7;                            // STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_NAN
      if (nR < atol) break;
      if (nR < res_old) {
        res_old = nR;
#pragma unroll
        for (int k = 0; k < 9; ++k) lo.set(k, Lg[k]);
        step = 1.0;
      } else {
        step = nm.r_linesearch_Lp * step;
#pragma unroll
        for (int k = 0; k < 9; ++k) Lg[k] = fma(dl.get(k), step, lo.get(k));
        continue;
      }
    }
    double X[9];
    if (jaco % nm.f_update_jacobi_Lp == 0) {
      ++jaco;
      // K: columns k of u-u products (symmetric: 15) and v-u products (15)
      double Ku[15], Kv[15];
#pragma unroll
      for (int i = 0; i < 15; ++i) Ku[i] = Kv[i] = 0.0;
#pragma unroll 1
      for (int s = 0; s < NS; ++s) {
        const double2 u01 = sc[s].u01, u23 = sc[s].u23, u4v0 = sc[s].u4v0, v12 = sc[s].v12;
        const double u[5] = {u01.x, u01.y, u23.x, u23.y, u4v0.x};
        const double v[3] = {u4v0.y, v12.x, v12.y};
        const double w = sw[s * T];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          const double wu = w * u[k];
#pragma unroll
          for (int i = 0; i <= k; ++i) Ku[k * (k + 1) / 2 + i] = fma(wu, u[i], Ku[k * (k + 1) / 2 + i]);
#pragma unroll
          for (int i = 0; i < 3; ++i) Kv[3 * k + i] = fma(wu, v[i], Kv[3 * k + i]);
        }
      }
      double M[9];
      {
        double A[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) A[k] = sA[k * T];
        mtm33(A, Fe, M);                                  // M = A^T Fe
      }
      // zeta(M^T Y) but for the factors c1, c1, c4, c4, c4
      auto zeta = [&](const double* Y, double* o) {
        const double g33 = dot3(M[6], Y[6], M[7], Y[7], M[8], Y[8]);
        o[0] = dot3(M[0], Y[0], M[1], Y[1], M[2], Y[2]) - g33;
        o[1] = dot3(M[3], Y[3], M[4], Y[4], M[5], Y[5]) - g33;
        o[2] = dot3(M[3], Y[6], M[4], Y[7], M[5], Y[8]) + dot3(M[6], Y[3], M[7], Y[4], M[8], Y[5]);
        o[3] = dot3(M[0], Y[6], M[1], Y[7], M[2], Y[8]) + dot3(M[6], Y[0], M[7], Y[1], M[8], Y[2]);
        o[4] = dot3(M[0], Y[3], M[1], Y[4], M[2], Y[5]) + dot3(M[3], Y[0], M[4], Y[1], M[5], Y[2]);
      };
      // K goes to the slots of the weights, which are spent, so that J and the factorisation have the registers
#pragma unroll
      for (int i = 0; i < 15; ++i) {
        sw[i * T] = Ku[i];
        sw[(15 + i) * T] = Kv[i];
      }
      asm volatile("" ::: "memory");                      // keep K there: no forwarding from the registers
      auto ku = [&](int k, int i) { return sw[(i <= k ? k * (k + 1) / 2 + i : i * (i + 1) / 2 + k) * T]; };
      auto kv = [&](int k, int i) { return sw[(15 + 3 * k + i) * T]; };
      double y[5];
      zeta(R, y);
#pragma unroll
      for (int i = 0; i < 5; ++i) y[i] *= i < 2 ? c1 : c4;
#pragma unroll
      for (int k = 0; k < 9; ++k) dl.set(k, R[k]);
      asm volatile("" ::: "memory");                      // and R
      double J[25];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        double u[5], v[3];
#pragma unroll
        for (int i = 0; i < 5; ++i) u[i] = ku(k, i);
#pragma unroll
        for (int i = 0; i < 3; ++i) v[i] = kv(k, i);
        const double Y[9] = {u[0], u[4] - v[2], u[3] - v[1], u[4] + v[2], u[1], u[2] - v[0], u[3] + v[1], u[2] + v[0],
                             -(u[0] + u[1])};
        double o[5];
        zeta(Y, o);
#pragma unroll
        for (int i = 0; i < 5; ++i) J[5 * i + k] = fma(i < 2 ? c1 : c4, o[i], i == k ? 1.0 : 0.0);
      }
      if (qr_solve<5>(J, y)) return 8;                   // singular: STATUS_FAIL_PHASE_MECHANICAL_STRESS_LP_DGESV
      double d[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int k = 0; k < 5; ++k) {
#pragma unroll
        for (int i = 0; i < 5; ++i) d[i] = fma(ku(k, i), y[k], d[i]);
#pragma unroll
        for (int i = 0; i < 3; ++i) d[5 + i] = fma(kv(k, i), y[k], d[5 + i]);
      }
      const double D[9] = {d[0], d[4] - d[7], d[3] - d[6], d[4] + d[7], d[1], d[2] - d[5], d[3] + d[6], d[2] + d[5],
                           -(d[0] + d[1])};
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        X[k] = D[k] - dl.get(k);
        dl.set(k, X[k]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) X[k] = dl.get(k);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) Lg[k] = fma(X[k], step, lo.get(k));
  }
  double s6[6];
  hooke_S<NS>(pc, Fe, s6);
  if (stress_end(Fp0g, N, B, Fe, s6, Fp, Pout)) return 5;
#pragma unroll
  for (int k = 0; k < 9; ++k) Lp[k] = Lg[k];
#pragma unroll
  for (int k = 0; k < 6; ++k) S[k] = s6[k];
  return 0;
}

// Hardening matrix staged in shared memory once per block (row = reacting system),
// read with uniform addresses (broadcast) in the control kernels.
// doubles of shared memory for the hardening matrix: staged up to 24 systems; at 48 (18 KB) the
// control and begin kernels read it from device memory (uniform addresses, L1 resident), so that
// four 64-thread blocks fit per SM instead of three
template <int NS>
__host__ __device__ constexpr size_t hard_smem_doubles() { return NS <= 24 ? size_t(NS) * NS : 0; }

template <int NS>
__device__ __forceinline__ void stage_hardening(const PhaseConst<NS>& pc, double* hs) {
  for (int i = threadIdx.x; i < NS * NS; i += blockDim.x) hs[i] = pc.hmat[i];
}

// phenopowerlaw_dotState (Fi = I => Mp = S; no twins => sumF = 0) at the given
// stress and state (state(i): value i of the voxel), written to this thread's slots: xi rates first, then
// |dot_gamma|.  hs: the hardening matrix (shared memory, or device memory read with uniform
// addresses).  adg_in (element s at adg_in[s * adg_stride]), when given, holds |dot_gamma| at
// this stress and state already (the kinetics of the converged integrateStress); otherwise
// the kinetics are evaluated.  Returns true if any rate is NaN.
template <int NS, class State>
__device__ __forceinline__ bool dot_state_slots(const PhaseConst<NS>& pc, const double* __restrict__ hs,
                                                const double s6[6], const State& state, double* xs,
                                                const double* adg_in, int64_t adg_stride) {
  double adg[NS];
  if (adg_in) {
#pragma unroll
    for (int s = 0; s < NS; ++s) adg[s] = adg_in[s * adg_stride];
  } else {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const double tp = dot6(s6, pc.p6[0][s]), tn = dot6(s6, pc.p6[1][s]);
      const double tmax = tp > tn ? tp : tn;
      adg[s] = fabs(pc.dg0[s] * powr(tmax / state(s), pc.n[s], pc.n_int[s]));
    }
  }
  bool bad = false;
  // xi of every system into the slots first, so that the loads overlap
#pragma unroll 8
  for (int l = 0; l < NS; ++l) xs[l * pass_threads<NS>()] = state(l);
#pragma unroll 2
  for (int l = 0; l < NS; ++l) {
    const double x = fma(-xs[l * pass_threads<NS>()], pc.ixiinf[l], 1.0);  // 1 - xi/xi_inf
    const double left = copysign(powr(fabs(x), pc.a[l], pc.a_int[l]), x);
    const double2* hrow = reinterpret_cast<const double2*>(hs + l * NS);
    double hg = 0.0;
#pragma unroll
    for (int k = 0; k < NS / 2; ++k) {
      const double2 hh = hrow[k];
      hg = fma(hh.x, adg[2 * k], hg);
      hg = fma(hh.y, adg[2 * k + 1], hg);
    }
    const double d = pc.h0f[l] * left * hg;
    bad |= isnan(d);
    xs[l * pass_threads<NS>()] = d;
  }
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    bad |= isnan(adg[s]);
    xs[(NS + s) * pass_threads<NS>()] = adg[s];
  }
  return bad;
}

// damper, phase_mechanical.f90:653-674
__device__ __forceinline__ double damper(double d01, double d12, double d22) {
  if (fmin(d01, d12) < 0.0 && d22 > 0.0) return 0.75 + 0.25 * tanh(2.0 + 4.0 * d12 / d22);
  return 1.0;
}

// Substep-start values (subF0, subFp0, subLp0, subState0 of phase_mechanical_constitutive).
// Until the first substep of an evaluation has advanced (stepFrac == 0) they equal the
// increment-start values F0, Fp0, Lp0, state0 and are read from there; the first advance
// writes them to the pass records, which are read from then on.
struct SubStart {
  const double *F0, *Fp0, *Lp0, *st0;
};
__device__ __forceinline__ SubStart sub_start(const Fields& f, const PassWork& w, double stepFrac) {
  const bool first = stepFrac == 0.0;
  return {first ? f.F0 : w.F0s, first ? f.Fp0 : w.Fp0s, first ? f.Lp0 : w.Lp0s, first ? f.state0 : w.st0s};
}

// dotState generations of the state iteration alternate between two 2NS-plane arrays:
// iteration it (0 = the start) stores its damped rate in array it % 2, which then holds
// dotState_last(:,1) for iteration it + 1 and dotState_last(:,2) for iteration it + 2.
__device__ __forceinline__ double* dot_gen(const PassWork& w, int it, int NST, int64_t N) {
  return w.D + int64_t(it & 1) * NST * N;
}

// Advances voxel v through the control flow of phase_mechanical_constitutive and
// integrateStateFPI until its next integrateStress (phase PH_STRESS) or its end
// (PH_DONE).  Entered in PH_CTRL (substep control after an integration attempt) or
// PH_DOT1 (state update after a successful integrateStress, whose |dot_gamma| is at
// adg[s * adg_stride]).
template <int NS>
__device__ void advance(const PhaseConst<NS>& pc, const double* __restrict__ hs, const Numerics& nm, const Fields& f,
                        const PassWork& w, int64_t v, double dt, VoxelCtl& c, double* xs, const double* adg,
                        int64_t adg_stride) {
  constexpr int NST = 2 * NS;
  const int64_t N = f.N;
  // every control step shrinks the substep or advances stepFrac; the bound only guards against
  // numerics (r_cutback >= 1) under which the reference loops forever, within one call (the calls of
  // an evaluation: Numerics::max_passes)
  for (int guard = 0; c.phase != PH_STRESS && c.phase != PH_DONE; ++guard) {
    if (guard > 4096) { c.status = 3; c.phase = PH_DONE; break; }
    if (c.phase == PH_CTRL) {
      // substep control, phase_mechanical.f90:1040-1080
      c.from_start = false;
      bool todo;
      if (c.status == 0) {
        c.stepFrac = c.stepFrac + c.step;
        c.step = fmin(1.0 - c.stepFrac, nm.r_increase * c.step);
        todo = c.step > 0.0;
        if (todo) {
#pragma unroll
          for (int k = 0; k < 9; ++k) {
            w.F0s[k * N + v] = w.Fs[k * N + v];
            w.Lp0s[k * N + v] = f.Lp[k * N + v];
            w.Fp0s[k * N + v] = f.Fp[k * N + v];
          }
#pragma unroll 12
          for (int i = 0; i < NST; ++i) w.st0s[i * N + v] = f.state[i * N + v];
        }
      } else {
        c.step = nm.r_cutback * c.step;
        const SubStart ss = sub_start(f, w, c.stepFrac);
#pragma unroll
        for (int k = 0; k < 9; ++k) f.Fp[k * N + v] = ss.Fp0[k * N + v];
#pragma unroll
        for (int k = 0; k < 6; ++k) f.S[k * N + v] = f.S0[k * N + v];
        if (c.step < 1.0)
#pragma unroll
          for (int k = 0; k < 9; ++k) f.Lp[k * N + v] = ss.Lp0[k * N + v];
#pragma unroll 12
        for (int i = 0; i < NST; ++i) f.state[i * N + v] = ss.st0[i * N + v];
        todo = c.step > nm.r_cutback_min;
      }
      if (!todo) { c.phase = PH_DONE; break; }
      ++c.nsub;
      const double* F0s = sub_start(f, w, c.stepFrac).F0;
#pragma unroll
      for (int k = 0; k < 9; ++k)
        w.Fs[k * N + v] = fma(c.step, f.F[k * N + v] - f.F0[k * N + v], F0s[k * N + v]);
      c.phase = PH_DOT0;
    } else {
      // dotState at the current stress and state: start (DOT0) or update (DOT1) of a state
      // iteration; after a converged integrateStress its kinetics are stored already
      double s6[6];
      const bool after_stress = c.phase == PH_DOT1;
      if (!after_stress)
#pragma unroll
        for (int k = 0; k < 6; ++k) s6[k] = f.S[k * N + v];
      const double dts = c.step * dt;
      // the first update after a start from the increment-start values
      const bool fresh = after_stress && c.from_start && c.it == 1;
      const double* st0 = sub_start(f, w, c.stepFrac).st0 + v;
      const double* stv = fresh ? w.dot0 + v : f.state + v;
      auto state = [&](int i) {
        const double x = stv[i * N];
        return fresh ? fma(x, dts, st0[i * N]) : x;
      };
      const bool bad = dot_state_slots<NS>(pc, hs, s6, state, xs, after_stress ? adg : nullptr, adg_stride);
      if (c.phase == PH_DOT0) {
        // integrateStateFPI:616-620
        if (bad) { c.status = 3; c.phase = PH_CTRL; continue; }   // STATUS_FAIL_PHASE_MECHANICAL_STATE
        double* D0 = dot_gen(w, 0, NST, N) + v;
#pragma unroll 12
        for (int i = 0; i < NST; ++i) {
          const double d = xs[i * pass_threads<NS>()];
          f.state[i * N + v] = fma(d, dts, st0[i * N]);
          D0[i * N] = d;
        }
        c.it = 0;
        c.phase = PH_STRESS;
      } else {
        // integrateStateFPI:631-646 (the stress integration of this iteration succeeded: status 0)
        if (bad) {
          // the state stays what this iteration started from, which a fresh start has not stored
          if (fresh)
#pragma unroll 1
            for (int i = 0; i < NST; ++i) f.state[i * N + v] = state(i);
          c.phase = PH_CTRL;
          continue;
        }
        // generations: dotState of the last iteration (it - 1) and the one before (it - 2,
        // whose storage receives the damped rate of this iteration)
        const double* L1 = fresh ? w.dot0 + v : dot_gen(w, c.it + 1, NST, N) + v;
        double* L2 = dot_gen(w, c.it, NST, N) + v;
        const double* L2r = c.from_start && c.it == 2 ? w.dot0 + v : L2;
        double d01 = 0.0, d12 = 0.0, d22 = 0.0;
#pragma unroll 24
        for (int i = 0; i < NST; ++i) {
          const double d = xs[i * pass_threads<NS>()];
          const double l1 = L1[i * N];                                 // dotState_last(:,1)
          const double l2 = c.it > 1 ? L2r[i * N] : 0.0;              // dotState_last(:,2)
          const double a = d - l1, b = l1 - l2;
          d12 = fma(a, b, d12);
          d22 = fma(b, b, d22);
          d01 = fma(d, l1, d01);
        }
        const double zeta = damper(d01, d12, d22);
        if (zeta != 1.0)                                              // rarely: the damped rate
#pragma unroll 12
          for (int i = 0; i < NST; ++i)
            xs[i * pass_threads<NS>()] = fma(xs[i * pass_threads<NS>()], zeta, L1[i * N] * (1.0 - zeta));
        bool conv = true;
#pragma unroll 12
        for (int i = 0; i < NST; ++i) {
          const double d = xs[i * pass_threads<NS>()];
          const double x0 = st0[i * N];
          const double x = stv[i * N];
          const double st = fresh ? fma(x, dts, x0) : x;
          const double r = fma(-d, dts, st - x0);
          const double stn = st - r;
          f.state[i * N + v] = stn;
          const double atol = i < NS ? pc.atol_xi : pc.atol_gamma;
          conv = conv && (fabs(r) <= fmax(atol, nm.eps_rel_state * fabs(stn)));
        }
        // the rate of this iteration is read by the next ones only
        if (!conv && c.it < nm.N_iter_state_max)
#pragma unroll 12
          for (int i = 0; i < NST; ++i) L2[i * N] = xs[i * pass_threads<NS>()];
        c.phase = (conv || c.it >= nm.N_iter_state_max) ? PH_CTRL : PH_STRESS;
      }
    }
  }
}

}  // namespace dmk
