// mrr.cuh -- dislocation-density hardening: twelve dislocation densities, one per slip system
// of a 12-system crystal, as the slip resistance variables.  Ma-Roters-Raabe (h_type 7,
// stress_mrr.cu) and ORNL (h_type 4, stress_ornl.cu: the same hardening law with the
// temperature-dependent shear modulus mu(T) = mu_0 - D_0 / (exp(T_0 / T) - 1), and its own
// slip law, mm10_slipinc_ornl .. mm10_dgdh_ornl, src/mm10_b.f:3457-4347).  Included by
// stress.cu when it is compiled with CPFFT_LAW 7 or 4.
//
// The slip law, hardening law and their derivatives follow mm10_slipinc_mrr ..
// mm10_dgdd_mrr (src/mm10_b.f:2343-3325); the local solve is mm10_solve
// (src/mm10_a.f:2860-3295) with 6 + 12 unknowns, the tangent mm10_tangent (:658-815) with
// ed = dgammadd = 0.  exact_j22 = 0 forms the Jacobian with the reference's formulas
// (sqrt(rho_F) in d h / d sigma and d h / d rho where mm10_h_mrr has sqrt(rho_P); no sign
// of tau on estress's c8 term; the fract > 1 branch of dgdt / dgdh drops terms), which
// slow the local Newton to linear convergence; exact_j22 = 1 differentiates the residual.
//
// Layout: half a warp per voxel, a lane per slip system.  One thread per voxel kept the
// 18 x 18 Jacobian and its LU in 15.7 KB of local memory, and 32 voxels' line searches and
// iteration counts diverged (10.5 of 32 lanes active, ncu): 46 ms for an implicit pass at
// 32^3, 60 % FP64 pipe.  Here each lane holds its system's slip, its rows of J21 and J22 in
// registers; the twelve rows are eliminated by Gauss-Jordan with the pivot row broadcast by
// shuffles, the 6 x 6 Schur complement S = J11 - J12 J22^-1 J21 is summed through shared memory
// and solved the same way, and S of the last iteration is the consistent tangent's matrix.
// d slip_a / d rho_q and J22's row are linear in the interaction matrices' rows, so an entry
// takes two products where the reference's formulas take about forty.  The two voxels of a
// warp run one loop whose every round is one residual evaluation, each in its own phase.
// The work that has no lanes to share (kinematics; rotation, P, dP/dF) runs in kernels with a
// thread per voxel before and after.  32^3, one implicit pass: 45.3 to 10.6 ms.

constexpr int NH = 12;  // dislocation densities
constexpr bool ORNL = CPFFT_LAW == 4;
constexpr double MRR_PI = 3.141592653589793;
constexpr double MRR_NU = 0.3;  // Poisson's ratio of the dipole distance (mm10_h_mrr)

// per-voxel scratch that mrr_solve hands to mrr_post in the voxel's K4 words
enum { MT_CEP = 0, MT_WB = 36, MT_STATE = 39 };
enum { MS_SOLVED = 0, MS_FAILED = 1, MS_EXPLICIT = 2 };

// constants of the law at a (sub)step, one set per voxel in shared memory
enum { LC_DT, LC_IDT, LC_QK, LC_G0, LC_PASS, LC_CUT, LC_DIP, LC_M, LC_E, LC_C4B, LC_C6B, LC_D0, LC_N };

constexpr int MRR_NT = 128, MRR_VB = MRR_NT / 16;  // voxels per block

struct MrrShared {
  double M[NH][9];    // per system: ms 0, 1, 3, 4, 5 (trace free), qc 0..2
  double W[NH][14];   // per system: wv 0..5, z 0..5, u_y
  double S[6][8];     // Schur complement and right-hand side
  double Sl[6][6];    // S of the last coupled iteration (the tangent's)
  double C[36];
  double lc[LC_N];
};

__device__ __forceinline__ double half_sum(double v) {
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// one system at (sigma, rho): mm10_slipinc_mrr (src/mm10_b.f:2477-2546) and the pieces of
// its derivatives
struct MrrLane {
  double rs, rhoF, rhoP, sF, sP, g0, tpass, itcut, fract, slip, sg0, dsf, m, gd, gdc8, h;
};

__device__ __forceinline__ void mrr_eval(const CrysRec& c, const double* lc, const double* Gr,
                                         const double* Hr, const double* ms, const double* sig,
                                         double rho, double nrho, int sl, MrrLane& y) {
  y.rs = (sig[0] - sig[2]) * ms[0] + (sig[1] - sig[2]) * ms[1] + sig[3] * ms[2] + sig[4] * ms[3] +
         sig[5] * ms[4];
  double f = 0.0, p = 0.0;
#pragma unroll
  for (int q = 0; q < NH; q++) {
    const double r = __shfl_sync(0xffffffffu, rho, q, 16);
    f += __ldg(Gr + q) * r;
    p += __ldg(Hr + q) * r;
  }
  y.rhoF = f;
  y.rhoP = p;
  y.sF = sqrt(f);
  y.sP = sqrt(p);
  // ORNL: mobile density 0.1 rho_a, cutting stress tau_0 mu(T) / mu_0
  y.g0 = lc[LC_G0] * (ORNL ? rho : y.sP);
  y.tpass = lc[LC_PASS] * y.sP;
  y.itcut = 1.0 / (ORNL ? lc[LC_CUT] : lc[LC_CUT] * y.sF);
  const double ars = fabs(y.rs), sg = sgn1(y.rs), Qk = lc[LC_QK], dt = lc[LC_DT];
  y.fract = (ars - y.tpass) * y.itcut;
  y.sg0 = 0.0;
  y.dsf = 0.0;
  y.m = 0.0;
  y.slip = 0.0;
  if (y.fract > 1.0) {  // linear extrapolation past fract = 1
    y.m = y.g0 * (c.q_v * Qk * c.p_v) * sg * y.itcut;
    y.slip = dt * (y.m * y.fract + y.g0);
  } else if (ars > 0.0) {
    // exp(-Q / kT (1 - fract^p)^q); ORNL takes p = 1 below the passing stress
    const double pe = ORNL && y.fract < 0.0 ? 1.0 : c.p_v;
    double fp, fp1;
    if (pe == 1.0) { fp = y.fract; fp1 = 1.0; }
    else if (pe == 0.5) { fp = sqrt(y.fract); fp1 = 1.0 / fp; }
    else { fp = pow(y.fract, pe); fp1 = pow(y.fract, pe - 1.0); }
    const double base = 1.0 - fp;
    const double bq1 = c.q_v == 2.0 ? base : pow(base, c.q_v - 1.0);
    const double bq = c.q_v == 2.0 ? base * base : pow(base, c.q_v);
    y.sg0 = dt * sg * exp(-Qk * bq);
    y.slip = y.sg0 * y.g0;
    y.dsf = y.slip * Qk * c.q_v * bq1 * pe * fp1;
  }
  // mm10_h_mrr's four terms (src/mm10_b.f:2549-2646)
  y.gd = fabs(y.slip * lc[LC_IDT]);
  y.gdc8 = c.tab_c8 ? tpow(c.tab_c8, y.gd) : pow(y.gd, c.tau_hat_v);
  const double ddip = lc[LC_DIP] / ars, rhoM = lc[LC_M] * y.sF * y.sP;
  const double tem = (lc[LC_C4B] * y.sP + lc[LC_C6B] * ddip * rhoM - c.u5 * rho) * y.gd -
                     lc[LC_E] * ars * rho * rho * y.gdc8;
  y.h = nrho + dt * tem;
}

// Derivatives of system a at y: dsl = d slip / d rs; d slip / d rho_q = aH H_aq + aG G_aq +
// (a == q) aD (mm10_dgdt_mrr, mm10_dgdh_mrr, src/mm10_b.f:3111-3306, mm10_dgdh_ornl
// :4224-4347); et = d h / d rs (mm10_estress_mrr :2859-2963); J22's row jH H_aq + jG G_aq +
// (a == q) jD (mm10_ehard_mrr :2966-3092)
struct MrrDeriv {
  double dsl, aH, aG, aD, et, jH, jG, jD;
};

__device__ __forceinline__ void mrr_deriv(const CrysRec& c, const double* lc, const MrrLane& y,
                                          double rho, MrrDeriv& d) {
  const double sg = sgn1(y.rs), sgs = sgn1(y.slip), ars = fabs(y.rs), dt = lc[LC_DT];
  const double iP = 1.0 / y.sP, iF = 1.0 / y.sF;
  const double gH = ORNL ? 0.0 : 0.5 * y.g0 * iP * iP, D0 = ORNL ? lc[LC_D0] : 0.0;
  const double pH = 0.5 * y.tpass * iP * iP * y.itcut;            // d tau_pass / tau_cut
  const double cG = ORNL ? 0.0 : 0.5 * iF * iF;                   // d tau_cut / tau_cut
  const bool exact = c.exact_j22 != 0;
  d.dsl = d.aH = d.aG = d.aD = 0.0;
  if (y.fract > 1.0) {
    const double K = c.q_v * lc[LC_QK] * c.p_v * sg * y.itcut;
    if (exact) {
      d.dsl = dt * y.m * sg * y.itcut;
      d.aH = dt * (K * gH * y.fract - y.m * pH + gH);
      d.aG = dt * (-K * y.g0 * cG * y.fract - y.m * y.fract * cG);
      d.aD = dt * D0 * (K * y.fract + 1.0);
    } else {
      d.dsl = dt * y.m;
      d.aH = dt * K * gH;
      d.aG = -dt * K * y.g0 * cG;
      d.aD = dt * K * D0;
    }
  } else if (ars > 0.0) {
    d.dsl = y.dsf * sg * y.itcut;
    d.aH = y.sg0 * gH - y.dsf * pH;
    d.aG = -y.dsf * y.fract * cG;
    d.aD = y.sg0 * D0;
  }
  const double ddip = lc[LC_DIP] / ars, dddip = -ddip / ars * sg;
  const double rhoM = lc[LC_M] * y.sF * y.sP, hM = 0.5 * lc[LC_M] * iP * iF;
  const double gdc8 = y.gd == 0.0 ? 0.0 : y.gdc8;              // gd^c8 (0 at gd = 0, c8 > 0)
  const double gdc81 = y.gd == 0.0 ? 0.0 : y.gdc8 / y.gd;      // gd^(c8 - 1), only where gd != 0
  const double s4 = exact ? y.sP : y.sF;                        // the reference differentiates sqrt(rho_F)
  const double sd = (exact ? sgs : sg) * (d.dsl * lc[LC_IDT]);  // d gd / d rs
  const double bad = c.tau_hat_v * ars * gdc81 * (exact ? sd : d.dsl * lc[LC_IDT]);
  d.et = dt * (lc[LC_C4B] * s4 * sd + lc[LC_C6B] * rhoM * (ddip * sd + dddip * y.gd) -
               c.u5 * rho * sd - lc[LC_E] * rho * rho * (bad + sg * gdc8));
  const double eS = -(exact ? sgs : sg) *
                    (lc[LC_C4B] * s4 + lc[LC_C6B] * ddip * rhoM - c.u5 * rho -
                     lc[LC_E] * ars * rho * rho * c.tau_hat_v * gdc81);
  const double dip = lc[LC_C6B] * ddip * y.gd * hM;
  const double e4 = lc[LC_C4B] * 0.5 * (exact ? iP : iF) * y.gd;
  const double eH = -dt * ((exact ? e4 : 0.0) + dip * y.rhoF);
  const double eG = -dt * ((exact ? 0.0 : e4) + dip * y.rhoP);
  const double ed = 1.0 + dt * (c.u5 * y.gd + lc[LC_E] * ars * 2.0 * rho * gdc8);
  d.jH = eH + d.aH * eS;
  d.jG = eG + d.aG * eS;
  d.jD = ed + d.aD * eS;
}

// Gauss-Jordan of K rows spread over the lanes 0 .. K - 1 of each half warp, a row of K + R
// columns a lane, with partial pivoting and no row exchange: on return lane a's m[K ..]
// holds row a of (K x K block)^-1 (the R right-hand columns).  The pivot is the largest
// high word (magnitude to 2^-16) among the rows not yet used.
template <int K, int R>
__device__ __forceinline__ void half_solve(double* m, int sl) {
  const unsigned half = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  double ipiv = 1.0;
  int used = sl < K ? -1 : K, where = 0;  // step at which this lane's row was the pivot
#pragma unroll
  for (int k = 0; k < K; k++) {
    unsigned key = 0u;
    if (used < 0) key = (((unsigned)__double2hiint(m[k]) & 0x7ffffff0u) | (unsigned)(15 - sl));
    const unsigned best = __reduce_max_sync(half, key);
    const int p = 15 - (int)(best & 15u);
    const double piv = __shfl_sync(0xffffffffu, m[k], p, 16);
    const double inv = 1.0 / piv;
    const bool mine = sl == p;
    const double f = mine ? 0.0 : m[k] * inv;
    if (mine) { used = k; ipiv = inv; }
    if (sl == k) where = p;  // unknown k is solved in lane p
#pragma unroll
    for (int j = k + 1; j < K + R; j++) {
      const double r = __shfl_sync(0xffffffffu, m[j], p, 16);
      m[j] -= f * r;
    }
  }
#pragma unroll
  for (int j = K; j < K + R; j++) {
    m[j] *= ipiv;
    m[j] = __shfl_sync(0xffffffffu, m[j], where, 16);
  }
}

// kinematics of every voxel: the unrotated increment into the history's D words at n+1 and
// the rotation at n+1 into its Rp words (mrr_post writes the plastic rotation there)
__global__ void __launch_bounds__(128) mrr_pre(StressArgs a) {
  const long long v = (long long)blockIdx.x * 128 + threadIdx.x, N3 = a.N3;
  if (v >= N3 || (a.mises && __ldg(a.mises + v) >= 0)) return;
  double Fn[9], Fn1[9], rnh[9], rn1[9], fnhinv[9], uddt[6];
  for (int i = 0; i < 9; i++) {
    Fn[i] = __ldg(a.Fn + i * N3 + v);
    Fn1[i] = __ldg(a.Fn1 + i * N3 + v);
  }
  kinematics(Fn, Fn1, rnh, rn1, fnhinv, uddt);
  for (int i = 0; i < 6; i++) a.hist_np1[(H_D + i) * N3 + v] = uddt[i];
  for (int i = 0; i < 9; i++) a.hist_np1[(H_RP + i) * N3 + v] = rn1[i];
}

// mm10_solve_strup with mm10_solve and the tangent, two voxels a warp
__global__ void __launch_bounds__(MRR_NT) mrr_solve(StressArgs a) {
  __shared__ MrrShared sh_all[MRR_VB];
  const long long N3 = a.N3;
  const int sl = threadIdx.x & 15, sys = sl < NH ? sl : 0;
  const unsigned halfmask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  MrrShared& sh = sh_all[threadIdx.x >> 4];
  unsigned long long st_it = 0, st_pit = 0, st_fail = 0, st_cut = 0;
  const long long groups = (N3 + MRR_VB - 1) / MRR_VB;
  for (long long grp = blockIdx.x; grp < groups; grp += gridDim.x) {
    const long long vi = grp * MRR_VB + (threadIdx.x >> 4), v = vi < N3 ? vi : N3 - 1;
    const bool mine = vi < N3 && (!a.mises || __ldg(a.mises + v) < 0);
    const OriRec* rec = a.oris + __ldg(a.ori + v);
    const CrysRec& c = a.cryss[__ldg(a.crys + v)];
    const double* Gr = c.Gm + NH * sys;
    const double* Hr = c.Hm + NH * sys;
    // ---- state at n (step 1: mm10_init_mrr, src/mm10_a.f:2205-2223)
    double nsig[6], nD[6], D[6], nRp[9], nrho, nrate, R[9];
    for (int i = 0; i < 6; i++) D[i] = mine ? a.hist_np1[(H_D + i) * N3 + v] : 0.0;
    for (int i = 0; i < 9; i++) R[i] = mine ? a.hist_np1[(H_RP + i) * N3 + v] : 0.0;
    if (a.step == 1 || !mine) {
      for (int i = 0; i < 6; i++) { nsig[i] = 0.0; nD[i] = 0.0; }
      nrho = c.theta_0 == 0.0 ? 1.0e8 : c.theta_0;
      nrate = 0.0;
      for (int i = 0; i < 9; i++) nRp[i] = (i % 4 == 0) ? 1.0 : 0.0;
    } else {
      for (int i = 0; i < 6; i++) nsig[i] = a.hist_n[(H_SIG + i) * N3 + v];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) nRp[3 * i + j] = a.hist_n[(H_RP + 3 * j + i) * N3 + v];
      for (int i = 0; i < 6; i++) nD[i] = a.hist_n[(H_D + i) * N3 + v];
      nrho = a.hist_n[(H_RHO + sys) * N3 + v];
      nrate = a.hist_n[(H_RHO + NH + sys) * N3 + v];
    }
    // ---- this lane's system: Schmid tensor, spin vector and C ms (setup_np1)
    double ms[5], qc[3], Cms[6], qs[3];  // ms: components 0, 1, 3, 4, 5
    __syncwarp();
    for (int i = sl; i < 36; i += 16) sh.C[i] = __ldg(rec->C + i);
    {
      double tr[9], work[9], RW[9], RE[36], q0[3], m0[6];
      for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) tr[3 * i + j] = nRp[3 * j + i];
      for (int k = 0; k < 6; k++) m0[k] = __ldg(rec->ms + 6 * sys + k);
      for (int k = 0; k < 3; k++) q0[k] = __ldg(rec->qs + 3 * sys + k);
      rt2rve(tr, RE);
      double mf[6];
      for (int i = 0; i < 6; i++) {
        double s = 0.0;
        for (int j = 0; j < 6; j++) s += RE[6 * i + j] * m0[j];
        mf[i] = s;
      }
      ms[0] = mf[0]; ms[1] = mf[1]; ms[2] = mf[3]; ms[3] = mf[4]; ms[4] = mf[5];
      mm3(R, tr, work);
      rt2rvw(work, RW);
      for (int k = 0; k < 3; k++) qc[k] = RW[3 * k] * q0[0] + RW[3 * k + 1] * q0[1] + RW[3 * k + 2] * q0[2];
      rt2rvw(tr, RW);
      for (int k = 0; k < 3; k++) qs[k] = RW[3 * k] * q0[0] + RW[3 * k + 1] * q0[1] + RW[3 * k + 2] * q0[2];
      __syncwarp();
      for (int i = 0; i < 6; i++) {
        double s = 0.0;
        for (int j = 0; j < 6; j++) s += sh.C[6 * i + j] * mf[j];
        Cms[i] = s;
      }
    }
    if (sl < NH) {
      for (int k = 0; k < 5; k++) sh.M[sl][k] = ms[k];
      for (int k = 0; k < 3; k++) sh.M[sl][5 + k] = qc[k];
    }
    double t1 = 0, t2 = 0;
    for (int i = 0; i < 6; i++) { t1 += D[i] * D[i]; t2 += nsig[i] * nsig[i]; }
    const bool no_load = t1 == 0.0 && t2 == 0.0;
    const bool expl = a.iter == 0 || no_load;
    // cos of the angle between the deviators of D and D_n (mm10_solve, :2975-3010); the
    // scale of a sub-step's D cancels
    double cosang = 0.0;
    {
      double d1[6], d2[6];
      for (int i = 0; i < 6; i++) { d1[i] = D[i]; d2[i] = nD[i]; }
      for (int k = 0; k < 2; k++) {
        double* d = k ? d2 : d1;
        const double dtr = (d[0] + d[1] + d[2]) / 3.0;
        d[0] -= dtr; d[1] -= dtr; d[2] -= dtr;
        double s = 0.0;
        for (int i = 0; i < 6; i++) s += d[i] * d[i];
        const double is = s == 0.0 ? 0.0 : 1.0 / sqrt(s);
        for (int i = 0; i < 6; i++) d[i] = s == 0.0 ? 0.0 : d[i] * is;
      }
      for (int i = 0; i < 6; i++) cosang += d1[i] * d2[i];
      cosang = fmax(cosang, 0.0);
    }
    // ---- the loop: one residual evaluation a round, each voxel in its own phase
    enum { PREDICT, UPDATE, DONE };
    int mode = mine ? PREDICT : DONE, it = 0, ls = 0, cuts = 0, iters = 0, piters = 0;
    bool first = true, fail = false, start = true;
    double frac = 0.0, stp = 1.0, sfr = 1.0;  // sfr: the sub-step's end as a fraction of the step
    double ost[6], orho = nrho, orate = 0.0;  // the last accepted sub-step's state
    for (int i = 0; i < 6; i++) ost[i] = nsig[i];
    double x[6], xn[6], dx[6], rho = nrho, rhon = nrho, drho = 0.0;
    for (int i = 0; i < 6; i++) { x[i] = nsig[i]; xn[i] = nsig[i]; dx[i] = 0.0; }
    double alpha = 1.0, ls1 = 0.0, stop2 = 0.0, inP2 = 0.0;
    MrrLane y;
    double R1 = 0.0;  // lane r < 6: component r of the stress residual
    for (;;) {
      if (start) {  // a sub-step (the whole step first): its constants and the predictor's start
        start = false;
        first = true;
        mode = mode == DONE ? DONE : PREDICT;
        it = 0;
        sfr = expl ? 1.0 : stp + frac;
        const double th = TEMP * sfr;  // n's temperature is zero (:2769)
        const double k = c.boltzman, b = c.burgers;
        const double G = ORNL ? c.mu_0 - c.D_0 / (exp(c.T_0 / th) - 1.0) : c.mu_0;
        const double dt = a.dt * sfr;
        __syncwarp(halfmask);
        if (sl == 0) {
          double* lc = sh.lc;
          lc[LC_DT] = dt;
          lc[LC_IDT] = 1.0 / dt;
          lc[LC_QK] = c.G_0_v / k / th;
          // ORNL: the attack frequency, exp(-G_0_y) when negative
          const double vs = c.G_0_y < 0.0 ? exp(-c.G_0_y) : c.G_0_y;
          lc[LC_D0] = 0.1 * vs * (c.u2 * b);
          lc[LC_G0] = ORNL ? lc[LC_D0] : c.G_0_y * k * th / (c.u1 * c.u3 * G * b * b);
          lc[LC_PASS] = c.u1 * G * b;
          lc[LC_CUT] = ORNL ? c.u3 * G / c.mu_0 : c.G_0_v / (c.u2 * c.u3 * b * b);
          lc[LC_DIP] = sqrt(3.0) * G * b / (16.0 * MRR_PI * (1.0 - MRR_NU));
          lc[LC_M] = (2.0 * k / (c.u1 * c.u2 * c.u3 * G * b * b * b)) * th;
          lc[LC_E] = c.tau_hat_y * exp(-c.tau_a / k / th) / (k * th);
          lc[LC_C4B] = c.u4 / b;
          lc[LC_C6B] = c.u6 / b;
        }
        __syncwarp(halfmask);
        for (int i = 0; i < 6; i++) { x[i] = ost[i]; xn[i] = ost[i]; }
        rho = expl ? nrho : nrho + cosang * nrate * (a.dt * stp);
        rhon = rho;
      }
      __syncwarp();
      // ---- residual at (xn, rhon)
      mrr_eval(c, sh.lc, Gr, Hr, ms, xn, rhon, nrho, sl, y);
      const double slip = sl < NH ? y.slip : 0.0;
      {
        // lanes 0 .. 7: dbar 0, 1, 3, 4, 5 and w 0 .. 2
        double o = 0.0;
        const int col = sl < 8 ? sl : 0;
#pragma unroll
        for (int q = 0; q < NH; q++) o += __shfl_sync(0xffffffffu, slip, q, 16) * sh.M[q][col];
        double db[6], w[3], sw[6];
        db[0] = __shfl_sync(0xffffffffu, o, 0, 16);
        db[1] = __shfl_sync(0xffffffffu, o, 1, 16);
        db[2] = -(db[0] + db[1]);
        for (int k = 0; k < 3; k++) {
          db[3 + k] = __shfl_sync(0xffffffffu, o, 2 + k, 16);
          w[k] = __shfl_sync(0xffffffffu, o, 5 + k, 16);
        }
        symsw(xn, w, sw);
        const int r = sl < 6 ? sl : 0;
        double t = 0.0;
        for (int j = 0; j < 6; j++) t += sh.C[6 * r + j] * (D[j] * sfr - db[j]);
        double xr = xn[0], nr = nsig[0], sr = sw[0];
#pragma unroll
        for (int k = 1; k < 6; k++)
          if (r == k) { xr = xn[k]; nr = nsig[k]; sr = sw[k]; }
        R1 = xr - nr - t + 2.0 * sr;
      }
      if (expl && mode != DONE) {  // mm10_solve_strup_a (src/mm10_a.f:2721-2743)
        for (int k = 0; k < 6; k++) {
          const double rk = __shfl_sync(halfmask, R1, k, 16);
          if (!no_load) x[k] = nsig[k] - rk;
        }
        rho = nrho;
        mode = DONE;
      }
      const double R2 = rhon - y.h;
      const double d1 = half_sum(sl < 6 ? R1 * R1 : 0.0);
      const double d2 = d1 + half_sum(sl < NH ? R2 * R2 : 0.0);
      bool need = false;
      if (mode != DONE) {
        const double dot = mode == PREDICT ? d1 : d2;
        if (first || 0.5 * dot <= ls1 * (1.0 - 2.0e-4 * alpha) || ls > 10) {
          bool bad = false;
          if (first) {
            inP2 = d1;
            stop2 = fmax(c.atol1 * c.atol1, c.rtol1 * c.rtol1 * d1);
            first = false;
          } else {
            for (int i = 0; i < 6; i++) x[i] = xn[i];
            rho = rhon;
            it++;
            const bool nan = anynan(x, 6) || (sl < NH && isnan(rho));
            bad = it > c.miter || __any_sync(halfmask, nan);
          }
          if (bad) {
            if (mode == PREDICT) piters += it;
            else iters += it;
            fail = true;
          } else if (mode == PREDICT) {
            need = true;
            if (!(d1 > stop2)) {  // on to the coupled Newton, from this point's residual
              piters += it;
              mode = UPDATE;
              it = 0;
              stop2 = fmax(c.atol * c.atol, c.rtol * c.rtol * (d2 == 0.0 ? inP2 : d2));
            }
          } else if (d2 > stop2) {
            need = true;
          } else {  // converged: accept the sub-step
            iters += it;
            for (int i = 0; i < 6; i++) ost[i] = x[i];
            orho = rho;
            orate = (y.h - nrho) * sh.lc[LC_IDT];
            frac += stp;
            if (frac < 1.0) start = true;
            else mode = DONE;
          }
          if (fail) {  // halve the sub-step, at most 4 times
            stp *= 0.5;
            if (++cuts > 4) {
              mode = DONE;
            } else {
              fail = false;
              start = true;
            }
          }
          ls1 = 0.5 * (mode == PREDICT ? d1 : d2);
          alpha = 1.0;
          ls = 0;
        } else {
          alpha *= 0.5;
          ls++;
          for (int i = 0; i < 6; i++) xn[i] = x[i] + alpha * dx[i];
          if (mode == UPDATE) rhon = rho + alpha * drho;
        }
      }
      if (!__any_sync(0xffffffffu, mode != DONE)) break;
      if (!__any_sync(0xffffffffu, need)) continue;
      // ---- Newton direction at (x, rho) = (xn, rhon), whose residual and slips are current
      const bool coupled = __any_sync(0xffffffffu, need && mode == UPDATE);
      MrrDeriv d;
      mrr_deriv(c, sh.lc, y, rhon, d);
      double wv[6], z[7];
      {
        double sq[6];
        symsw(xn, qc, sq);
        for (int r = 0; r < 6; r++) wv[r] = Cms[r] + 2.0 * sq[r];
        z[0] = d.dsl * ms[0];
        z[1] = d.dsl * ms[1];
        z[2] = -(z[0] + z[1]);
        for (int k = 0; k < 3; k++) z[3 + k] = d.dsl * ms[2 + k];
        z[6] = 0.0;
      }
      double B[7] = {0, 0, 0, 0, 0, 0, 0};  // this lane's row of J22^-1 [J21 | R2]
      if (coupled) {
        double m[NH + 7];
#pragma unroll
        for (int q = 0; q < NH; q++)
          m[q] = __ldg(Hr + q) * d.jH + __ldg(Gr + q) * d.jG + (q == sl ? d.jD : 0.0);
        m[NH + 0] = -d.et * ms[0];
        m[NH + 1] = -d.et * ms[1];
        m[NH + 2] = -(m[NH + 0] + m[NH + 1]);
        for (int k = 0; k < 3; k++) m[NH + 3 + k] = -d.et * ms[2 + k];
        m[NH + 6] = R2;
        half_solve<NH, 7>(m, sl);
        // z -= (d slip / d rho) B, u_y = (d slip / d rho) y
        double u[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < NH; q++) {
          const double s = __ldg(Hr + q) * d.aH + __ldg(Gr + q) * d.aG + (q == sl ? d.aD : 0.0);
#pragma unroll
          for (int k = 0; k < 7; k++) u[k] += s * __shfl_sync(0xffffffffu, m[NH + k], q, 16);
        }
        if (mode == UPDATE) {
          for (int k = 0; k < 6; k++) z[k] -= u[k];
          z[6] = u[6];
          for (int k = 0; k < 7; k++) B[k] = m[NH + k];
        }
      }
      __syncwarp();
      if (sl < NH) {
        for (int r = 0; r < 6; r++) sh.W[sl][r] = wv[r];
        for (int k = 0; k < 7; k++) sh.W[sl][6 + k] = z[k];
      }
      __syncwarp();
      {
        // S = I + IW + sum_a wv_a (x) z_a, right-hand side -R1 + sum_a wv_a u_y: lane 7 h + k
        // forms column k of rows 3 h .. 3 h + 2
        const int k = sl < 14 ? sl % 7 : 0, r0 = sl < 14 ? 3 * (sl / 7) : 0;
        double o0 = 0.0, o1 = 0.0, o2 = 0.0;
#pragma unroll
        for (int q = 0; q < NH; q++) {
          const double zz = sh.W[q][6 + k];
          o0 += sh.W[q][r0] * zz;
          o1 += sh.W[q][r0 + 1] * zz;
          o2 += sh.W[q][r0 + 2] * zz;
        }
        if (sl < 14) {
          sh.S[r0][k] = o0;
          sh.S[r0 + 1][k] = o1;
          sh.S[r0 + 2][k] = o2;
        }
        __syncwarp();
      }
      double m6[7];
      {
        // mm10_iw (src/mm10_b.f:1590-1634) with w = sum slip qc, and the identity
        double w[3] = {0, 0, 0};
        double o = 0.0;
        const int col = sl < 3 ? 5 + sl : 5;
#pragma unroll
        for (int q = 0; q < NH; q++) o += __shfl_sync(0xffffffffu, slip, q, 16) * sh.M[q][col];
        for (int k = 0; k < 3; k++) w[k] = __shfl_sync(0xffffffffu, o, k, 16);
        const int r = sl < 6 ? sl : 0;
        double iw[6] = {0, 0, 0, 0, 0, 0};
        if (r == 0) { iw[3] = 2.0 * w[2]; iw[5] = -2.0 * w[1]; }
        else if (r == 1) { iw[3] = 2.0 * w[2]; iw[4] = -2.0 * w[0]; }
        else if (r == 2) { iw[4] = 2.0 * w[0]; iw[5] = 2.0 * w[1]; }
        else if (r == 3) { iw[0] = w[2]; iw[1] = -w[2]; iw[4] = -w[1]; iw[5] = w[0]; }
        else if (r == 4) { iw[1] = w[0]; iw[2] = -w[0]; iw[3] = w[1]; iw[5] = w[2]; }
        else { iw[0] = w[1]; iw[2] = -w[1]; iw[3] = w[0]; iw[4] = -w[2]; }
#pragma unroll
        for (int k = 0; k < 6; k++) m6[k] = sh.S[r][k] + iw[k] + (k == r ? 1.0 : 0.0);
        m6[6] = sh.S[r][6] - R1;
        if (need && mode == UPDATE && sl < 6)
          for (int k = 0; k < 6; k++) sh.Sl[sl][k] = m6[k];
      }
      half_solve<6, 1>(m6, sl);
      if (need) {
        for (int k = 0; k < 6; k++) {
          dx[k] = __shfl_sync(halfmask, m6[6], k, 16);
          xn[k] = x[k] + dx[k];
        }
        if (mode == UPDATE) {
          drho = -B[6];
          for (int k = 0; k < 6; k++) drho -= B[k] * dx[k];
          rhon = rho + drho;
        }
      }
    }
    // ---- results
    const bool ok = expl || !(fail || __any_sync(halfmask, anynan(ost, 6) || (sl < NH && isnan(orho))));
    // slips at the converged state (the last residual's) for the plastic rotation
    double wb[3];
    for (int k = 0; k < 3; k++) wb[k] = half_sum(sl < NH ? y.slip * qs[k] : 0.0);
    __syncwarp();
    // mm10_tangent (:658-815): T = S^-1 C with S of the last coupled iteration, symmetrised
    double T[12];
    const int r6 = sl < 6 ? sl : 0;
    for (int k = 0; k < 6; k++) {
      T[k] = ok && !expl ? sh.Sl[r6][k] : (k == r6 ? 1.0 : 0.0);
      T[6 + k] = sh.C[6 * r6 + k];
    }
    half_solve<6, 6>(T, sl);
    __syncwarp();
    if (sl < 6)
      for (int k = 0; k < 6; k++) sh.Sl[sl][k] = T[6 + k];
    __syncwarp();
    if (mine) {
      for (int e = sl; e < 36; e += 16) {
        const int r = e / 6, k = e % 6;
        const double t = ok && !expl ? (sh.Sl[r][k] + sh.Sl[k][r]) * 0.5 : sh.C[e];
        a.K4[(MT_CEP + e) * N3 + v] = t;
      }
      if (sl < 6) {
        double s = ost[0];
#pragma unroll
        for (int k = 0; k < 6; k++)
          if (sl == k) s = !ok ? nsig[k] : expl ? x[k] : ost[k];
        a.hist_np1[(H_SIG + sl) * N3 + v] = s;
      }
      if (sl < NH) {
        a.hist_np1[(H_RHO + sl) * N3 + v] = !ok || expl ? nrho : orho;
        a.hist_np1[(H_RHO + NH + sl) * N3 + v] = !ok || expl ? 0.0 : orate;
      }
      if (sl < 3) {
        a.K4[(MT_WB + sl) * N3 + v] = sl == 0 ? wb[0] : sl == 1 ? wb[1] : wb[2];
      } else if (sl == 3) {
        a.K4[MT_STATE * N3 + v] = expl ? MS_EXPLICIT : ok ? MS_SOLVED : MS_FAILED;
      }
      if (sl == 0) {
        st_it += iters;
        st_pit += piters;
        st_fail += ok ? 0 : 1;
        st_cut += cuts ? 1 : 0;
      }
    }
    __syncwarp();
  }
  if (a.stats) {  // lanes 0 and 16 hold their voxels' counts
    st_it += __shfl_down_sync(0xffffffffu, st_it, 16);
    st_pit += __shfl_down_sync(0xffffffffu, st_pit, 16);
    st_fail += __shfl_down_sync(0xffffffffu, st_fail, 16);
    st_cut += __shfl_down_sync(0xffffffffu, st_cut, 16);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(a.stats + 0, st_it);
      atomicAdd(a.stats + 1, st_fail);
      atomicAdd(a.stats + 2, st_pit);
      if (st_cut) atomicAdd(a.stats + 4, st_cut);
    }
  }
}

// plastic rotation (mm10_update_rotation, src/mm10_a.f:3310-3327), the remaining history
// words, P and dP/dF of every voxel
__global__ void __launch_bounds__(128) mrr_post(StressArgs a) {
  const long long v = (long long)blockIdx.x * 128 + threadIdx.x, N3 = a.N3;
  if (v >= N3 || (a.mises && __ldg(a.mises + v) >= 0)) return;
  double Fn[9], Fn1[9], rnh[9], rn1[9], fnhinv[9], uddt[6], cep[36], stress[6];
  for (int i = 0; i < 9; i++) {
    Fn[i] = __ldg(a.Fn + i * N3 + v);
    Fn1[i] = __ldg(a.Fn1 + i * N3 + v);
  }
  kinematics(Fn, Fn1, rnh, rn1, fnhinv, uddt);
  for (int i = 0; i < 36; i++) cep[i] = a.K4[(MT_CEP + i) * N3 + v];
  for (int i = 0; i < 6; i++) stress[i] = a.hist_np1[(H_SIG + i) * N3 + v];
  const int state = (int)a.K4[MT_STATE * N3 + v];
  double nRp[9], Rp[9];
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++)
      nRp[3 * i + j] = a.step == 1 ? (i == j ? 1.0 : 0.0) : a.hist_n[(H_RP + 3 * j + i) * N3 + v];
  if (state == MS_FAILED) {
    for (int i = 0; i < 9; i++) Rp[i] = nRp[i];
  } else if (state == MS_EXPLICIT) {
    for (int i = 0; i < 9; i++) Rp[i] = 0.0;
  } else {
    double wb[3];
    for (int k = 0; k < 3; k++) wb[k] = a.K4[(MT_WB + k) * N3 + v];
    const double W[9] = {0.0, wb[2], wb[1], -wb[2], 0.0, wb[0], -wb[1], -wb[0], 0.0};
    const double al = sqrt(W[5] * W[5] + W[2] * W[2] + W[1] * W[1]);
    double ex[9];
    if (al < 1.0e-16) {
      for (int i = 0; i < 9; i++) ex[i] = 0.0;
    } else {
      double WW[9];
      mm3(W, W, WW);
      const double ca = (1.0 - cos(al)) / (al * al), sa = sin(al) / al;
      for (int i = 0; i < 9; i++) ex[i] = ca * WW[i] + sa * W[i];
    }
    ex[0] += 1.0; ex[4] += 1.0; ex[8] += 1.0;
    mm3(ex, nRp, Rp);
  }
  a.hist_np1[H_TT * N3 + v] = 0.0;
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) a.hist_np1[(H_RP + 3 * j + i) * N3 + v] = Rp[3 * i + j];
  a.hist_np1[H_TTR * N3 + v] = 0.0;
  a.hist_np1[H_U * N3 + v] = 0.0;
  a.hist_np1[(H_U + 1) * N3 + v] = 0.0;
  for (int i = 0; i < 6; i++)
    a.hist_np1[(H_EPS + i) * N3 + v] = (a.step == 1 ? 0.0 : a.hist_n[(H_EPS + i) * N3 + v]) + uddt[i];
  store_P_K4(a, v, Fn, Fn1, stress, cep, rnh, rn1, fnhinv);
}
