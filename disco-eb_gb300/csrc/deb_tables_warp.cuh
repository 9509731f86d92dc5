// deb_tables_warp.cuh -- the ionisation history of one parameter set by a warp
// (device only): solve_ionization of deb_tables_core.cuh with the expressions
// of one RHS evaluation spread over the lanes.
//
// What bounds it.  A history is a chain of ~800 small adaptive steps, each with
// three RHS evaluations (one of them with the 3x3 Jacobian), and a warp gets one
// FP64 instruction per 64 cycles however many of its lanes are active: a pow
// takes ~6000 cycles, an exp ~1000, a division ~370.  On one lane an evaluation
// was ~9 pow (18 with derivatives), ~12 exp and ~40 divisions in sequence.
//
// The split.  Every function of one kind is taken by all lanes at once, each
// lane with its own argument: one division, one square root, one pow and one exp
// per evaluation.  The rest is evaluated for three species at once (lane & 3:
// HeI singlet, HeI triplet, H -- their rates have one form with different
// constants) and for the three derivative directions at once ((lane >> 2) % 3),
// so the Jacobian costs twice a plain evaluation instead of four times.  What
// depends on the scale factor alone is evaluated once per step, not once per
// stage.  All branch conditions are on values every lane holds.  26 sets of 256
// samples, leaders then followers: 252.6 ms on one lane, 79.6 ms.
#pragma once

#include "deb_tables_core.cuh"

#ifdef __CUDACC__

namespace debt {

// value and the derivative in this lane's direction
struct D1 {
  double v, d;
  __device__ D1() : v(0.0), d(0.0) {}
  __device__ D1(double x) : v(x), d(0.0) {}
  __device__ D1(double x, double y) : v(x), d(y) {}
};
__device__ __forceinline__ D1 operator+(D1 a, D1 b) { return D1(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ D1 operator-(D1 a, D1 b) { return D1(a.v - b.v, a.d - b.d); }
__device__ __forceinline__ D1 operator*(D1 a, D1 b) { return D1(a.v * b.v, a.d * b.v + a.v * b.d); }
__device__ __forceinline__ D1 operator/(D1 a, D1 b) {
  const double q = a.v / b.v;
  return D1(q, (a.d - q * b.d) / b.v);
}
__device__ __forceinline__ D1 operator+(D1 a, double b) { return D1(a.v + b, a.d); }
__device__ __forceinline__ D1 operator+(double a, D1 b) { return D1(a + b.v, b.d); }
__device__ __forceinline__ D1 operator-(D1 a, double b) { return D1(a.v - b, a.d); }
__device__ __forceinline__ D1 operator-(double a, D1 b) { return D1(a - b.v, -b.d); }
__device__ __forceinline__ D1 operator*(D1 a, double b) { return D1(a.v * b, a.d * b); }
__device__ __forceinline__ D1 operator*(double a, D1 b) { return b * a; }
__device__ __forceinline__ D1 operator/(D1 a, double b) { return D1(a.v / b, a.d / b); }
__device__ __forceinline__ double val(const D1& a) { return a.v; }
__device__ __forceinline__ double der(const D1& a) { return a.d; }
__device__ __forceinline__ double der(double) { return 0.0; }
__device__ __forceinline__ D1 sel(bool c, D1 a, D1 b) { return D1(c ? a.v : b.v, c ? a.d : b.d); }
__device__ __forceinline__ double sel(bool c, double a, double b) { return c ? a : b; }
template <class S> struct Mk { static __device__ __forceinline__ S of(double v, double d) { return S(v, d); } };
template <> struct Mk<double> { static __device__ __forceinline__ double of(double v, double) { return v; } };

struct IonWarp {
  static constexpr unsigned FULL = 0xffffffffu;
  // shared scratch: bases of the powers and their T derivatives, square roots,
  // powers, T derivatives of the powers, exponentials and theirs, constants
  enum { BV = 0, BD = 16, SV = 32, SD = 36, PV = 40, PD = 72, EV = 80, ED = 96, KC = 104, SHARED = KC + DEB_TC_COUNT };

  const Bk& B;
  double* sh;
  TC K;
  int lane, sp, dir;
  // this lane's task in the shared function passes
  double dc, dm, pe;
  int i1, i2;
  // this lane's species
  double A2p, tc, tf, g2n, g2d, ahc, ahn, rdn, rf, cU, lam, fu;
  int ia, ib, ie, il;
  double HO, Nnow;
  // functions of the scale factor at the last a
  double a = -1.0, zt, n, n_He, Trad, Trad4, Hz, Hzz, KK, timeH, dzda, tden;

  __device__ IonWarp(const TC& Kg, const Bk& B_, double* sh_, int lane_)
      : B(B_), sh(sh_), K{sh_ + KC}, lane(lane_), sp(lane_ & 3), dir((lane_ >> 2) % 3) {
    for (int i = lane; i < DEB_TC_COUNT; i += 32) sh[KC + i] = Kg[i];
    if (lane < 16) { sh[BV + lane] = 1.0; sh[BD + lane] = 0.0; }
    __syncwarp();
    const double c2 = K[DEB_TC_C] * K[DEB_TC_C];
    // divisions: constant / T (lanes 0 .. 7), T / constant (8 .. 11)
    const int nidx[8] = {DEB_TC_CDB, DEB_TC_CDB_HE, DEB_TC_BFACT, DEB_TC_HCL_HE2ST_ION_KB,
                         DEB_TC_CL, DEB_TC_CL_HE, DEB_TC_CL_PST, DEB_TC_HCL_HE2ST_KB};
    dc = 1.0; dm = 1.0; i1 = i2 = 0;
    for (int l = 0; l < 8; ++l) if (lane == l) dc = K[nidx[l]];
    if (lane == 8) { dc = 1e4; i1 = 1; i2 = 2; }
    if (lane == 9) { dc = K[DEB_TC_T0]; i1 = 3; i2 = 5; }
    if (lane == 10) { dc = K[DEB_TC_T1]; i1 = 4; i2 = 6; }
    if (lane == 11) { dm = 2.0 * K[DEB_TC_KB]; dc = K[DEB_TC_MH] * K[DEB_TC_MHE_MH] * c2; }
    // powers: exponent p on lane l, p - 1 (the derivative's) on lane 16 + l
    const double ex[11] = {1.5, K[DEB_TC_B_PPB], K[DEB_TC_D_PPB], 1.0 - K[DEB_TC_B_VF], 1.0 + K[DEB_TC_B_VF],
                           1.0 - K[DEB_TC_B_TRIP], 1.0 + K[DEB_TC_B_TRIP], 0.86, 0.9, 1.5, -3.0 * (1.0 + B.w0 + B.wa)};
    pe = 1.0;
    for (int l = 0; l < 11; ++l) {
      if (lane == l) pe = ex[l];
      if (lane == 16 + l) pe = ex[l] - 1.0;
    }
    const bool tr = sp == 1, h = sp >= 2;
    A2p = K[tr ? DEB_TC_A2P_T : DEB_TC_A2P_S];
    const double L = K[tr ? DEB_TC_L_HE_2PT : DEB_TC_L_HE_2P], cl = K[DEB_TC_C] * L;
    tc = tr ? 3.0 * A2p : A2p * K[DEB_TC_CK_HE] * 3.0;
    tf = tr ? 8.0 * K[DEB_TC_PI] * (L * L * L) : 1.0;
    g2n = 3.0 * A2p * B.fHe * c2;
    g2d = K[DEB_TC_SQRT_PI] * K[tr ? DEB_TC_SIGMA_HE_2PT : DEB_TC_SIGMA_HE_2PS] * 8.0 * K[DEB_TC_PI] * cl * (cl * cl);
    ahc = tr ? 0.66 : 0.36;
    ahn = tr ? A2p / 3.0 : A2p;
    rdn = h ? 1e-19 * K[DEB_TC_A_PPB] : K[tr ? DEB_TC_A_TRIP : DEB_TC_A_VF];
    rf = h ? 1.0 : (tr ? 4.0 / 3.0 : 4.0);
    cU = tr ? 3.0 : 1.0;
    lam = K[h ? DEB_TC_LAMBDA_H : DEB_TC_LAMBDA_HE];
    fu = h ? K[DEB_TC_FU] : 1.0;
    ia = h ? 2 : (tr ? 5 : 3);
    ib = h ? 1 : (tr ? 6 : 4);
    ie = h ? 0 : (tr ? 3 : 1);
    il = h ? 4 : (tr ? 7 : 5);
    const double H = B.H0 / 100.0, mu_H = 1.0 / (1.0 - B.YHe);
    HO = H * K[DEB_TC_BIG_H];
    Nnow = K[DEB_TC_DENS_FAC] * H * H * B.Ob / mu_H;
  }

  __device__ __forceinline__ double bc(double x, int src) const { return __shfl_sync(FULL, x, src); }
  __device__ __forceinline__ double row(const double* v) const { return dir == 0 ? v[0] : (dir == 1 ? v[1] : v[2]); }
  __device__ __forceinline__ void spread(double x, double* v) const { v[0] = bc(x, 0); v[1] = bc(x, 4); v[2] = bc(x, 8); }

  // functions of a alone; the powers of a and 1/a come from the evaluation's pass
  __device__ __forceinline__ void at_a(double an, double powzt, double powa) {
    const double lg = log(lane == 0 ? an : zt);
    const double la = bc(lg, 0), lz = bc(lg, 1);
    const double g1 = (lz - K[DEB_TC_ZGAUSS1]) / K[DEB_TC_WGAUSS1], g2 = (lz - K[DEB_TC_ZGAUSS2]) / K[DEB_TC_WGAUSS2];
    const double sl = spl_ab(B.lx, B.ly, B.lS, B.nnu, la);
    const double e = exp(lane == 0 ? sl : (lane == 1 ? 3.0 * (an - 1.0) * B.wa : (lane == 2 ? -(g1 * g1) : -(g2 * g2))));
    const double rhonu = bc(e, 0), rde = powa * bc(e, 1);
    const double grho = B.grhom * B.Om / an + (B.grhog + B.grhor * (B.Neff + B.Nmnu * rhonu)) / (an * an) +
                        B.grhom * B.ODE * rde * an * an + B.grhom * B.Ok;
    const double aH = sqrt(grho / 3.0);
    n = Nnow * zt * zt * zt;
    n_He = B.fHe * n;
    Trad = B.Tcmb * zt;
    Trad4 = Trad * Trad * Trad * Trad;
    Hz = (1e-5 * aH) / an * K[DEB_TC_C] * K[DEB_TC_BIG_H];
    Hzz = Hz * zt;
    KK = K[DEB_TC_CK] / Hz * (1.0 + K[DEB_TC_AGAUSS1] * bc(e, 2) + K[DEB_TC_AGAUSS2] * bc(e, 3));
    timeH = 2.0 / (3.0 * HO * powzt);
    dzda = -1.0 / (an * an);
    tden = tf * Hz;
    a = an;
  }

  // ion_rhs at (an, y); y and the values of f are held by every lane, the
  // derivatives of f by the lanes of their direction
  template <class S>
  __device__ void rhs(double an, const double* y, S* f, Br* br) {
    constexpr bool DER = sizeof(S) == sizeof(D1);
    const double fHe = B.fHe;
    const bool fresh = an != a;
    if (fresh) zt = 1.0 + (1.0 / an - 1.0);
    const S x_H = Mk<S>::of(y[0], dir == 0 ? 1.0 : 0.0), x_He = Mk<S>::of(y[1], dir == 1 ? 1.0 : 0.0);
    const S x = x_H + fHe * x_He;
    const double sT = take(br, BR_TSIGN, y[2] >= 0.0) ? 1.0 : -1.0, T = sT * y[2];
    const S Tmat = Mk<S>::of(T, dir == 2 ? sT : 0.0);
    // one division, one square root
    const double den = lane < 8 ? T : dc;
    const double q = (lane < 8 ? dc : dm * T) / den;
    double dq = 0.0;
    if (DER) dq = (lane < 8 ? -(q * sT) : dm * sT) / den;
    const double s = sqrt(q);
    double ds = 0.0;
    if (DER) ds = 0.5 * dq / s;
    if (lane >= 8 && lane < 12) {
      if (lane > 8) { sh[SV + lane - 9] = s; sh[SD + lane - 9] = ds; }
      if (lane < 11) {
        const double b = lane == 8 ? q : 1.0 + s, bd = lane == 8 ? dq : ds;
        sh[BV + i1] = b; sh[BV + i2] = b;
        sh[BD + i1] = bd; sh[BD + i2] = bd;
      }
    }
    if (lane == 0) { sh[BV] = K[DEB_TC_CR] * T; sh[BD] = K[DEB_TC_CR] * sT; sh[BV + 9] = zt; sh[BV + 10] = an; }
    __syncwarp();
    auto tdual = [&](int v, int d) { return Mk<S>::of(sh[v], dir == 2 ? sh[d] : 0.0); };
    const S omxHe = 1.0 - x_He, omxH = 1.0 - x_H;
    const S g2 = (g2n * omxHe) / (g2d * tdual(SV + 2, SD + 2) * omxH);
    if (lane < 2) sh[BV + 7 + lane] = val(g2);
    __syncwarp();
    // one power
    sh[PV + lane] = pow(sh[BV + (lane & 15)], pe);
    __syncwarp();
    if (fresh) at_a(an, sh[PV + 9], sh[PV + 10]);
    if (DER && lane < 7) sh[PD + lane] = (pe * sh[PV + 16 + lane]) * sh[BD + lane];
    // one exponential
    const S nHe1 = n_He * omxHe;
    const S tau = (tc * nHe1) / tden;
    const bool clip = !take(br, BR_BOLTZ, bc(q, 2) < 680.0);
    const double arg = lane < 8 ? (lane == 2 ? (clip ? 680.0 : q) : -q) : -val(tau);
    const double e = exp(arg);
    if (lane < 16) sh[EV + lane] = e;
    if (DER && lane < 8) sh[ED + lane] = lane == 2 ? (clip ? 0.0 : e * dq) : e * -dq;
    __syncwarp();
    auto te = [&](int i) { return tdual(EV + i, ED + i); };
    auto tp = [&](int i) { return tdual(PV + i, PD + i); };
    const bool h = sp >= 2, tr = sp == 1;
    const double xHe_r = y[1], xH_r = y[0];
    const bool he_edge = take(br, BR_HE_EDGE, (xHe_r < 5e-9) || (xHe_r > 0.98));
    const bool partial = he_edge ? false : take(br, BR_H_PARTIAL, xH_r < 0.9999999);
    const bool saha = take(br, BR_H_SAHA, xH_r > 0.99);
    const bool peebles0 = saha ? false : take(br, BR_H_PEEBLES0, xH_r > 0.985);
    const bool he_zero = take(br, BR_HE_ZERO, xHe_r < 1e-8);
    const bool full = (he_zero || he_edge) ? false : take(br, BR_H_FULL, xH_r > 0.99999);
    // recombination and ionisation rates
    const S X1 = tp(ia), X2 = tp(ib);
    const S rden = sel(h, 1.0 + K[DEB_TC_C_PPB] * X1, tdual(SV, SD) * X1 * X2);
    const S Rd = sel(h, rdn * X2, S(rdn)) / rden;
    const S Rup = rf * Rd * tp(0) * te(ie);
    const S xs = sel(h, x_H, x_He), om = sel(h, omxH, omxHe);
    const S rate = x * xs * n * Rd - cU * Rup * om * te(il);
    // HeI: escape probabilities, then K_He (singlet) and C_He (triplet)
    S Q = S(K[DEB_TC_CK_HE] / Hz);
    if (!he_edge) {
      const double ev = sh[EV + 8 + (tr ? 1 : 0)];
      const S et = Mk<S>::of(ev, ev * -der(tau));
      S M = A2p * ((1.0 - et) / tau);
      if (partial || !full) {
        const int ip = tr ? 8 : 7;
        const double p = tr ? 0.9 : 0.86;
        const S gp = Mk<S>::of(sh[PV + ip], DER ? (p * sh[PV + 16 + ip]) * der(g2) : 0.0);
        M = sel(tr ? !full : partial, M + ahn / (S(1.0) + ahc * gp), M);
      }
      const S num = sel(tr, M * te(6), S(1.0));
      Q = num / sel(tr, Rup + num, 3.0 * M * nHe1);
    }
    const S G = sel(h, KK * n * omxH, Q * nHe1 * te(2));
    const S KL = G * lam;
    S mult = sel(tr, Q, 1.0 + KL), den3 = sel(tr, S(1.0), 1.0 / fu + KL / fu + G * Rup);
    if (peebles0 && h) { mult = S(1.0); den3 = S(1.0); }
    const S F = rate * mult / (Hzz * den3);
    const int g = lane & ~3;
    auto of_species = [&](int s_) {
      if constexpr (DER) return S(bc(F.v, g | s_), bc(F.d, g | s_));
      else return bc(F, g | s_);
    };
    const S F0 = of_species(0), F1 = of_species(1), F2 = of_species(2);
    const S f0 = saha ? S(0.0) : F2;
    const S f1 = he_zero ? S(0.0) : (he_edge ? F0 : F0 + F1);
    const double timeTh = (1.0 / (K[DEB_TC_CT] * Trad4)) * (1.0 + val(x) + fHe) / val(x);
    S f2;
    if (take(br, BR_TM_LOCK, timeTh < K[DEB_TC_H_FRAC] * timeH)) {
      f2 = Tmat / zt;
    } else {
      f2 = K[DEB_TC_CT] * Trad4 * x / (1.0 + x + fHe) * (Tmat - Trad) / Hzz + 2.0 * Tmat / zt;
    }
    f[0] = f0 * dzda;
    f[1] = f1 * dzda;
    f[2] = f2 * dzda;
    __syncwarp();   // the scratch is written again by the next evaluation
  }

  // inverse of the 3x3 matrix whose rows every lane holds, by Gauss-Jordan with
  // partial pivoting (inv3), a column of (A | 1) per lane; X: this lane's row
  __device__ __forceinline__ void inverse_row(const double A[3][3], double* X) const {
    const int c6 = lane % 6;
    double m[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) m[i] = c6 == 0 ? A[i][0] : (c6 == 1 ? A[i][1] : (c6 == 2 ? A[i][2] : (c6 == i + 3 ? 1.0 : 0.0)));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double p[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) p[i] = bc(m[i], c);
      int pr = c;
      double best = fabs(p[c]);
#pragma unroll
      for (int r = c + 1; r < 3; ++r) if (fabs(p[r]) > best) { pr = r; best = fabs(p[r]); }
#pragma unroll
      for (int r = c + 1; r < 3; ++r)
        if (pr == r) { double t = m[c]; m[c] = m[r]; m[r] = t; t = p[c]; p[c] = p[r]; p[r] = t; }
      m[c] *= 1.0 / p[c];
#pragma unroll
      for (int r = 0; r < 3; ++r) if (r != c) m[r] -= p[r] * m[c];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double v[3] = {bc(m[0], 3 + j), bc(m[1], 3 + j), bc(m[2], 3 + j)};
      X[j] = row(v);
    }
  }

  static __device__ __forceinline__ double dot3(const double* r, const double* v) { return r[0] * v[0] + r[1] * v[1] + r[2] * v[2]; }

  // grk4a_step, a row of the 3-vectors per lane; y1 and err in every lane
  __device__ __forceinline__ void step(double t0, double dt, const double* y0, double* y1, double& err, Br* br3) {
    D1 fd[3];
    rhs<D1>(t0, y0, fd, br3);
    double Jr[3], Ar[3];
    {
      double A[3][3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double v[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          v[i] = bc(fd[i].d, 4 * j) * dt;
          A[i][j] = (i == j ? 1.0 : 0.0) - K[DEB_TC_G] * v[i];
        }
        Jr[j] = row(v);
      }
      inverse_row(A, Ar);
    }
    const double f0[3] = {fd[0].v * dt, fd[1].v * dt, fd[2].v * dt};
    const double yr = row(y0);
    double k1[3], k2[3], k3[3], u[3], o[3], t[3];
    const double k1r = dot3(Ar, f0);
    spread(k1r, k1);
    const double J1 = dot3(Jr, k1);
    spread(yr + K[DEB_TC_A21] * k1r, u);
    rhs<double>(t0, u, o, br3 ? br3 + 1 : nullptr);
    spread(row(o) * dt + K[DEB_TC_G21] * J1, t);
    const double k2r = dot3(Ar, t);
    spread(k2r, k2);
    const double J2 = dot3(Jr, k2);
    spread(yr + K[DEB_TC_A31] * k1r + K[DEB_TC_A32] * k2r, u);
    rhs<double>(t0, u, o, br3 ? br3 + 2 : nullptr);
    const double f2 = row(o) * dt;
    spread(f2 + K[DEB_TC_G31] * J1 + K[DEB_TC_G32] * J2, t);
    const double k3r = dot3(Ar, t);
    spread(k3r, k3);
    const double J3 = dot3(Jr, k3);
    spread(f2 + K[DEB_TC_G41] * J1 + K[DEB_TC_G42] * J2 + K[DEB_TC_G43] * J3, t);
    const double k4r = dot3(Ar, t);
    spread(yr + K[DEB_TC_C1] * k1r + K[DEB_TC_C2] * k2r + K[DEB_TC_C3] * k3r + K[DEB_TC_C4] * k4r, y1);
    err = (K[DEB_TC_C1] - K[DEB_TC_CH1]) * k1r + (K[DEB_TC_C2] - K[DEB_TC_CH2]) * k2r +
          (K[DEB_TC_C3] - K[DEB_TC_CH3]) * k3r + K[DEB_TC_C4] * k4r;
  }

  // solve_ionization
  __device__ bool solve(double astart, double aend, const double* ystart, double rtol, double atol, int max_steps,
                        double* out, StepLog slog = StepLog(), const double* rep = nullptr, int nrep = 0,
                        double rep_fin = 0.0) {
    double t0 = astart;
    double t1 = fmin(astart + fabs(astart) * 1e-3, aend);
    double y[3] = {ystart[0], ystart[1], ystart[2]};
    Br fin;
    bool ok = true;
    for (int j = 0, steps = 0; rep ? j < nrep : (t0 < aend && steps < max_steps); ++j, ++steps) {
      if (rep) t1 = rep[2 * j];
      const double dt = t1 - t0;
      double y1[3], er;
      Br b3[3];
      if (rep) unpack3(rep[2 * j + 1], b3);
      else for (int i = 0; i < 3; ++i) b3[i].mode = 1;
      step(t0, dt, y, y1, er, b3);
      const bool nan1 = isnan(y1[0]) || isnan(y1[1]) || isnan(y1[2]);
      if (rep) {
        ok = ok && !nan1;
        y[0] = y1[0]; y[1] = y1[1]; y[2] = y1[2];
        t0 = t1;
        continue;
      }
      const double yr = row(y), yc = nan1 ? yr : row(y1);
      const double sc = er / (atol + rtol * fmax(fabs(yr), fabs(yc)));
      double s3[3];
      spread(sc, s3);
      double ss = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) ss += s3[i] * s3[i];
      const double en = sqrt(ss / 3.0);
      const bool keep = en < 1.0;
      const double inv = en == 0.0 ? HUGE_VAL : 1.0 / en;
      double fac = 0.9 * pow(inv, 1.0 / 3.0);
      fac = fmin(fmax(fac, keep ? 1.0 : 0.2), 10.0);
      if (keep) {
        y[0] = y1[0]; y[1] = y1[1]; y[2] = y1[2];
        t0 = t1;
        if (slog.pos) {
          if (*slog.pos < slog.cap && lane == 0) { slog.steps[2 * *slog.pos] = t1; slog.steps[2 * *slog.pos + 1] = pack3(b3); }
          ++*slog.pos;
        }
      }
      t1 = t0 + dt * fac;
      if (t1 > aend - 1e-10) t1 = aend;
    }
    fin.mode = rep ? 2 : 1;
    fin.bits = rep ? (unsigned)rep_fin : 0u;
    double dy[3];
    rhs<double>(aend, y, dy, &fin);
    if (slog.fin && lane == 0) *slog.fin = (double)fin.bits;
    out[0] = y[0]; out[1] = y[1]; out[2] = y[2]; out[3] = dy[0]; out[4] = dy[1]; out[5] = dy[2];
    return rep ? ok && t0 == aend : t0 >= aend;
  }
};

}  // namespace debt

#endif
