// deb_block.cuh -- one Rodas5 step of one k-mode by a thread block (device
// only; structured solver).  Same arithmetic as step_attempt of deb_core.cuh,
// operation by operation, so both take the same steps; what differs is which
// thread evaluates which expression.  (Output fields agree to 1e-15: their
// conversion is compiled separately in the two kernels.)
//
// What bounds a step.  GB300 issues one FP64 instruction per 64 cycles to a
// warp, however many of its lanes are active, and one per ~19 cycles to an SM
// with four or more warps (measured with dependent and independent FMA
// chains).  A mode run by one warp is therefore limited to under a third of
// its SM's FP64 rate, and a launch with few modes -- or the last, longest modes
// of a large one -- by that warp's ~3600 (nvar 72) to ~9600 (nvar 1098) FP64
// instructions per step in sequence.
//
// The split.  The last warp of the block is the producer: the scale factor's
// equation (row 0) depends on a alone, so all eight stage values of a, and
// every RHS coefficient that depends on (a, tau) only, are known before any
// other row is touched.  The producer runs that scalar chain for the whole
// step, ahead of the other warps, and finishes with the forward-mode
// background of the next step's starting point.  The other warps (the team)
// run the vector work: the first one the reductions and metric sums, the
// others the hierarchies; in a solve the first takes the neutrino chains, the
// second the photon tails and the photon-baryon core, the third the scalar
// blocks.  The producer hands its coefficients over through two named barriers
// (stages 1-3, stages 4-7).  In the first stage the factorisation runs beside
// the right-hand side.
//
// Measured (whole calls, against one warp per mode): nvar 80, 64 modes 252 ->
// 81 ms; nvar 323, 256 modes 423 -> 155 ms and 4096 modes 777 -> 583 ms; nvar
// 265, 512 modes 201 -> 95 ms; nvar 72, 512 modes 54 -> 31 ms.
#pragma once

#include "deb_core.cuh"

namespace deb {

#ifdef __CUDACC__

constexpr int BAR_TEAM = 1, BAR_CO1 = 2, BAR_CO2 = 3;
constexpr int kCoSplit = 3;   // stages 1 .. kCoSplit are handed over first

__device__ __forceinline__ void bar_sync(int id, int n) { __syncwarp(); asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { __syncwarp(); asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// coefficients of one stage's RHS that depend on (a, tau) only
enum { CO_A = 0, CO_LA, CO_RHONU, CO_RHOQ, CO_IA, CO_IA2, CO_IAH, CO_AH, CO_RQ, CO_WRQ, CO_CA2, CO_OP, CO_ITAU, CO_SG,
       NCO = CO_SG + NSIG };

// Shared state of a block beside the mode's slot.
struct BlkS {
  ModeConst m;
  Cosmo c;
  Run r, rn;
  Bg<Dual> bg[2];        // forward-mode background at the start of this step and of the next
  double co[8][NCO];
  double dv[NDV];        // h', eta', alpha, P1, 1 of the current stage
  double dpnu;           // its momentum sum of the neutrino pressure
  double cc[8][8];       // C_sq / dt
  double fun[6];         // functionals of Z_h, Z_e and of stage 0's solution
  double th, te;
  double ss;
  double f0[6];          // entries -lo, up of the massless neutrinos' rows l = 0 .. 2
  double dtt[3];         // d f / d tau of the truncation rows of photon T, P and massless nu
  Tab T;
  double kap[NLEAD][NLT], lk[NLEAD * NLT];   // lk: times the current stage's scalars
  short src[NLEAD][NLT], sig[NLEAD][NLT], tgt[NLEAD];
  int cur;               // which of bg[] is this step's
  int q, item, go, keep, more, nout_hit;
  int bad;
};

template <int NW>
struct Blk {
  static constexpr int NT = 32 * NW, TT = NT - 32, HT = TT - 32;   // block, team, team without its first warp

  BlkS& S;
  WS<32> w;
  double* vqs;      // per stage s = 1 .. 7 and momentum bin: k v, v, v s^2 at [((s - 1) 3 + i) nq + q]
  Dims D;
  const Rodas& R;
  int tid, wi, lane;
  int ih, ie, ir1;   // this lane's elements of the h', eta' and row-1 lists (fewer than 33 entries)

  __device__ __forceinline__ bool producer() const { return wi == NW - 1; }
  __device__ __forceinline__ void team_sync() const { bar_sync(BAR_TEAM, TT); }
  __device__ __forceinline__ double& V(int vec, int j) const { return w.p[vec * D.n + j]; }
  __device__ __forceinline__ double& K(int s, int j) const { return w.kp[s * D.n + j]; }
  __device__ __forceinline__ double* vq(int s, int which) const { return vqs + ((s - 1) * 3 + which) * D.nq; }

  // once per launch: hierarchy coefficients and the lead rows' table in shared memory
  __device__ void init_tables(const Tab& T) {
    const bool in = lane < D.nq + 6;
    ih = in ? gather_index(D, GL_H, lane) : 0;
    ie = in ? gather_index(D, GL_E, lane) : 0;
    ir1 = in ? gather_index(D, GL_R1, lane) : 0;
    for (int l = tid; l < LMAX_TABLE + 2; l += NT) { S.T.lo[l] = T.lo[l]; S.T.up[l] = T.up[l]; }
    for (int e = tid; e < NLEAD * NLT; e += NT) {
      const int r = e / NLT, t = e - r * NLT;
      const LeadTerm& lt = lead_term(r, t);
      S.kap[r][t] = lt.kap;
      S.src[r][t] = (short)lead_index(D, lt.base, lt.off);
      S.sig[r][t] = (short)lt.sig;
      if (t == 0) S.tgt[r] = (short)lead_index(D, lead_tgt(r, 0), lead_tgt(r, 1));
    }
  }

  // ------------------------------------------------------------------ producer
  // ln of the dark-energy density a^(-3(1+w0+wa)) exp(3(a-1) wa), rounded as background_grp rounds it
  static __device__ __forceinline__ double de_exponent(const ModeConst& m, double a, double la) {
    return __fma_rn(3.0 * (a - 1.0), m.wa, __dmul_rn(m.pQ, la));
  }
  // a'/a and its inverse of a stage point, rounded as background_grp rounds them
  static __device__ __forceinline__ void hubble(const ModeConst& m, Bg<double>& g, double rhonu, double rhoQ) {
    const double X = __fma_rn(m.grM, rhonu, m.grr);
    const double s = __fma_rn(m.gOm, g.ia, __dmul_rn(X, g.ia2));
    const double rQ = __dmul_rn(__dmul_rn(m.gODE, rhoQ), g.a2);
    const double g3 = __dmul_rn(__dadd_rn(__dadd_rn(s, rQ), m.gOk), 1.0 / 3.0);
    g.iaH = rsqrt_(g3);
    g.aH = __dmul_rn(g3, g.iaH);
  }

  // a b whose derivative rounds a' b before the sum, or (mul1) a b'
  static __device__ __forceinline__ Dual mul2(Dual a, Dual b) { return Dual(a.v * b.v, __fma_rn(a.v, b.d, __dmul_rn(a.d, b.v))); }
  static __device__ __forceinline__ Dual mul1(Dual a, Dual b) { return Dual(a.v * b.v, __fma_rn(a.d, b.v, __dmul_rn(a.v, b.d))); }

  // spl_eval's value and derivative, every product rounded as there
  static __device__ __forceinline__ Dual spline_dual(const Spl& s, Dual x) {
    const int i = spl_locate(s, x.v);
    const double* cf = s.c + 4 * i;
    const double c1 = LDG(cf + 1), c2 = LDG(cf + 2), c3 = LDG(cf + 3);
    const double u = x.v - LDG(s.x + i);
    const double q2 = __fma_rn(u, c3, c2), q1 = __fma_rn(u, q2, c1);
    const double q1d = __fma_rn(u, __dmul_rn(x.d, c3), __dmul_rn(x.d, q2));
    return Dual(__fma_rn(u, q1, LDG(cf)), __fma_rn(x.d, q1, __dmul_rn(u, q1d)));
  }

  __device__ void bg_dual(double a, Bg<Dual>& out) {
    const Grp<32> gp{lane};
    const ModeConst& m = S.m;
    Bg<Dual> g;
    const Dual ad = make_var<Dual>(a);
    background_start(ad, g);
    const int which = lane == 1 ? SP_XE_LOGA : (lane == 2 ? SP_LRHONU_LOGA : SP_CS2A_LOGA);
    const Dual sv = spline_dual(S.c.sp[which], g.la);
    const Dual cs2a = gp.bcast(sv, 0), xe = gp.bcast(sv, 1), lrhonu = gp.bcast(sv, 2);
    const Dual ed(de_exponent(m, a, g.la.v), __fma_rn(3.0, m.wa, __dmul_rn(m.pQ, g.la.d)));
    const Dual ev = dexp(lane == 0 ? lrhonu : ed);
    const Dual rhonu = gp.bcast(ev, 0), rhoQ = gp.bcast(ev, 1);
    background_finish(m, ad, g, cs2a, xe, rhonu, rhoQ);
    // the density sum and a'/a with every product that a sum absorbs named:
    // the roundings the step sequence of a mode depends on
    const Dual X(__fma_rn(m.grM, rhonu.v, m.grr), __dmul_rn(m.grM, rhonu.d));
    const Dual r2(__dmul_rn(m.gODE, rhoQ.v), __dmul_rn(m.gODE, rhoQ.d));
    const double gv = __dadd_rn(__dadd_rn(__fma_rn(m.gOm, g.ia.v, __dmul_rn(X.v, g.ia2.v)),
                                          __dmul_rn(r2.v, g.a2.v)), m.gOk);
    const double td = __fma_rn(X.v, g.ia2.d, __dmul_rn(X.d, g.ia2.v));
    const double qd = __fma_rn(r2.v, g.a2.d, __dmul_rn(r2.d, g.a2.v));
    const double gd = __dadd_rn(__fma_rn(m.gOm, g.ia.d, td), qd);
    const Dual g3(__dmul_rn(gv, 1.0 / 3.0), __dmul_rn(gd, 1.0 / 3.0));
    g.iaH = drsqrt(g3);
    g.aH = Dual(__dmul_rn(g3.v, g.iaH.v), __fma_rn(g3.d, g.iaH.v, __dmul_rn(g3.v, g.iaH.d)));
    g.cs2.d = mul2(cs2a, g.ia).d;
    g.opac.d = mul2(xe * m.akthom, g.ia2).d;
    const Dual wQp(__dmul_rn(__dmul_rn(-m.wa, g.aH.v), a),
                   __fma_rn(__dmul_rn(-m.wa, g.aH.d), a, __dmul_rn(-m.wa, g.aH.v)));
    const Dual t2 = mul1(wQp * (1.0 / 3.0), drcp((1.0 + g.wQ) + 1e-6));
    g.ca2 = Dual(__fma_rn(-t2.v, g.iaH.v, g.wQ.v), g.wQ.d - mul2(t2, g.iaH).d);
    if (lane == 0) out = g;
    __syncwarp();
  }

  // element 0 (the scale factor) of stage SG before its RHS, as stage_prep forms it
  template <int SG>
  __device__ __forceinline__ void prep0(int vy, double idt, double ulast, double& u, double& p) const {
    double a[SG], cc[SG], kq[SG];
#pragma unroll
    for (int q = 0; q < SG; ++q) { a[q] = R.a[SG][q]; cc[q] = R.C[SG][q] * idt; }
#pragma unroll
    for (int q = 0; q < SG; ++q) kq[q] = K(q, 0);
    p = cc[0] * kq[0];
#pragma unroll
    for (int q = 1; q < SG; ++q) p += cc[q] * kq[q];
    if constexpr (SG <= 5) {
      u = V(vy, 0);
#pragma unroll
      for (int q = 0; q < SG; ++q) u += a[q] * kq[q];
    } else {
      u = ulast + kq[SG - 1];
    }
  }

  // stages s0 .. s1: one lane each for the coefficients, then the momentum bins
  __device__ void coefficients(int s0, int s1, double t0, double dt) {
    const ModeConst& m = S.m;
    const int s = s0 + lane;
    if (s <= s1) {
      double* co = S.co[s];
      Bg<double> g;
      g.a = co[CO_A];
      g.ia = rcp(g.a);
      g.ia2 = g.ia * g.ia;
      g.a2 = g.a * g.a;
      g.la = co[CO_LA];
      const double cs2a = spl_eval(S.c.sp[SP_CS2A_LOGA], g.la), xe = spl_eval(S.c.sp[SP_XE_LOGA], g.la);
      g.rhonu = co[CO_RHONU];
      g.rhoQ = co[CO_RHOQ];
      hubble(m, g, g.rhonu, g.rhoQ);
      g.cs2 = cs2a * g.ia;
      g.wQ = m.w0 + m.wa * (1.0 - g.a);
      const double wQp = -m.wa * g.aH * g.a;
      g.ca2 = __dadd_rn(g.wQ, -__dmul_rn(wQp * (1.0 / 3.0) * rcp((1.0 + g.wQ) + 1e-6), g.iaH));
      g.opac = xe * m.akthom * g.ia2;
      g.pb43 = m.pb43c * g.ia;
      const double itau = rcp(t0 + R.c[s] * dt);
      const double rQ = m.gODE * g.rhoQ * g.a2;
      const double w1 = 1.0 + g.wQ;
      const double k = m.k, k2 = m.k2;
      co[CO_IA] = g.ia; co[CO_IA2] = g.ia2; co[CO_IAH] = g.iaH; co[CO_AH] = g.aH; co[CO_RQ] = rQ; co[CO_WRQ] = w1 * rQ;
      co[CO_CA2] = g.ca2; co[CO_OP] = g.opac; co[CO_ITAU] = itau;
      const double sg[NSIG] = {1.0, k, k2, g.opac, g.aH, g.a, g.aH * g.a, k2 * g.cs2, g.pb43 * g.opac,
                               -(D.lg + 1.0) * itau, -(D.lgp + 1.0) * itau, -(D.lr + 1.0) * itau, w1,
                               3.0 * (m.cs2Q - g.wQ) * g.aH, 9.0 * w1 * (m.cs2Q - g.ca2) * g.aH * g.aH * m.ik2,
                               (1.0 - 3.0 * m.cs2Q) * g.aH, m.cs2Q * drcp(w1) * k2};
#pragma unroll
      for (int i = 0; i < NSIG; ++i) co[CO_SG + i] = sg[i];
    }
    const int nq = D.nq;
    for (int e = lane; e < (s1 - s0 + 1) * nq; e += 32) {
      const int se = s0 + e / nq, i = e - (se - s0) * nq;
      const double aq = S.co[se][CO_A] * w.m(M_Q + Q_AMQ * nq + i);
      const double s2 = 1.0 + aq * aq;
      const double v = drsqrt(s2);
      vq(se, 0)[i] = m.k * v;
      vq(se, 1)[i] = v;
      vq(se, 2)[i] = s2 * v;
    }
    __syncwarp();
  }

  // all of it for one step; with_next: also the forward-mode background at y1
  __device__ void produce(double t0, double dt, int vy, int vu, bool with_next) {
    const ModeConst& m = S.m;
    const Bg<Dual>& g0 = S.bg[S.cur];
    const double d = rcp(dt * R.gamma), idt = rcp(dt);
    // row 0: f = aH a, d f / d a
    const Dual f0 = g0.aH * Dual(g0.a.v, 1.0);
    const double w00i = 1.0 / (d - f0.d);
    if (lane == 0) K(0, 0) = f0.v * w00i;
    __syncwarp();
    double u = 0.0;
    for (int s = 1; s <= 7; ++s) {
      double p;
      switch (s) {
        case 1: prep0<1>(vy, idt, u, u, p); break;
        case 2: prep0<2>(vy, idt, u, u, p); break;
        case 3: prep0<3>(vy, idt, u, u, p); break;
        case 4: prep0<4>(vy, idt, u, u, p); break;
        case 5: prep0<5>(vy, idt, u, u, p); break;
        case 6: prep0<6>(vy, idt, u, u, p); break;
        default: prep0<7>(vy, idt, u, u, p); break;
      }
      Bg<double> g;
      background_start(u, g);
      const double lrhonu = spl_eval(S.c.sp[SP_LRHONU_LOGA], g.la);
      const double ev = dexp(lane == 0 ? lrhonu : de_exponent(m, u, g.la));
      const double rhonu = __shfl_sync(0xffffffffu, ev, 0), rhoQ = __shfl_sync(0xffffffffu, ev, 1);
      hubble(m, g, rhonu, rhoQ);
      if (lane == 0) {
        double* co = S.co[s];
        co[CO_A] = u; co[CO_LA] = g.la; co[CO_RHONU] = rhonu; co[CO_RHOQ] = rhoQ;
        const double f = __dadd_rn(p, __dmul_rn(g.aH, u));
        K(s, 0) = f * w00i;
      }
      __syncwarp();
      if (s == kCoSplit) { coefficients(1, kCoSplit, t0, dt); bar_arrive(BAR_CO1, NT); }
    }
    coefficients(kCoSplit + 1, 7, t0, dt);
    bar_arrive(BAR_CO2, NT);
    const double a1 = u + K(7, 0);
    if (with_next) bg_dual(a1, S.bg[S.cur ^ 1]);
    // y1 of row 0, after the team has read the previous contents (it reads u[0] nowhere)
    if (lane == 0) V(vu, 0) = a1;
  }

  // ------------------------------------------------------------------ team: stage 0, forward mode
  // f(t0, y0) into k1 (with the d f / d tau term and column 0 moved over, as
  // the solve wants it), d f / d a into JC0, and the factorisation of W; ends
  // with stage 0's, Z_h's and Z_e's M^-1 applied
  __device__ void stage0(double t0, double dt, int vy) {
    const ModeConst& m = S.m;
    const int n = D.n, nq = D.nq, iq0 = D.iq0, iq1 = iq0 + nq, iq2 = iq1 + nq, iq3 = iq2 + nq;
    const int igp = D.igp, ir = D.ir, lg = D.lg, lgp = D.lgp, lr = D.lr, lnu = D.lnu;
    const double k = m.k, k2 = m.k2;
    const Grp<32> gp{lane};
    auto Y = [&](int j) -> double { return V(vy, j); };
    const double d = rcp(dt * R.gamma);
    const double itau = rcp(t0);
    Bg<Dual> g = S.bg[S.cur];
    g.a.d = 1.0;
    const Dual f0 = g.aH * g.a;
    const double w00i = 1.0 / (d - f0.d);
    const double x0 = f0.v * w00i;
    const double it2 = rcp(t0 * t0), dd = dt * R.d[0];
    // f of row j, then dd dT where the row has a truncation term, then column 0
    auto put = [&](int j, Dual f) {
      V(V_JC0, j) = f.d;
      K(0, j) = __fma_rn(f.d, x0, f.v);
    };
    auto put_top = [&](int j, Dual f, double lmax) {
      const double dT = (lmax + 1.0) * it2 * Y(j);
      V(V_JC0, j) = f.d;
      K(0, j) = __fma_rn(f.d, x0, __fma_rn(dd, dT, f.v));
      return dT;
    };
    for (int j = tid; j < n; j += TT) { V(V_ZH, j) = 0.0; V(V_ZE, j) = 0.0; }
    if (wi == 2) {
      if (lane == 0) {
        S.f0[0] = 0.0; S.f0[1] = 0.25 * k2; S.f0[2] = 8.0 / 15.0;
        S.f0[3] = 4.0 / 3.0; S.f0[4] = 0.5 * k2; S.f0[5] = 0.6 * k;
      }
      const double idt = rcp(dt);
      for (int e = lane; e < 64; e += 32) S.cc[e >> 3][e & 7] = R.C[e >> 3][e & 7] * idt;
    }
    Dual drhonu = 0.0, dpnu = 0.0, fnu = 0.0;
    if (wi == 0) {
      for (int i = lane; i < nq; i += 32) {
        Dual aq = g.a * w.m(M_Q + Q_AMQ * nq + i);
        const Dual s2 = 1.0 + aq * aq;
        Dual v = drsqrt(s2);
        const double wq = LDG(S.c.w + i);
        const double wp0 = wq * Y(iq0 + i);
        drhonu = drhonu + wp0 * (s2 * v);
        dpnu = dpnu + wp0 * v;
        fnu = fnu + wq * Y(iq1 + i);
        w.m(M_Q + Q_V * nq + i) = v.v;
        w.m(M_Q + Q_DV * nq + i) = v.d;
      }
    } else {
      const int nt = lg - 3, np = lgp - 3, nr = lr - 3;
      for (int e = tid - 32; e < nt + np + nr; e += HT) {
        const bool ph = e < nt + np;
        const int l = 3 + (e < nt ? e : (ph ? e - nt : e - nt - np));
        const int j = (e < nt ? 7 : (ph ? igp : ir)) + l;
        const Dual damp = ph ? g.opac : Dual(0.0);
        put(j, k * (S.T.lo[l] * Y(j - 1) - S.T.up[l] * Y(j + 1)) - damp * Y(j));
      }
    }
    team_sync();
    auto kvq = [&](int i) -> Dual { return Dual(w.m(M_Q + Q_V * nq + i), w.m(M_Q + Q_DV * nq + i)); };
    if (wi == 0) {
      gp.sum3(drhonu.v, dpnu.v, fnu.v);
      gp.sum3(drhonu.d, dpnu.d, fnu.d);
      dpnu = dpnu * (1.0 / 3.0);
      const double eta = Y(2), dc = Y(3), tc = Y(4), db = Y(5), tb = Y(6), dg = Y(7), tg = Y(8);
      const double dr = Y(ir), tr = Y(ir + 1);
      const double dq = Y(n - 2), tq = Y(n - 1);
      const Dual rQ = mul2(m.gODE * g.rhoQ, g.a2);
      const Dual w1rQ = mul2(1.0 + g.wQ, rQ);
      const Dual rptQ(w1rQ.v * tq, __dmul_rn(w1rQ.d, tq));
      Dual dgrho = (m.gOc * dc + m.gOb * db) * g.ia + (m.grhog * dg + m.grN * dr + m.grM * drhonu) * g.ia2 + rQ * dq;
      Dual hp = (2.0 * k2 * eta + dgrho) * g.iaH;
      Dual dgtheta = (m.gOc * tc + m.gOb * tb) * g.ia + (m.g43g * tg + m.g43N * tr + m.grMk * fnu) * g.ia2 + rptQ;
      Dual etap = 0.5 * dgtheta * m.ik2;
      if (lane == 0) {
        const Dual dgpres = ((m.grhog * dg + m.grN * dr) * (1.0 / 3.0) + m.grM * dpnu) * g.ia2 +
                            (m.cs2Q * rQ * dq + (m.cs2Q - g.ca2) * (3.0 * g.aH * rptQ * m.ik2));
        const Dual w1 = 1.0 + g.wQ;
        const Dual sg[NSIG] = {Dual(1.0), Dual(k), Dual(k2), g.opac, g.aH, g.a, g.aH * g.a, k2 * g.cs2, mul1(g.pb43, g.opac),
                               Dual(-(lg + 1.0) * itau), Dual(-(lgp + 1.0) * itau), Dual(-(lr + 1.0) * itau), w1,
                               mul1(3.0 * (m.cs2Q - g.wQ), g.aH), mul2(mul2(mul1(9.0 * w1, m.cs2Q - g.ca2), g.aH), g.aH) * m.ik2,
                               (1.0 - 3.0 * m.cs2Q) * g.aH, m.cs2Q * drcp(w1) * k2};
        const Dual dv[NDV] = {hp, etap, (hp + 6.0 * etap) * 0.5 * m.ik2, dgrho + 3.0 * dgpres, Dual(1.0)};
        for (int i = 0; i < NSIG; ++i) {
          w.m(M_SCAL + S_LEAD + i) = sg[i].v;
          w.m(M_SCAL + S_LEADD + i) = sg[i].d;
        }
        for (int i = 0; i < NDV; ++i) {
          w.m(M_SCAL + S_LEAD + NSIG + i) = dv[i].v;
          w.m(M_SCAL + S_LEADD + NSIG + i) = dv[i].d;
        }
      }
      __syncwarp();
      auto scal = [&](int i) -> Dual { return Dual(w.m(M_SCAL + S_LEAD + i), w.m(M_SCAL + S_LEADD + i)); };
      // lead rows
      if (lane < NLEAD) {
        const int r = lane, tgt = S.tgt[r];
        Dual acc = 0.0;
#pragma unroll
        for (int t = 0; t < NLT; ++t) {
          const int src = S.src[r][t];
          const Dual x = src >= 0 ? Dual(Y(src)) : scal(NSIG - 1 - src);
          acc = acc + mul2(S.kap[r][t] * scal(S.sig[r][t]), x);
        }
        if (r == 10) S.dtt[0] = put_top(tgt, acc, lg);
        else if (r == 14) S.dtt[1] = put_top(tgt, acc, lgp);
        else if (r == 18) S.dtt[2] = put_top(tgt, acc, lr);
        else if (r > 0) put(tgt, acc);
        else V(V_JC0, 0) = acc.d;
      }
      // massive-neutrino rows l = 0 .. 2 and lnu
      const Dual hps = scal(NSIG + DV_HP), etaps = scal(NSIG + DV_ETAP);
      const Dual hp6 = hps * (1.0 / 6.0);
      const Dual hp_eta = hps * (1.0 / 15.0) + 0.4 * etaps;
      for (int i = lane; i < nq; i += 32) {
        const Dual kv = k * kvq(i);
        const double dlf = w.m(M_Q + Q_DLF * nq + i);
        put(iq0 + i, -kv * Y(iq1 + i) + hp6 * dlf);
        put(iq2 + i, kv * (2.0 * Y(iq1 + i) - 3.0 * Y(iq3 + i)) * 0.2 - hp_eta * dlf);
        const int jt = iq0 + lnu * nq + i;
        put(iq1 + i, kv * (Y(iq0 + i) - 2.0 * Y(iq2 + i)) * (1.0 / 3.0));
        w.m(M_Q + Q_DT * nq + i) = put_top(jt, kv * Y(jt - nq) - (lnu + 1.0) * itau * Y(jt), lnu);
      }
    } else {
      Bg<double> gv;
      gv.a = g.a.v; gv.ia = g.ia.v; gv.ia2 = g.ia2.v; gv.a2 = g.a2.v; gv.la = g.la.v; gv.cs2 = g.cs2.v; gv.xe = g.xe.v;
      gv.rhonu = g.rhonu.v; gv.rhoQ = g.rhoQ.v; gv.aH = g.aH.v; gv.iaH = g.iaH.v; gv.wQ = g.wQ.v; gv.ca2 = g.ca2.v;
      gv.opac = g.opac.v; gv.pb43 = g.pb43.v;
      if (wi == 1) {
        // photon tails' factors, the core's inverse, the momentum bins of the functionals
        chain_entries_tails();
        if (lane < 2) factor_chain(nq + 1 + lane, d, itau, gv.opac);
        __syncwarp();
        if (lane == 0) {
          double core[64], de[4];
          core_entries(m, S.T, gv, d, core, de);
          core[36] -= w.m(M_SCAL + S_FT);
          core[63] -= w.m(M_SCAL + S_FP);
          for (int i = 0; i < 64; ++i) w.m(M_CORE + (i & 7) * 8 + (i >> 3)) = core[i];   // column-major
        }
        __syncwarp();
        core_invert_warp();
        factor_bins(gv);
      } else {
        // neutrino chains' factors; scalar blocks of W, functional coefficients
        chain_entries_nu();
        for (int ch = lane; ch <= nq; ch += 32) factor_chain(ch, d, itau, gv.opac);
        factor_scalars(d, w00i, gv);
      }
      const int ngen = (lnu - 3) * nq;
      for (int e = tid - 32; e < ngen; e += HT) {
        const int l = 3 + e / nq, i = e - (l - 3) * nq;
        const int j = iq3 + e;
        put(j, k * kvq(i) * (S.T.lo[l] * Y(j - nq) - S.T.up[l] * Y(j + nq)));
      }
    }
    team_sync();
    // M^-1 of Z_h, Z_e and stage 0's vector together
    sweep_many();
    team_sync();
    if (wi < 3) {
      double sh, se;
      functionals_of(wi == 0 ? &V(V_ZH, 0) : (wi == 1 ? &K(0, 0) : &V(V_ZE, 0)), sh, se);
      if (lane == 0) { S.fun[2 * wi] = sh; S.fun[2 * wi + 1] = se; }
    }
    team_sync();
    if (wi == 0) {
      if (lane == 0) {
        const double hh = S.fun[0], eh = S.fun[1], he = S.fun[4], ee = S.fun[5];
        const double c00 = 1.0 - hh, c01 = -he, c10 = -eh, c11 = 1.0 - ee;
        const double idet = 1.0 / (c00 * c11 - c01 * c10);
        w.m(M_CINV + 0) = c11 * idet; w.m(M_CINV + 1) = -c01 * idet;
        w.m(M_CINV + 2) = -c10 * idet; w.m(M_CINV + 3) = c00 * idet;
      }
      __syncwarp();
      woodbury(S.fun[2], S.fun[3]);
    }
    team_sync();
  }

  __device__ __forceinline__ void woodbury(double sh, double se) {
    const double th = w.m(M_CINV + 0) * sh + w.m(M_CINV + 1) * se;
    const double te = w.m(M_CINV + 2) * sh + w.m(M_CINV + 3) * se;
    if (lane == 0) { S.th = th; S.te = te; }
  }

  // raw entries of the neutrino chains (by one warp) into V_LO, V_UP: what does
  // not depend on the elimination is taken off its serial loop
  __device__ __forceinline__ void chain_entries_nu() const {
    const int nq = D.nq, nm = (D.lnu + 1) * nq, tot = nm + D.lr + 1;
    const double k = S.m.k;
    for (int e = lane; e < tot; e += 32) {
      const bool mass = e < nm;
      const int l = mass ? e / nq : e - nm, lmax = mass ? D.lnu : D.lr;
      const bool fl = !mass && l <= 2;
      const double kf = mass ? k * w.m(M_Q + Q_V * nq + e - l * nq) : (fl ? 1.0 : k);
      const double el = l == lmax ? 1.0 : (fl ? S.f0[l] : S.T.lo[l]), eu = fl ? S.f0[3 + l] : S.T.up[l];
      const int j = mass ? D.iq0 + e : D.ir + l;
      V(V_LO, j) = -__dmul_rn(kf, el);
      V(V_UP, j) = __dmul_rn(kf, eu);
    }
    __syncwarp();
  }
  // the same of the photon tails
  __device__ __forceinline__ void chain_entries_tails() const {
    const int nt = D.lg - 2, tot = nt + D.lgp - 2;
    const double k = S.m.k;
    for (int e = lane; e < tot; e += 32) {
      const int l = 3 + (e < nt ? e : e - nt), j = (e < nt ? 7 : D.igp) + l;
      V(V_LO, j) = -__dmul_rn(k, l == (e < nt ? D.lg : D.lgp) ? 1.0 : S.T.lo[l]);
      V(V_UP, j) = __dmul_rn(k, S.T.up[l]);
    }
    __syncwarp();
  }

  // factors of chain ch from its raw entries (chain_factor of deb_core.cuh): a
  // reciprocal and two dependent FP64 operations per element
  __device__ __forceinline__ void factor_chain(int ch, double d, double itau, double op) const {
    const Chain c = chain_of<32>(S.m, D, w, ch);
    const double d_rest = c.attach >= 0 ? d + op : d;
    double *UP = &V(V_UP, 0), *LO = &V(V_LO, 0), *PI = &V(V_PI, 0);
    int i = c.start + (c.cnt - 1) * c.stride;
    double lo = LO[i];
    double pinv = rcp(__fma_rn(c.lmax + 1.0, itau, d_rest));
    PI[i] = pinv;
    LO[i] = __dmul_rn(lo, pinv);
    i -= c.cnt > 1 ? c.stride : 0;
    double up = UP[i], l2 = LO[i];
#pragma unroll 1
    for (int j = c.cnt - 2; j >= 0; --j) {
      const int nx = j > 0 ? i - c.stride : i;
      const double un = UP[nx], ln = LO[nx];
      const double qf = __dmul_rn(up, pinv);
      pinv = rcp(__fma_rn(-qf, lo, d_rest));
      lo = l2;
      UP[i] = qf;
      PI[i] = pinv;
      LO[i] = __dmul_rn(lo, pinv);
      i = nx; up = un; l2 = ln;
    }
    if (c.attach >= 0) {
      const double qa = 0.6 * S.m.k * pinv;
      UP[c.attach] = qa;
      w.m(M_SCAL + (ch == D.nq + 1 ? S_FT : S_FP)) = qa * lo;
    }
  }

  // the scalar blocks of W, the functionals' coefficients, row 1 and the
  // columns u_h, u_e but for the momentum bins (one lane)
  __device__ void factor_scalars(double d, double w00i, const Bg<double>& g) {
    const ModeConst& m = S.m;
    const int n = D.n, nq = D.nq, ir = D.ir;
    const double a = g.a, iaH = g.iaH, h2 = 0.5 * m.ik2;
    if (lane == 0) {
      w.m(M_SCAL + S_D) = d;
      w.m(M_SCAL + S_W00I) = w00i;
      const int oh = gl_off(nq, GL_H) + nq, oe = gl_off(nq, GL_E) + nq, o1 = gl_off(nq, GL_R1) + nq;
      const double rQ = m.gODE * g.rhoQ * g.a2;
      w.m(oh + 0) = 2.0 * m.k2 * iaH;
      w.m(oh + 1) = m.gOc * g.ia * iaH;
      w.m(oh + 2) = m.gOb * g.ia * iaH;
      w.m(oh + 3) = m.grhog * g.ia2 * iaH;
      w.m(oh + 4) = m.grN * g.ia2 * iaH;
      w.m(oh + 5) = rQ * iaH;
      w.m(oe + 0) = m.gOc * g.ia * h2;
      w.m(oe + 1) = m.gOb * g.ia * h2;
      w.m(oe + 2) = m.g43g * g.ia2 * h2;
      w.m(oe + 3) = m.g43N * g.ia2 * h2;
      w.m(oe + 4) = (1.0 + g.wQ) * rQ * h2;
      w.m(oe + 5) = 0.0;
      w.m(o1 + 0) = -m.gOc;
      w.m(o1 + 1) = -m.gOb;
      w.m(o1 + 2) = -2.0 * m.grhog * g.ia;
      w.m(o1 + 3) = -2.0 * m.grN * g.ia;
      w.m(o1 + 4) = -rQ * a * (1.0 + 3.0 * m.cs2Q);
      w.m(o1 + 5) = -9.0 * (m.cs2Q - g.ca2) * g.aH * (1.0 + g.wQ) * rQ * a * m.ik2;
      double core[64], de[4];
      core_entries(m, S.T, g, d, core, de);
      double a00 = de[0], a01 = de[1], a10 = de[2], a11 = de[3];
      double sw = 0.0;
      if (fabs(a10) > fabs(a00)) { double t0_ = a00, t1_ = a01; a00 = a10; a01 = a11; a10 = t0_; a11 = t1_; sw = 1.0; }
      const double i00 = rcp(a00), l = a10 * i00;
      w.m(M_DE + 0) = i00; w.m(M_DE + 1) = a01; w.m(M_DE + 2) = l; w.m(M_DE + 3) = rcp(a11 - l * a01);
      w.m(M_DE + 4) = sw;
      w.m(M_SCAL + S_ID) = rcp(d);
      w.m(M_SCAL + S_IDAH) = rcp(d + g.aH);
      V(V_ZH, 3) = -0.5; V(V_ZH, 5) = -0.5; V(V_ZH, 7) = -2.0 / 3.0; V(V_ZH, 9) = 4.0 / 15.0;
      V(V_ZH, ir) = -2.0 / 3.0; V(V_ZH, ir + 2) = 4.0 / 15.0; V(V_ZH, n - 2) = -0.5 * (1.0 + g.wQ);
      V(V_ZE, 2) = 1.0; V(V_ZE, 9) = 1.6; V(V_ZE, ir + 2) = 1.6;
    }
  }
  // the momentum bins' coefficients and their rows of u_h and u_e (one warp)
  __device__ void factor_bins(const Bg<double>& g) {
    const ModeConst& m = S.m;
    const int nq = D.nq, iq0 = D.iq0;
    const double iaH = g.iaH, h2 = 0.5 * m.ik2;
    for (int i = lane; i < nq; i += 32) {
      const double v = w.m(M_Q + Q_V * nq + i);
      const double iv = rcp(v);
      const double wq = LDG(S.c.w + i);
      w.m(gl_off(nq, GL_H) + i) = m.grM * wq * iv * g.ia2 * iaH;
      w.m(gl_off(nq, GL_E) + i) = m.grMk * wq * g.ia2 * h2;
      w.m(gl_off(nq, GL_R1) + i) = -m.grM * wq * (iv + v) * g.ia;
      const double dlf = w.m(M_Q + Q_DLF * nq + i);
      V(V_ZH, iq0 + i) = dlf / 6.0;
      V(V_ZH, iq0 + 2 * nq + i) = -dlf / 15.0;
      V(V_ZE, iq0 + 2 * nq + i) = -0.4 * dlf;
    }
  }

  // explicit inverse of the 8x8 core (core_invert of deb_core.cuh) with the
  // 8 x 16 elimination spread over the warp: lane = row + 8 (column group), its
  // four columns of (A | 1) in registers, so a step is one reciprocal, one
  // multiply and four multiply-adds; the pivot row and column go through the
  // slot.  Columns left of the pivot are eliminated too and read by nothing.
  __device__ void core_invert_warp() {
    const unsigned full = 0xffffffffu;
    const int i = lane & 7, cg = lane >> 3;
    double* A = &w.m(M_CORE);
    double* X = &w.m(M_CINV8);
    double* C = cg < 2 ? A + 32 * cg : X + 32 * (cg - 2);   // this group's columns
    double e[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (cg >= 2) C[8 * c + i] = 4 * (cg - 2) + c == i ? 1.0 : 0.0;
      e[c] = C[8 * c + i];
    }
    __syncwarp();
    unsigned done = 0u;
    int prow = 0;
    double pinv = 0.0;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      // largest key, lowest row among equals
      const int key = (lane < 8 && !((done >> lane) & 1u)) ? abs_key(A[kk * 8 + i]) : -1;
      const int top = __reduce_max_sync(full, key);
      const int p = __ffs(__ballot_sync(full, key == top)) - 1;
      done |= 1u << p;
      const double pv = A[kk * 8 + p], fv = A[kk * 8 + i];
      double r[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) r[c] = C[8 * c + p];
      __syncwarp();
      const double pi = rcp(pv), f = fv * pi;
      if (i != p) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          e[c] = __fma_rn(-f, r[c], e[c]);
          C[8 * c + i] = e[c];
        }
      }
      if (i == kk) { prow = p; pinv = pi; }
      __syncwarp();
    }
    double z[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) z[q] = X[8 * (cg + 4 * q) + prow] * pinv;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; ++q) X[8 * (cg + 4 * q) + i] = z[q];
    __syncwarp();
  }

  // Elimination x_i = r_i - up_i x_prev downwards over cnt elements from i, a
  // stride st apart; x is the element before them.  One dependent multiply-add
  // per element (two upwards) with the next element's loads under it: 64 cycles
  // each is the floor, 95 and 170 are measured.  Unrolling by four with padded
  // trip counts was slower (5.9 against 4.9 thousand cycles for 18 elements down
  // and up), a select on x inside the chain more so (107 against 64 per element).
  static __device__ __forceinline__ void sweep_down(double* r, const double* up, int i, int st, int cnt, double x) {
    double rv = r[i], uv = up[i];
#pragma unroll 1
    for (int j = 1; j <= cnt; ++j) {
      const int nx = j < cnt ? i - st : i;
      const double rn = r[nx], un = up[nx];
      x = __fma_rn(-uv, x, rv);
      r[i] = x;
      i = nx; rv = rn; uv = un;
    }
  }
  // Back-substitution z_i = r_i / p_i - lo_i z_prev upwards from element i (the
  // product lo_i z_prev is the rounded one)
  static __device__ __forceinline__ void sweep_up(double* r, const double* pi, const double* lo, int i, int st, int cnt,
                                                  double z) {
    double rv = r[i], pv = pi[i], lv = lo[i];
#pragma unroll 1
    for (int j = 1; j <= cnt; ++j) {
      const int nx = j < cnt ? i + st : i;
      const double rn = r[nx], pn = pi[nx], ln = lo[nx];
      z = __fma_rn(rv, pv, -__dmul_rn(lv, z));
      r[i] = z;
      i = nx; rv = rn; pv = pn; lv = ln;
    }
  }

  // neutrino chain ch of vector r
  __device__ __forceinline__ void chain_sweep(double* r, int ch) const {
    const int st = ch == 0 ? 1 : D.nq, cnt = ch == 0 ? D.lr + 1 : D.lnu + 1;
    const int first = ch == 0 ? D.ir : D.iq0 + ch - 1, top = first + (cnt - 1) * st;
    sweep_down(r, &V(V_UP, 0), top - st, st, cnt - 1, r[top]);
    const double z = r[first] * V(V_PI, first);
    r[first] = z;
    sweep_up(r, &V(V_PI, 0), &V(V_LO, 0), first + st, st, cnt - 1, z);
  }

  // photon tail t (0: T, 1: P) of vector r folded into its core row
  __device__ __forceinline__ void tail_fold(double* r, int t) const {
    const int start = t == 0 ? 10 : D.igp + 3, cnt = t == 0 ? D.lg - 2 : D.lgp - 2, top = start + cnt - 1;
    sweep_down(r, &V(V_UP, 0), top - 1, 1, cnt, r[top]);   // the last element is the core row
  }
  __device__ __forceinline__ void tail_back(double* r, int t) const {
    const int start = t == 0 ? 10 : D.igp + 3, cnt = t == 0 ? D.lg - 2 : D.lgp - 2;
    sweep_up(r, &V(V_PI, 0), &V(V_LO, 0), start, 1, cnt, r[start - 1]);
  }

  __device__ __forceinline__ int core_index(int j) const { return j < 5 ? 5 + j : D.igp + j - 5; }

  // eta, CDM and dark-energy blocks of vector r
  __device__ __forceinline__ void scalar_blocks(double* r) const {
    const int n = D.n;
    const double id = w.m(M_SCAL + S_ID);
    r[2] = r[2] * id;
    const double z4 = r[4] * w.m(M_SCAL + S_IDAH);
    r[4] = z4;
    r[3] = (r[3] - z4) * id;
    double r0 = r[n - 2], r1 = r[n - 1];
    if (w.m(M_DE + 4) != 0.0) { double t = r0; r0 = r1; r1 = t; }
    r1 -= w.m(M_DE + 2) * r0;
    const double z1 = r1 * w.m(M_DE + 3);
    const double z0 = (r0 - w.m(M_DE + 1) * z1) * w.m(M_DE + 0);
    r[n - 2] = z0; r[n - 1] = z1;
  }

  // photon tails and core of nv <= 4 vectors (one warp): 2 nv, 8 nv, 2 nv lanes
  template <class VecFn>
  __device__ __forceinline__ void photon_block(int nv, VecFn vec) const {
    if (lane < 2 * nv) tail_fold(vec(lane >> 1), lane & 1);
    __syncwarp();
    const int cv = lane >> 3, row = lane & 7;
    double z = 0.0;
    if (cv < nv) {
      const double* r = vec(cv);
#pragma unroll
      for (int j = 0; j < 8; ++j) z += w.m(M_CINV8 + j * 8 + row) * r[core_index(j)];
    }
    __syncwarp();
    if (cv < nv) vec(cv)[core_index(row)] = z;
    __syncwarp();
    if (lane < 2 * nv) tail_back(vec(lane >> 1), lane & 1);
  }

  // M^-1 of Z_h, Z_e and stage 0's vector
  __device__ void sweep_many() const {
    auto vec = [&](int v) -> double* { return v == 0 ? &V(V_ZH, 0) : (v == 1 ? &V(V_ZE, 0) : &K(0, 0)); };
    if (wi == 1) {
      photon_block(3, vec);
    } else {
      if (wi == 2 && lane < 3) scalar_blocks(vec(lane));
      const int nch = D.nq + 1;
      for (int e = wi == 0 ? lane : tid - 32; e < 3 * nch; e += TT - 32) {
        const int v = e / nch;
        chain_sweep(vec(v), e - v * nch);
      }
    }
  }

  // M^-1 of stage s's vector
  __device__ void sweep_one(int s) const {
    double* r = &K(s, 0);
    if (wi == 1) {
      photon_block(1, [&](int) { return r; });
    } else {
      if (wi == 2 && lane == 0) scalar_blocks(r);
      for (int ch = wi == 0 ? lane : tid - 32; ch <= D.nq; ch += TT - 32) chain_sweep(r, ch);
    }
  }

  // sums of the momentum bins (one per lane, nq <= 32) in the order of
  // Grp::sum3, without its additions of lanes that hold no bin
  __device__ __forceinline__ void bin_sums(double& a, double& b, double& c) const {
    const unsigned full = 0xffffffffu;
    if (D.nq <= 8) {
      const int g = lane >> 3, l = lane & 7;
      const double vb = __shfl_sync(full, b, l), vc = __shfl_sync(full, c, l);
      double v = g == 0 ? a : (g == 1 ? vb : vc);
      if (D.nq > 4) v += __shfl_xor_sync(full, v, 4);
      if (D.nq > 2) v += __shfl_xor_sync(full, v, 2);
      v += __shfl_xor_sync(full, v, 1);
      a = __shfl_sync(full, v, 0);
      b = __shfl_sync(full, v, 8);
      c = __shfl_sync(full, v, 16);
    } else if (D.nq <= 16) {
      const bool lo = lane < 16, q = (lane & 8) == 0;
      const double vb = __shfl_xor_sync(full, b, 16);
      const double k1 = lo ? a : vb, k2 = lo ? c : 0.0;
      double k = (q ? k1 : k2) + __shfl_xor_sync(full, q ? k2 : k1, 8);
      for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(full, k, o);
      a = __shfl_sync(full, k, 0);
      c = __shfl_sync(full, k, 8);
      b = __shfl_sync(full, k, 16);
    } else {
      const Grp<32> gp{lane};
      gp.sum3(a, b, c);
    }
  }

  // g_h . r and g_e . r
  __device__ __forceinline__ void functionals_of(const double* r, double& sh, double& se) const {
    const int nq = D.nq;
    const Grp<32> gp{lane};
    double h = 0.0, e = 0.0;
    if (nq + 6 <= 32) {
      if (lane < nq + 6) {
        h = w.m(gl_off(nq, GL_H) + lane) * r[ih];
        e = w.m(gl_off(nq, GL_E) + lane) * r[ie];
      }
      if (nq + 6 <= 16) {
        const unsigned full = 0xffffffffu;
        const double eo = __shfl_xor_sync(full, e, 16);
        double k = lane < 16 ? h : eo;
        for (int o = 8; o > 0; o >>= 1) k += __shfl_xor_sync(full, k, o);
        sh = __shfl_sync(full, k, 0);
        se = __shfl_sync(full, k, 16);
        return;
      }
    } else {
      for (int t = lane; t < nq + 6; t += 32) {
        h += w.m(gl_off(nq, GL_H) + t) * r[gather_index(D, GL_H, t)];
        e += w.m(gl_off(nq, GL_E) + t) * r[gather_index(D, GL_E, t)];
      }
    }
    gp.sum2(h, e);
    sh = h;
    se = e;
  }

  // ------------------------------------------------------------------ team: stages 1 .. 7
  // k_{SG-1} += Woodbury term, then stage SG's point and the sum over the
  // earlier stages for this thread's elements (rows 2 ..)
  template <int SG>
  __device__ __forceinline__ void update_prep(int vy, int vu, double idt) const {
    const int n = D.n;
    const double th = S.th, te = S.te;
    double a[SG], cc[SG];
#pragma unroll
    for (int q = 0; q < SG; ++q) { a[q] = R.a[SG][q]; cc[q] = S.cc[SG][q]; }
    for (int j = 2 + tid; j < n; j += TT) {
      double kq[SG];
#pragma unroll
      for (int q = 0; q < SG; ++q) kq[q] = K(q, j);
      kq[SG - 1] += V(V_ZH, j) * th + V(V_ZE, j) * te;
      K(SG - 1, j) = kq[SG - 1];
      double p = cc[0] * kq[0];
#pragma unroll
      for (int q = 1; q < SG; ++q) p += cc[q] * kq[q];
      double u;
      if constexpr (SG <= 5) {
        u = V(vy, j);
#pragma unroll
        for (int q = 0; q < SG; ++q) u += a[q] * kq[q];
      } else {
        u = V(vu, j) + kq[SG - 1];
      }
      V(vu, j) = u;
      K(SG, j) = p;
    }
  }

  // the RHS of row 1 at stage s, -(dgrho + 3 dgpres) a: read by nothing in this
  // stage, so a warp without chains forms it during the solve
  __device__ __forceinline__ void row1_rhs(int s, int vu) const {
    if (lane == 0) {
      const ModeConst& m = S.m;
      const double* co = S.co[s];
      const double dg = V(vu, 7), dr = V(vu, D.ir), dq = V(vu, D.n - 2), rptQ = co[CO_WRQ] * V(vu, D.n - 1);
      const double dgpres = ((m.grhog * dg + m.grN * dr) * (1.0 / 3.0) + m.grM * (S.dpnu * (1.0 / 3.0))) * co[CO_IA2] +
                            (m.cs2Q * co[CO_RQ] * dq + (m.cs2Q - co[CO_CA2]) * (3.0 * co[CO_AH] * rptQ * m.ik2));
      const double f = -co[CO_A] * (S.dv[DV_P1] + 3.0 * dgpres);
      K(s, 1) = __fma_rn(V(V_JC0, 1), K(s, 0), K(s, 1) + f);
    }
    __syncwarp();
  }

  // row 1 of stage s's solution (never read by the RHS), by one warp
  __device__ __forceinline__ void row1(int s) const {
    const int nq = D.nq, o1 = gl_off(nq, GL_R1);
    const Grp<32> gp{lane};
    double s1 = 0.0;
    if (nq + 6 <= 32) {
      if (lane < nq + 6) s1 = w.m(o1 + lane) * K(s, ir1);
    } else {
      for (int t = lane; t < nq + 6; t += 32) s1 += w.m(o1 + t) * K(s, gather_index(D, GL_R1, t));
    }
    s1 = gp.sum(s1);
    if (lane == 0) K(s, 1) = (K(s, 1) + s1) * w.m(M_SCAL + S_ID);
    __syncwarp();
  }

  // row 1 of stage SG's point and sum
  template <int SG>
  __device__ __forceinline__ void prep1(int vy, int vu, double idt) const {
    double a[SG], cc[SG], kq[SG];
#pragma unroll
    for (int q = 0; q < SG; ++q) { a[q] = R.a[SG][q]; cc[q] = R.C[SG][q] * idt; }
#pragma unroll
    for (int q = 0; q < SG; ++q) kq[q] = K(q, 1);
    double p = cc[0] * kq[0];
#pragma unroll
    for (int q = 1; q < SG; ++q) p += cc[q] * kq[q];
    double u;
    if constexpr (SG <= 5) {
      u = V(vy, 1);
#pragma unroll
      for (int q = 0; q < SG; ++q) u += a[q] * kq[q];
    } else {
      u = V(vu, 1) + kq[SG - 1];
    }
    if (lane == 0) { V(vu, 1) = u; K(SG, 1) = p; }
  }

  __device__ void stage(int s, double dt, double idt, int vy, int vu) {
    switch (s) {
      case 1: update_prep<1>(vy, vu, idt); break;
      case 2: update_prep<2>(vy, vu, idt); break;
      case 3: update_prep<3>(vy, vu, idt); break;
      case 4: update_prep<4>(vy, vu, idt); break;
      case 5: update_prep<5>(vy, vu, idt); break;
      case 6: update_prep<6>(vy, vu, idt); break;
      default: update_prep<7>(vy, vu, idt); break;
    }
    if (s == 1) bar_sync(BAR_CO1, NT);
    else if (s == kCoSplit + 1) bar_sync(BAR_CO2, NT);
    else team_sync();
    const ModeConst& m = S.m;
    const double* co = S.co[s];
    const int n = D.n, nq = D.nq, iq0 = D.iq0, iq1 = iq0 + nq, iq2 = iq1 + nq, iq3 = iq2 + nq;
    const int igp = D.igp, ir = D.ir, lg = D.lg, lgp = D.lgp, lr = D.lr, lnu = D.lnu;
    const double k = m.k, k2 = m.k2;
    const double x0 = K(s, 0);
    const Grp<32> gp{lane};
    auto Y = [&](int j) -> double { return V(vu, j); };
    auto fin = [&](int j, double t) { K(s, j) = __fma_rn(V(V_JC0, j), x0, t); };
    const double dd = dt * R.d[s];
    if (wi == 0) {
      double drhonu = 0.0, dpnu = 0.0, fnu = 0.0;
      for (int i = lane; i < nq; i += 32) {
        const double wq = LDG(S.c.w + i);
        const double wp0 = wq * Y(iq0 + i);
        drhonu = drhonu + wp0 * vq(s, 2)[i];
        dpnu = dpnu + wp0 * vq(s, 1)[i];
        fnu = fnu + wq * Y(iq1 + i);
      }
      // dgrho (even lanes) and dgtheta (odd lanes) have one form
      //   (Oc y1 + Ob y2) / a + (c3 y3 + c4 y4 + c5 S) / a^2 + c6 y6
      const bool odd = (lane & 1) != 0;
      const double y1 = Y(odd ? 4 : 3), y2 = Y(odd ? 6 : 5), y3 = Y(odd ? 8 : 7), y4 = Y(ir + (odd ? 1 : 0)),
                   y6 = Y(n - (odd ? 1 : 2)), eta = Y(2);
      const double c3 = odd ? m.g43g : m.grhog, c4 = odd ? m.g43N : m.grN, c5 = odd ? m.grMk : m.grM;
      const double c6 = odd ? co[CO_WRQ] : co[CO_RQ], ia = co[CO_IA], ia2 = co[CO_IA2];
      const double A = __fma_rn(m.gOc, y1, __dmul_rn(m.gOb, y2));
      const double G = __fma_rn(c3, y3, __dmul_rn(c4, y4));
      bin_sums(drhonu, dpnu, fnu);
      const double T = __fma_rn(A, ia, __dmul_rn(__fma_rn(c5, odd ? fnu : drhonu, G), ia2));
      const double d = odd ? __dadd_rn(T, __dmul_rn(c6, y6)) : __fma_rn(c6, y6, T);
      // h' = (2 k^2 eta + dgrho) / aH; eta' = dgtheta / (2 k^2)
      const double z = __dmul_rn(odd ? d : __fma_rn(2.0 * k2, eta, d), odd ? 0.5 * m.ik2 : co[CO_IAH]);
      const double etap = __shfl_sync(0xffffffffu, z, 1);
      if (lane == 0) {
        const double hp = z;
        S.dv[DV_HP] = hp;
        S.dv[DV_ETAP] = etap;
        S.dv[DV_ALPHA] = (hp + 6.0 * etap) * 0.5 * m.ik2;
        S.dv[DV_P1] = d;                           // dgrho (row1_rhs)
        S.dv[DV_ONE] = 1.0;
        S.dpnu = dpnu;
      }
    } else {
      if (wi == 2) {
        row1(s - 1);
        switch (s) {
          case 1: prep1<1>(vy, vu, idt); break;
          case 2: prep1<2>(vy, vu, idt); break;
          case 3: prep1<3>(vy, vu, idt); break;
          case 4: prep1<4>(vy, vu, idt); break;
          case 5: prep1<5>(vy, vu, idt); break;
          case 6: prep1<6>(vy, vu, idt); break;
          default: prep1<7>(vy, vu, idt); break;
        }
      }
      const double opac = co[CO_OP];
      const int nt = lg - 3, np = lgp - 3, nr = lr - 3;
      for (int e = tid - 32; e < nt + np + nr; e += HT) {
        const bool ph = e < nt + np;
        const int l = 3 + (e < nt ? e : (ph ? e - nt : e - nt - np));
        const int j = (e < nt ? 7 : (ph ? igp : ir)) + l;
        const double damp = ph ? opac : 0.0;
        double t = K(s, j);
        t += k * (S.T.lo[l] * Y(j - 1) - S.T.up[l] * Y(j + 1)) - damp * Y(j);
        fin(j, t);
      }
      const double* kv = vq(s, 0);
      const int ngen = (lnu - 3) * nq;
      for (int e = tid - 32; e < ngen; e += HT) {
        const int l = 3 + e / nq, i = e - (l - 3) * nq;
        const int j = iq3 + e;
        double t = K(s, j);
        t += kv[i] * (S.T.lo[l] * Y(j - nq) - S.T.up[l] * Y(j + nq));
        fin(j, t);
      }
      if (wi == 1) {
        const double itau = co[CO_ITAU];
        for (int i = lane; i < nq; i += 32) {
          const int jt = iq0 + lnu * nq + i;
          double t = K(s, iq1 + i);
          t += kv[i] * (Y(iq0 + i) - 2.0 * Y(iq2 + i)) * (1.0 / 3.0);
          fin(iq1 + i, t);
          t = K(s, jt);
          t += kv[i] * Y(jt - nq) - (lnu + 1.0) * itau * Y(jt);
          if (s <= 4) t = __fma_rn(dd, w.m(M_Q + Q_DT * nq + i), t);
          fin(jt, t);
        }
      }
    }
    // the lead rows' coefficients, before the metric is known
    if (wi == 2)
      for (int e = lane; e < NLEAD * NLT; e += 32) S.lk[e] = (&S.kap[0][0])[e] * co[CO_SG + (&S.sig[0][0])[e]];
    team_sync();
    if (wi == 2) {
      if (lane < NLEAD && lane > 1) {
        const int r = lane, tgt = S.tgt[r];
        double acc = 0.0;
#pragma unroll
        for (int t = 0; t < NLT; ++t) {
          const int src = S.src[r][t];
          acc = __fma_rn(S.lk[r * NLT + t], src >= 0 ? Y(src) : S.dv[-1 - src], acc);
        }
        double t = __dadd_rn(K(s, tgt), acc);
        if (s <= 4) {
          if (r == 10) t = __fma_rn(dd, S.dtt[0], t);
          else if (r == 14) t = __fma_rn(dd, S.dtt[1], t);
          else if (r == 18) t = __fma_rn(dd, S.dtt[2], t);
        }
        fin(tgt, t);
      }
    } else if (wi == 0) {
      const double* kv = vq(s, 0);
      const double hp6 = S.dv[DV_HP] * (1.0 / 6.0);
      for (int i = lane; i < nq; i += 32) {
        const double dlf = w.m(M_Q + Q_DLF * nq + i);
        double t = K(s, iq0 + i);
        t += -kv[i] * Y(iq1 + i) + hp6 * dlf;
        fin(iq0 + i, t);
      }
    } else if (wi == 1) {
      const double* kv = vq(s, 0);
      const double hp = S.dv[DV_HP], etap = S.dv[DV_ETAP];
      const double hp_eta = hp * (1.0 / 15.0) + 0.4 * etap;
      for (int i = lane; i < nq; i += 32) {
        const double dlf = w.m(M_Q + Q_DLF * nq + i);
        double t = K(s, iq2 + i);
        t += kv[i] * (2.0 * Y(iq1 + i) - 3.0 * Y(iq3 + i)) * 0.2 - hp_eta * dlf;
        fin(iq2 + i, t);
      }
    }
    team_sync();
    sweep_one(s);
    if (wi == 2) row1_rhs(s, vu);
    team_sync();
    if (wi == 0) {
      double sh, se;
      functionals_of(&K(s, 0), sh, se);
      woodbury(sh, se);
    }
    team_sync();
  }

  // The team's part of a step from (t0, y0 = vy): y1 into vu, stages and
  // factors in the slot; whether this thread saw a non-finite entry of y1.
  __device__ bool advance(double t0, double dt, int vy, int vu) {
    const double idt = rcp(dt);
    stage0(t0, dt, vy);
    for (int s = 1; s < 8; ++s) stage(s, dt, idt, vy, vu);
    // y1 = u + k8
    const int n = D.n;
    const double th = S.th, te = S.te;
    bool bad = false;
    for (int j = 2 + tid; j < n; j += TT) {
      double kk = K(7, j);
      kk += V(V_ZH, j) * th + V(V_ZE, j) * te;
      K(7, j) = kk;
      const double v = V(vu, j) + kk;
      V(vu, j) = v;
      bad = bad || !isfinite_(v);
    }
    team_sync();
    if (wi == 2) {
      row1(7);
      if (lane == 0) {
        const double v = V(vu, 1) + K(7, 1);
        V(vu, 1) = v;
        bad = bad || !isfinite_(v);
      }
    }
    return bad;
  }

  // One attempted step from (t0, y0 = vy) over dt: S.ss the sum of squares of
  // the scaled errors and S.bad whether y1 has a non-finite entry.  All
  // threads of the block call it after a block barrier; it ends with one.
  __device__ void step(double t0, double dt, int vy, int vu, double rtol, double atol) {
    if (tid == 0) S.bad = 0;
    if (producer()) {
      produce(t0, dt, vy, vu, true);
    } else if (advance(t0, dt, vy, vu)) {
      S.bad = 1;
    }
    __syncthreads();
    if (wi == 0) {
      const bool bad = S.bad != 0 || !isfinite_(V(vu, 0));
      // the six entries of the error norm on six lanes, their squares summed in order
      const int q = lane < 6 ? lane : 5;
      const int j = q == 0 ? 0 : (q < 3 ? q + 1 : q + 2);
      const double ew = q == 1 ? S.m.k2 : (q == 4 ? S.m.ik2 : 1.0);
      const double y0 = fabs(V(vy, j));
      const double y1 = bad ? y0 : fabs(V(vu, j));
      const double sc = K(7, j) * rcp(__fma_rn(y0 > y1 ? y0 : y1, rtol, atol)) * ew;
      double ss = 0.0;
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const double x = __shfl_sync(0xffffffffu, sc, e);
        ss = __fma_rn(x, x, ss);
      }
      if (lane == 0) { S.ss = ss; S.bad = bad; }
      __syncwarp();
    }
  }

  // ------------------------------------------------------------------ driver
  // The PID decision of step_decide (deb_core.cuh) by the first warp: the
  // next step into S.rn, and whether the step is kept, whether any output
  // time lies in it and whether the mode needs more steps.
  __device__ void decide(const Ctl& ctl, const double* tau_out) {
    Run r = S.r;
    const bool bad = S.bad != 0;
    const double err = ctl.replay ? 0.0 : sqrt(S.ss / 6.0);
    const double dt = r.t1 - r.t0;
    const double t0 = r.t0, t1 = r.t1;
    bool keep = false, go = false;
    int hit = 0;
    ++r.steps;
    if (!isfinite_(err) || (ctl.replay && bad)) {
      r.status = ST_NONFINITE;
    } else {
      keep = ctl.replay ? true : err < 1.0;
      const double linv = -log(err);
      double lf = 0.0;
      if (ctl.b1 != 0.0) lf += ctl.b1 * linv;
      if (ctl.b2 != 0.0) lf += ctl.b2 * r.lprev;
      if (ctl.b3 != 0.0) lf += ctl.b3 * r.lprev_prev;
      double factor = ctl.safety * exp(lf);
      const double fmin = keep ? 1.0 : ctl.fmin;
      factor = factor < fmin ? fmin : factor;
      factor = factor > ctl.fmax ? ctl.fmax : factor;
      const double linv_kept = isfinite_(linv) ? linv : 0.0;
      bool done = false;
      if (keep) {
        ++r.acc;
        for (int o = lane; o < ctl.nout; o += 32) {
          const double tt = LDG(tau_out + o);
          hit |= tt > t0 && tt <= t1;
        }
        hit = __any_sync(0xffffffffu, hit);
        const int vy = r.vy;
        r.vy = r.vu; r.vu = vy;
        r.t0 = r.t1;
        r.lprev_prev = r.lprev;
        r.lprev = linv_kept;
        if (ctl.record && lane == 0 && r.acc < r.rec_cap) r.rec[r.acc] = r.t1_out >= 0 ? -(r.t1_out + 1.0) : r.t1;
        if (ctl.replay) {
          if (r.t0 < r.T1) {
            double tn = r.acc + 1 < r.nrec ? replay_time(r, tau_out, r.acc + 1) : r.T1;
            if (r.acc + 1 >= r.nrec || tn >= r.T1) tn = r.T1;
            r.t1 = tn;
            go = true;
          }
          done = true;
        }
      } else {
        ++r.rej;
        if (ctl.hist_on_reject) { r.lprev_prev = r.lprev; r.lprev = linv_kept; }
      }
      if (!done) {
        double tn = __fma_rn(dt, factor, r.t0);
        r.t1_out = -1;
        if (ctl.step_ts) {
          int o;
          const double to = next_output(tau_out, ctl.nout, r.t0, o);
          if (tn >= to) { tn = to; r.t1_out = o; }
        }
        if (tn > r.T1 - 1e-10) tn = r.T1;
        if (!(tn > r.t0) && r.t0 < r.T1) {
          r.status = ST_DT_UNDERFLOW;
        } else {
          r.t1 = tn;
          go = r.t0 < r.T1;
        }
      }
    }
    if (lane == 0) { S.rn = r; S.keep = keep; S.go = go; S.nout_hit = hit; }
    __syncwarp();
  }

  // next_output_after of deb_core.cuh with the output times over the lanes
  __device__ double next_output(const double* tau_out, int nout, double t, int& which) {
    double best = 1e300;
    int bi = -1;
    for (int o = lane; o < nout; o += 32) {
      const double to = LDG(tau_out + o);
      if (to > t && to < best) { best = to; bi = o; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (oi >= 0 && (bi < 0 || ob < best || (ob == best && oi < bi))) { best = ob; bi = oi; }
    }
    which = bi;
    return best;
  }

  // One mode from its start to its last output; S.c, S.m and S.r (record
  // pointers) set, every thread of the block calls it after a barrier.
  __device__ void solve(const Ctl& ctl, const double* tau_out, double* yout) {
    const int n = D.n;
    const Grp<NT> gp{tid};
    WS<NT> wb;
    wb.p = w.p; wb.kp = w.kp; wb.n = n; wb.misc0 = w.misc0; wb.dp = nullptr;
    {
      Run r = S.r;
      __syncthreads();
      mode_begin<NT>(gp, S.c, S.m, D, ctl, wb, tau_out, r);
      __syncthreads();
      if (producer()) bg_dual(V(V_Y, 0), S.bg[0]);
      if (tid == 0) { S.r = r; S.cur = 0; }
    }
    __syncthreads();
    for (;;) {
      if (!(S.r.t0 < S.r.T1)) break;
      if (S.r.steps >= ctl.max_steps) {
        __syncthreads();
        if (tid == 0) S.r.status = ST_MAX_STEPS;
        break;
      }
      step(S.r.t0, S.r.t1 - S.r.t0, S.r.vy, S.r.vu, ctl.rtol, ctl.atol);
      if (wi == 0) decide(ctl, tau_out);
      __syncthreads();
      if (S.keep) {
        if (S.nout_hit) {
          const double t0 = S.r.t0, t1 = S.r.t1;
          const int vy = S.r.vy, vy1 = S.r.vu;
          for (int o = 0; o < ctl.nout; ++o) {
            const double tt = LDG(tau_out + o);
            if (tt > t0 && tt <= t1) {
              const double cf = (tt - t0) / (t1 - t0);
              double* dst = yout + (long)o * (ctl.return_full ? n : 20);
              if (ctl.return_full) {
                for (int j = tid; j < n; j += NT) { const double y0 = V(vy, j); dst[j] = y0 + cf * (V(vy1, j) - y0); }
              } else {
                for (int j = tid; j < n; j += NT) { const double y0 = V(vy, j); K(0, j) = y0 + cf * (V(vy1, j) - y0); }
                __syncthreads();
                if (tid == 0) outputs<32>(S.c, S.m, D, w, V_K0, dst, 1);
              }
              __syncthreads();
            }
          }
        }
        if (ctl.record && S.rn.ck) {
          Run r = S.rn;
          checkpoint_store<NT>(gp, wb, n, r, r.vy, r.acc);
          if (tid == 0) S.rn.ck_stride = r.ck_stride;
        }
        __syncthreads();
      }
      const bool go = S.go != 0;
      if (tid == 0) { S.r = S.rn; if (S.keep) S.cur ^= 1; }
      __syncthreads();
      if (!go) break;
    }
    __syncthreads();
  }
};

#endif  // __CUDACC__

}  // namespace deb
