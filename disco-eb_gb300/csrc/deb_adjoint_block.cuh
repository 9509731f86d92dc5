// deb_adjoint_block.cuh -- the discrete adjoint of one k-mode by a thread block
// (device only).  The mathematics is that of deb_adjoint.cuh; this file splits
// it over the warps of a block.
//
// What bounds a backward step.  On one warp it took ~45 k FP64 instructions in
// sequence (64 cycles each) at any hierarchy size: evaluating the RHS
// coefficients for every stage and every theta +- eps table set, a few lanes at
// a time, cost more than the vectors.  None of those coefficients depends on
// the adjoint variables, and r^T f = Phi(coefficients) . B is linear in the
// bilinear form B.  So the block's last warp (the producer of deb_block.cuh)
// evaluates, while the others re-attempt the forward step and run the stages
// backwards,
//   * the nominal coefficients of all eight stages at once, one lane per stage,
//     as second-order Taylor numbers in a;
//   * the weights Phi of B for every (stage, table set), one lane each, and
//     keeps their theta differences;
//   * the forward-mode background of the next (earlier) step's start.
// The other warps (the team) are left with the vectors: the transposed solve
// (neutrino chains, photon tails with the core, scalar blocks on one warp
// each), the two bilinear forms in one pass, and one fused pass over the stage
// vectors that also applies J^T's hierarchy couplings and forms the next
// stage's right-hand side.  The theta gradient is a dot product of the kept
// differences with the stages' forms, once per step.
#pragma once

#include "deb_adjoint.cuh"
#include "deb_block.cuh"
#include "deb_warp_sums.cuh"

namespace deb {

#ifdef __CUDACC__

// second-order Taylor number in one variable
struct Tay2 {
  double v, d, e;   // value, first and second derivative
  __device__ __forceinline__ Tay2() {}
  __device__ __forceinline__ Tay2(double x) : v(x), d(0.0), e(0.0) {}
  __device__ __forceinline__ Tay2(double x, double y, double z) : v(x), d(y), e(z) {}
};
__device__ __forceinline__ Tay2 operator+(const Tay2& a, const Tay2& b) { return Tay2(a.v + b.v, a.d + b.d, a.e + b.e); }
__device__ __forceinline__ Tay2 operator-(const Tay2& a, const Tay2& b) { return Tay2(a.v - b.v, a.d - b.d, a.e - b.e); }
__device__ __forceinline__ Tay2 operator*(const Tay2& a, const Tay2& b) {
  return Tay2(a.v * b.v, a.d * b.v + a.v * b.d, a.e * b.v + 2.0 * a.d * b.d + a.v * b.e);
}
__device__ __forceinline__ Tay2 operator+(const Tay2& a, double b) { return Tay2(a.v + b, a.d, a.e); }
__device__ __forceinline__ Tay2 operator+(double a, const Tay2& b) { return Tay2(a + b.v, b.d, b.e); }
__device__ __forceinline__ Tay2 operator-(const Tay2& a, double b) { return Tay2(a.v - b, a.d, a.e); }
__device__ __forceinline__ Tay2 operator-(double a, const Tay2& b) { return Tay2(a - b.v, -b.d, -b.e); }
__device__ __forceinline__ Tay2 operator*(const Tay2& a, double b) { return Tay2(a.v * b, a.d * b, a.e * b); }
__device__ __forceinline__ Tay2 operator*(double a, const Tay2& b) { return Tay2(a * b.v, a * b.d, a * b.e); }
// f(a) from f, f', f'' at a.v
__device__ __forceinline__ Tay2 tay_chain(const Tay2& a, double f, double f1, double f2) {
  return Tay2(f, f1 * a.d, f2 * a.d * a.d + f1 * a.e);
}
__device__ __forceinline__ Tay2 jexp(const Tay2& a) { const double e = exp(a.v); return tay_chain(a, e, e, e); }
__device__ __forceinline__ Tay2 jlog(const Tay2& a) { const double r = rcp(a.v); return tay_chain(a, log(a.v), r, -r * r); }
__device__ __forceinline__ Tay2 jrcp(const Tay2& a) { const double r = rcp(a.v); return tay_chain(a, r, -r * r, 2.0 * r * r * r); }
__device__ __forceinline__ Tay2 jrsqrt(const Tay2& a) {
  const double r = rsqrt_(a.v), r3 = r * r * r;
  return tay_chain(a, r, -0.5 * r3, 0.75 * r3 * r * r);
}
__device__ __forceinline__ double val(const Tay2& x) { return x.v; }

// weights of the bilinear form's entries: r^T f = sum_j Phi_j B_j; put(j, Phi_j)
template <class S, class F>
__device__ __forceinline__ void phi_weights(const Coef<S>& C, double k, F put) {
#pragma unroll
  for (int i = 0; i < NSIG; ++i) put(B_SIG + i, C.sg[i]);
  put(B_OP, C.opac);
  put(B_FREE, S(1.0));
  put(B_IT, C.itau);
  const S d2 = 0.5 * (C.dmu * C.dmu);
  put(B_V, S(k));
  put(B_V + 1, k * C.dmu);
  put(B_V + 2, k * d2);
  const S &w1 = C.sg[SG_W1], &a = C.sg[SG_A];
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    put(B_H1 + j, C.ch[j]);
    put(B_HW + j, w1 * C.ch[j]);
    put(B_P + j, a * C.cp[j]);
  }
  const S wx = w1 * C.xh, ax = a * C.xp;
  put(B_H1T, C.xh); put(B_H1T + 1, C.xh * C.dmu); put(B_H1T + 2, C.xh * d2);
  put(B_HWT, wx); put(B_HWT + 1, wx * C.dmu); put(B_HWT + 2, wx * d2);
  put(B_P1V, ax); put(B_P1V + 1, ax * C.dmu); put(B_P1V + 2, ax * d2);
  put(B_PV, ax); put(B_PV + 1, ax * C.dmu); put(B_PV + 2, ax * d2);
#pragma unroll
  for (int j = 0; j < 5; ++j) put(B_E + j, C.ce[j]);
  put(B_EF, C.xe);
}

constexpr int NCOEF = sizeof(Coef<double>) / sizeof(double);
constexpr int BAR_ADJ = 4;
constexpr int LEAD_MAXE = 72;      // nonzero lead-row terms
constexpr int MAXPAR = 12;

// one theta +- eps table set as a mode sees it
struct SetCtx { Cosmo c; ModeConst m; };

// The lead rows' table by scalar and by source element (LeadInv) with the
// indices of one hierarchy resolved: entries of list i at [at[i], at[i + 1]).
struct LeadLists {
  int sig_at[NSIG + 1], slot_at[LINV_NSLOT + 1];
  double sig_kap[LEAD_MAXE], slot_kap[LEAD_MAXE], der_kap[LINV_NDER];
  short sig_tgt[LEAD_MAXE], sig_src[LEAD_MAXE], slot_tgt[LEAD_MAXE], slot_sig[LEAD_MAXE], slot_dst[LINV_NSLOT];
  short der_tgt[LINV_NDER], der_kind[LINV_NDER];
  int nslot, nder;
};

// shared state of an adjoint block
struct AdjS {
  BlkS blk;
  LeadLists lead;
  double C[8][NCOEF];        // nominal coefficients of the stages
  double dphi[8][NB];        // d Phi / d a of the stages
  double C1[NCOEF];          // d / d a of the coefficients at y0
  double ddphi0[NB];         // d2 Phi / d a2 at y0
  double B[8][NB], BW[NB], BR[NB];   // r_s^T f(u_s); sum_s (r_s, k_s); (rho, y0)
  double part[2][4][8];      // a warp's partial sums of a form: op, free, v (3)
  double qs[2][8];           // bin sums of a form: t (3), s (3), fnu, it
  double xk[5], hn, en;      // weights of the derived values, momentum sums
  double s0[4], tmp[4][20];
  double th, te;
  double sts, tbn, tb_left, tb_right;   // time adjoints: tau_start, this step's ends
  double to[64];             // output times
  double ft[3 + 64];
  double out[MAXPAR];
  int hits;
  unsigned hitmask[2];
};

template <int NW>
struct AdjBlk {
  static constexpr int NT = 32 * NW, TT = NT - 32;
  static_assert(NW == 4, "roles are written for a team of three warps");

  AdjS& S;
  Blk<NW>& Bk;
  Dims D;
  const Rodas& R;
  int tid, wi, lane;
  double *lam, *rb, *rbn, *ub, *yh, *ye, *rho, *u, *yo2, *kb;   // n each, kb: 7 n; rb, rbn: r and the next r
  double* vv;       // [8 stages][6][nq]: v, dv, ddv, 1/v, d(1/v), dd(1/v) in mu
  double* dth;      // [NB][8][npar] theta differences of Phi
  double* dth1;     // [NB][npar] theta differences of d Phi / d a at y0
  SetCtx* sets;     // [2 npar]
  const AdjItem* it;
  double pc, pk, pf;    // shares of the step-length terms

  __device__ __forceinline__ double& V(int v, int j) const { return Bk.V(v, j); }
  __device__ __forceinline__ double& K(int s, int j) const { return Bk.K(s, j); }
  __device__ __forceinline__ double* KB(int s) const { return kb + (long)s * D.n; }
  __device__ __forceinline__ void team_sync() const { Bk.team_sync(); }

  __device__ void init_lists() {
    if (tid == 0) {
      const LeadInv& L = linv();
      LeadLists& Q = S.lead;
      int e = 0;
      for (int i = 0; i < NSIG; ++i) {
        Q.sig_at[i] = e;
        for (int q = 0; q < L.nsig[i]; ++q, ++e) {
          const int code = L.sig_ent[i][q], r = code / NLT, t = code - r * NLT;
          const LeadTerm& lt = lead_term(r, t);
          Q.sig_kap[e] = lt.kap;
          Q.sig_tgt[e] = (short)lead_index(D, lead_tgt(r, 0), lead_tgt(r, 1));
          Q.sig_src[e] = lt.base == IB_DV ? (short)-1 : (short)lead_index(D, lt.base, lt.off);
        }
      }
      Q.sig_at[NSIG] = e;
      e = 0;
      for (int s = 0; s < L.nslot; ++s) {
        Q.slot_at[s] = e;
        Q.slot_dst[s] = (short)lead_index(D, L.slot_base[s], L.slot_off[s]);
        for (int q = 0; q < L.slot_n[s]; ++q, ++e) {
          const int code = L.slot_ent[s][q], r = code / NLT, t = code - r * NLT;
          Q.slot_kap[e] = lead_term(r, t).kap;
          Q.slot_sig[e] = (short)lead_term(r, t).sig;
          Q.slot_tgt[e] = (short)lead_index(D, lead_tgt(r, 0), lead_tgt(r, 1));
        }
      }
      Q.slot_at[L.nslot] = e;
      Q.nslot = L.nslot;
      Q.nder = L.nder;
      for (int q = 0; q < L.nder; ++q) {
        const int code = L.der_ent[q], r = code / NLT, t = code - r * NLT;
        Q.der_kap[q] = lead_term(r, t).kap;
        Q.der_tgt[q] = (short)lead_index(D, lead_tgt(r, 0), lead_tgt(r, 1));
        Q.der_kind[q] = L.der_kind[q];
      }
    }
  }

  // ------------------------------------------------------------------ producer
  // coefficients of the stages at the nominal tables, Phi' and (at y0) Phi''
  __device__ void produce_nominal(double t0, double dt, double a0) {
    const ModeConst& m = S.blk.m;
    if (lane < 8) {
      const int s = lane;
      const double a = s == 0 ? a0 : S.blk.co[s][CO_A];
      const Coef<Tay2> C = coef<Tay2>(S.blk.c, m, D, Tay2(a, 1.0, 0.0), Tay2(t0 + R.c[s] * dt), a * m.amnu);
      const Tay2* p = reinterpret_cast<const Tay2*>(&C);
      for (int i = 0; i < NCOEF; ++i) S.C[s][i] = p[i].v;
      if (s == 0) for (int i = 0; i < NCOEF; ++i) S.C1[i] = p[i].d;
      phi_weights(C, m.k, [&](int j, const Tay2& w) {
        S.dphi[s][j] = w.d;
        if (s == 0) S.ddphi0[j] = w.e;
      });
    }
    __syncwarp();
    const int nq = D.nq;
    for (int e = lane; e < 8 * nq; e += 32) {
      const int s = e / nq, i = e - s * nq;
      const double a = s == 0 ? a0 : S.blk.co[s][CO_A];
      const double iq = rcp(LDG(S.blk.c.q + i)), xx = a * m.amnu * iq, v = rsqrt_(1.0 + xx * xx);
      const double v3 = v * v * v, iq2 = iq * iq;
      double* o = vv + (s * 6) * nq + i;
      o[0] = v;
      o[nq] = -xx * v3 * iq;
      o[2 * nq] = (-v3 + 3.0 * xx * xx * v3 * v * v) * iq2;
      o[3 * nq] = (1.0 + xx * xx) * v;
      o[4 * nq] = xx * v * iq;
      o[5 * nq] = v3 * iq2;
    }
    __syncwarp();
  }

  // theta differences of Phi at every stage and of Phi' at y0
  __device__ void produce_theta(double t0, double dt, double a0) {
    const int npar = it->npar, ns = 2 * npar;
    const double amnu = S.blk.m.amnu;
    for (int e0 = 0; e0 < 8 * ns; e0 += 32) {
      const int e = e0 + lane < 8 * ns ? e0 + lane : 8 * ns - 2 + (lane & 1);
      const int s = e / ns, b = e - s * ns;
      const double a = s == 0 ? a0 : S.blk.co[s][CO_A];
      const SetCtx& X = sets[b];
      const Coef<double> C = coef<double>(X.c, X.m, D, a, t0 + R.c[s] * dt, a * amnu);
      const double i2e = 0.5 / LDG(it->eps + (b >> 1));
      const bool keep = e0 + lane < 8 * ns && !(lane & 1);
      phi_weights(C, X.m.k, [&](int j, double w) {
        const double o = __shfl_xor_sync(0xffffffffu, w, 1);
        if (keep) dth[(j * 8 + s) * npar + (b >> 1)] = (w - o) * i2e;
      });
    }
    {
      const int b = lane < ns ? lane : ns - 2 + (lane & 1);
      const SetCtx& X = sets[b];
      typedef Jet<double> J1;
      const Coef<J1> C = coef<J1>(X.c, X.m, D, J1(a0, 1.0), J1(t0), a0 * amnu);
      const double i2e = 0.5 / LDG(it->eps + (b >> 1));
      phi_weights(C, X.m.k, [&](int j, const J1& w) {
        const double o = __shfl_xor_sync(0xffffffffu, w.d, 1);
        if (lane < ns && !(lane & 1)) dth1[j * npar + (b >> 1)] = (w.d - o) * i2e;
      });
    }
    __syncwarp();
  }

  // ------------------------------------------------------------------ transposed solve (solve_Mt by parts)
  __device__ __forceinline__ void chain_sweep_t(double* r, int ch) const {
    const int nq = D.nq;
    const double *UP = &V(V_UP, 0), *LO = &V(V_LO, 0), *PI = &V(V_PI, 0);
    const int start = ch == 0 ? D.ir : D.iq0 + ch - 1;
    const int stride = ch == 0 ? 1 : nq;
    const int cnt = ch == 0 ? D.lr + 1 : D.lnu + 1;
    int i = start + (cnt - 1) * stride;
    double rn = r[i];
    int j = cnt - 2;
    for (; j >= 7; j -= 8) {
      double rv[8], lv[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) { rv[q] = r[i - (q + 1) * stride]; lv[q] = LO[i - q * stride]; }
#pragma unroll
      for (int q = 0; q < 8; ++q) { rn = rv[q] - lv[q] * rn; r[i - (q + 1) * stride] = rn; }
      i -= 8 * stride;
    }
    for (; j >= 0; --j) {
      const int ip = i;
      i -= stride;
      rn = r[i] - LO[ip] * rn;
      r[i] = rn;
    }
    double z = rn * PI[start];
    r[start] = z;
    int jb = 1;
    for (; jb + 7 < cnt; jb += 8) {
      double sv[8], uv[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int ii = i + (q + 1) * stride;
        sv[q] = __dmul_rn(r[ii], PI[ii]);
        uv[q] = UP[ii - stride];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) { z = __fma_rn(-uv[q], z, sv[q]); r[i + (q + 1) * stride] = z; }
      i += 8 * stride;
    }
    for (; jb < cnt; ++jb) {
      i += stride;
      z = __fma_rn(-UP[i - stride], z, __dmul_rn(r[i], PI[i]));
      r[i] = z;
    }
  }
  __device__ __forceinline__ void tail_fold_t(double* r, int t) const {
    const double* LO = &V(V_LO, 0);
    const int start = t == 0 ? 10 : D.igp + 3, cnt = t == 0 ? D.lg - 2 : D.lgp - 2;
    int i = start + cnt - 1;
    double rn = r[i];
    for (int j = cnt - 2; j >= 0; --j) {
      const double l = LO[i];
      --i;
      rn = r[i] - l * rn;
      r[i] = rn;
    }
    r[start - 1] -= LO[start] * rn;
  }
  __device__ __forceinline__ void tail_back_t(double* r, int t) const {
    const double *UP = &V(V_UP, 0), *PI = &V(V_PI, 0);
    const int start = t == 0 ? 10 : D.igp + 3, cnt = t == 0 ? D.lg - 2 : D.lgp - 2;
    double z = r[start - 1];
    for (int j = 0; j < cnt; ++j) {
      const int i = start + j;
      const double sv = __dmul_rn(r[i], PI[i]);
      z = __fma_rn(-UP[i - 1], z, sv);
      r[i] = z;
    }
  }
  template <class VecFn>
  __device__ __forceinline__ void photon_block_t(int nv, VecFn vec) const {
    if (lane < 2 * nv) tail_fold_t(vec(lane >> 1), lane & 1);
    __syncwarp();
    const int cv = lane >> 3, row = lane & 7;
    double z = 0.0;
    if (cv < nv) {
      const double* r = vec(cv);
#pragma unroll
      for (int j = 0; j < 8; ++j) z += Bk.w.m(M_CINV8 + row * 8 + j) * r[Bk.core_index(j)];
    }
    __syncwarp();
    if (cv < nv) vec(cv)[Bk.core_index(row)] = z;
    __syncwarp();
    if (lane < 2 * nv) tail_back_t(vec(lane >> 1), lane & 1);
  }
  __device__ __forceinline__ void scalar_blocks_t(double* r) const {
    const int n = D.n;
    const WS<32>& w = Bk.w;
    const double id = w.m(M_SCAL + S_ID);
    r[2] = r[2] * id;
    const double z3 = r[3] * id;
    r[3] = z3;
    r[4] = (r[4] - z3) * w.m(M_SCAL + S_IDAH);
    const double i00 = w.m(M_DE + 0), a01 = w.m(M_DE + 1), l10 = w.m(M_DE + 2), i11 = w.m(M_DE + 3);
    const double v0 = r[n - 2] * i00;
    const double v1 = (r[n - 1] - a01 * v0) * i11;
    double w0 = v0 - l10 * v1, w1 = v1;
    if (w.m(M_DE + 4) != 0.0) { const double t = w0; w0 = w1; w1 = t; }
    r[n - 2] = w0;
    r[n - 1] = w1;
  }
  template <class VecFn>
  __device__ __forceinline__ void sweep_t(int nv, VecFn vec) const {
    if (wi == 1) {
      photon_block_t(nv, vec);
    } else {
      if (wi == 2 && lane < nv) scalar_blocks_t(vec(lane));
      const int nch = D.nq + 1;
      for (int e = wi == 0 ? lane : tid - 32; e < nv * nch; e += TT - 32) {
        const int v = e / nch;
        chain_sweep_t(vec(v), e - v * nch);
      }
    }
  }

  // Y_h = M^-T g_h, Y_e = M^-T g_e
  __device__ void prep_wt() {
    const int n = D.n, nq = D.nq;
    for (int j = tid; j < n; j += TT) { yh[j] = 0.0; ye[j] = 0.0; }
    team_sync();
    for (int t = tid; t < nq + 6; t += TT) {
      yh[gather_index(D, GL_H, t)] = Bk.w.m(gl_off(nq, GL_H) + t);
      if (t < nq + 5) ye[gather_index(D, GL_E, t)] = Bk.w.m(gl_off(nq, GL_E) + t);
    }
    team_sync();
    sweep_t(2, [&](int v) -> double* { return v == 0 ? yh : ye; });
    team_sync();
  }

  // rb <- W^-T rb (rows 1 ..; row 0 is finished by row0())
  __device__ void solve_wt(double wQ) {
    const int n = D.n, nq = D.nq;
    const WS<32>& w = Bk.w;
    const double z1 = rb[1] * w.m(M_SCAL + S_ID);
    if (wi == 0)
      for (int t = lane; t < nq + 6; t += 32) rb[gather_index(D, GL_R1, t)] += w.m(gl_off(nq, GL_R1) + t) * z1;
    team_sync();
    sweep_t(1, [&](int) -> double* { return rb; });
    team_sync();
    if (wi == 0) {
      const Grp<32> gp{lane};
      double sh = 0.0, se = 0.0;
      visit_u_lanes<32>(gp, D, w, wQ, [&](int i, double uh, double ue) { sh += uh * rb[i]; se += ue * rb[i]; });
      gp.sum2(sh, se);
      if (lane == 0) {
        S.th = w.m(M_CINV + 0) * sh + w.m(M_CINV + 2) * se;
        S.te = w.m(M_CINV + 1) * sh + w.m(M_CINV + 3) * se;
      }
    }
    team_sync();
    const double th = S.th, te = S.te;
    double s0 = tid == 0 ? V(V_JC0, 1) * z1 : 0.0;
    for (int j = 2 + tid; j < n; j += TT) {
      const double b = rb[j] + (yh[j] * th + ye[j] * te);
      rb[j] = b;
      s0 += V(V_JC0, j) * b;
    }
    for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    if (lane == 0) S.s0[wi] = s0;
    if (tid == 0) rb[1] = z1;
    team_sync();
  }
  // row 0 of the solution: every thread may ask for it until the next barrier
  __device__ __forceinline__ double row0() const {
    return (rb[0] + (S.s0[0] + S.s0[1] + S.s0[2])) * Bk.w.m(M_SCAL + S_W00I);
  }

  // ------------------------------------------------------------------ bilinear forms
  // Partial sums of (x, Y1) and, with TWO, of (x, Y2): a pass over the
  // hierarchies by the whole team, the momentum-bin sums by the first warp,
  // the derived values' weights by the second, the lead rows by scalar on the
  // third.  x0: x[0] (it may still be unfinished in memory).
  template <bool TWO>
  __device__ void forms(const double* x, double x0, const double* Y1, const double* v1, bool row0_1, double* B1,
                        const double* Y2, const double* v2, double* B2) {
    const int nq = D.nq, iq0 = D.iq0, iq1 = iq0 + nq, igp = D.igp, ir = D.ir, lg = D.lg, lgp = D.lgp, lr = D.lr, lnu = D.lnu;
    const double k = S.blk.m.k;
    const Tab& T = S.blk.T;
    double p[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) p[i] = 0.0;
    {
      const int nt = lg - 3, np = lgp - 3, nr = lr - 3;
      for (int e = tid; e < nt + np + nr; e += TT) {
        const bool ph = e < nt + np;
        const int l = 3 + (e < nt ? e : (ph ? e - nt : e - nt - np));
        const int j = (e < nt ? 7 : (ph ? igp : ir)) + l;
        const double xj = x[j], kl = k * T.lo[l], ku = k * T.up[l];
        p[1] += xj * (kl * Y1[j - 1] - ku * Y1[j + 1]);
        if (ph) p[0] -= xj * Y1[j];
        if constexpr (TWO) {
          p[6] += xj * (kl * Y2[j - 1] - ku * Y2[j + 1]);
          if (ph) p[5] -= xj * Y2[j];
        }
      }
    }
    for (int e = tid; e < (lnu + 1) * nq; e += TT) {
      const int l = e / nq, i = e - l * nq, j = iq0 + e;
      const double xj = x[j], lo = l == lnu ? 1.0 : T.lo[l], up = l == lnu ? 0.0 : T.up[l];
      const int jm = l > 0 ? j - nq : j, jp = l < lnu ? j + nq : j;
      const double w1 = xj * (lo * Y1[jm] - up * Y1[jp]);
      p[2] += w1 * v1[i];
      p[3] += w1 * v1[nq + i];
      p[4] += w1 * v1[2 * nq + i];
      if constexpr (TWO) {
        const double w2 = xj * (lo * Y2[jm] - up * Y2[jp]);
        p[7] += w2 * v2[i];
        p[8] += w2 * v2[nq + i];
        p[9] += w2 * v2[2 * nq + i];
      }
    }
    // slots 0 .. 4 of part[0] / part[1]
    warp_sums<TWO ? 10 : 5>(p, lane, S.tmp[wi]);
    if (lane < 5) {
      S.part[0][wi][lane] = S.tmp[wi][lane];
      if constexpr (TWO) S.part[1][wi][lane] = S.tmp[wi][5 + lane];
    }
    if (wi == 0) {
      double q[TWO ? 18 : 10];
#pragma unroll
      for (int i = 0; i < (TWO ? 18 : 10); ++i) q[i] = 0.0;
      for (int i = lane; i < nq; i += 32) {
        const double wq = LDG(S.blk.c.w + i), dlf = Bk.w.m(M_Q + Q_DLF * nq + i);
        const double xa = x[iq0 + i], xc = x[iq0 + 2 * nq + i], xt = x[iq0 + lnu * nq + i] * (lnu + 1.0);
        q[0] += dlf * (xa * (1.0 / 6.0) - xc * (1.0 / 15.0));
        q[1] -= 0.4 * dlf * xc;
        double wy = wq * Y1[iq0 + i];
        q[2] += wy * v1[3 * nq + i]; q[3] += wy * v1[4 * nq + i]; q[4] += wy * v1[5 * nq + i];
        q[5] += wy * v1[i]; q[6] += wy * v1[nq + i]; q[7] += wy * v1[2 * nq + i];
        q[8] += wq * Y1[iq1 + i];
        q[9] -= xt * Y1[iq0 + lnu * nq + i];
        if constexpr (TWO) {
          wy = wq * Y2[iq0 + i];
          q[10] += wy * v2[3 * nq + i]; q[11] += wy * v2[4 * nq + i]; q[12] += wy * v2[5 * nq + i];
          q[13] += wy * v2[i]; q[14] += wy * v2[nq + i]; q[15] += wy * v2[2 * nq + i];
          q[16] += wq * Y2[iq1 + i];
          q[17] -= xt * Y2[iq0 + lnu * nq + i];
        }
      }
      warp_sums<TWO ? 18 : 10>(q, lane, S.tmp[3]);
      if (lane == 0) { S.hn = S.tmp[3][0]; S.en = S.tmp[3][1]; }
      if (lane < 8) {
        S.qs[0][lane] = S.tmp[3][2 + lane];
        if constexpr (TWO) S.qs[1][lane] = S.tmp[3][10 + lane];
      }
    } else if (wi == 1) {
      const LeadLists& Q = S.lead;
      if (lane < 5) {
        double s = 0.0;
        for (int e = 0; e < Q.nder; ++e)
          if (Q.der_kind[e] == lane) s += Q.der_kap[e] * x[Q.der_tgt[e]];
        S.xk[lane] = s;
      }
    } else if (wi == 2) {
      const LeadLists& Q = S.lead;
      if (lane < NSIG) {
        double s1 = 0.0, s2 = 0.0;
        for (int e = Q.sig_at[lane]; e < Q.sig_at[lane + 1]; ++e) {
          const int src = Q.sig_src[e];
          const double kx = Q.sig_kap[e] * (Q.sig_tgt[e] == 0 ? x0 : x[Q.sig_tgt[e]]);
          if (src >= 0) {
            s1 += kx * Y1[src];
            if constexpr (TWO) s2 += kx * Y2[src];
          } else if (row0_1) {
            s1 += kx;
          }
        }
        B1[B_SIG + lane] = s1;
        if constexpr (TWO) B2[B_SIG + lane] += s2;
      }
    }
    team_sync();
    if (wi == 0) assemble(Y1, 0, B1, false);
    else if (TWO && wi == 1) assemble(Y2, 1, B2, true);
  }

  // the remaining entries of a form from its sums (one warp)
  __device__ void assemble(const double* Y, int f, double* B, bool add) {
    const double xh1 = S.xk[DK_HP1] + 0.5 * S.xk[DK_ALPHA] + S.hn, xhw = S.xk[DK_HPW];
    const double xe = S.xk[DK_E] + 3.0 * S.xk[DK_ALPHA] + S.en, xp = S.xk[DK_P1];
    for (int e = lane; e < NB - NSIG; e += 32) {
      const int j = NSIG + e;
      double v;
      if (j == B_OP || j == B_FREE || (j >= B_V && j < B_V + 3)) {
        const int i = j == B_OP ? 0 : (j == B_FREE ? 1 : 2 + j - B_V);
        v = S.part[f][0][i] + S.part[f][1][i] + S.part[f][2][i];
      } else if (j == B_IT) {
        v = S.qs[f][7];
      } else {
        double c, s;
        if (j >= B_H1 && j < B_H1 + 6) { c = xh1; s = Y[gather_fixed(0, j - B_H1)]; }
        else if (j >= B_H1T && j < B_H1T + 3) { c = xh1; s = S.qs[f][j - B_H1T]; }
        else if (j >= B_HW && j < B_HW + 6) { c = xhw; s = Y[gather_fixed(0, j - B_HW)]; }
        else if (j >= B_HWT && j < B_HWT + 3) { c = xhw; s = S.qs[f][j - B_HWT]; }
        else if (j >= B_E && j < B_E + 5) { c = xe; s = Y[gather_fixed(1, j - B_E)]; }
        else if (j == B_EF) { c = xe; s = S.qs[f][6]; }
        else if (j >= B_P && j < B_P + 6) { c = xp; s = Y[gather_fixed(2, j - B_P)]; }
        else if (j >= B_P1V && j < B_P1V + 3) { c = xp; s = S.qs[f][j - B_P1V]; }
        else { c = xp; s = S.qs[f][3 + j - B_PV]; }
        v = c * s;
      }
      B[j] = add ? B[j] + v : v;
    }
    __syncwarp();
  }
  // the fixed elements the functionals read: h' (0), eta' (1), P1 (2)
  __device__ __forceinline__ int gather_fixed(int which, int i) const { return gather_index(D, which, D.nq + i); }

  __device__ __forceinline__ double dot(const double* a, const double* b) const {
    double s = lane < NB ? a[lane] * b[lane] : 0.0;
    if (lane + 32 < NB) s += a[lane + 32] * b[lane + 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  }

  // ------------------------------------------------------------------ J^T
  // lead-row sources and the metric functionals of J^T x, added to z by one
  // warp; with DER the a-derivative (C1 beside C)
  template <bool DER>
  __device__ void jt_special(const double* Cv, const double* C1v, const double* x, const double* v, double* z) {
    const Coef<double>& C = *reinterpret_cast<const Coef<double>*>(Cv);
    const Coef<double>& E = *reinterpret_cast<const Coef<double>*>(C1v);
    const LeadLists& Q = S.lead;
    const int nq = D.nq, iq0 = D.iq0;
    for (int sl = lane; sl < Q.nslot; sl += 32) {
      double s = 0.0;
      for (int e = Q.slot_at[sl]; e < Q.slot_at[sl + 1]; ++e)
        s += (DER ? E.sg[Q.slot_sig[e]] : C.sg[Q.slot_sig[e]]) * (Q.slot_kap[e] * x[Q.slot_tgt[e]]);
      z[Q.slot_dst[sl]] += s;
    }
    __syncwarp();
    const double h0 = S.xk[DK_HP1] + 0.5 * S.xk[DK_ALPHA] + S.hn, hw = S.xk[DK_HPW], xp = S.xk[DK_P1];
    const double we = S.xk[DK_E] + 3.0 * S.xk[DK_ALPHA] + S.en;
    const double wh = h0 + C.sg[SG_W1] * hw, wp = C.sg[SG_A] * xp;
    const double wh1 = DER ? E.sg[SG_W1] * hw : 0.0, wp1 = DER ? E.sg[SG_A] * xp : 0.0;
    if (lane < 11) {
      // z[2, 3, 5, 7, ir, n-2] from h', z[3, 5, 7, ir, n-2, n-1] from P1, z[4, 6, 8, ir+1, n-1] from eta'
      double s;
      int j;
      if (lane < 6) {
        j = gather_fixed(0, lane);
        s = DER ? wh * E.ch[lane] + wh1 * C.ch[lane] : wh * C.ch[lane];
        if (lane > 0) s += DER ? wp * E.cp[lane - 1] + wp1 * C.cp[lane - 1] : wp * C.cp[lane - 1];
      } else {
        const int q = lane - 6;
        j = gather_fixed(1, q);
        s = we * (DER ? E.ce[q] : C.ce[q]);
        if (q == 4) s += DER ? wp * E.cp[5] + wp1 * C.cp[5] : wp * C.cp[5];
      }
      z[j] += s;
    }
    for (int i = lane; i < nq; i += 32) {
      const double wq = LDG(S.blk.c.w + i), vi = v[i], iv = v[3 * nq + i];
      double s, e;
      if (DER) {
        const double am = S.blk.m.amnu, vd = v[nq + i] * am, ivd = v[4 * nq + i] * am;   // d mu / d a = m_nu
        s = (wh1 * C.xh + wh * E.xh) * wq * iv + wh * C.xh * wq * ivd + (wp1 * C.xp + wp * E.xp) * wq * (iv + vi) +
            wp * C.xp * wq * (ivd + vd);
        e = we * E.xe * wq;
      } else {
        s = wh * C.xh * wq * iv + wp * C.xp * wq * (iv + vi);
        e = we * C.xe * wq;
      }
      z[iq0 + i] += s;
      z[iq0 + nq + i] += e;
    }
    __syncwarp();
  }

  // hierarchy couplings of (J^T x)_j: opac and kv (k v_q, or their
  // a-derivatives), itau the truncation (0 for the derivative)
  __device__ __forceinline__ double jt_hier(const double* x, int j, double k, double opac, const double* v, double kf,
                                            double itau) const {
    const int nq = D.nq, iq0 = D.iq0, lnu = D.lnu;
    const Tab& T = S.blk.T;
    double s = 0.0;
    if (j >= iq0 && j < D.n - 2) {
      const int e = j - iq0, l = e / nq, i = e - l * nq;
      const double kv = kf * v[i];
      if (l >= 1) s -= T.up[l - 1] * x[j - nq] * kv;
      if (l < lnu) s += (l + 1 == lnu ? 1.0 : T.lo[l + 1]) * x[j + nq] * kv;
      else s -= ((lnu + 1.0) * x[j]) * itau;
    } else if (j >= 7 && j < iq0) {
      const int which = j < D.igp ? 0 : (j < D.ir ? 1 : 2);
      const int l = j - (which == 0 ? 7 : (which == 1 ? D.igp : D.ir));
      const int lmax = which == 0 ? D.lg : (which == 1 ? D.lgp : D.lr);
      if (l + 1 >= 3 && l + 1 <= lmax - 1) s += (k * T.lo[l + 1]) * x[j + 1];
      if (l - 1 >= 3 && l - 1 <= lmax - 1) s -= (k * T.up[l - 1]) * x[j - 1];
      if (which < 2 && l >= 3 && l <= lmax - 1) s -= opac * x[j];
    }
    return s;
  }

  // ------------------------------------------------------------------ stage vectors
  // One pass over the stage vectors after stage SG's r is known: J^T's
  // hierarchy part into the stage point's cotangent, kbar_q += C / dt r, the
  // shares of the dt terms, rho += k_s[0] r, the cotangent passed on
  // (adj_stage_post), and then stage SG - 1's right-hand side and point
  // (adj_stage_pre).
  template <int SG>
  __device__ __forceinline__ void post_pre(double idt) {
    const int n = D.n;
    const Coef<double>& C = *reinterpret_cast<const Coef<double>*>(&S.C[SG][0]);
    const double k = S.blk.m.k, opac = C.opac, itau = C.itau, ks0 = K(SG, 0);
    const double* v = vv + SG * 6 * D.nq;
    constexpr int NP = SG >= 1 ? SG : 1;
    double cs[NP], ci[NP], aa[NP];
#pragma unroll
    for (int q = 0; q < SG; ++q) {
      cs[q] = R.C[SG][q];
      ci[q] = R.C[SG][q] * idt;
      aa[q] = SG <= 5 ? R.a[SG][q] : 0.0;
    }
    constexpr int SP = SG - 1;                       // the next stage
    constexpr int SB = SP <= 5 ? (SP > 0 ? SP : 0) : 5;
    double an[SB > 0 ? SB : 1];
#pragma unroll
    for (int q = 0; q < SB; ++q) an[q] = R.a[SB][q];
    for (int j = tid; j < n; j += TT) {
      double kk[NP], kbv[NP];
#pragma unroll
      for (int q = 0; q < SG; ++q) {
        kk[q] = K(q, j);
        kbv[q] = SG == 7 ? 0.0 : KB(q)[j];
      }
      const double rj = rb[j], kj = K(SG, j), y0 = SP >= 1 ? V(V_Y, j) : 0.0;
      double uj = (SG >= 1 ? ub[j] : lam[j]) + jt_hier(rb, j, k, opac, v, k, itau);
      pk += rj * kj;
      rho[j] = (SG == 7 ? 0.0 : rho[j]) + ks0 * rj;
      if constexpr (SG == 0) {
        lam[j] = uj;
      } else {
        double ck = 0.0;
#pragma unroll
        for (int q = 0; q < SG; ++q) {
          ck += cs[q] * kk[q];
          kbv[q] += ci[q] * rj;
        }
        pc += rj * ck;
        if constexpr (SG >= 6) {
          kbv[SG - 1] += uj;
          ub[j] = uj;
        } else {
          lam[j] = (SG == 5 ? 0.0 : lam[j]) + uj;
#pragma unroll
          for (int q = 0; q < SG; ++q) kbv[q] += aa[q] * uj;
          ub[j] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < SG; ++q) if (q < SG - 1) KB(q)[j] = kbv[q];
        rbn[j] = kbv[SG - 1];
        if constexpr (SP >= 1) {
          double uu = y0;
#pragma unroll
          for (int q = 0; q < SB; ++q) uu += an[q] * kk[q];
          if constexpr (SP >= 6) uu = uu + kk[5];
          if constexpr (SP >= 7) uu = uu + kk[6];
          u[j] = uu;
        }
      }
    }
  }

  // truncation rows of d f / d tau and their coefficient (lmax + 1) / t0^2
  __device__ __forceinline__ void trunc_row(int e, double it2, int& row, double& cf) const {
    if (e == 0) { row = 7 + D.lg; cf = (D.lg + 1.0) * it2; }
    else if (e == 1) { row = D.igp + D.lgp; cf = (D.lgp + 1.0) * it2; }
    else if (e == 2) { row = D.ir + D.lr; cf = (D.lr + 1.0) * it2; }
    else { row = D.iq0 + D.lnu * D.nq + (e - 3); cf = (D.lnu + 1.0) * it2; }
  }

  template <int SG>
  __device__ __forceinline__ void stage_back(double dt, double idt, double it2, double wQ) {
    solve_wt(wQ);
    const double x0 = row0();
    const int nq = D.nq;
    const double* y0 = &V(V_Y, 0);
    const double* us = SG >= 1 ? u : y0;
    forms<true>(rb, x0, us, vv + SG * 6 * nq, true, S.B[SG], &K(SG, 0), vv, S.BW);
    double* tgt = SG >= 1 ? ub : lam;
    if (wi == 0) {
      const double r0 = dot(S.dphi[SG], S.B[SG]);
      if (lane == 0) {
        tgt[0] += r0;
        rb[0] = x0;
      }
    } else if (wi == 1) {
      if constexpr (SG <= 4) {
        for (int e = lane; e < 3 + nq; e += 32) {
          int row;
          double cf;
          trunc_row(e, it2, row, cf);
          S.ft[e] += dt * R.d[SG] * rb[row];
          pf += R.d[SG] * (rb[row] * cf * y0[row]);
        }
      }
    } else if (wi == 2) {
      jt_special<false>(S.C[SG], S.C1, rb, vv + SG * 6 * nq, tgt);
    }
    team_sync();
    post_pre<SG>(idt);
    team_sync();
    double* t = rb;
    rb = rbn;
    rbn = t;
  }

  // One step backwards (the team): lam goes from dL/dy1 to dL/dy0 (without
  // yo2), S.tb_left / S.tb_right collect dL/dt0 and dL/dt1.
  __device__ void step_back(double t0, double dt) {
    const int n = D.n, nq = D.nq;
    const double idt = 1.0 / dt, it2 = 1.0 / (t0 * t0);
    const double wQ = S.blk.bg[S.blk.cur].wQ.v;
    const double* y0 = &V(V_Y, 0);
    // stage 7: kbar = ubar = dL/dy1 and its point
    for (int j = tid; j < n; j += TT) {
      const double l = lam[j];
      rb[j] = l;
      ub[j] = l;
      double uu = V(V_Y, j);
#pragma unroll
      for (int q = 0; q < 5; ++q) uu += R.a[5][q] * K(q, j);
      u[j] = (uu + K(5, j)) + K(6, j);
    }
    for (int i = tid; i < NB; i += TT) S.BW[i] = 0.0;
    for (int i = tid; i < 3 + nq; i += TT) S.ft[i] = 0.0;
    pc = 0.0; pk = 0.0; pf = 0.0;
    prep_wt();
    stage_back<7>(dt, idt, it2, wQ);
    stage_back<6>(dt, idt, it2, wQ);
    stage_back<5>(dt, idt, it2, wQ);
    stage_back<4>(dt, idt, it2, wQ);
    stage_back<3>(dt, idt, it2, wQ);
    stage_back<2>(dt, idt, it2, wQ);
    stage_back<1>(dt, idt, it2, wQ);
    stage_back<0>(dt, idt, it2, wQ);
    // W = I / (gamma dt) - J(t0, y0): the a-derivative of J(y0) on (rho, y0)
    forms<false>(rho, rho[0], y0, vv, true, S.BR, nullptr, nullptr, nullptr);
    if (wi == 0) {
      const double da0 = dot(S.dphi[0], S.BW) + dot(S.ddphi0, S.BR);
      if (lane == 0) lam[0] += da0;
    } else if (wi == 2) {
      jt_special<true>(S.C[0], S.C1, rho, vv, lam);
    }
    {
      double x[3] = {pc, pk, pf};
      warp_sums<3>(x, lane, S.tmp[wi]);
    }
    team_sync();
    const Coef<double>& E = *reinterpret_cast<const Coef<double>*>(S.C1);
    const double kam = S.blk.m.k * S.blk.m.amnu;
    for (int j = tid; j < n; j += TT) lam[j] += jt_hier(rho, j, 0.0, E.opac, vv + nq, kam, 0.0);
    team_sync();
    if (wi == 0) {
      double pt = 0.0;
      for (int e = lane; e < 3 + nq; e += 32) {
        int row;
        double cf;
        trunc_row(e, it2, row, cf);
        const double fb = S.ft[e];
        lam[row] += cf * fb;
        pt -= 2.0 * cf / t0 * y0[row] * fb;
      }
      // d/dt of Phi: 1/t enters three scalars and the truncation sum
      double tbs = 0.0, cs = 0.0;
      if (lane < 9) {
        const int s = lane < 8 ? lane : 0;
        const double* B = lane < 8 ? S.B[s] : S.BW;
        const double itau = reinterpret_cast<const Coef<double>*>(S.C[s])->itau;
        tbs = -(itau * itau) * (B[B_IT] - (D.lg + 1.0) * B[B_SIG + SG_ITG] - (D.lgp + 1.0) * B[B_SIG + SG_ITP] -
                                (D.lr + 1.0) * B[B_SIG + SG_ITR]);
        cs = lane < 8 ? R.c[s] * tbs : 0.0;
      }
      pt += tbs;
      for (int o = 16; o > 0; o >>= 1) {
        pt += __shfl_xor_sync(0xffffffffu, pt, o);
        cs += __shfl_xor_sync(0xffffffffu, cs, o);
      }
      if (lane == 0) {
        const double pcs = S.tmp[0][0] + S.tmp[1][0] + S.tmp[2][0], pks = S.tmp[0][1] + S.tmp[1][1] + S.tmp[2][1],
                     pfs = S.tmp[0][2] + S.tmp[1][2] + S.tmp[2][2];
        const double db = cs - pcs * idt * idt + pfs + pks * Bk.w.m(M_SCAL + S_D) * idt;
        S.tb_right += db;
        S.tb_left += pt - db;
      }
    }
  }

  // The step's theta gradient (all warps, after a block barrier): summed over
  // the form's entries and stages before it joins the earlier steps', since
  // the entries' terms cancel.  A warp's sum goes to S.tmp[wi].
  __device__ void add_theta() {
    const int npar = it->npar;
    double th[MAXPAR];
#pragma unroll
    for (int p = 0; p < MAXPAR; ++p) th[p] = 0.0;
    for (int e = tid; e < 8 * NB; e += NT) {
      const int s = e & 7, j = e >> 3;
      const double b = S.B[s][j] + (s == 0 ? S.BW[j] : 0.0);
      const double* t = dth + e * npar;
#pragma unroll
      for (int p = 0; p < MAXPAR; ++p)
        if (p < npar) th[p] += t[p] * b;
    }
    if (tid < NB) {
      const double b = S.BR[tid];
      const double* t = dth1 + tid * npar;
#pragma unroll
      for (int p = 0; p < MAXPAR; ++p)
        if (p < npar) th[p] += t[p] * b;
    }
    warp_sums<MAXPAR>(th, lane, S.tmp[wi]);
  }

  // a boundary's time adjoint into tau_start (scaled times), an output time or T1
  __device__ void boundary(int j, double tbar, double T1, int omax) {
    if (j == 0) { S.sts += tbar; return; }
    if (j >= it->nrec) { S.to[omax] += tbar; return; }
    const double v = LDG(it->rec + j);
    if (v < 0.0) { S.to[(int)(-v) - 1] += tbar; return; }
    if (v >= T1) { S.to[omax] += tbar; return; }
    S.sts += tbar * v / LDG(it->rec);
  }

  // The item: adjoint_item of deb_adjoint.cuh.  A: the vectors as output_adjoint
  // names them; sc its scratch.
  __device__ int run(const AdjItem& item, int nout, const AWS<32>& A, double* seg, int seg_cap, double* gth) {
    it = &item;
    const int n = D.n, N = item.nrec, Sd = item.ck_stride, npar = item.npar;
    double* sc = A.sc;
    {
      Cosmo c;
      if (N < 1 || Sd < 1 || Sd > seg_cap || !load_cosmo(item.blob0, item.blob_len, c) || c.nq != D.nq) return ST_BAD_INPUT;
      ModeConst m;
      mode_const(c, item.k, m);
      m.grr = __fma_rn(m.grhor, m.Neff, m.grhog);
      __syncthreads();
      if (tid == 0) { S.blk.c = c; S.blk.m = m; }
    }
    bool ok = true;
    for (int b = tid; b < 2 * npar; b += NT) {
      SetCtx x;
      ok = item_cosmo(item, b, x.c) && x.c.nq == D.nq;
      if (ok) { mode_const(x.c, item.k, x.m); sets[b] = x; }
    }
    if (__syncthreads_or(!ok)) return ST_BAD_INPUT;
    double T1 = LDG(item.tau0);
    int omax = 0;
    for (int o = 1; o < nout; ++o) { const double t = LDG(item.tau0 + o); if (t > T1) { T1 = t; omax = o; } }
    const double ts0 = LDG(item.rec);
    Ctl ctl;
    ctl.dense = 0; ctl.nout = nout; ctl.replay = 1; ctl.record = 0; ctl.step_ts = 0; ctl.return_full = 0;
    const Grp<NT> gp{tid};
    const Grp<32> gw{lane};
    WS<NT> wb;
    wb.p = Bk.w.p; wb.kp = Bk.w.kp; wb.n = n; wb.misc0 = Bk.w.misc0; wb.dp = nullptr;
    initial_conditions<NT>(gp, S.blk.c, S.blk.m, D, ts0, wb, V_Y);   // momentum-bin constants
    for (int j = tid; j < n; j += NT) lam[j] = 0.0;
    for (int i = tid; i < 16; i += NT) sc[SC_TH + i] = 0.0;
    for (int i = tid; i < nout; i += NT) S.to[i] = 0.0;
    if (tid == 0) { S.sts = 0.0; S.tbn = 0.0; S.blk.cur = 0; }
    if (tid < MAXPAR) S.out[tid] = 0.0;
    __syncthreads();
    const int nseg = (N + Sd - 1) / Sd;
    if (Bk.producer()) Bk.bg_dual(LDG(item.ck + (long)(nseg - 1) * n), S.blk.bg[0]);
    for (int sg = nseg - 1; sg >= 0; --sg) {
      const int c = sg * Sd, e = (c + Sd < N) ? c + Sd : N;
      // states of the segment from its checkpoint
      const double* ck = item.ck + (long)sg * n;
      for (int j = tid; j < n; j += NT) { const double y = LDG(ck + j); seg[j] = y; V(V_Y, j) = y; }
      __syncthreads();
      for (int j = c; j + 1 < e; ++j) {
        const double tj = adj_time(item, T1, j), dtj = adj_time(item, T1, j + 1) - tj;
        if (Bk.producer()) Bk.produce(tj, dtj, V_Y, V_U, true);
        else Bk.advance(tj, dtj, V_Y, V_U);
        __syncthreads();
        double* s1 = seg + (long)(j - c + 1) * n;
        for (int q = tid; q < n; q += NT) { const double y = V(V_U, q); s1[q] = y; V(V_Y, q) = y; }
        if (tid == 0) S.blk.cur ^= 1;
        __syncthreads();
      }
      for (int j = e - 1; j >= c; --j) {
        const double tj = adj_time(item, T1, j), tj1 = adj_time(item, T1, j + 1), dtj = tj1 - tj;
        if (j < e - 1) {
          const double* sj = seg + (long)(j - c) * n;
          for (int q = tid; q < n; q += NT) V(V_Y, q) = sj[q];
          __syncthreads();
        }
        const double a0 = V(V_Y, 0);
        if (Bk.producer()) {
          const double an = j > c ? seg[(long)(j - 1 - c) * n] : (sg > 0 ? LDG(ck - n) : a0);
          Bk.produce(tj, dtj, V_Y, V_U, false);
          produce_nominal(tj, dtj, a0);
          bar_arrive(BAR_ADJ, NT);
          produce_theta(tj, dtj, a0);
          Bk.bg_dual(an, S.blk.bg[S.blk.cur ^ 1]);
        } else {
          Bk.advance(tj, dtj, V_Y, V_U);
          // outputs inside (tj, tj1] with a cotangent
          if (wi == 0) {
            int hits = 0;
            for (int h = 0; h < 2; ++h) {
              const int o = lane + 32 * h;
              bool in = false;
              if (o < nout) {
                const double to = LDG(item.tau0 + o);
                in = to > tj && to <= tj1;
                if (in) {
                  bool any = false;
                  for (int f = 0; f < NFIELD; ++f) any = any || LDG(item.gy + (long)o * NFIELD + f) != 0.0;
                  in = any;
                }
              }
              const unsigned msk = __ballot_sync(0xffffffffu, in);
              if (lane == 0) S.hitmask[h] = msk;
              hits |= msk != 0u;
            }
            if (lane == 0) { S.hits = hits; S.tb_left = 0.0; S.tb_right = S.tbn; }
          }
          bar_sync(BAR_ADJ, NT);
          if (S.hits) {
            for (int q = tid; q < n; q += TT) yo2[q] = 0.0;
            team_sync();
            if (wi == 0) {
              const VecRef yv = A.fv(V_Y), uv = A.fv(V_U);
              for (int o = 0; o < nout; ++o) {
                if (!((S.hitmask[o >> 5] >> (o & 31)) & 1u)) continue;
                const double to = LDG(item.tau0 + o);
                const double cf = (to - tj) / dtj;
                const double dcf = output_adjoint<32>(gw, item, S.blk.c, S.blk.m, D, A, o, cf, yv, uv);
                if (lane == 0) {
                  S.to[o] += dcf / dtj;
                  S.tb_left += dcf * (to - tj1) / (dtj * dtj);
                  S.tb_right -= dcf * (to - tj) / (dtj * dtj);
                }
                __syncwarp();
              }
            }
            team_sync();
          }
          step_back(tj, dtj);
        }
        __syncthreads();
        add_theta();
        if (S.hits)
          for (int q = tid; q < n; q += NT) lam[q] += yo2[q];
        if (tid == 0) {
          boundary(j + 1, S.tb_right, T1, omax);
          S.tbn = S.tb_left;
          S.blk.cur ^= 1;
        }
        __syncthreads();
        if (tid < npar) S.out[tid] += (S.tmp[0][tid] + S.tmp[1][tid]) + (S.tmp[2][tid] + S.tmp[3][tid]);
      }
    }
    if (tid == 0) boundary(0, S.tbn, T1, omax);
    // tau_start, the ICs and the output times of each table set
    __syncthreads();
    // (a warp per parameter as far as the stage vectors hold their states)
    const long per = n + NQARR * D.nq;
    const int nw = 4L * n / per < NW ? (int)(4L * n / per) : NW;
    for (int p = wi; p < npar && wi < nw; p += nw) {
      double* y = Bk.w.kp + 2 * wi * per;
      double ts[2];
      for (int e = 0; e < 2; ++e) {
        const SetCtx& X = sets[2 * p + e];
        ts[e] = mode_start(X.c, X.m, ctl, item.taus + (long)(2 * p + e) * nout);
        initial_state(gw, X.c, X.m, ts[e], y + e * per);
      }
      // lam . (y+ - y-): the difference first, whose rounding is relative to
      // it and not to lam . y (of the size of the whole signal) over 2 eps
      double dotp = 0.0;
      for (int j = lane; j < n; j += 32) dotp += lam[j] * (y[j] - y[per + j]);
      for (int o = 16; o > 0; o >>= 1) dotp += __shfl_xor_sync(0xffffffffu, dotp, o);
      if (lane == 0) { sc[SC_RES + p] = dotp; sc[SC_CF + p] = ts[0] - ts[1]; }
      __syncwarp();
    }
    __syncthreads();
    if (tid < npar) {
      const int p = tid;
      const double i2e = 1.0 / (2.0 * LDG(item.eps + p));
      double g = sc[SC_TH + p] + S.out[p];
      g += sc[SC_RES + p] * i2e;
      g += S.sts * sc[SC_CF + p] * i2e;
      for (int o = 0; o < nout; ++o)
        g += S.to[o] * (LDG(item.taus + (long)(2 * p) * nout + o) - LDG(item.taus + (long)(2 * p + 1) * nout + o)) * i2e;
      gth[p] = g;
    }
    const bool fin = isfinite_(lam[0]);
    __syncthreads();
    return fin ? ST_OK : ST_NONFINITE;
  }

  // the adiabatic initial state of a table set, by one warp, into y: n + NQARR
  // nq doubles (the state, then the momentum bins' constants, which must not
  // overwrite the nominal ones)
  __device__ __forceinline__ void initial_state(const Grp<32>& gw, const Cosmo& c, const ModeConst& m, double tau,
                                                double* y) {
    WS<32> v;
    v.p = y;
    v.n = D.n;
    v.misc0 = D.n - M_Q;    // of MISC only the bins' arrays (from M_Q on) are written
    v.kp = nullptr;
    v.dp = nullptr;
    initial_conditions<32>(gw, c, m, D, tau, v, V_Y);
  }
};

#endif  // __CUDACC__

}  // namespace deb
