// flint_fixkin.cuh -- warp-per-cell kinetics on the fixed-point image.
//
// The same quantities as warp_kinetics (flint_dev.cuh), with every exponent,
// exponential and logarithm and the thermo polynomials in 64-bit fixed point
// (flint_fix.cuh).  What remains on the FP64 pipe per cell: the concentrations,
// four products per reaction round, the falloff blend, the species sums, and
// (JAC) the Jacobian.  A mechanism without the fixed-point image, and a cell
// outside its temperature range, go through warp_kinetics.
#pragma once
#include "flint_dev.cuh"

namespace flint {

// Index word of a reaction: bits 0-17 three reactant factors, 18-35 three
// product factors (6 bits each, `dummy` where absent), 36-39 dn + 8, 40-41
// type, 42 reversible, 43 A < 0, 44 and 45 both reactant and both product factors
// of a plain reaction are one species, 46 power form (the factors' orders are
// f_ord), 48-55 third-body row.
__device__ __forceinline__ int fix_type(uint64_t w) { return (int)(w >> 40) & 3; }
__device__ __forceinline__ bool fix_rev(uint64_t w) { return (w >> 42) & 1; }
__device__ __forceinline__ bool fix_power(uint64_t w) { return (w >> 46) & 1; }
__device__ __forceinline__ bool fix_twice_r(uint64_t w) { return (w >> 44) & 1; }
__device__ __forceinline__ bool fix_twice_p(uint64_t w) { return (w >> 45) & 1; }
__device__ __forceinline__ int fix_tbrow(uint64_t w) { return (int)(w >> 48) & 0xff; }
__device__ __forceinline__ int fix_idx(uint64_t w, int slot) { return (int)(w >> (6 * slot)) & 63; }
__device__ __forceinline__ int fix_dn(uint64_t w) { return ((int)(w >> 36) & 15) - 8; }

struct FixView {
  int ns, nr, nrpad, nsp, nfall, dummy, w3, ntb, seg_len;
  double inv_r_eos, r_eos, r_thermo, Tlo, Thi;
  int64_t lC;
  const double *mw, *invmw, *tr, *tbd, *tbv;
  const int64_t *tmid, *a, *ra;
  const uint64_t *g, *h, *c, *b, *e, *rb, *re, *et, *lt, *ix, *cx, *cy, *ord;
  const int *tbp, *tbs, *rs, *rw, *piece;
  const double *rv, *segv, *coef;
  const uint32_t *seg, *term;
  const uint16_t* target;
  int term_len;
  __device__ __forceinline__ void bind(const ImageLayout& L, const uint8_t* base) {
    ns = L.ns; nr = L.nr; nrpad = L.nrpad; nsp = L.nsp; nfall = L.nfall; dummy = fix_dummy(L.nsp); w3 = L.fix_w3;
    ntb = L.fix_ntb; seg_len = L.seg_len;
    inv_r_eos = L.inv_r_eos; r_eos = L.r_eos; r_thermo = L.r_thermo; Tlo = L.fix_Tlo; Thi = L.fix_Thi; lC = L.fix_lC;
    auto D = [&](int o) { return (const double*)(base + o); };
    auto I = [&](int o) { return (const int64_t*)(base + o); };
    auto U = [&](int o) { return (const uint64_t*)(base + o); };
    mw = D(L.f_mw); invmw = D(L.f_invmw); tr = D(L.f_tr); tbd = D(L.f_tbd); tbv = D(L.f_tbv);
    tmid = I(L.f_tmid); a = I(L.f_a); ra = I(L.f_ra);
    b = U(L.f_b); e = U(L.f_e);
    bind_thermo(L, base);
    rb = U(L.f_rb); re = U(L.f_re); et = U(L.f_exp); lt = U(L.f_log); ix = U(L.f_ix); ord = U(L.f_ord); cx = U(L.f_cx); cy = U(L.f_cy);
    tbp = (const int*)(base + L.f_tbp); tbs = (const int*)(base + L.f_tbs);
    rs = (const int*)(base + L.f_rs); rw = (const int*)(base + L.f_rw); rv = D(L.f_rv);
    seg = (const uint32_t*)(base + L.f_seg); segv = D(L.f_segv); piece = (const int*)(base + L.f_piece);
    bind_terms(L, base);
  }
  __device__ __forceinline__ void bind_thermo(const ImageLayout& L, const uint8_t* base) {
    g = (const uint64_t*)(base + L.f_g); h = (const uint64_t*)(base + L.f_h); c = (const uint64_t*)(base + L.f_c);
  }
  __device__ __forceinline__ void bind_terms(const ImageLayout& L, const uint8_t* base) {
    term = (const uint32_t*)(base + L.f_term); target = (const uint16_t*)(base + L.f_target);
    coef = (const double*)(base + L.f_coef); term_len = L.term_len;
  }
  __device__ __forceinline__ bool covers(double T) const { return T >= Tlo && T < Thi; }
};

// Sum over the warp in 64-bit integers: every lane's value aligned to the
// largest exponent of the warp (58 bits below it), three 32-bit warp reductions
// of its 24-bit pieces, one rounding at the end.  The result is the exact sum to
// 2^-57 of the largest term, the same on every lane, with no FP64 instruction
// (the FP64 butterfly took five DADDs of 19 cycles and ten shuffles).
static __device__ __noinline__ double warp_sum_slow(double v) { return warp_sum(v); }
__device__ __forceinline__ double warp_isum(double v) {
  const int64_t b = __double_as_longlong(v);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  const unsigned emax = __reduce_max_sync(FULL, e);
  if (emax - 128u > 1900u) return warp_sum_slow(v);   // zeros, subnormal, huge, inf, NaN
  int64_t m = (b & 0xfffffffffffffll) | (e ? ONE52 : 0);
  const unsigned sh = emax - (e ? e : 1u);
  m = sh < 58 ? (m << 5) >> sh : 0;
  m = b < 0 ? -m : m;
  const unsigned lo = __reduce_add_sync(FULL, (unsigned)m & 0xffffffu);
  const unsigned mi = __reduce_add_sync(FULL, (unsigned)(m >> 24) & 0xffffffu);
  const int hi = __reduce_add_sync(FULL, (int)(m >> 48));
  const int64_t S = ((int64_t)hi << 48) + ((int64_t)mi << 24) + (int64_t)lo;
  return fix2d(S, 1080 - (int)emax);
}

__device__ __forceinline__ double fix_tb_conc(const FixView& m, int t, double ctot, const double* c) {
  double M = m.tbd[t] * ctot;
  for (int e = m.tbp[t]; e < m.tbp[t + 1]; ++e) M = fma(m.tbv[e], c[m.tbs[e]], M);
  return M;
}

// Constants of the Troe blend with all logarithms in octaves (base 2): x = log Pr
// - 0.4 - 0.67 log Fc, n = 0.75 - 1.27 log Fc, den = n - 0.14 x and log F = log Fc
// den^2 / (den^2 + x^2); x, n and den carry the factor log2(10), which cancels.
constexpr int64_t TROE_C40 = 5984253652114523ll;        // 0.40 log2(10)  Q52
constexpr int64_t TROE_C75 = 11220475597714730ll;       // 0.75 log2(10)  Q52
constexpr int64_t TROE_M67 = 6179659264692699791ll;     // 0.67  Q63
constexpr int64_t TROE_M127 = 5856841243402782638ll;    // 1.27  Q62
constexpr int64_t TROE_M14 = 1291272085159668613ll;     // 0.14  Q63

// x, or 1e-300 where x is smaller (compared as bit patterns: no FP64 slot).
__device__ __forceinline__ double floor_tiny(double x) {
  return __double_as_longlong(x) > 0x01a56e1fc2f8f359ll ? x : 1e-300;
}

__device__ __forceinline__ int64_t mulhi_s(int64_t a, int64_t b) { return __mul64hi(a, b); }

// The blend from log2 Fc and log2 Pr (Q52).
__device__ __forceinline__ double troe_blend_raw(int64_t lg, int64_t lgP, const uint64_t* et) {
  const int64_t xx = lgP - TROE_C40 - (mulhi_s(lg, TROE_M67) << 1);
  const int64_t den = TROE_C75 - (mulhi_s(lg, TROE_M127) << 2) - (mulhi_s(xx, TROE_M14) << 1);
  const double dx = fix2d(xx, 52), dd = fix2d(den, 52), d2 = dd * dd;
  return exp2_q52(d2fix52(fix2d(lg, 52) * (d2 * recip(fma(dx, dx, d2)))), et);
}

__device__ __forceinline__ double troe_blend(double Fc, double Pr, const uint64_t* lt, const uint64_t* et) {
  return troe_blend_raw(log2_q52(floor_tiny(Fc), lt), log2_q52(floor_tiny(Pr), lt), et);
}

// Effective rate coefficient of a falloff reaction (i-th, reaction word w) from
// its high-pressure limit's exponent xinf (Q52; SUB: below the normal range too).
template <bool SUB = false>
__device__ __forceinline__ double cell_falloff(const FixView& m, int i, int type, int64_t xinf, double M, const FixT& f,
                                               double T, double Tinv) {
  const double kinf = exp2_q52<SUB>(xinf, m.et);
  const double kratio = exp2_q52(fix_arrhenius(m.ra[i], m.rb[i], m.re[i], f), m.et);
  const double Pr = kratio * M;
  const double k = kinf * (Pr * recip(1.0 + Pr));
  if (type != 3) return k;
  const double z2 = m.tr[64 + i];
  double Fc = z2 != 0.0 ? exp2_q52(-d2fix52(z2 * Tinv), m.et) : 0.0;
  Fc = fma(m.tr[16 + i], exp2_q52(-d2fix52(m.tr[48 + i] * T), m.et), Fc);
  Fc = fma(m.tr[i], exp2_q52(-d2fix52(m.tr[32 + i] * T), m.et), Fc);
  return k * troe_blend(Fc, Pr, m.lt, m.et);
}

// What a cell's fixed pressure (cv: density) contributes: the reactor forms it
// once per cell.
struct FixPress {
  double pr;      // p, or rho (cv)
  double a;       // p / r_eos
  double b;       // r_eos / p, or 1 / rho (cv); for the right-hand side and the Jacobian
  bool cv;
  template <bool INV>
  __device__ __forceinline__ static FixPress of(const FixView& m, double pr, bool cv) {
    FixPress q;
    q.pr = pr;
    q.a = pr * m.inv_r_eos;
    q.b = INV ? (cv ? recip(pr) : m.r_eos * recip(pr)) : 0.0;
    q.cv = cv;
    return q;
  }
};

// One cell (see warp_kinetics for the meaning of pr, cv and s.Jr).  RHS: form
// out.f and out.fT; want_h: form out.cp_mass and out.h_mass.  JAC: the Jacobian is
// written to dst by columns of dld doubles; img: the global image, for its FP64
// coefficients.
template <bool JAC, int SPL, bool RHS>
__device__ __forceinline__ void kinetics_fix(const FixView& m, const uint8_t* __restrict__ img, const ImageLayout& L,
                                             const WarpScratch& s, int lane, const double (&Yk)[SPL], double T,
                                             const FixPress& pr, CellOutT<SPL>& out, bool want_h, double* dst, int dld) {
  const bool cv = pr.cv;
  const int ns = m.ns, nsp = m.nsp, nrpad = m.nrpad;
  const bool thermo = JAC || RHS || want_h;
  int64_t* G = reinterpret_cast<int64_t*>(s.gRT);
  double yw[SPL];
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    yw[j] = k < ns ? Yk[j] * m.invmw[k] : 0.0;
  }
  const double sumYW = warp_isum(SPL == 1 ? yw[0] : yw[0] + yw[SPL - 1]);
  const FixT f = fix_T(T, m.lt);
  const double X = T * sumYW;
  const double rho = cv ? pr.pr : pr.a * recip(X);
  const double ctot = rho * sumYW;
  // ---- species k = lane + 32 j
  double my_cpR[SPL], my_hRT[SPL], my_c[SPL];
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    my_cpR[j] = 0.0; my_hRT[j] = 0.0; my_c[j] = 0.0;
    int64_t gk = 0;
    double ck = k == m.dummy ? 1.0 : 0.0;
    if (k < ns) {
      ck = rho * yw[j];
      my_c[j] = ck;
      const bool lo = __double_as_longlong(T) <= m.tmid[k];
      const uint64_t t = lo ? f.t11 : f.t13;
      gk = fix_gibbs(m.g + (lo ? 0 : 7 * nsp) + k, nsp, t, f);
      if (thermo) {
        my_hRT[j] = fix2d(fix_enthalpy(m.h + (lo ? 0 : 6 * nsp) + k, nsp, t, f), 52);
        my_cpR[j] = fix2d(fix_poly5(m.c + (lo ? 0 : 5 * nsp) + k, nsp, t), 52);
      }
    }
    if (k < nsp) {
      s.c[k] = ck;
      G[k] = gk;
      if (JAC) s.hRT[k] = my_hRT[j];
    }
  }
  if (lane == 0 && m.dummy == nsp) { s.c[nsp] = 1.0; G[nsp] = 0; if (JAC) s.hRT[nsp] = 0.0; }
  __syncwarp();
  double invT = 0.0;
  const double *gb = nullptr, *gE = nullptr, *gb0 = nullptr, *gE0 = nullptr;   // FP64 Arrhenius data (JAC)
  if (JAC) {
    invT = recip(T);
    gb = (const double*)(img + L.o_b); gE = (const double*)(img + L.o_E);
    gb0 = (const double*)(img + L.o_b0); gE0 = (const double*)(img + L.o_E0);
  }
  // ---- falloff: the last nfall reactions (<= 16), as in warp_kinetics.  Pass 1
  // spreads their five exponentials each over the lanes, pass 2 forms M, Pr and
  // Fcent on lane i, pass 3 takes log2 of Fcent (lane i) and Pr (lane nfall + i)
  // together, pass 4 blends.
  const int NF = m.nfall, f0 = m.nr - NF;
  double* fo = JAC ? s.Jr : s.fo;
  // third-body concentrations, each row once, kept in the rate's place until the
  // rate itself is known; formed on one lane and read on another, so a barrier lies
  // between: the falloff passes' first one or, without falloff reactions, the else's
  for (int t = lane; t < m.ntb; t += WARP) s.q[m.nr - m.ntb + t] = fix_tb_conc(m, t, ctot, s.c);
  if (NF > 0) {
    const double Tinv = JAC ? invT : fix2d((int64_t)f.v, 70);
    for (int jb = lane; jb < 5 * NF; jb += WARP) {
      const int i = jb / 5, kind = jb - 5 * i, r = f0 + i;
      int64_t x;
      double keep = 1.0;
      if (kind < 2) {
        x = fix_arrhenius(kind == 0 ? m.a[r] : m.ra[i], kind == 0 ? m.b[r] : m.rb[i], kind == 0 ? m.e[r] : m.re[i], f);
      } else {
        const double z = m.tr[16 * kind + i];      // log2e/T3, log2e/T1, T2 log2e
        x = -d2fix52(z * (kind == 4 ? Tinv : T));
        if (kind == 4 && z == 0.0) keep = 0.0;
      }
      const double v = exp2_q52(x, m.et);
      fo[kind * WARP + i] = keep != 0.0 ? v : 0.0;
    }
    __syncwarp();
    double Pr = 1.0, Fc = 1.0, kinf = 0.0, kratio = 0.0;
    bool troe = false;
    if (lane < NF) {
      const uint64_t w = m.ix[f0 + lane];
      troe = fix_type(w) == 3;
      kinf = fo[lane];
      kratio = fo[WARP + lane];
      Pr = kratio * s.q[f0 + lane];
      if (troe) Fc = fma(m.tr[lane], fo[2 * WARP + lane], fma(m.tr[16 + lane], fo[3 * WARP + lane], fo[4 * WARP + lane]));
    }
    const double Pr_src = __shfl_sync(FULL, Pr, lane >= NF && lane < 2 * NF ? lane - NF : 0);
    double lg_in = lane < NF ? Fc : (lane < 2 * NF ? Pr_src : 1.0);
    lg_in = floor_tiny(lg_in);
    // octaves; Pr = inf or NaN gives a finite garbage exponent, and the NaN of
    // Pr / (1 + Pr) below makes the rate NaN as before
    const int64_t lg = log2_q52(lg_in, m.lt);
    const int64_t lgP = __shfl_sync(FULL, lg, lane < NF ? lane + NF : 0);
    double dx = 0.0, dden = 1.0, lgd = 0.0, nnd = 0.0, d2 = 1.0;
    if (troe) {
      const int64_t xx = lgP - TROE_C40 - (mulhi_s(lg, TROE_M67) << 1);
      const int64_t nn = TROE_C75 - (mulhi_s(lg, TROE_M127) << 2);
      const int64_t den = nn - (mulhi_s(xx, TROE_M14) << 1);
      dx = fix2d(xx, 52);
      dden = fix2d(den, 52);
      lgd = fix2d(lg, 52);
      d2 = dden * dden;
      if (JAC) nnd = fix2d(nn, 52);
    }
    // one reciprocal for both: den^2 + x^2 on lane i, 1 + Pr on lane nfall + i
    const double rc = recip(lane < NF ? fma(dx, dx, d2) : 1.0 + (lane < 2 * NF ? Pr_src : 0.0));
    const double iopr = __shfl_sync(FULL, rc, lane < NF ? lane + NF : 0);
    if (lane < NF) {
      const double R = d2 * rc;
      const double Fb = troe ? exp2_q52(d2fix52(lgd * R), m.et) : 1.0;
      fo[5 * WARP + lane] = kinf * (Pr * iopr) * Fb;
      if (JAC) {
        const int r = f0 + lane;
        const double dlnkinf = fma(gE[r], invT, gb[r]) * invT, dlnPr = fma(gE0[r], invT, gb0[r]) * invT;
        double Gf = 0.0, dlnF_T = 0.0;
        if (troe) {
          // d ln F: with f1 = x/den, Aq = 2 lgF f1 / ((1 + f1^2)^2 den^2) and
          // 1 + f1^2 = (den^2 + x^2)/den^2; lgF, x, n, den all carry the factor
          // log2(10), and Aq n, Aq x are free of it
          const double iden = recip(dden);
          const double f1 = dx * iden;
          const double Aq = 2.0 * lgd * f1 * (R * R) * (iden * iden);
          Gf = -Aq * nnd;
          const double e3 = fo[2 * WARP + lane], e1 = fo[3 * WARP + lane], e2 = fo[4 * WARP + lane];
          constexpr double LN2 = 0.6931471805599453;
          const double k3 = m.tr[32 + lane] * LN2, k1 = m.tr[48 + lane] * LN2, k2 = m.tr[64 + lane] * LN2;
          const double dFc = -m.tr[lane] * k3 * e3 - m.tr[16 + lane] * k1 * e1 + k2 * invT * invT * e2;
          dlnF_T = (R + Aq * (0.67 * nnd - 1.27 * dx)) * dFc / Fc;
        }
        fo[6 * WARP + lane] = dlnkinf + dlnPr * iopr + Gf * dlnPr + dlnF_T;
        fo[7 * WARP + lane] = kinf * Fb * iopr * (iopr + Gf) * kratio;
      }
    }
    __syncwarp();
  } else {
    __syncwarp();
  }
  // ---- reactions: rates of progress
  for (int r = lane; r < nrpad; r += WARP) {
    double q = 0.0;
    if (r < m.nr) {
      const uint64_t w = m.ix[r];
      const int type = fix_type(w);
      const bool rev = fix_rev(w);
      const int r0 = fix_idx(w, 0), r1 = fix_idx(w, 1), p0 = fix_idx(w, 3), p1 = fix_idx(w, 4);
      const double c0 = s.c[r0], c1 = s.c[r1], d0 = s.c[p0], d1 = s.c[p1];
      int64_t a = fix_arrhenius(m.a[r], m.b[r], m.e[r], f);
      a = type >= 2 ? 0 : a;
      // 1/Kc = 2^(dG - dn log2(p_ref/RT)), kr = kf / Kc
      int64_t ar = a + G[p0] + G[p1] - G[r0] - G[r1] - (int64_t)fix_dn(w) * (m.lC - (int64_t)(f.L >> 9));
      double c2 = 1.0, d2 = 1.0;
      if (m.w3) {
        const int r2 = fix_idx(w, 2), p2 = fix_idx(w, 5);
        ar += G[p2] - G[r2];
        c2 = s.c[r2];
        d2 = s.c[p2];
      }
      double kf = exp2_q52(a, m.et);
      double kr = rev ? exp2_q52(ar, m.et) : 0.0;
      const int sgn = ((int)(w >> 43) & 1) << 31;
      kf = __hiloint2double(__double2hiint(kf) ^ sgn, __double2loint(kf));
      kr = __hiloint2double(__double2hiint(kr) ^ sgn, __double2loint(kr));
      const double iKc = kr;                      // (falloff reactions: a = 0)
      double Mfac = 1.0;
      if (type == 1) {
        Mfac = s.q[r];
      } else if (type >= 2) {
        kf = fo[5 * WARP + r - f0];
        kr *= kf;
      }
      double Pf = c0 * c1, Pr = d0 * d1;
      if (m.w3) { Pf *= c2; Pr *= d2; }
      const double fwd = kf * Pf;
      q = fma(-kr, Pr, fwd);
      if (JAC) {
        // derivatives by factor; by the third body; T times the one by T
        const int ns2 = m.w3 ? 3 : 2;
        const double kfM = type == 1 ? kf * Mfac : kf, krM = type == 1 ? kr * Mfac : kr;
        const double rvs = krM * Pr;
        if (m.w3) {
          s.dq[r] = kfM * c1 * c2;
          s.dq[nrpad + r] = kfM * c0 * c2;
          s.dq[2 * nrpad + r] = kfM * (c0 * c1);
          s.dq[3 * nrpad + r] = -krM * d1 * d2;
          s.dq[4 * nrpad + r] = -krM * d0 * d2;
          s.dq[5 * nrpad + r] = -krM * (d0 * d1);
        } else {
          s.dq[r] = kfM * c1;
          s.dq[nrpad + r] = kfM * c0;
          s.dq[2 * nrpad + r] = -krM * d1;
          s.dq[3 * nrpad + r] = -krM * d0;
        }
        double dlnk, tb = 0.0;
        if (type >= 2) {
          dlnk = fo[6 * WARP + r - f0] * T;
          tb = fo[7 * WARP + r - f0] * fma(-iKc, Pr, Pf);   // dkeff/dM (Pf - Pr/Kc)
        } else {
          dlnk = fma(gE[r], invT, gb[r]);
          if (type == 1) tb = q;
        }
        double dH = s.hRT[p0] + s.hRT[p1] - s.hRT[r0] - s.hRT[r1] - (double)fix_dn(w);
        if (m.w3) dH += s.hRT[fix_idx(w, 5)] - s.hRT[fix_idx(w, 2)];
        s.dq[2 * ns2 * nrpad + r] = tb;
        // fwd dlnk - rvs (dlnk - dlnKc) = q dlnk + rvs dlnKc
        s.dq[(2 * ns2 + 1) * nrpad + r] = fma(type == 1 ? q * Mfac : q, dlnk, rvs * dH);
      }
      if (type == 1) q *= Mfac;
    }
    s.q[r] = q;
  }
  __syncwarp();
  // ---- species: production rates.  The entries of all species are dealt out
  // evenly over the lanes (19 each at 31 species and 160 reactions, where the
  // longest species list has 34); a lane writes the sum of each piece of a
  // species' list and the species' lane adds the pieces.
  double* part = fo;
  {
    double acc = 0.0;
    for (int e = 0; e < m.seg_len; ++e) {
      const uint32_t w = m.seg[32 * e + lane];
      const double q = s.q[w & 0xffffu], v = m.segv[(w >> 17) & 127u];
      acc = fma(v, __hiloint2double(__double2hiint(q) ^ (int)((w << 15) & 0x80000000u), __double2loint(q)), acc);
      if ((int)w < 0) {
        part[(w >> 24) & 127u] = acc;
        acc = 0.0;
      }
    }
  }
  __syncwarp();
  const double cvone = cv ? 1.0 : 0.0;
  double wm[SPL];
  double Ql = 0.0, Dl = 0.0, cpl = 0.0, hl = 0.0;
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    wm[j] = 0.0;
    if (k < ns) {
      const int e0 = m.piece[k], e1 = m.piece[k + 1];
      if (e0 < e1) wm[j] = part[e0];
      for (int e = e0 + 1; e < e1; ++e) wm[j] += part[e];
      if (RHS || JAC) {
        // constant volume: u_k/RT = h_k/RT - 1, cv_k/R = cp_k/R - 1
        Ql = fma(cv ? my_hRT[j] - 1.0 : my_hRT[j], wm[j], Ql);
        Dl = fma(my_c[j], cv ? my_cpR[j] - 1.0 : my_cpR[j], Dl);
      }
      if (want_h) {
        cpl = fma(yw[j], my_cpR[j], cpl);
        hl = fma(yw[j], my_hRT[j], hl);
      }
    }
    out.wmol[j] = wm[j];
  }
  out.rho = rho;
  if (want_h) {
    out.cp_mass = warp_isum(cpl) * m.r_thermo;
    out.h_mass = warp_isum(hl) * m.r_thermo * T;
  }
  if (!RHS && !JAC) return;
  const double Q = warp_isum(Ql), D = warp_isum(Dl);
  const double invD = recip(D);
  const double fT = -T * Q * invD;
  const double irho = cv ? pr.b : pr.b * X;
  out.fT = fT;
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    out.cpR[j] = my_cpR[j];
    out.f[j] = (k < ns) ? m.mw[k] * wm[j] * irho : (k == ns ? fT : 0.0);
  }
  if (!JAC) return;

  // ---- Jacobian in concentration space: row k = species k ------------------
  // Every entry is a run of terms, the runs dealt out evenly over the lanes (88
  // multiply-adds a lane at 31 species and 160 reactions, where a row per lane
  // took about 380: the longest species list times four, and third-body rows met
  // at different places of different lists).  Column ns collects what a third
  // body adds to every column, row ns T times the derivative by T.
  __syncwarp();   // the pieces lie in the rows
  // SPL 2: the work area lies in global memory and its entries by columns, so that
  // lanes (rows) that go along a row read whole sectors (54 species, 320 reactions,
  // 20,011 cells: 2.30 -> 2.21 ms).  With the derivatives in shared memory instead
  // the L1 left over is too small for the rows: 2.61.
  constexpr bool COL = SPL > 1;
  constexpr int ld = 32 * SPL + 1;
  constexpr int rs = COL ? 1 : ld, cs = COL ? ld : 1;   // strides of a row and of a column
  for (int i = lane; i < (ns + 1) * ld; i += WARP) s.Jr[i] = 0.0;
  __syncwarp();
  {
    double acc = 0.0;
    const uint16_t* target = m.target + lane;
    for (int e = 0; e < m.term_len; ++e) {
      const uint32_t w = m.term[32 * e + lane];
      acc = fma(m.coef[(w >> 16) & 0xfffu], s.dq[w & 0xffffu], acc);
      if ((int)w < 0) {
        const int t = *target;   // row * ld + column
        s.Jr[COL ? t / ld + t % ld * ld : t] = acc;
        target += WARP;
        acc = 0.0;
      }
    }
  }
  __syncwarp();
  // S_k = sum_j c_j Jc[k][j] (row k); HJ_m = sum_k hRT_k Jc[k][m] (column m)
  double Sk[SPL], HJ[SPL], tball[SPL], JT[SPL];
  double HSl = 0.0, dQTl = 0.0, dDTl = 0.0, HTl = 0.0;
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    Sk[j] = 0.0; HJ[j] = 0.0; tball[j] = 0.0; JT[j] = 0.0;
    if (k < ns) {
      const double* Jrow = s.Jr + k * rs;
      tball[j] = Jrow[ns * cs];
      JT[j] = s.Jr[ns * rs + k * cs] * invT;
      const double* a = (const double*)(img + L.o_nasa) + k;
      const double tm = a[14 * nsp];
      a += __double_as_longlong(T) <= __double_as_longlong(tm) ? 0 : 7 * nsp;
      const double dcp = fma(T, fma(T, fma(4.0 * T, a[4 * nsp], 3.0 * a[3 * nsp]), 2.0 * a[2 * nsp]), a[nsp]);
      if (cv) {
        // rho fixed: no dependence of c on T or through rho on Y (Sk = 0)
        for (int kk = 0; kk < ns; ++kk) HJ[j] = fma(s.hRT[kk] - 1.0, s.Jr[kk * rs + k * cs], HJ[j]);
        HTl += (my_hRT[j] - 1.0) * tball[j];
        dQTl += (my_cpR[j] - my_hRT[j]) * invT * wm[j] + (my_hRT[j] - 1.0) * JT[j];
        dDTl += my_c[j] * dcp;
      } else {
        Sk[j] = tball[j] * ctot;
        for (int jj = 0; jj < ns; ++jj) Sk[j] = fma(s.c[jj], Jrow[jj * cs], Sk[j]);
        for (int kk = 0; kk < ns; ++kk) HJ[j] = fma(s.hRT[kk], s.Jr[kk * rs + k * cs], HJ[j]);
        HTl = fma(my_hRT[j], tball[j], HTl);
        HSl = fma(my_hRT[j], Sk[j], HSl);
        dQTl += (my_cpR[j] - my_hRT[j]) * invT * wm[j] + my_hRT[j] * (JT[j] - Sk[j] * invT);
        dDTl += my_c[j] * (dcp - my_cpR[j] * invT);
      }
    }
  }
  const double HS = warp_isum(HSl), HT = warp_isum(HTl);
  const double wbar = recip(sumYW);
  const double wr = cv ? 0.0 : wbar * irho;
  const double dQT = warp_isum(dQTl), dDT = warp_isum(dDTl);
  const double QD = Q * invD, TD = T * invD;
  const double JTT = -QD - TD * (dQT - QD * dDT);
  // the T row by columns, then row by row (lanes = rows) into (Y, T) variables:
  // W_k (Jc + tball - wr t_k) / W_j, t_k = S_k - w_k
  double Wk[SPL], off[SPL], last[SPL];
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    Wk[j] = off[j] = last[j] = 0.0;
    if (k < ns) {
      const double rw = rho * m.invmw[k], ww = cv ? 0.0 : wbar * m.invmw[k];
      const double dQ = rw * (HJ[j] + HT) - ww * HS;
      const double dD = rw * (my_cpR[j] - cvone) - ww * D;
      s.q[k] = -TD * (dQ - QD * dD);
      const double tk = Sk[j] - wm[j];
      Wk[j] = m.mw[k];
      off[j] = Wk[j] * (tball[j] - wr * tk);
      last[j] = (Wk[j] * irho) * (cv ? JT[j] : JT[j] - tk * invT);
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    if (k <= ns) {
      const double* Jrow = s.Jr + k * rs;
#pragma unroll 4
      for (int jj = 0; jj < ns; ++jj) {
        const double v = fma(Wk[j], Jrow[jj * cs], off[j]) * m.invmw[jj];
        dst[(int64_t)jj * dld + k] = k < ns ? v : s.q[jj];
      }
      dst[(int64_t)ns * dld + k] = k < ns ? last[j] : JTT;
    }
  }
  __syncwarp();
}

// The FP64 path of one cell for kernels whose shared memory holds the
// fixed-point image: the mechanism is read from global memory.
template <bool JAC, int SPL>
__device__ __noinline__ void kinetics_general(const uint8_t* __restrict__ img, const ImageLayout& L,
                                              const WarpScratch& s, int lane, const double (&Yk)[SPL], double T,
                                              double pr, CellOutT<SPL>& out, bool cv) {
  MechView g;
  g.bind(L, img);
  warp_kinetics<JAC, SPL>(g, s, lane, Yk, T, pr, out, cv);
}

// The fixed-point path where the cell's temperature allows it.  Returns whether
// the Jacobian was written to dst (else its rows are in s.Jr).
template <bool JAC, int SPL, bool RHS>
__device__ __forceinline__ bool kinetics_cell(const FixView& m, const uint8_t* __restrict__ img, const ImageLayout& L,
                                              const WarpScratch& s, int lane, const double (&Yk)[SPL], double T,
                                              const FixPress& pr, CellOutT<SPL>& out, bool want_h, double* dst = nullptr,
                                              int dld = 0) {
  if (m.covers(T) && (!JAC || m.term_len > 0)) {
    kinetics_fix<JAC, SPL, RHS>(m, img, L, s, lane, Yk, T, pr, out, want_h, dst, dld);
    return true;
  }
  CellOutT<SPL> o;
  double yk[SPL];
#pragma unroll
  for (int j = 0; j < SPL; ++j) yk[j] = Yk[j];
  WarpScratch sc = s;
  kinetics_general<JAC, SPL>(img, L, sc, lane, yk, T, pr.pr, o, pr.cv);
  out = o;
  return false;
}

}  // namespace flint
