// flint_kernels.cu -- batched source-term, Jacobian and thermo kernels.
//
//  k_wdot_small   one thread per cell, for small mechanisms (ns <= 16): the
//                 2-step CH4/air case.  Every thread reads the same reaction
//                 word at the same time (broadcast), per-thread species arrays
//                 live in shared memory as [species][thread] (conflict-free).
//                 k_wdot_small_fix on the fixed-point image, k_wdot_small in
//                 FP64 for a mechanism without one.
//  k_wdot_warp    one warp per cell (ns <= 63, species k on lane k % 32): reaction-parallel rates of
//                 progress, species-parallel sums; optional analytic Jacobian
//                 written coalesced (lane = row, one column per store); FIX: on
//                 the fixed-point image (flint_fixkin.cuh); RHS: the reactor's
//                 right-hand side.  Source terms of large batches go to
//                 flint_cell.cu.
//
// All kernels are grid-stride loops over cells sized to whole waves of the 152
// SMs, so any N (including 0 and ragged tails) is handled without a tail kernel.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <unordered_map>
#include "flint_dev.cuh"
#include "flint_fixkin.cuh"
#include "flint_host.h"

namespace flint {

constexpr int SMALL_NSMAX = 16;
constexpr int SMALL_THREADS = 128;
constexpr int WARP_THREADS = 256;

// ---------------------------------------------------------------- small
// One cell of a small mechanism on the FP64 path, by one thread.  cs, gs, ws:
// the thread's columns of shared memory (stride S).
__device__ inline void small_cell(const MechView& m, int64_t i, int64_t n, int layout, const double* __restrict__ Tg,
                                  const double* __restrict__ pg, const double* __restrict__ Yg,
                                  double* __restrict__ wdot, double* __restrict__ cpo, double* __restrict__ ho,
                                  int roi_mode, double* roi_io, double* cs, double* gs, double* ws, int S) {
  const int ns = m.ns, P = m.nrpad;
#define CS(k) cs[(k) * S]
#define GS(k) gs[(k) * S]
#define WS(k) ws[(k) * S]
  const double T = Tg[i];
  const double lnT = flog(T, m.logtab), invT = 1.0 / T;
  double rho;
  double cpm = 0.0, hm = 0.0, ctot = 0.0;
  if (roi_mode) {
    // chemistry_source(roi, T, omegadot): c = max(roi,0)/W (WD.f90:18-21)
    rho = 0.0;
    for (int k = 0; k < ns; ++k) {
      double r = roi_io[i * ns + k];
      r = r > 0.0 ? r : 0.0;
      roi_io[i * ns + k] = r;
      CS(k) = r * m.invmw[k];
      ctot += CS(k);
    }
  } else {
    double sumYW = 0.0;
    for (int k = 0; k < ns; ++k) {
      double y = (layout == 1) ? Yg[(int64_t)k * n + i] : Yg[i * ns + k];
      CS(k) = y;
      sumYW += y * m.invmw[k];
    }
    rho = pg[i] / (m.r_eos * T * sumYW);
    for (int k = 0; k < ns; ++k) {
      double y = CS(k);
      SpThermo th = nasa7(m, k, T, lnT, invT);
      cpm += y * th.cpR * m.invmw[k];
      hm += y * th.hRT * m.invmw[k];
      CS(k) = rho * y * m.invmw[k];
      ctot += CS(k);
      GS(k) = th.hRT - th.sR;
    }
  }
  if (roi_mode) {
    for (int k = 0; k < ns; ++k) {
      SpThermo th = nasa7(m, k, T, lnT, invT);
      GS(k) = th.hRT - th.sR;
    }
  }
  for (int k = 0; k < ns; ++k) WS(k) = 0.0;
  const double lnC0 = m.lnpref_rth - lnT;
  for (int r = 0; r < m.nr; ++r) {
    const uint32_t w = m.code[r];
    const int type = rx_type(w);
    double kf = m.A[r] * fexp(m.b[r] * lnT - m.E[r] * invT, m.exptab);
    double Pf = 1.0, d;
#pragma unroll
    for (int sl = 0; sl < MAXSIDE; ++sl) {
      int sp = m.rsp[sl * P + r];
      if (sp >= 0) Pf *= powc(CS(sp), rx_ordcode(w, sl), m.rord[sl * P + r], &d, m.exptab, m.logtab);
    }
    double rvsf = 0.0;
    if (rx_rev(w)) {
      double dG = 0.0, Pr = 1.0;
#pragma unroll
      for (int sl = 0; sl < MAXSIDE; ++sl) {
        int sp = m.psp[sl * P + r];
        if (sp >= 0) {
          double nu = m.pnu[sl * P + r];
          dG += nu * GS(sp);
          Pr *= powc(CS(sp), (m.pcode[r] >> (4 * sl)) & 0xf, nu, &d, m.exptab, m.logtab);
        }
        int sq = m.rsp[sl * P + r];
        if (sq >= 0) dG -= m.rnu[sl * P + r] * GS(sq);
      }
      rvsf = fexp(dG - m.dnu[r] * lnC0, m.exptab) * Pr;
    }
    double keff = kf, Mfac = 1.0;
    if (type != 0) {
      const int row = rx_tbrow(w);
      double M = m.tbd[row] * ctot;
      for (int e = m.tbp[row]; e < m.tbp[row + 1]; ++e) M = fma(m.tbv[e], CS(m.tbs[e]), M);
      if (type == 1) Mfac = M;
      else keff = falloff_eval(m, r, type, kf, 0.0, M, T, lnT, invT).keff;
    }
    const double q = Mfac * keff * (Pf - rvsf);
#pragma unroll
    for (int sl = 0; sl < MAXSIDE; ++sl) {
      int sp = m.rsp[sl * P + r];
      if (sp >= 0) WS(sp) -= m.rnu[sl * P + r] * q;
      int sq = m.psp[sl * P + r];
      if (sq >= 0) WS(sq) += m.pnu[sl * P + r] * q;
    }
  }
  if (wdot) {
    for (int k = 0; k < ns; ++k) {
      double v = m.mw[k] * WS(k);
      if (roi_mode || layout == 0) wdot[i * ns + k] = v;
      else wdot[(int64_t)k * n + i] = v;
    }
  }
  (void)rho;
  if (cpo) cpo[i] = cpm * m.r_thermo;
  if (ho) ho[i] = hm * m.r_thermo * T;
#undef CS
#undef GS
#undef WS
}

__global__ void __launch_bounds__(SMALL_THREADS)
k_wdot_small(const uint8_t* __restrict__ img, ImageLayout L, int64_t n, int layout,
             const double* __restrict__ Tg, const double* __restrict__ pg,
             const double* __restrict__ Yg, double* __restrict__ wdot,
             double* __restrict__ cpo, double* __restrict__ ho, int roi_mode, double* roi_io) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img, L.bytes);
  MechView m;
  m.bind(L, smem);
  double* cs = reinterpret_cast<double*>(smem + L.bytes) + threadIdx.x;      // [NSMAX][threads]
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    small_cell(m, i, n, layout, Tg, pg, Yg, wdot, cpo, ho, roi_mode, roi_io, cs, cs + SMALL_NSMAX * SMALL_THREADS,
               cs + 2 * SMALL_NSMAX * SMALL_THREADS, SMALL_THREADS);
}

__device__ __noinline__ void small_cell_general(const uint8_t* __restrict__ img, const ImageLayout& L, int64_t i,
                                                int64_t n, int layout, const double* __restrict__ Tg,
                                                const double* __restrict__ pg, const double* __restrict__ Yg,
                                                double* __restrict__ wdot, double* __restrict__ cpo,
                                                double* __restrict__ ho, int roi_mode, double* roi_io, double* cs, int S) {
  MechView m;
  m.bind(L, img);
  small_cell(m, i, n, layout, Tg, pg, Yg, wdot, cpo, ho, roi_mode, roi_io, cs, cs + L.ns * S, cs + 2 * L.ns * S, S);
}

// The same on the fixed-point image (flint_fix.cuh).  A rate with other than
// integer orders is one exponential of log2 k + sum of order x log2 c, so the
// 2-step CH4/air source term leaves about 60 operations of a thread on the FP64
// pipe (concentrations, sums, cp and h) where it took about 300, half of them
// logarithms and exponentials.  The mechanism's few words are read through the
// read-only cache: staging them cost a block more than they are worth.  A thread
// whose temperature leaves the formats, or a concentration in power form the normal
// range (subnormal, inf or NaN), takes the FP64 path.
__global__ void __launch_bounds__(SMALL_THREADS)
k_wdot_small_fix(const uint8_t* __restrict__ img, const __grid_constant__ ImageLayout L, int64_t n, int layout,
                 const double* __restrict__ Tg, const double* __restrict__ pg, const double* __restrict__ Yg,
                 double* __restrict__ wdot, double* __restrict__ cpo, double* __restrict__ ho, int roi_mode,
                 double* roi_io) {
  extern __shared__ __align__(16) uint8_t smem[];
  FixView m;
  m.bind(L, img + L.o_fix);
  const int ns = m.ns, nsp = m.nsp, S = blockDim.x, P = m.nrpad, f0 = m.nr - m.nfall;
  double* cs = reinterpret_cast<double*>(smem) + threadIdx.x;      // c, G, w, log2 c: [ns][threads] each
  int64_t* gs = reinterpret_cast<int64_t*>(cs + ns * S);
  double* ws = cs + 2 * ns * S;
  uint64_t* ls = reinterpret_cast<uint64_t*>(cs + 3 * ns * S);
  const bool thermo = cpo || ho;
  for (int64_t i = (int64_t)blockIdx.x * S + threadIdx.x; i < n; i += (int64_t)gridDim.x * S) {
    const double T = Tg[i];
    bool in = m.covers(T);
    const FixT f = fix_T(in ? T : 1000.0, m.lt);
    double cpm = 0.0, hm = 0.0, ctot = 0.0;
    if (roi_mode) {
      // chemistry_source(roi, T, omegadot): c = max(roi,0)/W (WD.f90:18-21)
      for (int k = 0; k < ns; ++k) {
        double r = roi_io[i * ns + k];
        r = r > 0.0 ? r : 0.0;
        roi_io[i * ns + k] = r;
        cs[k * S] = r * m.invmw[k];
      }
    } else {
      double sumYW = 0.0;
      for (int k = 0; k < ns; ++k) {
        const double yw = (layout == 1 ? Yg[(int64_t)k * n + i] : Yg[i * ns + k]) * m.invmw[k];
        cs[k * S] = yw;
        sumYW += yw;
      }
      const double rho = pg[i] * m.inv_r_eos * recip(T * sumYW);
      for (int k = 0; k < ns; ++k) {
        const double yw = cs[k * S];
        if (thermo) {
          const bool lo = __double_as_longlong(T) <= m.tmid[k];
          const uint64_t t = lo ? f.t11 : f.t13;
          cpm = fma(yw, fix2d(fix_poly5(m.c + (lo ? 0 : 5 * nsp) + k, nsp, t), 52), cpm);
          hm = fma(yw, fix2d(fix_enthalpy(m.h + (lo ? 0 : 6 * nsp) + k, nsp, t, f), 52), hm);
        }
        cs[k * S] = rho * yw;
      }
    }
    if (m.ntb)
      for (int k = 0; k < ns; ++k) ctot += cs[k * S];
    if (L.fix_rev)
      for (int k = 0; k < ns; ++k) {
        const bool lo = __double_as_longlong(T) <= m.tmid[k];
        gs[k * S] = fix_gibbs(m.g + (lo ? 0 : 7 * nsp) + k, nsp, lo ? f.t11 : f.t13, f);
      }
    for (int k = 0; k < ns; ++k) {
      ws[k * S] = 0.0;
      ls[k * S] = 0;       // log2 c not formed yet
    }
    const int64_t lC0 = m.lC - (int64_t)(f.L >> 9);
    for (int r = 0; r < m.nr; ++r) {
      const uint64_t w = m.ix[r];
      const int type = fix_type(w);
      int64_t a = fix_arrhenius(m.a[r], m.b[r], m.e[r], f);
      double Pf = 1.0;
      bool none = false;
      int minus = 0;             // last bit: the factors' sign
      if (fix_power(w)) {
        // the sum modulo 2^64 and, against leaving the format, in Q32
        int64_t wide = a >> 20;
#pragma unroll
        for (int sl = 0; sl < 3; ++sl) {
          const int s = fix_idx(w, sl);
          if (s >= ns) continue;
          const double c = cs[s * S];
          uint64_t l = ls[s * S];
          if (l == 0) {
            // log2 |c| with its sign flipped: Q57 (last bit 0) from 2^-63 to 2^63, Q53
            // (last bit 1) beyond; 1 where c = 0
            const unsigned e = (unsigned)(__double2hiint(c) >> 20) & 0x7ffu;
            l = 1;
            if (e - 1u < 0x7feu) {
              int ex;
              const int64_t fr = log2_q62(fabs(c), m.lt, &ex);
              l = e - 960u < 126u ? (((uint64_t)(int64_t)ex << 57) + ((uint64_t)fr >> 6 << 1)) ^ 0x8000000000000000ull
                                  : ((((uint64_t)(int64_t)ex << 53) + ((uint64_t)fr >> 9)) ^ 0x8000000000000000ull) | 1u;
            } else if ((__double_as_longlong(c) << 1) != 0) {
              in = false;
            }
            ls[s * S] = l;
          }
          const uint64_t o = m.ord[sl * P + r];
          // a negative c to an order of 1, 2 or 3 has a sign, to any other it is absent
          none |= l == 1;
          if (__double2hiint(c) < 0) {
            none |= (o << 4) != 0 || o >> 60 > 3;
            minus ^= (int)(o >> 60);
          }
          const int64_t x = (int64_t)(mulhi_u(o, l) - (o >> 1));      // Q60 x Q57 -> Q53, x Q53 -> Q49
          a += l & 1 ? (int64_t)((uint64_t)x << 3) : x >> 1;
          wide += l & 1 ? x >> 17 : x >> 21;
        }
        if (wide >= 2040ll << 32) a = 2040ll << 52;
        if (wide <= -(2040ll << 32)) a = -(2040ll << 52);
      } else {
#pragma unroll
        for (int sl = 0; sl < 3; ++sl) {
          const int s = fix_idx(w, sl);
          if (s < ns) Pf *= cs[s * S];
        }
      }
      double M = 1.0;
      if (type != 0) {
        const int row = fix_tbrow(w);
        M = m.tbd[row] * ctot;
        for (int e = m.tbp[row]; e < m.tbp[row + 1]; ++e) M = fma(m.tbv[e], cs[m.tbs[e] * S], M);
      }
      double kf;
      if (none) kf = 0.0;      // (of any type: the absent factor is not in the exponent)
      else if (type < 2) kf = exp2_q52<true>(a, m.et);
      else kf = cell_falloff<true>(m, r - f0, type, a, M, f, T, fix2d((int64_t)f.v, 70));
      const int sgn = (((int)(w >> 43) ^ minus) & 1) << 31;
      kf = __hiloint2double(__double2hiint(kf) ^ sgn, __double2loint(kf));
      double q = kf * Pf;
      if (fix_rev(w)) {
        int64_t ar = (type < 2 ? a : 0) - (int64_t)fix_dn(w) * lC0;
        double Pr = 1.0;
#pragma unroll
        for (int sl = 0; sl < 3; ++sl) {
          const int s = fix_idx(w, sl), p = fix_idx(w, 3 + sl);
          if (s < ns) ar -= gs[s * S];
          if (p < ns) { ar += gs[p * S]; Pr *= cs[p * S]; }
        }
        double kr = exp2_q52(ar, m.et);
        if (type < 2) kr = __hiloint2double(__double2hiint(kr) ^ sgn, __double2loint(kr));
        else kr *= kf;
        q = fma(-kr, Pr, q);
      }
      if (type == 1) q *= M;
      for (int e = m.rs[r]; e < m.rs[r + 1]; ++e) {
        const int word = m.rw[e], code = word >> 8;
        double* wk = ws + (word & 0xff) * S;
        *wk = fma(code == 1 ? 1.0 : (code == -1 ? -1.0 : m.rv[code - 2]), q, *wk);
      }
    }
    if (!in) {
      small_cell_general(img, L, i, n, layout, Tg, pg, Yg, wdot, cpo, ho, roi_mode, roi_io, cs, S);
      continue;
    }
    if (wdot)
      for (int k = 0; k < ns; ++k) {
        const double v = m.mw[k] * ws[k * S];
        if (roi_mode || layout == 0) wdot[i * ns + k] = v;
        else wdot[(int64_t)k * n + i] = v;
      }
    if (cpo) cpo[i] = cpm * m.r_thermo;
    if (ho) ho[i] = hm * m.r_thermo * T;
  }
}

// ---------------------------------------------------------------- warp
// SPL species per lane; GJ: the Jacobian work area is a per-warp slot of
// global memory (mechanisms of 32-63 species, and smaller ones whose shared
// memory layout would not fit a block).  FIX: the fixed-point kinetics
// (flint_fixkin.cuh); the block then stages only that image.  RHS: rhs_out is
// wanted.
template <bool JAC, int SPL, bool GJ, bool FIX, bool RHS>
__global__ void __launch_bounds__(WARP_THREADS, JAC ? 1 : 2)
k_wdot_warp(const uint8_t* __restrict__ img, const __grid_constant__ ImageLayout L, int64_t n, int layout,
            const double* __restrict__ Tg, const double* __restrict__ pg,
            const double* __restrict__ Yg, double* __restrict__ wdot, double* __restrict__ cpo,
            double* __restrict__ ho, double* __restrict__ jac, double* __restrict__ rhs_out,
            double* __restrict__ gscratch, int cv) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int base = FIX ? (JAC ? L.fix_bytes : L.fix_bytes_rate) : L.bytes;
  stage_image(smem, FIX ? img + L.o_fix : img, base);
  MechView m;
  FixView x;
  if (FIX) x.bind(L, smem);
  else m.bind(L, smem);
  const double* mw = FIX ? x.mw : m.mw;
  const int nsp = L.nsp, nrpad = L.nrpad;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  WarpScratch s;
  if (!GJ) {
    const int sd = scratch_doubles(L, JAC);
    s = carve<FIX>(reinterpret_cast<double*>(smem + base) + wid * sd, L, JAC);
  } else {
    const int sd = scratch_small_doubles(L);
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + wid;
    s = carve2<FIX>(reinterpret_cast<double*>(smem + base) + wid * sd,
               JAC ? gscratch + gw * scratch_jac_doubles(L) : nullptr, L);
  }
  const int ns = L.ns, nv = ns + 1;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t cell = (int64_t)blockIdx.x * (blockDim.x >> 5) + wid; cell < n; cell += nwarps) {
    const double T = Tg[cell], p = pg[cell];
    double Yk[SPL];
#pragma unroll
    for (int j = 0; j < SPL; ++j) {
      const int k = lane + 32 * j;
      Yk[j] = 0.0;
      if (k < ns) Yk[j] = (layout == 1) ? Yg[(int64_t)k * n + cell] : Yg[cell * ns + k];
    }
    CellOutT<SPL> o;
    // Fortran (nv, nv, N): column c of this cell is contiguous; lanes = rows.
    double* dst = JAC ? jac + cell * (int64_t)nv * nv : nullptr;
    bool stored = false;
    if (FIX)
      stored = kinetics_cell<JAC, SPL, RHS>(x, img, L, s, lane, Yk, T, FixPress::of<JAC || RHS>(x, p, cv != 0), o,
                                            cpo != nullptr || ho != nullptr, dst, nv);
    else
      warp_kinetics<JAC, SPL>(m, s, lane, Yk, T, p, o, cv != 0);
#pragma unroll
    for (int j = 0; j < SPL; ++j) {
      const int k = lane + 32 * j;
      if (wdot && k < ns) {
        const double v = mw[k] * o.wmol[j];
        if (layout == 1) wdot[(int64_t)k * n + cell] = v;
        else wdot[cell * ns + k] = v;
      }
      if (RHS && k < nv) rhs_out[cell * nv + k] = o.f[j];
    }
    if (lane == 0) {
      if (cpo) cpo[cell] = o.cp_mass;
      if (ho) ho[cell] = o.h_mass;
    }
    if (JAC && !stored) {
#pragma unroll
      for (int j = 0; j < SPL; ++j) {
        const int r = lane + 32 * j;
        if (r < nv)
          for (int c = 0; c < nv; ++c) dst[(int64_t)c * nv + r] = s.Jr[r * s.ldj + c];
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------- thermo
// Mixture cp [J/kg/K] and h [J/kg] of N cells, one thread per cell
// (f_cp / H of Lib_ThermoTransport.f90:251-271, :40-52 on NASA-7 data).
__global__ void __launch_bounds__(SMALL_THREADS)
k_thermo(const uint8_t* __restrict__ img, ImageLayout L, int64_t n, int layout, const double* __restrict__ Tg,
         const double* __restrict__ Yg, double* __restrict__ cpo, double* __restrict__ ho) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img, L.bytes);
  MechView m;
  m.bind(L, smem);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double T = Tg[i], lnT = log(T), invT = 1.0 / T;
    double cpm = 0.0, hm = 0.0;
    for (int k = 0; k < m.ns; ++k) {
      const double y = (layout == 1) ? Yg[(int64_t)k * n + i] : Yg[i * m.ns + k];
      SpThermo th = nasa7(m, k, T, lnT, invT);
      cpm += y * th.cpR * m.invmw[k];
      hm += y * th.hRT * m.invmw[k];
    }
    if (cpo) cpo[i] = cpm * m.r_thermo;
    if (ho) ho[i] = hm * m.r_thermo * T;
  }
}

// ---------------------------------------------------------------- species thermo
// Species cp, h, s (at p_ref) and g = h - T s in mass units for N
// temperatures (cpi, H0i, S0i of Lib_ThermoTransport.f90:40-97, :233-248, from
// the polynomials): one thread per (cell, species), outputs cell-major (N, ns).
__global__ void k_species_thermo(const uint8_t* __restrict__ img, ImageLayout L, int64_t n,
                                 const double* __restrict__ Tg, double* __restrict__ cpo,
                                 double* __restrict__ ho, double* __restrict__ so, double* __restrict__ go) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img, L.bytes);
  MechView m;
  m.bind(L, smem);
  const int ns = m.ns;
  const int64_t total = n * ns;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t cell = i / ns;
    const int k = (int)(i - cell * ns);
    const double T = Tg[cell], lnT = log(T), invT = 1.0 / T;
    const SpThermo th = nasa7(m, k, T, lnT, invT);
    const double rw = m.r_thermo * m.invmw[k];
    if (cpo) cpo[i] = th.cpR * rw;
    if (ho) ho[i] = th.hRT * rw * T;
    if (so) so[i] = th.sR * rw;
    if (go) go[i] = (th.hRT - th.sR) * rw * T;
  }
}

// ---------------------------------------------------------------- exp self-test
__global__ void k_exp_selftest(const uint8_t* __restrict__ img, ImageLayout L, int64_t n,
                               const double* __restrict__ x, double* __restrict__ y) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img, L.bytes);
  MechView m;
  m.bind(L, smem);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    y[2 * i] = fexp(x[i], m.exptab);
    y[2 * i + 1] = exp(x[i]);
  }
}

cudaError_t launch_exp_selftest(const uint8_t* img, const ImageLayout& L, int64_t n, const double* x, double* y,
                                cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  cudaError_t e = set_smem((const void*)k_exp_selftest, L.bytes);
  if (e != cudaSuccess) return e;
  k_exp_selftest<<<256, 256, L.bytes, st>>>(img, L, n, x, y);
  count_launch();
  return cudaGetLastError();
}

__global__ void k_log_selftest(const uint8_t* __restrict__ img, ImageLayout L, int64_t n,
                               const double* __restrict__ x, double* __restrict__ y) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img, L.bytes);
  MechView m;
  m.bind(L, smem);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    y[2 * i] = flog(x[i], m.logtab);
    y[2 * i + 1] = log(x[i]);
  }
}

cudaError_t launch_log_selftest(const uint8_t* img, const ImageLayout& L, int64_t n, const double* x, double* y,
                                cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  cudaError_t e = set_smem((const void*)k_log_selftest, L.bytes);
  if (e != cudaSuccess) return e;
  k_log_selftest<<<256, 256, L.bytes, st>>>(img, L, n, x, y);
  count_launch();
  return cudaGetLastError();
}

__global__ void k_recip_selftest(int64_t n, const double* __restrict__ x, double* __restrict__ y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    y[4 * i] = recip(x[i]);
    y[4 * i + 1] = 1.0 / x[i];
    y[4 * i + 2] = sqrt_fast(x[i]);
    y[4 * i + 3] = sqrt(x[i]);
  }
}

cudaError_t launch_recip_selftest(int64_t n, const double* x, double* y, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_recip_selftest<<<256, 256, 0, st>>>(n, x, y);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------- FP64 probe
// Independent FMA chains: the FP64 pipe's throughput, the denominator of the
// FP64 roofline the benchmarks report.
__global__ void k_dfma_probe(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-3, x1 = x0 + 1.0, x2 = x0 + 2.0, x3 = x0 + 3.0;
  double x4 = x0 + 4.0, x5 = x0 + 5.0, x6 = x0 + 6.0, x7 = x0 + 7.0;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  out[(int64_t)blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}

cudaError_t probe_fp64(double* tflops) {
  const int blocks = device_sms() * 8, threads = 256, iters = 2048;
  double* buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, (size_t)blocks * threads * sizeof(double));
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_dfma_probe<<<blocks, threads>>>(buf, 64, 0.999, 1e-3);
  float best = 1e30f;
  for (int rep = 0; rep < 3; ++rep) {
    cudaEventRecord(e0);
    k_dfma_probe<<<blocks, threads>>>(buf, iters, 0.999, 1e-3);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) best = ms;
  }
  count_launch();
  e = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(buf);
  *tflops = 2.0 * 8.0 * iters * (double)blocks * threads / (best * 1e-3) / 1e12;
  return e;
}

// ---------------------------------------------------------------- launchers
// Device properties, cached per device (the current device of the calling
// thread); the cache entries are atomics, so concurrent first calls are safe.
constexpr int MAX_DEV_CACHE = 64;
static std::atomic<int> g_sms[MAX_DEV_CACHE];
static std::atomic<int> g_optin[MAX_DEV_CACHE];

static int cached_attr(std::atomic<int>* cache, cudaDeviceAttr attr, int fallback) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV_CACHE) dev = 0;
  int v = cache[dev].load(std::memory_order_relaxed);
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess || v <= 0) {
      (void)cudaGetLastError();
      v = fallback;
    }
    cache[dev].store(v, std::memory_order_relaxed);
  }
  return v;
}

int device_sms() { return cached_attr(g_sms, cudaDevAttrMultiProcessorCount, 1); }

size_t device_smem_optin() {
  return (size_t)cached_attr(g_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, 48 * 1024);
}

namespace {
struct LaunchKey {
  const void* fn;
  size_t smem;
  int threads, dev;
  bool operator==(const LaunchKey& o) const {
    return fn == o.fn && smem == o.smem && threads == o.threads && dev == o.dev;
  }
};
struct LaunchKeyHash {
  size_t operator()(const LaunchKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.fn);
    h = h * 0x9E3779B97F4A7C15ull + k.smem;
    return (h * 0x9E3779B97F4A7C15ull + (size_t)k.threads) * 0x9E3779B97F4A7C15ull + (size_t)k.dev;
  }
};
// one entry per kernel, launch shape and device: a few dozen in all
std::mutex g_launch_mu;
std::unordered_map<LaunchKey, int, LaunchKeyHash> g_resident;
std::unordered_map<LaunchKey, size_t, LaunchKeyHash> g_opted;   // threads = 0, smem = 0 in the key
}  // namespace

cudaError_t set_smem(const void* fn, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const LaunchKey key{fn, 0, 0, dev};
  std::lock_guard<std::mutex> lk(g_launch_mu);
  auto it = g_opted.find(key);
  if (it != g_opted.end() && it->second >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) (void)cudaGetLastError();
  else g_opted[key] = bytes;
  return e;
}

int resident_blocks(const void* fn, int threads, size_t smem) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const LaunchKey key{fn, smem, threads, dev};
  std::lock_guard<std::mutex> lk(g_launch_mu);
  auto it = g_resident.find(key);
  if (it != g_resident.end()) return it->second;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  if (per_sm > 0) g_resident[key] = per_sm;
  return per_sm;
}

static int64_t grid_for(const void* fn, int threads, size_t smem, int64_t work_items) {
  int per_sm = resident_blocks(fn, threads, smem);
  if (per_sm < 1) per_sm = 1;
  int64_t full = (int64_t)device_sms() * per_sm;
  int64_t need = (work_items + threads - 1) / threads;
  if (need < 1) need = 1;
  return need < full ? need : full;
}

size_t small_smem(const ImageLayout& L) { return L.bytes + 3 * SMALL_NSMAX * SMALL_THREADS * sizeof(double); }
// Whether a launch of the warp kernels takes the fixed-point form.  A Jacobian takes
// it where the mechanism's term lists were packed and the image with them leaves a
// block of 256 threads room, or where the FP64 image does not either: the lists grow
// with reactions x species x third-body efficiencies (255 three-body reactions of 20
// efficiencies each: 233 KB, the FP64 image 139).
static bool use_fix(const ImageLayout& L, bool jac) {
  if (!L.fix || !jac) return L.fix;
  const size_t warps = (WARP_THREADS / 32) * scratch_small_doubles(L) * sizeof(double);
  const bool fp64_fits = L.bytes + warps <= device_smem_optin();
  return !fp64_fits || (L.term_len > 0 && L.fix_bytes + warps <= device_smem_optin());
}
// The image a block of the warp kernels stages.
static size_t image_bytes(const ImageLayout& L, bool jac) {
  return use_fix(L, jac) ? (jac ? L.fix_bytes : L.fix_bytes_rate) : L.bytes;
}
// Jacobian work area in global memory: 32-63 species, or a shared-memory
// layout too large for a block of 256 threads (the choice does not depend on
// the block size a caller tunes, so one kernel serves every block size).
static bool warp_gj(const ImageLayout& L, bool jac) {
  if (L.nsp > 32) return true;
  if (!jac) return false;
  return image_bytes(L, true) + (WARP_THREADS / 32) * scratch_doubles(L, true) * sizeof(double) >
         device_smem_optin();
}

static int warp_block(int threads) { return threads == 64 || threads == 128 ? threads : WARP_THREADS; }

size_t warp_smem(const ImageLayout& L, bool jac, int threads) {
  const int wpb = warp_block(threads) / 32;
  if (warp_gj(L, jac)) return image_bytes(L, jac) + wpb * scratch_small_doubles(L) * sizeof(double);
  return image_bytes(L, jac) + wpb * scratch_doubles(L, jac) * sizeof(double);
}

int warp_block_candidates(int* out) {
  out[0] = 64; out[1] = 128; out[2] = WARP_THREADS;
  return 3;
}

typedef void (*WarpKernel)(const uint8_t*, ImageLayout, int64_t, int, const double*, const double*, const double*,
                           double*, double*, double*, double*, double*, double*, int);

template <bool JAC, bool RHS>
static WarpKernel warp_fn(const ImageLayout& L) {
  const bool fix = use_fix(L, JAC);
  if (L.nsp > 32) return fix ? k_wdot_warp<JAC, 2, true, true, RHS> : k_wdot_warp<JAC, 2, true, false, RHS>;
  if (JAC && warp_gj(L, JAC)) return fix ? k_wdot_warp<JAC, 1, true, true, RHS> : k_wdot_warp<JAC, 1, true, false, RHS>;
  return fix ? k_wdot_warp<JAC, 1, false, true, RHS> : k_wdot_warp<JAC, 1, false, false, RHS>;
}

// Global Jacobian work area needed by the warp kernels (doubles), for a grid
// of full waves; 0 when it lives in shared memory.
// (enough for the resident warps of every block size)
int64_t warp_jac_scratch_doubles(const ImageLayout& L) {
  if (!warp_gj(L, true)) return 0;
  const void* fn = (const void*)warp_fn<true, false>(L);
  int64_t most = 0;
  int cand[4];
  const int nc = warp_block_candidates(cand);
  for (int c = 0; c < nc; ++c) {
    const size_t sm = warp_smem(L, true, cand[c]);
    if (set_smem(fn, sm) != cudaSuccess) return 0;
    int per_sm = resident_blocks(fn, cand[c], sm);
    if (per_sm < 1) per_sm = 1;
    most = std::max(most, (int64_t)per_sm * device_sms() * (cand[c] / 32));
  }
  return most * scratch_jac_doubles(L);
}

template <bool JAC, bool RHS>
static cudaError_t launch_warp(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                               const double* p, const double* Y, double* wdot, double* cp, double* h, double* jac,
                               double* rhs, double* gscratch, cudaStream_t st, int cv = 0, int threads = 0) {
  const int bt = warp_block(threads);
  size_t sm = warp_smem(L, JAC, bt);
  const WarpKernel fn = warp_fn<JAC, RHS>(L);
  cudaError_t e = set_smem((const void*)fn, sm);
  if (e != cudaSuccess) return e;
  const bool gj = warp_gj(L, JAC);
  if (gj && JAC && !gscratch) return cudaErrorInvalidValue;
  int64_t g = grid_for((const void*)fn, bt, sm, n * 32);
  fn<<<(unsigned)g, bt, sm, st>>>(img, L, n, layout, T, p, Y, wdot, cp, h, jac, rhs, gj ? gscratch : nullptr, cv);
  count_launch();
  return cudaGetLastError();
}

// Thread per cell, small mechanisms.  Fixed point: blocks small enough that a
// small batch reaches every SM.
static cudaError_t launch_small(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                                const double* p, const double* Y, double* wdot, double* cp, double* h, int roi_mode,
                                double* roi, cudaStream_t st) {
  if (L.sfix) {
    const int64_t per_sm = (n + device_sms() - 1) / device_sms();
    const int bt = per_sm <= 32 ? 32 : (per_sm <= 64 ? 64 : SMALL_THREADS);
    const size_t sm = (size_t)4 * L.ns * bt * sizeof(double);
    cudaError_t e = set_smem((const void*)k_wdot_small_fix, (size_t)4 * L.ns * SMALL_THREADS * sizeof(double));
    if (e != cudaSuccess) return e;
    const int64_t g = grid_for((const void*)k_wdot_small_fix, bt, sm, n);
    k_wdot_small_fix<<<(unsigned)g, bt, sm, st>>>(img, L, n, layout, T, p, Y, wdot, cp, h, roi_mode, roi);
  } else {
    const size_t sm = small_smem(L);
    set_smem((const void*)k_wdot_small, sm);
    const int64_t g = grid_for((const void*)k_wdot_small, SMALL_THREADS, sm, n);
    k_wdot_small<<<(unsigned)g, SMALL_THREADS, sm, st>>>(img, L, n, layout, T, p, Y, wdot, cp, h, roi_mode, roi);
  }
  count_launch();
  return cudaGetLastError();
}

bool use_small_kernel(const ImageLayout& L) { return L.ns <= SMALL_NSMAX && L.ns <= 8; }

int wdot_kernel(const ImageLayout& L, int64_t n) {
  return use_small_kernel(L) ? FLINT_WDOT_SMALL : use_cell_kernel(L, n) ? FLINT_WDOT_CELL : FLINT_WDOT_WARP;
}

cudaError_t launch_wdot(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                        const double* p, const double* Y, double* wdot, double* cp, double* h,
                        cudaStream_t st, int threads) {
  if (n <= 0) return cudaSuccess;
  const int kernel = wdot_kernel(L, n);
  if (kernel == FLINT_WDOT_SMALL) return launch_small(img, L, n, layout, T, p, Y, wdot, cp, h, 0, nullptr, st);
  if (kernel == FLINT_WDOT_CELL) return launch_wdot_cell(img, L, n, layout, T, p, Y, wdot, cp, h, false, 0, st);
  return launch_warp<false, false>(img, L, n, layout, T, p, Y, wdot, cp, h, nullptr, nullptr, nullptr, st, 0, threads);
}

cudaError_t launch_thermo(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                          const double* Y, double* cp, double* h, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  size_t sm = L.bytes;
  set_smem((const void*)k_thermo, sm);
  int64_t g = grid_for((const void*)k_thermo, SMALL_THREADS, sm, n);
  k_thermo<<<(unsigned)g, SMALL_THREADS, sm, st>>>(img, L, n, layout, T, Y, cp, h);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_species_thermo(const uint8_t* img, const ImageLayout& L, int64_t n, const double* T, double* cp,
                                  double* h, double* s, double* g, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  size_t sm = L.bytes;
  set_smem((const void*)k_species_thermo, sm);
  const int64_t blocks = grid_for((const void*)k_species_thermo, SMALL_THREADS, sm, n * L.ns);
  k_species_thermo<<<(unsigned)blocks, SMALL_THREADS, sm, st>>>(img, L, n, T, cp, h, s, g);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_chemistry_source(const uint8_t* img, const ImageLayout& L, int64_t n, double* roi,
                                    const double* T, double* omegadot, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  return launch_small(img, L, n, 0, T, nullptr, nullptr, omegadot, nullptr, nullptr, 1, roi, st);
}

cudaError_t launch_wdot_jac(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                            const double* p, const double* Y, double* wdot, double* jac, double* gscratch,
                            cudaStream_t st, int cv, int threads) {
  if (n <= 0) return cudaSuccess;
  return launch_warp<true, false>(img, L, n, layout, T, p, Y, wdot, nullptr, nullptr, jac, nullptr, gscratch, st, cv,
                                  threads);
}

cudaError_t launch_rhs(const uint8_t* img, const ImageLayout& L, int64_t n, const double* T, const double* p,
                       const double* Y, double* f, cudaStream_t st, int cv) {
  if (n <= 0) return cudaSuccess;
  if (use_cell_kernel(L, n)) return launch_wdot_cell(img, L, n, 0, T, p, Y, f, nullptr, nullptr, true, cv, st);
  return launch_warp<false, true>(img, L, n, 0, T, p, Y, nullptr, nullptr, nullptr, nullptr, f, nullptr, st, cv);
}

}  // namespace flint
