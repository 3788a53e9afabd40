// flint_cell.cu -- source terms, one thread per cell, on the fixed-point image.
//
// For batches that fill the GPU the warp-per-cell kernel wastes FP64 slots:
// per-cell scalars are computed by all 32 lanes, falloff reactions occupy a few
// lanes of a round and the species sums run to the longest list.  Here a thread
// owns a cell and every lane of an FP64 instruction does needed work: 4 products
// and 4 multiply-adds per reversible reaction.  31 species, 160 reactions: 53
// FP64 warp instructions per cell (ncu) where the warp kernel takes 132; 1 M cells
// with cp and h 4.6 ms against 6.1, 66 % of the FP64 pipe.  Of that the 142
// plain reactions are 2.2 ms (86 % of the pipe), the 18 third-body and falloff
// ones 1.1, cp and h 0.4 and loads, concentrations and Gibbs exponents 0.9.
//
// Memory: a warp keeps the concentration, the Gibbs exponent and the production
// sum of every species of its 32 cells in shared memory, one row per species
// (CELL_ROW doubles), so that a lane's own values are conflict-free and a
// row-contiguous transfer to or from global memory (cell-major arrays) is too.
// 8 warps per SM at 31 species; the reactions' data are broadcast reads.  Two plain
// reactions are evaluated side by side, for want of warps to hide the integer chains
// behind.
//
// A cell whose temperature the fixed-point path does not cover is evaluated by
// its warp afterwards, on the FP64 path, with the warp's columns as scratch.
#include <algorithm>
#include "flint_fixkin.cuh"
#include "flint_host.h"

namespace flint {

constexpr int CELL_MAX_WARPS = 8;

// doubles of shared memory per warp: ns + 1 rows (the last for absent factors);
// the FP64 path's scratch aliases them
static __host__ __device__ int cell_warp_doubles(int ns) { return (ns + 1) * CELL_ROW; }

// A multiplier the compiler does not know: fma(one, q, w) stays a DFMA (16.2
// cycles per SM and warp), where w + q would be a DADD (19.1).
__device__ __forceinline__ double opaque(double x) {
  asm("" : "+d"(x));
  return x;
}

// One cell of the batch on the FP64 path, by the whole warp; scratch: the warp's
// columns.
template <bool RHS, int SPL>
__device__ __noinline__ void cell_general(const uint8_t* __restrict__ img, const ImageLayout& L, double* scratch,
                                          int lane, int64_t n, int layout, int64_t cell, const double* __restrict__ Tg,
                                          const double* __restrict__ pg, const double* __restrict__ Yg,
                                          double* __restrict__ out, double* __restrict__ cpo, double* __restrict__ ho,
                                          int cv) {
  const int ns = L.ns, nv = ns + 1;
  const double* mw = reinterpret_cast<const double*>(img + L.o_mw);
  const WarpScratch s = carve2<true>(scratch, nullptr, L);
  double Yk[SPL];
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    Yk[j] = k < ns ? (layout == 1 ? Yg[(int64_t)k * n + cell] : Yg[cell * ns + k]) : 0.0;
  }
  CellOutT<SPL> o;
  kinetics_general<false, SPL>(img, L, s, lane, Yk, Tg[cell], pg[cell], o, cv != 0);
#pragma unroll
  for (int j = 0; j < SPL; ++j) {
    const int k = lane + 32 * j;
    if (RHS) {
      if (k < nv) out[cell * nv + k] = o.f[j];
    } else if (k < ns) {
      out[layout == 1 ? (int64_t)k * n + cell : cell * ns + k] = mw[k] * o.wmol[j];
    }
  }
  if (lane == 0) {
    if (cpo) cpo[cell] = o.cp_mass;
    if (ho) ho[cell] = o.h_mass;
  }
}

// RHS: out is f (n, ns + 1) = (dY/dt, dT/dt), else the production rates;
// THERMO: the mixture cp and h are wanted.
template <bool RHS, bool THERMO>
__global__ void __launch_bounds__(32 * CELL_MAX_WARPS)
k_wdot_cell(const uint8_t* __restrict__ img, const __grid_constant__ ImageLayout L, int64_t n, int layout,
            const double* __restrict__ Tg, const double* __restrict__ pg, const double* __restrict__ Yg,
            double* __restrict__ out, double* __restrict__ cpo, double* __restrict__ ho, int cv, int staged) {
  extern __shared__ __align__(16) uint8_t smem[];
  stage_image(smem, img + L.o_fix, staged);
  FixView m;
  m.bind(L, smem);
  if (staged < L.fix_bytes_thermo) m.bind_thermo(L, img + L.o_fix);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int ns = m.ns, nsp = m.nsp, nr = m.nr, f0 = nr - m.nfall, nv = ns + 1;
  double* base = reinterpret_cast<double*>(smem + staged) + wid * cell_warp_doubles(ns);
  double* c = base + lane;                 // row k: c[k * CELL_ROW], G and w one and two paddings on
  int64_t* G = reinterpret_cast<int64_t*>(c + CELL_PAD);
  double* w = c + 2 * CELL_PAD;
  const double one = opaque(1.0), mone = opaque(-1.0), two = opaque(2.0), mtwo = opaque(-2.0);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t c0 = 32 * ((int64_t)blockIdx.x * (blockDim.x >> 5) + wid); c0 < n; c0 += 32 * nwarps) {
    const int nc = (int)(n - c0 < 32 ? n - c0 : 32);
    const int64_t cell = c0 + (lane < nc ? lane : nc - 1);   // idle lanes repeat the last cell
    // ---- mass fractions into the columns
    __syncwarp();
    if (layout == 1) {
      for (int k = 0; k < ns; ++k) c[k * CELL_ROW] = Yg[(int64_t)k * n + cell];
    } else {
      const double* src = Yg + c0 * ns;
      int row = 0, k = lane;
      while (k >= ns) { k -= ns; ++row; }
      for (int i = lane; i < nc * ns; i += 32) {
        base[k * CELL_ROW + row] = src[i];
        k += 32;
        while (k >= ns) { k -= ns; ++row; }
      }
      __syncwarp();
      if (lane >= nc)
        for (int k2 = 0; k2 < ns; ++k2) c[k2 * CELL_ROW] = base[k2 * CELL_ROW + nc - 1];
    }
    const double T = Tg[cell], p = pg[cell];
    const bool in = m.covers(T);
    const double Ts = in ? T : 1000.0;
    // ---- concentrations
    double sumYW = 0.0;
    for (int k = 0; k < ns; ++k) {
      const double yw = c[k * CELL_ROW] * m.invmw[k];
      c[k * CELL_ROW] = yw;
      sumYW = fma(one, yw, sumYW);
    }
    const double rho = cv ? p : p * m.inv_r_eos * recip(Ts * sumYW);
    const double ctot = rho * sumYW;
    const FixT f = fix_T(Ts, m.lt);
    double cpm = 0.0, hm = 0.0, D = 0.0;
    for (int k = 0; k < ns; ++k) {
      const double yw = c[k * CELL_ROW];
      const bool lo = __double_as_longlong(Ts) <= m.tmid[k];
      const uint64_t t = lo ? f.t11 : f.t13;
      G[k * CELL_ROW] = fix_gibbs(m.g + (lo ? 0 : 7 * nsp) + k, nsp, t, f);
      if (THERMO || RHS) {
        const double cpR = fix2d(fix_poly5(m.c + (lo ? 0 : 5 * nsp) + k, nsp, t), 52);
        if (THERMO) hm = fma(yw, fix2d(fix_enthalpy(m.h + (lo ? 0 : 6 * nsp) + k, nsp, t, f), 52), hm);
        cpm = fma(yw, cv ? cpR - 1.0 : cpR, cpm);   // (cv only with RHS: cv_k/R)
      }
      c[k * CELL_ROW] = rho * yw;
      w[k * CELL_ROW] = 0.0;
    }
    D = rho * cpm;
    c[ns * CELL_ROW] = 1.0;
    w[ns * CELL_ROW] = 0.0;
    G[ns * CELL_ROW] = 0;
    const double Tinv = m.nfall ? fix2d((int64_t)f.v, 70) : 0.0;
    const int64_t lC0 = m.lC - (int64_t)(f.L >> 9);       // log2(p_ref / RT)
    // ---- reactions
    // plain ones: rate = kf c c - kr c c, production to at most four species (an
    // absent factor's row ns reads c = 1, g = 0 and collects what nobody reads)
    auto at = [&](uint64_t x, int slot) { return c + ((unsigned)(x >> (16 * slot)) & 0xffffu); };
    auto g_of = [&](const double* p) { return __double_as_longlong(p[CELL_PAD]); };
    auto rate = [&](int r, bool rev, uint64_t x) {
      const int64_t a = fix_arrhenius(m.a[r], m.b[r], m.e[r], f);
      const double *r0 = at(x, 0), *r1 = at(x, 1), *p0 = at(x, 2), *p1 = at(x, 3);
      const double fwd = exp2_q52(a, m.et) * (*r0 * *r1);
      if (!rev) return fwd;
      const int64_t ar = a + g_of(p0) + g_of(p1) - g_of(r0) - g_of(r1) - (int64_t)fix_dn(m.ix[r]) * lC0;
      return fma(-exp2_q52(ar, m.et), *p0 * *p1, fwd);
    };
    // production to the (distinct) rows of word y; a doubled factor has one row
    auto produce = [&](uint64_t y, uint64_t ix, double q) {
      double *r0 = at(y, 0) + 2 * CELL_PAD, *r1 = at(y, 1) + 2 * CELL_PAD;
      double *p0 = at(y, 2) + 2 * CELL_PAD, *p1 = at(y, 3) + 2 * CELL_PAD;
      const double a0 = *r0, a1 = *r1, b0 = *p0, b1 = *p1;
      *r0 = fma(fix_twice_r(ix) ? mtwo : mone, q, a0);
      *r1 = fma(mone, q, a1);
      *p0 = fma(fix_twice_p(ix) ? two : one, q, b0);
      *p1 = fma(one, q, b1);
    };
    // the rates of the next pair come before the production of this one: their
    // integer work fills the time that the FP64 results take
    const int nrev = L.fix_plain_rev, nplain = nrev + L.fix_plain_irr;
    int r = 0;
    if (nrev >= 2) {
      double q0 = rate(0, true, m.cx[0]), q1 = rate(1, true, m.cx[1]);
      for (r = 2; r + 1 < nrev; r += 2) {
        const double n0 = rate(r, true, m.cx[r]), n1 = rate(r + 1, true, m.cx[r + 1]);
        produce(m.cy[r - 2], m.ix[r - 2], q0);
        produce(m.cy[r - 1], m.ix[r - 1], q1);
        q0 = n0;
        q1 = n1;
      }
      produce(m.cy[r - 2], m.ix[r - 2], q0);
      produce(m.cy[r - 1], m.ix[r - 1], q1);
    }
    for (; r < nplain; ++r) produce(m.cy[r], m.ix[r], rate(r, r < nrev, m.cx[r]));
    for (; r < nr; ++r) {
      const uint64_t ix = m.ix[r];
      const int type = fix_type(ix);
      const int r0 = min(fix_idx(ix, 0), ns), r1 = min(fix_idx(ix, 1), ns), r2 = min(fix_idx(ix, 2), ns);
      const int p0 = min(fix_idx(ix, 3), ns), p1 = min(fix_idx(ix, 4), ns), p2 = min(fix_idx(ix, 5), ns);
      const int64_t a = fix_arrhenius(m.a[r], m.b[r], m.e[r], f);
      double Pf = c[r0 * CELL_ROW] * c[r1 * CELL_ROW];
      if (r2 != ns) Pf *= c[r2 * CELL_ROW];
      double M = 1.0;
      if (type != 0) {
        const int row = fix_tbrow(ix);
        M = m.tbd[row] * ctot;
        for (int e = m.tbp[row]; e < m.tbp[row + 1]; ++e) M = fma(m.tbv[e], c[m.tbs[e] * CELL_ROW], M);
      }
      double kf = type < 2 ? exp2_q52(a, m.et) : cell_falloff(m, r - f0, type, a, M, f, Ts, Tinv);
      const int sgn = ((int)(ix >> 43) & 1) << 31;
      kf = __hiloint2double(__double2hiint(kf) ^ sgn, __double2loint(kf));
      double q;
      if (fix_rev(ix)) {
        // falloff: kr = kf / Kc, else 2^(a + dG) in one exponential
        int64_t ar = (type < 2 ? a : 0) + G[p0 * CELL_ROW] + G[p1 * CELL_ROW] - G[r0 * CELL_ROW] - G[r1 * CELL_ROW] -
                     (int64_t)fix_dn(ix) * lC0;
        if (r2 != ns || p2 != ns) ar += G[p2 * CELL_ROW] - G[r2 * CELL_ROW];
        double kr = exp2_q52(ar, m.et);
        if (type < 2) kr = __hiloint2double(__double2hiint(kr) ^ sgn, __double2loint(kr));
        else kr *= kf;
        double Pr = c[p0 * CELL_ROW] * c[p1 * CELL_ROW];
        if (p2 != ns) Pr *= c[p2 * CELL_ROW];
        q = fma(-kr, Pr, kf * Pf);
      } else {
        q = kf * Pf;
      }
      if (type == 1) q *= M;
      // production: the net coefficients of the reaction (species sums of
      // Lib_Chemistry_wdot.f90:203-215)
      for (int e = m.rs[r]; e < m.rs[r + 1]; ++e) {
        const int word = m.rw[e];
        double* wk = w + (word & 0xff) * CELL_ROW;
        const int code = word >> 8;                     // +1, -1, else an index of the value list
        const double nu = code == 1 ? one : (code == -1 ? mone : m.rv[code - 2]);
        *wk = fma(nu, q, *wk);
      }
    }
    // ---- outputs
    unsigned left = __ballot_sync(FULL, lane < nc && !in);
    if (RHS) {
      // dT/dt = -T sum_k (h_k/RT) w_k / sum_k c_k cp_k/R (u and cv at constant volume)
      double Q = 0.0;
      const double irho = recip(rho);
      for (int k = 0; k < ns; ++k) {
        const bool lo = __double_as_longlong(Ts) <= m.tmid[k];
        const double hr = fix2d(fix_enthalpy(m.h + (lo ? 0 : 6 * nsp) + k, nsp, lo ? f.t11 : f.t13, f) - (cv ? ONE52 : 0), 52);
        const double wk = w[k * CELL_ROW];
        Q = fma(hr, wk, Q);
        w[k * CELL_ROW] = m.mw[k] * wk * irho;
      }
      if (lane < nc && in) {
        for (int k = 0; k < ns; ++k) out[cell * nv + k] = w[k * CELL_ROW];
        out[cell * nv + ns] = -Ts * Q * recip(D);
      }
    } else {
      for (int k = 0; k < ns; ++k) w[k * CELL_ROW] *= m.mw[k];
      if (THERMO && lane < nc && in) {
        if (cpo) cpo[cell] = cpm * m.r_thermo;
        if (ho) ho[cell] = hm * m.r_thermo * Ts;
      }
      // (cells left to the FP64 path keep their row: it may hold their Y still)
      if (layout == 1) {
        if (lane < nc && in)
          for (int k = 0; k < ns; ++k) out[(int64_t)k * n + cell] = w[k * CELL_ROW];
      } else {
        __syncwarp();
        double* dst = out + c0 * ns;
        const double* wr = w - lane;
        int row = 0, k = lane;
        while (k >= ns) { k -= ns; ++row; }
        auto store = [&](bool all) {
          for (int i = lane; i < nc * ns; i += 32) {
            if (all || !(left >> row & 1u)) dst[i] = wr[k * CELL_ROW + row];
            k += 32;
            while (k >= ns) { k -= ns; ++row; }
          }
        };
        // (the test in the loop of every warp costs 1 M cells 0.9 %)
        if (left == 0) store(true);
        else store(false);
      }
    }
    // ---- cells outside the fixed-point range: the whole warp, one at a time
    while (left) {
      const int64_t ci = c0 + (__ffs(left) - 1);
      left &= left - 1;
      __syncwarp();
      if (nsp > 32) cell_general<RHS, 2>(img, L, base, lane, n, layout, ci, Tg, pg, Yg, out, cpo, ho, cv);
      else cell_general<RHS, 1>(img, L, base, lane, n, layout, ci, Tg, pg, Yg, out, cpo, ho, cv);
    }
  }
}

// Warps per block: what fits a block's shared memory, at most 8.
static int cell_warps(const ImageLayout& L, int staged) {
  const size_t room = device_smem_optin(), per = cell_warp_doubles(L.ns) * sizeof(double);
  if (room < staged + per) return 0;
  return (int)std::min<size_t>(CELL_MAX_WARPS, (room - staged) / per);
}

// When the thread-per-cell kernel is the faster one.  A warp's pass over the
// reactions takes about the same time for one cell as for 32 (31 species, 160
// reactions: 121 us with four warps on an SM, 145 with eight), so each round of
// warps has to bring enough cells: as many as the warp-per-cell kernel does in that
// time, about 145 per SM (thread against warp: 20,000 cells 136 against
// 125 us, 24,000 136 against 146, 32,000 145 against 193; 197 reactions: 20,000 167
// against 152, 24,000 167 against 177).  At 1 M cells it takes 4.6 ms against 6.1.
// Mechanisms of 13-25 species and 44-110 reactions could change earlier: 56-112 us at
// 22,100 cells, where the warp kernel takes 83-123 at 20,000.
// With 4 resident warps (54 species) there is too little to hide latencies
// behind (100,003 cells: 1.37 ms against 0.97 with the warp kernel), so six or more are
// asked for.
bool use_cell_kernel(const ImageLayout& L, int64_t n) {
  const int64_t sms = device_sms(), w = cell_warps(L, L.fix_bytes_cell);
  if (!L.fix || w < 6 || scratch_small_doubles(L) > cell_warp_doubles(L.ns)) return false;
  const int64_t rounds = (n + 32 * w * sms - 1) / (32 * w * sms);
  return n >= 145 * sms * rounds;
}

cudaError_t launch_wdot_cell(const uint8_t* img, const ImageLayout& L, int64_t n, int layout, const double* T,
                             const double* p, const double* Y, double* out, double* cp, double* h, bool rhs, int cv,
                             cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t tasks = (n + 31) / 32, sms = device_sms();
  // the thermo polynomials are read once per cell, at the same place on every
  // lane: they stay in global memory where staging them would cost a warp (1 M
  // cells of 31 species: 4.57 ms staged, 4.76 not, both with 8 warps; 4.9 staged with 7)
  const int wmax = cell_warps(L, L.fix_bytes_cell);
  const int staged = cell_warps(L, L.fix_bytes_thermo) == wmax ? L.fix_bytes_thermo : L.fix_bytes_cell;
  const int w = (int)std::min<int64_t>(wmax, (tasks + sms - 1) / sms);
  const size_t sm = staged + (size_t)w * cell_warp_doubles(L.ns) * sizeof(double);
  auto* fn = rhs ? k_wdot_cell<true, false> : (cp || h ? k_wdot_cell<false, true> : k_wdot_cell<false, false>);
  cudaError_t e = set_smem((const void*)fn, sm);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::min<int64_t>(sms, (tasks + w - 1) / w);
  fn<<<(unsigned)blocks, 32 * w, sm, st>>>(img, L, n, layout, T, p, Y, out, cp, h, cv, staged);
  count_launch();
  return cudaGetLastError();
}

}  // namespace flint
