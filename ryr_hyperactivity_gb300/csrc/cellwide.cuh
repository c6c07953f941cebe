// cellwide.cuh — the whole-cell update of one cell by four warps (the
// one-warp form is cell_update, tile.cuh; the arithmetic of both is
// membrane_update and step_coef, cellmodel.cuh).
//
// What bounds it: a warp issues one FP64 instruction every 64 cycles on this
// GPU, whatever its independent work, so one warp's membrane model (some 440
// FP64 instructions) takes 14 us before the lattice sums are needed and 7 us
// after.  Where the lattice update of a step is shorter than that (a cell or
// a few small ones), the cell update is the step's critical path.  Each of an
// SM's four schedulers has its own FP64 unit: four warps take the model's four
// independent parts (INa; IKr and IKs; Ito and IK1; INaK, the logarithms and
// the step's flags) at once, and within a warp the operands of each group of
// exponentials and quotients are formed one per lane.  A window of 100 steps
// with the one-warp update and with this one: one 100x20x10 cell in mixed
// precision 2.32 and 1.61 ms, 20 cells of 20x10x5 2.22 and 1.67 ms, one
// 20x10x5 cell in FP64 6.37 and 5.90 ms.  Four warps do not fit beside a full
// SM's lattice CTAs, so ensembles that fill the GPU keep the one-warp form,
// which hides there.
#pragma once

#include "tile.cuh"

namespace rh {

constexpr int kWideThreads = 128;

template <class R>
struct CellWideShared {
  double ena, eks, ek;
  double xina, xikr, xiks, xik1, xitos, xitof, xinak, stim;  // currents of the old state
  double xr, xs1, xs2;        // the gates the record prints, updated
  double qks_num, tauqks;
  double rdt, dth, rdt95, rdth95;
  double fm[6];
  int beat;
  double v, xnai, csubt, xicatto, xinacato, qks;  // after the sums
  double out_ica, out_ncx, out_ina;
  double osum[NOUT];
  StepCoef<R> k;
  BeatTracker bt;
};

__device__ __forceinline__ double from_lane(double x, int lane) {
  return __shfl_sync(0xffffffffu, x, lane);
}

// A gate relaxing to `inf`: g = exp(-dt / tau).
__device__ __forceinline__ double relax(double inf, double x, double g) {
  return inf - (inf - x) * g;
}

// One exponential of the membrane tables per lane.
__device__ __forceinline__ double table_exp(const ExpArg& ea, double v, double vek) {
  const double u = ea.src == kSrcV ? v : (ea.src == kSrcVek ? vek : XNAO);
  const double t = u + ea.a;
  double z = ea.div ? Math<double>::div(t, ea.d) : t * ea.c;
  z = z * ea.c2;
  return exp(ea.sq ? (-z) * z : z);
}

// ---- the four parts before the sums; `m` is the old state, `lane` the lane.
//      Updated gates go to `dm`, which the lattice update does not read. ----

__device__ __forceinline__ void wide_ina(const rh_membrane& m, double dt, rh_membrane* dm, int lane,
                                         double& conductance) {
  using M = Math<double>;
  const double v = m.v;
  const bool low = v < -40.0;
  const double E = table_exp(low ? kMemExpLow[lane] : kMemExpHigh[lane], v, 0.0);
  // quotients of lanes 0-2: am; low: the aj factor and bj; high: bh and bj
  const double ed = from_lane(E, lane == 0 ? 0 : lane == 1 ? (low ? 7 : 2) : (low ? 9 : 4));
  const double en = from_lane(E, low ? 8 : 3);
  double d = fma(lane == 0 ? -1.0 : 1.0, ed, 1.0);
  if (!low && lane == 1) d = 0.130 * d;
  double n = v + (lane == 0 ? 47.13 : 37.78);
  if (lane == 2) n = en;
  n = n * (lane == 0 ? 0.32 : lane == 1 ? 1.0 : (low ? 0.1212 : 0.3));
  if (!low && lane == 1) n = 1.00;
  const double q = M::div(n, lane < 3 ? d : 1.0);
  const double am = from_lane(q, 0), q1 = from_lane(q, 1), bj = from_lane(q, 2);
  const double bm = __dmul_rn(0.08, from_lane(E, 1));
  double ah = 0.00, bh = q1, aj = 0.00;
  if (low) {
    ah = __dmul_rn(0.135, from_lane(E, 2));
    bh = sum_of_products(3.56, from_lane(E, 3), 310000.0, from_lane(E, 4));
    aj = __dmul_rn(sum_of_products(-127140.0, from_lane(E, 5), -0.00003474, from_lane(E, 6)), q1);
  }
  // lanes 0-2: the time constants of h, j, m; lanes 3-5: their steady states
  const int g = lane % 3;
  const double a = g == 0 ? ah : g == 1 ? aj : am, b = g == 0 ? bh : g == 1 ? bj : bm;
  const double r = M::div(lane < 3 ? 1.00 : a, a + b);
  const double arg = M::div(-dt, r);
  const double G = exp(lane < 3 ? arg : 0.0);
  const double inf = from_lane(r, g + 3);
  const double x = relax(inf, g == 0 ? m.xh : g == 1 ? m.xj : m.xm, G);
  if (lane < 3) *(g == 0 ? &dm->xh : g == 1 ? &dm->xj : &dm->xm) = x;
  conductance = 15 * m.xh * m.xj * m.xm * m.xm * m.xm;
}

__device__ __forceinline__ void wide_ik(const rh_membrane& m, double dt, rh_membrane* dm, int lane,
                                        double& rg, double& xr, double& xs1, double& xs2) {
  using M = Math<double>;
  const double v = m.v;
  // lanes 0-6: the exponentials of table entries 10-16
  const double E = table_exp(kMemExpLow[lane < 7 ? 10 + lane : 31], v, 0.0);
  const bool minus = lane == 0 || lane == 5, grow = lane == 1 || lane == 6;
  const double d = fma(minus ? -1.0 : 1.0, E, grow ? -1.0 : 1.0);
  const double t = v + (lane == 0 ? 7.00 : lane == 1 ? 10.00 : 30.00);
  double n = t * (lane == 0 ? 0.001380 : lane == 1 ? 0.000610 : lane == 5 ? 0.0000719 : 0.0001310);
  if (!minus && !grow) n = 1.00;
  const double q = M::div(n, lane < 7 ? d : 1.0);
  rg = from_lane(q, 3);
  const double xkrinf = from_lane(q, 2), xs1ss = from_lane(q, 4);
  // lane 0: taukr, lanes 1-: tauxs
  const double s = from_lane(q, lane ? 5 : 0) + from_lane(q, lane ? 6 : 1);
  double tau = M::div(1.00, s);
  if (lane) tau = 0.95 * tau;
  const double G = exp(M::div(-dt, tau));
  const double x = relax(lane ? xs1ss : xkrinf, lane == 0 ? m.xr : lane == 1 ? m.xs1 : m.xs2, G);
  xr = from_lane(x, 0);
  xs1 = from_lane(x, 1);
  xs2 = from_lane(x, 2);
  if (lane < 3) *(lane == 0 ? &dm->xr : lane == 1 ? &dm->xs1 : &dm->xs2) = x;
}

__device__ __forceinline__ void wide_ito(const rh_membrane& m, double dt, rh_membrane* dm, int lane,
                                         double& ek, double& xik1, double& xitos, double& xitof) {
  using M = Math<double>;
  const double v = m.v;
  const double xki = 140.0, xko = 5.40;
  ek = __dmul_rn(1.00 / FRT, log(M::div(xko, xki)));
  const double vek = v - ek;
  // lanes 0-8: the exponentials of table entries 17-25
  const double E = table_exp(kMemExpLow[lane < 9 ? 17 + lane : 31], v, vek);
  // quotients: aki, bki, xtos_inf, ytos_inf, and those of txs, tys, tyf
  const double ed = from_lane(E, lane == 0 ? 0 : lane == 1 ? 3 : lane == 6 ? 5 : lane + 2);
  const double e18 = from_lane(E, 1), e19 = from_lane(E, 2), e25 = from_lane(E, 8);
  const double d = 1.0 + ed;
  const double n = lane == 0 ? 1.02 : lane == 1 ? 0.49124 * e18 + e19 : lane == 4 ? 9.00
                 : lane == 5 ? 3000.00 : lane == 6 ? 20.0 : 1.00;
  const double q = M::div(n, lane < 7 ? d : 1.0);
  const double aki = from_lane(q, 0), bki = from_lane(q, 1);
  const double xtos_inf = from_lane(q, 2), ytos_inf = from_lane(q, 3);
  // lanes 0-3: -dt over txs, tys, txf, tyf; lane 4: xkin
  const double qt = from_lane(q, lane == 0 ? 4 : lane == 1 ? 5 : 6);
  const double tau = fma(lane == 2 ? 3.50 : 1.0, lane == 2 ? e25 : qt,
                         lane == 0 ? 0.50 : lane == 1 ? 30.00 : lane == 2 ? 1.50 : 20.00);
  const double r = M::div(lane == 4 ? aki : -dt, lane == 4 ? aki + bki : tau);
  const double xkin = from_lane(r, 4);
  const double G = exp(lane < 4 ? r : 0.0);
  const double x = relax(lane & 1 ? ytos_inf : xtos_inf,
                         lane == 0 ? m.xtos : lane == 1 ? m.ytos : lane == 2 ? m.xtof : m.ytof, G);
  if (lane < 4)
    *(lane == 0 ? &dm->xtos : lane == 1 ? &dm->ytos : lane == 2 ? &dm->xtof : &dm->ytof) = x;
  const double gki = 0.600 * (sqrt(xko / 5.4));
  xik1 = (1.0) * gki * xkin * vek;
  xitos = 1.0 * 0.040 * m.xtos * (m.ytos + 0.50 * ytos_inf) * vek;
  xitof = 1.0 * 0.10 * m.xtof * m.ytof * vek;
}

template <class R>
__device__ __forceinline__ void wide_rest(const rh_membrane& m, double dt, const CellConst& c,
                                          int lane, CellWideShared<R>& sh) {
  using M = Math<double>;
  const double t = m.t, v = m.v, xnai = m.xnai;
  const double xki = 140.0, xko = 5.40, prnak = 0.0183300;
  // quotients: ena's and eks's arguments, INaK's 12/xnai, the time-step
  // constants and the beat
  const double q = M::div(lane == 0   ? XNAO
                          : lane == 1 ? xko + prnak * XNAO
                          : lane == 2 ? 12.00
                          : lane == 4 ? dt
                          : lane == 5 ? 0.95
                          : lane == 6 ? t - kStimStart
                                      : 1.0,
                          lane == 0 || lane == 2 ? xnai
                          : lane == 1            ? xki + prnak * xnai
                          : lane == 3 || lane == 5 ? dt
                          : lane == 4              ? 5.0
                          : lane == 6              ? c.pcl
                                                   : 1.0);
  const double lg = __dmul_rn(1.0 / FRT, log(lane < 2 ? q : 1.0));
  const double pow_nak = from_lane(q, 2), dth = from_lane(q, 4);
  // lanes 0-2: the exponentials of table entries 26-28
  const double E = table_exp(kMemExpLow[lane < 3 ? 26 + lane : 31], v, 0.0);
  const double e26 = from_lane(E, 0), e27 = from_lane(E, 1), e28 = from_lane(E, 2);
  const double r = M::div(lane == 0 ? e26 - 1.00 : lane == 1 ? 1.0 : 0.95,
                          lane == 0 ? 7.00 : lane == 1 ? 1.0 + pow_nak : dth);
  const double sigma = from_lane(r, 0), nak_f = from_lane(r, 1), rdth95 = from_lane(r, 2);
  const double fnak = M::div(1.00, 1.0 + 0.1245 * e27 + 0.0365 * sigma * e28);
  const double xinak = M::div(1. * 1.5000 * fnak * nak_f * xko, xko + 1.50);
  // fmods: stimulus phase (:689, iso :683) and the next update's window,
  // output, cadist and iso LCC flags (:1244, :777, :1002, :1213)
  const double tn = t + dt;
  const double f = fmod(lane == 0   ? (c.iso ? t : t + c.pcl - 100)
                        : lane == 1 ? tn - dt
                        : lane == 5 ? tn + 10 * c.pcl
                                    : tn + 0.0000001,
                        lane == 0   ? c.pcl
                        : lane == 3 ? 5.0
                        : lane == 4 ? c.pcl
                        : lane == 5 ? 15.5 * c.pcl
                                    : OUTT);
  if (lane < 6) sh.fm[lane] = f;
  const double f0 = from_lane(f, 0);
  const double beat = from_lane(q, 6), ena = from_lane(lg, 0), eks = from_lane(lg, 1);
  const double rdt = from_lane(q, 3), rdt95 = from_lane(q, 5);
  if (lane == 0) {
    sh.ena = ena;
    sh.eks = eks;
    sh.xinak = xinak;
    sh.stim = stimulus(c, t, f0);
    sh.beat = t < kStimStart ? -1 : (int)floor(beat);
    sh.qks_num = c.slowncx ? 1.6 : 0.8;      // :537, :541
    sh.tauqks = c.slowncx ? 2000 : 1000.00;  // :538, :542
    sh.rdt = rdt;
    sh.dth = dth;
    sh.rdt95 = rdt95;
    sh.rdth95 = rdth95;
  }
}

// The quotients of the step's exact sums (:447-456) in lanes 0-2: csubt,
// xicatto, xinacato, broadcast to the warp.
__device__ __forceinline__ void wide_sums(const CellDyn* dyn, const CellConst& c, int lane,
                                          double& csubt, double& xicatto, double& xinacato) {
  const int q = lane < 3 ? lane : 0;
  const double tot = fx_to_double(__ldcg(&dyn->acc[2 * q]), __ldcg(&dyn->acc[2 * q + 1]));
  const double s = Math<double>::div(tot, q == 0 ? (double)c.n : CM);
  const double r1 = s * 0.0965 * (q == 1 ? VP : VS);
  const double r2 = r1 * 2.0 * (ICAGAMMA + 1.);
  csubt = from_lane(s, 0);
  xicatto = from_lane(r2, 1);
  xinacato = from_lane(r1, 2);
}

// LCC gate rates of the FP64 lattice's coefficients (step_coef).
__device__ __forceinline__ void wide_coef_lcc(StepCoef<double>& k, double v, bool iso2, int lane) {
  using M = Math<double>;
  const double dv5 = iso2 ? 0 : 5, dvk = 8, fv5 = iso2 ? -28 : -22.8;
  const double fvk = iso2 ? 8.5 : 9.1;
  const double tq = 0.0337 * (v + 10.5);
  const double x = M::div(lane == 0 ? -(v - dv5) : lane == 1 ? -(v - fv5) : lane == 2 ? v - 60 : 1.0,
                          lane == 0 ? dvk : lane == 1 ? fvk : lane == 2 ? 12. : 1.0);
  const double X = exp(lane == 3 ? -tq * tq : x);
  const double x0 = from_lane(X, 0), x2 = from_lane(X, 2), x3 = from_lane(X, 3);
  const double inner = 0.035 * (v - dv5);
  const double q = M::div(lane == 2 ? 1.0 - x0 : 1.0, lane < 2 ? 1.0 + X : lane == 2 ? inner : 1.0);
  const double dinf = from_lane(q, 0), f_a = from_lane(q, 1), td_in = from_lane(q, 2);
  const double r = M::div(lane == 0 ? f_a : lane == 1 ? 1.0 : 0.035 * dvk,
                          lane == 0 ? 1. + x2 : lane == 1 ? td_in * dinf : dinf);
  const bool v_tiny = (v < 0.0001) && (v > -0.0001);
  const double finf = 1. - from_lane(r, 0);
  const double taudin = from_lane(r, v_tiny ? 2 : 1);
  const double taufin = (0.02 - 0.007 * x3);
  if (lane == 0) {
    k.alphac = 0.22;
    k.betac = iso2 ? 2 : 4;
    k.alphad = dinf * taudin;
    k.betad = (1 - dinf) * taudin;
    k.alphaf = finf * taufin;
    k.betaf = (1 - finf) * taufin;
  }
}

// GHK and NCX factors and the rest of the FP64 lattice's coefficients.
__device__ __forceinline__ void wide_coef_za(StepCoef<double>& k, double v, double xnai, double t,
                                             double dt, const CellConst& c, const double* fm,
                                             int lane) {
  using M = Math<double>;
  const double q = M::div(lane == 1 ? xnai : v * FARAD, lane == 1 ? KMNAI : XRGAS);
  const double r = from_lane(q, 1);
  const double za = M::div(from_lane(q, 0), TEMPER);
  const double X = exp((lane == 0 ? 2.0 : lane == 1 ? ETA : ETA - 1.0) * za);
  const double e2z = from_lane(X, 0), e1 = from_lane(X, 1), e2 = from_lane(X, 2);
  const double w = M::div(lane == 0 ? 4.0 * PCA * za * FARAD * GAMMAI : e2z,
                          lane == 0 ? e2z - 1.0 : 1000.0);
  const double k0 = from_lane(w, 0), k1 = from_lane(w, 1);
  const double xn3 = xnai * xnai * xnai;
  if (lane == 0) {
    k.lcc_k = fabs(za) < 0.001 ? 2.0 * PCA * FARAD * GAMMAI : k0;
    k.lcc_e2z_k = k1;
    k.ncx_num_a = e1 * xn3 * c.cao;
    k.ncx_num_b = e2 * (XNAO * XNAO * XNAO);
    k.ncx_t1 = KMCAI * (XNAO * XNAO * XNAO) * (1.0 + r * r * r);
    k.ncx_t3a = (KMCAO + c.cao) * xn3;
    k.ncx_den2 = 1.0 + KSAT * e2;
    option_coef(k, c, v, t, dt, fm[5]);
  }
}

// The four-warp update of `cell`; the steps and their order are those of
// cell_update, without its persistent form.
template <class R, bool OUT>
__device__ __forceinline__ void cell_update_wide(const StepArgs<R>& a, int cell, int nw,
                                                 CellWideShared<R>& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  CellDyn* dyn = a.dyn + cell;
  if (dyn->done) return;
  const StepCoef<R>* kc = coef_ptr<R>(dyn);
  const bool out_step = OUT && kc->output_step && !a.lattice_only && !a.no_output;
  const bool cadist = out_step && kc->cadist_step && a.out_cd != nullptr;
  const CellConst& cc = a.cells[cell];
  const double dt = a.dt;
  const rh_membrane m = dyn->m;
  const double t_next = m.t + dt;  // :1083
  if (a.lattice_only) {
    wait_for_prerequisite_grid();
  } else {
    double gna = 0.0, rg = 0.0, xr = 0.0, xs1 = 0.0, xs2 = 0.0;
    if (warp == 0) {
      wide_ina(m, dt, &dyn->m, lane, gna);
    } else if (warp == 1) {
      wide_ik(m, dt, &dyn->m, lane, rg, xr, xs1, xs2);
      if (lane == 0) {
        sh.xr = xr;
        sh.xs1 = xs1;
        sh.xs2 = xs2;
      }
    } else if (warp == 2) {
      double ek, xik1, xitos, xitof;
      wide_ito(m, dt, &dyn->m, lane, ek, xik1, xitos, xitof);
      if (lane == 0) {
        sh.ek = ek;
        sh.xik1 = xik1;
        sh.xitos = xitos;
        sh.xitof = xitof;
      }
      if (a.stats) {  // the beat in progress, read ahead
        const int* src = reinterpret_cast<const int*>(&dyn->bt);
        for (int i = lane; i < (int)(sizeof(BeatTracker) / 4); i += 32)
          reinterpret_cast<int*>(&sh.bt)[i] = src[i];
      }
    } else {
      wide_rest(m, dt, cc, lane, sh);
    }
    __syncthreads();
    const double v = m.v;
    if (warp == 0) {
      const double d = v - sh.ena;
      const double xina = sum_of_products(gna, d, 0.3e-3 * 5, d);
      if (lane == 0) {
        sh.xina = xina;
        dyn->m.xina = xina;
      }
    } else if (warp == 1) {
      const double gss = sqrt(5.40 / 5.40), gkr = 0.0078360;
      const double xikr = cc.svikr * gkr * gss * m.xr * rg * (v - sh.ek);
      const double xiks = 1.0 * 1. * 0.2000 * m.qks * m.xs1 * m.xs2 * (v - sh.eks);
      if (lane == 0) {
        sh.xikr = xikr;
        sh.xiks = xiks;
        dyn->m.xikr = xikr;
        dyn->m.xiks = xiks;
      }
    } else if (warp == 2) {
      if (lane == 0) {
        dyn->m.xik1 = sh.xik1;
        dyn->m.xitos = sh.xitos;
        dyn->m.xitof = sh.xitof;
        dyn->m.xinak = sh.xinak;
      }
    } else {  // the coefficients that need neither the sums nor the new voltage
      if constexpr (sizeof(R) == 4) {
        if (lane == 0) coef_known_f32(sh.k, cc, t_next, dt, sh.fm + 1, sh.rdt, sh.dth, sh.rdt95,
                                      sh.rdth95);
      } else if (lane == 0) {
        sh.k.rdt = sh.rdt;
        sh.k.dth = sh.dth;
        sh.k.rdt95 = sh.rdt95;
        sh.k.rdth95 = sh.rdth95;
        sh.k.svica = cc.svica;
        sh.k.svncx = cc.svncx;
        sh.k.cao = cc.cao;
        sh.k.ku = cc.ku;
        sh.k.ku2 = cc.ku2;
        sh.k.kb = cc.kb;
        sh.k.dt = dt;
        sh.k.reset_window = sh.fm[1] < dt;
        sh.k.output_step = sh.fm[2] < dt;
        sh.k.perm = cc.perm;
        sh.k.cadist_step = sh.k.output_step && sh.fm[3] < dt && sh.fm[4] < 500;
      }
    }
    __syncthreads();
    const double xina = sh.xina, xinak = sh.xinak;
    const double sum6 = xina + sh.xik1 + sh.xikr + sh.xiks + sh.xitos + sh.xitof;
    const double na = xina + 3.0 * xinak;

    wait_for_prerequisite_grid();

    uint32_t status = __ldcg(&dyn->status);
    if (warp == 0) {  // [Na]i and V (:701-738)
      double csubt, xicatto, xinacato;
      wide_sums(dyn, cc, lane, csubt, xicatto, xinacato);
      const double xrr = 1.0 * (1.0 / (1.0 / 50.0) / (0.18 * 12500)) / 1000.0;
      const double dvh = -(sum6 + xinacato + xicatto + xinak) + sh.stim;
      const double v1 = protocol_voltage(cc, m.t, dt, v + dvh * dt);
      const double dnai = -xrr * (na + 3.0 * xinacato);
      const double xnai1 = m.xnai + dnai * dt;
      if (lane == 0) {
        sh.v = v1;
        sh.xnai = xnai1;
        sh.csubt = csubt;
        sh.xicatto = xicatto;
        sh.xinacato = xinacato;
      }
    } else if (warp == 1) {  // the qks update and the window accumulators
      double csubt, xicatto, xinacato;
      wide_sums(dyn, cc, lane, csubt, xicatto, xinacato);
      double qks;
      if constexpr (sizeof(R) == 8) {
        const double q28 = Math<double>::div(0.28, csubt);
        const double qks_inf = 0.2 * (1 + Math<double>::div(sh.qks_num, 1 + q28 * q28 * q28));
        qks = m.qks + Math<double>::div(dt * (qks_inf - m.qks), sh.tauqks);
      } else {
        qks = m.qks + qks_increment(csubt, m.qks, sh.qks_num, sh.tauqks, dt);
      }
      if (lane == 0) {
        sh.qks = qks;
        sh.out_ica = m.out_ica + xicatto;
        sh.out_ncx = m.out_ncx + xinacato;
        sh.out_ina = m.out_ina + xina;
      }
    } else if (warp == 3 && out_step) {
      output_sums_warp(a.partials + (size_t)cc.tile_begin * nw * P_COUNT, cc.tile_count * nw,
                       sh.osum, lane);
    }
    __syncthreads();
    const double v1 = sh.v, xnai1 = sh.xnai;
    if (warp == 0) {
      if constexpr (sizeof(R) == 8) {
        wide_coef_lcc(sh.k, v1, cc.iso2, lane);
      } else {
        coef_voltage_f32(sh.k, cc, v1, xnai1);
      }
    } else if (warp == 1) {
      if constexpr (sizeof(R) == 8) wide_coef_za(sh.k, v1, xnai1, t_next, dt, cc, sh.fm, lane);
    } else if (warp == 2) {
      if (lane == 0 && a.stats) {  // per-beat detectors on the (t, V) sample of this step
        rh_beat_stats rec;
        if (beat_sample(sh.bt, sh.beat, m.t, v1, &rec)) {
          a.stats[(size_t)cell * a.stats_cap + dyn->stats_count % a.stats_cap] = rec;
          dyn->stats_count += 1;
        }
      }
      if (lane == 0) {
        if (extreme_high(v1) || extreme_high(xnai1) || extreme_high(sh.csubt) ||
            extreme_high(sh.xicatto) || extreme_high(sh.xinacato))
          status |= RH_STATUS_NAN;
        if (out_step && sh.osum[O_CIHIGH - P_STEP_END] > 0) status |= RH_STATUS_CI_HIGH;
        if (!(t_next < cc.tend)) {
          dyn->done = 1;
          status |= RH_STATUS_DONE;
        }
        dyn->status = status;
        dyn->m.t = t_next;
        dyn->m.step = m.step + 1;
        dyn->m.v = v1;
        dyn->m.xnai = xnai1;
        dyn->m.csubt = sh.csubt;
        dyn->m.xicatto = sh.xicatto;
        dyn->m.xinacato = sh.xinacato;
        dyn->m.qks = sh.qks;
      }
    } else if (!out_step) {
      if (lane == 0) {
        dyn->m.out_ica = sh.out_ica;
        dyn->m.out_ncx = sh.out_ncx;
        dyn->m.out_ina = sh.out_ina;
      }
    } else {
      double* w = a.out_wc + ((size_t)cell * a.out_cap + dyn->out_count % a.out_cap) * RH_WHOLECELL_COLS;
      rh_membrane mo = m;
      mo.sparksum = m.sparksum + (long long)sh.osum[O_SPARK - P_STEP_END];
      mo.v = v1;
      mo.xnai = xnai1;
      mo.csubt = sh.csubt;
      mo.qks = sh.qks;
      mo.xr = sh.xr;
      mo.xs1 = sh.xs1;
      mo.xiks = sh.xiks;
      mo.xikr = sh.xikr;
      mo.xik1 = sh.xik1;
      mo.xinak = xinak;
      mo.xitos = sh.xitos;
      mo.xitof = sh.xitof;
      mo.out_ica = sh.out_ica;
      mo.out_ncx = sh.out_ncx;
      mo.out_ina = sh.out_ina;
      wholecell_columns_warp(w, sh.osum, mo, cc.n, dt, lane);
      if (lane == 0) {
        if (cadist) {  // record header: t and V of this output step (:1005)
          double* h = a.out_cd + cc.cd_off + (dyn->cd_count % a.cd_cap) * (2 + 6 * (long long)cc.n);
          h[0] = m.t;
          h[1] = v1;
          dyn->cd_count += 1;
        }
        dyn->out_count += 1;
        dyn->m.sparksum = 0;  // :1074-1077
        dyn->m.out_ica = 0;
        dyn->m.out_ncx = 0;
        dyn->m.out_ina = 0;
      }
    }
    __syncthreads();
    if (warp == 0) {  // the next lattice update's coefficients
      const int* src = reinterpret_cast<const int*>(&sh.k);
      int* dst = sizeof(R) == 8 ? reinterpret_cast<int*>(&dyn->cd) : reinterpret_cast<int*>(&dyn->cf);
      for (int i = lane; i < (int)(sizeof(StepCoef<R>) / 4); i += 32) dst[i] = src[i];
    } else if (warp == 2 && a.stats) {
      if (out_step && lane == 0) {
        const double* w = a.out_wc + ((size_t)cell * a.out_cap +
                                      (dyn->out_count - 1) % a.out_cap) * RH_WHOLECELL_COLS;
        beat_on_output(sh.bt, w);  // written by warp 3 before the barrier
      }
      __syncwarp();
      int* dst = reinterpret_cast<int*>(&dyn->bt);
      for (int i = lane; i < (int)(sizeof(BeatTracker) / 4); i += 32)
        dst[i] = reinterpret_cast<const int*>(&sh.bt)[i];
    }
  }
  if (a.lattice_only) __syncthreads();  // every thread has read `done`
  if (tid < 6) dyn->acc[tid] = 0ull;  // the next step starts from zero
  if (tid == 32) dyn->parity ^= 1;
}

}  // namespace rh
