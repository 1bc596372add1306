// load_kernels.cu — the Newton-load kernels for sm_103a.
//
// One thread per device instance evaluates the model in FP64 (updateState) and
// writes every stamp term of that instance (loadDAEVectors/loadDAEMatrices) to
// a per-load term buffer laid out term-major, term[term0 + q*n + i], so a warp
// stores 32 consecutive doubles per term.  A second kernel sums the terms of
// each output (F, Q, dFdxdVp, dQdxdVp rows and dF/dx, dQ/dx non-zeros) in the
// reference's order — device type, instance, statement — from a precomputed
// list, one thread per output.  No atomics: results are identical run to run.
//
// This file is compiled twice: with -fmad=false into namespace xg::exact (each
// product and sum rounded on its own, as the serial CPU load does) and with
// -fmad=true into xg::fast (contracted to FMA).  XG_NS names the namespace.
// The fast build also splits each long output (a supply rail collects a term
// from every device on it) over the 256 threads of a block, each thread
// summing every 256th term in order, and adds the thread sums in a fixed
// butterfly and warp order: a serial chain of dependent FP64 adds (and
// gathers) is the slowest thing a GB300 can be asked to do.  The result is the same on every run, but not the reference's
// rounding, which the exact build keeps.

#include <cuda_runtime.h>

#include <algorithm>

#include <cstdint>

#include "xg_dcmp.cuh"
#include "xg_fast_rcp.cuh"
#include "xg_launch.cuh"
#include "xg_internal.h"

#ifndef XG_NS
#error "compile with -DXG_NS=exact or -DXG_NS=fast"
#endif
#ifndef XG_SPLIT_SUMS
#define XG_SPLIT_SUMS 0
#endif

namespace xg {
namespace XG_NS {

namespace {

constexpr double kMaxExpArg = 100.0;             // CONSTMAX_EXP_ARG
constexpr double kE = 2.718281828459045;         // CONSTe = exp(1.0), correctly rounded

__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }  // Xycemin

// Loads of what stays as it is while the kernel runs.  kStill: no kernel that
// is still running when this one starts may have written it, and the loads may
// be taken for constant; without it they are ordered behind await_previous()
// (few_kernel starts early, and a caller's kernel or a slot's set-up may have
// written any of it just ahead: vectors, parameters, circuit numbers).
template <bool kStill, typename T>
__device__ __forceinline__ T ld(const T *p) { return kStill ? __ldg(p) : *p; }

// ---- SPICE3 junction limiting, DeviceSupport (N_DEV_DeviceSupport.C:186-430);
// the MOSFETs' limiters in a form without divergence stand with level 1 ------
__device__ __forceinline__ double pnjlim(double vnew, double vold, double vt, double vcrit,
                                         int *icheck) {
  if ((vnew > vcrit) && (fabs(vnew - vold) > (vt + vt))) {
    if (vold > 0) {
      double arg = 1 + (vnew - vold) / vt;
      vnew = arg > 0 ? vold + vt * log(arg) : vcrit;
    } else {
      vnew = vt * log(vnew / vt);
    }
    *icheck = 1;
  } else {
    *icheck = 0;
  }
  return vnew;
}

// Term writer: term q of instance i at [q][i], so a warp's store of one term
// fills whole sectors; the reduction gathers them.
struct Terms {
  double *__restrict__ base;
  int n;
  __device__ __forceinline__ void put(int q, int i, double v) const { base[(int64_t)q * n + i] = v; }
};

// Batched loads: take instance i's circuit flags; false when the instance is
// not evaluated (no circuit: an unused place in a slot; or a finished one).
template <bool kStill>
__device__ __forceinline__ bool instance_flags(const DevType &t, int i, Flags &f) {
  if (!t.cid) return true;
  const int c = ld<kStill>(t.cid + i);
  if (c < 0) return false;
  if (!t.cflags) return true;
  f = t.cflags[c];
  return !f.skip;
}
template <bool kStill>
__device__ __forceinline__ bool instance_live(const DevType &t, int i) {
  if (!t.cid) return true;
  const int c = ld<kStill>(t.cid + i);
  return c >= 0 && !(t.cflags && t.cflags[c].skip);
}

// ---- resistor (N_DEV_Resistor.C:1073-1135) ---------------------------------
template <bool kStill>
__device__ __forceinline__ void res_one(const DevType &t, const LoadIO &io, int i) {
  if (i >= t.n || !instance_live<kStill>(t, i)) return;
  const int n = t.n;
  int lp = ld<kStill>(t.lid + i), ln = ld<kStill>(t.lid + n + i);
  double G = ld<kStill>(t.p + i);
  double i0 = (io.sol[lp] - io.sol[ln]) * G;
  Terms T{io.terms + t.term0, n};
  T.put(0, i, i0);
  T.put(1, i, -i0);
  T.put(2, i, G);
  T.put(3, i, -G);
  T.put(4, i, -G);
  T.put(5, i, G);
}

// ---- capacitor, constant C, no IC (N_DEV_Capacitor.C:1821-2040) -------------
template <bool kStill>
__device__ __forceinline__ void cap_one(const DevType &t, const LoadIO &io, int i) {
  if (i >= t.n || !instance_live<kStill>(t, i)) return;
  const int n = t.n;
  int lp = ld<kStill>(t.lid + i), ln = ld<kStill>(t.lid + n + i);
  double C = ld<kStill>(t.p + i);
  double vcap = io.sol[lp] - io.sol[ln];
  double q0 = C * vcap;
  io.sta[t.sta0 + i] = q0;
  Terms T{io.terms + t.term0, n};
  T.put(0, i, q0);
  T.put(1, i, -q0);
  T.put(2, i, C);
  T.put(3, i, -C);
  T.put(4, i, -C);
  T.put(5, i, C);
}

// PulseData::updateSource (N_DEV_SourceData.C:928-1031) with bpTol = 0.
template <bool kStill>
__device__ double pulse_value(const double *p, int n, int i, double t) {
  const double bpTol = 0.0;
  double V1 = ld<kStill>(p + XG_V_V1 * n + i), V2 = ld<kStill>(p + XG_V_V2 * n + i);
  double TD = ld<kStill>(p + XG_V_TD * n + i), TR = ld<kStill>(p + XG_V_TR * n + i);
  double TF = ld<kStill>(p + XG_V_TF * n + i), PW = ld<kStill>(p + XG_V_PW * n + i);
  double PER = ld<kStill>(p + XG_V_PER * n + i);
  double time = t - TD;
  if (time > PER && PER != 0.0) time -= PER * floor(time / PER);
  if (time <= 0 || (time > (TR + PW + TF) && (fabs(time - (TR + PW + TF)) > bpTol))) return V1;
  if ((time > TR && fabs(time - TR) > bpTol) && (time < (TR + PW) || fabs(time - (TR + PW)) < bpTol))
    return V2;
  if (time > 0 && (time < TR || fabs(time - TR) < bpTol))
    return TR != 0.0 ? V1 + (V2 - V1) * (time) / TR : V1;
  return TF != 0.0 ? V2 + (V1 - V2) * (time - (TR + PW)) / TF : V2;
}

// ---- independent voltage source (N_DEV_Vsrc.C:941-1045) ---------------------
template <bool kStill>
__device__ __forceinline__ void vsrc_one(const DevType &t, Flags f, const LoadIO &io, int i) {
  if (i >= t.n || !instance_flags<kStill>(t, i, f)) return;
  const int n = t.n;
  int lp = ld<kStill>(t.lid + i), ln = ld<kStill>(t.lid + n + i), lb = ld<kStill>(t.lid + 2 * n + i);
  double source;
  if ((f.tranop || f.transient) && ld<kStill>(t.p + XG_V_KIND * n + i) == XG_SRC_PULSE)
    source = pulse_value<kStill>(t.p, n, i, f.time);
  else
    source = ld<kStill>(t.p + XG_V_V1 * n + i);
  double srcCurrent = io.sol[lb];
  double srcDrop = (io.sol[lp] - io.sol[ln]);
  Terms T{io.terms + t.term0, n};
  T.put(0, i, srcCurrent);
  T.put(1, i, -srcCurrent);
  T.put(2, i, srcDrop);
  T.put(3, i, -source);
  T.put(4, i, 1.0);
  T.put(5, i, -1.0);
  T.put(6, i, 1.0);
  T.put(7, i, -1.0);
}

// ---- independent current source (N_DEV_ISRC.C:774-800) ----------------------
// The source value goes into F at both terminals; there are no matrix entries.
template <bool kStill>
__device__ __forceinline__ void isrc_one(const DevType &t, Flags f, const LoadIO &io, int i) {
  if (i >= t.n || !instance_flags<kStill>(t, i, f)) return;
  const int n = t.n;
  double source;
  if ((f.tranop || f.transient) && ld<kStill>(t.p + XG_V_KIND * n + i) == XG_SRC_PULSE)
    source = pulse_value<kStill>(t.p, n, i, f.time);
  else
    source = ld<kStill>(t.p + XG_V_V1 * n + i);
  Terms T{io.terms + t.term0, n};
  T.put(0, i, source);
  T.put(1, i, -source);
}

// ---- junction diode, level 1 (N_DEV_Diode.C:873-1331, 2007-2128) ------------
template <bool kStill>
__device__ __forceinline__ void diode_one(const DevType &t, const DevOptions &o, Flags f, const LoadIO &io, int i) {
  if (i >= t.n || !instance_flags<kStill>(t, i, f)) return;
  const int n = t.n;
  const double *p = t.p;
#define PRM(k) ld<kStill>(p + (k) * n + i)
  const int li_Pos = ld<kStill>(t.lid + i), li_Neg = ld<kStill>(t.lid + n + i), li_Pri = ld<kStill>(t.lid + 2 * n + i);
  const double gmin = o.gmin;
  const double M = PRM(XG_D_M), BV = PRM(XG_D_BV), N = PRM(XG_D_N), TT = PRM(XG_D_TT);
  const double tVcrit = PRM(XG_D_TVCRIT), tBrkdwnV = PRM(XG_D_TBRKDWNV);
  const double tJctCap = PRM(XG_D_TJCTCAP);
  const int flags = (int)PRM(XG_D_FLAGS);
  const int BVGiven = flags & 1, InitCondGiven = (flags >> 1) & 1, off = (flags >> 2) & 1;
  double *sto = io.sto + t.sto0 + i;

  // Master::updateState stores the previous limited Vd before the update.
  const double vd_member = io.diode_vd[i];
  *sto = vd_member;
  double Vpp = io.sol[li_Pri], Vn = io.sol[li_Neg], Vp = io.sol[li_Pos];
  double Vd = Vpp - Vn;
  double Isat = PRM(XG_D_ISAT);
  double Vte = N * PRM(XG_D_VT);
  const double Vd_orig = Vd;
  double Vd_old;
  if (f.newton_iter == 0) {
    if (f.init_jct && o.voltlim) {
      if (InitCondGiven) Vd = PRM(XG_D_INITCOND);
      else if (off) Vd = 0.0;
      else Vd = tVcrit;
    }
    Vd_old = f.dcop ? Vd : io.sto_curr[t.sto0 + i];
  } else {
    Vd_old = vd_member;
  }
  if (o.voltlim && f.newton_iter >= 0) {
    int ichk = 0;
    if (BVGiven && (Vd < dmin(0.0, -BV + 10.0 * Vte))) {
      double Vdtmp = -(BV + Vd);
      Vdtmp = pnjlim(Vdtmp, -(Vd_old + BV), Vte, tVcrit, &ichk);
      Vd = -(Vdtmp + BV);
    } else {
      Vd = pnjlim(Vd, Vd_old, Vte, tVcrit, &ichk);
    }
  }
  double Id, Gd;
  if (Vd >= -3.0 * Vte) {
    double evd = exp(dmin(kMaxExpArg, Vd / Vte));
    Id = Isat * (evd - 1.0) + gmin * Vd;
    Gd = Isat * evd / Vte + gmin;
  } else {
    Isat *= PRM(XG_D_TIRF);
    if (!tBrkdwnV || (Vd >= -tBrkdwnV)) {
      double arg = 3.0 * Vte / (Vd * kE);
      arg = arg * arg * arg;
      Id = -Isat * (1.0 + arg) + gmin * Vd;
      Gd = Isat * 3.0 * arg / Vd + gmin;
    } else {
      double evrev = exp(dmin(kMaxExpArg, -(tBrkdwnV + Vd) / Vte));
      double arg2 = 3.0 * Vte / (kE * tBrkdwnV);
      arg2 = arg2 * arg2 * arg2;
      double Isat_tBrkdwnV = Isat * (1 - arg2);
      Id = -Isat_tBrkdwnV * evrev + gmin * Vd;
      Gd = Isat_tBrkdwnV * evrev / Vte + gmin;
    }
  }
  double Qd = 0.0, Cd = 0.0;
  const double Vc = Vd;
  if (tJctCap != 0.0) {
    double Area = PRM(XG_D_AREA), tJctPot = PRM(XG_D_TJCTPOT), tDepCap = PRM(XG_D_TDEPCAP);
    double Czero = tJctCap * Area;
    if (Vc < tDepCap) {
      double arg = 1.0 - Vc / tJctPot;
      double sarg = exp(dmin(kMaxExpArg, -M * log(arg)));
      Qd = TT * Id + tJctPot * Czero * (1.0 - arg * sarg) / (1.0 - M);
      Cd = TT * Gd + Czero * sarg;
    } else {
      double F2 = PRM(XG_D_F2), F3 = PRM(XG_D_F3);
      double Czof2 = Czero / F2;
      double MotJctPot = M / tJctPot;
      Qd = TT * Id + Czero * PRM(XG_D_TF1) +
           Czof2 * (F3 * (Vc - tDepCap) + (0.5 * MotJctPot) * (Vc * Vc - tDepCap * tDepCap));
      Cd = TT * Gd + Czof2 * (F3 + MotJctPot * Vc);
    }
  }
  io.diode_vd[i] = Vd;

  // Master::loadDAEVectors / loadDAEMatrices
  const double Gspr = PRM(XG_D_GSPR);
#undef PRM
  double Ir = Gspr * (Vp - Vpp);
  Terms T{io.terms + t.term0, n};
  T.put(0, i, -(-Ir));
  T.put(1, i, -Id);
  T.put(2, i, -(-Id + Ir));
  T.put(3, i, -Qd);
  T.put(4, i, -(-Qd));
  double Gd_Jdxp = 0.0, Cd_Jdxp = 0.0;
  if (o.voltlim) {
    double Vd_diff = Vd - Vd_orig;
    Cd_Jdxp = -(Cd)*Vd_diff;
    Gd_Jdxp = -(Gd)*Vd_diff;
  }
  T.put(5, i, Gd_Jdxp);
  T.put(6, i, -Gd_Jdxp);
  T.put(7, i, Cd_Jdxp);
  T.put(8, i, -Cd_Jdxp);
  T.put(9, i, Gspr);
  T.put(10, i, -Gspr);
  T.put(11, i, Gd);
  T.put(12, i, -Gd);
  T.put(13, i, -Gspr);
  T.put(14, i, -Gd);
  T.put(15, i, Gspr + Gd);
  T.put(16, i, Cd);
  T.put(17, i, -Cd);
  T.put(18, i, -Cd);
  T.put(19, i, Cd);
}

// ---- MOSFET level 1 (N_DEV_MOSFET1.C:2618-3427, 4103-4722), newMeyer off ----
// Bound by FP64 issue, and a warp pays for every instruction any of its lanes
// takes: with the model's branches as branches, most of what a warp of the
// random netlist issued was for other lanes' alternatives.  So each alternative is a choice of operands for one evaluation (the direction of
// the channel, the junction that is limited, saturation or not) with the
// arithmetic of the branch it stands for; comparisons are made on the bits
// and polarity and mode are sign flips (xg_dcmp.cuh); quotients by vt share
// one reciprocal; and a warp whose instances all have M = 1 skips the
// products by M.  Nothing is formed that a card without body effect
// (GAMMA = 0) or oxide capacitance would multiply by that zero.  On a million
// devices a warp issues 244 FP64 instructions (FMA build; exact 259), 84% of
// the FP64 pipe's cycles: 1.532 -> 0.470 ms (exact 0.502; ncu,
// profiles/mos1_reduce_single_load_mos1_1M.md).

// fetlim: the limit is a bound on the step (s) or on the value (t).
__device__ __forceinline__ double fetlim_select(double vnew, double vold, double vto) {
  const double hi = fma(2.0, magnitude(vold - vto), 2.0);  // (exact products)
  const double lo = fma(0.5, hi, 2.0);
  const double vtox = vto + 3.5, delv = vnew - vold;
  const bool down = le0(delv), on = ge(vold, vto), strong = ge(vold, vtox);
  const double s = vold + (on ? (down ? -lo : hi) : (down ? -hi : lo));
  const double t = vto + (on ? (strong ? 2.0 : down ? -0.5 : 4.0) : 0.5);
  if (on ? strong && (!down || ge(vnew, vtox)) : down || le(vnew, t)) {
    const double step = down ? -delv : delv, bound = on ? (down ? lo : hi) : (down ? hi : lo);
    return (on && !down ? ge(step, bound) : gt(step, bound)) ? s : vnew;
  }
  if (!on) return t;
  return down ? (gt(vnew, t) ? vnew : t) : (lt(vnew, t) ? vnew : t);
}

__device__ __forceinline__ double limvds_select(double vnew, double vold) {
  const bool strong = ge(vold, 3.5), up = gt(vnew, vold);
  double lim = up ? 4.0 : -0.5;
  if (strong) lim = up ? (3.0 * vold) + 2.0 : 2.0;
  if (up) return lt(vnew, lim) ? vnew : lim;
  if (strong && !lt(vnew, 3.5)) return vnew;
  return gt(vnew, lim) ? vnew : lim;
}

// pnjlim with y the reciprocal of vt; one logarithm for both of its forms.
__device__ __forceinline__ double pnjlim_select(double vnew, double vold, double vt, double y, double vcrit) {
  const double delv = vnew - vold;
  if (!(gt(vnew, vcrit) && gt(magnitude(delv), vt + vt))) return vnew;
  const bool pos = gt0(vold);
  const double q = xg::quotient(pos ? delv : vnew, vt, y);
  const double arg = pos ? 1 + q : q;
  if (pos && !gt0(arg)) return vcrit;
  return (pos ? vold : 0.0) + vt * log(arg);
}

// DeviceSupport::qmeyer (N_DEV_DeviceSupport.C:545-631); the caller exchanges
// the gate-source and gate-drain sides in reverse mode.
__device__ __forceinline__ void qmeyer_select(double vgs, double vgd, double von, double vdsat, double &capgs,
                                              double &capgd, double &capgb, double phi, double cox) {
  const double vgst = vgs - von;
  capgs = capgd = 0.0;
  if (le0(vgst)) {
    if (le(vgst, -phi)) {
      capgb = 0.5 * cox;
    } else {
      const double c = vgst * cox;
      capgb = -c / (2 * phi);
      if (!le(vgst, -0.5 * phi)) capgs = c / (1.5 * phi) + cox / 3;
    }
  } else {
    const double vds = vgs - vgd;
    capgb = 0;
    if (le(vdsat, vds)) {
      capgs = cox / 3;
    } else {
      const double vddif = 2.0 * vdsat - vds, vddif1 = vdsat - vds, vddif2 = vddif * vddif;
      capgd = cox * (1.0 - vdsat * vdsat / vddif2) / 3;
      capgs = cox * (1.0 - vddif1 * vddif1 / vddif2) / 3;
    }
  }
}

// One junction: conductance and current from its voltage v (sat the
// saturation current, y the reciprocal of vt).  Without forward bias the
// exponential is 1, which leaves sat / vt and the current gbv v.
__device__ __forceinline__ void junction(double v, double sat, double vt, double y, double gmin, double &g, double &c) {
  const bool fwd = !le0(v);
  double ev = 1.0;
  if (fwd) {
    const double q = xg::quotient(v, vt, y);
    ev = exp(lt(kMaxExpArg, q) ? kMaxExpArg : q);
  }
  g = xg::quotient(sat * ev, vt, y) + gmin;
  const double cv = (fwd ? gmin : g) * v;
  c = fwd ? sat * (ev - 1) + gmin * v : cv;
}

template <bool kStill>
__device__ __forceinline__ void mos1_one(const DevType &t, const DevOptions &o, Flags f, const LoadIO &io, int i) {
  if (i >= t.n || !instance_flags<kStill>(t, i, f)) return;
  const int n = t.n;
  const double *p = t.p;
#define PRM(k) ld<kStill>(p + (k) * n + i)
  auto sol = [&](int k) { return ld<kStill>(io.sol + k); };
  const int li_d = ld<kStill>(t.lid + i), li_g = ld<kStill>(t.lid + n + i), li_s = ld<kStill>(t.lid + 2 * n + i);
  const int li_b = ld<kStill>(t.lid + 3 * n + i), li_dp = ld<kStill>(t.lid + 4 * n + i), li_sp = ld<kStill>(t.lid + 5 * n + i);
  // the polarity (+-1) as a sign to flip
  const int pol = __double2hiint(PRM(XG_M1_DTYPE)) & int(0x80000000);
  const double gamma = PRM(XG_M1_GAMMA);
  const double vt = PRM(XG_M1_VT), tPhi = PRM(XG_M1_TPHI);
  const double gmin = o.gmin;
  const int flags = (int)PRM(XG_M1_FLAGS);
  const int OFF = flags & 1, IC_GIVEN = (flags >> 1) & 1;
  double *sta = io.sta + t.sta0 + (int64_t)i * 8;
  double *sto = io.sto + t.sto0 + (int64_t)i * 5;
  const double *csta = io.sta_curr + t.sta0 + (int64_t)i * 8;
  const double *csto = io.sto_curr + t.sto0 + (int64_t)i * 5;
  enum { S_QGS, S_QGD, S_QGB, S_CAPGS, S_CAPGD, S_CAPGB, S_QBD, S_QBS };
  enum { O_VBD, O_VBS, O_VGS, O_VDS, O_VON };

  const double Vd = sol(li_d), Vg = sol(li_g), Vs = sol(li_s);
  const double Vb = sol(li_b), Vsp = sol(li_sp), Vdp = sol(li_dp);
  double vbs = flip(Vb - Vsp, pol), vgs = flip(Vg - Vsp, pol), vds = flip(Vdp - Vsp, pol);
  double vbd = vbs - vds, vgd = vgs - vds;
  const double vgs_orig = vgs, vds_orig = vds, vbs_orig = vbs, vbd_orig = vbd, vgd_orig = vgd;

  bool forced = false;  // origFlag cleared by the initial-condition branch
  if (f.init_jct && !OFF && o.voltlim) {
    if (IC_GIVEN) {
      forced = true;
      vds = flip(PRM(XG_M1_ICVDS), pol);
      vgs = flip(PRM(XG_M1_ICVGS), pol);
      vbs = flip(PRM(XG_M1_ICVBS), pol);
    } else {
      vbs = -1;
      vgs = flip(PRM(XG_M1_TVTO), pol);
      vds = 0;
    }
    vbd = vbs - vds;
    vgd = vgs - vds;
  } else if ((f.init_fix || f.init_jct) && OFF) {
    vbs = vgs = vds = 0;
    vbd = vgd = 0;
  }

  double Von, vbs_old, vbd_old, vgs_old, vds_old;
  if (f.newton_iter == 0) {
    if (!f.dcop) {
      vbs_old = ld<kStill>(csto + O_VBS); vbd_old = ld<kStill>(csto + O_VBD);
      vgs_old = ld<kStill>(csto + O_VGS); vds_old = ld<kStill>(csto + O_VDS);
      Von = flip(ld<kStill>(csto + O_VON), pol);
    } else {
      vbs_old = vbs; vbd_old = vbd; vgs_old = vgs; vds_old = vds;
      Von = 0.0;
    }
  } else {
    vbs_old = sto[O_VBS]; vbd_old = sto[O_VBD];
    vgs_old = sto[O_VGS]; vds_old = sto[O_VDS];
    Von = flip(sto[O_VON], pol);
  }
  const double y = 1.0 / vt;

  if (o.voltlim && !(f.init_fix && OFF)) {
    // forward: vgs is limited, then vds, and vgd follows; reverse: vgd, -vds, vgs
    const bool fwd = ge0(vds_old);
    const int rev = fwd ? 0 : int(0x80000000);
    const double vgd_old = vgs_old - vds_old;
    const double vg = fetlim_select(fwd ? vgs : vgd, fwd ? vgs_old : vgd_old, Von);
    vds = (fwd ? vg : vgs) - (fwd ? vgd : vg);
    vds = flip(limvds_select(flip(vds, rev), flip(vds_old, rev)), rev);
    const double other = vg + flip(vds, fwd ? int(0x80000000) : 0);
    vgs = fwd ? vg : other;
    vgd = fwd ? other : vg;
    const bool pos = ge0(vds);
    const double vb = pnjlim_select(pos ? vbs : vbd, pos ? vbs_old : vbd_old, vt, y,
                                    pos ? PRM(XG_M1_SOURCEVCRIT) : PRM(XG_M1_DRAINVCRIT));
    vbs = pos ? vb : vb + vds;
  }
  vbd = vbs - vds;
  vgd = vgs - vds;
  const double Vgb = vgs - vbs;
  const bool origFlag = !(forced || ne(vgs_orig, vgs) || ne(vds_orig, vds) || ne(vbs_orig, vbs) ||
                          ne(vbd_orig, vbd) || ne(vgd_orig, vgd));

  double gbs, cbs, gbd, cbd;
  junction(vbs, PRM(XG_M1_SOURCESATCUR), vt, y, gmin, gbs, cbs);
  junction(vbd, PRM(XG_M1_DRAINSATCUR), vt, y, gmin, gbd, cbd);
  // an infinite or NaN voltage takes every operation, zeros times it included
  const bool wild = !finite_bits(vbs) || !finite_bits(vgs) || !finite_bits(vds) || !finite_bits(vbs_orig) ||
                    !finite_bits(vgs_orig) || !finite_bits(vds_orig);
  const bool fwd = ge0(vds);  // mode
  const int rev = fwd ? 0 : int(0x80000000);
  const double vds_m = flip(vds, rev);
  double Vdsat, cdrain, gm, gds, gmbs;
  {
    const double vbx = fwd ? vbs : vbd;
    const double tVbi = flip(PRM(XG_M1_TVBI), pol);
    double arg = 0.0;
    Von = tVbi;
    if (wild || ne0(gamma)) {
      const bool neg = le0(vbx);
      double sarg = sqrt(neg ? tPhi - vbx : tPhi);
      if (!neg) {
        sarg = sarg - vbx / (sarg + sarg);
        sarg = lt0(sarg) ? 0.0 : sarg;
      }
      Von = tVbi + gamma * sarg;
      arg = le0(sarg) ? 0 : gamma / (sarg + sarg);
    }
    const double vgst = (fwd ? vgs : vgd) - Von;
    Vdsat = gt0(vgst) ? vgst : 0.0;
    const bool off = le0(vgst), sat = le(vgst, vds_m);
    const double lambda = PRM(XG_M1_LAMBDA), Beta = PRM(XG_M1_BETA);
    // with w = vgst in saturation, vds below it: gm = betap w, the current
    // gm (vgst - w/2), gds = betap (vgst - w) + lambda Beta w (vgst - w/2)
    const double w = sat ? vgst : vds_m;
    const double z = fma(-0.5, w, vgst);  // (exact product)
    double betap = Beta, lb = 0.0;
    if (wild || ne0(lambda)) {
      betap = Beta * (1 + lambda * vds_m);
      lb = lambda * Beta;
    }
    gm = betap * w;
    cdrain = gm * z;
    gds = sat ? 0.0 : betap * (vgst - w);
    if (wild || ne0(lambda)) gds += lb * w * z;
    gmbs = wild || ne0(arg) ? gm * arg : 0.0;
    if (off) {
      cdrain = 0; gm = 0; gds = 0; gmbs = 0;
    }
  }

  double qbs = 0, capbs = 0, qbd = 0, capbd = 0;
  {
    const double Cbs = PRM(XG_M1_CBS), Cbssw = PRM(XG_M1_CBSSW);
    const double Cbd = PRM(XG_M1_CBD), Cbdsw = PRM(XG_M1_CBDSW);
    if (ne0(Cbs) || ne0(Cbssw) || ne0(Cbd) || ne0(Cbdsw)) {
      const double MJ = PRM(XG_M1_MJ), MJSW = PRM(XG_M1_MJSW);
      const double tDepCap = PRM(XG_M1_TDEPCAP), tBulkPot = PRM(XG_M1_TBULKPOT);
      double sarg, sargsw, arg;
      if (ne0(Cbs) || ne0(Cbssw)) {
        if (lt(vbs, tDepCap)) {
          arg = 1 - vbs / tBulkPot;
          if (MJ == MJSW) {
            sarg = sargsw = (MJ == .5) ? 1 / sqrt(arg) : exp(-MJ * log(arg));
          } else {
            sarg = (MJ == .5) ? 1 / sqrt(arg) : exp(-MJ * log(arg));
            sargsw = (MJSW == .5) ? 1 / sqrt(arg) : exp(-MJSW * log(arg));
          }
          qbs = tBulkPot * (Cbs * (1 - arg * sarg) / (1 - MJ) + Cbssw * (1 - arg * sargsw) / (1 - MJSW));
          capbs = Cbs * sarg + Cbssw * sargsw;
        } else {
          const double f2s = PRM(XG_M1_F2S), f3s = PRM(XG_M1_F3S);
          qbs = PRM(XG_M1_F4S) + vbs * (f2s + vbs * (f3s / 2));
          capbs = f2s + f3s * vbs;
        }
      }
      if (ne0(Cbd) || ne0(Cbdsw)) {
        if (lt(vbd, tDepCap)) {
          arg = 1 - vbd / tBulkPot;
          if (MJ == .5 && MJSW == .5) {
            sarg = sargsw = 1 / sqrt(arg);
          } else {
            sarg = (MJ == .5) ? 1 / sqrt(arg) : exp(-MJ * log(arg));
            sargsw = (MJSW == .5) ? 1 / sqrt(arg) : exp(-MJSW * log(arg));
          }
          qbd = tBulkPot * (Cbd * (1 - arg * sarg) / (1 - MJ) + Cbdsw * (1 - arg * sargsw) / (1 - MJSW));
          capbd = Cbd * sarg + Cbdsw * sargsw;
        } else {
          const double f2d = PRM(XG_M1_F2D), f3d = PRM(XG_M1_F3D);
          qbd = PRM(XG_M1_F4D) + vbd * (f2d + vbd * f3d / 2);
          capbd = f2d + vbd * f3d;
        }
      }
    }
  }

  double capgs = 0.0, capgd = 0.0, capgb = 0.0;
  const double OxideCap = PRM(XG_M1_OXIDECAP);
  if (wild || ne0(OxideCap)) {
    double c1, c2;
    qmeyer_select(fwd ? vgs : vgd, fwd ? vgd : vgs, Von, Vdsat, c1, c2, capgb, tPhi, OxideCap);
    capgs = fwd ? c1 : c2;
    capgd = fwd ? c2 : c1;
  }

  double Capgs, Capgd, Capgb;
  {
    const double cgso = PRM(XG_M1_CGSO), cgdo = PRM(XG_M1_CGDO), cgbo = PRM(XG_M1_CGBO);
    if (f.dcop) {
      Capgs = 2.0 * capgs + cgso;
      Capgd = 2.0 * capgd + cgdo;
      Capgb = 2.0 * capgb + cgbo;
    } else {
      Capgs = (capgs + ld<kStill>(csta + S_CAPGS) + cgso);
      Capgd = (capgd + ld<kStill>(csta + S_CAPGD) + cgdo);
      Capgb = (capgb + ld<kStill>(csta + S_CAPGB) + cgbo);
    }
    Capgs = magnitude(Capgs);
    Capgd = magnitude(Capgd);
    Capgb = magnitude(Capgb);
  }
  const double drainConductance = PRM(XG_M1_GD), sourceConductance = PRM(XG_M1_GS);
  const double Idrain = wild || ne0(drainConductance) ? drainConductance * (Vd - Vdp) : 0.0;
  const double Isource = wild || ne0(sourceConductance) ? sourceConductance * (Vs - Vsp) : 0.0;
  const double Gm = flip(gm, rev), Gmbs = flip(gmbs, rev);
  const double gsum = ne0(gmbs) ? Gm + Gmbs : Gm;
  const double nrmsum = fwd ? gsum : 0.0, revsum = fwd ? 0.0 : -gsum;
  const double cdreq = flip(cdrain, pol ^ rev);

  // Master::updateState store / state writes
  sto[O_VBD] = vbd; sto[O_VBS] = vbs; sto[O_VGS] = vgs; sto[O_VDS] = vds; sto[O_VON] = flip(Von, pol);
  sta[S_CAPGS] = capgs; sta[S_CAPGD] = capgd; sta[S_CAPGB] = capgb;
  double qgs, qgd, qgb;
  if (f.dcop) {
    qgs = Capgs * vgs; qgd = Capgd * vgd; qgb = Capgb * Vgb;
  } else {
    qgs = ld<kStill>(csta + S_QGS); qgd = ld<kStill>(csta + S_QGD); qgb = ld<kStill>(csta + S_QGB);
    double vgs1 = ld<kStill>(csto + O_VGS), vbs1 = ld<kStill>(csto + O_VBS), vds1 = ld<kStill>(csto + O_VDS);
    if (wild || ne0(Capgs) || ne0(Capgd) || ne0(Capgb) || !finite_bits(vgs1) || !finite_bits(vbs1) ||
        !finite_bits(vds1)) {
      double vgb1 = vgs1 - vbs1, vgd1 = vgs1 - vds1;
      qgs += Capgs * (vgs - vgs1);
      qgd += Capgd * (vgd - vgd1);
      qgb += Capgb * (Vgb - vgb1);
    }
  }
  sta[S_QGS] = qgs; sta[S_QGD] = qgd; sta[S_QGB] = qgb; sta[S_QBD] = qbd; sta[S_QBS] = qbs;

  // Master::loadDAEVectors and loadDAEMatrices (pointer path; `-=` stored as
  // the negated term), each value times M
  const double numberParallel = PRM(XG_M1_M);
#undef PRM
  Terms T{io.terms + t.term0, n};
  const bool cap_on = f.tranop || f.acop || f.transient;
  const double gcgd = cap_on ? Capgd : 0.0, gcgs = cap_on ? Capgs : 0.0, gcgb = cap_on ? Capgb : 0.0;
  const double gcbs = cap_on ? capbs : 0.0, gcbd = cap_on ? capbd : 0.0;
  const bool caps = wild || ne0(gcgd) || ne0(gcgs) || ne0(gcgb) || ne0(gcbs) || ne0(gcbd);
  auto stamp = [&](auto times) {
    auto put = [&](int q, double v) { T.put(q, i, times(v)); };
    auto both = [&](int q, int r, double v) {  // v and -v
      const double a = times(v);
      T.put(q, i, a);
      T.put(r, i, -a);
    };
    const double ceqbs = flip(cbs, pol), ceqbd = flip(cbd, pol);
    put(0, ne0(drainConductance) ? Idrain : 0.0);
    put(1, 0.0);
    put(2, ne0(sourceConductance) ? Isource : 0.0);
    put(3, ceqbs + ceqbd);
    put(4, -Idrain - (ceqbd - cdreq));
    put(5, -Isource - (ceqbs + cdreq));
    put(6, flip(qgs + qgd + qgb, pol));
    put(7, flip(qbs + qbd - qgb, pol));
    put(8, -flip(qbd + qgd, pol));
    put(9, -flip(qbs + qgs, pol));
    if (!origFlag) {
      const double dvgs = vgs - vgs_orig, dvgd = vgd - vgd_orig, dvbs = vbs - vbs_orig;
      const double dvbd = vbd - vbd_orig, dvds = vds - vds_orig;
      const double dvg = fwd ? dvgs : dvgd, dvb = fwd ? dvbs : dvbd;
      const double jd = (gbd - gmin) * dvbd, js = (gbs - gmin) * dvbs;
      put(10, flip(jd + js, pol));
      put(11, flip(-jd + gds * dvds + Gm * dvg + Gmbs * dvb, pol));
      put(12, flip(-js - gds * dvds - Gm * dvg - Gmbs * dvb, pol));
      if (!caps) {
#pragma unroll
        for (int q = 13; q <= 16; ++q) T.put(q, i, 0.0);
      } else {
        const double dvgsb = vgs - vgs_orig - vbs + vbs_orig;
        put(13, flip(gcgd * dvgd + gcgs * dvgs + gcgb * dvgsb, pol));
        put(14, flip(-gcgb * dvgsb + gcgb * dvbd + gcbs * dvbs, pol));
        put(15, flip(-gcgd * dvgd - gcbd * dvbd, pol));
        put(16, flip(-gcgs * dvgs - gcbs * dvbs, pol));
      }
    } else {
#pragma unroll
      for (int q = 10; q <= 16; ++q) T.put(q, i, 0.0);
    }
    both(17, 18, drainConductance);
    both(19, 20, sourceConductance);
    put(21, gbs + gbd);
    put(22, -gbd);
    put(23, -gbs);
    put(24, -drainConductance);
    both(25, 29, Gm);
    put(26, -gbd + Gmbs);
    put(27, drainConductance + gds + gbd + revsum);
    put(28, -gds - nrmsum);
    put(30, -sourceConductance);
    put(31, -(gbs + Gmbs));
    put(32, -(gds + revsum));
    put(33, sourceConductance + gds + gbs + nrmsum);
    if (!caps) {
#pragma unroll
      for (int q = 34; q <= 47; ++q) T.put(q, i, 0.0);
      return;
    }
    put(34, gcgd + gcgs + gcgb);
    put(35, -gcgb);
    put(36, -gcgd);
    put(37, -gcgs);
    put(38, -gcgb);
    put(39, gcbs + gcbd + gcgb);
    put(40, -gcbd);
    put(41, -gcbs);
    put(42, -gcgd);
    put(43, -gcbd);
    put(44, gcbd + gcgd);
    put(45, -gcgs);
    put(46, -gcbs);
    put(47, gcbs + gcgs);
  };
  if (numberParallel == 1.0) stamp([](double v) { return v; });
  else stamp([&](double v) { return v * numberParallel; });
}

#include "bsim3_eval.cuh"

// ---- launches ------------------------------------------------------------------
__global__ void __launch_bounds__(256) res_kernel(DevType t, LoadIO io) {
  res_one<true>(t, io, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(256) cap_kernel(DevType t, LoadIO io) {
  cap_one<true>(t, io, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(256) vsrc_kernel(DevType t, Flags f, LoadIO io) {
  vsrc_one<true>(t, f, io, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(256) isrc_kernel(DevType t, Flags f, LoadIO io) {
  isrc_one<true>(t, f, io, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(256) diode_kernel(DevType t, DevOptions o, Flags f, LoadIO io) {
  diode_one<true>(t, o, f, io, blockIdx.x * blockDim.x + threadIdx.x);
}
__global__ void __launch_bounds__(128) mos1_kernel(DevType t, DevOptions o, Flags f, LoadIO io) {
  mos1_one<true>(t, o, f, io, blockIdx.x * blockDim.x + threadIdx.x);
}

// All light types of a small circuit in one launch: where every instance is
// resident at once a launch per type costs its start and its slowest warp in
// turn.  Blocks of one warp spread the MOSFETs' FP64 instructions, 66 cycles
// each on a sub-partition, over as many SMs as there are.  The MOSFETs' blocks
// come first.  A load of a 101-stage chain (sources, MOSFETs, capacitors):
// 26.6 us with three launches, 18.3 us with one, 13.6 us with the reduction
// close behind it (xg_launch.cuh); above one wave of warps the launches' cost
// no longer shows.
constexpr int kFewThreads = 32, kFewWarpsPerSm = 16;
struct FewArgs {
  int count;
  int type[XG_NUM_DEV_TYPES], block0[XG_NUM_DEV_TYPES + 1];
  DevType t[XG_NUM_DEV_TYPES];
  DevOptions o;
  Flags f;
  LoadIO io;
};
__global__ void __launch_bounds__(kFewThreads) few_kernel(const __grid_constant__ FewArgs a) {
  int k = 0;
  while (k + 1 < a.count && (int)blockIdx.x >= a.block0[k + 1]) ++k;
  const int i = ((int)blockIdx.x - a.block0[k]) * kFewThreads + (int)threadIdx.x;
  const DevType t = a.t[k];
  await_previous();
  switch (a.type[k]) {
    case XG_DEV_RES: res_one<false>(t, a.io, i); break;
    case XG_DEV_CAP: cap_one<false>(t, a.io, i); break;
    case XG_DEV_VSRC: vsrc_one<false>(t, a.f, a.io, i); break;
    case XG_DEV_ISRC: isrc_one<false>(t, a.f, a.io, i); break;
    case XG_DEV_DIODE: diode_one<false>(t, a.o, a.f, a.io, i); break;
    default: mos1_one<false>(t, a.o, a.f, a.io, i); break;
  }
}


// ---- fixed-order reduction ---------------------------------------------------
// Each output is the sum of its terms in the reference's statement order,
// s = ((0 + t1) + t2) + ..., so the result is bit-identical to a serial load.
// Short outputs take a thread each.  Outputs with more than kLongSegment
// terms (a supply node collects a term from every device on it) take a warp
// each: the warp gathers the terms, 256 at a time, into shared memory with
// independent loads, and one lane adds them in order.  Blocks [0, long_blocks)
// serve the long outputs, the rest the short ones.
constexpr int kRedThreads = 256;
constexpr int kRedWarps = kRedThreads / 32;
constexpr int kRedChunk = 256;

__global__ void __launch_bounds__(kRedThreads) reduce_kernel(ReduceArgs a, int long_blocks) {
  if ((int)blockIdx.x < long_blocks) {
    await_previous();
#if XG_SPLIT_SUMS
    // a block per long output: every thread sums a strided share of its terms,
    // then a fixed butterfly per warp and the warps in order
    __shared__ double part[kRedWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t w = blockIdx.x; w < a.n_long; w += long_blocks) {
      const int64_t o = a.long_out[w];
      const int64_t b = __ldg(a.red_ptr + o), e = __ldg(a.red_ptr + o + 1);
      double s = 0.0;
#pragma unroll 4
      for (int64_t j = b + threadIdx.x; j < e; j += blockDim.x)
        s += a.terms[__ldg(a.red_idx + j)];
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
      if (lane == 0) part[wid] = s;
      __syncthreads();
      if (threadIdx.x == 0) {
        double t = part[0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) t += part[k];
        a.out[o] = t;
      }
      __syncthreads();
    }
    return;
#else
    __shared__ double buf[kRedWarps][kRedChunk];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t w = (int64_t)blockIdx.x * kRedWarps + wid; w < a.n_long;
         w += (int64_t)long_blocks * kRedWarps) {
      const int64_t o = a.long_out[w];
      const int64_t b = __ldg(a.red_ptr + o), e = __ldg(a.red_ptr + o + 1);
      double s = 0.0;
      for (int64_t base = b; base < e; base += kRedChunk) {
        const int cnt = (int)(e - base < kRedChunk ? e - base : kRedChunk);
        for (int j = lane; j < cnt; j += 32)
          buf[wid][j] = a.terms[__ldg(a.red_idx + base + j)];
        __syncwarp();
        if (lane == 0)
          for (int j = 0; j < cnt; ++j) s += buf[wid][j];
        __syncwarp();
      }
      if (lane == 0) a.out[o] = s;
    }
    return;
#endif
  }
  // two short outputs per thread (kEllThreads apart), their bucket found by
  // the block; every term number loaded coalesced, the two outputs' term
  // loads interleaved so that twice as many are in flight, each output
  // summed in its own order
  static_assert(kEllPerThread == 2, "the loop below takes two outputs per thread");
  const int64_t g = a.ell_block0 + ((int64_t)blockIdx.x - long_blocks);
  int lo = a.b0, hi = a.b1 - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&a.ell[mid].block0) <= g) lo = mid;
    else hi = mid - 1;
  }
  const EllBucket B = a.ell[lo];
  const int64_t k0 = (g - B.block0) * kEllPerBlock + threadIdx.x, k1 = k0 + kEllThreads;
  const uint32_t *ix = a.ell_idx + B.idx0;
  await_previous();
  if (k0 >= B.m) return;
  if (k1 < B.m) {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
    for (int j = 0; j < B.c; ++j) {
      const int64_t row = (int64_t)j * B.m;
      const double t0 = a.terms[__ldg(ix + row + k0)];
      const double t1 = a.terms[__ldg(ix + row + k1)];
      s0 += t0;
      s1 += t1;
    }
    a.out[__ldg(a.ell_out + B.out0 + k0)] = s0;
    a.out[__ldg(a.ell_out + B.out0 + k1)] = s1;
  } else {
    double s = 0.0;
#pragma unroll 8
    for (int j = 0; j < B.c; ++j) s += a.terms[__ldg(ix + (int64_t)j * B.m + k0)];
    a.out[__ldg(a.ell_out + B.out0 + k0)] = s;
  }
}

int grid_for(int64_t n, int block) { return (int)((n + block - 1) / block); }

}  // namespace

static int launch_type(int dev_type, const DevType &t, const DevOptions &o, const Flags &f, const LoadIO &io,
                       void *stream) {
  if (t.n <= 0) return XG_OK;
  cudaStream_t s = (cudaStream_t)stream;
  switch (dev_type) {
    case XG_DEV_RES: res_kernel<<<grid_for(t.n, 256), 256, 0, s>>>(t, io); xg::count_launches(1); break;
    case XG_DEV_CAP: cap_kernel<<<grid_for(t.n, 256), 256, 0, s>>>(t, io); xg::count_launches(1); break;
    case XG_DEV_VSRC: vsrc_kernel<<<grid_for(t.n, 256), 256, 0, s>>>(t, f, io); xg::count_launches(1); break;
    case XG_DEV_ISRC: isrc_kernel<<<grid_for(t.n, 256), 256, 0, s>>>(t, f, io); xg::count_launches(1); break;
    case XG_DEV_DIODE: diode_kernel<<<grid_for(t.n, 256), 256, 0, s>>>(t, o, f, io); xg::count_launches(1); break;
    case XG_DEV_MOS1: mos1_kernel<<<grid_for(t.n, 128), 128, 0, s>>>(t, o, f, io); xg::count_launches(1); break;
    case XG_DEV_BSIM3: bsim3_kernel<<<grid_for(t.n, 128), 128, 0, s>>>(t, o, f, io); xg::count_launches(1); break;
    default: return XG_ERR_UNSUPPORTED;
  }
  return cudaGetLastError() == cudaSuccess ? XG_OK : XG_ERR_CUDA;
}

// Evaluates the given types: one launch for the light ones where they leave
// every SM at most kFewWarpsPerSm warps and there are two or more, else a
// launch each.
int launch_evals(const EvalType *types, int n, const DevOptions &o, const Flags &f, const LoadIO &io, void *stream) {
  FewArgs a;
  a.count = 0;
  int64_t blocks = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int k = 0; k < n; ++k) {
      const EvalType &e = types[k];
      if (e.t.n <= 0 || e.type == XG_DEV_BSIM3 || (e.type == XG_DEV_MOS1) != (pass == 0)) continue;
      if (e.type < 0 || e.type >= XG_NUM_DEV_TYPES || a.count >= XG_NUM_DEV_TYPES) return XG_ERR_UNSUPPORTED;
      a.type[a.count] = e.type;
      a.block0[a.count] = (int)std::min<int64_t>(blocks, INT32_MAX);
      a.t[a.count++] = e.t;
      blocks += (e.t.n + kFewThreads - 1) / kFewThreads;
    }
  const bool few = a.count > 1 && blocks <= (int64_t)sm_count() * kFewWarpsPerSm;
  if (few) {
    a.o = o;
    a.f = f;
    a.io = io;
    if (launch_close(few_kernel, blocks, kFewThreads, 0, 0, (cudaStream_t)stream, a) != cudaSuccess)
      return XG_ERR_CUDA;
  }
  for (int k = 0; k < n; ++k) {
    if (few && types[k].type != XG_DEV_BSIM3) continue;
    const int rc = launch_type(types[k].type, types[k].t, o, f, io, stream);
    if (rc) return rc;
  }
  return XG_OK;
}

int launch_reduce(const ReduceArgs &a, void *stream) {
  if (a.n_long <= 0 && a.ell_blocks <= 0) return XG_OK;
  const int sms = sm_count();
  const int64_t grid = a.ell_blocks;  // one thread per short output
  static_assert(kEllThreads == kRedThreads, "the ELL buckets are cut in blocks of the reduction's size");
#if XG_SPLIT_SUMS
  const int long_blocks = (int)std::min<int64_t>(a.n_long, sms * 8);  // a block per long output
#else
  const int long_blocks = (int)std::min<int64_t>((a.n_long + kRedWarps - 1) / kRedWarps, sms * 8);
#endif
  if (grid + long_blocks <= 0) return XG_OK;
  return launch_close(reduce_kernel, grid + long_blocks, kRedThreads, 0, 0, (cudaStream_t)stream, a, long_blocks) ==
                 cudaSuccess
             ? XG_OK
             : XG_ERR_CUDA;
}

}  // namespace XG_NS
}  // namespace xg
