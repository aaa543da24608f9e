// One-electron matrix H, two-electron integrals W and core-core repulsion on
// the GPU for sp atoms under PM7 -- the step before the SCF path
// (integrals/hcore.F90:150-297 with rotate -> rotatd, reppd, spcore, elenuc,
// ccrep, h1elec -> diat/diat2/set/coe, wstore; integrals/mndod.F90).
//
//   hcore_pairs  one thread per atom pair (i > j): the W block in the
//                reference layout (i's pair index outer, j's inner), the
//                resonance block H(i-orbitals, j-orbitals) and the pair's
//                core-core energy.
//   hcore_diag   one warp per atom A: A's diagonal H block, accumulating
//                U_ss/U_pp and the electron-core terms of every partner in
//                the reference's order (partners below A, then above A), and
//                the one-centre W block (wstore).
//   enuc_sum     fixed-order reduction of the pair energies.
#include <algorithm>

#include "mb_common.cuh"
#include "pm7_params.h"

namespace {

struct DevParams {
  Pm7Elem el[9];
  double xfac[9][9], alpb[9][9];
  double par1, par2, par3, par4;
};
__constant__ DevParams c_P;

__constant__ double c_fact[18] = {1.0, 1.0, 2.0, 6.0, 24.0, 120.0, 720.0, 5040.0, 40320.0, 362880.0,
                                  3628800.0, 39916800.0, 479001600.0, 6227020800.0, 87178291200.0,
                                  1307674368000.0, 20922789888000.0, 355687428096000.0};

__device__ __forceinline__ double ipow(double x, int m) {
  double r = 1.0;
  for (int i = 0; i < m; ++i) r *= x;
  return r;
}

// The pair functions below are templates on the two atoms' orbital counts (1 or 4):
// with constant loop bounds every array is in registers (before, 3 KB of local
// memory a thread; hcore_pairs of (H2O)512 took 8.5 ms, now 1.4, one B200).
// by_kind picks the instance of a pair.  Where a sum of two products could be
// contracted either way, it is written out, so a value does not depend on the
// kernel its function is inlined into.
template <int N>
struct Orb {
  static constexpr int n = N;
};
template <class F>
__device__ __forceinline__ void by_kind(int ni, int nj, F&& f) {
  if (c_P.el[ni].natorb == 1) {
    if (c_P.el[nj].natorb == 1) f(Orb<1>{}, Orb<1>{});
    else f(Orb<1>{}, Orb<4>{});
  } else {
    if (c_P.el[nj].natorb == 1) f(Orb<4>{}, Orb<1>{});
    else f(Orb<4>{}, Orb<4>{});
  }
}

// ------------------------------------------------------------ overlaps
template <int K>
struct Ovl {
  double a[K + 2], b[K + 2], sa, sb;  // from 1
};

template <int K>
__device__ __forceinline__ void aintgs(Ovl<K>& o, double x) {
  const double c = exp(-x);
  o.a[1] = c / x;
#pragma unroll
  for (int i = 1; i <= K; ++i) o.a[i + 1] = (o.a[i] * i + c) / x;
}

template <int K>
__device__ __forceinline__ void bintgs(Ovl<K>& o, double x) {
  const double ax = fabs(x);
  int last = 0, mode = 0;
  if (ax > 3.0) mode = 0;
  else if (ax > 2.0) { if (K <= 10) mode = 0; else { last = 15; mode = 1; } }
  else if (ax > 1.0) { if (K <= 7) mode = 0; else { last = 12; mode = 1; } }
  else if (ax > 0.5) { if (K <= 5) mode = 0; else { last = 7; mode = 1; } }
  else if (ax <= 1.0e-6) mode = 2;
  else { last = 6; mode = 1; }
  if (mode == 0) {
    const double expx = exp(x), expmx = 1.0 / expx;
    o.b[1] = (expx - expmx) / x;
#pragma unroll
    for (int i = 1; i <= K; ++i) o.b[i + 1] = (i * o.b[i] + ((i & 1) ? -1.0 : 1.0) * expx - expmx) / x;
  } else if (mode == 1) {
    // sum over m of (-x)^m 2 / (m! (m + i + 1)), m + i even, in ascending m
#pragma unroll
    for (int i = 0; i <= K; ++i) o.b[i + 1] = 0.0;
    double pw = 1.0;
    for (int m = 0; m <= last; ++m) {
      const double xf = m != 0 ? c_fact[m] : 1.0;
#pragma unroll
      for (int i = 0; i <= K; ++i)
        if (((m + i) & 1) == 0) o.b[i + 1] = o.b[i + 1] + pw * 2.0 / (xf * (double)(m + i + 1));
      pw *= -x;
    }
  } else {
#pragma unroll
    for (int i = 0; i <= K; ++i) o.b[i + 1] = (double)(2 * ((i + 1) % 2)) / (i + 1.0);
  }
}

// swap: the first atom has the higher atomic number
template <int K>
__device__ __forceinline__ void set_ovl(Ovl<K>& o, double s1, double s2, bool swap, double rab) {
  o.sa = swap ? s2 : s1;
  o.sb = swap ? s1 : s2;
  aintgs(o, 0.5 * rab * (o.sa + o.sb));
  bintgs(o, 0.5 * rab * (o.sb - o.sa));
}

// Local overlaps of first-row sp atoms (diat2 cases 1, 2, 4).
struct Overlap {
  double ss, sp, ps, pps, ppp;  // first atom's orbital first; pps sigma, ppp pi
};
template <int NI, int NJ>
__device__ __forceinline__ Overlap diat2(int na, double esa, double epa, double r12, int nb, double esb, double epb) {
  Overlap s{0.0, 0.0, 0.0, 0.0, 0.0};
  const double rab = r12 / PM7_A0;
  if constexpr (NI == 1 && NJ == 1) {
    Ovl<2> o;
    const double *a = o.a, *b = o.b;
    set_ovl(o, esa, esb, na > nb, rab);
    s.ss = 0.25 * sqrt(ipow(o.sa * o.sb * rab * rab, 3)) * (a[3] * b[1] - b[3] * a[1]);
  } else if constexpr (NI == 1 || NJ == 1) {
    Ovl<3> o;
    const double *a = o.a, *b = o.b;
    set_ovl(o, esa, esb, NI > 1, rab);
    const double rab4 = ipow(rab, 4) * 0.125;
    double w = sqrt(ipow(o.sa, 3) * ipow(o.sb, 5)) * rab4;
    s.ss = w * sqrt(1.0 / 3.0) * (a[4] * b[1] - b[4] * a[1] + a[3] * b[2] - b[3] * a[2]);
    set_ovl(o, NI > 1 ? epa : esa, NI > 1 ? esb : epb, NI > 1, rab);
    w = sqrt(ipow(o.sa, 3) * ipow(o.sb, 5)) * rab4;
    const double v = w * (a[3] * b[1] - b[3] * a[1] + a[4] * b[2] - b[4] * a[2]);
    if (NI > 1) s.ps = v;
    else s.sp = v;
  } else {
    Ovl<4> o;
    const double *a = o.a, *b = o.b;
    const bool swap = na > nb;
    set_ovl(o, esa, esb, swap, rab);
    const double rab4 = ipow(rab, 5) * 0.0625;
    double w = sqrt(ipow(o.sa * o.sb, 5)) * rab4;
    s.ss = w * (a[5] * b[1] + b[5] * a[1] - 2.0 * a[3] * b[3]) / 3.0;
    set_ovl(o, swap ? epa : esa, swap ? esb : epb, swap, rab);
    w = sqrt(ipow(o.sa * o.sb, 5)) * rab4;
    const double rt3 = 1.0 / sqrt(3.0);
    double d = a[4] * (b[1] - b[3]) - a[2] * (b[3] - b[5]);
    double e = b[4] * (a[1] - a[3]) - b[2] * (a[3] - a[5]);
    const double u = w * rt3 * (d + e);
    set_ovl(o, swap ? esa : epa, swap ? epb : esb, swap, rab);
    w = sqrt(ipow(o.sa * o.sb, 5)) * rab4;
    d = a[4] * (b[1] - b[3]) - a[2] * (b[3] - b[5]);
    e = b[4] * (a[1] - a[3]) - b[2] * (a[3] - a[5]);
    const double v = w * rt3 * (d - e);
    s.sp = swap ? v : u;
    s.ps = swap ? u : v;
    set_ovl(o, epa, epb, swap, rab);
    w = sqrt(ipow(o.sa * o.sb, 5)) * rab4;
    s.pps = -w * (b[3] * (a[5] + a[1]) - a[3] * (b[5] + b[1]));
    s.ppp = 0.5 * w * (a[5] * (b[1] - b[3]) - b[5] * (a[1] - a[3]) - a[3] * b[1] + b[3] * a[1]);
  }
  return s;
}

// Resonance block di[a][b] (orbitals s, px, py, pz) of atom i (a) with atom j (b)
// at xj - xi.
template <int NI, int NJ>
__device__ __forceinline__ void h1elec(int ni, int nj, const double* xi, const double* xj, double (&di)[NI][NJ]) {
#pragma unroll
  for (int a = 0; a < NI; ++a)
#pragma unroll
    for (int b = 0; b < NJ; ++b) di[a][b] = 0.0;
  const double x2 = xj[0] - xi[0], y2 = xj[1] - xi[1], z2 = xj[2] - xi[2];
  const double rr = x2 * x2 + y2 * y2 + z2 * z2;
  if (rr > 1.0e4 || rr >= 225.0) return;  // cutofs (h1elec) and cutof1 (diat)
  double xy = x2 * x2 + y2 * y2;
  const double r = sqrt(xy + z2 * z2);
  xy = sqrt(xy);
  double ca, cb, sa, sb;
  if (xy >= 1.0e-10) { ca = x2 / xy; cb = z2 / r; sa = y2 / xy; sb = xy / r; }
  else if (z2 < 0.0) { ca = -1.0; cb = -1.0; sa = 0.0; sb = 0.0; }
  else if (z2 == 0.0) { ca = 0.0; cb = 0.0; sa = 0.0; sb = 0.0; }
  else { ca = 1.0; cb = 1.0; sa = 0.0; sb = 0.0; }
  if (r < 0.001) return;
  // px, py, pz along sigma, pi, pi'
  const double cs[4] = {0.0, ca * sb, sa * sb, cb}, cp[4] = {0.0, ca * cb, sa * cb, -sb}, cq[4] = {0.0, -sa, ca, 0.0};
  const Pm7Elem& A = c_P.el[ni];
  const Pm7Elem& B = c_P.el[nj];
  const Overlap s = diat2<NI, NJ>(ni, A.zs, A.zp, r, nj, B.zs, B.zp);
#pragma unroll
  for (int a = 0; a < NI; ++a)
#pragma unroll
    for (int b = 0; b < NJ; ++b) {
      double v;
      if (a == 0 && b == 0) v = s.ss;
      else if (a == 0) v = -(s.sp * cs[b]);
      else if (b == 0) v = s.ps * cs[a];
      else v = __fma_rn(s.ppp, __fma_rn(cp[a], cp[b], __dmul_rn(cq[a], cq[b])), -__dmul_rn(s.pps, __dmul_rn(cs[a], cs[b])));
      di[a][b] = v * ((a == 0 ? A.betas : A.betap) * 0.5 + (b == 0 ? B.betas : B.betap) * 0.5);
    }
}

// ------------------------------------------------------- local integrals
__device__ __forceinline__ void to_point(double r, double* point, double* cst) {
  *point = PM7_EV * PM7_A0 / r;
  *cst = (r < 7.0) ? 1.0 - exp(-(r - 7.0) * (r - 7.0) * 0.22) : 0.0;
}

// 22 local-frame repulsion integrals (reppd, l_feather) and G_AB.
template <int NI, int NJ>
__device__ __forceinline__ void reppd(int ni, int nj, double rij, double ri[23], double* gab) {
  const double ev1 = PM7_EV / 2, ev2 = ev1 / 2, ev3 = ev2 / 2, ev4 = ev3 / 2, td = 2.0, pp = 0.5;
#pragma unroll
  for (int i = 0; i < 23; ++i) ri[i] = 0.0;
  const Pm7Elem& A = c_P.el[ni];
  const Pm7Elem& B = c_P.el[nj];
  const double r = rij / PM7_A0;
  constexpr bool si = NI == 4, sj = NJ == 4;
  const double rsq = __dmul_rn(r, r);
  double aee = A.po9 + B.po9;
  *gab = PM7_EV / sqrt(__fma_rn(aee, aee, rsq));
  aee = pp / A.am + pp / B.am;
  aee = __dmul_rn(aee, aee);
  if constexpr (!si && !sj) {
    ri[1] = PM7_EV / sqrt(rsq + aee);
  } else if constexpr (si && !sj) {
    const double da = A.dd, qa = A.qq * td;
    double ade = pp / A.ad + pp / B.am; ade *= ade;
    double aqe = pp / A.aq + pp / B.am; aqe *= aqe;
    const double s1 = sqrt(rsq + aee), s2 = sqrt((r + da) * (r + da) + ade), s3 = sqrt((r - da) * (r - da) + ade),
                 s4 = sqrt((r + qa) * (r + qa) + aqe), s5 = sqrt((r - qa) * (r - qa) + aqe), a6 = rsq + aqe,
                 s6 = sqrt(a6), s7 = sqrt(a6 + qa * qa);
    const double ee = PM7_EV / s1;
    ri[1] = ee;
    ri[2] = ev1 / s2 - ev1 / s3;
    ri[3] = ee + ev2 / s4 + ev2 / s5 - ev1 / s6;
    ri[4] = ee + ev1 / s7 - ev1 / s6;
  } else if constexpr (!si && sj) {
    const double db = B.dd, qb = B.qq * td;
    double aed = pp / A.am + pp / B.ad; aed *= aed;
    double aeq = pp / A.am + pp / B.aq; aeq *= aeq;
    const double s1 = sqrt(rsq + aee), s2 = sqrt((r - db) * (r - db) + aed), s3 = sqrt((r + db) * (r + db) + aed),
                 s4 = sqrt((r - qb) * (r - qb) + aeq), s5 = sqrt((r + qb) * (r + qb) + aeq), a6 = rsq + aeq,
                 s6 = sqrt(a6), s7 = sqrt(a6 + qb * qb);
    const double ee = PM7_EV / s1;
    ri[1] = ee;
    ri[5] = ev1 / s2 - ev1 / s3;
    ri[11] = ee + ev2 / s4 + ev2 / s5 - ev1 / s6;
    ri[12] = ee + ev1 / s7 - ev1 / s6;
  } else {
    const double da = A.dd, db = B.dd;
    double qa = A.qq * td, qb = B.qq * td;
    double ade = pp / A.ad + pp / B.am; ade *= ade;
    double aqe = pp / A.aq + pp / B.am; aqe *= aqe;
    double aed = pp / A.am + pp / B.ad; aed *= aed;
    double aeq = pp / A.am + pp / B.aq; aeq *= aeq;
    double axx = pp / A.ad + pp / B.ad; axx *= axx;
    double adq = pp / A.ad + pp / B.aq; adq *= adq;
    double aqd = pp / A.aq + pp / B.ad; aqd *= aqd;
    double aqq = pp / A.aq + pp / B.aq; aqq *= aqq;
    double sq[73];
    double xxx, yyy, zzz, www;
#define SQ(i, v) sq[i] = sqrt(v)
    SQ(1, rsq + aee);
    xxx = r + da; SQ(2, xxx * xxx + ade);
    xxx = r - da; SQ(3, xxx * xxx + ade);
    xxx = r - qa; SQ(4, xxx * xxx + aqe);
    xxx = r + qa; SQ(5, xxx * xxx + aqe);
    double a6 = rsq + aqe; SQ(6, a6);
    SQ(7, a6 + qa * qa);
    xxx = r - db; SQ(8, xxx * xxx + aed);
    xxx = r + db; SQ(9, xxx * xxx + aed);
    xxx = r - qb; SQ(10, xxx * xxx + aeq);
    xxx = r + qb; SQ(11, xxx * xxx + aeq);
    double a12 = rsq + aeq; SQ(12, a12);
    SQ(13, a12 + qb * qb);
    xxx = da - db; SQ(14, rsq + axx + xxx * xxx);
    xxx = da + db; SQ(15, rsq + axx + xxx * xxx);
    xxx = r + da - db; SQ(16, xxx * xxx + axx);
    xxx = r - da + db; SQ(17, xxx * xxx + axx);
    xxx = r - da - db; SQ(18, xxx * xxx + axx);
    xxx = r + da + db; SQ(19, xxx * xxx + axx);
    xxx = r + da; double a20 = xxx * xxx + adq; SQ(20, a20);
    SQ(21, a20 + qb * qb);
    xxx = r - da; double a22 = xxx * xxx + adq; SQ(22, a22);
    SQ(23, a22 + qb * qb);
    xxx = r - db; double a24 = xxx * xxx + aqd; SQ(24, a24);
    SQ(25, a24 + qa * qa);
    xxx = r + db; double a26 = xxx * xxx + aqd; SQ(26, a26);
    SQ(27, a26 + qa * qa);
    xxx = r + da - qb; SQ(28, xxx * xxx + adq);
    xxx = r - da - qb; SQ(29, xxx * xxx + adq);
    xxx = r + da + qb; SQ(30, xxx * xxx + adq);
    xxx = r - da + qb; SQ(31, xxx * xxx + adq);
    xxx = r + qa - db; SQ(32, xxx * xxx + aqd);
    xxx = r + qa + db; SQ(33, xxx * xxx + aqd);
    xxx = r - qa - db; SQ(34, xxx * xxx + aqd);
    xxx = r - qa + db; SQ(35, xxx * xxx + aqd);
    const double a36 = rsq + aqq; SQ(36, a36);
    xxx = qa - qb; SQ(37, a36 + xxx * xxx);
    xxx = qa + qb; SQ(38, a36 + xxx * xxx);
    const double a39 = a36 + qa * qa; SQ(39, a39);
    SQ(40, a36 + qb * qb);
    SQ(41, a39 + qb * qb);
    xxx = r - qb; double a42 = xxx * xxx + aqq; SQ(42, a42);
    SQ(43, a42 + qa * qa);
    xxx = r + qb; double a44 = xxx * xxx + aqq; SQ(44, a44);
    SQ(45, a44 + qa * qa);
    xxx = r + qa; double a46 = xxx * xxx + aqq; SQ(46, a46);
    SQ(47, a46 + qb * qb);
    xxx = r - qa; double a48 = xxx * xxx + aqq; SQ(48, a48);
    SQ(49, a48 + qb * qb);
    xxx = r + qa - qb; SQ(50, xxx * xxx + aqq);
    xxx = r + qa + qb; SQ(51, xxx * xxx + aqq);
    xxx = r - qa - qb; SQ(52, xxx * xxx + aqq);
    xxx = r - qa + qb; SQ(53, xxx * xxx + aqq);
    qa = A.qq;
    qb = B.qq;
    xxx = da - qb; xxx = xxx * xxx;
    yyy = r - qb; yyy = yyy * yyy;
    zzz = da + qb; zzz = zzz * zzz;
    www = r + qb; www = www * www;
    SQ(54, xxx + yyy + adq);
    SQ(55, xxx + www + adq);
    SQ(56, zzz + yyy + adq);
    SQ(57, zzz + www + adq);
    xxx = qa - db; xxx = xxx * xxx;
    yyy = qa + db; yyy = yyy * yyy;
    zzz = r + qa; zzz = zzz * zzz;
    www = r - qa; www = www * www;
    SQ(58, zzz + xxx + aqd);
    SQ(59, www + xxx + aqd);
    SQ(60, zzz + yyy + aqd);
    SQ(61, www + yyy + aqd);
    xxx = qa - qb; xxx = xxx * xxx;
    yyy = qa + qb; yyy = yyy * yyy;
    zzz = r + qa - qb; zzz = zzz * zzz;
    SQ(65, zzz + xxx + aqq);
    SQ(66, zzz + yyy + aqq);
    zzz = r + qa + qb; zzz = zzz * zzz;
    SQ(67, zzz + xxx + aqq);
    SQ(68, zzz + yyy + aqq);
    zzz = r - qa - qb; zzz = zzz * zzz;
    SQ(69, zzz + xxx + aqq);
    SQ(70, zzz + yyy + aqq);
    zzz = r - qa + qb; zzz = zzz * zzz;
    SQ(71, zzz + xxx + aqq);
    SQ(72, zzz + yyy + aqq);
#undef SQ
    const double ee = PM7_EV / sq[1];
    const double dze = (-ev1 / sq[2]) + ev1 / sq[3];
    const double qzze = ev2 / sq[4] + ev2 / sq[5] - ev1 / sq[6];
    const double qxxe = ev1 / sq[7] - ev1 / sq[6];
    const double edz = (-ev1 / sq[8]) + ev1 / sq[9];
    const double eqzz = ev2 / sq[10] + ev2 / sq[11] - ev1 / sq[12];
    const double eqxx = ev1 / sq[13] - ev1 / sq[12];
    const double dxdx = ev1 / sq[14] - ev1 / sq[15];
    const double dzdz = ev2 / sq[16] + ev2 / sq[17] - ev2 / sq[18] - ev2 / sq[19];
    const double dzqxx = ev2 / sq[20] - ev2 / sq[21] - ev2 / sq[22] + ev2 / sq[23];
    const double qxxdz = ev2 / sq[24] - ev2 / sq[25] - ev2 / sq[26] + ev2 / sq[27];
    const double dzqzz = (-ev3 / sq[28]) + ev3 / sq[29] - ev3 / sq[30] + ev3 / sq[31] - ev2 / sq[22] + ev2 / sq[20];
    const double qzzdz = (-ev3 / sq[32]) + ev3 / sq[33] - ev3 / sq[34] + ev3 / sq[35] + ev2 / sq[24] - ev2 / sq[26];
    const double qxxqxx = ev3 / sq[37] + ev3 / sq[38] - ev2 / sq[39] - ev2 / sq[40] + ev2 / sq[36];
    const double qxxqyy = ev2 / sq[41] - ev2 / sq[39] - ev2 / sq[40] + ev2 / sq[36];
    const double qxxqzz = ev3 / sq[43] + ev3 / sq[45] - ev3 / sq[42] - ev3 / sq[44] - ev2 / sq[39] + ev2 / sq[36];
    const double qzzqxx = ev3 / sq[47] + ev3 / sq[49] - ev3 / sq[46] - ev3 / sq[48] - ev2 / sq[40] + ev2 / sq[36];
    const double qzzqzz = ev4 / sq[50] + ev4 / sq[51] + ev4 / sq[52] + ev4 / sq[53] - ev3 / sq[48] - ev3 / sq[46] -
                          ev3 / sq[42] - ev3 / sq[44] + ev2 / sq[36];
    const double dxqxz = (-ev2 / sq[54]) + ev2 / sq[55] + ev2 / sq[56] - ev2 / sq[57];
    const double qxzdx = (-ev2 / sq[58]) + ev2 / sq[59] + ev2 / sq[60] - ev2 / sq[61];
    const double qxzqxz = ev3 / sq[65] - ev3 / sq[67] - ev3 / sq[69] + ev3 / sq[71] - ev3 / sq[66] + ev3 / sq[68] +
                          ev3 / sq[70] - ev3 / sq[72];
    ri[1] = ee; ri[2] = -dze; ri[3] = ee + qzze; ri[4] = ee + qxxe; ri[5] = -edz; ri[6] = dzdz; ri[7] = dxdx;
    ri[8] = (-edz) - qzzdz; ri[9] = (-edz) - qxxdz; ri[10] = -qxzdx; ri[11] = ee + eqzz; ri[12] = ee + eqxx;
    ri[13] = (-dze) - dzqzz; ri[14] = (-dze) - dzqxx; ri[15] = -dxqxz; ri[16] = ee + eqzz + qzze + qzzqzz;
    ri[17] = ee + eqzz + qxxe + qxxqzz; ri[18] = ee + eqxx + qzze + qzzqxx; ri[19] = ee + eqxx + qxxe + qxxqxx;
    ri[20] = qxzqxz; ri[21] = ee + eqxx + qxxe + qxxqyy; ri[22] = pp * (qxxqxx - qxxqyy);
  }
  double point, cst;
  to_point(rij, &point, &cst);
  const double far = __dmul_rn(1.0 - cst, point);
  const unsigned coul = (1u << 1) | (1u << 3) | (1u << 4) | (1u << 11) | (1u << 12) | (1u << 16) | (1u << 17) |
                        (1u << 18) | (1u << 19) | (1u << 21);
  const unsigned neg = (1u << 2) | (1u << 5) | (1u << 8) | (1u << 9) | (1u << 10) | (1u << 13) | (1u << 14) |
                       (1u << 15);
#pragma unroll
  for (int i = 1; i <= 22; ++i) {
    ri[i] = ((coul >> i) & 1u) ? __fma_rn(ri[i], cst, far) : __dmul_rn(ri[i], cst);
    if ((neg >> i) & 1u) ri[i] = -ri[i];
  }
  *gab = __fma_rn(*gab, cst, far);
}

// core[k][n]: electron-core attraction, local frame (spcore) with feathering.
template <int NI, int NJ>
__device__ __forceinline__ void core_terms(int ni, int nj, double rij, double core[5][3]) {
  const Pm7Elem& A = c_P.el[ni];
  const Pm7Elem& B = c_P.el[nj];
  const double pxy[8] = {0, 1.0, -0.5, -0.5, 0.5, 0.25, 0.25, 0.5};
#pragma unroll
  for (int x = 0; x < 5; ++x) core[x][1] = core[x][2] = 0.0;
  const double r = rij / PM7_A0, r2 = __dmul_rn(r, r);
  const double aci = A.po9, acj = B.po9;
  const double ssi = (aci + B.po1) * (aci + B.po1), ssj = (acj + A.po1) * (acj + A.po1);
  core[1][1] = -B.tore * PM7_EV / sqrt(r2 + ssj);
  core[1][2] = -A.tore * PM7_EV / sqrt(r2 + ssi);
  if constexpr (NI == 4) {
    const double ppj = (acj + A.po7) * (acj + A.po7), da = A.ddp2, qa = A.ddp3 / sqrt(2.0), twoqa = qa + qa;
    const double adj = (A.po2 + acj) * (A.po2 + acj), aqj = (A.po3 + acj) * (A.po3 + acj);
    double x[8];
    x[1] = r2 + ppj; x[2] = r2 + aqj; x[3] = (r + da) * (r + da) + adj; x[4] = (r - da) * (r - da) + adj;
    x[5] = (r - twoqa) * (r - twoqa) + aqj; x[6] = (r + twoqa) * (r + twoqa) + aqj; x[7] = r2 + twoqa * twoqa + aqj;
#pragma unroll
    for (int i = 1; i <= 7; ++i) x[i] = pxy[i] / sqrt(x[i]);
    core[2][1] = -B.tore * ((x[3] + x[4]) * PM7_EV);
    core[3][1] = -B.tore * ((x[1] + x[2] + x[5] + x[6]) * PM7_EV);
    core[4][1] = -B.tore * ((x[1] + x[2] + x[7]) * PM7_EV);
  }
  if constexpr (NJ == 4) {
    const double ppi = (aci + B.po7) * (aci + B.po7), db = B.ddp2, qb = B.ddp3 / sqrt(2.0), twoqb = qb + qb;
    const double adi = (B.po2 + aci) * (B.po2 + aci), aqi = (B.po3 + aci) * (B.po3 + aci);
    double x[8];
    x[1] = r2 + ppi; x[2] = r2 + aqi; x[3] = (r + db) * (r + db) + adi; x[4] = (r - db) * (r - db) + adi;
    x[5] = (r - twoqb) * (r - twoqb) + aqi; x[6] = (r + twoqb) * (r + twoqb) + aqi; x[7] = r2 + twoqb * twoqb + aqi;
#pragma unroll
    for (int i = 1; i <= 7; ++i) x[i] = pxy[i] / sqrt(x[i]);
    core[2][2] = -A.tore * (-(x[3] + x[4]) * PM7_EV);
    core[3][2] = -A.tore * ((x[1] + x[2] + x[5] + x[6]) * PM7_EV);
    core[4][2] = -A.tore * ((x[1] + x[2] + x[7]) * PM7_EV);
  }
  double point, cst;
  to_point(rij, &point, &cst);
  point = -(PM7_EV / r) * B.tore;
  core[1][1] = core[1][1] * cst + (1.0 - cst) * point;
  core[2][1] = core[2][1] * cst;
  core[3][1] = core[3][1] * cst + (1.0 - cst) * point;
  core[4][1] = core[4][1] * cst + (1.0 - cst) * point;
  point = -(PM7_EV / r) * A.tore;
  core[1][2] = core[1][2] * cst + (1.0 - cst) * point;
  core[2][2] = core[2][2] * cst;
  core[3][2] = core[3][2] * cst + (1.0 - cst) * point;
  core[4][2] = core[4][2] * cst + (1.0 - cst) * point;
}

// Rotation matrix of the pair axis (rotmat): p[k][m], k = local axis
// (sigma, pi, pi'), m = molecular x, y, z; returns the distance.
__device__ double rotmat(const double* ci, const double* cj, double p[4][4]) {
  const double x11 = cj[0] - ci[0], x22 = cj[1] - ci[1], x33 = cj[2] - ci[2];
  const double b = x11 * x11 + x22 * x22;
  const double r = sqrt(b + x33 * x33);
  const double sqb = sqrt(b);
  double sb = sqb / r, ca, sa, cb;
  if (sb > 1.0e-7) { ca = x11 / sqb; sa = x22 / sqb; cb = x33 / r; }
  else {
    sa = 0.0; sb = 0.0;
    if (x33 < 0.0) { ca = -1.0; cb = -1.0; }
    else if (x33 > 0.0) { ca = 1.0; cb = 1.0; }
    else { ca = 0.0; cb = 0.0; }
  }
  p[1][1] = ca * sb; p[2][1] = ca * cb; p[3][1] = -sa;
  p[1][2] = sa * sb; p[2][2] = sa * cb; p[3][2] = ca;
  p[1][3] = cb;      p[2][3] = -sb;     p[3][3] = 0.0;
  return r;
}

// pp(t, k, l) products of rotation rows (rotmat :1484-1501)
__device__ __forceinline__ double ppf(const double p[4][4], int t, int k, int l) {
  const int ta[7] = {0, 1, 2, 3, 1, 1, 2}, tb[7] = {0, 1, 2, 3, 2, 3, 3};
  const int a = ta[t], b = tb[t];
  if (k == l) return __dmul_rn(p[k][a], p[k][b]);
  if (t <= 3) return __dmul_rn(2.0 * p[k][a], p[l][a]);
  return __fma_rn(p[k][a], p[l][b], __dmul_rn(p[k][b], p[l][a]));
}

// The electron-core blocks e1b (atom i) / e2a (atom j), packed local order.
template <int NI, int NJ>
__device__ __forceinline__ void elenuc(const double p[4][4], const double core[5][3], double* e1b, double* e2a) {
  const int indpp[4][4] = {{0, 0, 0, 0}, {0, 1, 4, 5}, {0, 4, 2, 6}, {0, 5, 6, 3}};
#pragma unroll
  for (int nn = 1; nn <= 2; ++nn) {
    const int lim = nn == 1 ? NI : NJ;
    double* out = nn == 1 ? e1b : e2a;
#pragma unroll
    for (int a = 0; a < lim; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b) {
        double h;
        if (a == 0) h = core[1][nn];
        else if (b == 0) h = p[1][a] * core[2][nn];
        else {
          const int t = indpp[a][b];
          const int u = t == 4 || t == 5 ? 1 : t == 6 ? 2 : t, v = t == 4 ? 2 : t == 5 || t == 6 ? 3 : t;
          const double q = __fma_rn(p[2][u], p[2][v], __dmul_rn(p[3][u], p[3][v]));
          h = __fma_rn(core[3][nn], __dmul_rn(p[1][u], p[1][v]), __dmul_rn(core[4][nn], q));
        }
        out[a * (a + 1) / 2 + b] = 0.0 + h;
      }
  }
}

// ccrep (PM7): r in Bohr on entry; z3: the sum of the two atomic numbers' powers 0.3333
__device__ __forceinline__ double ccrep_z(int ni, int nj, double rb, double gab, double z3) {
  const double r = rb * PM7_A0;
  const Pm7Elem& A = c_P.el[ni];
  const Pm7Elem& B = c_P.el[nj];
  const double enuc = A.tore * B.tore * gab;
  double fff = c_P.xfac[ni][nj], abond = c_P.alpb[ni][nj];
  if (fabs(fff) < 1.0e-5) {
    fff = 0.5 * (c_P.xfac[ni][ni] + c_P.xfac[nj][nj]);
    abond = 0.5 * (c_P.alpb[ni][ni] + c_P.alpb[nj][nj]);
  }
  double enuclr, scale;
  if (fabs(fff) > 1.0e-5) {
    if (abond < 1.0e-6) abond = 1.2;
    scale = 1.0 + 2.0 * fff * exp(-abond * (r + (double)0.0003f * ipow(r, 6)));
    const int i = ni > nj ? ni : nj, j = ni < nj ? ni : nj;
    if (j == 1) {
      if (i == 6 || i == 7) scale = 1.0 + 2.0 * fff * exp(-abond * r * r);
      else if (i == 8) scale = 1.0 + 2.0 * fff * exp(-abond * r * r) - c_P.par3 * exp(-c_P.par4 * r * 2);
    } else if (j == 6 && i == 6) {
      scale = scale + c_P.par1 * exp(-c_P.par2 * r);
    }
    enuclr = __dmul_rn(enuc, scale);
  } else {
    scale = 10.0 * exp(-2.18 * r);
    enuclr = fabs(scale * enuc) + enuc;
  }
  scale = 0.0;
  double ax = A.g2 * (r - A.g3) * (r - A.g3);
  if (ax < 25.0) scale = scale + A.tore * B.tore / r * A.g1 * exp(-ax);
  ax = B.g2 * (r - B.g3) * (r - B.g3);
  if (ax < 25.0) scale = scale + A.tore * B.tore / r * B.g1 * exp(-ax);
  enuclr = enuclr + scale;
  ax = r / z3;
  if (ax < 3.0) {
    scale = 1.0e-8 / ipow(ax, 12);
    enuclr = enuclr + (scale < 1.0e5 ? scale : 1.0e5);
  }
  return enuclr;
}

__device__ __forceinline__ double ccrep(int ni, int nj, double rb, double gab) {
  return ccrep_z(ni, nj, rb, gab, pow((double)ni, 0.3333) + pow((double)nj, 0.3333));
}

// W block of pair (ni first, nj second) in molecular frame, a column at a time:
// col(kl, w) gets w[ij] of molecular pair kl of the second atom, kl ascending.
// Pairs of each atom, local or molecular: ss, ps, pp' in packed order.
template <int NI, int NJ, class Col>
__device__ __forceinline__ void w_block(const double p[4][4], const double ri[23], Col&& col) {
  constexpr int LI = NI == 1 ? 1 : 10, LJ = NJ == 1 ? 1 : 10;
  // rep index for (local pair on A, local pair on B); 0 where it vanishes
  const int rep[10][10] = {
      // B: ss  ps  pp  pis pisg pipi pi's pi'sg pi'pi pi'pi'
      {1, 5, 11, 0, 0, 12, 0, 0, 0, 12},       // A ss
      {2, 6, 13, 0, 0, 14, 0, 0, 0, 14},       // A sigma-s
      {3, 8, 16, 0, 0, 18, 0, 0, 0, 18},       // A sigma-sigma
      {0, 0, 0, 7, 15, 0, 0, 0, 0, 0},         // A pi-s
      {0, 0, 0, 10, 20, 0, 0, 0, 0, 0},        // A pi-sigma
      {4, 9, 17, 0, 0, 19, 0, 0, 0, 21},       // A pi-pi
      {0, 0, 0, 0, 0, 0, 7, 15, 0, 0},         // A pi'-s
      {0, 0, 0, 0, 0, 0, 10, 20, 0, 0},        // A pi'-sigma
      {0, 0, 0, 0, 0, 0, 0, 0, 22, 0},         // A pi'-pi
      {4, 9, 17, 0, 0, 21, 0, 0, 0, 19}};      // A pi'-pi'
  const int sp[10] = {0, 1, 0, 2, 0, 0, 3, 0, 0, 0};  // pair (p_k, s): k
  const int pt[10] = {0, 0, 1, 0, 4, 2, 0, 5, 6, 3};  // pair (p, p): ppf's molecular product
  const int pk[10] = {0, 0, 1, 0, 2, 2, 0, 3, 3, 3}, pl[10] = {0, 0, 1, 0, 1, 2, 0, 1, 2, 3};  // its local axes
#pragma unroll
  for (int kl = 0; kl < LJ; ++kl) {
    double v[LI], w[LI];
#pragma unroll
    for (int a = 0; a < LI; ++a) {  // B rotated
      v[a] = 0.0;
      if (kl == 0 && rep[a][0]) v[a] = ri[rep[a][0]];
#pragma unroll
      for (int b = 1; b < LJ; ++b) {
        if (!rep[a][b]) continue;
        if (sp[kl] && sp[b]) v[a] = __fma_rn(p[sp[b]][sp[kl]], ri[rep[a][b]], v[a]);
        if (pt[kl] && pt[b]) v[a] = __fma_rn(ppf(p, pt[kl], pk[b], pl[b]), ri[rep[a][b]], v[a]);
      }
    }
    w[0] = v[0];
#pragma unroll
    for (int ij = 1; ij < LI; ++ij) {  // A rotated
      w[ij] = 0.0;
#pragma unroll
      for (int a = 1; a < LI; ++a) {
        if (sp[ij] && sp[a]) w[ij] = __fma_rn(p[sp[a]][sp[ij]], v[a], w[ij]);
        if (pt[ij] && pt[a]) w[ij] = __fma_rn(ppf(p, pt[ij], pk[a], pl[a]), v[a], w[ij]);
      }
    }
    col(kl, w);
  }
}

// The pair's resonance block through hput(a, b, value), its W block in the
// reference layout (i's pair index outer, j's inner) to wb, and its core-core
// energy.
template <class HPut>
__device__ __forceinline__ double pair_integrals(int ni, int nj, const double* xi, const double* xj, double* wb,
                                                 HPut&& hput) {
  double enuc = 0.0;
  by_kind(ni, nj, [&](auto oi, auto oj) {
    constexpr int NI = decltype(oi)::n, NJ = decltype(oj)::n, LI = NI == 1 ? 1 : 10, LJ = NJ == 1 ? 1 : 10;
    double di[NI][NJ];
    h1elec<NI, NJ>(ni, nj, xi, xj, di);
#pragma unroll
    for (int a = 0; a < NI; ++a)
#pragma unroll
      for (int b = 0; b < NJ; ++b) hput(a, b, di[a][b]);
    const double dx = xi[0] - xj[0], dy = xi[1] - xj[1], dz = xi[2] - xj[2];
    if (dx * dx + dy * dy + dz * dz < 0.00002) {
      for (int x = 0; x < LI * LJ; ++x) wb[x] = 0.0;
      return;
    }
    double p[4][4];
    const double r = rotmat(xi, xj, p);
    double ri[23], gab;
    reppd<NI, NJ>(ni, nj, r, ri, &gab);
    w_block<NI, NJ>(p, ri, [&](int kl, const double* w) {
#pragma unroll
      for (int ij = 0; ij < LI; ++ij) wb[ij * LJ + kl] = w[ij];
    });
    enuc = ccrep(ni, nj, r / PM7_A0, gab);
  });
  return enuc;
}

// The electron-core blocks of atoms i and j, packed.
__device__ __forceinline__ void pair_cores(int ni, int nj, const double* xi, const double* xj, double* e1b,
                                           double* e2a) {
  double p[4][4], core[5][3];
  const double r = rotmat(xi, xj, p);
  by_kind(ni, nj, [&](auto oi, auto oj) {
    constexpr int NI = decltype(oi)::n, NJ = decltype(oj)::n;
    core_terms<NI, NJ>(ni, nj, r, core);
    elenuc<NI, NJ>(p, core, e1b, e2a);
  });
}

// reppd for a pair of any kind
__device__ __forceinline__ void reppd_any(int ni, int nj, double rij, double ri[23], double* gab) {
  by_kind(ni, nj, [&](auto oi, auto oj) { reppd<decltype(oi)::n, decltype(oj)::n>(ni, nj, rij, ri, gab); });
}

// Off-diagonal H block, two-centre W block and core-core energy of pair q.
__device__ void hcore_pair_one(long long q, const int* __restrict__ nat, const double* __restrict__ coord,
                               const MbAtomsDev& at, double* __restrict__ h, double* __restrict__ w,
                               double* __restrict__ enuc_pairs) {
  {
    // pair q -> (i, j), i > j, in the reference loop order
    long long i = (long long)((sqrt(8.0 * (double)q + 1.0) + 1.0) * 0.5);
    while (i * (i - 1) / 2 > q) --i;
    while ((i + 1) * i / 2 <= q) ++i;
    const int ia = (int)i, ja = (int)(q - i * (i - 1) / 2);
    const int ni = nat[ia], nj = nat[ja];
    const double* xi = coord + 3 * ia;
    const double* xj = coord + 3 * ja;
    const int fi = at.first[ia], fj = at.first[ja];
    double* wb = w + at.wrow[ia] + (long long)at.lim[ia] * at.cum[ja];
    enuc_pairs[q] = pair_integrals(ni, nj, xi, xj, wb,
                                   [&](int a, int b, double v) { h[mb_tri(fi + a, fj + b)] = v; });
  }
}

__global__ void hcore_pairs(int numat, const int* __restrict__ nat, const double* __restrict__ coord, MbAtomsDev at,
                            double* __restrict__ h, double* __restrict__ w, double* __restrict__ enuc_pairs) {
  const long long npair = (long long)numat * (numat - 1) / 2;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < npair; q += (long long)gridDim.x * blockDim.x)
    hcore_pair_one(q, nat, coord, at, h, w, enuc_pairs);
}

// Contribution of partner B to atom A's diagonal H block; false when B is A or
// on top of it.
__device__ __forceinline__ bool hcore_partner(int A, int B, const int* __restrict__ nat,
                                              const double* __restrict__ coord, const MbAtomsDev& at, double* c) {
  if (B == A) return false;
  const double *xa = coord + 3 * A, *xb = coord + 3 * B;
  const double dx = xa[0] - xb[0], dy = xa[1] - xb[1], dz = xa[2] - xb[2];
  if (dx * dx + dy * dy + dz * dz < 0.00002) return false;
  const int nA = nat[A], nB = nat[B];
  double other[10];
  if (B < A) pair_cores(nA, nB, xa, xb, c, other);  // pair (A first, B second): A receives e1b
  else pair_cores(nB, nA, xb, xa, other, c);        // pair (B first, A second): A receives e2a
  return true;
}

// Diagonal H block and one-centre W of atom A, by the calling warp.  The
// partners come 32 at a time, one a lane, and each lane's terms are then added
// in lane order, so the block is summed over B in the reference loop's order.
// A thread per atom, with the partners one after another, took 0.50 ms for the 72
// atoms of (H2O)24, this 0.06 (one B200); the bits are the same.
__device__ void hcore_atom_warp(int A, int numat, const int* __restrict__ nat, const double* __restrict__ coord,
                                const MbAtomsDev& at, double* __restrict__ h, double* __restrict__ w) {
  const int lane = threadIdx.x & 31;
  const int fA = at.first[A], noA = at.nor[A], lA = at.lim[A];
  const Pm7Elem& E = c_P.el[nat[A]];
  double blk[10];
  for (int x = 0; x < 10; ++x) blk[x] = 0.0;
  blk[0] = E.uss;
  if (noA == 4) { blk[2] = E.upp; blk[5] = E.upp; blk[9] = E.upp; }
  for (int b0 = 0; b0 < numat; b0 += 32) {
    double c[10];
    for (int x = 0; x < 10; ++x) c[x] = 0.0;
    const bool has = b0 + lane < numat && hcore_partner(A, b0 + lane, nat, coord, at, c);
    const unsigned mask = __ballot_sync(0xffffffffu, has);
    for (int src = 0; src < 32; ++src) {
      if (!((mask >> src) & 1u)) continue;
#pragma unroll
      for (int x = 0; x < 10; ++x)
        if (x < lA) blk[x] = blk[x] + __shfl_sync(0xffffffffu, c[x], src);
    }
  }
  if (lane != 0) return;
  for (int a = 0, x = 0; a < noA; ++a)
    for (int b = 0; b <= a; ++b, ++x) h[mb_tri(fA + a, fA + b)] = blk[x];
  // wstore (mndod.F90:2027)
  double* w1 = w + at.wrow[A] + (long long)lA * at.cum[A];
  for (int x = 0; x < lA * lA; ++x) w1[x] = 0.0;
#define WS(a, b) w1[((a) - 1) + lA * ((b) - 1)]
  WS(1, 1) = E.gss;
  if (noA == 4) {
    const int ipx = 3, ipy = 6, ipz = 10;
    WS(ipx, 1) = E.gsp; WS(ipy, 1) = E.gsp; WS(ipz, 1) = E.gsp;
    WS(1, ipx) = E.gsp; WS(1, ipy) = E.gsp; WS(1, ipz) = E.gsp;
    WS(ipx, ipx) = E.gpp; WS(ipy, ipy) = E.gpp; WS(ipz, ipz) = E.gpp;
    WS(ipy, ipx) = E.gp2; WS(ipz, ipx) = E.gp2; WS(ipz, ipy) = E.gp2;
    WS(ipx, ipy) = E.gp2; WS(ipx, ipz) = E.gp2; WS(ipy, ipz) = E.gp2;
    WS(2, 2) = E.hsp; WS(4, 4) = E.hsp; WS(7, 7) = E.hsp;
    WS(5, 5) = 0.5 * (E.gpp - E.gp2); WS(8, 8) = 0.5 * (E.gpp - E.gp2); WS(9, 9) = 0.5 * (E.gpp - E.gp2);
  }
#undef WS
}

__global__ void __launch_bounds__(128) hcore_diag(int numat, const int* __restrict__ nat,
                                                  const double* __restrict__ coord, MbAtomsDev at,
                                                  double* __restrict__ h, double* __restrict__ w) {
  const int A = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (A < numat) hcore_atom_warp(A, numat, nat, coord, at, h, w);
}

// ---- many molecules in one launch: a global pair or atom index is mapped to
// its molecule by a binary search over the prefix offsets.
__device__ __forceinline__ int batch_find(const long long* off, int nmol, long long q) {
  int lo = 0, hi = nmol;  // largest m < nmol with off[m] <= q
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= q) lo = mid; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ MbAtomsDev batch_atoms(const MbHcoreBatch& B, int m) {
  const long long a0 = B.atom_off[m];
  MbAtomsDev at;
  at.numat = (int)(B.atom_off[m + 1] - a0);
  at.first = B.first + a0;
  at.nor = B.nor + a0;
  at.lim = B.lim + a0;
  at.wrow = B.wrow + a0;
  at.cum = B.cum + a0;
  return at;
}

__global__ void hcore_pairs_batch(MbHcoreBatch B) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < B.pair_off[B.nmol];
       q += (long long)gridDim.x * blockDim.x) {
    const int m = batch_find(B.pair_off, B.nmol, q);
    const MbAtomsDev at = batch_atoms(B, m);
    const long long a0 = B.atom_off[m];
    hcore_pair_one(q - B.pair_off[m], B.nat + a0, B.coord + 3 * a0, at, B.h + B.hoff[m], B.w + B.woff[m],
                   B.enuc_pairs + B.pair_off[m]);
  }
}

__global__ void hcore_diag_batch(MbHcoreBatch B) {
  for (long long g = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; g < B.atom_off[B.nmol];
       g += ((long long)gridDim.x * blockDim.x) >> 5) {
    const int m = batch_find(B.atom_off, B.nmol, g);
    const MbAtomsDev at = batch_atoms(B, m);
    const long long a0 = B.atom_off[m];
    hcore_atom_warp((int)(g - a0), at.numat, B.nat + a0, B.coord + 3 * a0, at, B.h + B.hoff[m], B.w + B.woff[m]);
  }
}

// Fixed-order two-level reduction of the pair energies.
__global__ void enuc_sum(long long npair, const double* __restrict__ e, double* __restrict__ out) {
  __shared__ double sh[1024];
  double s = 0.0;
  for (long long q = threadIdx.x; q < npair; q += blockDim.x) s += e[q];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// enuc_sum for every molecule (block m: molecule m, the same order).
__global__ void enuc_sum_batch(MbHcoreBatch B) {
  const int m = blockIdx.x;
  const long long p0 = B.pair_off[m], np = B.pair_off[m + 1] - p0;
  __shared__ double sh[1024];
  double s = 0.0;
  for (long long q = threadIdx.x; q < np; q += blockDim.x) s += B.enuc_pairs[p0 + q];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) B.enuclr[m] = np > 0 ? sh[0] : 0.0;
}

// ---- hcore_for_MOZYME (MOZYME/hcore_for_MOZYME.F90, molecular, mode 0) on
// fillij's pair-block storage.  Stored pairs get the full integrals (the
// bodies above); the diagonal blocks take every partner's core attraction
// in the reference's order (with PM7's feathering the exact term beyond 7 A
// is the point charge outer1/outer2 use); the core-core energy of a pair
// that is not stored is outer1's or outer2's (tore_i tore_j times the
// point-charge or monopole integral).
__global__ void mz_hcore_pairs(MbMzLayout L, const int* __restrict__ nat, const double* __restrict__ coord,
                               double* __restrict__ h, double* __restrict__ w, double* __restrict__ enuc_entry) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < L.npairs;
       e += (long long)gridDim.x * blockDim.x) {
    const int ia = L.pair_i[e], ja = L.pair_j[e];
    if (ia == ja) {
      enuc_entry[e] = 0.0;
      continue;
    }
    const int ni = nat[ia], nj = nat[ja];
    const double* xi = coord + 3 * ia;
    const double* xj = coord + 3 * ja;
    const int noj = L.iorbs[ja];
    double* hb = h + L.pair_off[e];
    enuc_entry[e] = pair_integrals(ni, nj, xi, xj, w + L.pair_woff[e],
                                   [&](int a, int b, double v) { hb[a * noj + b] = v; });
  }
}

// The diagonal-block terms of a pair outside cutof2: outer2 (MOZYME/outer2.F90,
// mode 0: reppd's monopole and dipoles along the unit vector j -> i) in
// cutof1's band, outer1 (MOZYME/outer1.F90, mode 0: a feathered point charge)
// beyond it.  e1b: atom i's block, e2a: atom j's (packed, 10 for sp).
__device__ void mz_outer_terms(int ni, int nj, const double* ci, const double* cj, bool band, double* e1b,
                               double* e2a) {
  for (int k = 0; k < 10; ++k) { e1b[k] = 0.0; e2a[k] = 0.0; }
  const Pm7Elem& I = c_P.el[ni];
  const Pm7Elem& J = c_P.el[nj];
  if (!band) {
    const double rij = sqrt((ci[0] - cj[0]) * (ci[0] - cj[0]) + (ci[1] - cj[1]) * (ci[1] - cj[1]) +
                            (ci[2] - cj[2]) * (ci[2] - cj[2]));
    const double r = rij / PM7_A0;
    double aee = 0.5 / I.am + 0.5 / J.am;
    aee = aee * aee;
    double ww = PM7_EV / sqrt(r * r + aee), point, cst;
    to_point(rij, &point, &cst);
    ww = ww * cst + (1.0 - cst) * point;
    const int dg[4] = {0, 2, 5, 9};
    for (int k = 0; k < 4; ++k) {
      e1b[dg[k]] = -ww * J.tore;
      e2a[dg[k]] = -ww * I.tore;
    }
    return;
  }
  double x[3] = {ci[0] - cj[0], ci[1] - cj[1], ci[2] - cj[2]};
  const double rij = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
  double ri[23], gab;
  reppd_any(ni, nj, rij, ri, &gab);
  const double a = 1.0 / rij;
  x[0] *= a; x[1] *= a; x[2] *= a;
  if (fabs(x[2]) > 0.99999999) x[2] = x[2] >= 0.0 ? 1.0 : -1.0;
  const double w1 = ri[1];
  e1b[0] = -w1 * J.tore;
  e2a[0] = -w1 * I.tore;
  if (J.natorb > 1) {
    const double w2 = -ri[5] * x[0], w3 = -ri[5] * x[1], w4 = -ri[5] * x[2];
    e2a[1] = -w2 * I.tore; e2a[2] = -w1 * I.tore; e2a[3] = -w3 * I.tore;
    e2a[5] = -w1 * I.tore; e2a[6] = -w4 * I.tore; e2a[9] = -w1 * I.tore;
  }
  if (I.natorb > 1) {
    const double w5 = -ri[2] * x[0], w6 = -ri[2] * x[1], w7 = -ri[2] * x[2];
    e1b[1] = -w5 * J.tore; e1b[2] = -w1 * J.tore; e1b[3] = -w6 * J.tore;
    e1b[5] = -w1 * J.tore; e1b[6] = -w7 * J.tore; e1b[9] = -w1 * J.tore;
  }
}

// A warp per atom A; the partners B are taken 32 at a time, one per lane,
// and every lane's terms are then added in lane order, so the one-centre
// block and the core-core energy are summed over B in ascending order, the
// reference loop's order, bit for bit.
__global__ void __launch_bounds__(128) mz_hcore_diag(MbMzLayout L, const int* __restrict__ nat,
                                                     const double* __restrict__ coord, double* __restrict__ h,
                                                     double* __restrict__ w, const double* __restrict__ enuc_entry,
                                                     double* __restrict__ enuc_atom) {
  __shared__ int entry_of[4][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int A = blockIdx.x * 4 + wib;
  if (A >= L.numat) return;  // warp-uniform
  const int nA = nat[A], noA = L.iorbs[A], lA = noA * (noA + 1) / 2;
  const Pm7Elem& E = c_P.el[nA];
  double blk[10];
  for (int x = 0; x < 10; ++x) blk[x] = 0.0;
  blk[0] = E.uss;
  if (noA == 4) { blk[2] = E.upp; blk[5] = E.upp; blk[9] = E.upp; }
  const double* xa = coord + 3 * A;
  int ep = L.pair_ptr[A];                 // A's stored partners (ascending), then its own block
  const int ediag = L.pair_ptr[A + 1] - 1;
  double en = 0.0;
  for (int b0 = 0; b0 < L.numat; b0 += 32) {
    const int B = b0 + lane;
    // which partners of this chunk are stored pairs, and their entries
    entry_of[wib][lane] = -1;
    __syncwarp();
    {
      const int e = ep + lane;
      const int pj = e < ediag ? L.pair_j[e] : -1;
      const bool in = pj >= b0 && pj < b0 + 32;
      if (in) entry_of[wib][pj - b0] = e;
      ep += __popc(__ballot_sync(0xffffffffu, in));
    }
    __syncwarp();
    const int my_entry = entry_of[wib][lane];
    double cen = 0.0;        // this lane's core-core term (B < A)
    double c[10];            // this lane's contribution to A's one-centre block
    for (int x = 0; x < 10; ++x) c[x] = 0.0;
    bool has_c = false;
    if (B < L.numat && B != A) {
      const double* xb = coord + 3 * B;
      const double dx = xa[0] - xb[0], dy = xa[1] - xb[1], dz = xa[2] - xb[2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      const int nB = nat[B];
      if (B < A) {
        if (my_entry >= 0) {
          cen = enuc_entry[my_entry];
        } else if (r2 < L.cutof1) {       // outer2: monopole term
          double ri[23], gab;
          reppd_any(nA, nB, sqrt(r2), ri, &gab);
          cen = c_P.el[nA].tore * c_P.el[nB].tore * ri[1];
        } else {                          // outer1: feathered point charge
          const double rij = sqrt(r2), rb = rij / PM7_A0;
          double aee = 0.5 / E.am + 0.5 / c_P.el[nB].am;
          aee = aee * aee;
          double ww = PM7_EV / sqrt(rb * rb + aee), point, cst;
          to_point(rij, &point, &cst);
          ww = ww * cst + (1.0 - cst) * point;
          cen = c_P.el[nA].tore * c_P.el[nB].tore * ww;
        }
      }
      if (!(r2 < 0.00002)) {
        double e1b[10], e2a[10];
        has_c = true;
        if (!(r2 < L.cutof2) && sqrt(r2) < 7.0) {
          // a far pair inside PM7's 7 A feathering radius (a cutoff below
          // 7 A): outer1's or outer2's terms; beyond 7 A elenuc's feathered
          // integrals are the same point charges
          if (B < A) {
            mz_outer_terms(nA, nB, xa, xb, r2 < L.cutof1, e1b, e2a);
            for (int x = 0; x < 10; ++x) if (x < lA) c[x] = e1b[x];
          } else {
            mz_outer_terms(nB, nA, xb, xa, r2 < L.cutof1, e1b, e2a);
            for (int x = 0; x < 10; ++x) if (x < lA) c[x] = e2a[x];
          }
        } else {
          if (B < A) {
            pair_cores(nA, nB, xa, xb, e1b, e2a);
            for (int x = 0; x < 10; ++x) if (x < lA) c[x] = e1b[x];
          } else {
            pair_cores(nB, nA, xb, xa, e1b, e2a);
            for (int x = 0; x < 10; ++x) if (x < lA) c[x] = e2a[x];
          }
        }
      }
    }
    // the lanes' terms in ascending B
    const unsigned cmask = __ballot_sync(0xffffffffu, has_c);
    const unsigned emask = __ballot_sync(0xffffffffu, B < A);
    for (int src = 0; src < 32; ++src) {
      const double ce = __shfl_sync(0xffffffffu, cen, src);
      if ((emask >> src) & 1u) en += ce;
#pragma unroll
      for (int x = 0; x < 10; ++x) {
        if (x < lA) {  // lA is the warp's own, so every lane takes the shuffle or none
          const double v = __shfl_sync(0xffffffffu, c[x], src);
          if ((cmask >> src) & 1u) blk[x] = blk[x] + v * 1.0;
        }
      }
    }
    __syncwarp();
  }
  if (lane != 0) return;
  enuc_atom[A] = en;
  double* hd = h + L.pair_off[ediag];
  for (int x = 0; x < lA; ++x) hd[x] = blk[x];
  double* w1 = w + L.pair_woff[ediag];
  for (int x = 0; x < lA * lA; ++x) w1[x] = 0.0;
#define WS(a, b) w1[((a) - 1) + lA * ((b) - 1)]
  WS(1, 1) = E.gss;
  if (noA == 4) {
    const int ipx = 3, ipy = 6, ipz = 10;
    WS(ipx, 1) = E.gsp; WS(ipy, 1) = E.gsp; WS(ipz, 1) = E.gsp;
    WS(1, ipx) = E.gsp; WS(1, ipy) = E.gsp; WS(1, ipz) = E.gsp;
    WS(ipx, ipx) = E.gpp; WS(ipy, ipy) = E.gpp; WS(ipz, ipz) = E.gpp;
    WS(ipy, ipx) = E.gp2; WS(ipz, ipx) = E.gp2; WS(ipz, ipy) = E.gp2;
    WS(ipx, ipy) = E.gp2; WS(ipx, ipz) = E.gp2; WS(ipy, ipz) = E.gp2;
    WS(2, 2) = E.hsp; WS(4, 4) = E.hsp; WS(7, 7) = E.hsp;
    WS(5, 5) = 0.5 * (E.gpp - E.gp2); WS(8, 8) = 0.5 * (E.gpp - E.gp2); WS(9, 9) = 0.5 * (E.gpp - E.gp2);
  }
#undef WS
}

// ---------------------------------------------------------------- gradients
// Density blocks of the diatomic (atom 1 = jj, atom 2 = ii > jj): atom 1's,
// atom 2's, and rows of atom 2 by columns of atom 1.
struct PairDens {
  double p1[4][4], p2[4][4], p21[4][4];
};

__device__ __forceinline__ int pairix(int a, int b) {  // 0-based pair index of local orbitals a, b
  return a > b ? a * (a + 1) / 2 + b : b * (b + 1) / 2 + a;
}

// Energy of the diatomic in dhc's form (forces/dhc.F90:59-173, a molecule,
// RHF): h1elec's resonance block, the electron-core blocks, the two-centre
// Coulomb and exchange terms with the density fixed, helect over the pair's
// orbitals (doubled), and ccrep's core-core term; eV.  Like dhc it leaves out
// every term that does not depend on the pair's geometry.
//
// N1, N2: the atoms' orbital counts.  sw: room for the W block, element
// (ij, kl) at sw[(ij * lim1 + kl) * SW]; z3 as in ccrep_z.
template <int N1, int N2, int SW>
__device__ __forceinline__ double dhc_energy(int n1, int n2, const double* x1, const double* x2, const PairDens& d,
                                             double* sw, double z3) {
  constexpr int L1 = N1 == 1 ? 1 : 10, L2 = N2 == 1 ? 1 : 10;
  double enuc = 0.0, e = 0.0;
  double h1[10], h2[10], ri[23], p[4][4];
  const double dx = x2[0] - x1[0], dy = x2[1] - x1[1], dz = x2[2] - x1[2];
  const bool apart = dx * dx + dy * dy + dz * dz >= 0.00002;
#pragma unroll
  for (int x = 0; x < 10; ++x) h1[x] = h2[x] = 0.0;
  if (apart) {
    const double r = rotmat(x2, x1, p);  // rotate(ni = atom 2, nj = atom 1) as dhc calls it
    double core[5][3], gab;
    core_terms<N2, N1>(n2, n1, r, core);
    elenuc<N2, N1>(p, core, h2, h1);  // atom 2's electrons: e1b; atom 1's: e2a
    reppd<N2, N1>(n2, n1, r, ri, &gab);
    enuc = ccrep_z(n2, n1, r / PM7_A0, gab, z3);
  } else {
#pragma unroll
    for (int x = 0; x < 23; ++x) ri[x] = 0.0;
#pragma unroll
    for (int x = 0; x < 16; ++x) (&p[0][0])[x] = 0.0;
  }
  // Coulomb terms on each atom's block from the other atom's density, and the
  // energy of the diagonal blocks: sum' P (H + F), F = H + G
  w_block<N2, N1>(p, ri, [&](int q, const double* w) {  // atom 1's pair q
#pragma unroll
    for (int ij = 0; ij < L2; ++ij) sw[(ij * L1 + q) * SW] = w[ij];
    double g = 0.0;
#pragma unroll
    for (int x = 0; x < N2; ++x)
#pragma unroll
      for (int y = 0; y < N2; ++y) g += d.p2[x][y] * w[pairix(x, y)];
#pragma unroll
    for (int a = 0; a < N1; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b)
        if (pairix(a, b) == q) {
          const double wgt = a == b ? 0.5 : 1.0;
          e += wgt * d.p1[a][b] * (2.0 * h1[q] + g);
        }
  });
#pragma unroll
  for (int a = 0; a < N2; ++a)
#pragma unroll
    for (int b = 0; b <= a; ++b) {
      const int q = pairix(a, b);
      double g = 0.0;
#pragma unroll
      for (int x = 0; x < N1; ++x)
#pragma unroll
        for (int y = 0; y < N1; ++y) g += d.p1[x][y] * sw[(q * L1 + pairix(x, y)) * SW];
      const double wgt = a == b ? 0.5 : 1.0;
      e += wgt * d.p2[a][b] * (2.0 * h2[q] + g);
    }
  // the off-diagonal block: resonance and exchange (kab), PA = P / 2
  double di[N1][N2];
  h1elec<N1, N2>(n1, n2, x1, x2, di);  // di[a][b]: a on atom 1, b on atom 2
#pragma unroll
  for (int mu = 0; mu < N2; ++mu)
#pragma unroll
    for (int nu = 0; nu < N1; ++nu) {
      double k = 0.0;
#pragma unroll
      for (int la = 0; la < N2; ++la)
#pragma unroll
        for (int si = 0; si < N1; ++si)
          k += 0.5 * d.p21[la][si] * sw[(pairix(mu, la) * L1 + pairix(nu, si)) * SW];
      e += d.p21[mu][nu] * (2.0 * di[nu][mu] - k);
    }
  // 2 * helect(PA, H, F) with PA = P/2 is sum' P (H + F) = e
  return e + enuc;
}

// The k-th (from 0) atom of numat that has four orbitals (heavy) or one: cum
// counts ten pairs or one, so cum[a] - a is nine times the heavy atoms below a.
__device__ __forceinline__ int kth_atom(const int* __restrict__ cum, int numat, int k, bool heavy) {
  int lo = 0, hi = numat - 1;  // the largest a with at most k of the kind below it
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1, nh = (cum[mid] - mid) / 9;
    if ((heavy ? nh : mid - nh) <= k) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// q -> (i, j), i > j, q = i (i - 1) / 2 + j
__device__ __forceinline__ void pair_of(long long q, int* ii, int* jj) {
  long long i = (long long)((sqrt(8.0 * (double)q + 1.0) + 1.0) * 0.5);
  while (i * (i - 1) / 2 > q) --i;
  while ((i + 1) * i / 2 <= q) ++i;
  *ii = (int)i;
  *jj = (int)(q - i * (i - 1) / 2);
}

// dcart (forces/dcart.F90:60-300) for a molecule with the default finite
// difference (no FORCE keyword): pair q = (ii, jj), jj < ii, with atom jj
// moved by chnge/2 along all three axes, then atom ii by chnge along each
// axis in turn; deriv = (E0 - Ek) * fpc_9 / chnge, kcal/mol/A.
//
// A lane per (pair, geometry), four lanes a pair, and a launch per kind of pair:
// two heavy atoms (KIND 0), mixed (1; the light partners of a heavy atom in a
// row), two light ones (2), so that the loops have constant lengths and the lanes
// of a warp take the same branches.  The W block of two heavy atoms (100
// numbers) is in shared memory.  The rest is in registers, of which two heavy atoms
// take all 255 and spill (1.1 KB of stores and 1.2 of loads a thread); the other
// kinds do not (149 and 80).  Bound by the FP64 pipe's latency, a few hundred square
// roots and quotients an energy, at 8, 11 and 18 warps an SM.  (H2O)200, one B200:
// 0.25 ms; a thread per pair, with the kinds mixed
// in a warp and the arrays in local memory, took 3.4, that split by kind and
// geometry alone 1.0.
template <int KIND>
__global__ void __launch_bounds__(KIND == 0 ? 32 : 128) dcart_pairs(int numat, const int* __restrict__ nat,
                                                                    const double* __restrict__ coord, MbAtomsDev at,
                                                                    const double* __restrict__ ptot,
                                                                    double* __restrict__ deriv) {
  __shared__ double z3[9], sw[KIND == 0 ? 100 * 32 : 1];
  if (threadIdx.x < 9) z3[threadIdx.x] = pow((double)threadIdx.x, 0.3333);
  __syncthreads();
  const double chnge = 1.0e-4, chnge2 = chnge * 0.5;
  const long long nh = (at.cum[numat - 1] + at.lim[numat - 1] - numat) / 9, nl = numat - nh;
  const long long count = KIND == 0 ? nh * (nh - 1) / 2 : KIND == 1 ? nh * nl : nl * (nl - 1) / 2;
  const int geo = threadIdx.x & 3;
  // whole warps iterate, for the shuffle: lanes past the end repeat the last pair
  for (long long t0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x - (threadIdx.x & 31)) >> 2; t0 < count;
       t0 += (long long)gridDim.x * blockDim.x >> 2) {
    long long t = t0 + ((threadIdx.x & 31) >> 2);
    const bool live = t < count;
    if (!live) t = count - 1;
    int ii, jj;
    if (KIND == 1) {
      const int a = kth_atom(at.cum, numat, (int)(t / nl), true), b = kth_atom(at.cum, numat, (int)(t % nl), false);
      ii = a > b ? a : b;
      jj = a > b ? b : a;
    } else {
      pair_of(t, &ii, &jj);
      ii = kth_atom(at.cum, numat, ii, KIND == 0);
      jj = kth_atom(at.cum, numat, jj, KIND == 0);
    }
    const int n1 = nat[jj], n2 = nat[ii];
    const double zz = z3[n2] + z3[n1];
    double x1[3], x2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x1[k] = coord[3 * jj + k] + chnge2;
      // dcart moves ii forth and back on one axis after another, in place
      const double x = coord[3 * ii + k];
      x2[k] = k + 1 > geo ? x : k + 1 == geo ? x + chnge : x + chnge - chnge2 - chnge2;
    }
    auto energy = [&](auto o1, auto o2) {
      constexpr int N1 = decltype(o1)::n, N2 = decltype(o2)::n;
      const int f1 = at.first[jj], f2 = at.first[ii];
      PairDens d;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          d.p1[a][b] = (a < N1 && b < N1) ? ptot[mb_tri(f1 + (a > b ? a : b), f1 + (a > b ? b : a))] : 0.0;
          d.p2[a][b] = (a < N2 && b < N2) ? ptot[mb_tri(f2 + (a > b ? a : b), f2 + (a > b ? b : a))] : 0.0;
          d.p21[a][b] = (a < N2 && b < N1) ? ptot[mb_tri(f2 + a, f1 + b)] : 0.0;
        }
      if constexpr (KIND == 0) {
        return dhc_energy<N1, N2, 32>(n1, n2, x1, x2, d, sw + threadIdx.x, zz);
      } else {
        double w[10];
        return dhc_energy<N1, N2, 1>(n1, n2, x1, x2, d, w, zz);
      }
    };
    double e;
    if constexpr (KIND == 0) e = energy(Orb<4>{}, Orb<4>{});
    else if constexpr (KIND == 2) e = energy(Orb<1>{}, Orb<1>{});
    else if (at.nor[ii] == 1) e = energy(Orb<4>{}, Orb<1>{});
    else e = energy(Orb<1>{}, Orb<4>{});
    const double aa = __shfl_sync(0xffffffffu, e, threadIdx.x & 28);
    if (live && geo > 0) deriv[3 * ((long long)ii * (ii - 1) / 2 + jj) + geo - 1] = (aa - e) * PM7_FPC9 / chnge;
  }
}

// dxyz of atom a in dcart's accumulation order: the pairs (a, jj < a), then
// the pairs (ii > a, a), each ascending.  A warp per atom loads the terms of 32
// partners at a time and its first three lanes add them in order, a coordinate
// each; bound by the chain of additions.  600 atoms: 16 us; a thread per
// coordinate, straight from global memory, 98.
__global__ void __launch_bounds__(128) dcart_sum(int numat, const double* __restrict__ deriv,
                                                 double* __restrict__ dxyz) {
  __shared__ double term[4][96];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, a = blockIdx.x * 4 + warp;
  if (a >= numat) return;  // warp-uniform
  double next[3], g = 0.0;
  auto load = [&](int b) {
    const long long q = b < a ? (long long)a * (a - 1) / 2 + b : (long long)b * (b - 1) / 2 + a;
    for (int k = 0; k < 3; ++k) next[k] = (b < numat && b != a) ? deriv[3 * q + k] : 0.0;
  };
  load(lane);
  for (int b0 = 0; b0 < numat; b0 += 32) {
    for (int k = 0; k < 3; ++k) term[warp][3 * lane + k] = next[k];
    __syncwarp();
    load(b0 + 32 + lane);
    if (lane < 3) {
      const int nb = numat - b0 < 32 ? numat - b0 : 32;
#pragma unroll 8
      for (int x = 0; x < nb; ++x) {
        const double v = term[warp][3 * x + lane];
        if (b0 + x != a) g = b0 + x < a ? g - v : g + v;
      }
    }
    __syncwarp();
  }
  if (lane < 3) dxyz[3 * a + lane] = g;
}

bool g_params_uploaded = false;

int upload_params() {
  if (g_params_uploaded) return MB_OK;
  Pm7Params P;
  pm7_init(&P);
  DevParams D;
  memcpy(D.el, P.el, sizeof(D.el));
  memcpy(D.xfac, P.xfac, sizeof(D.xfac));
  memcpy(D.alpb, P.alpb, sizeof(D.alpb));
  D.par1 = P.par1; D.par2 = P.par2; D.par3 = P.par3; D.par4 = P.par4;
  MB_CUDA(cudaMemcpyToSymbol(c_P, &D, sizeof(D)));
  g_params_uploaded = true;
  return MB_OK;
}

}  // namespace

extern "C" int mb_hcore_dev(const int* nat_d, const double* coord_d, const MbAtomsDev* at, int numat, double* h,
                            double* w, double* enuc_pairs, cudaStream_t stream) {
  MB_TRY(upload_params());
  const long long npair = (long long)numat * (numat - 1) / 2;
  if (npair > 0) {
    int blocks = (int)((npair + 127) / 128);
    if (blocks > 148 * 32) blocks = 148 * 32;
    hcore_pairs<<<blocks, 128, 0, stream>>>(numat, nat_d, coord_d, *at, h, w, enuc_pairs);
    MB_LAUNCH_CHECK();
  }
  hcore_diag<<<(numat + 3) / 4, 128, 0, stream>>>(numat, nat_d, coord_d, *at, h, w);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

extern "C" int mb_hcore_batch_dev(const MbHcoreBatch* b, cudaStream_t stream) {
  if (!b || b->nmol <= 0) return mb_set_error(MB_ERR_ARG, "mb_hcore_batch_dev: bad args");
  MB_TRY(upload_params());
  const long long npair = b->npair_tot, natom = b->natom_tot;
  if (npair > 0) {
    const int blocks = (int)std::min<long long>((npair + 127) / 128, 148LL * 32);
    hcore_pairs_batch<<<blocks, 128, 0, stream>>>(*b);
    MB_LAUNCH_CHECK();
  }
  const int blocks = (int)std::min<long long>((natom + 3) / 4, 148LL * 32);
  hcore_diag_batch<<<blocks, 128, 0, stream>>>(*b);
  MB_LAUNCH_CHECK();
  enuc_sum_batch<<<b->nmol, 1024, 0, stream>>>(*b);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

extern "C" int mb_hcore_finish(int numat, const MbAtomsDev* at, const int* nat_d, double* h, const double* e1b,
                               double* enuclr_dev, const double* enuc_pairs, cudaStream_t stream) {
  (void)at; (void)nat_d; (void)h; (void)e1b;
  const long long npair = (long long)numat * (numat - 1) / 2;
  if (npair == 0) {
    MB_CUDA(cudaMemsetAsync(enuclr_dev, 0, sizeof(double), stream));
    return MB_OK;
  }
  enuc_sum<<<1, 1024, 0, stream>>>(npair, enuc_pairs, enuclr_dev);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

// hcore_for_MOZYME on the pair blocks: h (layout mpack), w (layout nw: the
// stored pairs' two-centre blocks and every atom's one-centre block),
// *enuclr_dev (device) the core-core energy over every atom pair.  ws:
// mb_mz_hcore_ws_bytes(layout) bytes of device scratch.
extern "C" size_t mb_mz_hcore_ws_bytes(const MbMzLayout* L) {
  return L ? sizeof(double) * (size_t)(L->npairs + L->numat) : 0;
}

extern "C" int mb_mz_hcore_dev(const MbMzLayout* L, const int* nat_d, const double* coord_d, double* h, double* w,
                               double* enuclr_dev, void* ws, cudaStream_t stream) {
  if (!L || !nat_d || !coord_d || !h || !w || !enuclr_dev || !ws || L->numat <= 0)
    return mb_set_error(MB_ERR_ARG, "mb_mz_hcore_dev: bad args");
  // Far pairs past PM7's 7 A feathering (mndod.F90:800-822) take the
  // rotated core attraction, which there is outer1's and outer2's point
  // charge; those inside 7 A (a cutoff below 7 A) take outer1's and outer2's
  // own terms, and every far pair the outer core-core term.
  MB_TRY(upload_params());
  double* enuc_entry = (double*)ws;
  double* enuc_atom = enuc_entry + L->npairs;
  if (L->npairs > 0) {
    const int blocks = (int)std::min<long long>((L->npairs + 127) / 128, 148LL * 32);
    mz_hcore_pairs<<<blocks, 128, 0, stream>>>(*L, nat_d, coord_d, h, w, enuc_entry);
    MB_LAUNCH_CHECK();
  }
  mz_hcore_diag<<<(L->numat + 3) / 4, 128, 0, stream>>>(*L, nat_d, coord_d, h, w, enuc_entry, enuc_atom);
  MB_LAUNCH_CHECK();
  enuc_sum<<<1, 1024, 0, stream>>>(L->numat, enuc_atom, enuclr_dev);
  MB_LAUNCH_CHECK();
  return MB_OK;
}

extern "C" size_t mb_dcart_ws_bytes(int numat) {
  if (numat < 2) return 0;
  return sizeof(double) * 3 * ((size_t)numat * (numat - 1) / 2);
}

// Cartesian gradient of the SCF energy (dcart, forces/dcart.F90:16-300, a
// molecule, RHF): dxyz_dev[3a + k] in kcal/mol/A for the packed density p.
extern "C" int mb_dcart_dev(const int* nat_d, const double* coord_d, const MbAtomsDev* at, int numat, const double* p,
                            double* dxyz_dev, void* ws, size_t ws_bytes, cudaStream_t stream) {
  if (!at || numat <= 0 || !nat_d || !coord_d || !p || !dxyz_dev) return mb_set_error(MB_ERR_ARG, "mb_dcart_dev: bad args");
  if (ws_bytes < mb_dcart_ws_bytes(numat) || (numat > 1 && !ws))
    return mb_set_error(MB_ERR_ARG, "mb_dcart_dev: workspace smaller than mb_dcart_ws_bytes(numat)");
  MB_TRY(upload_params());
  const long long npair = (long long)numat * (numat - 1) / 2;
  if (npair > 0) {
    // how many pairs are of which kind is known on the device only
    const int b32 = (int)std::min<long long>((npair + 7) / 8, 148 * 16);
    const int b128 = (int)std::min<long long>((npair + 31) / 32, 148 * 8);
    dcart_pairs<0><<<b32, 32, 0, stream>>>(numat, nat_d, coord_d, *at, p, (double*)ws);
    MB_LAUNCH_CHECK();
    dcart_pairs<1><<<b128, 128, 0, stream>>>(numat, nat_d, coord_d, *at, p, (double*)ws);
    MB_LAUNCH_CHECK();
    dcart_pairs<2><<<b128, 128, 0, stream>>>(numat, nat_d, coord_d, *at, p, (double*)ws);
    MB_LAUNCH_CHECK();
    dcart_sum<<<(numat + 3) / 4, 128, 0, stream>>>(numat, (const double*)ws, dxyz_dev);
    MB_LAUNCH_CHECK();
  } else {
    MB_CUDA(cudaMemsetAsync(dxyz_dev, 0, sizeof(double) * 3 * (size_t)numat, stream));
  }
  return MB_OK;
}
