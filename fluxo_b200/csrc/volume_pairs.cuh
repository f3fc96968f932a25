// Per-node records and symmetric two-point volume fluxes for the split-form volume kernel.
//
// Each volume node stores a record of the quantities its pair fluxes need (primitive variables,
// the logarithms of the log-averaged quantities, the metric terms of the three directions), so a
// pair evaluation does no logarithm and at most one division.  The fluxes are the reference's
// VolumeFluxAverageVec family (src/equation/navierstokes/flux_average.f90); results agree with
// the reference formulas to roundoff:
//  - the logarithmic mean LN_MEAN (flux_average.f90:1945-1965) keeps its series branch for
//    u = ((b-a)/(b+a))^2 < 1e-4, as a product with a series in u (ln_series, inv_ln_series), and
//    otherwise uses (b-a)/(log b - log a) with per-node logarithms;
//  - the divisions of one pair flux are merged into a single reciprocal (rcp_nr).
#pragma once
#include "common.cuh"

namespace fluxo {

// Reciprocal of x (nonzero, normal, not huge) for the pair fluxes: the hardware's approximate reciprocal
// (PTX rcp.approx.ftz.f64) refined by two Newton-Raphson steps for f(y) = 1/y - x,
// y <- y + y (1 - x y), each computed with fused multiply-adds.  The approximation's relative error
// is squared by every step, so two steps reach double precision (within an ulp of the rounded
// quotient); the denominators here are products of the sums of densities and inverse temperatures
// (off the log mean's series branch: their differences), far from zero and from overflow.  It replaces the longer IEEE division sequence (one per pair).
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// Logarithmic mean (LN_MEAN) of a and b from s = a + b, and its reciprocal from is = 1/s, on the series
// branch u = ((b-a)/s)^2 < 1e-4, where the mean is s/2 / (1 + u/3 + u^2/5 + u^3/7): ln_series multiplies by
// the series of that reciprocal, 1 - u/3 - 4u^2/45 - 44u^3/945 (the next term is below 1e-17), and
// inv_ln_series by the polynomial itself, so neither divides: one reciprocal 1/(s_a s_b) serves both means
// of a pair.
__device__ __forceinline__ double ln_series(double s, double u) {
  return s * fma(u, fma(u, fma(u, -22. / 945., -2. / 45.), -1. / 6.), 0.5);
}
__device__ __forceinline__ double inv_ln_series(double is, double u) {
  return is * fma(u, fma(u, fma(u, 2. / 7., 2. / 5.), 2. / 3.), 2.);
}
// The two means of a pair: M = LN(a) and I = 1 / LN(b).  ln_pair forms both by their series and tells whether
// both are on that branch; ln_pair_fix replaces those that are not by (b-a)/(log b - log a), with the
// logarithms of the nodes' records (read only here: in smooth flows nearly every pair is on the series
// branch).  Two steps, so that several pairs share one rare branch and their straight-line parts overlap.
__device__ __forceinline__ bool ln_pair(double La, double Ra, double sa, double isa, double Lb, double Rb, double isb,
                                        double& M, double& I) {
  const double fa = (Ra - La) * isa, fb = (Rb - Lb) * isb;
  const double ua = fa * fa, ub = fb * fb;
  M = ln_series(sa, ua);
  I = inv_ln_series(isb, ub);
  return ua < 1.0e-4 && ub < 1.0e-4;
}
__device__ __forceinline__ void ln_pair_fix(double La, double Ra, const double* lLa, const double* lRa, double Lb,
                                            double Rb, const double* lLb, const double* lRb, double& M, double& I) {
  const double da = Ra - La, sa = La + Ra, db = Rb - Lb, sb = Lb + Rb;
  if (!(da * da < 1.0e-4 * (sa * sa))) M = da * rcp_nr(*lRa - *lLa);
  if (!(db * db < 1.0e-4 * (sb * sb))) I = (*lRb - *lLb) * rcp_nr(db);
}

// Record of a node in shared memory: NQ flux quantities at [0, NQ) (the first NF without
// the logarithms, which come last), the metric terms Ja^1..Ja^3
// (x,y,z each) at [MO, MO+9), RS doubles per node.  The odd stride RS spreads the records of the
// nodes of a line over the shared-memory banks (padded 16-byte-aligned records read with 16-byte
// loads measured 19 % slower on the N=7 volume kernel).
template <int VF>
struct VolRec;
// standard DG (0) and dealiased metric (1): rho, rho u, rho v, rho w, rho E, u, v, w, p
template <> struct VolRec<0> { static constexpr int NQ = 9, NF = 9, MO = 9, RS = 19; };
template <> struct VolRec<1> { static constexpr int NQ = 9, NF = 9, MO = 9, RS = 19; };
// Kennedy-Gruber (2): rho, u, v, w, p, e = E/rho
template <> struct VolRec<2> { static constexpr int NQ = 6, NF = 6, MO = 6, RS = 15; };
// Ducros (3): halves of rho, u, v, w, p, rho u, rho v, rho w, rho E (every average is arithmetic)
template <> struct VolRec<3> { static constexpr int NQ = 9, NF = 9, MO = 9, RS = 19; };
// Morinishi (4): rho, u, v, w, p, |v|^2
template <> struct VolRec<4> { static constexpr int NQ = 6, NF = 6, MO = 6, RS = 15; };
// EC-KEP (5): rho, u/2, v/2, w/2, beta = rho/(2p), |v|^2/2, log rho, log beta (the halves make the
// pair averages plain sums; halving is exact, so the averages are bit-identical)
template <> struct VolRec<5> { static constexpr int NQ = 8, NF = 6, MO = 8, RS = 17; };
// approximate EC-KEP (6): rho/2, u/2, v/2, w/2, beta, |v|^2/2
template <> struct VolRec<6> { static constexpr int NQ = 6, NF = 6, MO = 6, RS = 15; };
// EC-KEP with pressure average (7): rho/2, u/2, v/2, w/2, p/2, beta, |v|^2/2, log beta
template <> struct VolRec<7> { static constexpr int NQ = 8, NF = 7, MO = 8, RS = 17; };
// Kennedy-Gruber, Pirozzoli form (8): halves of rho, u, v, w, p, H = (rho E + p)/rho
template <> struct VolRec<8> { static constexpr int NQ = 6, NF = 6, MO = 6, RS = 15; };
// Gassner-Winters-Walch (9): halves of sqrt(rho) times (1, u, v, w, H)
template <> struct VolRec<9> { static constexpr int NQ = 5, NF = 5, MO = 5, RS = 15; };
// Ismail-Roe (10): z1 = sqrt(rho/p), u, v, w, z5 = z1 p, log z1, log z5
template <> struct VolRec<10> { static constexpr int NQ = 7, NF = 5, MO = 7, RS = 17; };
// Ranocha (32): rho, u, v, w, p, rho/p, log rho, log(rho/p)
template <> struct VolRec<32> { static constexpr int NQ = 8, NF = 6, MO = 8, RS = 17; };

// the flux quantities of record r (shared memory) without the trailing logarithms
template <int VF>
__device__ __forceinline__ void load_rec(const double* r, double* q) {
#pragma unroll
  for (int z = 0; z < VolRec<VF>::NF; ++z) q[z] = r[z];
}

// the metric triple Ja^(dir+1) of record r
template <int VF>
__device__ __forceinline__ void load_metric(const double* r, int dir, double* m) {
  const int off = VolRec<VF>::MO + 3 * dir;
  m[0] = r[off]; m[1] = r[off + 1]; m[2] = r[off + 2];
}

template <int VF>
__device__ __forceinline__ void make_record(const KParams& P, const double* U, double* r) {
  const double srho = 1. / U[0];
  const double u = U[1] * srho, v = U[2] * srho, w = U[3] * srho;
  const double v2 = u * u + v * v + w * w;
  const double p = P.kappaM1 * (U[4] - 0.5 * U[0] * v2);
  if constexpr (VF == 0 || VF == 1) {
    r[0] = U[0]; r[1] = U[1]; r[2] = U[2]; r[3] = U[3]; r[4] = U[4];
    r[5] = u; r[6] = v; r[7] = w; r[8] = p;
  } else if constexpr (VF == 2) {
    r[0] = U[0]; r[1] = u; r[2] = v; r[3] = w; r[4] = p; r[5] = srho * U[4];
  } else if constexpr (VF == 3) {
    r[0] = 0.5 * U[0]; r[1] = 0.5 * u; r[2] = 0.5 * v; r[3] = 0.5 * w; r[4] = 0.5 * p;
    r[5] = 0.5 * U[1]; r[6] = 0.5 * U[2]; r[7] = 0.5 * U[3]; r[8] = 0.5 * U[4];
  } else if constexpr (VF == 4) {
    r[0] = U[0]; r[1] = u; r[2] = v; r[3] = w; r[4] = p; r[5] = v2;
  } else if constexpr (VF == 6) {
    r[0] = 0.5 * U[0]; r[1] = 0.5 * u; r[2] = 0.5 * v; r[3] = 0.5 * w; r[4] = 0.5 * U[0] / p; r[5] = 0.5 * v2;
  } else if constexpr (VF == 7) {
    const double beta = 0.5 * U[0] / p;
    r[0] = 0.5 * U[0]; r[1] = 0.5 * u; r[2] = 0.5 * v; r[3] = 0.5 * w; r[4] = 0.5 * p; r[5] = beta;
    r[6] = 0.5 * v2; r[7] = log(beta);
  } else if constexpr (VF == 8) {
    r[0] = 0.5 * U[0]; r[1] = 0.5 * u; r[2] = 0.5 * v; r[3] = 0.5 * w; r[4] = 0.5 * p;
    r[5] = 0.5 * ((U[4] + p) * srho);
  } else if constexpr (VF == 9) {
    const double w1 = sqrt(U[0]);
    r[0] = 0.5 * w1; r[1] = 0.5 * (w1 * u); r[2] = 0.5 * (w1 * v); r[3] = 0.5 * (w1 * w);
    r[4] = 0.5 * (w1 * srho * (U[4] + p));
  } else if constexpr (VF == 5) {
    const double beta = 0.5 * U[0] / p;
    r[0] = U[0]; r[1] = 0.5 * u; r[2] = 0.5 * v; r[3] = 0.5 * w; r[4] = beta; r[5] = 0.5 * v2;
    r[6] = log(U[0]); r[7] = log(beta);
  } else if constexpr (VF == 10) {
    const double z1 = sqrt(U[0] / p);
    const double z5 = z1 * p;
    r[0] = z1; r[1] = u; r[2] = v; r[3] = w; r[4] = z5; r[5] = log(z1); r[6] = log(z5);
  } else if constexpr (VF == 32) {
    const double rsp = U[0] / p;
    r[0] = U[0]; r[1] = u; r[2] = v; r[3] = w; r[4] = p; r[5] = rsp; r[6] = log(U[0]); r[7] = log(rsp);
  }
}

// Entries of a record that take a log mean (A, logarithm LA) and the reciprocal of one (B, LB)
template <int VF> struct VolMeans { static constexpr bool USED = false; static constexpr int A = 0, LA = 0, B = 0, LB = 0; };
template <> struct VolMeans<5> { static constexpr bool USED = true; static constexpr int A = 0, LA = 6, B = 4, LB = 7; };
template <> struct VolMeans<7> { static constexpr bool USED = true; static constexpr int A = 5, LA = 7, B = 5, LB = 7; };
template <> struct VolMeans<10> { static constexpr bool USED = true; static constexpr int A = 4, LA = 6, B = 0, LB = 5; };
template <> struct VolMeans<32> { static constexpr bool USED = true; static constexpr int A = 0, LA = 6, B = 5, LB = 7; };

// The means of a pair's flux: mn[0] = LN(A), mn[1] = 1/LN(B) on the series branch (returns whether both
// are on it), mn[2] = 1/(B_L + B_R)
template <int VF>
__device__ __forceinline__ bool pair_means(const double* L, const double* R, double* mn) {
  using V = VolMeans<VF>;
  if constexpr (!V::USED) return true;
  else {
    const double sa = L[V::A] + R[V::A], sb = L[V::B] + R[V::B];
    double isa;
    if constexpr (V::A == V::B) isa = mn[2] = rcp_nr(sa);
    else {
      const double inv = rcp_nr(sa * sb);
      isa = sb * inv;
      mn[2] = sa * inv;
    }
    return ln_pair(L[V::A], R[V::A], sa, isa, L[V::B], R[V::B], mn[2], mn[0], mn[1]);
  }
}
// off the series branch: lL, lR are the nodes' records, read for their logarithms
template <int VF>
__device__ __forceinline__ void pair_means_fix(const double* L, const double* R, const double* lL, const double* lR,
                                               double* mn) {
  using V = VolMeans<VF>;
  if constexpr (V::USED)
    ln_pair_fix(L[V::A], R[V::A], lL + V::LA, lR + V::LA, L[V::B], R[V::B], lL + V::LB, lR + V::LB, mn[0], mn[1]);
}

// F = F#(L, R) . metric, symmetric in (L, R), from the pair's means mn
template <int VF>
__device__ __forceinline__ void pair_flux_from(const KParams& P, const double* L, const double* R, const double* mn,
                                               const double* mL, const double* mR, double* F) {
  if constexpr (VF == 0) {  // StandardDGFluxVec :394-439
    const double qL = L[5] * mL[0] + L[6] * mL[1] + L[7] * mL[2];
    const double qR = R[5] * mR[0] + R[6] * mR[1] + R[7] * mR[2];
    F[0] = 0.5 * (L[0] * qL + R[0] * qR);
    F[1] = 0.5 * (L[1] * qL + R[1] * qR + mL[0] * L[8] + mR[0] * R[8]);
    F[2] = 0.5 * (L[2] * qL + R[2] * qR + mL[1] * L[8] + mR[1] * R[8]);
    F[3] = 0.5 * (L[3] * qL + R[3] * qR + mL[2] * L[8] + mR[2] * R[8]);
    F[4] = 0.5 * ((L[4] + L[8]) * qL + (R[4] + R[8]) * qR);
  } else {
    // the records of these fluxes hold half metrics: the dealiased metric 1/2 (Ja_L + Ja_R) is a sum
    const double m1 = mL[0] + mR[0], m2 = mL[1] + mR[1], m3 = mL[2] + mR[2];
    if constexpr (VF == 1) {  // StandardDGFluxDealiasedMetricVec :446-494
      const double qL = L[5] * m1 + L[6] * m2 + L[7] * m3;
      const double qR = R[5] * m1 + R[6] * m2 + R[7] * m3;
      const double ps = L[8] + R[8];
      F[0] = 0.5 * (L[0] * qL + R[0] * qR);
      F[1] = 0.5 * (L[1] * qL + R[1] * qR + m1 * ps);
      F[2] = 0.5 * (L[2] * qL + R[2] * qR + m2 * ps);
      F[3] = 0.5 * (L[3] * qL + R[3] * qR + m3 * ps);
      F[4] = 0.5 * ((L[4] + L[8]) * qL + (R[4] + R[8]) * qR);
    } else if constexpr (VF == 2) {  // KennedyAndGruberFluxVec1 :731-803
      const double rhoHat = 0.5 * (L[0] + R[0]);
      const double uH = 0.5 * (L[1] + R[1]), vH = 0.5 * (L[2] + R[2]), wH = 0.5 * (L[3] + R[3]);
      const double p1 = 0.5 * (L[4] + R[4]);
      const double eH = 0.5 * (L[5] + R[5]);
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoHat * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = F[0] * eH + p1 * q;
    } else if constexpr (VF == 3) {  // DucrosFluxVec :986-1059 (records hold halves)
      const double q = (L[1] + R[1]) * m1 + (L[2] + R[2]) * m2 + (L[3] + R[3]) * m3;
      const double p1 = L[4] + R[4];
      F[0] = (L[0] + R[0]) * q;
      F[1] = (L[5] + R[5]) * q + m1 * p1;
      F[2] = (L[6] + R[6]) * q + m2 * p1;
      F[3] = (L[7] + R[7]) * q + m3 * p1;
      F[4] = ((L[8] + R[8]) + p1) * q;
    } else if constexpr (VF == 4) {  // MorinishiFluxVec :1121-1205
      const double uH = 0.5 * (L[1] + R[1]), vH = 0.5 * (L[2] + R[2]), wH = 0.5 * (L[3] + R[3]);
      const double p1 = 0.5 * (L[4] + R[4]);
      const double qL = L[1] * m1 + L[2] * m2 + L[3] * m3;
      const double qR = R[1] * m1 + R[2] * m2 + R[3] * m3;
      const double rq2L = 0.5 * L[0] * qL, rq2R = 0.5 * R[0] * qR;
      F[0] = rq2L + rq2R;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = 0.5 * (P.kappa * P.sKappaM1 * (L[4] * qL + R[4] * qR) - (rq2L * L[5] + rq2R * R[5])) +
             rq2L * (L[1] * uH + L[2] * vH + L[3] * wH) + rq2R * (R[1] * uH + R[2] * vH + R[3] * wH);
    } else if constexpr (VF == 6) {  // EntropyAndEnergyConservingFluxVec2 :1427-1504 (halves)
      const double rhoM = L[0] + R[0];
      const double sbM = 2. * rcp_nr(L[4] + R[4]);
      const double uH = L[1] + R[1], vH = L[2] + R[2], wH = L[3] + R[3];
      const double p1 = 0.5 * rhoM * sbM;
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoM * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = F[0] * 0.5 * (P.sKappaM1 * sbM - (L[5] + R[5])) + uH * F[1] + vH * F[2] + wH * F[3];
    } else if constexpr (VF == 7) {  // ggFluxVec :1575-1653 (halves)
      const double sbHat = mn[1];
      const double rhoM = L[0] + R[0];
      const double uH = L[1] + R[1], vH = L[2] + R[2], wH = L[3] + R[3];
      const double p1 = L[4] + R[4];
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoM * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = F[0] * 0.5 * (P.sKappaM1 * sbHat - (L[6] + R[6])) + uH * F[1] + vH * F[2] + wH * F[3];
    } else if constexpr (VF == 8) {  // KennedyAndGruberFluxVec2 :857-929 (halves)
      const double uH = L[1] + R[1], vH = L[2] + R[2], wH = L[3] + R[3];
      const double p1 = L[4] + R[4];
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = (L[0] + R[0]) * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = F[0] * (L[5] + R[5]);
    } else if constexpr (VF == 9) {  // GassnerWintersWalchFluxVec :1724-1799 (halves)
      const double rhoH = L[0] + R[0];
      const double uH = L[1] + R[1], vH = L[2] + R[2], wH = L[3] + R[3];
      const double HH = L[4] + R[4];
      const double p1 = P.kappaM1 * P.sKappa * (rhoH * HH - 0.5 * (uH * uH + vH * vH + wH * wH));
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoH * q;
      F[1] = q * uH + m1 * p1;
      F[2] = q * vH + m2 * p1;
      F[3] = q * wH + m3 * p1;
      F[4] = q * HH;
    } else if constexpr (VF == 5) {  // EntropyAndEnergyConservingFluxVec :1277-1356
      const double rhoHat = mn[0], sbHat = mn[1];        // LN(rho), 1/LN(beta)
      const double p1 = 0.5 * (L[0] + R[0]) * mn[2];     // 0.5*rho_mean/beta_mean
      const double uH = L[1] + R[1], vH = L[2] + R[2], wH = L[3] + R[3];  // records hold u/2, v/2, w/2
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoHat * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = F[0] * 0.5 * (P.sKappaM1 * sbHat - (L[5] + R[5])) + uH * F[1] + vH * F[2] + wH * F[3];
    } else if constexpr (VF == 10) {  // TwoPointEntropyConservingFluxVec :574-673
      const double z5LN = mn[0], is1 = mn[2];  // is1 = 1/(z1_L + z1_R)
      const double ratio = z5LN * mn[1];       // z5LN / z1LN
      const double rhoHat = 0.5 * (L[0] + R[0]) * z5LN;
      const double uH = (L[0] * L[1] + R[0] * R[1]) * is1;
      const double vH = (L[0] * L[2] + R[0] * R[2]) * is1;
      const double wH = (L[0] * L[3] + R[0] * R[3]) * is1;
      const double p1 = (L[4] + R[4]) * is1;
      const double q = uH * m1 + vH * m2 + wH * m3;
      F[0] = rhoHat * q;
      F[1] = F[0] * uH + m1 * p1;
      F[2] = F[0] * vH + m2 * p1;
      F[3] = F[0] * wH + m3 * p1;
      F[4] = 0.5 * (q * P.kappaP1 * P.sKappaM1 * ratio + uH * F[1] + vH * F[2] + wH * F[3]);
    } else if constexpr (VF == 32) {  // RanochaFluxVec :1876-1929
      const double rhoLN = mn[0], srspM = mn[1];  // LN(rho), 1/LN(rho/p)
      const double va1 = 0.5 * (L[1] + R[1]), va2 = 0.5 * (L[2] + R[2]), va3 = 0.5 * (L[3] + R[3]);
      const double v2zip = 0.5 * (L[1] * R[1] + L[2] * R[2] + L[3] * R[3]);
      const double pavg = 0.5 * (L[4] + R[4]);
      const double vmL = L[1] * m1 + L[2] * m2 + L[3] * m3;
      const double vmR = R[1] * m1 + R[2] * m2 + R[3] * m3;
      F[0] = rhoLN * 0.5 * (vmL + vmR);
      F[1] = F[0] * va1 + m1 * pavg;
      F[2] = F[0] * va2 + m2 * pavg;
      F[3] = F[0] * va3 + m3 * pavg;
      F[4] = F[0] * (v2zip + srspM * P.sKappaM1) + 0.5 * (L[4] * vmR + R[4] * vmL);
    }
  }
}

// the flux of one pair; lL, lR are the nodes' records (L and R may be copies without the logarithms)
template <int VF>
__device__ __forceinline__ void pair_flux(const KParams& P, const double* L, const double* R, const double* lL,
                                          const double* lR, const double* mL, const double* mR, double* F) {
  double mn[3];
  if (!pair_means<VF>(L, R, mn)) pair_means_fix<VF>(L, R, lL, lR, mn);
  pair_flux_from<VF>(P, L, R, mn, mL, mR, F);
}

// The fluxes F and H of the pairs (x0, y0) and (x1, y1), side by side: one branch off the series for both
template <int VF>
__device__ __forceinline__ void pair_flux2(const KParams& P, const double* x0, const double* y0, const double* l0,
                                           const double* k0, const double* m0, const double* n0, const double* x1,
                                           const double* y1, const double* l1, const double* k1, const double* m1,
                                           const double* n1, double* F, double* H) {
  double a[3], b[3];
  const bool sa = pair_means<VF>(x0, y0, a), sb = pair_means<VF>(x1, y1, b);
  if (!(sa && sb)) {
    pair_means_fix<VF>(x0, y0, l0, k0, a);
    pair_means_fix<VF>(x1, y1, l1, k1, b);
  }
  pair_flux_from<VF>(P, x0, y0, a, m0, n0, F);
  pair_flux_from<VF>(P, x1, y1, b, m1, n1, H);
}

}  // namespace fluxo
