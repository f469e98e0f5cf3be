// Adjoint of the step's microphysics (moist_physics_prep_em, WSM6 and
// moist_physics_finish_em: wrf_physics.py:27-91, 137-1214, 2106-2137).
//
// Every output of the block in a column (theta, qv .. qg, h_diabatic) is a
// function of that column's inputs only (t, qv .. qg, al, p below the top
// level and ph on every level; alb, pb and phb are data), so its reverse
// product is formed column by column, one thread per column.  The column is
// restated here as plain per-column code templated on its scalar type
// (column arrays in a global workspace) in the order of the reference's
// statements: the instantaneous processes, the source and sink rates with
// their limiters, the saturation adjustment, and the semi-Lagrangian
// sedimentation (nislfv_rain_plm / _plm6, wrf_physics.py:1216-1583) with its
// interface fall speeds, departure cells and overlap remap.  The derivative
// is that of the branch taken.
//
// With one time-split loop (the ordinary case) only the sedimentation couples
// the levels, so the block is reversed in two parts.  The masses that fall
// are taped column by column (tape.cuh) in the columns that hold some.  All
// else -- prep, the saturation ratios, melting, the point processes, finish --
// is reversed per level on a thread of its own by forward-mode tangents with
// respect to the level's nine inputs (temperature, vapour, cloud water,
// pressure, density and the four fallen masses): the cotangents of the fallen
// masses seed the tape, whose one reverse sweep gives the falling species'.
// With several loops the whole column runs on taped scalars, the outputs'
// cotangents seed the adjoints of their entries, and one reverse sweep yields
// every input's cotangent.
// Columns are taped in chunks that bound the tape's memory.  A column whose
// tape outgrows the capacity is finished by forward-mode tangents instead:
// the same code on Dual<N> numbers with N inputs seeded per pass, the
// cotangent of each seeded input the dot product of the outputs' cotangents
// with their tangents, ceil(n_inputs / N) passes per column.
#include "dual.cuh"
#include "kernels.cuh"
#include "tape.cuh"
#include "wsm6_const.cuh"

#include <algorithm>

namespace wrf {
namespace mpt {

using namespace mp;

// column arrays of one thread: array a, level k at base[(a * kst + k) * ncol]
template <class T>
struct Col {
  T* base;
  int ncol, kst;
  __device__ __forceinline__ T& operator()(int a, int k) const { return base[((size_t)a * kst + k) * ncol]; }
  __device__ __forceinline__ const T& temp(int k) const;
  __device__ __forceinline__ const T& den(int k) const;
  __device__ __forceinline__ const T& delz(int k) const;
  __device__ __forceinline__ const T& denfac(int k) const;
};

enum {
  A_TIN, A_TH, A_PII, A_T, A_Q, A_QC, A_QI, A_QR, A_QS, A_QG, A_DEN, A_P, A_DELZ, A_CPM, A_XL, A_DENFAC, A_QS0,
  A_QS1, A_RH0, A_RH1, A_XNI, A_R1, A_R2, A_R3, A_W1, A_W2, A_ZI, A_WI, A_ZA, A_DZA, A_QA, A_QA2, A_WD, A_WWW,
  A_SR3, A_SRS, A_COUNT
};
template <class T>
__device__ __forceinline__ const T& Col<T>::temp(int k) const { return (*this)(A_T, k); }
template <class T>
__device__ __forceinline__ const T& Col<T>::den(int k) const { return (*this)(A_DEN, k); }
template <class T>
__device__ __forceinline__ const T& Col<T>::delz(int k) const { return (*this)(A_DELZ, k); }
template <class T>
__device__ __forceinline__ const T& Col<T>::denfac(int k) const { return (*this)(A_DENFAC, k); }

template <class T>
__device__ __forceinline__ T cst(float x) {
  return Lift<T>::c(x);
}

template <class T>
__device__ __forceinline__ T n0sfac(const T& t) {
  return vmax(vmin(vexp(F(ALPHA) * (F(T0C) - t)), F(N0SMAX / N0S)), 1.0f);
}

// terminal velocity of one precipitating species (the slope with the rain
// caps), kind 0 rain, 1 snow, 2 graupel
template <class T>
__device__ T vt_of(int kind, const T& q, const T& den, const T& denfac, const T& t) {
  const float pidn0 = kind == 0 ? F(PIDN0R) : (kind == 1 ? F(PIDN0S) : F(PIDN0G));
  const float bv = kind == 0 ? F(BVTR) : (kind == 1 ? F(BVTS) : F(BVTG));
  const float pv = kind == 0 ? F(PVTR) : (kind == 1 ? F(PVTS) : F(PVTG));
  const bool small = val(q) <= F(QCRMIN);
  T rb;
  if (small) {
    rb = cst<T>(F(RSLOPERBMAX));
  } else {
    const T num = kind == 1 ? pidn0 * n0sfac(t) : cst<T>(pidn0);
    const T lam = vpow(num / (q * den), 0.25f);
    rb = vpow(1.0f / lam, bv);
  }
  return val(q) <= 0.f ? cst<T>(0.f) : pv * rb * denfac;
}

// whether any directional derivative of x is nonzero (always true for a
// plain float, whose value path is the point of running the code)
__device__ __forceinline__ bool live(float) { return true; }
template <int N>
__device__ __forceinline__ bool live(const Dual<N>& x) {
  bool any = false;
#pragma unroll
  for (int n = 0; n < N; ++n) any |= x.d[n] != 0.f;
  return any;
}
__device__ __forceinline__ bool live(const Tv& x) { return x.id >= 0; }

template <class T>
struct Slope3 {
  T rs[3], rb[3], r2[3], r3[3];
};

// slope_wsm6 (wrf_physics.py:2048-2104) at one level
template <class T>
__device__ void slope3(const T& qr, const T& qs, const T& qg, const T& den, const T& t, Slope3<T>& o) {
  const T q[3] = {qr, qs, qg};
  const float bv[3] = {F(BVTR), F(BVTS), F(BVTG)};
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    if (val(q[m]) <= F(QCRMIN)) {
      o.rs[m] = cst<T>(F(RSLOPERMAX));
      o.rb[m] = cst<T>(F(RSLOPERBMAX));
      o.r2[m] = cst<T>(F(RSLOPER2MAX));
      o.r3[m] = cst<T>(F(RSLOPER3MAX));
    } else {
      const T num = m == 0 ? cst<T>(F(PIDN0R)) : (m == 1 ? F(PIDN0S) * n0sfac(t) : cst<T>(F(PIDN0G)));
      const T a = 1.0f / vpow(num / (q[m] * den), 0.25f);
      o.rs[m] = a;
      o.rb[m] = vpow(a, bv[m]);
      o.r2[m] = a * a;
      o.r3[m] = a * a * a;
    }
  }
}

// saturation mixing ratios over water and (below the triple point) ice
template <class T>
__device__ void fpvs(const T& t, const T& p, T& qs0, T& qs1) {
  const double ttp = T0C + 0.01;
  const double dldt = CPV - CLIQ, xa = -dldt / RV, xb = xa + XLV0 / (RV * ttp);
  const double dldti = CPV - CICE, xai = -dldti / RV, xbi = xai + XLS / (RV * ttp);
  const T tr = F(ttp) / t;
  const T w1 = F(PSAT) * vexp(vlog(tr) * F(xa)) * vexp(F(xb) * (1.0f - tr));
  T a = vmin(w1, 0.99f * p);
  a = F(EP2) * a / (p - a);
  qs0 = vmax(a, F(QMIN));
  T b = w1;
  if (val(t) < F(ttp)) b = F(PSAT) * vexp(vlog(tr) * F(xai)) * vexp(F(xbi) * (1.0f - tr));
  b = vmin(b, 0.99f * p);
  b = F(EP2) * b / (p - b);
  qs1 = vmax(b, F(QMIN));
}

template <class T>
__device__ __forceinline__ T viscos(const T& t, const T& den) {
  return 1.496e-6f * (t * vsqrt(t)) / (t + 120.0f) / den;
}
template <class T>
__device__ __forceinline__ T diffus(const T& t, const T& p) {
  return 8.794e-5f * vexp(vlog(t) * 1.81f) / p;
}
template <class T>
__device__ __forceinline__ T xka(const T& t, const T& den) {
  return 1.414e3f * viscos(t, den) * den;
}
template <class T, class A>
__device__ __forceinline__ T diffac(const A& a, const T& p, const T& t, const T& den, const T& qs) {
  return den * a * a / (xka(t, den) * F(RV) * t * t) + 1.0f / (qs * diffus(t, p));
}
template <class T>
__device__ __forceinline__ T venfac(const T& p, const T& t, const T& den) {
  return vexp(vlog(viscos(t, den) / diffus(t, p)) * 0.3333333f) / vsqrt(viscos(t, den)) * vsqrt(vsqrt(F(DEN0) / den));
}

// interface fall speeds: 3rd-order interpolation of the cell speeds (www),
// the ww == 0 fallback and the downward CFL limiter (wrf_physics.py:1269-1293)
template <class T, class C_>
__device__ void fall_interfaces(const C_& C, int km, float dt) {
  const float fa1 = 9.0f / 16.0f, fa2 = 1.0f / 16.0f;
  C(A_WI, 0) = C(A_WWW, 0);
  C(A_WI, 1) = 0.5f * (C(A_WWW, 1) + C(A_WWW, 0));
  for (int k = 2; k < km - 1; ++k)
    C(A_WI, k) = fa1 * (C(A_WWW, k) + C(A_WWW, k - 1)) - fa2 * (C(A_WWW, k + 1) + C(A_WWW, k - 2));
  C(A_WI, km - 1) = 0.5f * (C(A_WWW, km - 1) + C(A_WWW, km - 2));
  C(A_WI, km) = C(A_WWW, km - 1);
  for (int k = 1; k < km; ++k)
    if (val(C(A_WWW, k)) == 0.f) C(A_WI, k) = C(A_WWW, k - 1);
  for (int k = km - 1; k >= 0; --k) {
    const T dz = C.delz(k);
    const T decfl = (C(A_WI, k + 1) - C(A_WI, k)) * dt / dz;
    if (val(decfl) > 0.05f) C(A_WI, k) = C(A_WI, k + 1) - 0.05f * dz / dt;
  }
}

// the piecewise-constant overlap remap of the departure cells' mass (array
// qa, the top cell's zeroed) onto the grid (wrf_physics.py:1339-1357, the
// last layers 3800 m deep), written into array out.  A pair of cells whose
// overlap is not positive contributes the constant 0 (value and
// derivatives), so the pairs are screened on the values first: only the
// few overlapping departure cells of a level enter the dual arithmetic.
template <class T, class C_>
__device__ void remap(const C_& C, int km, int qa, int out) {
  float za[kMaxNz + 1];
  for (int k = 0; k <= km; ++k) za[k] = val(C(A_ZA, k));
  for (int k = 0; k < km; ++k) {
    const T zlo = C(A_ZI, k);
    const T zhi = k < km - 1 ? C(A_ZI, k + 1) : C(A_ZI, km - 1) + 3800.0f;
    const float zlov = val(zlo), zhiv = val(zhi);
    T acc = cst<T>(0.f);
    for (int ka = 0; ka < km; ++ka) {
      const float alov = za[ka], ahiv = ka < km - 1 ? za[ka + 1] : za[km - 1] + 3800.0f;
      if (!(vmin(zhiv, ahiv) - vmax(zlov, alov) > 0.0f)) continue;
      const T alo = C(A_ZA, ka);
      const T ahi = ka < km - 1 ? C(A_ZA, ka + 1) : C(A_ZA, km - 1) + 3800.0f;
      const T ov = vmax(0.0f, vmin(zhi, ahi) - vmax(zlo, alo));
      acc = acc + C(qa, ka) * ov;
    }
    C(out, k) = acc / C.delz(k);
  }
}

// nislfv_rain_plm (kind 0, rain; kind 2, cloud ice with iter 0) and
// nislfv_rain_plm6 (kind 1: snow in r1 and graupel in r2 with the shared
// mass-weighted speed): the cell speeds are in A_W1, the masses (den q) in
// r1 (and r2), replaced by the sedimented masses.  (The surface flux feeds
// the precipitation accumulators only, which are not differentiated.)
template <class T, class C_>
__device__ void nislfv(const C_& C, int km, int kind, int r1, int r2, float dt, int iter) {
  float allold = 0.f;
  for (int k = 0; k < km; ++k) allold = allold + val(C(r1, k));
  if (kind == 1)
    for (int k = 0; k < km; ++k) allold = allold + val(C(r2, k));
  if (!(allold > 0.f)) {
    // nothing to fall: the scheme's result is zero (value and derivatives)
    for (int k = 0; k < km; ++k) {
      C(r1, k) = cst<T>(0.f);
      if (kind == 1) C(r2, k) = cst<T>(0.f);
    }
    return;
  }
  C(A_ZI, 0) = cst<T>(0.f);
  for (int k = 0; k < km; ++k) C(A_ZI, k + 1) = C(A_ZI, k) + C.delz(k);
  for (int k = 0; k < km; ++k) {
    C(A_WD, k) = C(A_W1, k);
    C(A_WWW, k) = C(A_W1, k);
  }
  const int npass = iter >= 1 ? 2 : 1;
  for (int n = 1; n <= npass; ++n) {
    fall_interfaces<T>(C, km, dt);
    for (int k = 0; k <= km; ++k) C(A_ZA, k) = C(A_ZI, k) - C(A_WI, k) * dt;
    for (int k = 0; k < km; ++k) C(A_DZA, k) = C(A_ZA, k + 1) - C(A_ZA, k);
    C(A_DZA, km) = C(A_ZI, km) - C(A_ZA, km);
    for (int k = 0; k < km; ++k) {
      C(A_QA, k) = C(r1, k) * C.delz(k) / C(A_DZA, k);
      if (kind == 1) C(A_QA2, k) = C(r2, k) * C.delz(k) / C(A_DZA, k);
    }
    C(A_QA, km) = cst<T>(0.f);
    if (kind == 1) C(A_QA2, km) = cst<T>(0.f);
    if (n <= iter) {
      for (int k = 0; k < km; ++k) {
        const T den = C.den(k), denfac = C.denfac(k);
        const T qr = C(A_QA, k) / den;
        T wa;
        if (kind == 1) {
          const T qr2 = C(A_QA2, k) / den;
          const T wa1 = vt_of(1, qr, den, denfac, C.temp(k));
          const T wa2 = vt_of(2, qr2, den, denfac, C.temp(k));
          const T tmp = vmax(qr + qr2, 1.0e-15f);
          wa = val(tmp) > 1.0e-15f ? (wa1 * qr + wa2 * qr2) / tmp : cst<T>(0.f);
        } else {
          wa = vt_of(0, qr, den, denfac, C.temp(k));
        }
        C(A_WWW, k) = 0.5f * (C(A_WD, k) + wa);
      }
    }
  }
  for (int sp = 0; sp < (kind == 1 ? 2 : 1); ++sp) {
    const int qa = sp == 0 ? A_QA : A_QA2, r = sp == 0 ? r1 : r2;
    C(qa, km - 1) = cst<T>(0.f);
    remap<T>(C, km, qa, r);
  }
}

// the rates' limiter: where source > value (and cnd), every listed rate is
// scaled by value / source
template <class T, int M>
__device__ __forceinline__ void limit(const T& value, const T& source, bool cnd, T* const (&r)[M]) {
  if (cnd && val(source) > val(value)) {
    const T f = value / source;
#pragma unroll
    for (int m = 0; m < M; ++m) *r[m] = *r[m] * f;
  }
}

// the processes after the sedimentation at one level (wrf_physics.py:
// 596-1203): instantaneous melting / freezing, the source and sink rates,
// the mass-conserving limiters and updates for T <= t0c and T > t0c, and the
// saturation adjustment.  t, q, qc, qi, qr, qs, qg are updated in place.
template <class T>
__device__ void point_processes(T& t, T& q, T& qc, T& qi, T& qr, T& qs, T& qg, const T& den, const T& p,
                                const T& denfac, const T& cpm, const T& xl, const T& qs0, const T& qs1,
                                const T& rh0, const T& rh1, const Slope3<T>& sl0, float dtcld) {
  const T zero = cst<T>(0.f);
  // instantaneous melting / freezing (supcol from the temperature on entry)
  T supcol = F(T0C) - t;
  T xlf3 = F(XLS) - xl;
  if (val(supcol) < 0.f && val(qi) > 0.f) {
    qc = qc + qi;
    t = t - xlf3 / cpm * qi;
    qi = zero;
  }
  if (val(supcol) > 40.f && val(qc) > 0.f) {
    qi = qi + qc;
    t = t + xlf3 / cpm * qc;
    qc = zero;
  }
  if (val(supcol) > 0.f && val(qc) > F(QMIN)) {
    const T pf = vmin(F(PFRZ1) * (vexp(F(PFRZ2) * vmin(supcol, 50.0f)) - 1.0f) * den / F(DENR) / F(XNCR) * qc * qc *
                          dtcld, qc);
    qi = qi + pf;
    t = t + xlf3 / cpm * pf;
    qc = qc - pf;
  }
  if (val(supcol) > 0.f && val(qr) > 0.f) {
    const T pf = vmin(F(20.0 * PI * PI * PFRZ1 * N0R * DENR) / den * (vexp(F(PFRZ2) * vmin(supcol, 50.0f)) - 1.0f) *
                          sl0.r3[0] * sl0.r3[0] * sl0.rs[0] * dtcld, qr);
    qg = qg + pf;
    t = t + xlf3 / cpm * pf;
    qr = qr - pf;
  }
  // rates
  Slope3<T> sl;
  slope3(qr, qs, qg, den, t, sl);
  // (terms of processes that cannot act at this point are not formed: most
  // points hold no precipitation, and these are most of the work)
  const bool precip = val(qr) > 0.f || val(qs) > 0.f || val(qg) > 0.f;
  T work1_0 = cst<T>(1.f), work1_1 = cst<T>(1.f), work2 = zero;
  if (precip) {
    work1_0 = diffac(xl, p, t, den, qs0);
    work2 = venfac(p, t, den);
  }
  if (val(t) < F(T0C) && (precip || val(qi) > 0.f)) work1_1 = diffac(F(XLS), p, t, den, qs1);
  T supsat = vmax(q, F(QMIN)) - qs0;
  T praut = zero, pracw = zero, prevp = zero;
  if (val(qc) > F(QC0)) praut = vmin(F(QCK1) * vpow(qc, 7.0f / 3.0f), qc / dtcld);
  if (val(qr) > F(QCRMIN) && val(qc) > F(QMIN))
    pracw = vmin(F(PACRR) * sl.r3[0] * sl.rb[0] * qc * denfac, qc / dtcld);
  if (val(qr) > 0.f) {
    const T coeres = sl.r2[0] * vsqrt(sl.rs[0] * sl.rb[0]);
    prevp = (rh0 - 1.0f) * (F(PRECR1) * sl.r2[0] + F(PRECR2) * work2 * coeres) / work1_0;
    if (val(prevp) < 0.f) {
      prevp = vmax(prevp, -qr / dtcld);
      prevp = vmax(prevp, supsat / dtcld / 2.0f);
    } else {
      prevp = vmin(prevp, supsat / dtcld / 2.0f);
    }
  }
  supcol = F(T0C) - t;
  T n0s = cst<T>(1.f);
  if (val(qs) > 0.f) n0s = vmax(vmin(vexp(F(ALPHA) * supcol), F(N0SMAX / N0S)), 1.0f);
  supsat = vmax(q, F(QMIN)) - qs1;
  const T satdt = supsat / dtcld;
  bool ifsat = false;
  T xni = cst<T>(1.0e3f), diameter = zero, vt2i = zero;
  if (val(supcol) > 0.f && val(qi) > 0.f) {
    xni = vmin(vmax(5.38e7f * vpow(den * vmax(qi, F(QMIN)), 0.75f), 1.0e3f), 1.0e6f);
    const T xmi = den * qi / xni;
    diameter = vmin(F(DICON) * vsqrt(xmi), F(DIMAX));
    if (precip) vt2i = 1.49e4f * vpow(diameter, 1.31f);
  }
  const T vt2r = F(PVTR) * sl.rb[0] * denfac;
  const T vt2s = F(PVTS) * sl.rb[1] * denfac;
  const T vt2g = F(PVTG) * sl.rb[2] * denfac;
  const T qsum = vmax(qs + qg, 1.0e-15f);
  const T vt2ave = val(qsum) > 1.0e-15f ? (vt2s * qs + vt2g * qg) / qsum : zero;
  T praci = zero, piacr = zero, psaci = zero, pgaci = zero, psacw = zero, pgacw = zero, paacw = zero;
  T pracs = zero, psacr = zero, pgacr = zero, pgacs = zero, pseml = zero, pgeml = zero;
  T pidep = zero, psdep = zero, pgdep = zero, pigen = zero, psaut = zero, pgaut = zero, psevp = zero, pgevp = zero;
  const bool cold = val(supcol) > 0.f;
  if (cold && val(qi) > F(QMIN)) {
    if (val(qr) > F(QCRMIN)) {
      const T acrfac = 2.0f * sl.r3[0] + 2.0f * diameter * sl.r2[0] + diameter * diameter * sl.rs[0];
      praci = vmin(F(PI) * qi * F(N0R) * vabs(vt2r - vt2i) * acrfac, qi / dtcld);
      piacr = vmin(F(PI * PI * AVTR * N0R * DENR) * xni * denfac * F(G6PBR) * (sl.r3[0] * sl.r3[0]) * sl.rb[0] /
                       24.0f / den,
                   qr / dtcld);
    }
    if (val(qs) > F(QCRMIN)) {
      const T eacrs = vexp(0.07f * (-supcol));
      const T acrfac = 2.0f * sl.r3[1] + 2.0f * diameter * sl.r2[1] + diameter * diameter * sl.rs[1];
      psaci = vmin(F(PI) * qi * eacrs * F(N0S) * n0s * vabs(vt2ave - vt2i) * acrfac / 4.0f, qi / dtcld);
    }
    if (val(qg) > F(QCRMIN)) {
      const T egi = vexp(-0.07f * supcol);
      const T acrfac = 2.0f * sl.r3[2] + 2.0f * diameter * sl.r2[2] + diameter * diameter * sl.rs[2];
      pgaci = vmin(F(PI) * egi * qi * F(N0G) * vabs(vt2ave - vt2i) * acrfac / 4.0f, qi / dtcld);
    }
  }
  if (val(qs) > F(QCRMIN) && val(qc) > F(QMIN))
    psacw = vmin(F(PACRC) * n0s * sl.r3[1] * sl.rb[1] * qc * denfac, qc / dtcld);
  if (val(qg) > F(QCRMIN) && val(qc) > F(QMIN)) pgacw = vmin(F(PACRC) * sl.r3[2] * sl.rb[2] * qc * denfac, qc / dtcld);
  if (val(qsum) > 1.0e-15f) paacw = (qs * psacw + qg * pgacw) / qsum;
  if (val(qs) > F(QCRMIN) && val(qr) > F(QCRMIN)) {
    if (cold) {
      const T acrfac = 5.0f * (sl.r3[1] * sl.r3[1]) * sl.rs[0] + 2.0f * sl.r3[1] * sl.r2[1] * sl.r2[0] +
                       0.5f * (sl.r2[1] * sl.r2[1]) * sl.r3[0];
      pracs = vmin(F(PI * PI * N0R * N0S) * n0s * vabs(vt2r - vt2ave) * (F(DENS) / den) * acrfac, qs / dtcld);
    }
    const T acrfac = 5.0f * (sl.r3[0] * sl.r3[0]) * sl.rs[1] + 2.0f * sl.r3[0] * sl.r2[0] * sl.r2[1] +
                     0.5f * (sl.r2[0] * sl.r2[0]) * sl.r3[1];
    psacr = vmin(F(PI * PI * N0R * N0S) * n0s * vabs(vt2r - vt2ave) * (F(DENR) / den) * acrfac, qr / dtcld);
  }
  if (val(qg) > F(QCRMIN) && val(qr) > F(QCRMIN)) {
    const T acrfac = 5.0f * (sl.r3[0] * sl.r3[0]) * sl.rs[2] + 2.0f * sl.r3[0] * sl.r2[0] * sl.r2[2] +
                     0.5f * (sl.r2[0] * sl.r2[0]) * sl.r3[2];
    pgacr = vmin(F(PI * PI * N0R * N0G) * vabs(vt2r - vt2ave) * (F(DENR) / den) * acrfac, qr / dtcld);
  }
  if (!cold) {  // supcol <= 0
    const T melt = F(CLIQ) * supcol * (paacw + psacr) / F(XLF0);
    if (val(qs) > 0.f) pseml = vmin(vmax(melt, -qs / dtcld), 0.0f);
    if (val(qg) > 0.f) pgeml = vmin(vmax(melt, -qg / dtcld), 0.0f);
  }
  if (cold) {
    if (val(qi) > 0.f && !ifsat) {
      pidep = 4.0f * diameter * xni * (rh1 - 1.0f) / work1_1;
      const T supice = satdt - prevp;
      if (val(pidep) < 0.f)
        pidep = vmax(vmax(vmax(pidep, satdt / 2.0f), supice), -qi / dtcld);
      else
        pidep = vmin(vmin(pidep, satdt / 2.0f), supice);
      if (fabsf(val(prevp + pidep)) >= fabsf(val(satdt))) ifsat = true;
    }
    if (val(qs) > 0.f && !ifsat) {
      const T coeres = sl.r2[1] * vsqrt(sl.rs[1] * sl.rb[1]);
      psdep = (rh1 - 1.0f) * n0s * (F(PRECS1) * sl.r2[1] + F(PRECS2) * work2 * coeres) / work1_1;
      const T supice = satdt - prevp - pidep;
      if (val(psdep) < 0.f)
        psdep = vmax(vmax(vmax(psdep, -qs / dtcld), satdt / 2.0f), supice);
      else
        psdep = vmin(vmin(psdep, satdt / 2.0f), supice);
      if (fabsf(val(prevp + pidep + psdep)) >= fabsf(val(satdt))) ifsat = true;
    }
    if (val(qg) > 0.f && !ifsat) {
      const T coeres = sl.r2[2] * vsqrt(sl.rs[2] * sl.rb[2]);
      pgdep = (rh1 - 1.0f) * (F(PRECG1) * sl.r2[2] + F(PRECG2) * work2 * coeres) / work1_1;
      const T supice = satdt - prevp - pidep - psdep;
      if (val(pgdep) < 0.f)
        pgdep = vmax(vmax(vmax(pgdep, -qg / dtcld), satdt / 2.0f), supice);
      else
        pgdep = vmin(vmin(pgdep, satdt / 2.0f), supice);
      if (fabsf(val(prevp + pidep + psdep + pgdep)) >= fabsf(val(satdt))) ifsat = true;
    }
    if (val(supsat) > 0.f && !ifsat) {
      const T supice = satdt - prevp - pidep - psdep - pgdep;
      const T roqi0 = 4.92e-11f * vpow(1.0e3f * vexp(0.1f * supcol), 1.33f);
      T pg = vmax(0.0f, (roqi0 / den - vmax(qi, 0.0f)) / dtcld);
      pigen = vmin(vmin(pg, satdt), supice);
    }
    if (val(qi) > 0.f) psaut = vmax(0.0f, (qi - F(ROQIMAX) / den) / dtcld);
    if (val(qs) > 0.f) pgaut = vmin(vmax(0.0f, 1.0e-3f * vexp(-0.09f * supcol) * (qs - F(QS0))), qs / dtcld);
  }
  if (val(supcol) < 0.f && val(rh0) < 1.f) {
    if (val(qs) > 0.f) {
      const T coeres = sl.r2[1] * vsqrt(sl.rs[1] * sl.rb[1]);
      psevp = vmin(vmax((rh0 - 1.0f) * n0s * (F(PRECS1) * sl.r2[1] + F(PRECS2) * work2 * coeres) / work1_0,
                        -qs / dtcld),
                   0.0f);
    }
    if (val(qg) > 0.f) {
      const T coeres = sl.r2[2] * vsqrt(sl.rs[2] * sl.rb[2]);
      pgevp = vmin(vmax((rh0 - 1.0f) * (F(PRECG1) * sl.r2[2] + F(PRECG2) * work2 * coeres) / work1_0, -qg / dtcld),
                   0.0f);
    }
  }
  // limiters and update, T <= t0c
  const float delta2 = (val(qr) < 1.0e-4f && val(qs) < 1.0e-4f) ? 1.f : 0.f;
  const float delta3 = val(qr) < 1.0e-4f ? 1.f : 0.f;
  bool cnd = val(t) <= F(T0C);
  {
    T* const r1[3] = {&praut, &pracw, &paacw};
    limit(vmax(F(QMIN), qc), (praut + pracw + paacw + paacw) * dtcld, cnd, r1);
    T* const r2[6] = {&psaut, &pigen, &pidep, &praci, &psaci, &pgaci};
    limit(vmax(F(QMIN), qi), (psaut - pigen - pidep + praci + psaci + pgaci) * dtcld, cnd, r2);
    T* const r3[6] = {&praut, &prevp, &pracw, &piacr, &psacr, &pgacr};
    limit(vmax(F(QMIN), qr), (-praut - prevp - pracw + piacr + psacr + pgacr) * dtcld, cnd, r3);
    const T src4 = -(psdep + psaut - pgaut + paacw + piacr * delta3 + praci * delta3 - pracs * (1.0f - delta2) +
                     psacr * delta2 + psaci - pgacs) * dtcld;
    T* const r4[10] = {&psdep, &psaut, &pgaut, &paacw, &piacr, &praci, &psaci, &pracs, &psacr, &pgacs};
    limit(vmax(F(QMIN), qs), src4, cnd, r4);
    const T src5 = -(pgdep + pgaut + piacr * (1.0f - delta3) + praci * (1.0f - delta3) + psacr * (1.0f - delta2) +
                     pracs * (1.0f - delta2) + pgaci + paacw + pgacr + pgacs) * dtcld;
    T* const r5[10] = {&pgdep, &pgaut, &piacr, &praci, &psacr, &pracs, &paacw, &pgaci, &pgacr, &pgacs};
    limit(vmax(F(QMIN), qg), src5, cnd, r5);
  }
  if (cnd) {
    work2 = -(prevp + psdep + pgdep + pigen + pidep);
    q = q + work2 * dtcld;
    qc = vmax(qc - (praut + pracw + paacw + paacw) * dtcld, 0.0f);
    qr = vmax(qr + (praut + pracw + prevp - piacr - pgacr - psacr) * dtcld, 0.0f);
    qi = vmax(qi - (psaut + praci + psaci + pgaci - pigen - pidep) * dtcld, 0.0f);
    qs = vmax(qs + (psdep + psaut + paacw - pgaut + piacr * delta3 + praci * delta3 + psaci - pgacs -
                    pracs * (1.0f - delta2) + psacr * delta2) * dtcld,
              0.0f);
    qg = vmax(qg + (pgdep + pgaut + piacr * (1.0f - delta3) + praci * (1.0f - delta3) + psacr * (1.0f - delta2) +
                    pracs * (1.0f - delta2) + pgaci + paacw + pgacr + pgacs) * dtcld,
              0.0f);
    xlf3 = F(XLS) - xl;
    const T xlwork2 = -F(XLS) * (psdep + pgdep + pidep + pigen) - xl * prevp -
                      xlf3 * (piacr + paacw + paacw + pgacr + psacr);
    t = t - xlwork2 / cpm * dtcld;
  }
  // T > t0c
  cnd = val(t) > F(T0C);
  {
    T* const r1[3] = {&praut, &pracw, &paacw};
    limit(vmax(F(QMIN), qc), (praut + pracw + paacw + paacw) * dtcld, cnd, r1);
    T* const r2[6] = {&praut, &prevp, &pracw, &paacw, &pseml, &pgeml};
    limit(vmax(F(QMIN), qr), (-paacw - praut + pseml + pgeml - pracw - paacw - prevp) * dtcld, cnd, r2);
    T* const r3[3] = {&pgacs, &psevp, &pseml};
    limit(vmax(F(QCRMIN), qs), (pgacs - pseml - psevp) * dtcld, cnd, r3);
    T* const r4[3] = {&pgacs, &pgevp, &pgeml};
    limit(vmax(F(QCRMIN), qg), -(pgacs + pgevp + pgeml) * dtcld, cnd, r4);
  }
  if (cnd) {
    work2 = -(prevp + psevp + pgevp);
    q = q + work2 * dtcld;
    qc = vmax(qc - (praut + pracw + paacw + paacw) * dtcld, 0.0f);
    qr = vmax(qr + (praut + pracw + prevp + paacw + paacw - pseml - pgeml) * dtcld, 0.0f);
    qs = vmax(qs + (psevp - pgacs + pseml) * dtcld, 0.0f);
    qg = vmax(qg + (pgacs + pgevp + pgeml) * dtcld, 0.0f);
    xlf3 = F(XLS) - xl;
    const T xlwork2 = -xl * (prevp + psevp + pgevp) - xlf3 * (pseml + pgeml);
    t = t - xlwork2 / cpm * dtcld;
  }
  // saturation adjustment
  T a0, a1;
  fpvs(t, p, a0, a1);
  const T w1 = (vmax(q, F(QMIN)) - a0) / (1.0f + xl * xl / (F(RV) * cpm) * a0 / (t * t));
  T pcond = vmin(vmax(w1 / dtcld, 0.0f), vmax(q, 0.0f) / dtcld);
  if (val(qc) > 0.f && val(w1) < 0.f) pcond = vmax(w1, -qc) / dtcld;
  q = q - pcond * dtcld;
  qc = vmax(qc + pcond * dtcld, 0.0f);
  t = t + pcond * xl / cpm * dtcld;
  if (val(qc) <= F(QMIN)) qc = zero;
  if (val(qi) <= F(QMIN)) qi = zero;
}

// melting of snow, then graupel (wrf_physics.py:415-470) at one level, and
// rain's slope before it (the others' are read where they melt only)
template <class T>
__device__ void melt_level(T& t, T& qr, T& qs, T& qg, const T& den, const T& p, const T& cpm, Slope3<T>& sl,
                           float dtcld) {
  const float xlf = F(XLF0);
  const bool warm = val(t) > F(T0C) && (val(qs) > 0.f || val(qg) > 0.f);
  const T none = cst<T>(0.f);
  slope3(qr, warm ? qs : none, warm ? qg : none, den, t, sl);
  if (!warm) return;
  const T n0s = val(qs) > 0.f ? n0sfac(t) : none;
  const T work2 = venfac(p, t, den);
  if (val(qs) > 0.f) {
    const T coeres = sl.r2[1] * vsqrt(sl.rs[1] * sl.rb[1]);
    T ps = xka(t, den) / xlf * (F(T0C) - t) * F(PI) / 2.0f * n0s *
           (F(PRECS1) * sl.r2[1] + F(PRECS2) * work2 * coeres) / den;
    ps = vmin(vmax(ps * dtcld / 1.0f, -qs / 1.0f), 0.0f);
    qs = qs + ps;
    qr = qr - ps;
    t = t + xlf / cpm * ps;
  }
  if (val(qg) > 0.f) {
    const T coeres = sl.r2[2] * vsqrt(sl.rs[2] * sl.rb[2]);
    T pg = xka(t, den) / xlf * (F(T0C) - t) * (F(PRECG1) * sl.r2[2] + F(PRECG2) * work2 * coeres) / den;
    pg = vmin(vmax(pg * dtcld / 1.0f, -qg / 1.0f), 0.0f);
    qg = qg + pg;
    qr = qr - pg;
    t = t + xlf / cpm * pg;
  }
}

// wsm6 (wrf_physics.py:137-1214) on one column of km levels: the arrays
// A_T (temperature), A_Q, A_QC, A_QI, A_QR, A_QS, A_QG, A_DEN, A_P and
// A_DELZ hold the inputs and receive the results
template <class T>
__device__ void wsm6_column(const Col<T>& C, int km, float delt, bool skip_dead = false) {
  for (int k = 0; k < km; ++k) {
    const T q = C(A_Q, k), t = C(A_T, k);
    C(A_CPM, k) = val(q) >= F(QMIN) ? F(CPV) * q + (1.0f - q) * F(CPD) : cst<T>(F(CPD * (1.0 - QMIN) + CPV * QMIN));
    C(A_XL, k) = F(XLV0) - F(XLV1) * (t - F(T0C));
    C(A_QC, k) = vmax(C(A_QC, k), 0.0f);
    C(A_QI, k) = vmax(C(A_QI, k), 0.0f);
    C(A_QR, k) = vmax(C(A_QR, k), 0.0f);
    C(A_QS, k) = vmax(C(A_QS, k), 0.0f);
    C(A_QG, k) = vmax(C(A_QG, k), 0.0f);
  }
  const float loops = fmaxf(delt / F(DTCLDCR), 1.0f);
  const float dtcld = delt <= F(DTCLDCR) ? delt : delt / loops;
  const int nloop = (int)loops;
  for (int it = 0; it < nloop; ++it) {
    bool rain = false, snow = false, ice = false;
    for (int k = 0; k < km; ++k) {
      rain |= val(C(A_QR, k)) > 0.f;
      snow |= val(C(A_QS, k)) > 0.f || val(C(A_QG, k)) > 0.f;
      ice |= val(C(A_QI, k)) > 0.f;
    }
    for (int k = 0; k < km; ++k) {
      const T den = C(A_DEN, k), t = C(A_T, k), q = C(A_Q, k);
      const T denfac = vsqrt(1.0f / den * F(DEN0));
      C(A_DENFAC, k) = denfac;
      T qs0, qs1;
      fpvs(t, C(A_P, k), qs0, qs1);
      C(A_QS0, k) = qs0;
      C(A_QS1, k) = qs1;
      C(A_RH0, k) = vmax(q / qs0, F(QMIN));
      C(A_RH1, k) = vmax(q / qs1, F(QMIN));
      const T qi = C(A_QI, k);
      if (val(qi) > 0.f)
        C(A_XNI, k) = vmin(vmax(5.387e7f * vpow(den * vmax(qi, F(QMIN)), 0.75f), 1.0e3f), 1.0e6f);
      const T qr = C(A_QR, k), qs = C(A_QS, k), qg = C(A_QG, k);
      C(A_W1, k) = vt_of(0, qr, den, denfac, t);
      const T qsum = vmax(qs + qg, 1.0e-15f);
      C(A_W2, k) = val(qsum) > 1.0e-15f
                       ? (vt_of(1, qs, den, denfac, t) * qs + vt_of(2, qg, den, denfac, t) * qg) / qsum
                       : cst<T>(0.f);
      // (the masses of a species that the column does not hold fall nowhere)
      C(A_R1, k) = rain ? den * qr : cst<T>(0.f);
      C(A_R2, k) = snow ? den * qs : cst<T>(0.f);
      C(A_R3, k) = snow ? den * qg : cst<T>(0.f);
    }
    nislfv<T>(C, km, 0, A_R1, -1, dtcld, 1);
    for (int k = 0; k < km; ++k) C(A_W1, k) = C(A_W2, k);
    nislfv<T>(C, km, 1, A_R2, A_R3, dtcld, 1);
    for (int k = 0; k < km; ++k) {
      const T den = C(A_DEN, k), p = C(A_P, k), cpm = C(A_CPM, k);
      T qr = vmax(C(A_R1, k) / den, 0.0f), qs = vmax(C(A_R2, k) / den, 0.0f), qg = vmax(C(A_R3, k) / den, 0.0f);
      T t = C(A_T, k);
      Slope3<T> sl;
      melt_level(t, qr, qs, qg, den, p, cpm, sl, dtcld);
      C(A_SR3, k) = sl.r3[0];
      C(A_SRS, k) = sl.rs[0];
      C(A_QR, k) = qr;
      C(A_QS, k) = qs;
      C(A_QG, k) = qg;
      C(A_T, k) = t;
      // cloud-ice fall speed and mass
      const T qi = C(A_QI, k);
      if (val(qi) <= 0.f) {
        C(A_W1, k) = cst<T>(0.f);
      } else {
        T wt = vmax(vmin(F(DICON) * vsqrt(den * qi / C(A_XNI, k)), F(DIMAX)), 1.0e-25f);
        C(A_W1, k) = 1.49e4f * vexp(vlog(wt) * 1.31f);
      }
      C(A_R1, k) = ice ? den * qi : cst<T>(0.f);
    }
    nislfv<T>(C, km, 2, A_R1, -1, dtcld, 0);
    for (int k = 0; k < km; ++k) {
      T t = C(A_T, k), q = C(A_Q, k), qc = C(A_QC, k), qr = C(A_QR, k), qs = C(A_QS, k), qg = C(A_QG, k);
      const T den = C(A_DEN, k);
      T qi = vmax(C(A_R1, k) / den, 0.0f);
      // a level whose every operand has zero tangents keeps zero tangents
      // through the processes; its values are not needed when only the
      // derivatives are wanted and no later time-split loop reads them
      if (skip_dead && it == nloop - 1 && !(live(t) || live(q) || live(qc) || live(qr) || live(qs) || live(qg) || live(den) ||
                         live(qi) || live(C(A_P, k)) || live(C(A_DENFAC, k)) || live(C(A_CPM, k)) ||
                         live(C(A_XL, k)) || live(C(A_QS0, k)) || live(C(A_QS1, k)) || live(C(A_RH0, k)) ||
                         live(C(A_RH1, k)) || live(C(A_SR3, k)) || live(C(A_SRS, k))))
        continue;
      Slope3<T> sl0;
      sl0.r3[0] = C(A_SR3, k);
      sl0.rs[0] = C(A_SRS, k);
      point_processes(t, q, qc, qi, qr, qs, qg, den, C(A_P, k), C(A_DENFAC, k), C(A_CPM, k), C(A_XL, k),
                      C(A_QS0, k), C(A_QS1, k), C(A_RH0, k), C(A_RH1, k), sl0, dtcld);
      C(A_T, k) = t;
      C(A_Q, k) = q;
      C(A_QC, k) = qc;
      C(A_QI, k) = qi;
      C(A_QR, k) = qr;
      C(A_QS, k) = qs;
      C(A_QG, k) = qg;
    }
  }
}

// the columns of moist_physics_prep_em's block ([jds+1, jde-1) x [ids+1,
// ide-1)), numbered row by row; WSM6 runs on [jds+1, jde-2) x [ids+1,
// ide-2) of them (run), the others only take the prep and finish
struct ColPos {
  int c2;
  bool run;
};
__device__ __forceinline__ bool col_pos(const Grid& g, int col, ColPos& o) {
  const int wi = g.ide - 1 - (g.ids + 1), wj = g.jde - 1 - (g.jds + 1);
  if (col >= wi * wj) return false;
  const int j = g.jds + 1 + col / wi, i = g.ids + 1 + col % wi;
  o.c2 = g.i2(j, i);
  o.run = j < g.jde - 2 && i < g.ide - 2;
  return true;
}

// the column's inputs are numbered t, qv, qc, qr, qi, qs, qg, al, p at
// levels < km (9 km indices: field f at level k is f km + k), then ph at
// levels < km + 1
__host__ __device__ __forceinline__ int mp_inputs(const Grid& g) { return 9 * (g.nz - 1) + g.nz; }

// moist_physics_prep_em (wrf_physics.py:27-91): theta, Exner function,
// temperature, density, pressure and layer depths of the column and its
// moisture into the column arrays; in(idx, value) makes input idx
template <class T, class In>
__device__ void prep_column(const Grid& g, const S& s, const Col<T>& C, int c2, In in) {
  const int km = g.nz - 1;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const int slot_of[6] = {A_Q, A_QC, A_QR, A_QI, A_QS, A_QG};
  for (int k = 0; k < km; ++k) {
    const size_t p = k * lev + c2;
    const T tin = in(k, s[WF_T][p]);
    C(A_TIN, k) = tin;
    const T th = tin + (float)T0;
    C(A_TH, k) = th;
    const T pfull = in(8 * km + k, s[WF_P][p]) + s[WF_PB][p];
    const T pii = vpow(pfull / (float)P0, F(RCP));
    C(A_PII, k) = pii;
    C(A_T, k) = th * pii;
    C(A_DEN, k) = 1.0f / (in(7 * km + k, s[WF_AL][p]) + s[WF_ALB][p]);
    C(A_P, k) = pfull;
    const T zlo = (in(9 * km + k, s[WF_PH][p]) + s[WF_PHB][p]) / (float)G;
    const T zhi = (in(9 * km + k + 1, s[WF_PH][p + lev]) + s[WF_PHB][p + lev]) / (float)G;
    C(A_DELZ, k) = zhi - zlo;
    for (int m = 1; m < 7; ++m) C(slot_of[m - 1], k) = in(m * km + k, s[WF_MOIST][m * n3 + p]);
  }
}

// moist_physics_finish_em (wrf_physics.py:2106-2137) at level k: theta's
// new value replaces A_TIN, h_diabatic replaces A_TH
template <class T>
__device__ __forceinline__ void finish_level(const Col<T>& C, int k, float dt) {
  const T mpten = C(A_T, k) / C(A_PII, k) - C(A_TH, k);
  C(A_TIN, k) = C(A_TIN, k) + mpten;
  C(A_TH, k) = mpten / dt;
}

// the array holding moist species m (1 qv .. 6 qg) in the column
__device__ __forceinline__ int moist_slot(int m) {
  const int slot_of[6] = {A_Q, A_QC, A_QR, A_QI, A_QS, A_QG};
  return slot_of[m - 1];
}

// a column that takes no process at all: no cloud, rain, ice, snow or
// graupel at any level, and qv below both saturation mixing ratios
// everywhere.  Every rate is zero, nothing falls, the saturation adjustment
// condenses nothing, and its reverse product is theta's and qv's
// cotangents passed through, zero for the hydrometeors (their results are
// constants: the zero of the empty sedimentation and the final zeroing of
// cloud and ice) and for h_diabatic.
__device__ bool quiet_column(const Grid& g, const S& s, int c2) {
  const int km = g.nz - 1;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  for (int k = 0; k < km; ++k) {
    const size_t p = k * lev + c2;
    for (int m = 2; m < 7; ++m)
      if (s[WF_MOIST][m * n3 + p] > 0.f) return false;
    const float th = s[WF_T][p] + (float)T0;
    const float pfull = s[WF_P][p] + s[WF_PB][p];
    const float t = th * wpow(pfull / (float)P0, F(RCP));
    float qs0, qs1;
    fpvs(t, pfull, qs0, qs1);
    const float qv = s[WF_MOIST][n3 + p];
    if (!(qv < qs0 && qv < qs1)) return false;
  }
  return true;
}

// the cotangent v of input idx into the cotangent table: assigned for t and
// the moisture (the block overwrites them), added for al, p and ph
__device__ __forceinline__ void put_input_cot(const Grid& g, const S& b, int c2, int idx, float v) {
  const int km = g.nz - 1;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  if (idx >= 9 * km) {
    b[WF_PH][(size_t)(idx - 9 * km) * lev + c2] += v;
    return;
  }
  const int f = idx / km, k = idx - f * km;
  const size_t p = k * lev + c2;
  if (f == 0) b[WF_T][p] = v;
  else if (f < 7) b[WF_MOIST][f * n3 + p] = v;
  else if (f == 7) b[WF_AL][p] += v;
  else b[WF_P][p] += v;
}

// the taped forward over the columns [c0, c0 + nc) (lane l of the launch
// takes column c0 + l; tape and column arrays interleaved with the
// context's stride): the column runs once on taped scalars and the
// outputs' cotangents yb (theta, qv .. qg, h_diabatic) seed their entries'
// adjoints.  Columns outside WSM6's block pass t and q through and set
// h_diabatic to zero; quiet columns pass theta's and qv's cotangents
// through (unless the values are wanted); both are done here.  vo (when
// its T is not null) receives the outputs' values.  used[col] receives the
// entries the column's tape took (0 when none) and done[col] whether its
// cotangents are (or, after k_mp_tape_rev, will be) written: not when the
// tape outgrew the capacity.
__global__ void __launch_bounds__(kTapeBlock) k_mp_tape(Grid g, S s, S yb, S b, float dt, Tv* ws, TapeCtx tc,
                                                        int c0, int nc, S vo, int* done, int* used) {
  tape_open(tc);
  const int lane = tape_lane(), col = c0 + lane;
  ColPos cp;
  if (lane >= nc || !col_pos(g, col, cp)) return;
  const int km = g.nz - 1, c2 = cp.c2;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const bool want = vo[WF_T] != nullptr;
  used[col] = 0;
  done[col] = 1;
  if (!cp.run) {
    for (int k = 0; k < km; ++k) {
      const size_t p = k * lev + c2;
      b[WF_T][p] = yb[WF_T][p];
      for (int m = 1; m < 7; ++m) b[WF_MOIST][m * n3 + p] = yb[WF_MOIST][m * n3 + p];
      b[WF_H_DIABATIC][p] = 0.f;
      if (want) {
        vo[WF_T][p] = s[WF_T][p];
        for (int m = 1; m < 7; ++m) vo[WF_MOIST][m * n3 + p] = s[WF_MOIST][m * n3 + p];
        vo[WF_H_DIABATIC][p] = 0.f;
      }
    }
    return;
  }
  if (!want && quiet_column(g, s, c2)) {
    for (int k = 0; k < km; ++k) {
      const size_t p = k * lev + c2;
      b[WF_T][p] = yb[WF_T][p];
      b[WF_MOIST][n3 + p] = yb[WF_MOIST][n3 + p];
      for (int m = 2; m < 7; ++m) b[WF_MOIST][m * n3 + p] = 0.f;
      b[WF_H_DIABATIC][p] = 0.f;
    }
    return;
  }
  const Col<Tv> C{ws + lane, tc.stride, km + 1};
  tape_reserve(mp_inputs(g));
  prep_column(g, s, C, c2, [](int idx, float v) { return Tv{v, idx, 1.f}; });
  wsm6_column(C, km, dt);
  for (int k = 0; k < km; ++k) finish_level(C, k, dt);
  const int n = g_tape_n[threadIdx.x];
  used[col] = n;
  if (want)
    for (int k = 0; k < km; ++k) {
      const size_t p = k * lev + c2;
      vo[WF_T][p] = C(A_TIN, k).v;
      vo[WF_H_DIABATIC][p] = C(A_TH, k).v;
      for (int m = 1; m < 7; ++m) vo[WF_MOIST][m * n3 + p] = C(moist_slot(m), k).v;
    }
  for (int k = 0; k < km; ++k) b[WF_H_DIABATIC][k * lev + c2] = 0.f;
  if (n > tc.cap) {
    done[col] = 0;
    return;
  }
  auto seed = [&](const Tv& y, float w) {
    if (y.id >= 0 && w != 0.f) *tc.adj(y.id, lane) += w * y.s;
  };
  for (int k = 0; k < km; ++k) {
    const size_t p = k * lev + c2;
    seed(C(A_TIN, k), yb[WF_T][p]);
    seed(C(A_TH, k), yb[WF_H_DIABATIC][p]);
    for (int m = 1; m < 7; ++m) seed(C(moist_slot(m), k), yb[WF_MOIST][m * n3 + p]);
  }
}

// ---- one time-split loop: the sedimentation on a tape, the rest per level

// the level's values that the kernels below share (float arrays in the slots
// of the column arrays)
enum { B_T, B_PII, B_DEN, B_DELZ, B_COUNT };
struct Base {
  float* base;
  int ncol, kst;
  __device__ __forceinline__ float& operator()(int a, int k) const {
    return base[((size_t)a * kst + k) * ncol];
  }
};
__device__ __forceinline__ Base base_of(Tv* ws, int lane, int stride, int kst) {
  return Base{reinterpret_cast<float*>(ws) + lane, stride, kst};
}

// The three falls -- rain, snow with graupel, cloud ice -- read the level's
// values only, so each is taped by a thread of its own, on a tape of its own
// (a share of the column's capacity) over column arrays of its own: A_R1,
// A_R2 the masses, A_W2 the density factor, the rest as in nislfv.  Its inputs
// are density and depth, then the species' and, for snow, the temperature.
enum { FALL_RAIN, FALL_SNOW, FALL_ICE, FALLS };
enum { I_DEN, I_DELZ, I_Q, I_Q2, I_T };
constexpr int kFallArrays = A_WWW - A_R1 + 1;
constexpr int kFallSlots = FALLS * kFallArrays + (B_COUNT + 2) / 3;  // arrays of Tv
__host__ __device__ constexpr int fall_inputs(int f) { return f == FALL_SNOW ? 5 : 3; }
// entries per level: at most 45, 82 and 26 where each level overlaps two
// departure cells, and as much again for those that overlap more
__host__ __device__ constexpr int fall_share(int f) { return f == FALL_RAIN ? 75 : (f == FALL_SNOW ? 138 : 53); }
__device__ __forceinline__ TapeCtx fall_tape(const TapeCtx& tc, int f) {
  constexpr int all = fall_share(0) + fall_share(1) + fall_share(2);
  auto part = [&](int shares) { return (int)((long long)tc.cap * shares / all); };
  const int c0 = f == FALL_RAIN ? 0 : part(f == FALL_SNOW ? fall_share(0) : fall_share(0) + fall_share(1));
  const int c1 = f == FALL_RAIN ? part(fall_share(0)) : (f == FALL_SNOW ? part(fall_share(0) + fall_share(1)) : tc.cap);
  return TapeCtx{tc.rec + (size_t)c0 * tc.stride, tc.stride, c1 - c0};
}

struct FallCol {
  Tv* base;  // array A_R1
  int ncol, kst, km;
  Base B;
  __device__ __forceinline__ Tv& operator()(int a, int k) const {
    return base[((size_t)(a - A_R1) * kst + k) * ncol];
  }
  __device__ __forceinline__ Tv in(int f, int k, float v) const { return Tv{v, f * km + k, 1.f}; }
  __device__ __forceinline__ Tv den(int k) const { return in(I_DEN, k, B(B_DEN, k)); }
  __device__ __forceinline__ Tv delz(int k) const { return in(I_DELZ, k, B(B_DELZ, k)); }
  __device__ __forceinline__ Tv temp(int k) const { return in(I_T, k, B(B_T, k)); }
  __device__ __forceinline__ const Tv& denfac(int k) const { return (*this)(A_W2, k); }
};
__device__ __forceinline__ FallCol fall_col(Tv* ws, int f, int lane, int stride, int km) {
  const size_t array = (size_t)(km + 1) * stride;
  return FallCol{ws + ((B_COUNT + 2) / 3 + f * kFallArrays) * array + lane, stride, km + 1, km,
                 base_of(ws, lane, stride, km + 1)};
}

// moist_physics_prep_em of one level per thread (neighbouring threads take
// neighbouring columns); used[f * ncol + col] (zero on entry) becomes 1
// where fall f has mass, done[col] 1, or 0 where the tapes are too small for any
// column.  Columns outside WSM6's block pass t and q through and set
// h_diabatic to zero.
__global__ void __launch_bounds__(128) k_mp_levels(Grid g, S s, S yb, S b, Tv* ws, TapeCtx tc, int c0, int nc, S vo,
                                                   int* done, int* used, int ncol) {
  const int km = g.nz - 1;
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(x / nc), lane = (int)(x - (long long)k * nc);
  if (k >= km) return;
  const int col = c0 + lane;
  ColPos cp;
  col_pos(g, col, cp);
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3(), p = k * lev + cp.c2;
  if (k == 0) done[col] = !cp.run || tc.cap >= mp_inputs(g);
  if (!cp.run) {
    b[WF_T][p] = yb[WF_T][p];
    for (int m = 1; m < 7; ++m) b[WF_MOIST][m * n3 + p] = yb[WF_MOIST][m * n3 + p];
    b[WF_H_DIABATIC][p] = 0.f;
    if (vo[WF_T]) {
      vo[WF_T][p] = s[WF_T][p];
      for (int m = 1; m < 7; ++m) vo[WF_MOIST][m * n3 + p] = s[WF_MOIST][m * n3 + p];
      vo[WF_H_DIABATIC][p] = 0.f;
    }
    return;
  }
  const Base B = base_of(ws, lane, tc.stride, km + 1);
  const float pii = wpow((s[WF_P][p] + s[WF_PB][p]) / (float)P0, F(RCP));
  B(B_PII, k) = pii;
  B(B_T, k) = (s[WF_T][p] + (float)T0) * pii;
  B(B_DEN, k) = 1.0f / (s[WF_AL][p] + s[WF_ALB][p]);
  B(B_DELZ, k) = (s[WF_PH][p + lev] + s[WF_PHB][p + lev]) / (float)G - (s[WF_PH][p] + s[WF_PHB][p]) / (float)G;
  const float* q = s[WF_MOIST];
  if (q[3 * n3 + p] > 0.f) used[FALL_RAIN * ncol + col] = 1;
  if (q[5 * n3 + p] > 0.f || q[6 * n3 + p] > 0.f) used[FALL_SNOW * ncol + col] = 1;
  if (q[4 * n3 + p] > 0.f) used[FALL_ICE * ncol + col] = 1;
}

// The sedimentation of the columns that hold falling species, taped: one
// thread per column and fall (blockIdx.y), the fallen masses (den q) left in
// A_R1 and A_R2 of the fall's arrays.  used receives the entries each tape
// took, 0 without a tape; done[col] becomes 0 where one outgrew its capacity.
// A column's chain of levels is bound by its own latencies: the three falls
// side by side take 1.1 and 0.6 ms (tape and sweep) at 101x101x35 where one
// after another they took 2.0 and 1.1, and 2.1 and 1.2 against 3.8 and 1.4 at
// 240x240x41.
__global__ void __launch_bounds__(kTapeBlock) k_mp_fall(Grid g, S s, float dt, Tv* ws, TapeCtx tc, int c0, int nc,
                                                        int* done, int* used, int ncol) {
  const int f = blockIdx.y;
  const TapeCtx tf = fall_tape(tc, f);
  tape_open(tf);
  const int lane = tape_lane(), col = c0 + lane, km = g.nz - 1;
  ColPos cp;
  if (lane >= nc || !col_pos(g, col, cp)) return;
  int& entries = used[f * ncol + col];
  if (!cp.run || !entries) return;
  if (tc.cap < mp_inputs(g)) {
    entries = 0;
    return;
  }
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const FallCol C = fall_col(ws, f, lane, tc.stride, km);
  const float loops = fmaxf(dt / F(DTCLDCR), 1.0f);
  const float dtcld = dt <= F(DTCLDCR) ? dt : dt / loops;
  tape_reserve(fall_inputs(f) * km);
  const float* q = s[WF_MOIST] + cp.c2;
  const Tv none = cst<Tv>(0.f);
  for (int k = 0; k < km; ++k, q += lev) {
    const Tv den = C.den(k), denfac = f == FALL_ICE ? none : vsqrt(1.0f / den * F(DEN0));
    if (f != FALL_ICE) C(A_W2, k) = denfac;
    if (f == FALL_RAIN) {
      const Tv qr = vmax(C.in(I_Q, k, q[3 * n3]), 0.0f);
      C(A_W1, k) = vt_of(0, qr, den, denfac, none);
      C(A_R1, k) = den * qr;
    } else if (f == FALL_SNOW) {
      const Tv t = C.temp(k), qs = vmax(C.in(I_Q, k, q[5 * n3]), 0.0f), qg = vmax(C.in(I_Q2, k, q[6 * n3]), 0.0f);
      const Tv qsum = vmax(qs + qg, 1.0e-15f);
      C(A_W1, k) = val(qsum) > 1.0e-15f
                       ? (vt_of(1, qs, den, denfac, t) * qs + vt_of(2, qg, den, denfac, t) * qg) / qsum
                       : none;
      C(A_R1, k) = den * qs;
      C(A_R2, k) = den * qg;
    } else {
      const Tv qi = vmax(C.in(I_Q, k, q[4 * n3]), 0.0f);
      Tv w = none;
      if (val(qi) > 0.f) {
        const Tv xni = vmin(vmax(5.387e7f * vpow(den * vmax(qi, F(QMIN)), 0.75f), 1.0e3f), 1.0e6f);
        const Tv wt = vmax(vmin(F(DICON) * vsqrt(den * qi / xni), F(DIMAX)), 1.0e-25f);
        w = 1.49e4f * vexp(vlog(wt) * 1.31f);
      }
      C(A_W1, k) = w;
      C(A_R1, k) = den * qi;
    }
  }
  // kinds 0, 1 and 2 as the falls; cloud ice takes no second pass
  nislfv<Tv>(C, km, f, A_R1, f == FALL_SNOW ? A_R2 : -1, dtcld, f == FALL_ICE ? 0 : 1);
  const int n = g_tape_n[threadIdx.x];
  entries = n;
  if (n > tf.cap) done[col] = 0;
}

// All but the sedimentation of one level, reversed by forward-mode tangents:
// one thread per (column, level) evaluates the level in Dual<N> arithmetic
// with N of its nine inputs seeded per pass -- temperature, vapour, cloud
// water, pressure, density and the fallen masses -- forms their cotangents
// from the outputs' (yb: theta, qv .. qg, h_diabatic), adds those of the
// fallen masses into the adjoints of the tape entries they come from, and
// writes prep's inputs' cotangents (the falling species' own are the tape's).
// vo (when its T is not null) receives the level's output values.
//
// The evaluation is a chain of powers, divisions and selections: what counts
// is how often it runs.  Only inputs that can act are seeded, packed over the
// passes (nine at most, where the saturation ratios, slopes and heat
// capacities as inputs of their own made eighteen), and a level with nothing
// to condense, freeze or fall runs it not at all: its derivatives are the
// identity.  A warp runs every branch that one of its points takes, so a block
// first sorts its points: the quiet ones are done on the spot, those with
// precipitation are listed from the front, the others from the back, and the
// evaluations run down the list.  The code is larger than the instruction
// caches, and three directions at a time keep it smallest for its use: 2.5 ms
// at 240x240x41 with three, 3.1 with two, 3.2 with four, 3.1 with six; 4.5
// unsorted with four.
enum { X_T, X_Q, X_QC, X_P, X_DEN, X_RR, X_RS, X_RG, X_RI, X_COUNT };
constexpr int kLvBlock = 128;
template <int N, int kLvPoints>  // directions, points per thread
__global__ void __launch_bounds__(kLvBlock) k_mp_levels_adj(Grid g, S s, S yb, S b, Tv* ws, TapeCtx tc, int c0, int nc,
                                                            S vo, const int* done, const int* used, int ncol, float dt) {
  __shared__ int list[kLvBlock * kLvPoints], nfront, nback;
  const int km = g.nz - 1;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  const long long x0 = (long long)blockIdx.x * (kLvBlock * kLvPoints);
  if (threadIdx.x == 0) nfront = nback = 0;
  __syncthreads();
  // a point's place and inputs
  struct Point {
    int k, lane, col;
    size_t p;
    float v[X_COUNT], tin, pii;
    Tv fall[4];
  };
  auto point = [&](int e, Point& o) {
    const long long x = x0 + e;
    o.k = (int)(x / nc);
    o.lane = (int)(x - (long long)o.k * nc);
    if (o.k >= km) return false;
    o.col = c0 + o.lane;
    ColPos cp;
    col_pos(g, o.col, cp);
    if (!cp.run || !done[o.col]) return false;
    const size_t p = o.p = o.k * lev + cp.c2;
    const Base B = base_of(ws, o.lane, tc.stride, km + 1);
    o.tin = s[WF_T][p];
    o.pii = B(B_PII, o.k);
    o.v[X_T] = B(B_T, o.k);
    o.v[X_Q] = s[WF_MOIST][n3 + p];
    o.v[X_QC] = s[WF_MOIST][2 * n3 + p];
    o.v[X_P] = s[WF_P][p] + s[WF_PB][p];
    o.v[X_DEN] = B(B_DEN, o.k);
#pragma unroll
    for (int q = 0; q < 4; ++q) o.fall[q] = cst<Tv>(0.f);
    // (X_RR, X_RS, X_RG, X_RI)
    if (used[FALL_RAIN * ncol + o.col]) o.fall[0] = fall_col(ws, FALL_RAIN, o.lane, tc.stride, km)(A_R1, o.k);
    if (used[FALL_SNOW * ncol + o.col]) {
      const FallCol C = fall_col(ws, FALL_SNOW, o.lane, tc.stride, km);
      o.fall[1] = C(A_R1, o.k);
      o.fall[2] = C(A_R2, o.k);
    }
    if (used[FALL_ICE * ncol + o.col]) o.fall[3] = fall_col(ws, FALL_ICE, o.lane, tc.stride, km)(A_R1, o.k);
#pragma unroll
    for (int q = 0; q < 4; ++q) o.v[X_RR + q] = o.fall[q].v;
    return true;
  };
  // the fallen masses' cotangents into the tapes
  auto to_tape = [&](const Point& o, const float* cot) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (o.fall[q].id >= 0 && cot[X_RR + q] != 0.f)
        atomicAdd(fall_tape(tc, q == 0 ? FALL_RAIN : (q == 3 ? FALL_ICE : FALL_SNOW)).adj(o.fall[q].id, o.lane),
                  cot[X_RR + q] * o.fall[q].s);
  };
  // moist_physics_finish_em: mpten = t / pii - th is added to theta and
  // gives h_diabatic = mpten / dt
  auto theta_out = [&](const Point& o, float tout) {
    const float mpten = tout / o.pii - (o.tin + (float)T0);
    vo[WF_T][o.p] = o.tin + mpten;
    vo[WF_H_DIABATIC][o.p] = mpten / dt;
  };
  // no hydrometeors, no condensation; no nucleation of ice
  auto is_dry = [](const float* v) {
    return v[X_QC] <= 0.f && v[X_RR] == 0.f && v[X_RS] == 0.f && v[X_RG] == 0.f && v[X_RI] == 0.f;
  };
  bool own = false;  // (one point a thread) the evaluation is this thread's
#pragma unroll 1
  for (int e = threadIdx.x; e < kLvBlock * kLvPoints; e += kLvBlock) {
    Point o;
    if (!point(e, o)) continue;
    const float* v = o.v;
    float qs0, qs1;
    fpvs(v[X_T], v[X_P], qs0, qs1);
    const float qm = vmax(v[X_Q], F(QMIN));
    if (!(is_dry(v) && (qm <= qs1 || v[X_T] >= F(T0C)) && qm < qs0)) {
      if (kLvPoints == 1) {
        own = true;
      } else {
        const bool precip = v[X_RR] > 0.f || v[X_RS] > 0.f || v[X_RG] > 0.f;
        list[precip ? atomicAdd(&nfront, 1) : kLvBlock * kLvPoints - 1 - atomicAdd(&nback, 1)] = e;
      }
      continue;
    }
    const size_t p = o.p;
    float cot[X_COUNT];
    const float rden = 1.0f / v[X_DEN];
    cot[X_RR] = yb[WF_MOIST][3 * n3 + p] * rden;
    cot[X_RS] = yb[WF_MOIST][5 * n3 + p] * rden;
    cot[X_RG] = yb[WF_MOIST][6 * n3 + p] * rden;
    cot[X_RI] = 0.f;
    if (vo[WF_T]) {
      theta_out(o, v[X_T]);
      vo[WF_MOIST][n3 + p] = v[X_Q];
      for (int m = 2; m < 7; ++m) vo[WF_MOIST][m * n3 + p] = 0.f;
    }
    b[WF_T][p] = yb[WF_T][p];
    b[WF_MOIST][n3 + p] = yb[WF_MOIST][n3 + p];
#pragma unroll
    for (int m = 2; m < 7; ++m) b[WF_MOIST][m * n3 + p] = 0.f;
    b[WF_H_DIABATIC][p] = 0.f;
    to_tape(o, cot);
  }
  if (kLvPoints > 1) __syncthreads();
  // the time-split loop's step (one loop: dt itself up to the split step)
  const float loops = fmaxf(dt / F(DTCLDCR), 1.0f);
  const float dtcld = dt <= F(DTCLDCR) ? dt : dt / loops;
  const int front = nfront, gap = (front + 31) / 32 * 32, all = kLvPoints > 1 ? gap + nback : (own ? kLvBlock : 0);
#pragma unroll 1
  for (int e = threadIdx.x; e < all; e += kLvBlock) {
    if (kLvPoints > 1 && e >= front && e < gap) continue;
    Point o;
    point(kLvPoints == 1 ? e : list[e < front ? e : kLvBlock * kLvPoints - 1 - (e - gap)], o);
    const float* v = o.v;
    const size_t p = o.p;
    float ym[7];
#pragma unroll
    for (int m = 1; m < 7; ++m) ym[m] = yb[WF_MOIST][m * n3 + p];
    const float yt = yb[WF_T][p], ympten = yt + yb[WF_H_DIABATIC][p] / dt;
    const float th = o.tin + (float)T0, rp = 1.0f / o.pii;
    float cot[X_COUNT];
#pragma unroll
    for (int q = 0; q < X_COUNT; ++q) cot[q] = 0.f;
    float tout = v[X_T];
    using D = Dual<N>;
    int seeds = 1 << X_T | 1 << X_Q | 1 << X_P;
    if (!(v[X_QC] < 0.f)) seeds |= 1 << X_QC;
    float qs0, qs1;
    fpvs(v[X_T], v[X_P], qs0, qs1);
    const float qm = vmax(v[X_Q], F(QMIN));
    if (!(is_dry(v) && (qm <= qs1 || v[X_T] >= F(T0C)))) seeds |= 1 << X_DEN;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (o.fall[q].id >= 0) seeds |= 1 << (X_RR + q);
#pragma unroll 1
    for (int pass = 0; seeds; ++pass) {
      int at[N];  // the inputs seeded in this pass
#pragma unroll
      for (int d = 0; d < N; ++d) {
        at[d] = seeds ? __ffs(seeds) - 1 : -1;
        seeds &= seeds - 1;
      }
      auto seed = [&](int q) {
        D x = dconst<N>(v[q]);
#pragma unroll
        for (int d = 0; d < N; ++d) x.d[d] = q == at[d] ? 1.f : 0.f;
        return x;
      };
      D t = seed(X_T), q = seed(X_Q), qc = vmax(seed(X_QC), 0.0f);
      const D pp = seed(X_P), den = seed(X_DEN);
      const D cpm = val(q) >= F(QMIN) ? F(CPV) * q + (1.0f - q) * F(CPD) : cst<D>(F(CPD * (1.0 - QMIN) + CPV * QMIN));
      const D xl = F(XLV0) - F(XLV1) * (t - F(T0C));
      const D denfac = vsqrt(1.0f / den * F(DEN0));
      D s0, s1;
      fpvs(t, pp, s0, s1);
      const D rh0 = vmax(q / s0, F(QMIN)), rh1 = vmax(q / s1, F(QMIN));
      D qr = vmax(seed(X_RR) / den, 0.0f), qs = vmax(seed(X_RS) / den, 0.0f), qg = vmax(seed(X_RG) / den, 0.0f);
      Slope3<D> sl0;
      melt_level(t, qr, qs, qg, den, pp, cpm, sl0, dtcld);
      D qi = vmax(seed(X_RI) / den, 0.0f);
      point_processes(t, q, qc, qi, qr, qs, qg, den, pp, denfac, cpm, xl, s0, s1, rh0, rh1, sl0, dtcld);
#pragma unroll
      for (int d = 0; d < N; ++d) {
        const float c = ympten * (t.d[d] * rp) + ym[1] * q.d[d] + ym[2] * qc.d[d] + ym[3] * qr.d[d] +
                        ym[4] * qi.d[d] + ym[5] * qs.d[d] + ym[6] * qg.d[d];
#pragma unroll
        for (int e = 0; e < X_COUNT; ++e)
          if (e == at[d]) cot[e] = c;
      }
      if (pass == 0) {
        tout = t.v;
        if (vo[WF_T]) {
          theta_out(o, tout);
          const float mv[7] = {0.f, q.v, qc.v, qr.v, qi.v, qs.v, qg.v};
          for (int m = 1; m < 7; ++m) vo[WF_MOIST][m * n3 + p] = mv[m];
        }
      }
    }
    // prep: the cotangents through the temperature th pii and the Exner
    // function
    const float cpii = fmaf(cot[X_T], th, -ympten * (tout * rp) * rp);
    b[WF_P][p] += cot[X_P] + cpii * (F(RCP) * o.pii / v[X_P]);
    b[WF_AL][p] -= cot[X_DEN] * (v[X_DEN] * v[X_DEN]);
    b[WF_T][p] = yt + fmaf(cot[X_T], o.pii, -ympten);
    b[WF_MOIST][n3 + p] = cot[X_Q];
    b[WF_MOIST][2 * n3 + p] = cot[X_QC];
#pragma unroll
    for (int m = 3; m < 7; ++m) b[WF_MOIST][m * n3 + p] = 0.f;
    b[WF_H_DIABATIC][p] = 0.f;
    to_tape(o, cot);
  }
}

// the reverse sweep of the sedimentation's tapes: the inputs' cotangents into
// the adjoints of the first entries
constexpr int kSweepBlock = 32, kSweepWindow = 16, kSweepRing = 64;
__global__ void __launch_bounds__(kSweepBlock) k_mp_fall_rev(Grid g, TapeCtx tc, int c0, int nc, const int* done,
                                                             const int* used, int ncol) {
  __shared__ float acc[kSweepRing * kSweepBlock];
  const int lane = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;
  if (lane >= nc) return;
  const int n = used[f * ncol + c0 + lane];
  if (n == 0 || !done[c0 + lane]) return;
  tape_sweep<kSweepWindow, kSweepRing, kSweepBlock>(fall_tape(tc, f), lane, fall_inputs(f) * (g.nz - 1), n, acc);
}

// and from there through prep, one level per thread
__global__ void __launch_bounds__(128) k_mp_fall_inputs(Grid g, S s, S b, Tv* ws, TapeCtx tc, int c0, int nc,
                                                        const int* done, const int* used, int ncol) {
  const int km = g.nz - 1;
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(x / nc), lane = (int)(x - (long long)k * nc);
  if (k > km) return;
  const int col = c0 + lane;
  ColPos cp;
  col_pos(g, col, cp);
  if (!cp.run || !done[col]) return;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3(), p = k * lev + cp.c2;
  float below = 0.f, at = 0.f, aden = 0.f, adz = 0.f;
  bool any = false;
#pragma unroll
  for (int f = 0; f < FALLS; ++f) {
    if (!used[f * ncol + col]) continue;
    any = true;
    const TapeCtx tf = fall_tape(tc, f);
    auto a = [&](int in, int kk) { return *tf.adj(in * km + kk, lane); };
    if (k > 0) below += a(I_DELZ, k - 1);
    if (k == km) continue;
    aden += a(I_DEN, k);
    adz += a(I_DELZ, k);
    b[WF_MOIST][(f == FALL_RAIN ? 3 : (f == FALL_SNOW ? 5 : 4)) * n3 + p] += a(I_Q, k);
    if (f == FALL_SNOW) {
      b[WF_MOIST][6 * n3 + p] += a(I_Q2, k);
      at += a(I_T, k);
    }
  }
  if (!any) return;
  b[WF_PH][p] += (below - adz) / (float)G;
  if (k == km) return;
  const Base B = base_of(ws, lane, tc.stride, km + 1);
  const float den = B(B_DEN, k);
  b[WF_T][p] += at * B(B_PII, k);
  b[WF_P][p] += at * (B(B_T, k) * F(RCP) / (s[WF_P][p] + s[WF_PB][p]));
  b[WF_AL][p] -= aden * (den * den);
}

// the reverse sweep of the tapes k_mp_tape left (same chunk and lanes):
// the inputs' cotangents from the adjoints of entries [0, n_inputs)
__global__ void __launch_bounds__(kSweepBlock) k_mp_tape_rev(Grid g, S b, TapeCtx tc, int c0, int nc,
                                                             const int* used) {
  __shared__ float acc[kSweepRing * kSweepBlock];
  const int lane = blockIdx.x * blockDim.x + threadIdx.x, col = c0 + lane;
  ColPos cp;
  if (lane >= nc || !col_pos(g, col, cp)) return;
  const int n = used[col];
  if (n == 0 || n > tc.cap) return;
  const int nin = mp_inputs(g);
  tape_sweep<kSweepWindow, kSweepRing, kSweepBlock>(tc, lane, nin, n, acc);
  for (int idx = 0; idx < nin; ++idx) put_input_cot(g, b, cp.c2, idx, __ldcg(tc.adj(idx, lane)));
}

// the passes of forward-mode tangents over the columns that the tape left
// undone (usually none: one launch finds that out): each pass seeds the inputs
// with indices [pass N, pass N + N) and forms their cotangents from the
// outputs' cotangents yb
template <int N>
__global__ void __launch_bounds__(64) k_mp_tangent(Grid g, S s, S yb, S b, float dt, Dual<N>* ws, int ncol,
                                                   const int* done) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  ColPos cp;
  if (col >= ncol || !col_pos(g, col, cp) || done[col] || !cp.run) return;
  const int nin = mp_inputs(g);
  const int km = g.nz - 1, c2 = cp.c2;
  const size_t lev = (size_t)g.ny * g.nx, n3 = g.n3();
  using T = Dual<N>;
  const Col<T> C{ws + col, ncol, km + 1};
  for (int j0 = 0; j0 < nin; j0 += N) {
    prep_column(g, s, C, c2, [&](int idx, float v) {
      T x = dconst<N>(v);
      const int d = idx - j0;
      if (d >= 0 && d < N) x.d[d] = 1.f;
      return x;
    });
    wsm6_column(C, km, dt, true);
    float acc[N];
#pragma unroll
    for (int n = 0; n < N; ++n) acc[n] = 0.f;
    for (int k = 0; k < km; ++k) {
      finish_level(C, k, dt);
      const size_t p = k * lev + c2;
      const T tnew = C(A_TIN, k), h = C(A_TH, k);
      const float yt = yb[WF_T][p], yh = yb[WF_H_DIABATIC][p];
#pragma unroll
      for (int n = 0; n < N; ++n) acc[n] += yt * tnew.d[n] + yh * h.d[n];
      for (int m = 1; m < 7; ++m) {
        const T qo = C(moist_slot(m), k);
        const float y = yb[WF_MOIST][m * n3 + p];
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n] += y * qo.d[n];
      }
    }
#pragma unroll
    for (int n = 0; n < N; ++n)
      if (j0 + n < nin) put_input_cot(g, b, c2, j0 + n, acc[n]);
  }
}

}  // namespace mpt

namespace {

constexpr int kMpDirections = 8;
// entries a column's tape may take per level by default (of the
// sedimentation with one time-split loop, of the whole column per loop with
// several), and the memory the tapes of one chunk of columns may take
constexpr int kTapeEntriesPerLevel = 480, kTapeSplitPerLevel = 256;
constexpr size_t kTapeChunkBytes = size_t(24) << 30;
// the capacity set through set_microphysics_tape_capacity (0: default)
int g_tape_capacity = 0;

// the adjoint's workspace, in floats: the outputs' cotangents (9 n3), the
// per-column done flags and the tapes' sizes, then one region shared by the
// chunk's tapes and column arrays and (afterwards) the tangent passes'
// column arrays
struct MpAdjWork {
  size_t done, used, region, tangent, rec, cols, total;
  int ncol, width, cap;
};

MpAdjWork mp_adj_work(const Grid& g) {
  MpAdjWork w;
  const int km = g.nz - 1;
  w.ncol = (g.ide - 1 - (g.ids + 1)) * (g.jde - 1 - (g.jds + 1));
  const int nloop = (int)fmaxf(g.dt / F(mp::DTCLDCR), 1.0f);
  const int per_level = nloop == 1 ? kTapeSplitPerLevel : kTapeEntriesPerLevel * nloop;
  w.cap = g_tape_capacity > 0 ? std::min(kTapeMaxEntries, g_tape_capacity)
                              : std::min(kTapeMaxEntries, per_level * km + mpt::mp_inputs(g));
  const int arrays = std::max<int>(mpt::A_COUNT, mpt::kFallSlots);
  const size_t per_col = (size_t)w.cap * 16 + (size_t)arrays * (km + 1) * sizeof(Tv);
  const size_t fit = std::max<size_t>(64, kTapeChunkBytes / per_col / 64 * 64);
  w.width = (int)std::min<size_t>(fit, ((size_t)w.ncol + 63) / 64 * 64);
  w.done = 9 * g.n3();
  w.used = w.done + w.ncol;
  w.region = (w.used + (size_t)mpt::FALLS * w.ncol + 3) / 4 * 4;
  w.tangent = (size_t)mpt::A_COUNT * g.nz * w.ncol * (kMpDirections + 1);
  const size_t ent = (size_t)w.cap * w.width;
  w.rec = w.region;
  w.cols = w.rec + 4 * ent;
  const size_t tape = 4 * ent + sizeof(Tv) / sizeof(float) * (size_t)arrays * (km + 1) * w.width;
  w.total = w.region + std::max(w.tangent, tape);
  return w;
}

}  // namespace

size_t microphysics_adj_work_floats(const Grid& g) { return mp_adj_work(g).total; }

int set_microphysics_tape_capacity(int entries) {
  const int prev = g_tape_capacity;
  g_tape_capacity = entries;
  return prev;
}

int launch_physics_adj(const Grid& g, const S& s, const S& post, const S& b, float* work, float dt, cudaStream_t st,
                       const S* values) {
  const size_t n3 = g.n3();
  const MpAdjWork w = mp_adj_work(g);
  int n = launch_eos_adj(g, post, b, st);
  // the outputs' cotangents, kept while the kernels write the inputs'
  S yb{};
  yb.f[WF_T] = work;
  yb.f[WF_MOIST] = work + n3;
  yb.f[WF_H_DIABATIC] = work + 8 * n3;
  cudaMemcpyAsync(yb.f[WF_T], b[WF_T], n3 * sizeof(float), cudaMemcpyDeviceToDevice, st);
  cudaMemcpyAsync(yb.f[WF_MOIST], b[WF_MOIST], 7 * n3 * sizeof(float), cudaMemcpyDeviceToDevice, st);
  cudaMemcpyAsync(yb.f[WF_H_DIABATIC], b[WF_H_DIABATIC], n3 * sizeof(float), cudaMemcpyDeviceToDevice, st);
  int* done = reinterpret_cast<int*>(work + w.done);
  int* used = reinterpret_cast<int*>(work + w.used);
  S vo{};
  if (values) vo = *values;
  TapeCtx tc;
  tc.rec = reinterpret_cast<TapeRec*>(work + w.rec);
  tc.stride = w.width;
  tc.cap = w.cap;
  auto* cols = reinterpret_cast<Tv*>(work + w.cols);
  const bool split = (int)fmaxf(dt / F(mp::DTCLDCR), 1.0f) == 1;
  for (int c0 = 0; c0 < w.ncol; c0 += w.width) {
    const int nc = std::min(w.width, w.ncol - c0);
    const unsigned columns = (nc + kTapeBlock - 1) / kTapeBlock, sweeps = (nc + mpt::kSweepBlock - 1) / mpt::kSweepBlock;
    if (split) {
      const unsigned levels = (unsigned)(((long long)nc * (g.nz - 1) + 127) / 128);
      const dim3 falls(columns, mpt::FALLS), fsweeps(sweeps, mpt::FALLS);
      const unsigned ends = (unsigned)(((long long)nc * g.nz + 127) / 128);
      if (c0 == 0) cudaMemsetAsync(used, 0, mpt::FALLS * w.ncol * sizeof(int), st);
      mpt::k_mp_levels<<<levels, 128, 0, st>>>(g, s, yb, b, cols, tc, c0, nc, vo, done, used, w.ncol);
      mpt::k_mp_fall<<<falls, kTapeBlock, 0, st>>>(g, s, dt, cols, tc, c0, nc, done, used, w.ncol);
      // sorting pays where it leaves enough blocks to even out (two per SM at
      // a time); elsewhere a thread runs its own point: 2.5 ms sorted, 3.4 not,
      // at 240x240x41 (4062 blocks of sorted points); 0.53 and 0.38 at 101x101x35
      // (527)
      const bool deep = levels >= 4 * 148 * 2 * 8;
      const unsigned sorted = deep ? (levels + 3) / 4 : levels;
      (deep ? mpt::k_mp_levels_adj<3, 4> : mpt::k_mp_levels_adj<3, 1>)<<<sorted, mpt::kLvBlock, 0, st>>>(g, s, yb, b, cols, tc, c0, nc, vo, done, used, w.ncol, dt);
      mpt::k_mp_fall_rev<<<fsweeps, mpt::kSweepBlock, 0, st>>>(g, tc, c0, nc, done, used, w.ncol);
      mpt::k_mp_fall_inputs<<<ends, 128, 0, st>>>(g, s, b, cols, tc, c0, nc, done, used, w.ncol);
      n += 5;
      continue;
    }
    mpt::k_mp_tape<<<columns, kTapeBlock, 0, st>>>(g, s, yb, b, dt, cols, tc, c0, nc, vo, done, used);
    mpt::k_mp_tape_rev<<<sweeps, mpt::kSweepBlock, 0, st>>>(g, b, tc, c0, nc, used);
    n += 2;
  }
  // the columns whose tape outgrew the capacity, by tangent passes
  auto* ws = reinterpret_cast<Dual<kMpDirections>*>(work + w.region);
  mpt::k_mp_tangent<kMpDirections><<<(w.ncol + 63) / 64, 64, 0, st>>>(g, s, yb, b, dt, ws, w.ncol, done);
  return n + 1;
}

}  // namespace wrf
