// salsa_kernel_impl.cuh -- the fused SALSA microphysics step for sm_103a (templates;
// instantiated by salsa_k_*.cu and salsa_l_*.cu, one translation unit per form).
//
// One launch advances every interior grid cell by one SALSA call
// (UCLALES-SALSA src/src_salsa/mo_salsa_driver.f90:180-427 -> mo_salsa.f90:45-153).
//
// Execution model: two forms of the same templates (LS lanes advance one cell)
//   * warp form (LS = 32, salsa_step_kernel): block = SALSA_CPG warps = SALSA_CPG interior
//     cells ("group"); the block stages the group's bin-major input rows into shared memory
//     with sector-complete loads, every warp advances its own cell out of shared memory,
//     lanes split bins (diameters, condensation, activation, freezing) and bin pairs
//     (collision kernels), and the block writes the tendency rows back.  The Gauss-Seidel
//     bin sweep of the coagulation update stays ordered; each target bin's partner sums are
//     lane-parallel and reduced with warp shuffles.
//   * lane form (LS = 1, salsa_lane_kernel): every lane advances a cell of its own out of a
//     workspace in global memory, for calls with enough cells to fill the lanes.  The FP64
//     pipe, which bounds both forms, takes as long for one lane as for 32.
//   * KT is the arithmetic type of the collision kernels and of the condensation
//     mass-transfer coefficients: double for the parity form, float for the mixed
//     form (whose partner sums are compensated float sums; denominators, the water
//     budget and all state updates stay double).
//   * a pre-pass orders the cells so that the cells of one block or warp share a class
//     (dry clear, moist clear or cloudy); they are then not always neighbours.
#pragma once
#include "salsa_device.cuh"
#include "salsa_math.cuh"
#include <cstdio>
#include <type_traits>

namespace salsa {
namespace {   // internal linkage: every instantiation unit carries its own copy

// ----------------------------------------------------------------------------------------
// per-warp workspace
// ----------------------------------------------------------------------------------------
// LS lanes advance one cell:
//   LS = 32 (warp form)  one warp per cell, the workspace in shared memory, rows contiguous;
//   LS = 1  (lane form)  one lane per cell, the workspaces of a warp's 32 cells interleaved in
//                        global memory: row r of lane l at r * 32 + l, so that a warp's access
//                        to a row is one 256-byte (128 for float) segment.
template <typename T>
struct Col {
  T *p;
  __device__ __forceinline__ T &operator[](int i) const { return p[i * 32]; }
  __device__ __forceinline__ Col operator+(int k) const { return {p + k * 32}; }
  template <typename U> __device__ __forceinline__ operator Col<U>() const { return {p}; }   // T -> const T
};
template <typename T, int LS> using Ptr = typename std::conditional<LS == 1, Col<T>, T *>::type;
// the same memory as rows of another type
template <typename U, typename T> __device__ __forceinline__ U *row_cast(T *p) { return reinterpret_cast<U *>(p); }
template <typename U, typename T> __device__ __forceinline__ Col<U> row_cast(Col<T> c) {
  const int l = threadIdx.x & 31;
  return {reinterpret_cast<U *>(c.p - l) + l};
}

template <typename KT, int LS>
struct WS {
  using D = Ptr<double, LS>;
  D raw, numc, volc, dwet, ddry, dins, dnsp, rhomean, indef, ctime, scr, misc;
  Ptr<KT, LS> K;
  int *pbuf;   // warp form
  int NB;
  bool live;   // lane form, last warp: lanes past the last cell repeat it and write nothing
  long long off;   // lane form: the cell's offset inside a field plane
  // lane form: bins that reach their number limit in some cell of the warp before coagulation
  // (bins 0-63, 64-95); pairs with the others have K = 0 and their terms are skipped
  unsigned long long am0;
  unsigned am1;
  __device__ __forceinline__ bool on(int b) const {
    if constexpr (LS == 1) return b < 64 ? (am0 >> b) & 1ull : (am1 >> (b - 64)) & 1u;
    else return true;
  }
  // float copies of numc and volc that the mixed form's coagulation update sums from
  // (in the scratch rows, valid from shadow_all to the end of the update)
  Ptr<float, LS> nf, vf;
  Ptr<float, LS> lf;   // lane form of the mixed form: the leaves of the partner sums
  __device__ __forceinline__ double &v(int s, int b) const { return volc[s * NB + b]; }
  __device__ __forceinline__ D sc(int k) const { return scr + k * NB; }
  // partner values in the kernel type: the state itself (FP64 form) or its float copy
  __device__ __forceinline__ KT nk(int b) const {
    if constexpr (sizeof(KT) == 4) return nf[b];
    else return numc[b];
  }
  __device__ __forceinline__ KT vk(int s, int b) const {
    if constexpr (sizeof(KT) == 4) return vf[s * NB + b];
    else return volc[s * NB + b];
  }
};

// reductions and barriers of the lanes of one cell
template <int LS> __device__ __forceinline__ double wsum(double v) { return LS == 1 ? v : warp_sum(v); }
template <int LS> __device__ __forceinline__ bool wany(bool b) { return LS == 1 ? b : (bool)warp_any(b); }
template <int LS> __device__ __forceinline__ void wsync() { if constexpr (LS != 1) __syncwarp(); }

// misc slots (doubles)
enum {
  M_DIAG = 0,              // 17 diagnostic accumulators
  M_FLAGS = 17,            // F_* per-cell condition counters
  M_RV = 24,               // water vapour mixing ratio of the cell
  M_PF = 32,               // precipitation-formation accumulators (7 + 9 * nprc, nprc <= 23)
  M_PFSLOT = M_PF + 216,   // 8 partner slots * 10
  M_GAS = M_PFSLOT + 80,   // the cell's five gases [#/m3] (gas condensation only)
  M_END = M_GAS + 8
};
enum { F_NEG = 0, F_EQUIL, F_DISTR, F_NEGFRAC, F_COND };
#define SALSA_MISC_DOUBLES 336
#define SALSA_NSCR 13

__device__ __forceinline__ int phase_of(const DevParams &P, int b) {
  return b < P.nbins ? 1 : (b < P.nbins + P.ncld ? 2 : (b < P.nliquid ? 3 : 4));
}
__device__ __forceinline__ double nlim_of(int ph) { return ph <= 2 ? K_NLIM : K_PRLIM; }
__device__ __forceinline__ double dlim_of(int ph) {
  return ph == 1 ? 30.e-6 : (ph == 2 ? 100.e-6 : (ph == 3 ? 5.e-3 : 10.e-3));
}
// Comparisons of a number with a positive constant, and minima and maxima of non-negative
// ones, on the bit patterns: an FP64 comparison occupies the FP64 pipe as long as a sum
// does.  The results equal the FP64 ones over the stated ranges, infinities and the positive
// quiet NaN of the GPU's arithmetic included (-0 counts as 0).
#define FM_INF 0x7ff0000000000000ll
__device__ __forceinline__ bool num_ge(double x, double c) {
  const long long b = __double_as_longlong(x);
  return b >= __double_as_longlong(c) && b <= FM_INF;
}
__device__ __forceinline__ bool num_gt(double x, double c) {
  const long long b = __double_as_longlong(x);
  return b > __double_as_longlong(c) && b <= FM_INF;
}
__device__ __forceinline__ bool num_lt(double x, double c) { return __double_as_longlong(x) < __double_as_longlong(c); }
__device__ __forceinline__ double min_pos(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b) ? a : b; }
// fmax(0., x)
__device__ __forceinline__ double pos_part(double x) {
  return (unsigned long long)__double_as_longlong(x) > (unsigned long long)FM_INF ? 0. : x;
}
// fmax(c, x) of x >= 0 (or NaN: c)
__device__ __forceinline__ double max_pos(double c, double x) { return num_gt(x, c) ? x : c; }
// fmin(fmax(x, -t), t) of t >= 0 (NaN x: -t)
__device__ __forceinline__ double limit_pos(double x, double t) {
  const long long b = __double_as_longlong(x), m = b & 0x7fffffffffffffffll, bt = __double_as_longlong(t);
  const long long sign = m > FM_INF ? (long long)0x8000000000000000ull : b ^ m;
  return m > bt ? __longlong_as_double(bt | sign) : x;
}
__device__ __forceinline__ int tri(int i, int j, int NB) {  // i <= j
  return i * NB - (i * (i - 1)) / 2 + (j - i);
}
template <typename KT, int LS>
__device__ __forceinline__ KT kget(const WS<KT, LS> &w, int i, int j) {
  if (!(w.on(i) && w.on(j))) return (KT)0;
  return i <= j ? w.K[tri(i, j, w.NB)] : w.K[tri(j, i, w.NB)];
}

// ----------------------------------------------------------------------------------------
// classSection.f90:91-159 updateDiameter(limit=.TRUE., type="all") and :169-195 updateRhomean.
// With limit set, dnsp = MIN(dwet, dlim) overwrites the non-spherical diameter (:149-150),
// so getDiameter's value never survives a type="all" update and is not evaluated here.
// ----------------------------------------------------------------------------------------
// CUDA_ROOT: the wet diameter by CUDA's cbrt (see the condensation coefficients).
template <bool CUDA_ROOT = false, typename KT, int LS>
__device__ __forceinline__ void updateDiameterAll(const DevParams &P, const WS<KT, LS> &w, const double *dmid, int b) {
  int ph = phase_of(P, b);
  double n = w.numc[b];
  double dw, dd, di;
  if (num_gt(n, nlim_of(ph))) {
    double vs = 0., vd = 0., vi = 0.;
    for (int s = 0; s < P.nused; s++) vs += w.v(s, b);
    for (int s = 0; s < P.ndry; s++) vd += w.v(s, b);
    for (int k = 0; k < P.ninsoluble; k++) vi += w.v(P.ind_insoluble[k], b);
    // (v / numc / pi6)^(1/3) with one division for the three diameters
    const double q = drcp(n * K_PI6);
    dw = CUDA_ROOT ? ::cbrt(vs * q) : dcbrt(vs * q);
    dd = dcbrt(vd * q);
    di = dcbrt(vi * q);
  } else {
    dw = dd = di = dmid[b];
  }
  double dl = dlim_of(ph);
  dw = min_pos(dw, dl);
  w.dwet[b] = dw;
  w.dnsp[b] = dw;
  w.ddry[b] = min_pos(dd, dl);
  w.dins[b] = min_pos(di, dl);
}

__device__ __forceinline__ double rhomean_of(const DevParams &P, int ph, double n, double vw, double vr) {
  if (ph > 3) {
    if (num_gt(n, nlim_of(ph))) {
      double mp = K_RHOIC * vw, mr = K_RHORI * vr, mt = mp + mr;
      double r = ddiv(mp * K_RHOIC + mr * K_RHORI, max_pos(7.e-25, mt));
      return fmin(r, K_RHOIC);
    }
    return K_RHOIC;
  }
  return K_RHOWA;
}

// classSection.f90:202-224 getRimeFraction
__device__ __forceinline__ double rimefrac(const DevParams &P, double n, double vw, double vr, int ph) {
  double r = 0.;
  if (ph == 4 && num_gt(vw, 1.e-23) && num_gt(vr, 1.e-23) && num_gt(n, nlim_of(ph))) r = ddiv(vr * K_RHORI, vw * K_RHOIC + vr * K_RHORI);
  return r;
}

// ----------------------------------------------------------------------------------------
// Terminal velocity: mo_particle_external_properties.f90:237-352 (+ ice shape
// coefficients, mo_ice_shape.f90:145-191)
// ----------------------------------------------------------------------------------------
template <typename T>
struct Shape { T alpha, beta, gamma, sigma; };

// float selects the cancellation-free single-precision forms; every other arithmetic
// type (double, and the dual numbers of the gradient kernels) takes the FP64 forms
template <typename T> struct is_f32 { static constexpr bool value = false; };
template <> struct is_f32<float> { static constexpr bool value = true; };

template <typename T>
__device__ __forceinline__ T t_exp(T x);
template <> __device__ __forceinline__ double t_exp<double>(double x) { return dexp(x); }
template <> __device__ __forceinline__ float t_exp<float>(float x) { return expf(x); }
template <typename T>
__device__ __forceinline__ T t_log(T x);
template <> __device__ __forceinline__ double t_log<double>(double x) { return dlog(x); }
template <> __device__ __forceinline__ float t_log<float>(float x) { return logf(x); }
template <typename T>
__device__ __forceinline__ T t_sqrt(T x);
template <> __device__ __forceinline__ double t_sqrt<double>(double x) { return dsqrt(x); }
template <> __device__ __forceinline__ float t_sqrt<float>(float x) { return sqrtf(x); }
template <typename T>
__device__ __forceinline__ T t_cbrt(T x);
template <> __device__ __forceinline__ double t_cbrt<double>(double x) { return dcbrt(x); }
template <> __device__ __forceinline__ float t_cbrt<float>(float x) { return cbrtf(x); }
template <typename T>
__device__ __forceinline__ T t_pow(T x, T y);
template <> __device__ __forceinline__ double t_pow<double>(double x, double y) { return dpow(x, y); }
template <> __device__ __forceinline__ float t_pow<float>(float x, float y) { return powf(x, y); }

template <typename T>
__device__ void shape_coeffs(const DevParams &P, Shape<T> &s, double mpri, double mrim, double numc) {
  s.alpha = (T)(K_PI6 * K_RHOIC);
  s.beta = (T)3.;
  s.gamma = (T)(K_PI / 4.);
  s.sigma = (T)2.;
  if (numc < 1.e-6) return;
  double Mtot = ddiv(mpri + mrim, numc);
  double Fr = fmax(fmin(ddiv(mrim, Mtot * numc), 0.9999), 0.0001);
  double rho_b = Fr * K_RHORI + (1. - Fr) * K_RHOIC;
  double Dth = dpow(ddiv(K_PI6 * K_RHOIC, P.iceShapeAlpha), drcp(P.iceShapeBeta - 3.));
  double Dgr = dpow(ddiv(P.iceShapeAlpha, K_PI6 * rho_b), drcp(3. - P.iceShapeBeta));
  double Dcr = dpow(ddiv((drcp(1. - Fr)) * P.iceShapeAlpha, K_PI6 * rho_b), drcp(3. - P.iceShapeBeta));
  double Mth = K_RHOIC * K_PI6 * cube(Dth), Mgr = rho_b * K_PI6 * cube(Dgr), Mcr = rho_b * K_PI6 * cube(Dcr);
  if (Mtot >= Mth && Mtot < Mgr) {
    s.alpha = (T)P.iceShapeAlpha; s.beta = (T)P.iceShapeBeta; s.gamma = (T)P.iceShapeGamma; s.sigma = (T)P.iceShapeSigma;
  } else if (Mtot > Mcr) {
    double hlp = drcp(1. - Fr);
    s.alpha = (T)(P.iceShapeAlpha * hlp);
    s.beta = (T)P.iceShapeBeta;
    s.gamma = (T)(P.iceShapeGamma * (1. - Fr) + K_PI / 4. * Fr);
    s.sigma = (T)(P.iceShapeSigma * (1. - Fr) + 2. * Fr);
  }
}

template <typename T>
__device__ T terminal_vel(T diam, T rhop, T rhoa, T visc, T beta, int flag, const Shape<T> &sh, T dnsp) {
  const T grav = (T)K_GRAV;
  T tv = 0;
  if (flag <= 3) {
    if (diam <= (T)19E-6) {
      tv = ddiv(sq(diam) * (rhop - rhoa) * grav * beta, (T)18. * visc);
    } else if (diam < (T)1.07E-3) {
      T NDa = ddiv((T)4. / (T)3. * cube(diam) * grav * (rhop - rhoa) * rhoa, sq(visc));
      T X = t_log(NDa);
      T X2 = sq(X);
      T Y = (T)-0.318657E1 + (T)0.992696 * X - (T)0.153193E-2 * X2 - (T)0.987059E-3 * X2 * X -
            (T)0.578878E-3 * sq(X2) + (T)0.855176E-4 * sq(X2) * X - (T)0.327815E-5 * cube(X2);
      T Re2 = beta * t_exp(Y);
      tv = ddiv(ddiv(visc, rhoa), diam) * Re2;
    } else {
      T Np = ddiv(cube((T)K_SURFW0) * sq(rhoa), sq(sq(visc)) * (rhop - rhoa) * grav);
      T Bo = divc((T)4. / (T)3. * (rhop - rhoa) * grav, (T)K_SURFW0) * sq(diam);
      T Np6 = t_sqrt(t_cbrt(Np));
      T X3 = t_log(Bo * Np6);
      T X32 = sq(X3);
      T Y3 = (T)-0.500015E1 + (T)0.523778E1 * X3 - (T)0.204914E1 * X32 + (T)0.475294 * X32 * X3 -
             (T)0.542819E-1 * sq(X32) + (T)0.238449E-2 * sq(X32) * X3;
      T Re3 = Np6 * t_exp(Y3);
      tv = fmin(ddiv(ddiv(visc, rhoa), diam) * Re3, (T)9.2);
    }
  } else {
    // Khvorostyanov and Curry 2002 (kc1213/kcbre/kcare/kcAv/kcBv/kcVt :297-352)
    T Vb = (T)K_PI6 * cube(diam);
    T Ap = sh.gamma * t_pow(dnsp, sh.sigma);
    T X = ddiv((T)2. * Vb * (rhop - rhoa) * grav * sq(dnsp), Ap * rhoa * sq(visc));
    const T c1 = (T)0.0902, delta0 = (T)9.06;
    T k12, km1, bre;
    if (!is_f32<T>::value) {
      k12 = t_sqrt((T)1. + c1 * t_sqrt(X));
      km1 = k12 - (T)1.;
      bre = (T)0.5 * c1 * t_sqrt(X);
      bre = ddiv(bre, km1);
      bre = ddiv(bre, k12);
    } else {
      // float: sqrt(1+y)-1 = y/(sqrt(1+y)+1) and b_Re = (1 + 1/k12)/2, free of cancellation
      T y = c1 * t_sqrt(X);
      k12 = t_sqrt((T)1. + y);
      km1 = ddiv(y, k12 + (T)1.);
      bre = (T)0.5 * ((T)1. + ddiv((T)1., k12));
    }
    T are = (T)0.25 * sq(delta0);
    are = are * sq(km1);
    are = ddiv(are, t_pow(X, bre));
    T Av = are * t_pow(visc, (T)1. - (T)2. * bre);
    Av = Av * t_pow(ddiv((T)2. * sh.alpha * grav, rhoa * sh.gamma), bre);
    T Bv = bre * (sh.beta - sh.sigma + (T)2.) - (T)1.;
    tv = Av * t_pow(dnsp, Bv);
  }
  return tv;
}

// per-cell constants of the collision kernel (mo_salsa_coagulation_kernels.f90:282-284, 343-345, 389-391)
template <typename T>
struct CoagCell { T T_, visc, mfp, zrhoa, vkin, shearA, turbB; };

// Per-bin collision properties (the particle-dependent part of coagc :263-364), in the
// form the pair evaluation uses: the squared mean thermal velocity, and the per-bin
// factors of the convective Brownian term and of the collision efficiency, so that a pair
// takes no cube root and one division less.  Nine values (the gradient harness stores
// and differentiates them as a row each).
template <typename T>
struct BinProps { T diam, fre, cschm, dfpart, mtvel2, omega, termv, reyn, ire; };
// fre = Re^(1/3) for Re <= 1, else Re^(1/2) (:350-355); cschm = Sc^(1/3); ire = 1/(60 + Re)

template <typename T>
__device__ void bin_props(const CoagCell<T> &cc, int ph, T diam, T dsph, T mass, T rhomean, const Shape<T> &sh,
                          BinProps<T> &o) {
  o.diam = diam;
  T knud = ddiv((T)2. * cc.mfp, diam);
  const T beta = (T)1. + knud * ((T)1.142 + (T)0.558 * t_exp(ddiv((T)-0.999, knud)));
  o.dfpart = ddiv(beta * (T)K_BOLTZ * cc.T_, (T)3. * (T)K_PI * cc.visc * diam);
  const T mtvel = t_sqrt(ddiv((T)8. * (T)K_BOLTZ * cc.T_, (T)K_PI * mass));
  o.mtvel2 = sq(mtvel);
  o.omega = ddiv((T)8. * o.dfpart, (T)K_PI * mtvel);
  if constexpr (is_f32<T>::value) {
    // the fall speed stays FP64 in the mixed form: collision kernels of pairs with close
    // fall speeds take their difference, which would magnify float rounding of the Beard
    // exponent (exp of up to ~10) into the kernel
    Shape<double> shd;
    shd.alpha = sh.alpha; shd.beta = sh.beta; shd.gamma = sh.gamma; shd.sigma = sh.sigma;
    const double vd = ph < 4 ? terminal_vel<double>(diam, rhomean, cc.zrhoa, cc.visc, beta, ph, shd, 0.)
                             : terminal_vel<double>(dsph, rhomean, cc.zrhoa, cc.visc, beta, ph, shd, diam);
    o.termv = (T)vd;
  } else {
    if (ph < 4) o.termv = terminal_vel<T>(diam, rhomean, cc.zrhoa, cc.visc, beta, ph, sh, (T)0);
    else o.termv = terminal_vel<T>(dsph, rhomean, cc.zrhoa, cc.visc, beta, ph, sh, diam);
  }
  o.reyn = ddiv(diam * o.termv, cc.vkin);
  const T schm = ddiv(cc.vkin, o.dfpart);
  o.fre = o.reyn <= (T)1. ? t_cbrt(o.reyn) : t_sqrt(o.reyn);
  o.cschm = t_cbrt(schm);
  o.ire = ddiv((T)1., (T)60. + o.reyn);
}

// ((m+w)^3 - (m^2+w^2)^(3/2)) / (3 m w) - m without cancellation (float form of :305-313):
// with u = min(m,w)/max(m,w) and E = (1+u^2)^(3/2) - 1 = expm1(1.5 log1p(u^2)),
// w <= m: m (u + u^2/3 - E/(3u));  w > m: w (1 + u^2/3 - E/(3u)).
__device__ __forceinline__ float flux_match_stable(float m, float w) {
  bool small = w <= m;
  float u = small ? w / m : m / w;
  float u2 = u * u;
  float E = expm1f(1.5f * log1pf(u2));
  float core = u2 * (1.f / 3.f) - E / (3.f * u);
  return small ? m * (u + core) : w * (1.f + core);
}
__device__ __forceinline__ double flux_match_stable(double m, double w) { return 0.; }

// pair part of coagc (:298-416)
template <typename T>
__device__ T coag_pair(const CoagCell<T> &cc, const BinProps<T> &a, const BinProps<T> &b) {
  T mdiam = (T)0.5 * (a.diam + b.diam);
  T flux1 = (T)4. * (T)K_PI * mdiam * (a.dfpart + b.dfpart);
  T flux2 = (T)K_PI * t_sqrt(a.mtvel2 + b.mtvel2) * sq(mdiam);
  T tva1, tva2;
  if (!is_f32<T>::value) {
    T m2 = sq(mdiam);
    T oa2 = m2 + sq(a.omega), ob2 = m2 + sq(b.omega);
    tva1 = ddiv(cube(mdiam + a.omega) - oa2 * t_sqrt(oa2), (T)3. * mdiam * a.omega) - mdiam;
    tva2 = ddiv(cube(mdiam + b.omega) - ob2 * t_sqrt(ob2), (T)3. * mdiam * b.omega) - mdiam;
  } else {
    tva1 = flux_match_stable(mdiam, a.omega);
    tva2 = flux_match_stable(mdiam, b.omega);
  }
  T fmdist = t_sqrt(sq(tva1) + sq(tva2));
  bool first_large = a.diam >= b.diam;
  const BinProps<T> &L = first_large ? a : b;
  const BinProps<T> &S = first_large ? b : a;
  T dv = fabs(a.termv - b.termv);
  T stok = ddiv((T)2. * S.termv * dv, L.diam * (T)K_GRAV);
  // flux1 / (mdiam/(mdiam+fmdist) + flux1/flux2) as one quotient in FP64; the float form
  // keeps the reference's shape (the products would leave float's range)
  T zbrown;
  if (!is_f32<T>::value) {
    const T mf = mdiam + fmdist;
    zbrown = ddiv(flux1 * flux2 * mf, mdiam * flux2 + flux1 * mf);
  } else {
    zbrown = ddiv(flux1, ddiv(mdiam, mdiam + fmdist) + ddiv(flux1, flux2));
  }
  // Re <= 1: (Re Sc)^(1/3), else Re^(1/2) Sc^(1/3), from the per-bin factors
  const T zbrconv = (T)0.45 * zbrown * L.fre * S.cschm;
  T hd = (T)0.5 * (a.diam + b.diam);
  T ztshear = cc.shearA * cube(hd);
  T zturb = cc.turbB * sq(hd) * dv;
  T zea = ddiv(sq(stok), sq(stok + (T)0.5));
  T zev = 0;
  if (stok > (T)1.214) {
    zev = ddiv((T)0.75 * t_log((T)2. * stok), stok - (T)1.214);
    zev = ddiv((T)1., sq((T)1. + zev));
  }
  T zecoll = ((T)60. * zev + zea * L.reyn) * L.ire;
  T zgrav = zecoll * (T)K_PI * sq(mdiam);
  zgrav = zgrav * dv;
  return zbrown + zbrconv + t_sqrt(sq(zgrav) + sq(ztshear) + sq(zturb));
}

// ---- the FP64 step's form of the pair kernel ----
// The same kernel as coag_pair in fewer FP64 operations (64 instead of 92 a pair, 48 instead
// of 75 a bin): what depends on one particle is taken once per bin, per-cell factors once per
// cell, and common factors leave the sums.  With m the mean diameter, w the mean free path of
// a particle (omega), D4 four times its diffusion coefficient, v2 its squared thermal speed:
//   flux matching   ((m+w)^3 - (m^2+w^2)^(3/2)) / (3 m w) - m, by the reciprocals of m and 3 w
//                     (the differences as coag_pair rounds them: they cancel to 1e-14 for a
//                     drop and an Aitken particle, and condensation magnifies that)
//   Brownian        pi X Y / (X + Y),  X = m^2 sqrt(v2_a + v2_b),  Y = (D4_a + D4_b) (m + f)
//   gravity, shear, turbulence  m^2 sqrt((pi E dv)^2 + (A m)^2 + (B dv)^2)
// On grid384x384x160 the collision kernels were 42 % of the lane form's time.
struct PairProps {
  double h, D4, v2, om, i3om, tv;   // half diameter, D4, v2, omega, 1/(3 omega), fall speed
  double fre, cs, rre, G;   // Re^(1/3 or 1/2); 0.45 pi Sc^(1/3); pi Re/(60 + Re); 2/(d g)
};
// per-cell factors
struct PairCell {
  CoagCell<double> c;
  double mfp2, kx, kD4, kv2, k18, ivkin, vkin4;   // 2 mfp, 0.999/(2 mfp), 4kT/(3 pi mu), 8kT/pi, g/(18 mu), 1/nu, 4 nu
};

__device__ __forceinline__ bool bits_ge(double a, double b) {   // a >= b of non-negative numbers
  return __double_as_longlong(a) >= __double_as_longlong(b);
}

// rd = 1/diam, im = 1/mass
__device__ __forceinline__ void pair_props(const PairCell &k, int ph, double diam, double rd, double im, double dsph,
                                           double rho, const Shape<double> &sh, PairProps &o) {
  const double beta = fma(k.mfp2 * rd, fma(0.558, dexp(-(k.kx * diam)), 1.142), 1.);
  o.h = 0.5 * diam;
  o.D4 = beta * rd * k.kD4;
  o.v2 = k.kv2 * im;
  const double v = dsqrt(o.v2);
  o.om = ddiv((2. / K_PI) * o.D4, v);
  o.i3om = drcp(3. * o.om);
  if (ph < 4 && bits_ge(19E-6, diam)) o.tv = diam * diam * (rho - k.c.zrhoa) * beta * k.k18;
  else if (ph < 4) o.tv = terminal_vel<double>(diam, rho, k.c.zrhoa, k.c.visc, beta, ph, sh, 0.);
  else o.tv = terminal_vel<double>(dsph, rho, k.c.zrhoa, k.c.visc, beta, ph, sh, diam);
  const double re = diam * o.tv * k.ivkin;
  o.fre = re <= 1. ? dcbrt(re) : dsqrt(re);
  o.cs = (0.45 * K_PI) * dcbrt(ddiv(k.vkin4, o.D4));
  o.rre = ddiv(K_PI * re, 60. + re);
  o.G = (2. / K_GRAV) * rd;
}

__device__ __forceinline__ double pair_kernel(const PairCell &k, const PairProps &a, const PairProps &b) {
  const double m = a.h + b.h, m2 = m * m, im = drcp(m);
  const double oa = fma(a.om, a.om, m2), ob = fma(b.om, b.om, m2), sa = m + a.om, sb = m + b.om;
  const double ta = fma(fma(sa * sa, sa, -(oa * dsqrt(oa))) * im, a.i3om, -m);
  const double tb = fma(fma(sb * sb, sb, -(ob * dsqrt(ob))) * im, b.i3om, -m);
  const double X = m2 * dsqrt(a.v2 + b.v2), Y = (a.D4 + b.D4) * (m + dsqrt(fma(tb, tb, ta * ta)));
  const double zb = ddiv(X * Y, X + Y);
  const bool al = bits_ge(a.h, b.h);
  const double Lrre = al ? a.rre : b.rre;
  const double dv = fabs(a.tv - b.tv);
  const double stok = (al ? b.tv : a.tv) * dv * (al ? a.G : b.G);
  const double q = ddiv(stok, stok + 0.5);
  double e = q * q * Lrre;   // pi times the collision efficiency
  if (stok > 1.214) {
    double z = ddiv(0.75 * dlog(2. * stok), stok - 1.214);
    z = drcp(sq(1. + z));
    e = fma(z, K_PI - Lrre, e);   // 60/(60 + Re) = 1 - Re/(60 + Re)
  }
  const double g = e * dv, t1 = k.c.shearA * m, t2 = k.c.turbB * dv;
  return fma(zb, fma(al ? a.fre : b.fre, al ? b.cs : a.cs, K_PI), m2 * dsqrt(fma(g, g, fma(t1, t1, t2 * t2))));
}

// What the two kernel types use: properties of a bin, rows that hold them, cell constants
template <typename KT> struct KForm;
template <> struct KForm<float> {
  typedef BinProps<float> Props;
  struct Cell { CoagCell<double> cd; CoagCell<float> cc; };
  static constexpr int NROW = 9;
};
template <> struct KForm<double> {
  typedef PairProps Props;
  typedef PairCell Cell;
  static constexpr int NROW = 10;
};
template <typename KT> using KProps = typename KForm<KT>::Props;
template <typename KT> using KCell = typename KForm<KT>::Cell;

template <typename KT, typename PT>
__device__ __forceinline__ void load_props(const PT &S, int NB, int b, KProps<KT> &o) {
  KT *po = reinterpret_cast<KT *>(&o);
#pragma unroll
  for (int k = 0; k < KForm<KT>::NROW; k++) po[k] = S[k * NB + b];
}
template <typename KT, typename PT>
__device__ __forceinline__ void store_props(const PT &S, int NB, int b, const KProps<KT> &o) {
  const KT *po = reinterpret_cast<const KT *>(&o);
#pragma unroll
  for (int k = 0; k < KForm<KT>::NROW; k++) S[k * NB + b] = po[k];
}
__device__ __forceinline__ void to_float(const BinProps<double> &d, BinProps<float> &o) {
  const double *pd = &d.diam;
  float *po = &o.diam;
#pragma unroll
  for (int k = 0; k < 9; k++) po[k] = (float)pd[k];
}

// per-cell constants of the collision kernel
__device__ __forceinline__ void coag_cell(const DevParams &P, double T, double pres, CoagCell<double> &cd) {
  double visc = ddiv(7.44523e-3 * dsqrt(cube(T)), 5093. * (T + 110.4));
  double mfp = ddiv((1.656e-10 * T + 1.828e-8) * K_PSTAND, pres);
  double zrhoa = ddiv(pres, K_RD * T);
  double vkin = ddiv(visc, zrhoa);
  cd.T_ = T; cd.visc = visc; cd.mfp = mfp; cd.zrhoa = zrhoa; cd.vkin = vkin;
  cd.shearA = dsqrt(ddiv(8. * K_PI * P.eddy_dis, 15. * vkin));
  cd.turbB = ddiv(K_PI * dpow(P.eddy_dis, 0.75), K_GRAV * dsqrt(dsqrt(vkin)));
}
__device__ __forceinline__ void kcell(const DevParams &P, double T, double pres, KCell<float> &k) {
  coag_cell(P, T, pres, k.cd);
  const CoagCell<double> &cd = k.cd;
  CoagCell<float> &cc = k.cc;
  cc.T_ = (float)cd.T_; cc.visc = (float)cd.visc; cc.mfp = (float)cd.mfp; cc.zrhoa = (float)cd.zrhoa;
  cc.vkin = (float)cd.vkin; cc.shearA = (float)cd.shearA; cc.turbB = (float)cd.turbB;
}
__device__ __forceinline__ void kcell(const DevParams &P, double T, double pres, KCell<double> &k) {
  coag_cell(P, T, pres, k.c);
  const double imu = drcp(k.c.visc);
  k.mfp2 = 2. * k.c.mfp;
  k.kx = ddiv(0.999, k.mfp2);
  k.kD4 = (4. * K_BOLTZ / (3. * K_PI)) * T * imu;
  k.kv2 = (8. * K_BOLTZ / K_PI) * T;
  k.k18 = (K_GRAV / 18.) * imu;
  k.ivkin = drcp(k.c.vkin);
  k.vkin4 = 4. * k.c.vkin;
}

template <typename KT, int LS>
__device__ __forceinline__ void shape_of_bin(const DevParams &P, const WS<KT, LS> &w, int b, Shape<double> &sh) {
  if (phase_of(P, b) == 4) {
    double mp = 0.;
    for (int s = 0; s < P.nused - 1; s++) mp += w.v(s, b) * K_RHOIC;
    shape_coeffs<double>(P, sh, mp, w.v(P.nused - 1, b) * K_RHORI, w.numc[b]);
  } else {
    sh.alpha = sh.beta = sh.gamma = sh.sigma = 0.;
  }
}

// Collision properties of bin b (diam == dwet: dnsp equals it after a limited "all" update)
template <int LS>
__device__ __forceinline__ void props_of_bin(const DevParams &P, const WS<float, LS> &w, const KCell<float> &k, int b,
                                             const Shape<double> &sh, BinProps<float> &o) {
  const int ph = phase_of(P, b);
  const double diam = w.dwet[b];
  if (ph < 4) {
    // the mixed form evaluates the per-bin properties of the liquid bins in float as
    // well; ice keeps FP64 (the Khvorostyanov-Curry fall speed carries float rounding
    // of its exponents into ice-drop speed differences, which cancel)
    const float df = (float)diam;
    const float mass = (float)w.rhomean[b] * (float)K_PI6 * cube(df);
    const Shape<float> shf = {0.f, 0.f, 0.f, 0.f};
    bin_props<float>(k.cc, ph, df, df, mass, (float)w.rhomean[b], shf, o);
    return;
  }
  BinProps<double> od;
  bin_props<double>(k.cd, ph, diam, diam, w.rhomean[b] * K_PI6 * cube(diam), w.rhomean[b], sh, od);
  to_float(od, o);
}
template <int LS>
__device__ __forceinline__ void props_of_bin(const DevParams &P, const WS<double, LS> &w, const KCell<double> &k, int b,
                                             const Shape<double> &sh, PairProps &o) {
  const double d = w.dwet[b], rho = w.rhomean[b], rd = drcp(d);
  const double im = rd * rd * rd * (phase_of(P, b) < 4 ? 1. / (K_RHOWA * K_PI6) : drcp(rho * K_PI6));
  pair_props(k, phase_of(P, b), d, rd, im, d, rho, sh, o);
}
// Properties of the first particle of a pair of equal-size bins (i, j), the self-coagulation
// offset (:273-276): 1.1 times the diameter and 1.33 times the mass of particle 2; sh is bin
// i's shape.  For liquid bins they depend on bin j alone: the fall speed takes the same
// branch for every liquid phase, every liquid density is that of water and the
// sphere-equivalent diameter enters only for ice.
template <int LS>
__device__ __forceinline__ void offset_props(const DevParams &P, const WS<float, LS> &w, const KCell<float> &k,
                                             const Shape<double> &sh, int i, int j, BinProps<float> &a) {
  if (phase_of(P, i) < 4) {
    const float dj = (float)w.dwet[j], mj = (float)w.rhomean[j] * (float)K_PI6 * cube(dj);
    const Shape<float> shf = {0.f, 0.f, 0.f, 0.f};
    bin_props<float>(k.cc, phase_of(P, i), 1.1f * dj, (float)w.dwet[i], 1.33f * mj, (float)w.rhomean[i], shf, a);
    return;
  }
  const double dj = w.dwet[j], mj = w.rhomean[j] * K_PI6 * cube(dj);
  BinProps<double> ad;
  bin_props<double>(k.cd, phase_of(P, i), 1.1 * dj, w.dwet[i], 1.33 * mj, w.rhomean[i], sh, ad);
  to_float(ad, a);
}
template <int LS>
__device__ __forceinline__ void offset_props(const DevParams &P, const WS<double, LS> &w, const KCell<double> &k,
                                             const Shape<double> &sh, int i, int j, PairProps &a) {
  const double dj = w.dwet[j], rdj = drcp(dj);
  const double im = rdj * rdj * rdj *
                    (phase_of(P, j) < 4 ? 1. / (1.33 * K_RHOWA * K_PI6) : drcp(1.33 * K_PI6 * w.rhomean[j]));
  pair_props(k, phase_of(P, i), 1.1 * dj, (1. / 1.1) * rdj, im, w.dwet[i], w.rhomean[i], sh, a);
}
__device__ __forceinline__ float pair_kernel(const KCell<float> &k, const BinProps<float> &a, const BinProps<float> &b) {
  return coag_pair<float>(k.cc, a, b);
}

// charging enhancement (:411-416)
template <typename KT, int LS>
__device__ __forceinline__ KT charged(const DevParams &P, const WS<KT, LS> &w, KT k, int i, int j) {
  if (P.lcharge) {
    double kd = (double)k;
    kd = kd + ddiv(kd * P.chargeCollEnh * 0.5 * (w.ctime[i] + w.ctime[j]), P.chargeTimeMax);
    k = (KT)kd;
  }
  return k;
}

template <typename KT, bool OFFSET>
__device__ void eval_pairs(const DevParams &P, const WS<KT, 32> &w, const KCell<KT> &kc, const KT *S, const int *list,
                           int n, int lane) {
  const int NB = w.NB;
  if (lane < n) {
    int q = list[lane];
    int i = q & 0xff, j = (q >> 8) & 0xff;
    KProps<KT> a, b;
    load_props<KT>(S, NB, j, b);
    if (OFFSET) {
      Shape<double> sh;
      shape_of_bin(P, w, i, sh);
      offset_props(P, w, kc, sh, i, j, a);
    } else {
      load_props<KT>(S, NB, i, a);
    }
    w.K[tri(i, j, NB)] = charged(P, w, pair_kernel(kc, a, b), i, j);
  }
}

// ----------------------------------------------------------------------------------------
// Collision kernels for all enabled bin pairs: mo_salsa_coagulation_kernels.f90:24-180
// (buildKernelSelf/buildKernel: pairs whose partner has numc < nlim are zero).
// Scratch: the rows of the bins' properties (KForm<KT>::NROW of them).
// ----------------------------------------------------------------------------------------
template <typename KT>
__device__ __forceinline__ void build_kernels(const DevParams &P, const WS<KT, 32> &w, double T, double pres, int lane) {
  const int NB = w.NB;
  KCell<KT> kc;
  kcell(P, T, pres, kc);
  KT *S = reinterpret_cast<KT *>(w.scr);   // KT-typed scratch, NROW * NB entries
  // per-bin properties of the populated bins only (a pair with an empty bin has K = 0)
  const unsigned lt = (1u << lane) - 1u;
  int nact = 0;
  for (int base = 0; base < P.ntotal; base += 32) {
    int b = base + lane;
    bool act = b < P.ntotal && num_ge(w.numc[b], nlim_of(phase_of(P, b)));
    unsigned bal = __ballot_sync(0xffffffffu, act);
    if (act) w.pbuf[nact + __popc(bal & lt)] = b;
    nact += __popc(bal);
  }
  __syncwarp();
  for (int e = lane; e < nact; e += 32) {
    const int b = w.pbuf[e];
    Shape<double> sh;
    KProps<KT> o;
    shape_of_bin(P, w, b, sh);
    props_of_bin(P, w, kc, b, sh, o);
    store_props<KT>(S, NB, b, o);
  }
  __syncwarp();
  // Scan the pair table, compact the active pairs into pbuf and evaluate them 32 at a
  // time.  The table lists the pairs of equal-size bins (self-coagulation offset) last,
  // so those evaluate in batches of their own.
  for (int sec = 0; sec < 2; sec++) {
    const int p0 = sec == 0 ? 0 : P.npairs_plain, p1 = sec == 0 ? P.npairs_plain : P.npairs;
    int nbuf = 0;
    for (int base = p0; base < p1; base += 32) {
      bool act = false;
      int pk = 0;
      int t = base + lane;
      if (t < p1) {
        pk = __ldg(P.pairs + t);
        int i = pk & 0xff, j = (pk >> 8) & 0xff;
        act = num_ge(w.numc[i], nlim_of(phase_of(P, i))) && num_ge(w.numc[j], nlim_of(phase_of(P, j)));
        if (!act) w.K[tri(i, j, NB)] = (KT)0;
      }
      unsigned bal = __ballot_sync(0xffffffffu, act);
      if (act) w.pbuf[nbuf + __popc(bal & lt)] = pk;
      nbuf += __popc(bal);
      __syncwarp();
      if (nbuf >= 32) {
        if (sec == 0) eval_pairs<KT, false>(P, w, kc, S, w.pbuf + nbuf - 32, 32, lane);
        else eval_pairs<KT, true>(P, w, kc, S, w.pbuf + nbuf - 32, 32, lane);
        nbuf -= 32;
        __syncwarp();
      }
    }
    if (nbuf > 0) {
      if (sec == 0) eval_pairs<KT, false>(P, w, kc, S, w.pbuf, nbuf, lane);
      else eval_pairs<KT, true>(P, w, kc, S, w.pbuf, nbuf, lane);
    }
    __syncwarp();
  }
}


// The lane form: the pair table in order (its entries are sorted by the first bin, whose
// properties stay in registers), every cell of the warp at the same pair.  The kernel of an
// equal-size pair of liquid bins is that of the larger bin with itself, evaluated once per
// bin with the properties.
template <typename KT>
__device__ __forceinline__ void build_kernels(const DevParams &P, const WS<KT, 1> &w, double T, double pres, int) {
  const int NB = w.NB;
  KCell<KT> kc;
  kcell(P, T, pres, kc);
  const Col<KT> S = row_cast<KT>(w.scr);
  const bool eq = P.npairs > P.npairs_plain;
  for (int b = 0; b < P.ntotal; b++) {
    if (!w.on(b) || !(num_ge(w.numc[b], nlim_of(phase_of(P, b))))) continue;
    Shape<double> sh;
    KProps<KT> o;
    shape_of_bin(P, w, b, sh);
    props_of_bin(P, w, kc, b, sh, o);
    store_props<KT>(S, NB, b, o);
    if (eq) {
      KProps<KT> a;
      offset_props(P, w, kc, sh, b, b, a);
      w.K[tri(b, b, NB)] = pair_kernel(kc, a, o);
    }
  }
  KProps<KT> a;
  int ia = -1;
  for (int t = 0; t < P.npairs; t++) {
    const int pk = __ldg(P.pairs + t), i = pk & 0xff, j = (pk >> 8) & 0xff, ij = tri(i, j, NB);
    if (!w.on(i) || !w.on(j)) {
      if (P.kc_mode == 1) w.K[ij] = (KT)0;   // the stored triangle; no sum reads it here
      continue;
    }
    if (t < P.npairs_plain && i != ia) {
      load_props<KT>(S, NB, i, a);   // every lane, whether its bin i is populated or not
      ia = i;
    }
    KT k = (KT)0;
    if (num_ge(w.numc[i], nlim_of(phase_of(P, i))) && num_ge(w.numc[j], nlim_of(phase_of(P, j)))) {
      if (t < P.npairs_plain) {
        KProps<KT> b;
        load_props<KT>(S, NB, j, b);
        k = pair_kernel(kc, a, b);
      } else if (i == j || phase_of(P, j) < 4) {
        k = w.K[tri(j, j, NB)];   // pairs (i, j) come before (j, j), which is charged last
      } else {
        // a drop and a crystal bin of the same size
        Shape<double> sh;
        shape_of_bin(P, w, i, sh);
        KProps<KT> c, b;
        load_props<KT>(S, NB, j, b);
        offset_props(P, w, kc, sh, i, j, c);
        k = pair_kernel(kc, c, b);
      }
      k = charged(P, w, k, i, j);
    }
    w.K[ij] = k;
  }
}


// ----------------------------------------------------------------------------------------
// Semi-implicit coagulation update: mo_salsa_coagulation_processes.f90:24-702 and the
// driver mo_salsa_dynamics.f90:92-202.  Target bins are visited in the reference order
// (ice, precipitation, aerosol, cloud; ascending bins); every partner sum of one target
// is accumulated lane-parallel and reduced once.  Only the diagnostics that reach the
// output fields are accumulated (the number-only rate tallies of accumulateSink never do).
// ----------------------------------------------------------------------------------------
// Sum eight per-lane values over the warp with 9 adds: each butterfly step keeps half of
// the values and exchanges the other half, after which every lane receives all totals.
__device__ __forceinline__ void warp_sum8(double (&v)[8], int lane) {
  const unsigned F = 0xffffffffu;
  const bool h = lane & 16, g = lane & 8, f = lane & 4;
  double a[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    double send = h ? v[i] : v[i + 4];
    double keep = h ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(F, send, 16);
  }
  double b[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    double send = g ? a[i] : a[i + 2];
    double keep = g ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(F, send, 8);
  }
  double c = (f ? b[1] : b[0]) + __shfl_xor_sync(F, f ? b[0] : b[1], 4);
  c += __shfl_xor_sync(F, c, 2);
  c += __shfl_xor_sync(F, c, 1);
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = __shfl_sync(F, c, ((i >> 2) << 4) | (((i >> 1) & 1) << 3) | ((i & 1) << 2));
}

// Compensated (Kahan) float accumulator of the mixed form's partner sums: the running
// sum and the correction of its rounding.  After the warp reduction it holds the total.
struct KahanF {
  float s, c;
  __device__ __forceinline__ KahanF &operator=(float x) { s = x; c = 0.f; return *this; }
  __device__ __forceinline__ KahanF &operator+=(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
    return *this;
  }
  __device__ __forceinline__ operator double() const { return (double)s; }
};

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// warp_sum8 for compensated float sums: every exchange adds the high parts exactly
// (two_sum) and carries the low parts, so the totals keep float accuracy whatever the
// cancellation between lanes; every lane receives the eight totals (high + low).
__device__ __forceinline__ void warp_sum8_comp(float (&hi)[8], float (&lo)[8], int lane) {
  const unsigned F = 0xffffffffu;
  const bool h = lane & 16, g = lane & 8, f = lane & 4;
  float ah[4], al[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float sh = h ? hi[i] : hi[i + 4], kh = h ? hi[i + 4] : hi[i];
    const float sl = h ? lo[i] : lo[i + 4], kl = h ? lo[i + 4] : lo[i];
    const float rh = __shfl_xor_sync(F, sh, 16), rl = __shfl_xor_sync(F, sl, 16);
    float e;
    two_sum(kh, rh, ah[i], e);
    al[i] = kl + rl + e;
  }
  float bh[2], bl[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float sh = g ? ah[i] : ah[i + 2], kh = g ? ah[i + 2] : ah[i];
    const float sl = g ? al[i] : al[i + 2], kl = g ? al[i + 2] : al[i];
    const float rh = __shfl_xor_sync(F, sh, 8), rl = __shfl_xor_sync(F, sl, 8);
    float e;
    two_sum(kh, rh, bh[i], e);
    bl[i] = kl + rl + e;
  }
  float ch, cl;
  {
    const float sh = f ? bh[0] : bh[1], kh = f ? bh[1] : bh[0];
    const float sl = f ? bl[0] : bl[1], kl = f ? bl[1] : bl[0];
    const float rh = __shfl_xor_sync(F, sh, 4), rl = __shfl_xor_sync(F, sl, 4);
    float e;
    two_sum(kh, rh, ch, e);
    cl = kl + rl + e;
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1) {
    const float rh = __shfl_xor_sync(F, ch, o), rl = __shfl_xor_sync(F, cl, o);
    float sh, e;
    two_sum(ch, rh, sh, e);
    ch = sh;
    cl = cl + rl + e;
  }
  const float c = ch + cl;
#pragma unroll
  for (int i = 0; i < 8; i++) hi[i] = __shfl_sync(F, c, ((i >> 2) << 4) | (((i >> 1) & 1) << 3) | ((i & 1) << 2));
}

// Partner sums of one target bin: FP64 in the FP64 form; compensated float sums in the
// mixed form, from float kernels and float copies of the partner state.
template <typename KT, int LS>
struct TAccT {
  using A = typename std::conditional<sizeof(KT) == 4, KahanF, double>::type;
  A sink, self;
  A src[SALSA_NSV];
  A dg[7];   // 0 autoc(abs) 1 autoc80 2 autoc50 3 accr 4 accr80 5 accr50 6 coll mass
  KT cm;     // the lane's part of dg[6], added at the end
  // additions of a partner's term; `leaf` is its lane in the warp form (see the lane form's
  // float sums below)
  __device__ __forceinline__ void add_sink(KT x, int) { sink += x; }
  __device__ __forceinline__ void add_self(KT x, int) { self += x; }
  __device__ __forceinline__ void add_src(int s, KT x, int) { src[s] += x; }
  __device__ __forceinline__ void add_dg(int d, KT x, int) { dg[d] += x; }
  __device__ __forceinline__ KT cm_get(int) const { return cm; }
  __device__ __forceinline__ void cm_put(int, KT x) { cm = x; }
  __device__ __forceinline__ void cm_add() { dg[6] += cm; }
  template <typename W> __device__ __forceinline__ void zero(const W &) {
    cm = (KT)0;
    sink = (KT)0; self = (KT)0;
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++) src[s] = (KT)0;
#pragma unroll
    for (int d = 0; d < 7; d++) dg[d] = (KT)0;
  }
  __device__ __forceinline__ void reduce(bool diag, int lane) {
    if constexpr (LS == 1) {
      // one lane holds the totals
    } else if constexpr (sizeof(KT) == 4) {
      float h[8], l[8];
#pragma unroll
      for (int s = 0; s < 7; s++) { h[s] = src[s].s; l[s] = -src[s].c; }
      h[7] = sink.s; l[7] = -sink.c;
      warp_sum8_comp(h, l, lane);
#pragma unroll
      for (int s = 0; s < 7; s++) src[s] = h[s];
      sink = h[7];
      if (diag) {
        h[0] = self.s; l[0] = -self.c;
#pragma unroll
        for (int d = 0; d < 7; d++) { h[d + 1] = dg[d].s; l[d + 1] = -dg[d].c; }
        warp_sum8_comp(h, l, lane);
        self = h[0];
#pragma unroll
        for (int d = 0; d < 7; d++) dg[d] = h[d + 1];
      } else {
        self = __shfl_sync(0xffffffffu, self.s - self.c, 0);   // self terms are accumulated on lane 0 only
      }
    } else {
      double v[8];
#pragma unroll
      for (int s = 0; s < 7; s++) v[s] = src[s];
      v[7] = sink;
      warp_sum8(v, lane);
#pragma unroll
      for (int s = 0; s < 7; s++) src[s] = v[s];
      sink = v[7];
      if (diag) {
        double u[8];
        u[0] = self;
#pragma unroll
        for (int d = 0; d < 7; d++) u[d + 1] = dg[d];
        warp_sum8(u, lane);
        self = u[0];
#pragma unroll
        for (int d = 0; d < 7; d++) dg[d] = u[d + 1];
      } else {
        self = __shfl_sync(0xffffffffu, self, 0);   // self terms are accumulated on lane 0 only
      }
    }
  }
};

// The mixed form's sums in the lane form.  Each of the warp form's 32 lanes adds its partners
// in a compensated float pair and the pairs are added over the lanes in a fixed tree, with
// one rounding to float at the end; the lane form keeps those pairs in its workspace
// (`leaf`: the warp form's lane of a partner) and adds them in the same tree, so that both
// forms round alike.
struct LeafSums {
  static constexpr int SINK = 7, SELF = 8, DG = 9, CM = 16, N = 17;   // slots; 0-6 are the species
  Col<float> lf;
  unsigned m[N];   // leaves that hold something
  float src[SALSA_NSV], sink, self, dg[7];
  __device__ __forceinline__ void acc(int i, float x, int leaf) {
    const Col<float> q = lf + (leaf * N + i) * 2;
    KahanF k;
    k = 0.f;
    if ((m[i] >> leaf) & 1u) { k.s = q[0]; k.c = q[1]; }
    m[i] |= 1u << leaf;
    k += x;
    q[0] = k.s;
    q[1] = k.c;
  }
  __device__ __forceinline__ void add_sink(float x, int leaf) { acc(SINK, x, leaf); }
  __device__ __forceinline__ void add_self(float x, int leaf) { acc(SELF, x, leaf); }
  __device__ __forceinline__ void add_src(int s, float x, int leaf) { acc(s, x, leaf); }
  __device__ __forceinline__ void add_dg(int d, float x, int leaf) { acc(DG + d, x, leaf); }
  __device__ __forceinline__ float cm_get(int leaf) const { return (m[CM] >> leaf) & 1u ? lf[(leaf * N + CM) * 2] : 0.f; }
  __device__ __forceinline__ void cm_put(int leaf, float x) {
    lf[(leaf * N + CM) * 2] = x;
    m[CM] |= 1u << leaf;
  }
  __device__ __forceinline__ void cm_add() {
    for (int l = 0; l < 32; l++)
      if ((m[CM] >> l) & 1u) acc(DG + 6, lf[(l * N + CM) * 2], l);
  }
  template <typename W> __device__ __forceinline__ void zero(const W &w) {
    lf = w.lf;
#pragma unroll
    for (int i = 0; i < N; i++) m[i] = 0u;
  }
  // the total of slot i over the leaves (warp_sum8_comp's tree)
  __device__ __forceinline__ float total(int i) const {
    if (m[i] == 0u) return 0.f;
    float h4 = 0.f, l4 = 0.f, h3 = 0.f, l3 = 0.f, h2 = 0.f, l2 = 0.f, h1 = 0.f, l1 = 0.f, h0 = 0.f, l0 = 0.f;
    float h = 0.f, l = 0.f;
    auto merge = [&](float a, float b) {   // (a, b) + (h, l)
      float t, e;
      two_sum(a, h, t, e);
      l = b + l + e;
      h = t;
    };
#pragma unroll 1
    for (int k = 0; k < 32; k++) {
      const int leaf = (int)(__brev((unsigned)k) >> 27);
      h = 0.f;
      l = 0.f;
      if ((m[i] >> leaf) & 1u) {
        const Col<float> q = lf + (leaf * N + i) * 2;
        h = q[0];
        l = -q[1];
      }
      if (!(k & 1)) { h4 = h; l4 = l; continue; }
      merge(h4, l4);
      if (!(k & 2)) { h3 = h; l3 = l; continue; }
      merge(h3, l3);
      if (!(k & 4)) { h2 = h; l2 = l; continue; }
      merge(h2, l2);
      if (!(k & 8)) { h1 = h; l1 = l; continue; }
      merge(h1, l1);
      if (!(k & 16)) { h0 = h; l0 = l; continue; }
      merge(h0, l0);
    }
    return h + l;
  }
  __device__ __forceinline__ void reduce(bool diag, int) {
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++) src[s] = total(s);
    sink = total(SINK);
    if (diag) {
      self = total(SELF);
#pragma unroll
      for (int d = 0; d < 7; d++) dg[d] = total(DG + d);
    } else {
      self = m[SELF] & 1u ? lf[SELF * 2] - lf[SELF * 2 + 1] : 0.f;   // lane 0 alone
    }
  }
};
template <> struct TAccT<float, 1> : LeafSums {};
static_assert(SALSA_LEAF_ROWS == 32 * LeafSums::N, "32 leaves of N float pairs");

// float copies of the partner state for the mixed form's coagulation update: every bin
// before the sweep, then each bin again whenever the sweep changes it
template <typename KT, int LS>
__device__ __forceinline__ void shadow_all(const DevParams &P, const WS<KT, LS> &w, int lane) {
  if constexpr (sizeof(KT) == 4) {
    const int NB = w.NB, n = P.ntotal;
    for (int b = lane; b < n; b += LS) w.nf[b] = (float)w.numc[b];
    for (int e = lane; e < P.nused * NB; e += LS) w.vf[e] = (float)w.volc[e];
    wsync<LS>();
  }
}
template <typename KT, int LS>
__device__ __forceinline__ void shadow_bin(const DevParams &P, const WS<KT, LS> &w, int b, int lane) {
  if constexpr (sizeof(KT) == 4) {
    for (int s = lane; s <= P.nused; s += LS) {
      if (s < P.nused) w.vf[s * w.NB + b] = (float)w.v(s, b);
      else w.nf[b] = (float)w.numc[b];
    }
    wsync<LS>();
  }
}

// ----------------------------------------------------------------------------------------
// Secondary ice (mo_salsa_secondary_ice.f90:6-40).  Only the SIP instantiations of the
// step compile this code.  Coagulation tallies the collisions the three schemes read,
// at the point of its Gauss-Seidel sweep where the reference does; the schemes then
// run on lane 0 after coagulation.  The per-cell tallies and the schemes' scratch sit
// at the end of the warp's workspace (P.sip_off doubles after its start); n = nice,
// p = nprc, V = SALSA_NSV:
//   nfrzn_rs, mfrzn_rs, nfrzn_df, mfrzn_df  p x n each (precipitation or cloud row, ice bin)
//   nii_ibr, mii_ibr                        n x n each
//   scratch                                 7 n + 3 n V
//   tracers SIP_drfr, SIP_rmspl, SIP_iibr   3 n (per m3 of air during the step)
//   the schemes' rates, melting flags       4, n
// ----------------------------------------------------------------------------------------
#define SIP_DLLIQ_RS 24.0e-6   // mo_salsa_SIP_RS.f90:17: smallest drop that splinters on riming
#define SIP_DLLIQ_DF 100.e-6   // mo_salsa_SIP_DF.f90:18: smallest drop that fractures on freezing
#define SALSA_DIAG_SIPDRFR_SLOT 17   // diagnostic slot of s_n_sipdrfr (then s_n_siprmspl, s_n_sipiibr)

template <typename D>
struct SipT {
  D nrs, mrs, ndf, mdf, nii, mii, scr, tr, rate, melt;
};
template <typename D>
__device__ __forceinline__ SipT<D> sip_tallies(const DevParams &P, D wsbase) {
  const int n = P.nice, pn = P.nprc * n, nn = n * n;
  const D t = wsbase + P.sip_off;
  const D scr = t + (4 * pn + 2 * nn), tr = scr + (7 * n + 3 * n * SALSA_NSV);
  return {t, t + pn, t + 2 * pn, t + 3 * pn, t + 4 * pn, t + (4 * pn + nn), scr, tr, tr + 3 * n, tr + (3 * n + 4)};
}

// zero tallies and rates; the tracers from their rows, per m3 of air (mo_salsa_driver.f90:258-262)
template <typename KT, int LS>
__device__ void sip_clear(const DevParams &P, const WS<KT, LS> &w, double dn, int lane) {
  const auto t = w.raw + P.sip_off;
  const int n = 4 * P.nprc * P.nice + 2 * P.nice * P.nice;
  for (int e = lane; e < n; e += LS) t[e] = 0.;
  const auto s = sip_tallies(P, w.raw);
  for (int e = lane; e < 3 * P.nice; e += LS) s.tr[e] = w.raw[P.raw_sip + e] * dn;
  for (int e = lane; e < 4; e += LS) s.rate[e] = 0.;
  wsync<LS>();
}

// accumulateSink's secondary-ice block (coagulation_processes.f90:863-944) for the liquid
// target tg (a cloud or precipitation bin) and its ice collectors: the frozen-drop
// numbers of drop fracturing (drops larger than the crystal) and rime splintering
// (drops not larger), in row `row` (the precipitation bin, or 0 for every cloud bin).
// tnlim is the target's number limit.  Lane 0.
template <typename KT, int LS>
__device__ void sip_drop_numbers(const DevParams &P, const WS<KT, LS> &w, int tg, int row, double tnlim) {
  const int I0 = P.nliquid, nice = P.nice;
  const auto s = sip_tallies(P, w.raw);
  double sum = 0.;
  for (int l = 0; l < nice; l++) sum += (double)kget(w, tg, I0 + l) * w.numc[I0 + l];
  const double fix = fmax(1. - sum, 0.1);
  const double Dt = w.dwet[tg], Nt = w.numc[tg];
  for (int ll = 0; ll < nice; ll++) {
    const int g = I0 + ll;
    const double Nl = w.numc[g], Dl = w.dwet[g];
    const double r = (double)kget(w, tg, g) * Nl * Nt * fix;
    if (P.st_sipdf && Nl > K_PRLIM && Dl < Dt && Dt > SIP_DLLIQ_DF && Nt > tnlim) s.ndf[row * nice + ll] += r;
    // :916-921, :936-941: Phillips' full scheme also counts drops collected by larger crystals
    if (P.st_sipdf && P.sip_df_mode == 4 && Nl > K_PRLIM && Dl >= Dt && Dt > SIP_DLLIQ_DF && Nt > tnlim)
      s.ndf[row * nice + ll] += r;
    if (P.st_siprs && Dl >= Dt && Dt > SIP_DLLIQ_RS && Nt > tnlim && Nl > K_PRLIM) s.nrs[row * nice + ll] += r;
  }
}

// accumulateSink's ice-ice breakup block (:881-896) for ice target kk: collisions with the
// larger crystals kk+1..nice-1, with the aggregation efficiency of the pair.  Lane 0.
template <typename KT, int LS>
__device__ void sip_iibr_numbers(const DevParams &P, const WS<KT, LS> &w, int kk, double rf_t) {
  const int I0 = P.nliquid, nice = P.nice, tg = I0 + kk;
  const auto s = sip_tallies(P, w.raw);
  double sum = 0.;
  for (int l = 0; l < nice; l++) sum += (double)kget(w, tg, I0 + l) * w.numc[I0 + l];
  const double fix = fmax(1. - sum, 0.1);
  for (int ll = kk + 1; ll < nice; ll++) {
    const int g = I0 + ll;
    if (w.dnsp[tg] < w.dnsp[g] && w.numc[tg] > K_PRLIM && w.numc[g] > K_PRLIM) {
      const double rf = fmax(rimefrac(P, w.numc[g], w.v(P.iwa, g), w.v(P.irim, g), 4), rf_t);
      const double E = P.Eiagg_max - rf * (P.Eiagg_max - P.Eiagg_min);
      s.nii[ll * nice + kk] += E * (double)kget(w, g, tg) * w.numc[g] * w.numc[tg] * fix;
    }
  }
}

// accumulateSourcePhaseChange's secondary-ice block (:1285-1378) for ice target kk and the
// liquid collectors c0 + istr..iend of a category with nb bins (cloud or precipitation):
// the ice target's diameters are updated (:1291-1308), then the frozen-drop masses are
// tallied; drops from cloud bins use the kernel of cloud bin 1 (ix = 1), as the
// reference writes it.  Lane 0.
template <typename KT, int LS>
__device__ void sip_drop_masses(const DevParams &P, const WS<KT, LS> &w, const double *dmid, int kk, int c0, int nb,
                                int istr, int iend, bool precip) {
  const int nice = P.nice, iwa = P.iwa, tg = P.nliquid + kk;
  const auto s = sip_tallies(P, w.raw);
  double sum = 0.;
  for (int l = 0; l < nb; l++) sum += (double)kget(w, c0 + l, tg) * w.numc[c0 + l];
  const double fix = fmax(1. - sum, 0.1);
  updateDiameterAll(P, w, dmid, tg);
  const double Dt = w.dnsp[tg], Nt = w.numc[tg];
  const double lnlim = precip ? K_PRLIM : K_NLIM;
  for (int ll = istr; ll <= iend; ll++) {
    const int g = c0 + ll, ix = precip ? ll : 0;
    const double Dl = w.dwet[g];
    const double r = (double)kget(w, c0 + ix, tg) * w.v(iwa, g) * Nt * K_RHOWA * fix;
    if (P.st_sipdf && Dt < Dl && Dl > SIP_DLLIQ_DF && Nt > K_PRLIM && w.numc[g] > lnlim) s.mdf[ix * nice + kk] += r;
    // :1331-1343: Phillips' full scheme, drops collected by more massive crystals
    if (P.st_sipdf && P.sip_df_mode == 4 && Dt >= Dl && Dl > SIP_DLLIQ_DF && w.numc[g] > lnlim && Nt > K_PRLIM)
      s.mdf[ix * nice + kk] += r;
    if (P.st_siprs && Dl >= SIP_DLLIQ_RS && Dl < Dt) s.mrs[ix * nice + kk] += r;
  }
}

// accumulateSourceIce's ice-ice breakup block (:1429-1447) for ice target kk: the ice and
// rime mass collected from the smaller crystals 0..kk-1.  Lane 0.
template <typename KT, int LS>
__device__ void sip_iibr_masses(const DevParams &P, const WS<KT, LS> &w, const double *dmid, int kk, double rf_t) {
  const int I0 = P.nliquid, nice = P.nice, tg = I0 + kk;
  const auto s = sip_tallies(P, w.raw);
  updateDiameterAll(P, w, dmid, tg);
  for (int ll = 0; ll < kk; ll++) {
    const int g = I0 + ll;
    if (w.dnsp[tg] > w.dnsp[g] && w.numc[tg] > K_PRLIM && w.numc[g] > K_PRLIM) {
      const double rf = fmax(rimefrac(P, w.numc[g], w.v(P.iwa, g), w.v(P.irim, g), 4), rf_t);
      const double E = P.Eiagg_max - rf * (P.Eiagg_max - P.Eiagg_min);
      s.mii[kk * nice + ll] +=
          E * (double)kget(w, tg, g) * (w.v(P.iwa, g) * K_RHOIC + w.v(P.irim, g) * K_RHORI) * w.numc[tg];
    }
  }
}

// The schemes' common end (mo_salsa_SIP_RS.f90:152-201, _DF.f90:183-237,
// _IIBR.f90:195-250): per source bin, the sink is capped at the bin's content and scaled
// to 99 % of its volume; then fragments are added and sinks removed.
template <typename D>
__device__ void sip_cap_sink(const DevParams &P, const D &numc, const D &volc, int NB, int g, double &sinkn,
                             const D &sinkv) {
  const int nspec = P.nused;
  if (numc[g] < sinkn) {
    sinkn = numc[g];
    for (int s = 0; s < nspec; s++) sinkv[s] = volc[s * NB + g];
  }
  double ssk = 0., sv = 0.;
  for (int s = 0; s < nspec; s++) { ssk += sinkv[s]; sv += volc[s * NB + g]; }
  if (ssk > sv) {
    const double frconst = ddiv(0.99 * sv, ssk);
    for (int s = 0; s < nspec; s++) sinkv[s] = sinkv[s] * frconst;
    sinkn = sinkn * frconst;
    sinkn = fmin(sinkn, 0.99 * numc[g]);
  }
}
template <typename D>
__device__ void sip_apply(const DevParams &P, const D &numc, const D &volc, int NB, const D &fragn, const D &fragv,
                          const D &sinkn, const D &sinkv) {
  const int I0 = P.nliquid, nspec = P.nused;
  for (int bb = 0; bb < P.nice; bb++) {
    const int g = I0 + bb;
    double n = numc[g] + fragn[bb];
    n = n - sinkn[bb];
    numc[g] = fmax(0., n);
    for (int s = 0; s < nspec; s++) {
      double v = volc[s * NB + g] + fragv[bb * SALSA_NSV + s];
      v = v - sinkv[bb * SALSA_NSV + s];
      volc[s * NB + g] = fmax(0., v);
    }
  }
}

// Scratch of the schemes (inside the tally region).
template <typename D>
struct SipScr {
  D fragn, sinkn, fragn_loc, dNb, dVb, diams, bw, fragv, sinkv, fragv_loc;
};
template <typename D>
__device__ __forceinline__ SipScr<D> sip_scratch(const DevParams &P, const SipT<D> &t) {
  const int n = P.nice, V = SALSA_NSV;
  const D p = t.scr;
  SipScr<D> q;
  q.fragn = p; q.sinkn = p + n; q.fragn_loc = p + 2 * n; q.dNb = p + 3 * n; q.dVb = p + 4 * n;
  q.diams = p + 5 * n; q.bw = p + 6 * n;
  q.fragv = p + 7 * n; q.sinkv = q.fragv + n * V; q.fragv_loc = q.sinkv + n * V;
  for (int e = 0; e < 7 * n + 3 * n * V; e++) p[e] = 0.;
  return q;
}
// ice bin centres and widths in diameter (DF :82-88, IIBR :75-81)
template <typename D>
__device__ void sip_bin_geometry(const DevParams &P, const double *tb, SipScr<D> &q) {
  const int I0 = P.nliquid;
  for (int bb = 0; bb < P.nice; bb++) {
    q.diams[bb] = tb[TAB_DMID * P.nb_pad + I0 + bb];
    q.bw[bb] = dpow(divc(tb[TAB_VHI * P.nb_pad + I0 + bb], K_PI6), 1. / 3) - dpow(divc(tb[TAB_VLO * P.nb_pad + I0 + bb], K_PI6), 1. / 3);
  }
}
// Fragments dN spread over the ice bins 0..npmax-1 as d^-3 in number (DF :131-146, IIBR
// :141-156): adds the fragment numbers and volumes (the source bin's composition);
// returns the fragments' total volume sdv, and sv, the source bin g's.
template <typename D>
__device__ double sip_spread(const DevParams &P, const D &volc, int NB, int g, double dN, int npmax, SipScr<D> &q,
                             double &sv) {
  const int nspec = P.nused;
  for (int k = 0; k < P.nice; k++) q.dNb[k] = q.dVb[k] = 0.;
  double Nnorm = 0.;
  for (int k = 0; k < npmax; k++) q.dNb[k] = drcp(cube(q.diams[k]));
  for (int k = 0; k < npmax; k++) Nnorm += q.dNb[k] * q.bw[k];
  for (int k = 0; k < npmax; k++) q.dNb[k] = ddiv(dN * q.dNb[k] * q.bw[k], Nnorm);
  for (int k = 0; k < npmax; k++) q.dVb[k] = q.dNb[k] * K_PI6 * cube(q.diams[k]);
  double sdv = 0.;
  sv = 0.;
  for (int s = 0; s < nspec; s++) sv += volc[s * NB + g];
  for (int k = 0; k < npmax; k++) sdv += q.dVb[k];
  for (int k = 0; k < npmax; k++) {
    q.fragn_loc[k] = q.fragn_loc[k] + q.dNb[k];
    for (int s = 0; s < nspec; s++)
      q.fragv_loc[k * SALSA_NSV + s] = q.fragv_loc[k * SALSA_NSV + s] + volc[s * NB + g] * (ddiv(q.dVb[k], sv));
  }
  return sdv;
}
// the per-source-bin fragments join the totals before the sink safeguard (DF :175-176,
// IIBR :187-188)
template <typename D>
__device__ void sip_fold_local(const DevParams &P, SipScr<D> &q) {
  for (int k = 0; k < P.nice; k++) {
    q.fragn[k] = q.fragn[k] + q.fragn_loc[k];
    for (int s = 0; s < SALSA_NSV; s++) q.fragv[k * SALSA_NSV + s] = q.fragv[k * SALSA_NSV + s] + q.fragv_loc[k * SALSA_NSV + s];
    q.fragn_loc[k] = 0.;
    for (int s = 0; s < SALSA_NSV; s++) q.fragv_loc[k * SALSA_NSV + s] = 0.;
  }
}

// mo_salsa_SIP_RS.f90:28-215 rimesplintering (Hallett-Mossop per kg of rime, mode 1;
// Mossop per frozen drop, mode 2; dltemp_rs = 5: no temperature shape).  Lane 0.
template <typename KT, int LS>
__device__ void sip_rimesplintering(const DevParams &P, const WS<KT, LS> &w, double T, double dt) {
  const int nprc = P.nprc, nice = P.nice, nspec = P.nused, I0 = P.nliquid, NB = w.NB;
  const auto t = sip_tallies(P, w.raw);
  auto q = sip_scratch(P, t);
  const double v_i = 3.405365461487051e-16;   // a 10 um hexagonal column of bulk ice
  const int splbin = P.sip_splbin;
  for (int e = 0; e < nprc * nice; e++) {
    t.mrs[e] = t.mrs[e] * dt;
    t.nrs[e] = t.nrs[e] * dt;
  }
  for (int bb = 0; bb < nice; bb++) {
    const int g = I0 + bb;
    double vall = 0.;
    for (int s = 0; s < nspec; s++) vall += w.v(s, g);
    const auto sinkv = q.sinkv + bb * SALSA_NSV;
    for (int cc = 0; cc < nprc; cc++) {
      const double nf = t.nrs[cc * nice + bb], mf = t.mrs[cc * nice + bb];
      if (T < 238.15 || T > 273.15 || nf < 1.e-12 || vall < 1.e-15 || w.numc[g] < K_PRLIM || bb + 1 < splbin + 2)
        continue;
      const double ddmean = dpow(divc(divc(ddiv(mf, nf), K_RHOWA), K_PI6), 1. / 3.);
      if (ddmean < SIP_DLLIQ_RS) continue;
      const double dN = P.sip_rs_mode == 1 ? 3.5E8 * mf : 4.0E-3 * nf;
      const double dV = dN * v_i;
      q.fragn[splbin - 1] = q.fragn[splbin - 1] + dN;
      double sv = 0.;
      for (int s = 0; s < nspec; s++) sv += w.v(s, g);
      const double f = fmin(ddiv(dV, sv), 1.);
      double ss = 0.;
      for (int s = 0; s < nspec; s++) {
        q.fragv[(splbin - 1) * SALSA_NSV + s] = q.fragv[(splbin - 1) * SALSA_NSV + s] + w.v(s, g) * f;
        const double sk = w.v(s, g) * f;
        sinkv[s] = sinkv[s] + sk;
        ss += sk;
      }
      q.sinkn[bb] = q.sinkn[bb] + ddiv(ss, K_PI6 * dpow(ddmean, 3.0));
      t.tr[nice + splbin - 1] = t.tr[nice + splbin - 1] + dN;   // :134-136
      t.rate[1] += ddiv(dN, dt);
    }
    sip_cap_sink(P, w.numc, w.volc, NB, g, q.sinkn[bb], sinkv);
  }
  sip_apply(P, w.numc, w.volc, NB, q.fragn, q.fragv, q.sinkn, q.sinkv);
}

// mo_salsa_SIP_DF.f90:370-398 fragments per frozen drop: Lawson (mode 1), Sullivan
// (mode 2), Phillips' simple form (mode 3)
__device__ double sip_df_fragments(int mode, double T, double nf, double ddmean) {
  if (mode == 1) return nf * 2.5e-11 * dpow(fmin(ddmean, 3.e-3) * 1.e6, 4.);
  if (mode == 2) {
    // f_gauss(T, 10, 258) / f_gauss(258, 10, 258)
    const double a = sqrt(2. * K_PI_FULL) * 10.;
    double b = (T - 258.) * (T - 258.);
    b = divc(b, 10. * 10.);
    const double hT = ((1. / a) * dexp(-0.5 * b)) / ((1. / a) * exp(-0.5 * 0.));
    return nf * 0.2 * hT * 2.5e-11 * dpow(fmin(ddmean, 3.e-3) * 1.e6, 4.);
  }
  const double t0 = -24. + 273.15, t1 = -20. + 273.15, t2 = -16. + 273.15, t3 = -10. + 273.15, t4 = -6. + 273.15;
  double hT = 0.;
  if (T >= t0 && T < t1) hT = (0.24 - 0.6) * (divc(T - t0, 4.)) + 0.6;
  else if (T >= t1 && T < t2) hT = (2.6 - 0.24) * (divc(T - t2, 4.)) + 2.6;
  else if (T >= t2 && T < t3) hT = (0.43 - 2.6) * (divc(T - t3, 6.)) + 0.43;
  else if (T >= t3 && T < t4) hT = (0.35 - 0.43) * (divc(T - t4, 4.)) + 0.35;
  return nf * ((4. / 9.) * 1.e4 * hT * ddmean);
}

// mo_salsa_SIP_DF.f90:29-260 dropfracturing.  Lane 0.
// Phillips et al. (2018) drop fracturing (mode 4, mo_salsa_SIP_DF.f90:313-608).  Fits in
// x = log10 of the drop diameter in mm, limited to 0.06-1.6 mm (beta: 0 below 0.4 mm).
__device__ __forceinline__ double sip_ph_cubic(double x, double c1, double c2, double c3, double c4) {
  return (c1 * cube(x)) + (c2 * sq(x)) + (c3 * x) + c4;
}
// :431-451 fragments per frozen drop when the drop is heavier than the crystal (eq. 1)
__device__ double sip_df_phillips_mode1(double d, double T) {
  const double tc = T - 273.15, x = log10(fmax(fmin(d * 1.e3, 1.6), 0.06));
  const double T0 = sip_ph_cubic(x, -1.3999, -5.3285, -3.9847, -15.0332);
  const double zeta = dpow(10., sip_ph_cubic(x, 2.4268, 3.3274, 2.0783, 1.2927));
  const double eta = dpow(10., sip_ph_cubic(x, 0.1242, -0.2316, -0.9874, -0.0827));
  double beta = 0.;
  if (!(d < 0.4e-3)) {
    const double xb = log10(fmin(d * 1.e3, 1.6));
    beta = (-0.1839 * sq(xb)) + (-0.2017 * xb) + -0.0512;
  }
  return beta * tc + ddiv(zeta * sq(eta), sq(tc - T0) + sq(eta));
}
// :479-532 the crystal heavier than the drop (eq. 7): the collision's kinetic energy over
// the drop's surface energy
__device__ double sip_df_phillips_mode2(const DevParams &P, double p, double T, double d, double disph, double dinsph,
                                        double mrim, double mpri, double ncice, double rhoip) {
  const double rhoa = ddiv(p, K_RD * T);
  const double visc = ddiv(7.44523e-3 * dsqrt(cube(T)), 5093. * (T + 110.4));
  const double mfp = ddiv((1.656e-10 * T + 1.828e-8) * K_PSTAND, p);
  double knud = ddiv(2. * mfp, dinsph);
  double beta = 1. + knud * (1.142 + 0.558 * dexp(-ddiv(0.999, knud)));
  Shape<double> ish;
  shape_coeffs<double>(P, ish, mpri, mrim, ncice);
  const double vti = terminal_vel<double>(disph, rhoip, rhoa, visc, beta, 4, ish, dinsph);
  knud = ddiv(2. * mfp, d);
  beta = 1. + knud * (1.142 + 0.558 * dexp(-ddiv(0.999, knud)));
  const double vtd = terminal_vel<double>(d, K_RHOWA, rhoa, visc, beta, 3, ish, d);
  const double mip = ddiv(mrim + mpri, ncice), mdp = K_RHOWA * K_PI6 * cube(d);
  const double K0 = 0.5 * (ddiv(mip * mdp, mdp + mip)) * sq(vtd - vti);
  const double DE = ddiv(K0, K_SURFW0 * K_PI * sq(d));
  const double fT = -divc(4200. * (T - 273.15), 3.3e5);   // cwa, alf (mo_submctl.f90:268, 281)
  return 3. * fmin(4. * fT, 1.) * (1. - fT) * fmax(DE - 0.2, 0.);
}
// :313-372 the regime by the masses of drop and crystal (ice bin g)
template <typename KT, int LS>
__device__ double sip_df_phillips_full(const DevParams &P, const WS<KT, LS> &w, double p, double T, double d, int g,
                                       double nf) {
  double sv = 0.;
  for (int s = 0; s < P.nused - 1; s++) sv += w.v(s, g);
  const double mrim = w.v(P.nused - 1, g) * K_RHORI, mpri = sv * K_RHOIC, ncice = w.numc[g];
  const double mip = ddiv(mrim + mpri, ncice), mdp = K_RHOWA * K_PI6 * cube(d);
  if (mdp > mip) {
    if (d < 50.e-6 && T > 267.15) return 0.;
    return fmin(sip_df_phillips_mode1(d, T), 100.) * nf;
  }
  if (d < 150.e-6) return 0.;
  const double rhoip = ddiv(mrim * K_RHORI + mpri * K_RHOIC, mrim + mpri);
  return fmin(sip_df_phillips_mode2(P, p, T, d, w.dwet[g], w.dnsp[g], mrim, mpri, ncice, rhoip), 100.) * nf;
}

template <typename KT, int LS>
__device__ void sip_dropfracturing(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double pres,
                                   double dt) {
  const int nprc = P.nprc, nice = P.nice, nspec = P.nused, I0 = P.nliquid, NB = w.NB;
  const auto t = sip_tallies(P, w.raw);
  auto q = sip_scratch(P, t);
  sip_bin_geometry(P, tb, q);
  for (int e = 0; e < nprc * nice; e++) {
    t.mdf[e] = t.mdf[e] * dt;
    t.ndf[e] = t.ndf[e] * dt;
  }
  for (int bb = 0; bb < nice; bb++) {
    const int g = I0 + bb;
    double vall = 0.;
    for (int s = 0; s < nspec; s++) vall += w.v(s, g);
    const auto sinkv = q.sinkv + bb * SALSA_NSV;
    for (int cc = 0; cc < nprc; cc++) {
      const double nf = t.ndf[cc * nice + bb], mf = t.mdf[cc * nice + bb];
      if (T < 248.15 || T > 271.15 || nf < 1.e-12 || vall < 1.e-15 || w.numc[g] < K_PRLIM) continue;
      const double ddmean = dpow(divc(divc(ddiv(mf, nf), K_RHOWA), K_PI6), 1. / 3.);
      if (ddmean < SIP_DLLIQ_DF) continue;
      int npmax = 0;
      for (int k = 0; k < nice; k++) npmax += q.diams[k] <= ddmean;
      npmax = npmax - 1 > 1 ? npmax - 1 : 1;
      if (npmax <= 2) continue;
      const double dN = P.sip_df_mode == 4 ? sip_df_phillips_full<KT>(P, w, pres, T, ddmean, g, nf)
                                           : sip_df_fragments(P.sip_df_mode, T, nf, ddmean);
      double sv;
      const double sdv = sip_spread(P, w.volc, NB, g, dN, npmax, q, sv);
      double ss = 0.;
      for (int s = 0; s < nspec; s++) {
        const double sk = ddiv(w.v(s, g) * sdv, sv);
        sinkv[s] = sinkv[s] + sk;
        ss += sk;
      }
      q.sinkn[bb] = q.sinkn[bb] + ddiv(ss, divc(ddiv(mf, nf), K_RHOWA));
      double sdn = 0.;                                           // :165-167
      for (int k = 0; k < npmax; k++) t.tr[k] = t.tr[k] + q.dNb[k];
      for (int k = 0; k < nice; k++) sdn += q.dNb[k];
      t.rate[0] += ddiv(sdn, dt);
    }
    sip_fold_local(P, q);
    sip_cap_sink(P, w.numc, w.volc, NB, g, q.sinkn[bb], sinkv);
  }
  sip_apply(P, w.numc, w.volc, NB, q.fragn, q.fragv, q.sinkn, q.sinkv);
}

// mo_salsa_SIP_IIBR.f90:262-291 fragments per collision: Sullivan (mode 1), Sotiropoulou
// (mode 2), at most 100
__device__ double sip_iibr_imf(int mode, double T, double dmin) {
  const double fbr = 280., Tmin = 252., D0 = 0.02;
  double imf;
  if (mode == 1) imf = T < Tmin ? 0. : fmax(0., fbr * dpow(T - Tmin, 1.2) * dexp(-divc(T - Tmin, 5.)));
  else imf = T <= Tmin ? 0. : fmax(0., divc(fbr * dpow(T - Tmin, 1.2) * dexp(-divc(T - Tmin, 5.)) * dmin, D0));
  return fmin(imf, 100.0);
}

// mo_salsa_SIP_IIBR.f90:23-258 iceicecollbreak: each pair (smaller bb, larger cc) breaks
// the smaller crystal; the source bin's diameters are updated first.  Lane 0.
// mo_salsa_SIP_IIBR.f90:588-607 mip and :552-585 getvelocity: mean crystal mass of ice
// bin g, and its fall speed with the bin's shape coefficients and rime-weighted density
template <typename KT, int LS>
__device__ __forceinline__ void sip_iibr_masses(const DevParams &P, const WS<KT, LS> &w, int g, double &mrim, double &mpri) {
  double v = 0.;
  for (int k = 0; k <= P.iwa; k++) v += w.v(k, g);
  mrim = w.v(P.irim, g) * K_RHORI;
  mpri = v * K_RHOIC;
}
template <typename KT, int LS>
__device__ double sip_iibr_velocity(const DevParams &P, const WS<KT, LS> &w, int g, double visc, double rhoa, double mfp) {
  const double knud = ddiv(2. * mfp, w.dnsp[g]);
  const double beta = 1. + knud * (1.142 + 0.558 * dexp(-ddiv(0.999, knud)));
  double mrim, mpri;
  sip_iibr_masses(P, w, g, mrim, mpri);
  const double rhoip = ddiv(mrim * K_RHORI + mpri * K_RHOIC, mrim + mpri);
  Shape<double> sh;
  shape_coeffs<double>(P, sh, mpri, mrim, w.numc[g]);
  return terminal_vel<double>(w.dwet[g], rhoip, rhoa, visc, beta, 4, sh, w.dnsp[g]);
}
// :323-401 imf_phillips_mod: Phillips et al. (2017) breakup with the corrections of
// Sotiropoulou et al. (2020); asperity parameters by the rime fraction of bin `small`, the
// supersaturation over ice ssi and the distance from -15 C; the collision's kinetic energy
// from both bins' fall speeds (:505-548)
template <typename KT, int LS>
__device__ double sip_imf_phillips(const DevParams &P, const WS<KT, LS> &w, double p, double T, int large, int small,
                                   double disphmin, double ssi) {
  const double T0 = 258.15;
  double mrim, mpri;
  sip_iibr_masses(P, w, small, mrim, mpri);
  const double rimfrac = ddiv(mrim, mrim + mpri);
  double a0, C, gg, Nmax;
  if (rimfrac > 0.5) {
    a0 = dexp(14.74 * ssi + 14.28);
    C = dexp(20.15 * ssi + 13.78);
    gg = ssi + 0.55;
    Nmax = 600.;
  } else {
    a0 = 4.75E7;
    C = 1.0E08;
    gg = 0.78;
    Nmax = 500.;
  }
  const double Am = divc(a0, 3.) + fmax(2. / 3. * a0 - 1. / 9. * a0 * fabs(T - T0), 0.);
  const double alpha = K_PI * sq(disphmin);
  const double rhoa = ddiv(p, K_RD * T);
  const double visc = ddiv(7.44523e-3 * dsqrt(cube(T)), 5093. * (T + 110.4));
  const double mfp = ddiv((1.656e-10 * T + 1.828e-8) * K_PSTAND, p);
  const double v1 = sip_iibr_velocity(P, w, large, visc, rhoa, mfp);
  double mr1, mp1;
  sip_iibr_masses(P, w, large, mr1, mp1);
  const double m1 = ddiv(mr1 + mp1, w.numc[large]);
  const double v2 = sip_iibr_velocity(P, w, small, visc, rhoa, mfp);
  const double m2 = ddiv(mrim + mpri, w.numc[small]);
  const double K0 = (ddiv(m1 * m2, m1 + m2)) * (1.7 * sq(v1 - v2) + 0.3 * v1 * v2);
  return fmin(alpha * Am * (1 - dexp(-dpow(ddiv(ddiv(C * K0, alpha), Am), gg))), Nmax);
}

template <typename KT, int LS>
__device__ void sip_iceicecollbreak(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double pres,
                                    double rv, double rsi, double dt) {
  const int nice = P.nice, nspec = P.nused, I0 = P.nliquid, NB = w.NB;
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  const auto t = sip_tallies(P, w.raw);
  auto q = sip_scratch(P, t);
  sip_bin_geometry(P, tb, q);
  for (int e = 0; e < nice * nice; e++) {
    t.mii[e] = t.mii[e] * dt;
    t.nii[e] = t.nii[e] * dt;
  }
  for (int bb = 0; bb < nice; bb++) {
    const int g = I0 + bb;
    const auto sinkv = q.sinkv + bb * SALSA_NSV;
    for (int cc = bb; cc < nice; cc++) {
      const int h = I0 + cc;
      const double nii = t.nii[cc * nice + bb], mii = t.mii[cc * nice + bb];
      double vb = 0., vc = 0.;
      for (int s = 0; s < nspec; s++) { vb += w.v(s, g); vc += w.v(s, h); }
      if (T < 248.15 || T > 270.15 || nii < 1.e-12 || mii < 1.e-15 || vb < 1.e-15 || w.numc[g] < K_PRLIM ||
          vc < 1.e-15 || w.numc[h] < K_PRLIM)
        continue;
      updateDiameterAll(P, w, dmid, g);
      const double v_i = ddiv(ddiv(mii, nii), w.rhomean[g]);
      const double dinsphmin = dpow(divc(v_i, K_PI6), 1. / 3.);
      int npmax = 0;
      for (int k = 0; k < nice; k++) npmax += q.diams[k] <= dinsphmin;
      npmax = npmax - 1;
      if (npmax <= 2) continue;
      double dN;
      if (P.sip_ib_mode == 3) {   // :148-155: bb passes as the larger crystal, as the reference writes it
        const double disphmin = dpow(divc(ddiv(ddiv(mii, nii), w.rhomean[g]), K_PI6), 1. / 3.);
        const double ssi = fmax(0., ddiv(rv, rsi) - 1.0);
        dN = fmin(sip_imf_phillips<KT>(P, w, pres, T, g, h, disphmin, ssi), 600.0) * nii;
      } else {
        dN = sip_iibr_imf(P.sip_ib_mode, T, dinsphmin) * nii;
      }
      double sv;
      const double sdv = sip_spread(P, w.volc, NB, g, dN, npmax, q, sv);
      double ss = 0.;
      for (int s = 0; s < nspec; s++) {
        const double sk = ddiv(w.v(s, g) * sdv, sv);
        sinkv[s] = sinkv[s] + sk;
        ss += sk;
      }
      q.sinkn[bb] = q.sinkn[bb] + ddiv(ss, v_i);
      double sdn = 0.;                                           // :187-189
      for (int k = 0; k < npmax; k++) t.tr[2 * nice + k] = t.tr[2 * nice + k] + q.dNb[k];
      for (int k = 0; k < nice; k++) sdn += q.dNb[k];
      t.rate[2] += ddiv(sdn, dt);
    }
    sip_fold_local(P, q);
    sip_cap_sink(P, w.numc, w.volc, NB, g, q.sinkn[bb], sinkv);
  }
  sip_apply(P, w.numc, w.volc, NB, q.fragn, q.fragv, q.sinkn, q.sinkv);
}

// secondary_ice (mo_salsa_secondary_ice.f90:6-40), after coagulation (mo_salsa.f90:98-99)
template <typename KT, int LS>
__device__ void secondary_ice(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double pres, double rv,
                              double rsi, double dt, int lane) {
  wsync<LS>();
  if (lane == 0) {
    if (P.st_siprs) sip_rimesplintering<KT>(P, w, T, dt);
    if (P.st_sipdf) sip_dropfracturing<KT>(P, w, tb, T, pres, dt);
    if (P.st_sipib) sip_iceicecollbreak<KT>(P, w, tb, T, pres, rv, rsi, dt);
  }
  wsync<LS>();
}

template <typename KT, int LS>
__device__ __forceinline__ void source_range(const WS<KT, LS> &w, int t, int g0, int istr, int iend, int nspec,
                                             TAccT<KT, LS> &a, int lane) {
  for (int ll = istr + lane; ll <= iend; ll += LS) {
    int g = g0 + ll;
    const int leaf = (ll - istr) & 31;
    if (!w.on(g)) continue;
    const KT k = kget(w, g, t);
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++)
      if (s < nspec) a.add_src(s, k * w.vk(s, g), leaf);
  }
}

// Partner lists of target bin t (built by the host from the partner ranges of the
// reference's accumulateSink / accumulateSource calls): header [4 t .. 4 t + 3] =
// sink offset, sink count, source offset, source count; entries are global bin indices.
__device__ __forceinline__ const int16_t *partner_lists(const DevParams &P, const double *tb) {
  return reinterpret_cast<const int16_t *>(tb + P.list_off);
}

template <typename KT, int LS>
__device__ __forceinline__ void list_sinks(const WS<KT, LS> &w, const int16_t *L, int t, TAccT<KT, LS> &a, int lane) {
  const int off = L[4 * t], n = L[4 * t + 1];
  for (int e = lane; e < n; e += LS) {
    const int g = L[off + e], leaf = e & 31;
    if (!w.on(g)) continue;
    a.add_sink(kget(w, t, g) * w.nk(g), leaf);
  }
}

template <typename KT, int LS>
__device__ __forceinline__ void list_sources(const WS<KT, LS> &w, const int16_t *L, int t, int nspec, TAccT<KT, LS> &a,
                                             int lane) {
  const int off = L[4 * t + 2], n = L[4 * t + 3];
  for (int e = lane; e < n; e += LS) {
    const int g = L[off + e], leaf = e & 31;
    if (!w.on(g)) continue;
    const KT k = kget(w, g, t);
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++)
      if (s < nspec) a.add_src(s, k * w.vk(s, g), leaf);
  }
}

// applyCoag (:539-559): lanes 0..nspec-1 update the volumes and lane nspec the number,
// all in one division.
template <typename KT, int LS>
__device__ __forceinline__ void apply_coag(const DevParams &P, const WS<KT, LS> &w, int t, int nspec, double dt,
                                           const TAccT<KT, LS> &a, int lane) {
  if constexpr (LS == 1) {
    const double n = w.numc[t], sink = a.sink, self = a.self;
    const double den = 1. + dt * sink, r = drcp(den);
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++)
      if (s < nspec) w.v(s, t) = ddiv_r(w.v(s, t) + dt * (double)a.src[s] * n, den, r);
    w.numc[t] = ddiv(n, 1. + dt * (sink + self));
    shadow_bin<KT>(P, w, t, lane);
    return;
  }
  double my = 0.;
#pragma unroll
  for (int s = 0; s < SALSA_NSV; s++)
    if (lane == s) my = a.src[s];
  const double n = w.numc[t];
  const double sink = a.sink, self = a.self;
  const bool vol = lane < nspec;
  const double num = vol ? w.v(lane, t) + dt * my * n : n;
  const double den = vol ? 1. + dt * sink : 1. + dt * (sink + self);
  const double q = ddiv(num, den);
  wsync<LS>();
  if (vol) w.v(lane, t) = q;
  else if (lane == nspec) w.numc[t] = q;
  wsync<LS>();
  shadow_bin<KT>(P, w, t, lane);
}

template <typename KT, int LS>
__device__ void coag_aero(const DevParams &P, const WS<KT, LS> &w, const double *tb, double dt, int lane) {
  const int nspec = P.nwet;
  const int16_t *L = partner_lists(P, tb);
  for (int kk = P.in1a; kk <= P.fn2b; kk++) {
    if (num_lt(w.numc[kk], K_NLIM)) continue;
    TAccT<KT, LS> a;
    a.zero(w);
    if (P.lscgaa && lane == 0) a.add_self((KT)0.5 * kget(w, kk, kk) * w.nk(kk), 0);
    list_sinks(w, L, kk, a, lane);
    list_sources(w, L, kk, nspec, a, lane);
    a.reduce(false, lane);
    apply_coag(P, w, kk, nspec, dt, a, lane);
  }
}

// accumulatePrecipFormation (:1457-1584) for the partners istr..iend (cloud-local) of
// target t (cloud-local).  Per-partner contributions are staged in partner slots and
// summed per precipitation bin in partner order, which keeps the result deterministic.
template <typename KT, int LS>
__device__ void precip_formation(const DevParams &P, const WS<KT, LS> &w, const double *tb, int t, int istr, int iend,
                                 double fix, bool selfcoll, TAccT<KT, LS> &a, bool diag, int lane) {
  const int C0 = P.nbins, nspec = P.nwet, nprc = P.nprc, iwa = P.iwa;
  const double *pbins = tb + TAB_PRECPBINS * P.nb_pad;
  const auto pf = w.misc + M_PF;                // [0..6] volsink, then vol_prc[nprc][7], num_prc[nprc], INFnum[nprc]
  const auto vol_prc = pf + 7, num_prc = pf + (7 + 7 * nprc), inf_prc = num_prc + nprc;
  const auto slot = w.misc + M_PFSLOT;          // 8 slots x 10: tp, dvol[7], dnum, x*dnum
  const int tg = C0 + t;
  if constexpr (LS == 1) {
    const double dt3 = cube(w.dwet[tg]);
    for (int ll = istr; ll <= iend; ll++) {
      const int lg = C0 + ll, leaf = (ll - istr) & 7;   // partners in chunks of eight lanes
      if (!w.on(lg)) continue;
      const double D_new = dcbrt(dt3 + cube(w.dwet[lg]));
      int cnt = 0;
      for (int i = 0; i < nprc; i++) cnt += num_gt(D_new, pbins[i]);
      const double klt = (double)kget(w, lg, tg), nt = w.numc[tg], nl = w.numc[lg];
      if (cnt > 0) {
        const int tp = cnt - 1;
        double dvw = 0., dnum, xin;
        for (int s = 0; s < nspec; s++) {
          const double dv = selfcoll ? w.v(s, lg) * nt * klt * fix : (w.v(s, lg) * nt + w.v(s, tg) * nl) * klt * fix;
          vol_prc[tp * 7 + s] += dv;
          if (selfcoll) pf[s] += dv;   // volsink_slf
          if (s == iwa) dvw = dv;
        }
        if (selfcoll) {
          dnum = (0.5 * klt * nl * nt) * fix;
          xin = w.indef[lg] * dnum;
          a.add_self((KT)(0.5 * klt * nt), leaf);
        } else {
          dnum = (klt * nl * nt) * fix;
          xin = 0.5 * (w.indef[lg] + w.indef[tg]) * dnum;
          a.add_sink((KT)(klt * nl), leaf);
        }
        num_prc[tp] += dnum;
        inf_prc[tp] += xin;
        if (diag) {
          a.add_dg(0, (KT)dvw, leaf);
          if (num_gt(D_new, 50.e-6)) a.add_dg(2, (KT)dvw, leaf);
          if (num_gt(D_new, 80.e-6)) a.add_dg(1, (KT)dvw, leaf);
        }
      } else if (selfcoll) {
        a.add_self((KT)(0.5 * klt * nl), leaf);
      } else {
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s < nspec) a.add_src(s, (KT)(klt * w.v(s, lg)), leaf);
      }
    }
    return;
  }
  for (int c0 = istr; c0 <= iend; c0 += 8) {
    int np = min(8, iend - c0 + 1);
    if (lane < np) {
      int ll = c0 + lane, lg = C0 + ll;
      double dt3 = cube(w.dwet[tg]) + cube(w.dwet[lg]);
      double D_new = dcbrt(dt3);
      int cnt = 0;
      for (int i = 0; i < nprc; i++) cnt += (D_new > pbins[i]);
      double klt = (double)kget(w, lg, tg);
      double nt = w.numc[tg], nl = w.numc[lg];
      const auto sl = slot + lane * 10;
      sl[0] = (double)(cnt - 1);
      double dnum = 0.;
      if (D_new > pbins[0]) {
        double dvw = 0.;
        if (selfcoll) {
          for (int s = 0; s < nspec; s++) sl[1 + s] = w.v(s, lg) * nt * klt * fix;
          dnum = (0.5 * klt * nl * nt) * fix;
          sl[9] = w.indef[lg] * dnum;
          a.add_self((KT)(0.5 * klt * nt), lane);
        } else {
          for (int s = 0; s < nspec; s++) sl[1 + s] = (w.v(s, lg) * nt + w.v(s, tg) * nl) * klt * fix;
          dnum = (klt * nl * nt) * fix;
          sl[9] = 0.5 * (w.indef[lg] + w.indef[tg]) * dnum;
          a.add_sink((KT)((double)kget(w, tg, lg) * nl), lane);
        }
        dvw = sl[1 + iwa];
        if (diag) {
          a.add_dg(0, (KT)dvw, lane);
          if (D_new > 50.e-6) a.add_dg(2, (KT)dvw, lane);
          if (D_new > 80.e-6) a.add_dg(1, (KT)dvw, lane);
        }
      } else {
        sl[0] = -1.;
        if (selfcoll) a.add_self((KT)(0.5 * (double)kget(w, tg, lg) * nl), lane);
        else {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < nspec) a.add_src(s, (KT)(klt * w.v(s, lg)), lane);
        }
      }
      sl[8] = dnum;
    }
    wsync<LS>();
    // sum the staged contributions per precipitation bin (partner order)
    for (int e = lane; e < nprc * (nspec + 2); e += LS) {
      int tp = e / (nspec + 2), q = e % (nspec + 2);
      double acc = 0.;
      bool any = false;
      for (int j = 0; j < np; j++) {
        const auto sl = slot + j * 10;
        if ((int)sl[0] == tp) { acc += (q < nspec) ? sl[1 + q] : (q == nspec ? sl[8] : sl[9]); any = true; }
      }
      if (any) {
        if (q < nspec) vol_prc[tp * 7 + q] += acc;
        else if (q == nspec) num_prc[tp] += acc;
        else inf_prc[tp] += acc;
      }
    }
    if (selfcoll && lane < nspec) {
      // volsink_slf: the single self partner's contribution (same expression as dvol)
      const auto sl = slot;
      if ((int)sl[0] >= 0) pf[lane] += sl[1 + lane];
    }
    wsync<LS>();
  }
}

template <typename KT, bool SIP, int LS>
__device__ void coag_cloud(const DevParams &P, const WS<KT, LS> &w, const double *tb, double dt, bool diag, int lane) {
  const int nspec = P.nwet, C0 = P.nbins, P0 = P.nbins + P.ncld, nprc = P.nprc;
  const bool autoc1 = P.st_auto && P.auto_mode == 1;
  const int16_t *L = partner_lists(P, tb);
  const auto pf = w.misc + M_PF;
  for (int reg = 0; reg < 2; reg++) {
    int kfirst = reg == 0 ? P.ica_cur : P.icb_cur;
    int klast = reg == 0 ? P.fca_cur : P.fcb_cur;
    int o_first = reg == 0 ? P.icb_cur : P.ica_cur;
    int o_last = reg == 0 ? P.fcb_cur : P.fca_cur;
    for (int kk = kfirst; kk <= klast; kk++) {
      int tg = C0 + kk;
      if (num_lt(w.numc[tg], K_NLIM)) continue;
      TAccT<KT, LS> a;
      a.zero(w);
      if (autoc1) {
        for (int e = lane; e < 7 + nprc * 9; e += LS) pf[e] = 0.;
        wsync<LS>();
      }
      int other = o_first + (kk - kfirst);
      int rel = kk - kfirst;
      list_sinks(w, L, tg, a, lane);
      if constexpr (SIP) {
        if (P.st_secice && P.lscgic && lane == 0) sip_drop_numbers<KT>(P, w, tg, 0, K_NLIM);
        wsync<LS>();
      }
      if (P.lscgcc) {
        if (autoc1) {
          double n = w.numc[tg];
          double fix = fmax(1. - dt * (ddiv(0.5 * (double)kget(w, tg, tg) * (n * n), n)), 0.1);
          precip_formation(P, w, tb, kk, kk, kk, fix, true, a, diag, lane);
        } else if (lane == 0) {
          a.add_self((KT)0.5 * kget(w, tg, tg) * w.nk(tg), 0);
        }
      }
      if (P.lscgca) {
        int iaa = P.ica_par + rel, iab = P.icb_par + rel;
        for (int ll = P.in1a + lane; ll <= iaa; ll += LS) {
          const int leaf = (ll - P.in1a) & 31;
          if (!w.on(ll)) continue;
          const KT k = kget(w, ll, tg);
          {
#pragma unroll
            for (int s = 0; s < SALSA_NSV; s++)
              if (s < nspec) a.add_src(s, k * w.vk(s, ll), leaf);
          }
          if (diag) {
            KT cm = a.cm_get(leaf);
            for (int s = 0; s < P.ndry; s++) cm += k * w.vk(s, ll) * (KT)P.rholiq[s];
            a.cm_put(leaf, cm);
          }
        }
        for (int ll = P.in2b + lane; ll <= iab; ll += LS) {
          const int leaf = (ll - P.in2b) & 31;
          if (!w.on(ll)) continue;
          const KT k = kget(w, ll, tg);
          {
#pragma unroll
            for (int s = 0; s < SALSA_NSV; s++)
              if (s < nspec) a.add_src(s, k * w.vk(s, ll), leaf);
          }
          if (diag) {
            KT cm = a.cm_get(leaf);
            for (int s = 0; s < P.ndry; s++) cm += k * w.vk(s, ll) * (KT)P.rholiq[s];
            a.cm_put(leaf, cm);
          }
        }
        a.cm_add();
      }
      if (P.lscgcc && kk > kfirst) {
        if (autoc1) {
          double s1 = 0.;
          for (int i = kfirst + lane; i <= klast; i += LS) s1 += (double)kget(w, tg, C0 + i) * w.numc[C0 + i];
          s1 = wsum<LS>(s1);
          double fix = fmax(1. - dt * s1, 0.1);
          precip_formation(P, w, tb, kk, kfirst, kk - 1, fix, false, a, diag, lane);
          double s2 = 0.;
          for (int i = o_first + lane; i <= o_last; i += LS) s2 += (double)kget(w, tg, C0 + i) * w.numc[C0 + i];
          s2 = wsum<LS>(s2);
          fix = fmax(1. - dt * s2, 0.1);
          precip_formation(P, w, tb, kk, o_first, other, fix, false, a, diag, lane);
        } else {
          source_range(w, tg, C0, kfirst, kk - 1, nspec, a, lane);
          source_range(w, tg, C0, o_first, other, nspec, a, lane);
        }
      }
      a.reduce(diag, lane);
      if (diag && lane == 0) {
        double nt = w.numc[tg];
        w.misc[M_DIAG + DG_ACCOLL] += a.dg[6] * nt;
        w.misc[M_DIAG + DG_AUTOC] += a.dg[0];
        w.misc[M_DIAG + DG_AUTOC80] += a.dg[1];
        w.misc[M_DIAG + DG_AUTOC50] += a.dg[2];
      }
      apply_coag(P, w, tg, nspec, dt, a, lane);
      if (autoc1) {
        // applyCoagPrecipFormation (:654-702)
        const auto vol_prc = pf + 7, num_prc = pf + (7 + 7 * nprc), inf_num = num_prc + nprc;
        for (int s = lane; s < nspec; s += LS) w.v(s, tg) = w.v(s, tg) - dt * pf[s];
        for (int e = lane; e < nprc * nspec; e += LS) {
          int cc = e / nspec, s = e % nspec;
          w.v(s, P0 + cc) = w.v(s, P0 + cc) + dt * vol_prc[cc * 7 + s];
        }
        wsync<LS>();
        for (int cc = lane; cc < nprc; cc += LS) {
          int g = P0 + cc;
          double nrate = num_prc[cc];
          double inf = nrate > 0. ? ddiv(inf_num[cc], nrate) : 0.;
          double n = w.numc[g] + dt * nrate;
          w.numc[g] = n;
          if (n > K_PRLIM) w.indef[g] = ddiv(w.indef[g] * (n - dt * nrate) + inf * dt * nrate, n);
        }
        wsync<LS>();
        shadow_bin<KT>(P, w, tg, lane);
        for (int cc = 0; cc < nprc; cc++) shadow_bin<KT>(P, w, P0 + cc, lane);
      }
    }
  }
}

template <typename KT, bool SIP, int LS>
__device__ void coag_precp(const DevParams &P, const WS<KT, LS> &w, const double *tb, double dt, bool diag, int lane) {
  const int nspec = P.nwet, C0 = P.nbins, P0 = P.nbins + P.ncld, nprc = P.nprc, iwa = P.iwa;
  const double *pbins = tb + TAB_PRECPBINS * P.nb_pad;
  const int16_t *L = partner_lists(P, tb);
  for (int kk = 0; kk < nprc; kk++) {
    int tg = P0 + kk;
    if (num_lt(w.numc[tg], K_PRLIM)) continue;
    TAccT<KT, LS> a;
    a.zero(w);
    double num_slf = 0.;
    list_sinks(w, L, tg, a, lane);
    if constexpr (SIP) {
      if (P.st_secice && P.lscgip && lane == 0) sip_drop_numbers<KT>(P, w, tg, kk, K_PRLIM);
      wsync<LS>();
    }
    if (P.lscgpp && kk == nprc - 1 && lane == 0) a.add_self((KT)0.5 * kget(w, tg, tg) * w.nk(tg), 0);
    const double D = w.dwet[tg], D3 = cube(D);
    const bool lt80 = num_gt(D, 0.) && num_lt(D, 80.e-6), lt50 = num_gt(D, 0.) && num_lt(D, 50.e-6);
    const bool bin80 = num_gt(pbins[kk], 80.e-6), bin50 = num_gt(pbins[kk], 50.e-6);
    if (P.lscgpa) {
      for (int ll = P.in1a + lane; ll <= P.fn2b; ll += LS) {
        const int leaf = (ll - P.in1a) & 31;
        if (!w.on(ll)) continue;
        const KT k = kget(w, ll, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < nspec) a.add_src(s, k * w.vk(s, ll), leaf);
        }
        if (diag) {
          KT cm = a.cm_get(leaf);
          for (int s = 0; s < P.ndry; s++) cm += k * w.vk(s, ll) * (KT)P.rholiq[s];
          a.cm_put(leaf, cm);
        }
      }
      a.cm_add();
    }
    if (P.lscgpc) {
      // source from cloud; accretion and autoconversion diagnostics (:1086-1215, coll phase 2)
      for (int ll = lane; ll < P.ncld; ll += LS) {
        int g = C0 + ll;
        const int leaf = ll & 31;
        if (!w.on(g)) continue;
        const KT k = kget(w, g, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < nspec) a.add_src(s, k * w.vk(s, g), leaf);
        }
        if (diag) {
          const KT kw = k * w.vk(iwa, g);
          a.add_dg(3, kw, leaf);
          double dd = D3 + cube(w.dwet[g]);
          if (lt80 && num_gt(dd, cube(80.e-6))) a.add_dg(1, kw, leaf);
          if (lt50 && num_gt(dd, cube(50.e-6))) a.add_dg(2, kw, leaf);
          if (bin80) a.add_dg(4, kw, leaf);
          if (bin50) a.add_dg(5, kw, leaf);
        }
      }
    }
    if (P.lscgpp && kk > 0) {
      int ex80 = min(kk - 1, P.cnt80 - 1), ex50 = min(kk - 1, P.cnt50 - 1);
      for (int ll = lane; ll <= kk - 1; ll += LS) {
        int g = P0 + ll;
        const int leaf = ll & 31;
        if (!w.on(g)) continue;
        const KT k = kget(w, g, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < nspec) a.add_src(s, k * w.vk(s, g), leaf);
        }
        if (diag) {
          const KT kw = k * w.vk(iwa, g);
          double dd = D3 + cube(w.dwet[g]);
          if (ll <= ex80 && lt80 && num_gt(dd, cube(80.e-6))) a.add_dg(1, kw, leaf);
          if (ll <= ex50 && lt50 && num_gt(dd, cube(50.e-6))) a.add_dg(2, kw, leaf);
          if (ll <= ex80 && bin80) a.add_dg(4, kw, leaf);
          if (ll <= ex50 && bin50) a.add_dg(5, kw, leaf);
        }
      }
    }
    a.reduce(diag, lane);
    if (diag && lane == 0) {
      double nt = w.numc[tg];
      w.misc[M_DIAG + DG_APCOLL] += a.dg[6] * nt;
      w.misc[M_DIAG + DG_ACCR] += a.dg[3] * nt;
      w.misc[M_DIAG + DG_AUTOC80] += a.dg[1] * nt;
      w.misc[M_DIAG + DG_AUTOC50] += a.dg[2] * nt;
      w.misc[M_DIAG + DG_ACCR80] += a.dg[4] * nt;
      w.misc[M_DIAG + DG_ACCR50] += a.dg[5] * nt;
    }
    // precipSelfCoag (:1588-1611) with the pre-update state
    double kself = (P.lscgpp && kk < nprc - 1) ? (double)kget(w, tg, tg) : 0.;
    double nold = w.numc[tg];
    double vs_my[LS == 1 ? SALSA_NSV : 1];
    if constexpr (LS == 1) {
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++) vs_my[s] = s < nspec ? w.v(s, tg) * nold * kself : 0.;
    } else {
      vs_my[0] = (lane < nspec) ? w.v(lane, tg) * nold * kself : 0.;
    }
    num_slf = 0.5 * kself * nold * nold;
    apply_coag(P, w, tg, nspec, dt, a, lane);
    if (P.lscgpp && kk < nprc - 1) {
      // applyCoagPrecp (:584-599): self-coagulation products go to the next bin
      if constexpr (LS == 1) {
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s < nspec) {
            w.v(s, tg + 1) = w.v(s, tg + 1) + dt * vs_my[s];
            w.v(s, tg) = w.v(s, tg) - dt * vs_my[s];
          }
      } else if (lane < nspec) {
        w.v(lane, tg + 1) = w.v(lane, tg + 1) + dt * vs_my[0];
        w.v(lane, tg) = w.v(lane, tg) - dt * vs_my[0];
      }
      if (lane == 0) {
        w.numc[tg + 1] = w.numc[tg + 1] + dt * num_slf;
        w.numc[tg] = w.numc[tg] - dt * num_slf;
      }
      wsync<LS>();
      shadow_bin<KT>(P, w, tg, lane);
      shadow_bin<KT>(P, w, tg + 1, lane);
    }
  }
}

template <typename KT, bool SIP, int LS>
__device__ void coag_ice(const DevParams &P, const WS<KT, LS> &w, const double *tb, double dt, int lane) {
  const int nspec = P.nused, C0 = P.nbins, P0 = P.nbins + P.ncld, I0 = P.nliquid, nice = P.nice;
  const int iwa = P.iwa, irim = P.irim, ndry = P.ndry;
  (void)C0; (void)P0; (void)tb;
  for (int kk = 0; kk < nice; kk++) {
    int tg = I0 + kk;
    if (num_lt(w.numc[tg], K_PRLIM)) continue;
    TAccT<KT, LS> a;
    a.zero(w);
    double rf_t = rimefrac(P, w.numc[tg], w.v(iwa, tg), w.v(irim, tg), 4);
    if (P.lscgii) {
      // Eagg from the larger rime fraction of the pair (:758-769)
      for (int ll = kk + 1 + lane; ll <= nice - 1; ll += LS) {
        int g = I0 + ll;
        const int leaf = (ll - (kk + 1)) & 31;
        if (!w.on(g)) continue;
        double rf = fmax(rimefrac(P, w.numc[g], w.v(iwa, g), w.v(irim, g), 4), rf_t);
        double E = P.Eiagg_max - rf * (P.Eiagg_max - P.Eiagg_min);
        a.add_sink((KT)E * (KT)1.0 * kget(w, tg, g) * w.nk(g), leaf);
      }
      if (lane == 0) {
        double E = P.Eiagg_max - fmax(rf_t, rf_t) * (P.Eiagg_max - P.Eiagg_min);
        a.add_self((KT)E * (KT)0.5 * kget(w, tg, tg) * w.nk(tg), 0);
      }
    }
    if constexpr (SIP) {
      // the secondary-ice tallies of this target, in the reference's order: breakup
      // numbers (accumulateSink), frozen-drop masses (accumulateSourcePhaseChange),
      // breakup masses (accumulateSourceIce)
      if (P.st_secice && lane == 0) {
        const double *dmid = tb + TAB_DMID * P.nb_pad;
        if (P.lscgii && P.st_sipib) sip_iibr_numbers<KT>(P, w, kk, rf_t);
        if (P.lscgic) sip_drop_masses<KT>(P, w, dmid, kk, C0, P.ncld, P.ica_cur, P.fcb_cur, false);
        if (P.lscgip) sip_drop_masses<KT>(P, w, dmid, kk, P0, P.nprc, 0, P.nprc - 1, true);
        if (P.lscgii && kk > 0 && P.st_sipib) sip_iibr_masses<KT>(P, w, dmid, kk, rf_t);
      }
      wsync<LS>();
    }
    // accumulateSourcePhaseChange (:1244-1280)
    if (P.lscgia)
      for (int ll = P.in1a + lane; ll <= P.fn2b; ll += LS) {
        const int leaf = (ll - P.in1a) & 31;
        if (!w.on(ll)) continue;
        const KT k = kget(w, ll, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < ndry) a.add_src(s, k * w.vk(s, ll), leaf);
        }
        const KT xw = divc(k * w.vk(iwa, ll) * (KT)K_RHOWA, (KT)K_RHOIC);
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s == iwa) a.add_src(s, xw, leaf);
      }
    if (P.lscgic)
      for (int ll = lane; ll < P.ncld; ll += LS) {
        int g = C0 + ll;
        const int leaf = ll & 31;
        if (!w.on(g)) continue;
        const KT k = kget(w, g, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < ndry) a.add_src(s, k * w.vk(s, g), leaf);
        }
        const KT xw = divc(k * w.vk(iwa, g) * (KT)K_RHOWA, (KT)K_RHORI);
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s == irim) a.add_src(s, xw, leaf);
      }
    if (P.lscgip)
      for (int ll = lane; ll < P.nprc; ll += LS) {
        int g = P0 + ll;
        const int leaf = ll & 31;
        if (!w.on(g)) continue;
        const KT k = kget(w, g, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < ndry) a.add_src(s, k * w.vk(s, g), leaf);
        }
        const KT xw = divc(k * w.vk(iwa, g) * (KT)K_RHOWA, (KT)K_RHORI);
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s == irim) a.add_src(s, xw, leaf);
      }
    // accumulateSourceIce (:1385-1427)
    if (P.lscgii && kk > 0)
      for (int ll = lane; ll <= kk - 1; ll += LS) {
        int g = I0 + ll;
        const int leaf = ll & 31;
        if (!w.on(g)) continue;
        double rf = fmax(rimefrac(P, w.numc[g], w.v(iwa, g), w.v(irim, g), 4), rf_t);
        double E = P.Eiagg_max - rf * (P.Eiagg_max - P.Eiagg_min);
        const KT k = kget(w, g, tg);
        {
#pragma unroll
          for (int s = 0; s < SALSA_NSV; s++)
            if (s < nspec) a.add_src(s, (KT)E * k * w.vk(s, g), leaf);
        }
      }
    a.reduce(false, lane);
    // applyCoagIce (:605-651): every species slot with the same semi-implicit form
    apply_coag(P, w, tg, nspec, dt, a, lane);
    if (lane == 0) w.rhomean[tg] = rhomean_of(P, 4, w.numc[tg], w.v(iwa, tg), w.v(irim, tg));
    wsync<LS>();
  }
}

// the bins that reach their limit in some cell of the warp (all of them when the kernels come
// from the storage, whose pairs were populated at another step); all 32 lanes arrive together
template <typename KT>
__device__ __forceinline__ void mark_populated(const DevParams &P, WS<KT, 1> &w) {
  unsigned m[3] = {0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < 3; k++)
    for (int b = 32 * k; b < min(P.ntotal, 32 * k + 32); b++)
      if (P.kc_mode == 2 || num_ge(w.numc[b], nlim_of(phase_of(P, b)))) m[k] |= 1u << (b - 32 * k);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 3; k++) m[k] = __reduce_or_sync(0xffffffffu, m[k]);
  w.am0 = (unsigned long long)m[0] | ((unsigned long long)m[1] << 32);
  w.am1 = m[2];
}

template <typename KT, bool SIP, int LS>
__device__ __forceinline__ void coagulation(const DevParams &P, WS<KT, LS> &w, const double *tb, double dt, double T, double pres,
                            bool diag, long long cell, int lane) {
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  if constexpr (LS == 1) mark_populated(P, w);
  // updateDiameter("all") on every bin (:146-152) and rhomean of the kernel categories
  for (int b = lane; b < P.ntotal; b += LS) {
    updateDiameterAll(P, w, dmid, b);
    int ph = phase_of(P, b);
    bool inker = (ph == 1 && (P.lscgaa || P.lscgca || P.lscgpa || P.lscgia)) ||
                 (ph == 2 && (P.lscgcc || P.lscgca || P.lscgpc || P.lscgic)) ||
                 (ph == 3 && (P.lscgpp || P.lscgpa || P.lscgpc || P.lscgip)) ||
                 (ph == 4 && (P.lscgii || P.lscgia || P.lscgic || P.lscgip));
    if (inker) w.rhomean[b] = rhomean_of(P, ph, w.numc[b], w.v(P.iwa, b), w.v(P.irim, b));
  }
  wsync<LS>();
#ifdef SALSA_STAGE_TIMERS
  long long t_k0 = clock64();
#endif
  if (P.kc_mode == 2) {
    // fetch_coag (mo_salsa_driver.f90:297-298, 676-697): the kernels stored at the last
    // update step of the low-frequency kernel mode
    const KT *src = static_cast<const KT *>(P.kcache) + (P.kc_base + cell) * (long long)P.kc_stride;
    for (int e = lane; e < P.kc_stride; e += LS) w.K[e] = src[e];
    wsync<LS>();
  } else {
    build_kernels<KT>(P, w, T, pres, lane);
    if (P.kc_mode == 1) {   // store_coag (:421-423, 655-674); the kernels do not change later in the step
      KT *dst = static_cast<KT *>(P.kcache) + (P.kc_base + cell) * (long long)P.kc_stride;
      for (int e = lane; e < P.kc_stride; e += LS) dst[e] = w.K[e];
    }
  }
#ifdef SALSA_STAGE_TIMERS
  if ((threadIdx.x & 31) == 0 && P.stage_clocks) atomicAdd(P.stage_clocks + 8, (unsigned long long)(clock64() - t_k0));
#endif
  bool any_aero = P.lscgaa || P.lscgca || P.lscgpa || P.lscgia;
  bool any_cloud = P.lscgcc || P.lscgca || P.lscgpc || P.lscgic;
  bool any_precp = P.lscgpp || P.lscgpa || P.lscgpc || P.lscgip;
  bool any_ice = P.lscgii || P.lscgia || P.lscgic || P.lscgip;
  shadow_all<KT>(P, w, lane);
  if (any_ice && T < 273.15) coag_ice<KT, SIP>(P, w, tb, dt, lane);
  if (any_precp) coag_precp<KT, SIP>(P, w, tb, dt, diag, lane);
  if (any_aero) coag_aero<KT>(P, w, tb, dt, lane);
  if (any_cloud) coag_cloud<KT, SIP>(P, w, tb, dt, diag, lane);
  bool neg = false;
  for (int b = lane; b < P.ntotal; b += LS) {
    const double n = w.numc[b];
    if (num_gt(-n, 1.e-6)) neg = true;
    w.numc[b] = pos_part(n);
    for (int s = 0; s < P.nused; s++) w.v(s, b) = pos_part(w.v(s, b));
  }
  if (wany<LS>(neg) && lane == 0) w.misc[M_FLAGS + F_NEG] = 1.;
  wsync<LS>();
}


// ----------------------------------------------------------------------------------------
// Water uptake: mo_salsa_properties.f90:73-380 equilibration.
// Regime 1a carries the Kelvin factor zke from bin to bin (:170, set once before
// the bin loop), so its bins are visited in order; regime 2 (init) restarts zke per
// bin and runs lane-parallel.
// ----------------------------------------------------------------------------------------
template <typename KT, int LS>
__device__ __forceinline__ double zvolc_of(const DevParams &P, const WS<KT, LS> &w, int which, int b) {
  const int ix[7] = {P.ix_so4, P.ix_oc, P.ix_bc, P.ix_du, P.ix_ss, P.ix_no, P.ix_nh};
  int d = ix[which];
  return (d >= 0 && which < 5) ? w.v(d, b) : 0.;   // only the first five are copied (:148)
}

template <typename KT, int LS>
__device__ double equil_iterate(const DevParams &P, const WS<KT, LS> &w, int b, double zrh, double T, double &zke,
                                double tol, bool regime2, double &zdwet_out, double &zcore_out, int &nonconv) {
  double numc = w.numc[b];
  double zv0 = zvolc_of(P, w, 0, b), zv1 = zvolc_of(P, w, 1, b), zv4 = zvolc_of(P, w, 4, b);
  double zvp[7];
  for (int i = 0; i < 7; i++) zvp[i] = ddiv(zvolc_of(P, w, i, b), numc);
  double zcore = regime2 ? (zvp[0] + zvp[1] + zvp[2] + zvp[3] + zvp[4]) : (zvp[0] + zvp[1]);
  double zdwet = w.dwet[b];
  double zdold = 1.;
  double zlwc = 0.;
  int count = 0;
  const double rhosu_msu = 1830. / 98.08e-3, rhooc_moc = 1400. / 150.e-3, rhoss_mss = 2165. / 58.44e-3;
  while (fabs(ddiv(zdwet, zdold) - 1.) > tol) {
    zdold = fmax(zdwet, 1.e-20);
    double zaw = ddiv(zrh, zke);
    double a2 = zaw * zaw, a3 = a2 * zaw, a4 = a2 * a2;
    double bm1 = +1.1065495e+2 - 3.6759197e+2 * zaw + 5.0462934e+2 * a2 - 3.1543839e+2 * a3 + 6.770824e+1 * a4;
    double bm2 = drcp(zaw * K_MWA) - 1. / K_MWA;
    // nitric acid molality only multiplies a zero NO volume (NO not copied, :148) -> its term is zero
    zlwc = ddiv(zv0 * rhosu_msu, bm1) + ddiv(K_EPSOC * zv1 * rhooc_moc, bm2);
    if (regime2) {
      double bm5 = +5.875248e+1 - 1.8781997e+2 * zaw + 2.7211377e+2 * a2 - 1.8458287e+2 * a3 + 4.153689e+1 * a4;
      zlwc += ddiv(zv4 * rhoss_mss, bm5);
    }
    zdwet = dcbrt(divc(divc(ddiv(zlwc, numc), K_RHOWA), K_PI6) + divc(zvp[5] + zvp[6], K_PI6) + divc(zcore, K_PI6));
    zke = dexp(ddiv(2. * K_SURFW0 * K_MVWA, K_BOLTZ * T * zdwet));
    count++;
    if (count > 100) { nonconv = 1; break; }
  }
  zdwet_out = zdwet;
  zcore_out = zcore;
  return zlwc;
}

// State of one fixed-point solve of equil_iterate, advanced one iteration at a time so
// that the regime-1a chain (sequential: zke carries from bin to bin) runs on its own lane
// next to the independent regime-2 solves.  The iteration carries 1/zke = exp(-c/dwet)
// rather than zke, so that zaw = zrh/zke is a product.
struct EqJob {
  int kk, count;
  bool r2;
  double tol, zrh, izke, numc, zv0, zv1, zv4, zvp56, zcore, zdwet, zdold, zlwc;
  double q0, q1, q4, ppc, rinv;   // per-bin invariants of the iteration, computed once
};

template <typename KT, int LS>
__device__ __forceinline__ void eq_load(const DevParams &P, const WS<KT, LS> &w, int b, EqJob &j) {
  j.kk = b;
  j.count = 0;
  j.numc = w.numc[b];
  j.zv0 = zvolc_of(P, w, 0, b); j.zv1 = zvolc_of(P, w, 1, b); j.zv4 = zvolc_of(P, w, 4, b);
  double zvp[7];
  for (int i = 0; i < 7; i++) zvp[i] = ddiv(zvolc_of(P, w, i, b), j.numc);
  j.zcore = j.r2 ? (zvp[0] + zvp[1] + zvp[2] + zvp[3] + zvp[4]) : (zvp[0] + zvp[1]);
  j.zvp56 = zvp[5] + zvp[6];
  {
    const double rhosu_msu = 1830. / 98.08e-3, rhooc_moc = 1400. / 150.e-3, rhoss_mss = 2165. / 58.44e-3;
    j.q0 = j.zv0 * rhosu_msu;
    j.q1 = K_EPSOC * j.zv1 * rhooc_moc * K_MWA;
    j.q4 = j.zv4 * rhoss_mss;
    j.ppc = divc(j.zvp56, K_PI6) + divc(j.zcore, K_PI6);
    j.rinv = drcp(j.numc * (K_RHOWA * K_PI6));   // zlwc / numc / rhowa / pi6 as one product
  }
  j.zdwet = w.dwet[b];
  j.zdold = 1.;
  j.zlwc = 0.;
}

// one pass of the equil_iterate loop body (mo_salsa_properties.f90:196-230, :305-340) in 32
// FP64 operations: one division for the water content and one for the Kelvin exponent.  The
// molality quotients share one denominator, with 1/bm2 = aw M/(1 - aw) for
// bm2 = 1/(aw M) - 1/M; the factor 1/(numc rhowa pi6) and c = 2 sigma v_w / kT are computed
// once, and 1/zke = exp(-c/dwet) is carried.  The values move by an ulp or so against the
// reference's operation order.  UNI: the lanes are all in one regime (lane form); the warp
// form runs regime 1a as regime 2 with bm5 = 1 and no sea salt, on the same code.
template <bool UNI>
__device__ __forceinline__ void eq_step(EqJob &j, double ckt) {
  j.zdold = max_pos(1.e-20, j.zdwet);
  const double zaw = j.zrh * j.izke;
  const double bm1 = fma(fma(fma(fma(6.770824e+1, zaw, -3.1543839e+2), zaw, 5.0462934e+2), zaw, -3.6759197e+2), zaw,
                         1.1065495e+2);
  const double b2 = 1. - zaw;
  if (UNI && !j.r2) {
    j.zlwc = ddiv(fma(j.q1 * zaw, bm1, j.q0 * b2), bm1 * b2);
  } else {
    double bm5 = fma(fma(fma(fma(4.153689e+1, zaw, -1.8458287e+2), zaw, 2.7211377e+2), zaw, -1.8781997e+2), zaw,
                     5.875248e+1);
    if (!UNI) bm5 = j.r2 ? bm5 : 1.;
    const double q4 = (UNI || j.r2) ? j.q4 : 0., b12 = bm1 * b2;
    j.zlwc = ddiv(fma(q4, b12, fma(j.q1 * zaw, bm1 * bm5, j.q0 * (b2 * bm5))), b12 * bm5);
  }
  j.zdwet = dcbrt(fma(j.zlwc, j.rinv, j.ppc));
  j.izke = dexp(-(ddiv(ckt, j.zdwet)));
  j.count++;
}

// ---- the mixed form's water-uptake iteration in FP32 ----
// The ZSR molality polynomials in aw (mo_salsa_properties.f90:202-227, 311-341) cancel
// to a few parts in 1e4 of their terms as aw -> 1, so the float iteration evaluates them
// in u = 1 - aw with the Taylor-shifted coefficients below, and carries
// em = 1 - 1/zke = -expm1(-c/dwet), so that u = (1 - zrh) + zrh em keeps its relative
// accuracy.  The callers clamp zrh to <= 0.98, so u >= 0.02 and the shifted polynomials
// do not cancel.  Regime 2 (tolerance 1e-12) then takes two FP64 passes from the float
// result; regime 1a (tolerance 1e-2) ends in float.
#define ZSR_D0(a0, a1, a2, a3, a4) ((a0) + (a1) + (a2) + (a3) + (a4))
#define ZSR_D1(a0, a1, a2, a3, a4) (-((a1) + 2. * (a2) + 3. * (a3) + 4. * (a4)))
#define ZSR_D2(a0, a1, a2, a3, a4) ((a2) + 3. * (a3) + 6. * (a4))
#define ZSR_D3(a0, a1, a2, a3, a4) (-((a3) + 4. * (a4)))
#define ZSR_D4(a0, a1, a2, a3, a4) (a4)
#define ZSR_SHIFTED(u, ...)                                                                          \
  fmaf(fmaf(fmaf(fmaf((float)ZSR_D4(__VA_ARGS__), u, (float)ZSR_D3(__VA_ARGS__)), u,                 \
                 (float)ZSR_D2(__VA_ARGS__)), u, (float)ZSR_D1(__VA_ARGS__)), u, (float)ZSR_D0(__VA_ARGS__))
// bm1 (sulphate, :211-212) and bm5 (sea salt, :318-319) in u = 1 - aw
__device__ __forceinline__ float zsr1_u(float u) {
  return ZSR_SHIFTED(u, +1.1065495e+2, -3.6759197e+2, +5.0462934e+2, -3.1543839e+2, +6.770824e+1);
}
__device__ __forceinline__ float zsr5_u(float u) {
  return ZSR_SHIFTED(u, +5.875248e+1, -1.8781997e+2, +2.7211377e+2, -1.8458287e+2, +4.153689e+1);
}

struct EqJobF {
  int kk, count;
  bool r2;
  float tol, zrh, omrh, em, zdwet, zdold, zlwc;
  float q0, q1, q4, p56, pc, rinv;
};

template <typename KT, int LS>
__device__ __forceinline__ void eq_load_f(const DevParams &P, const WS<KT, LS> &w, int b, EqJobF &j) {
  j.kk = b;
  j.count = 0;
  const float numc = (float)w.numc[b], in = ddiv(1.f, numc);
  float zv[7];
  for (int i = 0; i < 7; i++) zv[i] = (float)zvolc_of(P, w, i, b);
  const float zcore = j.r2 ? (zv[0] + zv[1] + zv[2] + zv[3] + zv[4]) * in : (zv[0] + zv[1]) * in;
  const float rhosu_msu = (float)(1830. / 98.08e-3), rhooc_moc = (float)(1400. / 150.e-3),
              rhoss_mss = (float)(2165. / 58.44e-3), ipi6 = (float)(1. / K_PI6);
  j.q0 = zv[0] * rhosu_msu;
  j.q1 = (float)K_EPSOC * zv[1] * rhooc_moc;
  j.q4 = zv[4] * rhoss_mss;
  j.p56 = (zv[5] + zv[6]) * in * ipi6;
  j.pc = zcore * ipi6;
  j.rinv = in * (float)(1. / (K_RHOWA * K_PI6));
  j.zdwet = (float)w.dwet[b];
  j.zdold = 1.f;
  j.zlwc = 0.f;
}

__device__ __forceinline__ void eq_step_f(EqJobF &j, float ckt) {
  j.zdold = fmaxf(j.zdwet, 1.e-20f);
  const float u = fmaf(j.zrh, j.em, j.omrh);   // 1 - zrh / zke
  const float zaw = 1.f - u;
  const float bm1 = zsr1_u(u);
  const float bm2 = ddiv(u, zaw * (float)K_MWA);   // 1/(aw M) - 1/M
  const float bm5 = j.r2 ? zsr5_u(u) : 1.f;
  const float q4 = j.r2 ? j.q4 : 0.f;
  const float zlwc = ddiv(fmaf(q4, bm1 * bm2, fmaf(j.q1, bm1 * bm5, j.q0 * (bm2 * bm5))), bm1 * bm2 * bm5);
  j.zlwc = zlwc;
  j.zdwet = cbrtf(fmaf(zlwc, j.rinv, j.p56) + j.pc);
  j.em = -expm1f(-(ddiv(ckt, j.zdwet)));
  j.count++;
}

// next regime-1a bin after b with numc > nlim; empty bins take dmid when initialising
template <typename KT, int LS>
__device__ __forceinline__ int eq_next_1a(const DevParams &P, const WS<KT, LS> &w, const double *dmid, int b, bool init) {
  for (int k = b + 1; k <= P.fn1a; k++) {
    if (num_gt(w.numc[k], K_NLIM)) return k;
    if (init) w.dwet[k] = dmid[k];
  }
  return -1;
}

template <typename KT, int LS>
__device__ void equilibration(const DevParams &P, const WS<KT, LS> &w, const double *tb, double prh, double T, bool init,
                              int lane) {
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  int nonconv = 0;
  const int n2 = init ? P.fn2b - P.in2a + 1 : 0;
  const double ckt = ddiv(2. * K_SURFW0 * K_MVWA, K_BOLTZ * T);
  if constexpr (LS == 1) {
    // the regime-1a bins in order (1/zke carries from bin to bin), then the regime-2 bins
    const double zrh1 = fmin(fmax(prh, 0.05), 0.98), zrh2 = fmin(fmax(prh, 0.37), 0.98);
    if constexpr (sizeof(KT) == 4) {
      const float cktf = (float)ckt;
      EqJobF j;
      j.em = (float)(1. - 1. / 1.001);
      for (int k = eq_next_1a(P, w, dmid, P.in1a - 1, init); k >= 0; k = eq_next_1a(P, w, dmid, k, init)) {
        j.r2 = false; j.tol = 1.e-2f; j.zrh = (float)zrh1; j.omrh = (float)(1. - zrh1);
        eq_load_f(P, w, k, j);
        while (fabsf(j.zdwet - j.zdold) > j.tol * j.zdold) {
          eq_step_f(j, cktf);
          if (j.count > 100) { nonconv = 1; break; }
        }
        w.v(P.iwa, k) = (double)j.zlwc * (1. / K_RHOWA);
        if (init) w.dwet[k] = (double)j.zdwet;
      }
      for (int k = P.in2a; k < P.in2a + n2; k++) {
        if (!num_gt(w.numc[k], K_NLIM)) { w.dwet[k] = dmid[k]; continue; }
        j.r2 = true; j.tol = 1.e-6f; j.zrh = (float)zrh2; j.omrh = (float)(1. - zrh2); j.em = (float)(1. - 1. / 1.02);
        eq_load_f(P, w, k, j);
        while (fabsf(j.zdwet - j.zdold) > j.tol * j.zdold) {
          eq_step_f(j, cktf);
          if (j.count > 100) { nonconv = 1; break; }
        }
        EqJob d;   // two FP64 passes from the float result
        d.r2 = true; d.tol = 1.e-12; d.zrh = zrh2;
        eq_load(P, w, k, d);
        d.zdwet = (double)j.zdwet;
        d.izke = dexp(-(ddiv(ckt, d.zdwet)));
        eq_step<true>(d, ckt);
        eq_step<true>(d, ckt);
        w.v(P.iwa, k) = divc(d.zlwc, K_RHOWA);
        w.dwet[k] = d.zdwet;
      }
    } else {
      EqJob j;
      j.izke = 1. / 1.001;
      for (int k = eq_next_1a(P, w, dmid, P.in1a - 1, init); k >= 0; k = eq_next_1a(P, w, dmid, k, init)) {
        j.r2 = false; j.tol = 1.e-2; j.zrh = zrh1;
        eq_load(P, w, k, j);
        while (fabs(j.zdwet - j.zdold) > j.tol * j.zdold) {
          eq_step<true>(j, ckt);
          if (j.count > 100) { nonconv = 1; break; }
        }
        w.v(P.iwa, k) = divc(j.zlwc, K_RHOWA);
        if (init) w.dwet[k] = j.zdwet;
      }
      for (int k = P.in2a; k < P.in2a + n2; k++) {
        if (!num_gt(w.numc[k], K_NLIM)) { w.dwet[k] = dmid[k]; continue; }
        j.r2 = true; j.tol = 1.e-12; j.zrh = zrh2; j.izke = 1. / 1.02;
        eq_load(P, w, k, j);
        while (fabs(j.zdwet - j.zdold) > j.tol * j.zdold) {
          eq_step<true>(j, ckt);
          if (j.count > 100) { nonconv = 1; break; }
        }
        w.v(P.iwa, k) = divc(j.zlwc, K_RHOWA);
        w.dwet[k] = j.zdwet;
      }
    }
  } else if (n2 <= 31 && sizeof(KT) == 4) {
    // the mixed form: lane 31 runs the regime-1a chain, lanes 0..n2-1 the regime-2 bins,
    // all in float; then the regime-2 lanes take two FP64 passes from the float result
    EqJobF j;
    j.kk = -1;
    const float cktf = (float)ckt;
    if (lane == 31) {
      const double zrh = fmin(fmax(prh, 0.05), 0.98);
      j.r2 = false; j.tol = 1.e-2f; j.zrh = (float)zrh; j.omrh = (float)(1. - zrh); j.em = (float)(1. - 1. / 1.001);
      int k = eq_next_1a(P, w, dmid, P.in1a - 1, init);
      if (k >= 0) eq_load_f(P, w, k, j);
    } else if (lane < n2) {
      int k = P.in2a + lane;
      if (w.numc[k] > K_NLIM) {
        const double zrh = fmin(fmax(prh, 0.37), 0.98);
        j.r2 = true; j.tol = 1.e-6f; j.zrh = (float)zrh; j.omrh = (float)(1. - zrh); j.em = (float)(1. - 1. / 1.02);
        eq_load_f(P, w, k, j);
      } else {
        w.dwet[k] = dmid[k];
      }
    }
    int r2k = -1;   // the regime-2 bin a lane polishes
    while (__any_sync(0xffffffffu, j.kk >= 0)) {
      if (j.kk >= 0) {
        bool go = fabsf(j.zdwet - j.zdold) > j.tol * j.zdold;
        if (go) {
          eq_step_f(j, cktf);
          if (j.count > 100) { nonconv = 1; go = false; }
        }
        if (!go) {
          if (j.r2) {
            r2k = j.kk;
            j.kk = -1;
          } else {
            w.v(P.iwa, j.kk) = (double)j.zlwc * (1. / K_RHOWA);
            if (init) w.dwet[j.kk] = (double)j.zdwet;
            int k = eq_next_1a(P, w, dmid, j.kk, init);
            if (k >= 0) eq_load_f(P, w, k, j);
            else j.kk = -1;
          }
        }
      }
    }
    if (__any_sync(0xffffffffu, r2k >= 0)) {
      EqJob d;
      if (r2k >= 0) {
        d.r2 = true; d.tol = 1.e-12; d.zrh = fmin(fmax(prh, 0.37), 0.98);
        eq_load(P, w, r2k, d);
        d.zdwet = (double)j.zdwet;
        d.izke = dexp(-(ddiv(ckt, d.zdwet)));
        eq_step<false>(d, ckt);
        eq_step<false>(d, ckt);
        w.v(P.iwa, r2k) = divc(d.zlwc, K_RHOWA);
        w.dwet[r2k] = d.zdwet;
      }
    }
    wsync<LS>();
  } else if (n2 <= 31) {
    // lane 31: the regime-1a chain in bin order; lanes 0..n2-1: regime-2 bins
    EqJob j;
    j.kk = -1;
    if (lane == 31) {
      j.r2 = false; j.tol = 1.e-2; j.zrh = fmin(fmax(prh, 0.05), 0.98); j.izke = 1. / 1.001;
      int k = eq_next_1a(P, w, dmid, P.in1a - 1, init);
      if (k >= 0) eq_load(P, w, k, j);
    } else if (lane < n2) {
      int k = P.in2a + lane;
      if (w.numc[k] > K_NLIM) {
        j.r2 = true; j.tol = 1.e-12; j.zrh = fmin(fmax(prh, 0.37), 0.98); j.izke = 1. / 1.02;
        eq_load(P, w, k, j);
      } else {
        w.dwet[k] = dmid[k];
      }
    }
    while (__any_sync(0xffffffffu, j.kk >= 0)) {
      if (j.kk >= 0) {
        bool go = fabs(j.zdwet - j.zdold) > j.tol * j.zdold;   // |zdwet/zdold - 1| > tol, zdold > 0
        if (go) {
          eq_step<false>(j, ckt);
          if (j.count > 100) { nonconv = 1; go = false; }
        }
        if (!go) {
          w.v(P.iwa, j.kk) = divc(j.zlwc, K_RHOWA);
          if (init) w.dwet[j.kk] = j.zdwet;
          int k = j.r2 ? -1 : eq_next_1a(P, w, dmid, j.kk, init);
          if (k >= 0) eq_load(P, w, k, j);
          else j.kk = -1;
        }
      }
    }
    wsync<LS>();
  } else {
    // regime 1a, in bin order (all lanes run it; lane 0 writes)
    double zke = 1.001;
    for (int kk = P.in1a; kk <= P.fn1a; kk++) {
      if (w.numc[kk] > K_NLIM) {
        double zrh = fmin(fmax(prh, 0.05), 0.98);
        double zd, zc;
        double zlwc = equil_iterate<KT>(P, w, kk, zrh, T, zke, 1.e-2, false, zd, zc, nonconv);
        wsync<LS>();
        if (lane == 0) {
          w.v(P.iwa, kk) = divc(zlwc, K_RHOWA);
          if (init) w.dwet[kk] = zd;
        }
      } else if (init && lane == 0) {
        w.dwet[kk] = dmid[kk];
      }
      wsync<LS>();
    }
    for (int kk = P.in2a + lane; kk <= P.fn2b; kk += LS) {
      if (w.numc[kk] > K_NLIM) {
        double zke = 1.02;
        double zrh = fmin(fmax(prh, 0.37), 0.98);
        double zd, zc;
        double zlwc = equil_iterate<KT>(P, w, kk, zrh, T, zke, 1.e-12, true, zd, zc, nonconv);
        w.v(P.iwa, kk) = divc(zlwc, K_RHOWA);
        w.dwet[kk] = zd;
      } else {
        w.dwet[kk] = dmid[kk];
      }
    }
  }
  if (wany<LS>(nonconv) && lane == 0) w.misc[M_FLAGS + F_EQUIL] = 1.;
  wsync<LS>();
}

// ----------------------------------------------------------------------------------------
// Condensation of water: mo_salsa_dynamics.f90:691-1125 gpparth2o, :1127-1157 acth2o.
// Scratch (per global bin): 0 kelvin 1 cwsurf 2 mt 3 wsat 4 cw (current) 5 zns (solute
// moles in acth2o) 6 orgic 7 orgri
// ----------------------------------------------------------------------------------------
template <typename KT, int LS>
__device__ __forceinline__ double solute_moles(const DevParams &P, const WS<KT, LS> &w, int b, double kappa) {
  double zns = 0.;
  if (P.has_kappa) {
    double vs = 0.;
    for (int nn = 0; nn < P.ndry; nn++) if (P.diss[nn] > 0.) vs += w.v(nn, b);
    zns = divc(kappa * vs * K_RHOWA, K_MWA);
  } else {
    for (int nn = 0; nn < P.ndry; nn++) zns = zns + ddiv(P.diss[nn] * w.v(nn, b) * P.rholiq[nn], P.MM[nn]);
  }
  return zns;
}
__device__ __forceinline__ double acth2o_w(double znw, double zns) {
  return max_pos(0.1, ddiv(znw, max_pos(K_EPS, znw + zns)));
}

// ----------------------------------------------------------------------------------------
// Gas condensation: mo_salsa_dynamics.f90:348-685 (condgas).  H2SO4 and the non- and
// semi-volatile organic vapours condense onto every bin in proportion to its
// Fuchs-Sutugin collision rate; the gas phase takes one implicit step.  zg holds the
// five gases in #/m3 (SO4, HNO3, NH3, OC non-volatile, OC semi-volatile) in shared memory.
// The smallest-bin nucleation terms (Jacobson 16.73, 16.75) read condgas's own zj3n3
// and zxocnv, which it declares locally and zeroes (:433-444): zn_vs_c stays 0, the
// collision rate of the smallest bin and the sinks gain 0/c.  zxsa, the H2SO4 fraction of
// the 3 nm clusters from nucleation, only multiplies that zero.  Collision rates go to
// scratch row 0, the non-volatile organic increments of the aerosol bins to row 1.
// ----------------------------------------------------------------------------------------
template <typename KT, int LS>
__device__ __forceinline__ void condgas(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double pres,
                                        double dt, const Ptr<double, LS> &gas, double zxsa, int lane) {
  double zg[5];
  for (int i = 0; i < 5; i++) zg[i] = gas[i];
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  const int ntot = P.ntotal, in1a = P.in1a, in2a = P.in2a, fn2b = P.fn2b;
  const int C0 = P.nbins, P0 = P.nbins + P.ncld, I0 = P.nliquid;
  const int ioc = P.ix_oc, iso4 = P.ix_so4;
  const auto cr = w.scr, dvoc = w.scr + w.NB;
  const double zvisc = ddiv(7.44523e-3 * dsqrt(cube(T)), 5093. * (T + 110.4));
  const double zdfvap = ddiv(5.1111e-10 * dpow(T, 1.75) * K_PSTAND, pres);
  const double zmfp = 3. * zdfvap * dsqrt(ddiv(K_PI * K_MSU, 8. * K_RG * T));
  for (int b = lane; b < ntot; b += LS) {
    // updateDiameter(limit=.TRUE., type="wet") (:446-448)
    const int ph = phase_of(P, b);
    const double n = w.numc[b];
    double dw = dmid[b];
    if (n > nlim_of(ph)) {
      double vs = 0.;
      for (int sp = 0; sp < P.nused; sp++) vs += w.v(sp, b);
      dw = dcbrt(divc(ddiv(vs, n), K_PI6));
    }
    dw = fmin(dw, dlim_of(ph));
    w.dwet[b] = dw;
    // collision rate of the vapour molecules with the bin's particles [1/s] (:461-541)
    double r = 0.;
    if (ph == 1) {
      const bool small = b <= in1a + 1;   // molecule size and particle diffusion count below 20 nm
      const double kn = small ? ddiv(2. * zmfp, dw + K_DSA) : ddiv(2. * zmfp, dw);
      const double beta = ddiv(kn + 1., 0.377 * kn + 1. + 4. / (3. * K_MASSACC) * (kn + sq(kn)));
      if (small) {
        const double zdfpart = ddiv(K_BOLTZ * T * beta, 3. * K_PI * zvisc * dw);
        if (n > K_NLIM) r = 2. * K_PI * (dw + K_DSA) * (zdfvap + zdfpart) * beta * n;
      } else if (n > K_NLIM) {
        r = 2. * K_PI * dw * zdfvap * beta * n;
      }
      dvoc[b] = 0.;
    } else {
      const double kn = ddiv(2. * zmfp, dw);
      double beta = 1. + ddiv(kn * (1.33 + (ddiv(0.71, kn))), 1. + (drcp(kn)));
      beta = drcp(beta);
      if (n > (ph == 2 ? K_NLIM : K_PRLIM)) r = 2. * K_PI * dw * zdfvap * beta * n;
    }
    cr[b] = r;
  }
  wsync<LS>();
  // condensation sinks, summed in bin order as Fortran's SUM (:545, :603-606)
  double sa = 0., sca = 0., spa = 0., sia = 0., sa2 = 0.;
  for (int k = in1a; k <= fn2b; k++) sa += cr[k];
  for (int k = 0; k < P.ncld; k++) sca += cr[C0 + k];
  for (int k = 0; k < P.nprc; k++) spa += cr[P0 + k];
  for (int k = 0; k < P.nice; k++) sia += cr[I0 + k];
  for (int k = in2a; k <= fn2b; k++) sa2 += cr[k];
  const double zcs_tot = sa + sca + spa + sia;
  const double zn_vs_c = 0.;
  // non-volatile organics onto every bin (:552-598)
  if (zg[3] > 1.e-10 && zcs_tot > 1.e-30 && ioc >= 0) {
    const double zcs = zcs_tot;
    const double cnew = ddiv(zg[3], 1. + dt * zcs);
    const double dv = zg[3] - cnew;
    zg[3] = cnew;
    for (int b = lane; b < ntot; b += LS) {
      const double inc = ddiv(cr[b], zcs) * K_MVOC * dv;
      if (b <= fn2b) dvoc[b] = inc;
      w.v(ioc, b) = w.v(ioc, b) + inc;
    }
  }
  // semi-volatile organics onto regimes 2a/2b and the hydrometeors (:603-632); the aerosol
  // update adds the whole increment row, which still holds the non-volatile increments
  const double zcs_ocsv = sa2 + sca + spa + sia;
  if (zg[4] > 1.e-10 && zcs_ocsv > 1.e-30 && ioc >= 0) {
    const double cnew = ddiv(zg[4], 1. + dt * zcs_ocsv);
    const double dv = zg[4] - cnew;
    zg[4] = cnew;
    for (int b = lane; b < ntot; b += LS) {
      if (b <= fn2b) {
        double d = dvoc[b];
        if (b >= in2a) d = d + ddiv(cr[b], zcs_ocsv) * K_MVOC * dv;
        w.v(ioc, b) = w.v(ioc, b) + d;
      } else {
        w.v(ioc, b) = w.v(ioc, b) + ddiv(cr[b], zcs_ocsv) * K_MVOC * dv;
      }
    }
  }
  // sulphuric acid onto every bin (:636-679)
  if (zg[0] > 1.e-10 && zcs_tot > 1.e-30 && iso4 >= 0) {
    const double zcs = zcs_tot;
    const double cnew = ddiv(zg[0], 1. + dt * zcs);
    const double dv = zg[0] - cnew;
    zg[0] = cnew;
    for (int b = lane; b < ntot; b += LS) {
      const double inc = ddiv(cr[b], zcs) * K_MVSU * dv;
      w.v(iso4, b) = w.v(iso4, b) + inc;
      if (b == in1a && zxsa > 0.) w.numc[b] = w.numc[b] + ddiv(divc(zn_vs_c * inc, K_MVSU), K_N3 * zxsa);
    }
  }
  wsync<LS>();
  for (int i = 0; i < 5; i++)
    if (LS == 1 || lane == i) gas[i] = zg[i];
  wsync<LS>();
}

// Two sums over the bins 0..n-1 in the order of the warp form's lane partial sums and
// butterfly (bins l, l + 32, .. of leaf l; leaves paired over 16, 8, 4, 2, 1 apart).  The
// explicit substeps take the vapour as a difference of such sums and magnify their rounding
// in the Aitken bins' water by orders of magnitude, so both forms round alike.  f(b, first,
// x, y) sets (first) or adds to the leaf's two partial sums.
template <typename F>
__device__ __forceinline__ void tree_sum2(int n, F f, double &X, double &Y) {
  double x0 = 0., y0 = 0., x1 = 0., y1 = 0., x2 = 0., y2 = 0.;
#pragma unroll 1
  for (int o = 0; o < 8; o++) {   // bits 0, 1, 2 of the leaf from the outside in
    const int l3 = (o >> 2) | (o & 2) | ((o & 1) << 2);
    double x3 = 0., y3 = 0.;
#pragma unroll
    for (int i3 = 0; i3 < 2; i3++) {
      double x4 = 0., y4 = 0.;
#pragma unroll
      for (int i4 = 0; i4 < 2; i4++) {
        double x = 0., y = 0.;
        bool first = true;
        for (int b = l3 + 8 * i3 + 16 * i4; b < n; b += 32) {
          f(b, first, x, y);
          first = false;
        }
        x4 = i4 ? x4 + x : x;
        y4 = i4 ? y4 + y : y;
      }
      x3 = i3 ? x3 + x4 : x4;
      y3 = i3 ? y3 + y4 : y4;
    }
    if (o & 1) { x2 += x3; y2 += y3; } else { x2 = x3; y2 = y3; }
    if (o & 1) {
      if (o & 2) { x1 += x2; y1 += y2; } else { x1 = x2; y1 = y2; }
      if (o & 2) {
        if (o & 4) { x0 += x1; y0 += y1; } else { x0 = x1; y0 = y1; }
      }
    }
  }
  X = x0;
  Y = y0;
}
// one sum in that order; f(b) is bin b's term
template <int LS, typename F>
__device__ __forceinline__ double bins_sum(int n, int lane, F f) {
  double X, Y;
  if constexpr (LS == 1) {
    tree_sum2(n, [&](int b, bool first, double &x, double &) { x = first ? f(b) : x + f(b); }, X, Y);
  } else {
    X = 0.;
    for (int b = lane; b < n; b += LS) X += f(b);
    X = warp_sum(X);
  }
  return X;
}

template <typename KT, int LS>
__device__ void gpparth2o(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double pres, double prs,
                          double prsi, double &prv, double dt, double kappa, bool diag, int lane) {
  const int nbins = P.nbins, ncld = P.ncld, nprc = P.nprc, nice = P.nice, ntot = P.ntotal;
  const int iwa = P.iwa, irim = P.irim, C0 = nbins, P0 = nbins + ncld, I0 = P.nliquid;
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  const double zrh = ddiv(prv, prs);
  // aerosol water before/after the equilibrium update
  double zaelwc1 = bins_sum<LS>(P.fn2b + 1, lane, [&](int b) { return w.v(iwa, b); }) * K_RHOWA;
  // The init-form call repeats the 1a update with identical inputs (dwet untouched by
  // the first call, zke restarted at 1.001), so running it alone gives the same state.
#ifdef SALSA_STAGE_TIMERS
  long long t_eq0 = clock64();
#endif
  if (zrh < 0.98 || !P.lscndh2oae) equilibration<KT>(P, w, tb, zrh, T, true, lane);
  else equilibration<KT>(P, w, tb, zrh, T, false, lane);
#ifdef SALSA_STAGE_TIMERS
  if ((threadIdx.x & 31) == 0 && P.stage_clocks) atomicAdd(P.stage_clocks + 10, (unsigned long long)(clock64() - t_eq0));
#endif
  double zaelwc2 = bins_sum<LS>(P.fn2b + 1, lane, [&](int b) { return w.v(iwa, b); }) * K_RHOWA;
  prv = prv - ddiv(zaelwc2 - zaelwc1, ddiv(pres * K_MAIR, K_RG * T));

  bool anycl = false, anypr = false, anyic = false, anyae = false;
  for (int b = lane; b < ntot; b += LS) {
    int ph = phase_of(P, b);
    double n = w.numc[b];
    const bool on = num_gt(n, nlim_of(ph));
    if (ph == 1) anyae |= on;
    else if (ph == 2) anycl |= on;
    else if (ph == 3) anypr |= on;
    else anyic |= on;
  }
  anyae = wany<LS>(anyae); anycl = wany<LS>(anycl); anypr = wany<LS>(anypr); anyic = wany<LS>(anyic);
  if (!((anycl || (anypr && P.lscndh2ocl)) || (anyic && P.lscndh2oic) || (anyae && zrh > 0.98 && P.lscndh2oae)))
    return;

  const double rhoair = ddiv(K_MAIR * pres, K_RG * T);
  double zdfh2o = (ddiv(5., 16. * K_AVOG * rhoair * 1.e-3 * sq(3.11e-8))) *
                  dsqrt(divc(K_RG * 1.e7 * T * K_MAIR * 1.e3 * (K_MWA + K_MAIR) * 1.e3, 2. * K_PI * K_MWA * 1.e3));
  zdfh2o = zdfh2o * 1.e-4;
  const double zmfph2o = 3. * zdfh2o * dsqrt(ddiv(K_PI * K_MWA, 8. * K_RG * T));
  const double zthcond = 0.023807 + 7.1128e-5 * (T - 273.16);
  const int NB = w.NB;
  const auto kel = w.sc(0), amt = w.sc(1), mt = w.sc(2), wsat = w.sc(3), cw = w.sc(4), zns = w.sc(5),
             orgic = w.sc(6), orgri = w.sc(7);
  (void)NB;
  const double sfl = divc(prs * rhoair, K_MWA), sfi = divc(prsi * rhoair, K_MWA);   // saturation, liquid and ice
  const double adt = 2.e-2;                                                         // substep [s]
  // diameters and densities (:819-822), then per-bin coefficients (:826-955).  The explicit
  // substeps magnify a last-bit difference of the diameter or the Kelvin term of the
  // smallest wet aerosol to as much as 1e-3 of the bin's water in a few cells in 1e5, so both
  // come from CUDA's functions (once per bin and step: no measurable time).
  for (int b = lane; b < ntot; b += LS) {
    updateDiameterAll<true>(P, w, dmid, b);
    int ph = phase_of(P, b);
    w.rhomean[b] = rhomean_of(P, ph, w.numc[b], w.v(iwa, b), w.v(irim, b));
    double n = w.numc[b];
    double k_ = 1., m = 0., ws = 0.;
    double ns_ = (ph <= 3) ? solute_moles(P, w, b, kappa) : 0.;
    bool act;
    if (ph == 1) act = zrh > 0.98 && P.lscndh2oae;
    else if (ph <= 3) act = P.lscndh2ocl;
    else act = P.lscndh2oic && T < 273.15;
    act = act && num_gt(n, nlim_of(ph));
    if (act) {
      if (ph <= 3) {
        double dwet = w.dwet[b];
        double znw = ddiv(w.v(iwa, b) * P.rholiq[iwa], P.MM[iwa]);
        double zact = acth2o_w(znw, ns_);
        k_ = ::exp(ddiv(4. * K_SURFW0 * K_MWA, K_RG * T * K_RHOWA * dwet));
        const double sf = sfl;
        ws = zact * k_;
        KT zknud = ddiv((KT)2. * (KT)zmfph2o, (KT)dwet);
        KT zbeta = ddiv(zknud + (KT)1., (KT)0.377 * zknud + (KT)1. + (KT)4. / ((KT)3. * (KT)1.) * (zknud + zknud * zknud));
        KT h1 = (KT)n * (KT)2. * (KT)K_PI * (KT)dwet * (KT)zdfh2o * zbeta;
        KT h2 = ddiv((KT)K_MWA * (KT)zdfh2o * (KT)K_ALV * (KT)ws * (KT)sf, (KT)zthcond * (KT)T);
        KT h3 = (ddiv((KT)K_ALV * (KT)K_MWA, (KT)K_RG * (KT)T)) - (KT)1.;
        m = (double)(ddiv(h1, h2 * h3 + (KT)1.));
      } else {
        double dwet = w.dnsp[b];
        double cap = 0.5 * dwet;
        k_ = ::exp(ddiv(4. * K_SURFI0 * K_MWA, K_RG * T * K_RHOWA * dwet));
        const double sf = sfi;
        ws = 1.0 * k_;
        KT zknud = ddiv((KT)2. * (KT)zmfph2o, (KT)dwet);
        KT zbeta = ddiv(zknud + (KT)1., (KT)0.377 * zknud + (KT)1. + (KT)4. / (KT)3. * (zknud + zknud * zknud));
        KT h1 = (KT)n * (KT)4. * (KT)K_PI * (KT)cap * (KT)zdfh2o * zbeta;
        KT h2 = ddiv((KT)K_MWA * (KT)zdfh2o * (KT)K_ALS * (KT)ws * (KT)sf, (KT)zthcond * (KT)T);
        KT h3 = (ddiv((KT)K_ALS * (KT)K_MWA, (KT)K_RG * (KT)T)) - (KT)1.;
        m = (double)(ddiv(h1, h2 * h3 + (KT)1.));
      }
    }
    kel[b] = k_; amt[b] = adt * m; mt[b] = m; wsat[b] = ws; zns[b] = ns_;
    if (ph <= 3) {
      cw[b] = divc(w.v(iwa, b) * K_RHOWA, K_MWA);
      orgic[b] = orgri[b] = 0.;
    } else {
      double c1 = divc(w.v(iwa, b) * K_RHOIC, K_MWA);
      cw[b] = c1 + divc(w.v(irim, b) * K_RHORI, K_MWA);
      orgic[b] = divc(w.v(iwa, b) * K_RHOIC, K_MWA);
      orgri[b] = divc(w.v(irim, b) * K_RHORI, K_MWA);
    }
  }
  wsync<LS>();
  // categories updated inside the substep loop (:1002-1031)
  bool upd_ae = false, upd_cl = false, upd_pr = false, upd_ic = false;
  {
    bool a = false, c = false, p = false, i = false;
    for (int b = lane; b < ntot; b += LS) {
      int ph = phase_of(P, b);
      double n = w.numc[b];
      const bool on = num_gt(n, nlim_of(ph));
      if (ph == 1) a |= on; else if (ph == 2) c |= on; else if (ph == 3) p |= on; else i |= on;
    }
    upd_ae = wany<LS>(a) && zrh > 0.98; upd_cl = wany<LS>(c); upd_pr = wany<LS>(p); upd_ic = wany<LS>(i);
  }
  double zcwc = divc(prv * rhoair, K_MWA);
  const double zcwtot = zcwc + bins_sum<LS>(ntot, lane, [&](int b) { return cw[b]; });
  // the substep sums skip regime 1a (nstr = in2a)
  const double mtot = bins_sum<LS>(ntot, lane, [&](int b) { return b >= P.in2a ? mt[b] : 0.; });
  double ttot = 0., zcwint = 0.;
  int counter = 0;
#ifdef SALSA_STAGE_TIMERS
  long long t_sub0 = clock64();
#endif
  // The sum of mt*wsat*surf that opens a substep is formed at the end of the previous
  // one and reduced together with its vapour sum: one paired butterfly of 5 adds
  // instead of two of 5.  Lane l holds bins l, l+32 (the same partial sums for both),
  // so the totals are those of two separate butterflies over those partial sums.
  double spsum;
  if constexpr (LS == 1) {
    double unused;
    tree_sum2(ntot, [&](int b, bool first, double &x, double &) {
      const double p = b >= P.in2a ? mt[b] * wsat[b] : 0., sf = b < I0 ? sfl : sfi;
      x = first ? p * sf : fma(p, sf, x);
    }, spsum, unused);
  } else {
    double sp = 0.;
    for (int b = lane; b < ntot; b += LS)
      if (b >= P.in2a) sp += mt[b] * wsat[b] * (b < I0 ? sfl : sfi);
    spsum = warp_sum(sp);
  }
  while (ttot < dt) {
    double zhlp1 = zcwc + adt * spsum;
    double zhlp2 = 1. + adt * mtot;
    zcwint = fmin(ddiv(zhlp1, zhlp2), zcwtot);
    struct SubBin { double c, am, ws, zn, ke, m; };
    auto load = [&](int b) -> SubBin { return {cw[b], amt[b], wsat[b], zns[b], kel[b], mt[b]}; };
    auto substep_bin = [&](int b, SubBin &q) {   // bin b through the substep: water q.c and activity q.ws
      const int ph = phase_of(P, b);
      const bool upd = (ph == 1) ? (upd_ae && b >= P.in2a) : (ph == 2 ? upd_cl : (ph == 3 ? upd_pr : upd_ic));
      if (upd) {
        const double x = q.am * (zcwint - q.ws * (ph <= 3 ? sfl : sfi));
        const double t = 1.e-1 * q.c;
        const double ci = q.c + (__double2hiint(t) >= 0 ? limit_pos(x, t) : fmin(fmax(x, -t), t));
        q.ws = (ph <= 3) ? acth2o_w(ci, q.zn) * q.ke : q.ke;
        wsat[b] = q.ws;
        q.c = pos_part(ci);
        cw[b] = q.c;
      }
    };
    if constexpr (LS == 1) {
      // tree_sum2's order, the next bin's values loaded ahead of the current bin's stores
      double cs = 0., sp = 0., x4 = 0., y4 = 0., x3 = 0., y3 = 0., x2 = 0., y2 = 0., x1 = 0., y1 = 0., x0 = 0., y0 = 0.;
      SubBin nx = load(0);
      int have = 0;   // the bin in nx
#pragma unroll 1
      for (int k = 0; k < 32; k++) {
        double x = 0., y = 0.;
        const int l = (int)(__brev((unsigned)k) >> 27), ln = (int)(__brev((unsigned)k + 1u) >> 27);
#pragma unroll 1
        for (int b = l; b < ntot; b += 32) {
          SubBin q = nx;
          if (have != b) q = load(b);   // layouts of fewer than 32 bins leave some leaves empty
          have = b + 32 < ntot ? b + 32 : ln;
          if (have < ntot) nx = load(have);
          // a bin without transfer coefficient keeps its water and adds nothing to the vapour sum
          const bool still = __double_as_longlong(q.am) == 0 && __double_as_longlong(q.c) >= 0;
          double ps = 0.;
          if (!still) {
            substep_bin(b, q);
            const double p = b >= P.in2a ? q.m * q.ws : 0., sf = b < I0 ? sfl : sfi;
            ps = b == l ? p * sf : fma(p, sf, y);
          } else if (b != l) {
            ps = y;
          }
          x = b == l ? q.c : x + q.c;
          y = ps;
        }
        if (!(k & 1)) { x4 = x; y4 = y; continue; }
        x = x4 + x; y = y4 + y;
        if (!(k & 2)) { x3 = x; y3 = y; continue; }
        x = x3 + x; y = y3 + y;
        if (!(k & 4)) { x2 = x; y2 = y; continue; }
        x = x2 + x; y = y2 + y;
        if (!(k & 8)) { x1 = x; y1 = y; continue; }
        x = x1 + x; y = y1 + y;
        if (!(k & 16)) { x0 = x; y0 = y; continue; }
        cs = x0 + x; sp = y0 + y;
      }
      zcwint = zcwtot - cs;
      spsum = sp;
    } else {
      double cs = 0., sp = 0.;
      for (int b = lane; b < ntot; b += LS) {
        SubBin q = load(b);
        substep_bin(b, q);
        cs += q.c;
        if (b >= P.in2a) sp += q.m * q.ws * (b < I0 ? sfl : sfi);
      }
      // lanes 0-15 reduce cs, lanes 16-31 reduce sp
      const bool hi = lane & 16;
      double v = (hi ? sp : cs) + __shfl_xor_sync(0xffffffffu, hi ? cs : sp, 16);
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      zcwint = zcwtot - __shfl_sync(0xffffffffu, v, 0);
      spsum = __shfl_sync(0xffffffffu, v, 16);
    }
    zcwc = zcwint;
    ttot = ttot + adt;
    counter++;
    if (counter >= 200000) break;   // the C-ABI bounds tstep, so this cap is never the exit path
  }
  if (counter > 100 && lane == 0) w.misc[M_FLAGS + F_COND] = 1.;
#ifdef SALSA_STAGE_TIMERS
  if ((threadIdx.x & 31) == 0 && P.stage_clocks) atomicAdd(P.stage_clocks + 9, (unsigned long long)(clock64() - t_sub0));
#endif
  prv = ddiv(zcwint * K_MWA, rhoair);
  // Cond_i diagnostic (:1086-1112): vrate(irim) is only assigned on sublimation and keeps
  // its previous value on later deposition bins; the sum follows the ice bins in order.
  double dci = 0.;
  if (diag && lane == 0) {
    double vr_last = 0.;
    for (int k = 0; k < nice; k++) {
      int b = I0 + k;
      double dvitot = cw[b] - (orgic[b] + orgri[b]);
      if (dvitot > 0.) {
        dci += divc(dvitot * K_MWA, K_RHOIC) * K_RHOIC + vr_last * K_RHORI;
      } else if (dvitot < 0.) {
        double f = (ddiv(cw[b], orgic[b] + orgri[b])) - 1.;
        vr_last = divc(f * orgri[b] * K_MWA, K_RHORI);
        dci += divc(f * orgic[b] * K_MWA, K_RHOIC) * K_RHOIC + vr_last * K_RHORI;
      }
    }
  }
  wsync<LS>();
  // write back and diagnostics (:1061-1117)
  double dca = 0., dcc = 0., dcp = 0.;
  for (int b = lane; b < ntot; b += LS) {
    int ph = phase_of(P, b);
    if (ph <= 3) {
      double nv = pos_part(divc(cw[b] * K_MWA, K_RHOWA));
      double d = nv - w.v(iwa, b);
      if (ph == 1) dca += d; else if (ph == 2) dcc += d; else dcp += d;
      w.v(iwa, b) = nv;
    } else {
      double dvitot = cw[b] - (orgic[b] + orgri[b]);
      if (dvitot > 0.) {
        double dv = divc(dvitot * K_MWA, K_RHOIC);
        w.v(iwa, b) = w.v(iwa, b) + dv;
      } else if (dvitot < 0.) {
        double f = (ddiv(cw[b], orgic[b] + orgri[b])) - 1.;
        double dvice = f * orgic[b], dvrime = f * orgri[b];
        w.v(iwa, b) = w.v(iwa, b) + divc(dvice * K_MWA, K_RHOIC);
        w.v(irim, b) = w.v(irim, b) + divc(dvrime * K_MWA, K_RHORI);
      }
    }
    if (num_gt(w.numc[b], nlim_of(ph))) w.rhomean[b] = rhomean_of(P, ph, w.numc[b], w.v(iwa, b), w.v(irim, b));
  }
  if (diag) {
    dca = wsum<LS>(dca); dcc = wsum<LS>(dcc); dcp = wsum<LS>(dcp);
    if (lane == 0) {
      w.misc[M_DIAG + DG_CONDA] += dca;
      w.misc[M_DIAG + DG_CONDC] += dcc;
      w.misc[M_DIAG + DG_CONDP] += dcp;
      w.misc[M_DIAG + DG_CONDI] += dci;
    }
  }
  wsync<LS>();
}

// ----------------------------------------------------------------------------------------
// Interstitial activation: mo_salsa_cloud.f90:859-1195 actInterst (+ intgN/intgV :1381-1398)
// Lanes own cloud bins; the transfer touches only the parallel aerosol bin.
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ double intgN(double k, double c, double lo, double hi) {
  return 0.5 * k * fmax(hi * hi - lo * lo, 0.) + c * fmax(hi - lo, 0.);
}
__device__ __forceinline__ double intgV(double k, double c, double lo, double hi) {
  return (1. / 3.) * k * fmax(cube(hi) - cube(lo), 0.) + 0.5 * c * fmax(hi * hi - lo * lo, 0.);
}

// ----------------------------------------------------------------------------------------
// Cloud-base activation: mo_salsa_cloud.f90:161-375 (ActCloudBase: Abdul-Razzak & Ghan,
// sectional form) and :1199-1378 (activate3).  The updraft sets the parcel's maximum
// supersaturation, which gives a critical diameter per bin; the activated number and
// volume of each cloud bin are integrals of piecewise-linear number densities in dry
// volume above the critical volume.  The state does not change: the results go to the
// activated-droplet outputs (raw rows, per kg of air).  One lane per aerosol bin, then
// one lane per cloud bin; sums run in bin order on every lane.
// ----------------------------------------------------------------------------------------
template <typename KT, int LS>
__device__ __forceinline__ void act_cloudbase(const DevParams &P, const WS<KT, LS> &w, const double *tb, double pres,
                                              double T, double wvel, double dn, const Ptr<double, LS> &raw, int lane) {
  const int in1a = P.in1a, fn2a = P.fn2a, in2b = P.in2b, fn2b = P.fn2b, ndry = P.ndry, nwet = P.nwet;
  const int iwa = P.iwa, ncld = P.ncld;
  const double *dmid = tb + TAB_DMID * P.nb_pad, *vlo = tb + TAB_VLO * P.nb_pad, *vhi = tb + TAB_VHI * P.nb_pad;
  const double *vrlo = tb + TAB_VRLO * P.nb_pad, *vrhi = tb + TAB_VRHI * P.nb_pad;
  const auto ns = w.sc(0), zdcrit = w.sc(1), zdcrlo = w.sc(2), zdcrhi = w.sc(3), frac = w.sc(4), term = w.sc(5);
  const double bb = 6. * K_MWA / (K_PI * K_RHOWA);   // Raoult term per mole of solute [m3]
  // getSolute (:116-157): moles of dissolved solute per particle
  for (int k = lane; k <= fn2b; k += LS) {
    double n_ = 0.;
    if (w.numc[k] > K_NLIM) {
      for (int nn = 0; nn < ndry; nn++) n_ = n_ + ddiv(P.diss[nn] * w.v(nn, k) * P.rholiq[nn], P.MM[nn]);
      n_ = ddiv(n_, w.numc[k]);
    }
    ns[k] = n_;
    frac[k] = zdcrit[k] = zdcrlo[k] = zdcrhi[k] = 0.;
  }
  wsync<LS>();
  int bcrita = fn2a;
  double zdcstar = 0.;
  if (wvel > 0.) {
    const double aa = ddiv(4. * K_MWA * K_SURFW0, K_RG * K_RHOWA * T);   // Kelvin term [m]
    const double x = divc(4. * cube(aa), 27. * bb);
    for (int k = in1a + lane; k <= fn2b; k += LS) {
      const double scrit = dexp(dsqrt(ddiv(x, fmax(K_EPS, ns[k])))) - 1.;
      term[k] = ddiv(w.numc[k], dpow(scrit, 2. / 3.));
    }
    wsync<LS>();
    double ntot = 0., sum1 = 0.;   // part 3, eq. (8)
    for (int k = in1a; k <= fn2b; k++) ntot += w.numc[k];
    for (int k = in1a; k <= fn2b; k++) sum1 += term[k];
    if (!(ntot < K_NLIM)) {
      const double V = wvel;
      const double L = 2.501e6 - 2370. * (T - 273.15);
      const double a1 = 1. - (ddiv(373.15, T));
      const double ps = 101325. * dexp(13.3185 * a1 - 1.976 * sq(a1) - 0.6445 * cube(a1) - 0.1299 * sq(sq(a1)));
      const double alpha = ddiv(K_GRAV * K_MWA * L, K_CPA * K_RG * sq(T)) - ddiv(K_GRAV * K_MAIR, K_RG * T);
      const double gamma = ddiv(K_RG * T, ps * K_MWA) + ddiv(K_MWA * sq(L), K_CPA * pres * K_MAIR * T);
      const double x1 = divc(pres, 101325.);
      const double dv1 = 1.e-4 * (ddiv(0.211, x1)) * dpow(divc(T, 273.), 1.94);
      const double ka1 = 1.e-3 * (4.39 + 0.071 * T);
      const double Gc = drcp(ddiv(K_RHOWA * K_RG * T, ps * dv1 * K_MWA) +
                              ddiv(L * K_RHOWA, ka1 * T) * (ddiv(L * K_MWA, T * K_RG) - 1.));
      const double s_eff = dsqrt(cube(ddiv(ntot, sum1)));
      const double theta = ddiv(dsqrt(cube(ddiv(alpha * V, Gc))), 2. * K_PI * K_RHOWA * gamma * ntot);
      const double khi = (2. / 3.) * aa * dsqrt(ddiv(alpha * V, Gc));
      const double s_max = ddiv(s_eff, dsqrt(0.5 * dsqrt(cube(ddiv(khi, theta))) + dpow(ddiv(sq(s_eff), theta + 3. * khi), 0.75)));
      zdcstar = ddiv(2. * aa, 3. * s_max);
      for (int kk = in1a + lane; kk <= fn2b; kk += LS) {
        if (num_lt(w.numc[kk], K_NLIM)) continue;
        const double nshi = ns[kk] * vrhi[kk];
        const double sil = dexp(dsqrt(ddiv(x, nshi))) - 1.;
        if (s_max < sil) continue;
        const double nslo = ns[kk] * vrlo[kk];
        const double siu = dexp(dsqrt(ddiv(x, nslo))) - 1.;
        frac[kk] = fmin(1., ddiv(dlog(ddiv(s_max, sil)), dlog(ddiv(siu, sil))));
        zdcrlo[kk] = 2. * dsqrt(ddiv(3. * nslo * bb, aa));
        zdcrhi[kk] = 2. * dsqrt(ddiv(3. * nshi * bb, aa));
        zdcrit[kk] = 2. * dsqrt(ddiv(3. * ns[kk] * bb, aa));
      }
      wsync<LS>();
      for (int kk = in1a; kk <= fn2a; kk++)   // the critical bin of regime a
        if (frac[kk] < 1. && frac[kk] > 0.) { bcrita = kk; break; }
    }
  }
  // activate3: nothing activates when no bin has a critical diameter
  bool big = false;
  for (int k = lane; k <= fn2b; k += LS) big |= !(zdcrit[k] < K_EPS);
  if (!wany<LS>(big)) return;
  double Vmid, Vlo, Vhi;
  if (w.numc[bcrita] < K_NLIM) {
    Vmid = K_PI6 * cube(dmid[bcrita]);
  } else {
    double sd = 0.;
    for (int i = 0; i < ndry; i++) sd += w.v(i, bcrita);
    Vmid = ddiv(sd, fmax(K_NLIM, w.numc[bcrita]));
  }
  Vhi = vhi[bcrita];
  Vlo = vlo[bcrita];
  double zvcstar = 0.;
  const double dc = zdcrit[bcrita];
  if (zdcstar >= dc) {
    const double zhlp = ddiv(K_PI6 * cube(zdcstar) - K_PI6 * cube(dc), fmax(K_EPS, K_PI6 * cube(zdcrhi[bcrita]) - K_PI6 * cube(dc)));
    zvcstar = Vmid + zhlp * (Vhi - Vmid);
  } else if (zdcstar < dc) {
    const double zhlp = ddiv(K_PI6 * cube(dc) - K_PI6 * cube(zdcstar), fmax(K_EPS, K_PI6 * cube(dc) - K_PI6 * cube(zdcrlo[bcrita])));
    zvcstar = Vmid - zhlp * (Vmid - Vlo);
  }
  zvcstar = fmax(zvcstar, vlo[bcrita]);
  zvcstar = fmin(zvcstar, vhi[bcrita]);
  for (int cb = lane; cb < ncld; cb += LS) {
    const int ab = (cb <= P.fca_cur) ? P.ica_par + (cb - P.ica_cur) : P.icb_par + (cb - P.icb_cur);
    if (w.numc[ab] < K_NLIM) continue;
    const double Nmid = fmax(w.numc[ab], K_NLIM);
    double sd = 0.;
    for (int i = 0; i < ndry; i++) sd += w.v(i, ab);
    const double Vm = ddiv(sd, Nmid), Vl = vlo[ab], Vh = vhi[ab];
    double Nim1, Vim1, Vlom1, Vhim1, Nip1, Vip1, Vlop1, Vhip1;
    if (ab == in1a || ab == in2b) {
      Nim1 = K_NLIM; Vim1 = divc(Vl, 2.); Vlom1 = 0.; Vhim1 = Vl;
    } else {
      Nim1 = fmax(w.numc[ab - 1], K_NLIM);
      if (Nim1 > K_NLIM) {
        double v = 0.;
        for (int i = 0; i < ndry; i++) v += w.v(i, ab - 1);
        Vim1 = ddiv(v, Nim1);
      } else {
        Vim1 = K_PI6 * cube(dmid[ab - 1]);
      }
      Vlom1 = vlo[ab - 1]; Vhim1 = vhi[ab - 1];
    }
    if (ab == fn2a || ab == fn2b) {
      Nip1 = K_NLIM; Vip1 = Vh + 0.5 * (Vh - Vl); Vlop1 = Vh; Vhip1 = Vh + (Vh - Vl);
    } else {
      Nip1 = fmax(w.numc[ab + 1], K_NLIM);
      if (Nip1 > K_NLIM) {
        double v = 0.;
        for (int i = 0; i < ndry; i++) v += w.v(i, ab + 1);
        Vip1 = ddiv(v, Nip1);
      } else {
        Vip1 = K_PI6 * cube(dmid[ab + 1]);
      }
      Vlop1 = vlo[ab + 1]; Vhip1 = vhi[ab + 1];
    }
    Vip1 = fmax(Vlop1, fmin(Vip1, Vhip1));
    Vim1 = fmax(Vlom1, fmin(Vim1, Vhim1));
    const double dNim1 = ddiv(Nim1, Vhim1 - Vlom1), dNip1 = ddiv(Nip1, Vhip1 - Vlop1), dNmid = ddiv(Nmid, Vh - Vl);
    const double zs1 = ddiv(dNmid - dNim1, Vm - Vim1), zs2 = ddiv(dNip1 - dNmid, Vip1 - Vm);
    const double N01 = dNmid - zs1 * Vm, N02 = dNip1 - zs2 * Vip1;
    const double Nnorm = intgN(zs1, N01, Vl, Vm) + intgN(zs2, N02, Vm, Vh);
    const double Vnorm = intgV(zs1, N01, Vl, Vm) + intgV(zs2, N02, Vm, Vh);
    double nact = 0., zactvol = 0.;
    bool set = false;
    if (zvcstar < Vm) {
      const double zvcint = fmax(zvcstar, Vl);
      nact = (ddiv(Nmid, Nnorm)) * (intgN(zs1, N01, zvcint, Vm) + intgN(zs2, N02, Vm, Vh));
      zactvol = (ddiv(Nmid * Vm, Vnorm)) * (intgV(zs1, N01, zvcint, Vm) + intgV(zs2, N02, Vm, Vh));
      set = true;
    } else if (zvcstar >= Vm) {
      const double zvcint = fmin(zvcstar, Vh);
      nact = (ddiv(Nmid, Nnorm)) * (intgN(zs2, N02, zvcint, Vh));
      zactvol = (ddiv(Nmid * Vm, Vnorm)) * (intgV(zs2, N02, zvcint, Vh));
      set = true;
    }
    nact = fmax(0., set ? nact : 0.);
    for (int ss = 0; ss < nwet; ss++) {
      double v = set ? zactvol * (ddiv(w.v(ss, ab), Vm * Nmid)) : 0.;
      v = fmax(0., v);
      if (ss == iwa)   // the activated droplets' water (:1366-1367)
        v = nact * K_PI6 * cube(zdcrit[ab]) * fmin(2., sq(ddiv(3.e-6, fmax(K_EPS, zdcrit[ab]))));
      raw[P.raw_vact + ss * ncld + cb] = ddiv(v * P.rholiq[ss], dn);
    }
    raw[P.raw_nact + cb] = ddiv(nact, dn);
  }
}

template <typename KT, int LS>
__device__ void act_interst(const DevParams &P, const WS<KT, LS> &w, const double *tb, double prv, double prs, double T,
                            bool diag, int lane) {
  if (ddiv(prv, prs) <= 1.000) return;
  const int ndry = P.ndry, nwet = P.nwet, iwa = P.iwa, C0 = P.nbins;
  const double *dmid = tb + TAB_DMID * P.nb_pad, *vrlo = tb + TAB_VRLO * P.nb_pad, *vrhi = tb + TAB_VRHI * P.nb_pad;
  const double THvol = 1.e-28;
  double zkelvin = ddiv(4. * K_MWA * K_SURFW0, K_RG * K_RHOWA * T);
  double zdcstar = ddiv(2. * zkelvin, 3. * ((ddiv(prv, prs)) - 1.));
  double zvcstar = K_PI6 * cube(zdcstar);
  const auto actn = w.sc(8);        // per cloud bin
  const auto actv = w.sc(0);        // [s * NB + cb] (reuses condensation scratch 0..nwet-1)
  double nsum = 0.;
  for (int cb = lane; cb < P.ncld; cb += LS) {
    int ab = (cb <= P.fca_cur) ? P.ica_par + (cb - P.ica_cur) : P.icb_par + (cb - P.icb_cur);
    double an = 0.;
    double av[SALSA_NSV];
    for (int s = 0; s < SALSA_NSV; s++) av[s] = 0.;
    double vol_sol = 0.;
    for (int i = 0; i < P.nsoluble; i++) vol_sol += w.v(P.ind_soluble[i], ab);
    double Nmid = w.numc[ab];
    bool go = !(Nmid < K_NLIM) && !(vol_sol < Nmid * THvol) && !(w.v(iwa, ab) < Nmid * THvol);
    if (go) {
      double Vwmid = 0., Vmid = 0.;
      for (int s = 0; s < nwet; s++) Vwmid += w.v(s, ab);
      Vwmid /= Nmid;
      for (int s = 0; s < ndry; s++) Vmid += w.v(s, ab);
      Vmid /= Nmid;
      double Vlo = Vmid * vrlo[ab], Vhi = Vmid * vrhi[ab];
      double Nim1, Vim1, Vlom1, Vhim1, Vwim1, Nip1, Vip1, Vlop1, Vhip1, Vwip1;
      if (ab == P.in1a || ab == P.in2b) {
        Nim1 = K_NLIM; Vim1 = divc(Vlo, 2.); Vlom1 = 0.; Vhim1 = Vlo; Vwim1 = Vim1;
      } else {
        Nim1 = w.numc[ab - 1];
        if (Nim1 > K_NLIM) {
          double vd = 0., vw = 0.;
          for (int s = 0; s < ndry; s++) vd += w.v(s, ab - 1);
          for (int s = 0; s < nwet; s++) vw += w.v(s, ab - 1);
          Vim1 = ddiv(vd, Nim1); Vwim1 = ddiv(vw, Nim1);
        } else {
          Vim1 = K_PI6 * cube(dmid[ab - 1]); Vwim1 = K_PI6 * cube(dmid[ab - 1]);
        }
        Vlom1 = Vim1 * vrlo[ab - 1]; Vhim1 = Vim1 * vrhi[ab - 1];
      }
      if (ab == P.fn2a || ab == P.fn2b) {
        Nip1 = K_NLIM; Vip1 = Vhi + 0.5 * (Vhi - Vlo); Vlop1 = Vhi; Vhip1 = Vhi + (Vhi - Vlo); Vwip1 = Vip1;
      } else {
        Nip1 = w.numc[ab + 1];
        if (Nip1 > K_NLIM) {
          double vd = 0., vw = 0.;
          for (int s = 0; s < ndry; s++) vd += w.v(s, ab + 1);
          for (int s = 0; s < nwet; s++) vw += w.v(s, ab + 1);
          Vip1 = ddiv(vd, Nip1); Vwip1 = ddiv(vw, Nip1);
        } else {
          Vip1 = K_PI6 * cube(dmid[ab + 1]); Vwip1 = K_PI6 * cube(dmid[ab + 1]);
        }
        Vlop1 = Vip1 * vrlo[ab + 1]; Vhip1 = Vip1 * vrhi[ab + 1];
      }
      Vip1 = fmax(Vhi, Vip1);
      Vim1 = fmin(Vlo, Vim1);
      double zs1 = ddiv(Vwmid - fmax(Vwim1, 0.), Vmid - Vim1);
      double zs2 = ddiv(fmax(Vwip1, 0.) - Vwmid, Vip1 - Vmid);
      double V01 = Vwmid - zs1 * Vmid, V02 = Vwmid - zs2 * Vmid;
      double Vwlo = fmax(V01 + zs1 * Vlo, Vlo), Vwhi = fmax(V02 + zs2 * Vhi, Vhi);
      double vint1, vint2;
      bool r1, r2, r3, r4;
      if (zvcstar < Vwlo && zvcstar < Vwmid && zvcstar < Vwhi) {
        vint1 = Vlo; vint2 = Vhi; r1 = r2 = r3 = r4 = true;
      } else if (zvcstar > Vwlo && zvcstar > Vwmid && zvcstar > Vwhi) {
        vint1 = 999.; vint2 = 999.; r1 = r2 = r3 = r4 = false;
      } else {
        double vcut = ddiv(zvcstar - V01, zs1);
        vint1 = (vcut < Vlo || vcut > Vmid) ? Vlo : vcut;
        vcut = ddiv(zvcstar - V02, zs2);
        vint2 = (vcut < Vmid || vcut > Vhi) ? Vmid : vcut;
        r1 = Vwlo > zvcstar; r2 = Vwmid > zvcstar; r3 = Vwmid > zvcstar; r4 = Vwhi > zvcstar;
      }
      double dNim1 = ddiv(Nim1, Vhim1 - Vlom1), dNip1 = ddiv(Nip1, Vhip1 - Vlop1), dNmid = ddiv(Nmid, Vhi - Vlo);
      zs1 = ddiv(dNmid - dNim1, Vmid - Vim1);
      zs2 = ddiv(dNip1 - dNmid, Vip1 - Vmid);
      double N01 = dNmid - zs1 * Vmid, N02 = dNmid - zs2 * Vmid;
      double Nnorm = intgN(zs1, N01, Vlo, Vmid) + intgN(zs2, N02, Vmid, Vhi);
      double Vnorm = intgV(zs1, N01, Vlo, Vmid) + intgV(zs2, N02, Vmid, Vhi);
      double zactvol = 0., Nact = 0.;
      if (r1) { Nact += (ddiv(Nmid, Nnorm)) * intgN(zs1, N01, Vlo, vint1); zactvol += (ddiv(Nmid * Vmid, Vnorm)) * intgV(zs1, N01, Vlo, vint1); }
      if (r2) { Nact += (ddiv(Nmid, Nnorm)) * intgN(zs1, N01, vint1, Vmid); zactvol += (ddiv(Nmid * Vmid, Vnorm)) * intgV(zs1, N01, vint1, Vmid); }
      if (r3) { Nact += (ddiv(Nmid, Nnorm)) * intgN(zs2, N02, Vmid, vint2); zactvol += (ddiv(Nmid * Vmid, Vnorm)) * intgV(zs2, N02, Vmid, vint2); }
      if (r4) { Nact += (ddiv(Nmid, Nnorm)) * intgN(zs2, N02, vint2, Vhi); zactvol += (ddiv(Nmid * Vmid, Vnorm)) * intgV(zs2, N02, vint2, Vhi); }
      an = fmin(Nact, Nmid);
      for (int s = 0; s < nwet; s++) av[s] = fmin(zactvol * (ddiv(w.v(s, ab), Vmid * Nmid)), w.v(s, ab));
    }
    actn[cb] = an;
    for (int s = 0; s < nwet; s++) actv[s * w.NB + cb] = av[s];
    nsum += an;
  }
  wsync<LS>();
  if (diag) {
    nsum = wsum<LS>(nsum);
    if (lane == 0) w.misc[M_DIAG + DG_ACTIV] += nsum;
  }
  for (int cb = lane; cb < P.ncld; cb += LS) {
    int ab = P.ica_par + cb, cg = C0 + cb;
    double an = actn[cb];
    if (an > 0.) w.ctime[cg] = ddiv(an * P.chargeTimeMax + w.numc[cg] * w.ctime[cg], an + w.numc[cg]);
    w.numc[ab] = fmax(0., w.numc[ab] - an);
    double nc = w.numc[cg] + an;
    w.numc[cg] = nc;
    for (int s = 0; s < nwet; s++) {
      double av = actv[s * w.NB + cb];
      w.v(s, ab) = fmax(0., w.v(s, ab) - av);
      w.v(s, cg) = w.v(s, cg) + av;
    }
    if (nc > 0.) w.indef[cg] = ddiv(w.indef[cg] * (nc - an) + w.indef[ab] * an, nc);
  }
  wsync<LS>();
}

// mo_salsa_cloud.f90:1401-1477 autoconv2 (cloud bins from the largest; all move to precip bin 1)
template <typename KT, int LS>
__device__ void autoconv2(const DevParams &P, const WS<KT, LS> &w, double dt, int lane) {
  if (lane == 0) {
    const double zd0 = 50.e-6, sigmag = 1.2, max_rate_autoc = 1.0e10;
    const int C0 = P.nbins, P0 = P.nbins + P.ncld;
    for (int cc = P.ncld - 1; cc >= 0; cc--) {
      int g = C0 + cc;
      double tot = 0.;
      double Ntot = w.numc[g], Vtot = 0.;
      for (int s = 0; s < P.nwet; s++) Vtot += w.v(s, g);
      if (Ntot > K_NLIM && Vtot > 0.) {
        double ls = log(sigmag);
        double dvg = dcbrt(divc(ddiv(Vtot, Ntot), K_PI6)) * exp((3. * ls * ls) / 2.);
        double dg = dvg * exp(-3. * ls * ls);
        double hlp2 = sqrt(2.) * ls;
        double Vrem = Vtot * (1. - (0.5 + 0.5 * erf(ddiv(log(zd0) - dlog(dvg), hlp2))));
        double Nrem = Ntot * (1. - (0.5 + 0.5 * erf(ddiv(log(zd0) - dlog(dg), hlp2))));
        if (Vrem > 0. && Nrem > K_PRLIM) {
          for (int s = 0; s < P.ndry; s++) {
            w.v(s, P0) = w.v(s, P0) + w.v(s, g) * (ddiv(Nrem, Ntot));
            w.v(s, g) = w.v(s, g) * (1. - (ddiv(Nrem, Ntot)));
          }
          w.v(P.iwa, P0) = w.v(P.iwa, P0) + w.v(P.iwa, g) * (ddiv(Vrem, Vtot));
          w.v(P.iwa, g) = w.v(P.iwa, g) * (1. - (ddiv(Vrem, Vtot)));
          w.numc[P0] = w.numc[P0] + Nrem;
          w.numc[g] = w.numc[g] - Nrem;
          tot = tot + Nrem;
          if (tot > max_rate_autoc * dt) break;
        }
      }
    }
  }
  wsync<LS>();
}


// ----------------------------------------------------------------------------------------
// Ice nucleation with contact-angle distributions: mo_salsa_cloud_ice_SE.f90:28-555.
// Lanes own liquid bins; each lane stages what its bin hands to the ice bins, and the
// ice bins then add the staged amounts in liquid-bin order (the reference order).
// ----------------------------------------------------------------------------------------
__device__ __constant__ double c_gl_x[10] = {-0.973908239224106, -0.865060566454542, -0.679410688379483,
                                             -0.433395397408358, -0.148874339007507, 0.148874339007507,
                                             0.433395397408358,  0.679410688379483,  0.865060566454542,
                                             0.973908239224106};
__device__ __constant__ double c_gl_w[10] = {0.066667031481273176, 0.14945422671662059, 0.21908574324601154,
                                             0.26926671836765848,  0.29552422471242434, 0.29552422471242434,
                                             0.26926671836765848,  0.21908574324601154, 0.14945422671662059,
                                             0.066667031481273176};

// Products that must not fuse with a following add: the freezing rates below take
// exp(-crit/kT) of terms that cancel (het_sf), so a fused rounding there moves the
// frozen fraction far more than any input rounding does.  The rest of the FP64 form
// contracts multiply-adds.
__device__ __forceinline__ double mrn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double cube_rn(double x) { return __dmul_rn(__dmul_rn(x, x), x); }

__device__ double erfm1(double x) {   // math_functions.f90:494-510
  const double a = 0.140012;
  double sgn = x < 0. ? -1. : 1.;
  double xx = fmax(1.e-20, 1. - x * x);
  double t1 = dlog(xx), t2 = 2. / (K_PI_FULL * a);
  double t3 = t2 + mrn(0.5, t1), t4 = divc(t1, a), t5 = t2 + mrn(0.5, t1);
  return sgn * dsqrt(dsqrt(mrn(t3, t3) - t4) - t5);
}
// f_gauss (:515-524) with its per-configuration factors 1/(sqrt(2 pi) sig) and 1/sig^2
// taken once per cell
struct GaussC { double ra, rs2, mean; };
__device__ __forceinline__ GaussC gauss_c(double sig, double mean) {
  GaussC g;
  g.ra = drcp(sqrt(2. * K_PI_FULL) * sig);
  g.rs2 = drcp(sig * sig);
  g.mean = mean;
  return g;
}
__device__ __forceinline__ double f_gauss(double x, const GaussC &g) {
  double b = (x - g.mean) * (x - g.mean);
  b = b * g.rs2;
  return g.ra * dexp(-0.5 * b);
}
__device__ double het_sf(double x, double mis) {   // SE :375-390
  if (x > 100.) return divc(cube_rn(mis) - mrn(3., mis) + 2., 4.);
  double fii = dsqrt(1. - mrn(mrn(2., mis), x) + mrn(x, x));
  double fpsi = ddiv(x - mis, fii);
  return 0.5 * (1. + cube_rn(ddiv(1. - mrn(mis, x), fii)) + mrn(2. - mrn(3., fpsi) + cube_rn(fpsi), cube_rn(x)) +
                mrn(mrn(mrn(mrn(3., mis), fpsi - 1.), x), x));
}

// Temperature-only parts of J_imm (:210-278), evaluated once per cell and bin
struct JimmPre { double act_energy, sigma_is, d_g; bool ok; };
__device__ JimmPre jimm_pre(double Tk, double Seq) {
  JimmPre r;
  const double rho_ice = 900., T0 = 273.15;
  double Tc = Tk - T0;
  r.act_energy = divc(K_RG * Tk * (ddiv(347., Tk - 177.) - log(4.14 / 349.)), K_AVOG);
  r.sigma_is = 28.e-3 + mrn(0.25e-3, Tc);
  double Lefm = (79.7 + mrn(0.708, Tc) - mrn(mrn(2.5e-3, Tc), Tc)) * 4.1868e3;
  double GG = ddiv(divc(K_RG * Tk, K_MWA), Lefm);
  double sg = dpow(Seq, GG);
  r.ok = !((ddiv(T0, Tk)) * sg < 1.0001);
  r.d_g = r.ok ? ddiv(4. * r.sigma_is, mrn(mrn(rho_ice, Lefm), dlog((ddiv(T0, Tk)) * sg)) - 1.7e10 * 0.) : 0.;
  if (r.d_g <= 1e-10) r.ok = false;
  return r;
}
// kth = K_BOLTZ * Tk / K_PLANCK, taken once per cell; x = Din / d_g, once per bin
__device__ double J_imm(const JimmPre &q, double theta, double Tk, double Din, double x, double kth) {
  if (Din < 1e-10 || !q.ok) return 0.;
  double costh = cos(divc(theta * K_PI, 180.));
  double sf = het_sf(x, costh);
  double crit = mrn(mrn(mrn((K_PI / 3.), q.sigma_is), mrn(q.d_g, q.d_g)), sf) -
                mrn(mrn(mrn((1. / 4.) * 0.0, (1. - costh)), Din), Din);
  return kth * 1.e19 * K_PI * (Din * Din) * dexp(-ddiv(q.act_energy + crit, K_BOLTZ * Tk));
}
__device__ double J_dep(double theta, double Tk, double Din, double Seq) {   // :282-331
  if (Din < 1e-10 || Seq < 1.0001) return 0.;
  double Tc = Tk - 273.15;
  double sigma_iv = ((76.1 - mrn(0.155, Tc)) + (28.5 + mrn(0.25, Tc))) * 1.e-3;
  double d_g = ddiv(4. * sigma_iv, mrn(K_RG * K_RHOIC / K_MWA * Tk, dlog(Seq)) - 1.7e10 * 0.);
  if (d_g <= 1e-10) return 0.;
  double costh = cos(divc(theta * K_PI, 180.));
  double sf = het_sf(ddiv(Din, d_g), costh);
  double crit = (K_PI / 3.) * sigma_iv * (d_g * d_g) * sf;
  return (1. / 4.) * 1.e30 * (Din * Din) * dexp(-ddiv(0. + crit, K_BOLTZ * Tk));
}
__device__ double J_hf(double Tk, double Sw) {   // :335-371
  const double Nc = 5.85e16, T0 = 273.15;
  double Tc = Tk - T0;
  double act = 0.694e-19 * (1. + mrn(0.027, (Tc + 30.)));
  double Lefm = (79.7 + mrn(0.708, Tc) - mrn(mrn(2.5e-3, Tc), Tc)) * 4.1868e3;
  double GG = divc(ddiv(K_RG * Tk, Lefm), K_MWA);
  double sg = dpow(Sw, GG);
  if ((ddiv(T0, Tk)) * sg < 1.0001) return 0.;
  double sigma_is = 28.e-3 + mrn(0.25e-3, Tc);
  double d_g = ddiv(4. * sigma_is, K_RHOIC * Lefm * dlog((ddiv(T0, Tk)) * sg));
  if (d_g <= 1e-10) return 0.;
  double crit = (K_PI / 3.) * sigma_is * d_g * d_g;
  return 2.0 * Nc * (divc(divc(K_RHOWA * K_BOLTZ * Tk, K_RHOIC), K_PLANCK)) * dsqrt(ddiv(divc(sigma_is, K_BOLTZ), Tk)) *
         dexp(-ddiv(crit + act, K_BOLTZ * Tk));
}

// calcSweq (mo_particle_external_properties.f90:402-447)
template <typename KT, int LS>
__device__ double calc_sweq(const DevParams &P, const WS<KT, LS> &w, int b, double T, double kappa) {
  double n = w.numc[b];
  if (num_lt(n, nlim_of(phase_of(P, b)))) return 0.;
  double vs = 0.;
  for (int s = 0; s < P.nused; s++) vs += w.v(s, b);
  double dwet = dcbrt(divc(ddiv(vs, n), K_PI6));
  double znw = divc(w.v(P.iwa, b) * K_RHOWA, K_MWA), zvw = w.v(P.iwa, b);
  double zns = 0., zvs = 0., zvtot = 0.;
  for (int i = 0; i < P.ndry; i++) {
    zns = zns + ddiv(P.diss[i] * w.v(i, b) * P.rholiq[i], P.MM[i]);
    zvs = zvs + mrn(fmin(1., P.diss[i]), w.v(i, b));
    zvtot = zvtot + w.v(i, b);
  }
  if (P.has_kappa) zns = solute_moles(P, w, b, kappa);
  double kel = dexp(ddiv(4. * K_SURFW0 * K_MWA, K_RG * T * K_RHOWA * dwet));
  if (zvw > 1.e-28 * n || zvs > 1.e-28 * n) return (ddiv(znw, zns + znw)) * kel;
  if (zvtot - zvs > 1.e-28 * n) return kel;
  return (ddiv(znw, K_EPS + zns + znw)) * kel;
}

__device__ __forceinline__ int ice_bin_of(const DevParams &P, const double *vlo, double dwet) {   // :542-555
  double vol = divc(K_PI6 * cube(dwet) * K_RHOWA, K_RHOIC);
  int ii = 0;
  for (int k = 0; k < P.nice; k++) ii += (vlo[P.nliquid + k] < vol);
  return min(max(1, ii), P.nice) - 1;
}
__device__ __forceinline__ int precip_bin_of(const DevParams &P, const double *vlo, double dwet, double dens) {
  double vol = divc(K_PI6 * cube(dwet) * dens, K_RHOWA);   // :559-573
  int ii = 0;
  for (int k = 0; k < P.nprc; k++) ii += (vlo[P.nbins + P.ncld + k] < vol);
  return min(max(1, ii), P.nprc) - 1;
}

// staged ice contribution of one liquid bin: [0] target ice bin (-1 none), [1..nused] volumes, [8] number
template <typename KT, int LS>
__device__ void ice_apply_staged(const DevParams &P, const WS<KT, LS> &w, const Ptr<double, LS> &stage, int nsrc, int lane) {
  if constexpr (LS == 1) {
    // sources in order; each goes to one ice bin
    for (int k = 0; k < nsrc; k++) {
      const auto st = stage + k * 10;
      const int ib = (int)st[0];
      if (ib < 0) continue;
      const int g = P.nliquid + ib;
      const bool all = st[9] != 0.;
      for (int q = 0; q <= P.nused; q++) {
        const double add = (q < P.nused) ? st[1 + q] : st[8];
        if (add == 0. && !all) continue;
        if (q < P.nused) w.v(q, g) = fmax(0., w.v(q, g) + add);
        else w.numc[g] = fmax(0., w.numc[g] + add);
      }
    }
    return;
  }
  // one lane per ice bin and component, sources in order
  const int ncomp = P.nused + 1;
  for (int e = lane; e < P.nice * ncomp; e += LS) {
    int ib = e / ncomp, q = e % ncomp, g = P.nliquid + ib;
    double val = (q < P.nused) ? w.v(q, g) : w.numc[g];
    for (int k = 0; k < nsrc; k++) {
      const auto st = stage + k * 10;
      if ((int)st[0] != ib) continue;
      double add = (q < P.nused) ? st[1 + q] : st[8];
      if (add != 0. || st[9] != 0.) val = fmax(0., val + add);
    }
    if (q < P.nused) w.v(q, g) = val; else w.numc[g] = val;
  }
  wsync<LS>();
}

// SE ice nucleation (mo_salsa_SecondaryIce / iceNucleation, :394-538).  Pass A (lanes
// over liquid bins) evaluates the per-bin quantities and decides which bins need the
// Gauss-Legendre integral over contact angles; pass B evaluates the integrands with one
// lane per (bin, node), three bins per warp pass, and sums each bin's ten terms in node
// order; pass C (lanes over bins) applies the frozen fractions.
template <typename KT, int LS>
__device__ void ice_nucl_SE(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double prv, double prs,
                            double prsi, double dt, double kappa, bool diag, int lane) {
  if (P.ninsoluble <= 0) return;
  const double *dmid = tb + TAB_DMID * P.nb_pad, *vlo = tb + TAB_VLO * P.nb_pad;
  const double dmin = 1.e-10, tmax_homog = 237.9, minVin = K_PI6 * cube(1.e-8);
  const int nl = P.nliquid, ndry = P.ndry, iwa = P.iwa, irim = P.irim, idu = P.ix_du;
  const unsigned F = 0xffffffffu;
  const auto stage = w.scr;   // nl * 10 doubles
  // per-bin records in the (now unused) collision-kernel area: 8 doubles per bin
  const auto rec = row_cast<double>(w.K);
  enum { R_MODE = 0, R_THMIN, R_DIN, R_AE, R_SIG, R_DG, R_FHOM, R_FINT };
  const double Si = ddiv(prv, prsi);
  // The lane form's short cuts leave out bins that cannot freeze.  A bin that freezes by nothing
  // still sets negative values of the crystal bin of its size to zero (fmax of the sum), so
  // they are for cells without negative ice: every cell, unless coagulation is off and
  // advection left some.
  bool quick = LS == 1;
  if constexpr (LS == 1) {
    auto ok = [](double x) {   // zero, positive or infinite
      const unsigned long long b = (unsigned long long)__double_as_longlong(x);
      return b <= (unsigned long long)FM_INF || b << 1 == 0ull;
    };
    if (P.st_icenucl)
      for (int g = nl; g < P.ntotal; g++) {
        quick = quick && ok(w.numc[g]);
        for (int s = 0; s < P.nused; s++) quick = quick && ok(w.v(s, g));
      }
  }
  // pass A
  for (int kk = lane; kk < nl; kk += LS) {
    const auto st = stage + kk * 10;
    st[0] = -1.;
    const auto r = rec + kk * 8;
    if constexpr (LS == 1) {
      // no scheme can freeze this bin (dry aerosol with immersion freezing alone, empty bins)
      const int ph = phase_of(P, kk);
      const bool cnt = !(T > 273.15) && !num_lt(w.numc[kk], nlim_of(ph));
      if (quick && !((P.lsicehom && T < tmax_homog) || (cnt && ph > 1 && P.lsiceimm) || (cnt && ph == 1 && P.lsicedep))) {
        r[R_FHOM] = 0.;
        r[R_MODE] = 0.;
        continue;
      }
    }
    for (int q = 1; q < 10; q++) st[q] = 0.;
    updateDiameterAll(P, w, dmid, kk);
    const double dwet = w.dwet[kk], dins_ = w.ddry[kk];
    const double n = w.numc[kk];
    const int ph = phase_of(P, kk);
    const bool countable = !(T > 273.15) && !num_lt(n, nlim_of(ph));
    const bool hom = dwet - dins_ > dmin && T < tmax_homog && P.lsicehom;
    const bool imm = P.lsiceimm && (ph == 2 || ph == 3) && (w.dins[kk] > dmin) && countable;
    const bool dep = P.lsicedep && (ph == 1 && ddiv(prv, prs) < 1.0) && (w.dwet[kk] - w.dins[kk] < dmin) &&
                     (w.dins[kk] > dmin) && countable;
    double Seq = 0.;
    if (hom || imm) Seq = calc_sweq(P, w, kk, T, kappa);
    double f_hom = 0.;
    if (hom) {
      double Jh = J_hf(T, Seq);
      f_hom = 1. - dexp(-Jh * K_PI6 * (cube_rn(dwet) - cube_rn(dins_)) * dt);
    }
    r[R_FHOM] = f_hom;
    r[R_MODE] = imm ? 1. : (dep ? 2. : 0.);
    r[R_DIN] = w.ddry[kk];
    double fint = 0.;
    if (imm) {
      // low_theta (:394-417)
      double th00 = P.mean_theta_imm + mrn(sqrt(2.) * P.sigma_theta_imm, erfm1(mrn(2., w.indef[kk]) - 1.));
      th00 = fmin(fmax(th00, 0.), 180.);
      if (!P.st_freeTheta) th00 = fmax(P.initMinTheta, th00);
      JimmPre q = jimm_pre(T, Seq);
      r[R_THMIN] = th00; r[R_AE] = q.act_energy; r[R_SIG] = q.sigma_is; r[R_DG] = q.ok ? q.d_g : -1.;
      fint = q.ok ? ddiv(r[R_DIN], q.d_g) : 0.;   // the integrand's size ratio, until the integral takes its place
    } else if (dep) {
      double th00 = P.mean_theta_dep + mrn(sqrt(2.) * P.sigma_theta_dep, erfm1(mrn(2., w.indef[kk]) - 1.));
      th00 = fmin(fmax(th00, 0.), 180.);
      if (!P.st_freeTheta) th00 = fmax(P.initMinTheta, th00);
      r[R_THMIN] = th00;
    }
    r[R_FINT] = fint;
  }
  wsync<LS>();
  // pass B: gauss_legendre (:131-206) for the bins that need it
  const GaussC g_imm = gauss_c(P.sigma_theta_imm, P.mean_theta_imm);
  const GaussC g_dep = gauss_c(P.sigma_theta_dep, P.mean_theta_dep);
  const double kth = divc(K_BOLTZ * T, K_PLANCK);
  auto node_term = [&](const Ptr<double, LS> &r, int node) {
    const double thmin = r[R_THMIN], thmax = 180.;
    const double th1 = mrn(0.5 * (thmax - thmin), c_gl_x[node]) + 0.5 * (thmax + thmin);
    double J, ft;
    if (r[R_MODE] == 1.) {
      JimmPre q;
      q.act_energy = r[R_AE]; q.sigma_is = r[R_SIG]; q.d_g = r[R_DG]; q.ok = r[R_DG] >= 0.;
      J = J_imm(q, th1, T, r[R_DIN], r[R_FINT], kth);
      ft = th1 > thmin ? f_gauss(th1, g_imm) : 0.;
    } else {
      J = J_dep(th1, T, r[R_DIN], Si);
      ft = th1 > thmin ? f_gauss(th1, g_dep) : 0.;
    }
    return ft * c_gl_w[node] * (1. - dexp(-J * dt));
  };
  if constexpr (LS == 1) {
    for (int kk = 0; kk < nl; kk++) {
      const auto r = rec + kk * 8;
      if (r[R_MODE] == 0.) continue;
      double acc = 0.;
      for (int node = 0; node < 10; node++) acc = acc + node_term(r, node);
      r[R_FINT] = 0.5 * (180. - r[R_THMIN]) * acc;
    }
  } else {
    const unsigned lt = (1u << lane) - 1u;
    int nlist = 0;
    int *list = w.pbuf;
    for (int base = 0; base < nl; base += LS) {
      int kk = base + lane;
      bool need = kk < nl && rec[kk * 8 + R_MODE] != 0.;
      unsigned bal = __ballot_sync(F, need);
      if (need) list[nlist + __popc(bal & lt)] = kk;
      nlist += __popc(bal);
    }
    wsync<LS>();
    const int grp = lane / 10, node = lane - grp * 10;
    for (int b0 = 0; b0 < nlist; b0 += 3) {
      const int slot = b0 + grp;
      const bool on = grp < 3 && slot < nlist;
      const int kk = on ? list[slot] : 0;
      double term = 0.;
      if (on) {
        term = node_term(rec + kk * 8, node);
      }
      double acc = 0.;
      const int g10 = (grp < 3 ? grp : 0) * 10;
#pragma unroll
      for (int i = 0; i < 10; i++) acc = acc + __shfl_sync(F, term, g10 + i);
      if (on && node == 0) {
        const auto r = rec + kk * 8;
        r[R_FINT] = 0.5 * (180. - r[R_THMIN]) * acc;
      }
    }
    wsync<LS>();
  }
  // pass C: iceNucleation (:421-538)
  double dh = 0., dd = 0., di = 0.;
  for (int kk = lane; kk < nl; kk += LS) {
    const auto st = stage + kk * 10;
    const auto r = rec + kk * 8;
    const double dwet = w.dwet[kk];
    const double n = w.numc[kk];
    const int ph = phase_of(P, kk);
    if constexpr (LS == 1) {
      if (quick && (__double_as_longlong(r[R_MODE]) | __double_as_longlong(r[R_FHOM])) == 0) {
        // nothing freezes: what is left of the update below are its limits, and an IN deficit
        // of 0/0 -> 0 without dust
        if (num_lt(n, nlim_of(ph))) continue;
        double vins = 0.;
        for (int k = 0; k < P.ninsoluble; k++) vins += w.v(P.ind_insoluble[k], kk);
        if (num_lt(vins, minVin)) continue;
        w.indef[kk] = __double_as_longlong(w.v(idu, kk)) << 1 == 0 ? 0. : min_pos(pos_part(w.indef[kk]), 1.);
        for (int s = 0; s < P.nwet; s++) w.v(s, kk) = pos_part(w.v(s, kk));
        w.numc[kk] = pos_part(n);
        continue;
      }
    }
    const double f_hom = r[R_FHOM];
    const double f_imm = r[R_MODE] == 1. ? r[R_FINT] : 0.;
    const double f_dep = r[R_MODE] == 2. ? r[R_FINT] : 0.;
    dh += mrn(n, f_hom); dd += mrn(n, f_dep); di += mrn(n, f_imm);
    double frac = fmax(0., fmin(0.99, f_imm + f_hom + f_dep - mrn((f_imm + f_dep), f_hom)));
    if (num_lt(n, nlim_of(ph))) continue;
    double vins = 0.;
    for (int k = 0; k < P.ninsoluble; k++) vins += w.v(P.ind_insoluble[k], kk);
    if (vins < minVin) continue;
    int bb = ice_bin_of(P, vlo, dwet);
    double vdry = 0.;
    for (int s = 0; s < ndry; s++) vdry += w.v(s, kk);
    double V_tot = frac * vdry;
    double frac_DU = ddiv(w.v(idu, kk), vdry);
    double frac2, ncur0;
    if (frac_DU <= 0.1) { frac2 = frac * frac_DU; ncur0 = n * frac_DU; }
    else { frac2 = frac; ncur0 = n; }
    double nnuc = frac2 * n;
    double f1 = nnuc + mrn((ncur0 - nnuc), w.indef[kk]);
    f1 = ddiv(f1, ncur0);
    w.indef[kk] = fmin(fmax(f1, 0.), 1. - 1.e-20);
    st[0] = (double)bb;
    st[9] = 1.;
    bool mk = P.st_icenucl;
    if (frac_DU <= 0.1) {
      if (mk) st[1 + idu] = V_tot * frac_DU;
      w.v(idu, kk) = fmax(0., w.v(idu, kk) - mrn(V_tot, frac_DU));
    } else {
      for (int s = 0; s < ndry; s++) {
        if (mk) st[1 + s] = w.v(s, kk) * frac2;
        w.v(s, kk) = fmax(0., w.v(s, kk) * (1. - frac2));
      }
    }
    if (ph == 1 || ph == 2) {
      if (mk) st[1 + iwa] = divc(w.v(iwa, kk) * frac2 * K_RHOWA, K_RHOIC);
    } else {
      if (mk) st[1 + irim] = divc(w.v(iwa, kk) * frac2 * K_RHOWA, K_RHORI);
    }
    w.v(iwa, kk) = fmax(0., w.v(iwa, kk) * (1. - frac2));
    if (mk) st[8] = n * frac2;
    w.numc[kk] = fmax(0., n * (1. - frac2));
    if (!mk) st[9] = 0.;
  }
  wsync<LS>();
  if (diag) {
    dh = wsum<LS>(dh); dd = wsum<LS>(dd); di = wsum<LS>(di);
    if (lane == 0) {
      w.misc[M_DIAG + DG_ICEHOM] += dh;
      w.misc[M_DIAG + DG_ICEDEP] += dd;
      w.misc[M_DIAG + DG_ICEIMM] += di;
    }
  }
  if (P.st_icenucl) ice_apply_staged(P, w, stage, nl, lane);
}

// classic ice nucleation (mo_salsa_cloud_ice.f90:26-140 with calc_Jhet/Jdep/Jhf :146-291)
__device__ double calc_Jhet(double rn, double temp, double Sw) {
  const double rho_ice = 900., c_1s = 1e32, T0 = 273.15, mis = 0.5;
  if (rn < 1e-10) return 0.;
  double Tc = temp - T0;
  double act = divc(K_RG * temp * (ddiv(347., temp - 177.) - log(4.14 / 349.)), K_AVOG);
  double Lefm = (79.7 + mrn(0.708, Tc) - mrn(mrn(2.5e-3, Tc), Tc)) * 4.1868e3;
  double GG = ddiv(divc(K_RG * temp, K_MWA), Lefm);
  double sg = dpow(Sw, GG);
  if ((ddiv(T0, temp)) * sg < 1.0001) return 0.;
  double sigma_is = 28.e-3 + mrn(0.25e-3, Tc);
  double r_g = ddiv(4. * sigma_is, mrn(mrn(rho_ice, Lefm), dlog((ddiv(T0, temp)) * sg)) - 1.7e10 * 0.);
  if (r_g <= 1e-10) return 0.;
  double sf = het_sf(ddiv(rn, r_g), mis);
  double crit = mrn(mrn(mrn(mrn((K_PI / 3.), sigma_is), r_g), r_g), sf) -
                mrn(mrn(mrn((1. / 4.) * 0.0, (1. - mis)), rn), rn);
  return divc(K_BOLTZ * temp, K_PLANCK) * c_1s * K_PI * rn * rn * dexp(ddiv(-act - crit, K_BOLTZ * temp));
}
__device__ double calc_Jdep(double rn, double temp, double Si) {
  const double rho_ice = 900., mis = 0.5;
  if (rn < 1e-10 || Si < 1.0001) return 0.;
  double Tc = temp - 273.15;
  double sigma_iv = ((76.1 - mrn(0.155, Tc)) + (28.5 + mrn(0.25, Tc))) * 1e-3;
  double r_g = ddiv(4. * sigma_iv, mrn(K_RG * rho_ice / K_MWA * temp, dlog(Si)) - 1.7e10 * 0.);
  if (r_g <= 1e-10) return 0.;
  double sf = het_sf(ddiv(rn, r_g), mis);
  double crit = (K_PI / 3.) * sigma_iv * r_g * r_g * sf;
  return (1. / 4.) * 1.e30 * rn * rn * dexp(ddiv(-0. - crit, K_BOLTZ * temp));
}
__device__ double calc_Jhf(double temp, double Sw) {
  const double Nc = 5.85e16, rho_ice = 900., T0 = 273.15;
  double Tc = temp - T0;
  double act = 0.694e-19 * (1. + mrn(0.027, (Tc + 30.)));
  double Lefm = (79.7 + mrn(0.708, Tc) - mrn(mrn(2.5e-3, Tc), Tc)) * 4.1868e3;
  double GG = divc(ddiv(K_RG * temp, Lefm), K_MWA);
  double sg = dpow(Sw, GG);
  if ((ddiv(T0, temp)) * sg < 1.0001) return 0.;
  double sigma_is = 28.e-3 + mrn(0.25e-3, Tc);
  double r_g = ddiv(2. * sigma_is, rho_ice * Lefm * dlog((ddiv(T0, temp)) * sg));
  if (r_g <= 1e-10) return 0.;
  double crit = 4. * K_PI / 3. * sigma_is * r_g * r_g;
  return 2.0 * Nc * (divc(divc(K_RHOWA * K_BOLTZ * temp, rho_ice), K_PLANCK)) * dsqrt(ddiv(divc(sigma_is, K_BOLTZ), temp)) *
         dexp(ddiv(-crit - act, K_BOLTZ * temp));
}

template <typename KT, int LS>
__device__ void ice_nucl_classic(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, double prv,
                                 double prs, double prsi, double dt, double kappa, bool diag, int lane) {
  const double *dmid = tb + TAB_DMID * P.nb_pad, *vlo = tb + TAB_VLO * P.nb_pad;
  const double tmax_homog = 237.9, dmin = 1.e-10;
  const int nl = P.nliquid, ndry = P.ndry, iwa = P.iwa, irim = P.irim;
  const auto stage = w.scr;
  double dh = 0., dd = 0., di = 0.;
  for (int kk = lane; kk < nl; kk += LS) {
    const auto st = stage + kk * 10;
    for (int q = 0; q < 10; q++) st[q] = 0.;
    st[0] = -1.;
    int ph = phase_of(P, kk);
    if (T > 273.15 || w.numc[kk] < nlim_of(ph)) continue;
    updateDiameterAll(P, w, dmid, kk);
    double dins_ = w.dins[kk], dwet = w.dwet[kk];
    double Sw = calc_sweq(P, w, kk, T, kappa);
    double pf_imm = 0., pf_dep = 0., pf_hom = 0.;
    if (dins_ > dmin && P.lsiceimm && (ph == 2 || ph == 3)) pf_imm = 1. - dexp(-calc_Jhet(dins_, T, Sw) * dt);
    if (dins_ > dmin && dwet - dins_ < dmin && ddiv(prv, prs) < 1.0 && ph == 1 && P.lsicedep)
      pf_dep = 1. - dexp(-calc_Jdep(dins_, T, ddiv(prv, prsi)) * dt);
    if (dwet - dins_ > dmin && T < tmax_homog && P.lsicehom)
      pf_hom = 1. - dexp(-calc_Jhf(T, Sw) * K_PI6 * (cube_rn(dwet) - cube_rn(dins_)) * dt);
    double frac = fmax(0., fmin(0.99, pf_imm + pf_hom + pf_dep - mrn((pf_imm + pf_dep), pf_hom)));
    int bb = ice_bin_of(P, vlo, dwet);
    bool mk = P.st_icenucl;
    st[0] = (double)bb;
    st[9] = mk ? 1. : 0.;
    for (int s = 0; s < ndry; s++) {
      if (mk) st[1 + s] = w.v(s, kk) * frac;
      w.v(s, kk) = fmax(0., w.v(s, kk) * (1. - frac));
    }
    if (ph == 1 || ph == 2) { if (mk) st[1 + iwa] = divc(w.v(iwa, kk) * frac * K_RHOWA, K_RHOIC); }
    else { if (mk) st[1 + irim] = divc(w.v(iwa, kk) * frac * K_RHOWA, K_RHORI); }
    w.v(iwa, kk) = fmax(0., w.v(iwa, kk) * (1. - frac));
    if (mk) st[8] = w.numc[kk] * frac;
    double nn = fmax(0., w.numc[kk] * (1. - frac));
    w.numc[kk] = nn;
    // iceDiagnostics is called after iceNucleation (:130-132): the reduced number
    dh += nn * pf_hom; dd += nn * pf_dep; di += nn * pf_imm;
  }
  wsync<LS>();
  if (diag) {
    dh = wsum<LS>(dh); dd = wsum<LS>(dd); di = wsum<LS>(di);
    if (lane == 0) {
      w.misc[M_DIAG + DG_ICEHOM] += dh;
      w.misc[M_DIAG + DG_ICEDEP] += dd;
      w.misc[M_DIAG + DG_ICEIMM] += di;
    }
  }
  ice_apply_staged(P, w, stage, nl, lane);
  for (int b = P.nliquid + lane; b < P.ntotal; b += LS)
    w.rhomean[b] = rhomean_of(P, 4, w.numc[b], w.v(iwa, b), w.v(irim, b));
  wsync<LS>();
}

// ice_melt (mo_salsa_cloud_ice.f90:393-462): ice bins staged per lane, precip bins add in ice order
template <typename KT, int LS>
__device__ void ice_melt(const DevParams &P, const WS<KT, LS> &w, const double *tb, double T, int lane) {
  if (T < 273.15) return;
  const double *dmid = tb + TAB_DMID * P.nb_pad, *vlo = tb + TAB_VLO * P.nb_pad;
  const double maxfrac = 0.999;
  const int ndry = P.ndry, iwa = P.iwa, irim = P.irim, I0 = P.nliquid, P0 = P.nbins + P.ncld;
  const auto stage = w.scr;   // nice * 10
  for (int k = lane; k < P.nice; k += LS) {
    int g = I0 + k;
    const auto st = stage + k * 10;
    for (int q = 0; q < 10; q++) st[q] = 0.;
    st[0] = -1.;
    if (w.numc[g] < K_PRLIM) continue;
    // updateDiameter(limit, "wet") and updateRhomean
    double n = w.numc[g];
    double dw;
    if (n > K_PRLIM) {
      double vs = 0.;
      for (int s = 0; s < P.nused; s++) vs += w.v(s, g);
      dw = dcbrt(divc(ddiv(vs, n), K_PI6));
    } else {
      dw = dmid[g];
    }
    dw = fmin(dw, 10.e-3);
    w.dwet[g] = dw;
    double rm = rhomean_of(P, 4, n, w.v(iwa, g), w.v(irim, g));
    w.rhomean[g] = rm;
    int bb = precip_bin_of(P, vlo, dw, rm);
    st[0] = (double)bb;
    for (int s = 0; s < ndry; s++) {
      st[1 + s] = maxfrac * w.v(s, g);
      w.v(s, g) = (1. - maxfrac) * w.v(s, g);
    }
    double liqvol = divc(w.v(iwa, g) * K_RHOIC + w.v(irim, g) * K_RHORI, K_RHOWA);
    st[8] = maxfrac * n;
    w.numc[g] = (1. - maxfrac) * n;
    st[1 + iwa] = maxfrac * liqvol;
    w.v(iwa, g) = (1. - maxfrac) * w.v(iwa, g);
    w.v(irim, g) = (1. - maxfrac) * w.v(irim, g);
  }
  wsync<LS>();
  // precip bin gets dry species, number, water in ice-bin order
  for (int e = lane; e < P.nprc * (P.nwet + 1); e += LS) {
    int pb = e / (P.nwet + 1), q = e % (P.nwet + 1), g = P0 + pb;
    double val = (q < P.nwet) ? w.v(q, g) : w.numc[g];
    for (int k = 0; k < P.nice; k++) {
      const auto st = stage + k * 10;
      if ((int)st[0] != pb) continue;
      val = val + ((q < P.nwet) ? st[1 + q] : st[8]);
    }
    if (q < P.nwet) w.v(q, g) = val; else w.numc[g] = val;
  }
  wsync<LS>();
}

// ----------------------------------------------------------------------------------------
// distr_update: mo_salsa_update.f90:21-433.  A sweep visits the bins of a category in
// descending order; a bin's move depends on what it holds when the sweep reaches it.
// Moves go to the next bin up (visited already) or to a lower bin (visited later), so
// every bin from the top down to the highest downward move holds its sweep-start
// content when visited.  Those bins are processed by one lane each with the same
// arithmetic as the sequential sweep; the bins below that point follow sequentially on
// lane 0.  The bin-limit flag is overwritten by every checked bin (:132, 224, 322, 418):
// the last checked bin decides whether another sweep follows.
// ----------------------------------------------------------------------------------------
enum { DC_AERO = 0, DC_CLOUD, DC_PRECP, DC_ICE };

struct DStep {
  int dir;              // 0 stays, 1 moves up, -1 moves down
  int target;           // global index of the receiving bin
  bool check, within, neg;
  double own_n, push_n;
  double own[SALSA_NSV], push[SALSA_NSV];
};

// One bin of one sweep given its current content (n, v): kk is the index inside the
// category, g the global bin index.  Aerosols :66-136, cloud :150-226, precipitation
// :240-324 (wet volume), ice :338-420 (total volume).
template <int CAT>
__device__ __forceinline__ void distr_bin(const DevParams &P, const double *tb, int kk, int g, double n,
                                          const double (&v)[SALSA_NSV], DStep &o) {
  const double *vlo = tb + TAB_VLO * P.nb_pad, *vhi = tb + TAB_VHI * P.nb_pad, *dmid = tb + TAB_DMID * P.nb_pad;
  const int nmove = (CAT == DC_ICE) ? P.nused : P.nwet;
  const int nsum = (CAT <= DC_CLOUD) ? P.ndry : nmove;
  o.dir = 0; o.target = g; o.check = false; o.within = true; o.neg = false;
  o.own_n = n; o.push_n = 0.;
#pragma unroll
  for (int s = 0; s < SALSA_NSV; s++) { o.own[s] = v[s]; o.push[s] = 0.; }
  double sd = 0.;
#pragma unroll
  for (int s = 0; s < SALSA_NSV; s++) if (s < nsum) sd += v[s];
  if (CAT == DC_AERO) {
    if (!num_gt(n, K_NLIM) || g == P.fn2a) return;
    const double zvpart = ddiv(sd, n);
    if (vlo[g] > zvpart) {
      if (g == P.in1a) return;
      o.dir = -1; o.target = (g == P.in2b) ? P.fn1a : g - 1;
      o.own_n = 0.; o.push_n = n;
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++) if (s < nmove) { o.own[s] = 0.; o.push[s] = v[s]; }
      return;
    }
    if (zvpart <= K_PI6 * cube(dmid[g])) return;
    const double zVrat = ddiv(vhi[g], vlo[g]);
    const double zVilo = ddiv(2. * zvpart, 1. + zVrat);
    const double zVihi = zVrat * zVilo;
    const double zVexc = 0.5 * (zVihi + vhi[g]);
    const double znfrac = fmin(1., ddiv(zVihi - vhi[g], zVihi - zVilo));
    const double zvfrac = fmin(0.99, ddiv(znfrac * zVexc, zvpart));
    o.neg = zvfrac < 0.;
    const double f = znfrac * n * zVexc;
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++)
      if (s < nmove) { double mv = ddiv(f * v[s], sd); o.push[s] = mv; o.own[s] = v[s] - mv; }
    o.dir = 1; o.target = g + 1;
    o.push_n = znfrac * n;
    o.own_n = n * (1. - znfrac);
    if (o.own_n > K_NLIM) {
      double s2 = 0.;
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++) if (s < nsum) s2 += o.own[s];
      const double zp = ddiv(s2, o.own_n);
      o.check = true; o.within = (vlo[g] < zp && zp < vhi[g]);
    }
    return;
  }
  const double lim = (CAT == DC_CLOUD) ? K_NLIM : K_PRLIM;
  if (!num_gt(n, lim) || (CAT == DC_CLOUD && !num_gt(sd, 1.e-30))) return;
  const double zvpart = ddiv(sd, n);
  const double zVrat = ddiv(vhi[g], vlo[g]);
  const double zVilo = ddiv(2. * zvpart, 1. + zVrat);
  const double zVihi = zVrat * zVilo;
  double zVexc, znfrac;
  if (CAT == DC_CLOUD) {
    if (zvpart < vlo[g] && (kk != P.ica_cur && kk != P.icb_cur)) {
      zVexc = 0.5 * (zVilo + vlo[g]);
      znfrac = fmin(1., ddiv(vlo[g] - zVilo, zVihi - zVilo));
      o.dir = -1;
    } else if (zvpart > vhi[g] && (kk != P.fca_cur && kk != P.fcb_cur)) {
      zVexc = 0.5 * (zVihi + vhi[g]);
      znfrac = fmin(1., ddiv(zVihi - vhi[g], zVihi - zVilo));
      o.dir = 1;
    } else {
      return;
    }
  } else {
    const int ntop = (CAT == DC_PRECP) ? P.nprc - 1 : P.nice - 1;
    const double vm = K_PI6 * cube(dmid[g]);
    const double zvdec = vm - 0.2 * (vm - vlo[g]);
    if (zvpart < zvdec && kk != 0) {
      zVexc = 0.5 * (zVilo + vlo[g]);
      znfrac = fmin(1., ddiv(vlo[g] - zVilo, zVihi - zVilo));
      o.dir = -1;
    } else if (zvpart > vm && kk != ntop) {
      zVexc = 0.5 * (zVihi + vhi[g]);
      znfrac = fmin(0.99, ddiv(zVihi - vhi[g], zVihi - zVilo));
      o.dir = 1;
    } else {
      return;
    }
  }
  o.target = g + o.dir;
  const double zvfrac = fmin(0.99, ddiv(znfrac * zVexc, zvpart));
  o.neg = zvfrac < 0.;
#pragma unroll
  for (int s = 0; s < SALSA_NSV; s++)
    if (s < nmove) { o.push[s] = zvfrac * v[s]; o.own[s] = v[s] - zvfrac * v[s]; }
  o.push_n = znfrac * n;
  o.own_n = n - znfrac * n;
  double s2 = 0.;
#pragma unroll
  for (int s = 0; s < SALSA_NSV; s++) if (s < nsum) s2 += o.own[s];
  const bool chk = (CAT == DC_PRECP) ? (o.own_n > lim) : (o.own_n > lim && s2 > 1.e-30);
  if (chk) {
    const double zp = ddiv(s2, o.own_n);
    o.check = true; o.within = (vlo[g] < zp && zp < vhi[g]);
  }
}

// Sequential part of a sweep (one thread): bins kk = from .. lo in descending order.
template <int CAT, typename KT, int LS>
__device__ void distr_serial(const DevParams &P, const WS<KT, LS> &w, const double *tb, int base, int from, int lo,
                             bool &has_check, bool &within, bool &neg) {
  const int nmove = (CAT == DC_ICE) ? P.nused : P.nwet;
  for (int kk = from; kk >= lo; kk--) {
    const int g = base + kk;
    double v[SALSA_NSV];
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++) v[s] = (s < nmove) ? w.v(s, g) : 0.;
    DStep o;
    distr_bin<CAT>(P, tb, kk, g, w.numc[g], v, o);
    if (o.dir != 0) {
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++)
        if (s < nmove) { w.v(s, o.target) = w.v(s, o.target) + o.push[s]; w.v(s, g) = o.own[s]; }
      w.numc[o.target] = w.numc[o.target] + o.push_n;
      w.numc[g] = o.own_n;
    }
    if (o.check) { has_check = true; within = o.within; }
    neg = neg || o.neg;
  }
}

// One sweep over bins lo..hi of a category (global index base + kk); hi_recv > hi when
// the bin above the sweep range can receive particles.  Returns the bin-limit flag.
template <int CAT, typename KT, int LS>
__device__ bool distr_sweep(const DevParams &P, const WS<KT, LS> &w, const double *tb, int lane, int base, int lo,
                            int hi, int hi_recv, bool &neg_flag) {
  const unsigned F = 0xffffffffu;
  const int nmove = (CAT == DC_ICE) ? P.nused : P.nwet;
  bool has_check = false, within = true, neg = false;
  if (LS == 1 || hi_recv >= 32) {
    if (lane == 0) distr_serial<CAT>(P, w, tb, base, hi, lo, has_check, within, neg);
  } else {
    const int kk = lane, g = base + lane;
    const bool inr = kk >= lo && kk <= hi_recv;
    const bool dec = kk >= lo && kk <= hi;
    double v[SALSA_NSV];
    double n = 0.;
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++) v[s] = (inr && s < nmove) ? w.v(s, g) : 0.;
    if (inr) n = w.numc[g];
    DStep o;
    if (dec) {
      distr_bin<CAT>(P, tb, kk, g, n, v, o);
    } else {
      o.dir = 0; o.target = g; o.check = false; o.within = true; o.neg = false;
      o.own_n = n; o.push_n = 0.;
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++) { o.own[s] = v[s]; o.push[s] = 0.; }
    }
    const unsigned down = __ballot_sync(F, dec && o.dir < 0);
    const int D = down ? 31 - __clz(down) : -1;
    const bool par = inr && kk >= D;
    const bool up = par && o.dir > 0;
    const bool in_up = (__shfl_up_sync(F, up ? 1 : 0, 1) != 0) && lane > 0;
    const double pn = __shfl_up_sync(F, o.push_n, 1);
    double pv[SALSA_NSV];
#pragma unroll
    for (int s = 0; s < SALSA_NSV; s++) pv[s] = __shfl_up_sync(F, o.push[s], 1);
    if (par) {
#pragma unroll
      for (int s = 0; s < SALSA_NSV; s++)
        if (s < nmove) w.v(s, g) = in_up ? o.own[s] + pv[s] : o.own[s];
      w.numc[g] = in_up ? o.own_n + pn : o.own_n;
      if (kk == D) {
#pragma unroll
        for (int s = 0; s < SALSA_NSV; s++)
          if (s < nmove) w.v(s, o.target) = w.v(s, o.target) + o.push[s];
        w.numc[o.target] = w.numc[o.target] + o.push_n;
      }
    }
    const unsigned cm = __ballot_sync(F, par && o.check);
    if (cm) within = __shfl_sync(F, o.within, __ffs(cm) - 1);
    neg = __any_sync(F, par && o.neg);
    wsync<LS>();
    if (lane == 0 && D > lo) {
      bool hc = false, wi = true;
      distr_serial<CAT>(P, w, tb, base, D - 1, lo, hc, wi, neg);
      if (hc) within = wi;
    }
  }
  wsync<LS>();
  if constexpr (LS != 1) {
    within = __shfl_sync(F, within, 0);
    neg = __shfl_sync(F, neg, 0);
  }
  neg_flag = neg_flag || neg;
  return within;
}

template <typename KT, int LS>
__device__ void distr_update(const DevParams &P, const WS<KT, LS> &w, const double *tb, int lane) {
  bool f_distr = false, f_neg = false;
#pragma unroll 1
  for (int c = 0; c < 4; c++) {
    if (c == DC_ICE && P.level < 5) break;
    bool within = false;
    int count = 0;
    while (!within) {
      switch (c) {
        case DC_AERO: within = distr_sweep<DC_AERO>(P, w, tb, lane, 0, P.in1a, P.fn2b - 1, P.fn2b, f_neg); break;
        case DC_CLOUD: within = distr_sweep<DC_CLOUD>(P, w, tb, lane, P.nbins, P.ica_cur, P.ncld - 1, P.ncld - 1, f_neg); break;
        case DC_PRECP: within = distr_sweep<DC_PRECP>(P, w, tb, lane, P.nbins + P.ncld, 0, P.nprc - 1, P.nprc - 1, f_neg); break;
        default: within = distr_sweep<DC_ICE>(P, w, tb, lane, P.nliquid, 0, P.nice - 1, P.nice - 1, f_neg); break;
      }
      if (++count > 100) { f_distr = true; break; }
    }
  }
  if (lane == 0) {
    if (f_distr) w.misc[M_FLAGS + F_DISTR] = 1.;
    if (f_neg) w.misc[M_FLAGS + F_NEGFRAC] = 1.;
  }
  wsync<LS>();
}


// ----------------------------------------------------------------------------------------
// One cell: the body of the run_SALSA cell loop (mo_salsa_driver.f90:185-419) around
// salsa() (mo_salsa.f90:89-149).  Every cell starts from the post-initialisation module
// state (bin templates), i.e. each cell sees allSALSA as the reference's first cell does.
// Inlined into the kernel with everything it calls: a call would pass the workspace
// descriptor by reference through the stack, and the callee would reload its pointers
// from local memory (the mixed form ran 10-14 % slower that way).
// ----------------------------------------------------------------------------------------
#ifdef SALSA_STAGE_TIMERS
#define STAGE_MARK(k)                                                              \
  do {                                                                             \
    long long t_ = clock64();                                                      \
    if ((threadIdx.x & 31) == 0 && P.stage_clocks) atomicAdd(P.stage_clocks + (k), (unsigned long long)(t_ - t_stage)); \
    t_stage = t_;                                                                  \
  } while (0)
#else
#define STAGE_MARK(k) do { } while (0)
#endif

// The lane form's warps of a block meet between the stages: a stage's code then stays in the
// instruction cache while they run it (without the meetings a 1.1 M-cell block of
// grid384x384x160 took 127 ms instead of 105, with each warp on a tile of its own 179 ms).
template <int LS> __device__ __forceinline__ void stage_sync() {
  if constexpr (LS == 1) { __syncwarp(); __syncthreads(); }
}
// ---- the lane form's unit conversion, straight between the fields and the workspace ----
// x a and x a b, without FP64 products for the zeros of unpopulated bins (rounded as in the
// warp form: the substeps magnify last-bit differences of the water); z = 0 a, NaN when a is
// not finite
__device__ __forceinline__ double scaled(double x, double a, double z) { return __double_as_longlong(x) == 0 ? z : x * a; }
__device__ __forceinline__ double scaled(double x, double a, double b, double z) {
  return __double_as_longlong(x) == 0 ? z : x * a * b;
}

// (mo_salsa_driver.f90:196-283) the cell's bins in particles and volume per m3 of air
template <typename KT>
__device__ __forceinline__ void lane_unpack(const DevParams &P, const WS<KT, 1> &w, const double *dmid, double dn) {
  const double zero = 0. * dn;
  int b0 = 0;
#pragma unroll 1
  for (int c = 0; c < 4; c++) {
    const int nb = c == 0 ? P.nbins : (c == 1 ? P.ncld : (c == 2 ? P.nprc : P.nice));
    const bool absent = c == 3 && P.level < 5;
    const double *fn = absent ? nullptr : P.fin[FI_NAERO + c] + w.off;
    const double *fi = c < 3 && P.raw_indef >= 0 ? P.fin[FI_INDEF] + w.off : nullptr;
    const double *fc = c < 3 && P.fin[FI_CHARGE] ? P.fin[FI_CHARGE] + w.off : nullptr;
#pragma unroll 4
    for (int b = 0; b < nb; b++) {
      const int g = b0 + b;
      const double n = fn ? __ldg(fn + P.plane * b) : 0.;
      const double d = fi ? __ldg(fi + P.plane * g) : 0.;
      const double t = fc ? __ldg(fc + P.plane * g) : 0.;
      w.dwet[g] = dmid[g];
      w.ddry[g] = 0.;
      w.dins[g] = 0.;
      w.dnsp[g] = 0.;
      w.numc[g] = absent ? 0. : scaled(n, dn, zero);
      w.indef[g] = d;
      w.ctime[g] = t;
    }
    const int ns = absent ? 0 : (c == 3 ? P.nwet + 1 : P.nwet);
    const double *fm = absent ? nullptr : P.fin[FI_MAERO + c] + w.off;
#pragma unroll 1
    for (int s = 0; s < P.nused; s++) {
      const double irho = c < 3 ? P.irholiq[s] : (s < P.nwet ? P.irhoice[s] : 1. / K_RHORI);
      const double *f = s < ns ? fm + P.plane * ((long long)s * nb) : nullptr;
#pragma unroll 8
      for (int b = 0; b < nb; b++) w.v(s, b0 + b) = f ? scaled(__ldg(f + P.plane * b), dn, irho, zero) : 0.;
    }
    for (int b = 0; b < nb; b++) {
      const int g = b0 + b;
      w.rhomean[g] = absent ? 0. : rhomean_of(P, c + 1, w.numc[g], w.v(P.iwa, g), w.v(P.irim, g));
    }
    b0 += nb;
  }
}

// (mo_salsa_driver.f90:310-349) tendencies (new - old) / dt into the fields, the IN deficit
// and the charge times in place; returns whether a number is not finite
template <typename KT>
__device__ __forceinline__ bool lane_output(const DevParams &P, const WS<KT, 1> &w, double idn) {
  const double dt = P.dt, idt = P.inv_dt != 0. ? P.inv_dt : drcp(dt);
  const long long degenerate = (__double_as_longlong(idn) & FM_INF) == FM_INF;   // no finite 1/dn: 0/dn is NaN
  auto add = [&](double *f, double x, double v, double rho) {   // f += (v rho / dn - x) / dt
    if ((__double_as_longlong(v) | __double_as_longlong(x) | degenerate) == 0 || !w.live) return;
    const double d = (v * rho * idn) - x;
    *f = *f + (P.inv_dt != 0. ? d * idt : ddiv_r(d, dt, idt));
  };
  bool bad = false;
  int b0 = 0;
#pragma unroll 1
  for (int c = 0; c < 4; c++) {
    const int nb = c == 0 ? P.nbins : (c == 1 ? P.ncld : (c == 2 ? P.nprc : P.nice));
    if (c == 3 && P.level < 5) break;
    const double *fn = P.fin[FI_NAERO + c] + w.off;
    double *tn = P.fout[FO_NAEROT + c] + w.off;
#pragma unroll 4
    for (int b = 0; b < nb; b++) {
      const double n = w.numc[b0 + b];
      bad |= (__double_as_longlong(n) & FM_INF) == FM_INF;
      add(tn + P.plane * b, __ldg(fn + P.plane * b), n, 1.);
    }
    const int ns = c == 3 ? P.nwet + 1 : P.nwet;
    const double *fm = P.fin[FI_MAERO + c] + w.off;
    double *tm = P.fout[FO_MAEROT + c] + w.off;
#pragma unroll 1
    for (int s = 0; s < ns; s++) {
      const double rho = c < 3 ? P.rholiq[s] : (s < P.nwet ? P.rhoice[s] : K_RHORI);
      const long long r = P.plane * ((long long)s * nb);
#pragma unroll 4
      for (int b = 0; b < nb; b++) add(tm + r + P.plane * b, __ldg(fm + r + P.plane * b), w.v(s, b0 + b), rho);
    }
    if (c < 3 && w.live) {
      double *oi = P.raw_indef >= 0 ? P.fout[FO_INDEF] : nullptr, *oc = P.fout[FO_CHARGE];
      for (int b = b0; b < b0 + nb; b++) {
        if (oi) oi[w.off + P.plane * b] = w.indef[b];
        if (oc) oc[w.off + P.plane * b] = w.ctime[b];
      }
    }
    b0 += nb;
  }
  return bad;
}

template <typename KT, bool SIP, int LS>
__device__ __forceinline__ void cell_step(const DevParams &P, WS<KT, LS> &w, const double *tb, long long cell,
                                          int lane) {
#ifdef SALSA_STAGE_TIMERS
  long long t_stage = clock64();
#endif
  const double *dmid = tb + TAB_DMID * P.nb_pad;
  const auto raw = w.raw;
  const double T = raw[RW_T], pres = raw[RW_P], rs = raw[RW_RS], rsi = raw[RW_RSI], dn = raw[RW_DN];
  const double kappa = raw[RW_KAPPA];
  const double dt = P.dt;
  double rv = P.st_freeRH ? raw[RW_RV] : fmin(raw[RW_RV], rs * P.rhlim);
  const double rv_old = rv;
  const int nwet = P.nwet, irim = P.irim;
  const int bstart[4] = {0, P.nbins, P.nbins + P.ncld, P.nliquid};
  const int bnum[4] = {P.nbins, P.ncld, P.nprc, P.nice};
  const int ncat = P.level == 5 ? 4 : 3;
  const int m0 = P.raw_mbase[0];
  const int nmrow = (ncat == 4 ? P.raw_mbase[3] + (nwet + 1) * P.nice : P.raw_mbase[2] + nwet * P.nprc) - m0;
  if constexpr (LS == 1) {
    lane_unpack(P, w, dmid, dn);
  } else {
    for (int b = lane; b < P.ntotal; b += LS) {
      int icat = phase_of(P, b) - 1;
      w.dwet[b] = dmid[b];
      w.ddry[b] = w.dins[b] = w.dnsp[b] = 0.;
      for (int s = 0; s < SALSA_NSV; s++) w.v(s, b) = 0.;
      const bool absent = icat == 3 && P.level < 5;
      w.numc[b] = absent ? 0. : raw[P.raw_num + b] * dn;
      w.indef[b] = (!absent && icat < 3 && P.raw_indef >= 0) ? raw[P.raw_indef + b] : 0.;
      w.ctime[b] = (!absent && icat < 3 && P.raw_charge >= 0) ? raw[P.raw_charge + b] : 0.;
    }
    wsync<LS>();
    // mass rows of all categories, one lane per (category, species, bin) row
    for (int e = lane; e < nmrow; e += LS) {
      const int r = m0 + e;
      const int icat = (ncat == 4 && r >= P.raw_mbase[3]) ? 3 : (r >= P.raw_mbase[2] ? 2 : (r >= P.raw_mbase[1] ? 1 : 0));
      const int loc = r - P.raw_mbase[icat], nbc = bnum[icat];
      const int sp = loc / nbc, b = bstart[icat] + (loc - sp * nbc);
      const double irho = icat < 3 ? P.irholiq[sp] : (sp < nwet ? P.irhoice[sp] : 1. / K_RHORI);
      w.v(sp, b) = raw[r] * dn * irho;
    }
    wsync<LS>();
    for (int b = lane; b < P.ntotal; b += LS) {
      int icat = phase_of(P, b) - 1;
      w.rhomean[b] = (icat == 3 && P.level < 5) ? 0. : rhomean_of(P, icat + 1, w.numc[b], w.v(P.iwa, b), w.v(irim, b));
    }
  }
  for (int i = lane; i < M_PF; i += LS) w.misc[i] = 0.;
  wsync<LS>();
  if constexpr (SIP) {
    if (P.st_secice) sip_clear<KT>(P, w, dn, lane);
  }
  if (P.initialize) equilibration<KT>(P, w, tb, 0.3, T, true, lane);
  // gases in #/m3 (mo_salsa_driver.f90:285-290)
  if (P.raw_gas >= 0)
    for (int i = lane; i < 5; i += LS) w.misc[M_GAS + i] = raw[P.raw_gas + i] * dn;
  stage_sync<LS>();
  STAGE_MARK(0);

  // ---- salsa() ----
  if (P.st_coag) coagulation<KT, SIP>(P, w, tb, dt, T, pres, true, cell, lane);
  if constexpr (SIP) {
    if (P.st_secice) secondary_ice<KT>(P, w, tb, T, pres, rv, rsi, dt, lane);
  }
  stage_sync<LS>();
  STAGE_MARK(1);
  if (P.st_cnd) {
    // condensation (mo_salsa_dynamics.f90:276-342): nucleation returns only the 3 nm
    // formation rates, which condgas does not read, and the H2SO4 fraction of the
    // clusters: 1 for nsnucl = 1-3; for the mixed schemes it only multiplies condgas's
    // vanishing nucleation term, and 1 stands in
    if (P.lscndgas) condgas<KT>(P, w, tb, T, pres, dt, w.misc + M_GAS, P.nsnucl > 0 ? 1. : 0., lane);
    if (P.lscndh2ocl || P.lscndh2oae || P.lscndh2oic) gpparth2o<KT>(P, w, tb, T, pres, rs, rsi, rv, dt, kappa, true, lane);
  }
  stage_sync<LS>();
  STAGE_MARK(2);
  if (P.st_auto && P.auto_mode == 2) autoconv2<KT>(P, w, dt, lane);
  if (P.st_activ && P.activ_mode == 1) act_interst<KT>(P, w, tb, rv, rs, T, true, lane);
  if (P.st_activ && P.activ_mode == 2) act_cloudbase<KT>(P, w, tb, pres, T, raw[RW_W], dn, raw, lane);
  stage_sync<LS>();
  STAGE_MARK(3);
  if ((P.st_icenucl || P.icenucl_mode == 2) && (P.lsicehom || P.lsiceimm || P.lsicedep)) {
    if (P.ice_theta_dist) ice_nucl_SE<KT>(P, w, tb, T, rv, rs, rsi, dt, kappa, true, lane);
    else ice_nucl_classic<KT>(P, w, tb, T, rv, rs, rsi, dt, kappa, true, lane);
  }
  if constexpr (SIP) {
    // ice_melt's bins (numbers not below prlim) before it runs: their tracers melt with them
    if (P.st_secice && P.st_icemelt) {
      const auto s = sip_tallies(P, w.raw);
      for (int k = lane; k < P.nice; k += LS) s.melt[k] = w.numc[P.nliquid + k] < K_PRLIM ? 0. : 1.;
      wsync<LS>();
    }
  }
  if (P.st_icemelt) ice_melt<KT>(P, w, tb, T, lane);
  if constexpr (SIP) {
    if (P.st_secice && P.st_icemelt && T >= 273.15) {   // mo_salsa_cloud_ice.f90:453-456
      const auto s = sip_tallies(P, w.raw);
      for (int e = lane; e < 3 * P.nice; e += LS)
        if (s.melt[e % P.nice] != 0.) s.tr[e] = (1. - 0.999) * s.tr[e];
      wsync<LS>();
    }
  }
  stage_sync<LS>();
  STAGE_MARK(4);
  if (P.lsdistupdate) distr_update<KT>(P, w, tb, lane);
  stage_sync<LS>();
  STAGE_MARK(5);

  // ---- tendencies and outputs (mo_salsa_driver.f90:310-419) into the raw slots ----
  // (x / dn - old) / dt: one division for 1/dn per cell, and the quotient by dt as a
  // product when dt is a power of two (then it is the same number)
  bool bad = false;
  const double idn = drcp(dn);
  if constexpr (LS == 1) {
    bad = lane_output(P, w, idn);
  } else {
    for (int e = lane; e < nmrow; e += LS) {
      const int r = m0 + e;
      const int icat = (ncat == 4 && r >= P.raw_mbase[3]) ? 3 : (r >= P.raw_mbase[2] ? 2 : (r >= P.raw_mbase[1] ? 1 : 0));
      const int loc = r - P.raw_mbase[icat], nbc = bnum[icat];
      const int sp = loc / nbc, b = bstart[icat] + (loc - sp * nbc);
      const double rho = icat < 3 ? P.rholiq[sp] : (sp < nwet ? P.rhoice[sp] : K_RHORI);
      const double d = (w.v(sp, b) * rho * idn) - raw[r];
      raw[r] = P.inv_dt != 0. ? d * P.inv_dt : ddiv(d, dt);
    }
    for (int b = lane; b < P.ntotal; b += LS) {
      int icat = phase_of(P, b) - 1;
      if (icat == 3 && P.level < 5) continue;
      if (icat < 3) {
        if (P.raw_indef >= 0) raw[P.raw_indef + b] = w.indef[b];
        if (P.raw_charge >= 0) raw[P.raw_charge + b] = w.ctime[b];
      }
      double &on = raw[P.raw_num + b];
      const double d = (w.numc[b] * idn) - on;
      on = P.inv_dt != 0. ? d * P.inv_dt : ddiv(d, dt);
      bad |= !isfinite(w.numc[b]);
    }
  }
  // interstitial activation leaves the activated-droplet outputs at zero (:879, local pactd);
  // cloud-base activation has written them
  if (LS != 1 && !(P.st_activ && P.activ_mode == 2))
    for (int i = lane; i < P.ncld * (1 + nwet); i += LS) raw[P.raw_nact + i] = 0.;
  if (lane == 0) raw[RW_RV] = ddiv(rv - rv_old, dt);
  if constexpr (SIP) {
    if (P.st_secice) {   // :345-349 and :412-416
      const auto s = sip_tallies(P, w.raw);
      for (int e = lane; e < 3 * P.nice; e += LS) raw[P.raw_sip + e] = ddiv(s.tr[e], dn);
      if (P.raw_diag >= 0)
        for (int e = lane; e < 3; e += LS) raw[P.raw_diag + SALSA_DIAG_SIPDRFR_SLOT + e] = ddiv(s.rate[e], dn);
    }
  }
  if (P.raw_gas >= 0)   // :369-384
    for (int i = lane; i < 5; i += LS)
      raw[P.raw_gas + i] = ddiv((ddiv(w.misc[M_GAS + i], dn)) - raw[P.raw_gas + i], dt);
  if (P.raw_diag >= 0 && lane == 0) {
    const auto d = w.misc + M_DIAG;
    const auto o = raw + P.raw_diag;
    o[DG_AUTOC] = ddiv(d[DG_AUTOC] * K_RHOWA, dn);
    o[DG_AUTOC80] = ddiv(d[DG_AUTOC80] * K_RHOWA, dn);
    o[DG_AUTOC50] = ddiv(d[DG_AUTOC50] * K_RHOWA, dn);
    o[DG_ACCR] = ddiv(d[DG_ACCR] * K_RHOWA, dn);
    o[DG_ACCR80] = ddiv(d[DG_ACCR80] * K_RHOWA, dn);
    o[DG_ACCR50] = ddiv(d[DG_ACCR50] * K_RHOWA, dn);
    o[DG_ACCOLL] = ddiv(d[DG_ACCOLL], dn);
    o[DG_APCOLL] = ddiv(d[DG_APCOLL], dn);
    o[DG_ACTIV] = ddiv(d[DG_ACTIV], dn);
    o[DG_CONDA] = ddiv(d[DG_CONDA], dn);
    o[DG_CONDC] = ddiv(d[DG_CONDC], dn);
    o[DG_CONDP] = ddiv(d[DG_CONDP], dn);
    if (P.level == 5) {
      o[DG_AICOLL] = 0.;   // AIcoll%volc is never accumulated on this path (coag_ice uses the phase-change source)
      o[DG_ICEHOM] = ddiv(d[DG_ICEHOM], dn);
      o[DG_ICEDEP] = ddiv(d[DG_ICEDEP], dn);
      o[DG_ICEIMM] = ddiv(d[DG_ICEIMM], dn);
      o[DG_CONDI] = ddiv(d[DG_CONDI], dn);
    }
  }
  bad = wany<LS>(bad);
  stage_sync<LS>();
  STAGE_MARK(6);
  if (lane == 0 && P.status && w.live) {
    const auto f = w.misc + M_FLAGS;
    if (f[F_EQUIL] != 0.) atomicAdd(P.status + ST_EQUIL, 1ull);
    if (f[F_DISTR] != 0.) atomicAdd(P.status + ST_DISTR, 1ull);
    if (f[F_NEGFRAC] != 0.) atomicAdd(P.status + ST_NEGFRAC, 1ull);
    if (f[F_COND] != 0.) atomicAdd(P.status + ST_COND, 1ull);
    if (f[F_NEG] != 0.) atomicAdd(P.status + ST_NEG, 1ull);
    if (bad) atomicAdd(P.status + ST_NONFINITE, 1ull);
  }
  wsync<LS>();
}

template <typename KT, int LS>
__device__ __forceinline__ WS<KT, LS> make_ws(const DevParams &P, Ptr<double, LS> base) {
  WS<KT, LS> w;
  w.am0 = ~0ull;
  w.am1 = ~0u;
  w.live = true;
  const int NB = P.nb_pad;
  w.NB = NB;
  Ptr<double, LS> p = base;
  w.raw = p; p = p + ((P.nraw + 1) & ~1);
  w.numc = p; p = p + NB;
  w.volc = p; p = p + SALSA_NSV * NB;
  w.dwet = p; p = p + NB;
  w.ddry = p; p = p + NB;
  w.dins = p; p = p + NB;
  w.dnsp = p; p = p + NB;
  w.rhomean = p; p = p + NB;
  w.indef = p; p = p + NB;
  w.ctime = p; p = p + NB;
  w.scr = p; p = p + SALSA_NSCR * NB;
  w.nf = row_cast<float>(w.scr);   // NB floats, then SALSA_NSV * NB floats (4 scratch rows)
  w.vf = w.nf + NB;
  w.misc = p; p = p + SALSA_MISC_DOUBLES;
  if constexpr (LS != 1) w.pbuf = reinterpret_cast<int *>(p);
  p = p + 64;   // 128 ints: bin lists (<= 96) and pair batches (<= 63)
  w.K = row_cast<KT>(p);
  if constexpr (LS == 1 && sizeof(KT) == 4) w.lf = row_cast<float>(base + P.ws_doubles);
  return w;
}


template <typename KT, bool SIP>
__global__ void __launch_bounds__(SALSA_THREADS, 2) salsa_step_kernel(const DevParams P) {
  extern __shared__ double smem[];
  if (P.choose && lane_pays(P)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double *tb = smem;
  for (int i = tid; i < P.tab_doubles; i += SALSA_THREADS) tb[i] = P.tables[i];
  double *wsbase = smem + P.tab_doubles;
  WS<KT, 32> w = make_ws<KT, 32>(P, wsbase + (size_t)warp * P.ws_doubles);
  __syncthreads();
  for (long long g = blockIdx.x; g < P.ngroups; g += gridDim.x) {
    // stage the group's input rows: consecutive threads read the group's cells of one row
    const int c = tid % SALSA_CPG;
    const long long qc = g * SALSA_CPG + c;
    const bool okc = qc < P.ncells;
    const long long offc = okc ? cell_offset(P, cell_at(P, qc)) : 0;
    if (okc)
      for (int r = tid / SALSA_CPG; r < P.nrows; r += SALSA_THREADS / SALSA_CPG) {
        const Row row = P.rows[r];
        double v = 0.;
        if (row.fin >= 0) {
          const double *f = P.fin[row.fin];
          if (f) v = __ldg(f + offc + P.plane * row.idx);
        }
        wsbase[(size_t)c * P.ws_doubles + r] = v;
      }
    __syncthreads();
    long long q = g * SALSA_CPG + warp;
    if (q < P.ncells) cell_step<KT, SIP>(P, w, tb, cell_at(P, q), lane);
    __syncthreads();
    // write the group's output rows
    if (okc)
      for (int r = tid / SALSA_CPG; r < P.nrows; r += SALSA_THREADS / SALSA_CPG) {
        const Row row = P.rows[r];
        if (row.fout < 0) continue;
        double *f = P.fout[row.fout];
        if (!f) continue;
        const double v = wsbase[(size_t)c * P.ws_doubles + r];
        double *a = f + offc + P.plane * row.idx;
        if (row.mode == ROW_TEND) *a = *a + v;
        else *a = v;
      }
    if (tid == 0 && P.status) atomicAdd(P.status + ST_CELLS, (unsigned long long)min((long long)SALSA_CPG, P.ncells - g * SALSA_CPG));
    __syncthreads();
  }
}

// The lane form: one cell per lane, a warp's 32 cells side by side from the order list.  Every
// FP64 instruction then serves 32 cells, where the warp form leaves half of the lanes idle,
// adds up partial sums across them and repeats per-cell scalars on all of them; the FP64 pipe
// takes as long for one active lane as for 32.  The workspaces (about 25 KB a cell) live in
// global memory, a slot per resident warp, interleaved by lane: HBM and L2 have bandwidth to
// spare (they are 5-15 % busy).  Blocks take four tiles of 32 cells at a time, the cloudy end
// of the list first (its cells take several times as long as clear ones): the first ones by
// block index, which puts the cloudy tiles of a small call on different SMs, the others from
// a counter.  With the counter alone the blocks that start first, those of the same SMs, took
// them all: grid384x384x160 with 10 % of the cells cloudy, scattered, took 13.1 ms at 24,576
// cells and 18.3 at 49,152 (the warp form 6.1 and 12.4); now 9.6 and 10.5.
// FP64 instructions per cell of grid384x384x160: 6,190 in the warp form, about 1,000 here; a
// 1.1 M cell block takes 76 ms, where the warp form took 299 ms (FP32-mixed: 69 and 226 ms).  Four blocks of 128 threads
// per SM (128 registers) measured better than three (164 registers): clear cells 39.3
// against 43.9 ns a cell, cloudy ones 397 against 455 (372 since); the FP64 pipe is 71-80 %
// busy.
template <typename KT, bool SIP>
__global__ void __launch_bounds__(32 * SALSA_LANE_WARPS, SALSA_LANE_MINBLOCKS) salsa_lane_kernel(const DevParams P) {
  extern __shared__ double smem[];
  if (P.choose && !lane_pays(P)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double *tb = smem;
  for (int i = tid; i < P.tab_doubles; i += 32 * SALSA_LANE_WARPS) tb[i] = P.tables[i];
  __syncthreads();
  WS<KT, 1> w = make_ws<KT, 1>(
      P, Col<double>{P.lane_ws + ((size_t)blockIdx.x * SALSA_LANE_WARPS + warp) * (size_t)P.lane_rows * 32 + lane});
  const long long ntiles = (P.ncells + 31) / 32;
  __shared__ unsigned long long next;
  for (bool first = true;; first = false) {
    // the block's warps take neighbouring tiles together, the first ones by block index (see above)
    if (tid == 0)
      next = first ? (unsigned long long)blockIdx.x * SALSA_LANE_WARPS
                   : (unsigned long long)gridDim.x * SALSA_LANE_WARPS +
                         atomicAdd(P.status + ST_TILE, (unsigned long long)SALSA_LANE_WARPS);
    __syncthreads();
    const long long k0 = (long long)next, k = k0 + warp;
    __syncthreads();
    if (k0 >= ntiles) break;
    // warps past the last tile repeat it
    const long long q = (ntiles - 1 - min(k, ntiles - 1)) * 32 + lane;
    w.live = k < ntiles && q < P.ncells;
    const long long cell = cell_at(P, min(q, P.ncells - 1));
    w.off = cell_offset(P, cell);
    // thermodynamics, gases and tracers through the workspace; the bins in lane_unpack
    auto stage = [&](int r0, int r1) {
#pragma unroll 4
      for (int r = r0; r < r1; r++) {
        const Row row = P.rows[r];
        const double *f = row.fin >= 0 ? P.fin[row.fin] : nullptr;
        w.raw[r] = f ? __ldg(f + w.off + P.plane * row.idx) : 0.;
      }
    };
    const bool nact0 = !(P.st_activ && P.activ_mode == 2);   // no activated droplets to report
    stage(0, P.raw_num);
    stage(nact0 ? P.raw_diag : P.raw_nact, P.nrows);
    cell_step<KT, SIP>(P, w, tb, cell, 0);
    __syncwarp();
    if (w.live) {
      for (int r = 0; r < P.nrows; r = r + 1 == P.raw_num ? P.raw_nact : r + 1) {
        const Row row = P.rows[r];
        double *f = row.fout >= 0 ? P.fout[row.fout] : nullptr;
        if (!f) continue;
        double *o = f + w.off + P.plane * row.idx;
        const double v = nact0 && r >= P.raw_nact && r < P.raw_diag ? 0. : w.raw[r];
        *o = row.mode == ROW_TEND ? *o + v : v;
      }
    }
    const unsigned nlive = __popc(__ballot_sync(0xffffffffu, w.live));
    if (lane == 0) atomicAdd(P.status + ST_LANE_CELLS, (unsigned long long)nlive);
  }
}

// Host-side launch helpers, instantiated per form in salsa_k_*.cu.
inline size_t smem_bytes(const DevParams &P) {
  return sizeof(double) * ((size_t)P.tab_doubles + (size_t)SALSA_CPG * P.ws_doubles);
}

template <typename KT, bool SIP = false>
cudaError_t launch_t(const DevParams &P, cudaStream_t st, int grid) {
  size_t sm = smem_bytes(P);
  cudaError_t e =
      cudaFuncSetAttribute(salsa_step_kernel<KT, SIP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  salsa_step_kernel<KT, SIP><<<grid, SALSA_THREADS, sm, st>>>(P);
  return cudaGetLastError();
}

template <typename KT, bool SIP = false>
cudaError_t launch_lane_t(const DevParams &P, cudaStream_t st, int grid) {
  salsa_lane_kernel<KT, SIP><<<grid, 32 * SALSA_LANE_WARPS, sizeof(double) * (size_t)P.tab_doubles, st>>>(P);
  return cudaGetLastError();
}
template <typename KT, bool SIP = false>
int lane_blocks_per_sm_t(const DevParams &P) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, salsa_lane_kernel<KT, SIP>, 32 * SALSA_LANE_WARPS,
                                                    sizeof(double) * (size_t)P.tab_doubles) != cudaSuccess)
    return 0;
  return nb;
}

template <typename KT, bool SIP = false>
int blocks_per_sm_t(const DevParams &P) {
  size_t sm = smem_bytes(P);
  if (cudaFuncSetAttribute(salsa_step_kernel<KT, SIP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) !=
      cudaSuccess)
    return 0;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, salsa_step_kernel<KT, SIP>, SALSA_THREADS, sm) !=
      cudaSuccess)
    return 0;
  return nb;
}

}  // namespace
}  // namespace salsa
