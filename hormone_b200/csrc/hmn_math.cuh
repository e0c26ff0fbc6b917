// hmn_math.cuh -- per-cell and per-face arithmetic of HORMONE's explicit step,
// in the operation order of the Fortran reference (every product, sum and
// quotient below is one IEEE binary64 operation; the including translation
// unit is compiled with --fmad=false so nothing is fused).
//
// Reference routines (paths in the HORMONE tree):
//   minmod / modified_mc   src/main/fluxlimiter.f90:40-56, 58-75
//   get_eint               src/main/eos.f90:846-866
//   get_cf                 src/main/eos.f90:351-365
//   eos_p_cs (ideal gas)   src/main/eos.f90:195-242
//   hlldflux + fstar       src/main/hlldflux.f90:19-179
#pragma once
#include <cuda_runtime.h>

namespace hmn {

// Fortran SIGN(a,b): |a| with the sign bit of b (honours -0).
template <typename T>
__device__ __forceinline__ T fsign(T a, T b) { return copysign(fabs(a), b); }
// MIN/MAX in the argument order the reference evaluates them.
template <typename T>
__device__ __forceinline__ T fmin2(T a, T b) { return a < b ? a : b; }
template <typename T>
__device__ __forceinline__ T fmax2(T a, T b) { return a > b ? a : b; }

// Division policies: div(a, b, r) is a/b, where r = rec(b) was formed once
// for every quotient with the denominator b, and root(x) is sqrt(x).
// PlainDiv divides (r is b itself); FastDiv (hmn_div.cuh) forms RN(1/b) once
// and corrects each quotient to RN(a/b), flagging operands it cannot take.
// FastDiv takes positive denominators only, so expressions are written with
// the positive one of b and -b (negating both operands changes no bit of the
// quotient).
struct PlainDiv {
  static constexpr bool flags = false;
  template <int LO, int HI, typename T>
  __device__ __forceinline__ void need_pos(T) {}
  template <int HI, typename T>
  __device__ __forceinline__ void need_below(T) {}
  template <typename T>
  __device__ __forceinline__ T rec(T b) { return b; }
  template <typename T>
  __device__ __forceinline__ T div(T a, T b, T) { return a / b; }
  template <typename T>
  __device__ __forceinline__ T root(T x) { return sqrt(x); }
};

// x with its sign flipped where s is negative: sign(1, s) * x, exactly.
__device__ __forceinline__ double flip(double x, double s) {
  return __hiloint2double(__double2hiint(x) ^ (__double2hiint(s) & (int)0x80000000), __double2loint(x));
}

// Generalised minmod with theta = 1.4 on inverse spacings (fluxlimiter.f90:40-56).
// i0 = 1/dx(c), i1 = 1/dx(c+1), isum = i0 + i1; risum = dv.rec(isum).  The
// reference multiplies by sign(1, x); that product is a flip of the sign bit,
// and a factor taken as |x| costs nothing, so four FP64 multiplications per
// variable become three logic operations (here as in lim_mmc, where the
// quotient's numerator takes its sign by copysign).
template <class D>
__device__ __forceinline__ double lim_minmod(double u0, double u1, double u2, double i0, double i1, double isum,
                                             D& dv, double risum) {
  const double x = 1.4 * (u2 - u1) * i1;
  const double y = 1.4 * (u1 - u0) * i0;
  const double z = dv.div((u2 - u0) * i0 * i1, isum, risum);
  double m = fabs(x);
  m = fmin2(m, flip(y, x));
  m = fmin2(m, flip(z, x));
  return copysign(fmax2(0.0, m), x);
}
__device__ __forceinline__ double lim_minmod(double u0, double u1, double u2, double i0, double i1, double isum) {
  PlainDiv dv;
  return lim_minmod(u0, u1, u2, i0, i1, isum, dv, isum);
}

// Modified MC (fluxlimiter.f90:58-75).  Grid factors precomputed per cell:
// cf = (x(c+1)-x(c))/(xi(c)-x(c)), cb = (x(c)-x(c-1))/(x(c)-xi(c-1)),
// ga = x(c+1)-x(c), gb = x(c)-x(c-1).
// With a division policy: rga = dv.rec(ga), rgb = dv.rec(gb).
template <class D>
__device__ __forceinline__ double lim_mmc(double u0, double u1, double u2, double cf, double cb, double ga, double gb,
                                          D& dv, double rga, double rgb) {
  const double bot = u2 - u1, a = fabs(bot);
  const double t = flip(dv.div((u1 - u0) * ga, gb, rgb), bot);
  double m = 0.5 * (a + t);
  m = fmin2(m, cf * a);
  m = fmin2(m, cb * t);
  return dv.div(copysign(fmax2(0.0, m), bot), ga, rga);
}
__device__ __forceinline__ double lim_mmc(double u0, double u1, double u2, double cf, double cb, double ga,
                                          double gb) {
  PlainDiv dv;
  return lim_mmc(u0, u1, u2, cf, cb, ga, gb, dv, ga, gb);
}

// Internal energy from total energy (eos.f90:846-866).
template <bool MAG>
__device__ __forceinline__ double get_eint(double etot, double d, double v1, double v2, double v3, double b1,
                                           double b2, double b3) {
  double vsq = v1 * v1 + v2 * v2 + v3 * v3;
  double ei = etot - 0.5 * d * vsq;
  if (MAG) {
    double bsq = b1 * b1 + b2 * b2 + b3 * b3;
    ei = ei - 0.5 * bsq;
  }
  return ei;
}

// Fast magnetosonic speed along b1 (eos.f90:351-365); rd = dv.rec(d).
template <typename T, class D>
__device__ __forceinline__ T get_cf(T d, T cs, T b1, T b2, T b3, D& dv, T rd) {
  T asq = cs * cs;
  T bb1 = dv.div(b1 * b1, d, rd);
  T bb2 = dv.div(b2 * b2, d, rd);
  T bb3 = dv.div(b3 * b3, d, rd);
  T bbsq = bb1 + bb2 + bb3;
  T t = asq + bbsq;
  return dv.root(T(0.5) * (t + dv.root(t * t - T(4.0) * asq * bb1)));
}
template <typename T>
__device__ __forceinline__ T get_cf(T d, T cs, T b1, T b2, T b3) {
  T asq = cs * cs;
  T bb1 = b1 * b1 / d;
  T bb2 = b2 * b2 / d;
  T bb3 = b3 * b3 / d;
  T bbsq = bb1 + bb2 + bb3;
  T t = asq + bbsq;
  return sqrt(T(0.5) * (t + sqrt(t * t - T(4.0) * asq * bb1)));
}

// Face flux of one interface: HLLD (Miyoshi & Kusano 2005) with the GLM mixing
// of the normal field and phi (hlldflux.f90:19-150), then the flux of the
// selected state (fstar, hlldflux.f90:156-179).  f[0..8] = mass, normal and
// two tangential momenta, energy, phi-flux (normal B), two tangential B,
// ch^2*B_n.  rch = 1/ch, correctly rounded (the same for every face of a
// launch).  T = double in the FP64 path; the mixed-precision path
// instantiates it for float.
template <typename T, class D>
__device__ __forceinline__ void hlld(T f[9], T cfl, T cfr, T v1l, T v1r, T v2l, T v2r, T v3l, T v3r, T dl, T dr, T el,
                                     T er, T ptl, T ptr, T b1l, T b1r, T b2l, T b2r, T b3l, T b3r, T phil, T phir,
                                     T ch, T rch, D& dvp) {
  const T h = T(0.5), one = T(1.0), zero = T(0.0);
  const T b1 = h * ((b1l + b1r) - dvp.div(phir - phil, ch, rch));
  const T phi = h * ((phil + phir) - (b1r - b1l) * ch);
  const T sl = fmin2(fmin2(v1r - cfr, v1l - cfl), zero);
  const T sr = fmax2(fmax2(v1r + cfr, v1l + cfl), zero);
  const T wl = sl - v1l, wr = sr - v1r;  // S - v on each side
  const T den = wr * dr - wl * dl;
  const T rden = dvp.rec(den);
  const T sm = dvp.div(wr * dr * v1r - wl * dl * v1l - ptr + ptl, den, rden);
  // FastDiv takes the left wave distance as sm - sl, which is positive (sl -
  // sm otherwise: the FP32 solver's rounding depends on how it is written)
  constexpr bool pos = D::flags;
  const T smsl = pos ? sm - sl : sl - sm, srsm = sr - sm;
  const T rsmsl = dvp.rec(smsl), rsrsm = dvp.rec(srsm);
  const T dla0 = dvp.div(pos ? -(dl * wl) : dl * wl, smsl, rsmsl);
  const T dra0 = dvp.div(dr * wr, srsm, rsrsm);
  const T sqla = dvp.root(dla0), sqra = dvp.root(dra0);
  const T sla = sm - dvp.div(fabs(b1), sqla, dvp.rec(sqla));
  const T sra = sm + dvp.div(fabs(b1), sqra, dvp.rec(sqra));
  const T pta = dvp.div(wr * dr * ptl - wl * dl * ptr + dl * dr * wr * wl * (v1r - v1l), den, rden);
  const T b1b1 = b1 * b1;
  const T denl = dl * wl * (sl - sm) - b1b1;
  const T denr = dr * wr * (sr - sm) - b1b1;
  const T rdenl = dvp.rec(denl), rdenr = dvp.rec(denr);
  const T v2la = v2l - dvp.div(b1 * b2l * (sm - v1l), denl, rdenl);
  const T v2ra = v2r - dvp.div(b1 * b2r * (sm - v1r), denr, rdenr);
  const T v3la = v3l - dvp.div(b1 * b3l * (sm - v1l), denl, rdenl);
  const T v3ra = v3r - dvp.div(b1 * b3r * (sm - v1r), denr, rdenr);
  const T numl = dl * wl * wl - b1b1;
  const T numr = dr * wr * wr - b1b1;
  const T b2la = dvp.div(b2l * numl, denl, rdenl);
  const T b2ra = dvp.div(b2r * numr, denr, rdenr);
  const T b3la = dvp.div(b3l * numl, denl, rdenl);
  const T b3ra = dvp.div(b3r * numr, denr, rdenr);
  const T wela = wl * el - ptl * v1l + pta * sm +
                 b1 * ((v1l * b1 + v2l * b2l + v3l * b3l) - (sm * b1 + v2la * b2la + v3la * b3la));
  const T ela = dvp.div(pos ? -wela : wela, smsl, rsmsl);
  const T era = dvp.div(wr * er - ptr * v1r + pta * sm +
                           b1 * ((v1r * b1 + v2r * b2r + v3r * b3r) - (sm * b1 + v2ra * b2ra + v3ra * b3ra)),
                       srsm, rsrsm);
  const T s1 = fsign(one, b1);
  const T sqsum = sqla + sqra;
  const T rsqsum = dvp.rec(sqsum);
  const T v2aa = dvp.div(sqla * v2la + sqra * v2ra + (b2ra - b2la) * s1, sqsum, rsqsum);
  const T v3aa = dvp.div(sqla * v3la + sqra * v3ra + (b3ra - b3la) * s1, sqsum, rsqsum);
  const T sqlr = dvp.root(dla0 * dra0);
  const T b2aa = dvp.div(sqla * b2ra + sqra * b2la + sqlr * (v2ra - v2la) * s1, sqsum, rsqsum);
  const T b3aa = dvp.div(sqla * b3ra + sqra * b3la + sqlr * (v3ra - v3la) * s1, sqsum, rsqsum);
  const T vbaa = v2aa * b2aa + v3aa * b3aa;
  const T eraa = era + s1 * sqra * ((v2ra * b2ra + v3ra * b3ra) - vbaa);
  const T elaa = ela - s1 * sqla * ((v2la * b2la + v3la * b3la) - vbaa);
  T d, v2, v3, bb2, bb3, e;
  if constexpr (D::flags) {
    // The reference adds each state times 0 or 1, by the signs of sm, sla <= sm
    // and sra >= sm.  A finite state times 0 adds nothing, so the state can be
    // picked: 24 selects instead of 42 FP64 operations.  All are finite unless
    // refused: the quotients by their operands, the energies here.  (Where a
    // zero's sign picks otherwise there, every flux has a zero factor.)
    dvp.template need_below<1000>(elaa);
    dvp.template need_below<1000>(eraa);
    const bool ml = !(sm < zero), la = !(sla < zero), ra = sra < zero;
    d = ml ? dla0 : dra0;
    v2 = la ? v2la : (ra ? v2ra : v2aa);
    v3 = la ? v3la : (ra ? v3ra : v3aa);
    bb2 = la ? b2la : (ra ? b2ra : b2aa);
    bb3 = la ? b3la : (ra ? b3ra : b3aa);
    e = la ? ela : (ra ? era : (ml ? elaa : eraa));
  } else {
    // branch-free selection of the state at x/t = 0 (hlldflux.f90:113-145)
    const T signsm = fsign(h, sm);
    const T wsla = h + fsign(h, sla);
    const T wsra = h + fsign(h, -sra);
    const T wslr = h - fsign(h, sla * sra);
    d = (h + signsm) * dla0 + (h - signsm) * dra0;
    v2 = wsla * v2la + wslr * v2aa + wsra * v2ra;
    v3 = wsla * v3la + wslr * v3aa + wsra * v3ra;
    bb2 = wsla * b2la + wslr * b2aa + wsra * b2ra;
    bb3 = wsla * b3la + wslr * b3aa + wsra * b3ra;
    e = wsla * ela + (h - fsign(h, sla * sm)) * elaa + (h + fsign(h, -(sm * sra))) * eraa +
                     (h - fsign(h, sra)) * era;
  }
  const T v1 = sm, p = pta;
  const T dv = d * v1;
  f[0] = dv;
  f[1] = dv * v1 + p - b1 * b1;
  f[2] = dv * v2 - b1 * bb2;
  f[3] = dv * v3 - b1 * bb3;
  f[4] = (e + p) * v1 - b1 * (v1 * b1 + v2 * bb2 + v3 * bb3);
  f[5] = phi;
  f[6] = bb2 * v1 - b1 * v2;
  f[7] = bb3 * v1 - b1 * v3;
  f[8] = ch * ch * b1;
}

// The same flux without a magnetic field (every B and phi zero), f[0..4]:
// what is left of the expressions above once the terms that are exactly zero
// are gone.  With B = 0 the fast speed is the sound speed (the square root of
// a rounded square is its argument), sla = sra = sm, each star state keeps its
// tangential velocities, and the state at x/t = 0 is the left star state for
// sm >= 0 and the right one for sm < 0.  So the side is chosen first and one
// star state is formed: 4 reciprocals, 12 quotients and 2 square roots per
// face instead of 11, 35 and 9.  A result equals that of hlld as long as no
// dropped term is NaN or infinite: the policy refuses operands for which one
// might be (densities outside [2^-150, 2^200), velocities from 2^150 on, wave
// distances outside [2^-200, 2^200), a star density that is not positive).  Where
// sm = -0, hlld takes the state between the Alfven waves, but every flux then has
// the factor sm.
//
// T = float (the mixed form): there the compiler contracts both solvers, and not
// alike, so the bits differ from hlld<float> while the error does not grow.
// Against 64 bits, over 4 M faces in each of 15 ranges (jumps of 0 to e^2 in density
// and pressure, Mach 0.1 to 5), the rms error of every flux is 0.95 to 1.00 of
// hlld<float>'s (2e-8 to 6e-7 of the local scale) and the largest 0.87 to 1.10; a
// mixed step of 160x150x140 cells takes 1.82 ms instead of 2.13.
template <typename T, class D>
__device__ __forceinline__ void hllc(T f[5], T csl, T csr, T v1l, T v1r, T v2l, T v2r, T v3l, T v3r, T dl, T dr, T el,
                                     T er, T ptl, T ptr, D& dvp) {
  const T zero = T(0.0);
  const T sl = fmin2(fmin2(v1r - csr, v1l - csl), zero);
  const T sr = fmax2(fmax2(v1r + csr, v1l + csl), zero);
  const T wl = sl - v1l, wr = sr - v1r;
  const T wdl = wl * dl, wdr = wr * dr;
  const T den = wdr - wdl;
  const T rden = dvp.rec(den);
  const T sm = dvp.div(wdr * v1r - wdl * v1l - ptr + ptl, den, rden);
  const T pta = dvp.div(wdr * ptl - wdl * ptr + dl * dr * wr * wl * (v1r - v1l), den, rden);
  const T smsl = sm - sl, srsm = sr - sm;
  dvp.template need_pos<-200, 200>(smsl);
  dvp.template need_pos<-200, 200>(srsm);
  dvp.template need_pos<-200, 200>(-wdl);
  dvp.template need_pos<-200, 200>(wdr);
  const bool left = sm >= zero;
  const T s = left ? smsl : srsm, w = left ? -wl : wr, wd = left ? -wdl : wdr;
  const T v1 = left ? v1l : v1r, e0 = left ? el : er, pt = left ? ptl : ptr;
  const T sg = left ? -sm : sm;
  const T rs = dvp.rec(s);
  const T d = dvp.div(wd, s, rs);
  // (w e - pt v1 + pta sm) / (S - sm) with both operands negated on the left
  const T e = dvp.div(w * e0 - (left ? -pt : pt) * v1 + pta * sg, s, rs);
  const T dv = d * sm;
  f[0] = dv;
  f[1] = dv * sm + pta;
  f[2] = dv * (left ? v2l : v2r);
  f[3] = dv * (left ? v3l : v3r);
  f[4] = (e + pta) * sm;
}

// The same with plain division (every caller without a division policy).
template <typename T>
__device__ __forceinline__ void hlld(T f[9], T cfl, T cfr, T v1l, T v1r, T v2l, T v2r, T v3l, T v3r, T dl, T dr, T el,
                                     T er, T ptl, T ptr, T b1l, T b1r, T b2l, T b2r, T b3l, T b3r, T phil, T phir,
                                     T ch) {
  PlainDiv dv;
  hlld(f, cfl, cfr, v1l, v1r, v2l, v2r, v3l, v3r, dl, dr, el, er, ptl, ptr, b1l, b1r, b2l, b2r, b3l, b3r, phil, phir, ch,
       ch, dv);
}

}  // namespace hmn
