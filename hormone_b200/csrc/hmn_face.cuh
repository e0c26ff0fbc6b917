// hmn_face.cuh -- the limited slopes of one cell and the flux through one
// face in the reference's operation order, with every quotient formed by
// FastDiv (hmn_div.cuh) and an exact fallback; shared by the march
// (hmn_march.cu) and tile (hmn_kernels.cu) stages.  Results are bitwise
// those of IEEE division.
#pragma once
#include <cuda_runtime.h>

#include "hmn_div.cuh"
#include "hmn_math.cuh"
#include "hmn_tile.cuh"

namespace hmn {
namespace {

// What every face of a launch (of a simulation, in a batch) shares: a copy in
// shared memory, so that the face function takes one pointer instead of four
// values in registers.
struct FluxConst {
  double gamma, gm1, ch, rch;  // rch: 1/ch, correctly rounded
};
__device__ __forceinline__ void set_flux_const(FluxConst& fc, const StageArgs& A) {
  const double ch = A.sc->ch;
  fc.gamma = A.gamma;
  fc.gm1 = A.gm1;
  fc.ch = ch;
  fc.rch = 1.0 / ch;
}

// Limited slopes of one cell along one axis from its two neighbours
// (interpolation.f90:49-163 with fluxlimiter.f90:40-75): pm, p0, pp point at
// staged quantity 0 of the cells, quantity q at [q * QS].  g points at the
// cell in the axis's first array, array q at g[q * len] (GEO_*).
template <bool MAG, int LIM, int QS, class D>
__device__ __forceinline__ void slopes_with(const double* pm, const double* p0, const double* pp, const double* g,
                                            int len, double sl[NS], D& dv) {
  constexpr int nsl = MAG ? NS : S_B;
#pragma unroll
  for (int q = 0; q < NS; q++) sl[q] = 0.0;
  if constexpr (LIM == 0) {
    return;
  } else {
    constexpr int qmap[NS] = {Q_D, Q_E, Q_M + 0, Q_M + 1, Q_M + 2, Q_B + 0, Q_B + 1, Q_B + 2};
    const double hl = g[GEO_HL * len], hr = g[GEO_HR * len];
    double L[NS], R[NS];
    if constexpr (LIM == 1) {
      const double i0 = g[GEO_IDX * len], i1 = g[GEO_IDX * len + 1], is = g[GEO_ISUM * len];
      const double ris = dv.rec(is);
#pragma unroll
      for (int q = 0; q < nsl; q++) {
        const double u0 = pm[qmap[q] * QS], u1 = p0[qmap[q] * QS], u2 = pp[qmap[q] * QS];
        const double du = lim_minmod(u0, u1, u2, i0, i1, is, dv, ris);
        sl[q] = du;
        L[q] = u1 - hl * du;
        R[q] = u1 + hr * du;
      }
    } else {
      const double cf = g[GEO_MCF * len], cb = g[GEO_MCB * len], ga = g[GEO_GA * len], gb = g[GEO_GB * len];
      const double rga = dv.rec(ga), rgb = dv.rec(gb);
#pragma unroll
      for (int q = 0; q < nsl; q++) {
        const double u0 = pm[qmap[q] * QS], u1 = p0[qmap[q] * QS], u2 = pp[qmap[q] * QS];
        const double du = lim_mmc(u0, u1, u2, cf, cb, ga, gb, dv, rga, rgb);
        sl[q] = du;
        L[q] = u1 - hl * du;
        R[q] = u1 + hr * du;
      }
    }
    double eintl = L[S_E] - dv.div(0.5 * (L[S_M] * L[S_M] + L[S_M + 1] * L[S_M + 1] + L[S_M + 2] * L[S_M + 2]),
                                   L[S_D], dv.rec(L[S_D]));
    double eintr = R[S_E] - dv.div(0.5 * (R[S_M] * R[S_M] + R[S_M + 1] * R[S_M + 1] + R[S_M + 2] * R[S_M + 2]),
                                   R[S_D], dv.rec(R[S_D]));
    if (MAG) {
      eintl = eintl - 0.5 * (L[S_B] * L[S_B] + L[S_B + 1] * L[S_B + 1] + L[S_B + 2] * L[S_B + 2]);
      eintr = eintr - 0.5 * (R[S_B] * R[S_B] + R[S_B + 1] * R[S_B + 1] + R[S_B + 2] * R[S_B + 2]);
    }
    const double em = pm[Lay<MAG>::EINT * QS], e0 = p0[Lay<MAG>::EINT * QS], ep = pp[Lay<MAG>::EINT * QS];
    if (eintl >= fmax2(em, e0) || eintl <= fmin2(em, e0) || eintr >= fmax2(e0, ep) || eintr <= fmin2(e0, ep)) {
#pragma unroll
      for (int q = 0; q < NS; q++) sl[q] = 0.0;
    }
  }
}

// What a caller of the out-of-line functions below vouches for: staged cells,
// slopes and fluxes lie in shared memory.  (A pointer argument is generic; with
// this the accesses need no address-space test.)
__device__ __forceinline__ void in_shared(const void* p) { __builtin_assume(__isShared(p)); }

// The slopes with IEEE division, out of line: the rare path of slopes_fast.
// Slope q goes to out[q * OS].
template <bool MAG, int LIM, int QS, int OS>
__device__ __noinline__ void slopes_ieee(const double* pm, const double* p0, const double* pp, const double* g, int L,
                                         double* out) {
  PlainDiv pd;
  double sl[NS];
  slopes_with<MAG, LIM, QS>(pm, p0, pp, g, L, sl, pd);
#pragma unroll
  for (int q = 0; q < Lay<MAG>::NS; q++) out[q * OS] = sl[q];
}

// The slopes with every quotient formed by FastDiv, recomputed with IEEE
// division where FastDiv could not vouch for one (bitwise the same result).
// One out-of-line copy serves every call site of a kernel, so that warps in
// different phases share instruction cache lines.  Slope q goes straight to
// out[q * OS]: with every stride a constant and the axis's arrays reached from
// one pointer, a call spends no multiplications on addresses and loads no
// pointer that it then has to wait for.  (Before, with run-time strides, four
// solver constants in registers and the march's z slopes and fluxes on the
// stack: 256^3 MHD stage 7.10 -> 6.60 ms, 97x75x62 box 15.2 -> 14.3 ms for 16
// steps, 160^3 polytrope 51.1 -> 48.5 ms.)
template <bool MAG, int LIM, int QS, int OS>
__device__ __noinline__ void slopes_fast(const double* pm, const double* p0, const double* pp, const double* g, int L,
                                         double* out) {
  in_shared(pm), in_shared(p0), in_shared(pp), in_shared(out);
  FastDiv fd;
  double sl[NS];
  slopes_with<MAG, LIM, QS>(pm, p0, pp, g, L, sl, fd);
  if (fd.bad) {
    slopes_ieee<MAG, LIM, QS, OS>(pm, p0, pp, g, L, out);
    return;
  }
#pragma unroll
  for (int q = 0; q < Lay<MAG>::NS; q++) out[q * OS] = sl[q];
}

// The slopes of the cell at global coordinate cg along the axis, n cells long.
template <bool MAG, int LIM, int QS, int OS>
__device__ __forceinline__ void slopes_to(const double* pm, const double* p0, const double* pp, const AxisGeo& g, int n,
                                          int cg, double* out) {
  if constexpr (LIM == 0) {
#pragma unroll
    for (int q = 0; q < Lay<MAG>::NS; q++) out[q * OS] = 0.0;
  } else {
    slopes_fast<MAG, LIM, QS, OS>(pm, p0, pp, g.x + cg + 2, n + 4, out);
  }
}

// Flux through one face (numflux.f90:65-198 + hlldflux.f90): pl/pr give the
// staged quantities of the left and right cells, sl/sr their slopes (index
// functors), dx1 = xi - x(left), dx2 = x(right) - xi, (cn, c1, c2) the
// normal and tangential components.  fl[0..8] in the solver's order (mass,
// normal and tangential momenta, energy, normal B (phi flux), tangential B,
// ch^2 B_n).  Returns false (fl zero) where a face state has eint <= 0 or
// rho <= 0 (numflux.f90:117 -> error_flux).
template <bool MAG, class D, class PL, class PR, class SL, class SR>
__device__ __forceinline__ bool face_flux_with(PL pl, PR pr, SL sl, SR sr, double dx1, double dx2, int cn, int c1,
                                               int c2, const FluxConst& fc, double fl[9], D& dv) {
  const double gamma = fc.gamma, gm1 = fc.gm1;
  const double dl = pl(Q_D) + dx1 * sl(S_D);
  const double dr = pr(Q_D) - dx2 * sr(S_D);
  const double el = pl(Q_E) + dx1 * sl(S_E);
  const double er = pr(Q_E) - dx2 * sr(S_E);
  const double rdl = dv.rec(dl), rdr = dv.rec(dr);
  const double v1l = dv.div(pl(Q_M + cn) + dx1 * sl(S_M + cn), dl, rdl);
  const double v1r = dv.div(pr(Q_M + cn) - dx2 * sr(S_M + cn), dr, rdr);
  const double v2l = dv.div(pl(Q_M + c1) + dx1 * sl(S_M + c1), dl, rdl);
  const double v2r = dv.div(pr(Q_M + c1) - dx2 * sr(S_M + c1), dr, rdr);
  const double v3l = dv.div(pl(Q_M + c2) + dx1 * sl(S_M + c2), dl, rdl);
  const double v3r = dv.div(pr(Q_M + c2) - dx2 * sr(S_M + c2), dr, rdr);
  double b1l = 0.0, b1r = 0.0, b2l = 0.0, b2r = 0.0, b3l = 0.0, b3r = 0.0, phil = 0.0, phir = 0.0;
  if (MAG) {
    b1l = pl(Q_B + cn) + dx1 * sl(S_B + cn);
    b1r = pr(Q_B + cn) - dx2 * sr(S_B + cn);
    b2l = pl(Q_B + c1) + dx1 * sl(S_B + c1);
    b2r = pr(Q_B + c1) - dx2 * sr(S_B + c1);
    b3l = pl(Q_B + c2) + dx1 * sl(S_B + c2);
    b3r = pr(Q_B + c2) - dx2 * sr(S_B + c2);
    // phi is never reconstructed: its slope is identically zero (allocations.f90)
    phil = pl(Q_PHI);
    phir = pr(Q_PHI);
  }
  const double eil = get_eint<MAG>(el, dl, v1l, v2l, v3l, b1l, b2l, b3l);
  const double eir = get_eint<MAG>(er, dr, v1r, v2r, v3r, b1r, b2r, b3r);
  if (eil <= 0.0 || dl <= 0.0 || eir <= 0.0 || dr <= 0.0) {
#pragma unroll
    for (int q = 0; q < 9; q++) fl[q] = 0.0;
    return false;
  }
  // eos_p_cs (eos.f90:209-219) with erad = 0
  const double ptl0 = gm1 * eil, ptr0 = gm1 * eir;
  const double csl = dv.root(dv.div(gamma * ptl0, dl, rdl)), csr = dv.root(dv.div(gamma * ptr0, dr, rdr));
  if constexpr (!MAG && D::flags) {  // the policy that recomputes what it refuses with the full solver
    dv.template need_pos<-150, 200>(dl);
    dv.template need_pos<-150, 200>(dr);
    dv.template need_below<150>(v1l);
    dv.template need_below<150>(v1r);
    dv.template need_below<150>(v2l);
    dv.template need_below<150>(v2r);
    dv.template need_below<150>(v3l);
    dv.template need_below<150>(v3r);
    hllc(fl, csl, csr, v1l, v1r, v2l, v2r, v3l, v3r, dl, dr, el, er, ptl0, ptr0, dv);
    return true;
  }
  const double ptl = ptl0 + 0.5 * (b1l * b1l + b2l * b2l + b3l * b3l);
  const double ptr = ptr0 + 0.5 * (b1r * b1r + b2r * b2r + b3r * b3r);
  const double cfl = get_cf(dl, csl, b1l, b2l, b3l, dv, rdl);
  const double cfr = get_cf(dr, csr, b1r, b2r, b3r, dv, rdr);
  const double ch = fc.ch;
  dv.template need_pos<-500, 501>(ch);
  hlld(fl, cfl, cfr, v1l, v1r, v2l, v2r, v3l, v3r, dl, dr, el, er, ptl, ptr, b1l, b1r, b2l, b2r, b3l, b3r, phil, phir,
       ch, fc.rch, dv);
  return true;
}

// Store a face flux rotated back into the conserved slots
// (numflux.f90:186-198, 359-371, 531-543), slot v to out[v * OS].
template <bool MAG, int OS>
__device__ __forceinline__ void put_flux(const double fl[9], int cn, int c1, int c2, double* out) {
  double *on = out + cn * OS, *o1 = out + c1 * OS, *o2 = out + c2 * OS;
  out[ICNT * OS] = fl[0];
  on[IMO1 * OS] = fl[1];
  o1[IMO1 * OS] = fl[2];
  o2[IMO1 * OS] = fl[3];
  out[IENE * OS] = fl[4];
  if constexpr (MAG) {
    on[IMG1 * OS] = fl[5];
    o1[IMG1 * OS] = fl[6];
    o2[IMG1 * OS] = fl[7];
    out[I9WV * OS] = fl[8];
  }
}

// The flux through a face normal to axis cn from staged cells (quantity 0 at
// pl, pr, stride QS) and slopes (slope 0 at sl, sr, stride SS).
template <bool MAG, int QS, int SS, class D>
__device__ __forceinline__ bool face_flux_at(const double* pl, const double* pr, const double* sl, const double* sr,
                                             double dx1, double dx2, int cn, int c1, int c2, const FluxConst* fc,
                                             double fl[9], D& dv) {
  return face_flux_with<MAG>([&](int q) { return pl[q * QS]; }, [&](int q) { return pr[q * QS]; },
                             [&](int q) { return sl[q * SS]; }, [&](int q) { return sr[q * SS]; }, dx1, dx2, cn, c1,
                             c2, *fc, fl, dv);
}

// The face flux with IEEE division, out of line: the rare path of
// face_flux_fast; arguments as there.
template <bool MAG, int QS, int SS, int OS>
__device__ __noinline__ bool face_flux_ieee(const double* pl, const double* pr, const double* sl, const double* sr,
                                            double dx1, double dx2, int cn, const FluxConst* fc, double* out) {
  PlainDiv pd;
  const int c1 = cn == 2 ? 0 : cn + 1, c2 = cn == 0 ? 2 : cn - 1;
  double fl[9];
  const bool ok = face_flux_at<MAG, QS, SS>(pl, pr, sl, sr, dx1, dx2, cn, c1, c2, fc, fl, pd);
  put_flux<MAG, OS>(fl, cn, c1, c2, out);
  return ok;
}

// The face flux with every quotient formed by FastDiv, recomputed with IEEE
// division where FastDiv could not vouch for one (bitwise the same result);
// one out-of-line copy for the x, y and z faces of a kernel.  The flux goes to
// out[slot * OS]; out may be where sl or sr is, for every operand is read
// before the first store.  Returns false (flux zero) where a face state has
// eint <= 0 or rho <= 0.
template <bool MAG, int QS, int SS, int OS>
__device__ __noinline__ bool face_flux_fast(const double* pl, const double* pr, const double* sl, const double* sr,
                                            double dx1, double dx2, int cn, const FluxConst* fc, double* out) {
  in_shared(pl), in_shared(pr), in_shared(sl), in_shared(sr), in_shared(fc), in_shared(out);
  FastDiv fd;
  const int c1 = cn == 2 ? 0 : cn + 1, c2 = cn == 0 ? 2 : cn - 1;
  double fl[9];
  const bool ok = face_flux_at<MAG, QS, SS>(pl, pr, sl, sr, dx1, dx2, cn, c1, c2, fc, fl, fd);
  if (fd.bad) return face_flux_ieee<MAG, QS, SS, OS>(pl, pr, sl, sr, dx1, dx2, cn, fc, out);
  put_flux<MAG, OS>(fl, cn, c1, c2, out);
  return ok;
}

}  // namespace
}  // namespace hmn
