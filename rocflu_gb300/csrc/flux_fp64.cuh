// The interior fluxes of RFLU_PREC_FP64 with the fewest FP64 instructions.
//
// Same fluxes as physics.cuh's roeFlux, hllcFlux and ausmFlux (the reference
// routines cited there), which keep the reference's operation order for the
// bit-exact mode.  The FP64 pipe binds the face kernel (84% busy), so common
// factors are taken out (one reciprocal per density, the face area and the
// factor 1/2 once per component, the acoustic terms of the Roe dissipation
// combined), and divisions and roots run on the integer pipe (dual.cuh): about
// 105 FP64 instructions per HLLC face instead of 150, 140 instead of 205 for
// Roe.  Results differ from the reference order by rounding only.  S is double
// or a dual number over it (the tangent's and the adjoint's derivatives are
// those of the same expressions); normals and gas parameters carry none.
// Measured: 2 steps of 421,875 hexahedra (HLLC) 9.02 -> 8.30 ms, 40 first-order
// Roe steps of 6,400 cells 3.23 -> 3.05 ms; the tangent's Roe faces of 196,608
// tetrahedra (kTanFlux) 625 -> 405 us.
#pragma once
#include "dual.cuh"

namespace rflu {

// HLLC; e: total energy per mass, a: sound speed, H: enthalpy as the caller
// forms them, irl = 1/rl; g1 = gamma - 1.
template <typename S>
__host__ __device__ inline void hllcFluxShort(double g1, double nx, double ny, double nz, double nm, S rl, S ul, S vl,
                                              S wl, S pl, S el, S al, S Hl, S irl, S rr, S ur, S vr, S wr, S pr, S er,
                                              S ar, S Hr, S *flx) {
  const S ql = ul * nx + vl * ny + wl * nz, qr = ur * nx + vr * ny + wr * nz;
  const S w1 = sqrt_(rr * irl), w2 = div_(1.0, 1.0 + w1);
  const S us = w2 * (ul + w1 * ur), vs = w2 * (vl + w1 * vr), ws = w2 * (wl + w1 * wr);
  const S qs = w2 * (ql + w1 * qr), Hs = w2 * (Hl + w1 * Hr);
  const S as = sqrt_(g1 * (Hs - 0.5 * (us * us + vs * vs + ws * ws)));
  const S sl = fmin2(ql - al, qs - as), sr = fmax2(qr + ar, qs + as);
  // mass flux a, normal coefficient b and energy flux of the three cases:
  // F = (a, a u + b n, f4)
  S a, b, f4, u, v, w;
  if (pos_(sl) || neg_(sr)) {
    const bool left = pos_(sl);
    const S q = left ? ql : qr, r = left ? rl : rr, e = left ? el : er;
    b = left ? pl : pr;
    u = left ? ul : ur;
    v = left ? vl : vr;
    w = left ? wl : wr;
    a = q * r;
    f4 = q * (r * e + b);
  } else {
    const S ml = rl * (sl - ql), mr = rr * (sr - qr);
    const S sm = div_(mr * qr - ml * ql - pr + pl, mr - ml);
    const S ps = pl + ml * (sm - ql);
    const bool left = pos_(sm);
    const S q = left ? ql : qr, p = left ? pl : pr, k = left ? ml : mr, e = left ? el : er;
    u = left ? ul : ur;
    v = left ? vl : vr;
    w = left ? wl : wr;
    const S c = div_(sm, (left ? sl : sr) - sm);
    const S pm = ps * sm;
    a = c * k;
    b = ps + c * (ps - p);
    f4 = a * e + (pm + c * (pm - p * q));
  }
  a = a * nm;
  b = b * nm;
  flx[0] = a;
  flx[1] = a * u + b * nx;
  flx[2] = a * v + b * ny;
  flx[3] = a * w + b * nz;
  flx[4] = f4 * nm;
}

// Roe with the Harten-Hyman fix; H: enthalpy as the caller forms it.
template <typename S>
__host__ __device__ inline void roeFluxShort(double g1, double epsentr, double dissFact, double nx, double ny,
                                             double nz, double nm, S rl, S ul, S vl, S wl, S pl, S Hl, S rr, S ur,
                                             S vr, S wr, S pr, S Hr, S *flx) {
  const S ql = ul * nx + vl * ny + wl * nz, qr = ur * nx + vr * ny + wr * nz;
  const S rh = sqrt_(rl * rr), wt = div_(rl, rl + rh);
  const S dr = rr - rl, du = ur - ul, dv = vr - vl, dw = wr - wl, dp = pr - pl;
  const S dq = du * nx + dv * ny + dw * nz;
  // wt X_l + (1 - wt) X_r
  const S uh = ur - wt * du, vh = vr - wt * dv, wh = wr - wt * dw, Hh = Hr - wt * (Hr - Hl);
  const S qh = uh * nx + vh * ny + wh * nz;
  const S sh = 0.5 * (uh * uh + vh * vh + wh * wh);
  const S ah = sqrt_(g1 * (Hh - sh));
  S l1 = fabs_(qh - ah), l2 = fabs_(qh), l5 = fabs_(qh + ah);
  const S efc = epsentr * l5;
  l1 = entropyFixHH(l1, efc);
  l2 = entropyFixHH(l2, efc);
  l5 = entropyFixHH(l5, efc);
  const S ih = div_(0.5, ah * ah), x = rh * ah * dq;
  const S t1 = l1 * ((dp - x) * ih), t5 = l5 * ((dp + x) * ih);
  const S t2 = l2 * (dr - dp * (ih + ih)), t3 = l2 * rh;
  const S t15 = t1 + t5, t = t15 + t2, s = (t5 - t1) * ah, b = s - t3 * dq;
  const S al = ql * rl, ar = qr * rr, ps = pl + pr;
  const double h = 0.5 * nm;
  // half the area times (convective part - dissFact x dissipative part)
  flx[0] = h * (al + ar - dissFact * t);
  const S td = dissFact * t, t3d = dissFact * t3, pn = ps - dissFact * b;
  flx[1] = h * (al * ul + ar * ur + pn * nx - (td * uh + t3d * du));
  flx[2] = h * (al * vl + ar * vr + pn * ny - (td * vh + t3d * dv));
  flx[3] = h * (al * wl + ar * wr + pn * nz - (td * wh + t3d * dw));
  flx[4] = h * (al * Hl + ar * Hr -
                dissFact * (t15 * Hh + s * qh + t2 * sh + t3 * (uh * du + vh * dv + wh * dw - qh * dq)));
}

// AUSM+; a: sound speeds, H: enthalpies.
template <typename S>
__host__ __device__ inline void ausmFluxShort(double nx, double ny, double nz, double nm, S rl, S ul, S vl, S wl,
                                              S pl, S Hl, S al, S rr, S ur, S vr, S wr, S pr, S Hr, S ar, S *flx) {
  const S ql = ul * nx + vl * ny + wl * nz, qr = ur * nx + vr * ny + wr * nz;
  const S af = 0.5 * (al + ar), iaf = div_(1.0, af);
  const S ml = ql * iaf, mr = qr * iaf;
  S mp, mm, wp, wm;
  if (lessEq_(fabs_(ml), S(1.0))) {
    const S s = ml + 1.0, d = ml * ml - 1.0, d2 = d * d, s2 = 0.25 * (s * s);
    mp = s2 + 0.125 * d2;
    wp = s2 * (2.0 - ml) + 0.1875 * ml * d2;
  } else {
    mp = 0.5 * (ml + fabs_(ml));
    wp = pos_(ml) ? 1.0 : 0.0;
  }
  if (lessEq_(fabs_(mr), S(1.0))) {
    const S s = mr - 1.0, d = mr * mr - 1.0, d2 = d * d, s2 = 0.25 * (s * s);
    mm = -s2 - 0.125 * d2;
    wm = s2 * (2.0 + mr) - 0.1875 * mr * d2;
  } else {
    mm = 0.5 * (mr - fabs_(mr));
    wm = pos_(mr) ? 0.0 : 1.0;
  }
  const S mf = mp + mm, an = af * nm;
  const S a = pos_(mf) ? an * mf * rl : 0.0, b = pos_(mf) ? 0.0 : an * mf * rr;
  const S pn = (wp * pl + wm * pr) * nm;
  flx[0] = a + b;
  flx[1] = a * ul + b * ur + pn * nx;
  flx[2] = a * vl + b * vr + pn * ny;
  flx[3] = a * wl + b * wr + pn * nz;
  flx[4] = a * Hl + b * Hr;
}

}  // namespace rflu
