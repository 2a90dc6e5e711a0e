// Hand-written reverse mode of the second-order HLLC face flux.
//
// Forward: RFLU_HLLC_ComputeFlux2_TCP (modflu/RFLU_ModHLLCFlux.F90:2131-2434)
// on the reconstructed states L = (rl,ul,vl,wl,pl), R = (rr,ur,vr,wr,pr), with
// e = p/((g-1) rho) + |u|^2/2, a = sqrt(g p/rho) and H = e + ir p, ir the
// cells' 1/rho.  Reverse: given fbar = dJ/dF (5), writes dJ/d(L, irl) and
// dJ/d(R, irr), six values each, in one forward and one backward sweep whose
// intermediates stay in registers (the dual-number form seeds six directions
// per side through the whole flux at 255 registers).  Derivatives follow the
// branch the forward sweep takes (wave speeds, side of the contact).
#pragma once
#include "dual.cuh"

namespace rflu {

template <typename T>
__host__ __device__ inline void hllc2Adjoint(T g, T nx, T ny, T nz, T nm, const T *L, T irl, const T *R, T irr,
                                             const T *fbar, T *Lb, T *Rb) {
  const T g1 = g - T(1), half = T(0.5);
  const T rl = L[0], ul = L[1], vl = L[2], wl = L[3], pl = L[4];
  const T rr = R[0], ur = R[1], vr = R[2], wr = R[3], pr = R[4];
  // ---------------- forward ----------------
  const T cl = div_(pl, rl * g1), cr = div_(pr, rr * g1);  // internal energies
  const T el = cl + half * (ul * ul + vl * vl + wl * wl), er = cr + half * (ur * ur + vr * vr + wr * wr);
  const T al = sqrt_(div_(g * pl, rl)), ar = sqrt_(div_(g * pr, rr));
  const T Hl = el + irl * pl, Hr = er + irr * pr;
  const T ql = ul * nx + vl * ny + wl * nz, qr = ur * nx + vr * ny + wr * nz;
  const T w1 = sqrt_(div_(rr, rl)), w2 = div_(T(1), T(1) + w1);
  const T us = w2 * (ul + w1 * ur), vs = w2 * (vl + w1 * vr), ws = w2 * (wl + w1 * wr);
  const T qs = w2 * (ql + w1 * qr), Hs = w2 * (Hl + w1 * Hr);
  const T as = sqrt_(g1 * (Hs - half * (us * us + vs * vs + ws * ws)));
  const T sl1 = ql - al, sl2 = qs - as, sr1 = qr + ar, sr2 = qs + as;
  const bool slRoe = less_(sl2, sl1), srRoe = less_(sr1, sr2);
  const T sl = slRoe ? sl2 : sl1, sr = srRoe ? sr2 : sr1;
  // ---------------- reverse ----------------
  const T f0 = fbar[0] * nm, f1 = fbar[1] * nm, f2 = fbar[2] * nm, f3 = fbar[3] * nm, f4 = fbar[4] * nm;
  const T fn = f1 * nx + f2 * ny + f3 * nz;
  // adjoints of one side's (rho, u, v, w, p, e, q); the other side's start at 0
  T rlb = T(0), ulb = T(0), vlb = T(0), wlb = T(0), plb = T(0), elb = T(0), qlb = T(0);
  T rrb = T(0), urb = T(0), vrb = T(0), wrb = T(0), prb = T(0), erb = T(0), qrb = T(0);
  T slb = T(0), srb = T(0);
  auto plain = [&](T r, T u, T v, T w, T p, T e, T q, T &rb, T &ub, T &vb, T &wb, T &pb, T &eb, T &qb) {
    const T fu = f1 * u + f2 * v + f3 * w;
    qb = r * (f0 + fu) + f4 * (r * e + p);
    rb = q * (f0 + fu + f4 * e);
    const T qr_ = q * r;
    ub = f1 * qr_;
    vb = f2 * qr_;
    wb = f3 * qr_;
    pb = fn + f4 * q;
    eb = f4 * qr_;
  };
  if (pos_(sl)) {
    plain(rl, ul, vl, wl, pl, el, ql, rlb, ulb, vlb, wlb, plb, elb, qlb);
  } else if (neg_(sr)) {
    plain(rr, ur, vr, wr, pr, er, qr, rrb, urb, vrb, wrb, prb, erb, qrb);
  } else {
    const T dl = sl - ql, dr = sr - qr;
    const T idn = div_(T(1), rr * dr - rl * dl);
    const T sm = (rr * qr * dr - rl * ql * dl - pr + pl) * idn;
    const T ps = pl + rl * (ql - sl) * (ql - sm);
    T smb, psb;
    auto star = [&](T r, T u, T v, T w, T p, T e, T q, T S, T &rb, T &ub, T &vb, T &wb, T &pb, T &eb, T &qb, T &Sb) {
      const T term = div_(T(1), S - sm);
      const T k = (S - q) * r, dp = ps - p;
      const T rs = term * k, rus = term * (k * u + dp * nx), rvs = term * (k * v + dp * ny),
              rws = term * (k * w + dp * nz), res = term * (k * e + (ps * sm - p * q));
      const T b0 = f0 * sm, b1 = f1 * sm, b2 = f2 * sm, b3 = f3 * sm, b4 = f4 * sm;
      smb = f0 * rs + f1 * rus + f2 * rvs + f3 * rws + f4 * (res + ps);
      psb = fn + b4;
      const T tt = (b0 * rs + b1 * rus + b2 * rvs + b3 * rws + b4 * res) * term;  // -dJ/dS through the quotient
      const T kb = term * (b0 + b1 * u + b2 * v + b3 * w + b4 * e), tk = term * k, t4 = term * b4;
      const T x = term * (b1 * nx + b2 * ny + b3 * nz);
      ub = b1 * tk;
      vb = b2 * tk;
      wb = b3 * tk;
      eb = b4 * tk;
      psb += x + t4 * sm;
      pb = -x - t4 * q;
      smb += tt + t4 * ps;
      qb = -t4 * p - kb * r;
      rb = kb * (S - q);
      Sb = kb * r - tt;
    };
    if (pos_(sm)) star(rl, ul, vl, wl, pl, el, ql, sl, rlb, ulb, vlb, wlb, plb, elb, qlb, slb);
    else star(rr, ur, vr, wr, pr, er, qr, sr, rrb, urb, vrb, wrb, prb, erb, qrb, srb);
    // ps = pl + rl (ql - sl)(ql - sm)
    const T ls = ql - sl, lm = ql - sm;
    plb += psb;
    rlb += psb * ls * lm;
    qlb += psb * rl * (ls + lm);
    slb -= psb * rl * lm;
    smb -= psb * rl * ls;
    // sm = (rr qr dr - rl ql dl - pr + pl) / (rr dr - rl dl)
    const T nb = smb * idn, db = -nb * sm;
    rrb += dr * (nb * qr + db);
    qrb += rr * (nb * (dr - qr) - db);
    srb += rr * (nb * qr + db);
    prb -= nb;
    rlb -= dl * (nb * ql + db);
    qlb -= rl * (nb * (dl - ql) - db);
    slb -= rl * (nb * ql + db);
    plb += nb;
  }
  // wave speeds
  T alb = T(0), arb = T(0), asb = T(0), qsb = T(0);
  if (slRoe) { qsb += slb; asb -= slb; } else { qlb += slb; alb = -slb; }
  if (srRoe) { qsb += srb; asb += srb; } else { qrb += srb; arb = srb; }
  // Roe averages: as = sqrt(g1 (Hs - |us|^2/2)), Xs = w2 (Xl + w1 Xr)
  const T Hsb = nonZero_(asb) && pos_(as) ? div_(half * g1 * asb, as) : T(0);
  const T usb = -Hsb * us, vsb = -Hsb * vs, wsb = -Hsb * ws;
  const T w1b = w2 * (usb * (ur - us) + vsb * (vr - vs) + wsb * (wr - ws) + qsb * (qr - qs) + Hsb * (Hr - Hs));
  const T w12 = w2 * w1;
  ulb += w2 * usb; vlb += w2 * vsb; wlb += w2 * wsb; qlb += w2 * qsb;
  urb += w12 * usb; vrb += w12 * vsb; wrb += w12 * wsb; qrb += w12 * qsb;
  const T Hlb = w2 * Hsb, Hrb = w12 * Hsb;
  const T irL = div_(T(1), rl), irR = div_(T(1), rr), hw = half * w1b * w1;
  rlb -= hw * irL;
  rrb += hw * irR;
  // H = e + ir p; a = sqrt(g p/rho); e = p/((g-1) rho) + |u|^2/2; q = u.n
  elb += Hlb;
  erb += Hrb;
  plb += Hlb * irl;
  prb += Hrb * irr;
  const T ha = half * alb * al, hb = half * arb * ar;
  // a root at zero (p = 0) counts as a derivative of zero, as in dual.cuh
  if (nonZero_(ha)) plb += div_(ha, pl);
  if (nonZero_(hb)) prb += div_(hb, pr);
  const T ig1 = div_(T(1), g1);
  plb += elb * irL * ig1;
  prb += erb * irR * ig1;
  rlb -= (ha + elb * cl) * irL;
  rrb -= (hb + erb * cr) * irR;
  Lb[0] = rlb;
  Lb[1] = ulb + elb * ul + qlb * nx;
  Lb[2] = vlb + elb * vl + qlb * ny;
  Lb[3] = wlb + elb * wl + qlb * nz;
  Lb[4] = plb;
  Lb[5] = Hlb * pl;
  Rb[0] = rrb;
  Rb[1] = urb + erb * ur + qrb * nx;
  Rb[2] = vrb + erb * vr + qrb * ny;
  Rb[3] = wrb + erb * wr + qrb * nz;
  Rb[4] = prb;
  Rb[5] = Hrb * pr;
}

}  // namespace rflu
