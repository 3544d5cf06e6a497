// Strain rates of compute_Sij (subgrid.f90:1014-1072) at the centres of a
// column of planes, from fixed-point velocities.
//
// The four edge strains around a centre are sums of differences of four faces
// each, collected per spacing:
//   8 S12 = ry(jc-1) A + ry(jc) B + rx(i) C,  A, B the y differences of
//     U(i-1) + U(i) below and above, C = V(i+1) - V(i-1) on both y faces,
//   8 S13 = rz(k) D + rx(i) E,  D = U(k+1) - U(k-1) on both x faces,
//     E = W(i+1) - W(i-1) on both z faces,
//   8 S23 = ry(jc-1) G + ry(jc) H + rz(k) K,  likewise of W and V,
// sums and differences that are exact in integers.  x and z are uniform only
// within 1e-9 (chl_create), and the edges below i and k have spacings of their
// own: the lower half of C, D, E, K takes the difference of the reciprocals,
// (rx(i-1) - rx(i)) C_lo, for which 32 bits of either are enough.  Each centre
// scales its fifteen differences by their largest and its six strain rates by
// theirs, so that the products keep 54 bits or more of the largest.  A thread
// marches through planes and carries what they share: 17 loads per centre.
#pragma once
#include "chl_fix.cuh"

// t: S_11, S_22, S_33 and 2 S_12, 2 S_13, 2 S_23 in units of 2^e; s: |S| / sqrt(2)
struct Strain { fx t[6]; int e; double s; };

struct StrainColumn {
  const ChlInst& I;
  const fx *U, *V, *W;
  int eu, ev, ew;               // exponents of U, V, W
  int i, im, ip, jc, er;
  fx rx, rxc, ryl, ryh, ryc;    // reciprocal spacings, last bit 2^er
  int dx, sz;                   // rx(i-1) - rx(i), last bit 2^(er+3); shift of its like along z
  fx um, u0, us, usb;           // plane k: U at both x faces and their sum, the sum on plane k-1
  fx vm, v0, vs, vsb;           // V at both y faces
  fx wb, xwb, xlb, ylb, yhb;    // plane k-1: W and its x (whole, lower half) and y differences
  fx w0;                        // plane k: W (valid after point())

  __device__ __forceinline__ fx u(int a, int j, int k) const { return LDG(U + cidx(I, a, j, k)); }
  __device__ __forceinline__ fx v(int a, int j, int k) const { return LDG(V + vidx(I, a, j, k)); }
  __device__ __forceinline__ fx w(int a, int j, int k) const { return LDG(W + cidx(I, a, j, k)); }

  // column (i, jc), first plane k
  __device__ __forceinline__ StrainColumn(const ChlInst& I_, const fx* U_, const fx* V_, const fx* W_, int eu_, int ev_,
                                          int ew_, int i_, int jc_, int k)
      : I(I_), U(U_), V(V_), W(W_), eu(eu_), ev(ev_), ew(ew_), i(i_), jc(jc_) {
    im = wrap(i - 1, I.Nx); ip = wrap(i + 1, I.Nx);
    const int el = I.eyf[jc - 1], eh = I.eyf[jc], ec = I.eyc[jc];
    er = max(max(max(el, eh), max(ec, I.exf)), max(max(I.exc, I.ezf), I.ezc));
    ryl = LDG(I.fxryf + jc - 1) >> min(63, er - el);
    ryh = LDG(I.fxryf + jc) >> min(63, er - eh);
    ryc = LDG(I.fxryc + jc) >> min(63, er - ec);
    rx = LDG(I.fxrxf + i) >> min(63, er - I.exf);
    rxc = LDG(I.fxrxc + i) >> min(63, er - I.exc);
    dx = LDG(I.dxr + i) >> min(31, er - I.exf);
    sz = min(31, er - I.ezf);
    const int kb = k == 0 ? I.Nz - 1 : k - 1;
    um = u(im, jc, k); u0 = u(i, jc, k); us = um + u0; usb = u(im, jc, kb) + u(i, jc, kb);
    vm = v(i, jc - 1, k); v0 = v(i, jc, k); vs = vm + v0; vsb = v(i, jc - 1, kb) + v(i, jc, kb);
    wb = w(i, jc, kb);
    const fx wl = w(im, jc, kb);
    xwb = w(ip, jc, kb) - wl; xlb = wb - wl;
    ylb = wb - w(i, jc - 1, kb); yhb = w(i, jc + 1, kb) - wb;
  }

  // the strain of plane k; the face sums 2 u, 2 v, 2 w of its centre in c
  __device__ __forceinline__ Strain point(int k, fx (&c)[3]) {
    const int kp = k + 1 == I.Nz ? 0 : k + 1;
    const fx ump = u(im, jc, kp), u0p = u(i, jc, kp), vmp = v(i, jc - 1, kp), v0p = v(i, jc, kp);
    w0 = w(i, jc, k);
    const fx wl = w(im, jc, k), xw = w(ip, jc, k) - wl, xl = w0 - wl, yl = w0 - w(i, jc - 1, k), yh = w(i, jc + 1, k) - w0;
    const fx usp = ump + u0p, vsp = vmp + v0p;
    fx A = us - (u(im, jc - 1, k) + u(i, jc - 1, k)), B = (u(im, jc + 1, k) + u(i, jc + 1, k)) - us;
    fx D = usp - usb, K = vsp - vsb;
    const fx vl = v(im, jc - 1, k) + v(im, jc, k);
    fx C = (v(ip, jc - 1, k) + v(ip, jc, k)) - vl;
    // the lower halves of C, D, E, K
    const fx Cl = vs - vl, Dl = us - usb, El = xlb + xl, Kl = vs - vsb;
    fx E = xwb + xw, G = ylb + yl, H = yhb + yh;
    fx d1 = u0 - um, d2 = v0 - vm, d3 = w0 - wb;
    c[0] = us; c[1] = vs; c[2] = wb + w0;
    usb = us; us = usp; um = ump; u0 = u0p;
    vsb = vs; vs = vsp; vm = vmp; v0 = v0p;
    wb = w0; xwb = xw; xlb = xl; ylb = yl; yhb = yh;
    // |difference| < 2^60 in units of 2^et
    unsigned mu = 0u, mv = 0u, mw = 0u;
    top_or(mu, d1); top_or(mu, A); top_or(mu, B); top_or(mu, D); top_or(mu, Dl);
    top_or(mv, d2); top_or(mv, C); top_or(mv, K); top_or(mv, Cl); top_or(mv, Kl);
    top_or(mw, d3); top_or(mw, E); top_or(mw, G); top_or(mw, H); top_or(mw, El);
    const int et = max(max(eu + 64 - __clz((int)mu), ev + 64 - __clz((int)mv)), ew + 64 - __clz((int)mw)) - 60;
    const int su = eu - et, sv = ev - et, sw = ew - et;
    const fx rz = LDG(I.fxrzf + k) >> min(63, er - I.ezf), rzc = LDG(I.fxrzc + k) >> min(63, er - I.ezc);
    const int dz = LDG(I.dzr + k) >> sz;
    // strain rates: 4 S_ii, 8 S_ij, |x| < 2^61
    fx s1 = 4 * fx_mul(scale2(d1, su), rxc), s2 = 4 * fx_mul(scale2(d2, sv), ryc), s3 = 4 * fx_mul(scale2(d3, sw), rzc);
    fx t1 = fx_mul(scale2(A, su), ryl) + fx_mul(scale2(B, su), ryh) + fx_mul(scale2(C, sv), rx) + ((long long)scale2_hi(Cl, sv) * dx >> 29);
    fx t2 = fx_mul(scale2(D, su), rz) + fx_mul(scale2(E, sw), rx) +
            ((long long)scale2_hi(Dl, su) * dz + (long long)scale2_hi(El, sw) * dx >> 29);
    fx t3 = fx_mul(scale2(G, sw), ryl) + fx_mul(scale2(H, sw), ryh) + fx_mul(scale2(K, sv), rz) + ((long long)scale2_hi(Kl, sv) * dz >> 29);
    unsigned md = 0u;
    top_or(md, s1); top_or(md, s2); top_or(md, s3); top_or(md, t1); top_or(md, t2); top_or(md, t3);
    const int sd = __clz((int)md) - 3;
    s1 <<= sd; s2 <<= sd; s3 <<= sd; t1 <<= sd; t2 <<= sd; t3 <<= sd;
    // |S|^2 / 2 = d.d + (o.o)/32, here 16 x
    const fx q = (fx_mul(s1, s1) + fx_mul(s2, s2) + fx_mul(s3, s3) + 6) +
                 ((fx_mul(t1, t1) + fx_mul(t2, t2) + fx_mul(t3, t3)) >> 1);
    const int e = et + er + 64 - sd;
    Strain r;
    r.s = chl_sqrt(fx_to(q, 2 * e + 60));
    r.t[0] = s1; r.t[1] = s2; r.t[2] = s3; r.t[3] = t1; r.t[4] = t2; r.t[5] = t3;
    r.e = e - 2;
    return r;
  }
};
