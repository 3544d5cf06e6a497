// Anisotropic minimum-dissipation (AMD) and Vreman eddy viscosities, one
// fused kernel each, a thread per column of a few planes at an interior centre
// (rows 1..Ny).  Both write
// the unclipped nu_t into S and, in the same pass, nu + nu_t with k_nut's
// rules for these models (write_nut_rows): max(., 0) and the ghost-row rule of
// Dirichlet_nu_t - so there is no separate nu_t pass.
//
// AMD (subgrid.f90:632-874):
//   nu_t = max(0, -C N / D),  C = 0.3,
//   N = sum_k (d^_k u_i)(d^_k u_j) S_ij,   D = sum_kl (d_k u_l)^2,
// d^_k = grid-scaled difference, d_k = derivative; off-diagonal entries are
// interpolated to the centre from the four surrounding edges in the order the
// reference's interpolate_x/y/z calls use (interpolation.f90:24-105), and
// the three mixed products of each S_ij row are formed as written: two from
// centre values, one interpolated after the product.  S_ij is compute_Sij's
// (subgrid.f90:1014-1072), formed from the same edge sums.  The halves and
// quarters of the interpolations are exponents of the fixed-point values.
//
// Vreman (subgrid.f90:897-1004):
//   nu_t = C sqrt(B_b / a_ij a_ij),  C = 2.5 * 0.1^2,
//   b_ij = sum_m dx_m^2 a_mi a_mj,  B_b = b11 b22 - b12^2 + b11 b33 - b13^2 + b22 b33 - b23^2,
// a_ij = du_j/dx_i at the centre, off-diagonals the mean of four edge
// derivatives.  Two U sections of the reference are written 2:ny, 1:ny-1
// where 2:nx, 1:nx-1 are meant (subgrid.f90:930-931,946-947); they start at
// the same index, so element-wise they read the intended values, which is
// what is computed here.
#include "chl_nut.cuh"

namespace {

// Edge differences around the centres of a column of planes, exact integers
// from the fixed-point copies (k_fix).  For each off-diagonal velocity gradient
// the four edge differences are summed in two pairs: ?L/?H are the two-point
// sums on the near/far edge in the derivative direction (2 x the reference's
// first interpolation), their sum 4 x the centre difference.  The centre
// strain of compute_Sij (subgrid.f90:1014-1072) is the same sums.  A thread
// marches through a few planes and carries what they share (pair sums of U
// and V, differences of W): 17 loads per centre.
struct Diffs {
  fx dux, dvy, dwz;                      // diagonal differences
  fx uyL, uyH, uzL, uzH;                 // U: y and z edge pair sums
  fx vxL, vxR, vzL, vzH;                 // V: x and z
  fx wxL, wxR, wyL, wyH;                 // W: x and y
};

struct GradColumn {
  const ChlInst& I;
  int i, im, ip, jc, er;
  fx rxf, rxc, ryl, ryh, ryc;            // reciprocal spacings, last bit 2^er
  fx um, u0, uzL, vm, v0, vzL;           // plane k: U and V faces, their z differences to the plane below
  fx wm, wxl, wxr, wyl, wyh;             // plane k-1: W and its x and y differences

  __device__ __forceinline__ fx u(int a, int j, int k) const { return LDG(I.X[0] + cidx(I, a, j, k)); }
  __device__ __forceinline__ fx v(int a, int j, int k) const { return LDG(I.X[1] + vidx(I, a, j, k)); }
  __device__ __forceinline__ fx w(int a, int j, int k) const { return LDG(I.X[2] + cidx(I, a, j, k)); }

  __device__ __forceinline__ GradColumn(const ChlInst& I_, int i_, int jc_, int k) : I(I_), i(i_), jc(jc_) {
    im = wrap(i - 1, I.Nx); ip = wrap(i + 1, I.Nx);
    const int el = I.eyf[jc - 1], eh = I.eyf[jc], ec = I.eyc[jc];
    er = max(max(max(el, eh), max(ec, I.exf)), max(max(I.exc, I.ezf), I.ezc));
    ryl = LDG(I.fxryf + jc - 1) >> min(63, er - el);
    ryh = LDG(I.fxryf + jc) >> min(63, er - eh);
    ryc = LDG(I.fxryc + jc) >> min(63, er - ec);
    rxf = LDG(I.fxrxf + i - 1) >> min(63, er - I.exf);
    rxc = LDG(I.fxrxc + i) >> min(63, er - I.exc);
    const int kb = k == 0 ? I.Nz - 1 : k - 1;
    um = u(im, jc, k); u0 = u(i, jc, k);
    vm = v(i, jc - 1, k); v0 = v(i, jc, k);
    wm = w(i, jc, kb);
    uzL = (um + u0) - (u(im, jc, kb) + u(i, jc, kb));
    vzL = (vm + v0) - (v(i, jc - 1, kb) + v(i, jc, kb));
    wxl = wm - w(im, jc, kb); wxr = w(ip, jc, kb) - wm;
    wyl = wm - w(i, jc - 1, kb); wyh = w(i, jc + 1, kb) - wm;
  }
  __device__ __forceinline__ fx rzf(int k) const { return LDG(I.fxrzf + k - 1) >> min(63, er - I.ezf); }
  __device__ __forceinline__ fx rzc(int k) const { return LDG(I.fxrzc + k) >> min(63, er - I.ezc); }

  __device__ __forceinline__ Diffs point(int k) {
    const int kp = k + 1 == I.Nz ? 0 : k + 1;
    const fx ump = u(im, jc, kp), u0p = u(i, jc, kp), vmp = v(i, jc - 1, kp), v0p = v(i, jc, kp);
    const fx w0 = w(i, jc, k);
    const fx us = um + u0, vs = vm + v0;
    const fx xl = w0 - w(im, jc, k), xr = w(ip, jc, k) - w0, yl = w0 - w(i, jc - 1, k), yh = w(i, jc + 1, k) - w0;
    Diffs d;
    d.uyL = us - (u(im, jc - 1, k) + u(i, jc - 1, k)); d.uyH = (u(im, jc + 1, k) + u(i, jc + 1, k)) - us;
    d.vxL = vs - (v(im, jc - 1, k) + v(im, jc, k)); d.vxR = (v(ip, jc - 1, k) + v(ip, jc, k)) - vs;
    d.uzL = uzL; d.uzH = (ump + u0p) - us;
    d.vzL = vzL; d.vzH = (vmp + v0p) - vs;
    d.wxL = wxl + xl; d.wxR = wxr + xr; d.wyL = wyl + yl; d.wyH = wyh + yh;
    d.dux = u0 - um; d.dvy = v0 - vm; d.dwz = w0 - wm;
    uzL = d.uzH; vzL = d.vzH; wxl = xl; wxr = xr; wyl = yl; wyh = yh;
    um = ump; u0 = u0p; vm = vmp; v0 = v0p; wm = w0;
    return d;
  }
};

}  // namespace

// AMD in fixed point.  As FP64 code this kernel issued 114 FP64 instructions
// per point (0.97 ms per launch at 256x96x192, the FP64 pipe 90 % busy; 0.31 ms now).  The
// edge differences are exact integers from the fixed-point copies (k_fix);
// each point scales those of each component by their largest, so that a weak
// component keeps its digits, and forms the a_ij, the derivatives and D there.  The
// S_ii, N and the division are FP64 (one scale for the three components and the
// S_ii in integers beside the largest derivative took 0.28 ms and left nu_t of a
// nearly parallel flow 9 times as far off as in FP64, of turbulent ones 1.1 to 1.2
// times).  With none, three, six and twelve of N's twelve conversions on the FP64
// pipe 301, 300, 309 and 359 us (before the exact S_ii): all are on the integer pipe.
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 5)   // 2, 3, 4, 5, 6 blocks per SM took 417, 321, 289, 288, 290 us (312 now)
k_amd(ChlMap map, int s_in, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, M = map.planes;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k0 = p.k * M;
  const unsigned* vm = chl_vmax(I, s_in);
  const int eu = fx_exp<61>(vm[0]), ev = fx_exp<61>(vm[1]), ew = fx_exp<61>(vm[2]);
  const bool bad = fx_bad(vm[0]) || fx_bad(vm[1]) || fx_bad(vm[2]);
  GradColumn col(I, i, jc, min(k0, Nz - 1));       // lanes past the last plane repeat it
  const int er = col.er;
  unsigned hi = 0u;
  for (int q = 0; q < M; ++q) {
    const int k = min(k0 + q, Nz - 1);
    const bool valid = k0 + q < Nz;
    const Diffs d = col.point(k);
    fx dux = d.dux, dvy = d.dvy, dwz = d.dwz, uyL = d.uyL, uyH = d.uyH, vxL = d.vxL, vxR = d.vxR;
    fx wxL = d.wxL, wxR = d.wxR, wyL = d.wyL, wyH = d.wyH;
    // scale: each component's differences below 2^59 in units of 2^eU, 2^eV, 2^eW
    unsigned mu = 0u, mv = 0u, mw = 0u;
    top_or(mu, dux); top_or(mu, uyL); top_or(mu, uyH); top_or(mu, d.uzL); top_or(mu, d.uzH);
    top_or(mv, dvy); top_or(mv, vxL); top_or(mv, vxR); top_or(mv, d.vzL); top_or(mv, d.vzH);
    top_or(mw, dwz); top_or(mw, wxL); top_or(mw, wxR); top_or(mw, wyL); top_or(mw, wyH);
    const int su = __clz((int)mu) - 5, sv = __clz((int)mv) - 5, sw = __clz((int)mw) - 5;
    const int eU = eu - su, eV = ev - sv, eW = ew - sw, em = max(eU, max(eV, eW));
    dux = scale2(dux, su); uyL = scale2(uyL, su); uyH = scale2(uyH, su);
    const fx uL = scale2(d.uzL, su), uH = scale2(d.uzH, su);
    dvy = scale2(dvy, sv); vxL = scale2(vxL, sv); vxR = scale2(vxR, sv);
    const fx vL = scale2(d.vzL, sv), vH = scale2(d.vzH, sv);
    dwz = scale2(dwz, sw); wxL = scale2(wxL, sw); wxR = scale2(wxR, sw); wyL = scale2(wyL, sw); wyH = scale2(wyH, sw);
    // grid-scaled centre differences, 4 x
    const fx Yu = uyL + uyH, Zu = uL + uH, Xv = vxL + vxR, Zv = vL + vH, Xw = wxL + wxR, Yw = wyL + wyH;
    // exponents in N, whose differences are in units of 2^em
    const int cU = max(-300, eU - em), cV = max(-300, eV - em), cW = max(-300, eW - em);
    // D, a sum of squares, from the derivatives, 4 x, in units of 2^(em + er + 64 -
    // sd): scaled anew, as the spacings differ by up to the stretching of the grid
    const int du = min(63, em - eU), dv = min(63, em - eV), dw = min(63, em - eW);
    const fx rzf = col.rzf(k), rxf = col.rxf, ryl = col.ryl, ryh = col.ryh;
    fx s11 = 4 * fx_mul(dux, col.rxc) >> du, s22 = 4 * fx_mul(dvy, col.ryc) >> dv, s33 = 4 * fx_mul(dwz, col.rzc(k)) >> dw;
    fx dUy = fx_mul(uyL, ryl) + fx_mul(uyH, ryh) >> du, dWy = fx_mul(wyL, ryl) + fx_mul(wyH, ryh) >> dw;
    fx dUz = fx_mul(Zu, rzf) >> du, dVz = fx_mul(Zv, rzf) >> dv, dVx = fx_mul(Xv, rxf) >> dv, dWx = fx_mul(Xw, rxf) >> dw;
    unsigned md = 0u;
    top_or(md, s11); top_or(md, s22); top_or(md, s33);
    top_or(md, dUy); top_or(md, dUz); top_or(md, dVx); top_or(md, dVz); top_or(md, dWx); top_or(md, dWy);
    const int sd = __clz((int)md) - 3;     // |x| < 2^61; a derivative is below 2^61 already
    s11 <<= sd; s22 <<= sd; s33 <<= sd;
    dUy <<= sd; dUz <<= sd; dVx <<= sd; dVz <<= sd; dWx <<= sd; dWy <<= sd;
    // 16 x (2^64 units of the derivatives' square); 12 makes up for nine products
    const fx D = (fx_mul(s11, s11) + fx_mul(s22, s22) + fx_mul(s33, s33) + 12) +
                 (fx_mul(dUy, dUy) + fx_mul(dUz, dUz) + fx_mul(dVx, dVx)) +
                 (fx_mul(dVz, dVz) + fx_mul(dWx, dWx) + fx_mul(dWy, dWy));
    // N = sum a_ij S_ij, 64 x.  a_ii 16 x in 2^63 units, a_ij 4 x in 2^61 units of
    // the differences' products: sum_k (d^_k u_i)(d^_k u_j) with the reference's
    // product forms; the third mixed term of each is the edge product averaged.
    // S_ii 4 x, S_ij 8 x; S_ii in FP64 from the exact differences, because in a nearly
    // parallel flow a weak one times the largest a_ii is N's largest term.
    const fx a12 = fx_mul_shr<61>(Xv, dux) + fx_mul_shr<61>(Yu, dvy) + fx_mul_shr<62>(uL, vL) + fx_mul_shr<62>(uH, vH);
    const fx a13 = fx_mul_shr<61>(Xw, dux) + fx_mul_shr<61>(Zu, dwz) + fx_mul_shr<62>(uyL, wyL) + fx_mul_shr<62>(uyH, wyH);
    const fx a23 = fx_mul_shr<61>(Yw, dvy) + fx_mul_shr<61>(Zv, dwz) + fx_mul_shr<62>(vxL, wxL) + fx_mul_shr<62>(vxR, wxR);
    double No = fx_to(a12, cU + cV) * fx_raw<false>(dUy + dVx);
    No = fma(fx_to(a13, cU + cW), fx_raw<false>(dUz + dWx), No);
    No = fma(fx_to(a23, cV + cW), fx_raw<false>(dVz + dWy), No);
#define SQ(a) fx_mul_shr<63>(a, a)
    double Nd = fx_to(SQ(4 * dux) + SQ(Yu) + SQ(Zu), 2 * cU) * (fx_to<true>(d.dux, cU + su + 2) * LDG(I.rdxc + i));
    Nd = fma(fx_to(SQ(4 * dvy) + SQ(Xv) + SQ(Zv), 2 * cV), fx_to<true>(d.dvy, cV + sv + 2) * LDG(I.rdyc + jc), Nd);
    Nd = fma(fx_to(SQ(4 * dwz) + SQ(Xw) + SQ(Yw), 2 * cW), fx_to<true>(d.dwz, cW + sw + 2) * LDG(I.rdzc + k), Nd);
#undef SQ
    Nd = fma(No, pow2(min(1023, max(-1022, er + 64 - sd))), Nd);
    double v = (-0.3 * Nd) / fx_to(D, 0) * pow2(min(1023, max(-1022, em - 2 * er - 131 + 2 * sd)));
    if (bad) v = __longlong_as_double(0x7FF8000000000000LL);
    if (valid) I.S[cidx(I, i, jc, k)] = v;
    if (valid) hi = max(hi, write_nut_rows(I, i, jc, k, I.nu + chl_pos(v), [v] { return chl_pos(v); }, use_wm));
  }
  chl_line_max(I.nmax, (unsigned)(p.k * Ny + p.j), Ny, 1, hi);
}

// Vreman in fixed point (124 FP64 instructions per point before, 25 now).
// b_ij sums products of the grid-scaled differences h_m a_mi and h_m a_mj of
// components i and j, so each component is scaled by its own largest: b_22 of
// a weak V keeps its digits beside b_11.  The grid-scaled difference is the mean
// of the edge differences times h/d of their spacings (in x and z 1 but for the
// tolerance of a uniform grid).  B_b, which cancels, and the
// quotient are FP64.
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 5)
k_vreman(ChlMap map, int s_in, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, M = map.planes;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k0 = p.k * M;
  const unsigned* vm = chl_vmax(I, s_in);
  const int eu = fx_exp<61>(vm[0]), ev = fx_exp<61>(vm[1]), ew = fx_exp<61>(vm[2]);
  const bool bad = fx_bad(vm[0]) || fx_bad(vm[1]) || fx_bad(vm[2]);
  GradColumn col(I, i, jc, min(k0, Nz - 1));
  const fx wl = LDG(I.fxhyl + jc), wh = LDG(I.fxhyh + jc);      // h_y / dy below and above, 2^-62
  unsigned hi = 0u;
  for (int q = 0; q < M; ++q) {
    const int k = min(k0 + q, Nz - 1);
    const bool valid = k0 + q < Nz;
    const Diffs d = col.point(k);
    // differences of each component below 2^59 in units of 2^eU, 2^eV, 2^eW
    unsigned mu = 0u, mv = 0u, mw = 0u;
    top_or(mu, d.dux); top_or(mu, d.uyL); top_or(mu, d.uyH); top_or(mu, d.uzL); top_or(mu, d.uzH);
    top_or(mv, d.dvy); top_or(mv, d.vxL); top_or(mv, d.vxR); top_or(mv, d.vzL); top_or(mv, d.vzH);
    top_or(mw, d.dwz); top_or(mw, d.wxL); top_or(mw, d.wxR); top_or(mw, d.wyL); top_or(mw, d.wyH);
    const int su = __clz((int)mu) - 5, sv = __clz((int)mv) - 5, sw = __clz((int)mw) - 5;
    const int eU = eu - su, eV = ev - sv, eW = ew - sw;
    // grid-scaled differences, 4 x, below 2^61: rows x, y, z of u, v, w
    const fx xu = 4 * scale2(d.dux, su), yv = 4 * scale2(d.dvy, sv), zw = 4 * scale2(d.dwz, sw);
    const fx yu = 4 * (fx_mul(scale2(d.uyL, su), wl) + fx_mul(scale2(d.uyH, su), wh));
    const fx yw = 4 * (fx_mul(scale2(d.wyL, sw), wl) + fx_mul(scale2(d.wyH, sw), wh));
    // (in x and z h/dx is 1 to the 1e-9 that a grid may be off uniform)
    const int2 hx = LDG(I.hxe + i), hz = LDG(I.hze + k);
    auto mean = [](fx lo, fx hi, int s, int2 e) {
      lo = scale2(lo, s); hi = scale2(hi, s);
      return lo + hi + ((long long)(int)(lo >> 32) * e.x + (long long)(int)(hi >> 32) * e.y >> 27);
    };
    const fx zu = mean(d.uzL, d.uzH, su, hz), zv = mean(d.vzL, d.vzH, sv, hz);
    const fx xv = mean(d.vxL, d.vxR, sv, hx), xw = mean(d.wxL, d.wxR, sw, hx);
    // b_ij, 16 x, 2^64 units
    const double b11 = fx_to(fx_mul(xu, xu) + fx_mul(yu, yu) + fx_mul(zu, zu) + 4, 0);
    const double b22 = fx_to(fx_mul(xv, xv) + fx_mul(yv, yv) + fx_mul(zv, zv) + 4, 0);
    const double b33 = fx_to(fx_mul(xw, xw) + fx_mul(yw, yw) + fx_mul(zw, zw) + 4, 0);
    const double b12 = fx_to(fx_mul(xu, xv) + fx_mul(yu, yv) + fx_mul(zu, zv) + 4, 0);
    const double b13 = fx_to(fx_mul(xu, xw) + fx_mul(yu, yw) + fx_mul(zu, zw) + 4, 0);
    const double b23 = fx_to(fx_mul(xv, xw) + fx_mul(yv, yw) + fx_mul(zv, zw) + 4, 0);
    // B_b, 256 x: pairs of components with their own units
    const double q12 = b11 * b22 - b12 * b12, q13 = b11 * b33 - b13 * b13, q23 = b22 * b33 - b23 * b23;
    const int em = max(eU, max(eV, eW));
    const int n12 = max(-900, 2 * (eU + eV - 2 * em)), n13 = max(-900, 2 * (eU + eW - 2 * em)), n23 = max(-900, 2 * (eV + eW - 2 * em));
    const double Bb = fma(q12, pow2(n12), fma(q13, pow2(n13), q23 * pow2(n23)));
    // derivatives, 4 x, in units of 2^(em + er + 64), then scaled by their largest
    const fx rzc = col.rzc(k), rxc = col.rxc;
    const int du = eU - em, dv = eV - em, dw = eW - em;
    fx a1 = fx_mul(xu, rxc) >> min(63, -du), a7 = fx_mul(yu, col.ryc) >> min(63, -du), a8 = fx_mul(zu, rzc) >> min(63, -du);
    fx a4 = fx_mul(xv, rxc) >> min(63, -dv), a2 = fx_mul(yv, col.ryc) >> min(63, -dv), a9 = fx_mul(zv, rzc) >> min(63, -dv);
    fx a5 = fx_mul(xw, rxc) >> min(63, -dw), a6 = fx_mul(yw, col.ryc) >> min(63, -dw), a3 = fx_mul(zw, rzc) >> min(63, -dw);
    unsigned md = 0u;
    top_or(md, a1); top_or(md, a2); top_or(md, a3); top_or(md, a4); top_or(md, a5);
    top_or(md, a6); top_or(md, a7); top_or(md, a8); top_or(md, a9);
    const int sd = __clz((int)md) - 3;
    a1 <<= sd; a2 <<= sd; a3 <<= sd; a4 <<= sd; a5 <<= sd; a6 <<= sd; a7 <<= sd; a8 <<= sd; a9 <<= sd;
    // a_ij a_ij, 16 x, 2^64 units; 12 makes up for nine products
    const fx A = (fx_mul(a1, a1) + fx_mul(a2, a2) + fx_mul(a3, a3) + 12) +
                 (fx_mul(a4, a4) + fx_mul(a5, a5) + fx_mul(a6, a6)) +
                 (fx_mul(a7, a7) + fx_mul(a8, a8) + fx_mul(a9, a9));
    // C sqrt(B_b / a_ij a_ij): the quotient is 16 x and in units of
    // 2^(4 em + 128) / 2^(2 (em + er + 64 - sd) + 64)
    const double x = chl_sqrt(Bb / fx_to(A, 0));
    double v = (2.5 * (0.1 * 0.1) * 0.25) * x * pow2(min(1023, max(-1022, em - col.er - 32 + sd)));
    if (bad) v = __longlong_as_double(0x7FF8000000000000LL);
    if (valid) I.S[cidx(I, i, jc, k)] = v;
    if (valid) hi = max(hi, write_nut_rows(I, i, jc, k, I.nu + chl_pos(v), [v] { return chl_pos(v); }, use_wm));
  }
  chl_line_max(I.nmax, (unsigned)(p.k * Ny + p.j), Ny, 1, hi);
}

extern "C" {
void chl_launch_amd(const ChlMap& m, int nb, int s_in, int use_wm, cudaStream_t st) { chl_launch_pdl(k_amd, dim3(nb), dim3(CHL_FLUX_THREADS), 0, st, m, s_in, use_wm); }
void chl_launch_vreman(const ChlMap& m, int nb, int s_in, int use_wm, cudaStream_t st) { chl_launch_pdl(k_vreman, dim3(nb), dim3(CHL_FLUX_THREADS), 0, st, m, s_in, use_wm); }
}
