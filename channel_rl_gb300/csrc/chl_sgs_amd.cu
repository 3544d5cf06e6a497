// Anisotropic minimum-dissipation (AMD) and Vreman eddy viscosities, one
// fused kernel each, one thread per interior centre (rows 1..Ny).  Both write
// the unclipped nu_t into S and, in the same pass, nu + nu_t with k_nut's
// rules for these models (write_nut_rows): max(., 0), the ghost-row rule of
// Dirichlet_nu_t and, when use_wm, the wall-model rows - so the step runs the
// wall-stress kernels first and no separate nu_t pass.
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
// quarters of the interpolations are folded into constants (0.0625,
// 0.03125): the FP64 pipe bounds these kernels.
//
// Vreman (subgrid.f90:897-1004):
//   nu_t = C sqrt(B_b / a_ij a_ij),  C = 2.5 * 0.1^2,
//   b_ij = sum_m dx_m^2 a_mi a_mj,  B_b = b11 b22 - b12^2 + b11 b33 - b13^2 + b22 b33 - b23^2,
// a_ij = du_j/dx_i at the centre, off-diagonals the mean of four edge
// derivatives.  Two U sections of the reference are written 2:ny, 1:ny-1
// where 2:nx, 1:nx-1 are meant (subgrid.f90:930-931,946-947); they start at
// the same index, so element-wise they read the intended values, which is
// what is computed here.
#include "chl_fix.cuh"

namespace {

// Edge differences around a centre (device indices i, jc, k).  For each
// off-diagonal velocity gradient the four edge differences are summed in
// two pairs: s?L/s?H are the two-point sums on the near/far edge in the
// derivative direction (2 x the reference's first interpolation), s = sL+sH
// (4 x the centre value) and d = rl sL + rr sH (4 x the centre derivative,
// the edge differences divided by their centre-to-centre spacings first;
// along the uniform x and z that is r (sL + sH)).
// The centre strain of compute_Sij (subgrid.f90:1014-1072) is the same sums:
// S12 = (dUy + dVx)/8 from the four edges, etc.
struct Grad {
  double dux, dvy, dwz;                  // diagonal differences
  double uyL, uyH, uzL, uzH;             // U: y and z edge pair sums
  double vxL, vxR, vzL, vzH;             // V: x and z
  double wxL, wxR, wyL, wyH;             // W: x and y
  double dUy, dUz, dVx, dVz, dWx, dWy;   // 4 x centre derivatives
  double rxc, ryc, rzc;
};

__device__ __forceinline__ Grad gradients(const ChlInst& I, const double* U, const double* V, const double* W,
                                          int i, int jc, int k) {
  const int im = wrap(i - 1, I.Nx), ip = wrap(i + 1, I.Nx), km = wrap(k - 1, I.Nz), kp = wrap(k + 1, I.Nz);
  auto u = [&](int a, int j, int kk) { return LDG(U + cidx(I, a, j, kk)); };
  auto v = [&](int a, int j, int kk) { return LDG(V + vidx(I, a, j, kk)); };
  auto w = [&](int a, int j, int kk) { return LDG(W + cidx(I, a, j, kk)); };
  const double rxl = LDG(I.rdxf + i - 1), rxr = LDG(I.rdxf + i);
  const double ryl = LDG(I.rdyf + jc - 1), ryr = LDG(I.rdyf + jc);
  const double rzl = LDG(I.rdzf + k - 1), rzr = LDG(I.rdzf + k);
  Grad g;
  g.rxc = LDG(I.rdxc + i); g.ryc = LDG(I.rdyc + jc); g.rzc = LDG(I.rdzc + k);
  const double u0 = u(i, jc, k), um = u(im, jc, k);
  const double v0 = v(i, jc, k), vm = v(i, jc - 1, k);
  const double w0 = w(i, jc, k), wm = w(i, jc, km);
  g.dux = u0 - um; g.dvy = v0 - vm; g.dwz = w0 - wm;
  // U at x-faces im, i
  g.uyL = (um - u(im, jc - 1, k)) + (u0 - u(i, jc - 1, k));
  g.uyH = (u(im, jc + 1, k) - um) + (u(i, jc + 1, k) - u0);
  g.uzL = (um - u(im, jc, km)) + (u0 - u(i, jc, km));
  g.uzH = (u(im, jc, kp) - um) + (u(i, jc, kp) - u0);
  // V at y-faces jc-1, jc
  const double vmm = v(im, jc - 1, k), vm0 = v(im, jc, k);
  g.vxL = (vm - vmm) + (v0 - vm0);
  g.vxR = (v(ip, jc - 1, k) - vm) + (v(ip, jc, k) - v0);
  g.vzL = (vm - v(i, jc - 1, km)) + (v0 - v(i, jc, km));
  g.vzH = (v(i, jc - 1, kp) - vm) + (v(i, jc, kp) - v0);
  // W at z-faces km, k
  g.wxL = (wm - w(im, jc, km)) + (w0 - w(im, jc, k));
  g.wxR = (w(ip, jc, km) - wm) + (w(ip, jc, k) - w0);
  g.wyL = (wm - w(i, jc - 1, km)) + (w0 - w(i, jc - 1, k));
  g.wyH = (w(i, jc + 1, km) - wm) + (w(i, jc + 1, k) - w0);
  // y is stretched: each edge pair by its own spacing; x and z are uniform
  // (checked at creation), so one spacing times the pair sum
  (void)rxr; (void)rzr;
  g.dUy = fma(ryl, g.uyL, ryr * g.uyH); g.dUz = rzl * (g.uzL + g.uzH);
  g.dVx = rxl * (g.vxL + g.vxR); g.dVz = rzl * (g.vzL + g.vzH);
  g.dWx = rxl * (g.wxL + g.wxR); g.dWy = fma(ryl, g.wyL, ryr * g.wyH);
  return g;
}

// nu + nu_t for the interior centre (i, jc, k) from its unclipped value v,
// plus the ghost row next to the first and last interior rows; with the
// wall model on, rows 0, 1 and Ny, Ny+1 take the mean of the wall-model face
// values at x faces i-1 and i (face i-1 from the lane to the left when that
// lane is on the same row, i > 0).  Every lane of the warp reaches the
// shuffle; lanes past the instance's last centre carry valid = false.
// Returns the high word of the largest magnitude written; the ghost row's
// counts for the row next to it.
__device__ __forceinline__ unsigned write_nut_rows(const ChlInst& I, const double* U, int i, int jc, int k, double v,
                                                   int use_wm, bool valid) {
  const int Ny = I.Ny;
  const bool wmrow = valid && use_wm && I.wall_model != 0 && (jc == 1 || jc == Ny);
  const int wall = jc == 1 ? 0 : 1;
  const double f = wmrow ? wm_face(I, U, i, k, wall) : 0.0;
  const double f_left = __shfl_up_sync(0xffffffffu, f, 1);
  if (!valid) return 0u;
  const double nu = I.nu;
  double* nt = I.nut;
  if (wmrow) {
    const double fl = ((threadIdx.x & 31) > 0 && i > 0) ? f_left : wm_face(I, U, wrap(i - 1, I.Nx), k, wall);
    const double w = 0.5 * (fl + f);
    nt[cidx(I, i, jc, k)] = nu + w;
    nt[cidx(I, i, jc == 1 ? 0 : Ny + 1, k)] = nu + w;
    return chl_abshi(nu + w);
  }
  const double vc = chl_pos(v);
  nt[cidx(I, i, jc, k)] = nu + vc;
  unsigned hi = chl_abshi(nu + vc);
  if (jc == 1 || jc == Ny) {
    const double g = nu + nut_ghost(I, vc);
    if (jc == 1) nt[cidx(I, i, 0, k)] = g;
    if (jc == Ny) nt[cidx(I, i, Ny + 1, k)] = g;
    hi = max(hi, chl_abshi(g));
  }
  return hi;
}

}  // namespace

// AMD in fixed point.  As FP64 code this kernel issued 114 FP64 instructions
// per point (0.97 ms per launch at 256x96x192, the FP64 pipe 90 % busy).  The
// edge differences are exact integers from the fixed-point copies (k_fix);
// each point scales its fifteen by their largest, so that the products keep
// 54 bits or more of the largest product, and forms the derivatives, D and
// the a_ij there.  N and the division are FP64 (17 instructions).
// A thread marches through a few planes: what planes share (pair sums of
// U and V, differences of W) is carried.
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 5)   // 102 registers: 2, 3, 4, 5, 6 blocks per SM take 417, 321, 289, 288, 290 us
k_amd(ChlMap map, int s_in, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, M = map.planes;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k0 = p.k * M;
  const int im = wrap(i - 1, Nx), ip = wrap(i + 1, Nx);
  const fx* __restrict__ U = I.X[0];
  const fx* __restrict__ V = I.X[1];
  const fx* __restrict__ W = I.X[2];
#define UC(ii, jj, kk) LDG(U + cidx(I, ii, jj, kk))
#define WC(ii, jj, kk) LDG(W + cidx(I, ii, jj, kk))
#define VV(ii, jj, kk) LDG(V + vidx(I, ii, jj, kk))
  // reciprocal spacings with one exponent er
  const int el = I.eyf[jc - 1], eh = I.eyf[jc], ec = I.eyc[jc];
  const int er = max(max(max(el, eh), max(ec, I.exf)), max(max(I.exc, I.ezf), I.ezc));
  const fx ryl = LDG(I.fxryf + jc - 1) >> min(63, er - el), ryh = LDG(I.fxryf + jc) >> min(63, er - eh);
  const fx ryc = LDG(I.fxryc + jc) >> min(63, er - ec);
  const fx rxf = LDG(I.fxrxf + i - 1) >> min(63, er - I.exf), rxc = LDG(I.fxrxc + i) >> min(63, er - I.exc);
  const unsigned* vm = chl_vmax(I, s_in);
  const int eu = fx_exp<61>(vm[0]), ev = fx_exp<61>(vm[1]), ew = fx_exp<61>(vm[2]);
  const bool bad = fx_bad(vm[0]) || fx_bad(vm[1]) || fx_bad(vm[2]);
  const int ks = min(k0, Nz - 1), kb = ks == 0 ? Nz - 1 : ks - 1;    // lanes past the last plane repeat it
  fx um = UC(im, jc, ks), u0 = UC(i, jc, ks);
  fx vm0 = VV(i, jc - 1, ks), v0 = VV(i, jc, ks);
  fx wm = WC(i, jc, kb);
  fx uzL = (um + u0) - (UC(im, jc, kb) + UC(i, jc, kb));
  fx vzL = (vm0 + v0) - (VV(i, jc - 1, kb) + VV(i, jc, kb));
  fx wxl = wm - WC(im, jc, kb), wxr = WC(ip, jc, kb) - wm;          // W's x and y differences, plane below
  fx wyl = wm - WC(i, jc - 1, kb), wyh = WC(i, jc + 1, kb) - wm;
  unsigned hi = 0u;
  for (int q = 0; q < M; ++q) {
    const int k = min(k0 + q, Nz - 1), kp = k + 1 == Nz ? 0 : k + 1;
    const bool valid = k0 + q < Nz;
    const fx up_m = UC(im, jc, kp), up_0 = UC(i, jc, kp), vp_m = VV(i, jc - 1, kp), vp_0 = VV(i, jc, kp);
    const fx w0 = WC(i, jc, k), wim = WC(im, jc, k), wip = WC(ip, jc, k);
    const fx wjm = WC(i, jc - 1, k), wjp = WC(i, jc + 1, k);
    const fx us = um + u0, vs = vm0 + v0;
    fx uyL = us - (UC(im, jc - 1, k) + UC(i, jc - 1, k)), uyH = (UC(im, jc + 1, k) + UC(i, jc + 1, k)) - us;
    fx vxL = vs - (VV(im, jc - 1, k) + VV(im, jc, k)), vxR = (VV(ip, jc - 1, k) + VV(ip, jc, k)) - vs;
    const fx uzN = (up_m + up_0) - us, vzN = (vp_m + vp_0) - vs;
    const fx xl = w0 - wim, xr = wip - w0, yl = w0 - wjm, yh = wjp - w0;
    fx wxL = wxl + xl, wxR = wxr + xr, wyL = wyl + yl, wyH = wyh + yh;
    fx dux = u0 - um, dvy = v0 - vm0, dwz = w0 - wm;
    // scale: |x| < 2^60 in units of 2^et
    unsigned mu = 0u, mv = 0u, mw = 0u;
    top_or(mu, dux); top_or(mu, uyL); top_or(mu, uyH); top_or(mu, uzL); top_or(mu, uzN);
    top_or(mv, dvy); top_or(mv, vxL); top_or(mv, vxR); top_or(mv, vzL); top_or(mv, vzN);
    top_or(mw, dwz); top_or(mw, wxL); top_or(mw, wxR); top_or(mw, wyL); top_or(mw, wyH);
    const int et = max(max(eu + 64 - __clz((int)mu), ev + 64 - __clz((int)mv)), ew + 64 - __clz((int)mw)) - 60;
    const int su = eu - et, sv = ev - et, sw = ew - et;
    dux = scale2(dux, su); uyL = scale2(uyL, su); uyH = scale2(uyH, su);
    const fx uL = scale2(uzL, su), uH = scale2(uzN, su);
    dvy = scale2(dvy, sv); vxL = scale2(vxL, sv); vxR = scale2(vxR, sv);
    const fx vL = scale2(vzL, sv), vH = scale2(vzN, sv);
    dwz = scale2(dwz, sw); wxL = scale2(wxL, sw); wxR = scale2(wxR, sw); wyL = scale2(wyL, sw); wyH = scale2(wyH, sw);
    uzL = uzN; vzL = vzN; wxl = xl; wxr = xr; wyl = yl; wyh = yh;
    um = up_m; u0 = up_0; vm0 = vp_m; v0 = vp_0; wm = w0;
    // grid-scaled centre differences, 4 x
    const fx Yu = uyL + uyH, Zu = uL + uH, Xv = vxL + vxR, Zv = vL + vH, Xw = wxL + wxR, Yw = wyL + wyH;
    // derivatives, 4 x, scaled anew: the spacings differ by up to the
    // stretching of the grid (units 2^(et + er + 64 - sd))
    const fx rzf = LDG(I.fxrzf + k - 1) >> min(63, er - I.ezf), rzc = LDG(I.fxrzc + k) >> min(63, er - I.ezc);
    fx s11 = 4 * fx_mul(dux, rxc), s22 = 4 * fx_mul(dvy, ryc), s33 = 4 * fx_mul(dwz, rzc);
    fx dUy = fx_mul(uyL, ryl) + fx_mul(uyH, ryh), dWy = fx_mul(wyL, ryl) + fx_mul(wyH, ryh);
    fx dUz = fx_mul(Zu, rzf), dVz = fx_mul(Zv, rzf), dVx = fx_mul(Xv, rxf), dWx = fx_mul(Xw, rxf);
    unsigned md = 0u;
    top_or(md, s11); top_or(md, s22); top_or(md, s33);
    top_or(md, dUy); top_or(md, dUz); top_or(md, dVx); top_or(md, dVz); top_or(md, dWx); top_or(md, dWy);
    const int sd = __clz((int)md) - 3;     // |x| < 2^61; a derivative is below 2^61 already
    s11 <<= sd; s22 <<= sd; s33 <<= sd;
    dUy <<= sd; dUz <<= sd; dVx <<= sd; dVz <<= sd; dWx <<= sd; dWy <<= sd;
    // D, 16 x (2^64 units of the derivatives' square); 12 makes up for nine products
    const fx D = (fx_mul(s11, s11) + fx_mul(s22, s22) + fx_mul(s33, s33) + 12) +
                 (fx_mul(dUy, dUy) + fx_mul(dUz, dUz) + fx_mul(dVx, dVx)) +
                 (fx_mul(dVz, dVz) + fx_mul(dWx, dWx) + fx_mul(dWy, dWy));
    // a_ii 16 x in 2^63 units, a_ij 4 x in 2^61 units of the differences' square:
    // sum_k (d^_k u_i)(d^_k u_j) with the reference's product forms; the third
    // mixed term of each is the edge product averaged
#define SQ(a) fx_mul_shr<63>(a, a)
    const fx a11 = SQ(4 * dux) + SQ(Yu) + SQ(Zu), a22 = SQ(4 * dvy) + SQ(Xv) + SQ(Zv), a33 = SQ(4 * dwz) + SQ(Xw) + SQ(Yw);
#undef SQ
    const fx a12 = fx_mul_shr<61>(Xv, dux) + fx_mul_shr<61>(Yu, dvy) + fx_mul_shr<62>(uL, vL) + fx_mul_shr<62>(uH, vH);
    const fx a13 = fx_mul_shr<61>(Xw, dux) + fx_mul_shr<61>(Zu, dwz) + fx_mul_shr<62>(uyL, wyL) + fx_mul_shr<62>(uyH, wyH);
    const fx a23 = fx_mul_shr<61>(Yw, dvy) + fx_mul_shr<61>(Zv, dwz) + fx_mul_shr<62>(vxL, wxL) + fx_mul_shr<62>(vxR, wxR);
    // N = sum a_ij S_ij, 64 x (S_ii 4 x, a_ij 4 x with S_ij 8 x in 2^-2 units of a_ii)
    double Nd = fx_raw<true>(a11) * fx_raw<false>(s11);
    Nd = fma(fx_raw<true>(a22), fx_raw<false>(s22), Nd);
    Nd = fma(fx_raw<false>(a33), fx_raw<false>(s33), Nd);
    Nd = fma(fx_raw<false>(a12), fx_raw<false>(dUy + dVx), Nd);
    Nd = fma(fx_raw<false>(a13), fx_raw<false>(dUz + dWx), Nd);
    Nd = fma(fx_raw<false>(a23), fx_raw<false>(dVz + dWy), Nd);
    double v = (-0.3 * Nd) / fx_to(D, 0) * pow2(min(1023, max(-1022, et - er - 67 + sd)));
    if (bad) v = __longlong_as_double(0x7FF8000000000000LL);
    if (valid) I.S[cidx(I, i, jc, k)] = v;
    hi = max(hi, write_nut_rows(I, I.U[s_in], i, jc, k, v, use_wm, valid));
  }
#undef UC
#undef WC
#undef VV
  chl_line_max(I.nmax, (unsigned)(p.k * Ny + p.j), Ny, 1, hi);
}

__global__ void __launch_bounds__(256)
k_vreman(ChlMap map, int s_in, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const bool valid = t < (unsigned)(Nx * Ny * Nz);
  const ChlIdx p = chl_split(valid ? t : (unsigned)(Nx * Ny * Nz) - 1u, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k = p.k;
  const Grad g = gradients(I, I.U[s_in], I.V[s_in], I.W[s_in], i, jc, k);
  // a_ij = du_j/dx_i (reference layout 1 4 5 / 7 2 6 / 8 9 3); the
  // off-diagonal entries are kept 4 x (the 1/16 is folded below)
  const double a1 = g.dux * g.rxc, a2 = g.dvy * g.ryc, a3 = g.dwz * g.rzc;
  const double a4 = g.dVx, a5 = g.dWx, a7 = g.dUy, a6 = g.dWy, a8 = g.dUz, a9 = g.dVz;
  const double hx = LDG(I.hx2 + i), hy = LDG(I.hy2 + jc), hz = LDG(I.hz2 + k);
  const double qx = 0.0625 * hx, qy = 0.0625 * hy, qz = 0.0625 * hz;
  // b_ij = sum_m dx_m^2 a_mi a_mj
  const double b11 = fma(hx * a1, a1, fma(qy * a7, a7, qz * a8 * a8));
  const double b22 = fma(qx * a4, a4, fma(hy * a2, a2, qz * a9 * a9));
  const double b33 = fma(qx * a5, a5, fma(qy * a6, a6, hz * a3 * a3));
  const double hx4 = 0.25 * hx, hy4 = 0.25 * hy, hz4 = 0.25 * hz;
  const double b12 = fma(hx4 * a1, a4, fma(hy4 * a7, a2, qz * a8 * a9));
  const double b13 = fma(hx4 * a1, a5, fma(qy * a7, a6, hz4 * a8 * a3));
  const double b23 = fma(qx * a4, a5, fma(hy4 * a2, a6, hz4 * a9 * a3));
  const double Bb = b11 * b22 - b12 * b12 + b11 * b33 - b13 * b13 + b22 * b33 - b23 * b23;
  double Ab = a1 * a1;
  Ab = fma(a2, a2, Ab); Ab = fma(a3, a3, Ab);
  double Ao = a4 * a4;
  Ao = fma(a5, a5, Ao); Ao = fma(a6, a6, Ao); Ao = fma(a7, a7, Ao); Ao = fma(a8, a8, Ao); Ao = fma(a9, a9, Ao);
  Ab = fma(0.0625, Ao, Ab);
  const double v = 2.5 * (0.1 * 0.1) * chl_sqrt(Bb / Ab);
  if (valid) I.S[cidx(I, i, jc, k)] = v;
  chl_line_max(I.nmax, (unsigned)(k * Ny + jc - 1), Ny, 1, write_nut_rows(I, I.U[s_in], i, jc, k, v, use_wm, valid));
}

extern "C" {
void chl_launch_amd(const ChlMap& m, int nb, int s_in, int use_wm, cudaStream_t st) { chl_launch_pdl(k_amd, dim3(nb), dim3(CHL_FLUX_THREADS), 0, st, m, s_in, use_wm); }
void chl_launch_vreman(const ChlMap& m, int nb, int s_in, int use_wm, cudaStream_t st) { chl_launch_pdl(k_vreman, dim3(nb), dim3(m.tb), 0, st, m, s_in, use_wm); }
}
