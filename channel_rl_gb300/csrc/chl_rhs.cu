// Momentum right-hand side and Runge-Kutta stage update.
//
// Restates compute_rhs_u/v/w (equations.f90:24-468) - advection by the
// reference's interpolations (interpolation.f90:24-105: plain averages in x
// and z, weight_y_0/1 averages in y) plus variable-viscosity diffusion - and
// the stage update of compute_time_step_RK3 (time_integration.f90:42-81)
// with the Dirichlet ghost rows of apply_Dirichlet_bc_y
// (boundary_conditions.f90:239-254).
//
// The reference sums each derivative's advective and viscous part per
// component; here the same terms are grouped by the face they live on
// (flux form), so every face value is computed once:
//   * cell centres     : the diagonal fluxes of u (x), v (y), w (z);
//   * xy edges (x-face, y-face, z-centre): uv and the edge viscosity, shared
//                        by the y flux of u and the x flux of v;
//   * xz edges (x-face, y-centre, z-face): uw, shared by u (z) and w (x);
//   * yz edges (x-centre, y-face, z-face): vw, shared by v (z) and w (y).
// The edge viscosities are exactly the reference's averages (nu_y1/nu_y2 of
// compute_rhs_u equal nu_x1/nu_x2 of compute_rhs_v at the same edge, etc.).
// I.nut holds nu + nu_t, so no per-use "nu +" is needed.
//
// Both kernels work in 64-bit fixed point (chl_fix.cuh): as FP64 code they
// were bound by the FP64 pipe (52 and 24 instructions per point, 457 and 201
// us per launch at 256x96x192; 192 and 135 now).  The velocities are scaled by
// their rows' largest, the fluxes are kept as integers, and only the three
// components of F and the two FMAs of the stage update are FP64.  Halves and quarters of the averages are exponents.  The y-face
// value of u (and w) is u_a + w1 (u_b - u_a).
#include "chl_fix.cuh"

// flux fields: centre-like (rows 1..Ny): 0 GUx, 1 GVy, 2 GWz, 3 GUz, 4 GWx;
// V-like (rows 0..Ny): 5 GUy, 6 GVx, 7 GVz, 8 GWy
enum { G_UX = 0, G_VY, G_WZ, G_UZ, G_WX, G_UY, G_VX, G_VZ, G_WY };

// Exponents of the velocities that the fluxes of y-face j and centre row j take
// (U and W of rows j and j + 1, V of faces j - 1 and j), from those rows' largest.
// Next to a resolved wall V is a millionth of its largest and less, U a hundredth:
// in units of the field's largest the rows there had up to 35 roundings of error
// (FP64 and this 3), and more the stronger the grid is stretched.  x, y, z are the
// exponents, w whether a velocity is not finite; left in vexp by k_fix.
__device__ __forceinline__ int4 vel_exp(const ChlInst& I, int j) {
  const int a = max(j, 1), b = min(j + 1, I.Ny);
  const unsigned u = max(chl_row_max(I, 0, a), chl_row_max(I, 0, b));
  const unsigned v = max(chl_row_max(I, 1, max(j - 1, 0)), chl_row_max(I, 1, j));
  const unsigned w = max(chl_row_max(I, 2, a), chl_row_max(I, 2, b));
  return make_int4(fx_exp<61>(u), fx_exp<61>(v), fx_exp<61>(w), fx_bad(u) || fx_bad(v) || fx_bad(w));
}

// Exponents of the fluxes of row j, from those of its velocities and the largest
// |nu + nu_t| of the row and the one above.  Flux m = viscous - advective part: the
// advective product has last bit 2^adv[m], the viscous one 2^vis[m]; the
// fluxes of one momentum component are stored with last bit 2^G, one above
// the largest, so that |flux| < 2^62.  A row whose fluxes may exceed a double's
// range counts as not finite, as their overflow in FP64 would have it.
#define FLUX_G_MAX 962
__device__ constexpr int FLUX_A[9] = {0, 1, 2, 0, 2, 0, 1, 1, 2};   // momentum component
__device__ constexpr int FLUX_B[9] = {0, 1, 2, 2, 0, 1, 0, 2, 1};   // direction
struct RowExp { int adv[9], vis[9], G[3], n; bool bad; };
__device__ __forceinline__ RowExp row_exp(const ChlInst& I, int4 x, int j) {
  const unsigned nm = max(I.nmax[j], I.nmax[j + 1]);
  const int ev[3] = {x.x, x.y, x.z};
  const int ef[3] = {I.exf, I.eyf[j], I.ezf}, ec[3] = {I.exc, I.eyc[j], I.ezc};
  RowExp q;
  q.n = fx_exp<60>(nm);
  q.G[0] = q.G[1] = q.G[2] = -100000;
#pragma unroll
  for (int m = 0; m < 9; ++m) {
    const int a = FLUX_A[m], b = FLUX_B[m];
    // factors of the averages: one half in the products on y-face edges, a
    // quarter in the others; viscosity 1, 4 and 2 x at centres, xz and y-face edges
    q.adv[m] = ev[a] + ev[b] + (m >= G_UY ? 61 : 60);
    q.vis[m] = q.n + ev[a] + (m <= G_WZ ? ec[b] + 125 : m <= G_WX ? ef[b] + 123 : ef[b] + 124);
    q.G[a] = max(q.G[a], max(q.adv[m], q.vis[m]) + 1);
  }
  q.bad = x.w || fx_bad(nm) || max(q.G[0], max(q.G[1], q.G[2])) > FLUX_G_MAX;
  return q;
}

// Row coefficient of the static model, nu_t = coef |S|/sqrt(2): van Driest
// damping f = 1 - exp(-d/25/(nu/utau)), utau = dPdx^0.5 (subgrid.f90:581-599).
static __device__ __noinline__ double smag_coef(const ChlInst& I, int jc) {
  const double ut = sqrt(I.scal[CHL_S_DPDX]);
  double f = 1.0 - exp(-I.smag_dwall[jc] / 25.0 / (I.nu / ut));
  if (I.Dirichlet_nu_t == 0) f = 1.0;
  const double cd = I.smag_csdelta[jc] * f;   // Cs*Delta_j*f
  return cd * cd * 1.41421356237309504880;    // (Cs Delta f)^2 |S| with S holding |S|/sqrt(2)
}

// k_fix's work for row j.  A call, for the registers.
static __device__ __noinline__ void fix_row(const ChlInst& I, int s, int j, int prep) {
  if (prep) {
    I.nmax[j] = I.smax[j] = 0u;
    if (prep & 2) I.coef[j] = j >= 1 && j <= I.Ny ? smag_coef(I, j) : 0.0;
  }
  if (j > I.Ny) return;
  const int4 x = vel_exp(I, j);
  I.vexp[j] = x;
  if (j >= 1 && I.LES_model == 2) {      // dynamic model
    // centre row j with the rows of faces that the test filter brings into it
    const int a = max(j - 1, 1);
    const int u = max(x.x, fx_exp<61>(chl_row_max(I, 0, a))), w = max(x.z, fx_exp<61>(chl_row_max(I, 2, a)));
    const int v = max(x.y, fx_exp<61>(max(chl_row_max(I, 1, max(j - 2, 0)), chl_row_max(I, 1, min(j + 1, I.Ny)))));
    const unsigned* vm = chl_vmax(I, s);
    I.slack[j] = make_int4(min(24, fx_exp<61>(vm[0]) - u), min(24, fx_exp<61>(vm[1]) - v), min(24, fx_exp<61>(vm[2]) - w), 0);
  }
}

// Fixed-point copies of the velocity set that a stage works on (rows as
// stored, ghosts included).  prep: 1 clears the rows' largest |nu + nu_t|
// and |S| S_ij ahead of the kernels that form them, + 2 forms the static
// model's row coefficients.  Also forms the exponents of the rows' velocities for
// k_flux, from what the set's writer folded.  Moves 48 bytes per point: HBM-bound.
// An instance's first blocks do what goes by rows (a thread per row), beside the
// others: in blocks that also copy it added 1 us to a launch of 8.
__global__ void __launch_bounds__(256)
k_fix(ChlMap map, int s, int prep) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  // pairs of points (Nx is even)
  const unsigned nc = (unsigned)(I.Nx * (I.Ny + 2) * I.Nz) / 2, nv = (unsigned)(I.Nx * (I.Ny + 1) * I.Nz) / 2;
  // threads of the blocks of rows (blockDim is a power of two)
  const unsigned rows = ((unsigned)I.Ny + 1u + blockDim.x) & ~(blockDim.x - 1u);
  unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  if (t < rows) {
    if ((int)t <= I.Ny + 1) fix_row(I, s, (int)t, prep);
    return;
  }
  t -= rows;
  const unsigned* vm = chl_vmax(I, s);
  const int eu = fx_exp<61>(vm[0]), ev = fx_exp<61>(vm[1]), ew = fx_exp<61>(vm[2]);
  auto put = [t](fx* x, double2 v, int e) { reinterpret_cast<longlong2*>(x)[t] = make_longlong2(fx_from(v.x, e), fx_from(v.y, e)); };
  auto get = [t](const double* x) { return __ldg(reinterpret_cast<const double2*>(x) + t); };
  double2 u, v, w;
  if (t < nc) { u = get(I.U[s]); w = get(I.W[s]); }
  if (t < nv) v = get(I.V[s]);
  if (t < nc) { put(I.X[0], u, eu); put(I.X[2], w, ew); }
  if (t < nv) put(I.X[1], v, ev);
}

// Fluxes next to a wall whose nu + nu_t the wall model sets (y-faces 0, 1 and
// Ny-1, Ny, centre rows 1 and Ny).  It is tau dyw/du there, without a bound where
// the wall shear passes zero, and with one unit per row the largest of a row takes
// the digits of all its points: one with 1e-9 of the others' shear left 7 of them,
// one with none left NaN.  So each of these fluxes has a unit of its own, from the
// nu + nu_t of its edge, and is stored as a double.
__device__ __forceinline__ bool wall_face(const ChlInst& I, int j) { return I.wall_model != 0 && (j <= 1 || j >= I.Ny - 1); }
__device__ __forceinline__ bool wall_centre(const ChlInst& I, int j) { return I.wall_model != 0 && (j == 1 || j == I.Ny); }

// x as m 2^e, |m| < 2^61 (0 for a subnormal x)
struct Norm {
  fx m; int e; bool bad;
  __device__ __forceinline__ explicit Norm(double x) {
    const long long b = __double_as_longlong(x);
    const int x11 = (int)(b >> 52) & 0x7FF;
    const fx f = (fx)(((unsigned long long)b << 12 >> 4) | (1ULL << 60));
    m = x11 == 0 ? 0 : (b < 0 ? -f : f);
    e = x11 - 1083;
    bad = x11 == 0x7FF;
  }
};

// One of these: of y-face j (of a wall's only those that a row takes) or of centre
// row j at (i, k).  The averages of nu + nu_t are its only FP64 instructions, 4 and 3
// per point (in FP64 throughout, 28 and 24, they cost the 128x40x64 channel 6 % of a
// step).  A call, for the registers.
static __device__ __noinline__ void flux_wall(const ChlInst& I, int sin, int i, int j, int k, bool centre) {
  const int Nx = I.Nx, Nz = I.Nz, ip = wrap(i + 1, Nx), kp = wrap(k + 1, Nz);
  const int4 x = LDG(I.vexp + j);
  const int eu = x.x, ev = x.y, ew = x.z;
  auto u = [&](int a, int b, int kk) { return fx_from(LDG(I.U[sin] + cidx(I, a, b, kk)), eu); };
  auto v = [&](int a, int b, int kk) { return fx_from(LDG(I.V[sin] + vidx(I, a, b, kk)), ev); };
  auto w = [&](int a, int b, int kk) { return fx_from(LDG(I.W[sin] + cidx(I, a, b, kk)), ew); };
  auto n = [&](int a, int b, int kk) { return LDG(I.nut + cidx(I, a, b, kk)); };
  // viscous less advective part: vis 2^ev less adv 2^ea
  auto put = [&](int m, size_t q, fx adv, int ea, const Norm& nu, fx grad, int ev) {
    ev += nu.e;
    const int g = max(ea, ev) + 1;
    const double f = fx_to((fx_mul_shr<61>(nu.m, grad) >> min(63, g - ev)) - (adv >> min(63, g - ea)), g);
    reinterpret_cast<double*>(I.G[m])[q] = x.w || nu.bad || g > FLUX_G_MAX ? __longlong_as_double(0x7FF8000000000000LL) : f;
  };
  const fx rxf = LDG(I.fxrxf + i), rzf = LDG(I.fxrzf + k);
  const fx ua = u(i, j, k), wa = w(i, j, k), v0 = v(i, j, k);
  const double na = n(i, j, k), nx = n(ip, j, k), nz = n(i, j, kp);
  if (!centre) {
    const int jp = j + 1, eyf = I.eyf[j];
    const fx ryf = LDG(I.fxryf + j), w1 = LDG(I.fxw1 + j);
    const double w0x2 = LDG(I.w0x2 + j), w1x2 = LDG(I.w1x2 + j);
    const fx du = u(i, jp, k) - ua, dw = w(i, jp, k) - wa, vz = v(i, j, kp), vp = v(ip, j, k);
    const double nb = n(i, jp, k);
    const size_t e = vidx(I, i, j, k);
    // yz edge: 2 v w, 4 nu; xy edge: 2 u v, 4 nu
    const fx vw = fx_mul_shr<62>(wa + 2 * fx_mul(dw, w1), v0 + vz), uv = fx_mul_shr<62>(ua + 2 * fx_mul(du, w1), v0 + vp);
    const Norm nyz(fma(w0x2, na + nz, w1x2 * (nb + n(i, jp, kp))));
    const Norm nxy(fma(w0x2, na + nx, w1x2 * (nb + n(ip, jp, k))));
    put(G_WY, e, vw, ev + ew + 61, nyz, fx_mul(dw, ryf), ew + eyf + 123);
    put(G_UY, e, uv, eu + ev + 61, nxy, fx_mul(du, ryf), eu + eyf + 123);
    if (j != 0 && j != I.Ny) {
      put(G_VZ, e, vw, ev + ew + 61, nyz, fx_mul(vz - v0, rzf), ev + I.ezf + 123);
      put(G_VX, e, uv, eu + ev + 61, nxy, fx_mul(vp - v0, rxf), ev + I.exf + 123);
    }
    return;
  }
  const size_t c = cidx(I, i, j, k);
  const fx um = u(wrap(i - 1, Nx), j, k), vm = v(i, j - 1, k), wm = w(i, j, wrap(k - 1, Nz));
  const fx su = um + ua, sv = vm + v0, sw = wm + wa;
  const fx uz = u(i, j, kp), wp = w(ip, j, k), uw = fx_mul_shr<62>(ua + uz, wa + wp);
  // xz edge: 4 u w, 4 nu; cell centre: u u with both halves in the exponent, nu
  const Norm nxz((na + nx) + (nz + n(ip, j, kp))), nu(na);
  put(G_UX, c, fx_mul_shr<62>(su, su), 2 * eu + 60, nu, fx_mul(ua - um, LDG(I.fxrxc + i)), eu + I.exc + 125);
  put(G_VY, c, fx_mul_shr<62>(sv, sv), 2 * ev + 60, nu, fx_mul(v0 - vm, LDG(I.fxryc + j)), ev + I.eyc[j] + 125);
  put(G_WZ, c, fx_mul_shr<62>(sw, sw), 2 * ew + 60, nu, fx_mul(wa - wm, LDG(I.fxrzc + k)), ew + I.ezc + 125);
  put(G_UZ, c, uw, eu + ew + 60, nxz, fx_mul(uz - ua, rzf), eu + I.ezf + 123);
  put(G_WX, c, uw, eu + ew + 60, nxz, fx_mul(wp - wa, rxf), ew + I.exf + 123);
}

// 28 products and 4 conversions of nu + nu_t per point on the integer pipe, 9
// conversions of velocities: 7 on the FP64 pipe, which nothing else here uses, 2 on
// the integer pipe (9 and 0, 8 and 1, 4 and 5, 0 and 9: 2 to 4 % more); 104 bytes
// per point.  A thread marches through a few planes at its (i, j), so that what
// the next plane shares (U, V, nu + nu_t one plane up, W one down) is loaded and
// converted once.
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 6)
k_flux(ChlMap map, int sin) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const int M = map.planes;
  // with a wall model the first blocks form the walls' own fluxes, a point each,
  // and the others leave out rows 0, 1 and Ny
  const bool wm = I.wall_model != 0;
  const int nw = wm ? chl_wall_flux_blocks(Nx, Nz) : 0;
  if (lb < nw) {
    const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
    if (t >= (unsigned)(6 * Nx * Nz)) return;
    const ChlIdx p = chl_split(t, Nx, 6);       // centre rows 1, Ny; y-faces 1, Ny-1, 0, Ny
    flux_wall(I, sin, p.i, p.j == 4 ? 0 : ((p.j & 1) == 0 ? 1 : (p.j == 3 ? Ny - 1 : Ny)), p.k, p.j < 2);
    return;
  }
  const unsigned t = (unsigned)(lb - nw) * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, wm ? Ny - 2 : Ny + 1);
  const int i = p.i, j = p.j + (wm ? 2 : 0), k0 = p.k * M, k1 = min(Nz, k0 + M);
  const double* __restrict__ U = I.U[sin];
  const double* __restrict__ V = I.V[sin];
  const double* __restrict__ W = I.W[sin];
  const double* __restrict__ nt = I.nut;   // nu + nu_t
  const bool valid = k0 < Nz;
  const int4 x = LDG(I.vexp + j);
  const fx w1 = LDG(I.fxw1 + j), rxf = LDG(I.fxrxf + i), ryf = LDG(I.fxryf + j);
  const fx rxc = LDG(I.fxrxc + i), ryc = LDG(I.fxryc + j);
  const int ip = wrap(i + 1, Nx), im = wrap(i - 1, Nx);
  const int jp = min(j + 1, Ny + 1), jm = max(j - 1, 0);
  double u_a0 = 0.0, v_00 = 0.0, w_m0 = 0.0;
  double dn_a = 0.0, dn_b = 0.0, dn_p = 0.0;
  if (valid) {
    u_a0 = LDG(U + cidx(I, i, j, k0));
    v_00 = LDG(V + vidx(I, i, j, k0));
    w_m0 = LDG(W + cidx(I, i, j, k0 == 0 ? Nz - 1 : k0 - 1));
    dn_a = LDG(nt + cidx(I, i, j, k0)); dn_b = LDG(nt + cidx(I, i, jp, k0)); dn_p = LDG(nt + cidx(I, ip, j, k0));
  }
  if (!valid) return;
  const bool own = wm && j == Ny - 1;        // the face above this centre row is the wall's
  const FxConv cu(x.x), cv(x.y), cw(x.z);
  fx u_a = cu(u_a0), v_0 = cv(v_00), w_m = cw(w_m0);
  int sa[9], sv_[9];          // right shifts of the advective and viscous parts
  int en;
  {
    const RowExp q = row_exp(I, x, j);
    en = q.n;
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      sa[m] = min(63, q.G[FLUX_A[m]] - q.adv[m]);
      sv_[m] = min(63, q.G[FLUX_A[m]] - q.vis[m]);
    }
    if (i == 0 && k0 == 0) I.upd[j] = make_int4(q.G[0], q.G[1], q.G[2], q.bad);   // for k_rhs_update
  }
  fx n_a = fx_from(dn_a, en), n_b = fx_from(dn_b, en), n_p = fx_from(dn_p, en);
#define MUL fx_mul
#define ADV fx_mul_shr<62>
#define VIS fx_mul_shr<61>
#define PUT(m, e, adv, vis) I.G[m][e] = ((vis) >> sv_[m]) - ((adv) >> sa[m])
  for (int k = k0; k < k1; ++k) {
    const int kp = k + 1 == Nz ? 0 : k + 1;
    const size_t c = cidx(I, i, j, k), e = vidx(I, i, j, k);
    const fx u_b = cu(LDG(U + cidx(I, i, jp, k))), w_b = cw(LDG(W + cidx(I, i, jp, k)));
    const fx w_a = cw(LDG(W + c));
    const fx u_z = fx_from(LDG(U + cidx(I, i, j, kp)), x.x), v_z = cv(LDG(V + vidx(I, i, j, kp))), v_p = cv(LDG(V + vidx(I, ip, j, k)));
    const fx n_az = fx_from(LDG(nt + cidx(I, i, j, kp)), en), n_bz = fx_from(LDG(nt + cidx(I, i, jp, kp)), en);
    const fx n_pz = fx_from(LDG(nt + cidx(I, ip, j, kp)), en), n_bp = fx_from(LDG(nt + cidx(I, ip, jp, k)), en);
    const fx rzf = LDG(I.fxrzf + k);
    const fx nx_a = n_a + n_p;             // x pair of row j: the xy and xz edges share it
    if (!own) {  // yz edge (x-centre i, y-face j, z-face k): vw, nu -> GVz, GWy
      const fx dw = w_b - w_a;
      const fx vw = ADV(w_a + 2 * MUL(dw, w1), v_0 + v_z);                            // 2 v w
      const fx na = n_a + n_az;
      const fx nyz = na + 2 * MUL(n_b + n_bz - na, w1);                               // 2 nu
      PUT(G_VZ, e, vw, VIS(nyz, MUL(v_z - v_0, rzf)));
      PUT(G_WY, e, vw, VIS(nyz, MUL(dw, ryf)));
    }
    if (!own) {  // xy edge (x-face i, y-face j, z-centre k): uv, nu -> GUy, GVx
      const fx du = u_b - u_a;
      const fx uv = ADV(u_a + 2 * MUL(du, w1), v_0 + v_p);                            // 2 u v
      const fx nxy = nx_a + 2 * MUL(n_b + n_bp - nx_a, w1);                           // 2 nu
      PUT(G_UY, e, uv, VIS(nxy, MUL(du, ryf)));
      PUT(G_VX, e, uv, VIS(nxy, MUL(v_p - v_0, rxf)));
    }
    if (j >= 1) {
      {  // cell centre: diagonal fluxes
        const fx u_m = cu(LDG(U + cidx(I, im, j, k))), v_m = fx_from(LDG(V + vidx(I, i, jm, k)), x.y);
        const fx su = u_m + u_a, sv = v_m + v_0, sw = w_m + w_a;
        PUT(G_UX, c, ADV(su, su), VIS(n_a, MUL(u_a - u_m, rxc)));
        PUT(G_VY, c, ADV(sv, sv), VIS(n_a, MUL(v_0 - v_m, ryc)));
        PUT(G_WZ, c, ADV(sw, sw), VIS(n_a, MUL(w_a - w_m, LDG(I.fxrzc + k))));
      }
      {  // xz edge (x-face i, y-centre jc, z-face k): uw, nu -> GUz, GWx
        const fx w_p = cw(LDG(W + cidx(I, ip, j, k)));
        const fx uw = ADV(u_a + u_z, w_a + w_p);                                      // 4 u w
        const fx nxz = nx_a + (n_az + n_pz);                                          // 4 nu
        PUT(G_UZ, c, uw, VIS(nxz, MUL(u_z - u_a, rzf)));
        PUT(G_WX, c, uw, VIS(nxz, MUL(w_p - w_a, rxf)));
      }
    }
    u_a = u_z; v_0 = v_z; w_m = w_a; n_a = n_az; n_b = n_bz; n_p = n_pz;
  }
#undef MUL
#undef ADV
#undef VIS
#undef PUT
}

struct RhsArgs {
  int sbase, sout;        // velocity sets: stage base (U^n), output
  int stage;              // RK3 stage 0..2: out = base + dt (c1 F1 + c2 F) (chl_put_dt's products)
  int mode;               // 0: stage 1 (store F1), 1: stages 2/3, 2: actual-pressure RHS only
};

// A difference of y fluxes, whose rows have their own exponents.
__device__ __forceinline__ double row_diff(fx hi, int eh, fx lo, int el) {
  const int m = max(eh, el);
  return fx_to<true>((hi >> min(63, m - eh)) - (lo >> min(63, m - el)), m);
}

// A flux as a double: stored so (next to a modelled wall) or in its row's unit 2^e.
__device__ __forceinline__ double flux_val(fx f, bool dbl, int e) { return dbl ? __longlong_as_double(f) : fx_to<true>(f, e); }

// F at x points i (even) and i + 1 of row jc, plane k.  WALL: a row next to a
// modelled wall, where some of the fluxes are doubles.
struct Rhs { double2 u, v, w; };
template <bool WALL>
__device__ __forceinline__ Rhs rhs_pair(const ChlInst& I, int i, int jc, int k) {
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const int im = wrap(i - 1, Nx), ip = wrap(i + 2, Nx);
  const int km = wrap(k - 1, Nz), kp = wrap(k + 1, Nz);
  const fx* const* G = I.G;
  const bool hasv = jc <= Ny - 1;
  const size_t c = cidx(I, i, jc, k), e = vidx(I, i, jc, k), em = vidx(I, i, jc - 1, k);
  auto g2 = [](const fx* f, size_t q) { return __ldg(reinterpret_cast<const longlong2*>(f + q)); };
  const double rxc0 = LDG(I.rdxc + i), rxc1 = LDG(I.rdxc + i + 1), rxf0 = LDG(I.rdxf + i), rxf1 = LDG(I.rdxf + i + 1);
  const double ryc = LDG(I.rdyc + jc), ryf = LDG(I.rdyf + jc);
  const double rzc = LDG(I.rdzc + k), rzf = LDG(I.rdzf + k), dpdx = I.scal[CHL_S_DPDX];
  // exponents of the fluxes of rows jc - 1, jc, jc + 1
  const int4 e0 = LDG(I.upd + jc), el = LDG(I.upd + jc - 1), eh = LDG(I.upd + min(jc + 1, Ny));
  // stored as doubles: y-faces jc - 1 and jc, centre rows jc and jc + 1
  const bool dl = WALL && wall_face(I, jc - 1), dh = WALL && wall_face(I, jc), dc = WALL && wall_centre(I, jc);
  const bool dn = WALL && wall_centre(I, jc + 1);
  // difference of two fluxes of one row (of doubles on the integer pipe: the FP64
  // pipe has the products) and of two rows
  auto diff = [](fx hi, fx lo, bool d, int x) {
    return WALL && d ? fx_sub(__longlong_as_double(hi), __longlong_as_double(lo)) : fx_to<true>(hi - lo, x);
  };
  auto ydiff = [](fx hi, bool dhi, int ehi, fx lo, bool dlo, int elo) {
    return WALL ? flux_val(hi, dhi, ehi) - flux_val(lo, dlo, elo) : row_diff(hi, ehi, lo, elo);
  };
  Rhs F;
  F.v = make_double2(0.0, 0.0);
  {  // u at (x-face i, row jc, z-centre k)
    const longlong2 x = g2(G[G_UX], c), yh = g2(G[G_UY], e), yl = g2(G[G_UY], em);
    const longlong2 zh = g2(G[G_UZ], c), zl = g2(G[G_UZ], cidx(I, i, jc, km));
    const fx xp = LDG(G[G_UX] + cidx(I, ip, jc, k));
    F.u.x = fma(diff(x.y, x.x, dc, e0.x), rxf0, dpdx);
    F.u.y = fma(diff(xp, x.y, dc, e0.x), rxf1, dpdx);
    F.u.x = fma(ydiff(yh.x, dh, e0.x, yl.x, dl, el.x), ryc, F.u.x);
    F.u.y = fma(ydiff(yh.y, dh, e0.x, yl.y, dl, el.x), ryc, F.u.y);
    F.u.x = fma(diff(zh.x, zl.x, dc, e0.x), rzc, F.u.x);
    F.u.y = fma(diff(zh.y, zl.y, dc, e0.x), rzc, F.u.y);
  }
  {  // w at (x-centre i, row jc, z-face k)
    const longlong2 x = g2(G[G_WX], c), yh = g2(G[G_WY], e), yl = g2(G[G_WY], em);
    const longlong2 zl = g2(G[G_WZ], c), zh = g2(G[G_WZ], cidx(I, i, jc, kp));
    const fx xm = LDG(G[G_WX] + cidx(I, im, jc, k));
    F.w.x = diff(x.x, xm, dc, e0.z) * rxc0;
    F.w.y = diff(x.y, x.x, dc, e0.z) * rxc1;
    F.w.x = fma(ydiff(yh.x, dh, e0.z, yl.x, dl, el.z), ryc, F.w.x);
    F.w.y = fma(ydiff(yh.y, dh, e0.z, yl.y, dl, el.z), ryc, F.w.y);
    F.w.x = fma(diff(zh.x, zl.x, dc, e0.z), rzf, F.w.x);
    F.w.y = fma(diff(zh.y, zl.y, dc, e0.z), rzf, F.w.y);
  }
  if (hasv) {  // v at (x-centre i, y-face jv = jc, z-centre k)
    const longlong2 x = g2(G[G_VX], e), yl = g2(G[G_VY], c), yh = g2(G[G_VY], cidx(I, i, jc + 1, k));
    const longlong2 zh = g2(G[G_VZ], e), zl = g2(G[G_VZ], vidx(I, i, jc, km));
    const fx xm = LDG(G[G_VX] + vidx(I, im, jc, k));
    F.v.x = diff(x.x, xm, dh, e0.y) * rxc0;
    F.v.y = diff(x.y, x.x, dh, e0.y) * rxc1;
    F.v.x = fma(ydiff(yh.x, dn, eh.y, yl.x, dc, e0.y), ryf, F.v.x);
    F.v.y = fma(ydiff(yh.y, dn, eh.y, yl.y, dc, e0.y), ryf, F.v.y);
    F.v.x = fma(diff(zh.x, zl.x, dh, e0.y), rzc, F.v.x);
    F.v.y = fma(diff(zh.y, zl.y, dh, e0.y), rzc, F.v.y);
  }
  // a row marked non-finite by its maxima (none where its fluxes are doubles)
  const int bad = WALL ? (dc ? 0 : e0.w) | (dl ? 0 : el.w) | (dn ? 0 : eh.w) : e0.w | el.w | eh.w;
  if (bad) {
    const double q = __longlong_as_double(0x7FF8000000000000LL);
    F.u = F.v = F.w = make_double2(q, q);
  }
  return F;
}
// F and the stage update at x points i (even) and i + 1 of row jc, plane k.
template <bool WALL>
__device__ __forceinline__ void update_pair(const ChlInst& I, const RhsArgs& a, int i, int jc, int k) {
  const int Ny = I.Ny;
  const bool hasv = jc <= Ny - 1;
  const size_t c = cidx(I, i, jc, k), e = vidx(I, i, jc, k);
  auto d2 = [](const double* f, size_t q) { return *reinterpret_cast<const double2*>(f + q); };
  auto put = [](double* f, size_t q, double2 v) { *reinterpret_cast<double2*>(f + q) = v; };
  auto neg = [](double2 v) { return make_double2(chl_neg(v.x), chl_neg(v.y)); };
  const Rhs F = rhs_pair<WALL>(I, i, jc, k);
  if (a.mode == 2) {           // actual-pressure RHS: keep F only
    put(I.Fp[0], c, F.u); put(I.Fp[2], c, F.w);
    if (hasv) put(I.Fp[1], e, F.v);
    return;
  }
  // out = base + dt (c1 F1 + c2 F) as two FMAs per component; the products
  // dt c are formed once per step where dt is set
  const double dc1 = I.scal[CHL_S_DC + 2 * a.stage], dc2 = I.scal[CHL_S_DC + 2 * a.stage + 1];
  double* Uo = I.U[a.sout]; double* Vo = I.V[a.sout]; double* Wo = I.W[a.sout];
  auto axpy = [](double s, double2 x, double2 y) { return make_double2(fma(s, x.x, y.x), fma(s, x.y, y.y)); };
  double2 un = axpy(dc2, F.u, d2(I.U[a.sbase], c)), wn = axpy(dc2, F.w, d2(I.W[a.sbase], c)), vn;
  if (hasv) vn = axpy(dc2, F.v, d2(I.V[a.sbase], e));
  if (a.mode == 0) {
    put(I.F1[0], c, F.u); put(I.F1[2], c, F.w);
    if (hasv) put(I.F1[1], e, F.v);
  } else {
    un = axpy(dc1, d2(I.F1[0], c), un);
    wn = axpy(dc1, d2(I.F1[2], c), wn);
    if (hasv) vn = axpy(dc1, d2(I.F1[1], e), vn);
  }
  put(Uo, c, un); put(Wo, c, wn);
  if (hasv) put(Vo, e, vn);
  if (jc == 1) { put(Uo, cidx(I, i, 0, k), neg(un)); put(Wo, cidx(I, i, 0, k), neg(wn)); }
  if (jc == Ny) { put(Uo, cidx(I, i, Ny + 1, k), neg(un)); put(Wo, cidx(I, i, Ny + 1, k), neg(wn)); }
}
// a call: its FP64 instructions would be predicated into every row
static __device__ __noinline__ void update_pair_wall(const ChlInst& I, const RhsArgs& a, int i, int jc, int k) {
  update_pair<true>(I, a, i, jc, k);
}

// The flux differences are exact integers; each is rounded once to a double
// and multiplied by its reciprocal spacing there (with the products in
// integers as well, F lost two to four bits to their common exponent).  One
// thread per pair of x points: 16-byte loads, and the pair shares the fluxes
// between its points.
__global__ void __launch_bounds__(256, 4)
k_rhs_update(ChlMap map, RhsArgs a) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  if (t >= (unsigned)(I.Nx / 2 * I.Ny * I.Nz)) return;
  const ChlIdx p = chl_split(t, I.Nx / 2, I.Ny);
  const int i = 2 * p.i, jc = 1 + p.j;
  if (I.wall_model != 0 && (jc <= 2 || jc >= I.Ny - 1)) update_pair_wall(I, a, i, jc, p.k);
  else update_pair<false>(I, a, i, jc, p.k);
}

extern "C" {
void chl_launch_fix(const ChlMap& map, int nb_full, int s, int prep, cudaStream_t st) {
  chl_launch_pdl(k_fix, dim3(nb_full), dim3(map.tb), 0, st, map, s, prep);
}
void chl_launch_flux(const ChlMap& map, int nb_edge, int sin, cudaStream_t st) {
  chl_launch_pdl(k_flux, dim3(nb_edge), dim3(CHL_FLUX_THREADS), 0, st, map, sin);
}
void chl_launch_update(const ChlMap& map, int nb_pt, int sbase, int sout, int stage, int mode, cudaStream_t st) {
  RhsArgs a{sbase, sout, stage, mode};
  chl_launch_pdl(k_rhs_update, dim3(nb_pt), dim3(map.tb), 0, st, map, a);
}
}
