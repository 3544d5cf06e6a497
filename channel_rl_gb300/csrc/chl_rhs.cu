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
// us per launch at 256x96x192).  The velocities come as the fixed-point
// copies k_fix made of the stage's input, the fluxes are kept as integers,
// and only the three components of F and the two FMAs of the stage update
// are FP64.  Halves and quarters of the averages are exponents.  The y-face
// value of u (and w) is u_a + w1 (u_b - u_a).
#include "chl_fix.cuh"

// flux fields: centre-like (rows 1..Ny): 0 GUx, 1 GVy, 2 GWz, 3 GUz, 4 GWx;
// V-like (rows 0..Ny): 5 GUy, 6 GVx, 7 GVz, 8 GWy
enum { G_UX = 0, G_VY, G_WZ, G_UZ, G_WX, G_UY, G_VX, G_VZ, G_WY };

// Exponents of a launch, from the largest |U|, |V|, |W|, |nu + nu_t| of its
// input.  Flux m = viscous - advective part: the advective product has last
// bit 2^A, the viscous one 2^B, the stored flux 2^G, one above the larger,
// so that |flux| < 2^60.
struct FluxExp { int A, B, G; };
__device__ __forceinline__ FluxExp flux_exp(const ChlInst& I, int sin, int m) {
  const unsigned* vm = chl_vmax(I, sin);
  const int a = m == G_UX || m == G_UZ || m == G_UY ? 0 : (m == G_VY || m == G_VX || m == G_VZ ? 1 : 2);
  const int b = m == G_UX || m == G_VX || m == G_WX ? 0 : (m == G_UY || m == G_VY || m == G_WY ? 1 : 2);
  const int ea = fx_exp<61>(vm[a]), eb = fx_exp<61>(vm[b]), en = fx_exp<60>(*chl_nmax(I));
  const int er = m == G_UX ? I.exc : m == G_VY ? I.eyc : m == G_WZ ? I.ezc
               : b == 0 ? I.exf : b == 1 ? I.eyf : I.ezf;
  FluxExp q;
  // factors of the averages: one half in the products on y-face edges, a
  // quarter in the others; viscosity 1, 4 and 2 x at centres, xz and y-face edges
  q.A = ea + eb + (m >= G_UY ? 63 : 62);
  q.B = en + ea + er + (m <= G_WZ ? 128 : m <= G_WX ? 126 : 127);
  q.G = max(q.A, q.B) + 1;
  return q;
}

// Table of the stage update, written by k_flux's first block of the instance
// for k_rhs_update (so that none of its blocks waits for it): alignment
// shifts of the nine terms, the three exponents of F, and whether an input
// was not finite (F is then NaN, as its products would be).
enum { UPD_SHIFT = 0, UPD_EXP = 9, UPD_BAD = 12, UPD_N = 13 };
// Component c of F sums three flux differences times a reciprocal spacing,
// term q from flux field UPD_FLUX[c][q]; the products are aligned to 2^eF.
__device__ constexpr int UPD_FLUX[3][3] = {{G_UX, G_UY, G_UZ}, {G_VX, G_VY, G_VZ}, {G_WX, G_WY, G_WZ}};
__device__ __forceinline__ void write_upd(const ChlInst& I, int sin, int c) {   // c = 0..3
  if (c == 3) {
    const unsigned* vm = chl_vmax(I, sin);
    I.upd[UPD_BAD] = fx_bad(vm[0]) || fx_bad(vm[1]) || fx_bad(vm[2]) || fx_bad(*chl_nmax(I));
    return;
  }
  int e[3];
  for (int q = 0; q < 3; ++q) {
    const int er = q == 0 ? (c == 0 ? I.exf : I.exc) : q == 1 ? (c == 1 ? I.eyf : I.eyc) : (c == 2 ? I.ezf : I.ezc);
    e[q] = flux_exp(I, sin, UPD_FLUX[c][q]).G + er + 64;
  }
  const int eF = max(max(e[0], e[1]), e[2]) + 2;
  for (int q = 0; q < 3; ++q) I.upd[UPD_SHIFT + 3 * c + q] = min(63, eF - e[q]);
  I.upd[UPD_EXP + c] = eF;
}

// Fixed-point copies of the velocity set that a stage works on (rows as
// stored, ghosts included); reset_n clears the largest |nu + nu_t| ahead of
// the kernels that form it.  Moves 48 bytes per point: HBM-bound.
__global__ void __launch_bounds__(256)
k_fix(ChlMap map, int s, int reset_n) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  if (reset_n && t == 0) *chl_nmax(I) = 0u;
  const unsigned* vm = chl_vmax(I, s);
  const unsigned nc = (unsigned)(I.Nx * (I.Ny + 2) * I.Nz), nv = (unsigned)(I.Nx * (I.Ny + 1) * I.Nz);
  if (t < nc) {
    I.X[0][t] = fx_from(LDG(I.U[s] + t), fx_exp<61>(vm[0]));
    I.X[2][t] = fx_from(LDG(I.W[s] + t), fx_exp<61>(vm[2]));
  }
  if (t < nv) I.X[1][t] = fx_from(LDG(I.V[s] + t), fx_exp<61>(vm[1]));
}

// 28 products and 4 conversions of nu + nu_t per point on the integer pipe,
// no FP64 instruction; 104 bytes per point.  A thread marches through
// chl_planes planes at its (i, j), so that what the next plane shares (U, V,
// nu + nu_t one plane up, W one down) is loaded and converted once.
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 6)
k_flux(ChlMap map, int sin) {
  chl_pdl_wait();
  __shared__ int sh[20];      // right shifts of the advective (0..8) and viscous (9..17) parts, exponent of nu
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  if (threadIdx.x < 18) {
    const int m = threadIdx.x % 9;
    const FluxExp q = flux_exp(I, sin, m);
    sh[threadIdx.x] = min(63, q.G - (threadIdx.x < 9 ? q.A : q.B));
  } else if (threadIdx.x == 18) {
    sh[18] = fx_exp<60>(*chl_nmax(I));
  } else if (lb == 0 && threadIdx.x >= 32 && threadIdx.x < 36) {
    write_upd(I, sin, threadIdx.x - 32);
  }
  const int M = chl_planes(Nx, Ny, Nz);
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, Ny + 1);
  const int i = p.i, j = p.j, k0 = p.k * M, k1 = min(Nz, k0 + M);
  const fx* __restrict__ U = I.X[0];
  const fx* __restrict__ V = I.X[1];
  const fx* __restrict__ W = I.X[2];
  const double* __restrict__ nt = I.nut;   // nu + nu_t
  const bool valid = k0 < Nz;
  const fx w1 = LDG(I.fxw1 + j), rxf = LDG(I.fxrxf + i), ryf = LDG(I.fxryf + j);
  const fx rxc = LDG(I.fxrxc + i), ryc = LDG(I.fxryc + j);
  const int ip = wrap(i + 1, Nx), im = wrap(i - 1, Nx);
  const int jp = min(j + 1, Ny + 1), jm = max(j - 1, 0);
  fx u_a = 0, v_0 = 0, w_m = 0;
  double dn_a = 0.0, dn_b = 0.0, dn_p = 0.0;
  if (valid) {
    u_a = LDG(U + cidx(I, i, j, k0));
    v_0 = LDG(V + vidx(I, i, j, k0));
    w_m = LDG(W + cidx(I, i, j, k0 == 0 ? Nz - 1 : k0 - 1));
    dn_a = LDG(nt + cidx(I, i, j, k0)); dn_b = LDG(nt + cidx(I, i, jp, k0)); dn_p = LDG(nt + cidx(I, ip, j, k0));
  }
  __syncthreads();
  if (!valid) return;
  const int en = sh[18];
  fx n_a = fx_from(dn_a, en), n_b = fx_from(dn_b, en), n_p = fx_from(dn_p, en);
#define ADV(m, f) ((f) >> sh[m])
#define VIS(m, f) ((f) >> sh[9 + (m)])
#define PUT(m, e, adv, vis) I.G[m][e] = VIS(m, vis) - ADV(m, adv)
  for (int k = k0; k < k1; ++k) {
    const int kp = k + 1 == Nz ? 0 : k + 1;
    const size_t c = cidx(I, i, j, k), e = vidx(I, i, j, k);
    const fx u_b = LDG(U + cidx(I, i, jp, k)), w_b = LDG(W + cidx(I, i, jp, k));
    const fx w_a = LDG(W + c);
    const fx u_z = LDG(U + cidx(I, i, j, kp)), v_z = LDG(V + vidx(I, i, j, kp)), v_p = LDG(V + vidx(I, ip, j, k));
    const fx n_az = fx_from(LDG(nt + cidx(I, i, j, kp)), en), n_bz = fx_from(LDG(nt + cidx(I, i, jp, kp)), en);
    const fx n_pz = fx_from(LDG(nt + cidx(I, ip, j, kp)), en), n_bp = fx_from(LDG(nt + cidx(I, ip, jp, k)), en);
    const fx rzf = LDG(I.fxrzf + k);
    const fx nx_a = n_a + n_p;             // x pair of row j: the xy and xz edges share it
    {  // yz edge (x-centre i, y-face j, z-face k): vw, nu -> GVz, GWy
      const fx dw = w_b - w_a;
      const fx vw = fx_mul(w_a + 2 * fx_mul(dw, w1), v_0 + v_z);                      // 2 v w
      const fx na = n_a + n_az;
      const fx nyz = na + 2 * fx_mul(n_b + n_bz - na, w1);                            // 2 nu
      PUT(G_VZ, e, vw, fx_mul(nyz, fx_mul(v_z - v_0, rzf)));
      PUT(G_WY, e, vw, fx_mul(nyz, fx_mul(dw, ryf)));
    }
    {  // xy edge (x-face i, y-face j, z-centre k): uv, nu -> GUy, GVx
      const fx du = u_b - u_a;
      const fx uv = fx_mul(u_a + 2 * fx_mul(du, w1), v_0 + v_p);                      // 2 u v
      const fx nxy = nx_a + 2 * fx_mul(n_b + n_bp - nx_a, w1);                        // 2 nu
      PUT(G_UY, e, uv, fx_mul(nxy, fx_mul(du, ryf)));
      PUT(G_VX, e, uv, fx_mul(nxy, fx_mul(v_p - v_0, rxf)));
    }
    if (j >= 1) {
      {  // cell centre: diagonal fluxes
        const fx u_m = LDG(U + cidx(I, im, j, k)), v_m = LDG(V + vidx(I, i, jm, k));
        const fx su = u_m + u_a, sv = v_m + v_0, sw = w_m + w_a;
        PUT(G_UX, c, fx_mul(su, su), fx_mul(n_a, fx_mul(u_a - u_m, rxc)));
        PUT(G_VY, c, fx_mul(sv, sv), fx_mul(n_a, fx_mul(v_0 - v_m, ryc)));
        PUT(G_WZ, c, fx_mul(sw, sw), fx_mul(n_a, fx_mul(w_a - w_m, LDG(I.fxrzc + k))));
      }
      {  // xz edge (x-face i, y-centre j, z-face k): uw, nu -> GUz, GWx
        const fx w_p = LDG(W + cidx(I, ip, j, k));
        const fx uw = fx_mul(u_a + u_z, w_a + w_p);                                   // 4 u w
        const fx nxz = nx_a + (n_az + n_pz);                                          // 4 nu
        PUT(G_UZ, c, uw, fx_mul(nxz, fx_mul(u_z - u_a, rzf)));
        PUT(G_WX, c, uw, fx_mul(nxz, fx_mul(w_p - w_a, rxf)));
      }
    }
    u_a = u_z; v_0 = v_z; w_m = w_a; n_a = n_az; n_b = n_bz; n_p = n_pz;
  }
#undef ADV
#undef VIS
#undef PUT
}

struct RhsArgs {
  int sbase, sout;        // velocity sets: stage base (U^n), output
  int stage;              // RK3 stage 0..2: out = base + dt (c1 F1 + c2 F) (chl_put_dt's products)
  int mode;               // 0: stage 1 (store F1), 1: stages 2/3, 2: actual-pressure RHS only
};

__global__ void __launch_bounds__(256)
k_rhs_update(ChlMap map, RhsArgs a) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  if (t >= (unsigned)(Nx * Ny * Nz)) return;
  const ChlIdx p = chl_split(t, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k = p.k;
  const int im = wrap(i - 1, Nx), ip = wrap(i + 1, Nx);
  const int km = wrap(k - 1, Nz), kp = wrap(k + 1, Nz);
  const fx* const* G = I.G;
  const int* u = I.upd;
  const fx rxc = LDG(I.fxrxc + i), rxf = LDG(I.fxrxf + i);
  const fx rzc = LDG(I.fxrzc + k), rzf = LDG(I.fxrzf + k);
  const fx ryc = LDG(I.fxryc + jc);
  const size_t c = cidx(I, i, jc, k), e = vidx(I, i, jc, k), em = vidx(I, i, jc - 1, k);
  const bool hasv = jc <= Ny - 1;
#define TERM(q, m, hi, lo, r) (fx_mul(LDG(G[m] + (hi)) - LDG(G[m] + (lo)), r) >> LDG(u + UPD_SHIFT + (q)))
  // u at (x-face i, row jc, z-centre k), w at (x-centre i, row jc, z-face k),
  // v at (x-centre i, y-face jv = jc, z-centre k)
  double Fu = fx_to(TERM(0, G_UX, cidx(I, ip, jc, k), c, rxf) + TERM(1, G_UY, e, em, ryc)
                    + TERM(2, G_UZ, c, cidx(I, i, jc, km), rzc), LDG(u + UPD_EXP)) + I.scal[CHL_S_DPDX];
  double Fw = fx_to(TERM(6, G_WX, c, cidx(I, im, jc, k), rxc) + TERM(7, G_WY, e, em, ryc)
                    + TERM(8, G_WZ, cidx(I, i, jc, kp), c, rzf), LDG(u + UPD_EXP + 2));
  double Fv = 0.0;
  if (hasv)
    Fv = fx_to(TERM(3, G_VX, e, vidx(I, im, jc, k), rxc) + TERM(4, G_VY, cidx(I, i, jc + 1, k), c, LDG(I.fxryf + jc))
               + TERM(5, G_VZ, e, vidx(I, i, jc, km), rzc), LDG(u + UPD_EXP + 1));
#undef TERM
  if (LDG(u + UPD_BAD)) Fu = Fv = Fw = __longlong_as_double(0x7FF8000000000000LL);
  if (a.mode == 2) {           // actual-pressure RHS: keep F only
    I.Fp[0][c] = Fu; I.Fp[2][c] = Fw;
    if (hasv) I.Fp[1][e] = Fv;
    return;
  }
  // out = base + dt (c1 F1 + c2 F) as two FMAs per component; the products
  // dt c are formed once per step where dt is set
  const double dc1 = I.scal[CHL_S_DC + 2 * a.stage], dc2 = I.scal[CHL_S_DC + 2 * a.stage + 1];
  double* Uo = I.U[a.sout]; double* Vo = I.V[a.sout]; double* Wo = I.W[a.sout];
  const double* Ub = I.U[a.sbase]; const double* Vb = I.V[a.sbase]; const double* Wb = I.W[a.sbase];
  double un = fma(dc2, Fu, Ub[c]), wn = fma(dc2, Fw, Wb[c]), vn = hasv ? fma(dc2, Fv, Vb[e]) : 0.0;
  if (a.mode == 0) {
    I.F1[0][c] = Fu; I.F1[2][c] = Fw;
    if (hasv) I.F1[1][e] = Fv;
  } else {
    un = fma(dc1, I.F1[0][c], un);
    wn = fma(dc1, I.F1[2][c], wn);
    if (hasv) vn = fma(dc1, I.F1[1][e], vn);
  }
  Uo[c] = un; Wo[c] = wn;
  if (hasv) Vo[e] = vn;
  if (jc == 1) { Uo[cidx(I, i, 0, k)] = chl_neg(un); Wo[cidx(I, i, 0, k)] = chl_neg(wn); }
  if (jc == Ny) { Uo[cidx(I, i, Ny + 1, k)] = chl_neg(un); Wo[cidx(I, i, Ny + 1, k)] = chl_neg(wn); }
}

extern "C" {
void chl_launch_fix(const ChlMap& map, int nb_full, int s, int reset_n, cudaStream_t st) {
  chl_launch_pdl(k_fix, dim3(nb_full), dim3(map.tb), 0, st, map, s, reset_n);
}
void chl_launch_flux(const ChlMap& map, int nb_edge, int sin, cudaStream_t st) {
  chl_launch_pdl(k_flux, dim3(nb_edge), dim3(CHL_FLUX_THREADS), 0, st, map, sin);
}
void chl_launch_update(const ChlMap& map, int nb_pt, int sbase, int sout, int stage, int mode, cudaStream_t st) {
  RhsArgs a{sbase, sout, stage, mode};
  chl_launch_pdl(k_rhs_update, dim3(nb_pt), dim3(map.tb), 0, st, map, a);
}
}
