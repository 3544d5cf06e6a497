// Subgrid-scale eddy viscosity and wall models.
//
// Dynamic Smagorinsky (Lilly) as sgs_dynamic_Smagorinsky does it
// (subgrid.f90:379-537): test filter filter_xzy (subgrid.f90:140-190, the
// 1/6-2/3-1/6 rule in x, z and y, one-sided 2/3-1/3 at the first and last
// row), strain rates of compute_Sij (subgrid.f90:1014-1072), plane sums of
// L:M and M:M over i=2..nxg-1, k=2..nzg-1 (the duplicated periodic column
// and plane counted twice, subgrid.f90:492-509), nu_t = max(0,-1/2 <LM>/<MM>|S|)
// and the ghost-row rule of Dirichlet_nu_t.
//
// The strain, the filter and L are formed in fixed point (chl_fix.cuh,
// chl_strain.cuh): as FP64 code the dynamic model took 212 FP64 instructions
// per point and stage, which the FP64 pipe bounds; 43 are left.
//
// Static Smagorinsky with van Driest damping (subgrid.f90:563-612, which
// aborts in the reference) is written from its formula.  The stress wall
// model is compute_wall_model (wallmodel.f90:23-46); the equilibrium log-law
// wall stress that feeds it is new.
#include "chl_strain.cuh"
#include "chl_nut.cuh"

// ---------------------------------------------------------------- strain
// Strain magnitude and the DSM filter inputs at centres (rows 1..Ny): q3..8
// the products of the centre velocities' face sums in fixed point (last bit
// 2^(e_i + e_j + 64), less the row's slack of both: next to a resolved wall the
// products are 1e-8 of the field's largest and less), q9..14 = |S|*(S_ii, 2 S_ij)
// / sqrt(2) and their largest per row.
// With DSM = false (the static model, whose row coefficients do not depend on
// the strain) nu + nu_t instead, so that no pass reads |S| back: 14 us at
// 256x96x192 for the 37 that k_nut then took and the launch of the coefficients'
// own kernel.  218 and 170 us there (202 and 157 with one x and z spacing for both
// edges of a centre).
template <bool DSM>
__global__ void __launch_bounds__(CHL_FLUX_THREADS, 7)
k_strain(ChlMap map, int s_in, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, M = map.planes;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  const ChlIdx p = chl_split(t, Nx, Ny);
  const int i = p.i, jc = 1 + p.j, k0 = p.k * M;
  unsigned hi = 0u;
  const unsigned* vm = chl_vmax(I, s_in);
  const bool bad = fx_bad(vm[0]) || fx_bad(vm[1]) || fx_bad(vm[2]);
  StrainColumn col(I, I.X[0], I.X[1], I.X[2], fx_exp<61>(vm[0]), fx_exp<61>(vm[1]), fx_exp<61>(vm[2]), i, jc,
                   min(k0, Nz - 1));
  const double cj = DSM ? 0.0 : I.coef[jc], nu = I.nu;
  int4 sl = make_int4(0, 0, 0, 0);
  if (DSM) sl = LDG(I.slack + jc);
  for (int k = k0; k < min(Nz, k0 + M); ++k) {
    fx f[3];
    Strain s = col.point(k, f);
    if (bad) s.s = __longlong_as_double(0x7FF8000000000000LL);
    const size_t c = cidx(I, i, jc, k);
    I.S[c] = s.s;
    if (!DSM) {
      // nu + max(0, c |S|) as in k_nut
      const double v = chl_atleast(fma(cj, s.s, nu), nu);
      hi = max(hi, write_nut_rows(I, i, jc, k, v, [&] { return chl_pos(cj * s.s); }, use_wm));
      continue;
    }
    fx* const* q = reinterpret_cast<fx* const*>(I.q);
    f[0] <<= sl.x; f[1] <<= sl.y; f[2] <<= sl.z;
    q[3][c] = fx_mul_mean<64>(f[0], f[0]); q[4][c] = fx_mul_mean<64>(f[1], f[1]); q[5][c] = fx_mul_mean<64>(f[2], f[2]);
    q[6][c] = fx_mul_mean<64>(f[0], f[1]); q[7][c] = fx_mul_mean<64>(f[0], f[2]); q[8][c] = fx_mul_mean<64>(f[1], f[2]);
    const double se = s.s * pow2(min(1023, max(-1022, s.e)));
    // two of the six conversions on the FP64 pipe, which is the less busy
    const double d[6] = {se * fx_raw<true>(s.t[0]), se * fx_raw<true>(s.t[1]), se * fx_raw<false>(s.t[2]),
                         se * fx_raw<false>(s.t[3]), se * fx_raw<false>(s.t[4]), se * fx_raw<false>(s.t[5])};
#pragma unroll
    for (int n = 0; n < 6; ++n) { I.q[9 + n][c] = d[n]; hi = max(hi, chl_abshi(d[n])); }
  }
  chl_line_max(DSM ? I.smax : I.nmax, (unsigned)(p.k * Ny + p.j), Ny, 1, hi);
}

// ------------------------------------------------------------ test filter
// filter_xzy of fifteen fields in one pass over memory, in fixed point: the
// six products of the centre velocities (rows 1..Ny), the six |S| S_ij (rows
// 1..Ny, scaled by the largest of the group's rows) and the face velocities U
// and W (rows 0..Ny+1) and V (rows 0..Ny); each with the one-sided rule
// (4, 2)/6 at its first and last row.  Three separable FP64 passes took 2
// instructions of 64 clocks per pass, field and point and moved every field
// three times: 247 us per pass at 256x96x192.  Here a tap is an integer
// shift and two additions, and the three passes take 239 us together.
//
// A pass forms (a + 4 b + c) >> 3, rounded (up at a half in y and z, down in x: a
// mean error of L would not average out of its sums), so that a field starts and ends below 2^60
// and a filtered value is 512/216 times its integer.  A thread holds two
// points in x of two rows, filters them in y from the four rows it loads,
// exchanges with its neighbours in x through shared memory and marches in z,
// carrying the two planes behind.
//
// Rows 1 and Ny of the centre velocities need the one-sided rule in y, which
// the filtered faces next to them do not have: three more "fields" of two
// rows each hold (4 f_1 + 2 f_2) of U, W (and of the face sum of V), so that
// the final kernel forms the wall rows' filtered centre velocities from them
// like the others from the faces.
//
// Blocks per instance: for each of the 15 fields row blocks x plane chunks,
// then for each of the 3 wall fields one row block x plane chunks.
#define FILT_FIELDS 15
struct FiltShape { int nxp, RG, segs, rowblocks, M, nz, full; };   // full: blocks of one field
__host__ __device__ inline FiltShape filt_shape(int Nx, int Ny, int Nz, int T, int M) {
  FiltShape f;
  f.nxp = Nx / 2;
  f.RG = f.nxp <= T ? T / f.nxp : 1;                       // row groups per block
  f.segs = f.nxp <= T ? 1 : (f.nxp + T - 3) / (T - 2);     // longer rows: overlapping segments
  const int groups = (Ny + 3) / 2;                         // of U and W, the most
  f.rowblocks = (groups + f.RG - 1) / f.RG * f.segs;
  f.M = M;
  f.nz = (Nz + f.M - 1) / f.M;
  f.full = f.rowblocks * f.nz;
  return f;
}

// the exponent of |S| S_ij in the filter of row group g (rows 1 + 2 g, 2 + 2 g)
__device__ __forceinline__ int filt_exp(const ChlInst& I, int g) {
  unsigned m = I.smax[max(1, 2 * g)];
#pragma unroll
  for (int r = 1; r < 4; ++r) m = max(m, I.smax[min(I.Ny, 2 * g + r)]);
  return fx_exp<60>(m);
}

// bits by which the velocities of row group g's centre rows are shifted up
__device__ __forceinline__ int4 filt_slack(const ChlInst& I, int g) {
  int4 m = LDG(I.slack + max(1, 2 * g));
#pragma unroll
  for (int r = 1; r < 4; ++r) {
    const int4 s = LDG(I.slack + min(I.Ny, 2 * g + r));
    m.x = min(m.x, s.x); m.y = min(m.y, s.y); m.z = min(m.z, s.z);
  }
  return m;
}
// of the product of field 0..5: u u, v v, w w, u v, u w, v w
__device__ __forceinline__ int product_slack(int4 s, int field) {
  return (field == 1 || field == 5 ? s.y : field == 2 ? s.z : s.x) + (field == 0 ? s.x : field == 1 || field == 3 ? s.y : s.z);
}

struct Pair { fx x, y; };
__device__ __forceinline__ Pair tap(Pair a, Pair b, Pair c) {
  return Pair{(a.x + 4 * b.x + c.x + 4) >> 3, (a.y + 4 * b.y + c.y + 4) >> 3};
}
__device__ __forceinline__ Pair one_sided(Pair a, Pair b) { return Pair{(a.x >> 1) + (b.x >> 2), (a.y >> 1) + (b.y >> 2)}; }

__global__ void __launch_bounds__(256)
k_filter(ChlMap map) {
  chl_pdl_wait();
  __shared__ longlong2 sm[2][2][256];      // [parity][row][thread]
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const FiltShape f = filt_shape(Nx, Ny, Nz, blockDim.x, map.fplanes);
  // field, row block, segment, planes
  int field, rest;
  if (lb < FILT_FIELDS * f.full) { field = lb / f.full; rest = lb - field * f.full; }
  else {
    const int w = lb - FILT_FIELDS * f.full;
    field = FILT_FIELDS + w / (f.segs * f.nz);
    rest = w % (f.segs * f.nz);
  }
  const bool wall = field >= FILT_FIELDS;
  const int rb = wall ? rest % f.segs : rest % f.rowblocks, zc = wall ? rest / f.segs : rest / f.rowblocks;
  const int seg = rb % f.segs;
  const int tid = threadIdx.x;
  int rg, pi, left, right;
  bool out;
  if (f.segs == 1) {
    rg = tid / f.nxp;
    pi = tid - rg * f.nxp;
    out = rg < f.RG;
    left = pi == 0 ? tid + f.nxp - 1 : tid - 1;
    right = pi == f.nxp - 1 ? tid - (f.nxp - 1) : tid + 1;
    if (!out) { rg = 0; left = right = tid; }
  } else {
    rg = 0;
    pi = seg * ((int)blockDim.x - 2) + tid - 1;
    out = tid >= 1 && tid < (int)blockDim.x - 1 && pi < f.nxp;
    pi = pi < 0 ? pi + f.nxp : pi % f.nxp;
    left = max(tid - 1, 0); right = min(tid + 1, (int)blockDim.x - 1);
  }
  const int g = wall ? 0 : rb / f.segs * f.RG + rg;
  out = out && (!wall || rg == 0);
  // source, rows and layout
  const int comp = wall ? field - FILT_FIELDS : field - 12;     // 0, 1, 2: U, V, W
  const bool vlike = field >= 12 && comp == 1;
  const bool conv = field >= 6 && field < 12;
  const int nrow = vlike ? Ny + 1 : Ny + 2;
  const int first = field < 12 ? 1 : 0, last = field < 12 ? Ny : (vlike ? Ny : Ny + 1);
  const longlong2* src;
  longlong2* dst;
  if (field < 12) { src = reinterpret_cast<const longlong2*>(I.q[3 + field]); dst = reinterpret_cast<longlong2*>(I.r[3 + field]); }
  else {
    src = reinterpret_cast<const longlong2*>(I.X[comp]);
    dst = reinterpret_cast<longlong2*>(wall ? I.r[comp] : I.r[15 + comp]);
  }
  const int j0 = first + 2 * g;
  out = out && (wall || j0 <= last);
  const bool two = wall || j0 < last;
  int row[4];
  if (wall) {
    // U, W: f_1, f_2 next to each wall; V: the face sums there are V(1) and
    // V(1) + V(2) (V is zero on the wall)
    row[0] = 1; row[1] = 2;
    row[2] = vlike ? Ny - 1 : Ny; row[3] = row[2] - 1;
  } else {
    const int j = min(j0, last);
    row[1] = j;
    row[0] = j == first ? j + 1 : j - 1;
    row[2] = j == last ? j - 1 : j + 1;
    row[3] = j + 1 >= last ? j : j + 2;
  }
  const int e = conv ? filt_exp(I, min(g, (Ny - 1) / 2)) : 0;
  // the field indices of this kernel are offsets; the bounds-checked build checks
  // what they are made of (and the neighbours in shared memory as x and y of a block)
  int xi = 2 * pi, kz = zc * f.M;
#pragma unroll
  for (int q = 0; q < 4; ++q) chl_clamp(I, xi, row[q], kz, nrow - 1);
  pi = xi >> 1;
  chl_clamp_to(I, left, (int)blockDim.x); chl_clamp_to(I, right, (int)blockDim.x);
  const unsigned pitch = (unsigned)f.nxp * (unsigned)nrow;
  const unsigned off0 = f.nxp * row[0] + pi, off1 = f.nxp * row[1] + pi, off2 = f.nxp * row[2] + pi, off3 = f.nxp * row[3] + pi;
  auto get = [&](longlong2 v, int down) {
    if (conv) return Pair{fx_from(__longlong_as_double(v.x), e), fx_from(__longlong_as_double(v.y), e)};
    return Pair{v.x >> down, v.y >> down};
  };
  const int k0 = zc * f.M, k1 = min(Nz, k0 + f.M);
  int k = k0 == 0 ? Nz - 1 : k0 - 1;
  const longlong2* s = src + (size_t)pitch * k;
  longlong2 n0 = __ldg(s + off0), n1 = __ldg(s + off1), n2 = __ldg(s + off2), n3 = __ldg(s + off3);
  // right shifts of the four rows: the velocities' copies are below 2^61, products
  // come in the unit of their row and go in that of the group
  int4 down = make_int4(1, 1, 1, 1);
  if (field < 6) {
    const int to = product_slack(filt_slack(I, min(g, (Ny - 1) / 2)), field);
    auto by = [&](int r) { return max(0, product_slack(LDG(I.slack + min(max(r, 1), Ny)), field) - to); };
    down = make_int4(by(row[0]), by(row[1]), by(row[2]), by(row[3]));
  }
  Pair a0 = {0, 0}, a1 = {0, 0}, b0 = {0, 0}, b1 = {0, 0};      // the planes k - 2 and k - 1 of both rows
  for (int it = 0; it < k1 - k0 + 2; ++it) {
    const Pair v0 = get(n0, down.x), v1 = get(n1, down.y), v2 = get(n2, down.z), v3 = get(n3, down.w);
    k = k + 1 == Nz ? 0 : k + 1;
    if (it < k1 - k0 + 1) {
      chl_clamp_to(I, k, Nz);
      s = src + (size_t)pitch * k;
      n0 = __ldg(s + off0); n1 = __ldg(s + off1); n2 = __ldg(s + off2); n3 = __ldg(s + off3);
    }
    Pair y0, y1;
    if (wall) {
      y0 = one_sided(v0, vlike ? Pair{v0.x + v1.x, v0.y + v1.y} : v1);
      y1 = one_sided(v2, vlike ? Pair{v2.x + v3.x, v2.y + v3.y} : v3);
    } else {
      y0 = tap(v0, v1, v2);
      y1 = tap(v1, v2, v3);
    }
    longlong2 (*buf)[256] = sm[it & 1];
    buf[0][tid] = make_longlong2(y0.x, y0.y);
    buf[1][tid] = make_longlong2(y1.x, y1.y);
    __syncthreads();
    const fx l0 = buf[0][left].y, r0 = buf[0][right].x, l1 = buf[1][left].y, r1 = buf[1][right].x;
    const Pair x0 = {(l0 + 4 * y0.x + y0.y + 3) >> 3, (y0.x + 4 * y0.y + r0 + 3) >> 3};
    const Pair x1 = {(l1 + 4 * y1.x + y1.y + 3) >> 3, (y1.x + 4 * y1.y + r1 + 3) >> 3};
    if (it >= 2 && out) {
      const Pair z0 = tap(a0, b0, x0), z1 = tap(a1, b1, x1);
      // wall fields go to rows 1 and Ny of a centre-like field
      const int nr = wall ? Ny + 2 : nrow;
      int ra = wall ? 1 : j0, rc = wall ? Ny : j0 + 1, ko = k0 + it - 2;
      chl_clamp(I, xi, ra, ko, nr - 1);
      if (two) chl_clamp_to(I, rc, nr);
      longlong2* d = dst + (size_t)f.nxp * ((size_t)nr * ko) + pi;
      d[(size_t)f.nxp * ra] = make_longlong2(z0.x, z0.y);
      if (two) d[(size_t)f.nxp * rc] = make_longlong2(z1.x, z1.y);
    }
    a0 = b0; a1 = b1; b0 = x0; b1 = x1;
  }
}

// ------------------------------------------------------------ L:M, M:M
// One block of CHL_DSMF_THREADS per (centre row jc, chunk of the row's
// columns); a column is an x position and chl_dsm_planes planes, which its
// thread marches through (chl_strain.cuh, on the filtered faces).  Each
// thread writes its partial sums to part[0|1][jc][chunk][thread] (no
// reduction tree in every block: its mostly idle warps would issue an FP64
// instruction per level for a handful of lanes).  The last block of a row to
// finish (a counter per row) adds the row's partials - thread t the entries
// t, t + CHL_DSMF_THREADS, ... in order, then a fixed-order block tree - and
// writes the row's coefficient -1/2 <LM>/<MM>, then returns the counter to 0.
// L_ij is an integer difference (filtered products less products of filtered
// velocities, which cancel to a hundredth), M_ij and the sums are FP64.
__device__ __forceinline__ void block_sum2(double* sl, double* sm, double& a, double& b) {
  sl[threadIdx.x] = a; sm[threadIdx.x] = b;
  __syncthreads();
  for (int w = CHL_DSMF_THREADS / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) { sl[threadIdx.x] += sl[threadIdx.x + w]; sm[threadIdx.x] += sm[threadIdx.x + w]; }
    __syncthreads();
  }
  a = sl[0]; b = sm[0];
}

// -1/2 <LM>/<MM> (L and M both 216/512 of their values, M in units of
// 2^filt_exp).  Whole block; every
// thread gets it.  Thread t adds the partials of chunks t mod 4 = 0..3 into
// four chains (their loads in flight together: on a small instance this tail
// is latency, not throughput), then the chains in a fixed order.
__device__ __forceinline__ double dsm_row_coef(const ChlInst& I, int jc, double* sl, double* sm) {
  const int np = I.npart;
  const size_t n = (size_t)np * CHL_DSMF_THREADS;
  const double* pl = I.part + (size_t)jc * n + threadIdx.x;
  const double* pm = I.part + (size_t)(I.Ny + 2) * n + (size_t)jc * n + threadIdx.x;
  double l[4] = {0.0, 0.0, 0.0, 0.0}, m[4] = {0.0, 0.0, 0.0, 0.0};
  int c = 0;
  for (; c + 4 <= np; c += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      l[u] += __ldcg(pl + (size_t)(c + u) * CHL_DSMF_THREADS);
      m[u] += __ldcg(pm + (size_t)(c + u) * CHL_DSMF_THREADS);
    }
  }
  for (int u = 0; c < np; ++c, ++u) {
    l[u] += __ldcg(pl + (size_t)c * CHL_DSMF_THREADS);
    m[u] += __ldcg(pm + (size_t)c * CHL_DSMF_THREADS);
  }
  double lm = (l[0] + l[1]) + (l[2] + l[3]), mm = (m[0] + m[1]) + (m[2] + m[3]);
  __syncthreads();
  block_sum2(sl, sm, lm, mm);
  const int es = filt_exp(I, (jc - 1) / 2);
  return -0.5 * (lm / mm) * pow2(min(1023, max(-1022, -es)));
}

struct LMSums { double ld, lo, md, mo; };   // diagonal and off-diagonal parts of L:M and M:M
// Doubles a column's sums so far: the reference counts plane 0 (and x position
// 0) twice.  A call, so that its FP64 instructions are not predicated into
// every point.
static __device__ __noinline__ void twice(LMSums& s) { s.ld *= 2.0; s.lo *= 2.0; s.md *= 2.0; s.mo *= 2.0; }

#define DSM_C 0x4BDA12F684BDA12FLL     // 2048/216 / 32 2^64
__global__ void __launch_bounds__(CHL_DSMF_THREADS, 14)
k_dsm_final(ChlMap map, int s_in) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const int np = I.npart;
  const int jc = 1 + lb / np, chunk = lb % np;
  const unsigned col = (unsigned)chunk * CHL_DSMF_THREADS + threadIdx.x;
  const unsigned kc = col / (unsigned)Nx;
  const int i = (int)(col - kc * (unsigned)Nx), k0 = (int)kc * I.dsm_planes, k1 = min(Nz, k0 + I.dsm_planes);
  const bool wall = jc == 1 || jc == Ny;
  LMSums a = {0.0, 0.0, 0.0, 0.0};
  if (k0 < k1) {
    const unsigned* vm = chl_vmax(I, s_in);
    const int eu = fx_exp<60>(vm[0]), ev = fx_exp<60>(vm[1]), ew = fx_exp<60>(vm[2]);
    const int es = filt_exp(I, (jc - 1) / 2);
    const fx* const* R = reinterpret_cast<const fx* const*>(I.r);
    StrainColumn c(I, R[15], R[16], R[17], eu, ev, ew, i, jc, k0);
    const int4 sl = filt_slack(I, (jc - 1) / 2);
    const int lu = eu - sl.x, lv = ev - sl.y, lw = ew - sl.z;      // exponents in L
    for (int k = k0; k < k1; ++k) {
      fx f[3];
      const Strain h = c.point(k, f);
      const size_t o = cidx(I, i, jc, k);
      if (wall) {          // the centre velocities filtered in their own right
        f[0] = LDG(R[0] + cidx(I, c.im, jc, k)) + LDG(R[0] + o);
        f[1] = LDG(R[1] + o);
        f[2] = LDG(R[2] + cidx(I, i, jc, k == 0 ? Nz - 1 : k - 1)) + LDG(R[2] + o);
      }
      // M_ij: 4 |S^| S^_ij less the filtered |S| S_ij (off the diagonal twice
      // that), 216/512 of its value and in units of the filtered fields
      const double hs = h.s * scale_exp(4.0 * 512.0 / 216.0, min(900, max(-900, h.e - es)));
#define MIJ(n) fma(hs, fx_raw<false>(h.t[n]), -fx_raw<(n) < 3>(LDG(R[9 + (n)] + o)))
      const double M1 = MIJ(0), M2 = MIJ(1), M3 = MIJ(2), M4 = MIJ(3), M5 = MIJ(4), M6 = MIJ(5);
#undef MIJ
      // L_ij: f are the filtered face sums, 216/512 of their value and in
      // units twice the copies', shifted up by the group's slack; g = 512/216 f / 8
      f[0] <<= sl.x; f[1] <<= sl.y; f[2] <<= sl.z;
      const fx g0 = fx_mul_mean<64>(2 * f[0], DSM_C), g1 = fx_mul_mean<64>(2 * f[1], DSM_C), g2 = fx_mul_mean<64>(2 * f[2], DSM_C);
#define PROD(g, h) fx_mul_mean<62>(2 * (g), 2 * (h))
      const double L1 = fx_to<true>(LDG(R[3] + o) - PROD(g0, f[0]), lu + lu + 60);
      const double L2 = fx_to<true>(LDG(R[4] + o) - PROD(g1, f[1]), lv + lv + 60);
      const double L3 = fx_to<true>(LDG(R[5] + o) - PROD(g2, f[2]), lw + lw + 60);
      const double L4 = fx_to<true>(LDG(R[6] + o) - PROD(g0, f[1]), lu + lv + 60);
      const double L5 = fx_to<true>(LDG(R[7] + o) - PROD(g0, f[2]), lu + lw + 60);
      const double L6 = fx_to<true>(LDG(R[8] + o) - PROD(g1, f[2]), lv + lw + 60);
#undef PROD
      a.ld = fma(L1, M1, a.ld); a.ld = fma(L2, M2, a.ld); a.ld = fma(L3, M3, a.ld);
      a.lo = fma(L4, M4, a.lo); a.lo = fma(L5, M5, a.lo); a.lo = fma(L6, M6, a.lo);
      a.md = fma(M1, M1, a.md); a.md = fma(M2, M2, a.md); a.md = fma(M3, M3, a.md);
      a.mo = fma(M4, M4, a.mo); a.mo = fma(M5, M5, a.mo); a.mo = fma(M6, M6, a.mo);
      if (k == 0) twice(a);
    }
    if (i == 0) twice(a);
  }
  const size_t n = (size_t)np * CHL_DSMF_THREADS;
  const size_t q = (size_t)jc * n + (size_t)chunk * CHL_DSMF_THREADS + threadIdx.x;
  I.part[q] = a.lo + a.ld;
  I.part[(size_t)(Ny + 2) * n + q] = fma(0.5, a.mo, a.md);
  __threadfence();
  __shared__ double sl[CHL_DSMF_THREADS], sm[CHL_DSMF_THREADS];
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(I.dsm_cnt + jc, 1) == np - 1;     // the row's last block
  __syncthreads();
  if (last) {
    __threadfence();
    const double c = dsm_row_coef(I, jc, sl, sm);
    if (threadIdx.x == 0) { I.coef[jc] = c; I.dsm_cnt[jc] = 0; }
  }
}

// ------------------------------------------------------------ equilibrium log-law wall stress
#define EQWM_KAPPA 0.41
#define EQWM_B 5.2
#define EQWM_ITERS 12
// Newton on f(ut) = ut (ln(h ut/nu)/kappa + B) - |u|.  f is convex and
// increasing, so Newton converges from either side of the root (from the
// left the first step lands right of it, then the iterates decrease).  The
// log law applies only above its upper crossing with u+ = y+ (y+ ~ 11), i.e.
// where ln(y+)/kappa + B < y+ at the laminar y+ = sqrt(|u| h/nu); below it
// tau is the laminar |u| nu/h.
//
// The iteration in FP64 throughout, with a log and a division per step: for
// points next to the crossing and magnitudes outside FP32.  hn = h/nu.
static __device__ __noinline__ double eqlog_ut_fp64(double au, double hn) {
  const double inv_k = 1.0 / EQWM_KAPPA;   // folded at compile time
  const double ut_lam = sqrt(au / hn);
  const double yp_lam = hn * ut_lam;
  const double f0 = ut_lam * fma(log(yp_lam), inv_k, EQWM_B) - au;
  double ut = ut_lam;
  if (f0 < 0.0 && yp_lam >= 1.0) {
    for (int it = 0; it < 2 * EQWM_ITERS; ++it) {
      const double g = fma(log(hn * ut), inv_k, EQWM_B);          // u+ at ut
      const double d = fma(ut, g, -au) / (g + inv_k);             // f / f'
      ut = ut - d;
      if (fabs(d) <= 3e-8 * ut) break;
    }
  }
  return ut;
}
// The same root from FP32 iterates, which the idle FP32 pipe gives for
// nothing, and one FP64 step from them: with the iterate within 1e-6 of the
// root, Halley's step (Newton's with the f'' f/(2 f'^2) term, needed to 1e-10
// of itself only) leaves 1e-18.  One FP64 log per point instead of one per
// iteration, and no FP64 division.
__device__ __forceinline__ double eqlog_tau(double u, double hn, double prev) {
  const double inv_k = 1.0 / EQWM_KAPPA;
  const float ik = (float)(1.0 / EQWM_KAPPA), B = (float)EQWM_B;
  const double au = fabs(u);
  const float af = (float)au, hf = (float)hn;
  const float yp = sqrtf(af * hf);
  const float gap = yp - (logf(yp) * ik + B);          // > 0: log law (for yp >= 1)
  double ut;
  if (!(yp > 1e-12f && yp < 1e12f && hf > 1e-12f && hf < 1e12f && fabsf(gap) > 1e-4f * (yp + B))) {
    ut = eqlog_ut_fp64(au, hn);
  } else if (gap < 0.0f || yp < 1.0f) {
    const double tau = au / hn;
    return u < 0.0 ? -tau : tau;
  } else {
    const float lam = yp / hf, warm = sqrtf(fabsf((float)prev));
    float x = warm > lam ? warm : lam;
    for (int it = 0; it < 2 * EQWM_ITERS; ++it) {
      const float g = logf(hf * x) * ik + B;
      const float d = (x * g - af) / (g + ik);
      x -= d;
      if (fabsf(d) <= 1e-6f * x) break;
    }
    const double x0 = x;
    const double g = fma(log(hn * x0), inv_k, EQWM_B);   // u+
    const double r = fma(x0, g, -au), fp = g + inv_k;     // f and f'
    double q;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(q) : "d"(fp));
    double d = r * q;
    d = fma(fma(-d, fp, r), q, d);
    const double c = (0.5 * inv_k) * q * d;                        // f'' f / (2 f'^2) times ut
    ut = x0 - fma(d, c * (double)(1.0f / x), d);
  }
  const double tau = ut * ut;
  return u < 0.0 ? -tau : (u > 0.0 ? tau : 0.0);
}

// CHL_WALL_THREADS-wide blocks: the 2 Nx Nz wall points of a small channel
// are few, and the serial Newton chains are FP64-issue bound, so they are
// spread over as many SMs as there are blocks.
__global__ void __launch_bounds__(CHL_WALL_THREADS)
k_eqwm(ChlMap map, int s_in) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  if (t >= (unsigned)(2 * Nx * Nz)) return;
  const ChlIdx p = chl_split(t, Nx, Nz);
  const int a = p.i, k = p.j, wall = p.k;
  const double* U = I.U[s_in];
  const double u = wall == 0 ? U[cidx(I, a, 3, k)] : U[cidx(I, a, Ny - 2, k)];
  I.alpha[t] = eqlog_tau(u, wall == 0 ? I.hnb : I.hnt, I.alpha[t]);
}

// ------------------------------------------------------------ nu_t (+ wall model rows)
// nu + nu_t of every centre but the interior ones of the Smagorinsky models:
// no model, AMD and Vreman (S holds nu_t itself) and the ghost rows.  A call,
// so that its FP64 instructions are not predicated into the common path.
static __device__ __noinline__ double nut_other(const ChlInst& I, int i, int jc, int k) {
  if (I.LES_model == 0) return I.nu;
  if (jc == 0 || jc == I.Ny + 1) {         // ghost rows: the rule of Dirichlet_nu_t
    const int js = jc == 0 ? 1 : I.Ny;
    const double sv = I.S[cidx(I, i, js, k)];
    return I.nu + nut_ghost(I, chl_pos(I.LES_model >= 3 ? sv : I.coef[js] * sv));
  }
  return I.nu + chl_pos(I.S[cidx(I, i, jc, k)]);
}
// One thread per pair of x points of a row jc = 0..Ny+1 and `planes` planes: a
// stream of 16 bytes in and out per pair, 11 us of HBM at 256x96x192.  With one
// point per thread it took 52 us, with one pair 30 (blocks too short-lived for
// their start-up and their fold of the maximum), now 22.  With the wall model on,
// rows 0, 1 and Ny, Ny+1 are k_wall_rows's.
__global__ void __launch_bounds__(256)
k_nut(ChlMap map, int use_wm) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, nxp = Nx / 2, M = map.planes, nk = (Nz + M - 1) / M;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x, n = (unsigned)(nxp * (Ny + 2) * nk);
  const bool valid = t < n;
  // lanes past the end repeat the last column and write nothing
  const ChlIdx p = chl_split(valid ? t : n - 1u, nxp, Ny + 2);
  const int i = 2 * p.i, jc = p.j, k0 = p.k * M, k1 = min(Nz, k0 + M);
  const bool wm = use_wm && I.wall_model != 0 && (jc <= 1 || jc >= Ny);
  unsigned hi = 0u;
  if (valid && !wm) {
    // stored as nu + nu_t: every consumer adds nu (equations.f90:139-155)
    const double nu = I.nu;
    double2* nut = reinterpret_cast<double2*>(I.nut);
    if (I.LES_model == 0 || I.LES_model >= 3 || jc == 0 || jc == Ny + 1) {
      for (int k = k0; k < k1; ++k) {
        const double2 v = make_double2(nut_other(I, i, jc, k), nut_other(I, i + 1, jc, k));
        nut[cidx(I, i, jc, k) / 2] = v;
        hi = max(hi, max(chl_abshi(v.x), chl_abshi(v.y)));
      }
    } else {
      // nu + max(0, c |S|) as one FMA, nu + c |S|, clipped below at nu by the
      // bit patterns (both positive; a NaN, for which max gives 0, gives nu)
      const double cj = I.coef[jc];
      const double2* S = reinterpret_cast<const double2*>(I.S);
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        const size_t c = cidx(I, i, jc, k) / 2;
        const double2 s = __ldg(S + c);
        const double2 v = make_double2(chl_atleast(fma(cj, s.x, nu), nu), chl_atleast(fma(cj, s.y, nu), nu));
        nut[c] = v;
        hi = max(hi, max(chl_abshi(v.x), chl_abshi(v.y)));
      }
    }
  }
  chl_line_max(I.nmax, (unsigned)(p.k * (Ny + 2) + jc), Ny + 2, 0, hi);
}

// nu + nu_t on the wall-model rows, jc = 0, 1 and Ny, Ny+1: nu_t is the mean
// of the face values at x faces i-1 and i, the same in both rows of a wall.
// One thread per wall point; face i-1 comes from the lane to the left when
// that lane is on the same row, so no thread returns before the shuffle.  The
// values, which have no bound, stay out of the rows' largest (chl_rhs.cu:
// wall_face).  A kernel of its own, beside the model's: where k_amd and
// k_strain<false> did these rows, whose divisions the whole block waits for, they
// took 17 and 9 us more at 256x96x192.
__global__ void __launch_bounds__(256)
k_wall_rows(ChlMap map, int s_in) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x, n = (unsigned)(2 * Nx * Nz);
  const bool valid = t < n;                        // lanes past the end repeat the last point and write nothing
  const ChlIdx p = chl_split(valid ? t : n - 1u, Nx, Nz);
  const int i = p.i, k = p.j, wall = p.k;
  const double* U = I.U[s_in];
  const double f = wm_face(I, U, i, k, wall);
  const double f_left = __shfl_up_sync(0xffffffffu, f, 1);
  const double fl = ((threadIdx.x & 31) > 0 && i > 0) ? f_left : wm_face(I, U, wrap(i - 1, Nx), k, wall);
  const double v = I.nu + 0.5 * (fl + f);
  if (valid) I.nut[cidx(I, i, wall == 0 ? 0 : Ny, k)] = I.nut[cidx(I, i, wall == 0 ? 1 : Ny + 1, k)] = v;
}

// ------------------------------------------------------------ launchers
extern "C" {
void chl_launch_strain(const ChlMap& m, int nb, int s_in, int dsm, int use_wm, cudaStream_t st) {
  chl_launch_pdl(dsm ? k_strain<true> : k_strain<false>, dim3(nb), dim3(CHL_FLUX_THREADS), 0, st, m, s_in, use_wm);
}
int chl_filter_blocks(int Nx, int Ny, int Nz, int T, int M) {
  const FiltShape f = filt_shape(Nx, Ny, Nz, T, M);
  return FILT_FIELDS * f.full + 3 * f.segs * f.nz;
}
void chl_launch_filter(const ChlMap& m, int nb, int T, cudaStream_t st) { chl_launch_pdl(k_filter, dim3(nb), dim3(T), 0, st, m); }
void chl_launch_dsm_final(const ChlMap& m, int nb, int s_in, cudaStream_t st) {
  chl_launch_pdl(k_dsm_final, dim3(nb), dim3(CHL_DSMF_THREADS), 0, st, m, s_in);
}
void chl_launch_eqwm(const ChlMap& m, int nb, int s_in, cudaStream_t st) { chl_launch_pdl(k_eqwm, dim3(nb), dim3(CHL_WALL_THREADS), 0, st, m, s_in); }
void chl_launch_nut(const ChlMap& m, int nb, int use_wm, cudaStream_t st) { chl_launch_pdl(k_nut, dim3(nb), dim3(m.tb), 0, st, m, use_wm); }
void chl_launch_wall_rows(const ChlMap& m, int nb, int s_in, cudaStream_t st) { chl_launch_pdl(k_wall_rows, dim3(nb), dim3(256), 0, st, m, s_in); }
}
