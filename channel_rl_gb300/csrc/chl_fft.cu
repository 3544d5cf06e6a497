// Fractional-step projection: divergence, 2-D Fourier transform in x and z,
// one tridiagonal solve in y per wavenumber pair, inverse transform and the
// velocity correction.  Restates compute_projection_step
// (projection.f90:20-214) and, for the actual pressure, the right-hand side
// and solver that compute_pressure (pressure.f90:21-29) calls
// (pressure.f90:42-172).
//
// The reference transforms each y-plane with FFTW-MPI and calls LAPACK
// zgtsv per mode.  Here:
//  * x: two real rows are packed as one complex row, transformed by a
//    shared-memory Stockham FFT (radix 4/3/2, fixed point) and split into two
//    half-spectra (kx = 0..Nx/2) - fused with the divergence that produces
//    the rows;
//  * z: complex columns of the half-spectrum, staged up to 8 kx-columns at a time
//    in shared memory;
//  * y: one thread per real column of a mode runs the Thomas elimination with factors
//    precomputed once per grid (the matrix of a mode never changes between
//    steps), into which the 1/(Nx*Nz) of the inverse transform and the 2 of
//    the real-row packing are folded; the mode's column is staged in shared
//    memory by asynchronous copies when it fits;
//  * the inverse runs the same way back and the x pass writes the pressure.
#include "chl_fix.cuh"

#include <cooperative_groups.h>

// ------------------------------------------------------------ Stockham passes
// Autosort Stockham FFT of radix 4, 3, 2 in 64-bit fixed point (chl_fix.cuh),
// shared memory to shared memory.  On the FP64 pipe a radix-4 butterfly with
// twiddles took 22 instructions of 64 clocks; here it is 36 32-bit
// multiply-adds (IMAD.WIDE) and about 70 additions and shifts, which the
// integer pipes issue in a fifth of that.
//
// Every line is scaled by its own largest component (found while it is
// loaded), so a line's result does not depend on which lines share its block.
// The first pass (no twiddles) grows a line by at most its radix R; every
// later pass is halved, growth R/2, because the halved product is what the
// multiplication gives.  fft_bits(N) is the number of bits a line may start
// with so that no pass input exceeds 2^61: 56 for N = 256, three bits finer
// than a double's last bit at the line's largest component; the rounding of a
// pass (below one unit per product) stays there too.  Measured error of the
// projection: chl_fft's callers compare with FP64 in tests/test_fixed_point_gpu.py.
//
// Table of a length: per pass {R, Ns, 2^32/Ns, 2^32/(N/R)}, then the twiddles.
// Twiddles w = c + is as the words (high, low >> 1) of c 2^63 and s 2^63
// (2^63 - 1 for 1), per pass with twiddles and radix digit r = 1..R-1: entries
// jm = 0..Ns-1 for w = exp(-2 pi i jm r/(Ns R)).
typedef longlong2 fx2;
__device__ __forceinline__ fx2 add2(fx2 a, fx2 b) { return make_longlong2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ fx2 sub2(fx2 a, fx2 b) { return make_longlong2(a.x - b.x, a.y - b.y); }
// a / 2, ties to even: a constant bias of a quarter of a unit would add up over
// the rows of the low modes, which the Poisson solve amplifies most
__device__ __forceinline__ fx half_even(fx a) { return (a + (fx)(((unsigned)a >> 1) & 1u)) >> 1; }
__device__ __forceinline__ fx2 halve(fx2 a) { return make_longlong2(half_even(a.x), half_even(a.y)); }

// v w / 2 (INV: v conj(w) / 2).  The four cross terms of a component, at most
// 2^62.9 together for |v| < 2^61, are summed before their one shift.  The
// starting value r takes out the mean of what is dropped: half a unit each for
// the shift and the low products (2^31) and (c + s)/4 for the last bit of v's
// components, which the signed 32-bit factors have no room for.
template <bool INV>
__device__ __forceinline__ fx2 tw_mul(fx2 v, int4 w) {
  const long long r = (long long)(0x80000000u + (unsigned)((w.x >> 2) + (w.z >> 2)));
  const fx n = INV ? -v.x : -v.y;
  const int xh = (int)(v.x >> 32), xl = (int)((unsigned)v.x >> 1);
  const int yh = (int)(v.y >> 32), yl = (int)((unsigned)v.y >> 1);
  const int nh = (int)(n >> 32), nl = (int)((unsigned)n >> 1);
  const int ah = INV ? yh : nh, al = INV ? yl : nl;    // times s into the real part
  const int bh = INV ? nh : xh, bl = INV ? nl : xl;    // times s into the imaginary part
  long long t = r + (long long)xh * w.y + (long long)w.x * xl;
  t += (long long)ah * w.w;
  t += (long long)w.z * al;
  long long u = r + (long long)yh * w.y + (long long)w.x * yl;
  u += (long long)bh * w.w;
  u += (long long)w.z * bl;
  return make_longlong2((long long)xh * w.x + (long long)ah * w.z + (t >> 31),
                        (long long)yh * w.x + (long long)bh * w.z + (u >> 31));
}

// a sin(2 pi/3), |a| < 2^62.  The means of the dropped low product (0.380 of a
// unit), last bit of a (0.433) and shift (0.5) come back with the start of t.
__device__ __forceinline__ fx sin60_mul(fx a) {
  const fx w = 0x6ED9EBA16132A9CFLL;   // sin(2 pi/3) 2^63
  const int ah = (int)(a >> 32), wh = (int)(w >> 32);
  const int al = (int)((unsigned)a >> 1), wl = (int)((unsigned)w >> 1);
  const long long t = 1409783857LL + (long long)ah * wl + (long long)wh * al;
  return (fx)((unsigned long long)((long long)ah * wh) << 1) + (t >> 30);
}
// Butterfly of v[0..R): the first input as it is (pass one) or halved by the
// caller, the others twiddled.
template <int R, bool INV>
__device__ __forceinline__ void butterfly(fx2* v) {
  if (R == 2) {
    const fx2 a = v[0], b = v[1];
    v[0] = add2(a, b); v[1] = sub2(a, b);
  } else if (R == 4) {
    const fx2 a = add2(v[0], v[2]), b = sub2(v[0], v[2]);
    const fx2 c = add2(v[1], v[3]), e = sub2(v[1], v[3]);
    // d = e * (-i) forward, e * (+i) inverse
    v[0] = add2(a, c); v[2] = sub2(a, c);
    const fx2 p = make_longlong2(b.x + e.y, b.y - e.x), q = make_longlong2(b.x - e.y, b.y + e.x);
    v[1] = INV ? q : p; v[3] = INV ? p : q;
  } else {
    const fx2 t0 = add2(v[1], v[2]), d = sub2(v[1], v[2]);
    const fx2 t = sub2(v[0], halve(t0));
    const fx mx = sin60_mul(d.x), my = sin60_mul(d.y);
    v[0] = add2(v[0], t0);
    const fx2 p = make_longlong2(t.x + my, t.y - mx), q = make_longlong2(t.x - my, t.y + mx);
    v[1] = INV ? q : p; v[2] = INV ? p : q;
  }
}

// Shared memory, in 16-byte units; tiles and tables go by their offset in it
// (a pointer that alternates between the tiles would be a generic one).
__device__ __forceinline__ fx2* smem_fx() { extern __shared__ double2 sm[]; return reinterpret_cast<fx2*>(sm); }
__device__ __forceinline__ double2* smem_d2() { extern __shared__ double2 sm[]; return sm; }
__device__ __forceinline__ int4* smem_tw() { extern __shared__ double2 sm[]; return reinterpret_cast<int4*>(sm); }

// n / d for n < 2^16, 0 < d < 2^16 by one multiplication with m = 2^32/d rounded up (0
// stands for d = 1)
__device__ __forceinline__ int small_div(int n, unsigned m) { return m == 0u ? n : (int)__umulhi((unsigned)n, m); }
struct SmallDiv {
  int d; unsigned m;
  __device__ __forceinline__ explicit SmallDiv(int dd) : d(dd), m(0xFFFFFFFFu / (unsigned)dd + 1u) {}
  __device__ __forceinline__ int div(int n) const { return small_div(n, m); }
};

// One pass over nrows lines: butterfly inputs from ld(row, element), results
// to st(row, element, value).  Work items (row, butterfly j) are numbered so
// that consecutive threads touch neighbouring words: j fastest when a row is
// contiguous (the x lines), the row fastest when rows are interleaved (the z
// columns), which keeps the 16-byte accesses free of bank conflicts.
template <int R, bool TW, bool INV, class LD, class ST>
__device__ __forceinline__ void fx_pass(const LD& ld, const ST& st, const SmallDiv& rows, bool rowfast, int N, int4 pass,
                                        int tab) {
  const int nb = N / R, Ns = pass.y;
  const int d = rowfast ? rows.d : nb;
  const unsigned dm = rowfast ? rows.m : (unsigned)pass.w;
  for (int w = threadIdx.x; w < rows.d * nb; w += blockDim.x) {
    const int q = small_div(w, dm), m = w - q * d;
    const int row = rowfast ? m : q, j = rowfast ? q : m;
    fx2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(row, j + r * nb);
    int o = j * R, step = 1;
    if (TW) {
      const int g = small_div(j, (unsigned)pass.z), jm = j - g * Ns;
      v[0] = halve(v[0]);
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = tw_mul<INV>(v[r], smem_tw()[tab + (r - 1) * Ns + jm]);
      o = g * Ns * R + jm;
      step = Ns;
    }
    butterfly<R, INV>(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(row, o + r * step, v[r]);
  }
}

template <bool TW, bool INV, class LD, class ST>
__device__ __forceinline__ void fx_pass_any(const LD& ld, const ST& st, const SmallDiv& rows, bool rowfast, int N,
                                            int4 pass, int tab) {
  if (pass.x == 4) fx_pass<4, TW, INV>(ld, st, rows, rowfast, N, pass, tab);
  else if (pass.x == 3) fx_pass<3, TW, INV>(ld, st, rows, rowfast, N, pass, tab);
  else fx_pass<2, TW, INV>(ld, st, rows, rowfast, N, pass, tab);
}

// Conversions of a line.  Doubles come in on the integer pipe; of a result's
// two components one goes out on each pipe (scaled by the power of two after
// the hardware's conversion on the FP64 pipe, which nothing else here uses):
// at 256x96x192 the four transforms of a stage take 275 us with all
// conversions on the integer pipe, 262 us like this and 332 us with all of
// them on the FP64 pipe (230 us with what was made cheaper since).
struct LineIn {
  int bits; const unsigned* hi;
  __device__ __forceinline__ int exponent(int r) const { return fx_line_exp(hi[r], bits); }
};
__device__ __forceinline__ fx2 fx2_from(double2 d, int e) { return make_longlong2(fx_from(d.x, e), fx_from(d.y, e)); }

// shared-memory tile of lines: element e of row r at off + r*rs + e*es
struct TileLd {
  int off, rs, es;
  __device__ __forceinline__ fx2 operator()(int r, int e) const { return smem_fx()[off + r * rs + e * es]; }
};
struct TileSt {
  int off, rs, es;
  __device__ __forceinline__ void operator()(int r, int e, fx2 v) const { smem_fx()[off + r * rs + e * es] = v; }
};
// a tile that holds doubles, converted with the exponent of its line
struct RawLd {
  int off, rs, es; LineIn in;
  __device__ __forceinline__ fx2 operator()(int r, int e) const {
    return fx2_from(smem_d2()[off + r * rs + e * es], in.exponent(r));
  }
};
// a line's result as doubles: the passes with twiddles halved it `halvings`
// times; a line with a non-finite input is NaN throughout, one without a value of
// 2^-958 or more zero (the passes round zeros to a unit)
struct LineOut {
  int bits, halvings; const unsigned* hi;
  __device__ __forceinline__ double2 operator()(int r, fx2 v) const {
    const int x = fx_line_exp(hi[r], bits) + halvings;
    const bool special = hi[r] - (64u << 20) >= 0x7FF00000u - (64u << 20);
    const double s = !special ? pow2(x) : fx_bad(hi[r]) ? __longlong_as_double(0x7FF8000000000000LL) : 0.0;
    double a = fx_to(v.x, x);
    if (special) a = s;
    return make_double2(a, __ll2double_rn(v.y) * s);
  }
};
struct DoubleTileSt {
  int off, rs, es; LineOut out;
  __device__ __forceinline__ void operator()(int r, int e, fx2 v) const { smem_d2()[off + r * rs + e * es] = out(r, v); }
};

// Full transform of `passes` passes: the first from `first` into b, the ones
// between through the tiles b and a, the last to `last`.  tab: the length's
// table in shared memory.  Ends without a barrier.
template <bool INV, class LD, class ST>
__device__ __forceinline__ void fx_fft(const LD& first, const ST& last, int a, int b, int nrows, int rs, int es, int N,
                                       int passes, int tab) {
  const bool rowfast = rs < es;
  const SmallDiv rows(nrows);
  __syncthreads();
  if (passes == 1) {
    fx_pass_any<false, INV>(first, last, rows, rowfast, N, smem_tw()[tab], 0);
    return;
  }
  fx_pass_any<false, INV>(first, TileSt{b, rs, es}, rows, rowfast, N, smem_tw()[tab], 0);
  int src = b, dst = a, tw = tab + passes;
  for (int p = 1; p < passes - 1; ++p) {
    const int4 pass = smem_tw()[tab + p];
    __syncthreads();
    fx_pass_any<true, INV>(TileLd{src, rs, es}, TileSt{dst, rs, es}, rows, rowfast, N, pass, tw);
    tw += pass.y * (pass.x - 1);
    const int t = src; src = dst; dst = t;
  }
  __syncthreads();
  fx_pass_any<true, INV>(TileLd{src, rs, es}, last, rows, rowfast, N, smem_tw()[tab + passes - 1], tw);
}
// the tile that fx_fft's last pass may write (it reads the other one)
__device__ __forceinline__ int fx_last_tile(int a, int b, int passes) { return passes & 1 ? b : a; }

// Copies a length's twiddles into shared memory; the barrier ahead of the
// first pass orders it before any use.
__device__ __forceinline__ void stage_twiddles(int4* tws, const int4* __restrict__ tab, int len) {
  for (int w = threadIdx.x; w < len; w += blockDim.x) tws[w] = LDG(tab + w);
}

// Largest component of line `row` among the values of the calling warp's
// lanes (high words; all lanes call, those without a value pass 0).
__device__ __forceinline__ void fold_line(unsigned* hi, int row, unsigned v) {
  const unsigned full = 0xffffffffu;
  if (__all_sync(full, row == __shfl_sync(full, row, 0))) {
    v = __reduce_max_sync(full, v);
    if ((threadIdx.x & 31) == 0) atomicMax(hi + row, v);
  } else {
    atomicMax(hi + row, v);
  }
}
__device__ __forceinline__ unsigned abshi2(double2 v) { return max(chl_abshi(v.x), chl_abshi(v.y)); }

// ------------------------------------------------------------ divergence + forward x
// mode 0: div of velocity set s_in (compute_pseudo_pressure_rhs, projection.f90:40-55)
// mode 1: div of the actual-pressure RHS Fp with the wall rows of Fv set to
//         the pressure BC planes and the BC source terms of pressure.f90:138-139.
// mode 2: mode 0 without a velocity correction to follow (the tuner).  Mode 0
//         clears the set's largest velocities, which k_project forms anew.
// Two of the six differences of a pair of planes go to the integer pipe, beside
// the FP64 one: 88 -> 82 us at 256x96x192 (one, two, three, four, six of them
// 86, 82, 84, 86, 94 us).
__global__ void __launch_bounds__(256)
k_div_fftx(ChlMap map, int s_in, int mode, int xmb) {
  chl_pdl_wait();
  extern __shared__ double2 sm[];
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, Nxh = I.Nxh;
  const int nrow = Ny * (Nz / 2);
  const int CR = chl_fftx_rows(Nx, nrow, xmb);
  const int g0 = lb * CR;
  const int cr_n = min(CR, nrow - g0);
  const int A = 0, B = CR * (Nx + 2), T = B + CR * Nx;       // tiles, twiddles
  unsigned* hi = reinterpret_cast<unsigned*>(sm + T + I.lenx);
  stage_twiddles(smem_tw() + T, I.twx, I.lenx);
  for (int r = threadIdx.x; r < CR; r += blockDim.x) hi[r] = 0u;
  __syncthreads();
  const double *U, *V, *W;
  if (mode == 0) {
    if (lb == 0 && threadIdx.x < 3) chl_vmax(I, s_in)[threadIdx.x] = 0u;
    const int nb = (nrow + CR - 1) / CR;
    for (int w = lb * (int)blockDim.x + threadIdx.x; w < 3 * CHL_ROW_COPIES * (Ny + 2); w += nb * (int)blockDim.x)
      chl_row_words(I, 0, 0)[w] = 0u;
  }
  if (mode != 1) { U = I.U[s_in]; V = I.V[s_in]; W = I.W[s_in]; }
  else { U = I.Fp[0]; V = I.Fp[1]; W = I.Fp[2]; }
  const SmallDiv byNx(Nx);
  for (int w0 = 0; w0 < cr_n * Nx; w0 += blockDim.x) {
    const int w = min(w0 + (int)threadIdx.x, cr_n * Nx - 1);   // lanes past the end repeat the last point
    const int cr = byNx.div(w), i = w - cr * Nx;
    const unsigned g = g0 + cr;
    const int jz = (int)(g / (unsigned)(Nz / 2)), jc = 1 + jz, k0 = 2 * ((int)g - jz * (Nz / 2));
    const int im = wrap(i - 1, Nx);
    double dv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + h, km = wrap(k - 1, Nz);
      double vlo = LDG(V + vidx(I, i, jc - 1, k)), vhi = LDG(V + vidx(I, i, jc, k));
      if (mode == 1) {
        if (jc == 1) vlo = I.bc[(size_t)k * Nx + i];
        if (jc == Ny) vhi = I.bc[(size_t)Nx * Nz + (size_t)k * Nx + i];
      }
      const double uhi = LDG(U + cidx(I, i, jc, k)), ulo = LDG(U + cidx(I, im, jc, k));
      double d = (h == 0 ? fx_sub(uhi, ulo) : uhi - ulo) * LDG(I.rdxc + i)
               + (h == 0 ? fx_sub(vhi, vlo) : vhi - vlo) * LDG(I.rdyc + jc)
               + (LDG(W + cidx(I, i, jc, k)) - LDG(W + cidx(I, i, jc, km))) * LDG(I.rdzc + k);
      if (mode == 1) {
        if (jc == 1) d += I.cbc1 * I.bc[(size_t)k * Nx + i];
        if (jc == Ny) d -= I.cbc2 * I.bc[(size_t)Nx * Nz + (size_t)k * Nx + i];
      }
      dv[h] = d;
    }
    sm[cr * Nx + i] = make_double2(dv[0], dv[1]);
    fold_line(hi, cr, abshi2(make_double2(dv[0], dv[1])));
  }
  // one bit less than the transform allows: the split below adds two elements
  const int bits = I.bitsx - 1;
  const int last = fx_last_tile(A, B, I.passx);
  fx_fft<false>(RawLd{A, Nx, 1, LineIn{bits, hi}}, TileSt{last, Nx, 1}, A, B, cr_n, Nx, 1, Nx, I.passx, T);
  const fx2* res = smem_fx() + last;
  __syncthreads();
  // split the packed spectrum into the two half-spectra (each times 2)
  const LineOut out{bits, I.passx - 1, hi};
  const SmallDiv byNxh(Nxh);
  for (int w = threadIdx.x; w < cr_n * Nxh; w += blockDim.x) {
    const int cr = byNxh.div(w), kx = w - cr * Nxh;
    const unsigned g = g0 + cr;
    const int jz = (int)(g / (unsigned)(Nz / 2)), jc = 1 + jz, k0 = 2 * ((int)g - jz * (Nz / 2));
    const fx2 z = res[cr * Nx + kx];
    const fx2 zc = res[cr * Nx + (kx == 0 ? 0 : Nx - kx)];   // conj taken below
    I.spec[((size_t)jc * Nz + k0) * Nxh + kx] = out(cr, make_longlong2(z.x + zc.x, z.y - zc.y));
    I.spec[((size_t)jc * Nz + k0 + 1) * Nxh + kx] = out(cr, make_longlong2(z.y + zc.y, zc.x - z.x));
  }
}

// ------------------------------------------------------------ z transform of the half spectrum
// a column's element k straight to the spectrum
struct SpecSt {
  double2* spec; const size_t* coff; int pitch; LineOut out;
  __device__ __forceinline__ void operator()(int c, int k, fx2 v) const { spec[coff[c] + (size_t)k * pitch] = out(c, v); }
};

template <bool INV>
__global__ void __launch_bounds__(256)
k_fftz(ChlMap map, int zcw) {
  chl_pdl_wait();
  // The Ny x Nxh columns (jc, kx) of an instance are numbered jc-major and
  // cut into runs of zcw (chl_fftz_cols); a run may cross into the next
  // jc row, so every column is a full one and only the instance's last
  // block is short.
  extern __shared__ double2 sm[];
  __shared__ size_t coff[16];
  __shared__ unsigned hi[16];    // the columns' largest components
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nz = I.Nz, Nxh = I.Nxh;
  const int q0 = lb * zcw;
  const int cw = min(zcw, I.Ny * Nxh - q0);
  if (threadIdx.x < cw) {
    const int q = q0 + threadIdx.x;
    coff[threadIdx.x] = (size_t)(1 + q / Nxh) * Nz * Nxh + (q % Nxh);
    hi[threadIdx.x] = 0u;
  }
  __syncthreads();
  const int A = 0, B = Nz * zcw, T = 2 * Nz * zcw;           // tiles, twiddles
  stage_twiddles(smem_tw() + T, I.twz, I.lenz);
  double2* spec = I.spec;
  unsigned mine = 0u;
  const bool fixed_c = blockDim.x % cw == 0;     // a thread stays on one column
  const SmallDiv bycw(cw);
  for (int w = threadIdx.x; w < Nz * cw; w += blockDim.x) {
    const int k = bycw.div(w), c = w - k * cw;
    const double2 v = spec[coff[c] + (size_t)k * Nxh];
    sm[k * zcw + c] = v;
    mine = max(mine, abshi2(v));
    if (!fixed_c) { atomicMax(hi + c, mine); mine = 0u; }
  }
  if (fixed_c) atomicMax(hi + threadIdx.x % cw, mine);
  const int bits = I.bitsz;
  const RawLd first{A, 1, zcw, LineIn{bits, hi}};
  const SpecSt last{spec, coff, Nxh, LineOut{bits, I.passz - 1, hi}};
  fx_fft<INV>(first, last, A, B, cw, 1, zcw, Nz, I.passz, T);
}

// ------------------------------------------------------------ tridiagonal per mode
// The solves are serial chains of FP64 instructions, one of which holds a
// warp's scheduler for 64 clocks; a channel has few chains, so they are cut
// as fine as they go: the real and the imaginary part of a mode are columns
// of their own, in neighbouring lanes (column t = 2 mode + part, rows 2 ps
// doubles apart; the factors are shared).  With a mode per thread a warp
// issued 6 FP64 instructions per row where it now issues 3, and the last wave
// of 774 warps at 256x96x192 left 442 of the 608 schedulers with half the
// work: 57 us per launch there, now 40 (HBM floor 20); 23 and 17 us for the
// staged form at 64^3 (5 of them the launch between events).
// Forward, the product with inv is formed apart from the chain, which is one
// FMA per row.
// rows [j0, j0 + TB) of [lo, hi): v[q] = p[j stride]
template <int TB>
__device__ __forceinline__ void tri_up(double (&v)[TB], const double* p, size_t stride, int j0, int hi) {
#pragma unroll
  for (int q = 0; q < TB; ++q) if (j0 + q < hi) v[q] = p[(size_t)(j0 + q) * stride];
}
// rows j1, j1 - 1, ... down to lo
template <int TB>
__device__ __forceinline__ void tri_down(double (&v)[TB], const double* p, size_t stride, int j1, int lo) {
#pragma unroll
  for (int q = 0; q < TB; ++q) if (j1 - q >= lo) v[q] = p[(size_t)(j1 - q) * stride];
}
// Forward elimination y_j = inv_j d_j - m_j y_{j-1} over rows [lo, hi) of a
// column from y = prev (d: column and row stride; fi, fm: the mode's factors,
// rows ps apart); STORE: into d, else forms the affine map y_in -> y of the
// rows, A the product of the -m_j.  The recurrence is serial in j; the loads
// are not: TB rows are fetched together, and from global memory (GLOBAL) while
// the TB rows before them are in the chain (47 -> 40 us at 256x96x192; from
// shared memory it only costs registers).  Short columns leave the last TB
// early: a predicated-off FP64 instruction takes its 64 clocks all the same.
template <int TB, bool GLOBAL, bool STORE>
__device__ __forceinline__ double tri_forward(double* d, size_t ds, const double* __restrict__ fi,
                                              const double* __restrict__ fm, size_t ps, int lo, int hi, double prev,
                                              double& A) {
  double nx[TB], ni[TB], nm[TB];
  auto fetch = [&](int j) { tri_up(nx, d, ds, j, hi); tri_up(ni, fi, ps, j, hi); tri_up(nm, fm, ps, j, hi); };
  if (GLOBAL) fetch(lo);
  for (int j0 = lo; j0 < hi; j0 += TB) {
    if (!GLOBAL) fetch(j0);
    double x[TB], m[TB];
#pragma unroll
    for (int q = 0; q < TB; ++q) { if (GLOBAL) x[q] = nx[q] * ni[q]; m[q] = nm[q]; }
    if (GLOBAL) fetch(j0 + TB);
#pragma unroll
    for (int q = 0; q < TB; ++q) {
      if (!GLOBAL && j0 + q >= hi) break;
      if (j0 + q < hi) {
        prev = fma(-m[q], prev, GLOBAL ? x[q] : nx[q] * ni[q]);   // m = 0 on the first row
        if (STORE) d[(size_t)(j0 + q) * ds] = prev;
        else A = -m[q] * A;
      }
    }
  }
  return prev;
}
// back substitution x_j = y_j - c_j x_{j+1} from the top (c = 0 on the last row)
template <int TB, bool GLOBAL, bool STORE>
__device__ __forceinline__ double tri_backward(const double* y, size_t ys, double* d, size_t ds, const double* __restrict__ fc,
                                               size_t ps, int lo, int hi, double prev, double& A) {
  double nx[TB], nc[TB];
  auto fetch = [&](int j) { tri_down(nx, y, ys, j, lo); tri_down(nc, fc, ps, j, lo); };
  if (GLOBAL) fetch(hi - 1);
  for (int j1 = hi - 1; j1 >= lo; j1 -= TB) {
    if (!GLOBAL) fetch(j1);
    double x[TB], c[TB];
#pragma unroll
    for (int q = 0; q < TB; ++q) { x[q] = nx[q]; c[q] = nc[q]; }
    if (GLOBAL) fetch(j1 - TB);
#pragma unroll
    for (int q = 0; q < TB; ++q) {
      if (!GLOBAL && j1 - q < lo) break;
      if (j1 - q >= lo) {
        prev = fma(-c[q], prev, x[q]);
        if (STORE) d[(size_t)(j1 - q) * ds] = prev;
        else A = -c[q] * A;
      }
    }
  }
  return prev;
}

__global__ void __launch_bounds__(128, 4)
k_tri(ChlMap map) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x, mode = t >> 1;
  const size_t ps = (size_t)I.Nz * I.Nxh;       // row pitch of spec and factors
  if (mode >= ps) return;
  double* d = reinterpret_cast<double*>(I.spec + ps) + t;   // row jc = 1
  double A = 1.0;
  tri_forward<8, true, true>(d, 2 * ps, I.tri_inv + mode, I.tri_m + mode, ps, 0, I.Ny, 0.0, A);
  tri_backward<8, true, true>(d, 2 * ps, d, 2 * ps, I.tri_c + mode, ps, 0, I.Ny, 0.0, A);
}

// Staged form, for columns that fit in shared memory: TRI_W modes, 2 TRI_W
// threads per block.  Each thread copies its column and, with its neighbour,
// the mode's factors into shared memory with cp.async (all rows in flight at
// once, where the form above waits once per TB rows), runs both sweeps there
// and writes only the solution.  A warp reads back only what it copied
// itself, so the copies need a wait but no block barrier.  The arithmetic
// and its order are those of k_tri.
#define TRI_W 32
__device__ __forceinline__ void cp_async8(void* sdst, const void* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" :: "r"(s), "l"(gsrc) : "memory");
}

__global__ void __launch_bounds__(2 * TRI_W)
k_tri_staged(ChlMap map) {
  chl_pdl_wait();
  extern __shared__ double2 smt[];
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Ny = I.Ny;
  const size_t ps = (size_t)I.Nz * I.Nxh;       // row pitch of spec and factors
  const int t = threadIdx.x, m = t >> 1;
  const size_t mode = (size_t)lb * TRI_W + m;
  const bool valid = mode < ps;                 // lanes past the last mode copy nothing
  double* d = reinterpret_cast<double*>(I.spec + ps + mode) + (t & 1);   // row jc = 1
  // [Ny][2 TRI_W] right side, then [Ny][TRI_W] inv, m and c
  double* sd = reinterpret_cast<double*>(smt);
  double* si = sd + (size_t)Ny * 2 * TRI_W;
  double* sm = si + (size_t)Ny * TRI_W;
  double* sc = sm + (size_t)Ny * TRI_W;
  for (int j = 0; valid && j < Ny; ++j) {
    const size_t g = (size_t)j * ps + mode, l = (size_t)j * TRI_W + m;
    cp_async8(sd + (size_t)j * 2 * TRI_W + t, d + (size_t)j * 2 * ps);
    if (t & 1) {
      cp_async8(sc + l, I.tri_c + g);
    } else {
      cp_async8(si + l, I.tri_inv + g);
      cp_async8(sm + l, I.tri_m + g);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncwarp();
  if (!valid) return;
  double A = 1.0;
  tri_forward<8, false, true>(sd + t, 2 * TRI_W, si + m, sm + m, TRI_W, 0, Ny, 0.0, A);
  tri_backward<8, false, true>(sd + t, 2 * TRI_W, d, 2 * ps, sc + m, TRI_W, 0, Ny, 0.0, A);
}

// Lane-split form, for instances with few modes: chl_tri_lanes(modes, Ny) =
// P lanes per column (P = 1 for the larger instances of the same launch).
// Lane p owns rows [p L, (p+1) L), L = ceil(Ny / P).  Forward, the
// elimination maps the value entering a lane's rows affinely to the value
// leaving them: A y_in + B.  Each lane forms (A, B) from y_in = 0, an
// inclusive scan of these maps over the P lanes (warp shuffles within the lane
// group) gives every lane its y_in, and the lane reruns its rows from it,
// storing them.  The back substitution is split the same way from the top.
// With P = 1 the arithmetic is k_tri's; with P > 1 the scan rounds
// differently from the serial sweep (the multipliers are below 1 in
// magnitude, so the maps are contractions).  Every lane of a warp reaches the
// shuffles: a lane group belongs to one column, and lanes past the last
// carry no rows.
//
// The scan: the map (A, z) of lane p's rows in, the value entering them out
// (0 for the first lane).  UP: lane 0 first, else lane P - 1.
template <bool UP>
__device__ __forceinline__ double tri_lane_scan(double A, double z, int p, int P) {
  const unsigned full = 0xffffffffu;
  for (int off = 1; off < P; off <<= 1) {
    const double Ao = UP ? __shfl_up_sync(full, A, off, P) : __shfl_down_sync(full, A, off, P);
    const double b = UP ? __shfl_up_sync(full, z, off, P) : __shfl_down_sync(full, z, off, P);
    if (UP ? p >= off : p + off < P) { z = fma(A, b, z); A *= Ao; }
  }
  const double in = UP ? __shfl_up_sync(full, z, 1, P) : __shfl_down_sync(full, z, 1, P);
  return p == (UP ? 0 : P - 1) ? 0.0 : in;
}
__global__ void __launch_bounds__(128)
k_tri_scan(ChlMap map) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Ny = I.Ny;
  const size_t ps = (size_t)I.Nz * I.Nxh;           // row pitch of spec and factors
  const int P = chl_tri_lanes((long)ps, Ny);
  const unsigned g = (unsigned)lb * blockDim.x + threadIdx.x, col = g / P;
  const int p = (int)(g % P);
  const bool valid = col < 2 * ps;
  const int L = (Ny + P - 1) / P;
  const int lo = min(Ny, p * L);
  const int hi = valid ? min(Ny, lo + L) : lo;      // rows [lo, hi) of this lane
  const size_t c = valid ? col : 0, mode = c >> 1;
  double* d = reinterpret_cast<double*>(I.spec + ps) + c;       // row jc = 1
  const double* fi = I.tri_inv + mode;
  const double* fm = I.tri_m + mode;
  const double* fc = I.tri_c + mode;
  double A = 1.0, in = 0.0;
  if (P > 1) {
    const double z = tri_forward<8, true, false>(d, 2 * ps, fi, fm, ps, lo, hi, 0.0, A);
    in = tri_lane_scan<true>(A, z, p, P);
  }
  tri_forward<8, true, true>(d, 2 * ps, fi, fm, ps, lo, hi, in, A);
  A = 1.0; in = 0.0;
  if (P > 1) {
    const double z = tri_backward<8, true, false>(d, 2 * ps, d, 2 * ps, fc, ps, lo, hi, 0.0, A);
    in = tri_lane_scan<false>(A, z, p, P);
  }
  tri_backward<8, true, true>(d, 2 * ps, d, 2 * ps, fc, ps, lo, hi, in, A);
}

// ------------------------------------------------------------ fused z transform + tridiagonal + inverse z
// For instances whose wavenumber column block fits in shared memory: one
// thread-block cluster of P CTAs per (instance, kx), P = chl_tri_lanes of
// the instance (the lane count of k_tri_scan).  CTA r holds the rows that
// lane r of k_tri_scan owns, [r L, min(Ny, (r+1) L)) with L = ceil(Ny/P),
// for all Nz wavenumbers kz, and runs on them
//   the forward z transform (the Stockham passes of k_fftz),
//   the Thomas sweeps of k_tri_scan, whose lane maps (A, z) it exchanges
//     with the other CTAs of its cluster through distributed shared memory
//     and scans with the same warp shuffles (one thread per (kz, lane)),
//   the inverse z transform,
// so the result is bit-identical to k_fftz, the tridiagonal kernel and
// k_fftz again, in one launch and without the two round trips of the
// spectrum.  The cluster barriers are hardware barriers that every thread
// of the cluster reaches (no early exit).
namespace cg = cooperative_groups;

// hi[r] of the rows r of a tile (element e at r + e*es), one warp per row
__device__ __forceinline__ void line_max(const double2* p, int nrows, int es, int N, unsigned* hi) {
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < nrows; r += blockDim.x >> 5) {
    unsigned v = 0u;
    for (int e = lane; e < N; e += 32) v = max(v, abshi2(p[r + e * es]));
    v = __reduce_max_sync(0xffffffffu, v);
    if (lane == 0) hi[r] = v;
  }
}
// row r, wavenumber e of a spectrum column
struct RowSt {
  double2* p; size_t rowpitch, pitch; LineOut out;
  __device__ __forceinline__ void operator()(int r, int e, fx2 v) const { p[(size_t)r * rowpitch + (size_t)e * pitch] = out(r, v); }
};

// 64 registers: with 128 (eight rows fetched together) a step of 32x48x32 takes
// 241 us instead of 236, the block finding no room beside its predecessor's.
__global__ void __launch_bounds__(256, 4)
k_zsolve(ChlMap map) {
  chl_pdl_wait();
  extern __shared__ double2 sm[];
  cg::cluster_group cl = cg::this_cluster();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Ny = I.Ny, Nz = I.Nz, Nxh = I.Nxh;
  const long modes = (long)Nz * Nxh;
  const int P = chl_tri_lanes(modes, Ny);       // the cluster size (host-checked)
  const int r = lb % P, kx = lb / P;
  const int L = (Ny + P - 1) / P;
  const int lo = min(Ny, r * L), hi = min(Ny, lo + L), nr = hi - lo;
  const size_t ps = (size_t)modes;              // row pitch of spec and factors
  double2* A = sm;
  const int T = 2 * L * Nz;                                     // twiddles
  double* fz = reinterpret_cast<double*>(sm + T + I.lenz);   // per column: forward lane values
  double* bw = fz + 2 * Nz;                     // backward lane values
  double* in = bw + 2 * Nz;                     // values entering the rows, first upwards, then downwards
  double* fA = in + 2 * Nz;
  double* bA = fA + 2 * Nz;
  unsigned* top = reinterpret_cast<unsigned*>(bA + 2 * Nz);          // the lines' largest components
  const int t = threadIdx.x, bd = blockDim.x;
  const int bits = I.bitsz, halvings = I.passz - 1;
  stage_twiddles(smem_tw() + T, I.twz, I.lenz);
  // rows [lo, hi) of column kx: element (row l, kz) at l + kz*nr
  double2* spec = I.spec + ps + kx;             // row jc = 1
  for (int w = t; w < nr * Nz; w += bd) {
    const int l = w % nr, kz = w / nr;
    A[l + (size_t)kz * nr] = spec[(size_t)(lo + l) * ps + (size_t)kz * Nxh];
  }
  __syncthreads();
  line_max(A, nr, nr, Nz, top);
  const int r0 = fx_last_tile(0, L * Nz, I.passz);
  double2* res = sm + r0;
  // (the last CTAs of a cluster may have no rows)
  if (nr > 0)
    fx_fft<false>(RawLd{0, 1, nr, LineIn{bits, top}}, DoubleTileSt{r0, 1, nr, LineOut{bits, halvings, top}}, 0, L * Nz, nr, 1,
                  nr, Nz, I.passz, T);
  __syncthreads();
  // column w = 2 kz + part of this CTA's rows: element l at rows + 2 l (kz nr of them before)
  double* const rows = reinterpret_cast<double*>(res);
  auto column = [&](int w) { return rows + (size_t)(w >> 1) * 2 * nr + (w & 1); };
  auto factor = [&](const double* f, int w) { return f + (size_t)lo * ps + kx + (size_t)(w >> 1) * Nxh; };
  // ---- forward elimination: this CTA's lane maps
  double none = 1.0;
  if (P > 1) {
    for (int w = t; w < 2 * Nz; w += bd) {
      double Am = 1.0;
      fz[w] = tri_forward<4, false, false>(column(w), 2, factor(I.tri_inv, w), factor(I.tri_m, w), ps, 0, nr, 0.0, Am);
      fA[w] = Am;
    }
  }
  cl.sync();
  if (P > 1) {
    // one thread per (column, lane p): the inclusive scan of k_tri_scan
    for (int base = 0; base < 2 * Nz * P; base += bd) {
      const int w = (base + t) / P, p = (base + t) % P;
      const bool ok = w < 2 * Nz;
      const double A0 = ok ? cl.map_shared_rank(fA, p)[w] : 1.0, z = ok ? cl.map_shared_rank(fz, p)[w] : 0.0;
      const double y = tri_lane_scan<true>(A0, z, p, P);
      if (ok && p == r) in[w] = y;
    }
  }
  __syncthreads();
  for (int w = t; w < 2 * Nz; w += bd)
    tri_forward<4, false, true>(column(w), 2, factor(I.tri_inv, w), factor(I.tri_m, w), ps, 0, nr, P > 1 ? in[w] : 0.0, none);
  // ---- back substitution from the top (each thread on its own columns)
  if (P > 1) {
    for (int w = t; w < 2 * Nz; w += bd) {
      double Am = 1.0;
      bw[w] = tri_backward<4, false, false>(column(w), 2, nullptr, 0, factor(I.tri_c, w), ps, 0, nr, 0.0, Am);
      bA[w] = Am;
    }
  }
  cl.sync();
  if (P > 1) {
    for (int base = 0; base < 2 * Nz * P; base += bd) {
      const int w = (base + t) / P, p = (base + t) % P;
      const bool ok = w < 2 * Nz;
      const double A0 = ok ? cl.map_shared_rank(bA, p)[w] : 1.0, z = ok ? cl.map_shared_rank(bw, p)[w] : 0.0;
      const double x = tri_lane_scan<false>(A0, z, p, P);
      if (ok && p == r) in[w] = x;
    }
  }
  __syncthreads();
  for (int w = t; w < 2 * Nz; w += bd)
    tri_backward<4, false, true>(column(w), 2, column(w), 2, factor(I.tri_c, w), ps, 0, nr, P > 1 ? in[w] : 0.0, none);
  __syncthreads();
  line_max(res, nr, nr, Nz, top);
  if (nr > 0)
    fx_fft<true>(RawLd{r0, 1, nr, LineIn{bits, top}}, RowSt{spec + (size_t)lo * ps, ps, (size_t)Nxh, LineOut{bits, halvings, top}},
                 r0, L * Nz - r0, nr, 1, nr, Nz, I.passz, T);
  cl.sync();   // no CTA leaves while another may still read its lane values
}

// ------------------------------------------------------------ inverse x -> pressure field
// the packed line of two real rows from their half-spectra pa, pb (stored at
// kx and Nxh + kx): element kx is pa + i pb, element Nx - kx conj(pa) + i
// conj(pb).  At kx = 0 and Nx/2 both are real; the rounding that the z passes
// leave in their imaginary parts would go into the other row.
struct PackLd {
  int pitch, Nx; LineIn in;
  __device__ __forceinline__ fx2 operator()(int r, int e) const {
    const bool lo = e <= Nx / 2;
    const double2* q = smem_d2() + r * pitch + (lo ? e : Nx - e);
    const int s = in.exponent(r);
    fx2 a = fx2_from(q[0], s), b = fx2_from(q[Nx / 2 + 1], s);
    if (e == 0 || 2 * e == Nx) a.y = b.y = 0;
    return lo ? make_longlong2(a.x - b.y, a.y + b.x) : make_longlong2(a.x + b.y, b.x - a.y);
  }
};
// the two real rows (planes k0, k0 + 1) of a packed line
struct RealSt {
  const ChlInst* I; double* p; int g0; LineOut out;
  __device__ __forceinline__ void operator()(int r, int i, fx2 v) const {
    const unsigned g = g0 + r, h = I->Nz / 2;
    const int jc = 1 + (int)(g / h), k0 = 2 * (int)(g % h);
    const double2 z = out(r, v);
    p[cidx(*I, i, jc, k0)] = z.x;
    p[cidx(*I, i, jc, k0 + 1)] = z.y;
  }
};

__global__ void __launch_bounds__(256)
k_fftx_inv(ChlMap map, int dst, int xmb) {
  chl_pdl_wait();
  extern __shared__ double2 sm[];
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz, Nxh = I.Nxh;
  const int nrow = Ny * (Nz / 2);
  const int CR = chl_fftx_rows(Nx, nrow, xmb);
  const int g0 = lb * CR;
  const int cr_n = min(CR, nrow - g0);
  const int A = 0, B = CR * (Nx + 2), T = B + CR * Nx;       // tiles, twiddles
  unsigned* hi = reinterpret_cast<unsigned*>(sm + T + I.lenx);
  stage_twiddles(smem_tw() + T, I.twx, I.lenx);
  for (int r = threadIdx.x; r < CR; r += blockDim.x) hi[r] = 0u;
  __syncthreads();
  const SmallDiv byNxh(Nxh);
  for (int w0 = 0; w0 < cr_n * Nxh; w0 += blockDim.x) {
    const int w = min(w0 + (int)threadIdx.x, cr_n * Nxh - 1);
    const int cr = byNxh.div(w), kx = w - cr * Nxh;
    const unsigned g = g0 + cr;
    const int jz = (int)(g / (unsigned)(Nz / 2)), jc = 1 + jz, k0 = 2 * ((int)g - jz * (Nz / 2));
    const double2 pa = I.spec[((size_t)jc * Nz + k0) * Nxh + kx];
    const double2 pb = I.spec[((size_t)jc * Nz + k0 + 1) * Nxh + kx];
    sm[cr * (Nx + 2) + kx] = pa;
    sm[cr * (Nx + 2) + Nxh + kx] = pb;
    fold_line(hi, cr, max(abshi2(pa), abshi2(pb)));
  }
  const int bits = I.bitsx - 1;      // an element is a sum of two components
  const RealSt last{&I, dst == 0 ? I.p : I.P, g0, LineOut{bits, I.passx - 1, hi}};
  fx_fft<true>(PackLd{Nx + 2, Nx, LineIn{bits, hi}}, last, A, B, cr_n, Nx, 1, Nx, I.passx, T);
}

// ------------------------------------------------------------ velocity correction
// project_velocity (projection.f90:192-214) + Dirichlet ghost rows; folds
// the largest velocities of the set and its rows (cleared by k_div_fftx).
// The FP64 pipe bounds it (6 instructions per point, 71 % busy), so two of a
// pair's six differences are formed on the integer pipe: 60 -> 55 us at
// 256x96x192 (one, two, three, four, six of them 57, 55, 55, 61, 64 us; HBM floor
// 39), 61 since it folds the rows' largest too.
__global__ void __launch_bounds__(256)
k_project(ChlMap map, int s) {
  chl_pdl_wait();
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const unsigned t = (unsigned)lb * blockDim.x + threadIdx.x;
  unsigned hi[3] = {0u, 0u, 0u};
  const ChlIdx ix = chl_split(t, Nx / 2, Ny);
  if (t < (unsigned)(Nx / 2 * Ny * Nz)) {     // pairs of points
    const int i = 2 * ix.i, jc = 1 + ix.j, k = ix.k;
    const bool hasv = jc <= Ny - 1;
    auto at = [](const double* f, size_t c) { return *reinterpret_cast<const double2*>(f + c); };
    auto put = [](double* f, size_t c, double2 v) { *reinterpret_cast<double2*>(f + c) = v; };
    auto top = [](double2 v) { return max(chl_abshi(v.x), chl_abshi(v.y)); };
    auto neg = [](double2 v) { return make_double2(chl_neg(v.x), chl_neg(v.y)); };
    const double* p = I.p;
    double* U = I.U[s]; double* V = I.V[s]; double* W = I.W[s];
    const size_t c = cidx(I, i, jc, k), e = vidx(I, i, jc, k);
    const double2 p0 = at(p, c), pz = at(p, cidx(I, i, jc, wrap(k + 1, Nz)));
    const double2 py = hasv ? at(p, cidx(I, i, jc + 1, k)) : p0;
    const double px = LDG(p + cidx(I, wrap(i + 2, Nx), jc, k));
    const double2 u = at(U, c), w = at(W, c), v = at(V, e);
    const double rx0 = LDG(I.rdxf + i), rx1 = LDG(I.rdxf + i + 1), ry = LDG(I.rdyf + jc), rz = LDG(I.rdzf + k);
    const double2 un = make_double2(u.x - fx_sub(p0.y, p0.x) * rx0, u.y - fx_sub(px, p0.y) * rx1);
    const double2 wn = make_double2(w.x - (pz.x - p0.x) * rz, w.y - (pz.y - p0.y) * rz);
    put(U, c, un); put(W, c, wn);
    hi[0] = top(un); hi[2] = top(wn);
    if (hasv) {
      const double2 vn = make_double2(v.x - (py.x - p0.x) * ry, v.y - (py.y - p0.y) * ry);
      put(V, e, vn);
      hi[1] = top(vn);
    }
    if (jc == 1) { put(U, cidx(I, i, 0, k), neg(un)); put(W, cidx(I, i, 0, k), neg(wn)); }
    if (jc == Ny) { put(U, cidx(I, i, Ny + 1, k), neg(un)); put(W, cidx(I, i, Ny + 1, k), neg(wn)); }
  }
  chl_set_max(I, s, (unsigned)(ix.k * Ny + ix.j), 1 + ix.j, hi);
}

// ------------------------------------------------------------ actual pressure: wall BC planes
// compute_pressure_BC (pressure.f90:269-340): bc = d/dy(nu dV/dy) at both walls.
__global__ void k_pbc(ChlMap map, int s) {
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  long t = (long)lb * blockDim.x + threadIdx.x;
  if (t >= 2L * Nx * Nz) return;
  const int i = (int)(t % Nx), k = (int)((t / Nx) % Nz), wall = (int)(t / ((long)Nx * Nz));
  const double* V = I.V[s];
  const double* nt = I.nut;      // nu + nu_t
  double bcv;
  if (wall == 0) {
    const double g = I.gb1, g2 = I.gb2;
    const double nui = 0.5 * (nt[cidx(I, i, 0, k)] + nt[cidx(I, i, 1, k)]);
    const double dnu = (nt[cidx(I, i, 1, k)] - nt[cidx(I, i, 0, k)]) / I.dygb;
    const double v1 = V[vidx(I, i, 0, k)], v2 = V[vidx(I, i, 1, k)], v3 = V[vidx(I, i, 2, k)], v4 = V[vidx(I, i, 3, k)];
    const double dV = (-3.0 * v1 + 4.0 * v2 - v3) / 2.0 * (1.0 / g);
    double ddV = 2.0 * v1 - 5.0 * v2 + 4.0 * v3 - 1.0 * v4;
    ddV = (ddV - dV * g2) / (g * g);
    bcv = dnu * dV + nui * ddV;
  } else {
    const double g = I.gt1, g2 = I.gt2;
    const double nui = 0.5 * (nt[cidx(I, i, Ny + 1, k)] + nt[cidx(I, i, Ny, k)]);
    const double dnu = (nt[cidx(I, i, Ny + 1, k)] - nt[cidx(I, i, Ny, k)]) / I.dygt;
    const double v1 = V[vidx(I, i, Ny, k)], v2 = V[vidx(I, i, Ny - 1, k)], v3 = V[vidx(I, i, Ny - 2, k)], v4 = V[vidx(I, i, Ny - 3, k)];
    const double dV = (3.0 * v1 - 4.0 * v2 + v3) / 2.0 * (1.0 / g);
    double ddV = 2.0 * v1 - 5.0 * v2 + 4.0 * v3 - 1.0 * v4;
    ddV = (ddV - dV * g2) / (g * g);
    bcv = dnu * dV + nui * ddV;
  }
  I.bc[t] = bcv;
}

// P ghost rows (pressure.f90:158-159)
__global__ void k_pghost(ChlMap map) {
  int lb;
  const ChlInst& I = map.inst[chl_find(map, blockIdx.x, lb)];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  long t = (long)lb * blockDim.x + threadIdx.x;
  if (t >= (long)Nx * Nz) return;
  const int i = (int)(t % Nx), k = (int)(t / Nx);
  double* P = I.P;
  P[cidx(I, i, 0, k)] = P[cidx(I, i, 1, k)] - I.dygb * I.bc[t];
  P[cidx(I, i, Ny + 1, k)] = P[cidx(I, i, Ny, k)] + I.dygt * I.bc[(size_t)Nx * Nz + t];
}

extern "C" {
// two ping-pong tiles (an x line's raw half-spectra take Nx + 2 elements), the
// twiddles (twz: the longest z table of the launch's instances) and, for the
// x lines, their largest components
size_t chl_smem_fftx(int Nx, int nrow, int xmb) {
  const size_t rows = chl_fftx_rows(Nx, nrow, xmb);
  return rows * (2 * (size_t)Nx + 2) * sizeof(double2) + (size_t)chl_twf_len(Nx) * sizeof(int4) + rows * sizeof(unsigned);
}
size_t chl_smem_fftz(int maxNz, int zcw, int twz) {
  return (size_t)2 * zcw * maxNz * sizeof(double2) + (size_t)twz * sizeof(int4);
}
// kx columns staged per z-transform block: 8 (at 256x96x192 two, four, eight
// and sixteen columns take 48, 48, 46 and 57 us per launch), halved while two
// Nz x cols complex tiles would exceed the 227 KB a block may use, and halved (down
// to 2) while the grid over all `ncols` columns would have fewer than
// min_blocks blocks (CHL_FFT_MIN_BLOCKS, about four per SM, unless the
// tuner chose another)
int chl_fftz_cols(int maxNz, long ncols, int min_blocks, int twz) {
  int c = 8;
  while (c > 1 && chl_smem_fftz(maxNz, c, twz) > (size_t)227 * 1024) c /= 2;
  while (c > 2 && (ncols + c - 1) / c < min_blocks) c /= 2;
  return c;
}
int chl_fft_setup(size_t smx, size_t smz, size_t smt) {
  cudaError_t e1 = cudaFuncSetAttribute(k_div_fftx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smx);
  cudaError_t e2 = cudaFuncSetAttribute(k_fftx_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smx);
  cudaError_t e3 = cudaFuncSetAttribute(k_fftz<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smz);
  if (e3 == cudaSuccess) e3 = cudaFuncSetAttribute(k_fftz<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smz);
  cudaError_t e4 = smt ? cudaFuncSetAttribute(k_tri_staged, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smt)
                       : cudaSuccess;
  return (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess || e4 != cudaSuccess) ? 1 : 0;
}
void chl_launch_div_fftx(const ChlMap& m, int nb, int nt, size_t smem, int s_in, int mode, int xmb, cudaStream_t st) { chl_launch_pdl(k_div_fftx, dim3(nb), dim3(nt), smem, st, m, s_in, mode, xmb); }
void chl_launch_fftz(const ChlMap& m, int nb, int nt, size_t smem, int inv, int zcw, cudaStream_t st) { 
  if (inv) chl_launch_pdl(k_fftz<true>, dim3(nb), dim3(nt), smem, st, m, zcw);
  else chl_launch_pdl(k_fftz<false>, dim3(nb), dim3(nt), smem, st, m, zcw);
}
// smem > 0: the staged form with TRI_W-mode blocks (chl_tri_modes_per_block)
void chl_launch_tri(const ChlMap& m, int nb, size_t smem, cudaStream_t st) {
  if (smem) chl_launch_pdl(k_tri_staged, dim3(nb), dim3(2 * TRI_W), smem, st, m);
  else chl_launch_pdl(k_tri, dim3(nb), dim3(128), 0, st, m);
}
// Shared memory of the staged form for the tallest column (40 bytes per
// row and mode), or 0 for the row-batched form.  mode 0: row-batched;
// 1: staged whenever it fits; 2 (default): staged only while all `modes`
// fit in one wave of resident blocks - the staged form has one warp per
// block, and beyond one wave the row-batched form keeps more warps per SM.
size_t chl_smem_tri(int maxNy, long modes, int mode) {
  const size_t b = (size_t)maxNy * TRI_W * (sizeof(double2) + 3 * sizeof(double));
  if (mode == 0 || b > (size_t)CHL_TRI_SMEM_MAX) return 0;
  if (mode == 1) return b;
  const long per_sm = (long)((228 * 1024) / (b + 1024));   // + the 1 KB the runtime reserves per block
  const long blocks = (modes + TRI_W - 1) / TRI_W;
  return blocks <= per_sm * CHL_SMS ? b : 0;
}
int chl_tri_modes_per_block(size_t smem) { return smem ? TRI_W : 64; }
// Fused z solve: shared memory of a CTA for an instance (0 if its block does
// not fit, or its lane count is not a cluster size of 1, 2, 4 or 8), and its
// launch: cluster (P, 1, 1), Nxh x P CTAs per instance.
size_t chl_smem_zsolve(int Nx, int Ny, int Nz) {
  const int Nxh = Nx / 2 + 1;
  const int P = chl_tri_lanes((long)Nz * Nxh, Ny);
  if (P != 1 && P != 2 && P != 4 && P != 8) return 0;
  const int L = (Ny + P - 1) / P;
  const size_t b = (size_t)2 * L * Nz * sizeof(double2) + (size_t)chl_twf_len(Nz) * sizeof(int4) +
                   (size_t)10 * Nz * sizeof(double) + (size_t)L * sizeof(unsigned);
  return b <= (size_t)227 * 1024 ? b : 0;
}
int chl_zsolve_setup(size_t smem) {
  return cudaFuncSetAttribute(k_zsolve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess ? 0 : 1;
}
void chl_launch_zsolve(const ChlMap& m, int nb, int P, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nb); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = P; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, k_zsolve, m);
}
void chl_launch_tri_scan(const ChlMap& m, int nb, cudaStream_t st) { chl_launch_pdl(k_tri_scan, dim3(nb), dim3(128), 0, st, m); }
void chl_launch_fftx_inv(const ChlMap& m, int nb, int nt, size_t smem, int dst, int xmb, cudaStream_t st) { chl_launch_pdl(k_fftx_inv, dim3(nb), dim3(nt), smem, st, m, dst, xmb); }
void chl_launch_project(const ChlMap& m, int nb, int s, cudaStream_t st) { chl_launch_pdl(k_project, dim3(nb), dim3(m.tb), 0, st, m, s); }
void chl_launch_pbc(const ChlMap& m, int nb, int s, cudaStream_t st) { k_pbc<<<nb, 256, 0, st>>>(m, s); }
void chl_launch_pghost(const ChlMap& m, int nb, cudaStream_t st) { k_pghost<<<nb, 256, 0, st>>>(m); }
}
