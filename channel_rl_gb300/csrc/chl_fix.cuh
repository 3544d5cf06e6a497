// 64-bit fixed-point arithmetic on the integer pipe.
//
// GB300 issues one warp FP64 instruction per 64-67 clocks and SM
// sub-partition, whatever it is; in the same time the integer pipe issues
// 13 64-bit additions, 4 of the products below or 2.7 conversions (measured
// clocks per warp instruction: 5, 16, 24), and the two pipes run side by
// side.  Sums and products of quantities whose largest magnitude is known
// are therefore formed here in 64-bit integers F standing for F 2^e, e the
// exponent of the quantity's last bit, and only the result goes back to
// double.  A field is scaled by its own largest magnitude (kept with the
// velocity set, ChlInst::status), so that |F| < 2^61: eight bits finer than
// a double's last bit at that magnitude, and exact for every double down to
// 2^-8 of it (k_flux, whose rows differ by more, scales every row by its own).
// Sums and differences are exact; a product keeps 60 bits or more of its largest
// possible value.
#pragma once
#include "chl_common.cuh"

typedef long long fx;

// exponent of the last bit for a quantity whose largest |x| has the high
// word `hi` (bits of the double >> 32, sign cleared), such that |F| < 2^BITS;
// magnitudes below 2^-958 are scaled as that (they round to zero)
template <int BITS>
__device__ __forceinline__ int fx_exp(unsigned hi) {
  const int E = max((int)(hi >> 20), 64);
  return E - 1022 - BITS;
}
__device__ __forceinline__ int fx_line_exp(unsigned hi, int bits) { return max((int)(hi >> 20), 64) - 1022 - bits; }
__device__ __forceinline__ bool fx_bad(unsigned hi) { return hi >= 0x7FF00000u; }

// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// x as F 2^e, rounded toward zero
__device__ __forceinline__ fx fx_from(double x, int e) {
  const long long b = __double_as_longlong(x);
  const int r = e + 1086 - (((int)(b >> 52)) & 0x7FF);
  unsigned long long f;
  // shr clamps shift amounts above 63, which give 0 (also for x = 0)
  asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(((unsigned long long)b << 11) | 0x8000000000000000ULL), "r"(r));
  return b < 0 ? -(fx)f : (fx)f;
}

// The same for |x| < 2^(61+e) on the FP64 pipe (one conversion; the scaling is an
// addition to the exponent, clamped at zero so that zeros and tiny x stay below one
// unit), for kernels that leave it idle.
struct FxConv {
  int d;
  __device__ __forceinline__ explicit FxConv(int e) : d(-e * (1 << 20)) {}
  __device__ __forceinline__ fx operator()(double x) const {
    const int h = __double2hiint(x), a = max((int)((unsigned)(h & 0x7FFFFFFF) + (unsigned)d), 0);
    return __double2ll_rz(__hiloint2double(a | (h & (int)0x80000000), __double2loint(x)));
  }
};

// F 2^e as a double, rounded to nearest; exponents beyond a double's give its
// smallest and largest magnitudes.  EXACT = false takes the magnitude of a
// negative F one unit short, which saves the carry, for values whose last bits
// are rounding anyway and whose sums are not taken (it is a mean error).
template <bool EXACT = false>
__device__ __forceinline__ double fx_to(fx f, int e) {
  const int sign = (int)(f >> 63);
  if (EXACT) f -= (fx)((unsigned)sign & 1u);
  const unsigned hi = (unsigned)(f >> 32) ^ (unsigned)sign, lo = (unsigned)f ^ (unsigned)sign;
  const int lz = hi ? __clz((int)hi) : 32 + __clz((int)lo);
  unsigned long long n;
  asm("shl.b64 %0, %1, %2;" : "=l"(n) : "l"(((unsigned long long)hi << 32) | lo), "r"(lz));
  const int ef = min(max(e + 1085 - lz, 0), 2045);
  unsigned long long r = (n >> 11) + ((n >> 10) & 1ULL) + ((unsigned long long)(unsigned)ef << 52);
  unsigned rh = (unsigned)(r >> 32);
  if (lz == 64) rh = 0u;
  return __hiloint2double((int)(rh | ((unsigned)sign & 0x80000000u)), (int)(unsigned)r);
}
// a - b on the integer pipe: exact like the FP64 subtraction where that is
// (magnitudes within 2^8 of each other keep all their bits), else within 2^-61
// of the larger, 2^-1019 at least, before its one rounding; zeros of either sign
// are zero; NaN if a or b is not finite.
__device__ __forceinline__ double fx_sub(double a, double b) {
  const int m = max(max(__double2hiint(a) >> 20 & 0x7FF, __double2hiint(b) >> 20 & 0x7FF), 64);
  const double d = fx_to<true>(fx_from(a, m - 1084) - fx_from(b, m - 1084), m - 1084);
  return m == 0x7FF ? __longlong_as_double(0x7FF8000000000000LL) : d;
}
// F as a double, on the FP64 pipe (64 clocks, no other) or the integer pipe
template <bool HW>
__device__ __forceinline__ double fx_raw(fx f) { return HW ? __ll2double_rn(f) : fx_to(f, 0); }
// x 2^e for a normal x and result (an addition to the exponent)
__device__ __forceinline__ double scale_exp(double x, int e) {
  return __hiloint2double(__double2hiint(x) + (e << 20), __double2loint(x));
}


// (a b) >> 64, low by less than three units, for |a| < 2^62 and |b| < 2^63 (or
// |a| < 2^63 and 0 <= b < 2^63):
// the product of the high words plus the cross terms, whose low words enter
// with 31 bits so that they are signed 32-bit factors.
__device__ __forceinline__ fx fx_mul(fx a, fx b) {
  const int ah = (int)(a >> 32), bh = (int)(b >> 32);
  const int al = (int)((unsigned)a >> 1), bl = (int)((unsigned)b >> 1);
  const long long t = (long long)ah * bl + (long long)bh * al;
  return (long long)ah * bh + (t >> 31);
}

// (a b) >> S for 34 <= S <= 64, without a mean error where low words are random:
// half a unit for the last shift and a quarter of 2^(64-S) for the low words' product
// come back with the start of t.  For what sums over many points collect.
template <int S>
__device__ __forceinline__ fx fx_mul_mean(fx a, fx b) {
  const int ah = (int)(a >> 32), bh = (int)(b >> 32);
  const int al = (int)((unsigned)a >> 1), bl = (int)((unsigned)b >> 1);
  const long long t = (1LL << (S - 34)) + (1LL << 29) + (long long)ah * bl + (long long)bh * al;
  return (fx)((unsigned long long)((long long)ah * bh) << (64 - S)) + (t >> (S - 33));
}

// (a b) >> S for 34 <= S <= 64, |a b| < 2^(62+S): keeps 64 - S more bits of a
// product whose factors leave room for them.
template <int S>
__device__ __forceinline__ fx fx_mul_shr(fx a, fx b) {
  const int ah = (int)(a >> 32), bh = (int)(b >> 32);
  const int al = (int)((unsigned)a >> 1), bl = (int)((unsigned)b >> 1);
  const long long t = (long long)ah * bl + (long long)bh * al;
  return (fx)((unsigned long long)((long long)ah * bh) << (64 - S)) + (t >> (S - 33));
}

// High words of the largest |U|, |V|, |W| of a velocity set and of the largest
// |nu + nu_t| of every centre row.  Written with the fields by every kernel that
// leaves a velocity set behind (upload, projection, mass-flow shift) or nu + nu_t.
__device__ __forceinline__ unsigned* chl_vmax(const ChlInst& I, int set) {
  return reinterpret_cast<unsigned*>(I.status) + (set == 0 ? CHL_ST_VMAX0 : CHL_ST_VMAX12 + 3 * (set - 1));
}
// The same of every row of the set that was written last (U and W: centre rows
// 1..Ny, whose mirrors the ghost rows are; V: faces 0..Ny), of which only the
// exponent counts.  The writers fold them into one of CHL_ROW_COPIES words each,
// from which k_fix forms the rows' exponents: all warps reading and raising one
// word per row made k_project 55 -> 69 us at 256x96x192.
__device__ __forceinline__ unsigned* chl_row_words(const ChlInst& I, int comp, int row) {
  return reinterpret_cast<unsigned*>(I.status) + CHL_ST_ROWS + CHL_ROW_COPIES * (comp * (I.Ny + 2) + row);
}
__device__ __forceinline__ unsigned chl_row_max(const ChlInst& I, int comp, int row) {
  const uint4* p = reinterpret_cast<const uint4*>(chl_row_words(I, comp, row));
  const uint4 a = __ldcg(p), b = __ldcg(p + 1);
  return max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w)));
}
// raises *g to x where x has the larger exponent
__device__ __forceinline__ void chl_raise_exp(unsigned* g, unsigned x) {
  if ((x >> 20) > (__ldcg(g) >> 20)) atomicMax(g, x);
}
__device__ __forceinline__ unsigned chl_abshi(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

#define CHL_BLOCK_LINES 130
// Folds each thread's v into g[off + j], j = q mod rows the row of its x-line
// q = k rows + j (whole block, at most 256 threads; x-lines are numbered
// upwards through the block and hold two threads or more).
__device__ __forceinline__ void chl_line_max(unsigned* g, unsigned q, int rows, int off, unsigned v) {
  __shared__ unsigned sm[CHL_BLOCK_LINES];
  __shared__ unsigned q0;
  for (unsigned l = threadIdx.x; l < CHL_BLOCK_LINES; l += blockDim.x) sm[l] = 0u;
  if (threadIdx.x == 0) q0 = q;
  __syncthreads();
  const unsigned l = min(q - q0, (unsigned)CHL_BLOCK_LINES - 1u);
  if (__all_sync(0xffffffffu, l == __shfl_sync(0xffffffffu, l, 0))) {
    v = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) atomicMax(sm + l, v);
  } else {
    atomicMax(sm + l, v);
  }
  __syncthreads();
  for (unsigned w = threadIdx.x; w < CHL_BLOCK_LINES; w += blockDim.x) {
    unsigned* d = g + off + (q0 + w) % (unsigned)rows;
    if (sm[w] && sm[w] > __ldcg(d)) atomicMax(d, sm[w]);
  }
}

// Folds the magnitudes of each thread's U, V, W (of U alone with N = 1) in row j
// into the set's largest and the row's (whole block, at most 256 threads; x-line
// q = k Ny + j - 1, numbered upwards through the block, of Nx/2 threads).  The
// global words are read first: only blocks that raise one issue an atomic, or the
// tens of thousands of same-address atomics would take longer than the kernels.
template <int N>
__device__ __forceinline__ void chl_set_max(const ChlInst& I, int set, unsigned q, int j, const unsigned (&v)[N]) {
  __shared__ unsigned sm[N][CHL_BLOCK_LINES];
  __shared__ unsigned line[8], row[8], q0;
  const unsigned copy = blockIdx.x % CHL_ROW_COPIES;
  if (I.Nx % 64 == 0) {       // every warp is in one x-line
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned mine = 0u;
#pragma unroll
    for (int c = 0; c < N; ++c) {
      const unsigned x = __reduce_max_sync(0xffffffffu, v[c]);
      if (lane == c) mine = x;
    }
    if (lane < N) sm[lane][warp] = mine;
    if (lane == 0) { line[warp] = q; row[warp] = j; }
    __syncthreads();
    if (threadIdx.x >= 8 * N) return;
    // thread (c, w): the warps from w on that share its x-line; w = 7 all of them
    const unsigned c = threadIdx.x >> 3, w = threadIdx.x & 7;
    if (w < nw && (w == 0 || line[w - 1] != line[w])) {
      unsigned x = sm[c][w];
      for (unsigned k = w + 1; k < nw && line[k] == line[w]; ++k) x = max(x, sm[c][k]);
      chl_raise_exp(chl_row_words(I, c, row[w]) + copy, x);
    }
    if (w == 7) {
      unsigned x = sm[c][0];
      for (unsigned k = 1; k < nw; ++k) x = max(x, sm[c][k]);
      unsigned* all = chl_vmax(I, set) + c;
      if (x > __ldcg(all)) atomicMax(all, x);
    }
    return;
  }
  const unsigned nl = min((unsigned)CHL_BLOCK_LINES, blockDim.x / (unsigned)(I.Nx / 2) + 2u);   // lines of the block
  for (unsigned t = threadIdx.x; t < N * nl; t += blockDim.x) sm[t / nl][t % nl] = 0u;
  if (threadIdx.x == 0) q0 = q;
  __syncthreads();
  const unsigned l = q - q0;
#pragma unroll
  for (int c = 0; c < N; ++c) atomicMax(&sm[c][l], v[c]);
  __syncthreads();
  for (unsigned t = threadIdx.x; t < N * nl; t += blockDim.x) {
    const unsigned c = t / nl, w = t - c * nl, x = sm[c][w];
    if (x == 0u) continue;
    chl_raise_exp(chl_row_words(I, c, 1 + (q0 + w) % (unsigned)I.Ny) + copy, x);
    unsigned* all = chl_vmax(I, set) + c;
    if (x > __ldcg(all)) atomicMax(all, x);
  }
}

// One's-complement magnitudes of the high words, or-ed: the bit length of the
// result is that of the largest of them.
__device__ __forceinline__ void top_or(unsigned& m, fx a) {
  const int h = (int)(a >> 32);
  m |= (unsigned)(h ^ (h >> 31));
}
// a 2^s for s of either sign (toward minus infinity)
__device__ __forceinline__ fx scale2(fx a, int s) { return (a << max(s, 0)) >> max(-s, 0); }
// its high word, for s <= 31
__device__ __forceinline__ int scale2_hi(fx a, int s) {
  const int h = __funnelshift_l((unsigned)a, (unsigned)(a >> 32), (unsigned)max(s, 0));
  return h >> min(31, max(-s, 0));
}
