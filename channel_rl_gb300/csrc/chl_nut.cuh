// nu + nu_t written by the kernel that forms nu_t (static Smagorinsky, AMD, Vreman).
#pragma once
#include "chl_fix.cuh"

// nu + nu_t for the interior centre (i, jc, k), v with the clipped nu_t, plus
// the ghost row next to the first and last interior rows from that nu_t
// (nu_t(), asked for there only).  With the wall model on, rows 0, 1 and Ny,
// Ny+1 are k_wall_rows's.  Returns the high word of the largest magnitude
// written; the ghost row's counts for the row next to it.
template <class NUT>
__device__ __forceinline__ unsigned write_nut_rows(const ChlInst& I, int i, int jc, int k, double v, const NUT& nu_t,
                                                   int use_wm) {
  const int Ny = I.Ny;
  const bool wallrow = jc == 1 || jc == Ny;
  if (wallrow && use_wm && I.wall_model != 0) return 0u;
  double* nt = I.nut;
  nt[cidx(I, i, jc, k)] = v;
  unsigned hi = chl_abshi(v);
  if (wallrow) {
    const double g = I.nu + nut_ghost(I, nu_t());
    if (jc == 1) nt[cidx(I, i, 0, k)] = g;
    if (jc == Ny) nt[cidx(I, i, Ny + 1, k)] = g;
    hi = max(hi, chl_abshi(g));
  }
  return hi;
}
