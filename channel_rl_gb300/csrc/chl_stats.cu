// Statistics of compute_statistics (statistics.f90:22-145): plane means of
// U, V, W, their squares and UV per row, the wall shear, u_tau, Re_tau and
// the bulk flows (mass_flow.f90:24-98).  The reference's summation ranges
// are kept, including their duplicated periodic columns and planes:
//   U   : x faces 1..nx-2 (each unique face once), z centres 1..nzg-2 (plane nzg-2 twice)
//   W   : x centres 1..nxg-2 (centre nxg-2 twice), z faces 1..nz-2 (once each)
//   V,UV: x centres 2..nxg-1 and z centres 2..nzg-1 (centre 2 / plane 2 twice)
// The wall shear uses the bottom wall for both walls, as statistics.f90:108-116 does.
#include "chl_common.cuh"

#define NST 7
// sums of a row: the seven of the profiles, the plain sum of U (bulk flow) and,
// on row 0, the bottom wall's nu du/dy
#define NSUM 9
// parts of a row's x-z plane, each summed by one block: with one block per row
// a 108 x 54 plane left most SMs idle, and with one block per instance the
// bulk flows took 1.4 ms of a 45-row channel's sampling
#define STATS_PARTS 8

// block (row block, part): partial sums of Fortran row jj = r+1, r in [0, Ny]
__global__ void __launch_bounds__(256)
k_stats_rows(ChlMap map, int s, double* part) {
  int lb;
  const int q = chl_find(map, blockIdx.x, lb);
  const ChlInst& I = map.inst[q];
  const int Nx = I.Nx, Nz = I.Nz;
  const int r = lb;
  const double *U = I.U[s], *V = I.V[s], *W = I.W[s], *nt = I.nut;
  const double w0 = 0.5 * I.w0x2[r], w1 = 0.5 * I.w1x2[r];   // exact halvings
  const int n = Nx * Nz, chunk = (n + STATS_PARTS - 1) / STATS_PARTS;
  const int end = min(n, ((int)blockIdx.y + 1) * chunk);
  double acc[NSUM] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int w = blockIdx.y * chunk + threadIdx.x; w < end; w += blockDim.x) {
    const int k = (int)((unsigned)w / (unsigned)Nx), i = w - k * Nx;
    const double u = U[cidx(I, i, r, k)], up = U[cidx(I, i, r + 1, k)];
    const double wu = k == Nz - 1 ? 2.0 : 1.0;
    const double ww_ = W[cidx(I, i, r, k)];
    const double wwt = i == Nx - 1 ? 2.0 : 1.0;
    const double v = V[vidx(I, i, r, k)];
    const double wv = (i == 0 ? 2.0 : 1.0) * (k == 0 ? 2.0 : 1.0);
    const int im = wrap(i - 1, Nx);
    const double uyl = w0 * U[cidx(I, im, r, k)] + w1 * U[cidx(I, im, r + 1, k)];
    const double uyh = w0 * u + w1 * up;
    const double uc = 0.5 * (uyl + uyh);
    acc[0] += wu * u;  acc[1] += wv * v;  acc[2] += wwt * ww_;
    acc[3] += wu * u * u; acc[4] += wv * v * v; acc[5] += wwt * ww_ * ww_;
    acc[6] += wv * v * uc;
    acc[7] += u;
    if (r == 0) {
      const int ip = wrap(i + 1, Nx);
      const double ntf0 = 0.5 * (nt[cidx(I, i, 0, k)] + nt[cidx(I, ip, 0, k)]);
      const double ntf1 = 0.5 * (nt[cidx(I, i, 1, k)] + nt[cidx(I, ip, 1, k)]);
      const double ntw = w0 * ntf0 + w1 * ntf1;      // nu + nu_t at the wall (weights sum to 1)
      acc[8] += (up - u) / I.dyw * ntw;
    }
  }
  __shared__ double red[NSUM][256];
#pragma unroll
  for (int m = 0; m < NSUM; ++m) red[m][threadIdx.x] = acc[m];
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h)
#pragma unroll
      for (int m = 0; m < NSUM; ++m) red[m][threadIdx.x] += red[m][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x < NSUM) part[((size_t)blockIdx.x * STATS_PARTS + blockIdx.y) * NSUM + threadIdx.x] = red[threadIdx.x][0];
}

// one block per instance: the profiles, then tau (bottom wall), Qflow_x and
// Qflow_y, whose trapezoids over y are sums of the rows' plane sums
__global__ void __launch_bounds__(256)
k_stats_final(ChlMap map, const double* part, double* out, int pitch) {
  const int q = blockIdx.x;
  const ChlInst& I = map.inst[q];
  const int Nx = I.Nx, Ny = I.Ny, Nz = I.Nz;
  const double* P = part + (size_t)map.off[q] * STATS_PARTS * NSUM;
  double* o = out + (size_t)q * pitch;
  auto sum = [&](int r, int m) {
    double v = 0.0;
    for (int c = 0; c < STATS_PARTS; ++c) v += P[((size_t)r * STATS_PARTS + c) * NSUM + m];
    return v;
  };
  const double cu = (double)Nx * (Nz + 1), cv = (double)(Nx + 1) * (Nz + 1), cw = (double)(Nx + 1) * Nz;
  const double norm[NST] = {cu, cv, cw, cu, cv, cw, cv};
  for (int w = threadIdx.x; w < NST * (Ny + 1); w += blockDim.x) {
    const int m = w / (Ny + 1), r = w - m * (Ny + 1);
    o[w] = sum(r, m) / norm[m];
  }
  // U rows jc - 1, jc for jc = 2..Ny (yg spacing), V rows jv - 1, jv for jv = 1..Ny (y spacing)
  double qx = 0.0, nx_ = 0.0, qy = 0.0, ny_ = 0.0;
  for (int j = 1 + threadIdx.x; j <= Ny; j += blockDim.x) {
    const double dy = 1.0 / I.rdyc[j];               // y(j)-y(j-1), j_f = j+1
    qy += (sum(j, 1) + sum(j - 1, 1)) * 0.5 * dy;
    ny_ += dy;
    if (j >= 2) {
      const double dyg = I.dyf[j - 1];
      qx += (sum(j, 7) + sum(j - 1, 7)) * 0.5 * dyg;
      nx_ += dyg;
    }
  }
  __shared__ double red[4][256];
  red[0][threadIdx.x] = qx; red[1][threadIdx.x] = nx_; red[2][threadIdx.x] = qy; red[3][threadIdx.x] = ny_;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h)
      for (int m = 0; m < 4; ++m) red[m][threadIdx.x] += red[m][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double* t = o + (size_t)NST * (Ny + 1);
    t[0] = sum(0, 8) / ((double)Nx * Nz);
    t[1] = red[0][0] / (red[1][0] * ((double)Nx * Nz));
    t[2] = red[2][0] / (red[3][0] * cv);
  }
}

extern "C" {
size_t chl_stats_parts() { return STATS_PARTS * NSUM; }   // doubles per row block
void chl_launch_stats(const ChlMap& rows, int nrows_blocks, double* part, double* out, int pitch, int s,
                      cudaStream_t st) {
  k_stats_rows<<<dim3(nrows_blocks, STATS_PARTS), 256, 0, st>>>(rows, s, part);
  k_stats_final<<<rows.n, 256, 0, st>>>(rows, part, out, pitch);
}
}
