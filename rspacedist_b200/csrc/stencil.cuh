// stencil.cuh -- coefficient bundles and the per-point stencil evaluation
// shared by the stand-alone Laplacian and the fused H*psi kernels.
#pragma once
#include <algorithm>

#include "rs_common.cuh"

namespace rs {

template <class T>
struct StencilArgs {
  int nx, ny, nz, nf;
  T cx[9], cy[9], cz[9];
  T c0;  // cx[0] + cy[0] + cz[0], added left to right
};

struct HartreeCoefs {
  double cx[9], cy[9], cz[9];
  double diag;
};

struct GradCoefs {
  double a[9];
};

// i in (-n, 2n) wrapped into [0, n) (stencil offsets are below the grid size:
// rs_geom_create requires 2 nf < n on every axis)
__device__ __forceinline__ int wrap_near(int i, int n) {
  return i < 0 ? i + n : (i >= n ? i - n : i);
}

// acc + (-1/2 lap + veff) psi at (ix,iy,iz): x terms with the diagonal, then
// y, then z, one fma each (kslaplacian8f.F90:207-261).
template <class T>
__device__ __forceinline__ T stencil_point(const StencilArgs<T>& s, const T* __restrict__ v,
                                           int ix, int iy, int iz, T vloc, T acc) {
  const int nx = s.nx, ny = s.ny, nz = s.nz;
  const long plane = (long)nx * ny;
  const T* row = v + (long)iz * plane + (long)iy * nx;  // (iy, iz) row
  const T* col = v + (long)iy * nx + ix;                  // (ix, iy) column, z stride plane
  for (int m = s.nf; m >= 1; --m) acc = fma(s.cx[m], __ldg(row + wrap_near(ix - m, nx)), acc);
  const T diag = s.c0 + vloc;
  acc = fma(diag, __ldg(row + ix), acc);
  for (int m = 1; m <= s.nf; ++m) acc = fma(s.cx[m], __ldg(row + wrap_near(ix + m, nx)), acc);
  const T* pl = v + (long)iz * plane + ix;
  for (int m = s.nf; m >= 1; --m)
    acc = fma(s.cy[m], __ldg(pl + (long)wrap_near(iy - m, ny) * nx), acc);
  for (int m = 1; m <= s.nf; ++m)
    acc = fma(s.cy[m], __ldg(pl + (long)wrap_near(iy + m, ny) * nx), acc);
  for (int m = s.nf; m >= 1; --m)
    acc = fma(s.cz[m], __ldg(col + (long)wrap_near(iz - m, nz) * plane), acc);
  for (int m = 1; m <= s.nf; ++m)
    acc = fma(s.cz[m], __ldg(col + (long)wrap_near(iz + m, nz) * plane), acc);
  return acc;
}

// z run of a plane-marching stencil whose launch has ncol (tile, band)
// columns of nz planes and room for `slots` CTAs at once: the run that makes
// waves * (run + 8) smallest, 8 being the halo planes each run reads before its
// first output.  Few columns are so cut into enough runs to fill the SMs and
// two columns more than a wave do not cost a second full one; many columns keep
// whole runs (at most 160 planes, 64 of longer axes).  Results do not depend on
// the run.  Measured on one B200, H psi with whole runs and with
// these: FP32 Si8, 20 bands 41.0 and 27.4 us; Si64, 20 bands 64 and 33 us, 160 bands 202
// and 186 us; FP64 Si8, 1 band 41 and 24 us, 20 bands 50 and 35 us.
inline int stencil_zrun(long ncol, int nz, long slots) {
  const int most = nz <= 160 ? nz : 64;
  int best = most;
  long cost = -1;
  for (int n = (nz + most - 1) / most; n <= std::max(1, nz / 4); ++n) {
    const int run = (nz + n - 1) / n;
    const long c = ((ncol * ((nz + run - 1) / run) + slots - 1) / slots) * (run + 8);
    if (cost < 0 || c < cost) {
      cost = c;
      best = run;
    }
  }
  return best;
}

template <class T>
StencilArgs<T> make_stencil_args(const rs_geom* g);
GradCoefs grad_coefs(int nf, double h);
HartreeCoefs hartree_coefs(int nfh, double ddx, double ddy, double ddz);

template <class T>
int launch_kslaplacian(const rs_geom* g, const T* psi, const T* veff, T* out, int nb,
                       cudaStream_t st);
template <class T>
int launch_precondition(const rs_geom* g, const T* in, T* out, int nb, cudaStream_t st);
// r0 = h - lam s (DIIS; CG with cg: its negative, in double), lam of band b at
// lam[b * lstride], and out = ksprecondition(r0); either output may be null
template <class T>
int launch_resid_precond(const rs_geom* g, const T* h, const T* s, const double* lam, long lstride,
                         bool cg, T* r0, T* out, int nb, cudaStream_t st);
int launch_hartree_lap(int nx, int ny, int nz, int nfh, const HartreeCoefs& c, const double* v,
                       double* av, cudaStream_t st);
template <class T>
int launch_gradient(const rs_geom* g, int axis, const T* psi, T* out, int nb, cudaStream_t st);

}  // namespace rs
