// hartree_resident.cuh -- the one-launch mixed Hartree CG of grids that fit the
// SMs (hartree_resident.cu) as density.cu's solver calls it.
#pragma once
#include "stencil.cuh"

namespace rs {

constexpr int kResidentCtas = 148;

// device scratch of one solve (448 doubles; the caller checks that its array holds
// it): zeroed, then r1r = r.r of the first residual; iters, dp and err are read
// when the launch has finished
struct ResidentState {
  double r1r, dp;
  int iters, err;
  unsigned arrived, pad;
  double part[3][kResidentCtas];
};
static_assert(sizeof(ResidentState) == 448 * sizeof(double));

bool hartree_resident_ok(int nx, int ny, int nz, int nfh);
int launch_hartree_resident(int nx, int ny, int nz, const HartreeCoefs& hc, int ncgres, int ncgmin,
                            int ncgmax, double epsvh, double dv, double vol, const double* b,
                            double* vh, float* p, const float* r0, ResidentState* state,
                            cudaStream_t st);
bool hartree_resident64_ok(int nx, int ny, int nz, int nfh);
int launch_hartree_resident64(int nx, int ny, int nz, int nfh, const HartreeCoefs& hc, int ncgres,
                              int ncgmin, int ncgmax, double epsvh, double ddx, double ddy,
                              double ddz, double vol, const double* b, const double* avhs,
                              const double* r, double* vh, double* p, ResidentState* state,
                              cudaStream_t st);

}  // namespace rs
