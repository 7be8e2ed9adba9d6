// Interface of the on-chip sweep kernels (k_resident.cu).
#pragma once

#include "ib3d_internal.cuh"

namespace ib3d {

ResidentPlan plan_resident32(int nx, int ny, int nz, int nsm);
ResidentPlan plan_resident64(int nx, int ny, int nz, int nsm, bool exact);

// One launch of FP32 sweeps on A e = r from e = 0, ending with pc += e.
struct Resident32 {
  Dims d;
  const float4* axp[2][3];              // grouped x coefficients (Grid1D::axp)
  const float *ay[3], *az[3];           // 1-based by j-1, k-1 (Grid1D::acy32, acz32)
  const float* r[2];                    // right-hand side: entry 0 of row (j, k) = (2, 2) of each colour
  int rs, ps;                           // row and plane strides of r
  double* pc;
  unsigned long long* xch;              // exchange buffer (ResidentPlan::xch_words)
  unsigned seq0;                        // passes run before on this buffer
  int gy, gz, by, bz, zl;
  int nsweeps, nsmooth, nramp;          // sweeps at relaxation 1, then rising, then (om, om1)
  double wi;
  float om, om1;
  int* err;                             // set when a wait gave up
  int polls;                            // loads after which a wait gives up, checked every 256
  unsigned skew;                        // added to the numbers waited for: 0, or no wait ends
};
cudaError_t launch_resident32(const ResidentPlan& pl, Resident32 a, cudaStream_t st);

// One launch of FP64 sweeps on A pc = b/dt, from pc_in to pc_out (padded layout; pc_out's
// cells that are not fluid are left alone).
struct Resident64 {
  Dims d;
  const double *ax[3], *ay[3], *az[3];  // Poisson coefficients, 1-based by i-1, j-1, k-1
  const double* bdt;
  const double* pc_in;
  double* pc_out;
  const unsigned char* cell;
  unsigned long long* xch;
  unsigned seq0;
  int gy, gz, by, bz;
  int nsweeps, check;                   // check: sweeps between residuals, 0: update norm of every sweep
  long long sweep0;                     // sweeps of the solve before this launch
  double omega, om1;
  unsigned long long* errs;             // [nsweeps] largest update or residual (bit pattern)
  int* err;                             // as in Resident32
  int polls;
  unsigned skew;
};
cudaError_t launch_resident64(const ResidentPlan& pl, Resident64 a, bool exact, cudaStream_t st);

}  // namespace ib3d
