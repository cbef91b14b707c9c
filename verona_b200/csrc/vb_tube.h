// Every step of a call on a short ghosted 1D FP64 grid in one launch (vb_tube.cu).
#pragma once
#include "vb_internal.h"

namespace vb {

struct TubeRun {
    double* P[2];
    double *U0, *U1;
    int cur, rk, nsteps;       // P[cur]: the state at the start
    double t0, dt;
    double dtdx, half_dtdx;    // dt / dx, (dt / 2) / dx
};
bool tube_fits(int cells);
// cudaErrorNotSupported where the GPU grants no cluster of the grid's tiles (nothing launched)
cudaError_t launch_tube(int rec, int rs, const TubeRun& r, const int* bc_kind, const double (*bc_par)[16],
                        const StageParams& p, cudaStream_t s);

}  // namespace vb
