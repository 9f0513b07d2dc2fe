// column.h -- many steady-state steps of a 1 x 1 x NZ column in one launch.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace ehd {

// A column context's buffers (see ehd_ctx); parity: the buffer read first.
struct ColumnArgs {
    void *f[2], *h[2];
    double *wref[2], *mean[2];
    void *ktab[2];
    void *phip, *q, *rho, *u, *v, *w;
    double *phi00, *ez00;
    double dz, eps, voltage;
    int parity;
};

// whether the column kernel serves a grid
bool column_usable(int nx, int ny, int nz);
// sets its shared-memory attribute (prec: ehd_precision)
cudaError_t prepare_column(int prec);
// nsteps >= 1 steps; the state is then in buffer parity ^ (nsteps & 1)
cudaError_t launch_column_steps(int prec, const ColumnArgs &a, const StepConst &c, int nsteps,
                                cudaStream_t s);

}  // namespace ehd
