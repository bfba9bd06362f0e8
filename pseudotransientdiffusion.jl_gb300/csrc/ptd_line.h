// ptd_line.h -- host interface of the 1D kernel that holds whole steps (ptd_line.cu).
#pragma once

#include <cuda_runtime.h>

#include "ptd_kernels.h"

namespace ptd {

// A launch: `ctas` CTAs of `warps` warps, one cluster; windows of 32 c cells
// per warp of which `core` are written back after at most `tmax` iterations.
struct LinePlan {
    int c = 0, tmax = 0, core = 0, ctas = 0, warps = 0;
};

struct LineArgs {
    double* Hold;
    DevState* st;        // host-visible: the outcome of the launch (checks),
    HostSteps* out;      // its steps, and acc (sum R^2, or max |R|) of its first checks,
    double* errmore;     // device memory: of the others, each at its index
    int errcap, nchk, itmax, checks, niter;   // checks 0: niter iterations without checks
    int nsteps, itlimit; // steps at most, and none begun after that many iterations
    double tol, norm_den;
    double acc_above;    // an acc above it has err > tol
    int tmax, core, warps;
};

// False: the grid is too large for one cluster (or the device grants none).
bool line_plan(int model, int nx, int nchk, LinePlan& p);
cudaError_t launch_line(const PTArgs& a, const LineArgs& l, int model, const LinePlan& p, cudaStream_t s);

}  // namespace ptd
