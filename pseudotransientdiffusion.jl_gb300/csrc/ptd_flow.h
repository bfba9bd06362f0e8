// ptd_flow.h -- host interface of the one-launch 2D step (ptd_flow.cuh).
#pragma once

#include <cuda_runtime.h>

#include "ptd_kernels.h"

namespace ptd {

constexpr int kFlowWarps = 20;   // warps per CTA at most (96 registers a thread)

// A launch: `ctas` CTAs of `warps` warps, each warp owning 31 columns x `rows`
// rows, and one CTA that judges.
struct FlowPlan {
    int rows = 0, warps = 0, ctas = 0;   // rows 0: no plan
    int ntx = 0, nty = 0;                // warp tiles in x and y
};

struct FlowArgs {
    uint4* halo_y;             // [parity][warp][bottom, top][lane]
    uint4* halo_x;             // [parity][warp][left, right][row]
    uint4* parts;              // [parity][warp]: check residuals
    unsigned long long* ctl;   // [CTA][16]: the latest decision, one line per CTA
    DevState* st;              // host-visible: the outcome
    double* errhist;           // host-visible: err of the first errhost checks,
    double* errmore;           // device memory: of the others, each at its index
    int errhost, errcap;
    unsigned base;             // tags of this launch start above it
    int ntx, nwarps;           // warp tiles in x and in all
    int nchk, itmax, checks, niter;   // checks 0: niter iterations without checks
    double tol, norm_den;
};

// Done states of a launch besides DONE_*: a wait that gave up.
enum { FLOW_TIMEOUT = 4 };

// False: the grid does not fit the registers of the SMs (or the model has no flow kernel).
bool flow_plan(int model, int nx, int ny, FlowPlan& p);
size_t flow_bytes(const FlowPlan& p);           // device memory of the exchange buffers
void flow_buffers(const FlowPlan& p, void* mem, FlowArgs& f);
cudaError_t launch_flow(const PTArgs& a, const FlowArgs& f, int model, const FlowPlan& p, cudaStream_t s);

}  // namespace ptd
