// ptd_flow.h -- host interface of the 2D kernel that holds whole steps (ptd_flow.cuh).
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
    double* edge_y;            // [parity][warp][lane]: flux on a tile's lower edge at a check
    double* edge_x;            // [parity][warp][row]: flux on its left edge
    unsigned long long* ctl;   // [CTA][16]: the latest decision, one line per CTA
    DevState* st;              // host-visible: the outcome,
    HostSteps* out;            // the steps, and err of the first checks,
    double* errmore;           // device memory: of the others, each at its index
    int errcap;
    unsigned base;             // tags of this launch start above it
    int ntx, nwarps;           // warp tiles in x and in all
    int nchk, itmax, checks, niter;   // checks 0: niter iterations without checks
    int nsteps, itlimit;       // steps at most, and none begun after that many iterations
    double tol, norm_den;
};

// Done states besides DONE_*: a wait that gave up; a step that converged, and
// the next one begins in the same launch.
enum { FLOW_TIMEOUT = 4, FLOW_NEXT = 5 };

// Tags that a step of iter iterations uses: its warps run on until the
// decision reaches them, three check blocks at most, and the next step's first
// exchange has one.
__host__ __device__ inline unsigned flow_tags(int iter, int nchk) { return (unsigned)iter + 3u * (unsigned)nchk + 2u; }

// False: the grid does not fit the registers of the SMs (or the model has no flow kernel).
bool flow_plan(int model, int nx, int ny, FlowPlan& p);
size_t flow_bytes(const FlowPlan& p);           // device memory of the exchange buffers
void flow_buffers(const FlowPlan& p, void* mem, FlowArgs& f);
cudaError_t launch_flow(const PTArgs& a, const FlowArgs& f, int model, const FlowPlan& p, cudaStream_t s);

}  // namespace ptd
