// ptd_flow.h -- host interface of the 2D and 3D kernels that hold whole steps
// (ptd_flow.cuh, ptd_flow3.cuh).
#pragma once

#include <cuda_runtime.h>

#include "ptd_kernels.h"

namespace ptd {

constexpr int kFlowWarps = 20;   // warps per CTA at most (96 registers a thread)
// (3D tiles of two rows of cells: 28, 72 registers; of four: 16, 128)
__host__ __device__ constexpr int flow_warps(int rows, int planes)
{
    return planes < 2 ? kFlowWarps : (rows == 1 ? 28 : 16);
}

// A launch: `ctas` CTAs of `warps` warps, each warp owning 31 columns x `rows`
// rows (3D: x `planes` planes), and one CTA that judges.
struct FlowPlan {
    int rows = 0, planes = 0, warps = 0, ctas = 0;   // rows 0: no plan; planes 0: 2D
    int ntx = 0, nty = 0, ntz = 1;                   // warp tiles in x, y and z
};

struct FlowArgs {
    uint4* halo_y;             // [parity][warp][bottom, top][lane]; 3D: [parity][warp][front, back][plane][lane]
    uint4* halo_x;             // [parity][warp][left, right][row]; 3D: [parity][warp][left, right][plane][row]
    uint4* halo_z;             // 3D: [parity][warp][below, above][row][lane]
    uint4* parts;              // [parity][warp]: check residuals
    double* edge_y;            // [parity][warp][(plane)][lane]: flux on a tile's lower y edge at a check
    double* edge_x;            // [parity][warp][(plane)][row]: flux on its left edge
    double* edge_z;            // 3D: [parity][warp][row][lane]: flux on its lower z edge
    unsigned long long* ctl;   // [CTA][16]: the latest decision, one line per CTA
    DevState* st;              // host-visible: the outcome,
    HostSteps* out;            // the steps, and err of the first checks,
    double* errmore;           // device memory: of the others, each at its index
    int errcap;
    unsigned base;             // tags of this launch start above it
    int ntx, nty, nwarps;      // warp tiles in x, in y and in all
    int nchk, itmax, checks, niter;   // checks 0: niter iterations without checks
    int nsteps, itlimit;       // steps at most, and none begun after that many iterations
    int wait;                  // polls of one wait before it gives up
    double tol, norm_den;
};

constexpr int kFlowWait = 1 << 25;   // about 20 s: another kernel may hold an SM
// Iterations of a check block at most: the judge's wait spans one (4 s of the
// largest grids).  A context with a longer cadence runs one iteration per launch.
constexpr int kFlowCheck = 1 << 18;

// Done states besides DONE_*: a wait that gave up; a step that converged, and
// the next one begins in the same launch.
enum { FLOW_TIMEOUT = 4, FLOW_NEXT = 5 };

// Tags that a step of iter iterations uses: its warps run on until the
// decision reaches them, three check blocks at most, and the next step's first
// exchange has one.
__host__ __device__ inline unsigned flow_tags(int iter, int nchk) { return (unsigned)iter + 3u * (unsigned)nchk + 2u; }

// False: the grid does not fit the registers of the SMs (or the model has no flow kernel).
bool flow_plan(int model, int ndim, int nx, int ny, int nz, FlowPlan& p);
size_t flow_bytes(const FlowPlan& p);           // device memory of the exchange buffers
void flow_buffers(const FlowPlan& p, void* mem, FlowArgs& f);
cudaError_t launch_flow(const PTArgs& a, const FlowArgs& f, int model, const FlowPlan& p, cudaStream_t s);

}  // namespace ptd
