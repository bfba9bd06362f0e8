// ptd_flow.cu -- host side of the flow kernels (ptd_flow.cuh, ptd_flow3.cuh): the tile
// of a warp, the exchange buffers and the cooperative launch.
#include <algorithm>
#include <mutex>

#include "ptd_flow.h"
#include "ptd_internal.h"

namespace ptd {

const void* flow_kernel_lin(int rows, int planes, int warps);
const void* flow_kernel_linstep(int rows, int planes, int warps);
const void* flow_kernel_nonlin(int rows, int planes, int warps);

namespace {

const void* flow_kernel(int model, int rows, int planes, int warps)
{
    return model == LIN ? flow_kernel_lin(rows, planes, warps)
                        : (model == LINSTEP ? flow_kernel_linstep(rows, planes, warps)
                                            : (model == NONLIN ? flow_kernel_nonlin(rows, planes, warps) : nullptr));
}

// Elements of the exchange buffers (uint4) and of the edge fluxes (double).
size_t halo_y_len(const FlowPlan& p) { return 2ull * p.ntx * p.nty * p.ntz * 2 * std::max(p.planes, 1) * 32; }
size_t halo_x_len(const FlowPlan& p) { return 2ull * p.ntx * p.nty * p.ntz * 2 * std::max(p.planes, 1) * p.rows; }
size_t halo_z_len(const FlowPlan& p) { return p.planes ? 2ull * p.ntx * p.nty * p.ntz * 2 * p.rows * 32 : 0; }

}  // namespace

// The lowest tile whose warps fit (one SM is left to the judge): the more and
// smaller the tiles, the better the warps of an SM hide one another's latency
// (500x333 NONLIN: 2 rows 6.0 us per iteration, 3 6.1, 4 6.4, 6 7.9).  Taller
// tiles than 5 rows (468 K cells) are slower than one launch per iteration for
// NONLIN and LINSTEP (768x600 in 6 rows 17.8, 16.4; one launch each 15.2,
// 15.9), than 6 rows for LIN.  3D: 1 row x 1 plane, 1 x 2, and for LIN 2 x 2
// (299 K cells; NONLIN 64^3 in 1 x 2 11.9 us, in 2 x 2 15.8, one launch each
// 13.3).  3D grids under 32^3 cells keep one launch per iteration, although
// they would be faster here too: their launch counter (ptd_counters) is read
// as one launch per iteration and more.
bool flow_plan(int model, int ndim, int nx, int ny, int nz, FlowPlan& p)
{
    struct Tile {
        int rows, planes;
    };
    static const Tile tiles2[] = {{1, 0}, {2, 0}, {3, 0}, {4, 0}, {5, 0}, {6, 0}, {0, 0}};
    static const Tile tiles3[] = {{1, 1}, {1, 2}, {2, 2}, {0, 0}};
    const int most = sm_count() - 1;
    p = FlowPlan();
    if (ndim == 3 && (long long)nx * ny * nz < 32768) return false;
    for (const Tile* t = ndim == 3 ? tiles3 : tiles2; t->rows; ++t) {
        const long long ntx = (nx - 2 + 30) / 31, nty = (ny - 2 + t->rows - 1) / t->rows,
                        ntz = t->planes ? (nz - 2 + t->planes - 1) / t->planes : 1, n = ntx * nty * ntz;
        if (n > (long long)most * flow_warps(t->rows, t->planes)) continue;
        const int warps = (int)((n + most - 1) / most);
        const void* kernel = flow_kernel(model, t->rows, t->planes, warps);
        if (!kernel) return false;
        p.rows = t->rows;
        p.planes = t->planes;
        p.ntx = (int)ntx;
        p.nty = (int)nty;
        p.ntz = (int)ntz;
        p.warps = warps;
        p.ctas = (int)((n + p.warps - 1) / p.warps);
        int per_sm = 0;
        const bool ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32 * p.warps, 0) == cudaSuccess &&
                        per_sm >= 1;
        if (!ok) {
            cudaGetLastError();
            p = FlowPlan();
        }
        return ok;
    }
    return false;
}

size_t flow_bytes(const FlowPlan& p)
{
    const size_t n = (size_t)p.ntx * p.nty * p.ntz;
    const size_t halo = halo_y_len(p) + halo_x_len(p) + halo_z_len(p);
    return (halo + 2 * n) * sizeof(uint4) + halo / 2 * sizeof(double) + (size_t)p.ctas * 128;
}

void flow_buffers(const FlowPlan& p, void* mem, FlowArgs& f)
{
    const size_t n = (size_t)p.ntx * p.nty * p.ntz;
    f.halo_y = static_cast<uint4*>(mem);
    f.halo_x = f.halo_y + halo_y_len(p);
    f.halo_z = f.halo_x + halo_x_len(p);
    f.parts = f.halo_z + halo_z_len(p);
    f.edge_y = reinterpret_cast<double*>(f.parts + 2 * n);
    f.edge_x = f.edge_y + halo_y_len(p) / 2;
    f.edge_z = f.edge_x + halo_x_len(p) / 2;
    f.ctl = reinterpret_cast<unsigned long long*>(f.edge_z + halo_z_len(p) / 2);
    f.ntx = p.ntx;
    f.nty = p.nty;
    f.nwarps = (int)n;
}

// Launches of one process on one device run one after the other: each waits
// for all its CTAs to be resident, and two that held half the SMs each would
// wait for good.
cudaError_t launch_flow(const PTArgs& a, const FlowArgs& f, int model, const FlowPlan& p, cudaStream_t s)
{
    static std::mutex mu;
    static cudaEvent_t last[64] = {nullptr};   // per device, kept until the process ends
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ctas + (f.checks ? 1 : 0));
    cfg.blockDim = dim3(32, p.warps);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    PTArgs pa = a;
    FlowArgs fa = f;
    void* args[] = {&pa, &fa};
    std::lock_guard<std::mutex> lk(mu);
    if (!last[dev]) e = cudaEventCreateWithFlags(&last[dev], cudaEventDisableTiming);
    else e = cudaStreamWaitEvent(s, last[dev], 0);
    if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, flow_kernel(model, p.rows, p.planes, p.warps), args);
    if (e == cudaSuccess) e = cudaEventRecord(last[dev], s);
    return e;
}

}  // namespace ptd
