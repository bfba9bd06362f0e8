// ptd_flow.cu -- host side of the 2D flow kernel (ptd_flow.cuh): the tile
// of a warp, the exchange buffers and the cooperative launch.
#include <mutex>

#include "ptd_flow.h"
#include "ptd_internal.h"

namespace ptd {

const void* flow_kernel_lin(int rows);
const void* flow_kernel_linstep(int rows);
const void* flow_kernel_nonlin(int rows);

namespace {

const void* flow_kernel(int model, int rows)
{
    return model == LIN ? flow_kernel_lin(rows)
                        : (model == LINSTEP ? flow_kernel_linstep(rows)
                                            : (model == NONLIN ? flow_kernel_nonlin(rows) : nullptr));
}

}  // namespace

// The lowest tile whose warps fit (one SM is left to the judge): the more and
// smaller the tiles, the better the warps of an SM hide one another's latency
// (500x333 NONLIN: 2 rows 6.0 us per iteration, 3 6.1, 4 6.4, 6 7.9).  Taller
// tiles than 5 rows (468 K cells) are slower than one launch per iteration for
// NONLIN and LINSTEP (768x600 in 6 rows 17.8, 16.4; one launch each 15.2,
// 15.9), than 6 rows for LIN.
bool flow_plan(int model, int nx, int ny, FlowPlan& p)
{
    const int most = sm_count() - 1;
    for (int rows : {1, 2, 3, 4, 5, 6}) {
        p = FlowPlan();
        if (!flow_kernel(model, rows)) return false;
        const long long ntx = (nx - 2 + 30) / 31, nty = (ny - 2 + rows - 1) / rows, n = ntx * nty;
        if (n > (long long)most * kFlowWarps) continue;
        p.rows = rows;
        p.ntx = (int)ntx;
        p.nty = (int)nty;
        p.warps = (int)((n + most - 1) / most);
        p.ctas = (int)((n + p.warps - 1) / p.warps);
        int per_sm = 0;
        const bool ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, flow_kernel(model, rows), 32 * p.warps,
                                                                      0) == cudaSuccess && per_sm >= 1;
        if (!ok) {
            cudaGetLastError();
            p = FlowPlan();
        }
        return ok;
    }
    p = FlowPlan();
    return false;
}

size_t flow_bytes(const FlowPlan& p)
{
    const size_t n = (size_t)p.ntx * p.nty;
    return (2 * n * 2 * 32 + 2 * n * 2 * p.rows + 2 * n) * sizeof(uint4) + (2 * n * 32 + 2 * n * p.rows) * sizeof(double) +
           (size_t)p.ctas * 128;
}

void flow_buffers(const FlowPlan& p, void* mem, FlowArgs& f)
{
    const size_t n = (size_t)p.ntx * p.nty;
    f.halo_y = static_cast<uint4*>(mem);
    f.halo_x = f.halo_y + 2 * n * 2 * 32;
    f.parts = f.halo_x + 2 * n * 2 * p.rows;
    f.edge_y = reinterpret_cast<double*>(f.parts + 2 * n);
    f.edge_x = f.edge_y + 2 * n * 32;
    f.ctl = reinterpret_cast<unsigned long long*>(f.edge_x + 2 * n * p.rows);
    f.ntx = p.ntx;
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
    if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, flow_kernel(model, p.rows), args);
    if (e == cudaSuccess) e = cudaEventRecord(last[dev], s);
    return e;
}

}  // namespace ptd
