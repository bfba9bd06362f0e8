// ptd_line.cu -- whole physical steps of a 1D grid in one launch.
//
// A 1D grid is too small for one launch per PT iteration to do anything but
// wait: 512 cells take 3.1 us per iteration, nearly all of it launch gap and
// memory latency.  Here one thread-block cluster (up to 16 CTAs) keeps H and
// the fluxes in its shared memory from the first step to the last.  A warp loads a window
// of 32 C cells, runs up to `tmax` PT iterations on it in registers -- the
// outermost cells go stale one per iteration and side -- and writes back the
// cells in the middle, which are still exact; then one cluster barrier, and
// the next block.  The last block of a check also leaves the warp's residual
// in shared memory, and after the barrier every warp sums all of them in the
// same order and takes the same decision, so the step needs no judge and no
// second launch, and goes straight on to the next one with Hold = H (10 steps
// of 512 cells: 1.17 ms with a launch per step, 1.04 in one).  The arithmetic
// is pt1d_body's, operation for operation.
//
// Bound by the latency of a chain of six dependent FP64 instructions per
// iteration (64-76 cycles each, which is also what a scheduler needs to issue
// one): 0.32 us per iteration of 512 cells without checks, 0.47 with one
// every 10.  us per iteration, one launch per iteration / here (checks every
// 10): LIN 64 cells 2.4, 0.45; 512 2.9, 0.49; 2048 2.9, 0.77; 4096 2.9, 1.04;
// 8192 2.9, 1.95; NONLIN 512 3.3, 0.63; 4096 3.4, 1.37; 8192 3.3, 2.60.
#include <algorithm>
#include <cooperative_groups.h>

#include "ptd_internal.h"
#include "ptd_line.h"
#include "ptd_pt_body.cuh"

namespace cg = cooperative_groups;

namespace ptd {

namespace {

constexpr int kMaxWarps = 8;     // warps per CTA (13824 cells in all; at 16384 one launch per iteration is as fast)
constexpr int kMaxCluster = 16;  // CTAs (above 8 the size is not portable: granted by kernel attribute)

// Dynamic shared memory of a CTA.  The largest, 8 warps x 126 cells, is under
// the 48 KB that a kernel has without an attribute, and no plan sets that
// attribute: it belongs to the kernel, which all contexts share.
constexpr size_t line_smem(int warps, int core)
{
    return (size_t)(4 * warps * core + 2 * kMaxWarps + kHostErr) * sizeof(double);
}
static_assert(line_smem(kMaxWarps, 32 * 4 - 2) <= 48 * 1024, "a line CTA needs no shared-memory attribute");

// One cell window of a warp: C consecutive cells per lane.
template <int MODEL, int C>
__global__ void __launch_bounds__(32 * kMaxWarps) pt_line_kernel(PTArgs a, LineArgs l)
{
    using N = F64;
    constexpr bool HASD = ModelTraits<MODEL>::hasd;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ double smem[];
    // own slice of H and of the fluxes, double-buffered by block; the warps'
    // residuals of the two latest checks
    const int slice = l.warps * l.core;
    double* sH = smem;
    double* sW = smem + 2 * slice;
    double* sR = smem + 4 * slice;
    double* sE = sR + 2 * kMaxWarps;   // CTA 0: acc of the first kHostErr checks
    double* const Hg = static_cast<double*>(a.Hout);
    double* const Wg = static_cast<double*>(a.wout[0]);
    double* const Og = l.Hold;

    const int rank = (int)cluster.block_rank(), ncta = (int)cluster.num_blocks();
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int nx = a.nx;
    const int first = rank * slice;                    // first cell of this CTA's slice
    const int x0 = first + warp * l.core - l.tmax;     // first cell of this warp's window

    double H[C], W[C], Ho[C], D[C], Dr[C];
    bool face[C], upd[C], core[C];
    float e[C];
#pragma unroll
    for (int q = 0; q < C; ++q) {
        const int k = lane * C + q, j = x0 + k;
        face[q] = j >= 0 && j <= nx - 2;
        upd[q] = j >= 1 && j <= nx - 2;
        core[q] = k >= l.tmax && k < l.tmax + l.core && j < nx;
        const int jc = min(max(j, 0), nx - 1);
        Ho[q] = Og[jc];
        D[q] = HASD ? static_cast<const double*>(a.D)[jc] : 0.0;
        Dr[q] = HASD ? static_cast<const double*>(a.D)[min(jc + 1, nx - 1)] : 0.0;
        const float dl = HASD ? N::lo_f(static_cast<const double*>(a.D)[max(jc - 1, 0)]) : 0.0f;
        if (MODEL == LIN) e[q] = a.fe_lin;
        if (MODEL == LINSTEP) e[q] = linstep_cell_e(a.f, fmaxf(fmaxf(dl, N::lo_f(Dr[q])), N::lo_f(D[q])));
        if (core[q]) {
            sH[j - first] = Hg[j];
            sW[j - first] = Wg[j];
        }
    }
    // the shared-memory slice holding cell j, and j's place in it
    auto at = [&](double* base, int j) {
        const int r = j < first ? rank - 1 : (j >= first + slice ? rank + 1 : rank);
        return cluster.map_shared_rank(base, (unsigned)r) + (j - r * slice);
    };
    int iter = 0, nchecks = 0, done = DONE_RUNNING, buf = 0;
    int steps = 0;                                     // steps ended,
    unsigned total = 0;                                // their iterations
    const int blocks = l.itmax / max(l.nchk, 1);       // checks of a step at most
    bool begin = false;                                // a step begins: Hold = H
    double acc = 0.0;
    const int nchk = l.checks ? l.nchk : l.niter;      // iterations of one check block
    cluster.sync();
    // every pass runs 1..tmax iterations of a check block, so the loop ends
    // within nsteps * itmax (niter) passes
    for (int left = l.checks ? (nchk <= l.itmax ? nchk : 0) : l.niter; left > 0;) {
        const int n = min(left, l.tmax);
        const bool check = l.checks && n == left;
#pragma unroll
        for (int q = 0; q < C; ++q) {
            const int j = x0 + lane * C + q;
            const bool in = j >= 0 && j < nx;
            H[q] = in ? *at(sH + buf * slice, j) : 0.0;
            W[q] = in ? *at(sW + buf * slice, j) : 0.0;
            if (begin) Ho[q] = H[q];
        }
        begin = false;
        double part = 0.0;
        unsigned long long pmax = 0ull;
        auto iteration = [&](auto chk) {
            constexpr bool CHECK = decltype(chk)::value;
            double u[C];
            const double Hnext = N::shfl_down(H[0], 1);
#pragma unroll
            for (int q = 0; q < C; ++q) {
                const double Hr = q < C - 1 ? H[q + 1 < C ? q + 1 : q] : Hnext;
                u[q] = 0.0;
                const double w = face_t<N, MODEL, CHECK, false>(a, H[q], Hr, N::hf(H[q]) + N::hf(Hr), D[q], Dr[q],
                                                                W[q], u[q]);
                W[q] = face[q] ? w : 0.0;
            }
            const double Wprev = N::shfl_up(W[C - 1], 1);
            const double Uprev = CHECK ? N::shfl_up(u[C - 1], 1) : 0.0;
#pragma unroll
            for (int q = 0; q < C; ++q) {
                const double wl = q > 0 ? W[q > 0 ? q - 1 : 0] : Wprev;
                float eq = e[q];
                if (MODEL == NONLIN || MODEL == NONLIN_EXPM)
                    eq = cell_e<MODEL>(a, N::hf(H[q]), MODEL == NONLIN_EXPM ? N::lo_f(D[q]) : 0.0f);
                const double Hn = h_update_sq<N, false>(a, H[q], Ho[q], N::sub(W[q], wl), eq);
                if (CHECK && upd[q] && core[q]) {
                    const double ul = q > 0 ? u[q > 0 ? q - 1 : 0] : Uprev;
                    const double r = N::sub(N::mul(N::sub(u[q], ul), cst<N>(a, 0)), N::mul(N::hdn(Hn, Ho[q]), cst<N>(a, 3)));
                    accumulate_residual(r, part, pmax);
                }
                if (upd[q]) H[q] = Hn;
            }
        };
        for (int t = 0; t < n - (check ? 1 : 0); ++t) iteration(std::false_type{});
        if (check) iteration(std::true_type{});
        buf ^= 1;
#pragma unroll
        for (int q = 0; q < C; ++q) {
            if (core[q]) {
                const int j = x0 + lane * C + q;
                sH[buf * slice + j - first] = H[q];
                sW[buf * slice + j - first] = W[q];
            }
        }
        if (check) {
            double v = a.norm_max ? __longlong_as_double((long long)warp_max_u64(pmax)) : warp_sum(part);
            if (lane == 0) sR[(nchecks & 1) * kMaxWarps + warp] = v;
        }
        cluster.sync();
        left -= n;
        if (check) {
            // the residual of every warp of the cluster, in the same order in every warp
            double sum = 0.0;
            unsigned long long mx = 0ull;
            for (int k = lane; k < ncta * l.warps; k += 32) {
                const double v = *(cluster.map_shared_rank(sR, (unsigned)(k / l.warps)) + (nchecks & 1) * kMaxWarps +
                                   k % l.warps);
                const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
                mx = bits > mx ? bits : mx;
                sum += v;
            }
            acc = a.norm_max ? __longlong_as_double((long long)warp_max_u64(mx)) : warp_sum(sum);
            // the history takes acc (the host forms err = sqrt(acc) / sqrt(norm_den),
            // which would cost about 1 us of dependent FP64 here), in shared
            // memory until the end: the next barrier would wait for a store to
            // the host
            if (rank == 0 && warp == 0 && lane == 0) {
                if (nchecks < kHostErr) sE[nchecks] = acc;
                else if (nchecks < l.errcap) l.errmore[nchecks] = acc;
            }
            nchecks += 1;
            iter += nchk;
            // err is needed only where acc does not decide
            if (!(acc > l.acc_above)) {
                const double err = a.norm_max ? acc : sqrt(acc) / sqrt(l.norm_den);
                if (!(err > l.tol)) done = (err != err) ? DONE_NAN : DONE_CONVERGED;
            }
            if (done == DONE_RUNNING && iter + nchk > l.itmax) done = DONE_CAP;
            if (done != DONE_RUNNING) {
                if (rank == 0 && warp == 0 && lane == 0) l.out->iters[steps] = iter;
                steps += 1;
                total += iter;
                if (done == DONE_CONVERGED && steps < l.nsteps && total < (unsigned)l.itlimit && nchecks <= l.errcap - blocks) {
                    done = DONE_RUNNING;
                    begin = true;
                    iter = 0;
                }
            }
            left = done == DONE_RUNNING ? nchk : 0;
        }
    }
#pragma unroll
    for (int q = 0; q < C; ++q) {
        if (core[q]) {
            const int j = x0 + lane * C + q;
            Hg[j] = sH[buf * slice + j - first];
            Wg[j] = sW[buf * slice + j - first];
            // the next step's Hold; a step stopped by itmax goes on from its own
            if (l.checks) Og[j] = done == DONE_CAP ? Ho[q] : Hg[j];
        }
    }
    if (l.checks && rank == 0 && warp == 0) {
        __syncwarp();
        for (int k = lane; k < min(nchecks, kHostErr); k += 32) l.out->err[k] = sE[k];
    }
    if (l.checks && rank == 0 && warp == 0 && lane == 0) {
        l.st->done = done;
        l.st->nchecks = nchecks;
        l.st->iter = iter;
        l.st->acc = acc;
        l.out->nsteps = steps;
    }
    cluster.sync();   // no CTA leaves while another may read its shared memory
}

template <int MODEL>
const void* kernel_of(int c)
{
    return c == 1 ? (const void*)pt_line_kernel<MODEL, 1>
                  : (c == 2 ? (const void*)pt_line_kernel<MODEL, 2> : (const void*)pt_line_kernel<MODEL, 4>);
}

const void* line_kernel(int model, int c)
{
    switch (model) {
    case LIN: return kernel_of<LIN>(c);
    case LINSTEP: return kernel_of<LINSTEP>(c);
    case NONLIN: return kernel_of<NONLIN>(c);
    default: return kernel_of<NONLIN_EXPM>(c);
    }
}

cudaLaunchConfig_t launch_of(const LinePlan& p, cudaStream_t s, cudaLaunchAttribute* at)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ctas);
    cfg.blockDim = dim3(32, p.warps);
    cfg.dynamicSmemBytes = line_smem(p.warps, p.core);
    cfg.stream = s;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = p.ctas;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

// The window width and cluster of a grid: blocks of up to 10 iterations (at
// most a check block), and the cells per lane that give the fewest FP64
// instructions per scheduler and iteration, each of the cluster's 4
// schedulers per SM running one warp's instructions after another's.
bool line_plan(int model, int nx, int nchk, LinePlan& p)
{
    p = LinePlan();
    long long best = 0;
    for (int c = 1; c <= 4; c *= 2) {
        const int t = std::min(nchk, 10), core = 32 * c - 2 * t;
        const int need = (nx + core - 1) / core;                 // warps
        int ctas = 1;
        while (ctas < kMaxCluster && ctas < need) ctas *= 2;
        const int warps = (need + ctas - 1) / ctas;
        if (warps > kMaxWarps) continue;
        const long long cost = (long long)c * ((warps + 3) / 4);
        if (!p.ctas || cost < best) {
            best = cost;
            p.c = c;
            p.tmax = t;
            p.core = core;
            p.ctas = ctas;
            p.warps = warps;
        }
    }
    if (!p.ctas) return false;
    const void* f = line_kernel(model, p.c);
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = launch_of(p, nullptr, &at);
    int n = 0;
    bool ok = true;
    if (p.ctas > 8) ok = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    ok = ok && cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n >= 1;
    if (!ok) cudaGetLastError();
    return ok;
}

cudaError_t launch_line(const PTArgs& a, const LineArgs& l, int model, const LinePlan& p, cudaStream_t s)
{
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = launch_of(p, s, &at);
    PTArgs pa = a;
    LineArgs la = l;
    la.tmax = p.tmax;
    la.core = p.core;
    la.warps = p.warps;
    void* args[] = {&pa, &la};
    return cudaLaunchKernelExC(&cfg, line_kernel(model, p.c), args);
}

}  // namespace ptd
