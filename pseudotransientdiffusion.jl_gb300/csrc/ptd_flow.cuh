// ptd_flow.cuh -- whole physical steps of a 2D grid (native FP64) in one
// launch.
//
// One launch per iteration costs a grid that fits the chip about 4 us of
// launch gap, memory latency and ramp per iteration, several times its FP64
// work (0.3 us at 128^2).  Here every warp owns a tile of 31 columns x R rows
// for the whole step, H and the fluxes in registers, and exchanges only the
// edges of H with its four neighbours: each iteration it publishes its edge
// cells and waits for theirs.  An edge value travels with its tag (the
// iteration it belongs to) in the same 8 bytes, {32 bits of the double, tag}
// twice in one 16-byte store, so a reader that sees both tags has the value: no
// fence, no flag, no barrier, and a warp waits for its neighbours only.  The
// faces on a tile's left and lower edge are evolved by both tiles that touch
// them, from the same values.  Slots alternate by iteration parity; a warp
// publishes iteration k + 2 only after it has read its neighbours' k + 1,
// which they published after reading its k.
//
// Checks do not stop the warps: each leaves its residual in a tagged slot and
// a snapshot of its cells in the buffer of the check's parity, and goes on; a
// judging CTA sums the slots in a fixed order, takes the reference's decision
// and publishes it; the warps look for it once per iteration and leave when
// the step has stopped.  A snapshot is overwritten (two checks later) only
// once the decision on it is known.
//
// Between two steps of a launch a warp reads back the snapshot that the
// decision was on (its own stores), takes its H as Hold and exchanges edges:
// about 2 us, where the end of a launch, the host's wait, a copy of Hold and
// the next launch cost 38 (a solve of 5 steps of 128^2: 1.04 ms with a launch
// per step, 0.81 in one).
//
// All CTAs must run at once: the launch is cooperative, and every wait has a
// limit after which its warp gives up and the step ends with FLOW_TIMEOUT.
//
// The arithmetic is pt2d_body's, operation for operation: the same bits.
//
// Bound by the FP64 pipe and, on small grids, by the latency of an iteration
// (about 1700 cycles of dependent arithmetic for the first row of a tile, 1200
// for each other, and 1400-2000 of exchange through L2).  us per iteration
// with checks every 10, one launch per iteration / here: NONLIN 128^2 4.1, 2.5;
// 256^2 5.2, 3.2; 512^2 10.0, 7.3; 640^2 13.2, 10.3; 768x600 15.2, 11.9;
// LINSTEP 500x333 8.1, 5.5; 768x600 15.9, 12.2; LIN 768x600 15.0, 11.8; 730x740
// 16.3, 14.2.
// (Evaluating the faces of several rows as one branch-free group was no
// faster, and tiles of 10 rows in 8-warp CTAs slower: 128^2 2.6, 8.3.)
#pragma once

#include "ptd_flow.h"
#include "ptd_pt_body.cuh"

namespace ptd {

constexpr int kWarps = kFlowWarps;

// A slot is two 64-bit words, each {32 bits of the value, tag} (the layout of
// NCCL's low-latency protocol), moved by one vector instruction.  A vector
// access is one scalar access per element in the memory model, so a word
// arrives whole; as four 32-bit elements a value could part from its tag.
__device__ __forceinline__ uint4 flow_load(const uint4* p)
{
    uint4 v;
    asm volatile("{ .reg .b64 a, b; ld.volatile.global.v2.b64 {a,b}, [%4]; mov.b64 {%0,%1}, a; mov.b64 {%2,%3}, b; }"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void flow_store(uint4* p, double x, unsigned tag)
{
    asm volatile("{ .reg .b64 a, b; mov.b64 a, {%1,%3}; mov.b64 b, {%2,%3}; st.volatile.global.v2.b64 [%0], {a,b}; }" ::"l"(p),
                 "r"((unsigned)__double2loint(x)), "r"((unsigned)__double2hiint(x)), "r"(tag) : "memory");
}
__device__ __forceinline__ double flow_value(const uint4& v) { return __hiloint2double((int)v.z, (int)v.x); }
__device__ __forceinline__ bool flow_ready(const uint4& v, unsigned tag) { return v.y == tag && v.w == tag; }

// The judge, one CTA (the decision of judge_parts_kernel).
__device__ __forceinline__ void flow_judge(const PTArgs& a, const FlowArgs& f)
{
    __shared__ double s_sum[256];
    __shared__ unsigned long long s_max[256];
    __shared__ int s_done, s_lost;
    const int t = threadIdx.y * 32 + threadIdx.x, nt = min((int)blockDim.y * 32, 256);   // threads that sum
    if (t == 0) s_lost = 0;
    __syncthreads();
    int iter = 0, nchecks = 0, step = 0;   // of the step; of the launch
    unsigned base = f.base, total = 0;
    const int blocks = f.itmax / f.nchk;
    // every pass is a check block of nchk iterations, so a step ends within itmax/nchk passes
    for (int n = 0;; ++n) {
        const unsigned tag = base + (unsigned)n + 1u;
        const uint4* parts = f.parts + (size_t)(n & 1) * f.nwarps;
        double sum = 0.0;
        unsigned long long mx = 0ull;
        for (int i = t; t < nt && i < f.nwarps; i += nt) {
            uint4 v = flow_load(parts + i);
            for (int left = f.wait; !flow_ready(v, tag) && left > 0; --left) v = flow_load(parts + i);
            if (!flow_ready(v, tag)) {
                s_lost = 1;
                break;
            }
            const double x = flow_value(v);
            const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
            mx = bits > mx ? bits : mx;
            sum += x;
        }
        for (int q = t; t < nt && q < 256; q += nt) {
            s_sum[q] = q == t ? sum : 0.0;
            s_max[q] = q == t ? mx : 0ull;
        }
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            for (int q = t; t < nt && q < o; q += nt) {
                s_sum[q] += s_sum[q + o];
                s_max[q] = s_max[q + o] > s_max[q] ? s_max[q + o] : s_max[q];
            }
            __syncthreads();
        }
        iter += f.nchk;
        if (t == 0) {
            const double acc = a.norm_max ? __longlong_as_double((long long)s_max[0]) : s_sum[0];
            const double err = a.norm_max ? acc : sqrt(acc) / sqrt(f.norm_den);
            int done = DONE_RUNNING;
            if (!(err > f.tol)) done = (err != err) ? DONE_NAN : DONE_CONVERGED;
            else if (iter + f.nchk > f.itmax) done = DONE_CAP;
            if (s_lost) done = FLOW_TIMEOUT;
            if (done == DONE_CONVERGED && step + 1 < f.nsteps && total + (unsigned)iter < (unsigned)f.itlimit &&
                nchecks + 1 <= f.errcap - blocks)
                done = FLOW_NEXT;
            s_done = done;
            if (nchecks < kHostErr) f.out->err[nchecks] = err;
            else if (nchecks < f.errcap) f.errmore[nchecks] = err;
            if (done != DONE_RUNNING) f.out->iters[step] = iter;
            if (done != DONE_RUNNING && done != FLOW_NEXT) {
                f.st->done = done;
                f.st->nchecks = nchecks + 1;
                f.st->iter = iter;
                f.st->err = err;
                f.out->nsteps = step + 1;
            }
        }
        __syncthreads();
        const int done = s_done;
        const unsigned long long word = ((unsigned long long)tag << 32) | (unsigned)done;
        for (int c = t; c < (int)gridDim.x - 1; c += (int)blockDim.y * 32) *(volatile unsigned long long*)(f.ctl + 16 * c) = word;
        if (done != DONE_RUNNING && done != FLOW_NEXT) return;
        nchecks += 1;
        if (done == FLOW_NEXT) {
            base += flow_tags(iter, f.nchk);
            total += (unsigned)iter;
            step += 1;
            iter = 0;
            n = -1;
        }
        __syncthreads();   // s_sum of this check is read before the next one writes it
    }
}

template <int MODEL, int R>
__global__ void __launch_bounds__(32 * kWarps, 1) pt2d_flow_kernel(PTArgs a, FlowArgs f)
{
    using N = F64;
    constexpr bool HASD = ModelTraits<MODEL>::hasd;
    if (blockIdx.x == gridDim.x - 1 && f.checks) {
        flow_judge(a, f);
        return;
    }
    const int lane = threadIdx.x;
    const int w = blockIdx.x * blockDim.y + threadIdx.y;   // the warp's tile
    if (w >= f.nwarps) return;
    const int tx = w % f.ntx, ty = w / f.ntx, nty = f.nwarps / f.ntx;
    const int nx = a.nx, ny = a.ny;
    const int i = 31 * tx + lane, ic = min(i, nx - 1), ir = min(i + 1, nx - 1);
    const int j0 = 1 + ty * R;
    const bool xface = i <= nx - 2, upd = i >= 1 && i <= nx - 2 && lane >= 1;
    const bool own_x = xface && (lane >= 1 || tx == 0);
    const bool left = tx > 0, right = tx < f.ntx - 1, below = ty > 0, above = ty < nty - 1;   // neighbours
    const long long sy = a.sy;
    volatile unsigned long long* const ctl = f.ctl + 16 * blockIdx.x;

    // the tile: rows j0 .. j0+R-1 (those past ny-2 hold the boundary row and
    // never change), the rows below and above it; in shared memory what does
    // not change in a step, and the column right of the tile (read by lane 31)
    __shared__ double s_Ho[kWarps][R][32], s_Hr[kWarps][R];
    __shared__ double s_D[HASD ? kWarps : 1][R][32], s_Dr[HASD ? kWarps : 1][R][32];
    __shared__ float s_E[MODEL == LINSTEP ? kWarps : 1][R][32];
    double(*const sHo)[32] = s_Ho[threadIdx.y];
    double* const sHr = s_Hr[threadIdx.y];
    double(*const sD)[32] = s_D[HASD ? threadIdx.y : 0];
    double(*const sDr)[32] = s_Dr[HASD ? threadIdx.y : 0];
    float(*const sE)[32] = s_E[MODEL == LINSTEP ? threadIdx.y : 0];
    double H[R], wx[R], wy[R], Hb, Ht, wyb, Db = 0.0, Dt = 0.0;
    auto at = [&](int j) { return (long long)min(j, ny - 1) * sy; };
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const long long row = at(j0 + q);
        H[q] = N::ldh(a.Hin, row + ic);
        wx[q] = ld<N>(a.win[0], row + ic);
        wy[q] = ld<N>(a.win[1], row + ic);
        sHo[q][lane] = N::ldo(a.Hold, row + ic);
        if (lane == 31) sHr[q] = N::ldh(a.Hin, row + ir);
        if constexpr (HASD) {
            const double dc = ld<N>(a.D, row + ic), dr = ld<N>(a.D, row + ir);
            sD[q][lane] = dc;
            sDr[q][lane] = dr;
            if (MODEL == LINSTEP) {
                const double dl = ld<N>(a.D, row + max(ic - 1, 0)), db = ld<N>(a.D, at(j0 + q - 1) + ic),
                             du = ld<N>(a.D, at(j0 + q + 1) + ic);
                sE[q][lane] = linstep_cell_e(a.f, fmaxf(fmaxf(fmaxf(N::lo_f(dc), N::lo_f(dl)),
                                                              fmaxf(N::lo_f(dr), N::lo_f(db))), N::lo_f(du)));
            }
        }
    }
    Hb = N::ldh(a.Hin, at(j0 - 1) + ic);
    Ht = N::ldh(a.Hin, at(j0 + R) + ic);
    wyb = ld<N>(a.win[1], at(j0 - 1) + ic);
    if (HASD) {
        Db = ld<N>(a.D, at(j0 - 1) + ic);
        Dt = ld<N>(a.D, at(j0 + R) + ic);
    }
    __syncwarp();

    // the neighbours' slots this lane reads and its own
    auto hy = [&](int par, int tile, int side) {
        return f.halo_y + (((size_t)par * f.nwarps + tile) * 2 + side) * 32 + lane;
    };
    auto hx = [&](int par, int tile, int side) {
        return f.halo_x + (((size_t)par * f.nwarps + tile) * 2 + side) * R;
    };
    const bool getx = (lane == 0 && left) || (lane == 31 && right);
    const bool putx = (lane == 1 && left) || (lane == 31 && right);
    const bool gety_b = below && upd, gety_t = above && upd;

    // the tile's cells and faces in the buffers of parity par: stored (with
    // the faces that the neighbours own, in buffers of this warp), and read
    // back by the threads that stored them
    auto buf_h = [&](int par) { return static_cast<double*>(par ? a.Hout : const_cast<void*>(a.Hin)); };
    auto buf_x = [&](int par) { return static_cast<double*>(par ? a.wout[0] : const_cast<void*>(a.win[0])); };
    auto buf_y = [&](int par) { return static_cast<double*>(par ? a.wout[1] : const_cast<void*>(a.win[1])); };
    auto edge_y = [&](int par) { return f.edge_y + ((size_t)par * f.nwarps + w) * 32 + lane; };
    auto edge_x = [&](int par) { return f.edge_x + ((size_t)par * f.nwarps + w) * R; };
    auto snapshot = [&](int par) {
        double *const Hd = buf_h(par), *const X = buf_x(par), *const Y = buf_y(par);
        if (f.checks) *edge_y(par) = wyb;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (j0 + q <= ny - 2) {
                const long long c = at(j0 + q) + ic;
                if (own_x) X[c] = wx[q];
                else if (f.checks && lane == 0) edge_x(par)[q] = wx[q];
                if (upd) {
                    Y[c] = wy[q];
                    Hd[c] = H[q];
                }
            }
        }
        if (ty == 0 && upd) Y[ic] = wyb;
    };
    auto restore = [&](int par) {
        const double *const Hd = buf_h(par), *const X = buf_x(par), *const Y = buf_y(par);
        wyb = __ldcg(edge_y(par));
#pragma unroll
        for (int q = 0; q < R; ++q) {
            if (j0 + q <= ny - 2) {
                const long long c = at(j0 + q) + ic;
                if (own_x) wx[q] = __ldcg(X + c);
                else if (lane == 0) wx[q] = __ldcg(edge_x(par) + q);
                if (upd) {
                    wy[q] = __ldcg(Y + c);
                    H[q] = __ldcg(Hd + c);
                    sHo[q][lane] = H[q];   // the next step's Hold
                }
            }
        }
    };

    double part = 0.0;
    unsigned long long pmax = 0ull;
    // one iteration from the halos in place.  Row q's cells are updated once
    // both their faces are known; the next row's old H is read before.
    auto iteration = [&](auto chk) {
        constexpr bool C = decltype(chk)::value;
        double uyb = 0.0, uy = 0.0, Hcur = H[0];
        float hc = N::hf(Hcur);
        wyb = face_t<N, MODEL, C>(a, Hb, Hcur, N::hf(Hb) + hc, Db, HASD ? sD[0][lane] : 0.0, wyb, uyb);
        double wlow = wyb;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const double Hup = q < R - 1 ? H[q + 1 < R ? q + 1 : q] : Ht;
            const double Dc = HASD ? sD[HASD ? q : 0][lane] : 0.0;
            const double Dup = HASD ? (q < R - 1 ? sD[HASD && q + 1 < R ? q + 1 : 0][lane] : Dt) : 0.0;
            const double Dright = HASD ? sDr[HASD ? q : 0][lane] : 0.0;
            const float hu = N::hf(Hup);
            double Hright = N::shfl_down(Hcur, 1);
            float hr = __shfl_down_sync(FULL, hc, 1);
            if (lane == 31) {
                Hright = sHr[q];
                hr = N::hf(Hright);
            }
            double ux = 0.0;
            if (xface) wx[q] = face_t<N, MODEL, C>(a, Hcur, Hright, hc + hr, Dc, Dright, wx[q], ux);
            const double wup = face_t<N, MODEL, C>(a, Hcur, Hup, hc + hu, Dc, Dup, wy[q], uy);
            const double wxl = N::shfl_up(wx[q], 1), uxl = C ? N::shfl_up(ux, 1) : 0.0;
            if (upd && j0 + q <= ny - 2) {
                wy[q] = wup;
                const double dx = N::sub(wx[q], wxl), dy = N::sub(wup, wlow), Ho = sHo[q][lane];
                float e = a.fe_lin;
                if (MODEL == LINSTEP) e = sE[MODEL == LINSTEP ? q : 0][lane];
                if (MODEL == NONLIN) e = cell_e<MODEL>(a, hc, 0.0f);
                const double Hn =
                    a.sq ? h_update_sq<N>(a, Hcur, Ho, N::add(dy, dx), e)
                         : h_update<N>(a, Hcur, Ho, N::mad(dy, cst<N>(a, 1), N::mul(dx, cst<N>(a, 0))), e);
                if (C) {
                    const double divu = N::mad(N::sub(uy, uyb), cst<N>(a, 1), N::mul(N::sub(ux, uxl), cst<N>(a, 0)));
                    accumulate_residual(N::sub(divu, N::mul(N::hdn(Hn, Ho), cst<N>(a, 3))), part, pmax);
                }
                H[q] = Hn;
            }
            wlow = wup;
            if (C) uyb = uy;
            Hcur = Hup;
            hc = hu;
        }
    };

    unsigned base = f.base;   // tags of the step start above it
    // the decision published last: how many checks are decided, and the outcome
    // (a word of an earlier step counts as none); lane 0's reading for all
    auto decided = [&](unsigned long long word, int& n, int& done) {
        const unsigned d = (unsigned)(word >> 32) - base;
        n = __shfl_sync(FULL, d < 0x80000000u ? (int)d : 0, 0);
        done = __shfl_sync(FULL, (int)(unsigned)word, 0);
        if (n == 0) done = DONE_RUNNING;
    };
    int flip = 0;   // parity of the buffers that hold the step's first state
    // every pass is a step (a launch without checks: its iterations)
    for (bool first = true;; first = false) {
        int left_in_block = f.checks ? f.nchk : f.niter + 1;   // iterations to the next check
        int nchecks = 0, nd = 0, done = DONE_RUNNING;          // checks posted, decided
        bool stop = false;
        // every pass is one iteration (a step after the first begins with an
        // exchange alone); with checks the judge's decision ends it within itmax
        // iterations (plus those run before the decision arrives)
        for (int k = first ? 0 : -1; !stop && (f.checks || k < f.niter); ++k) {
            const unsigned long long word = f.checks && lane == 0 ? *ctl : 0ull;   // read now, looked at after the iteration
            if (k >= 0) {
                if (left_in_block == 1) iteration(std::true_type{});
                else iteration(std::false_type{});
            }
            const int par = (k + 1) & 1;
            const unsigned tag = base + (unsigned)k + 1u;
            // publish the edges, first of all
            if (below && upd) flow_store(hy(par, w, 0), H[0], tag);
            if (above && upd) flow_store(hy(par, w, 1), H[R - 1], tag);
            if (putx) {
                uint4* const o = hx(par, w, lane == 1 ? 0 : 1);
#pragma unroll
                for (int q = 0; q < R; ++q) flow_store(o + q, H[q], tag);
            }
            if (f.checks) decided(word, nd, done);
            if (k >= 0 && --left_in_block == 0) {
                left_in_block = f.nchk;
                // the snapshot of two checks ago is given up: its decision must be known
                for (int wait = f.wait; nd < nchecks - 1 && done == DONE_RUNNING; --wait) {
                    decided(lane == 0 ? *ctl : 0ull, nd, done);
                    if (wait == 0) done = FLOW_TIMEOUT;
                }
                if (done == DONE_RUNNING) {
                    snapshot((flip + nchecks + 1) & 1);
                    const double v = a.norm_max ? __longlong_as_double((long long)warp_max_u64(pmax)) : warp_sum(part);
                    if (lane == 0) flow_store(f.parts + (size_t)(nchecks & 1) * f.nwarps + w, v, base + (unsigned)nchecks + 1u);
                    nchecks += 1;
                    part = 0.0;
                    pmax = 0ull;
                }
            }
            stop = done != DONE_RUNNING;
            if (!f.checks && k == f.niter - 1) break;
            // the neighbours' edges of the same iteration
            bool ok = stop;
            for (int wait = f.wait; !ok; --wait) {
                uint4 vb = make_uint4(0, tag, 0, tag), vt = vb, vx[R];
                if (gety_b) vb = flow_load(hy(par, w - f.ntx, 1));
                if (gety_t) vt = flow_load(hy(par, w + f.ntx, 0));
                bool here = true;
                if (getx) {
                    const uint4* const src = hx(par, lane == 0 ? w - 1 : w + 1, lane == 0 ? 1 : 0);
#pragma unroll
                    for (int q = 0; q < R; ++q) vx[q] = flow_load(src + q);
#pragma unroll
                    for (int q = 0; q < R; ++q) here = here && flow_ready(vx[q], tag);
                }
                here = here && flow_ready(vb, tag) && flow_ready(vt, tag);
                ok = __all_sync(FULL, here);
                if (ok) {
                    if (gety_b) Hb = flow_value(vb);
                    if (gety_t) Ht = flow_value(vt);
                    if (getx) {
#pragma unroll
                        for (int q = 0; q < R; ++q) {
                            if (lane == 0) H[q] = flow_value(vx[q]);
                            else sHr[q] = flow_value(vx[q]);   // (read by this lane alone)
                        }
                    }
                } else {
                    // a neighbour may have left: the step has stopped
                    if (f.checks) decided(lane == 0 ? *ctl : 0ull, nd, done);
                    if (wait == 0) done = FLOW_TIMEOUT;
                    if (done != DONE_RUNNING) {
                        stop = true;
                        break;
                    }
                }
            }
            if (done == FLOW_TIMEOUT && lane == 0) f.st->pad = 1;
        }
        if (!f.checks) {
            snapshot(1);
            return;
        }
        flip = (flip + nd) & 1;
        if (done == DONE_CONVERGED || done == DONE_NAN || done == FLOW_NEXT) restore(flip);
        if (done != FLOW_NEXT) break;
        base += flow_tags(nd * f.nchk, f.nchk);
        part = 0.0;
        pmax = 0ull;
    }
    // Hold of the next step (a step stopped by itmax goes on from its own)
    double* const Od = static_cast<double*>(const_cast<void*>(a.Hold));
#pragma unroll
    for (int q = 0; q < R; ++q)
        if (upd && j0 + q <= ny - 2) Od[at(j0 + q) + ic] = sHo[q][lane];
}

template <int MODEL>
const void* flow_kernel_of(int rows)
{
    switch (rows) {
    case 1: return (const void*)pt2d_flow_kernel<MODEL, 1>;
    case 2: return (const void*)pt2d_flow_kernel<MODEL, 2>;
    case 3: return (const void*)pt2d_flow_kernel<MODEL, 3>;
    case 4: return (const void*)pt2d_flow_kernel<MODEL, 4>;
    case 5: return (const void*)pt2d_flow_kernel<MODEL, 5>;
    }
    if constexpr (MODEL == LIN)
        if (rows == 6) return (const void*)pt2d_flow_kernel<MODEL, 6>;
    return nullptr;
}

}  // namespace ptd
