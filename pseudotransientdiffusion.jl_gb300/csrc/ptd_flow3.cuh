// ptd_flow3.cuh -- whole physical steps of a 3D grid (native FP64) in one
// launch: the scheme of ptd_flow.cuh with a warp owning a tile of 31 columns x
// RY rows x RZ planes and exchanging edges with six neighbours.
//
// The arithmetic is pt3d_body's, operation for operation: the same bits.
//
// Bound by the FP64 pipe (16 instructions per row of 1 x 2 tiles, 13 without
// the faces that two tiles evolve) and, on small grids, by the latency of an
// iteration.  us per iteration with checks every 10, one launch per iteration
// / here: NONLIN 32^3 5.1, 3.4; 48^3 9.9, 7.2; 64^3 13.3, 11.9; LINSTEP 32^3
// 5.0, 3.1; 64^3 13.8, 11.2; LIN 32^3 4.3, 2.7; 64^3 11.5, 9.7; 62x72x66 14.0,
// 11.4.  (With 2 x 2 tiles, whose code of 16 faces is twice as long, NONLIN
// 64^3 took 15.8; with each look's loads stored before the next was issued
// 32^3 took 4.3.)
#pragma once

#include "ptd_flow.cuh"

namespace ptd {

template <int MODEL, int RY, int RZ, int W>
__global__ void __launch_bounds__(32 * W, 1) pt3d_flow_kernel(PTArgs a, FlowArgs f)
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
    const int tx = w % f.ntx, ty = w / f.ntx % f.nty, tz = w / (f.ntx * f.nty), ntz = f.nwarps / (f.ntx * f.nty);
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int i = 31 * tx + lane, ic = min(i, nx - 1), ir = min(i + 1, nx - 1);
    const int j0 = 1 + ty * RY, k0 = 1 + tz * RZ;
    const bool xface = i <= nx - 2, upd = i >= 1 && i <= nx - 2 && lane >= 1;
    const bool own_x = xface && (lane >= 1 || tx == 0);
    const bool left = tx > 0, right = tx < f.ntx - 1, front = ty > 0, back = ty < f.nty - 1;   // neighbours in x, y
    const bool below = tz > 0, above = tz < ntz - 1;                                            // in z
    const long long sy = a.sy, sz = a.sz;
    volatile unsigned long long* const ctl = f.ctl + 16 * blockIdx.x;
    auto at = [&](int j, int k) { return (long long)min(k, nz - 1) * sz + (long long)min(j, ny - 1) * sy; };
    auto inner = [&](int q, int p) { return j0 + q <= ny - 2 && k0 + p <= nz - 2; };   // uniform over the warp

    // the tile: rows past ny-2 and planes past nz-2 hold the boundary and never
    // change; in shared memory what does not change in a step, the column right
    // of the tile (read by lane 31), and H of the rows and planes around it
    __shared__ double s_Ho[W][RZ][RY][32], s_Hr[W][RZ][RY];
    __shared__ double s_D[HASD ? W : 1][RZ + 2][RY + 2][32], s_Dr[HASD ? W : 1][RZ][RY];
    __shared__ float s_E[MODEL == LINSTEP ? W : 1][RZ][RY][32];
    double(*const sHo)[RY][32] = s_Ho[threadIdx.y];
    double(*const sHr)[RY] = s_Hr[threadIdx.y];
    double(*const sD)[RY + 2][32] = s_D[HASD ? threadIdx.y : 0];   // rows j0-1 .. j0+RY, planes k0-1 .. k0+RZ
    double(*const sDr)[RY] = s_Dr[HASD ? threadIdx.y : 0];
    float(*const sE)[RY][32] = s_E[MODEL == LINSTEP ? threadIdx.y : 0];
    __shared__ double s_Hh[W][2 * (RZ + RY)][32];
    double(*const Hf)[32] = s_Hh[threadIdx.y];
    double(*const Hk)[32] = Hf + RZ;
    double(*const Hb)[32] = Hk + RZ;
    double(*const Ht)[32] = Hb + RY;
    double H[RZ][RY], wx[RZ][RY], wy[RZ][RY], wz[RZ][RY], wyf[RZ], wzb[RY];
    if constexpr (HASD) {
#pragma unroll
        for (int p = -1; p <= RZ; ++p)
#pragma unroll
            for (int q = -1; q <= RY; ++q) sD[p + 1][q + 1][lane] = ld<N>(a.D, at(j0 + q, k0 + p) + ic);
    }
#pragma unroll
    for (int p = 0; p < RZ; ++p) {
#pragma unroll
        for (int q = 0; q < RY; ++q) {
            const long long row = at(j0 + q, k0 + p);
            H[p][q] = N::ldh(a.Hin, row + ic);
            wx[p][q] = ld<N>(a.win[0], row + ic);
            wy[p][q] = ld<N>(a.win[1], row + ic);
            wz[p][q] = ld<N>(a.win[2], row + ic);
            sHo[p][q][lane] = N::ldo(a.Hold, row + ic);
            if (lane == 31) sHr[p][q] = N::ldh(a.Hin, row + ir);
            if constexpr (HASD) {
                const double dr = ld<N>(a.D, row + ir);
                if (lane == 31) sDr[p][q] = dr;
                if (MODEL == LINSTEP) {
                    const float dl = N::lo_f(ld<N>(a.D, row + max(ic - 1, 0)));
                    const float dy = fmaxf(N::lo_f(sD[p + 1][q][lane]), N::lo_f(sD[p + 1][q + 2][lane]));
                    const float dz = fmaxf(N::lo_f(sD[p][q + 1][lane]), N::lo_f(sD[p + 2][q + 1][lane]));
                    sE[p][q][lane] = linstep_cell_e(a.f, fmaxf(fmaxf(fmaxf(N::lo_f(sD[p + 1][q + 1][lane]), dl),
                                                                     N::lo_f(dr)), fmaxf(dy, dz)));
                }
            }
        }
        Hf[p][lane] = N::ldh(a.Hin, at(j0 - 1, k0 + p) + ic);
        Hk[p][lane] = N::ldh(a.Hin, at(j0 + RY, k0 + p) + ic);
        wyf[p] = ld<N>(a.win[1], at(j0 - 1, k0 + p) + ic);
    }
#pragma unroll
    for (int q = 0; q < RY; ++q) {
        Hb[q][lane] = N::ldh(a.Hin, at(j0 + q, k0 - 1) + ic);
        Ht[q][lane] = N::ldh(a.Hin, at(j0 + q, k0 + RZ) + ic);
        wzb[q] = ld<N>(a.win[2], at(j0 + q, k0 - 1) + ic);
    }
    __syncwarp();

    // the slots of a tile's edges: y [front, back][plane][lane], z [below, above][row][lane], x [left, right][plane][row]
    auto hy = [&](int par, int tile, int side) { return f.halo_y + (((size_t)par * f.nwarps + tile) * 2 + side) * RZ * 32 + lane; };
    auto hz = [&](int par, int tile, int side) { return f.halo_z + (((size_t)par * f.nwarps + tile) * 2 + side) * RY * 32 + lane; };
    auto hx = [&](int par, int tile, int side) { return f.halo_x + (((size_t)par * f.nwarps + tile) * 2 + side) * RZ * RY; };
    const bool getx = (lane == 0 && left) || (lane == 31 && right);
    const bool putx = (lane == 1 && left) || (lane == 31 && right);

    // the tile's cells and faces in the buffers of parity par: stored (with
    // the faces that the neighbours own, in buffers of this warp), and read
    // back by the threads that stored them
    auto buf = [&](const void* in, void* out, int par) { return static_cast<double*>(par ? out : const_cast<void*>(in)); };
    auto edge_x = [&](int par) { return f.edge_x + ((size_t)par * f.nwarps + w) * RZ * RY; };
    auto edge_y = [&](int par) { return f.edge_y + ((size_t)par * f.nwarps + w) * RZ * 32 + lane; };
    auto edge_z = [&](int par) { return f.edge_z + ((size_t)par * f.nwarps + w) * RY * 32 + lane; };
    auto snapshot = [&](int par) {
        double *const Hd = buf(a.Hin, a.Hout, par), *const X = buf(a.win[0], a.wout[0], par),
               *const Y = buf(a.win[1], a.wout[1], par), *const Z = buf(a.win[2], a.wout[2], par);
#pragma unroll
        for (int p = 0; p < RZ; ++p) {
            if (f.checks) edge_y(par)[32 * p] = wyf[p];
            if (ty == 0 && upd && k0 + p <= nz - 2) Y[at(0, k0 + p) + ic] = wyf[p];
#pragma unroll
            for (int q = 0; q < RY; ++q) {
                if (inner(q, p)) {
                    const long long c = at(j0 + q, k0 + p) + ic;
                    if (own_x) X[c] = wx[p][q];
                    else if (f.checks && lane == 0) edge_x(par)[p * RY + q] = wx[p][q];
                    if (upd) {
                        Y[c] = wy[p][q];
                        Z[c] = wz[p][q];
                        Hd[c] = H[p][q];
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < RY; ++q) {
            if (f.checks) edge_z(par)[32 * q] = wzb[q];
            if (tz == 0 && upd && j0 + q <= ny - 2) Z[at(j0 + q, 0) + ic] = wzb[q];
        }
    };
    auto restore = [&](int par) {
        const double *const Hd = buf(a.Hin, a.Hout, par), *const X = buf(a.win[0], a.wout[0], par),
                     *const Y = buf(a.win[1], a.wout[1], par), *const Z = buf(a.win[2], a.wout[2], par);
#pragma unroll
        for (int p = 0; p < RZ; ++p) {
            wyf[p] = __ldcg(edge_y(par) + 32 * p);
#pragma unroll
            for (int q = 0; q < RY; ++q) {
                if (inner(q, p)) {
                    const long long c = at(j0 + q, k0 + p) + ic;
                    if (own_x) wx[p][q] = __ldcg(X + c);
                    else if (lane == 0) wx[p][q] = __ldcg(edge_x(par) + p * RY + q);
                    if (upd) {
                        wy[p][q] = __ldcg(Y + c);
                        wz[p][q] = __ldcg(Z + c);
                        H[p][q] = __ldcg(Hd + c);
                        sHo[p][q][lane] = H[p][q];   // the next step's Hold
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < RY; ++q) wzb[q] = __ldcg(edge_z(par) + 32 * q);
    };

    double part = 0.0;
    unsigned long long pmax = 0ull;
    // one iteration from the halos in place: a row's cells are updated once
    // their faces are known; the rows behind and above still hold the old H
    auto iteration = [&](auto chk) {
        constexpr bool C = decltype(chk)::value;
        double wzl[RY], uzl[C ? RY : 1];   // new faces below the plane
#pragma unroll
        for (int q = 0; q < RY; ++q) {
            double u = 0.0;
            const double Hbq = Hb[q][lane];
            wzb[q] = face_t<N, MODEL, C>(a, Hbq, H[0][q], N::hf(Hbq) + N::hf(H[0][q]), HASD ? sD[0][q + 1][lane] : 0.0,
                                         HASD ? sD[1][q + 1][lane] : 0.0, wzb[q], u);
            wzl[q] = wzb[q];
            if (C) uzl[q] = u;
        }
#pragma unroll
        for (int p = 0; p < RZ; ++p) {
            double uyl = 0.0, Hcur = H[p][0];
            float hc = N::hf(Hcur);
            const double Hfp = Hf[p][lane];
            wyf[p] = face_t<N, MODEL, C>(a, Hfp, Hcur, N::hf(Hfp) + hc, HASD ? sD[p + 1][0][lane] : 0.0,
                                         HASD ? sD[p + 1][1][lane] : 0.0, wyf[p], uyl);
            double wyl = wyf[p];
#pragma unroll
            for (int q = 0; q < RY; ++q) {
                const double Hbk = q < RY - 1 ? H[p][q + 1 < RY ? q + 1 : q] : Hk[p][lane];
                const double Hup = p < RZ - 1 ? H[p + 1 < RZ ? p + 1 : p][q] : Ht[q][lane];
                const double Dc = HASD ? sD[p + 1][q + 1][lane] : 0.0;
                const float hk = N::hf(Hbk);
                double Hright = N::shfl_down(Hcur, 1);
                float hr = __shfl_down_sync(FULL, hc, 1);
                if (lane == 31) {
                    Hright = sHr[p][q];
                    hr = N::hf(Hright);
                }
                const double Drt = HASD ? N::shfl_down(Dc, 1) : 0.0;
                double ux = 0.0, uy = 0.0, uz = 0.0;
                if (xface)
                    wx[p][q] = face_t<N, MODEL, C>(a, Hcur, Hright, hc + hr, Dc, HASD && lane == 31 ? sDr[p][q] : Drt,
                                                   wx[p][q], ux);
                const double wyn = face_t<N, MODEL, C>(a, Hcur, Hbk, hc + hk, Dc, HASD ? sD[p + 1][q + 2][lane] : 0.0,
                                                       wy[p][q], uy);
                const double wzn = face_t<N, MODEL, C>(a, Hcur, Hup, hc + N::hf(Hup), Dc, HASD ? sD[p + 2][q + 1][lane] : 0.0,
                                                       wz[p][q], uz);
                const double wxl = N::shfl_up(wx[p][q], 1), uxl = C ? N::shfl_up(ux, 1) : 0.0;
                if (upd && inner(q, p)) {
                    wy[p][q] = wyn;
                    wz[p][q] = wzn;
                    const double dx = N::sub(wx[p][q], wxl), dy = N::sub(wyn, wyl), dz = N::sub(wzn, wzl[q]);
                    const double Ho = sHo[p][q][lane];
                    float e = a.fe_lin;
                    if (MODEL == LINSTEP) e = sE[MODEL == LINSTEP ? p : 0][q][lane];
                    if (MODEL == NONLIN) e = cell_e<MODEL>(a, hc, 0.0f);
                    const double Hn =
                        a.sq ? h_update_sq<N>(a, Hcur, Ho, N::add(N::add(dz, dy), dx), e)
                             : h_update<N>(a, Hcur, Ho, N::mad(dz, cst<N>(a, 2), N::mad(dy, cst<N>(a, 1), N::mul(dx, cst<N>(a, 0)))), e);
                    if (C) {
                        const double divu = N::mad(N::sub(uz, uzl[C ? q : 0]), cst<N>(a, 2),
                                                   N::mad(N::sub(uy, uyl), cst<N>(a, 1), N::mul(N::sub(ux, uxl), cst<N>(a, 0))));
                        accumulate_residual(N::sub(divu, N::mul(N::hdn(Hn, Ho), cst<N>(a, 3))), part, pmax);
                    }
                    H[p][q] = Hn;
                }
                wyl = wyn;
                wzl[q] = wzn;
                if (C) {
                    uyl = uy;
                    uzl[C ? q : 0] = uz;
                }
                Hcur = Hbk;
                hc = hk;
            }
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
#pragma unroll
            for (int p = 0; p < RZ; ++p) {
                if (front && upd) flow_store(hy(par, w, 0) + 32 * p, H[p][0], tag);
                if (back && upd) flow_store(hy(par, w, 1) + 32 * p, H[p][RY - 1], tag);
            }
#pragma unroll
            for (int q = 0; q < RY; ++q) {
                if (below && upd) flow_store(hz(par, w, 0) + 32 * q, H[0][q], tag);
                if (above && upd) flow_store(hz(par, w, 1) + 32 * q, H[RZ - 1][q], tag);
            }
            if (putx) {
                uint4* const o = hx(par, w, lane == 1 ? 0 : 1);
#pragma unroll
                for (int p = 0; p < RZ; ++p)
#pragma unroll
                    for (int q = 0; q < RY; ++q) flow_store(o + p * RY + q, H[p][q], tag);
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
                // (all loads first: what follows one waits for it)
                uint4 vf[RZ], vk[RZ], vb[RY], vt[RY], vx[RZ][RY];
#pragma unroll
                for (int p = 0; p < RZ; ++p) {
                    vf[p] = vk[p] = make_uint4(0, tag, 0, tag);
                    if (front && upd) vf[p] = flow_load(hy(par, w - f.ntx, 1) + 32 * p);
                    if (back && upd) vk[p] = flow_load(hy(par, w + f.ntx, 0) + 32 * p);
                }
#pragma unroll
                for (int q = 0; q < RY; ++q) {
                    vb[q] = vt[q] = make_uint4(0, tag, 0, tag);
                    if (below && upd) vb[q] = flow_load(hz(par, w - f.ntx * f.nty, 1) + 32 * q);
                    if (above && upd) vt[q] = flow_load(hz(par, w + f.ntx * f.nty, 0) + 32 * q);
                }
                bool here = true;
                if (getx) {
                    const uint4* const src = hx(par, lane == 0 ? w - 1 : w + 1, lane == 0 ? 1 : 0);
#pragma unroll
                    for (int p = 0; p < RZ; ++p)
#pragma unroll
                        for (int q = 0; q < RY; ++q) vx[p][q] = flow_load(src + p * RY + q);
#pragma unroll
                    for (int p = 0; p < RZ; ++p)
#pragma unroll
                        for (int q = 0; q < RY; ++q) here = here && flow_ready(vx[p][q], tag);
                }
#pragma unroll
                for (int p = 0; p < RZ; ++p) here = here && flow_ready(vf[p], tag) && flow_ready(vk[p], tag);
#pragma unroll
                for (int q = 0; q < RY; ++q) here = here && flow_ready(vb[q], tag) && flow_ready(vt[q], tag);
                ok = __all_sync(FULL, here);
                if (ok) {
#pragma unroll
                    for (int p = 0; p < RZ; ++p) {
                        if (front && upd) Hf[p][lane] = flow_value(vf[p]);
                        if (back && upd) Hk[p][lane] = flow_value(vk[p]);
                    }
#pragma unroll
                    for (int q = 0; q < RY; ++q) {
                        if (below && upd) Hb[q][lane] = flow_value(vb[q]);
                        if (above && upd) Ht[q][lane] = flow_value(vt[q]);
                    }
                    if (getx) {
#pragma unroll
                        for (int p = 0; p < RZ; ++p)
#pragma unroll
                            for (int q = 0; q < RY; ++q) {
                                if (lane == 0) H[p][q] = flow_value(vx[p][q]);
                                else sHr[p][q] = flow_value(vx[p][q]);   // (read by this lane alone)
                            }
                    }
                }
                if (!ok) {
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
    for (int p = 0; p < RZ; ++p)
#pragma unroll
        for (int q = 0; q < RY; ++q)
            if (upd && inner(q, p)) Od[at(j0 + q, k0 + p) + ic] = sHo[p][q][lane];
}

template <int MODEL>
const void* flow3_kernel_of(int ry, int rz, int warps)
{
    if (ry == 1 && rz == 1) return (const void*)pt3d_flow_kernel<MODEL, 1, 1, 20>;
    if (ry == 1 && rz == 2 && warps <= 20) return (const void*)pt3d_flow_kernel<MODEL, 1, 2, 20>;
    if (ry == 1 && rz == 2) return (const void*)pt3d_flow_kernel<MODEL, 1, 2, 28>;
    if constexpr (MODEL == LIN)
        if (ry == 2 && rz == 2) return (const void*)pt3d_flow_kernel<MODEL, 2, 2, 16>;
    return nullptr;
}

}  // namespace ptd
