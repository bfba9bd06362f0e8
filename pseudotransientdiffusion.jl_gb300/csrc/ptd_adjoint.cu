// ptd_adjoint.cu -- discrete adjoint of the implicit PT solve (3D, D = exp(m) H^3
// or D = H^3): gradient of L = 1/2 sum_inner (H^nt - H_target)^2 with respect
// to the per-cell log-coefficient m and the initial state H0.
//
// No reference counterpart (the reference has no adjoint); this is new work
// checked against central finite differences and the CPU FP64 reference
// adjoint of oracle/ptd_oracle.c.
//
// Per physical step n = nt..1 the forward residual is (scaled as in
// ptd_device.cuh) F_i = (H_i - Hold_i)/dt - sum_d sigma_d (u_{i+1/2} - u_{i-1/2}),
// u_f = K_f (H_R - H_L), K_f = (E_L + E_R) s^3, s = H_L + H_R, E = exp(m).
// The adjoint state solves J^T lam = g with J = dF/dH at the converged H^n:
//   (J^T lam)_j = lam_j/dt + sum_d sigma_d [ (w_{j+1/2} - w_{j-1/2})      -- symmetric part,
//                                            + (n_{j+1/2} + n_{j-1/2}) ]   -- transposed Newton term
// with v_f = lam_R - lam_L, w_f -> -K_f v_f (damped exactly like the forward
// flux) and n_f = 3 (E_L+E_R) s^2 (H_R - H_L) v_f (the 3H^2 derivative of
// D = H^3, transposed).  The transposed stencil is iterated with the same
// accelerated PT scheme and parameters as the forward (one fused kernel per
// iteration, z-march, device-side checks), then
//   dL/dm_j  -= sum_{f ∋ j} sigma v_f E_j s^3 (H_R - H_L)
//   dL/dH0_b -= sum_{f ∋ b} sigma v_f du_f/dH_b      (boundary cells: frozen at H0)
//   g <- lam / dt                                    (dL/dH^{n-1})
// and after step 1 dL/dH0 (inner cells) = g.  The forward keeps one FP64
// checkpoint of H per physical step; the adjoint sweep needs no recomputation.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "ptd_internal.h"
#include "ptd_pt_body.cuh"

namespace ptd {

struct AdjArgs {
    int nx, ny, nz;
    long long sy, sz;
    double rdt;
    double sig[3];
    float2 rdt_df;
    float2 sig_df[3];
    FParams f;
    const void* lin;    // lam (iteration k)
    void* lout;         // lam (iteration k+1)
    const void* win[3];
    void* wout[3];
    const void* H;      // H^n (frozen, number type of the kernel)
    const void* E;      // exp(m) (number type of the kernel); NULL for D = H^3
    const void* g;      // right-hand side (rebased form: minus the base update residual)
    const int* done;
    double* acc;
    double* parts;      // check-residual slots, one per CTA (summed in a fixed order by the judge)
    // rebased FP32 form (precision FP32_RB): the adjoint PT iteration on the
    // change since an FP64 base (lam_b, w_b), see ptd_rb.cu for the scheme
    float rdtf;
    float sigf[3];
    const void* tb[3];  // base flux defect w_b + K v_b per face (FP32)
    const double* Cb;   // base check residual (FP64)
};

// FP32 number type of the rebased adjoint iteration (ptd_num.cuh interface).
struct F32 {
    using T = float;
    static constexpr bool native = true;
    __device__ static __forceinline__ T add(T a, T b) { return a + b; }
    __device__ static __forceinline__ T sub(T a, T b) { return a - b; }
    __device__ static __forceinline__ T mul(T a, T b) { return a * b; }
    __device__ static __forceinline__ T mad(T a, T b, T c) { return fmaf(a, b, c); }
    __device__ static __forceinline__ float lo_f(T a) { return a; }
    __device__ static __forceinline__ double to_d(T a) { return f2d_exact(a); }
    __device__ static __forceinline__ T zero() { return 0.0f; }
    __device__ static __forceinline__ T shfl_down(T v, int d) { return __shfl_down_sync(0xffffffffu, v, d); }
    __device__ static __forceinline__ T shfl_up(T v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
};
__device__ __forceinline__ float nmadf(F32, float c, float t, float w) { return fmaf(-c, t, w); }

// done: 1 converged (err <= target), 2 itmax, 3 stalled at an arithmetic
// floor below the acceptable level (err <= accept, no 1 % improvement over
// `stall` checks)
struct AdjState {
    int done, nchecks, iter, best_at;
    int blocks, pad;    // check blocks run by the solve graph
    double acc, err, target, accept, best;
};

template <class N>
__device__ __forceinline__ typename N::T acst(const AdjArgs& a, int which);
template <>
__device__ __forceinline__ double acst<F64>(const AdjArgs& a, int which)
{
    return which < 3 ? a.sig[which] : a.rdt;
}
template <>
__device__ __forceinline__ float2 acst<DF64>(const AdjArgs& a, int which)
{
    return which < 3 ? a.sig_df[which] : a.rdt_df;
}
template <>
__device__ __forceinline__ float acst<F32>(const AdjArgs& a, int which)
{
    return which < 3 ? a.sigf[which] : a.rdtf;
}

// One adjoint face: damped symmetric flux, and the Newton-transpose value n.
// kv = K v (undamped, for the check).  DELTA: the rebased form, whose flux
// relaxes towards -(t_b + K v) (t_b: the base flux defect).
template <class N, bool EXPM, bool U, bool DELTA = false>
__device__ __forceinline__ typename N::T adj_face(const AdjArgs& a, typename N::T HL, typename N::T HR, float hsum,
                                                  typename N::T EL, typename N::T ER, typename N::T lL,
                                                  typename N::T lR, typename N::T w, typename N::T& n,
                                                  typename N::T& kv, typename N::T tb = typename N::T())
{
    using T = typename N::T;
    const T v = N::sub(lR, lL);
    const T s = N::add(HL, HR);
    const T s2 = N::mul(s, s);
    T K = N::mul(s2, s);
    T Kp = N::add(N::add(s2, s2), s2);   // K' = 3 s^2 (times E_L + E_R)
    float efac = 1.0f;
    if (EXPM) {
        const T e2 = N::add(EL, ER);
        K = N::mul(K, e2);
        Kp = N::mul(Kp, e2);
        efac = 0.5f * N::lo_f(e2);
    } else {
        // D = H^3 is the EXPM form with E = 1: (E_L + E_R) = 2, kappa 1/16
        K = N::add(K, K);
        Kp = N::add(Kp, Kp);
    }
    n = N::mul(N::mul(Kp, N::sub(HR, HL)), v);
    const T kvv = N::mul(K, v);
    if (U) kv = kvv;
    const float c = nonlin_face_c(a.f, hsum, efac);
    if (DELTA) return nmadf(N(), c, N::add(N::add(w, tb), kvv), w);
    return nmadf(N(), c, N::add(w, kvv), w);
}

template <class N, bool EXPM, bool CHECK, int R, bool DELTA = false>
__global__ void __launch_bounds__(32 * R) adj3d_kernel(const AdjArgs* __restrict__ ap, int chunk)
{
    using T = typename N::T;
    const AdjArgs a = *ap;   // (written by the host before the solve)
    pdl_begin();
    if (step_done(a.done)) return;
    __shared__ T sL[2][R][32];     // lam of the plane
    __shared__ T sH[2][R][32];     // H of the plane
    __shared__ T sE[EXPM ? 2 : 1][EXPM ? R : 1][32];
    __shared__ T sW[2][R][32];     // y faces: damped flux
    __shared__ T sN[2][R][32];     // y faces: Newton-transpose value
    __shared__ T sK[CHECK ? 2 : 1][CHECK ? R : 1][32];

    const int lane = threadIdx.x, r = threadIdx.y;
    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int i = 31 * blockIdx.x + lane;
    const int j = (R - 1) * blockIdx.y + r;
    const int k0 = 1 + blockIdx.z * chunk;
    const int k1 = min(k0 + chunk, nz - 1);
    double part = 0.0;
    unsigned long long pmax = 0ull;
    if (k0 < k1) {
        const int ic = min(i, nx - 1), jc = min(j, ny - 1);
        const bool inner_x = i >= 1 && i <= nx - 2, inner_y = j >= 1 && j <= ny - 2;
        const bool xface = i <= nx - 2 && inner_y && r >= 1;
        const bool yface = j <= ny - 2 && inner_x;
        const bool upd = inner_x && inner_y && lane >= 1 && r >= 1;
        const bool own_x = xface && (lane >= 1 || blockIdx.x == 0);
        const bool own_y = yface && lane >= 1 && (r >= 1 || blockIdx.y == 0);
        const bool top = r == R - 1, up_ok = jc + 1 < ny;
        const long long sy = a.sy, sz = a.sz;
        long long idx = (long long)k0 * sz + (long long)jc * sy + ic;
        T lc = ld<N>(a.lin, idx), Hc = ld<N>(a.H, idx);
        T Ec = EXPM ? ld<N>(a.E, idx) : N::zero();
        float hc = N::lo_f(Hc);
        T wzb = N::zero(), nzb = N::zero(), kzb = N::zero();
        if (upd) {
            const T lb = ld<N>(a.lin, idx - sz), Hb = ld<N>(a.H, idx - sz);
            const T Eb = EXPM ? ld<N>(a.E, idx - sz) : N::zero();
            wzb = adj_face<N, EXPM, CHECK, DELTA>(a, Hb, Hc, N::lo_f(Hb) + hc, Eb, Ec, lb, lc,
                                                  ld<N>(a.win[2], idx - sz), nzb, kzb,
                                                  DELTA ? ld<N>(a.tb[2], idx - sz) : N::zero());
            if (k0 == 1) st<N>(a.wout[2], idx - sz, wzb);
        }
        int p = 0;
        sL[0][r][lane] = lc;
        sH[0][r][lane] = Hc;
        if (EXPM) sE[0][r][lane] = Ec;
        __syncthreads();
        for (int k = k0; k < k1; ++k, idx += sz) {
            const T ln = ld<N>(a.lin, idx + sz), Hn = ld<N>(a.H, idx + sz);
            const T En = EXPM ? ld<N>(a.E, idx + sz) : N::zero();
            const T wx = ld<N>(a.win[0], idx), wy = ld<N>(a.win[1], idx), wz = ld<N>(a.win[2], idx);
            const T gg = ld<N>(a.g, idx);
            const T tbx = DELTA ? ld<N>(a.tb[0], idx) : N::zero();
            const T tby = DELTA ? ld<N>(a.tb[1], idx) : N::zero();
            const T tbz = DELTA ? ld<N>(a.tb[2], idx) : N::zero();
            T lu, Hu, Eu = N::zero();
            if (!top) {
                lu = sL[p][r + 1][lane];
                Hu = sH[p][r + 1][lane];
                if (EXPM) Eu = sE[p][r + 1][lane];
            } else {
                lu = up_ok ? ld<N>(a.lin, idx + sy) : lc;
                Hu = up_ok ? ld<N>(a.H, idx + sy) : Hc;
                if (EXPM) Eu = up_ok ? ld<N>(a.E, idx + sy) : Ec;
            }
            T lr = N::shfl_down(lc, 1), Hr = N::shfl_down(Hc, 1);
            T Er = EXPM ? N::shfl_down(Ec, 1) : N::zero();
            if (lane == 31) {
                const bool ok = ic + 1 < nx;
                lr = ok ? ld<N>(a.lin, idx + 1) : lc;
                Hr = ok ? ld<N>(a.H, idx + 1) : Hc;
                if (EXPM) Er = ok ? ld<N>(a.E, idx + 1) : Ec;
            }
            T nx_ = N::zero(), ny_ = N::zero(), nz_ = N::zero();
            T kx = N::zero(), ky = N::zero(), kz = N::zero();
            T wxn = N::zero(), wyn = N::zero(), wzn = N::zero();
            if (xface)
                wxn = adj_face<N, EXPM, CHECK, DELTA>(a, Hc, Hr, hc + N::lo_f(Hr), Ec, Er, lc, lr, wx, nx_, kx, tbx);
            if (yface)
                wyn = adj_face<N, EXPM, CHECK, DELTA>(a, Hc, Hu, hc + N::lo_f(Hu), Ec, Eu, lc, lu, wy, ny_, ky, tby);
            if (upd)
                wzn = adj_face<N, EXPM, CHECK, DELTA>(a, Hc, Hn, hc + N::lo_f(Hn), Ec, En, lc, ln, wz, nz_, kz, tbz);
            if (own_x) st<N>(a.wout[0], idx, wxn);
            if (own_y) st<N>(a.wout[1], idx, wyn);
            if (upd) st<N>(a.wout[2], idx, wzn);
            const T wxl = N::shfl_up(wxn, 1), nxl = N::shfl_up(nx_, 1);
            const T kxl = CHECK ? N::shfl_up(kx, 1) : N::zero();
            sW[p][r][lane] = wyn;
            sN[p][r][lane] = ny_;
            if (CHECK) sK[p][r][lane] = ky;
            sL[p ^ 1][r][lane] = ln;
            sH[p ^ 1][r][lane] = Hn;
            if (EXPM) sE[p ^ 1][r][lane] = En;
            __syncthreads();
            if (upd) {
                const T wyb = sW[p][r - 1][lane], nyb = sN[p][r - 1][lane];
                const float e = nonlin_cell_e<true>(a.f, hc, EXPM ? N::lo_f(Ec) : 1.0f);
                // sum_d sigma_d [(w_+ - w_-) + (n_+ + n_-)]
                T div = N::mul(N::add(N::sub(wxn, wxl), N::add(nx_, nxl)), acst<N>(a, 0));
                div = N::mad(N::add(N::sub(wyn, wyb), N::add(ny_, nyb)), acst<N>(a, 1), div);
                div = N::mad(N::add(N::sub(wzn, wzb), N::add(nz_, nzb)), acst<N>(a, 2), div);
                const T A = N::sub(N::mad(lc, acst<N>(a, 3), div), gg);
                const T lnew = nmadf(N(), e, A, lc);
                st<N>(a.lout, idx, lnew);
                if (CHECK) {
                    const T kyb = sK[p][r - 1][lane];
                    // R = g - lam rdt + sum sigma [(kv_+ - kv_-) - (n_+ + n_-)]
                    T q = N::mul(N::sub(N::sub(kx, kxl), N::add(nx_, nxl)), acst<N>(a, 0));
                    q = N::mad(N::sub(N::sub(ky, kyb), N::add(ny_, nyb)), acst<N>(a, 1), q);
                    q = N::mad(N::sub(N::sub(kz, kzb), N::add(nz_, nzb)), acst<N>(a, 2), q);
                    if (DELTA) {   // C_b + (the same terms of the changes)
                        accumulate_residual(fma(-N::to_d(lnew), a.rdt, a.Cb[idx] + N::to_d(q)), part, pmax);
                    } else {
                        const T res = N::add(N::sub(gg, N::mul(lnew, acst<N>(a, 3))), q);
                        accumulate_residual(N::to_d(res), part, pmax);
                    }
                }
            }
            lc = ln;
            Hc = Hn;
            hc = N::lo_f(Hn);
            if (EXPM) Ec = En;
            wzb = wzn;
            nzb = nz_;
            kzb = kz;
            p ^= 1;
        }
    }
    if (CHECK)
        block_reduce_residual(a.acc, 0, part, pmax, a.parts,
                              ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x);
}

// Gradient accumulation of one step (FP64, one thread per cell of the whole
// grid) and the next right-hand side g = lam/dt.
template <class N, bool EXPM>
__global__ void __launch_bounds__(256) adj_grad_kernel(AdjArgs a, const double* Hn, const double* Ed, double* gm,
                                                       double* gh, void* g_next, long long total_cells)
{
    const long long stp[3] = {1, a.sy, a.sz};
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total_cells;
         t += (long long)gridDim.x * blockDim.x) {
        const long long ix = t % a.nx, iy = (t / a.nx) % a.ny, iz = t / ((long long)a.nx * a.ny);
        const long long c = iz * a.sz + iy * a.sy + ix;
        const long long id[3] = {ix, iy, iz};
        const int n[3] = {a.nx, a.ny, a.nz};
        auto inner = [&](long long cc, int dd, int side) -> bool {
            long long q[3] = {id[0], id[1], id[2]};
            q[dd] += side;
            for (int e = 0; e < 3; ++e)
                if (q[e] < 1 || q[e] > n[e] - 2) return false;
            (void)cc;
            return true;
        };
        const bool ci = inner(c, 0, 0);
        const double lamc = ci ? N::to_d(ld<N>(a.lin, c)) : 0.0;
        double dm = 0.0, dh = 0.0;
        const double Hc = Hn[c];
        const double Ec = EXPM ? Ed[c] : 1.0;
        for (int d = 0; d < 3; ++d) {
            for (int side = -1; side <= 1; side += 2) {
                const long long q[3] = {id[0] + (d == 0 ? side : 0), id[1] + (d == 1 ? side : 0),
                                        id[2] + (d == 2 ? side : 0)};
                if (q[d] < 0 || q[d] > n[d] - 1) continue;
                const long long o = c + side * stp[d];
                // a face exists in the reference only between cells whose
                // other coordinates are inner
                bool face_ok = true;
                for (int e = 0; e < 3; ++e)
                    if (e != d && (id[e] < 1 || id[e] > n[e] - 2)) face_ok = false;
                if (!face_ok) continue;
                const bool oi = inner(o, d, side);
                const double lamo = oi ? N::to_d(ld<N>(a.lin, o)) : 0.0;
                const double Ho = Hn[o];
                const double Eo = EXPM ? Ed[o] : 1.0;
                // orient the face: L = lower index
                const double HL = side > 0 ? Hc : Ho, HR = side > 0 ? Ho : Hc;
                const double lL = side > 0 ? lamc : lamo, lR = side > 0 ? lamo : lamc;
                const double e2 = side > 0 ? Ec + Eo : Eo + Ec;
                const double s = HL + HR, gH = HR - HL, v = lR - lL;
                const double sv = a.sig[d] * v;
                if (EXPM) dm -= sv * Ec * s * s * s * gH;
                if (!ci) {
                    const double K = e2 * s * s * s, Kp = 3.0 * e2 * s * s;
                    const double du = side > 0 ? (-K + Kp * gH) : (K + Kp * gH);   // this cell is L (side>0) or R
                    dh -= sv * du;
                }
            }
        }
        if (EXPM) gm[c] += dm;
        if (!ci) gh[c] += dh;
        // next right-hand side
        if (ci) {
            const double gn = lamc * a.rdt;
            if (N::native) reinterpret_cast<double*>(g_next)[c] = gn;
            else reinterpret_cast<float2*>(g_next)[c] = split_df(gn);
        }
    }
}

__global__ void __launch_bounds__(256) adj_target_kernel(AdjState* st, const double* parts, long long nparts,
                                                         double rtol, double accept_rtol, double norm_den,
                                                         double floor_abs)
{
    const double gn = sqrt(sum_slots(parts, nparts, 0)) / sqrt(norm_den);
    if (threadIdx.x != 0) return;
    st->acc = 0.0;
    st->blocks = 0;
    st->target = fmax(rtol * gn, floor_abs);
    st->accept = fmax(accept_rtol * gn, floor_abs);
    st->done = gn == 0.0 ? 1 : 0;
    st->nchecks = 0;
    st->iter = 0;
    st->err = gn;
    st->best = gn;
    st->best_at = 0;
}

// After each check block: the err from the check launch's slots (fixed
// order); ends the solve graph's loop once the solve has stopped.  Every pass
// of a running solve adds nchk iterations and the solve stops (capped) before
// one would pass itmax, so the loop ends within itmax/nchk + 1 passes.
__global__ void __launch_bounds__(256) adj_judge_kernel(AdjState* st, const double* parts, long long nparts,
                                                        int nchk, int itmax, double norm_den, int stall,
                                                        cudaGraphConditionalHandle loop)
{
    // every thread reads the flag before thread 0 can change it
    pdl_begin();
    const bool idle = st->done != 0;
    __syncthreads();
    if (idle) {   // no PT kernel ran: the slots are stale
        if (threadIdx.x == 0) {
            st->blocks += 1;
            cudaGraphSetConditional(loop, 0);
        }
        return;
    }
    const double acc = sum_slots(parts, nparts, 0);
    if (threadIdx.x != 0) return;
    st->blocks += 1;
    const double err = sqrt(acc) / sqrt(norm_den);
    st->acc = 0.0;
    st->err = err;
    st->nchecks += 1;
    st->iter += nchk;
    if (err < 0.99 * st->best) {
        st->best = err;
        st->best_at = st->nchecks;
    }
    if (!(err > st->target)) st->done = 1;
    else if (err != err) st->done = 2;
    else if (st->nchecks - st->best_at >= stall && err <= st->accept) st->done = 3;
    else if (st->iter + nchk > itmax) st->done = 2;
    if (st->done) cudaGraphSetConditional(loop, 0);
}

// sum over inner cells of v^2 (v as N::T), one slot per CTA.
template <class N>
__global__ void __launch_bounds__(256) adj_sumsq_kernel(const void* v, double* parts, int nx, int ny, int nz,
                                                        long long sy, long long sz)
{
    const long long nix = nx - 2, niy = ny - 2, niz = nz - 2, total = nix * niy * niz;
    double part = 0.0;
    unsigned long long pm = 0ull;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long ix = 1 + t % nix, iy = 1 + (t / nix) % niy, iz = 1 + t / (nix * niy);
        const double x = N::to_d(ld<N>(v, iz * sz + iy * sy + ix));
        part = fma(x, x, part);
    }
    block_reduce_residual(nullptr, 0, part, pm, parts, blockIdx.x);
}

// ---------------------------------------------------------------------------
// Rebased FP32 adjoint (precision FP32_RB).  The adjoint system of a step is
// linear in lam, so the PT iteration runs in FP32 on the change since an FP64
// base (lam_b, w_b) exactly like the forward's rebased form (ptd_rb.cu): the
// FP32 flux relaxes towards -(t_b + K v) with the base flux defect
// t_b = w_b + K v_b, and the update uses the base residual
// R_b = lam_b/dt + div_b - g (passed as g = -R_b).  The base is rebased in
// FP64 when a phase has cut its residual 1e4-fold, when the FP32 check (from
// the FP64 base check residual C_b and the changes) reaches the target, or
// when it stalls below the acceptable level; the FP64 residual of the rebased
// base confirms the stop.
struct AdjRbState {
    int skip, done, iter, phase_iter, nchecks, capped, stalled, best_at;
    int blocks, passes, phases, pad;   // check blocks, loop passes, rebases of the solve graph
    double acc, acc64, err, err64, target, accept, best;
};

__global__ void adj_tofloat_kernel(const double* src, float* dst, long long n)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        dst[t] = __double2float_rn(src[t]);
}

struct AdjFold {
    long long n;
    double* lamb;
    double* wb[3];
    float* d[2];
    float* w[3][2];
};

// lam_b += delta, w_b += omega (the changes of buffer parity par); both
// buffers cleared, the next iteration may start on either parity
__global__ void adj_rb_fold_kernel(AdjFold f, const AdjRbState* st, int par)
{
    if (st->done) return;
    const float* dp = par ? f.d[1] : f.d[0];
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < f.n;
         t += (long long)gridDim.x * blockDim.x) {
        f.lamb[t] += (double)dp[t];
        f.d[0][t] = 0.0f;
        f.d[1][t] = 0.0f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float* wp = par ? f.w[d][1] : f.w[d][0];
            f.wb[d][t] += (double)wp[t];
            f.w[d][0][t] = 0.0f;
            f.w[d][1][t] = 0.0f;
        }
    }
}

struct AdjBase {
    int nx, ny, nz;
    long long sy, sz;
    double rdt;
    double sig[3];
    const double* H;     // H^n (FP64)
    const double* E;     // exp(m) (FP64); NULL for D = H^3
    const double* lamb;
    const double* wb[3];
    const double* g;     // right-hand side (FP64)
    float* tb[3];
    float* rbf;          // -R_b
    double* Cb;
    double* parts;       // FP64 residual slots, one per CTA
};

// FP64 base quantities (one thread per cell): t_b for the +d faces, and for
// inner cells -R_b, C_b = g - lam_b/dt + sum sigma [(Kv_+ - Kv_-) - (n_+ + n_-)]
// and |C_b|^2.
template <bool EXPM>
__global__ void __launch_bounds__(256) adj_rb_base_kernel(AdjBase b, const AdjRbState* st)
{
    if (st->done) return;
    const long long total = (long long)b.nx * b.ny * b.nz;
    const long long stp[3] = {1, b.sy, b.sz};
    double part = 0.0;
    unsigned long long pmax = 0ull;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int co[3] = {(int)(t % b.nx), (int)((t / b.nx) % b.ny), (int)(t / ((long long)b.nx * b.ny))};
        const int nn[3] = {b.nx, b.ny, b.nz};
        const long long c = co[2] * b.sz + co[1] * b.sy + co[0];
        bool in[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) in[d] = co[d] >= 1 && co[d] <= nn[d] - 2;
        const bool inner = in[0] && in[1] && in[2];
        auto face = [&](long long cL, long long cR, double& kv, double& n) {
            const double HL = b.H[cL], HR = b.H[cR];
            const double sm = HL + HR;
            const double e2 = EXPM ? b.E[cL] + b.E[cR] : 2.0;
            const double v = b.lamb[cR] - b.lamb[cL];
            kv = e2 * sm * sm * sm * v;
            n = 3.0 * e2 * sm * sm * (HR - HL) * v;
        };
        double div = 0.0, q = 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const bool others = (d == 0 || in[0]) && (d == 1 || in[1]) && (d == 2 || in[2]);
            double kvp = 0.0, np = 0.0;
            if (others && co[d] <= nn[d] - 2) {
                face(c, c + stp[d], kvp, np);
                b.tb[d][c] = (float)(b.wb[d][c] + kvp);
            }
            if (inner) {
                double kvm, nm;
                face(c - stp[d], c, kvm, nm);
                div = fma(b.wb[d][c] - b.wb[d][c - stp[d]] + (np + nm), b.sig[d], div);
                q = fma((kvp - kvm) - (np + nm), b.sig[d], q);
            }
        }
        if (inner) {
            const double lr = b.lamb[c] * b.rdt;
            b.rbf[c] = (float)(b.g[c] - lr - div);
            const double cb = b.g[c] - lr + q;
            b.Cb[c] = cb;
            accumulate_residual(cb, part, pmax);
        }
    }
    block_reduce_residual(nullptr, 0, part, pmax, b.parts, blockIdx.x);
}

__global__ void __launch_bounds__(256) adj_rb_init_kernel(AdjRbState* st, const double* parts, long long nparts,
                                                          double rtol, double accept_rtol, double norm_den)
{
    const double gn = sqrt(sum_slots(parts, nparts, 0)) / sqrt(norm_den);
    if (threadIdx.x != 0) return;
    st->acc = 0.0;
    st->blocks = st->passes = st->phases = 0;
    st->acc64 = 0.0;
    st->target = fmax(rtol * gn, 1e-300);
    st->accept = fmax(accept_rtol * gn, 1e-300);
    st->done = gn == 0.0 ? 1 : 0;
    st->skip = st->done;
    st->iter = st->phase_iter = st->nchecks = st->capped = st->stalled = st->best_at = 0;
    st->err = st->err64 = st->best = gn;
}

// After each check block: the FP32 err from the check launch's slots (fixed
// order); the phase ends (skip) on the conditions below, and the rebase that
// follows the block in the solve graph (its IF node) runs when it has.
__global__ void __launch_bounds__(256) adj_rb_check_judge_kernel(AdjRbState* st, const double* parts,
                                                                 long long nparts, int nchk, int itmax,
                                                                 double norm_den, int stall, int phase_cap,
                                                                 cudaGraphConditionalHandle rebase)
{
    pdl_begin();
    // every thread reads the flags before thread 0 can change them
    const bool idle = st->skip || st->done;
    __syncthreads();
    if (idle) {   // no PT kernel ran: the slots are stale
        if (threadIdx.x == 0) {
            st->blocks += 1;
            cudaGraphSetConditional(rebase, 0);
        }
        return;
    }
    const double acc = sum_slots(parts, nparts, 0);
    if (threadIdx.x != 0) return;
    st->blocks += 1;
    const double err = sqrt(acc) / sqrt(norm_den);
    st->acc = 0.0;
    st->err = err;
    st->nchecks += 1;
    st->iter += nchk;
    st->phase_iter += nchk;
    if (err < 0.99 * st->best) {
        st->best = err;
        st->best_at = st->nchecks;
    }
    if (err != err) {
        st->done = 2;
        st->skip = 1;
        cudaGraphSetConditional(rebase, 1);
        return;
    }
    if (!(err > st->target)) {
        st->skip = 1;
    } else if (st->nchecks - st->best_at >= stall && err <= st->accept) {
        st->skip = 1;
        st->stalled = 1;
    } else if (err <= 1e-4 * st->err64 || st->phase_iter >= phase_cap) {
        st->skip = 1;
    }
    if (st->iter + nchk > itmax) {
        st->skip = 1;
        st->capped = 1;
    }
    cudaGraphSetConditional(rebase, st->skip ? 1 : 0);
}

__global__ void __launch_bounds__(256) adj_rb_base_judge_kernel(AdjRbState* st, const double* parts,
                                                                long long nparts, double norm_den, int in_loop)
{
    // every thread reads the flag before thread 0 can change it
    const bool stopped = st->done != 0;
    __syncthreads();
    if (stopped) {   // the base kernel did not run: the slots are stale
        if (threadIdx.x == 0 && in_loop) st->phases += 1;
        return;
    }
    const double acc64 = sum_slots(parts, nparts, 0);
    if (threadIdx.x != 0) return;
    if (in_loop) st->phases += 1;
    const double err64 = sqrt(acc64) / sqrt(norm_den);
    st->acc64 = 0.0;
    st->err64 = err64;
    st->phase_iter = 0;
    if (err64 != err64) {
        st->done = 2;
        st->skip = 1;
    } else if (st->iter > 0 && !(st->err > st->target) && !(err64 > st->target)) {
        st->done = 1;
    } else if (st->stalled && !(err64 > st->accept)) {
        st->done = 3;
    } else if (st->capped) {
        st->done = 2;
    } else {
        st->skip = 0;
        st->stalled = 0;
        st->best_at = st->nchecks;
    }
}

// Last node of the rebased solve graph's loop body: ends the loop once the
// solve has stopped; a solve still running after max_passes passes
// (itmax/nchk + 2) has lost its stop and ends as capped.
__global__ void adj_rb_loop_judge_kernel(AdjRbState* st, int max_passes, cudaGraphConditionalHandle loop)
{
    st->passes += 1;
    if (!st->done && st->passes > max_passes) {
        st->done = 2;
        st->skip = 1;
    }
    if (st->done) cudaGraphSetConditional(loop, 0);
}

__global__ void __launch_bounds__(256) adj_misfit_kernel(const double* HN, const double* Ht, void* g, double* parts,
                                                         int nx, int ny, int nz, long long sy, long long sz, int df64)
{
    const long long nix = nx - 2, niy = ny - 2, niz = nz - 2, total = nix * niy * niz;
    double part = 0.0;
    unsigned long long pm = 0ull;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long ix = 1 + t % nix, iy = 1 + (t / nix) % niy, iz = 1 + t / (nix * niy);
        const long long c = iz * sz + iy * sy + ix;
        const double d = HN[c] - Ht[c];
        part = fma(d, d, part);
        if (g) {
            if (df64) reinterpret_cast<float2*>(g)[c] = split_df(d);
            else reinterpret_cast<double*>(g)[c] = d;
        }
    }
    block_reduce_residual(nullptr, 0, part, pm, parts, blockIdx.x);
}

__global__ void expd_kernel(const double* m, double* E, long long n)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x)
        E[t] = exp(m[t]);
}

}  // namespace ptd

using namespace ptd;

struct ptd_adj {
    ptd_params p;
    ptd_ctx* fwd = nullptr;
    ptd_ctx_base g;
    Derived dv;
    LaunchCfg cfg;
    cudaStream_t s = nullptr;
    bool df64 = false, expm = false;
    double* ck = nullptr;       // (nt+1) FP64 checkpoints
    double* Ht = nullptr;       // target (FP64, padded)
    double* Ed = nullptr;       // exp(m) FP64
    void* E = nullptr;          // exp(m) in the kernel number type
    void* Hk = nullptr;         // H^n in the kernel number type
    void* lam[2] = {nullptr, nullptr};
    void* w[3][2] = {{nullptr, nullptr}, {nullptr, nullptr}, {nullptr, nullptr}};
    void* gbuf = nullptr;       // right-hand side
    double* gm = nullptr;
    double* gh = nullptr;
    double* stage = nullptr;
    AdjState* st = nullptr;
    AdjState* h_st = nullptr;
    double* h_acc = nullptr;
    AdjArgs* d_args[2] = {nullptr, nullptr};
    cudaGraphExec_t graph = nullptr;   // one FP64 / DF64 adjoint solve
    int nchk = 20;
    double rtol = 1e-10;        // adjoint solve target, relative to its right-hand side
    double accept_rtol = 1e-7;  // a solve stalled at an arithmetic floor below this is accepted
    int stall = 10;             // checks without 1 % improvement that count as stalled
    bool have_fwd = false;
    long long launches = 0, iterations = 0;
    std::vector<double> step_err, step_target;   // last adjoint solve: final residual and target per step
    bool any_capped = false;
    // rebased FP32 form (precision FP32_RB): lam[], w[] hold the FP32
    // changes, Hk and E FP32 copies; the FP64 base and its defects below
    bool rb = false;
    double* lamb = nullptr;
    double* wb[3] = {nullptr, nullptr, nullptr};
    double* Hk64 = nullptr;                      // H^n of the current step (FP64)
    void* tbf[3] = {nullptr, nullptr, nullptr};
    void* rbf = nullptr;
    double* Cb = nullptr;
    AdjRbState* rbst = nullptr;
    AdjRbState* h_rbst = nullptr;
    AdjArgs* d_rbargs[2] = {nullptr, nullptr};
    cudaGraphExec_t gphase = nullptr;
    int phase_iters = 200;      // PT iterations of a rebased phase at most
    int blocks_per_pass = 1;    // check blocks per pass of a solve graph's loop
    double* parts = nullptr;    // check-residual slots of the check launches
    long long nparts = 0;
    double* parts64 = nullptr;  // slots of the grid-stride reductions (one per CTA)
    long long nparts64 = 0;
    double* h_parts64 = nullptr;
};

namespace {

#define ACK(call)                                                 \
    do {                                                          \
        cudaError_t _e = (call);                                  \
        if (_e != cudaSuccess) return cuda_fail(_e, #call);       \
    } while (0)

cudaError_t adj_launch_rb(ptd_adj* A, int par, bool check)
{
    const dim3 blk(32, 8);
    const int tx = (A->g.nx - 2 + 30) / 31, ty = (A->g.ny - 2 + 6) / 7;
    const int ch = A->cfg.chunk3d;
    const dim3 grid(tx, ty, (A->g.nz - 2 + ch - 1) / ch);
    const AdjArgs* ap = A->d_rbargs[par];
    if (A->expm) {
        if (check) return launch_pdl(adj3d_kernel<F32, true, true, 8, true>, grid, blk, A->s, ap, ch);
        return launch_pdl(adj3d_kernel<F32, true, false, 8, true>, grid, blk, A->s, ap, ch);
    }
    if (check) return launch_pdl(adj3d_kernel<F32, false, true, 8, true>, grid, blk, A->s, ap, ch);
    return launch_pdl(adj3d_kernel<F32, false, false, 8, true>, grid, blk, A->s, ap, ch);
}

cudaError_t adj_launch(ptd_adj* A, int par, bool check)
{
    const dim3 blk(32, 8);
    const int tx = (A->g.nx - 2 + 30) / 31, ty = (A->g.ny - 2 + 6) / 7;
    const int ch = A->cfg.chunk3d;
    const dim3 grid(tx, ty, (A->g.nz - 2 + ch - 1) / ch);
    const AdjArgs* ap = A->d_args[par];
#define ADJ(NT, EX)                                                                          \
    return check ? launch_pdl(adj3d_kernel<NT, EX, true, 8>, grid, blk, A->s, ap, ch)         \
                 : launch_pdl(adj3d_kernel<NT, EX, false, 8>, grid, blk, A->s, ap, ch)
    if (A->df64) {
        if (A->expm) ADJ(DF64, true);
        else ADJ(DF64, false);
    } else {
        if (A->expm) ADJ(F64, true);
        else ADJ(F64, false);
    }
#undef ADJ
}

void adj_fill(ptd_adj* A, int par, AdjArgs& a)
{
    std::memset(&a, 0, sizeof(a));
    a.nx = A->g.nx;
    a.ny = A->g.ny;
    a.nz = A->g.nz;
    a.sy = A->g.sy;
    a.sz = A->g.sz;
    a.rdt = A->dv.rdt;
    a.rdt_df = split_df(A->dv.rdt);
    for (int d = 0; d < 3; ++d) {
        // the adjoint uses kappa = 1/16 for both models (D = H^3 as E = 1)
        a.sig[d] = 0.0625 / (A->dv.h[d] * A->dv.h[d]);
        a.sig_df[d] = split_df(a.sig[d]);
    }
    a.f = fparams(A->dv);
    a.lin = A->lam[par];
    a.lout = A->lam[par ^ 1];
    for (int d = 0; d < 3; ++d) {
        a.win[d] = A->w[d][par];
        a.wout[d] = A->w[d][par ^ 1];
    }
    a.H = A->Hk;
    a.E = A->expm ? A->E : nullptr;
    a.g = A->gbuf;
    a.done = &A->st->done;
    a.acc = &A->st->acc;
    a.parts = A->parts;
}

void adj_fill_rb(ptd_adj* A, int par, AdjArgs& a)
{
    adj_fill(A, par, a);
    a.rdtf = (float)A->dv.rdt;
    for (int d = 0; d < 3; ++d) {
        a.sigf[d] = (float)a.sig[d];
        a.tb[d] = A->tbf[d];
    }
    a.g = A->rbf;
    a.Cb = A->Cb;
    a.done = &A->rbst->skip;
    a.acc = &A->rbst->acc;
}

AdjBase adj_base_args(ptd_adj* A)
{
    AdjBase b;
    std::memset(&b, 0, sizeof(b));
    b.nx = A->g.nx;
    b.ny = A->g.ny;
    b.nz = A->g.nz;
    b.sy = A->g.sy;
    b.sz = A->g.sz;
    b.rdt = A->dv.rdt;
    for (int d = 0; d < 3; ++d) {
        b.sig[d] = 0.0625 / (A->dv.h[d] * A->dv.h[d]);
        b.wb[d] = A->wb[d];
        b.tb[d] = static_cast<float*>(A->tbf[d]);
    }
    b.H = A->Hk64;
    b.E = A->expm ? A->Ed : nullptr;
    b.lamb = A->lamb;
    b.g = static_cast<const double*>(A->gbuf);
    b.rbf = static_cast<float*>(A->rbf);
    b.Cb = A->Cb;
    b.parts = A->parts64;
    return b;
}

cudaError_t adj_rebase(ptd_adj* A, int par, int in_loop)
{
    AdjFold f;
    std::memset(&f, 0, sizeof(f));
    f.n = A->g.nfield;
    f.lamb = A->lamb;
    for (int q = 0; q < 2; ++q) f.d[q] = static_cast<float*>(A->lam[q]);
    for (int d = 0; d < 3; ++d) {
        f.wb[d] = A->wb[d];
        for (int q = 0; q < 2; ++q) f.w[d][q] = static_cast<float*>(A->w[d][q]);
    }
    adj_rb_fold_kernel<<<fill_blocks(), 256, 0, A->s>>>(f, A->rbst, par);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (A->expm) adj_rb_base_kernel<true><<<fill_blocks(), 256, 0, A->s>>>(adj_base_args(A), A->rbst);
    else adj_rb_base_kernel<false><<<fill_blocks(), 256, 0, A->s>>>(adj_base_args(A), A->rbst);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    adj_rb_base_judge_kernel<<<1, 256, 0, A->s>>>(A->rbst, A->parts64, A->nparts64, A->dv.norm_den, in_loop);
    return cudaGetLastError();
}

// The WHILE node of a solve graph, and its body graph.
cudaError_t adj_loop_graph(cudaGraph_t* g, cudaGraphConditionalHandle* loop, cudaGraph_t* body)
{
    *g = nullptr;
    cudaError_t err = cudaGraphCreate(g, 0);
    if (err == cudaSuccess) err = cudaGraphConditionalHandleCreate(loop, *g, 1, cudaGraphCondAssignDefault);
    cudaGraphNodeParams np = {cudaGraphNodeTypeConditional};
    np.conditional.handle = *loop;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    if (err == cudaSuccess) err = cudaGraphAddNode(&node, *g, nullptr, nullptr, 0, &np);
    if (err == cudaSuccess) *body = np.conditional.phGraph_out[0];
    return err;
}

// End a capture that an error interrupted.
void adj_drop_capture(cudaStream_t s)
{
    cudaStreamCaptureStatus cs;
    if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
        cudaGraph_t dropped = nullptr;
        cudaStreamEndCapture(s, &dropped);
        if (dropped) cudaGraphDestroy(dropped);
    }
    cudaGetLastError();
}

// The rebased adjoint solve of one step as one CUDA graph: a WHILE node whose
// body is one check block (nchk FP32 launches and the check judge) followed by
// an IF node holding the FP64 rebase (fold, base quantities, base judge), run
// when the judge has ended the phase; two such blocks when nchk is odd, so
// that every pass starts on buffer parity 0; last, the loop judge.  No launch
// is issued past the end of a phase or of the solve.
int adj_capture_rb(ptd_adj* A)
{
    for (int q = 0; q < 2; ++q) {
        AdjArgs a;
        adj_fill_rb(A, q, a);
        ACK(cudaMemcpy(A->d_rbargs[q], &a, sizeof(a), cudaMemcpyHostToDevice));
    }
    cudaGraph_t g = nullptr, body = nullptr;
    cudaGraphConditionalHandle loop;
    cudaError_t err = adj_loop_graph(&g, &loop, &body);
    const int nblk = (A->nchk & 1) ? 2 : 1;
    int par = 0;
    cudaGraphNode_t prev = nullptr;   // the previous block's IF node
    for (int b = 0; b < nblk && err == cudaSuccess; ++b) {
        cudaGraphConditionalHandle rebase;
        err = cudaGraphConditionalHandleCreate(&rebase, body, 0, cudaGraphCondAssignDefault);
        if (err == cudaSuccess)
            err = cudaStreamBeginCaptureToGraph(A->s, body, prev ? &prev : nullptr, nullptr, prev ? 1 : 0,
                                                cudaStreamCaptureModeThreadLocal);
        if (err != cudaSuccess) break;
        for (int it = 0; it < A->nchk && err == cudaSuccess; ++it) {
            err = adj_launch_rb(A, par, it == A->nchk - 1);
            par ^= 1;
        }
        if (err == cudaSuccess) {
            err = launch_pdl(adj_rb_check_judge_kernel, 1, 256, A->s, A->rbst, A->parts, A->nparts, A->nchk, A->p.itmax,
                             A->dv.norm_den, A->stall, A->phase_iters, rebase);
        }
        // the judge is the capture's last node: the IF node follows it
        cudaStreamCaptureStatus cs;
        const cudaGraphNode_t* deps = nullptr;
        size_t nd = 0;
        const cudaError_t e1 = cudaStreamGetCaptureInfo(A->s, &cs, nullptr, nullptr, &deps, nullptr, &nd);
        cudaGraphNode_t leaf = (e1 == cudaSuccess && nd == 1) ? deps[0] : nullptr;
        cudaGraph_t captured = body;
        const cudaError_t e2 = cudaStreamEndCapture(A->s, &captured);
        if (err == cudaSuccess) err = e1 != cudaSuccess ? e1 : e2;
        if (err == cudaSuccess && !leaf) err = cudaErrorStreamCaptureInvalidated;
        cudaGraphNodeParams ip = {cudaGraphNodeTypeConditional};
        ip.conditional.handle = rebase;
        ip.conditional.type = cudaGraphCondTypeIf;
        ip.conditional.size = 1;
        cudaGraphNode_t ifn = nullptr;
        if (err == cudaSuccess) err = cudaGraphAddNode(&ifn, body, &leaf, nullptr, 1, &ip);
        if (err == cudaSuccess)
            err = cudaStreamBeginCaptureToGraph(A->s, ip.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                cudaStreamCaptureModeThreadLocal);
        if (err != cudaSuccess) break;
        err = adj_rebase(A, par, 1);
        cudaGraph_t ifbody = ip.conditional.phGraph_out[0];
        const cudaError_t e3 = cudaStreamEndCapture(A->s, &ifbody);
        if (err == cudaSuccess) err = e3;
        prev = ifn;
    }
    // the loop's condition, set at the body's level after the last rebase node
    if (err == cudaSuccess)
        err = cudaStreamBeginCaptureToGraph(A->s, body, &prev, nullptr, 1, cudaStreamCaptureModeThreadLocal);
    if (err == cudaSuccess) {
        adj_rb_loop_judge_kernel<<<1, 1, 0, A->s>>>(A->rbst, A->p.itmax / A->nchk + 2, loop);
        err = cudaGetLastError();
        cudaGraph_t captured = body;
        const cudaError_t e4 = cudaStreamEndCapture(A->s, &captured);
        if (err == cudaSuccess) err = e4;
    }
    if (err != cudaSuccess) {
        adj_drop_capture(A->s);
        if (g) cudaGraphDestroy(g);
        return cuda_fail(err, "adjoint capture (rebased)");
    }
    const cudaError_t e5 = cudaGraphInstantiate(&A->gphase, g, 0);
    cudaGraphDestroy(g);
    if (e5 != cudaSuccess) return cuda_fail(e5, "cudaGraphInstantiate");
    A->blocks_per_pass = nblk;
    return PTD_OK;
}

// The FP64 / DF64 adjoint solve of one step as one CUDA graph: a WHILE node
// whose body is one check block (nchk launches and the judge, which ends the
// loop once the solve has stopped); two blocks when nchk is odd, so that every
// pass starts on buffer parity 0.
int adj_capture(ptd_adj* A)
{
    for (int q = 0; q < 2; ++q) {
        AdjArgs a;
        adj_fill(A, q, a);
        ACK(cudaMemcpy(A->d_args[q], &a, sizeof(a), cudaMemcpyHostToDevice));
    }
    cudaGraph_t g = nullptr, body = nullptr;
    cudaGraphConditionalHandle loop;
    cudaError_t err = adj_loop_graph(&g, &loop, &body);
    if (err == cudaSuccess)
        err = cudaStreamBeginCaptureToGraph(A->s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
    const int nblk = (A->nchk & 1) ? 2 : 1;
    int par = 0;
    for (int b = 0; b < nblk && err == cudaSuccess; ++b) {
        for (int it = 0; it < A->nchk && err == cudaSuccess; ++it) {
            err = adj_launch(A, par, it == A->nchk - 1);
            par ^= 1;
        }
        if (err == cudaSuccess) {
            err = launch_pdl(adj_judge_kernel, 1, 256, A->s, A->st, A->parts, A->nparts, A->nchk, A->p.itmax,
                             A->dv.norm_den, A->stall, loop);
        }
    }
    if (err == cudaSuccess) {
        cudaGraph_t captured = body;
        err = cudaStreamEndCapture(A->s, &captured);
    }
    if (err != cudaSuccess) {
        adj_drop_capture(A->s);
        if (g) cudaGraphDestroy(g);
        return cuda_fail(err, "adjoint capture");
    }
    const cudaError_t e3 = cudaGraphInstantiate(&A->graph, g, 0);
    cudaGraphDestroy(g);
    if (e3 != cudaSuccess) return cuda_fail(e3, "cudaGraphInstantiate");
    A->blocks_per_pass = nblk;
    return PTD_OK;
}

void adj_free(ptd_adj* A)
{
    if (!A) return;
    if (A->s) cudaStreamSynchronize(A->s);
    if (A->graph) cudaGraphExecDestroy(A->graph);
    if (A->gphase) cudaGraphExecDestroy(A->gphase);
    if (A->fwd) ptd_destroy(A->fwd);
    void* ptrs[] = {A->ck, A->Ht, A->Ed, A->E, A->Hk, A->lam[0], A->lam[1], A->gbuf, A->gm, A->gh, A->stage,
                    A->st, A->d_args[0], A->d_args[1], A->lamb, A->Hk64, A->rbf, A->Cb, A->rbst, A->d_rbargs[0],
                    A->d_rbargs[1], A->parts, A->parts64};
    for (void* q : ptrs) cudaFree(q);
    for (int d = 0; d < 3; ++d) {
        for (int q = 0; q < 2; ++q) cudaFree(A->w[d][q]);
        cudaFree(A->wb[d]);
        cudaFree(A->tbf[d]);
    }
    if (A->h_st) cudaFreeHost(A->h_st);
    if (A->h_rbst) cudaFreeHost(A->h_rbst);
    if (A->h_parts64) cudaFreeHost(A->h_parts64);
    delete A;
}

}  // namespace

extern "C" int ptd_adj_create(ptd_adj** out, const ptd_params* p)
{
    if (!out) return set_error(PTD_EINVAL, "ptd_adj_create: out is NULL");
    *out = nullptr;
    int rc = validate(p);
    if (rc) return rc;
    if (p->ndim != 3) return set_error(PTD_EINVAL, "the adjoint solver is 3D");
    if (p->model != PTD_MODEL_NONLIN && p->model != PTD_MODEL_NONLIN_EXPM)
        return set_error(PTD_EINVAL, "the adjoint solver supports D = H^3 and D = exp(m) H^3");
    if (p->precision == PTD_PREC_FP32_DC || p->precision == PTD_PREC_DFH)
        return set_error(PTD_EINVAL, "the adjoint runs in FP64, DF64 or FP32_RB");
    ptd_adj* A = new (std::nothrow) ptd_adj();
    if (!A) return set_error(PTD_ENOMEM, "adjoint: host allocation failed");
    A->p = *p;
    A->df64 = p->precision == PTD_PREC_DF64;
    A->rb = p->precision == PTD_PREC_FP32_RB;
    A->expm = p->model == PTD_MODEL_NONLIN_EXPM;
    derive(A->p, A->dv);
    A->cfg.chunk3d = z_march8(A->p, A->rb ? 2 : 4);   // every form's kernel has 8-row CTAs
    {   // stagnation window: ~2 n_max iterations, the PT iteration's own time scale
        const int nmax = std::max(p->nx, std::max(p->ny, p->nz));
        A->stall = std::max(10, (2 * nmax + A->nchk - 1) / A->nchk);
    }
    A->g.nx = p->nx;
    A->g.ny = p->ny;
    A->g.nz = p->nz;
    A->g.sy = ((p->nx + 31) / 32) * 32;
    A->g.sz = A->g.sy * p->ny;
    A->g.nfield = A->g.sz * p->nz;
    ptd_params pf = *p;
    pf.nt = 1;
    rc = ptd_create(&A->fwd, &pf);
    if (rc) {
        adj_free(A);
        return rc;
    }
    A->s = static_cast<cudaStream_t>(ptd_stream(A->fwd));
    const size_t b = (size_t)A->g.nfield * sizeof(double);
    auto al = [&](void** q, size_t n) -> int {
        if (cudaMalloc(q, n) != cudaSuccess) {
            cudaGetLastError();
            return set_error(PTD_ENOMEM, "adjoint: cudaMalloc failed");
        }
        return cudaMemset(*q, 0, n) == cudaSuccess ? PTD_OK : set_error(PTD_ECUDA, "adjoint: cudaMemset failed");
    };
    rc = al((void**)&A->ck, b * (size_t)(p->nt + 1));
    if (!rc) rc = al((void**)&A->Ht, b);
    if (!rc) rc = al((void**)&A->Ed, b);
    if (!rc) rc = al(&A->E, b);
    if (!rc) rc = al(&A->Hk, b);
    for (int q = 0; q < 2 && !rc; ++q) rc = al(&A->lam[q], b);
    for (int d = 0; d < 3 && !rc; ++d)
        for (int q = 0; q < 2 && !rc; ++q) rc = al(&A->w[d][q], b);
    if (!rc) rc = al(&A->gbuf, b);
    if (!rc) rc = al((void**)&A->gm, b);
    if (!rc) rc = al((void**)&A->gh, b);
    if (!rc) rc = al((void**)&A->stage, b);
    if (!rc) rc = al((void**)&A->st, sizeof(AdjState));
    for (int q = 0; q < 2 && !rc; ++q) rc = al((void**)&A->d_args[q], sizeof(AdjArgs));
    if (!rc && cudaMallocHost((void**)&A->h_st, sizeof(AdjState)) != cudaSuccess)
        rc = set_error(PTD_ENOMEM, "adjoint: cudaMallocHost failed");
    // residual slots: one per CTA of a check launch, one per CTA of the
    // grid-stride reductions (sums of squares, misfit, rebase)
    A->nparts = (long long)((A->g.nx - 2 + 30) / 31) * ((A->g.ny - 2 + 6) / 7) *
                ((A->g.nz - 2 + A->cfg.chunk3d - 1) / A->cfg.chunk3d);
    A->nparts64 = fill_blocks();
    if (!rc) rc = al((void**)&A->parts, (size_t)A->nparts * sizeof(double));
    if (!rc) rc = al((void**)&A->parts64, (size_t)A->nparts64 * sizeof(double));
    if (!rc && cudaMallocHost((void**)&A->h_parts64, (size_t)A->nparts64 * sizeof(double)) != cudaSuccess)
        rc = set_error(PTD_ENOMEM, "adjoint: cudaMallocHost failed");
    if (A->rb) {
        if (!rc) rc = al((void**)&A->lamb, b);
        if (!rc) rc = al((void**)&A->Hk64, b);
        for (int d = 0; d < 3 && !rc; ++d) {
            rc = al((void**)&A->wb[d], b);
            if (!rc) rc = al(&A->tbf[d], b);
        }
        if (!rc) rc = al(&A->rbf, b);
        if (!rc) rc = al((void**)&A->Cb, b);
        if (!rc) rc = al((void**)&A->rbst, sizeof(AdjRbState));
        for (int q = 0; q < 2 && !rc; ++q) rc = al((void**)&A->d_rbargs[q], sizeof(AdjArgs));
        if (!rc && cudaMallocHost((void**)&A->h_rbst, sizeof(AdjRbState)) != cudaSuccess)
            rc = set_error(PTD_ENOMEM, "adjoint: cudaMallocHost failed");
        if (!rc) rc = adj_capture_rb(A);
    }
    if (!rc) rc = adj_capture(A);
    if (rc) {
        adj_free(A);
        return rc;
    }
    *out = A;
    return PTD_OK;
}

extern "C" void ptd_adj_destroy(ptd_adj* A) { adj_free(A); }

static int adj_loss(ptd_adj* A, double* loss)
{
    const double* HN = A->ck + (size_t)A->p.nt * A->g.nfield;
    adj_misfit_kernel<<<(int)A->nparts64, 256, 0, A->s>>>(HN, A->Ht, nullptr, A->parts64, A->g.nx, A->g.ny, A->g.nz,
                                                          A->g.sy, A->g.sz, 0);
    ACK(cudaGetLastError());
    ACK(cudaMemcpyAsync(A->h_parts64, A->parts64, (size_t)A->nparts64 * sizeof(double), cudaMemcpyDeviceToHost,
                        A->s));
    ACK(cudaStreamSynchronize(A->s));
    double acc = 0.0;   // the CTAs' partial sums in a fixed order
    for (long long i = 0; i < A->nparts64; ++i) acc += A->h_parts64[i];
    if (loss) *loss = 0.5 * acc;
    return PTD_OK;
}

// Forward solve of nt steps from H0 with log-coefficient m (NULL for D = H^3),
// keeping one FP64 checkpoint per step; L = 1/2 sum_inner (H^nt - Ht)^2.
extern "C" int ptd_adj_forward(ptd_adj* A, const double* H0, const double* m, const double* Ht, double* loss,
                               double* HN, int32_t* iters_per_step)
{
    if (!A || !H0 || !Ht) return set_error(PTD_EINVAL, "ptd_adj_forward: NULL argument");
    if (A->expm && !m) return set_error(PTD_EINVAL, "ptd_adj_forward: m is required");
    int rc = ptd_set_state(A->fwd, H0, m);
    if (rc) return rc;
    const size_t b = (size_t)A->g.nfield * sizeof(double);
    rc = copy_field_in(A->g, A->Ht, Ht, A->s);
    if (rc) return rc;
    if (A->expm) {
        rc = copy_field_in(A->g, A->stage, m, A->s);
        if (rc) return rc;
        expd_kernel<<<fill_blocks(), 256, 0, A->s>>>(A->stage, A->Ed, A->g.nfield);
        ACK(cudaGetLastError());
        if (A->rb) {   // exp(m) as FP32 for the rebased adjoint iteration
            adj_tofloat_kernel<<<fill_blocks(), 256, 0, A->s>>>(A->Ed, static_cast<float*>(A->E), A->g.nfield);
            ACK(cudaGetLastError());
        } else {
            ACK(launch_expm(A->stage, A->E, A->g.nfield, A->df64, A->s));
        }
    }
    ACK(cudaMemsetAsync(A->ck, 0, b, A->s));
    rc = copy_field_in(A->g, A->ck, H0, A->s);
    if (rc) return rc;
    for (int n = 1; n <= A->p.nt; ++n) {
        int32_t it = 0;
        rc = ptd_step(A->fwd, 1, &it, nullptr, 0, nullptr);
        if (rc && rc != PTD_ENOTCONV) return rc;
        if (iters_per_step) iters_per_step[n - 1] = it;
        rc = ctx_current_f64(A->fwd, A->ck + (size_t)n * A->g.nfield);
        if (rc) return rc;
    }
    A->have_fwd = true;
    rc = adj_loss(A, loss);
    if (rc) return rc;
    if (HN) {
        rc = copy_field_out(A->g, HN, A->ck + (size_t)A->p.nt * A->g.nfield, A->s);
        if (rc) return rc;
        ACK(cudaStreamSynchronize(A->s));
    }
    return PTD_OK;
}

// Adjoint sweep over the checkpoints of the last ptd_adj_forward: dL/dm (model
// exp(m) H^3) and dL/dH0 (all cells), each nullable.  adj_iters (nullable,
// nt entries): PT iterations of each adjoint solve, in step order.
extern "C" int ptd_adj_gradient(ptd_adj* A, double* grad_m, double* grad_H0, int32_t* adj_iters)
{
    if (!A) return set_error(PTD_EINVAL, "ptd_adj_gradient: NULL argument");
    if (!A->have_fwd) return set_error(PTD_ESTATE, "ptd_adj_gradient: run ptd_adj_forward first");
    const size_t b = (size_t)A->g.nfield * sizeof(double);
    A->step_err.assign(A->p.nt, 0.0);
    A->step_target.assign(A->p.nt, 0.0);
    A->any_capped = false;
    ACK(cudaMemsetAsync(A->gm, 0, b, A->s));
    ACK(cudaMemsetAsync(A->gh, 0, b, A->s));
    // g = H^nt - Ht on inner cells
    ACK(cudaMemsetAsync(A->gbuf, 0, b, A->s));
    const double* HN = A->ck + (size_t)A->p.nt * A->g.nfield;
    adj_misfit_kernel<<<(int)A->nparts64, 256, 0, A->s>>>(HN, A->Ht, A->gbuf, A->parts64, A->g.nx, A->g.ny,
                                                          A->g.nz, A->g.sy, A->g.sz, A->df64);
    ACK(cudaGetLastError());
    const long long cells = (long long)A->g.nx * A->g.ny * A->g.nz;
    for (int n = A->p.nt; n >= 1 && A->rb; --n) {
        // rebased FP32 adjoint solve of step n
        const double* Hn = A->ck + (size_t)n * A->g.nfield;
        ACK(cudaMemcpyAsync(A->Hk64, Hn, b, cudaMemcpyDeviceToDevice, A->s));
        adj_tofloat_kernel<<<fill_blocks(), 256, 0, A->s>>>(Hn, static_cast<float*>(A->Hk), A->g.nfield);
        ACK(cudaGetLastError());
        ACK(cudaMemsetAsync(A->lamb, 0, b, A->s));
        for (int d = 0; d < 3; ++d) ACK(cudaMemsetAsync(A->wb[d], 0, b, A->s));
        for (int q = 0; q < 2; ++q) {
            ACK(cudaMemsetAsync(A->lam[q], 0, b, A->s));
            for (int d = 0; d < 3; ++d) ACK(cudaMemsetAsync(A->w[d][q], 0, b, A->s));
        }
        adj_sumsq_kernel<F64><<<(int)A->nparts64, 256, 0, A->s>>>(A->gbuf, A->parts64, A->g.nx, A->g.ny, A->g.nz,
                                                                  A->g.sy, A->g.sz);
        ACK(cudaGetLastError());
        adj_rb_init_kernel<<<1, 256, 0, A->s>>>(A->rbst, A->parts64, A->nparts64, A->rtol, A->accept_rtol,
                                                A->dv.norm_den);
        ACK(cudaGetLastError());
        ACK(adj_rebase(A, 0, 0));   // base quantities of lam_b = 0 (the fold adds zeros)
        A->launches += 5;
        // the whole solve: one graph launch, ended on the device
        ACK(cudaGraphLaunch(A->gphase, A->s));
        ACK(cudaMemcpyAsync(A->h_rbst, A->rbst, sizeof(AdjRbState), cudaMemcpyDeviceToHost, A->s));
        ACK(cudaStreamSynchronize(A->s));
        A->launches += (long long)A->h_rbst->blocks * (A->nchk + 1) + A->h_rbst->passes + 3LL * A->h_rbst->phases;
        const AdjRbState& rs = *A->h_rbst;
        A->iterations += rs.iter;
        if (adj_iters) adj_iters[n - 1] = rs.iter;
        A->step_err[n - 1] = rs.err64;
        A->step_target[n - 1] = rs.target;
        if (rs.done == 2 || rs.done == 0) A->any_capped = true;
        AdjArgs a;
        adj_fill(A, 0, a);
        a.lin = A->lamb;   // the FP64 base holds the solution
        if (A->expm) adj_grad_kernel<F64, true><<<fill_blocks(), 256, 0, A->s>>>(a, Hn, A->Ed, A->gm, A->gh, A->gbuf, cells);
        else adj_grad_kernel<F64, false><<<fill_blocks(), 256, 0, A->s>>>(a, Hn, A->Ed, A->gm, A->gh, A->gbuf, cells);
        ACK(cudaGetLastError());
        A->launches += 1;
    }
    for (int n = A->p.nt; n >= 1 && !A->rb; --n) {
        const double* Hn = A->ck + (size_t)n * A->g.nfield;
        if (A->df64) ACK(launch_to_df64(Hn, A->Hk, A->g.nfield, A->s));
        else ACK(cudaMemcpyAsync(A->Hk, Hn, b, cudaMemcpyDeviceToDevice, A->s));
        for (int q = 0; q < 2; ++q) {
            ACK(cudaMemsetAsync(A->lam[q], 0, b, A->s));
            for (int d = 0; d < 3; ++d) ACK(cudaMemsetAsync(A->w[d][q], 0, b, A->s));
        }
        // target: rtol * ||g||_rms
        if (A->df64)
            adj_sumsq_kernel<DF64><<<(int)A->nparts64, 256, 0, A->s>>>(A->gbuf, A->parts64, A->g.nx, A->g.ny,
                                                                       A->g.nz, A->g.sy, A->g.sz);
        else
            adj_sumsq_kernel<F64><<<(int)A->nparts64, 256, 0, A->s>>>(A->gbuf, A->parts64, A->g.nx, A->g.ny, A->g.nz,
                                                                      A->g.sy, A->g.sz);
        ACK(cudaGetLastError());
        adj_target_kernel<<<1, 256, 0, A->s>>>(A->st, A->parts64, A->nparts64, A->rtol, A->accept_rtol,
                                               A->dv.norm_den, 1e-300);
        ACK(cudaGetLastError());
        A->launches += 3;
        // the whole solve: one graph launch, ended on the device
        ACK(cudaGraphLaunch(A->graph, A->s));
        ACK(cudaMemcpyAsync(A->h_st, A->st, sizeof(AdjState), cudaMemcpyDeviceToHost, A->s));
        ACK(cudaStreamSynchronize(A->s));
        A->launches += (long long)A->h_st->blocks * (A->nchk + 1);
        const int iters = A->h_st->iter;
        A->iterations += iters;
        if (adj_iters) adj_iters[n - 1] = iters;
        A->step_err[n - 1] = A->h_st->err;
        A->step_target[n - 1] = A->h_st->target;
        if (A->h_st->done == 2) A->any_capped = true;   // 3 (stalled below accept_rtol) is accepted
        AdjArgs a;
        adj_fill(A, iters & 1, a);
#define AGK(NT, EX) adj_grad_kernel<NT, EX><<<fill_blocks(), 256, 0, A->s>>>(a, Hn, A->Ed, A->gm, A->gh, A->gbuf, cells)
        if (A->df64) {
            if (A->expm) AGK(DF64, true);
            else AGK(DF64, false);
        } else {
            if (A->expm) AGK(F64, true);
            else AGK(F64, false);
        }
#undef AGK
        ACK(cudaGetLastError());
        A->launches += 1;
    }
    // dL/dH0 on inner cells = g (lam_1 / dt)
    if (grad_H0) {
        // gh += g on inner cells: fold through the staging field
        if (A->df64) ACK(launch_from_df64(A->gbuf, A->stage, A->g.nfield, A->s));
        else ACK(cudaMemcpyAsync(A->stage, A->gbuf, b, cudaMemcpyDeviceToDevice, A->s));
        ACK(add_fields(A->gh, A->stage, A->g.nfield, A->s));
        int rc = copy_field_out(A->g, grad_H0, A->gh, A->s);
        if (rc) return rc;
    }
    if (grad_m && A->expm) {
        int rc = copy_field_out(A->g, grad_m, A->gm, A->s);
        if (rc) return rc;
    }
    ACK(cudaStreamSynchronize(A->s));
    if ((A->p.flags & PTD_FLAG_STRICT) && A->any_capped)
        return set_error(PTD_ENOTCONV, "ptd_adj_gradient: an adjoint solve reached itmax");
    return PTD_OK;
}

extern "C" int ptd_adj_residuals(ptd_adj* A, double* err, double* target)
{
    if (!A) return set_error(PTD_EINVAL, "adjoint is NULL");
    for (int n = 0; n < A->p.nt; ++n) {
        if (err) err[n] = A->step_err[n];
        if (target) target[n] = A->step_target[n];
    }
    return PTD_OK;
}

extern "C" int ptd_adj_counters(ptd_adj* A, int64_t* launches, int64_t* iterations)
{
    if (!A) return set_error(PTD_EINVAL, "adjoint is NULL");
    int64_t fl = 0, fi = 0;
    ptd_counters(A->fwd, &fl, &fi);
    if (launches) *launches = A->launches + fl;
    if (iterations) *iterations = A->iterations + fi;
    return PTD_OK;
}
