"""Performance cases of the diffusion framework: what its users run, through
its public entry points (``ptdiff.Solver``, ``BatchSolver``, ``AdjointSolver``).

Kinds of case
  solve    ``nt`` implicit steps to the scripts' tolerance: set_state, step, get_state
  iterate  a fixed number of PT iterations, the reference's perf-script protocol
  batch    one implicit step of many uneven 2D step-diffusion grids
  adjoint  forward with checkpoints, then the gradients of the L2 misfit

Every field is a device tensor in x-fastest order (shape ``(nz, ny, nx)`` in
torch's C order), made from the seed: bumps of random height and place on the
scripts' domain of side 10, with the scripts' dt, tolerance and CFL.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "pseudotransientdiffusion.jl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import ptdiff  # noqa: E402
from ptdiff import scripts as S  # noqa: E402

DEVICE = "cuda"
SIDE = 10.0      # the scripts' domain length in every direction
DT = 0.2         # the scripts' physical time step
TOL = 1e-8       # the scripts' tolerance
D_OUT, D_IN = 1.0, 1e-4   # the step model's diffusivities
PI = math.pi


def grid(ndim, model, precision, n, *, nt=1, nchk=10, shift=1.0, niter=0, name=None):
    case = {"kind": "iterate" if niter else "solve", "model": model, "precision": precision, "nx": n[0],
            "ny": n[1] if ndim > 1 else 1, "nz": n[2] if ndim > 2 else 1, "ndim": ndim, "nt": nt, "nchk": nchk,
            "shift": shift, "niter": niter}
    return {"name": name, **case} if name else case


def listed():
    return [
        # the published 1D run: 512 cells, 5 steps; a 1D solve is the smallest
        # call there is, so launches and latency decide it
        grid(1, "lin", "fp64", (512,), nt=5, name="lin1d_512"),
        # an ordinary small 2D run of the nonlinear script with its own start
        # field (D = H^3 goes to zero away from the bump)
        grid(2, "nonlin", "fp64", (128, 128), nt=5, shift=0.0, name="nonlin2d_128"),
        # a ragged grid with cells that are not square, per-cell diffusivity
        grid(2, "linstep", "fp64", (500, 333), nt=2, name="linstep2d_500x333"),
        # the perf script's protocol on the large 2D grid of the benchmarks
        grid(2, "nonlin", "fp64", (4096, 4096), niter=40, name="nonlin2d_4096_iterate"),
        # the 3D script at its default size, all five steps
        grid(3, "nonlin", "fp64", (64, 64, 64), nt=5, name="nonlin3d_64"),
        # the headline: the 3D perf protocol at 512^3, the largest state
        grid(3, "nonlin", "fp64", (512, 512, 512), niter=20, name="nonlin3d_512_iterate"),
        # time to tolerance in the fast arithmetic, large 2D and ragged 3D
        grid(2, "nonlin", "fp32_rb", (2048, 2048), nchk=100, name="nonlin2d_2048_rb"),
        grid(3, "nonlin", "fp32_rb", (320, 255, 191), name="nonlin3d_320x255x191_rb"),
        # the double-float forms where they are used: FP64 state in 2D,
        # double-float state in 3D
        grid(2, "nonlin", "dfh", (1021, 1500), name="nonlin2d_1021x1500_dfh"),
        grid(3, "lin", "df64", (126, 126, 126), nt=2, name="lin3d_126_df64"),
        # many uneven grids at once
        {"name": "batch_48", "kind": "batch", "precision": "fp32_rb", "ninst": 48, "nmin": 64, "nmax": 512},
        # gradients of a misfit (forward and backward)
        {"name": "adjoint_72", "kind": "adjoint", "precision": "fp32_rb", "nx": 72, "ny": 72, "nz": 72, "nt": 3},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, ndim, lo, hi):
    """A box whose sides differ by up to a third."""
    n = _side(rng, lo, hi)
    return [max(lo, int(n * rng.uniform(0.67, 1.0))) if d else n for d in range(ndim)]


def draw(rng):
    kind = rng.choice(["1d", "2d", "2d", "3d", "iter2d", "iter3d", "fast2d", "fast3d", "batch", "adjoint"])
    model = rng.choice(["lin", "linstep", "nonlin"])
    shift = rng.choice([0.0, 1.0]) if model == "nonlin" else 1.0
    if kind == "1d":
        return grid(1, model, "fp64", (_side(rng, 32, 4096),), nt=rng.randint(1, 5), shift=shift)
    if kind == "2d":
        return grid(2, model, "fp64", _sides(rng, 2, 32, 768), nt=rng.randint(1, 2), shift=shift)
    if kind == "3d":
        return grid(3, model, "fp64", _sides(rng, 3, 24, 160), nt=rng.randint(1, 2), shift=shift)
    if kind == "iter2d":
        return grid(2, model, "fp64", _sides(rng, 2, 512, 4096), niter=rng.randint(20, 40), shift=shift)
    if kind == "iter3d":
        return grid(3, model, "fp64", _sides(rng, 3, 64, 480), niter=rng.randint(10, 20), shift=shift)
    if kind == "fast2d":
        return grid(2, model, rng.choice(["fp32_rb", "fp32_rb", "dfh"]), _sides(rng, 2, 256, 1800),
                    nchk=rng.choice([10, 100]))
    if kind == "fast3d":
        return grid(3, model, rng.choice(["fp32_rb", "fp32_rb", "dfh", "df64"]), _sides(rng, 3, 48, 288))
    if kind == "batch":
        nmin = _side(rng, 32, 128)
        return {"kind": "batch", "precision": "fp32_rb", "ninst": rng.randint(8, 48), "nmin": nmin,
                "nmax": _side(rng, nmin, 512)}
    n = _sides(rng, 3, 24, 72)
    return {"kind": "adjoint", "precision": rng.choice(["fp32_rb", "fp64"]), "nx": n[0], "ny": n[1], "nz": n[2],
            "nt": rng.randint(1, 3)}


# ---------------------------------------------------------------------------
# inputs
def _shape(case):
    """torch shape: x is the last (fastest) dimension."""
    return [case[k] for k in ("nz", "ny", "nx")][3 - case.get("ndim", 3):]


def _centres(n):
    return (torch.arange(n, dtype=torch.float64, device=DEVICE) + 0.5) * (SIDE / n)


def _bump(shape, rng, shift, width=1.0):
    """shift + A exp(-r^2/width) around a random centre; boundary cells at shift if it is not 0."""
    amp = float(rng.uniform(0.6, 1.4))
    H = torch.full([1] * len(shape), amp, dtype=torch.float64, device=DEVICE)
    for d, n in enumerate(shape):
        x = _centres(n) - float(rng.uniform(0.4, 0.6)) * SIDE
        H = H * torch.exp(-x * x / width).reshape([-1 if k == d else 1 for k in range(len(shape))])
    H = H + shift
    if shift:
        for d, n in enumerate(shape):
            H.narrow(d, 0, 1).fill_(shift)
            H.narrow(d, n - 1, 1).fill_(shift)
    return H.contiguous()


def _step_field(shape, rng):
    """The step model's field: D_IN below a random interface in each of the first two directions."""
    D = torch.full(shape, D_OUT, dtype=torch.float64, device=DEVICE)
    for d in range(len(shape) - 1, max(-1, len(shape) - 3), -1):
        n = shape[d]
        D.narrow(d, 0, max(1, int(n * rng.uniform(0.4, 0.5)))).fill_(D_IN)
    return D


def _log_coefficient(shape, rng, std=0.3):
    """A smooth random field: a few cosines of random wave vector and phase."""
    m = torch.zeros(shape, dtype=torch.float64, device=DEVICE)
    axes = [_centres(n).reshape([-1 if k == d else 1 for k in range(len(shape))]) for d, n in enumerate(shape)]
    for _ in range(6):
        k = rng.normal(0.0, 1.0, len(shape))
        m = m + torch.cos(sum(float(k[d]) * axes[d] for d in range(len(shape))) + float(rng.uniform(0, 2 * PI)))
    return (m * (std / math.sqrt(3.0))).contiguous()


def _script(case):
    name = {1: "diff_1D_%s", 2: "diff_2D_%s", 3: "diff_3D_%s_multixpu"}[case["ndim"]] % case["model"]
    return S.SCRIPTS[name]


def _grid_inputs(case, seed):
    rng = np.random.default_rng(seed)
    H0 = _bump(_shape(case), rng, case["shift"])
    D = _step_field(_shape(case), rng) if case["model"] == "linstep" else None
    return H0, D


def _batch_sides(case):
    """Sides log-uniform in [nmin, nmax]."""
    u = np.random.default_rng(case["ninst"] * 1000 + case["nmax"]).uniform(
        math.log(case["nmin"]), math.log(case["nmax"]), case["ninst"])
    return [int(n) for n in np.rint(np.exp(u))]


def _batch_inputs(case, seed):
    """The sizes belong to the case, the fields to the seed."""
    sides = _batch_sides(case)
    rng = np.random.default_rng(seed)
    Hs, Ds = [], []
    for n in sides:
        x = _centres(n)
        cx, cy = rng.uniform(0.25, 0.75, 2) * SIDE
        H = 1.0 + float(rng.uniform(0.5, 2.0)) * torch.exp(-(x[:, None] - cy) ** 2 - (x[None, :] - cx) ** 2)
        D = torch.full((n, n), D_IN, dtype=torch.float64, device=DEVICE)
        D[x < float(rng.uniform(0.3, 0.7)) * SIDE] = D_OUT
        Hs.append(H.reshape(-1))
        Ds.append(D.reshape(-1))
    return sides, Hs, Ds


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shape = _shape(case)
    return _bump(shape, rng, 1.0), _log_coefficient(shape, rng), _bump(shape, rng, 1.0, width=1.5)


def _adjoint_script(case):
    return S.SCRIPTS["diff_3D_nonlin_multixpu"].with_(
        name="adjoint", model=S.NONLIN_EXPM, shift=1.0, dirichlet=1.0, dt=0.1, ttot=0.1 * case["nt"], tol=1e-10,
        ic="linrange")


# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "batch":
        sides, Hs, Ds = _batch_inputs(case, seed)
        H0 = torch.cat(Hs)
        H = torch.empty_like(H0)
        parts = list(torch.split(H, [n * n for n in sides]))
        solver = ptdiff.BatchSolver(ptdiff.batch_params(len(sides), model=S.LINSTEP, precision=case["precision"], nt=1),
                                    sides, sides)
        return {"case": case, "solver": solver, "H0": H0, "H": H, "parts": parts, "D": Ds}
    if case["kind"] == "adjoint":
        H0, m, Ht = _adjoint_inputs(case, seed)
        solver = ptdiff.AdjointSolver(ptdiff.make_params(_adjoint_script(case), [case[k] for k in ("nx", "ny", "nz")],
                                                         precision=case["precision"], nt=case["nt"], nchk=10))
        return {"case": case, "solver": solver, "H0": H0, "m": m, "Ht": Ht, "gm": torch.empty_like(m),
                "gH": torch.empty_like(m)}
    H0, D = _grid_inputs(case, seed)
    s = _script(case)
    p = ptdiff.make_params(s, [case[k] for k in ("nx", "ny", "nz")], nt=case["nt"], nchk=case["nchk"],
                           precision=case["precision"])
    return {"case": case, "solver": ptdiff.Solver(p), "H0": H0, "D": D, "H": torch.empty_like(H0)}


def run(state):
    case, solver = state["case"], state["solver"]
    if case["kind"] == "batch":
        state["H"].copy_(state["H0"])
        torch.cuda.current_stream().synchronize()   # the solver works on streams of its own
        iters, err = solver.solve(state["parts"], state["D"])
        return {"H": state["H"], "iters": iters}
    if case["kind"] == "adjoint":
        loss = solver.forward(state["H0"], state["m"], state["Ht"])
        solver.gradient(out_m=state["gm"], out_H0=state["gH"])
        return {"loss": loss, "dm": state["gm"], "dH0": state["gH"]}
    solver.set_state(state["H0"], state["D"])
    if case["kind"] == "iterate":
        solver.iterate(case["niter"])
        return {"H": solver.get_state(state["H"])}
    iters, _ = solver.step(case["nt"])
    return {"H": solver.get_state(state["H"]), "iters": iters}


# ---------------------------------------------------------------------------
# PT iterations per physical step, per cell of the longest side (measured: the
# counts grow linearly with it)
ITERS_PER_CELL = {"lin": 1.2, "linstep": 1.2, "nonlin": 1.4, "expm": 1.2}


def _flops(ndim, model):
    """Floating-point operations of one PT iteration per cell: per direction the face (gradient, conductance,
    damped flux) and its part of the divergence, then the update."""
    face = {"lin": 4, "linstep": 6, "nonlin": 8, "expm": 10}[model]
    return ndim * (face + 2) + 6


def work(case):
    """Bytes: the fields handed over and returned, once each.  Operations: those of the PT iterations."""
    if case["kind"] == "batch":
        sides = _batch_sides(case)
        cells = sum(n * n for n in sides)
        return {"bytes": 24 * cells, "flops": _flops(2, "linstep") * sum(n * n * 1.2 * n for n in sides)}
    cells = case["nx"] * case["ny"] * case["nz"]
    n = max(case["nx"], case["ny"], case["nz"])
    if case["kind"] == "adjoint":
        its = 2 * case["nt"] * ITERS_PER_CELL["expm"] * n
        return {"bytes": 40 * cells, "flops": _flops(3, "expm") * cells * its}
    its = case["niter"] or case["nt"] * ITERS_PER_CELL[case["model"]] * n
    return {"bytes": (24 if case["model"] == "linstep" else 16) * cells,
            "flops": _flops(case["ndim"], case["model"]) * cells * its}


# ---------------------------------------------------------------------------
# The same computations in 64 bits with plain tensor operations.
class _Exact:
    """The accelerated PT iteration (damped flux, then the update) on one grid."""

    def __init__(self, H0, model, dt=DT, D=None, E=None, resc=None, cfl=None):
        self.H, self.Hold, self.model, self.D, self.E, self.dt = H0.clone(), H0, model, D, E, dt
        self.nd = nd = H0.dim()
        self.dims = list(range(nd - 1, -1, -1))
        self.h = {d: SIDE / H0.shape[d] for d in self.dims}
        cfl = cfl if cfl is not None else {1: 1.0 if model == "nonlin" else 0.99}.get(nd, 1.0 / math.sqrt(nd))
        self.vpdt = cfl * min(self.h.values())
        self.resc = resc if resc is not None else (1.0 / 1.2 if model in ("nonlin", "expm") and nd > 1 else 1.0)
        self.q = {d: torch.zeros_like(self._face(H0, d)[0]) for d in self.dims}
        self.re = PI + math.sqrt(PI * PI + SIDE * SIDE / D_OUT / dt)
        if model == "linstep":
            P = torch.nn.functional.pad(D[None, None], [1] * (2 * nd), mode="replicate")[0, 0]
            mx = D
            for d in self.dims:
                for off in (0, 2):
                    sl = [slice(1, 1 + n) for n in D.shape]
                    sl[d] = slice(off, off + D.shape[d])
                    mx = torch.maximum(mx, P[tuple(sl)])
            self.inv_dtau = mx * (self.re / (self.vpdt * SIDE))

    def _face(self, A, d):
        n = A.shape[d]
        return A.narrow(d, 0, n - 1), A.narrow(d, 1, n - 1)

    def _inner(self, A, but=None):
        for d in range(self.nd):
            if d != but:
                A = A.narrow(d, 1, A.shape[d] - 2)
        return A

    def conductance(self, d):
        """Face diffusivity, and the damping parameter theta."""
        H = self.H
        if self.model == "lin":
            return D_OUT, SIDE / self.vpdt / self.re
        if self.model == "linstep":
            a, b = self._face(self.D, d)
            return (a + b) * 0.5, SIDE / self.vpdt / self.re
        a, b = self._face(H, d)
        K = ((a + b) * 0.5) ** 3
        if self.model == "expm":
            e, f = self._face(self.E, d)
            K = K * ((e + f) * 0.5)
        re = PI + torch.sqrt(PI * PI + SIDE * SIDE / (K * self.dt))
        return K, SIDE * self.resc / self.vpdt / re

    def iterate(self, check=False):
        H, und = self.H, {}
        for d in self.dims:
            a, b = self._face(H, d)
            K, theta = self.conductance(d)
            u = -K * (b - a) / self.h[d]
            und[d] = u if check else None
            self.q[d] = (self.q[d] * theta + u) / (1.0 + theta)
        if self.model == "lin":
            inv = D_OUT * self.re / (self.vpdt * SIDE)
        elif self.model == "linstep":
            inv = self._inner(self.inv_dtau)
        else:
            c = self._inner(H) ** 3
            if self.model == "expm":
                c = c * self._inner(self.E)
            inv = (PI * c + torch.sqrt(PI * PI * c * c + SIDE * SIDE * c / self.dt)) / (self.vpdt * SIDE * self.resc)
        div = sum(self._inner(torch.diff(self.q[d], dim=d), but=d) / self.h[d] for d in self.dims)
        Hc, Ho = self._inner(H), self._inner(self.Hold)
        Hn = Hc - ((Hc - Ho) / self.dt + div) / (inv + 1.0 / self.dt)
        self.H = H.clone()
        self._inner(self.H).copy_(Hn)
        if check:
            r = -(Hn - Ho) / self.dt - sum(self._inner(torch.diff(und[d], dim=d), but=d) / self.h[d] for d in self.dims)
            return float(torch.sqrt(torch.mean(r * r)))

    def step(self, nchk, tol=TOL, itmax=100000):
        it, err = 0, 2 * tol
        while err > tol and it < itmax:
            for k in range(nchk):
                err_k = self.iterate(k == nchk - 1)
            it, err = it + nchk, err_k
        self.Hold = self.H


def _gradient_exact(case, seed):
    """Forward steps to a tight tolerance, then the transposed linear systems by BiCGSTAB on autograd's products."""
    H0, m, Ht = _adjoint_inputs(case, seed)
    E, dt, inner = torch.exp(m), 0.1, (slice(1, -1),) * 3
    pt = _Exact(H0, "expm", dt=dt, E=E)
    Hs = [H0]
    for _ in range(case["nt"]):
        pt.step(10, tol=1e-12, itmax=40 * max(H0.shape))
        Hs.append(pt.H)

    def residual(H, Hold, logD):
        e = torch.exp(logD)
        out = (H[inner] - Hold[inner]) / dt
        for d in range(3):
            n, h = H.shape[d], SIDE / H.shape[d]
            a, b = H.narrow(d, 0, n - 1), H.narrow(d, 1, n - 1)
            u = ((a + b) * 0.5) ** 3 * ((e.narrow(d, 0, n - 1) + e.narrow(d, 1, n - 1)) * 0.5) * (b - a) / h
            for k in range(3):
                if k != d:
                    u = u.narrow(k, 1, u.shape[k] - 2)
            out = out - torch.diff(u, dim=d) / h
        return out

    def solve_t(jt, b):
        x, r = torch.zeros_like(b), b.clone()
        r0, p, rho = r.clone(), r.clone(), torch.sum(r * r)
        stop = 1e-13 * float(torch.sqrt(rho))
        for _ in range(2000):
            v = jt(p)
            al = rho / torch.sum(r0 * v)
            s = r - al * v
            t = jt(s)
            om = torch.sum(t * s) / torch.sum(t * t)
            x, r = x + al * p + om * s, s - om * t
            if float(torch.linalg.vector_norm(r)) <= stop:
                break
            new = torch.sum(r0 * r)
            p = r + (new / rho) * (al / om) * (p - om * v)
            rho = new
        return x

    miss = Hs[-1][inner] - Ht[inner]
    g, gm, gb = miss.clone(), torch.zeros_like(m), torch.zeros_like(m)
    for n in range(case["nt"], 0, -1):
        H, logD = Hs[n].clone().requires_grad_(True), m.clone().requires_grad_(True)
        F = residual(H, Hs[n - 1], logD)
        jt = lambda v: torch.autograd.grad(F, H, v, retain_graph=True)[0][inner]  # noqa: B023, E731
        lam = solve_t(jt, g)
        vH, vm = torch.autograd.grad(F, (H, logD), lam)
        edge = -vH
        edge[inner] = 0.0
        gb, gm, g = gb + edge, gm - vm, lam / dt
    gb[inner] = g
    return {"loss": float(0.5 * torch.sum(miss * miss)), "dm": gm, "dH0": gb}


def exact(case, seed):
    if case["kind"] == "adjoint":
        return _gradient_exact(case, seed)
    if case["kind"] == "batch":
        sides, Hs, Ds = _batch_inputs(case, seed)
        out = []
        for n, H, D in zip(sides, Hs, Ds):
            pt = _Exact(H.reshape(n, n), "linstep", D=D.reshape(n, n))
            pt.step(10)
            out.append(pt.H.reshape(-1))
        return {"H": torch.cat(out), "iters": None}
    H0, D = _grid_inputs(case, seed)
    pt = _Exact(H0, case["model"], D=D)
    if case["kind"] == "iterate":
        for _ in range(case["niter"]):
            pt.iterate()
        return {"H": pt.H}
    for _ in range(case["nt"]):
        pt.step(case["nchk"])
    return {"H": pt.H, "iters": None}
