"""Workloads that stand for what a user has this propagator do.

Every case goes through the package's public entry points (the ``Solver`` call
surface, ``sweep_step``, the device-buffer right-hand side and the learned
self-energy's ``MLP``), on seeded synthetic tight-binding models of the sizes of
the repository's configurations, tests and bench:

  propagate   one propagation: initial density matrix in, n steps, final density
              matrix out (host memory on both sides, as every driver of the
              library does); RK4 and Adams-Bashforth, with and without the HSEX
              self-energy, one solve or a batch, full or Hermitian-plane form
  printed     the command line's loop: one step at a time with the populations,
              the velocity and the field read between the steps
  sweep       independent solves of uneven band count and grid, a model and a
              pulse each, stepped together
  rhs         one right-hand side on device buffers (no allocation)
  mlp         training steps, or one evaluation, of the self-energy network

The precision forms below FP64 (mixed, split) are left out: they miss the 1e-8
bar on the benchmark and no configuration runs them.  So are the Peierls gauge
and the k-space gradient, which no configuration selects.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
E = pkg.edus

DEVICE = "cuda:0"
BOHR_LATTICE = 6.0
# grid sides the plane transform handles (prime factors 2 to 13)
SIDES = [n for n in range(1, 1100) if all(n % p or p <= 13 for p in range(2, n + 1) if all(p % q for q in range(2, p)))]


# ---------------------------------------------------------------------------
# inputs
def _rng(seed, *more):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, *[int(x) for x in more]])


def _hermitian(rng, nb, scale):
    a = (rng.uniform(-1, 1, (nb, nb)) + 1j * rng.uniform(-1, 1, (nb, nb))) * scale
    return 0.5 * (a + a.conj().T)


def _shells(grid):
    """One lattice vector of every +-R pair the model hops along."""
    dims = [d for d in range(3) if grid[d] > 1]
    if len(dims) == 1:
        base = [(1,), (2,)]
    elif len(dims) == 2:
        base = [(1, 0), (0, 1), (1, -1), (1, 1), (2, -1), (1, -2), (2, 0), (0, 2), (2, -2)]
    else:
        base = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0)]
    out = []
    for v in base:
        R = [0, 0, 0]
        for d, x in zip(dims, v):
            R[d] = x
        out.append(R)
    return np.array(out, dtype=np.float64)


def _lattice(grid):
    a = BOHR_LATTICE
    if sum(n > 1 for n in grid) == 2 and grid[2] == 1:
        return np.array([[a * math.sqrt(3) / 2, a * math.sqrt(3) / 2, 0.0], [a / 2, -a / 2, 0.0], [0.0, 0.0, 40.0]])
    return np.array([[a, 0.2, 0.0], [0.1, 1.1 * a, 0.3], [0.0, 0.2, 0.9 * a]])


def _crystal_R(grid):
    """Gamma-centred coordinates of every R index."""
    ax = [np.arange(n) for n in grid]
    ax = [np.where(2 * j >= n, j - n, j) for j, n in zip(ax, grid)]
    return np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)


def _model(grid, nb, coulomb, seed, observables=False):
    """Host arrays of a gapped random model in the library's [k][n][m] layout:
    random Hermitian hoppings on a few shells, valence and conduction bands
    apart, on-site dipoles; the ground state; with HSEX a Rytova-Keldysh-like
    screened potential and the Hartree matrix of the bare one."""
    rng = _rng(seed, nb, *grid)
    nv = max(1, nb // 2)
    Nk = grid[0] * grid[1] * grid[2]
    dev = torch.device(DEVICE)
    A = _lattice(grid)
    k = np.stack(np.meshgrid(*[np.arange(n) / n for n in grid], indexing="ij"), -1).reshape(-1, 3)
    kt = torch.as_tensor(k, device=dev)
    on = _hermitian(rng, nb, 0.01) + np.diag(rng.uniform(-0.02, 0.02, nb))
    on += np.diag(np.where(np.arange(nb) < nv, -0.12, 0.12))
    H0 = torch.as_tensor(on, device=dev).expand(Nk, nb, nb).clone()
    vel = torch.zeros((3, Nk, nb, nb), dtype=torch.complex128, device=dev) if observables else None
    for R in _shells(grid):
        T = (rng.uniform(-1, 1, (nb, nb)) + 1j * rng.uniform(-1, 1, (nb, nb))) * 0.02 / np.linalg.norm(R) / math.sqrt(nb)
        T = torch.as_tensor(T, device=dev)
        ph = torch.exp(2j * math.pi * (kt @ torch.as_tensor(R, device=dev)))
        hop = ph[:, None, None] * T
        H0 += hop + hop.conj().transpose(-1, -2)
        if observables:
            for d, x in enumerate(A @ R):
                vel[d] += 1j * x * (hop - hop.conj().transpose(-1, -2))
    ndim = sum(n > 1 for n in grid)
    xi = torch.zeros((3, Nk, nb, nb), dtype=torch.complex128, device=dev)
    for d in range(ndim):
        D = _hermitian(rng, nb, 0.4)
        np.fill_diagonal(D, 0.0)
        xi[d] = torch.as_tensor(D, device=dev)
    _, U = torch.linalg.eigh(H0)
    occ = U[:, :, :nv]
    rho = occ @ occ.conj().transpose(-1, -2)
    m = {"grid": grid, "nb": nb, "A": A, "H0": H0.cpu().numpy(), "xi": xi.cpu().numpy(), "filled": nv,
         "W": None, "rho0R": None, "hartree": None, "rho": rho.cpu().numpy()}
    if observables:
        m["U"], m["vel"] = U.cpu().numpy(), vel.cpu().numpy()
    if coulomb:
        c = np.zeros((nb, 3))
        c[:, 0] = rng.uniform(0.0, 0.4 * BOHR_LATTICE, nb)
        off = torch.as_tensor(c[:, None] - c[None, :], device=dev)
        r = torch.as_tensor(_crystal_R(grid) @ A.T, device=dev)
        dist = torch.linalg.vector_norm(off[None] - r[:, None, None, :], dim=-1).clamp_min(1.0)
        r0 = 75.0
        W = (-torch.log(dist / (dist + r0)) - 0.116 * torch.exp(-dist / r0)) / r0
        hart = (2.0 / dist).sum(0)
        rR = torch.fft.fftn(rho.reshape(*grid, nb, nb), dim=(0, 1, 2)).reshape(Nk, nb, nb) / Nk
        m["W"] = W.to(torch.complex128).cpu().numpy()
        m["hartree"] = (0.5 * (hart + hart.T)).to(torch.complex128).cpu().numpy()
        m["rho0R"] = rR.cpu().numpy()
    return m


def _pulse(grid, rng, field):
    """A Gaussian pulse that is at its peak when the propagation starts."""
    ndim = sum(n > 1 for n in grid)
    pol = [0.0, 0.0, 0.0]
    for d in range(ndim):
        pol[d] = float(rng.uniform(0.4, 1.0))
    return E.Laser(intensity=float(field * rng.uniform(0.8, 1.2)) ** 2, omega=float(rng.uniform(0.05, 0.1)),
                   pol=tuple(pol), t0=0.0, phase=float(rng.uniform(0, 1)), fwhm=413.0, envelope=E.ENVELOPE_GAUSS)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.complex128, pin_memory=True).numpy()


def _grid(case):
    return (case["n0"], case["n1"], case["n2"])


# ---------------------------------------------------------------------------
# the same propagation in plain torch, FP64 (for `exact`)
class _Plain:
    def __init__(self, m, lasers):
        t = lambda a: None if a is None else torch.as_tensor(a, device=DEVICE)  # noqa: E731
        self.m, self.lasers = m, lasers
        self.H0, self.xi, self.W, self.r0R, self.hart = (t(m[x]) for x in ("H0", "xi", "W", "rho0R", "hartree"))
        self.R = t(_crystal_R(m["grid"]) @ m["A"].T)
        self.Nk = self.H0.shape[0]

    def field(self, t):
        e = np.zeros(3)
        for L in self.lasers:
            pol = np.array(L.pol) / np.linalg.norm(L.pol)
            x = t - L.t0
            e += math.sqrt(L.intensity) * math.exp(-2 * math.log(2.0) * x * x / L.fwhm ** 2) * math.cos(L.omega * x + L.phase) * pol
        return e

    def _fft(self, x, f):
        return f(x.reshape(*self.m["grid"], *x.shape[1:]), dim=(0, 1, 2)).reshape(x.shape)

    def rhs(self, t, rho):
        e = self.field(t)
        rR = self._fft(rho, torch.fft.fftn) / self.Nk
        RE = self.R @ torch.as_tensor(e, device=DEVICE)
        f = self._fft(1j * RE[:, None, None] * rR, torch.fft.ifftn) * self.Nk
        H = self.H0 + sum(float(e[d]) * self.xi[d] for d in range(3))
        if self.W is not None:
            hee = -self.W * (rR - self.r0R)
            d = torch.diagonal(rR[0] - self.r0R[0])
            hee[0] += torch.diag(self.hart @ d)
            H = H + self._fft(hee, torch.fft.ifftn) * self.Nk
        return f - 1j * (H @ rho - rho @ H)

    def rk4(self, t, y, dt):
        k1 = self.rhs(t, y)
        k2 = self.rhs(t + dt / 2, y + dt / 2 * k1)
        k3 = self.rhs(t + dt / 2, y + dt / 2 * k2)
        k4 = self.rhs(t + dt, y + dt * k3)
        return y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)

    def run(self, y, dt, steps, solver, order):
        y, t, hist = torch.as_tensor(y, device=DEVICE), 0.0, []
        beta = {4: (55 / 24, -59 / 24, 37 / 24, -3 / 8),
                5: (1901 / 720, -2774 / 720, 2616 / 720, -1274 / 720, 251 / 720)}.get(order)
        for _ in range(steps):
            if solver == "RK":
                y = self.rk4(t, y, dt)
            else:  # zero history at the start, as the reference's solver
                hist = [self.rhs(t, y)] + hist[: order - 1]
                y = y + dt * sum(b * f for b, f in zip(beta, hist))
            t += dt
        return y


def _work_steps(grid, nb, coulomb, rhs_count):
    """Of `rhs_count` right-hand sides with their stage updates: the stage input
    and the model read and the stage output written once; the transforms by
    5 N log2 N and two complex matrix products."""
    Nk = grid[0] * grid[1] * grid[2]
    S = Nk * nb * nb
    ndim = sum(n > 1 for n in grid)
    # with HSEX W (8 B) and rho0; without it H0(k) and xi(k)
    model = 24 * S if coulomb else 16 * S * (1 + ndim)
    fft = (3 if coulomb else 2) * 5.0 * S * max(1.0, math.log2(Nk))
    return {"bytes": rhs_count * (32 * S + model), "flops": rhs_count * (fft + 16.0 * S * nb)}


# ---------------------------------------------------------------------------
# propagate
def _propagate_inputs(case, seed, observables=False):
    grid = _grid(case)
    m = _model(grid, case["nb"], case["coulomb"], seed, observables)
    rng = _rng(seed, 99)
    lasers = [[_pulse(grid, rng, case["field"] * math.sqrt(1.0 + b / 4.0))] for b in range(case["batch"])]
    return m, lasers


def _solver(case, m, lasers):
    prec = E.PREC_HPLANES if case["form"] == "hplanes" else E.PREC_FP64
    s = E.Solver(m["grid"], m["nb"], case["dt"], solver=E.SOLVER_RK if case["solver"] == "RK" else E.SOLVER_AB,
                 order=case["order"], coulomb=case["coulomb"], batch=case["batch"], precision=prec)
    s.upload_model(m["H0"], m["xi"], m["A"], m["W"], m["rho0R"], m["hartree"])
    for b, L in enumerate(lasers):
        s.set_lasers(L, b)
    return s


def _prepare_propagate(case, seed):
    m, lasers = _propagate_inputs(case, seed)
    s = _solver(case, m, lasers)
    rho = _pinned(m["rho"].shape)
    rho[:] = m["rho"]
    outs = [_pinned(m["rho"].shape) for _ in range(case["batch"])]
    return {"s": s, "rho": rho, "outs": outs, "steps": case["steps"]}


def _run_propagate(st):
    s = st["s"]
    s.time = 0.0
    for b in range(s.batch):
        s.set_state(st["rho"], b)
    s.step(st["steps"])
    return [s.get_state(b, out=st["outs"][b]) for b in range(s.batch)]


def _exact_propagate(case, seed):
    m, lasers = _propagate_inputs(case, seed)
    return [_Plain(m, L).run(m["rho"], case["dt"], case["steps"], case["solver"], case["order"]).cpu().numpy()
            for L in lasers]


# ---------------------------------------------------------------------------
# printed: one step at a time, with what the command line prints between them
def _prepare_printed(case, seed):
    m, lasers = _propagate_inputs(case, seed, observables=True)
    s = _solver(case, m, lasers)
    s.upload_observables(U=m["U"], vel=m["vel"])
    rho = _pinned(m["rho"].shape)
    rho[:] = m["rho"]
    return {"s": s, "rho": rho, "out": _pinned(m["rho"].shape), "steps": case["steps"], "filled": m["filled"]}


def _run_printed(st):
    s = st["s"]
    s.time = 0.0
    s.set_state(st["rho"])
    field, bloch, wannier, vel = [], [], [], []
    for _ in range(st["steps"]):
        s.step(1)
        field.append(s.efield(s.time))
        pb, pw, v = s.observables(0, st["filled"])
        bloch.append(pb)
        wannier.append(pw)
        vel.append(v)
    return {"field": np.array(field), "bloch": np.array(bloch), "wannier": np.array(wannier), "velocity": np.array(vel),
            "rho": s.get_state(out=st["out"])}


def _exact_printed(case, seed):
    m, lasers = _propagate_inputs(case, seed, observables=True)
    p = _Plain(m, lasers[0])
    U, vel = torch.as_tensor(m["U"], device=DEVICE), torch.as_tensor(m["vel"], device=DEVICE)
    y, t = torch.as_tensor(m["rho"], device=DEVICE), 0.0
    field, bloch, wannier, vs = [], [], [], []
    for _ in range(case["steps"]):
        y = p.rk4(t, y, case["dt"])
        t += case["dt"]
        field.append(p.field(t))
        b = torch.einsum("kin,kij,kjn->n", U.conj(), y, U).real / p.Nk
        b[: m["filled"]] = 1.0 - b[: m["filled"]]
        bloch.append(b.cpu().numpy())
        wannier.append((torch.diagonal(y, dim1=1, dim2=2).real.sum(0) / p.Nk).cpu().numpy())
        vs.append((torch.einsum("dknm,kmn->d", vel, y) / p.Nk).cpu().numpy())
    return {"field": np.array(field), "bloch": np.array(bloch), "wannier": np.array(wannier), "velocity": np.array(vs),
            "rho": y.cpu().numpy()}


# ---------------------------------------------------------------------------
# sweep: independent solves grouped by shape into handles, a model and a pulse each
def _sweep_shapes(case):
    rng = _rng(case["mix"], 4242)
    bands, sides = pkg.workloads.SWEEP_BANDS, pkg.workloads.SWEEP_SIDES
    groups = {}
    for _ in range(case["solves"]):
        shape = (int(rng.choice(bands)), int(rng.choice(sides)))
        groups[shape] = groups.get(shape, 0) + 1
    return sorted(groups.items())


def _sweep_inputs(case, seed):
    for (nb, N), count in _sweep_shapes(case):
        grid = (N, N, 1)
        rng = _rng(seed, nb, N, 7)
        yield grid, nb, [(_model(grid, nb, False, int(seed) + 1000 * b),
                          [_pulse(grid, rng, float(10.0 ** rng.uniform(-4.0, -2.0)))]) for b in range(count)]


def _prepare_sweep(case, seed):
    st = {"solvers": [], "rho": [], "outs": [], "steps": case["steps"]}
    for grid, nb, solves in _sweep_inputs(case, seed):
        s = E.Solver(grid, nb, case["dt"], batch=len(solves))
        s.upload_model(solves[0][0]["H0"], solves[0][0]["xi"], solves[0][0]["A"])
        for b, (m, L) in enumerate(solves):
            if b:
                s.upload_model_solve(b, m["H0"], m["xi"])
            s.set_lasers(L, b)
        st["solvers"].append(s)
        rho = [_pinned(s.shape) for _ in solves]
        for r, (m, _) in zip(rho, solves):
            r[:] = m["rho"]
        st["rho"].append(rho)
        st["outs"].append([_pinned(s.shape) for _ in solves])
    return st


def _run_sweep(st):
    for s, rho in zip(st["solvers"], st["rho"]):
        s.time = 0.0
        for b, r in enumerate(rho):
            s.set_state(r, b)
    E.sweep_step(st["solvers"], st["steps"])
    return [s.get_state(b, out=o) for s, outs in zip(st["solvers"], st["outs"]) for b, o in enumerate(outs)]


def _exact_sweep(case, seed):
    return [_Plain(m, L).run(m["rho"], case["dt"], case["steps"], "RK", 4).cpu().numpy()
            for _, _, solves in _sweep_inputs(case, seed) for m, L in solves]


# ---------------------------------------------------------------------------
# rhs: the right-hand side on the caller's device buffers
def _rhs_inputs(case, seed):
    grid = _grid(case)
    m = _model(grid, case["nb"], case["coulomb"], seed)
    rng = _rng(seed, 5)
    # a state off the ground state by a small Hermitian part
    d = rng.normal(size=m["rho"].shape) + 1j * rng.normal(size=m["rho"].shape)
    m["rho"] = m["rho"] + 1e-3 * (d + np.conj(np.swapaxes(d, 1, 2)))
    return m, [_pulse(grid, rng, case["field"])]


def _prepare_rhs(case, seed):
    m, L = _rhs_inputs(case, seed)
    dev = lambda a: None if a is None else torch.as_tensor(np.ascontiguousarray(a), device=DEVICE)  # noqa: E731
    bufs = {n: dev(m[n]) for n in ("H0", "xi", "W", "rho0R", "hartree", "rho")}
    return {"lib": E.load_library(), "grid": (ctypes.c_int * 3)(*m["grid"]), "nb": m["nb"], "coulomb": int(case["coulomb"]),
            "A": np.ascontiguousarray(m["A"]), "E": _Plain(m, L).field(0.0), "bufs": bufs,
            "out": torch.empty_like(bufs["rho"]), "err": ctypes.create_string_buffer(256)}


def _run_rhs(st):
    ptr = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)  # noqa: E731
    dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    b = st["bufs"]
    rc = st["lib"].edus_rhs_noalloc(st["grid"], st["nb"], st["coulomb"], dp(st["A"]), dp(st["E"]), ptr(b["H0"]),
                                    ptr(b["xi"]), ptr(b["W"]), ptr(b["rho0R"]), ptr(b["hartree"]), ptr(b["rho"]),
                                    ptr(st["out"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), st["err"],
                                    len(st["err"]))
    if rc:
        raise E.EdusError(rc, st["err"].value.decode())
    return st["out"]


def _exact_rhs(case, seed):
    m, L = _rhs_inputs(case, seed)
    return _Plain(m, L).rhs(0.0, torch.as_tensor(m["rho"], device=DEVICE))


# ---------------------------------------------------------------------------
# mlp: the learned self-energy's network (pair rows of a state in, shells out)
def _mlp_inputs(case, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    n_in, n_out, rows = case["n_in"], case["n_out"], case["rows"]
    x = torch.empty((case["minibatches"], rows, n_in), device=DEVICE).uniform_(-1.0, 1.0, generator=g)
    mix = torch.empty((n_in, n_out), device=DEVICE).normal_(generator=g) / math.sqrt(n_in)
    t = torch.tanh(x @ mix) * 0.5
    return x.contiguous(), t.contiguous()


def _prepare_mlp(case, seed):
    x, t = _mlp_inputs(case, seed)
    net = pkg.surrogate.MLP(case["n_in"], case["n_out"], seed=int(seed) % 100003)
    return {"net": net, "x": x, "t": t, "p0": net.params(), "lr": 2e-3, "train": case["train"]}


def _run_mlp(st):
    net = st["net"]
    if not st["train"]:
        return [net.forward(x) for x in st["x"]]
    net.set_params(st["p0"])  # a fit from its initial weights
    losses = [net.train_step(x, t, st["lr"]) for x, t in zip(st["x"], st["t"])]
    return {"loss": np.array(losses, dtype=np.float32), "params": net.params()}


def _exact_mlp(case, seed):
    if case["train"]:
        return None  # Adam divides each gradient by its own size: no 64-bit value to hold BF16 products to
    st = _prepare_mlp(case, seed)
    p = torch.as_tensor(st["p0"], device=DEVICE).double()
    out = []
    for x in st["x"]:
        a, off = x.double(), 0
        for i, (n_in, n_out) in enumerate(st["net"].layer_shapes()):
            w = p[off: off + n_in * n_out].reshape(n_in, n_out)
            bias = p[off + n_in * n_out: off + n_in * n_out + n_out]
            off += n_in * n_out + n_out
            a = a @ w + bias
            if i < 3:
                a = torch.nn.functional.gelu(a)
        out.append(a)
    return out


# ---------------------------------------------------------------------------
def _case(name, nb, grid, coulomb, steps, dt, field, solver="RK", order=4, batch=1, form="fp64", kind="propagate"):
    c = {"kind": kind, "nb": nb, "n0": grid[0], "n1": grid[1], "n2": grid[2], "coulomb": coulomb, "steps": steps,
         "dt": dt, "field": field, "solver": solver, "order": order, "batch": batch, "form": form}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the two-band chain of the first configuration, its whole run: the smallest steps there are
        _case("chain64_rk4", 2, (64, 1, 1), False, 2000, 0.413, 0.01),
        # the reference's own integration test as the command line runs it: a printed line per step
        _case("hbn50_printed", 2, (50, 50, 1), False, 100, 0.413, 0.01, kind="printed"),
        # the same two-band material with HSEX on the reference's HSEX test grid, its run length
        _case("hbn40_hsex_rk4", 2, (40, 40, 1), True, 102, 0.413, 0.01),
        # the hBN-like configuration: two bands on a large grid
        _case("hbn120_rk4", 2, (120, 120, 1), False, 512, 0.413, 0.005),
        # ragged: odd band count, odd and unequal sides, the five-step Adams-Bashforth
        _case("odd13_hsex_ab5", 13, (45, 63, 1), True, 40, 0.05, 0.005, solver="AB", order=5),
        # the benchmark's model and grid, one solve (22 bands, HSEX, RK4)
        _case("tmd22_rk4", 22, (72, 72, 1), True, 32, 0.2067, 0.005),
        # the same as a laser-amplitude sweep of 8 solves (the bench's default)
        _case("tmd22_rk4_batch8", 22, (72, 72, 1), True, 16, 0.2067, 0.005, batch=8),
        # the third configuration's stepper (at a time step where it is stable)
        _case("tmd22_ab4", 22, (72, 72, 1), True, 64, 0.08, 0.005, solver="AB"),
        # the Hermitian-plane form on an odd grid, where it is the reference's generator
        _case("tmd22_hplanes81", 22, (81, 81, 1), True, 32, 0.2067, 0.005, form="hplanes"),
        # the batched laser sweep: uneven solves stepped together
        {"name": "sweep16", "kind": "sweep", "solves": 16, "mix": 3, "steps": 64, "dt": 0.2067},
        # one evaluation on a caller's own device buffers
        {"name": "rhs14_hsex", "kind": "rhs", "nb": 14, "n0": 48, "n1": 48, "n2": 1, "coulomb": True, "field": 0.005},
        # the surrogate's training loop at the configuration's feature sizes
        {"name": "mlp_train", "kind": "mlp", "n_in": 259, "n_out": 254, "rows": 4096, "minibatches": 8, "train": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(x):
    return min(SIDES, key=lambda n: abs(n - x))


def _draw_grid(rng, max_points):
    dims = rng.choice([1, 2, 2, 2, 2, 2, 3])
    if dims == 1:
        return (_side(_log(rng, 16, 1024)), 1, 1)
    while True:
        if dims == 2:
            n = _log(rng, 10, 100)
            g = (_side(n * rng.uniform(0.8, 1.25)), _side(n * rng.uniform(0.8, 1.25)), 1)
        else:
            n = _log(rng, 5, 16)
            g = tuple(_side(n * rng.uniform(0.7, 1.4)) for _ in range(3))
        if g[0] * g[1] * g[2] <= max_points:
            return g


def _stable_field(grid, dt, solver):
    """Largest field for which the gradient's rate E R_max times dt stays inside the stepper's stability interval."""
    return (1.2 if solver == "RK" else 0.2) / (dt * 0.87 * BOHR_LATTICE * max(grid) * 1.66)


def _draw_propagate(rng):
    while True:
        coulomb = rng.random() < 0.6
        grid = _draw_grid(rng, 7000 if coulomb else 14400)
        nb = round(_log(rng, 2, 24))
        Nk = grid[0] * grid[1] * grid[2]
        batch = rng.choice([1, 1, 1, 2, 3, 5, 8])
        points = Nk * nb * nb * batch
        if points > 9_000_000:
            continue
        form = "fp64"
        if grid[2] == 1 and grid[1] > 1 and rng.random() < 0.15:
            grid = tuple(n if n % 2 else _side(n - 1) if _side(n - 1) % 2 else 45 for n in grid[:2]) + (1,)
            form = "hplanes" if grid[0] * grid[1] <= 7000 else "fp64"
        solver = "AB" if rng.random() < 0.25 else "RK"
        dt = 0.2067 if solver == "RK" else 0.05
        steps = max(4, min(600, int(4e7 * _log(rng, 0.3, 1.0) / points)))
        return _case(None, nb, grid, coulomb, steps, dt, min(_log(rng, 1e-3, 1e-2), _stable_field(grid, dt, solver)),
                     solver=solver, order=rng.choice([4, 5]) if solver == "AB" else 4, batch=batch, form=form)


def draw(rng):
    kind = rng.choice(["propagate"] * 6 + ["printed", "sweep", "rhs", "mlp"])
    if kind == "propagate":
        return _draw_propagate(rng)
    if kind == "printed":
        grid = _draw_grid(rng, 5000)
        return _case(None, rng.randint(2, 8), grid, rng.random() < 0.5, rng.randint(20, 100), 0.2067,
                     min(0.01, _stable_field(grid, 0.2067, "RK")), kind="printed")
    if kind == "sweep":
        most = next(work(c) for c in listed() if c["kind"] == "sweep")["bytes"]
        while True:
            c = {"kind": "sweep", "solves": rng.randint(3, 16), "mix": rng.randint(10, 10_000), "steps": rng.randint(8, 64), "dt": 0.2067}
            if work(c)["bytes"] <= most:
                return c
    if kind == "rhs":
        while True:
            grid, nb = _draw_grid(rng, 3000), round(_log(rng, 2, 24))
            if grid[0] * grid[1] * grid[2] * nb * nb <= 600_000:
                return {"kind": "rhs", "nb": nb, "n0": grid[0], "n1": grid[1], "n2": grid[2],
                        "coulomb": rng.random() < 0.6, "field": 0.005}
    shells = rng.randint(7, 127)
    return {"kind": "mlp", "n_in": 2 * shells + 5, "n_out": 2 * shells, "rows": round(_log(rng, 16, 8192)),
            "minibatches": rng.randint(1, 8), "train": rng.random() < 0.5}


_PREPARE = {"propagate": _prepare_propagate, "printed": _prepare_printed, "sweep": _prepare_sweep, "rhs": _prepare_rhs, "mlp": _prepare_mlp}
_RUN = {"propagate": _run_propagate, "printed": _run_printed, "sweep": _run_sweep, "rhs": _run_rhs, "mlp": _run_mlp}
_EXACT = {"propagate": _exact_propagate, "printed": _exact_printed, "sweep": _exact_sweep, "rhs": _exact_rhs, "mlp": _exact_mlp}


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def work(case):
    kind = case["kind"]
    if kind in ("propagate", "printed"):
        rhs = case["steps"] * (4 if case["solver"] == "RK" else 1)
        w = _work_steps(_grid(case), case["nb"], case["coulomb"], rhs * case["batch"])
        if kind == "printed":  # the state and the eigenvectors and velocity operator, once a step
            S = case["n0"] * case["n1"] * case["n2"] * case["nb"] ** 2
            w["bytes"] += case["steps"] * 16 * S * 5
        return w
    if kind == "sweep":
        parts = [_work_steps((N, N, 1), nb, False, 4 * case["steps"] * count) for (nb, N), count in _sweep_shapes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "rhs":
        return _work_steps(_grid(case), case["nb"], case["coulomb"], 1)
    d = [case["n_in"], 128, 128, 128, case["n_out"]]
    weights = sum(a * b for a, b in zip(d, d[1:]))
    rows = case["rows"] * case["minibatches"]
    io = 4 * rows * (case["n_in"] + case["n_out"])
    if not case["train"]:
        return {"bytes": io + 4 * weights, "flops": 2.0 * rows * weights}
    return {"bytes": io + case["minibatches"] * 24 * weights, "flops": 6.0 * rows * weights}
