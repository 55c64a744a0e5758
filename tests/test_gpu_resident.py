"""Small problems stepped whole in one launch (csrc/resident.cuh) against the
oracle, at the edges of its splits: one CTA and clusters, rows that do not
divide by the CTAs, an axis of one point, 1-D, 2-D and 3-D grids, one to three
stages an axis, odd band counts, radices 11 and 13, models per solve, calls that
continue one another.  The FP64 bar of the other parity tests.  A profiled
handle keeps its launches per stage: the two paths agree to rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import lasers_of, make_pair, model_input, rel

pytestmark = pytest.mark.gpu

SHAPES = [  # nb, grid, coulomb, solver, order
    (1, (8, 4, 1), False, "RK", 4),
    (2, (64, 1, 1), False, "RK", 4),
    (2, (1, 24, 1), False, "RK", 4),
    (2, (50, 50, 1), False, "RK", 4),
    (2, (40, 40, 1), True, "RK", 4),
    (2, (11, 13, 1), True, "AB", 5),
    (3, (6, 9, 1), False, "AB", 4),
    (3, (7, 5, 1), True, "RK", 4),
    (3, (3, 4, 5), False, "RK", 4),
    (5, (9, 1, 1), False, "AB", 5),
    (2, (64, 60, 1), False, "RK", 4),
]


@pytest.mark.parametrize("nb,grid,coulomb,solver,order", SHAPES)
def test_resident_matches_oracle_and_launches(pkg, po, tmp_path, nb, grid, coulomb, solver, order):
    dims = sum(n > 1 for n in grid)
    inp = model_input(pkg, tmp_path, f"res{nb}{grid[0]}{grid[1]}", grid, nb=nb, dims=1 if grid[1] == 1 else max(dims, 2),
                      coulomb=coulomb, solver=solver, order=order, dt=0.005, envelope="gauss")
    if grid[0] == 1:  # the model's hoppings along the one axis the grid has
        uc, Rs, H, r = pkg.workloads.random_model(nb, 0, dims=1)
        Rs = [(0, R[0], 0) for R in Rs]
        pkg.workloads.write_tb(inp["tb_file"] + "_tb.dat", uc, Rs, H, r)
    cfg, o, s = make_pair(pkg, po, inp)
    rho0 = s.get_state()
    n0 = s.kernel_launches
    s.step(5)
    s.step(4)
    launches = s.kernel_launches - n0
    assert launches == 2, "this shape is meant to step in one launch a call"
    got = s.get_state()
    o.step(9)
    assert rel(got, o.get("rho")) < 1e-10
    if solver == "RK":
        s.set_profiling(True)
        s.time = 0.0
        s.set_state(rho0)
        s.step(9)
        assert rel(got, s.get_state()) < 1e-13
        s.set_profiling(False)


def test_resident_models_per_solve(pkg, po, tmp_path):
    E = pkg.edus
    pairs = []
    for seed in (3, 4, 5):
        cfg = po.load_input(model_input(pkg, tmp_path, f"rms{seed}", (10, 12, 1), nb=2, seed=seed, dt=0.01,
                                        envelope="gauss"))
        pairs.append((cfg, po.Oracle(cfg)))
    cfg0, o0 = pairs[0]
    s = E.Solver(cfg0.grid, o0.nb, cfg0.dt, batch=3)
    xi = lambda o: np.stack([o.get("xk"), o.get("yk"), o.get("zk")])  # noqa: E731
    s.upload_model(o0.get("H0k"), xi(o0), o0.lattice())
    for b, (cfg, o) in enumerate(pairs):
        if b:
            s.upload_model_solve(b, o.get("H0k"), xi(o))
        s.set_lasers(lasers_of(pkg, cfg), b)
        s.set_state(o.get("rho"), b)
    n0 = s.kernel_launches
    s.step(12)
    assert s.kernel_launches - n0 == 1
    for b, (cfg, o) in enumerate(pairs):
        o.step(12)
        assert rel(s.get_state(b), o.get("rho")) < 1e-10, b


@pytest.mark.parametrize("nb,grid", [(2, (50, 50, 1)), (8, (9, 13, 1)), (9, (9, 13, 1)), (22, (28, 25, 1))])
def test_observables_against_numpy(pkg, tmp_path, nb, grid):
    """Both observables kernels (a thread per k point up to 8 bands, a CTA above),
    twice (the counter of finished CTAs resets): sums of Nk nb^2 products of order
    one, so 1e-12 of the largest; the repeat is bitwise the same."""
    inp = model_input(pkg, tmp_path, f"obs{nb}", grid, nb=nb, dt=0.01, envelope="gauss")
    m = pkg.model.Model(pkg.model.parse_input(inp))
    s = m.solver()
    rng = np.random.default_rng(1)
    rho = rng.normal(size=s.shape) + 1j * rng.normal(size=s.shape)
    vel = rng.normal(size=(3,) + s.shape) + 1j * rng.normal(size=(3,) + s.shape)
    s.upload_observables(U=m.U, vel=vel)
    s.set_state(rho)
    nk = rho.shape[0]
    bl = np.einsum("kin,kij,kjn->n", m.U.conj(), rho, m.U).real / nk
    wn = np.einsum("knn->n", rho).real / nk
    v = np.einsum("dknl,kln->d", vel, rho) / nk
    first = s.observables(0, 0)
    for got, ref in zip(first, (bl, wn, v)):
        assert np.abs(got - ref).max() < 1e-12 * max(1.0, np.abs(ref).max())
    again = s.observables(0, 0)
    assert all(np.array_equal(a, b) for a, b in zip(first, again))
