"""States of 32 MB and more without HSEX (12 to 24 bands) take the TMA-fed
commutator, with H0 + E.xi written when E changes: against the oracle at the
FP64 bar, and against the same solves in small handles (the direct-load
kernel), with which they agree to rounding.  Odd and even band counts, k points
that do not divide by the tile of 4, a model per solve, both steppers, and a
right-hand side between steps (which leaves another field's H behind).
"""
import numpy as np
import pytest

from test_gpu_parity import lasers_of, model_input, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,grid,batch,solver", [(22, (40, 39, 1), 3, "RK"), (13, (55, 45, 1), 6, "RK"),
                                                  (12, (45, 45, 1), 8, "AB")])
def test_large_ipa_matches_oracle_and_small_handles(pkg, po, tmp_path, nb, grid, batch, solver):
    E = pkg.edus
    assert nb * nb * grid[0] * grid[1] * 16 * batch >= 32 << 20 > nb * nb * grid[0] * grid[1] * 16
    pairs = []
    for seed in (1, 2):
        cfg = po.load_input(model_input(pkg, tmp_path, f"ipa{nb}_{seed}", grid, nb=nb, seed=seed, solver=solver, dt=0.005,
                                        envelope="gauss"))
        pairs.append((cfg, po.Oracle(cfg)))
    xi = lambda o: np.stack([o.get("xk"), o.get("yk"), o.get("zk")])  # noqa: E731
    cfg0, o0 = pairs[0]
    big = E.Solver(cfg0.grid, nb, cfg0.dt, solver=cfg0.solver, order=cfg0.order, batch=batch)
    big.upload_model(o0.get("H0k"), xi(o0), o0.lattice())
    big.upload_model_solve(1, pairs[1][1].get("H0k"), xi(pairs[1][1]))
    which = lambda b: 1 if b == 1 else 0  # noqa: E731
    for b in range(batch):
        big.set_lasers(lasers_of(pkg, pairs[which(b)][0]), b)
        big.set_state(pairs[which(b)][1].get("rho"), b)
    small = []
    for cfg, o in pairs:
        s = E.Solver(cfg.grid, nb, cfg.dt, solver=cfg.solver, order=cfg.order)
        s.upload_model(o.get("H0k"), xi(o), o.lattice())
        s.set_lasers(lasers_of(pkg, cfg))
        s.set_state(o.get("rho"))
        small.append(s)
    rho = o0.get("rho")
    big.step(2)
    assert rel(big.rhs(9.0, rho), o0.rhs(9.0, rho)) < 1e-10
    big.step(1)
    for (cfg, o), s in zip(pairs, small):
        o.step(3)
        s.step(3)
    for b in range(batch):
        got = big.get_state(b)
        assert rel(got, pairs[which(b)][1].get("rho")) < 1e-10, b
        assert rel(got, small[which(b)].get_state()) < 1e-13, b
