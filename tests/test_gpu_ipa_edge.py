"""Where the TMA-fed commutator without HSEX begins: 12 MB of state, 14 MB under
Adams-Bashforth with 16 bands.  On either side of the edge the handle takes the
launches it should (the new form writes H0 + E.xi in one more launch a stage) and
matches the oracle; the same solve agrees across the edge to rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import lasers_of, model_input, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,grid,batches,solver,extra", [
    (22, (26, 21, 1), (2, 3), "RK", (0, 4)),     # millions of bytes: 8.5 and 12.7
    (13, (26, 30, 1), (5, 6), "AB", (0, 1)),     # 10.5 and 12.7
    (16, (28, 28, 1), (4, 5), "AB", (0, 1)),     # 12.8 and 16.1: the later edge
    (16, (28, 28, 1), (3, 4), "RK", (0, 4)),     # 9.6 and 12.8
])
def test_edge(pkg, po, tmp_path, nb, grid, batches, solver, extra):
    E = pkg.edus
    cfg = po.load_input(model_input(pkg, tmp_path, f"edge{nb}", grid, nb=nb, solver=solver, dt=0.005, envelope="gauss"))
    o = po.Oracle(cfg)
    base = {"RK": 8, "AB": 2}[solver]
    out = []
    for batch, more in zip(batches, extra):
        edge = (14 if solver == "AB" and nb == 16 else 12) << 20
        assert (nb * nb * grid[0] * grid[1] * 16 * batch >= edge) == bool(more)
        s = E.Solver(cfg.grid, nb, cfg.dt, solver=cfg.solver, order=cfg.order, batch=batch)
        s.upload_model(o.get("H0k"), np.stack([o.get("xk"), o.get("yk"), o.get("zk")]), o.lattice())
        for b in range(batch):
            s.set_lasers(lasers_of(pkg, cfg), b)
            s.set_state(o.get("rho"), b)
        n0 = s.kernel_launches
        s.step(3)
        assert s.kernel_launches - n0 == 3 * (base + more)
        out.append(s.get_state(batch - 1))
    o.step(3)
    assert rel(out[0], o.get("rho")) < 1e-10
    assert rel(out[1], out[0]) < 1e-13
