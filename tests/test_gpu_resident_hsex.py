"""One-launch steps with HSEX and several solves, on 2-D and 3-D grids (two arrays
exchanged between the CTAs of a cluster, rows that do not divide by them), against the same
handle's launches per stage (a profiled handle keeps them), which the oracle checks elsewhere.
Solves differ in state and field; both forms sum in FP64 in another order: 1e-13 of the largest.
"""
import numpy as np
import pytest

from test_gpu_parity import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,grid,batch,solver,order", [
    (3, (8, 8, 8), 8, "RK", 4),    # clusters of 8
    (4, (8, 8, 8), 8, "AB", 5),
    (3, (9, 8, 6), 12, "RK", 4),   # 9 rows over 5 CTAs
    (2, (36, 36, 1), 5, "RK", 4),  # clusters of 12
])
def test_batches_match_launches(pkg, nb, grid, batch, solver, order):
    E = pkg.edus
    rng = np.random.default_rng(nb + batch)
    nk = grid[0] * grid[1] * grid[2]

    def herm(*n):
        a = rng.normal(size=n + (nb, nb)) + 1j * rng.normal(size=n + (nb, nb))
        return 0.05 * (a + np.conj(np.swapaxes(a, -1, -2)))

    W = rng.uniform(0.0, 1e-2, (nk, nb, nb)).astype(complex)
    model = (herm(nk), herm(3, nk), np.diag([5.0, 6.0, 7.0]), W, herm(nk) / nk, herm().real.astype(complex))
    states = [herm(nk) for _ in range(batch)]
    out = []
    for profiled in (False, True):
        s = E.Solver(grid, nb, 0.02, solver=E.SOLVER_RK if solver == "RK" else E.SOLVER_AB, order=order, coulomb=True,
                     batch=batch)
        s.upload_model(*model)
        for b in range(batch):
            s.set_lasers([E.Laser(intensity=(1e-3 * (b + 1)) ** 2, omega=0.07, pol=(1.0, 0.5, 0.2), t0=0.0,
                                  phase=0.3 * b, fwhm=400.0, envelope=E.ENVELOPE_GAUSS)], b)
            s.set_state(states[b], b)
        s.set_profiling(profiled)
        n0 = s.kernel_launches
        s.step(11)
        assert (s.kernel_launches - n0 == 1) != profiled
        out.append([s.get_state(b) for b in range(batch)])
    for b in range(batch):
        assert rel(out[0][b], states[b]) > 1e-4  # it moved
        assert rel(out[0][b], out[1][b]) < 1e-13, b
