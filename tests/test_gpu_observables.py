"""Observables against numpy where the sums split: a thread or a CTA per k point
(four and five bands), one CTA, 32 and 33 (one group of sums or two), more groups
than a round of loads takes, and several k points a CTA.  Sums of Nk nb^2 products of order
one: 1e-12 of the largest; a repeat is bitwise the same (the counters reset).
"""
import numpy as np
import pytest

from test_gpu_parity import model_input

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,grid", [(1, (1, 3, 1)), (4, (64, 64, 1)), (4, (65, 63, 1)), (4, (100, 96, 1)),
                                     (5, (32, 1, 1)), (5, (33, 1, 1)), (5, (25, 33, 1)), (5, (72, 72, 1)),
                                     (24, (44, 45, 1)), (40, (9, 13, 1))])
def test_observables_against_numpy(pkg, tmp_path, nb, grid):
    E = pkg.edus
    s = E.Solver(grid, nb, 0.05)
    nk = grid[0] * grid[1] * grid[2]
    rng = np.random.default_rng(nb)
    rand = lambda *n: rng.normal(size=n) + 1j * rng.normal(size=n)  # noqa: E731
    rho, U, vel, H = rand(nk, nb, nb), rand(nk, nb, nb) / nb ** 0.5, rand(3, nk, nb, nb), rand(nk, nb, nb)
    s.upload_model(H, np.stack([H] * 3), np.eye(3) * 6.0)
    s.upload_observables(U=U, vel=vel)
    s.set_state(rho)
    bl = np.einsum("kin,kij,kjn->n", U.conj(), rho, U, optimize=True).real / nk
    wn = np.einsum("knn->n", rho).real / nk
    v = np.einsum("dknl,kln->d", vel, rho) / nk
    first = s.observables(0, 0)
    for got, ref in zip(first, (bl, wn, v)):
        assert np.abs(got - ref).max() < 1e-12 * max(1.0, np.abs(ref).max())
    assert all(np.array_equal(a, b) for a, b in zip(first, s.observables(0, 0)))


def test_sums_round_no_more_than_pairwise(pkg):
    """Wannier populations are sums of Nk given numbers: the CTAs' sums (20 on 50 x 50) are added
    pairwise, and so are the warps' lanes, so the error stays below 16 units of 2^-53 of
    the sum of magnitudes (about log2 of the 2500 terms, and 4 more for the CTA's warps)."""
    import math

    s = pkg.edus.Solver((50, 50, 1), 2, 0.05)
    H = np.zeros(s.shape, dtype=complex)
    s.upload_model(H, np.stack([H] * 3), np.eye(3) * 6.0)
    rng = np.random.default_rng(3)
    rho = rng.uniform(0.1, 1.0, s.shape).astype(complex)
    s.set_state(rho)
    wn = s.observables(0, 0)[1]
    for n in range(2):
        exact = math.fsum(rho[:, n, n].real) / 2500
        assert abs(wn[n] - exact) <= 16 * 2.0 ** -53 * exact
