"""Which handles the fused sweep's launches take, and that each solve equals the
same solve stepped alone, bit for bit.  The fused launches are counted on the first handle
they take, so the counts tell the handles apart.
"""
import numpy as np
import pytest

from test_gpu_parity import lasers_of, model_input

pytestmark = pytest.mark.gpu


def make(pkg, po, tmp_path, shapes):
    E = pkg.edus
    out = []
    for i, (nb, grid, batch) in enumerate(shapes):
        cfg = po.load_input(model_input(pkg, tmp_path, f"swf{i}", grid, nb=nb, seed=30 + i, dt=0.005, envelope="gauss"))
        o = po.Oracle(cfg)
        pair = []
        for _ in range(2):
            s = E.Solver(cfg.grid, nb, cfg.dt, batch=batch)
            s.upload_model(o.get("H0k"), np.stack([o.get("xk"), o.get("yk"), o.get("zk")]), o.lattice())
            for b in range(batch):
                s.set_lasers(lasers_of(pkg, cfg), b)
                s.set_state(o.get("rho"), b)
            pair.append(s)
        out.append(pair)
    return out


def check(pkg, pairs, steps, launches, **kw):
    n0 = [s.kernel_launches for s, _ in pairs]
    pkg.edus.sweep_step([s for s, _ in pairs], steps, **kw)
    assert [s.kernel_launches - n for (s, _), n in zip(pairs, n0)] == launches
    for s, alone in pairs:
        alone.step(steps)
        assert s.time == alone.time
        for b in range(s.batch):
            assert np.array_equal(s.get_state(b), alone.get_state(b)), (s.nb, b)


@pytest.mark.parametrize("steps", [3, 34])
def test_large_states_step_as_alone(pkg, po, tmp_path, steps):
    """22 bands on 48 x 48, two solves (36 MB): the TMA-fed commutator, in the
    sweep as alone, beside a fused shape."""
    pairs = make(pkg, po, tmp_path, [(22, (48, 48, 1), 2), (7, (36, 36, 1), 4)])
    check(pkg, pairs, steps, [12 * steps, 8 * steps], fused=True)


def test_handle_limit_counts_every_handle(pkg):
    """More than 64 handles are refused, however they would step (these: each in one launch)."""
    E = pkg.edus
    H = np.zeros((16, 2, 2), dtype=complex)
    ss = []
    for _ in range(65):
        s = E.Solver((4, 4, 1), 2, 0.05)
        s.upload_model(H, np.stack([H] * 3), np.eye(3))
        ss.append(s)
    with pytest.raises(E.EdusError) as ei:
        E.sweep_step(ss, 2, fused=True)
    assert ei.value.code == 5 and ss[0].time == 0.0
    E.sweep_step(ss[:64], 2, fused=True)
    assert ss[0].time == 0.1
