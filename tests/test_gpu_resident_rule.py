"""Which handles step in one launch, where graph replays of long calls are the
faster form: 3 bands on 64 x 64 without HSEX keep their launches under RK4 (17.3 us a
stage replayed, 19.9 in one launch) and step in one launch under Adams-Bashforth,
which has no graphs (28.9 us launched).  Calls of any length take the same form, so split calls agree bitwise.
"""
import numpy as np
import pytest

from test_gpu_parity import make_pair, model_input, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver,one_launch", [("RK", False), ("AB", True)])
def test_choice_and_split_calls(pkg, po, tmp_path, solver, one_launch):
    inp = model_input(pkg, tmp_path, "resrule" + solver, (64, 64, 1), nb=3, solver=solver, order=4, dt=0.002,
                      envelope="gauss")
    cfg, o, s = make_pair(pkg, po, inp)
    rho0 = s.get_state()
    n0 = s.kernel_launches
    s.step(6)
    assert s.kernel_launches - n0 == (1 if one_launch else 6 * 16)
    o.step(6)
    assert rel(s.get_state(), o.get("rho")) < 1e-10
    if solver == "RK":
        s.time = 0.0
        s.set_state(rho0)
        s.step(520)  # replayed
        whole = s.get_state()
        s.time = 0.0
        s.set_state(rho0)
        for _ in range(4):
            s.step(130)
        assert np.array_equal(s.get_state(), whole)
