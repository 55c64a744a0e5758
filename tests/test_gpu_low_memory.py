"""Calls that fit the device's memory with little to spare.  The rest of it is
held by one array of this process, so an allocation that does not fit returns an
error code.
"""
import numpy as np
import pytest

from test_gpu_parity import lasers_of, model_input, rel

pytestmark = pytest.mark.gpu

NB, GRID, BATCH = 22, (63, 64, 1), 4
STATE = NB * NB * GRID[0] * GRID[1] * 16 * BATCH  # 125 MB


@pytest.fixture
def hold_all_but():
    """hold_all_but(n): allocate device memory until n bytes are left."""
    import torch

    held = []

    def hold(n):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - n, dtype=torch.uint8, device="cuda"))
        return held

    yield hold
    held.clear()
    torch.cuda.empty_cache()


@pytest.mark.parametrize("late", [False, True])
def test_optional_array_gives_way(pkg, po, tmp_path, hold_all_but, late):
    """A large handle without HSEX keeps H0 + E.xi while there is room.  Where
    creation (late: an upload after it) needs that room, the array gives way and
    the steps agree to rounding (the direct-load commutator's)."""
    cfg = po.load_input(model_input(pkg, tmp_path, "lowmem", GRID, nb=NB, dt=0.005, envelope="gauss"))
    o = po.Oracle(cfg)

    def run(s):
        s.time = 0.0
        for b in range(BATCH):
            s.set_lasers(lasers_of(pkg, cfg), b)
            s.set_state(o.get("rho"), b)
        s.step(3)
        return s.get_state(1)

    def solver():
        s = pkg.edus.Solver(cfg.grid, NB, cfg.dt, batch=BATCH)
        s.upload_model(o.get("H0k"), np.stack([o.get("xk"), o.get("yk"), o.get("zk")]), o.lattice())
        return s

    s = solver()
    full, ref = s.device_bytes, run(s)
    if late:
        hold_all_but(STATE // 8)  # less than the eigenvectors, STATE / 4
        s.upload_observables(U=np.broadcast_to(np.eye(NB, dtype=complex), s.shape))
        assert s.device_bytes < full
    else:
        s.close()
        hold_all_but(full - STATE // 2)
        s = solver()
        assert s.device_bytes == full - STATE
    assert rel(run(s), ref) < 1e-13


def test_sets_of_buffers_are_completed_by_the_next_call(pkg, po, tmp_path, hold_all_but):
    """Buffers that serve together: when the allocation of the second fails, the
    call reports it and the next one, with room again, takes what is missing."""
    E = pkg.edus
    cfg = po.load_input(model_input(pkg, tmp_path, "lowset", GRID, nb=NB, coulomb=True, dt=0.005, envelope="gauss"))
    o = po.Oracle(cfg)
    s = E.Solver(cfg.grid, NB, cfg.dt, coulomb=True)
    s.upload_model(o.get("H0k"), np.stack([o.get("xk"), o.get("yk"), o.get("zk")]), o.lattice(), o.get("W"),
                   o.get("DM0R"), o.hartree())
    s.set_lasers(lasers_of(pkg, cfg))
    s.set_state(o.get("rho"))
    rho, one = o.get("rho"), STATE // BATCH

    def release(held):
        import torch

        held.clear()
        torch.cuda.empty_cache()

    held = hold_all_but(one + one // 2)
    vel = np.zeros((3,) + s.shape, dtype=complex)
    with pytest.raises(E.EdusError) as ei:
        s.upload_observables(vel=vel)  # room for one of its three arrays
    assert ei.value.code == 6
    s._has_vel = True  # the binding's own note of an upload: the library is asked
    with pytest.raises(E.EdusError) as ei:
        s.observables(0, 0)
    assert ei.value.code == 1
    release(held)
    held = hold_all_but(one + one // 2)
    with pytest.raises(E.EdusError) as ei:
        s.rhs(3.0, rho)  # room for one of its two arrays
    assert ei.value.code == 6
    release(held)
    assert rel(s.rhs(3.0, rho), o.rhs(3.0, rho)) < 1e-10
    s.upload_observables(vel=vel)
    assert np.array_equal(s.observables(0, 0)[2], np.zeros(3))
