"""A bounded wait of the network's kernels that runs out (poll limit zero: no
fault, no hang) leaves weights, moments and the step count as they were, is
reported as a timeout by the next call that returns host data, and by that call
only.  Both forms of the network: hidden width 128 and another.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,n_out,batch", [(128, 19, 300), (128, 400, 130), (48, 19, 300)])
def test_timed_out_step_changes_nothing_and_is_reported(pkg, hidden, n_out, batch):
    import torch

    E = pkg.edus
    rng = np.random.default_rng(7)
    x = torch.as_tensor(rng.normal(size=(batch, 24)).astype(np.float32), device="cuda")
    t = torch.as_tensor(rng.normal(size=(batch, n_out)).astype(np.float32), device="cuda")
    torch.cuda.synchronize()
    net, ref = (pkg.surrogate.MLP(24, n_out, hidden=hidden, seed=3) for _ in range(2))
    for m in (net, ref):
        m.train_step(x, t, 1e-3)
    before = net.params()
    net.set_wait_limit(0)
    with pytest.raises(E.EdusError) as ei:
        net.train_step(x, t, 1e-3)
    assert ei.value.code == 3
    assert np.array_equal(net.params(), before)
    # steps that do not read the loss: the weights are asked for later
    for _ in range(2):
        assert net._L.edus_mlp_train_step(net._h, batch, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(t.data_ptr()),
                                          ctypes.c_float(1e-3), None) == 0
    with pytest.raises(E.EdusError) as ei:
        net.params()
    assert ei.value.code == 3
    with pytest.raises(E.EdusError):
        net.forward(x)
    net.set_wait_limit(-1)
    assert np.array_equal(net.params(), before)
    # the next step is the second of both networks: Adam's moments and step count are those of one step
    net.train_step(x, t, 1e-3)
    ref.train_step(x, t, 1e-3)
    assert np.array_equal(net.params(), ref.params())


def test_parameters_set_while_a_timeout_is_pending(pkg):
    """Steps since a wait ran out are left out until that is reported, also after new parameters; the
    step count then is that of the new parameters: none."""
    import torch

    E = pkg.edus
    rng = np.random.default_rng(8)
    x = torch.as_tensor(rng.normal(size=(200, 24)).astype(np.float32), device="cuda")
    t = torch.as_tensor(rng.normal(size=(200, 19)).astype(np.float32), device="cuda")
    torch.cuda.synchronize()
    net, ref = (pkg.surrogate.MLP(24, 19, seed=3) for _ in range(2))

    def unread_step(m):
        assert m._L.edus_mlp_train_step(m._h, 200, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(t.data_ptr()),
                                        ctypes.c_float(1e-3), None) == 0

    start = net.params()
    net.set_wait_limit(0)
    for _ in range(3):
        unread_step(net)
    net.set_wait_limit(-1)
    net.set_params(start)
    unread_step(net)
    with pytest.raises(E.EdusError):
        net.params()
    assert np.array_equal(net.params(), start)
    for m in (net, ref):
        m.train_step(x, t, 1e-3)
    assert np.array_equal(net.params(), ref.params())
