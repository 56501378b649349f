"""Training past a completion wait that ran out: the epoch ends with the error,
and the network, its moments and its step count are those of the minibatches
that were applied."""
import ctypes as C

import numpy as np
import pytest

from pigfem_assignment_b200 import _lib, learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("times", [1, 3])
def test_training_goes_on_as_if_the_timed_out_epoch_had_not_been(times):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda:0").manual_seed(3)
    X = torch.randn(1000, 16, generator=g, device="cuda:0")
    T = -torch.rand(1000, 2, generator=g, device="cuda:0")
    nets = [learned.MLP(0, seed=5) for _ in range(2)]
    for net in nets:
        net.train(X, T, epochs=2, batch=300)
    before = nets[0].params()
    for _ in range(times):
        assert _lib.lib.pg_mlp_wait_selftest(nets[0].handle, 1000) == _lib.PG_ERR_STATE
        assert b"timed out" in _lib.lib.pg_last_error()
        assert np.array_equal(nets[0].params(), before)
    losses = [net.train(X, T, epochs=2, batch=300) for net in nets]
    assert np.array_equal(nets[0].params(), nets[1].params())
    assert np.array_equal(losses[0], losses[1])
