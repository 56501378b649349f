"""The inference kernel at the edges of its tiles and of its grid, and on
buffers without the alignment its wide loads and stores ask for."""
import ctypes as C

import numpy as np
import pytest

import mlp_oracle as mo
from pigfem_assignment_b200 import _lib

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one row, a tile's edges, and one tile more than the 148 x 7 CTAs of a full grid take at once
@pytest.mark.parametrize("n", [1, 127, 128, 129, 148 * 7 * 128 + 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward_at_tile_edges(n, shift):
    rng = np.random.default_rng(n)
    p = mo.init_params(1)
    p["W3"] = (rng.standard_normal((16, 64)) * 0.2).astype(np.float32)
    for k, size in (("b1", 64), ("b2", 64), ("b3", 16)):
        p[k] = (0.1 * rng.standard_normal(size)).astype(np.float32)
    h = C.c_void_p()
    _lib.check(_lib.lib.pg_mlp_create(0, 7, C.byref(h)))
    v = np.concatenate([p[k].ravel() for k in ("W1", "b1", "W2", "b2", "W3", "b3")]).astype(np.float32)
    _lib.check(_lib.lib.pg_mlp_params(h, v.ctypes.data_as(C.POINTER(C.c_float)), 1))
    x = rng.standard_normal((n, 16)).astype(np.float32)
    X = torch.zeros(16 * n + 1, device="cuda")
    X[shift:shift + 16 * n] = torch.from_numpy(x.ravel()).cuda()
    Y = torch.full((2 * n + 2,), 7.0, device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.lib.pg_mlp_forward(h, C.c_void_p(X.data_ptr() + 4 * shift), n, C.c_void_p(Y.data_ptr() + 4 * shift), None))
    y = Y.cpu().numpy()
    _lib.lib.pg_mlp_destroy(h)
    assert (y[2 * n + shift:] == 7.0).all() and (y[:shift] == 7.0).all()
    yo, _ = mo.forward(p, x)
    scale = np.abs(yo[:, :2]).max()
    assert np.abs(y[shift:shift + 2 * n].reshape(n, 2) - yo[:, :2]).max() <= 2e-2 * scale
