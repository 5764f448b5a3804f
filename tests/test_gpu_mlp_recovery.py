"""A network handle that met a non-finite minibatch gives the gradients of a
fresh one once its weights and inputs are finite again: no operand keeps
anything of an earlier pass.  Output and hidden widths are no multiples of 16,
so that every padding of an operand is in use, and the output layer's rows are
shorter, as long as and longer than a hidden layer's."""
import numpy as np
import pytest
from test_gpu_mlp import Dev

from nrpyelliptic_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n_in,width,depth,n_out,rows", [(13, 64, 2, 41, 20), (13, 40, 3, 41, 33), (7, 72, 4, 130, 17),
                                                         (5, 130, 1, 3, 31)])
def test_gradients_after_a_non_finite_minibatch(n_in, width, depth, n_out, rows, bad):
    lib = _lib.load()
    lib.nrpyell_clear_status()
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    t = rng.normal(size=(rows, n_out)).astype(np.float32)
    dx, dt = Dev(lib, x), Dev(lib, t)
    dbad = Dev(lib, np.full((64, n_in), bad, np.float32))
    dtbad = Dev(lib, np.full((64, n_out), bad, np.float32))
    out = []
    for spoil in (False, True):
        m = lib.nrpyell_mlp_create(n_in, width, depth, n_out, 64, 3)
        _lib.check(lib)
        n = lib.nrpyell_mlp_num_params(m)
        p, g = np.empty(n, np.float32), np.empty(n, np.float32)
        lib.nrpyell_mlp_get_params(m, p.ctypes.data)
        if spoil:
            lib.nrpyell_mlp_loss_grad(m, dbad.p, dtbad.p, 64, None)
            lib.nrpyell_mlp_train(m, dbad.p, dtbad.p, 64, 32, 1, np.float32(1e-3), 1, None)
            assert lib.nrpyell_mlp_set_params(m, p.ctypes.data) == 0
        loss = lib.nrpyell_mlp_loss_grad(m, dx.p, dt.p, rows, g.ctypes.data)
        out.append((loss, g))
        lib.nrpyell_mlp_destroy(m)
    _lib.check(lib)
    assert np.isfinite(out[0][1]).all()
    np.testing.assert_allclose(out[1][0], out[0][0], rtol=1e-12)  # the loss is summed in any order
    np.testing.assert_array_equal(out[1][1], out[0][1])
