"""The network's products at the edges of their tiles, and the POD
reconstruction's two variants.

Products: layers narrower and wider than a tile and than the ring of K chunks,
widths and outputs that are no multiple of 4, 8, 16 or 32, minibatches from one
row to more than one row tile, no hidden layer; against the BF16 restatement
and tolerances of test_gpu_mlp.py.  POD: odd and even point counts, mode counts
around the 16 that are loaded together, against float64 numpy (the kernel
accumulates in float64: 1e-13 of the largest value covers a sum of 300 terms)."""
import numpy as np
import pytest
from test_gpu_mlp import Dev, forward, grads, unpack

from nrpyelliptic_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = _lib.load()
    lib.nrpyell_clear_status()
    return lib


@pytest.mark.parametrize("n_in,width,depth,n_out,rows", [
    (1, 1, 1, 1, 1), (13, 33, 2, 7, 15), (13, 64, 1, 32, 16), (20, 130, 2, 41, 17), (13, 600, 2, 250, 129),
    (70, 40, 0, 36, 128), (13, 512, 2, 256, 200), (5, 1030, 1, 3, 31)])
def test_products(lib, n_in, width, depth, n_out, rows):
    dims = [n_in] + [width] * depth + [n_out]
    m = lib.nrpyell_mlp_create(n_in, width, depth, n_out, 200, 3)
    _lib.check(lib)
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    t = rng.normal(size=(rows, n_out)).astype(np.float32)
    p = np.empty(lib.nrpyell_mlp_num_params(m), np.float32)
    lib.nrpyell_mlp_get_params(m, p.ctypes.data)
    p += rng.normal(size=p.size).astype(np.float32) * 0.01  # biases too
    lib.nrpyell_mlp_set_params(m, p.ctypes.data)
    layers = unpack(p, dims)
    full = Dev(lib, np.ones((200, n_in)))  # a larger call first: its rows must not leak into the next
    dx, dt, dy = Dev(lib, x), Dev(lib, t), Dev(lib, np.zeros((200, n_out)))
    assert lib.nrpyell_mlp_predict(m, full.p, 200, dy.p) == 0
    assert lib.nrpyell_mlp_predict(m, dx.p, rows, dy.p) == 0
    y_ref = forward(layers, x)[-1]
    assert np.max(np.abs(dy.get((200, n_out))[:rows] - y_ref)) < 2e-3 * np.max(np.abs(y_ref))
    g = np.empty_like(p)
    loss = lib.nrpyell_mlp_loss_grad(m, dx.p, dt.p, rows, g.ctypes.data)
    _lib.check(lib)
    loss_ref, g_ref = grads(layers, x, t)
    assert abs(loss - loss_ref) < 1e-3 * loss_ref
    for (gW, gb), (rW, rb) in zip(unpack(g, dims), g_ref):
        assert np.max(np.abs(gW - rW)) < 2e-2 * np.max(np.abs(rW))
        assert np.max(np.abs(gb - rb)) < 2e-2 * np.max(np.abs(rb))
    for d in (full, dx, dt, dy):
        d.free()
    lib.nrpyell_mlp_destroy(m)


@pytest.mark.parametrize("ntot", [1, 2, 511, 512, 4097])
@pytest.mark.parametrize("K", [1, 15, 16, 17, 300])
def test_pod_reconstruction(lib, ntot, K):
    rng = np.random.default_rng(K)
    mean, basis, c = (rng.normal(size=s).astype(np.float32) for s in ((ntot,), (K, ntot), (K,)))
    dm, db, dc, dy = Dev(lib, mean), Dev(lib, basis), Dev(lib, c), Dev(lib, np.zeros(4 * ntot))
    assert lib.nrpyell_pod_guess(dm.p, db.p, K, ntot, dc.p, 7.0, dy.p) == 0
    y = dy.get((4 * ntot,)).view(np.float64).reshape(2, ntot)
    ref = mean.astype(np.float64) + c.astype(np.float64) @ basis.astype(np.float64)
    np.testing.assert_allclose(y[0], ref, rtol=0, atol=1e-13 * (1 + np.max(np.abs(ref))))
    np.testing.assert_array_equal(y[1], 7.0 * y[0])
    for d in (dm, db, dc, dy):
        d.free()
