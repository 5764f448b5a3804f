"""Marching substeps that sweep back and forth (fields larger than L2) take the
same steps, bit for bit, as those that always sweep upwards and as the
shared-memory planes kernel: a batch whose grids exceed L2 only together
against each grid alone, and one grid that exceeds it by itself."""
import ctypes as C

import numpy as np
import pytest

from nrpyelliptic_b200 import _lib
from nrpyelliptic_b200.batch import relax_batch, relax_batch_mixed
from nrpyelliptic_b200.problem import DeviceState, Problem, sample_sweep, with_grid

pytestmark = pytest.mark.gpu
PLANES, MARCH = 15, (20, 18)  # tile shapes


@pytest.fixture()
def lib():
    lib = _lib.load()
    lib.nrpyell_clear_status()
    yield lib
    lib.nrpyell_set_tile(-1)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("tile", MARCH)
def test_batch_beyond_l2_matches_single_grids(lib, tile, mixed):
    grids = [(130, 125, 14), (128, 128, 16), (144, 140, 18)] * 2 + [(144, 144, 18)]
    probs = [Problem(with_grid(c, g), lib=lib, host_aux=False, device_tables=True)
             for c, g in zip(sample_sweep(len(grids)), grids)]
    field_bytes = sum(p.Ntot for p in probs) * (13 * 4 if mixed else 11 * 8)
    assert field_bytes > 160e6 and max(p.Ntot for p in probs) * 88 < 100e6
    lib.nrpyell_set_tile(tile)
    run = lambda ps: (relax_batch_mixed(ps, tol=-30.0, switch=-30.0, fold_every=17, max_steps=30, lib=lib) if mixed
                      else relax_batch(ps, tol=-30.0, max_steps=21, lib=lib))
    together = run(probs)
    for i, p in enumerate(probs):
        one = run([p])
        np.testing.assert_array_equal(together[-1][i].download("y_n"), one[-1][0].download("y_n"), err_msg=str(grids[i]))
        together[-1][i].free()
        one[-1][0].free()


@pytest.mark.parametrize("grid", [(209, 215, 26), (224, 210, 28)])
def test_grid_beyond_l2_matches_planes_kernel(lib, grid):
    prob = Problem(with_grid(sample_sweep(2)[1], grid), lib=lib, host_aux=False, device_tables=True)
    assert prob.Ntot * 88 > 140e6
    ys = []
    for tile in (PLANES,) + MARCH:
        ds = DeviceState(prob, lib=lib)
        lib.nrpyell_set_tile(tile)
        n, f = C.c_int(0), C.c_double(0)
        lib.nrpyell_relax(C.byref(ds.g), prob.dt, -30.0, 19, prob.cfg.R_L2, C.byref(n), C.byref(f), None)
        _lib.check(lib)
        ys.append(ds.download("y_n"))
        ds.free()
    for y in ys[1:]:
        np.testing.assert_array_equal(y, ys[0])
