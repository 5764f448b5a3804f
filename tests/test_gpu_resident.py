"""On-chip relaxation (kernels_resident.cu) against the substep kernels: the
same steps bit for bit, the same stop decision and the residual history to
rounding (the residual sum is split over other blocks), on grids whose tiles
are full and ragged, a single tile along i1, the shortest i2, and sizes next
to the largest that fits.

History tolerance: each entry is log10 of a sum of at most 2^19 positive
terms, whose order changes its relative value by at most 2^19 * 2^-53, i.e.
log10 by 2e-11."""
import ctypes as C

import numpy as np
import pytest
from _util import ptr

from nrpyelliptic_b200 import _lib
from nrpyelliptic_b200.problem import CONFIGS, DeviceState, Problem, sample_sweep, with_grid

pytestmark = pytest.mark.gpu
SUBSTEP_TILE = 15  # a shared-memory planes shape: forcing it turns the on-chip form off
GRIDS = [(12, 5, 6), (17, 9, 6), (24, 17, 8), (33, 40, 12), (64, 64, 8), (90, 75, 10), (48, 200, 6), (100, 40, 14),
         (96, 96, 12), (128, 128, 16)]


@pytest.fixture(scope="module")
def lib():
    lib = _lib.load()
    lib.nrpyell_clear_status()
    yield lib
    lib.nrpyell_set_tile(-1)


def _relax(lib, prob, tile, call):
    """(return code, steps, final, history, y_n, launches) of call(ds, ...) with the tile forced (-1: on chip)."""
    ds = DeviceState(prob, lib=lib)
    steps, fin = C.c_int(-1), C.c_double(0)
    hist = np.zeros(4096)
    lib.nrpyell_set_tile(tile)
    before = lib.nrpyell_launch_count()
    try:
        rc = call(ds, steps, fin, hist)
        _lib.check(lib)
    finally:
        lib.nrpyell_set_tile(-1)
    launches = lib.nrpyell_launch_count() - before
    y = ds.download("y_n")
    ds.free()
    return rc, steps.value, fin.value, hist, y, launches


def _compare(lib, prob, call, max_launches, tile=SUBSTEP_TILE):
    a = _relax(lib, prob, -1, call)
    b = _relax(lib, prob, tile, call)
    assert a[5] <= max_launches < b[5] or b[1] < 4, (a[5], b[5])  # the on-chip form ran
    assert a[:2] == b[:2]
    np.testing.assert_allclose(a[3], b[3], rtol=0, atol=2e-11)
    np.testing.assert_allclose(a[2], b[2], rtol=0, atol=2e-11)
    np.testing.assert_array_equal(a[4], b[4])
    return a


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("steps", [0, 1, 300])
def test_steps_match_substep_kernels(lib, grid, steps):
    prob = Problem(with_grid(sample_sweep(3)[1], grid), lib=lib)

    def call(ds, n, fin, hist):
        return lib.nrpyell_relax(C.byref(ds.g), prob.dt, -12.0, steps, prob.cfg.R_L2, C.byref(n), C.byref(fin),
                                 ptr(hist))

    a = _compare(lib, prob, call, 8)
    assert a[0] == 1 and a[1] == steps


def test_whole_solve_and_thorn_rule(lib):
    prob = Problem(CONFIGS["shipped_64x64x8"], lib=lib)

    def relax(ds, n, fin, hist):
        return lib.nrpyell_relax(C.byref(ds.g), prob.dt, -10.0, 4000, prob.cfg.R_L2, C.byref(n), C.byref(fin),
                                 ptr(hist))

    a = _compare(lib, prob, relax, 16)
    assert a[0] == 0 and abs(a[1] - 1014) <= 1 and a[2] <= -10.0

    def thorn(ds, n, fin, hist):
        return lib.nrpyell_relax_et(C.byref(ds.g), prob.dt, -6.0, 2000, 7, prob.cfg.R_L2, C.byref(n), C.byref(fin))

    a = _compare(lib, prob, thorn, 16)
    assert a[0] == 0 and a[1] % 7 == 0 and a[2] < -6.0


def test_rest_pair_takes_no_step(lib):
    prob = Problem(CONFIGS["equal_mass_rest_64x64x8"], lib=lib)

    def relax(ds, n, fin, hist):
        return lib.nrpyell_relax(C.byref(ds.g), prob.dt, -10.0, 100, prob.cfg.R_L2, C.byref(n), C.byref(fin), ptr(hist))

    a = _compare(lib, prob, relax, 4)
    assert a[0] == 0 and a[1] == 0


MARCH_TILE = 20  # a marching shape: runs the FP32 correction form too


@pytest.mark.parametrize("grid", [(12, 5, 6), (33, 40, 12), (64, 64, 8), (90, 75, 10), (128, 128, 16)])
@pytest.mark.parametrize("switch", [-30.0, -4.0])
def test_correction_form_matches_substep_kernels(lib, grid, switch):
    """The FP32 correction form on chip: stretches of 48 steps and a shorter
    last one, and the switch to FP64."""
    prob = Problem(with_grid(sample_sweep(3)[1], grid), lib=lib)

    def call(ds, n, fin, hist):
        n32, n64 = C.c_int(0), C.c_int(0)
        rc = lib.nrpyell_relax_mixed(C.byref(ds.g), prob.dt, -12.0, switch, 48, 130, prob.cfg.R_L2, C.byref(n32),
                                     C.byref(n64), C.byref(fin), ptr(hist))
        n.value = 1000 * n32.value + n64.value
        return rc

    _compare(lib, prob, call, 60, MARCH_TILE)


@pytest.mark.parametrize("mixed", [False, True])
def test_batches_match_single_runs(lib, mixed):
    """Batches whose grids run on chip, in teams of equal grids and with a team
    cut short, beside grids too large for it: every grid's steps and solution
    are those of its own run."""
    from nrpyelliptic_b200.batch import relax_batch, relax_batch_mixed
    grids = [(24, 17, 8)] * 3 + [(128, 128, 16)] * 2 + [(160, 160, 20)] + [(64, 64, 8)] * 5
    probs = [Problem(with_grid(c, g), lib=lib) for c, g in zip(sample_sweep(len(grids)), grids)]
    if mixed:
        _, s32, s64, fin, states = relax_batch_mixed(probs, tol=-5.0, switch=-4.0, fold_every=100, max_steps=250, lib=lib)
        steps = s32 * 1000 + s64
    else:
        _, steps, fin, states = relax_batch(probs, tol=-5.0, max_steps=250, lib=lib)
    for i, p in enumerate(probs):

        def call(ds, n, f, hist):
            if not mixed:
                return lib.nrpyell_relax(C.byref(ds.g), p.dt, -5.0, 250, p.cfg.R_L2, C.byref(n), C.byref(f), None)
            n32, n64 = C.c_int(0), C.c_int(0)
            rc = lib.nrpyell_relax_mixed(C.byref(ds.g), p.dt, -5.0, -4.0, 100, 250, p.cfg.R_L2, C.byref(n32),
                                         C.byref(n64), C.byref(f), None)
            n.value = 1000 * n32.value + n64.value
            return rc

        one = _relax(lib, p, -1, call)
        assert one[1] == steps[i], grids[i]
        np.testing.assert_allclose(fin[i], one[2], rtol=0, atol=2e-11)
        np.testing.assert_array_equal(states[i].download("y_n"), one[4], err_msg=str(grids[i]))
        states[i].free()
