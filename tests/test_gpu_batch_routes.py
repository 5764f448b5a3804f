"""The two routes of a batch: batched launches with the shape that the tuner
picks over several grids, and on-chip teams whose grids stop in different
launches; and on-chip relaxations that alternate between FP64 and FP32.  Every
grid's steps and solution are those of the substep kernels, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from nrpyelliptic_b200 import _lib
from nrpyelliptic_b200.batch import relax_batch, relax_batch_mixed
from nrpyelliptic_b200.problem import DeviceState, Problem, sample_sweep, with_grid

pytestmark = pytest.mark.gpu
MARCH = 20  # forcing a marching shape turns the on-chip form off
STEPS_PER_LAUNCH = 512


@pytest.fixture()
def lib():
    lib = _lib.load()
    lib.nrpyell_clear_status()
    yield lib
    lib.nrpyell_set_tile(-1)


def _problems(lib, grids):
    return [Problem(with_grid(c, g), lib=lib, host_aux=False, device_tables=True)
            for c, g in zip(sample_sweep(len(grids)), grids)]


def _relax(lib, prob, ds, tol, max_steps):
    n, f = C.c_int(0), C.c_double(0)
    lib.nrpyell_relax(C.byref(ds.g), prob.dt, tol, max_steps, prob.cfg.R_L2, C.byref(n), C.byref(f), None)
    _lib.check(lib)
    return n.value, f.value


def _mixed(lib, prob, ds, tol, switch, fold, max_steps):
    a, b, f = C.c_int(0), C.c_int(0), C.c_double(0)
    lib.nrpyell_relax_mixed(C.byref(ds.g), prob.dt, tol, switch, fold, max_steps, prob.cfg.R_L2, C.byref(a),
                            C.byref(b), C.byref(f), None)
    _lib.check(lib)
    return a.value, b.value


@pytest.mark.parametrize("mixed", [False, True])
def test_tuned_batched_launches_match_single_grids(lib, mixed):
    """Grids too large for the chip, no shape forced: the tuner's shape over
    several grids of different sizes, with blocks of all of them in a launch."""
    grids = [(136, 136, 16), (144, 130, 18), (137, 150, 18), (160, 96, 24)]
    probs = _problems(lib, grids)
    before = lib.nrpyell_launch_count()
    if mixed:
        _, s32, s64, _, states = relax_batch_mixed(probs, tol=-30.0, switch=-30.0, fold_every=16, max_steps=40, lib=lib)
        assert np.all(s32 == 40) and np.all(s64 == 0)
    else:
        _, steps, _, states = relax_batch(probs, tol=-30.0, max_steps=40, lib=lib)
        assert np.all(steps == 40)
    assert lib.nrpyell_launch_count() - before > 4 * 40
    lib.nrpyell_set_tile(MARCH)
    for p, got, g in zip(probs, states, grids):
        ds = DeviceState(p, lib=lib)
        if mixed:
            _mixed(lib, p, ds, -30.0, -30.0, 16, 40)
        else:
            _relax(lib, p, ds, -30.0, 40)
        np.testing.assert_array_equal(got.download("y_n"), ds.download("y_n"), err_msg=str(g))
        ds.free()
        got.free()


@pytest.mark.parametrize("mixed", [False, True])
def test_team_members_stop_in_different_launches(lib, mixed):
    """Five equal grids, one team: one starts near the tolerance, two step with
    shorter time steps, so that they end in launches of their own."""
    probs = _problems(lib, [(24, 17, 8)] * 5)
    probs[1].dt *= 0.25
    probs[3].dt *= 0.5
    runs = []
    for tile in (-1, MARCH):
        states = [DeviceState(p, lib=lib) for p in probs]
        lib.nrpyell_set_tile(MARCH)
        _relax(lib, probs[2], states[2], -8.0, 20000)
        lib.nrpyell_set_tile(tile)
        before = lib.nrpyell_launch_count()
        if mixed:
            rc, s32, s64, _, _ = relax_batch_mixed(probs, states, tol=-8.5, switch=-5.0, fold_every=1024,
                                                   max_steps=20000, lib=lib)
            steps = list(zip(s32, s64))
        else:
            rc, n, _, _ = relax_batch(probs, states, tol=-8.5, max_steps=20000, lib=lib)
            steps = list(n)
            assert len({s // STEPS_PER_LAUNCH for s in steps}) >= 3, steps
        runs.append((rc, steps, [s.download("y_n") for s in states], lib.nrpyell_launch_count() - before))
        for s in states:
            s.free()
    (rc, steps, ys, few), (rc2, steps2, ys2, many) = runs
    assert rc == rc2 == 0 and few * 10 < many
    assert steps == steps2
    for a, b in zip(ys, ys2):
        np.testing.assert_array_equal(a, b)


def test_precisions_alternate_on_chip(lib):
    """FP64 and FP32 relaxations of two grids in turn, many launches of each: no
    exchanged value of one is taken for one of the other."""
    grids = [(33, 40, 12), (64, 64, 8)]
    probs = _problems(lib, grids)
    out = []
    for tile in (-1, MARCH):
        lib.nrpyell_set_tile(tile)
        states = [DeviceState(p, lib=lib) for p in probs]
        steps = []
        for k in range(8):
            for p, ds in zip(probs, states):
                steps.append(_mixed(lib, p, ds, -30.0, -30.0, 7, 50))
                steps.append(_relax(lib, p, ds, -30.0, 33)[0])
        out.append((steps, [s.download("y_n") for s in states]))
        for s in states:
            s.free()
    assert out[0][0] == out[1][0]
    for g, a, b in zip(grids, out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b, err_msg=str(g))
