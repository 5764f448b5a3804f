"""Host code of the GPU drivers, run without a GPU (see _hostlib.py)."""
import ctypes as C

import _hostlib
import numpy as np
import pytest


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return _hostlib.load(tmp_path_factory.mktemp("host"))


def test_exchange_words_hold_tags_of_one_form(lib):
    assert lib.check_exchange_roles() == 0


@pytest.mark.parametrize("stops", [[0], [511], [512], [1600], [0, 1, 1023, 1024], [700, 100], [1600, 0]])
def test_start_state_does_not_depend_on_when_it_is_read(lib, stops):
    assert lib.check_start_state((C.c_int * len(stops))(*stops), len(stops)) == 0


@pytest.mark.parametrize("check_every", [0, 1])
@pytest.mark.parametrize("volume", [0.0, 1e-300, 3.7e-3, 2.5e6])
@pytest.mark.parametrize("tol", [-np.inf, -400.0, -17.5, -16.0, -15.5, -14.9, -10.0, 0.0, 3.0, 154.5, 200.0, np.inf,
                                 np.nan])
def test_stop_test_follows_the_plain_rule(lib, tol, volume, check_every):
    """Sums on both sides of the tolerance, and those a volume without points
    (integration radius below the first cell) or a diverged run gives."""
    near = volume * 10.0 ** (2.0 * min(max(tol, -30.0), 150.0)) if np.isfinite(tol) else 1.0
    sums = np.array([0.0, np.inf, np.nan, 1e-320, 1e-30, 1.0, 1e300]
                    + [near * f for f in (0.5, 1 - 1e-6, 1 - 1e-8, 1 + 1e-8, 1 + 1e-6, 2.0)])
    assert lib.check_stop_rule(C.c_double(tol), C.c_double(volume), check_every,
                               sums.ctypes.data_as(C.POINTER(C.c_double)), len(sums)) == 0


def test_training_order_is_not_reshuffled_under_its_copy(lib):
    """Every epoch's row order reaches the GPU as it was drawn: the memory it is
    copied from stays as it is until the copy has happened."""
    n, epochs, seed = 83, 5, 7
    lib.nrpyell_mlp_create.restype = C.c_void_p
    lib.nrpyell_mlp_train.restype = C.c_double
    lib.fake_logged.restype = C.c_size_t
    q = C.c_void_p(lib.nrpyell_mlp_create(13, 32, 2, 8, 16, 3))
    rows = np.zeros((n, 13), np.float32)
    lib.fake_log_copies(C.c_size_t(4 * n))
    lib.nrpyell_mlp_train(q, rows.ctypes.data_as(C.c_void_p), rows.ctypes.data_as(C.c_void_p), n, 16, epochs,
                          C.c_float(1e-3), seed, None)
    got = np.zeros(2 * epochs * n, np.int32)
    used = lib.fake_logged(got.ctypes.data_as(C.c_void_p), C.c_size_t(got.nbytes))
    lib.fake_log_copies(C.c_size_t(0))
    lib.nrpyell_mlp_destroy(q)
    mask = (1 << 64) - 1
    s, perm, want = 0xD1B54A32D192ED03 ^ seed, list(range(n)), []
    for _ in range(epochs):
        for i in range(n - 1, 0, -1):
            s = (s * 6364136223846793005 + 1442695040888963407) & mask
            j = (s >> 33) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        want.append(list(perm))
    assert used == 4 * epochs * n
    np.testing.assert_array_equal(got[:epochs * n].reshape(epochs, n), want)


@pytest.mark.parametrize("grids,fp64,alternates", [
    ([(144, 144, 18)], 0, 0), ([(144, 144, 18)] * 3, 0, 0), ([(144, 144, 18)] * 5, 0, 1), ([(256, 256, 32)], 0, 1),
    ([(144, 144, 18)] * 2, 1, 0), ([(144, 144, 18)] * 3, 1, 1), ([(192, 192, 24)], 1, 0), ([(224, 224, 28)], 1, 1)])
def test_sweeps_alternate_beyond_l2_only(lib, grids, fp64, alternates):
    """Where the fields of a launch fit in L2 (126 MiB here), sweeping back and
    forth slows a batch by up to 8 %; beyond L2 it saves 3 to 6 %."""
    points = sum((a + 10) * (b + 10) * (c + 10) for a, b, c in grids)
    assert lib.check_alternates(fp64, C.c_double(points)) == alternates


CUBE = {g: (g, g, n2) for g, n2 in ((48, 6), (64, 8), (80, 10), (96, 12), (112, 14), (128, 16), (144, 18))}


@pytest.mark.parametrize("fp64,batch,chip", [
    # microseconds per RK4 step on chip against batched launches
    (1, [48, 64, 80], {48, 64, 80}),              # 38 / 45, and 54 with the smaller two in batched launches
    (1, [48, 64, 80] * 4, {48, 64, 80}),          # 76 / 93
    (1, [48, 48, 96] * 2, {48, 96}),              # 38 / 59
    (0, [48, 48, 96] * 2, {48, 96}),              # 34 / 52
    (0, [48, 48, 96] * 4, {48, 96}),              # 53 / 85
    (1, [48] * 16, {48}),                         # 41 / 77
    (0, [64] * 8, {64}),                          # 34 / 55
    (0, [64] * 16, {64}),                         # 69 / 91
    (0, [80] * 16, {80}),                         # 117 / 139
    (1, [112] * 16, {112}),                       # 328 / 394
    (1, [128] * 16, {128}),                       # 370 / 512
    (0, [128] * 16, {128}),                       # 356 / 371
    (0, [112] * 3, {112}),                        # 68 / 73
    (0, [112] * 4, set()),                        # 92 / 87
    (0, [112] * 8, set()),                        # 182 / 158
    (0, [112] * 16, set()),                       # 361 / 298
    (1, [64, 96, 144], set()),                    # a batch's fixed cost is paid in any case: 12 and 20 / 5 and 15
    (0, [112, 128, 144], set()),                  # 92 with 128 on chip / 88
    (0, [112, 128, 144] * 2, {128}),              # 159 / 165
    (1, [128, 128, 144, 144], {128})])            # 23 / 30 each
def test_batches_take_the_faster_route(lib, fp64, batch, chip):
    """Routes of batches for which both were measured."""
    nxx = np.array([CUBE[g] for g in batch], np.int32)
    team = np.zeros(len(batch), np.int32)
    ip = C.POINTER(C.c_int)
    lib.route_of(fp64, nxx.ctypes.data_as(ip), len(batch), team.ctypes.data_as(ip))
    assert {g for g, t in zip(batch, team) if t} == chip
    assert all(t > 0 for g, t in zip(batch, team) if g in chip)
