"""The first call on new tables gives the same result as the second: the tables
have arrived on the GPU before a kernel reads them."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

from nrpyelliptic_b200 import _lib, abi
from nrpyelliptic_b200.problem import Problem, sample_sweep, with_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(64, 64, 8), (252, 256, 6)])
def test_first_l2_norm_equals_second(grid):
    lib = _lib.load()
    prob = Problem(with_grid(sample_sweep(1)[0], grid), lib=lib, host_aux=False, device_tables=True)
    f = torch.rand(2 * prob.Ntot, dtype=torch.float64, generator=torch.Generator().manual_seed(1)).cuda()
    torch.cuda.synchronize()
    for i in range(30):  # each radius has volume weights of its own

        def norm():
            return lib.L2_norm_of_gf(C.byref(prob.params), abi.UUGF, 50.0 + i, prob.xx, C.cast(f.data_ptr(), abi.PREAL))

        first = norm()
        assert first == norm()
    _lib.check(lib)
