"""The first upload of a per-step round trip, which makes its staging buffers,
while steps are still running: the state is what was uploaded."""
import ctypes as C

import numpy as np
import pytest

from monomers2026_b200 import _lib
from monomers2026_b200.selm import Params, Selm

pytestmark = pytest.mark.gpu
DP = C.POINTER(C.c_double)


@pytest.mark.parametrize("form", ["plain64", "fused64", "fused32"])
@pytest.mark.parametrize("busy", [0, 300])
def test_first_upload_beside_running_steps(form, busy):
    n, M = 64, 5000
    rng = np.random.default_rng(4)
    p = Params(numMeshPtsPerDir=(n, n, n), box_lo=0.0, box_hi=float(n), form=form)
    s = Selm(p, rng.random((M, 3)) * n, np.ones(M))
    s.initial()
    x, v = rng.random((M, 3)) * n, rng.standard_normal((M, 3))
    s.run(1)
    s.synchronize()
    s.run(busy)
    _lib.check(_lib.load().selm_set_particles(s._h, M, x.ctypes.data_as(DP), v.ctypes.data_as(DP), None))
    gx, gv, _ = s.particles()
    np.testing.assert_array_equal(gx, x)
    np.testing.assert_array_equal(gv, v)
    assert s.status() == 0
    s.final()
