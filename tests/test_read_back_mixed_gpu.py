"""One read-back into arrays of different kinds: pageable, page-locked and
device memory in one call, just around the staging limit.  Each array gets what
it gets alone; an array that the copy refuses is an error, and never written
by the host."""
import ctypes as C
import itertools

import numpy as np
import pytest

from monomers2026_b200 import _lib
from monomers2026_b200.selm import Params, Selm, host_register, host_unregister

pytestmark = pytest.mark.gpu
DP = C.POINTER(C.c_double)


def _sim(M):
    rng = np.random.default_rng(M)
    p = Params(numMeshPtsPerDir=(16, 16, 16), box_lo=0.0, box_hi=16.0, form="fused32")
    s = Selm(p, rng.random((M, 3)) * 16.0, np.ones(M), v=rng.standard_normal((M, 3)))
    s.initial()
    s.run(2)
    s.synchronize()
    return s


@pytest.mark.parametrize("M", [37, 8192, 8193])
def test_page_locked_beside_pageable(M):
    s = _sim(M)
    ref = s.particles()
    for locked in itertools.product([False, True], repeat=3):
        out = [np.zeros((M, 3)) for _ in range(3)]
        for a, k in zip(out, locked):
            if k:
                host_register(a)
        _lib.check(_lib.load().selm_get_particles(s._h, *[a.ctypes.data_as(DP) for a in out]))
        for a, k in zip(out, locked):
            if k:
                host_unregister(a)
        for a, r in zip(out, ref):
            assert np.array_equal(a, r)
    s.final()


@pytest.mark.parametrize("where", [0, 1, 2])
@pytest.mark.parametrize("M", [37, 8193])
def test_device_array_beside_pageable(M, where):
    """The copy engine's answer for a device array (done, or refused with an
    error) is the same whatever the arrays beside it are."""
    torch = pytest.importorskip("torch")
    s = _sim(M)
    ref = s.particles()
    L = _lib.load()
    dev = torch.zeros((M, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    alone = [None] * 3
    alone[where] = C.cast(dev.data_ptr(), DP)
    rc_alone = L.selm_get_particles(s._h, *alone)
    out = [np.zeros((M, 3)) for _ in range(3)]
    mixed = [a.ctypes.data_as(DP) for a in out]
    mixed[where] = alone[where]
    rc = L.selm_get_particles(s._h, *mixed)
    assert rc == rc_alone
    if rc == 0:
        assert np.array_equal(dev.cpu().numpy(), ref[where])
        for i in range(3):
            if i != where:
                assert np.array_equal(out[i], ref[i])
    s.final()
