"""Read-backs into pageable and page-locked arrays, of few monomers and just
around the staging limit, by several threads at once: the same bytes."""
import ctypes as C
import threading

import numpy as np
import pytest

from monomers2026_b200 import _lib
from monomers2026_b200.selm import Params, Selm, host_register, host_unregister

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 37, 8192, 8193])
def test_read_back_is_the_same_through_every_path(M):
    rng = np.random.default_rng(M)
    p = Params(numMeshPtsPerDir=(16, 16, 16), box_lo=0.0, box_hi=16.0, form="fused32")
    sims = [Selm(p, rng.random((M, 3)) * 16.0, np.ones(M), v=rng.standard_normal((M, 3))) for _ in range(3)]
    dp = C.POINTER(C.c_double)
    ref = []
    for s in sims:
        s.initial()
        s.run(2)
        a = [np.zeros((M, 3)) for _ in range(3)]
        for q in a:
            host_register(q)
        _lib.check(_lib.load().selm_get_particles(s._h, *[q.ctypes.data_as(dp) for q in a]))
        for q in a:
            host_unregister(q)
        ref.append([q.copy() for q in a])
    got = [None] * 3

    def read(k):
        for _ in range(20):
            got[k] = sims[k].particles()

    ts = [threading.Thread(target=read, args=(k,)) for k in range(3)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for r, g in zip(ref, got):
        for a, b in zip(r, g):
            assert np.array_equal(a, b)
    only = np.zeros((M, 3))  # one of the three arrays
    _lib.check(_lib.load().selm_get_particles(sims[0]._h, None, only.ctypes.data_as(dp), None))
    assert np.array_equal(only, ref[0][1])
    [s.final() for s in sims]
