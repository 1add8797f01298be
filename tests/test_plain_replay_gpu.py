"""A read-back of the plain form after replays of steps that the caller
recorded is ordered after them, also where steps of the library's own lie
between the recording and the replays."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


def test_read_back_follows_the_replays():
    torch = pytest.importorskip("torch")
    wl = W.config(1, kT=1.0, grid=64, length=6, form="plain64")
    a, b = (Selm(wl.params, wl.x, wl.mass, topology=wl.topology) for _ in range(2))
    st = torch.cuda.Stream()
    a.set_stream(st.cuda_stream)
    a.initial()
    b.initial()
    a.run(2)
    a.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        a.run(2)
    a.run(2)
    with torch.cuda.stream(st):
        for _ in range(200):
            g.replay()
    got = a.particles()
    b.run(404)
    for p, q in zip(got, b.particles()):
        np.testing.assert_array_equal(p, q)
    a.synchronize()
    del g
    a.final()
    b.final()
