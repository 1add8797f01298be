"""The reference-structured form's captured step is the step kernel by kernel,
bit for bit, on the simulation's own stream, on the legacy default stream and
in a graph that the caller records."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stream", [(7, None), (24, None), (26, 1), (30, 1), (64, None)])
def test_overlapped_steps_equal_single_ones(n, stream):
    wl = W.config(1, kT=1.0, grid=n, length=6, form="plain64")

    def sim():
        s = Selm(wl.params, wl.x, wl.mass, topology=wl.topology)
        s.set_stream(stream)
        s.initial()
        return s

    a, b = sim(), sim()
    b.profile(True)
    for _ in range(3):
        a.run(20)  # captured, no wait between the steps
        for _ in range(20):  # kernel by kernel, one step a call
            b.run(1)
            b.synchronize()
        for p, q in zip(a.particles(), b.particles()):
            np.testing.assert_array_equal(p, q)
        np.testing.assert_array_equal(a.get_field(), b.get_field())
    assert a.status() == 0 and b.status() == 0
    a.final()
    b.final()


def test_steps_recorded_by_the_caller():
    """Two steps recorded into the caller's graph and replayed are the steps."""
    torch = pytest.importorskip("torch")
    wl = W.config(1, kT=1.0, grid=24, length=6, form="plain64")
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
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    b.run(8)
    for p, q in zip(a.particles(), b.particles()):
        np.testing.assert_array_equal(p, q)
    np.testing.assert_array_equal(a.get_field(), b.get_field())
    del g
    a.final()
    b.final()
