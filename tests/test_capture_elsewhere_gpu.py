"""The plain form's first steps while a stream of the caller's is being captured
in global mode, by this or another thread: the steps are taken, the capture
ends well, and both do what they do apart."""
import threading

import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other_thread", [False, True])
@pytest.mark.parametrize("n", [16, 22])  # compile-time and run-time factors
def test_first_steps_beside_a_capture(n, other_thread):
    torch = pytest.importorskip("torch")
    wl = W.config(1, kT=1.0, grid=n, length=6, form="plain64")
    a, b = (Selm(wl.params, wl.x, wl.mass, topology=wl.topology) for _ in range(2))
    for s in (a, b):
        s.initial()
        s.synchronize()
    a.run(3)
    t = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    failed = []

    def steps():
        try:
            b.run(3)
        except Exception as e:  # raised again below, after the capture has ended
            failed.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
        t += 1
        if other_thread:
            th = threading.Thread(target=steps)
            th.start()
            th.join()
        else:
            steps()
        t += 1
    assert not failed
    g.replay()
    torch.cuda.synchronize()
    assert bool((t == 2).all())
    for p, q in zip(a.particles(), b.particles()):
        np.testing.assert_array_equal(p, q)
    np.testing.assert_array_equal(a.get_field(), b.get_field())
    del g
    a.final()
    b.final()
