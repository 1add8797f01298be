"""The plain form's step as a host force provider sees it: positions, velocity
field and step count are those of the step just taken, and a provider that
fails leaves that step taken (grids of the compile-time, the run-time and the
axis-pass kernels)."""
import numpy as np
import pytest

from monomers2026_b200.selm import FIELD_U, Params, Selm

pytestmark = pytest.mark.gpu


def _sim(n, provider, M=5):
    rng = np.random.default_rng(n)
    p = Params(numMeshPtsPerDir=(n, n, n), box_lo=0.0, box_hi=float(n), form="plain64", dt=0.01, mu=1.0, rho=1.0, KB=1.0,
               T=1.0, flagStochasticDriving=1, SELM_Seed=5)
    s = Selm(p, rng.random((M, 3)) * n, np.ones(M), v=rng.standard_normal((M, 3)))
    s.set_force_callback(lambda x, v: provider(s, x, v))
    s.initial()
    return s


@pytest.mark.parametrize("n", [24, 26, 34])
def test_provider_sees_the_step_as_taken(n):
    seen = []

    def provider(s, x, v):
        px, pv, _ = s.particles()
        seen.append((s.nstep, x, v, px, pv, s.get_field(FIELD_U)))
        return np.full(x.shape, 0.1)

    s = _sim(n, provider)
    for k in range(1, 4):
        s.run(1)
        count, x, v, px, pv, u = seen[k]  # seen[0]: the initial forces
        assert count == k == s.nstep
        for a, b in ((x, px), (v, pv), (px, s.particles()[0]), (pv, s.particles()[1]), (u, s.get_field(FIELD_U))):
            np.testing.assert_array_equal(a, b)
    s.final()


@pytest.mark.parametrize("n", [24, 26, 34])
def test_failing_provider_leaves_the_step_taken(n):
    def steady(s, x, v):
        return np.full(x.shape, 0.1)

    def failing(s, x, v):
        if s.nstep == 2:
            raise RuntimeError("no forces")
        return steady(s, x, v)

    a, b = _sim(n, steady), _sim(n, failing)
    a.run(2)
    with pytest.raises(Exception):
        b.run(2)
    assert b.nstep == 2
    for q in range(2):
        np.testing.assert_array_equal(a.particles()[q], b.particles()[q])
    np.testing.assert_array_equal(a.get_field(FIELD_U), b.get_field(FIELD_U))
    a.final()
    b.final()
