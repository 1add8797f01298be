"""The largest compile-time grids of each form (one plane of shared memory an
SM, second factors up to 14): steps of a few monomers with thermal noise
against the oracle, tolerances as for the other sizes."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu

SIZES_64 = [126, 140, 144, 160]
SIZES_32 = SIZES_64 + [168, 192, 196, 224]


@pytest.mark.parametrize("n,forms", [(n, ("fused64", "plain64", "fused32") if n in SIZES_64 else ("fused32",))
                                     for n in SIZES_32])
def test_largest_planes_match_the_oracle(oracle, n, forms):
    wl = W.config(1, kT=1.0, grid=n, length=6, form="fused64")
    p = wl.params
    v0 = np.random.default_rng(n).normal(0.0, 0.5, wl.x.shape)
    ff = oracle.ForceField(wl.topology.as_dict(), p.box_lo, p.box_hi)
    o = oracle.Sim(p.numMeshPtsPerDir, p.box_lo, p.box_hi, p.dt, p.mu, p.rho, p.KB, p.T, wl.x, wl.mass, v=v0,
                   stochastic=True, seed=p.SELM_Seed, noise_mode=int(p.noise_mode == "exact"), ff=ff)
    o.initial()
    o.step(2)
    for form in forms:
        tol = 1e-5 if form == "fused32" else 1e-11
        p.form = form
        g = Selm(p, wl.x, wl.mass, v=v0, topology=wl.topology)
        g.initial()
        g.run(2)
        x, v, _ = g.particles()
        for a, b in ((x, o.x), (v, o.v), (g.get_field(), o.u)):
            assert np.abs(a - b).max() < tol * np.abs(b).max(), form
        assert g.status() == 0
        g.final()
