"""Grids with a prime factor above 13 (the Stockham passes' p-point DFT): the
prime alone, as the first or the last of several factors, odd and even, the
smallest and the largest, thermal noise on, against the oracle.  A p-point sum
rounds to about p eps of the field's maximum: 61 x 1e-16 and 61 x 6e-8 a pass
at worst, 1e-11 and 1e-5 as for the other sizes."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("fused64", 1e-11), ("fused32", 1e-5), ("plain64", 1e-11)])
@pytest.mark.parametrize("n", [17, 34, 51, 59, 61, 68])
def test_prime_sizes_match_the_oracle(oracle, n, form, tol):
    wl = W.config(1, kT=1.0, grid=n, length=6, form=form)
    p = wl.params
    p.noise_mode = "exact"
    ff = oracle.ForceField(wl.topology.as_dict(), p.box_lo, p.box_hi)
    o = oracle.Sim(p.numMeshPtsPerDir, p.box_lo, p.box_hi, p.dt, p.mu, p.rho, p.KB, p.T, wl.x, wl.mass,
                   stochastic=True, seed=p.SELM_Seed, noise_mode=1, ff=ff)
    o.initial()
    o.step(2)
    g = Selm(p, wl.x, wl.mass, topology=wl.topology)
    g.initial()
    g.run(2)
    assert np.abs(g.get_field() - o.u).max() < tol * np.abs(o.u).max()
    assert g.status() == 0
    g.final()
