"""The spectral update takes the modes of the planes i = 0 and i = nx/2 last in
each block: grids where a block holds several such columns, one of a pair, the
last or none, odd and even, thermal noise on, against the oracle (tolerances as
for the other sizes)."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("fused64", 1e-11), ("fused32", 1e-5)])
@pytest.mark.parametrize("n,integrator,noise", [(6, "inertial", "exact"), (9, "inertial", "exact"),
                                               (16, "quasi_steady", "exact"), (22, "inertial", "exact"),
                                               (30, "inertial", "ref_compat"), (34, "inertial", "exact"),
                                               (64, "inertial", "exact"),
                                               # plane kernels with more threads than equal rounds need
                                               (60, "inertial", "exact"), (84, "inertial", "ref_compat"),
                                               (112, "inertial", "exact")])
def test_edge_modes_match_the_oracle(oracle, n, integrator, noise, form, tol):
    wl = W.config(1, kT=1.0, grid=n, length=6, form=form)
    p = wl.params
    p.integrator, p.noise_mode = integrator, noise
    ff = oracle.ForceField(wl.topology.as_dict(), p.box_lo, p.box_hi)
    o = oracle.Sim(p.numMeshPtsPerDir, p.box_lo, p.box_hi, p.dt, p.mu, p.rho, p.KB, p.T, wl.x, wl.mass,
                   stochastic=True, seed=p.SELM_Seed, noise_mode=int(noise == "exact"), ff=ff,
                   integrator=int(integrator == "quasi_steady"))
    o.initial()
    o.step(3)
    g = Selm(p, wl.x, wl.mass, topology=wl.topology)
    g.initial()
    g.run(3)
    assert np.abs(g.get_field() - o.u).max() < tol * np.abs(o.u).max()
    g.final()
