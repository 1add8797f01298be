"""The three forms at grid sizes of the run-time factor kernels (one, two and
three factors, odd sizes, an odd number of row pairs) and of the compile-time
even sizes (second factors 5 to 9, odd and even), thermal noise on, against the
oracle.  Tolerances: a step's rounding is about 1e-15 (FP64) and
3e-7 (FP32) of the field's maximum; 1e-11 and 1e-5 as for the other sizes."""
import numpy as np
import pytest

from monomers2026_b200 import workloads as W
from monomers2026_b200.selm import Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,tol", [("fused64", 1e-11), ("fused32", 1e-5), ("plain64", 1e-11)])
@pytest.mark.parametrize("n,integrator,noise", [(7, "inertial", "ref_compat"), (13, "quasi_steady", "exact"),
                                               (20, "inertial", "exact"), (25, "inertial", "ref_compat"),
                                               (33, "quasi_steady", "ref_compat"), (42, "inertial", "ref_compat"),
                                               (125, "inertial", "exact"), (36, "inertial", "ref_compat"),
                                               (50, "inertial", "exact"), (54, "quasi_steady", "ref_compat"),
                                               (70, "inertial", "ref_compat"), (98, "inertial", "exact")])
def test_run_time_sizes_match_the_oracle(oracle, n, integrator, noise, form, tol):
    if form == "plain64" and integrator != "inertial":
        pytest.skip("the plain form has the inertial integrator only")
    wl = W.config(1, kT=1.0, grid=n, length=6, form=form)
    p = wl.params
    p.integrator, p.noise_mode = integrator, noise
    v0 = np.random.default_rng(n).normal(0.0, 0.5, wl.x.shape)
    ff = oracle.ForceField(wl.topology.as_dict(), p.box_lo, p.box_hi)
    o = oracle.Sim(p.numMeshPtsPerDir, p.box_lo, p.box_hi, p.dt, p.mu, p.rho, p.KB, p.T, wl.x, wl.mass, v=v0,
                   stochastic=True, seed=p.SELM_Seed, noise_mode=int(noise == "exact"), ff=ff,
                   integrator=int(integrator == "quasi_steady"))
    o.initial()
    o.step(3)
    g = Selm(p, wl.x, wl.mass, v=v0, topology=wl.topology)
    g.initial()
    g.run(3)
    x, v, _ = g.particles()
    for a, b in ((x, o.x), (v, o.v), (g.get_field(), o.u)):
        assert np.abs(a - b).max() < tol * np.abs(b).max()
    assert g.status() == 0
    g.final()
