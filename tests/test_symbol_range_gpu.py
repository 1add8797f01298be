"""Mode symbols beyond FP32's range: the spectral update's quotients and root
are FP64 whatever the form.  Cells of 2^-63 and 2^-64 (in the unit of the case)
put 2/dx^2, and with it the Laplacian's symbol, above the largest FP32 number,
while the velocity and the first differences stay inside; the viscosity
goes with dx^2, so that the viscous factor is that of unit cells.

Tolerance against the FP64 form: 1e-5 as for the other sizes.  1/L, stored in
FP32, is below FP32's normal numbers there: |L| <= 12 / dx^2 < 2^134 leaves it
above 2^-134, 15 bits or more, and 2^-15 of the projection's part of the modes
with the largest |L| only; at 2^-64 it is 17 bits, 8e-6."""
import numpy as np
import pytest

from monomers2026_b200.selm import Params, Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["inertial", "quasi_steady"])
@pytest.mark.parametrize("exponent", [0, -62, -63, -64])
@pytest.mark.parametrize("n", [21, 24, 36])  # run-time factors, tuned and other compile-time sizes
def test_small_cells(n, exponent, integrator):
    dx = 2.0 ** exponent
    u = []
    for form in ("fused64", "fused32"):
        p = Params(numMeshPtsPerDir=(n, n, n), box_lo=0.0, box_hi=n * dx, form=form, integrator=integrator, dt=0.01,
                   mu=dx * dx, rho=1.0, KB=1.0, T=dx ** (2 if integrator == "inertial" else 3), flagStochasticDriving=1,
                   SELM_Seed=7)
        s = Selm(p, np.full((1, 3), n * dx / 3), np.ones(1))
        s.initial()
        s.run(3)
        u.append(s.get_field())
        s.final()
    assert np.abs(u[0]).max() > 0.0
    assert np.abs(u[1] - u[0]).max() < 1e-5 * np.abs(u[0]).max()
