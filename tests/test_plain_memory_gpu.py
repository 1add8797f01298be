"""Device memory of the plain form's grid: two velocities, forcing and pressure
(ten values a cell), and the half spectra of the forcing's three components;
that of the pressure besides only where the captured step solves for it beside the draw."""
import numpy as np
import pytest

from monomers2026_b200.selm import Params, Selm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,parts", [(68, 3), (122, 3), (64, 4), (66, 4)])
def test_half_spectra(n, parts):
    p = Params(numMeshPtsPerDir=(n, n, n), box_lo=0.0, box_hi=float(n), form="plain64")
    s = Selm(p, np.full((1, 3), 1.0), np.ones(1))
    N, N2 = n**3, n * n * (n // 2 + 1)
    assert 0 <= s.device_bytes() - 8 * (10 * N + 2 * parts * N2) < 8 * N2
    s.final()
