"""Rounding of an FP64 fluid step (viscous step, projection, mean) against
extended precision, grids whose sizes have factors 3, 5 and 7.

Bound: with exact twiddles the rms error of a transform grows with the square
root of its butterfly levels, below 2^-53 for each; the step goes through 2 x 3
axes of log2 n levels: 2^-53 sqrt(6 log2 n) of the field.  Twiddles that are off
by more than their rounding add in the same direction on every axis."""
import numpy as np
import pytest

from monomers2026_b200.selm import Params, Selm

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _step(u, mu, rho, dt):
    n = u.shape[1]
    u = u.astype(LD)
    lap = sum(np.roll(u, s, a) for a in (1, 2, 3) for s in (1, -1)) - 6 * u
    us = u + LD(mu) * LD(dt) * lap / LD(rho)
    div = sum(np.roll(us[d], -1, 2 - d) - us[d] for d in range(3))
    s = -4 * np.sin(LD("3.14159265358979323846264338327950288") * np.arange(n).astype(LD) / n) ** 2
    L = s[:, None, None] + s[None, :, None] + s[None, None, : n // 2 + 1]
    L[0, 0, 0] = 1
    p = np.fft.irfftn(np.fft.rfftn(div, axes=(0, 1, 2)) / L, s=(n, n, n), axes=(0, 1, 2))
    for d in range(3):
        us[d] -= p - np.roll(p, 1, 2 - d)
    return us - us.mean(axis=(1, 2, 3), keepdims=True)


@pytest.mark.parametrize("form", ["fused64", "plain64"])
@pytest.mark.parametrize("n", [24, 25, 30, 42, 50, 72, 98, 100])
def test_fp64_step(n, form):
    p = Params(numMeshPtsPerDir=(n, n, n), box_lo=0.0, box_hi=float(n), form=form, dt=0.05, mu=1.3, rho=1.7,
               flagStochasticDriving=0)
    s = Selm(p, np.zeros((0, 3)), np.zeros(0))
    s.initial()
    u0 = np.random.default_rng(n).standard_normal((3, n, n, n))
    s.set_field(0, u0)
    s.run(1)
    want = _step(u0, p.mu, p.rho, p.dt)
    err = np.sqrt(((s.get_field() - want) ** 2).mean() / (want**2).mean())
    assert err < 2.0**-53 * np.sqrt(6 * np.log2(n))
    s.final()
