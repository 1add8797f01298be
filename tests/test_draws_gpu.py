"""The spectral update's draws against 64-bit references, by test kernels built
from the product's own headers."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("draws") / "libdraws.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Xcompiler", "-fPIC", "-shared", "--expt-relaxed-constexpr", "-o", so,
                    os.path.join(HERE, "draws_probe.cu")], check=True)
    return C.CDLL(so)


def normals(words):
    """The Box-Muller pairs of Philox words [..., 4] in extended precision, and their radius."""
    w = words.astype(np.uint64)
    x1, x2 = ((w[..., i] << np.uint64(20)) | (w[..., i + 1] >> np.uint64(12)) for i in (0, 2))
    x1, x2 = x1.astype(LD) + LD(0.5), x2.astype(LD) + LD(0.5)
    full = LD(2) ** 52
    r = np.sqrt(2 * np.where(x1 > full / 2, -np.log1p((x1 - full) / full), -np.log(x1 / full)))
    quarters = 4 * x2 / full
    n = np.rint(quarters)
    a = (quarters - n) * (PI / 2)
    n = n.astype(int) % 4
    s, c = np.sin(a), np.cos(a)
    return (r * np.choose(n, [c, -s, -c, s]), r * np.choose(n, [s, c, -s, -c])), r


def _words(probe, n, k, seed, steps):
    out = np.zeros((steps, 3, 4), np.uint32)
    q = k * n * (n // 2 + 1)
    assert probe.probe_words(C.c_ulonglong(seed), C.c_uint(q), C.c_ulonglong(1), steps, out.ctypes.data_as(C.c_void_p)) == 0
    return out


def _mode(probe, n, k, seed, steps, amp, exact):
    out = np.zeros((steps, 3, 2), np.float32)
    assert probe.probe_mode(n, k, C.c_ulonglong(seed), C.c_ulonglong(1), steps, C.c_double(amp), exact,
                            out.ctypes.data_as(C.c_void_p)) == 0
    return out


def test_fp32_grids_draw_fp64_normals(probe):
    """The FP32 grids that are not tuned draw in FP64 and round once: mode
    (0, 0, n/2), its own conjugate, of 200000 draws each the nearest FP32 number.
    (FP64 rounding, some 1e-15, moves one in 1e8 of them across.)"""
    n, amp = 10, 0.37
    got = _mode(probe, n, n // 2, 11, 100000, amp, 0)[:, :2]
    (z, _), _ = normals(_words(probe, n, n // 2, 11, 100000))
    want = (z[:, :2] * (LD(amp) * 2)).astype(np.float32)  # sqrt(lambda) = 2
    np.testing.assert_array_equal(got[..., 0], want)
    assert not got[..., 1].any()


@pytest.mark.parametrize("exact", [0, 1])
def test_fp32_grids_average_in_fp64(probe, exact):
    """The Hermitian average of mode (0, 0, k) with the conjugate of (0, 0, -k)
    on those grids: of 400000 values each the nearest FP32 number (an average
    of rounded draws is one in about half of them)."""
    n, k, amp = 10, 3, 0.37
    got = _mode(probe, n, k, 11, 100000, amp, exact)[:, :2]
    (zr, zi), _ = normals(_words(probe, n, k, 11, 100000))
    (cr, ci), _ = normals(_words(probe, n, n - k, 11, 100000))
    scale = LD(amp) * 2 * np.sin(PI * k / n) * np.sqrt(LD(0.5)) * (np.sqrt(LD(0.5)) if exact else LD(0.5))
    np.testing.assert_array_equal(got[..., 0], ((zr + cr) * scale)[:, :2].astype(np.float32))
    np.testing.assert_array_equal(got[..., 1], ((zi - ci) * scale)[:, :2].astype(np.float32))


def _normals(probe, fp32, words):
    words = np.ascontiguousarray(words, np.uint32)
    out = np.zeros((len(words), 2))
    assert probe.probe_normals(fp32, len(words), words.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p)) == 0
    return out


def test_fp32_angle_takes_all_bits_of_its_uniform(probe):
    """The angle's uniform has 52 bits, 20 of them in the fourth word: where the
    third leaves FP32 room for them (angles below 2^-14 turns) some draws
    change with the fourth word, to no more than the rounding of r sin."""
    words = np.random.default_rng(3).integers(0, 2**32, (200000, 4), np.uint64).astype(np.uint32)
    words[:, 2] >>= 14
    z = []
    for w3 in (0, 0xFFFFFFFF):
        words[:, 3] = w3
        z.append(_normals(probe, 1, words))
    assert (z[0] != z[1]).any()
    assert np.abs(z[0] - z[1]).max() < 9 * 2.0**-21
