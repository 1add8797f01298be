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


def _edge_words():
    """Both sides of u1 = 3/4 (the FP32 form's switch), 1/2, 1/sqrt 2 and
    1/(2 sqrt 2) (the FP64 form's), u1 and u2 next to 0 and 1, quarter and
    eighth turns, and whole words of zeros and ones below them."""
    hi = [0, 1, 2, 0x1FFFFFFF, 0x20000000, 0x3FFFFFFF, 0x40000000, 0x5A827999, 0x5A82799A, 0x5FFFFFFF, 0x60000000,
          0x7FFFFFFF, 0x80000000, 0x9FFFFFFF, 0xA0000000, 0xB504F333, 0xB504F334, 0xBFFFFFFF, 0xC0000000, 0xDFFFFFFF,
          0xE0000000, 0xFFFFFFFE, 0xFFFFFFFF]
    lo = [0, 0xFFF, 0x1000, 0x80000000, 0xFFFFF000, 0xFFFFFFFF]
    return np.stack(np.meshgrid(hi, lo, hi, lo, indexing="ij"), -1).reshape(-1, 4).astype(np.uint32)


def _random_words(where):
    words = np.random.default_rng(5).integers(0, 2**32, (500000, 4), np.uint64).astype(np.uint32)
    if where == "u1 near 0":
        words[:, 0] >>= 18
    elif where == "u1 near 1":
        words[:, 0] = ~(words[:, 0] >> 18)
    elif where == "u2 near 0":
        words[:, 2] >>= 18
    return words


@pytest.mark.parametrize("where", ["edges", "anywhere", "u1 near 0", "u1 near 1", "u2 near 0"])
def test_normals_match_extended_precision(probe, where):
    """FP64: relative error within 4 2^-52 (half an ulp from the logarithm, one
    each from the root, the angle and the sine, half from the product).  FP32:
    within 11 2^-23 of the radius: 2^-21.2 for the fast sine and cosine (3.5),
    pi 2^-23 for the rounding of their argument, and 4 for the radius (its
    fast quotient's 2 ulp, the sums, the root, the product)."""
    words = _edge_words() if where == "edges" else _random_words(where)
    want, r = normals(words)
    want = np.stack(want, 1)
    z64, z32 = (_normals(probe, fp32, words) for fp32 in (0, 1))
    assert (np.abs(z64 - want) <= 4 * LD(2) ** -52 * np.abs(want)).all()
    assert (np.abs(z32 - want) <= 11 * LD(2) ** -23 * r[:, None]).all()
