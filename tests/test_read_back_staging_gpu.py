"""Read-backs page-lock no memory: the staging buffers come with the
simulation's monomers, a bounded number of them, and go with the last
simulation.  A child process counts the runtime's page-locked allocations
through its own cudaHostAlloc and cudaFreeHost, which pass the calls on."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COUNTER = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int host_allocs = 0, host_frees = 0;
static void* runtime(const char* name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY), name); }
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
  __sync_fetch_and_add(&host_allocs, 1);
  return ((int (*)(void**, size_t, unsigned))runtime("cudaHostAlloc"))(p, n, flags);
}
int cudaFreeHost(void* p) {
  __sync_fetch_and_add(&host_frees, 1);
  return ((int (*)(void*))runtime("cudaFreeHost"))(p);
}
"""

CHILD = r"""
import ctypes as C, sys, threading
import numpy as np
from monomers2026_b200.selm import Params, Selm
count = C.CDLL(sys.argv[1])
allocs = lambda: C.c_int.in_dll(count, "host_allocs").value
frees = lambda: C.c_int.in_dll(count, "host_frees").value

def sim(M):
    rng = np.random.default_rng(M)
    p = Params(numMeshPtsPerDir=(16, 16, 16), box_lo=0.0, box_hi=16.0, form="fused32")
    s = Selm(p, rng.random((M, 3)) * 16.0, np.ones(M))
    s.initial()
    s.run(1)
    s.synchronize()
    return s

sims = [sim(M) for M in [37] * 10 + [8192, 8193]]
made = allocs()
assert made > 0
for _ in range(3):
    ref = [s.particles() for s in sims]
got = [None] * len(sims)
def read(k):
    for _ in range(10):
        got[k] = sims[k].particles()
ts = [threading.Thread(target=read, args=(k,)) for k in range(len(sims))]
[t.start() for t in ts]
[t.join() for t in ts]
for r, g in zip(ref, got):
    assert all(np.array_equal(a, b) for a, b in zip(r, g))
assert allocs() == made, (made, allocs())
assert made <= 8, made
[s.final() for s in sims]
assert frees() == made, (made, frees())
"""


def test_read_backs_page_lock_nothing(tmp_path):
    src, so = tmp_path / "count.c", tmp_path / "libcount.so"
    src.write_text(COUNTER)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD, str(so)], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
