"""Creation and the adjoint use host threads where the system gives them: without any they give the same results
(a process whose thread limit is reached).  A child process preloads a pthread_create that fails on request."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
PY = Path(__file__).resolve().parents[1] / "vocalsim-2p5d-fdtd_b200" / "python"
SHIM = """
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
static int refuse, refused;
int threads_refused(int on) { refuse = on; return refused; }
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    int (*real)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*) = dlsym(RTLD_NEXT, "pthread_create");
    if (refuse) { ++refused; return EAGAIN; }
    return real(t, a, f, x);
}
"""
CHILD = """
import ctypes, sys
import numpy as np
import vocalsim_b200 as V
from vocalsim_b200 import synthetic as S
shim = ctypes.CDLL(sys.argv[1])
seed = np.ones((6, 90), np.float32)
def go():
    b = V.Batch([V.params(cross_sectional_shape=2) for _ in range(6)], [V.Geometry(*S.batch_tube(k)[:2]) for k in range(6)])
    out = [b.forward_ckpt(90, 32)]
    maps, gz = b.adjoint(seed)
    b.close()
    return out + [gz] + [g for m in maps for g in m]
want = go()
shim.threads_refused(1)
got = go()
assert shim.threads_refused(0) > 0
for x, y in zip(got, want):
    np.testing.assert_array_equal(x, y)
print("same")
"""


def test_without_host_threads(tmp_path, cuda_ok):
    (tmp_path / "shim.c").write_text(SHIM)
    so = tmp_path / "shim.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(tmp_path / "shim.c"), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, str(so)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(PY)))
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
