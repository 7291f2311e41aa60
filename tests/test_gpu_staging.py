"""GPU: copies of pageable host arrays through the pinned slots.

From 4 MiB up and 8 MiB down a copy is shared out over worker threads.  Where the system refuses
threads (a process limit), the calling thread does the parts that are left: a
child process puts a pthread_create that can be told to fail in front of the
system's.
"""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
static int left = -1, refused = 0;
void allow_threads(int n) { left = n; }
int threads_refused(void) { return refused; }
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg)
{
    static int (*real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    if (!real) *(void **)&real = dlsym(RTLD_NEXT, "pthread_create");
    if (left == 0) { ++refused; return EAGAIN; }
    if (left > 0) --left;
    return real(t, a, f, arg);
}
"""

CHILD = r"""
import ctypes, sys
sys.path.insert(0, ROOT)
import numpy as np
import __graft_entry__ as e
e.load_package()
from milc_qphix_b200 import LIB_PATH, capi
shim = ctypes.CDLL(None)
dims = (24, 24, 24, 48)  # 15.2 MiB per parity
lib = capi.QphixLib(LIB_PATH)
assert lib.init(dims) == 0, lib.last_error()
a = np.random.default_rng(3).standard_normal(6 * int(np.prod(dims)))
lib.destroy_V("D", lib.create_V("D", a))  # makes the slots
for n in ALLOWED:
    out = np.zeros_like(a)
    shim.allow_threads(n)
    v = lib.create_V("D", a)
    shim.allow_threads(n)
    if v: lib.extract_V("D", v, out=out)
    shim.allow_threads(-1)
    assert v, lib.last_error()
    assert shim.threads_refused() > 0
    assert np.array_equal(out, a)
    lib.destroy_V("D", v)
lib.finalize()
"""


@pytest.mark.parametrize("allowed", [0, 3])
def test_copies_without_enough_threads(tmp_path, allowed):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    code = f"ROOT = {ROOT!r}\nALLOWED = [{allowed}]\n" + CHILD
    p = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, LD_PRELOAD=str(so)), capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
