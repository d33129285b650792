"""Runs a Python script in a child process whose cudaMalloc goes through a shim:
the script reads the sizes of the calls made so far and has chosen calls answer
cudaErrorMemoryAllocation, on the host, without asking the device for memory."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
static size_t lo = 1, hi, sizes[65536];
static int skip, fail, made;
/* of the calls for lo to hi bytes: the first `skip_` pass, the next `fail_` fail */
void shim_fail(size_t lo_, size_t hi_, int skip_, int fail_) { lo = lo_; hi = hi_; skip = skip_; fail = fail_; }
int shim_left(void) { return fail; }
int shim_made(void) { return made; }
size_t shim_size(int k) { return sizes[k]; }
int cudaMalloc(void **p, size_t n)
{
    static int (*real)(void **, size_t);
    if (!real) real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_NOW), "cudaMalloc");
    if (made < 65536) sizes[made++] = n;
    if (n >= lo && n <= hi && fail > 0) {
        if (skip > 0) skip--;
        else return fail--, 2;
    }
    return real(p, n);
}
"""

HEAD = """
import ctypes as C, sys
sys.path[:0] = [{root!r}, {root!r} + "/oracle", {root!r} + "/tests"]
import numpy as np
import __graft_entry__ as ge
import qmin_oracle as oracle
from cases import gpu_lattice, rel_err
qmin = ge.load_package()
oracle.build()
shim = C.CDLL({so!r})
shim.shim_size.restype = C.c_size_t
shim.shim_fail.argtypes = [C.c_size_t, C.c_size_t, C.c_int, C.c_int]
def sizes(since=0):
    return [shim.shim_size(k) for k in range(since, shim.shim_made())]
"""


def run(script, tmp_path):
    c, so, py = tmp_path / "shim.c", tmp_path / "shim.so", tmp_path / "script.py"
    c.write_text(SHIM)
    r = subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(c), "-o", str(so), "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    py.write_text(HEAD.format(root=ROOT, so=str(so)) + textwrap.dedent(script))
    r = subprocess.run([sys.executable, str(py)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0, r.stdout + r.stderr
