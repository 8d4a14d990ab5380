"""div_by as common.cuh has it (its host form, compiled here) against the division: the same bits for operands and
quotients well inside the normal range, and for a zero over anything."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_the_headers_own_form(tmp_path):
    src, so = tmp_path / "div.cu", tmp_path / "libdiv.so"
    src.write_text('#include "common.cuh"\n'
                   'extern "C" void quotients(long n, const double* a, const double* d, double* q){\n'
                   '    for(long i = 0; i < n; i++) q[i] = aturan::div_by(a[i], d[i], 1.0 / d[i]);\n}\n')
    subprocess.check_call([NVCC, "-std=c++17", "-O2", "-Xcompiler", "-fPIC,-ffp-contract=off", "-shared",
                           "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(ROOT, "include"),
                           "-I" + os.path.join(ROOT, "aturan_b200", "csrc"), "-o", str(so), str(src)])
    rng = np.random.default_rng(3)
    n = 400000
    a, d = (rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-200, 200, n) for _ in range(2))
    a[:1000] = 0.0
    a[1000:2000] = d[1000:2000] * rng.integers(1, 1 << 20, 1000)       # exact quotients
    a[2000:3000] = np.nextafter(a[1000:2000], np.inf)
    q = np.empty(n)
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    ctypes.CDLL(str(so)).quotients(ctypes.c_long(n), p(a), p(d), p(q))
    assert np.array_equal(q, a / d)
