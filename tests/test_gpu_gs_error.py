"""A bounded wait of the Gauss-Seidel sweep that ran out sets a word on the device; whatever the caller takes
first after the sweep reports it, not p_dyn alone, for the fields formed from it are as wrong. The word is set
here from the host, through the context's own structure, so no kernel has to hang."""
import os
import shutil
import subprocess

import ctypes
import numpy as np
import pytest

from aturan_b200 import api, params as P, state as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = (12, 20, 33)
PKG = os.path.dirname(os.path.abspath(api.__file__))


@pytest.fixture(scope="module")
def set_word(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("gs_word")
    src, so = d / "word.cu", d / "libgsword.so"
    src.write_text(f'#include "{PKG}/csrc/api.cu"\n'
                   'extern "C" int set_word(aturan_ctx* c, int v){\n'
                   '    return (int)cudaMemcpy(c->gs_err, &v, sizeof v, cudaMemcpyHostToDevice);\n}\n')
    subprocess.check_call([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                           "-I" + os.path.join(os.path.dirname(PKG), "include"), "--expt-relaxed-constexpr", "-shared",
                           "-o", str(so), str(src), "-L" + PKG, "-laturan_b200", "-Xlinker", "-rpath," + PKG])
    L = ctypes.CDLL(str(so))
    L.set_word.argtypes = [ctypes.c_void_p, ctypes.c_int]

    def put(ctx, v):
        torch.cuda.synchronize()                       # the sweep is over
        assert L.set_word(ctx.h, v) == 0
    return put


def _dev(n=1):
    return [torch.empty(SHAPE, dtype=torch.float64, device="cuda") for _ in range(n)]


def _adjoint(ctx):
    y, x = _dev(4), _dev(4)
    for t in y:
        t.fill_(1.0)
    torch.cuda.synchronize()
    ctx.rk4_adjoint([t.data_ptr() for t in y], [t.data_ptr() for t in x])


def _many(ctx, on_device):
    out = _dev(2) if on_device else [np.empty(SHAPE) for _ in range(2)]
    ctx.download_many(["t", "h2o"], [o.data_ptr() if on_device else o.ctypes.data for o in out], on_device=on_device)


TAKES = {
    "download": lambda c: c.download("t"),
    "download_device": lambda c: c.download_device("u", _dev()[0].data_ptr()),
    "download_many": lambda c: _many(c, False),
    "download_many_device": lambda c: _many(c, True),
    "buoy_ref": lambda c: c.buoy_ref_level(),
    "satadj_counts": lambda c: c.satadj(0xF),
    "chemistry_counts": lambda c: c.chemistry(api.CHEM_NH4SH_EQ, counts=True),
    "post_sums": lambda c: c.post_step(sums=True),
    "adjoint": _adjoint,
    "sync": lambda c: c.synchronize(),
}


@pytest.mark.parametrize("take", TAKES)
def test_what_is_taken_first_reports_it(set_word, take):
    p = P.default_params(*SHAPE)
    ctx = api.Context(p)
    ctx.upload_state(S.synthetic_state(p, seed=95))
    ctx.tape(1)
    ctx.step(P.PRESS_GS_LEX)
    set_word(ctx, 1)
    with pytest.raises(api.AturanError, match="GS sweep"):
        TAKES[take](ctx)
    TAKES[take](ctx)                                   # reported once
    ctx.step(P.PRESS_GS_LEX)
    TAKES[take](ctx)                                   # and a sound sweep is
    ctx.close()
