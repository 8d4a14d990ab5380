"""Kernels that need more dynamic shared memory than the default. The limit belongs to a kernel on a device:
asked for once per process it would be missing on a second device (read from the sources: the machines have
one), and fitted to one context it would be too low for another."""
import os
import re

import numpy as np
import pytest

from aturan_b200 import params as P, state as S

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aturan_b200", "csrc")


def test_the_limit_is_asked_for_at_each_launch_that_needs_it():
    text = "".join(re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
                   for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh")))
    assert text.count("cudaFuncAttributeMaxDynamicSharedMemorySize") == 1      # smem_opt_in's own
    assert not re.search(r"static\s+(?:const\s+)?\w+\s+\w+\s*=\s*smem_opt_in", text)
    dynamic = set(re.findall(r"(\w+_kernel)\s*\((?:[^(){}]|\([^()]*\))*\)\s*\{(?:[^{}]|\{[^{}]*\}){0,400}?extern __shared__", text))
    assert len(dynamic) >= 6
    for name in dynamic:
        via = "kern" if not re.search(r"smem_opt_in\(" + name, text) else name
        assert re.search(r"smem_opt_in\(" + via + r"\b", text), name


@pytest.mark.gpu
def test_a_smaller_context_leaves_a_larger_ones_solve_alone():
    """The column correction's block holds 8 (jm - 2) 24 bytes: 80 KB and 57 KB."""
    from aturan_b200 import api
    out = []
    for smaller in (False, True):
        p = P.default_params(5, 421, 9)
        ctx = api.Context(p)
        ctx.upload_state(S.synthetic_state(p, seed=91))
        other = api.Context(P.default_params(5, 300, 9)) if smaller else None
        rc, sweeps, _ = ctx.pressure(P.PRESS_RB_LINE, omega=1.0, max_sweeps=20, tol=1e-6)
        out.append((rc, sweeps, ctx.download("p_dyn")))
        ctx.close()
        if other:
            other.close()
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])
