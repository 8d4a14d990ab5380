"""The precipitation march at the edges of its branches: dry columns, fluxes at their cap and beyond the
reference flux from the top on, all cells warm, all cells frozen, saturated vapour (no evaporation), traces
whose fluxes are tiny, an infinite condensate in a single column. The bar of tests/test_gpu_precip.py
(1e-11 of each field's maximum outside 1 % of the columns); the infinite column value for value."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S
from tests.precip_case import GASES, PRECIP_OUT, precip_state
from tests.test_gpu_precip import compare, run_gpu

pytestmark = pytest.mark.gpu


def _scaled(st, p, kind):
    cond = [g + c for g in GASES for c in ("_cloud", "_ice")]
    for n in cond:
        if kind == "dry":
            st[n][:] = 0.0
        elif kind == "cap":
            st[n] = np.abs(st[n]) * 1e6 + 1.0
        elif kind == "trace":
            st[n] *= 1e-120
    if kind == "warm":
        st["t"][:] = 400.0 / p.t_ref
    if kind == "frozen":
        st["t"][:] = 60.0 / p.t_ref
    if kind == "moist":
        for g in GASES:
            st[g] = np.abs(st[g]) * 1e6 + 1.0
    return st


@pytest.mark.parametrize("shape", [(5, 6, 9), (14, 9, 35)])
@pytest.mark.parametrize("kind", ["dry", "cap", "trace", "warm", "frozen", "moist"])
def test_branches(oracle_lib, shape, kind):
    p, pp = P.default_params(*shape), P.default_precip_params()
    st = _scaled(precip_state(S.synthetic_state(p, seed=91), p, seed=92), p, kind)
    g = run_gpu(p, st, pp, PRECIP_OUT)
    oracle_lib.precipitation(p, pp, st)
    compare(g, st, PRECIP_OUT, 1e-11)


def test_an_infinite_condensate(oracle_lib):
    p, pp = P.default_params(10, 8, 17), P.default_precip_params()
    st = precip_state(S.synthetic_state(p, seed=93), p, seed=94)
    st["nh3_cloud"][5, 4, 7] = np.inf
    g = run_gpu(p, st, pp, PRECIP_OUT)
    oracle_lib.precipitation(p, pp, st)
    for n in PRECIP_OUT:
        a, b = g[n][:, 4, 7], st[n][:, 4, 7]
        same = (np.isnan(a) & np.isnan(b)) | (a == b) | (np.abs(a - b) <= 1e-11 * np.abs(st[n][np.isfinite(st[n])]).max())
        assert same.all(), (n, a, b)
