"""The moist convective adjustment where its quotients leave the ordinary range: temperatures at which
the saturation ratios underflow to 0 (and below the cp table's first entry), temperatures far above every
phase change, pressures many decades off, dry gas. Bars as tests/test_gpu_mca.py."""
import pytest

from aturan_b200 import params as P, state as S
from tests.test_gpu_mca import compare, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(12, 9, 17), (8, 97, 99)])
@pytest.mark.parametrize("t,p,q", [(0.03, 1.0, 1.0), (0.3, 1.0, 1.0), (8.0, 1.0, 1.0), (1.0, 1e-6, 1.0), (1.0, 1e6, 1.0),
                                   (1.0, 1.0, 0.0), (1.0, 1.0, 1e-200)])
def test_extreme_states_match_the_oracle(oracle_lib, shape, t, p, q):
    par = P.default_params(*shape)
    st = S.synthetic_state(par, seed=8)
    st["t"] *= t
    st["p_stat"] *= p
    for n in list(st):
        if n.split("_")[0] in ("h2o", "nh3", "h2s", "ch4") and not n.endswith("n"):
            st[n] *= q
    g = run_gpu(par, st)
    oracle_lib.mca(par, st)
    compare(par, g, st, 1e-11, 0.02)
