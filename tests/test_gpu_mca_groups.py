"""The moist convective adjustment's launches at the edges of their forms: a warp per column (few columns)
and eight columns per warp (many), the shallowest columns, a constant heat capacity, columns left alone
(a non-positive or non-finite level) next to adjusted ones. Bars as tests/test_gpu_mca.py: 1e-11 of each
field's maximum outside counted columns."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S
from tests.test_gpu_mca import NAMES, compare, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 9, 17), (6, 97, 99), (9, 95, 101), (34, 5, 7), (41, 97, 99)])
@pytest.mark.parametrize("cp_dyn", [1, 0])
def test_group_forms_match_oracle(oracle_lib, shape, cp_dyn):
    p = P.default_params(*shape)
    p.cp_dyn = cp_dyn
    st = S.synthetic_state(p, seed=shape[0] + 10 * shape[2])
    g = run_gpu(p, st)
    oracle_lib.mca(p, st)
    compare(p, g, st, 1e-11, 0.02)


@pytest.mark.parametrize("shape", [(21, 11, 17), (21, 97, 99)])
def test_unusable_columns_are_left_alone(oracle_lib, shape):
    """A level with T <= 0, a NaN temperature, p <= 0: the whole column keeps its bits; the others match."""
    p = P.default_params(*shape)
    st = S.synthetic_state(p, seed=5)
    st["t"][3, 2, 4] = -0.1
    st["t"][7, 3, 5] = np.nan
    st["p_stat"][4, 5, 6] = 0.0
    before = S.copy_state(st)
    g = run_gpu(p, st)
    cols = [(2, 4), (3, 5), (5, 6)]
    for n in NAMES:
        for j, k in cols:
            assert np.array_equal(g[n][:, j, k], before[n][:, j, k], equal_nan=True), (n, j, k)
    oracle_lib.mca(p, st)
    for n in NAMES:                          # out of the comparison's finiteness check
        for j, k in cols:
            g[n][:, j, k] = st[n][:, j, k] = 0.0
    compare(p, g, st, 1e-11, 0.02)
