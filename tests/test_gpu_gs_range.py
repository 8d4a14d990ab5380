"""The Gauss-Seidel sweep's defect-corrected source with quotients by reciprocals: infinities, NaNs, huge and
tiny values and signed zeros in the tendencies it differences. One sweep equals the oracle's, NaN for NaN."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["rhs_u", "rhs_v", "rhs_w"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e300, 1e-250, -0.0])
def test_one_sweep(oracle_lib, field, value):
    from aturan_b200.api import Context
    p = P.default_params(9, 14, 25)
    p.press_incr = 1
    st = S.synthetic_state(p, seed=31)
    st[field][4, 6, 11] = value
    ctx = Context(p)
    ctx.upload_state(st)
    ctx.pressure(P.PRESS_GS_LEX)
    g = ctx.download_state(["p_dyn"])["p_dyn"]
    ctx.close()
    oracle_lib.pressure_gs(p, st)
    assert np.array_equal(g, st["p_dyn"], equal_nan=True)
