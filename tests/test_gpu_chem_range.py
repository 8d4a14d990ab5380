"""The chemistry forcing's quotients by reciprocals outside the ordinary range: infinities and NaNs in the
temperature and the gases, a temperature of zero, values near the largest and far below any physical one,
negative zeros, exact zeros. Every value as the oracle's divisions give it (NaN for NaN)."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S
from tests.chem_case import FORCING_OUT, chem_state

pytestmark = pytest.mark.gpu

VALUES = [np.inf, -np.inf, np.nan, 0.0, -0.0, 1e300, -1e300, 1e-200, 5e-324]


@pytest.mark.parametrize("field", ["t", "nh3", "h2s", "nh4sh"])
def test_single_cells(oracle_lib, field):
    from aturan_b200.api import Context
    p, cp = P.default_params(12, 40, 65), P.default_chem_params()
    st = chem_state(S.synthetic_state(p, seed=21), p, seed=22)
    for n, v in enumerate(VALUES):                      # far enough apart that no stencil or filter sees two
        st[field][5, 3 + 4 * n, 7 + 6 * n] = v
    st["nh4sh"][:, 20:, 50:] = 0.0
    ctx = Context(p)
    ctx.upload_state(st)
    ctx.chemistry(2, cp, counts=False)
    g = ctx.download_state(FORCING_OUT)
    ctx.close()
    oracle_lib.chem_forcing(p, cp, st)
    for n in FORCING_OUT:
        assert np.array_equal(g[n], st[n], equal_nan=True), n
