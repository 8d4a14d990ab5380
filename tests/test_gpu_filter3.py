"""The fused three-axis filter of the chemistry forcing at the edges of its tiling: levels that are no
multiple of a block's, a single block of levels, rows and meridians one off the tile, both the short
and the long walk, with and without the periodic seam. The forcing's filtered fields are those of the
oracle bit for bit (FP64)."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S
from tests.chem_case import FORCING_OUT, chem_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per", [1, 0])
@pytest.mark.parametrize("shape", [(5, 5, 5), (7, 8, 33), (8, 9, 31), (15, 17, 65), (21, 121, 641), (22, 128, 611)])
def test_filtered_forcing_is_the_oracles(oracle_lib, shape, per):
    from aturan_b200.api import Context
    p, cp = P.default_params(*shape), P.default_chem_params()
    cp.phi_periodic = per
    st = chem_state(S.synthetic_state(p, seed=3), p, seed=4)
    ctx = Context(p)
    ctx.upload_state(st)
    ctx.chemistry(2, cp, counts=False)
    g = ctx.download_state(FORCING_OUT)
    ctx.close()
    oracle_lib.chem_forcing(p, cp, st)
    for n in FORCING_OUT:
        assert np.array_equal(g[n], st[n]), (n, np.abs(g[n] - st[n]).max())
