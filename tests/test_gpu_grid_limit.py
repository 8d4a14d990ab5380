"""The largest FP64 grid at 41 levels and 361 meridians: 2^31 elements of what the stage kernels address, the
Gauss-Seidel sweep's own buffers not counted. One row less or more on the other side of the line."""
import pytest

from aturan_b200 import api, params as P

pytestmark = pytest.mark.gpu


def test_the_largest_grid_is_accepted():
    ctx = api.Context(P.default_params(41, 986, 361))        # 17.2 GB
    ctx.pressure(P.PRESS_GS_LEX)
    ctx.synchronize()
    assert (ctx.download("p_dyn") == 0.0).all()
    ctx.close()


def test_one_row_more_is_refused():
    with pytest.raises(api.AturanError) as e:
        api.Context(P.default_params(41, 987, 361))
    assert e.value.code == api.E_UNSUPPORTED
