"""The reverse stage reads nothing off the interior: neither the boundary rows of the caller's aux cotangent
nor those of the stage inputs, which the RK4 step never writes and which other calls use as work space. With
NaN and infinities there the gradients have the bits they have without."""
import numpy as np
import pytest

from aturan_b200 import api, fields as F, params as P, state as S
from aturan_b200.autograd import DRY, MOIST

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPES = [(5, 5, 5), (7, 11, 37), (12, 20, 33)]


def _boundary(a, value):
    a[0], a[-1], a[:, 0], a[:, -1] = value, value, value, value
    return a


def _gradient(shape, moist, aux_off=0.0, leftovers=False, **params):
    """xbar and pbar of one taped step with random cotangents; aux_off: the aux cotangent off the interior."""
    p = P.default_params(*shape)
    for n, v in params.items():
        setattr(p, n, v)
    st = S.synthetic_state(p, seed=71)
    names = MOIST if moist else DRY
    ctx = api.Context(p)
    if leftovers:                     # the adjustment's and the chemistry's work fields hold them afterwards
        bad = S.copy_state(st)
        bad["nh4sh"][:, 0], bad["nh4sh"][:, -1] = np.nan, np.nan
        bad["h2o"][:, 0], bad["h2o"][:, -1] = np.inf, np.inf
        ctx.upload_state(bad)
        ctx.mca()
        nan = _boundary(np.zeros(shape), np.nan)
        for n in ("massflux_h2s", "massflux_nh3", "massflux_nh4sh", "fluxlim_nh4sh"):
            ctx.upload(n, nan)
        ctx.chemistry(api.CHEM_FORCING)
    zero = np.zeros(shape)
    for n in F.NAMES:
        ctx.upload(n, st.get(n, zero))
    ctx.tape(2 if moist else 1)
    ctx.restore_ncopies(1.0)
    ctx.rk4_step()
    rng = np.random.default_rng(72)
    ybar = [torch.tensor(rng.standard_normal(shape), device="cuda") for _ in names]
    aux = [torch.tensor(_boundary(rng.standard_normal(shape), aux_off), device="cuda") for _ in range(3)]
    xbar = [torch.empty(shape, dtype=torch.float64, device="cuda") for _ in names]
    pbar = torch.empty(shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    (ctx.moist_adjoint if moist else ctx.rk4_adjoint_ex)([y.data_ptr() for y in ybar], [a.data_ptr() for a in aux],
                                                         [x.data_ptr() for x in xbar], pbar.data_ptr())
    out = [x.cpu().numpy() for x in xbar] + [pbar.cpu().numpy()]
    ctx.close()
    return dict(zip((*names, "p_dyn"), out))


def _same(a, b):
    for n in a:
        assert np.isfinite(a[n]).all() and np.array_equal(a[n], b[n]), n


@pytest.mark.parametrize("moist", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_aux_cotangent_off_the_interior_is_not_read(shape, moist):
    want = _gradient(shape, moist)
    for value in (np.nan, np.inf):
        _same(want, _gradient(shape, moist, aux_off=value))


@pytest.mark.parametrize("moist", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_leftovers_in_the_stage_buffers_are_not_read(shape, moist):
    _same(_gradient(shape, moist), _gradient(shape, moist, leftovers=True))


@pytest.mark.parametrize("moist", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_a_pole_without_a_metric_floor(shape, moist):
    """sin = 0 on the pole's row and no floor: its weights are infinite, and nothing reads them."""
    p = P.default_params(*shape)
    assert p.the0 == 0.0
    for n, x in _gradient(shape, moist, sinthe_min=0.0).items():
        assert np.isfinite(x).all(), n
