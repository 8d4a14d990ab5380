"""The exact level means (the reference's serial sums, formed in parallel) where their steps can go wrong: fewer
cells than a chunk, a last colatitude whose sine rounds below zero or not, cells without a valid temperature
(zero terms), terms of very different size (many binades, a term above the running sum), whole levels without
a valid cell. Bit-equal to a serial sum in the reference's order."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S

pytestmark = pytest.mark.gpu


def serial_means(p, st):
    """RungeKutta_Uran_Turb.cpp:18-37 in numpy: one addition after another (cumsum adds in order)."""
    _, the = S.coords(p)
    w = np.broadcast_to(np.array([float(np.sin(x)) for x in the])[None, :, None], p.shape)
    out = np.zeros(p.im)
    for i in range(p.im):
        T, ps = st["t"][i].ravel(), st["p_stat"][i].ravel()
        with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
            b = p.g * ps / (p.r_mix * p.R_mix * T * p.t_ref)
        ok = (T > 0.0) & np.isfinite(b)
        wi = w[i].ravel()[ok]
        if wi.size:
            sw = np.cumsum(wi)[-1]
            out[i] = np.cumsum(wi * b[ok])[-1] / sw if sw > 0.0 else 0.0
    return out


@pytest.mark.parametrize("shape", [(5, 5, 5), (6, 16, 17), (9, 13, 21), (7, 91, 181), (5, 181, 361), (6, 46, 91)])
@pytest.mark.parametrize("kind", ["smooth", "wild"])
def test_level_means_are_the_serial_sums(shape, kind):
    from aturan_b200.api import Context
    p = P.default_params(*shape)
    st = S.synthetic_state(p, seed=shape[1])
    if kind == "wild":
        rng = np.random.default_rng(3)
        st["p_stat"] *= 2.0 ** rng.integers(-60, 60, shape)
        st["t"][rng.random(shape) < 0.1] = -1.0
        st["t"][1, :, :] = 0.0
        st["p_stat"][2, 1, 3] = 0.0
        st["p_stat"][3, 2, 1] *= 2.0 ** 300
    ctx = Context(p)
    ctx.upload_state(st)
    ctx.rk4_step()
    got = ctx.buoy_ref_level()
    ctx.close()
    assert np.array_equal(got, serial_means(p, st))
