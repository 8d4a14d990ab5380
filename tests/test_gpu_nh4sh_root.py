"""The NH4SH equilibrium where its root estimate is hardest: K_p so small that the root is within an
ulp of the smaller reactant, equal reactants (a double root as K_p goes to 0), reactants many orders
apart, roots in the middle of the bracket, decomposition from a trace up to all of the NH4SH, cells
with nothing to do. Newton's estimate only decides which midpoints of the reference's bisection need
their sign evaluated, so the result is the reference's: the same bar as for ordinary states (1e-12 of
each field's maximum, CUDA's pow against the host's in the evaluated signs), at three sizes of the
reactants."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S
from tests.chem_case import EQ_OUT

pytestmark = pytest.mark.gpu


def _cells(p, seed, t_lo, t_hi, kind, size):
    rng = np.random.default_rng(seed)
    st = S.synthetic_state(p, seed=seed)
    shape = (p.im, p.jm, p.km)
    st["t"] = rng.uniform(t_lo, t_hi, shape) / p.t_ref
    a = size * rng.uniform(0.5, 2.0, shape)
    st["nh3"] = 17.03052 * a
    if kind == "equal":
        st["h2s"] = 34.08088 * a
    elif kind == "near":
        st["h2s"] = 34.08088 * a * (1.0 + 10.0 ** rng.uniform(-15, -2, shape))
    else:
        st["h2s"] = 34.08088 * a * 10.0 ** rng.uniform(-8, 0, shape)
    st["nh4sh"] = np.where(rng.random(shape) < 0.3, 0.0, 51.1114 * size * 10.0 ** rng.uniform(-6, 0, shape))
    return st


@pytest.mark.parametrize("kind", ["equal", "near", "apart"])
@pytest.mark.parametrize("t_lo,t_hi", [(50.0, 90.0), (150.0, 260.0), (260.0, 420.0)])
@pytest.mark.parametrize("size", [1e-10, 1e-6, 1e-3])
def test_roots_match_the_oracle(oracle_lib, size, t_lo, t_hi, kind):
    from aturan_b200.api import Context
    p, cp = P.default_params(7, 9, 33), P.default_chem_params()
    st = _cells(p, 11, t_lo, t_hi, kind, size)
    ctx = Context(p)
    ctx.upload_state(st)
    gf, gd = ctx.chemistry(1, cp, counts=True)
    g = ctx.download_state(EQ_OUT)
    ctx.close()
    of, od = oracle_lib.nh4sh_eq(p, cp, st)
    assert (gf, gd) == (of, od) or abs(gf - of) + abs(gd - od) <= 0.001 * (of + od)
    for n in EQ_OUT:
        d = np.abs(g[n] - st[n]).max() / np.abs(st[n]).max()
        assert d <= 1e-12, (n, d)
