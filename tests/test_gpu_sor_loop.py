"""The solve loop of the folded pressure operator against the CPU restatement, sweep for sweep: the
chained point passes at the edges of their tiling (level counts that are no multiple of a thread's
cells, fewer cells than a block, folded rows on every side), and the sweeps that are enqueued before
a check's answer is known, which must leave no trace once that check has met the tolerance.

Both sides run the same sweeps, corrections and checks in FP64 and differ by rounding alone. A sweep
rounds each cell a few times and is no expansion; a correction solves a well-conditioned system of at
most ~40 rows per mode (growth <= 40^2). So after n sweeps the difference is below
n * 1600 * 2^-53 ~ 6e-12 of the largest value at n = 33: 1e-10 is asked."""
import numpy as np
import pytest

from aturan_b200 import params as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GRIDS = [(5, 5, 9), (6, 6, 17), (7, 9, 33), (8, 37, 15), (11, 13, 131)]
I = (slice(1, -1), slice(1, -1), slice(0, -1))


def _rhs(shape, seed):
    rng = np.random.default_rng(seed)
    b = np.zeros(shape)
    b[I] = rng.standard_normal((shape[0] - 2, shape[1] - 2, shape[2] - 1))
    return b


def _gpu(p, b, x0, kind, tr, omega, cap, tol):
    from aturan_b200 import api
    ctx = api.Context(P.default_params(p.im, p.jm, p.km, precision=P.FP64))
    bd, xd = torch.tensor(b, device="cuda"), torch.tensor(x0, device="cuda")
    torch.cuda.synchronize()
    out = ctx.pressure_solve(bd.data_ptr(), xd.data_ptr(), kind, tr, omega, cap, tol)
    ctx.close()
    return out, xd.cpu().numpy()


def _same(x, y):
    d = x[I] - y[I]
    assert np.abs(d - d.mean()).max() <= 1e-10 * np.abs(y[I]).max()


@pytest.mark.parametrize("tr", [False, True])
@pytest.mark.parametrize("kind,omega", [(P.PRESS_RB_SOR, 1.7), (P.PRESS_RB_LINE, 1.0)])
@pytest.mark.parametrize("shape", GRIDS)
def test_a_capped_solve_does_exactly_its_sweeps(oracle_lib, shape, kind, omega, tr):
    p = P.default_params(*shape)
    b = _rhs(shape, sum(shape))
    x0 = np.zeros(shape)
    x0[0], x0[-1], x0[:, 0], x0[:, -1] = (np.nan,) * 4       # boundary rows are no part of the operator
    for cap in (1, 2, 16, 17, 33):
        (rc, its, res), x = _gpu(p, b, x0, kind, tr, omega, cap, -1.0)
        y = np.zeros(shape)
        rc2, its2, res2 = oracle_lib.solve(p, b, y, tr, kind == P.PRESS_RB_LINE, omega, cap, -1.0)
        assert rc == rc2 == 1 and its == its2 == cap
        _same(x, y)
        assert abs(res - res2) <= 1e-8 * max(res2, 1e-3)


@pytest.mark.parametrize("tr", [False, True])
@pytest.mark.parametrize("kind,omega,tol", [(P.PRESS_RB_SOR, 1.7, 1e-3), (P.PRESS_RB_LINE, 1.0, 1e-2)])
@pytest.mark.parametrize("shape", GRIDS)
def test_the_sweeps_after_the_last_check_change_nothing(oracle_lib, shape, kind, omega, tol, tr):
    p = P.default_params(*shape)
    b = _rhs(shape, 7 + sum(shape))
    (rc, its, res), x = _gpu(p, b, np.zeros(shape), kind, tr, omega, 4000, tol)
    y = np.zeros(shape)
    rc2, its2, res2 = oracle_lib.solve(p, b, y, tr, kind == P.PRESS_RB_LINE, omega, 4000, tol)
    assert rc == 0 and rc2 == 0 and its == its2 and res <= tol
    _same(x, y)
    # a solution that already meets the tolerance comes back as it went in
    (rc, its, res), z = _gpu(p, b, x, kind, tr, omega, 50, 2.0 * tol)
    assert rc == 0 and its == 0 and np.array_equal(z[I], x[I])
