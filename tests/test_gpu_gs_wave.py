"""The one-launch lexicographic sweep (gs_wave_kernel) at the edges of its bands, chunks and column depths:
bit-exact with the oracle's serial sweep in FP64, on grids whose rows end inside a chunk, whose last band is
short, that take each count of sweeping threads, and too deep for it (the hyperplane launches); several sweeps
in a row (each has its own tag), with and without the defect correction."""
import numpy as np
import pytest

from aturan_b200 import params as P, state as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (5, 5, 5),          # one band of three rows, rows shorter than a chunk
    (9, 10, 17),        # exactly one band of eight rows, rows of one whole chunk
    (16, 11, 35),       # a second band of one row; 16 levels fill the padded column
    (17, 26, 33),       # three whole bands; rows of two whole chunks (the ring)
    (33, 14, 19),       # 256 / 384 sweeping threads: 48 padded levels
    (64, 11, 41),       # six rows per band
    (100, 9, 31),       # two rows per band
    (150, 7, 35),       # one row per band
    (240, 6, 9),        # deeper than the shared memory: hyperplane launches
])
@pytest.mark.parametrize("incr", [1, 0])
def test_sweeps_match_oracle_bit_for_bit(oracle_lib, shape, incr):
    from aturan_b200.api import Context
    p = P.default_params(*shape)
    p.press_incr = incr
    st = S.synthetic_state(p, seed=shape[0] + 7 * shape[2])
    ctx = Context(p)
    ctx.upload_state(st)
    for _ in range(3):
        rc, sweeps, _ = ctx.pressure(P.PRESS_GS_LEX)
        assert rc == 0 and sweeps == 1
        oracle_lib.pressure_gs(p, st)
    got = ctx.download("p_dyn")
    ctx.close()
    assert np.array_equal(got, st["p_dyn"]), np.abs(got - st["p_dyn"]).max()


def test_two_contexts_interleaved(oracle_lib):
    """Each context has its own ticket, tags and edge buffer: sweeps of two contexts in turn, both in flight."""
    from aturan_b200.api import Context
    p = P.default_params(21, 37, 73)
    states = [S.synthetic_state(p, seed=s) for s in (1, 2)]
    ctxs = [Context(p) for _ in states]
    for c, s in zip(ctxs, states):
        c.upload_state(s)
    for _ in range(4):
        for c in ctxs:
            c.pressure(P.PRESS_GS_LEX)
    for c, s in zip(ctxs, states):
        for _ in range(4):
            oracle_lib.pressure_gs(p, s)
        assert np.array_equal(c.download("p_dyn"), s["p_dyn"])
        c.close()
