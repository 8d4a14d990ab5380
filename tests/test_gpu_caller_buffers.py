"""The buffers of the adjoint and solve calls, in forms that a kernel cannot take: off the doubles' 8-byte
boundaries, overlapping outputs (the later field stays), and memory that is no device buffer (refused, the
context still usable)."""
import numpy as np
import pytest

from aturan_b200 import api, params as P, state as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = (8, 13, 19)
NB = int(np.prod(SHAPE)) * 8


class Buf:
    """A device array of SHAPE that starts `off` bytes into its allocation."""

    def __init__(self, a=None, off=0):
        self.raw = torch.zeros(NB + 16, dtype=torch.uint8, device="cuda")
        self.off = off
        if a is not None:
            self.raw[off:off + NB] = torch.tensor(np.ascontiguousarray(a).view(np.uint8).ravel(), device="cuda")
        self.ptr = self.raw.data_ptr() + off

    def get(self):
        return self.raw[self.off:self.off + NB].cpu().numpy().view(np.float64).reshape(SHAPE)


@pytest.fixture
def ctx():
    p = P.default_params(*SHAPE)
    st = S.synthetic_state(p, seed=81)
    c = api.Context(p)
    c.upload_state(st)
    c.tape(1)
    c.pressure(P.PRESS_RB_LINE, omega=1.0, max_sweeps=100, tol=1e-8)
    c.rk4_step()
    yield c
    c.close()


def _adjoint(ctx, off):
    rng = np.random.default_rng(82)
    yb = [Buf(rng.standard_normal(SHAPE), off) for _ in range(4)]
    ab = [Buf(rng.standard_normal(SHAPE), off) for _ in range(3)]
    xb, pb = [Buf(off=off) for _ in range(4)], Buf(off=off)
    gb = [Buf(off=off) for _ in range(3)]
    torch.cuda.synchronize()
    ctx.rk4_adjoint_ex([b.ptr for b in yb], [b.ptr for b in ab], [b.ptr for b in xb], pb.ptr)
    ctx.pressure_adjoint(pb.ptr, [b.ptr for b in gb], P.PRESS_RB_LINE, 1.0, 100, 1e-10)
    return [b.get() for b in (*xb, pb, *gb)]


@pytest.mark.parametrize("off", [4, 1, 8])
def test_adjoints_off_the_doubles_boundaries(ctx, off):
    want, got = _adjoint(ctx, 0), _adjoint(ctx, off)
    for a, b in zip(want, got):
        assert np.abs(a).max() > 0 and np.array_equal(a, b)


@pytest.mark.parametrize("off", [4, 1, 8])
def test_solve_off_the_doubles_boundaries(ctx, off):
    b = np.random.default_rng(83).standard_normal(SHAPE)
    out = []
    for o in (0, off):
        rhs, x = Buf(b, o), Buf(np.zeros(SHAPE), o)
        torch.cuda.synchronize()
        ctx.pressure_solve(rhs.ptr, x.ptr, P.PRESS_RB_LINE, omega=1.0, max_sweeps=100, tol=1e-8)
        out.append(x.get())
    assert np.abs(out[0]).max() > 0 and np.array_equal(out[0], out[1])


def test_overlapping_outputs_keep_the_later_field(ctx):
    want = _adjoint(ctx, 0)
    rng = np.random.default_rng(82)
    yb = [Buf(rng.standard_normal(SHAPE)) for _ in range(4)]
    ab = [Buf(rng.standard_normal(SHAPE)) for _ in range(3)]
    one, w, pb = Buf(), Buf(), Buf()
    torch.cuda.synchronize()
    ctx.rk4_adjoint_ex([b.ptr for b in yb], [b.ptr for b in ab], [one.ptr, one.ptr, one.ptr, w.ptr], pb.ptr)
    assert np.array_equal(one.get(), want[2]) and np.array_equal(w.get(), want[3])


def test_a_host_buffer_is_refused(ctx):
    host = np.zeros(SHAPE)
    xb, pb = [Buf() for _ in range(4)], Buf()
    good = [Buf(np.ones(SHAPE)) for _ in range(4)]
    torch.cuda.synchronize()
    with pytest.raises(api.AturanError):
        ctx.rk4_adjoint([*(b.ptr for b in good[:3]), host.ctypes.data], [b.ptr for b in xb])
    with pytest.raises(api.AturanError):
        ctx.rk4_adjoint([b.ptr for b in good], [*(b.ptr for b in xb[:3]), host.ctypes.data])
    with pytest.raises(api.AturanError):
        ctx.pressure_solve(host.ctypes.data, pb.ptr, P.PRESS_RB_LINE)
    with pytest.raises(api.AturanError):
        ctx.pressure_adjoint(host.ctypes.data, [b.ptr for b in xb[:3]])
    assert all(np.isfinite(a).all() for a in _adjoint(ctx, 0))
