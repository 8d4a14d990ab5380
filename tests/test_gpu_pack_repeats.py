"""upload_many / download_many on device buffers with a field given twice, or outputs that overlap: the later
one stays, as if the fields were moved one after the other."""
import numpy as np
import pytest

from aturan_b200 import params as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SHAPE = (21, 91, 181)
N = int(np.prod(SHAPE))


@pytest.fixture(params=[P.FP64, P.MIXED])
def ctx(request):
    from aturan_b200.api import Context
    c = Context(P.default_params(*SHAPE, precision=request.param))
    yield c
    c.close()


def test_a_field_given_many_times(ctx):
    dev = [torch.full(SHAPE, float(v), dtype=torch.float64, device="cuda") for v in range(70)]
    torch.cuda.synchronize()
    for names in (["t", "u", "t"], ["p_dyn"] * 70, ["u", "v"] * 35):
        ctx.upload_many(names, [d.data_ptr() for d in dev[:len(names)]], on_device=True)
        for n in set(names):
            last = max(q for q, m in enumerate(names) if m == n)
            assert (ctx.download(n) == float(last)).all(), (names[:3], n)


@pytest.mark.parametrize("shift", [0, 1, N - 1])
def test_overlapping_outputs(ctx, shift):
    names = ["u", "v", "p_dyn", "w"]
    for v, n in enumerate(names):
        ctx.upload(n, np.full(SHAPE, float(v + 1)))
    raw = torch.zeros(N + 4 * shift, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.download_many(names, [raw.data_ptr() + 8 * shift * q for q in range(4)], on_device=True)
    want = np.zeros(N + 4 * shift)
    for q in range(4):
        want[shift * q:shift * q + N] = q + 1
    assert np.array_equal(raw.cpu().numpy(), want)
