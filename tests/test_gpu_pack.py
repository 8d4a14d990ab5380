"""The batched layout change: every field through upload_many / download_many on device buffers, one launch per
64 fields, against what each storage type keeps of an FP64 value: all of it, its FP32 rounding, or (the mixed
form's t and tn) the pair's ~48 bits. Rows shorter than a warp, one block's worth and ragged ones; nothing
outside the destination is written."""
import numpy as np
import pytest

from aturan_b200 import fields as F, params as P

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FP64_IN_MIXED = {"p_dyn", "p_hydro", "p_baro", "p_b0", "p_bfollow"}


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
@pytest.mark.parametrize("shape", [(5, 5, 5), (9, 13, 17), (6, 11, 33), (8, 16, 129), (7, 9, 257)])
def test_round_trip(precision, shape):
    from aturan_b200.api import Context
    ctx = Context(P.default_params(*shape, precision=precision))
    rng = np.random.default_rng(shape[2])
    n = int(np.prod(shape))
    src = {f: rng.standard_normal(shape) * 10.0 ** rng.integers(-3, 4) for f in F.NAMES}
    dev = {f: torch.tensor(a, device="cuda") for f, a in src.items()}
    out = {f: torch.full((n + 2,), 7.0, dtype=torch.float64, device="cuda") for f in F.NAMES}
    torch.cuda.synchronize()
    ctx.upload_many(F.NAMES, [dev[f].data_ptr() for f in F.NAMES], on_device=True)
    ctx.download_many(F.NAMES, [out[f].data_ptr() + 8 for f in F.NAMES], on_device=True)
    for f in F.NAMES:
        got = out[f].cpu().numpy()
        assert got[0] == 7.0 and got[-1] == 7.0, f
        got = got[1:-1].reshape(shape)
        if precision == P.FP64 or f in FP64_IN_MIXED:
            assert np.array_equal(got, src[f]), f
        elif f in ("t", "tn"):
            hi = src[f].astype(np.float32).astype(np.float64)
            lo = (src[f] - hi).astype(np.float32).astype(np.float64)
            assert np.array_equal(got, hi + lo), f
        else:
            assert np.array_equal(got, src[f].astype(np.float32).astype(np.float64)), f
        assert np.array_equal(ctx.download(f), got), f          # the one-field host path
    ctx.close()
