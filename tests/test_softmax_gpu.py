"""Row softmax (llmt src/kernels/softmax.cu:33-50) where a row is not finite, at the widths of every form of the kernel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import llmt_b200 as L
from oracle import oracle
from tests.support import assert_close

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# registers of 8, 16, 32 and 64 values a lane, 16 bytes at a time and one value at a time, and the two passes of a long row
@pytest.mark.parametrize("t", [5, 64, 256, 300, 512, 1000, 1024, 1500, 2048, 2500])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_masked_columns_are_exact_zeros_beside_values_that_are_not_finite(t, dtype):
    x = torch.randn(2, t, t, device=DEV, generator=torch.Generator(device=DEV).manual_seed(t)).to(dtype)
    bad = {1: float("nan"), 2: float("inf"), t // 2: float("nan"), t - 2: float("inf")}
    for r, v in bad.items():
        x[0, r, r // 2] = v
    x[0, 3] = float("-inf")                   # nothing to choose from
    rows = sorted({*bad, 3})
    y = torch.full_like(x, 7.0)
    L.softmax_fwd(y, x, True)
    assert bool((torch.triu(y, 1) == 0).all())
    for r in rows:
        assert bool(torch.isnan(y[0, r, r // 2]))
    good = torch.ones(2, t, dtype=torch.bool)
    good[0, rows] = False
    ref = oracle.softmax(torch.where(good[:, :, None].to(DEV), x, torch.zeros_like(x)).float().cpu().numpy().astype(np.float64), True)
    got = y.float().cpu().numpy()
    tol = dict(rtol=1e-5, atol=1e-7) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=1e-7)
    assert_close(got[good.numpy()], ref.reshape(got.shape)[good.numpy()], what="rows without such values", **tol)
