"""fp32 products by FMAs at the edges of their tile forms, cluster splits and copy paths, and small ones on the tensor cores.

Bound: an fp32 sum of k products in any order differs from the exact one by at most k * 2^-24 of the sum of
magnitudes; for random signs the error grows with sqrt(k) instead.  8 sqrt(k) 2^-24 in the Frobenius norm
leaves a factor of several for the constant; it is 3e-6 at k = 40 and 7e-5 at k = 22000.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import llmt_b200 as L
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bound(k):
    return 8.0 * max(k, 1) ** 0.5 * 2.0 ** -24


# (m, n, k): one element; tile edges +- 1; one row; k below, at and beyond a stage and a split; the last split empty (k = 1088:
# 34 stages over 8 splits of 5); on the tensor cores one tile in 8 splits, an odd pitch with many tiles, a long reduction
SIZES = [(1, 1, 1), (128, 64, 16), (129, 65, 17), (63, 64, 15), (64, 63, 64), (3, 200, 300), (1, 128, 2176), (64, 64, 5000),
         (65, 130, 1088), (300, 2000, 131), (517, 771, 259), (130, 70, 22000)]
# Every form of the FMA kernel and every number of splits that its cost model gives it without a bias gradient
FORMS = [(462, 1176, 17, "128x64 warps=4 splits=1"), (131, 67, 70, "128x64 warps=4 splits=4"), (131, 67, 135, "128x64 warps=4 splits=8"),
         (1030, 1042, 17, "64x64 warps=4 splits=1"), (3, 1188, 129, "64x64 warps=4 splits=4"), (65, 67, 270, "64x64 warps=4 splits=8"),
         (67, 3, 17, "64x64 warps=8 splits=1"), (1188, 66, 194, "64x64 warps=8 splits=2"), (1158, 3, 387, "64x64 warps=8 splits=4"),
         (3, 978, 2307, "64x64 warps=8 splits=8")]


@pytest.mark.parametrize("m,n,k", SIZES)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_tiles_splits_and_pitches(m, n, k, ta, tb):
    rng = np.random.default_rng(m * 7 + n * 3 + k + 2 * ta + tb)
    a = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    b = rng.standard_normal((n, k) if tb else (k, n)).astype(np.float32)
    c0 = rng.standard_normal((m, n)).astype(np.float32)
    ref = oracle.gemm(a, b, bool(ta), bool(tb), 0.75, 0.5, c0)
    # as they are (16-byte copies where the pitch allows them) ...
    c = torch.from_numpy(c0).to(DEV)
    L.gemm(c, torch.from_numpy(a).to(DEV), torch.from_numpy(b).to(DEV), bool(ta), bool(tb), alpha=0.75, beta=0.5)
    assert oracle.rel_fro(c.cpu().numpy(), ref) <= _bound(k)
    # ... and as views that start one float into a row of odd pitch, in a frame that must stay untouched
    def frame(x):
        f = torch.full((x.shape[0], x.shape[1] + 2 + (x.shape[1] + 1) % 2), 7.0, device=DEV)
        f[:, 1:1 + x.shape[1]] = torch.from_numpy(x).to(DEV)
        return f, f[:, 1:1 + x.shape[1]]
    (_, av), (_, bv), (cf, cv) = frame(a), frame(b), frame(c0)
    L.gemm(cv, av, bv, bool(ta), bool(tb), alpha=0.75, beta=0.5)
    assert torch.equal(cv, c), "the copy path does not change the sums"
    assert bool((cf[:, 0] == 7.0).all()) and bool((cf[:, 1 + n:] == 7.0).all())


@pytest.mark.parametrize("m,n,k,form", FORMS)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_every_form_of_the_fma_kernel(m, n, k, form, ta, tb):
    a = np.empty((k, m) if ta else (m, k), dtype=np.float32)
    b = np.empty((n, k) if tb else (k, n), dtype=np.float32)
    assert f"fp32-simt tile={form} " in L.plan(L.make_desc(torch.empty(m, n), torch.from_numpy(a), torch.from_numpy(b), bool(ta), bool(tb)))
    test_tiles_splits_and_pitches(m, n, k, ta, tb)


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 5, 9), (200, 64, 5000), (129, 300, 70), (64, 64, 12000)])
def test_dbias_from_the_stages(m, n, k, ta):
    rng = np.random.default_rng(m + k)
    a = rng.standard_normal((k, m) if ta else (m, k)).astype(np.float32)
    b = rng.standard_normal((k, n)).astype(np.float32)
    db0 = rng.standard_normal(m).astype(np.float32)
    c = torch.zeros(m, n, device=DEV)
    db = torch.from_numpy(db0).to(DEV)
    L.gemm(c, torch.from_numpy(a).to(DEV), torch.from_numpy(b).to(DEV), bool(ta), False, beta=1.0, dbias=db, dbias_beta=1.0)
    ref = db0.astype(np.float64) + (a.astype(np.float64).sum(axis=0) if ta else a.astype(np.float64).sum(axis=1))
    assert oracle.rel_fro(db.cpu().numpy(), ref) <= _bound(k)
    assert oracle.rel_fro(c.cpu().numpy(), oracle.gemm(a, b, bool(ta), False)) <= _bound(k)


def test_empty_reduction():
    a, b = torch.ones(70, 4, device=DEV), torch.ones(4, 9, device=DEV)
    c = torch.full((70, 9), 2.0, device=DEV)
    d = L.make_desc(c, a, b, beta=0.5)
    d.k = 0
    L.gemm_desc(d, c, a, b)
    assert bool((c == 1.0).all())
