"""fp32 products large enough for the tensor-core form (three bf16 parts a value): its edges, splits, copy paths,
fused results, and the values that the split cannot carry.

Bound: a k-block of 64 leaves at most a few units of 2^-24 of its own magnitude (four truncating accumulations of
the leading terms), the k-blocks are added rounded to nearest: for random signs 4 * 2^-24 plus sqrt(k / 64) * 2^-24
in the Frobenius norm, 4.5e-7 at k = 768; fp32 FMAs in sequence reach about the same at k = 1500.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import llmt_b200 as L

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _healthy_device():
    yield
    assert L.device_status() == (0, 0)


def _bound(k):
    return (4.0 + (k / 64.0) ** 0.5) * 2.0 ** -24


def _rel(x, ref):
    return ((x.double() - ref).norm() / ref.norm()).item()


def _operands(m, n, k, ta, tb, batch=()):
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n * 3 + k + 2 * ta + tb)
    a = torch.randn(*batch, *((k, m) if ta else (m, k)), device=DEV, generator=g)
    b = torch.randn(*batch, *((n, k) if tb else (k, n)), device=DEV, generator=g)
    return a, b


def _product(a, b, ta, tb):
    a, b = a.double(), b.double()
    return (a.mT if ta else a) @ (b.mT if tb else b)


# edges of 128 x 128 and 128 x 64 tiles and of a k-block, one k-block, several tiles a CTA, splits of 2, 4 and 8
@pytest.mark.parametrize("m,n,k", [(1025, 2049, 64), (1024, 2048, 127), (257, 3073, 769), (300, 500, 777), (256, 768, 3072), (256, 2304, 768),
                                   (130, 1000, 2049), (2500, 1300, 191), (512, 768, 6003)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_against_64_bits_and_copy_paths(m, n, k, ta, tb):
    a, b = _operands(m, n, k, ta, tb)
    c0 = torch.randn(m, n, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    ref = 0.75 * _product(a, b, ta, tb) + 0.5 * c0.double()
    c = c0.clone()
    L.gemm(c, a, b, bool(ta), bool(tb), alpha=0.75, beta=0.5)
    assert _rel(c, ref) <= _bound(k)
    # views that start one float into a row of odd pitch, the result in a frame that must stay untouched: the same sums
    def frame(x):
        f = torch.full((x.shape[0], x.shape[1] + 2 + (x.shape[1] + 1) % 2), 7.0, device=DEV)
        f[:, 1:1 + x.shape[1]] = x
        return f, f[:, 1:1 + x.shape[1]]
    (_, av), (_, bv), (cf, cv) = frame(a), frame(b), frame(c0)
    L.gemm(cv, av, bv, bool(ta), bool(tb), alpha=0.75, beta=0.5)
    assert torch.equal(cv, c)
    assert bool((cf[:, 0] == 7.0).all()) and bool((cf[:, 1 + n:] == 7.0).all())


@pytest.mark.parametrize("m,n,k", [(1000, 1500, 200), (256, 768, 3072)])
def test_bias_and_gelu(m, n, k):
    a, b = _operands(m, n, k, 0, 1)
    a *= k ** -0.5
    bias = torch.randn(n, device=DEV)
    pre = _product(a, b, 0, 1) + bias.double()
    for gelu, ref in ((False, pre), (True, 0.5 * pre * (1 + torch.tanh(0.7978845608028654 * (pre + 0.044715 * pre ** 3))))):
        c = torch.empty(m, n, device=DEV)
        L.gemm(c, a, b, False, True, bias=bias, gelu=gelu)
        assert _rel(c, ref) <= _bound(k) + 2e-7 * gelu   # (tanhf and its argument: a few roundings more)


@pytest.mark.parametrize("m,n,k", [(3072, 768, 500), (768, 256, 4096), (129, 2000, 1500)])
def test_dbias(m, n, k):
    a, b = _operands(m, n, k, 1, 0)
    db0 = torch.randn(m, device=DEV)
    c, db = torch.zeros(m, n, device=DEV), db0.clone()
    L.gemm(c, a, b, True, False, beta=1.0, dbias=db, dbias_beta=1.0)
    assert _rel(c, _product(a, b, 1, 0)) <= _bound(k)
    assert _rel(db, db0.double() + a.double().sum(0)) <= 8.0 * k ** 0.5 * 2.0 ** -24   # k additions in some order


def test_batches():
    a, b = _operands(200, 190, 130, 0, 1, (37,))
    c = torch.empty(37, 200, 190, device=DEV)
    L.gemm(c, a, b, False, True)
    assert _rel(c, _product(a, b, 0, 1)) <= _bound(130)


@pytest.mark.parametrize("m,n,k", [(512, 3072, 300), (256, 768, 3072)])
def test_values_the_parts_cannot_carry(m, n, k):
    """Infinities, NaN, values next to the largest, overflowing sums and tiny operands give what fp32 FMAs give."""
    big = 3.4028234e38
    a0, b = _operands(m, n, k, 0, 1)
    def check(a, b):
        c = torch.empty(m, n, device=DEV)
        L.gemm(c, a, b, False, True)
        ref = _product(a, b, 0, 1)
        ref32 = ref.float()
        assert torch.equal(torch.isnan(c), torch.isnan(ref32))
        assert torch.equal(torch.isinf(c), torch.isinf(ref32))
        assert torch.equal(c[torch.isinf(c)], ref32[torch.isinf(ref32)])
        return c, ref
    a = a0.clone()
    a[3, 7], a[200, 5], a[m - 1, k - 1] = float("inf"), float("nan"), -float("inf")
    c, ref = check(a, b)
    fine = torch.isfinite(ref).all(1)
    assert int(fine.sum()) == m - 3 and _rel(c[fine], ref[fine]) <= 8.0 * k ** 0.5 * 2.0 ** -24
    # the leading part of a value this large rounds to infinity
    a, b1 = a0.clone(), b.clone()
    a[17] = 0.0
    a[17, 11] = big
    b1[:, 11] = 0.5
    c, ref = check(a, b1)
    assert _rel(c[17], ref[17]) <= 2.0 ** -23
    # sums beyond the largest value
    a, b1 = a0.clone(), b.clone()
    a[30], b1[40] = 1e38, 1.0
    c = torch.empty(m, n, device=DEV)
    L.gemm(c, a, b1, False, True)
    assert c[30, 40].item() == float("inf")
    # tiny operands: their parts, and the products of both, leave the normal range
    for sa, sb in ((2.0 ** -120, 2.0 ** 60), (2.0 ** -60, 2.0 ** -58), (2.0 ** 100, 2.0 ** -110)):
        c, ref = check(a0 * sa, b * sb)
        assert _rel(c, ref) <= 8.0 * k ** 0.5 * 2.0 ** -24
    # an operand of zeros
    c, ref = check(a0 * 0.0, b)
    assert bool((c == 0).all())


@pytest.mark.parametrize("m,n,k", [(512, 3072, 300), (256, 768, 3072)])
@pytest.mark.parametrize("ta,tb", [(0, 1), (1, 0)])
def test_rows_and_columns_of_any_size_side_by_side(m, n, k, ta, tb):
    """Every row and every column keeps its own precision, down to subnormal values, whatever size its neighbours in the tile
    have: the error of the block of each pair of sizes against its own norm.  Sums in the subnormal range are spaced 2^-149
    apart: half of that for the product's result and for each of the k additions that an FMA chain would make there."""
    a, b = _operands(m, n, k, ta, tb)
    rows, cols = (0, -55, -110, -116, -124, -140), (0, -55, -100, 60, -124)
    ra, cb = torch.arange(m, device=DEV) % len(rows), torch.arange(n, device=DEV) % len(cols)
    sa, sb = torch.tensor([2.0 ** e for e in rows], device=DEV)[ra], torch.tensor([2.0 ** e for e in cols], device=DEV)[cb]
    a, b = (a * sa if ta else a * sa[:, None]), (b * sb[:, None] if tb else b * sb)
    c = torch.empty(m, n, device=DEV)
    L.gemm(c, a, b, bool(ta), bool(tb))
    ref = _product(a, b, ta, tb)
    assert bool(torch.isfinite(c).all())
    for i in range(len(rows)):
        for j in range(len(cols)):
            got, want = c[ra == i][:, cb == j].double(), ref[ra == i][:, cb == j]
            spacing = 2.0 ** -150 * k * want.numel() ** 0.5
            assert (got - want).norm().item() <= 8.0 * k ** 0.5 * 2.0 ** -24 * want.norm().item() + spacing, (rows[i], cols[j])


@pytest.mark.parametrize("m,n,k", [(512, 3072, 300), (256, 768, 3072)])
def test_sums_near_the_largest_value(m, n, k):
    """Products and sums beyond what the scaled parts can carry, none of them beyond fp32: rows of 2^60 times columns of
    2^20 and 2^55, and a value of 2^110 among ordinary ones."""
    a, b = _operands(m, n, k, 0, 1)
    a[m // 2:] *= 2.0 ** 60
    b *= 2.0 ** 20
    b[n // 3:] *= 2.0 ** 35
    a[7, 3] = 2.0 ** 110
    b[:, 3] = 1.0
    c = torch.empty(m, n, device=DEV)
    L.gemm(c, a, b, False, True)
    ref = _product(a, b, 0, 1)
    assert bool(torch.isfinite(c).all())
    for rows in (slice(0, 7), slice(7, 8), slice(8, m // 2), slice(m // 2, m)):
        for cols in (slice(0, n // 3), slice(n // 3, n)):
            assert _rel(c[rows, cols], ref[rows, cols]) <= 8.0 * k ** 0.5 * 2.0 ** -24


def test_a_smaller_grid_gives_the_same_sums():
    """Tiles walked by 40 CTAs instead of all: the splits are the same, hence the bits."""
    a, b = _operands(1500, 1300, 700, 0, 1)
    c, d = torch.empty(1500, 1300, device=DEV), torch.empty(1500, 1300, device=DEV)
    L.gemm(c, a, b, False, True)
    prev = L.set_sm_budget(40)
    try:
        assert "splits=1 " in L.plan(L.make_desc(d, a, b, False, True)) and "grid=40" in L.plan(L.make_desc(d, a, b, False, True))
        L.gemm(d, a, b, False, True)
    finally:
        L.set_sm_budget(prev)
    assert torch.equal(c, d)


# rows and columns at the ends of the matrix and of a warp's block, k that is no multiple of the four taken at a time
@pytest.mark.parametrize("m,n,k", [(129, 3001, 130), (300, 500, 777), (256, 768, 3071)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_sums_formed_again_by_fmas(m, n, k, ta, tb):
    """An infinity in the first and the last row and in a column sends every block that they cross through the FMA form; what
    they do not touch there comes out as precise as an FMA chain makes it."""
    a, b = _operands(m, n, k, ta, tb)
    at, bt = (a.T if ta else a), (b.T if tb else b)
    at[0, k - 1], at[m - 1, 0], bt[k // 2, n - 1] = float("inf"), -float("inf"), float("inf")
    c = torch.empty(m, n, device=DEV)
    L.gemm(c, a, b, bool(ta), bool(tb))
    ref = _product(a, b, ta, tb)
    assert torch.equal(torch.isinf(c), torch.isinf(ref)) and torch.equal(torch.isnan(c), torch.isnan(ref))
    assert torch.equal(c[torch.isinf(c)].double(), ref[torch.isinf(ref)])
    fine = torch.isfinite(ref)
    assert int(fine.sum()) == (m - 2) * (n - 1)
    assert _rel(c[fine], ref[fine]) <= 8.0 * k ** 0.5 * 2.0 ** -24
    assert _rel(c[1:m - 1, :n - 1][:, -64:], ref[1:m - 1, :n - 1][:, -64:]) <= 8.0 * k ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("limit_ns", [500000, 2 ** 64 - 1])
def test_a_short_wait_limit_allows_for_sums_formed_again(limit_ns):
    """25000 k per split take milliseconds when they are formed again by FMAs, with the other warps waiting: no reason to give up,
    also where a caller allows a wait half a millisecond, or as long as it can say."""
    k = 200000
    a, b = _operands(128, 128, k, 0, 1)
    a[5, 7] = float("nan")
    c = torch.empty(128, 128, device=DEV)
    L.gemm(c, a, b, False, True)
    torch.cuda.synchronize()
    L.set_wait_limit_ns(gemm_ns=limit_ns)
    try:
        L.gemm(c, a, b, False, True)
        assert L.device_status() == (0, 0)
    finally:
        L.set_wait_limit_ns(gemm_ns=2000000000)
    ref = _product(a, b, 0, 1)
    rows = torch.arange(128, device=DEV) != 5
    assert bool(torch.isnan(c[5]).all()) and _rel(c[rows], ref[rows]) <= 8.0 * k ** 0.5 * 2.0 ** -24
