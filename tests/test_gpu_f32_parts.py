"""Float32 products on tensor-core parts: operands that two tf32 parts cannot hold."""
from __future__ import annotations

import pytest
import torch

import pamasun_util as pu

pytestmark = pytest.mark.gpu
INF = float("inf")


@pytest.fixture(scope="module")
def engine():
    model, _, _ = pu.engine_and_oracle(pu.config([pu.attn(heads=1, kv_heads=1, dim=8, vdim=8, ff=0)], vocab=33, width=16), seed=1)
    return model


# rows: a tile of 16 and of 64 rows, with remainders; few columns and a long sum: K shared by a cluster; sums of fewer than 72 k: on FMAs
@pytest.mark.parametrize("m,n,k", [(1, 40, 36), (17, 72, 68), (1, 33, 72), (33, 65, 76), (65, 130, 4100), (16, 64, 1536)])
def test_infinities_and_numbers_next_to_them(engine, m, n, k):
    g = torch.Generator().manual_seed(m)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g)
    w[0] = w[0].abs() + 0.5
    a[0, k // 2] = INF                                     # a signed infinity in all of row 0
    w[3, k - 1] = -INF                                     # and in all of column 3
    if m > 1:
        a[m - 1] = 0.0
        a[m - 1, 1] = torch.finfo(torch.float32).max       # in the last half step of tf32 below the largest float: its upper part rounds to infinity
        w[1] = 0.0
        w[1, 1] = 0.25
    got = engine.linear(a.cuda(), w.cuda()).cpu()
    want = (a.double() @ w.double().T).float()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    same = want.isfinite()
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    # sums of k products: k / 2 roundings of 2^-24 of the sum of their sizes, and 2^-21 of each product for the parts
    bound = (a.double().abs() @ w.double().abs().T) * (k / 2 * 2.0 ** -24 + 2.0 ** -21)
    assert bool(((got.double() - want.double()).abs()[same] <= bound[same]).all())
    if m > 1:
        assert got[m - 1, 1].item() == torch.finfo(torch.float32).max * 0.25


@pytest.mark.parametrize("size", [2.0 ** -118, 2.0 ** -122, 2.0 ** -125])
def test_small_operands_keep_their_bits(engine, size):
    """Products that nothing larger hides: operands whose lower part would be denormal."""
    g = torch.Generator().manual_seed(3)
    a, w = torch.randn(20, 96, generator=g) * size, torch.randn(40, 96, generator=g)
    got = engine.linear(a.cuda(), w.cuda()).cpu().double()
    want = a.double() @ w.double().T
    bound = (a.double().abs() @ w.double().abs().T) * 96 * 2.0 ** -24 + 96 * 2.0 ** -150
    assert bool(((got - want).abs() <= bound).all())
