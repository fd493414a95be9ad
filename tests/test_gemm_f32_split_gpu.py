"""32-bit products on the tensor cores: three exact bfloat16 parts a number, at the edges of its tiles and rings."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def k():
    from rapid_llm_b200.ops import kernels

    return kernels


def product(a, w, bias=None):
    out = torch.full((a.shape[0], w.shape[0] + 4), 7.0, device=DEV)
    fault = torch.zeros(1, dtype=torch.int32, device=DEV)
    k().gemm_f32(a, w, out[:, : w.shape[0]], bias, fault)
    assert int(fault) == 0 and bool((out[:, w.shape[0] :] == 7.0).all())
    return out[:, : w.shape[0]]


# weights on the line of the rule; rows that are no whole tile; columns of one to eight segments, of a last step with four columns
# (a sum of one step behind whole ones, steps of odd number) and of no whole 16 bytes of parts
@pytest.mark.parametrize("n,inner", [(8192, 1024), (2100, 4100), (1025, 8460), (24700, 1284)])
def test_rows_are_near_and_the_same_at_every_count(n, inner):
    torch.manual_seed(5)
    rows = [1, 16, 17, 32, 33, 64, 65, 112, 128, 129, 208, 209, 300, 1025]
    a, w, bias = torch.randn(max(rows), inner, device=DEV), torch.randn(n, inner, device=DEV), torch.randn(n, device=DEV)
    want = a.double() @ w.double().t() + bias.double()
    # Of the sum S of the products' magnitudes: a sum of 256 columns is cut off 16 times below 2^-23 of what it holds, the parts'
    # products that are left out stay within 2^-24, the small ones (2^-7 of the whole) are cut off 5 k / 16 times below 2^-23
    # of theirs, and the float32 sums of k / 256 such round to 2^-24
    magnitude = a.abs().double() @ w.abs().double().t() + bias.abs().double()
    bound = magnitude * (16 + 2 + 5 * inner / 16 / 128 + inner / 512 + 1) * 2.0 ** -23
    # and as random sums go, a small part of it: no further off than one multiply-add after the other would be on average
    typical = 0.5 * math.sqrt(inner) * 2.0 ** -24
    first = None
    for m in rows:
        got = product(a[:m], w, bias)
        assert bool(((got.double() - want[:m]).abs() <= bound[:m]).all()), m
        assert float((got.double() - want[:m]).norm() / want[:m].norm()) < typical, m
        first = got[:1].clone() if first is None else first
        assert torch.equal(got[:1], first), m


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_rows_off_a_16_byte_boundary(offset):
    torch.manual_seed(6)
    wide, w = torch.randn(70, 4101, device=DEV), torch.randn(2048, 4096, device=DEV)
    for m in (1, 20, 70):
        view = wide[:m, offset : offset + 4096]
        assert torch.equal(product(view, w), product(view.contiguous(), w))


@pytest.mark.parametrize("m", [3, 40, 130])
def test_what_is_not_finite_stays_in_its_row_and_column(m):
    torch.manual_seed(7)
    a, w = torch.randn(m, 4096, device=DEV), torch.randn(2048, 4096, device=DEV)
    clean = product(a, w)
    a[1, 5], w[7, 9] = math.inf, math.nan
    a[2, 11], w[9, 100] = 3.0e38, 3.0e38
    got = product(a, w)
    want = (a.double() @ w.double().t()).float()
    assert bool(got[:, 7].isnan().all()) and torch.equal(got[1].isinf(), want[1].isinf())
    assert torch.equal(got[1, want[1].isinf()], want[1, want[1].isinf()])
    kept = torch.ones_like(got, dtype=torch.bool)
    kept[1:3], kept[:, 7], kept[:, 9] = False, False, False
    assert torch.equal(got[kept], clean[kept])
    assert bool(torch.isfinite(got[2][torch.isfinite(want[2])]).all())


@pytest.mark.parametrize("n,inner", [(8192, 1024), (1025, 8460)])
def test_a_row_is_the_same_in_every_tile_and_pass(n, inner):
    torch.manual_seed(8)
    a, w = torch.randn(1100, inner, device=DEV), torch.randn(n, inner, device=DEV)
    for m in (33, 209, 416, 1024, 1060, 1100):
        got = product(a[:m], w)
        for at in {0, 15, 16, 31, 32, 104, 111, 112, 207, 208, 415, 831, 832, 1023, 1024, 1059, m - 1}:
            if at < m:
                assert torch.equal(got[at : at + 1], product(a[at : at + 1], w)), (m, at)


@pytest.mark.parametrize("rows", [5, 70, 209])
def test_a_product_by_itself_is_rounded_twice_at_most(rows):
    """Rows with a single number that is not zero: what the parts' products leave out and the rounding of their sum, 2^-24 each
    (a multiply-add has the second alone); either way as often as the other, and together hardly more than a rounding by itself."""
    torch.manual_seed(9)
    n, inner = 8192, 1028
    w, a = torch.randn(n, inner, device=DEV), torch.zeros(rows, inner, device=DEV)
    at = torch.randint(inner, (rows,), device=DEV)
    a[torch.arange(rows, device=DEV), at] = torch.randn(rows, device=DEV)
    a[0, at[0]] = 1 + 2.0 ** -7 - 2.0 ** -23           # cut off after 8 and 16 bits, both remainders are as large as they come
    w[::2, at[0]] = 1 + 2.0 ** -7 - 2.0 ** -23
    want = a.double() @ w.double().t()
    off = (product(a, w).double() - want) / want.abs()
    assert float(off.abs().max()) <= 2 * 2.0 ** -24 * (1 + 2.0 ** -5)
    rounded = (want.float().double() - want) / want.abs()
    assert float(off.norm()) <= 1.1 * float(rounded.norm())
    # of 10^4 numbers of at most 2^-23 and of a size of 2.6e-8: their mean is within five of its own deviations
    assert abs(float(off[1:].mean())) <= 5 * float(off[1:].std()) / (off[1:].numel() ** 0.5) + 2.0 ** -30


@pytest.mark.parametrize("rows", [1, 64, 203])
def test_what_is_not_finite_costs_no_more_than_a_few_products(rows):
    """A request that went astray holds up the others of its step: NaN in every row, infinities in one, NaN in a weight."""
    torch.manual_seed(10)
    n, inner = 24576, 4096
    w, spoilt = torch.randn(n, inner, device=DEV), torch.randn(n, inner, device=DEV)
    spoilt[::64, 3] = math.nan
    plain = torch.randn(rows, inner, device=DEV)
    nan, inf = plain.clone(), plain.clone()
    nan[:, 7], inf[rows // 2, 9] = math.nan, math.inf
    product(plain, w)
    for a, by in ((nan, w), (inf, w), (plain, spoilt)):
        product(a, by)
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        got = product(a, by)
        end.record()
        torch.cuda.synchronize()
        want = a.double() @ by.double().t()
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        # an infinity's row is 4.4 ms of sums; 203 rows of NaN would be 86 ms of them (with a buffer's filling and checking, 0.3 ms)
        assert begin.elapsed_time(end) < 15.0
