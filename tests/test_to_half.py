"""Keys and queries become float16 (or stay float32 where a value would not be finite in it) in one kernel: partial vectors of
eight, arrays that do not begin on a 16-byte boundary, every type it takes, and a bad value at either end."""

import pytest
import torch

from libcertex_b200.attention import _as_half_or_float

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float64])
@pytest.mark.parametrize("n,offset", [(0, 0), (1, 0), (7, 1), (8, 0), (1000, 3), (400_001, 0)])
def test_same_as_rounding_and_checking(n, offset, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = (torch.randn(n + offset, generator=g, device="cuda") * 1000).to(dtype)[offset:]
    for bad in (None, 0, n - 1):
        for value in (float("inf"), float("nan"), 65520.0):
            y = x.clone() if offset == 0 else torch.cat([x[:0].new_zeros(offset), x])[offset:]
            if bad is not None and n > 0:
                y[bad] = value
            h = y.to(torch.float16)
            want = h if bool(torch.isfinite(h).all()) else y.to(torch.float32)
            got = _as_half_or_float(y)
            assert got.dtype == want.dtype and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))
    if n > 8:
        t = x[: n // 8 * 8].reshape(8, -1).t()
        assert torch.equal(_as_half_or_float(t), t.to(torch.float16))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_views_that_negate_when_they_are_read(dtype):
    x = torch.randn((1000,), device="cuda").to(dtype)
    v = torch._neg_view(x)
    assert v.is_neg() and v.is_contiguous()
    got = _as_half_or_float(v)
    assert torch.equal(got, -x.to(torch.float16)) and not got.is_neg()
