"""RMSNorm of many short rows, a warp each: against float64, with gathered rows and at the edges of
the sizes that take this form (1,024 rows, 1,024 values)."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("R, H", [(1023, 1024), (1024, 1024), (1025, 4), (5000, 512), (4740, 516),
                                  (1100, 1028)])
@pytest.mark.parametrize("w_dtype, y_dtype", [("bfloat16", "bfloat16"), ("float32", "float32")])
@pytest.mark.parametrize("gather", [False, True])
def test_many_short_rows(R, H, w_dtype, y_dtype, gather):
    gen = torch.Generator().manual_seed(R + H)
    x = torch.randn((R + 7, H), generator=gen).to(DEV)
    w = torch.randn((H,), generator=gen).to(getattr(torch, w_dtype)).to(DEV)
    rows = torch.randperm(R + 7, generator=gen)[:R].to(torch.int32).to(DEV) if gather else None
    y = torch.full((R, H), float("nan"), dtype=getattr(torch, y_dtype), device=DEV)
    K.rmsnorm(x if gather else x[:R], w, 1e-6, y, rows, R, None)
    v = (x[rows.long()] if gather else x[:R]).double()
    want = w.double() * v / (v.square().mean(1, keepdim=True) + 1e-6).sqrt()
    # a rounding of the stored type on every value, and float32 sums
    tol = 2.0 ** -8 if y_dtype == "bfloat16" else 2e-6
    assert ((y.double() - want).abs() <= tol * want.abs() + 1e-6).all()


# the same sums in the same order whichever form the number of rows takes, so the same values
@pytest.mark.parametrize("H", [4, 260, 512, 516, 1000, 1024])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_a_rows_values_do_not_depend_on_how_many_there_are(H, dtype):
    gen = torch.Generator().manual_seed(H)
    R, dt = 2100, getattr(torch, dtype)
    x = (torch.randn((R, H), generator=gen) * torch.rand((R, 1), generator=gen).exp()).to(DEV)
    w = torch.randn((H,), generator=gen).to(dt).to(DEV)
    got, want = torch.empty((R, H), dtype=dt, device=DEV), torch.empty((R, H), dtype=dt, device=DEV)
    K.rmsnorm(x, w, 1e-6, got, None, R, None)
    for r in range(0, R, 700):
        K.rmsnorm(x[r:r + 700], w, 1e-6, want[r:r + 700], None, 700, None)
    assert torch.equal(got, want)
