"""Float32 products of more than 16 rows, whose values are cut into three bfloat16 parts: every tile
width and share of K, rows that are no whole tiles, bases off the 16-byte boundaries, infinities and
NaNs, and the error against float64 beside that of a chain of float32 multiply-adds."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def drawn(shape, seed, whole=False):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randint(-3, 4, shape, generator=gen).float() if whole else torch.randn(shape, generator=gen)
    return x.to(DEV)


# whole numbers: every sum is exact. Tiles of 16, 96 (four stages of the weight), 112 (three) and 128
# (two) rows; K shared by 1, 2, 5 and 8 CTAs, with ragged last stages
@pytest.mark.parametrize("cols, splits", [(16, 1), (16, 8), (96, 1), (96, 2), (112, 1), (112, 5), (128, 1), (128, 3)])
@pytest.mark.parametrize("M, N, Kd", [(17, 5, 1028), (129, 130, 1095), (300, 384, 1056)])
def test_plans(cols, splits, M, N, Kd):
    a, w = drawn((M, Kd), 1, True), drawn((2 * N, Kd), 2, True)
    error = torch.zeros(1, dtype=torch.int32, device=DEV)
    exact = a.double() @ w.double().t()
    out = torch.empty((M, 2 * N), device=DEV)
    K.gemm_split(a, w, out, K.EPI_STORE, error, cols, splits)
    assert torch.equal(out.double(), exact)
    K.gemm_split(a, w, out, K.EPI_ADD, error, cols, splits)
    assert torch.equal(out.double(), 2 * exact)
    a, w = a * 0.05, w * 0.25
    z = a.double() @ w.double().t()
    want = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2]
    for dtype, bound in ((torch.float32, 2e-6), (torch.bfloat16, 4e-3)):    # half a unit of the last place
        out = torch.empty((M, N), dtype=dtype, device=DEV)
        K.gemm_split(a, w, out, K.EPI_SWIGLU_PAIRS, error, cols, splits)
        assert (out.double() - want).norm() <= bound * want.norm()
    assert int(error) == 0


# tiles in several rounds of the device's CTAs
def test_many_tiles():
    a, w = drawn((1000, 96), 3, True), drawn((6000, 96), 4, True)
    out = torch.empty((1000, 6000), device=DEV)
    K.gemm_simt(a, w, out)
    assert torch.equal(out, a @ w.t())


@pytest.mark.parametrize("shift_a, shift_w, ld", [(1, 0, 200), (0, 1, 200), (0, 0, 203), (3, 2, 201)])
def test_rows_off_the_boundaries(shift_a, shift_w, ld):
    M, N, Kd = 70, 140, 200
    a = drawn((M * ld + 8,), 5, True)[shift_a:shift_a + M * ld].view(M, ld)[:, :Kd]
    w = drawn((N * Kd + 8,), 6, True)[shift_w:shift_w + N * Kd].view(N, Kd)
    out = torch.empty((M, N + 3), device=DEV)[:, :N]
    K.gemm_simt(a, w, out)
    assert torch.equal(out.double(), a.double() @ w.double().t())


# infinities, NaNs (one whose upper 16 bits are an infinity's), the largest and the smallest values
def test_values_that_are_no_numbers():
    M, N, Kd = 40, 130, 160
    a, w = drawn((M, Kd), 7), drawn((N, Kd), 8)
    a[3, 5], a[4, 7], a[5, 9] = float("inf"), float("-inf"), float("nan")
    a.view(torch.int32)[6, 11] = 0x7F800001
    a[7] *= 1e-38
    a[8, :], w[:, 0] = 0.0, 1.0
    a[8, 0] = torch.finfo(torch.float32).max
    w[9, 20], w[10, 21] = float("inf"), float("nan")
    out = torch.empty((M, N), device=DEV)
    K.gemm_simt(a, w, out)
    want = a.double() @ w.double().t()
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.isposinf(), want.isposinf()) and torch.equal(out.isneginf(), want.isneginf())
    fine = want.isfinite()
    rows = [m for m in range(M) if m != 7]      # 1e-38: its parts leave float32's normal range
    assert ((out.double() - want)[rows][fine[rows]].abs() <= 1e-5 * Kd ** 0.5 * want[rows][fine[rows]].abs()
            .clamp_min(1.0)).all()
    assert (out.double() - want)[7][fine[7]].abs().max() <= 1e-38


# Kd 2^-24 is what a chain of Kd multiply-adds may lose of the sum of magnitudes; four parts of it are far
# from what is measured (1.3e-7 to 1.9e-7 of the result for 1,024 to 12,288 values)
@pytest.mark.parametrize("Kd", [64, 1024, 12288])
def test_error_against_float64(Kd):
    a, w = drawn((130, Kd), 9), drawn((200, Kd), 10)
    out = torch.empty((130, 200), device=DEV)
    K.gemm_simt(a, w, out)
    want = a.double() @ w.double().t()
    assert (out.double() - want).norm() <= 4e-7 * want.norm()


# Values below 2^-110 have bits that no bfloat16 part holds: what they take part in is multiplied and added
# in float32, and errs by no more than such a chain: 4e-7 of the result as above, and of results below
# float32's normal range half a last place, 2^-150, a step
@pytest.mark.parametrize("M, N, Kd", [(40, 130, 160), (150, 70, 1095)])
@pytest.mark.parametrize("splits", [1, 3])
def test_small_values(M, N, Kd, splits):
    splits = splits if Kd >= 128 * splits else 0
    a, w, c = drawn((M, Kd), 11), drawn((N, Kd), 12), drawn((M, N), 13)
    small = {3: -104, 17: -111, 18: -120, 30: -126, 31: -140}
    for row, e in small.items():
        a[row] *= 2.0 ** e
    w[9] *= 2.0 ** -118
    a[6, 20] = 2.0 ** -119 * 1.0000001      # one beside others
    error, out = torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty((M, N), device=DEV)
    K.gemm_split(a, w, out, K.EPI_STORE, error, 0, splits)
    want = a.double() @ w.double().t()
    err = (out.double() - want).abs()
    near = lambda x, y: x.norm() <= 4e-7 * y.norm() + Kd * 2.0 ** -150 * y.numel() ** 0.5
    for row in (*small, 0, 6, M - 1):
        assert near(err[row], want[row]), (row, err[row].norm() / want[row].norm())
    assert near(err[:, 9], want[:, 9])
    a[0, 5], w[11, 5] = float("inf"), 2.0 ** -140      # infinity, not 0 * infinity, whose first part is zero
    K.gemm_split(a, w, c_add := c.clone(), K.EPI_ADD, error, 0, splits)
    want = c.double() + a.double() @ w.double().t()
    assert torch.equal(c_add.isposinf(), want.isposinf()) and torch.equal(c_add.isneginf(), want.isneginf())
    assert not c_add.isnan().any()
    fine = want.isfinite()
    assert (c_add.double() - want)[fine].norm() <= 4e-7 * want[fine].norm() and int(error) == 0


# the rows' parts take no more than SPLIT_SCRATCH: more rows go in bands of whole tiles through the same
# scratch, whole numbers so that every sum is exact
@pytest.mark.parametrize("rows", [1, 100, 128, 300])
@pytest.mark.parametrize("epilogue", [K.EPI_STORE, K.EPI_ADD, K.EPI_SWIGLU_PAIRS])
def test_bands(monkeypatch, rows, epilogue):
    M, N, Kd = 411, 260, 1090
    a, w, c = drawn((M, Kd + 3), 1, True)[:, :Kd], drawn((N, Kd), 2, True), drawn((M, N), 3, True)
    if epilogue == K.EPI_SWIGLU_PAIRS:
        a, w, c = a * 0.05, w * 0.25, c[:, :N // 2].bfloat16()
    want = c.clone()
    K.gemm_split(a, w, want, epilogue)
    monkeypatch.setattr(K, "SPLIT_SCRATCH", 6 * 1096 * rows + 7)
    if rows == 1:
        a, c, want = a[:5], c[:5], want[:5]
    K.gemm_split(a, w, c, epilogue, cols=0 if epilogue != K.EPI_SWIGLU_PAIRS else 128)
    if epilogue == K.EPI_SWIGLU_PAIRS:      # other tiles, other sums: half a place of bfloat16
        assert (c.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()
    else:
        assert torch.equal(c, want)


# a prefill of the default step size: 16,384 rows of 12,288 values
def test_memory():
    a, w = torch.zeros((16384, 12288), device=DEV), torch.zeros((128, 12288), device=DEV)
    out = torch.empty((16384, 128), device=DEV)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    K.gemm_simt(a, w, out)
    assert torch.cuda.max_memory_allocated() - before <= 256 << 20
    assert not out.any()
