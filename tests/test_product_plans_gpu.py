"""How the tensor-core products are cut up: bands of row tiles for many tokens, and K split
where few tiles leave the device idle. Small whole numbers as operands make every sum exact in
float32, whatever the order, so the results must equal the oracle's bit for bit."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


def whole(shape, seed, most=2):
    gen = torch.Generator().manual_seed(seed)
    return torch.randint(-most, most + 1, shape, generator=gen).to(torch.bfloat16).to(DEV)


def product(a, w, c, add, workspace):
    error = torch.zeros(1, dtype=torch.int32, device=DEV)
    splits = K.gemm_tc(a, w, c, add, workspace, error, SMS)
    assert int(error.item()) == 0
    return splits


# 18 row tiles of 4 MB (three bands of six, the last row tile ragged), and 130 of half a
# megabyte (bands of 44 and a shorter last one)
@pytest.mark.parametrize("M, N, Kd", [(4500, 272, 8192), (33100, 520, 1024)])
def test_bands_of_row_tiles(M, N, Kd):
    a, w = whole((M, Kd), 1), whole((N, Kd), 2)
    c = torch.zeros((M, N), dtype=torch.float32, device=DEV)
    product(a, w, c, True, None)
    assert torch.equal(c, a.float() @ w.float().t())


# around the edges of the forms (64 | 65 .. 128 | 129 tokens), where the sums are added up four
# at a time (N a multiple of 4) and one by one (N = 1,030)
@pytest.mark.parametrize("M", [65, 128, 129, 300, 513, 1500])
@pytest.mark.parametrize("N, Kd", [(1024, 2048), (260, 4096), (1030, 2048)])
@pytest.mark.parametrize("how", ["add", "float32", "bfloat16"])
def test_split_sums(M, N, Kd, how):
    a, w = whole((M, Kd), 3), whole((N, Kd), 4)
    workspace = torch.empty(16 << 20, dtype=torch.float32, device=DEV)
    exact = a.float() @ w.float().t()
    c = whole((M, N), 5, 100).to(torch.bfloat16 if how == "bfloat16" else torch.float32)
    want = exact + c if how == "add" else exact.to(c.dtype)
    splits = product(a, w, c, how == "add", workspace)
    assert torch.equal(c, want)
    if M <= 129:
        assert splits > 1      # one row tile of 128 (or 256) tokens leaves most of the device idle
