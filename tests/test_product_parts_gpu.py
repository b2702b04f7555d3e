"""How long the sums of one accumulator are where a product's tiles are fewer than the device takes
at once: K is cut, and whichever way its parts are brought together (in tensor memory by the
pair that has the tile, or through memory by a kernel of their own) the result is that of the parts'
sums added up in K's order, bit for bit."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K
from mormot2_ai_b200.csrc import build

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


def product(a, w, c, add, workspace):
    error = torch.zeros(1, dtype=torch.int32, device=DEV)
    K.gemm_tc(a, w, c, add, workspace, error, SMS)
    assert int(error.item()) == 0
    return build.load_library("gemm_tc").mb_gemm_tc_last()


# tokens, outputs, K, and the most blocks of 64 values of K in one sum: single CTAs (65 .. 128
# tokens), then pairs of them, with ragged last tiles, blocks and parts among them
@pytest.mark.parametrize("M, N, Kd, part", [
    (65, 1024, 2048, 4), (128, 4096, 4096, 4), (128, 300, 1000, 4),
    (129, 512, 12288, 6), (256, 1024, 1024, 4), (500, 2048, 2048, 7), (800, 1024, 2048, 7),
    (1024, 2048, 4096, 22), (2048, 2048, 2048, 11), (2048, 260, 1544, 5), (8000, 512, 1024, 6)])
@pytest.mark.parametrize("how", ["add", "float32", "bfloat16"])
def test_sums_are_those_of_the_parts(M, N, Kd, part, how):
    gen = torch.Generator(device=DEV).manual_seed(M + N)
    r = lambda *s, dt=torch.bfloat16: torch.randn(s, generator=gen, device=DEV).to(dt)
    a, w = r(M, Kd), r(N, Kd)
    c = r(M, N, dt=torch.bfloat16 if how == "bfloat16" else torch.float32)
    total = None
    for k in range(0, Kd, 64 * part):
        p = torch.empty((M, N), dtype=torch.float32, device=DEV)
        product(a[:, k:k + 64 * part], w[:, k:k + 64 * part].contiguous(), p, False, None)
        total = p if total is None else total + p
    want = c + total if how == "add" else total.to(c.dtype)
    workspace = torch.empty(16 << 20, dtype=torch.float32, device=DEV)
    assert product(a, w, c, how == "add", workspace) >> 16 == part
    assert torch.equal(c, want)
