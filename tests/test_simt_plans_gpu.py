"""The float32 products' forms at their edges: rows up to 16 (warps that share a weight row's K) and
more: float32 operands on the tensor cores where K is above 64 (test_split_products_gpu.py has that
form's own edges), an operand in bfloat16 in tiles of 64 x 128, K dealt out over a cluster. Small
whole numbers make every sum exact, so the results must equal the oracle's bit for bit; SwiGLU is
compared in float64."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def whole(shape, seed, most=3):
    gen = torch.Generator().manual_seed(seed)
    return torch.randint(-most, most + 1, shape, generator=gen).float().to(DEV)


# K = 1030 and 37 leave no whole pieces of four values, 132 a ragged last step, 2,048 splits
@pytest.mark.parametrize("M", [1, 9, 16, 17, 64, 65, 200])
@pytest.mark.parametrize("N, Kd", [(3, 37), (130, 132), (96, 1030), (1024, 2048), (260, 4096)])
def test_store_and_add(M, N, Kd):
    a, w, c = whole((M, Kd), 1), whole((N, Kd), 2), whole((M, N), 3, 50)
    exact = a @ w.t()
    out = torch.empty((M, N), device=DEV)
    K.gemm_simt(a, w, out)
    assert torch.equal(out, exact)
    K.gemm_simt(a, w, c_add := c.clone(), K.EPI_ADD)
    assert torch.equal(c_add, c + exact)


@pytest.mark.parametrize("M", [1, 16, 17, 70])
@pytest.mark.parametrize("N, Kd", [(5, 40), (65, 132), (512, 2048)])
@pytest.mark.parametrize("pairs", [True, False])
def test_swiglu(M, N, Kd, pairs):
    a, w = whole((M, Kd), 4) * 0.05, whole((2 * N, Kd), 5) * 0.25
    z = a.double() @ w.double().t()
    g, u = (z[:, 0::2], z[:, 1::2]) if pairs else (z[:, :N], z[:, N:])
    want = torch.nn.functional.silu(g) * u
    out = torch.empty((M, N), device=DEV)
    K.gemm_simt(a, w, out, K.EPI_SWIGLU_PAIRS if pairs else K.EPI_SWIGLU)
    # float32 sums of up to 2,048 terms: the error grows with their root
    assert (out.double() - want).norm() <= 5e-6 * want.norm()


# a weight that the library's kernel just before writes: read only after that kernel has ended
@pytest.mark.parametrize("M", [1, 16, 40])
def test_a_weight_of_the_kernel_before(M):
    N, Kd, inner = 512, 1024, 2048
    left, right, a = whole((N, inner), 7, 1), whole((Kd, inner), 8, 1), whole((M, Kd), 9, 2)
    w, out = torch.empty((N, Kd), device=DEV), torch.empty((M, N), device=DEV)
    exact = a.double() @ (left.double() @ right.double().t()).t()      # whole numbers below 2^24
    assert exact.abs().max() < 2 ** 24
    for _ in range(10):
        w.zero_()
        K.gemm_simt(left, right, w)
        K.gemm_simt(a, w, out)
        assert torch.equal(out.double(), exact)


# few rows of A: one or two, whose values are asked for with the weight's; up to eight and more than eight in
# shared memory (a large weight), the last of them in two passes a group; whole numbers, every pair of types
@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 13, 16])
@pytest.mark.parametrize("N, Kd", [(20001, 516), (6000, 1024), (7, 4096), (20, 64)])
@pytest.mark.parametrize("types", ["ff", "fb", "bb", "bf"])
def test_few_rows(M, N, Kd, types):
    kind = {"f": torch.float32, "b": torch.bfloat16}
    a, w, c = whole((M, Kd), 1).to(kind[types[0]]), whole((2 * N, Kd), 2).to(kind[types[1]]), whole((M, N), 3, 50)
    exact = a.float() @ w.float().t()
    out = torch.empty((M, 2 * N), device=DEV)
    K.gemm_simt(a, w, out, settled=True)
    assert torch.equal(out, exact)
    K.gemm_simt(a, w[:N], c_add := c.clone(), K.EPI_ADD)
    assert torch.equal(c_add, c + exact[:, :N])
    a, w = a * 0.0625, w * 0.25      # exact in bfloat16 too
    z = exact.double() / 64
    for epilogue, g, u in ((K.EPI_SWIGLU_PAIRS, z[:, 0::2], z[:, 1::2]), (K.EPI_SWIGLU, z[:, :N], z[:, N:])):
        K.gemm_simt(a, w, out := torch.empty((M, N), device=DEV), epilogue)
        want = torch.nn.functional.silu(g) * u
        assert (out.double() - want).norm() <= 2e-6 * want.norm()      # exact sums, expf and a division


# many rows with an operand in bfloat16: tiles of 64 x 128, K dealt out over up to eight CTAs (2,048 and 4,096),
# a ragged last step (132), no whole pieces of four values (1,030, 37)
@pytest.mark.parametrize("M", [17, 64, 65, 200])
@pytest.mark.parametrize("N, Kd", [(3, 37), (130, 132), (96, 1030), (1024, 2048), (260, 4096)])
@pytest.mark.parametrize("types", ["fb", "bb", "bf"])
def test_many_rows_in_bfloat16(M, N, Kd, types):
    kind = {"f": torch.float32, "b": torch.bfloat16}
    a, w, c = whole((M, Kd), 1).to(kind[types[0]]), whole((2 * N, Kd), 2).to(kind[types[1]]), whole((M, N), 3, 50)
    exact = a.float() @ w.float().t()
    K.gemm_simt(a, w, out := torch.empty((M, 2 * N), device=DEV))
    assert torch.equal(out, exact)
    K.gemm_simt(a, w[:N], c_add := c.clone(), K.EPI_ADD)
    assert torch.equal(c_add, c + exact[:, :N])
    z = exact.double() / 64
    for epilogue, g, u in ((K.EPI_SWIGLU_PAIRS, z[:, 0::2], z[:, 1::2]), (K.EPI_SWIGLU, z[:, :N], z[:, N:])):
        K.gemm_simt(a * 0.0625, w * 0.25, out := torch.empty((M, N), device=DEV), epilogue)
        want = torch.nn.functional.silu(g) * u
        assert (out.double() - want).norm() <= 2e-6 * want.norm()      # exact sums, expf and a division
