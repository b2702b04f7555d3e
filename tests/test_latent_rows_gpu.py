"""The latents' norms and rotation of many tokens, a warp a token, against float64 and against the form of
few tokens; sizes and places that the form does not take."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K
from tests.gpu_helpers import DEV, make_line, make_step

pytestmark = pytest.mark.gpu


# 256 tokens is where the form changes; ranks that fill a lane's pieces and that do not, no query latent,
# a part that does not rotate as a whole, columns off the 16-byte boundaries
@pytest.mark.parametrize("T", [255, 256, 301])
@pytest.mark.parametrize("qr, kvr, rd, dims, shift", [(768, 512, 64, 64, 0), (512, 256, 32, 32, 8), (1024, 264, 40, 24, 0),
                                                      (0, 128, 64, 32, 8), (8, 8, 8, 0, 0), (768, 512, 64, 64, 1), (1032, 512, 64, 64, 0)])
def test_latent_rows(T, qr, kvr, rd, dims, shift):
    gen = torch.Generator().manual_seed(T)
    draw = lambda *s: torch.randn(s, generator=gen).bfloat16().to(DEV)
    wide = (qr + kvr + rd + 24) // 8 * 8
    f, wq, wkv = draw(T, wide), draw(max(qr, 1)), draw(kvr)
    inv_freq = torch.rand(max(dims // 2, 1), generator=gen).to(DEV)
    past = 70
    step = make_step([(0, past, [0] * T, [])])
    got = []
    for n in (T, 100):      # all at once, and in steps of 100 tokens
        line = make_line(1, past + T, 1, kvr + rd, torch.bfloat16, seed=3)
        cq = torch.zeros((T, qr), dtype=torch.bfloat16, device=DEV)
        for a in range(0, T, n):
            m = min(n, T - a)
            part = step if n == T else make_step([(0, past + a, [0] * m, [])])
            K.latent_prep(f[a:a + m], shift, shift + qr, qr, kvr, rd, wq, wkv, 1e-5, inv_freq, dims, 1.5,
                          part, line, cq[a:a + m], True)
        table = line.page_table[0].long()
        rows = line.k[table, 0].reshape(-1, kvr + rd)[past:past + T]
        got.append(torch.cat([cq, rows], 1).double())
    x = f.double()
    norm = lambda v, w: v * torch.rsqrt(v.square().mean(1, keepdim=True) + 1e-5) * w.double()
    q, c, r = (x[:, shift + a:shift + b] for a, b in ((0, qr), (qr, qr + kvr), (qr + kvr, qr + kvr + rd)))
    half = dims // 2
    ang = (torch.arange(past, past + T, device=DEV, dtype=torch.float32)[:, None] * inv_freq[:half]).double()
    u, v = r[:, :half], r[:, half:dims]
    turned = torch.cat([1.5 * (u * ang.cos() - v * ang.sin()), 1.5 * (v * ang.cos() + u * ang.sin()), r[:, dims:]], 1)
    want = torch.cat(([norm(q, wq)] if qr else []) + [norm(c, wkv), turned], 1)
    # rounding to bfloat16's 8 bits: half a unit, 2^-8 of the value at most, and a little for float32 (the
    # angles' float32 products among it: some 370 radians times 2^-24)
    for g in got:
        assert ((g - want).abs() <= (2.0 ** -8 + 1e-5) * want.abs() + 2e-4).all()
    assert (got[0] - got[1]).norm() <= 1e-4 * want.norm()      # other sums: few values round otherwise


# both forms add the squares up in the same order: a step of many tokens leaves the bits that steps of few leave
@pytest.mark.parametrize("T", [256, 777])
@pytest.mark.parametrize("qr, kvr, rd, dims", [(768, 512, 64, 64), (512, 256, 32, 32), (1024, 264, 40, 24), (0, 128, 64, 32),
                                               (8, 8, 8, 0), (136, 24, 16, 16)])
def test_the_bits_of_few_tokens(T, qr, kvr, rd, dims):
    gen = torch.Generator().manual_seed(T + qr)
    draw = lambda *s: torch.randn(s, generator=gen).bfloat16().to(DEV)
    f, wq, wkv = draw(T, qr + kvr + rd), draw(max(qr, 1)), draw(kvr)
    f[3] *= 1e-3      # the norm's eps counts
    f[5, 0] = float("inf")
    inv_freq = torch.rand(max(dims // 2, 1), generator=gen).to(DEV)
    got = []
    for n in (T, 100):
        line = make_line(1, T, 1, kvr + rd, torch.bfloat16, seed=3)
        cq = torch.zeros((T, qr), dtype=torch.bfloat16, device=DEV)
        for a in range(0, T, n):
            m = min(n, T - a)
            K.latent_prep(f[a:a + m], 0, qr, qr, kvr, rd, wq, wkv, 1e-5, inv_freq, dims, 1.0,
                          make_step([(0, a, [0] * m, [])]), line, cq[a:a + m], True)
        got.append(torch.cat([cq.flatten().view(torch.int16), line.k.flatten().view(torch.int16)]))
    assert torch.equal(got[0], got[1])
