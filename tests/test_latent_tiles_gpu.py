"""Which row tiles a CTA of the latent prefill takes (neighbours, or one from each end) changes
nothing: against the kernels that never form keys and values, at the edges of row tiles."""
import pytest
import torch

from mormot2_ai_b200 import PartSpec, Runtime
from mormot2_ai_b200.parts import MIXERS, POSITIONS
from mormot2_ai_b200.parts.block import settle
from tests.gpu_helpers import DEV, make_step
from mormot2_ai_b200.cache.pages import PAGE, CacheBook, pages_for, plan_groups
from mormot2_ai_b200.cache.storage import CacheStorage

pytestmark = pytest.mark.gpu


# heads x pairs of row tiles: up to 148 CTAs one from each end, above them neighbours
@pytest.mark.parametrize("heads, lens", [(4, [128]), (4, [129]), (4, [257]), (8, [640, 1, 300]),
                                         (40, [1000]), (2, [1200, 130])])
@pytest.mark.parametrize("window", [0, 200])
def test_row_tiles(heads, lens, window):
    w, d, rd, vd, kvr, qr = 256, 64, 32, 64, 128, 128
    gen = torch.Generator().manual_seed(sum(lens))
    r = lambda *s, std=0.05, mean=0.0: (torch.randn(s, generator=gen) * std + mean).to(torch.bfloat16).to(DEV)
    weights = {"dq": r(qr, w), "dq_norm": r(qr, std=0.1, mean=1.0), "uq": r(heads * (d + rd), qr),
               "dkv": r(kvr + rd, w), "dkv_norm": r(kvr, std=0.1, mean=1.0), "uk": r(heads * d, kvr),
               "uv": r(heads * vd, kvr), "o": r(w, heads * vd), "g": r(heads * vd, w)}
    rt = Runtime(torch.bfloat16, DEV)
    rot = POSITIONS.build(PartSpec("rope_half", {"theta": 1e4, "rot_dim": rd}))
    rot.bind({}, rt)
    part = MIXERS.build(PartSpec("latent_attention", {
        "hidden_size": w, "heads": heads, "dim": d, "rot_dim": rd, "vdim": vd, "kv_rank": kvr,
        "q_rank": qr, "scale": (d + rd) ** -0.5, "latent_norm_eps": 1e-6, "gate": True,
        "window": window, "position": "rot", "names": {n: n for n in weights}}), "",
        positions={"rot": rot})
    part.bind(weights, rt)
    plans = plan_groups({0: (1, kvr + rd, window, 1, 0)}, 4096, pages_for(max(lens)) * PAGE,
                        len(lens), max(lens))
    book = CacheBook(plans, len(lens), pages_for(max(lens)) * PAGE)
    cache = CacheStorage(plans, len(lens), rt.dtype, rt.device, {})
    cache.map_pages(book.reserve([(book.open(), n) for n in lens]))
    step = make_step([(i, 0, [0] * n, []) for i, n in enumerate(lens)])
    h = r(sum(lens), w, std=1.0)
    got = []
    for expands in (True, False):
        part.expands = lambda step, e=expands: e
        x = torch.zeros((sum(lens), w), device=DEV)
        pending = part.forward(h, x, step, cache.lines[0], None, True)
        if pending is not None:
            settle(x, pending)
        got.append(x)
    rt.check()
    a, b = got
    # two chains of bfloat16 roundings (queries and outputs carried through the latents, or not)
    assert (a - b).norm() <= 2e-2 * b.norm()
