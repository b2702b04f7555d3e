"""Lists of the experts' rows and the sum of a token's experts at their edges: more experts than the
list's block has threads, experts without rows, columns that are no multiple of four."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("A, E, bm", [(1, 1, 8), (48, 64, 8), (300, 7, 128), (5000, 1025, 16),
                                      (900, 4096, 64)])
def test_lists(A, E, bm):
    ids = torch.randint(0, max(1, E // 2), (A,), generator=torch.Generator().manual_seed(A)) * 2 % E
    ids = ids.to(torch.int32)
    tiles_most = (A + bm - 1) // bm + E
    plan = torch.full((2 + E + A + 2 * tiles_most,), -7, dtype=torch.int32, device=DEV)
    K.moe_plan(ids.to(DEV).view(A, 1), E, bm, tiles_most, plan)
    got = plan.cpu().tolist()
    count = torch.bincount(ids.long(), minlength=E).tolist()
    offsets, tiles, at = [], [], 0
    for e in range(E):
        offsets.append(at)
        tiles += [(e, at + r) for r in range(0, count[e], bm)]
        at += count[e]
    assert got[1:2 + E] == offsets + [A] and got[0] == len(tiles)
    perm = got[2 + E:2 + E + A]
    for e in range(E):
        rows = sorted(perm[offsets[e]:offsets[e] + count[e]])
        assert rows == (ids == e).nonzero().view(-1).tolist()
    t0 = 2 + E + A
    assert list(zip(got[t0:t0 + len(tiles)],
                    got[t0 + tiles_most:t0 + tiles_most + len(tiles)])) == tiles


@pytest.mark.parametrize("T, H, top, parts", [(1, 8, 1, 1), (8, 2048, 6, 8), (5, 516, 5, 3), (3, 130, 2, 2)])
@pytest.mark.parametrize("store, identity", [(False, False), (True, False), (False, True)])
def test_sum_of_a_tokens_experts(T, H, top, parts, store, identity):
    gen = torch.Generator().manual_seed(H)
    r = lambda *s: torch.randn(s, generator=gen).to(DEV)
    x, y, shared, sg, w, h = r(T, H), r(T * top, H), r(parts, T, H), r(T), r(T, top), r(T, H)
    ids = torch.randint(0, 6, (T, top), generator=gen).to(torch.int32).to(DEV)
    terms = y.view(T, top, H).double()
    if identity:
        terms = torch.where((ids >= 4)[..., None], w.double()[..., None] * h.double()[:, None], terms)
    want = terms.sum(1) + sg.double()[:, None] * shared.double().sum(0)
    want = want if store else x.double() + want
    if identity:
        K.moe_combine(x, y, top, shared, sg, ids, w, 4, h, store=store)
    else:
        K.moe_combine(x, y, top, shared, sg, store=store)
    # float32 sums of at most 15 terms of the size of one
    assert (x.double() - want).abs().max() <= 1e-5
