"""The general attention of many new float32 tokens on the tensor cores (heads of 128 values): against
float64 with every option, against the float32 kernel where something is no number."""
import numpy as np
import pytest
import torch

from mormot2_ai_b200 import kernels as K
from tests import test_attention_plans_gpu as plans
from tests.gpu_helpers import DEV, fill_line, make_line, make_step

pytestmark = pytest.mark.gpu


# tiles of 128 tokens, pages of 64 keys: a whole tile, one token less and more, positions held that end
# inside a page; sequences of few tokens and of none that go in tiles beside them
@pytest.mark.parametrize("nh, nkv", [(4, 2), (3, 3)])
@pytest.mark.parametrize("seqs", [[(64, 0)], [(127, 1)], [(128, 64)], [(129, 700)], [(257, 63), (2, 9), (64, 130), (20, 0)]])
@pytest.mark.parametrize("options", ["plain", "window", "kept", "gates"])
def test_forms(nh, nkv, seqs, options, monkeypatch):
    monkeypatch.setattr(K, "ATTENTION_SPLIT", 0)
    error, inner = torch.zeros(1, dtype=torch.int32, device=DEV), K.attention_simt
    monkeypatch.setattr(K, "attention_simt", lambda *a, **k: inner(*a, **k, error=error))
    plans.test_forms_of_the_general_attention("float32", nh, nkv, 128, 128, seqs, options)
    assert int(error) == 0


def run(k, v, q, past, split, monkeypatch, nh=2, nkv=1, **options):
    monkeypatch.setattr(K, "ATTENTION_SPLIT", 0 if split else 1 << 30)
    n = q.shape[0]
    line = make_line(1, n + past, nkv, 128, torch.float32)
    fill_line(line, 0, k, v)
    out = torch.full((n, nh * 128), -7.0, device=DEV)
    error = torch.zeros(1, dtype=torch.int32, device=DEV)
    K.attention_simt(q.to(DEV), nh * 128, out, make_step([(0, past, [0] * n, [])]), line, nh, nkv, 128, 0, 128 ** -0.5,
                     error=error, **options)
    assert int(error) == 0
    return out


def draw(n, past, seed, nh=2, nkv=1):
    rng = np.random.default_rng(seed)
    f = lambda *s: torch.tensor(rng.standard_normal(s), dtype=torch.float32)
    return f(n + past, nkv, 128), f(n + past, nkv, 128), f(n, nh * 128)


# what is no number takes the tile through the float32 kernel: the same bits there, and nothing elsewhere
@pytest.mark.parametrize("where", ["q", "k", "v", "overflow", "no_key"])
def test_what_is_no_number(where, monkeypatch):
    n, past = 300, 20
    k, v, q = draw(n, past, 3)
    options = {}
    if where == "q":
        q[150, 3] = float("inf")
    elif where == "k":
        k[200, 0, 7] = float("nan")
    elif where == "v":
        v[200, 0, 7] = float("-inf")
    elif where == "overflow":
        q[140, 5], k[:, 0, 5] = 1e30, 1e30
    else:
        options["slopes"] = torch.tensor([0.0, float("inf")], device=DEV)      # inf * 0 = NaN on the diagonal
    want = run(k, v, q, past, False, monkeypatch, **options)
    got = run(k, v, q, past, True, monkeypatch, **options)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fine = want.isfinite()
    assert (got[fine] - want[fine]).abs().max() <= 1e-5 if fine.any() else True


# the error against float64 is at most a fifth above that of the float32 kernel's multiply-adds (measured:
# below it; single inputs vary)
@pytest.mark.parametrize("n, past", [(128, 0), (200, 1500)])
def test_error(n, past, monkeypatch):
    k, v, q = draw(n, past, 4, 4, 2)
    kd, vd = k.double().repeat_interleave(2, 1), v.double().repeat_interleave(2, 1)
    qd = q.double().view(n, 4, 128)
    s = torch.einsum("thd,khd->htk", qd, kd) * 128 ** -0.5
    s.masked_fill_(torch.arange(n + past)[None] > torch.arange(past, n + past)[:, None], -torch.inf)
    want = torch.einsum("htk,khd->thd", s.softmax(-1), vd).reshape(n, -1)
    errors = [((run(k, v, q, past, split, monkeypatch, 4, 2).double().cpu() - want).norm() / want.norm()).item()
              for split in (False, True)]
    assert errors[1] <= 1.2 * errors[0] and errors[1] <= 1e-6, errors


# queries, keys or values below 2^-110 may be no exact sums of three parts: their tiles go through the
# float32 kernel, the same bits
@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_small_values(where, monkeypatch):
    n, past = 300, 20
    k, v, q = draw(n, past, 5)
    if where == "q":
        q[130] *= 2.0 ** -118
        q[130, 128:] = 0.0      # the second head: zeros are cut exactly
    else:
        (k if where == "k" else v)[:, 0, 3] *= 2.0 ** -118
    want, got = (run(k, v, q, past, split, monkeypatch) for split in (False, True))
    if where == "q":
        assert torch.equal(got[128:256, :128], want[128:256, :128])
        assert not torch.equal(got[128:256, 128:], want[128:256, 128:])
    else:
        assert torch.equal(got, want)
