"""The general attention's two forms against float64: tiles of 64 new tokens, and clusters that
share out one token's keys, at the edges of tiles, pages and windows, with every option."""
import math

import numpy as np
import pytest
import torch

from mormot2_ai_b200 import kernels as K
from tests.gpu_helpers import DEV, fill_line, make_line, make_step

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def reference(q, k, v, pos, window, keep, scale, sink, cap, slopes, gate):
    """One token in float64: q [nh, hd], k and v [n, nkv, .], gate [nh, 1 or vd]."""
    nh, nkv = q.shape[0], k.shape[1]
    at = np.arange(pos + 1)
    at = at[(at > pos - window) | (at < keep)] if window else at
    out = []
    for h in range(nh):
        s = k[at, h // (nh // nkv)] @ q[h] * scale
        if cap:
            s = cap * np.tanh(s / cap)
        s = s - slopes[h] * (pos - at)
        m = max(s.max(), sink[h])
        p = np.exp(s - m)
        out.append(p @ v[at, h // (nh // nkv)] / (p.sum() + np.exp(sink[h] - m))
                   / (1 + np.exp(-gate[h])))
    return np.stack(out)


# (new tokens, positions held): 15 | 16 is where the form changes, 64 and 65 the tile's edges
STEPS = [[(1, 0), (1, 63), (1, 700)], [(15, 50), (3, 0)], [(16, 0), (1, 130), (65, 64)], [(129, 300)],
         [(2, 700), (20, 3), (15, 64), (1, 0), (16, 1)]]      # each sequence by its own tokens
SIZES = [(4, 2, 128, 128), (8, 1, 64, 64), (5, 5, 20, 12), (12, 2, 100, 128), (2, 1, 256, 196)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("nh, nkv, hd, vd", SIZES)
@pytest.mark.parametrize("seqs", STEPS)
@pytest.mark.parametrize("options", ["plain", "window", "kept", "gates"])
def test_forms_of_the_general_attention(dtype, nh, nkv, hd, vd, seqs, options):
    rng = np.random.default_rng(hd + len(seqs))
    dt = DT[dtype]
    window, keep = {"plain": (0, 0), "window": (70, 0), "kept": (70, 9), "gates": (0, 0)}[options]
    full = options in ("kept", "gates")
    sink = rng.standard_normal(nh) if full else np.full(nh, -np.inf)
    slopes = 2.0 ** -np.arange(3, nh + 3) if full else np.zeros(nh)
    cap = 3.0 if full else 0.0
    T = sum(n for n, _ in seqs)
    line = make_line(len(seqs), max(n + p for n, p in seqs), nkv, hd, dt, window=window, seed=hd)
    line.v = torch.zeros(line.v.shape[:3] + (vd,), dtype=dt, device=DEV)
    held = []
    for slot, (n, past) in enumerate(seqs):
        k = torch.tensor(rng.standard_normal((n + past, nkv, hd))).to(dt)
        v = torch.tensor(rng.standard_normal((n + past, nkv, vd))).to(dt)
        fill_line(line, slot, k.float(), v.float())
        held.append((k.double().numpy(), v.double().numpy()))
    q = torch.tensor(rng.standard_normal((T, nh * hd))).to(dt)
    per = vd if options == "gates" else 1
    gate = torch.tensor(rng.standard_normal((T, nh * per))).to(dt)
    step = make_step([(slot, past, [0] * n, []) for slot, (n, past) in enumerate(seqs)])
    out = torch.full((T, nh * vd), float("nan"), dtype=dt, device=DEV)
    f32 = lambda a: torch.tensor(a, dtype=torch.float32, device=DEV)
    K.attention_simt(q.to(DEV), nh * hd, out, step, line, nh, nkv, hd, window, hd ** -0.5, vd=vd,
                     sink=f32(sink) if full else None, softcap=cap,
                     gate=gate.to(DEV) if full else None, gate_stride=nh * per,
                     slopes=f32(slopes) if full else None, keep_first=keep,
                     gate_dim=per if options == "gates" else 0)
    got, row = out.double().cpu().numpy().reshape(T, nh, vd), 0
    for (n, past), (k, v) in zip(seqs, held):
        for pos in range(past, past + n):
            g = gate[row].double().numpy().reshape(nh, per) if full else np.full((nh, 1), np.inf)
            want = reference(q[row].double().numpy().reshape(nh, hd), k, v, pos, window, keep,
                             hd ** -0.5, sink.astype(np.float32).astype(np.float64), cap,
                             slopes, g)
            # float32: sums of up to 700 terms and the exponentials' last places; bfloat16: the
            # result's rounding, 2^-9
            tol = 4e-6 if dtype == "float32" else 5e-3
            assert np.linalg.norm(got[row] - want) <= tol * np.linalg.norm(want), (pos, row)
            row += 1


@pytest.mark.parametrize("n", [8, 40])
def test_an_infinite_value_reaches_only_the_tokens_that_see_it(n):
    nh, nkv, hd, bad = 2, 1, 64, 5
    rng = np.random.default_rng(0)
    line = make_line(1, n, nkv, hd, torch.float32)
    k, v = (torch.tensor(rng.standard_normal((n, nkv, hd)), dtype=torch.float32) for _ in range(2))
    v[bad, 0, 3] = math.inf
    fill_line(line, 0, k, v)
    step = make_step([(0, 0, [0] * n, [])])
    q = torch.tensor(rng.standard_normal((n, nh * hd)), dtype=torch.float32).to(DEV)
    out = torch.empty((n, nh * hd), dtype=torch.float32, device=DEV)
    K.attention_simt(q, nh * hd, out, step, line, nh, nkv, hd, 0, 0.125)
    got = out.cpu().reshape(n, nh, hd)
    assert torch.isfinite(got[:bad]).all()
    assert torch.isinf(got[bad:, :, 3]).all()
    got[bad:, :, 3] = 0
    assert torch.isfinite(got).all()


# more CTAs than run at once: they take the sequences by length, equal lengths among them
@pytest.mark.parametrize("count, splits", [(50, 1), (38, 1), (160, 1), (161, 1), (20, 2)])
def test_decode_takes_sequences_by_length(count, splits):
    nh, nkv, hd = 16, 8, 64
    rng = np.random.default_rng(count)
    lens = [int(n) for n in rng.choice([1, 2, 63, 64, 65, 130, 200], count)]
    line = make_line(count, 256, nkv, hd, torch.bfloat16, seed=count)
    line.k.copy_(torch.tensor(rng.standard_normal(line.k.shape)))
    line.v.copy_(torch.tensor(rng.standard_normal(line.v.shape)))
    step = make_step([(i, n - 1, [0], []) for i, n in enumerate(lens)], max_seqs=count)
    q = torch.tensor(rng.standard_normal((count, nh * hd))).to(torch.bfloat16).to(DEV)
    got, want = torch.empty_like(q), torch.empty((count, nh * hd), device=DEV)
    error = torch.zeros(1, dtype=torch.int32, device=DEV)
    K.attention_decode_clusters(q, nh * hd, got, step, line, nh, nkv, hd, 0, 0.125, splits, error)
    assert int(error.item()) == 0
    line32 = type(line)(line.k.float(), line.v.float(), line.page_table, line.max_pages, 0, 0, nkv, hd)
    K.attention_simt(q.float(), nh * hd, want, step, line32, nh, nkv, hd, 0, 0.125)
    # probabilities and outputs rounded to bfloat16, 2^-9 each
    assert ((got.float() - want).norm(dim=1) <= 1e-2 * want.norm(dim=1)).all()


# the keys of a whole tile of one warp overflow to -infinity: they weigh nothing, with a sink or none
@pytest.mark.parametrize("new", [1, 40])
@pytest.mark.parametrize("first, count", [(0, 16), (16, 16), (32, 64), (0, 127)])
@pytest.mark.parametrize("sink", [None, 0.5])
def test_scores_of_minus_infinity(new, first, count, sink):
    nh, nkv, hd, n = 2, 1, 64, 128
    rng = np.random.default_rng(first)
    line = make_line(1, n, nkv, hd, torch.float32)
    k, v = (torch.tensor(rng.standard_normal((n, nkv, hd)), dtype=torch.float32) for _ in range(2))
    q = torch.tensor(rng.standard_normal((new, nh * hd)), dtype=torch.float32)
    k[:, 0, 0], q[:, 0::hd] = 0.0, 1e20
    k[first:first + count, 0, 0] = -1e20
    fill_line(line, 0, k, v)
    sinks = None if sink is None else torch.full((nh,), sink, device=DEV)
    step = make_step([(0, n - new, [0] * new, [])])
    out = torch.empty((new, nh * hd), device=DEV)
    K.attention_simt(q.to(DEV), nh * hd, out, step, line, nh, nkv, hd, 0, 0.125, sink=sinks)
    ok = [i for i in range(n) if not first <= i < first + count]
    for row, pos in enumerate(range(n - new, n)):
        at = [i for i in ok if i <= pos]
        qd, kd, vd = q[row].view(nh, hd).double(), k[at, 0].double(), v[at, 0].double()
        s = qd @ kd.t() * 0.125
        if sinks is not None:
            s = torch.cat([s, torch.full((nh, 1), sink, dtype=torch.float64)], 1)
            vd = torch.cat([vd, torch.zeros((1, hd), dtype=torch.float64)])
        got = out[row].view(nh, hd).double().cpu()
        if s.shape[1] == 0:                 # nothing to weigh: 0 / 0
            assert torch.isnan(got).all()
            continue
        want = torch.softmax(s, 1) @ vd
        # float32 sums of at most 128 terms; the product with 1e20 leaves q·k of the others whole
        assert (got - want).norm() <= 4e-6 * want.norm() + 1e-12
