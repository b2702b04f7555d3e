"""The recurrences four tokens at a time against the same walked token by token: outputs and the
state that a step leaves, from a state that is not zero, at the edges of groups and chunks."""
import pytest
import torch

from mormot2_ai_b200 import kernels as K
from tests.gpu_helpers import DEV, make_step

pytestmark = pytest.mark.gpu


def rows(shape, seed, std=1.0, mean=0.0):
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=gen) * std + mean).to(DEV)


def run(mode, step, state, T, heads, dim, vdim, group, shift, dtype):
    out = torch.empty((T, heads * vdim), dtype=dtype, device=DEV)
    qkw, vw = heads // group * dim, heads * vdim
    z = rows((T, shift + 2 * qkw + 2 * vw + 2 * heads), 1)
    z[:, shift:shift + 2 * qkw] *= dim ** -0.25
    cols = [shift, shift + qkw, shift + 2 * qkw, shift + 2 * qkw + vw,
            shift + 2 * qkw + 2 * vw, shift + 2 * qkw + 2 * vw + heads]
    if mode == "mlstm":
        K.mlstm_scan(z, cols, rows((heads,), 2), rows((heads,), 3, mean=4.0), 15.0, dim ** -0.5,
                     rows((vw,), 4, 0.1, 1.0), 1e-6, state, step, out, heads, dim, vdim)
    elif mode == "wkv":
        r, k, v, g = (z[:, c:c + vw] for c in cols[:4])
        h = rows((T, 24), 5).to(dtype)
        lw = z.new_zeros(z.shape)[:, :vw]
        lw.copy_(rows((T, vw), 6))
        K.wkv_scan(r, k, v, lw, g, rows((vw,), 7, mean=-2.0), rows((vw,), 8), rows((vw,), 4, 0.1, 1.0),
                   1e-6, state, h, step, out, heads, dim)
    else:
        more = (dict(decay_logits=rows((T, heads * dim + 3), 6), decay_col=3,
                     decay_bias=rows((heads * dim,), 7), inv_tau=1 / 16) if mode == "gla" else
                dict(scalars=z, beta_col=cols[4], rate_col=cols[5], a_log=rows((heads,), 2),
                     dt_bias=rows((heads,), 3, mean=-2.0), unit_eps=1e-6))
        K.linear_state_scan(mode, z, cols[:3], group, z, cols[3], rows((vdim,), 4, 0.1, 1.0), 1e-6,
                            state, step, out, heads, dim, vdim, **more)
    return out


# 16 and 17 new tokens: a whole chunk and one more; 1 to 3: a group that is not full
LENGTHS = [[16], [17, 1, 2], [3, 50, 33, 64]]


@pytest.mark.parametrize("mode", ["gla", "delta", "mlstm", "wkv"])
@pytest.mark.parametrize("heads, dim, vdim, group", [(2, 20, 24, 1), (4, 64, 128, 2), (2, 128, 36, 1),
                                                     (1, 200, 72, 1), (40, 64, 64, 1)])
@pytest.mark.parametrize("lens", LENGTHS)
@pytest.mark.parametrize("shift", [0, 1])          # 1: rows that no 16-byte copy can take
def test_four_tokens_at_a_time(monkeypatch, mode, heads, dim, vdim, group, lens, shift):
    if mode in ("mlstm", "wkv"):
        group = 1
    if mode == "wkv":
        vdim = dim
    step = make_step([(i + 1, 5, [0] * n, []) for i, n in enumerate(lens)])
    size = {"mlstm": heads * (dim * vdim + dim + 1), "wkv": 24 + heads * dim * dim}.get(
        mode, heads * dim * vdim)
    start = rows((len(lens) + 2, size + 3), 9, 0.3)
    got = []
    for fours in (False, True):
        monkeypatch.setattr(K, "walks_by_fours", lambda *a: fours)
        state = start.clone()
        out = run(mode, step, state, sum(lens), heads, dim, vdim, group, shift, torch.float32)
        got.append((out, state))
    (want, state), (out, state4) = got
    # float32 sums over the head and the tokens in another order, divided by a root mean square
    assert (out - want).norm() <= 2e-5 * want.norm()
    assert (state4 - state).norm() <= 2e-6 * state.norm()
    assert torch.equal(state4[0], start[0]) and torch.equal(state4[-1], start[-1])
    assert torch.equal(state4[:, size:], start[:, size:])


def test_which_steps_go_by_fours():
    long, short = make_step([(0, 0, [0] * 16, [])]), make_step([(0, 0, [0] * 15, [])])
    assert K.walks_by_fours(long, 256)
    assert not K.walks_by_fours(long, 257) and not K.walks_by_fours(short, 64)


# four taps go four channels a thread in runs of 16 tokens, unless rows or channels do not allow it
@pytest.mark.parametrize("taps, channels, shift", [(4, 40, 0), (4, 520, 4), (4, 42, 0), (4, 40, 1),
                                                   (3, 40, 0)])
@pytest.mark.parametrize("lens", [[1], [2, 1, 3], [15, 18], [1, 40, 16, 5]])
def test_short_convolution(taps, channels, shift, lens):
    T = sum(lens)
    z = rows((T, channels + 8), 1)
    w = rows((channels, taps), 2)
    size = (taps - 1) * channels
    states = rows((len(lens) + 1, 8 + size), 3)
    step = make_step([(i + 1, 9, [0] * n, []) for i, n in enumerate(lens)])
    before = states.clone()
    out = torch.empty((T, channels), device=DEV)
    K.short_conv(z, shift, w, states[:, 8:], step, out)
    at = 0
    for i, n in enumerate(lens):
        past = before[i + 1, 8:].double().view(taps - 1, channels)
        x = torch.cat([past, z[at:at + n, shift:shift + channels].double()])
        want = torch.nn.functional.silu(sum(x[j:j + n] * w[:, j].double() for j in range(taps)))
        # four products and a sigmoid in float32
        assert (out[at:at + n].double() - want).abs().max() <= 1e-5
        assert torch.equal(states[i + 1, 8:].view(taps - 1, channels), x[n:].float())
        at += n


@pytest.mark.parametrize("mode", ["gla", "delta", "mlstm", "wkv"])
@pytest.mark.parametrize("bad", [1, 7, 18])
def test_an_infinity_does_not_reach_earlier_tokens(mode, bad):
    T, heads, dim = 20, 2, 64
    step = make_step([(0, 0, [0] * T, [])])
    size = {"mlstm": heads * (dim * dim + dim + 1), "wkv": 24 + heads * dim * dim}.get(
        mode, heads * dim * dim)
    args = (T, heads, dim, dim, 1, 0, torch.float32)
    clean = run(mode, step, torch.zeros((1, size), device=DEV), *args)
    real = globals()["rows"]
    try:
        def spoiled(shape, seed, *a, **k):
            t = real(shape, seed, *a, **k)
            if seed == 1:                 # a value of the token, in the second head
                t[bad, 2 * heads * dim + dim + 3] = float("inf")
            return t
        globals()["rows"] = spoiled
        out = run(mode, step, torch.zeros((1, size), device=DEV), *args)
    finally:
        globals()["rows"] = real
    assert torch.equal(out[:bad], clean[:bad])
    assert torch.equal(out[:, :dim], clean[:, :dim])
    assert not torch.isfinite(out[bad, dim:]).all()


# groups that a sequence does not fill, and no floor under the length that keys are divided by
@pytest.mark.parametrize("lens", [[17], [3, 50], [18, 1, 2], [16, 35]])
@pytest.mark.parametrize("group", [1, 2])
def test_delta_without_a_floor_under_the_keys_length(monkeypatch, lens, group):
    T, heads, dim, vdim = sum(lens), 4, 64, 32
    qkw, vw = heads // group * dim, heads * vdim
    z = rows((T, 2 * qkw + 2 * vw + 2 * heads), 1)
    step = make_step([(i, 5, [0] * n, []) for i, n in enumerate(lens)])
    start = rows((len(lens), heads * dim * vdim), 2, 0.3)
    got = []
    for fours in (False, True):
        monkeypatch.setattr(K, "walks_by_fours", lambda *a: fours)
        out, state = torch.empty((T, vw), device=DEV), start.clone()
        K.linear_state_scan("delta", z, [0, qkw, 2 * qkw], group, z, 2 * qkw + vw,
                            rows((vdim,), 4, 0.1, 1.0), 1e-6, state, step, out, heads, dim, vdim,
                            scalars=z, beta_col=2 * qkw + 2 * vw, rate_col=2 * qkw + 2 * vw + heads,
                            a_log=rows((heads,), 5), dt_bias=rows((heads,), 6, mean=-2.0))
        got.append((out, state))
    (want, state), (out, state4) = got
    # as above: float32 sums in another order
    assert (out - want).norm() <= 2e-5 * want.norm()
    assert (state4 - state).norm() <= 2e-6 * state.norm()


def plain(mode, start, lens, heads, dim, vdim, group, T):
    """``run`` token after token in float64: outputs [T, heads * vdim] and the sequences' states,
    without wkv's input row."""
    qkw, vw = heads // group * dim, heads * vdim
    z = rows((T, 2 * qkw + 2 * vw + 2 * heads), 1)
    z[:, :2 * qkw] *= dim ** -0.25
    z = z.double().cpu()
    f = lambda *a: rows(*a).double().cpu()
    head = lambda c, n, per: z[:, c:c + n].reshape(T, -1, per).repeat_interleave(heads * per // n, 1)
    q, k = head(0, qkw, dim), head(qkw, qkw, dim)
    v, gate = head(2 * qkw, vw, vdim), head(2 * qkw + vw, vw, vdim)
    s0, s1 = z[:, 2 * qkw + 2 * vw:].reshape(T, 2, heads).unbind(1)
    w0, w1 = f((heads,), 2), f((heads,), 3, 1.0, 4.0 if mode == "mlstm" else -2.0)
    if mode == "gla":
        a = torch.sigmoid(f((T, heads * dim + 3), 6)[:, 3:] + f((heads * dim,), 7)) ** (1 / 16)
        q = q * dim ** -0.5
    elif mode == "wkv":
        a = torch.exp(-torch.exp(f((T, vw), 6) + f((vw,), 7, 1.0, -2.0)))
        u = f((vw,), 8).view(heads, dim, 1)
    elif mode == "delta":
        q = q / (q.square().sum(-1, keepdim=True) + 1e-6).sqrt() * dim ** -0.5
        k = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
        a = torch.exp(-torch.exp(w0) * torch.nn.functional.softplus(s1 + w1))
        beta = torch.sigmoid(s0)
    else:
        q = q * dim ** -0.5
        gi = 15 * torch.tanh((s0 + w0) / 15)
        gf = torch.nn.functional.logsigmoid(15 * torch.tanh((s1 + w1) / 15))
    out, states, t = torch.empty((T, heads, vdim), dtype=torch.float64), [], 0
    for b, n in enumerate(lens):
        S = start[b].double().cpu()
        if mode == "mlstm":
            S = S[:heads * (dim * vdim + dim + 1)].view(heads, -1)
            S, nrm, m = S[:, :dim * vdim].view(heads, dim, vdim), S[:, -dim - 1:-1], S[:, -1]
        else:
            S = S[24 if mode == "wkv" else 0:][:heads * dim * vdim].view(heads, dim, vdim)
        for t in range(t, t + n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            if mode == "mlstm":
                top = torch.maximum(gf[t] + m, gi[t])
                keep, new, m = torch.exp(gf[t] + m - top), torch.exp(gi[t] - top), top
                S = keep[:, None, None] * S + new[:, None, None] * kv
                nrm = keep[:, None] * nrm + new[:, None] * k[t]
                den = torch.maximum((nrm * q[t]).sum(1).abs(), torch.exp(-m)) + 1e-6
                o = torch.einsum("hdv,hd->hv", S, q[t]) / den[:, None]
            elif mode == "wkv":
                o = torch.einsum("hdv,hd->hv", S + u * kv, q[t])
                S = a[t].view(heads, dim, 1) * S + kv
            elif mode == "gla":
                S = a[t].view(heads, dim, 1) * S + kv
                o = torch.einsum("hdv,hd->hv", S, q[t])
            else:
                S = a[t].view(heads, 1, 1) * S
                new = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
                S = S + k[t][:, :, None] * new[:, None, :]
                o = torch.einsum("hdv,hd->hv", S, q[t])
            out[t] = o / (o.square().mean(1, keepdim=True) + 1e-6).sqrt()
        t += 1
        states.append(torch.cat([S.reshape(heads, -1), nrm, m[:, None]], 1).view(-1)
                      if mode == "mlstm" else S.reshape(-1))
    per_head = mode in ("mlstm", "wkv")
    normw = f((vw if per_head else vdim,), 4, 0.1, 1.0).view(-1, vdim)
    gate = torch.sigmoid(gate) * (1 if mode == "mlstm" else gate)
    return (out * normw * gate).view(T, -1), torch.stack(states)


# from states that are not zero; the last lengths leave a group with one, two and three tokens
@pytest.mark.parametrize("mode", ["gla", "delta", "mlstm", "wkv"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("fours", [True, False])
@pytest.mark.parametrize("dim, vdim", [(64, 64), (36, 20)])
def test_recurrences_in_float64(monkeypatch, mode, dtype, fours, dim, vdim):
    lens, heads, group = [40, 17, 1, 22, 3], 4, 1 if mode in ("mlstm", "wkv") else 2
    vdim = dim if mode == "wkv" else vdim
    T = sum(lens)
    size = {"mlstm": heads * (dim * vdim + dim + 1), "wkv": 24 + heads * dim * dim}.get(
        mode, heads * dim * vdim)
    start = rows((len(lens), size), 9, 0.3)
    want, states = plain(mode, start, lens, heads, dim, vdim, group, T)
    monkeypatch.setattr(K, "walks_by_fours", lambda *a: fours)
    state, step = start.clone(), make_step([(i, 5, [0] * n, []) for i, n in enumerate(lens)])
    out = run(mode, step, state, T, heads, dim, vdim, group, 0, dtype).double().cpu()
    # float32 sums over the head, the tokens and the root mean square; bfloat16: the stored
    # output's rounding, 2^-9 of every value
    tol = 2e-5 if dtype == torch.float32 else 2.0 ** -8
    assert (out - want).norm() <= tol * want.norm()
    got = state.double().cpu()[:, 24 if mode == "wkv" else 0:]
    assert (got - states).norm() <= 1e-6 * states.norm() + (0 if mode != "mlstm" else 1e-6)
    if mode == "wkv":      # the last input row of every sequence, as it came
        last = rows((T, 24), 5).to(dtype).float()[torch.tensor(lens).cumsum(0) - 1]
        assert torch.equal(state[:, :24], last)


# GLA and the delta rule, the matrix memory, the decaying state: steps on both sides of the rule's edges
@pytest.mark.parametrize("lens, by", [
    ([16], (True, False, False)), ([47], (True, False, False)), ([48], (True, True, False)),
    ([96], (True, True, True)), ([16] * 8, (True, False, False)), ([79] * 8, (True, False, False)),
    ([96] * 8, (True, True, True)), ([48] * 16, (True, False, True)),
    ([47, 48], (True, True, False)), ([47] * 4, (True, False, False)),
    ([16] + [1] * 15, (False, False, False)), ([32] + [1] * 15, (True, False, False)),
    ([80] + [1] * 15, (True, True, True)), ([96] + [1] * 15, (True, True, True)),
    ([128] + [1] * 63, (True, True, False)), ([256] + [1] * 63, (True, True, True)),
    ([127] + [1] * 63, (False, False, False))])
def test_rule_of_the_walk(lens, by):
    step = make_step([(i, 0, [0] * n, []) for i, n in enumerate(lens)])
    modes = (K.WALK_GLA, K.WALK_MLSTM, K.WALK_WKV)
    assert tuple(K.walks_by_fours(step, 64, m, 8) for m in modes) == by
    assert K.walks_by_fours(step, 64, K.WALK_DELTA, 8) == by[0]
    assert not any(K.walks_by_fours(step, 257, m, 8) for m in modes)


# a block a token and runs of 16 tokens, whichever the step's size takes, give the same values
@pytest.mark.parametrize("lens", [[600], [300, 1, 2, 270], [1] * 20 + [1100]])
def test_convolutions_values_do_not_depend_on_the_steps_size(lens):
    channels, T = 2048, sum(lens)
    z, w = rows((T, channels), 1), rows((channels, 4), 2)
    states = rows((len(lens), 3 * channels), 3)
    after = states.clone()
    out, alone = torch.empty((T, channels), device=DEV), torch.empty((T, channels), device=DEV)
    K.short_conv(z, 0, w, after, make_step([(i, 9, [0] * n, []) for i, n in enumerate(lens)]), out)
    at = 0
    for i, n in enumerate(lens):          # parts of at most 64 tokens: far below a run's work
        for a in range(at, at + n, 64):
            m = min(64, at + n - a)
            K.short_conv(z[a:a + m], 0, w, states, make_step([(i, 9, [0] * m, [])]), alone[a:a + m])
        at += n
    assert torch.equal(out, alone) and torch.equal(after, states)
