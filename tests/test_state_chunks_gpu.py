"""The delta rule and the matrix memory in chunks of 32 tokens: outputs and states against float64 and
against the same four tokens at a time, in one pass and in several, and what is no number."""
from types import SimpleNamespace

import pytest
import torch

from mormot2_ai_b200 import kernels as K
from tests import test_state_walk_gpu as walk
from tests.gpu_helpers import DEV, make_step

pytestmark = pytest.mark.gpu


def size_of(mode, heads, dim, vdim):
    return heads * (dim * vdim + (dim + 1 if mode == "mlstm" else 0))


def route(monkeypatch, chunks, scratch=None):
    monkeypatch.setattr(K, "walks_by_fours", lambda *a: True)
    monkeypatch.setattr(K, "walks_in_chunks", lambda *a: chunks)
    if scratch is not None:
        monkeypatch.setattr(K, "CHUNK_SCRATCH", scratch)


# from states that are not zero; whole chunks, one token more and less, sequences of one token;
# scratch of 1: a chunk of every sequence a pass
@pytest.mark.parametrize("mode", ["delta", "mlstm"])
@pytest.mark.parametrize("heads, dim, vdim, group", [(4, 64, 64, 2), (2, 128, 128, 1), (2, 16, 48, 1), (3, 80, 16, 3)])
@pytest.mark.parametrize("scratch", [None, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_chunks_in_float64(monkeypatch, mode, heads, dim, vdim, group, scratch, dtype):
    lens = [64, 33, 1, 95, 32]
    group, T = 1 if mode == "mlstm" else group, sum(lens)
    start = walk.rows((len(lens), size_of(mode, heads, dim, vdim)), 9, 0.3)
    want, states = walk.plain(mode, start, lens, heads, dim, vdim, group, T)
    route(monkeypatch, True, scratch)
    state, step = start.clone(), make_step([(i, 5, [0] * n, []) for i, n in enumerate(lens)])
    out = walk.run(mode, step, state, T, heads, dim, vdim, group, 0, dtype).double().cpu()
    # the bounds of the walk by fours: float32 sums, and the rounding of a stored bfloat16
    tol = 2e-5 if dtype == torch.float32 else 2.0 ** -8
    assert (out - want).norm() <= tol * want.norm()
    assert (state.double().cpu() - states).norm() <= 1e-6 * states.norm() + (0 if mode != "mlstm" else 1e-6)


@pytest.mark.parametrize("mode", ["delta", "mlstm"])
def test_long_sequences_as_by_fours(monkeypatch, mode):
    lens, heads, dim, vdim = [700, 1, 129], 4, 128, 64
    T, group = sum(lens), 1 if mode == "mlstm" else 2
    start = walk.rows((5, size_of(mode, heads, dim, vdim) + 3), 9, 0.3)
    got = []
    for chunks in (False, True):
        route(monkeypatch, chunks)
        state, step = start.clone(), make_step([(i + 1, 5, [0] * n, []) for i, n in enumerate(lens)])
        got.append((walk.run(mode, step, state, T, heads, dim, vdim, group, 0, torch.float32), state))
    (want, state), (out, state32) = got
    assert (out - want).norm() <= 2e-5 * want.norm()
    assert (state32 - state).norm() <= 4e-6 * state.norm()
    assert torch.equal(state32[0], start[0]) and torch.equal(state32[4], start[4])


# Sums that lean to one side add up over the chunks: the delta rule's states and outputs are as near to
# float64 as by fours, in the mean over three inputs (a tenth more: what the mean of three can vary by)
def test_as_near_to_float64_as_by_fours(monkeypatch):
    heads, dim, lens, real = 2, 128, [2000], walk.rows
    errors = {False: [0.0, 0.0], True: [0.0, 0.0]}
    for more in (0, 100, 200):
        monkeypatch.setattr(walk, "rows", lambda shape, seed, *a, **k: real(shape, seed + more, *a, **k))
        start = walk.rows((1, heads * dim * dim), 9, 0.3)
        want, states = walk.plain("delta", start, lens, heads, dim, dim, 1, lens[0])
        for chunks in (False, True):
            route(monkeypatch, chunks)
            state, step = start.clone(), make_step([(0, 5, [0] * lens[0], [])])
            out = walk.run("delta", step, state, lens[0], heads, dim, dim, 1, 0, torch.float32)
            for i, (got, ref) in enumerate(((out, want), (state, states))):
                errors[chunks][i] += float((got.double().cpu() - ref).norm() / ref.norm())
    assert errors[True][0] <= 1.1 * errors[False][0] and errors[True][1] <= 1.1 * errors[False][1]


# an infinity among the values or the keys of a token, or in the state
@pytest.mark.parametrize("mode", ["delta", "mlstm"])
@pytest.mark.parametrize("what", ["value", "key", "state"])
@pytest.mark.parametrize("bad", [1, 31, 40])
def test_an_infinity_reaches_what_it_reaches_by_fours(monkeypatch, mode, what, bad):
    T, heads, dim = 70, 2, 64
    step = make_step([(0, 0, [0] * T, [])])
    column = {"value": 2 * heads * dim, "key": heads * dim, "state": 0}[what] + dim + 3
    real, outs = walk.rows, {}

    def spoiled(shape, seed, *a, **k):
        t = real(shape, seed, *a, **k)
        if seed == 1 and what != "state":
            t[bad, column] = float("inf")
        return t
    for name, rows, chunks in (("clean", real, True), ("fours", spoiled, False), ("chunks", spoiled, True)):
        route(monkeypatch, chunks)
        monkeypatch.setattr(walk, "rows", rows)
        state = torch.zeros((1, size_of(mode, heads, dim, dim)), device=DEV)
        if what == "state" and name != "clean":
            state[0, dim * dim + (dim + 1 if mode == "mlstm" else 0) + bad] = float("inf")
        outs[name] = walk.run(mode, step, state, T, heads, dim, dim, 1, 0, torch.float32)
    clean, fours, chunks = outs["clean"], outs["fours"], outs["chunks"]
    first = 0 if what == "state" else bad
    # a chunk with an infinity is taken token by token: other sums of the same values
    if first:
        assert (chunks[:first] - clean[:first]).abs().max() <= 1e-4
    assert (chunks[:, :dim] - clean[:, :dim]).abs().max() <= 1e-4      # the other head
    # in its head it spoils what it spoils by fours, but for the rest of a group of four tokens, which
    # four at a time sum up on their own and token by token do not
    same = [t for t in range(T) if t <= bad or t // 4 > bad // 4 or what == "state"]
    assert torch.equal(chunks[same].isfinite(), fours[same].isfinite())


def test_refusals():
    step = make_step([(0, 0, [0] * 80, [])])
    assert not K.walks_in_chunks(step, 130, 64, K.WALK_DELTA, 4) and not K.walks_in_chunks(step, 64, 40, K.WALK_DELTA, 4)
    assert not K.walks_in_chunks(step, 64, 64, K.WALK_GLA, 4) and not K.walks_in_chunks(step, 64, 64, K.WALK_WKV, 4)


# delta rule of 16 heads of 128, of 8 of 64, matrix memory of 8 heads: both sides of the rule's edges
@pytest.mark.parametrize("lens, by", [
    ([127], (False, False, True)), ([128], (True, True, True)), ([95], (False, False, False)),
    ([64] * 2, (True, False, False)), ([63] * 8, (False, False, False)), ([64] * 8, (True, False, True)),
    ([300] * 6, (True, True, True)), ([300] * 7, (True, False, True)), ([300] * 9, (False, False, True)),
    ([256] + [1] * 63, (False, False, True))])
def test_rule(lens, by):
    step = make_step([(i, 0, [0] * n, []) for i, n in enumerate(lens)])
    got = tuple(K.walks_in_chunks(step, dim, 128, mode, heads) for mode, heads, dim in
                ((K.WALK_DELTA, 16, 128), (K.WALK_DELTA, 8, 64), (K.WALK_MLSTM, 8, 128)))
    assert got == by


# States and values below 2^-110, which three bfloat16 parts do not hold: the state's error is that of the
# normal range (float32 roundings of the tokens' updates, whose size does not depend on the exponent)
@pytest.mark.parametrize("mode", ["delta", "mlstm"])
@pytest.mark.parametrize("exponent", [-100, -112, -118])
def test_small_states(monkeypatch, mode, exponent):
    lens, heads, dim, vdim = [96, 40], 2, 64, 32
    T, real, per = sum(lens), walk.rows, dim * vdim + (dim + 1 if mode == "mlstm" else 0)

    def small(shape, seed, *a, **k):
        t = real(shape, seed, *a, **k)
        if seed == 1:
            t[:, 2 * heads * dim:2 * heads * dim + heads * vdim] *= 2.0 ** exponent
        return t
    monkeypatch.setattr(walk, "rows", small)
    start = real((len(lens), size_of(mode, heads, dim, vdim)), 9, 0.3)
    start.view(len(lens), heads, per)[:, :, :dim * vdim] *= 2.0 ** exponent
    _, states = walk.plain(mode, start, lens, heads, dim, vdim, 1, T)
    route(monkeypatch, True)
    state, step = start.clone(), make_step([(i, 5, [0] * n, []) for i, n in enumerate(lens)])
    walk.run(mode, step, state, T, heads, dim, vdim, 1, 0, torch.float32)
    got, want = (s.double().cpu().view(len(lens), heads, per)[:, :, :dim * vdim] for s in (state, states))
    assert (got - want).norm() <= 1e-6 * want.norm()


# a state that overflows in a sequence's last token is an infinity, as by fours
def test_an_update_that_overflows(monkeypatch):
    T, heads, dim, real, states = 64, 2, 64, walk.rows, []

    def large(shape, seed, *a, **k):
        t = real(shape, seed, *a, **k)
        if seed == 1:
            t[T - 1, heads * dim:2 * heads * dim] *= 40.0
            t[T - 1, 2 * heads * dim:3 * heads * dim] *= 5e37
        return t
    monkeypatch.setattr(walk, "rows", large)
    step = make_step([(0, 0, [0] * T, [])])
    for chunks in (False, True):
        route(monkeypatch, chunks)
        state = torch.zeros((1, size_of("mlstm", heads, dim, dim)), device=DEV)
        walk.run("mlstm", step, state, T, heads, dim, dim, 1, 0, torch.float32)
        states.append(state)
    want, got = states
    assert want.isposinf().any() and want.isneginf().any() and not want.isnan().any()
    assert torch.equal(got.isposinf(), want.isposinf()) and torch.equal(got.isneginf(), want.isneginf())
    assert not got.isnan().any()


# the matrix memory's chunks take scratch for one chunk of every sequence at least (56 KB a head of 128 x 128):
# where that is more than CHUNK_SCRATCH the step goes by fours
def test_rule_of_the_scratch():
    got = [K.walks_in_chunks(SimpleNamespace(B=B, max_new=96), 128, 128, K.WALK_MLSTM, 8) for B in (64, 350, 380, 4000)]
    assert got == [True, True, False, False]
