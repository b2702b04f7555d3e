"""The filtered draw over rows whose shares lie in shared memory (up to 393,216 tokens) and over
longer ones: the token that the plain rule picks, at the edges of shares and of the sums' runs."""
import numpy as np
import pytest
import torch

from mormot2_ai_b200.sampling import DeviceSampler, Sampling
from tests.gpu_helpers import DEV

pytestmark = pytest.mark.gpu


def splitmix(state):
    mask = (1 << 64) - 1
    state = (state + 0x9E3779B97F4A7C15) & mask
    z = state
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
    return state, ((z ^ (z >> 31)) >> 11) / 9007199254740992.0


@pytest.mark.parametrize("vocab", [16384, 16391, 151936, 393216, 393217])
@pytest.mark.parametrize("settings", [dict(temperature=0.7, top_p=0.9), dict(temperature=1.0, top_k=50),
                                      dict(temperature=1.0, min_p=0.05),
                                      dict(temperature=2.0, top_k=700, top_p=0.95)])
def test_filtered_draws(vocab, settings):
    rng = np.random.default_rng(vocab)
    rows, draws = 3, 4
    logits = (rng.standard_normal((rows, vocab)) * 2).astype(np.float32)
    for r in range(rows):
        logits[r, rng.integers(0, vocab, 30)] += rng.uniform(2, 12, 30).astype(np.float32)
    logits[0, 5] = np.nan
    s = Sampling(seed=1, **settings)
    sampler = DeviceSampler(torch.device(DEV), rows, vocab)
    states = [1000 + r for r in range(rows)]
    for r, x in enumerate(states):
        sampler.start(r, x)
    dev, slots = torch.tensor(logits).to(DEV), torch.arange(rows, dtype=torch.int32, device=DEV)
    for _ in range(draws):
        got = sampler.pick(dev, slots, s).tolist()
        for r in range(rows):
            x = logits[r].astype(np.float64)
            x[np.isnan(x)] = -np.inf
            order = np.lexsort((np.arange(vocab), -x))
            w = np.exp((x[order] - x[order[0]]) / s.temperature)
            n = vocab
            if s.top_k:
                n = max(s.top_k, int((x[order] >= x[order[s.top_k - 1]]).sum()))
            if s.top_p < 1:
                n = min(n, int(np.searchsorted(np.cumsum(w[:n]), s.top_p * w[:n].sum())) + 1)
            if s.min_p > 0:
                n = min(n, int((w >= s.min_p * w[0]).sum()))
            states[r], u = splitmix(states[r])
            cum = np.cumsum(w[:n])
            assert got[r] == order[int(np.searchsorted(cum, u * cum[-1], side="right"))]
