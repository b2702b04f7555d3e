"""A decode step is captured while what an earlier engine left waits for Python's collector."""
import gc

import pytest
import torch

from mormot2_ai_b200 import Engine, Entry

pytestmark = pytest.mark.gpu


def test_an_earlier_engine_is_not_collected_under_a_capture(tiny):
    def decode(eager):
        eng = Engine.from_folder(tiny.folder, dtype="bfloat16", max_tokens=1024, max_slots=2)
        eng.mine = eng                      # only the collector frees it
        slots = [eng.open() for _ in range(2)]
        eng.step([Entry(s, tiny.tokens(5, seed=s)) for s in slots])
        forward = eng.model.forward

        def under_an_eager_collector(*args):
            if torch.cuda.is_current_stream_capturing():
                gc.set_threshold(1, 1, 1)
            return forward(*args)

        if eager:
            gc.enable()
            eng.model.forward = under_an_eager_collector
        return eng.step([Entry(s, [7]) for s in slots]).cpu()

    before = gc.get_threshold()
    gc.collect()
    gc.freeze()                             # all that is older is no business of the collector's
    gc.disable()
    gc.set_threshold(1 << 30, 1 << 30, 1 << 30)
    try:
        first, second = decode(False), decode(True)
        assert gc.isenabled()
    finally:
        gc.set_threshold(*before)
        gc.enable()
        gc.unfreeze()
        gc.collect()
    assert first.equal(second)
