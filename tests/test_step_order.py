"""A decode step packs its sequences the longest first where that matters; logits, slots and states
stay where the caller's entries put them."""
import pytest
import torch

from mormot2_ai_b200 import Engine, Entry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rows_stay_in_the_order_of_the_entries(tiny, dtype):
    lens, got = [3, 40, 7, 40, 21, 1], []
    for sort_from in (2, 1 << 30):
        eng = Engine.from_folder(tiny.folder, dtype=dtype, max_tokens=2048, max_slots=len(lens))
        eng.sort_from = sort_from
        slots = [eng.open() for _ in lens]
        for slot, n in zip(slots, lens):
            eng.step([Entry(slot, tiny.tokens(n, seed=n), [])])
        out = []
        # the same shape twice (the second is a replay), rows that nobody wants or that are
        # wanted twice, the longest first as they come, and one alone
        for pick, wants in (([0, 1, 2, 3, 4, 5], None), ([0, 1, 2, 3, 4, 5], None),
                            ([5, 1, 0, 3], [[0], [], [0, 0], [0]]), ([1, 4], None), ([2], None)):
            entries = [Entry(slots[i], [5 + i], None if wants is None else wants[j])
                       for j, i in enumerate(pick)]
            past = [eng.length(slots[i]) for i in pick]
            logits = eng.step(entries)
            out.append(logits.clone())
            assert eng.last_slots.tolist() == [slots[i] for i in pick]
            n = 4 * len(pick) + 3 * len(pick) + 1 + logits.shape[0]
            moved = sort_from == 2 and past != sorted(past, reverse=True)
            assert eng.last_h2d_bytes == 4 * (n + (len(pick) if moved else 0))
        eng.rt.check()
        got.append(out)
    for a, b in zip(*got):
        assert torch.equal(a, b)


def test_packing():
    from mormot2_ai_b200.engine.batch import StepBuffers
    buffers = StepBuffers(16, 8, torch.device("cuda:0"))
    seqs = [(3, 5, [11], [0]), (0, 9, [12], []), (7, 9, [13], [0, 0]), (1, 2, [14], [0])]
    for first in (False, True):
        step = buffers.fill(seqs, first)
        rows = [1, 2, 0, 3] if first else [0, 1, 2, 3]      # which sequence is in each row
        assert step.tok_ids.tolist() == [seqs[i][2][0] for i in rows]
        assert step.tok_pos.tolist() == step.seq_past.tolist() == [seqs[i][1] for i in rows]
        assert step.tok_slot.tolist() == step.seq_slot.tolist() == [seqs[i][0] for i in rows]
        assert step.tok_seq.tolist() == [0, 1, 2, 3] and step.seq_start.tolist() == [0, 1, 2, 3, 4]
        assert step.want_rows.tolist() == [rows.index(i) for i in (0, 2, 2, 3)]
        assert step.entry_slots.tolist() == [3, 0, 7, 1]
        assert step.decode and step.max_len == 10
