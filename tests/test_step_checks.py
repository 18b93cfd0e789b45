"""What a step refuses on the host, before anything is launched (no device needed: the check reads
only the vocabulary size)."""
from types import SimpleNamespace

import numpy as np
import pytest

from alpacca_b200.engine.engine import Engine
from alpacca_b200.engine.step import StepEntry


def check(entries, vocab=10):
    return Engine._check(SimpleNamespace(vocab_size=vocab), entries)


def test_good_entries_come_back_as_int32_arrays():
    arrays = check([StepEntry(0, [1, 2, 9], [0, 2]), StepEntry(3, np.array([0, 5]), [])])
    assert [a.dtype for a in arrays] == [np.int32, np.int32]
    assert arrays[0].tolist() == [1, 2, 9] and arrays[1].tolist() == [0, 5]


@pytest.mark.parametrize("entries,needle", [
    ([], "at least one sequence"),
    ([StepEntry(0, [1], [0]), StepEntry(0, [2], [0])], "appears twice"),
    ([StepEntry(0, [], [])], "at least one token"),
    ([StepEntry(0, [1, 10], [0])], "token id 10 lies outside the vocabulary of 10"),
    ([StepEntry(0, [3, -1], [0])], "token id -1 lies outside"),
    ([StepEntry(0, [1.5, 2.0], [0])], "integers"),
    ([StepEntry(0, [[1, 2]], [0])], "flat list"),
    ([StepEntry(0, [1, 2], [2])], "wanted place 2 is not among its 2 tokens"),
    ([StepEntry(0, [1, 2], [-1])], "wanted place -1"),
])
def test_faulty_entries_are_refused(entries, needle):
    with pytest.raises(ValueError, match=needle):
        check(entries)


def test_an_engine_cannot_have_more_positions_than_its_model_was_built_for():
    """Tables indexed by position (the rotation's angles) have as many rows as the model was built for;
    an engine that let sequences grow beyond them would have the kernels read past their end."""
    import torch
    from alpacca_b200.parts.base import BuildOptions
    model = SimpleNamespace(opts=BuildOptions(dtype=torch.float32, device="cpu", max_positions=128),
                            cache_entry_specs=lambda: [], spec=SimpleNamespace(vocab_size=10))
    eng = Engine(model, max_tokens=256, max_slots=2)
    assert eng.max_positions == 128
    assert Engine(model, max_tokens=256, max_slots=2, max_positions=64).max_positions == 64
    with pytest.raises(ValueError, match="built\\s+for 128"):
        Engine(model, max_tokens=256, max_slots=2, max_positions=129)


@pytest.mark.parametrize("room,lens", [(12, [8192] + [1] * 11), (18, [1] * 17 + [2048]), (12, [4000] + [300] * 6), (12, [2048]), (1, [500]),
                                       (18, [1500, 1000]), (296, [60000] + [1] * 99), (0, [5000, 3]), (12, [32768] * 8), (5, [1]),
                                       (40, [100] * 39 + [3000]), (37, [2000 + 250 * i for i in range(8)])])
def test_pieces_of_a_recurrent_prompt(room, lens):
    """One length for all sequences, a multiple of 8; what has more than one piece fits beside the others; the shortest such
    length; a long sequence is cut however many short ones stand beside it."""
    from alpacca_b200 import ops
    ctx = SimpleNamespace(host_q_lens=lens, extras={})
    length, items, kept = ops._piece_plan(ctx, room)
    pieces = [-(-n // length) for n in lens]
    assert length % 8 == 0 and length >= 32 and items == sum(pieces) and kept == sum(p for p in pieces if p > 1)

    def shortest(room):
        fits = (n for n in range(32, max(lens) + 8, 8)
                if sum(q / n if 4 * q <= n else -(-q // n) for q in lens) <= room)
        return next(fits, max(-(-max(lens) // 8) * 8, 32))
    one, two = shortest(room), shortest(2 * room)
    two_rounds = 2 * (5 * two + 120) < 0.9 * ((3 if one >= max(lens) else 5) * one + 120)
    assert length == (two if two_rounds else one) and kept <= 2 * room
    if room >= 12 and 4 * sum(lens) < 5 * max(lens):
        assert -(-max(lens) // length) >= room // 2
    assert ops._piece_plan(ctx, room) is ctx.extras["pieces", room]


def test_a_context_without_lengths_on_the_host_walks_in_order():
    from alpacca_b200 import ops
    ctx = SimpleNamespace(is_decode=False, n_tokens=500, n_seqs=1, host_q_lens=None, extras={})
    assert not ops._walks_pieces(ctx, 128, 128)


@pytest.mark.parametrize("H,K,seqs,pays", [
    (32, 8, [(0, 1024)], True), (32, 8, [(0, 700)], False), (32, 8, [(2000, 1000)], True), (32, 8, [(0, 512)] * 2, False),
    (32, 8, [(500, 160)] * 4, False), (32, 8, [(2000, 160)] * 4, True), (32, 32, [(500, 192)] * 4, False), (32, 32, [(2000, 192)] * 4, True),
    (32, 8, [(4000, 500)], False), (32, 8, [(0, 8192)], True), (32, 8, [(2000, 288)] * 4, False), (32, 8, [(2000, 320)] * 4, True),
    (32, 8, [(4000, 64)] + [(0, 500)] * 8, True), (32, 8, [(0, 1111)] * 3, False), (32, 2, [(0, 4096)], True), (32, 8, [(0, 1)], False)])
def test_which_prompts_take_two_query_tiles_per_block(H, K, seqs, pays):
    """On 148 processors; the sides that were measured (held and new tokens of each sequence)."""
    from alpacca_b200 import ops
    assert ops._pair_pays([n for _, n in seqs], [h + n for h, n in seqs], H, K, 148) is pays
