"""How many parts the prefill takes is a function of the shapes alone: the numbers themselves, at the lines of the rule."""
import pytest

from avelang_b200 import _lib
from test_prefill_schedule import _args


def _parts(B, T, heads, gated=False, *, seqs=0, longest=0, singles=0):
    """`seqs` > 0: a packed batch of T tokens, behind `singles` single tokens of a mixed step."""
    args = _args(B, T, heads, gated)
    a = args._obj
    if seqs:
        a.cu_seqlens, a.n_seqs, a.num_slots, a.max_seqlen, a.token_begin = 0x1000, seqs, seqs, longest, singles
    return _lib.load().ave_gdn_prefill_parts(args)


@pytest.mark.parametrize("B, T, heads, parts", [(1, 1024, 4, 4), (1, 1529, 16, 2), (2, 1990, 8, 4), (1, 2048, 24, 2), (1, 6144, 8, 8),  # test_scan_outputs_gpu's
                                                (1, 8192, 32, 2), (1, 32768, 4, 16), (1, 64 * 24, 16, 2), (1, 64 * 24, 18, 1), (1, 64 * 31, 24, 1), (1, 64 * 32, 24, 2)])
@pytest.mark.parametrize("gated", [False, True])
def test_dense_batches(built_lib, B, T, heads, parts, gated):
    assert _parts(B, T, heads, gated) == parts
    if B == 1:
        assert _parts(1, T, heads, gated, seqs=1) == parts
    if B == 2:
        assert _parts(1, 2 * T, heads, gated, seqs=2, longest=T) == parts


@pytest.mark.parametrize("T, heads, seqs", [(1950, 4, 3), (1950, 8, 2), (1200, 4, 2), (1984, 2, 4)])
def test_short_packed_sequences_without_a_bound_stay_whole(built_lib, T, heads, seqs):
    assert _parts(1, T, heads, seqs=seqs) == 1
    assert _parts(1, T, heads, seqs=seqs, longest=T - 40) > 1  # one of them known to be long
    assert _parts(1, 2048, heads, seqs=seqs) > 1


@pytest.mark.parametrize("heads, singles, prompt, parts", [(16, 200, 1700, 1), (8, 200, 1200, 1), (8, 200, 2500, 5), (4, 200, 1700, 5), (4, 64, 1500, 7)])
def test_a_mixed_steps_single_tokens_are_not_held_up(built_lib, heads, singles, prompt, parts):
    assert _parts(1, singles + prompt, heads, seqs=1, singles=singles) == parts


@pytest.mark.parametrize("gated", [False, True])
def test_every_chain_gets_an_sm(built_lib, gated):
    for heads in (2, 4, 6, 8, 12, 16, 24, 32, 48, 50, 74, 148, 200):
        for chunks in range(1, 80):
            parts = _parts(1, 64 * chunks, heads, gated)
            assert 1 <= parts <= 16 and (parts == 1 or (2 * parts - 1) * heads <= 148)
            assert chunks >= 12 or parts == 1
