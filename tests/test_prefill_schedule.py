"""The prefill's schedule is a function of the shapes alone, so the edges of its rules are tested without a GPU, by the scratch it asks
for: a record is 66304 bytes, and parallel parts keep 32 KiB of operand images beside each."""
import ctypes

import pytest

from avelang_b200 import _lib


def _parts(B, T, heads, gated):
    a = _lib.GdnArgs()
    a.struct_size = ctypes.sizeof(_lib.GdnArgs)
    for n in ("q", "k", "v", "g", "beta", "o"):
        setattr(a, n, 0x1000)  # never read: only shapes and the presence of a gate enter
    a.z = 0x1000 if gated else None
    a.B, a.T, a.Hk, a.Hv, a.dk, a.dv, a.n_seqs, a.num_slots, a.chunk = B, T, heads // 2, heads, 128, 128, B, B, 64
    chunks = B * ((T + 63) // 64) * heads
    scratch = _lib.load().ave_gdn_prefill_workspace_bytes(ctypes.byref(a))
    rows = B * T * heads * 128 * 4  # un-normalised rows wait in fp32 where there is a gate, or parts
    left = scratch - chunks * 66304 - (rows if gated else 0)
    return left > chunks * 32768


# the length of the longest chain, in 64-token chunks, at which two parts begin, with a gate and without
@pytest.mark.parametrize("gated, first", [(True, 112), (False, 64)])
@pytest.mark.parametrize("B, heads", [(1, 32), (2, 16), (1, 30)])
def test_two_parts_begin_where_the_chains_are_long_enough(built_lib, gated, first, B, heads):
    assert not _parts(B, 64 * (first - 1), heads, gated)
    assert _parts(B, 64 * (first - 1) + 1, heads, gated) and _parts(B, 64 * 512, heads, gated)


@pytest.mark.parametrize("gated", [False, True])
def test_more_chains_than_two_parts_leave_room_for_stay_whole(built_lib, gated):
    assert not _parts(1, 64 * 512, 34, gated) and not _parts(2, 64 * 512, 24, gated)
    assert _parts(1, 64 * 32, 28, gated) and not _parts(1, 64 * 31, 28, gated)  # three parts and more: from 32 chunks on
