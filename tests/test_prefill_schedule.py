"""The prefill's schedule is a function of the shapes alone, so the edges of its rules are tested without a GPU, and so is the scratch it asks for."""
import ctypes

import pytest

from avelang_b200 import _lib


def _args(B, T, heads, gated):
    a = _lib.GdnArgs()
    a.struct_size = ctypes.sizeof(_lib.GdnArgs)
    for n in ("q", "k", "v", "g", "beta", "o"):
        setattr(a, n, 0x1000)  # never read: only shapes and the presence of a gate enter
    a.z = 0x1000 if gated else None
    a.B, a.T, a.Hk, a.Hv, a.dk, a.dv, a.n_seqs, a.num_slots, a.chunk = B, T, heads // 2, heads, 128, 128, B, B, 64
    return ctypes.byref(a)


def _parts(B, T, heads, gated):
    parts = _lib.load().ave_gdn_prefill_parts(_args(B, T, heads, gated))
    assert parts >= 1
    return parts > 1


# per (chunk, value head): a record, 32 KiB of operand images of the transition chains with parts, and 32 KiB of fp32 rows that wait for the
# norm or the fix-up; with parts 64 KiB for each chain's state and for the image of each state that enters a part.  Two per cent for tables and alignment
@pytest.mark.parametrize("B, T, heads, gated", [(1, 8192, 32, True), (1, 8192, 32, False), (1, 32768, 4, True), (2, 1000, 32, False), (1, 64 * 40, 28, True)])
def test_scratch_is_what_the_schedule_uses(built_lib, B, T, heads, gated):
    args = _args(B, T, heads, gated)
    parts, chunks = _lib.load().ave_gdn_prefill_parts(args), B * ((T + 63) // 64) * heads
    need = chunks * 21504 + (B * T * heads * 512 if gated or parts > 1 else 0)
    if parts > 1:
        need += chunks * 32768 + B * heads * 65536 * (2 * parts - 1 + parts - 1)
    assert need <= _lib.load().ave_gdn_prefill_workspace_bytes(args) <= 1.02 * need + 65536


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
