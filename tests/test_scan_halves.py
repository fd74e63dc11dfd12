"""The prefill's second pass by halves: each chain-epilogue group has barriers of its own for the columns it converts, and the chain's issuer takes the
halves in turn.  The roles are walked in every order of their steps, the groups as roles of their own (see test_scan_barriers)."""
import pytest

import test_scan_barriers as whole

GROUPS = 2


def _programs(chunks, groups=GROUPS):
    """Of the roles of the whole walk: the chain's issuer and the epilogue by halves, the output issuer, which follows the last half of an increment, and
    the issuer's wait for the outputs of the chunk before in front of the products of X."""
    loader, chain, out_mma, epi, out = whole._programs(chunks, ragged=False)
    for i in [i for i, (k, w) in enumerate(chain) if k == "wait" and w[0][0] == "o_full"]:  # [wait x_ready, commit vn_full, wait o_full]
        chain[i - 2:i + 1] = [chain[i], chain[i - 2], chain[i - 1]]
    halves = {"h_ready", "x_ready", "vn_full", "vd_ready", "dh_full"}
    split = []
    i = 0
    while i < len(chain):
        kind, what = chain[i]
        name = what[0][0] if kind == "wait" else None
        if name in halves:  # wait g, what follows for g, next g
            after = chain[i + 1][1] if chain[i + 1][0] == "commit" else None
            for g in range(groups):
                split.append(("wait", [(f"{name}_{'ab'[g]}", what[0][1])]))
                if after == "vn_full":
                    split.append(("commit", f"vn_full_{'ab'[g]}"))
            if after == "dh_full":
                split += [("commit", f"dh_full_{'ab'[g]}") for g in range(groups)]
            elif after == "kh_full":
                split.append(("commit", "kh_full"))
            i += 2
        else:
            split.append((kind, what))
            i += 1
    out_mma = [(k, [(n + "_b" if n == "dh_full" else n, p) for n, p in w] if k == "wait" else w) for k, w in out_mma]
    epis = []
    for g in range(groups):
        mine = []
        for kind, what in epi:
            if kind == "put":
                mine.append((kind, what + "_" + "ab"[g] if what in halves else what))
            else:
                mine.append((kind, [(n + "_" + "ab"[g] if n in halves else n, p) for n, p in what]))
        epis.append(mine)
    return [loader, split, out_mma, *epis, out]


@pytest.mark.parametrize("chunks", [1, 2, 3, 4])
def test_no_order_of_the_halves_leaves_a_role_waiting(chunks, monkeypatch):
    monkeypatch.setitem(whole.COUNT, "vn_ready", GROUPS)
    assert not whole._stuck(_programs(chunks))


def test_the_walk_finds_an_output_issuer_that_does_not_wait_for_the_new_values(monkeypatch):
    monkeypatch.setitem(whole.COUNT, "vn_ready", GROUPS)
    programs = _programs(3)
    programs[2] = [(k, [x for x in w if x[0] != "vn_ready"] if k == "wait" else w) for k, w in programs[2]]
    assert whole._stuck(programs)
