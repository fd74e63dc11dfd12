"""The barriers of the prefill's second pass.  A wait on an mbarrier sees only the parity of its phase: a barrier that completes twice before
one of its waiters has looked leaves that waiter behind.  The roles of the kernel are walked here in every order of their steps, as lists of waits
and arrivals that are compared with the kernel's source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avelang_b200", "csrc", "prefill_scan.cuh")
STAGES = 3
COUNT = {"empty": 3}  # arrivals a phase: the two issuers and the output warps (a group of warps counts as one); 1 elsewhere
ROLES = {  # marker of the role's code -> its steps: `wait` barriers, `put` for an arrival, `commit` for one that comes when the MMAs are complete
    "loader:": ["wait empty", "commit when_full", "wait tail_full", "put full"],  # when_full: `tail_full` for the last chunk of a sequence that ends inside it
    "chain MMA issuer": ["wait full", "wait h_ready", "commit kh_full", "commit empty", "wait x_ready", "commit vn_full", "wait o_full",
                         "wait vd_ready", "commit dh_full", "wait full"],
    "output MMA issuer": ["wait kh_full o1_empty full", "commit o1_done", "wait vn_ready o2_empty dh_full", "commit o_full", "commit empty"],
    "chain epilogue:": ["put h_ready", "wait full kh_full", "put x_ready", "wait vn_full", "put vd_ready", "wait o_full", "put vn_ready", "wait dh_full o1_done"],
    "output warps:": ["wait o_full", "put o1_empty", "put o2_empty", "put empty"],
}


def _source_steps():
    text = open(SOURCE).read()
    at = sorted((text.index(mark, text.index("if (warp == 0) {")), mark) for mark in ROLES)
    steps = {}
    for i, (begin, mark) in enumerate(at):
        code = re.sub(r"//[^\n]*", "", text[begin:at[i + 1][0] if i + 1 < len(at) else None].split("\n", 1)[1])
        found = []
        for call, args in re.findall(r"tc::(mbar_wait(?:_warp|2|3)?|mbar_arrive|mma_commit|mbar_expect_tx)\(((?:[^()]|\([^()]*\))*)\)", code):
            names = re.findall(r"\b([a-z0-9_]*(?:full|empty|ready|done))\b", args)
            found.append({"w": "wait", "a": "put", "x": "commit"}["x" if call in ("mma_commit", "mbar_expect_tx") else call[5]] + " " + " ".join(names))
        steps[mark] = found
    return steps


def _programs(chunks, ordered=True, ragged=True):
    """One list of steps a role: (kind, [(barrier, phase)]), a wait naming the phase that has to be complete."""
    full, empty = (lambda c: f"full{c % STAGES}"), (lambda c: f"empty{c % STAGES}")
    loader, chain, out_mma, epi, out = [], [("wait", [(full(0), 0)])], [], [("put", "h_ready")], []
    for c in range(chunks):
        if c >= STAGES:
            loader.append(("wait", [(empty(c), c // STAGES - 1)]))
        loader.append(("commit", full(c) if c + 1 < chunks or not ragged else "tail_full"))
        chain += [("wait", [("h_ready", c)]), ("commit", "kh_full")] + ([("commit", empty(c - 1))] if c else [])
        chain += [("wait", [("x_ready", c)]), ("commit", "vn_full")] + ([("wait", [("o_full", c - 1)])] if ordered else [])
        chain += [("wait", [("vd_ready", c)]), ("commit", "dh_full")]
        if c + 1 < chunks:
            chain.append(("wait", [(full(c + 1), (c + 1) // STAGES)]))
        out_mma += [("wait", [("kh_full", c), ("o1_empty", c - 1), (full(c), c // STAGES)]), ("commit", "o1_done"),
                    ("wait", [("vn_ready", c), ("o2_empty", c - 1), ("dh_full", c)]), ("commit", "o_full"), ("commit", empty(c))]
        epi += [("wait", [(full(c), c // STAGES), ("kh_full", c)]), ("put", "x_ready")]
        epi += [("wait", [("vn_full", c)]), ("put", "vd_ready"), ("wait", [("o_full", c - 1)]), ("put", "vn_ready")]
        epi += [("wait", [("dh_full", c), ("o1_done", c)]), ("put", "h_ready")]
        out += [("wait", [("o_full", c)]), ("put", "o1_empty"), ("put", "o2_empty"), ("put", empty(c))]
    loader += [("wait", [("tail_full", 0)]), ("put", full(chunks - 1))] if ragged else []
    return [loader, chain, out_mma, epi, out]


def _stuck(programs):
    """Whether some order of the roles' steps ends with a role that waits for good, or lets one pass too early."""
    names = sorted({b for p in programs for k, x in p for b in ([n for n, _ in x] if k == "wait" else [x])})
    index = {n: i for i, n in enumerate(names)}
    start = ((0,) * len(programs), (0,) * len(programs), (0,) * len(names), ((),) * len(programs))  # step, waits passed, arrivals, commits on their way
    seen, todo = {start}, [start]

    def arrive(arrivals, name):
        return arrivals[:index[name]] + (arrivals[index[name]] + 1,) + arrivals[index[name] + 1:]

    def phase(arrivals, name):
        return arrivals[index[name]] // COUNT.get(name.rstrip("0123456789"), 1)

    while todo:
        state = todo.pop()
        at, mask, arrivals, flight = state
        moves = []
        for r, program in enumerate(programs):
            if flight[r]:  # the oldest commit of this role completes
                moves.append((at, mask, arrive(arrivals, flight[r][0]), flight[:r] + (flight[r][1:],) + flight[r + 1:]))
            if at[r] == len(program):
                continue
            kind, what = program[at[r]]
            step = at[:r] + (at[r] + 1,) + at[r + 1:]
            if kind == "put":
                moves.append((step, mask, arrive(arrivals, what), flight))
            elif kind == "commit":
                moves.append((step, mask, arrivals, flight[:r] + (flight[r] + (what,),) + flight[r + 1:]))
            else:
                for i, (name, want) in enumerate(what):
                    if not mask[r] >> i & 1 and (phase(arrivals, name) & 1) != (want & 1):  # what a parity wait sees
                        if phase(arrivals, name) <= want:
                            return True  # the other way round: passed a phase early
                        m = mask[r] | 1 << i
                        done = m == (1 << len(what)) - 1
                        moves.append((step if done else at, mask[:r] + (0 if done else m,) + mask[r + 1:], arrivals, flight))
        if not moves and any(a < len(p) for a, p in zip(at, programs)):
            return True
        for m in moves:
            if m not in seen:
                seen.add(m)
                todo.append(m)
    return False


def test_the_lists_are_the_kernels():
    assert _source_steps() == ROLES


@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("ragged", [False, True])
def test_no_order_leaves_a_role_waiting(chunks, ragged):
    assert not _stuck(_programs(chunks, ragged=ragged))


def test_the_walk_finds_a_wait_that_nothing_orders():
    assert _stuck(_programs(3, ordered=False))
