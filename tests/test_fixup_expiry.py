"""The fix-up of the prefill's parts when a bounded wait expires: no images are asked for again before they have landed, no rows are written from a product that part of
the group has not seen, and nothing is on its way into the shared memory or the accumulator of a CTA that ends.  How the kernel guards its steps is taken from the source."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "avelang_b200", "csrc", "prefill_tc.cu")


def _guards(text=None):
    text = text or open(SOURCE).read()
    text = re.sub(r"//[^\n]*", "", text[text.index("part_finish_kernel(const"):])
    text = text[:text.index("tmem_dealloc")]
    loop = text[text.index("for (int i = c_begin"):]
    load = re.search(r"if \(([^{;]*i \+ stride < c_end)\) \{? ?load_qt", loop).group(1)
    end = loop[loop.rindex("group_sync();"):]
    return {"loop": "&& ok" in loop[:loop.index("{")], "load": re.search(r"\bok\b", load) is not None, "group": "ok = group_all(ok)" in loop,
            "drained": {b for b in ("mma_bar", "q_full", "m0_full") if f"tc::drain({b}" in end}}


def _faults(g, chunks):
    """One group of warps, the first of which issues, and another; every wait may expire, at once when the flag is up (the other group may raise it)."""
    faults, seen = set(), set()
    # iteration, step, first warp landed and ok, other warp ok, products and images asked for, copies on their way (m0, images, product), flag
    todo = [(0, 0, True, True, True, 1, (True, True, False), False)]

    def waits(state, complete):  # -> (passed, flag) that may follow
        return [(True, state[7])] if complete else [(False, True)]

    while todo:
        s = todo.pop()
        if s in seen:
            continue
        seen.add(s)
        it, step, landed, ok0, ok1, asked, fly, flag = s
        for i in range(3):  # what is on its way arrives
            if fly[i]:
                todo.append((it, step, landed, ok0, ok1, asked, fly[:i] + (False,) + fly[i + 1:], flag))
        if step == 0:  # the first warp waits for its operands and issues
            for passed, f in waits(s, not fly[1] and (it > 0 or not fly[0])):
                if passed and fly[2]:
                    faults.add("again")
                todo.append((it, 1, passed, ok0, ok1, asked, fly[:2] + (passed or fly[2],), f))
        elif step in (1, 2):  # the first warp, then the other, wait for the product
            for passed, f in waits(s, landed and not fly[2]):
                todo.append((it, step + 1, landed, passed if step == 1 else ok0, passed if step == 2 else ok1, asked, fly, f))
        elif step == 3:
            if it + 1 < chunks and (ok0 or not g["load"]):
                if fly[1]:
                    faults.add("again")
                todo.append((it, 4, landed, ok0, ok1, asked + 1, (fly[0], True, fly[2]), flag))
            else:
                todo.append((it, 4, landed, ok0, ok1, asked, fly, flag))
        elif step == 4:  # the group meets, rows leave
            if g["group"]:
                ok0 = ok1 = ok0 and ok1
            if ok0 != ok1:
                faults.add("rows")
            more = it + 1 < chunks and (not g["loop"] or ok0)
            todo.append((it + 1, 0, landed, ok0, ok1, asked, fly, flag) if more else (it, 5, landed, ok0, ok1, asked, fly, flag))
        else:
            left = {b for b, on in zip(("m0_full", "q_full", "mma_bar"), fly) if on}
            if left - (g["drained"] if not (ok0 and ok1) else set()):
                faults.add("on its way")
    return faults


@pytest.mark.parametrize("chunks", [1, 2, 3, 4])
def test_an_expired_wait_ends_the_group(chunks):
    assert not _faults(_guards(), chunks)


@pytest.mark.parametrize("guard, fault", [("load", "again"), ("group", "rows")])
def test_the_walk_needs_the_guards(guard, fault):
    g = _guards()
    g[guard] = False
    if guard == "load":
        g["loop"] = g["group"] = False
    assert fault in _faults(g, 3)


def test_the_walk_needs_what_is_waited_for_at_the_end():
    for bar in ("mma_bar", "q_full", "m0_full"):
        g = _guards()
        g["drained"] = g["drained"] - {bar}
        assert "on its way" in _faults(g, 2)
