"""The prefill's second pass when a bounded wait expires: the CTA still reaches its end, no stage is asked for again before it has landed, and no role that has
not met an expiry goes on too early.  The roles' steps are taken from the kernel's source in the order in which they run (lambdas expanded at their calls, loops over
the groups unrolled), hardware barriers are counters of warps, and any wait may expire at any step."""
import re

import pytest

import test_scan_barriers as whole

NG, STAGES = 2, 2  # (a ring of two stages comes round within three chunks)
HARDWARE = ("h_ready", "x_ready", "vd_ready")  # one a group: its four warps and the issuer
STEP = re.compile(r"tc::(mbar_wait(?:_warp|2|3)?|mbar_arrive|mma_commit)\(((?:[^()]|\([^()]*\))*)\)")
NAME = re.compile(r"\b([a-z0-9_]*(?:full|empty|ready|done))\b")


def _source(text=None):
    """Role -> its code without comments."""
    text = text or open(whole.SOURCE).read()
    at = sorted((text.index(mark, text.index("if (warp == 0) {")), mark) for mark in whole.ROLES)
    code = {}
    for i, (begin, mark) in enumerate(at):
        body = text[begin:at[i + 1][0] if i + 1 < len(at) else None].split("\n", 1)[1]
        code[mark] = re.sub(r"^\s*#.*$", "", re.sub(r"//[^\n]*", "", body), flags=re.M)
    return code


def _parse(code):
    """Statements and blocks: a list of text, or (head, list).  Ends at the brace that closes the role."""
    stack, head, depth = [("", [])], "", 0
    for ch in code:
        if ch == "{" and depth == 0:
            stack.append((" ".join(head.split()), []))
            head = ""
        elif ch == "}" and depth == 0:
            if len(stack) == 1:
                break
            block = stack.pop()
            stack[-1][1].append(block)
            head = ""
        elif ch == ";" and depth == 0:
            if head.split():
                stack[-1][1].append(" ".join(head.split()))
            head = ""
        else:
            depth += {"(": 1, "[": 1, ")": -1, "]": -1}.get(ch, 0)
            head += ch
    return stack[0][1]


def _split(text):
    """`if (cond) rest` or `for (head) rest` -> inside of the parentheses, rest."""
    i = text.index("(")
    depth, j = 1, i + 1
    while depth:
        depth += {"(": 1, ")": -1}.get(text[j], 0)
        j += 1
    return text[i + 1:j - 1], text[j:].strip()


def _flat(nodes):
    return " ".join(n if isinstance(n, str) else n[0] + " " + _flat(n[1]) for n in ([nodes] if isinstance(nodes, (str, tuple)) else nodes))


def _steps(code, chunks, group=0):
    """The steps of one role, in the order in which they run: (kind, barriers, what an expiry or a role that has met one does here)."""
    lambdas, out, seen = {}, [], {}
    env = {"NG": NG, "HAND_OVERS": 3 * NG, "C": 64, "n_chunks": chunks, "grp": group}
    tail = "tc::named_sync(hand_over(" in code

    def value(expr):
        return eval(expr.replace("&&", " and ").replace("||", " or ").replace("/", "//"), {}, env)

    def barrier(arg, first):
        name = NAME.search(arg).group(1)
        if name in HARDWARE:
            return name + "ab"[value(re.search(r"_ready\((\w+)\)", arg).group(1))]
        index = re.search(name + r"\[(\w+)\]", arg)
        if name in ("vn_full", "dh_full"):
            return name + "ab"[value(index.group(1))]
        if name in ("full", "empty"):  # stage by stage
            k = seen.setdefault((name, first), 0)
            seen[name, first] += 1
            return f"{name}{k % STAGES}"
        return name

    def emit(text, expired):
        for call, args in STEP.findall(text):
            args = re.split(r",\s*(?![^()]*\))", args)
            if call.startswith("mbar_wait"):
                bars = []
                for arg, parity in zip(args[::2], args[1::2]):
                    if not NAME.search(arg):
                        continue
                    b = barrier(arg, "wait")
                    n = seen.setdefault((b, "phase"), -1 if "^ 1u" in parity or "+ 1) & 1u" in parity else 0)
                    seen[b, "phase"] += 1
                    bars.append((b, n))
                hardware = bars[0][0][:-1] in HARDWARE
                out.append(("meet" if hardware else "wait", bars, None if hardware else expired))
            else:
                b = barrier(args[0], call)
                if b[:-1] in HARDWARE:
                    out.append(("arrive", b, "meets" if len(args) > 1 else "arrives"))
                else:
                    out.append(("commit" if call == "mma_commit" else "put", b, "not" if "alive) tc::mbar_arrive" in text else "puts"))

    def has(nodes):
        text = _flat(nodes)
        return bool(STEP.search(text)) or any(re.search(rf"\b{n}\(", text) for n in lambdas)

    def call(text, expired):
        """Steps of a statement: its own, or those of the lambda that it calls."""
        for name, (params, body) in lambdas.items():
            hit = re.search(rf"\b{name}\(", text)
            if hit:
                run(body, expired)
                return
        emit(text, expired)

    def leaves(cond, body):
        """`if (!wait) ... break` or `return false`; the number of hand-overs that it names is that of those behind it."""
        met = re.search(r"\bmet = ([^;]*?)(?:;|$| break)", body)
        if met and "break" in body:
            assert value(met.group(1)) == sum(k == "meet" for k, _, _ in out)
        return "leave"

    def run(nodes, expired="ignore"):
        for node in nodes:
            if isinstance(node, tuple):
                head, body = node
                made = re.match(r"auto (\w+) = \[&\]\(([^)]*)\)", head)
                if made:
                    if has(body):
                        lambdas[made.group(1)] = (made.group(2), body)
                elif head.startswith("for") and has(body):
                    var, start, cond, by = re.match(r"int (\w+) = (\w+); ([^;]*); (?:\+\+\w+|\w+ \+= (\d+))$", _split(head)[0]).groups()
                    cond = " and ".join(x for x in cond.split("&&") if re.search(r"[<>]", x))
                    env[var] = value(start)
                    while value(cond):
                        run(body, expired)
                        env[var] += int(by or 1)
                elif re.match(r"(else )?if\b", head):
                    cond, _ = _split(head)
                    if has(cond):  # (the steps first, then what their expiry does)
                        call(cond, "leave")
                        leaves(cond, _flat(body))
                    elif has(body) and holds(cond):
                        run(body, expired)
                elif has(body):
                    run(body, expired)
            elif re.match(r"if\b", node):
                cond, rest = _split(node)
                if has(cond):
                    assert rest in ("break", "return false")
                    call(cond, "leave")
                elif has(rest) and holds(cond):
                    call(node if "alive" in cond else rest, expired)
            elif has(node):
                kind = "dead" if node.startswith("alive =") else "leave" if node.startswith("const bool landed") else expired if node.startswith("return") else "ignore"
                call(node, kind)

    def holds(cond):
        if re.fullmatch(r"(tc::elect_one\(\)|lane == 0( && alive)?|landed|alive)", cond):
            return True
        return bool(value(cond))

    run(_parse(code))
    assert not tail or sum(k == "meet" for k, _, _ in out) == 3 * NG * chunks
    return out, tail


def _programs(chunks, text=None):
    code = _source(text)
    loader = []
    for c in range(chunks):
        if c >= STAGES:
            loader.append(("wait", [(f"empty{c % STAGES}", c // STAGES - 1)], "leave"))
        loader.append(("load", f"full{c % STAGES}", None))
    programs, tails = [loader], [False]
    for mark in ("chain MMA issuer", "output MMA issuer", "output warps:"):
        steps, tail = _steps(code[mark], chunks)
        programs.append(steps)
        tails.append(tail)
    for g in range(NG):
        programs.append(_steps(code["chain epilogue:"], chunks, g)[0])
        tails.append(False)
    return programs, tails


COUNT = {"empty": 3, "vn_ready": NG}


def _faults(programs, tails, expiries=True, until=None):
    """(Up to the fault that is looked for.)  What some order of the steps leads to: `waits` for good, `early` past a phase that is not complete, `again`: a stage asked for before it has landed."""
    bars = sorted({b for p in programs for k, x, _ in p for b in ([n for n, _ in x] if k in ("wait", "meet") else [x])})
    index = {n: i for i, n in enumerate(bars)}
    n = len(programs)
    # position, met an expiry, left for the hand-overs alone, phase a hardware barrier has to reach, arrivals, warps at hardware barriers, copies on their way, flag
    start = ((0,) * n, (False,) * n, (False,) * n, (None,) * n, (0,) * len(bars), (0,) * len(bars), (), False)
    seen, todo, faults = {start}, [start], set()
    put = lambda t, i, v: t[:i] + (v,) + t[i + 1:]  # noqa: E731

    def join(arrivals, warps, name, count):
        """`count` warps come to a hardware barrier of five, one by one; also the phase that the last of them belongs to."""
        i, mine = index[name], None
        a, w = arrivals[i], warps[i]
        for _ in range(count):
            mine, w = a, w + 1
            if w == 5:
                a, w = a + 1, 0
        return put(arrivals, i, a), put(warps, i, w), mine

    while todo and until not in faults:
        state = todo.pop()
        at, dead, left, meets, arrivals, warps, flight, flag = state
        moves = [(at, dead, left, meets, put(arrivals, index[b], arrivals[index[b]] + 1), warps, flight[:i] + flight[i + 1:], flag) for i, b in enumerate(flight)]
        phase = lambda b: arrivals[index[b]] // COUNT.get(b.rstrip("0123456789"), 1)  # noqa: E731
        for r, program in enumerate(programs):
            p = at[r]
            if left[r]:  # takes part in the hand-overs only
                while p < len(program) and program[p][0] != "meet":
                    p += 1
            if p == len(program):
                if p != at[r]:
                    moves.append((put(at, r, p), *state[1:]))
                continue
            kind, what, how = program[p]
            step = put(at, r, p + 1)
            if meets[r] is not None:  # at a hardware barrier
                if arrivals[index[meets[r][0]]] > meets[r][1]:
                    moves.append((step, dead, left, put(meets, r, None), arrivals, warps, flight, flag))
            elif kind == "meet" or (kind == "arrive" and dead[r] and how == "meets"):
                b = what[0][0] if kind == "meet" else what
                a, w, mine = join(arrivals, warps, b, 1 if kind == "meet" else 4)
                moves.append((put(at, r, p), dead, left, put(meets, r, (b, mine)), a, w, flight, flag))
            elif kind == "arrive":
                a, w, _ = join(arrivals, warps, what, 4)
                moves.append((step, dead, left, meets, a, w, flight, flag))
            elif kind in ("put", "commit"):
                more = 0 if kind == "put" and how == "not" and dead[r] else 1
                moves.append((step, dead, left, meets, put(arrivals, index[what], arrivals[index[what]] + more), warps, flight, flag))
            elif kind == "load":
                if what in flight:
                    faults.add("again")
                moves.append((step, dead, left, meets, arrivals, warps, flight + (what,), flag))
            else:
                if all((phase(b) & 1) != (want & 1) for b, want in what):  # what a parity wait sees
                    if not dead[r] and any(phase(b) <= want for b, want in what):
                        faults.add("early")
                    moves.append((step, dead, left, meets, arrivals, warps, flight, flag))
                elif flag or expiries:
                    if how == "leave":
                        moves.append((step if tails[r] else put(at, r, len(program)), dead, put(left, r, True), meets, arrivals, warps, flight, True))
                    else:
                        moves.append((step, put(dead, r, dead[r] or how == "dead"), left, meets, arrivals, warps, flight, True))
        if not moves and any(a < len(q) for a, q in zip(at, programs)):
            faults.add("waits")
        for m in moves:
            if m not in seen:
                seen.add(m)
                todo.append(m)
    return faults


@pytest.mark.parametrize("chunks", [1, 2, 3])
def test_an_expired_wait_leaves_nobody_waiting(chunks):
    assert not _faults(*_programs(chunks))


@pytest.mark.parametrize("chunks", [1, 2, 4])
def test_the_steps_as_they_run_leave_nobody_waiting(chunks):
    assert not _faults(*_programs(chunks), expiries=False)


def test_the_walk_finds_a_call_that_is_missing():
    """Without its wait for the outputs of the chunk before, the issuer lets an increment complete twice before the output issuer has looked."""
    text = open(whole.SOURCE).read()
    call = re.search(r"\n[^\n]*\boutputs_before\(c\)[^\n]*;[^\n]*\n", text)
    assert call and _faults(*_programs(3, text.replace(call.group(0), "\n")), expiries=False)


def test_the_walk_finds_warps_that_pass_the_issuer():
    """A warp that arrives after an expiry, and waits for nothing any more, comes back before the issuer has gone through."""
    programs, tails = _programs(2)
    programs = [[(k, x, "arrives" if k == "arrive" else how) for k, x, how in p] for p in programs]
    assert "waits" in _faults(programs, tails, until="waits")
