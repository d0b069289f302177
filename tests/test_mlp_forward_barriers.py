"""The two groups of the TTT-MLP forward meet on mbarriers that are waited on by the parity of a phase.  A wait only works while the
barrier is at most one phase ahead of the waiter: with two the parity is the waiter's own again and the wait never ends.  The
kernel's barrier operations, taken from its source, run here on a model of mbarriers, with any one warp held up at any one of
them for as long as the others can go on."""
import re
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "ttt_rs_b200" / "csrc" / "ttt_mlp_fwd.cu"
NST, STAGES = 3, 6
OP = re.compile(r"(?:if \((?P<cond>(?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\)\s*\{?\s*)?\b(?P<op>wait_for|mbar_arrive_warp|mlp_group_sync<\d>|half_sync|issue|issue_first|form_m1|"
                r"issue_load)\((?P<args>(?:[^(){};]|\((?:[^()]|\([^()]*\))*\))*)[,)]")


def _block(text, start):
    """The braces that open at or after `start`: (body, end)."""
    a = text.index("{", start)
    depth, i = 0, a
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[a + 1:i], i + 1
        i += 1


def _ops(text):
    return [(m["cond"], m["op"], [a.strip() for a in m["args"].split(",")]) for m in OP.finditer(text)]


def _program():
    """{group: (lambdas, operations before the stage loop, in it, after it)}"""
    text = re.sub(r"//.*", "", SRC.read_text())
    text = text[text.index("if (!output_group) {"):]
    chain, end = _block(text, 0)
    output, _ = _block(text, end)
    groups = {}
    for name, body in (("chain", chain), ("output", output)):
        lambdas = {}
        for lam in ("issue_first", "form_m1", "issue_load", "issue", "half_sync"):
            at = body.find(f"auto {lam} = ")
            if at >= 0:
                inner, stop = _block(body, at)
                lambdas[lam] = _ops(inner) if lam in ("issue_first", "form_m1") else []
                body = body[:at] + body[stop:]
        loop = body.index("for (int s = s_lo;")
        inner, stop = _block(body, loop)
        groups[name] = (lambdas, _ops(body[:loop]), _ops(inner), _ops(body[stop:]))
    return groups


def _value(expr, env):
    expr = expr.replace("&&", " and ").replace("||", " or ").replace("(int)", "").replace("/", "//")
    return eval(expr, {"__builtins__": {}}, env)  # noqa: S307  (the kernel's own index arithmetic)


def _warp(group, w, program):
    """The operations of one warp over an item of STAGES stages: ("wait", barrier, phase) | ("arrive", barrier) | ("sync", id, warps)."""
    lambdas, before, loop, after = program[group]
    bars = {m: i << 16 for i, m in enumerate(("bar_full", "bar_pub", "bar_done", "bar_state", "bar_parts", "bar_zq", "bar_z", "bar_h", "bar_w1", "bar_w2", "bar_m1"))}
    consts = {"MLP_NST": NST, "warp": w, "half": w >> 2, "w_moves": True, "s_lo": 0, "s_hi": STAGES - 1, **bars}

    def run(ops, n, s):
        env = {**consts, "n": n, "s": s, "par": n & 1, "slot": n % NST, "more": s < STAGES - 1}
        for cond, op, args in ops:
            if cond is not None and "w_fail" not in cond and not _value(cond, env):
                continue
            if op == "wait_for":
                assert args[1].endswith("& 1"), args
                yield "wait", _value(args[0], env), _value(args[1][:-3], env)
            elif op == "mbar_arrive_warp":
                yield "arrive", _value(args[0], env)
            elif op == "half_sync":
                yield "sync", f"{group} half {w >> 2}", 4
            elif op.startswith("mlp_group_sync"):
                yield "sync", op, 8
            elif op == "issue":  # a commit, taken as done
                if w & 3 == int(args[0]):
                    yield "arrive", _value(args[1], env)
            elif op == "issue_load":
                if 2 <= w < 6 and ("s + 2" not in args[1] or s + 2 < STAGES):
                    yield "arrive", bars["bar_full"] + 8 * (_value(args[0], env) % NST)
            else:
                n2, s2 = _value(args[0], env), _value(args[1], env)
                if s2 < STAGES:
                    yield from run(lambdas[op], n2, s2)

    yield from run(before, 0, 0)
    for s in range(STAGES):
        yield from run(loop, s, s)
    yield from run(after, STAGES, STAGES)


def _arrivals(barrier):
    """What completes a phase: the four loads of a slot, one warp for M1', a commit of each half for products, else a group's eight warps."""
    return {0: 4, 10: 1}.get(barrier >> 16, 2 if 5 <= barrier >> 16 <= 9 else 8)


def _simulate(warps, held, at):
    """Runs all warps, `held` not beyond its operation `at` until nothing else can move; returns what went wrong, if anything."""
    pos = [0] * len(warps)
    count, phase, syncs, passed = {}, {}, {}, {}
    free = False
    while True:
        moved = False
        for i, ops in enumerate(warps):
            while pos[i] < len(ops) and (free or i != held or pos[i] < at):
                op = ops[pos[i]]
                if op[0] == "wait":
                    done = phase.get(op[1], 0)
                    if done != op[2] + 1:
                        if done > op[2] + 1 or (done & 1) != (op[2] & 1):
                            return f"warp {i} waits for phase {op[2]} of barrier {op[1] >> 16}, which is in phase {done}"
                        break
                elif op[0] == "arrive":
                    count[op[1]] = count.get(op[1], 0) + 1
                    if count[op[1]] == _arrivals(op[1]):
                        count[op[1]] = 0
                        phase[op[1]] = phase.get(op[1], 0) + 1
                else:
                    k = passed.get((i, op[1]), 0)
                    here = syncs.setdefault((op[1], k), set())
                    here.add(i)
                    if len(here) < op[2]:
                        break
                    passed[i, op[1]] = k + 1
                pos[i] += 1
                moved = True
        if not moved:
            if all(p == len(o) for p, o in zip(pos, warps)):
                return None
            if free:
                return f"stuck at {[o[p] if p < len(o) else None for p, o in zip(pos, warps)]}"
            free = True


def test_every_barrier_operation_is_in_the_model():
    program = _program()
    counted = {g: {op: sum(o[1] == op for o in program[g][2]) for op in ("wait_for", "mbar_arrive_warp", "issue")} for g in program}
    assert counted["chain"]["issue"] == 4 and counted["chain"]["wait_for"] >= 7 and counted["output"]["wait_for"] >= 4, counted
    text = re.sub(r"//.*", "", SRC.read_text())
    text = text[text.index("if (!output_group) {"):]
    modelled = sum(len(part) for g in program.values() for part in [*g[0].values(), *g[1:]])
    written = sum(len(re.findall(rf"\b{op}\(", text)) for op in ("wait_for", "mbar_arrive_warp", r"mlp_group_sync<\d>", "half_sync", "issue", "issue_first", "form_m1", "issue_load"))
    assert modelled == written


@pytest.mark.parametrize("held", range(16))
def test_a_warp_held_up_anywhere_finds_its_phase(held):
    program = _program()
    warps = [list(_warp("chain" if i < 8 else "output", i & 7, program)) for i in range(16)]
    for at in range(len(warps[held])):
        wrong = _simulate(warps, held, at)
        assert wrong is None, f"held before its operation {at}, {warps[held][at]}: {wrong}"


def test_products_end_before_tensor_memory_is_freed():
    """When a wait ran out nobody waits for the products behind it: on the way out every warp that issues products commits them once
    more, and the warp that frees tensor memory waits for all those commits."""
    text = re.sub(r"//.*", "", SRC.read_text())
    issuing = {int(i) for i in re.findall(r"\bissue\((\d),", text)}
    out = text[text.index("if (lds_word(w_fail) != 0u) break;"):text.index("tmem_dealloc(")]
    commit = re.search(r"if \(!output_group && \(warp & 3\) < (\d)\) \{\s*if \(elect_one\(\)\) umma_commit_to\((\w+)\);", out)
    assert commit and issuing == set(range(int(commit[1]))), issuing
    wait = re.search(rf"if \(threadIdx\.x < 32\) mbar_wait_bounded\({commit[2]}, 0\);", out)
    assert wait and commit.end() < wait.start()
    assert re.search(rf"mbar_init\({commit[2]}, {2 * len(issuing)}\);", text)  # (both halves of the hidden features)
