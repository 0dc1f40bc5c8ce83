"""How the three warpgroups of prompt attention at D = 256 wait for one another (csrc/prefill_attn.cu: m_ready, l_ready): the barriers and
parities as the source states them, in every order in which a quarter's three warps can go on.  A parity tells a phase from its
neighbours only, so nobody may be two phases ahead of somebody who has not looked yet."""
import itertools
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llmq_b200", "csrc", "prefill_attn.cu")
GROUPS, SW = 3, 12


def expressions():
    """(barrier, parity) of the waits and the barrier of the arrivals, as code in x, g, last, wg, i, quarter"""
    with open(SOURCE) as f:
        text = re.sub(r"//[^\n]*", "", f.read())

    def code(c):
        return compile(re.sub(r"\(uint32_t\)|(?<=\d)u\b", "", c).replace("/", "//"), c, "eval")

    found = {}
    for name in ("m_ready", "l_ready"):
        found[name] = ([(code(b), code(p)) for b, p in re.findall(r"\bwait\(%s \+ (.*?), (.*?)\);" % name, text)],
                       [code(b) for b in re.findall(r"mbar_arrive\(%s \+ (.*?)\);" % name, text)])
    (step, end), (mine,) = found["m_ready"]
    (sums,), (given,) = found["l_ready"]
    return {"step": step, "end": end, "mine": mine, "sums": sums, "given": given}


def program(wg, runs, e, quarter=1):
    """what a warp does, as (barrier, parity, arrivals that it means) for a wait and (barrier,) for an arrival"""
    ops, s_count = [], 0
    arrivals = {}                   # (by all warpgroups, as the order of the steps has it)

    def at(c, **names):
        return eval(c, {"GROUPS": GROUPS, "SW": SW, "wg": wg, "quarter": quarter, **names})

    for x, steps in enumerate(runs):
        for j in range(steps):
            g = s_count + j
            owner = g % GROUPS
            if owner == wg:
                if j > 0:
                    ops.append((("m", at(e["step"][0], g=g)), at(e["step"][1], g=g), arrivals[(g - 1) % GROUPS]))
                ops.append((("m", at(e["mine"], g=g)),))
            arrivals[owner] = arrivals.get(owner, 0) + 1
        s_count += steps
        last = s_count - 1
        if last % GROUPS != wg:
            ops.append((("m", at(e["end"][0], last=last)), at(e["end"][1], last=last), arrivals[last % GROUPS]))
        ops.append((("l", at(e["given"], x=x)),))
        for i in range(GROUPS):
            ops.append((("l", at(e["sums"][0], x=x, i=i)), at(e["sums"][1], x=x), None))
    return ops


@pytest.mark.parametrize("runs", list(itertools.product((1, 2, 3, 4), repeat=4)) + [(1,) * 7, (2,) * 7, (1, 2, 1, 1, 5, 1, 2)])
def test_every_order_ends(runs):
    e = expressions()
    programs = [program(wg, runs, e) for wg in range(GROUPS)]
    seen, todo = set(), [(0,) * GROUPS]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        phases = {}
        for wg in range(GROUPS):
            for op in programs[wg][:state[wg]]:
                if len(op) == 1:
                    phases[op[0]] = phases.get(op[0], 0) + 1
        on = 0
        for wg in range(GROUPS):
            if state[wg] == len(programs[wg]):
                continue
            op = programs[wg][state[wg]]
            if len(op) > 1:
                done = phases.get(op[0], 0)
                if done % 2 == op[1]:       # (the phase of this parity is not over)
                    continue
                assert op[2] is None or done == op[2], (state, op)
            on += 1
            todo.append(state[:wg] + (state[wg] + 1,) + state[wg + 1:])
        assert on or all(state[wg] == len(programs[wg]) for wg in range(GROUPS)), \
            f"run {runs}: warps stop at {[programs[wg][state[wg]:][:1] for wg in range(GROUPS)]}"
