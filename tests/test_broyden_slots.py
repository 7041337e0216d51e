"""Workspace of the charge mixing (common.cuh: broyden_slots; scc.cu: stage_mix), CPU only: over every
iteration of the fallback ladder's Broyden rungs (the first, and the last with at least 250 iterations) the
active vectors have slots of their own and the linear system fits the slots squared."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfn1-rs_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return fh.read()


def _slots(size, max_scc):
    """The batch's slots as capi.cu computes them."""
    line = re.search(r"b->cap = ([^;]*);", _source("capi.cu")).group(1)
    last = int(re.search(r"constexpr int kLastRungScc = (\d+);", _source("common.cuh")).group(1))
    assert line == "broyden_slots(o.scc_broyden_size, o.max_scc)"
    text = _source("common.cuh")
    body = text[text.index("inline int broyden_slots("):]
    env = {"broyden_size": size, "max_scc": max_scc, "kLastRungScc": last}
    for m in re.finditer(r"(?:const int (\w+) =|return) (\w+) ([<>]) (\w+) \? (\w+) : (\w+);", body[:body.index("\n}")]):
        name, a, op, b, x, y = m.groups()
        v = lambda t: int(t) if t.isdigit() else env[t]  # noqa: E731
        env[name or "result"] = v(x) if (v(a) < v(b) if op == "<" else v(a) > v(b)) else v(y)
    return env["result"], last


@pytest.mark.parametrize("size", [0, 1, 2, 3, 8, 16, 17, 64, 250, 400])
@pytest.mark.parametrize("max_scc", [1, 2, 3, 6, 15, 17, 100, 249, 250, 251, 600])
def test_active_vectors_fit(size, max_scc):
    cap, last = _slots(size, max_scc)
    memory = max(size, 2)
    for steps in (max_scc, max(max_scc, last)):
        for itn in {1, 2, 3, memory - 1, memory, memory + 1, memory + 2, steps // 2, steps - 2, steps - 1}:
            if not 1 <= itn <= steps - 1:  # the n-th Broyden step; the last iteration does not mix
                continue
            start = itn - memory + 1 if itn > memory else 1
            active = itn - start + 1
            used = [((start + r - 1) % memory) % cap for r in range(active)]
            assert active <= cap and len(set(used)) == active
