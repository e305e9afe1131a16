"""The bounded waits of the kernels, read from their sources: what has to hold so that a wait that runs out ends the kernel with a
status instead of leaving the GPU waiting. (Making one run out in a kernel that is wrong would hang the GPU, so nothing here runs.)"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "axolotl_b200" / "csrc"
WAIT = re.compile(r"\b(?:mbar_wait|mbar_wait_spin|mbar_wait_backoff|mbar_wait_partner|wait_sleeping)\(")
SOURCES = sorted(p.name for p in CSRC.glob("*.cu") if WAIT.search(p.read_text()))


def _code(name):
    text = re.sub(r"//[^\n]*", lambda m: " " * len(m.group()), (CSRC / name).read_text())
    return re.sub(r"/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text, flags=re.S)


def _waits(code):
    """(position, headers of the enclosing blocks, start of the outermost one) of every wait that is called, not defined."""
    stack, last = [], 0
    calls = {m.start() for m in WAIT.finditer(code)}
    for i, c in enumerate(code):
        if i in calls:
            if not code[last:i].strip().endswith("bool") and "bool mbar_wait" not in "".join(h for h, _ in stack):
                yield i, [h for h, _ in stack], next((at for h, at in stack if not re.match(r"\s*(extern|namespace)", h)), 0)
        if c == "{":
            stack.append((code[last:i].strip(), i))
            last = i + 1
        elif c == "}":
            stack.pop()
            last = i + 1
        elif c == ";":
            last = i + 1


@pytest.mark.parametrize("name", SOURCES)
def test_a_wait_ends_the_same_way_for_all_lanes_of_a_warp(name):
    """tcgen05.ld, elect.sync and __syncwarp wait for every lane of the warp, without a limit: unless a single lane walks the loop, the
    outcome of a wait is agreed on (warp_all) before anything depends on it."""
    code = _code(name)
    for at, headers, start in _waits(code):
        line = code.count("\n", 0, at) + 1
        statement = code[max(code.rfind(c, 0, at) for c in ";{}") + 1:at]
        held = re.search(r"(\w+) = (?:\w+ && )?$", statement)
        rest = code[at:at + 400]
        agreed = "warp_all(" in statement or (held and re.search(r"warp_all\(%s\)" % held.group(1), rest))
        if held and re.search(r"(\w+) = \1 && $", statement):      # remembered: nothing branches on it until the warp agrees
            agreed = re.search(r"\b(?:if|while|for) \([^{;]*\b%s\b" % held.group(1), code[at:]).group().startswith("if (warp_all(")
            agreed = agreed and not any(re.match(r"(if|while|for) \(.*\b%s\b" % held.group(1), h) for h in headers[-1:])
        one_lane = any("lane == 0)" in h or "elect_one()" in h for h in headers) or "lane != 0) return;" in code[start:at]
        assert agreed or one_lane, f"{name}:{line}: lanes of a warp may leave this wait on different ways"


@pytest.mark.parametrize("name", [n for n in SOURCES if "bar.sync" in _code(n)])
def test_a_warp_that_gives_up_still_meets_its_group(name):
    """A named barrier has no limit: a warp never leaves a loop with one because a wait ran out. Its lanes remember that and walk on."""
    code = _code(name)
    loops = 0
    for m in re.finditer(r"\bfor \(", code):
        depth, i = 0, code.index("{", m.end())
        body = i
        if ";" in re.sub(r"\([^()]*\)", "", code[m.start():i].split(")", 1)[-1]):     # a loop without braces
            continue
        while True:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
            if not depth:
                break
        block = code[body:i]
        if "bar.sync" not in block or not WAIT.search(block):
            continue
        loops += 1
        assert not re.search(r"\n\s*(break|return);", block), name                    # (those of a switch stand on its lines)
        assert "ok" not in re.findall(r"\w+", code[m.start():body]), name
        for w in WAIT.finditer(block):
            assert re.search(r"(ok = ok && |if \(!dead\) dead = !warp_all\()$", block[:w.start()]), name
    assert loops


def test_arrivals_on_another_cta_have_cluster_scope():
    """The default scope of mbarrier.arrive is the CTA: on the partner's barrier it would order nothing that the arriving CTA wrote
    before what the other one does. What such an arrival stands for has to be acquired at that scope too."""
    for name in sorted(p.name for p in CSRC.glob("*.cu*")):
        for m in re.finditer(r"mbarrier\.arrive[\w.:]*\.shared::cluster[\w.:]*", _code(name)):
            assert re.search(r"\.(release|relaxed)\.cluster\.", m.group()), f"{name}: {m.group()}"
    w4a16 = _code("grouped_w4a16.cu")
    for bar in ("w_full", "tempty_bar"):          # what the partner's converters and epilogue signal
        waits = re.findall(r"\b(mbar_\w+|wait_\w+)\(&%s\[" % bar, w4a16)
        assert [w for w in waits if "wait" in w] == ["mbar_wait_partner"], (bar, waits)
