"""A rule of the device code that can be read off the source: a lane's own answer from an mbarrier (probe or bounded wait)
never decides whether that lane takes part in something the whole warp does.  Lanes may see a phase end at different moments,
and a lane that waits in a vote, shuffle or matrix instruction for one that has gone past it waits without a limit."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "magnitude_b200" / "csrc"
PROBE = re.compile(r"\bmbar_(try|test)_wait\w*|\bmbar_wait_bounded\w*")
TOGETHER = re.compile(r"__(all|any|ballot|shfl\w*|reduce\w*)_sync\s*\(|__sync(warp|threads)\s*\(|\b(i?mma0?|consumers_sync)\s*\(")


def _matching(text, at, opening, closing):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == opening) - (text[i] == closing)
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced source")


def lane_branches(code):
    """(line, body) of every branch or loop whose condition is a lane's own probe, not a vote on it."""
    code = re.sub(r"//[^\n]*", "", code)
    found = []
    for m in re.finditer(r"\b(if|while|for)\s*\(", code):
        end = _matching(code, m.end() - 1, "(", ")")
        condition = code[m.end():end]
        if not PROBE.search(condition) or re.search(r"__(all|any)_sync", condition):
            continue
        rest = code[end:]
        body = rest[:_matching(rest, rest.index("{"), "{", "}")] if rest.lstrip().startswith("{") else rest[:rest.index(";") + 1]
        found.append((code.count("\n", 0, m.start()) + 1, body))
    return found


@pytest.mark.parametrize("path", sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh")), ids=lambda p: p.name)
def test_no_warp_wide_step_behind_a_lanes_own_probe(path):
    for line, body in lane_branches(path.read_text()):
        assert not TOGETHER.search(body), f"{path.name}, branch {line} (comments removed): {body.strip()[:200]}"


def test_the_rule_finds_what_it_is_for():
    bad = "if (!mbar_try_wait(b, p)) {\n if (!__all_sync(mask, mbar_wait_bounded(b, p))) return false;\n}"
    good = "if (!__all_sync(mask, mbar_try_wait(b, p))) {\n ok = __all_sync(mask, mbar_wait_bounded(b, p));\n}"
    assert TOGETHER.search(lane_branches(bad)[0][1])
    assert not lane_branches(good)
