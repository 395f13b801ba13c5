"""Warp-collective instructions of the kernels are reached by whole, converged warps.

``tcgen05.ld / .st / .wait / .alloc / .dealloc`` and the cluster barrier are ``.sync.aligned``: all lanes of a warp have to execute
them together.  A poll of an mbarrier that every lane runs for itself, or a branch that one lane takes, leaves the lanes apart until
something brings them together (``__syncwarp``, a vote, a block barrier).  On hardware this fails rarely and as a launch
failure, so it is checked in the source: the kernels are read in program order, loop bodies twice."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "torchure_b200" / "csrc"
KERNELS = sorted(p.name for p in CSRC.glob("*.cu") if "tmem_" in p.read_text())

APART = r"\bmbar_wait\(|\belect_one\(\)|if \(lane == 0\b"
TOGETHER = r"\bmbar_wait_warp\(|__syncwarp\(|__syncthreads\(|__all_sync\(|__any_sync\(|\} else if \(warp|\n  \} else \{"    # else: another warp's role
COLLECTIVE = r"\btmem_(?:ld|st|alloc|dealloc|relinquish)\w*\(|\bcluster_sync_all\(\)"
TOKEN = re.compile(f"(?P<apart>{APART})|(?P<together>{TOGETHER})|(?P<collective>{COLLECTIVE})|(?P<loop>\\bfor \\()|(?P<line>\n)")


def _closing(text, at, pair="{}"):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def _walk(text, apart, line, found):
    """What separated the lanes last (None: together) after ``text``; collectives reached that way are added to ``found``."""
    at = 0
    while m := TOKEN.search(text, at):
        at = m.end()
        kind = m.lastgroup
        if kind == "line":
            line += 1
        elif kind == "apart":
            apart = f"{m.group()} in line {line}"
        elif kind == "together":
            apart = None
        elif kind == "collective":
            if apart:
                found.add(f"line {line}: {m.group()} behind {apart}")
        else:
            head = _closing(text, m.end() - 1, "()") + 1
            line += text.count("\n", m.start(), head)
            if text[head:].lstrip(" ").startswith("{"):
                begin = text.index("{", head)
                end = _closing(text, begin)
                for _ in range(2):
                    apart = _walk(text[begin + 1:end], apart, line, found)
                line += text.count("\n", begin, end)
                at = end
            else:
                at = head
    return apart


def _code(name):
    """The file without comments and without the definitions of device helpers that stand before its first kernel."""
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


@pytest.mark.parametrize("name", KERNELS)
def test_collectives_are_reached_by_converged_warps(name):
    text, found = _code(name), set()
    for m in re.finditer(r"\n(?:__global__|__device__ __forceinline__) [^;{]*\{", text):
        begin = m.end() - 1
        _walk(text[begin + 1:_closing(text, begin)], None, text.count("\n", 0, begin) + 1, found)
    assert not found, "\n".join(sorted(found))


def test_whole_warps_do_not_poll_lane_by_lane():
    """Outside the one-lane roles every wait is the warp's."""
    for path in CSRC.glob("*.cu"):
        text = _code(path.name)
        one_lane = [(m.end(), _closing(text, text.index("{", m.end()))) for m in re.finditer(r"elect_one\(\)\)", text)]
        for m in re.finditer(r"\bmbar_wait(_warp)?\(", text):
            inside = any(a < m.start() < b for a, b in one_lane)
            assert inside != bool(m.group(1)), f"{path.name}:{text.count(chr(10), 0, m.start()) + 1}"


def test_named_barriers_take_whole_warps():
    """``bar.sync`` is aligned too; it stands in one helper, behind a ``__syncwarp``."""
    for path in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        text = _code(path.name)
        for m in re.finditer(r'"bar\.(?:sync|arrive)', text):
            body = text[text.rindex("{", 0, m.start()):m.start()]
            assert path.name == "common.cuh" and "__syncwarp();" in body, f"{path.name}: {m.group()}"


def test_the_check_sees_a_lane_that_is_apart():
    found = set()
    _walk("for (int i = 0; i < n; ++i) {\n tmem_ld_wait();\n if (lane == 0) store();\n}", None, 1, found)
    assert found == {"line 2: tmem_ld_wait( behind if (lane == 0 in line 3"}
