"""Properties of the CUDA sources that no run on a healthy GPU can show."""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "himuon_b200" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _loops(code):
    """Bodies of all braced for / while loops."""
    for m in re.finditer(r"\b(?:for|while)\s*\(", code):
        i, depth = m.end(), 1
        while depth:                                     # the closing parenthesis of the header
            depth += {"(": 1, ")": -1}.get(code[i], 0)
            i += 1
        while code[i].isspace():
            i += 1
        if code[i] != "{":
            continue
        start, depth = i, 0
        while True:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            i += 1
            if depth == 0:
                break
        yield code[start:i]


def _functions_with_named_barriers():
    names = set()
    for path in CSRC.glob("*.cuh"):
        code = _code(path)
        heads = [(m.start(), m.group(1)) for m in re.finditer(r"__device__[^;{]*?\b(\w+)\s*\([^;{]*\)\s*\{", code)]
        for (at, name), (end, _) in zip(heads, heads[1:] + [(len(code), "")]):
            if re.search(r"\bnamed_barrier\(", code[at:end]):
                names.add(name)
    return names


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_no_unbounded_barrier_in_a_loop_that_threads_leave_one_by_one(name):
    """A thread leaves such a loop by itself when its bounded wait runs out; a named barrier in the same loop (or in a
    function called there) would keep the other threads waiting for it for good."""
    barriers = "|".join(sorted({"named_barrier"} | _functions_with_named_barriers()))
    for body in _loops(_code(CSRC / name)):
        if re.search(r"if \(!mbar_wait\(", body) and "break;" in body:
            assert not re.search(rf"\b(?:{barriers})\s*(?:<[^;()]*>)?\(|\bbar\.sync\b", body), body[:400]
