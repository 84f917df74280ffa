"""Asynchronous copies in the kernel sources: every cp.async is committed before
the wait that is meant to cover it.

`cp.async.wait_group` counts committed groups only, so a wait that follows
copies without a commit waits for nothing, and the data is there or not by
timing: no numerical test shows it.  This reads the sources instead.  In each
function, after a copy the next commit or wait in the text must be a commit;
the commit may also stand in a loop that holds the copy and ends before the
wait (the copies of one pass are committed by the next).  Helpers and local
lambdas count as the copies and commits in their bodies.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bsofi_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _strip(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/|\"(?:\\.|[^\"\\])*\"", lambda m: " " * len(m.group()), text,
                  flags=re.S)


def _close(text, i, pair):
    """Index after the bracket that closes the one at i."""
    depth = 0
    while True:
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        i += 1
        if depth == 0:
            return i


def _bodies(text, pattern):
    """(name, start, end) of every brace body whose head matches the pattern."""
    for m in re.finditer(pattern, text):
        i = _close(text, m.end() - 1, "()")
        tail = re.match(r"[\s\w]*\{", text[i:])
        if tail:
            b = i + tail.end() - 1
            yield m.group("name"), b, _close(text, b, "{}")


def _loops(text):
    """Ranges of the bodies of for and while loops."""
    out = []
    for m in re.finditer(r"\b(?:for|while)\s*\(", text):
        i = _close(text, m.end() - 1, "()")
        while text[i].isspace():
            i += 1
        out.append((i, _close(text, i, "{}") if text[i] == "{" else text.index(";", i) + 1))
    return out


FUNCTION = r"(?P<name>[A-Za-z_]\w*)\s*\("
LAMBDA = r"(?P<name>[A-Za-z_]\w*)\s*=\s*\[&\]\s*\("


def _events(text, start, end, known):
    """(position, kind) of the copies, commits and waits between two positions."""
    out = []
    for m in re.finditer(r"\b([A-Za-z_]\w*)\s*(?:<[^;{}()]*>)?\s*\(", text[start:end]):
        for kind in known.get(m.group(1), ()):
            out.append((start + m.start(), kind))
    return out


def uncommitted(text):
    """Line numbers of copies that a wait follows without a commit."""
    text = _strip(text)
    known = {"cp_async16": ["copy"], "cp_async8": ["copy"], "cp_async_commit": ["commit"],
             "cp_async_wait": ["wait"]}
    keep = set(known)
    bodies = [b for b in _bodies(text, FUNCTION) if b[0] not in ("if", "for", "while", "switch")]
    lambdas = list(_bodies(text, LAMBDA))
    for name, b, e in bodies + lambdas:
        if name not in keep:
            kinds = [k for _, k in _events(text, b, e, known)]
            if kinds and "wait" not in kinds:  # a helper: what it leaves behind
                known[name] = [k for i, k in enumerate(kinds) if i == 0 or kinds[i - 1] != k]
    loops, bad = _loops(text), []
    for name, b, e in bodies:
        if name in keep:
            continue
        ev = _events(text, b, e, known)
        for i, (at, kind) in enumerate(ev):
            if kind != "copy":
                continue
            after = next(((p, k) for p, k in ev[i + 1:] if k != "copy"), None)
            if after is None or after[1] == "commit":
                continue
            again = any(s <= at < t and not s <= after[0] < t and
                        any(k == "commit" and s <= p < t for p, k in ev) for s, t in loops)
            if not again:
                bad.append(text.count("\n", 0, at) + 1)
    return bad


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_copies_are_committed_before_their_wait(path):
    with open(path) as f:
        assert uncommitted(f.read()) == []


def test_the_reader_sees_a_missing_commit():
    head = "BSOFI_DEVINL void f(double* a) {\n  for (int i = 0; i < 4; i++) {\n    cp_async16(a, a, 16);\n"
    assert uncommitted(head + "  }\n  cp_async_wait<0>();\n}\n") == [3]
    assert uncommitted(head + "  }\n  cp_async_commit();\n  cp_async_wait<0>();\n}\n") == []
    assert uncommitted(head + "    cp_async_commit();\n  }\n  cp_async_wait<0>();\n}\n") == []
