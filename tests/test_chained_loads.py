"""Kernels launched by launch_chained may be resident while the kernels in
front of them still write what they read, so neither they nor any device
function they call may read through __ldg or a __restrict__ pointer (the
read-only path is for memory nobody writes while the kernel is resident, and
griddepcontrol.wait does not order it)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "polysplat_gb300", "csrc")
KEYWORDS = {"if", "for", "while", "switch", "return", "sizeof", "decltype", "alignas", "asm", "static_assert"}


def _source(path):
    with open(path) as f:
        s = f.read()
    s = re.sub(r"/\*.*?\*/", "", s, flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


def _functions(s):
    """name -> [signature and body] of every function defined in `s`."""
    out = {}
    for m in re.finditer(r"\b([A-Za-z_]\w*)\s*\(", s):
        if m.group(1) in KEYWORDS:
            continue
        at, depth = m.end(), 1
        while at < len(s) and depth:
            depth += {"(": 1, ")": -1}.get(s[at], 0)
            at += 1
        tail = re.match(r"\s*(const\b)?\s*\{", s[at:])
        if not tail:
            continue
        end, depth = at + tail.end(), 1
        while end < len(s) and depth:
            depth += {"{": 1, "}": -1}.get(s[end], 0)
            end += 1
        out.setdefault(m.group(1), []).append(s[m.start():end])
    return out


FILES = {p: _source(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")))}
HEADERS = [_source(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")))]


def _chained():
    found = []
    for path, s in FILES.items():
        for m in re.finditer(r"launch_chained\(\s*(\w+)", s):
            names = [m.group(1)]
            if not names[0].startswith("k_"):  # a local holding the kernel, or one of several
                held = re.findall(r"\bauto\s+%s\s*=([^;]*);" % m.group(1), s[:m.start()])
                names = re.findall(r"\bk_\w+", held[-1])
            found += [(path, n) for n in names]
    return sorted(set(found))


def test_the_chain_is_found():
    names = {n for _, n in _chained()}
    assert {"k_emit_massive", "k_upsweep", "k_pass", "k_ranges_exact", "k_quad_starts", "k_quad_tiles",
            "k_quad_expand", "k_blend", "k_read_status"} <= names


@pytest.mark.parametrize("path,kernel", _chained(), ids=lambda v: os.path.basename(str(v)))
def test_chained_kernels_load_plainly(path, kernel):
    known = _functions(FILES[path])
    for h in HEADERS:
        for name, bodies in _functions(h).items():
            known.setdefault(name, []).extend(bodies)
    todo, seen = [kernel], set()
    while todo:
        name = todo.pop()
        if name in seen:
            continue
        seen.add(name)
        for body in known.get(name, []):
            assert "__ldg" not in body, "%s, reached from %s, reads through __ldg" % (name, kernel)
            assert "__restrict__" not in body.split("{")[0], "%s, reached from %s" % (name, kernel)
            todo += [n for n in re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^;(){}]*>)?\s*\(", body) if n in known]
    assert kernel in known
