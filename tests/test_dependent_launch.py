"""Kernels launched by launch_after (programmatic dependent launch), read as text.

Such a kernel may start while the one before it still runs.  It has to wait first, and the
compiler may move read-only loads (__ldg, const __restrict__) ahead of that wait unless the pointer
they use is taken after it (launch.cuh): an input read there would be the previous call's.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpurir_gb300", "csrc")


def _functions(text):
    """(name, parameters, body) of the functions defined in a source text without comments."""
    out = []
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        depth, i = 0, m.end() - 1
        while i < len(text):
            depth += (text[i] == "(") - (text[i] == ")")
            i += 1
            if depth == 0:
                break
        end = re.match(r"\s*\{", text[i:])
        if not end or m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            continue
        j = i + end.end()
        depth = 1
        while j < len(text) and depth:
            depth += (text[j] == "{") - (text[j] == "}")
            j += 1
        out.append((m.group(1), text[m.end():i - 1], text[i + end.end():j - 1]))
    return out


def _dependent():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        names = set(re.findall(r"launch_after\(\s*(\w+)", text))
        functions = _functions(text)
        reading = {"__ldg"}   # functions that load by __ldg, or call one that does
        while True:
            more = {n for n, _, body in functions if n not in names and any(re.search(r"\b%s\b" % r, body) for r in reading)}
            if more <= reading:
                break
            reading |= more
        for name, params, body in functions:
            if name in names:
                yield os.path.basename(path), name, params, body, any(re.search(r"\b%s\b" % r, body) for r in reading)


CASES = list(_dependent())


def test_every_kernel_is_found():
    launched = sum(len(set(re.findall(r"launch_after\(\s*(\w+)", open(p).read())))
                   for p in glob.glob(os.path.join(CSRC, "*.cu")))
    assert len(CASES) == launched > 10


@pytest.mark.parametrize("file,name,params,body,reads", CASES, ids=[c[1] for c in CASES])
def test_waits_before_it_reads(file, name, params, body, reads):
    first = re.sub(r"^(\s*(extern\s+)?__shared__[^;]*;)*\s*", "", body)
    assert first.startswith("after_previous();"), "%s: %s does not wait first" % (file, name)
    for p in params.split(","):
        pointer = re.search(r"\bconst\b.*\*\s*(__restrict__)?\s*(\w+)\s*$", p.strip())
        if pointer and (reads or pointer.group(1)):
            x = pointer.group(2)
            assert re.search(r"\b%s = after_wait\(%s\);" % (x, x), body), "%s: %s reads %s ahead of the wait" % (file, name, x)
