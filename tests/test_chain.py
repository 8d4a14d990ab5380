"""Launches chained by programmatic stream serialisation start beside the end of the kernel before
them. Every kernel launched so has to wait for that kernel before it touches memory: its first
statement is chain_wait(). The point pass of the pressure solves waits after reading what no pass
writes; whatever follows it is launched the plain way (the host code says so at those launches)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aturan_b200", "csrc")
FILES = [f for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh")) and f != "noalloc.cu"]
LATE = {"sor_colour_kernel"}                                  # waits further down


def _code(f):
    s = open(os.path.join(CSRC, f)).read()
    return re.sub(r"//[^\n]*", "", s)


def _launched():
    return {m for f in FILES for m in re.findall(r"chain(?:_if)?\(\s*(?:[^;]*?,\s*)?(\w+_kernel|kern)\b", _code(f))}


@pytest.mark.parametrize("f", FILES)
def test_every_chained_kernel_waits_first(f):
    s, launched = _code(f), _launched()
    for m in re.finditer(r"__global__", s):
        i, d = m.end(), 0
        while not (s[i] == "{" and d == 0):
            d += (s[i] == "(") - (s[i] == ")")
            i += 1
        name = re.search(r"(\w+_kernel)\s*\(", s[m.start():i]).group(1)
        body = s[i + 1:i + 4000]
        if name in LATE:
            assert 0 < body.find("chain_wait();") < body.find("oth + o[q]")
        elif body.lstrip().startswith("chain_wait();"):
            continue
        else:
            assert name not in launched, name
