"""Launches chained by programmatic serialisation (common.cuh): what a kernel that starts beside the end of
the one before it may and may not do, read from the sources.

* Every kernel waits first, whether its launch names it or a variable does; the point pass of the pressure
  solves, which waits further down, and the few kernels launched the plain way are listed.
* The launches that may follow a point pass are chained only to another point pass.
* What a launch writes is read by plain loads. The read-only path (__ldg, or a const pointer with
  __restrict__) is not held back by the wait: it is for the tables formed with the context, for what the
  point pass reads before its wait, and (ldr) for two kernels launched the plain way."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aturan_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
LATE = {"sor_colour_kernel"}
PLAIN = {"mca_H_kernel", "gs_hyperplane_kernel", "static_weights_kernel"}
# the tables' elements, the split right-hand side the point pass reads before its wait, ldr itself
READ_ONLY = (r"tab \+", r"&w->", r"&w\[", r"R2 \+", r"p\); \}")
# the kernels that read by ldr, and the functions only they call
LDR = {"rk_stage_kernel", "adj_stage_kernel"}
LDR_LOADS = {"load7c", "load_acc_nc", "load_momentum"}


def _code(f):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())


def _kernels():
    for f in FILES:
        s = _code(f)
        for m in re.finditer(r"__global__", s):
            i, d = m.end(), 0
            while not (s[i] == "{" and d == 0):
                d += (s[i] == "(") - (s[i] == ")")
                i += 1
            head = s[m.start():i]
            yield f, re.search(r"(\w+_kernel)\s*\(", head).group(1), head, s[i + 1:i + 400].lstrip()


def _functions(s):
    """(name, body) of the functions at namespace scope."""
    for m in re.finditer(r"\b(\w+)\s*\((?:[^(){};]|\([^()]*\))*\)\s*(?:const\s*)?\{", s):
        if m.group(1) in ("if", "for", "while", "switch"):
            continue
        d, i = 1, m.end()
        while d:
            d += (s[i] == "{") - (s[i] == "}")
            i += 1
        yield m.group(1), s[m.end():i]


def test_every_kernel_waits_first():
    names = set()
    for f, name, _, body in _kernels():
        names.add(name)
        if name not in LATE | PLAIN:
            assert body.startswith("chain_wait();"), (f, name)
    assert LATE | PLAIN <= names and len(names) > 40


def test_kernels_without_a_wait_are_launched_the_plain_way():
    text = "".join(_code(f) for f in FILES)
    for name in PLAIN | LDR:
        assert not re.search(r"chain(?:_if)?\([^;]*\b" + name, text), name
        assert re.search(name + r"(?:<[^;]*?>)?<<<", text), name


def test_only_a_point_pass_is_chained_to_a_point_pass():
    s = _code("api.cu")
    # the pass itself: chained behind the other colour's, or as the caller says
    assert len(re.findall(r"sor_colour_kernel<T, TR>", s)) == 1
    assert "chain_if(chained || colour == 1, sor_colour_kernel<T, TR>" in s
    # every run of sweeps starts unchained, and a merge (plain, to = false) follows it before anything else
    assert len(re.findall(r"sor_sweep<", s)) == 2
    assert "omega, line, n > 0)" in s and "omega, line, n > 0 && !now)" in s
    assert "chain_if(to, sor_split_kernel<T>" in s
    point = [m.start() for m in re.finditer(r"sor_sweep<\w+, TR>\(ctx", s)]
    for at in point:
        rest = s[at:]
        loop_end = rest.index("\n            }\n")
        after = rest[loop_end:loop_end + 400]
        first = re.search(r"\b(chain(?:_if)?\(|sor_\w+(?:<[^>]*>)?\()", after.replace("if(!line){ rc = sor_split(", "sor_split("))
        assert first.group(1).startswith("sor_split("), after
    # the correction in the middle of a run: behind a merge
    mid = s[s.index("if(now){"):]
    assert mid.index("sor_split(") < mid.index("sor_residual<float")


@pytest.mark.parametrize("f", FILES)
def test_the_read_only_path_is_for_tables(f):
    s = _code(f)
    for m in re.finditer(r"__ldg\(", s):
        assert re.match("|".join(READ_ONLY), s[m.end():]), (f, s[m.start():m.start() + 60])
    for name, body in _functions(s):
        if re.search(r"\bldr\(", body):
            assert name in LDR | LDR_LOADS, (f, name)
        if re.search(r"\b(?:" + "|".join(LDR_LOADS) + r")\b(?:<[^>]*>)?\(", body):
            assert name in LDR | LDR_LOADS, (f, name)
    assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", s), f
    assert not re.search(r"ld\.global\.nc|ld\.global\.L1::no_allocate", s), f
