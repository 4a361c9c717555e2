"""Rules of the kernels that no run can show reliably, checked in their
sources and in the compiler's report: what a kernel reads must stay behind the
wait for the kernel that wrote it, and dispatch rules count the CTAs that fit."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zsph_b200", "csrc")
SOURCES = {os.path.basename(p): re.sub(r"//[^\n]*", "", open(p).read())
           for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def _body(text, start):
    """The brace block that opens first at or after `start`."""
    a = text.index("{", start)
    depth = 0
    for k in range(a, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[a + 1:k]
    raise AssertionError("unbalanced braces")


def _kernels():
    """name -> body of every __global__ function."""
    out = {}
    for text in SOURCES.values():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\s*\(", text):
            out[m.group(1)] = _body(text, text.index(")", m.end()))
    return out


def test_inline_loads_are_volatile():
    """An asm load that is not volatile may move above griddepcontrol.wait or a grid barrier."""
    for name, text in SOURCES.items():
        for m in re.finditer(r"\basm\s*(volatile)?\s*\(", text):
            statement = text[m.start():text.index(";\n", m.end())]
            if re.search(r"\b(ld|ldmatrix|red|atom)\.", statement):
                assert m.group(1), (name, statement[:80])


def test_programmatic_kernels_wait_first():
    """A kernel launched while its predecessor drains touches no memory before pdl_wait()."""
    launched = set()
    for text in SOURCES.values():
        for m in re.finditer(r"\blaunch_pdl\(([^;]*?);", text):
            launched |= set(re.findall(r"\bk_\w+", m.group(1)))
    kernels = _kernels()
    assert len(launched) >= 10 and launched <= set(kernels)
    for name in launched:
        first = [s.strip() for s in kernels[name].split(";") if not s.strip().startswith("__shared__")][0]
        assert first == "pdl_wait()", (name, first)


def test_every_search_empties_the_wall_list():
    """A step that ended between a list build and the pass after it (a bounded
    barrier that ran out) leaves wall-list entries behind, which must not reach
    the lists of a new order; no call can be made to end there, so the sources
    are read: the last kernel of either search empties the list, as the
    persistent step does, and the wall pass leaves fluid records alone."""
    kernels = _kernels()
    for name in ("k_rank_gather", "k_gather_by_index", "k_batch_persistent"):
        assert re.search(r"misc\[kMiscWalls\]\s*=\s*0;", kernels[name]), name
    text = SOURCES["equations.cu"]
    body = _body(text, text.index("void walls_block("))
    assert "fluid_of(own.pr.w)" in body[:body.index("wall_sums<")]


def test_governing_budgets_fit_the_dispatch_rule():
    """The rule that takes six CTAs per SM counts five of the plain and the 5x5
    pass at the compiler's registers, and four of the precision form's: the
    build's own report must bear that out."""
    report = os.path.join(CSRC, "..", "_build", "equations.cu.o.ptxas.txt")
    if not os.path.exists(report):
        pytest.skip("no compiler report (the library was built elsewhere)")
    text = open(report).read()
    regs = {m.group(1): int(m.group(2)) for m in
            re.finditer(r"Compiling entry function '\w*k_governingI(\w+?)EEv\w*'.*?Used (\d+) registers", text, re.S)}

    def ctas(gf, mode, precise, minb):
        key = f"Li{gf}ELi{mode}ELb0ELb{precise}ELb0ELb0ELi{minb}ELb0E"
        return 65536 // (128 * -(-regs[key] // 8) * 8)

    for mode in (0, 1, 2):
        for gf, precise, fit in ((1, 0, 5), (2, 0, 5), (1, 1, 4)):
            assert ctas(gf, mode, precise, 1) == fit, (gf, mode, precise)
            assert ctas(gf, mode, precise, 6) == 6, (gf, mode, precise)
