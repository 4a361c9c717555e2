"""The list-reuse corrector's wall pass where walls' lists are past their
capacity (it filters their rows again), in both of its lane counts."""
import numpy as np
import pytest

import zsph_b200 as z
from oracle import pyoracle as po
from zsph_b200 import cases

pytestmark = pytest.mark.gpu


# 20,628 and 311,396 particles: 8 and 2 lanes per wall
@pytest.mark.parametrize("dx", [0.04, 0.013])
def test_reuse_walls_with_overflowed_lists(dx):
    """Fluid squeezed to half its spacing in the floor's corner.  The plain
    corrector is the reference: the two differ in the order of their sums, of
    at most some 300 FP32 terms (300 * 6e-8 = 2e-5 of the field's scale), and
    in pairs that crossed 2h within a half step, where the kernel vanishes.
    The bound is the kernel tests' 1e-4."""
    c = cases.dam_break(dx)
    p, k = c.state.pos, 0.04 / dx
    m = (c.state.type == 1) & (p[:, 0] < 0.3 / k) & (p[:, 1] < 0.3 / k) & (p[:, 2] < 0.5 / k)
    p[m, 0] *= 0.5
    p[m, 2] *= 0.5
    c.state.tmp_pos[:] = p
    o = po.Oracle(c.json, c.state, np.float32)
    o.search()
    assert ((o.neighbor_count("new", "governing") > 128) & (o.new["type"] != 1)).any()
    got = []
    for reuse in (False, True):
        sol = z.Solver.from_case(c)
        if reuse:
            sol.run_learned(None, 1, judge_every=0, corrector=z.CORR_REUSE_FRESH)
        else:
            sol.step()
        assert sol.status() & z.FLAG_NB_OVERFLOW
        st = sol.download("old")
        order = np.argsort(st.table + np.arange(c.n))
        got.append({a: getattr(st, a)[order] for a in ("pos", "vel", "rhop")})
        sol.close()
    for a in ("pos", "vel", "rhop"):
        want = got[0][a].reshape(c.n, -1)
        scale = np.abs(want).max(0)
        assert np.all(np.abs(got[1][a].reshape(c.n, -1) - want).max(0) <= 1e-4 * scale), a
