"""The precision form's step in the range of sizes whose governing pass takes
six CTAs per SM (75,777 to 113,664 particles on 148 SMs) and on either side."""
import dataclasses

import numpy as np
import pytest

import zsph_b200 as z
from oracle import pyoracle as po
from zsph_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx", [0.0235, 0.02, 0.0195])
def test_precision_step_matches_fp64_oracle(dx):
    """One step.  Tolerance: tests/test_gpu_precise.py's of the same comparison
    (1e-5 and 1e-3 after 60 steps)."""
    c = cases.dam_break(dx)
    pos64 = c.pos64 if c.pos64 is not None else c.state.pos.astype(np.float64)
    o = po.Oracle(c.json, dataclasses.replace(c.state, pos=pos64), dtype=np.float64)
    o.step(1)
    sol = z.Solver.from_case(c)
    sol.set_precision(True, pos64)
    sol.run(1)
    assert sol.status() == 0
    st, x = sol.download("old"), sol.positions64()
    sol.close()
    a, b = (np.argsort(t + np.arange(c.n)) for t in (st.table, o.old["table"]))
    assert np.abs(x[a] - o.old["pos"][b]).max() < 1e-5
    assert np.abs(st.vel[a] - o.old["vel"][b]).max() < 1e-3
