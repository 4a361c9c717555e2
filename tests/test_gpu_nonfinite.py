"""A density that is not finite stays where the equations put it: a particle
whose only neighbours lie outside the boundary rows has empty sums in the
boundary pass, whatever its own density."""
import numpy as np
import pytest

import zsph_b200 as z
from oracle import pyoracle as po
from zsph_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
@pytest.mark.parametrize("precise", [False, True], ids=["plain", "precision"])
def test_boundary_sums_of_a_particle_without_boundary_neighbours(value, precise):
    c = cases.random_cloud(150, 3)
    o = po.Oracle(c.json, c.state, np.float32)
    o.search()
    nb, ng = o.neighbor_count("new", "boundary"), o.neighbor_count("new", "governing")
    slots = np.where((nb == 0) & (ng > 0))[0]
    walls, fluid = (slots[o.new["type"][slots] == t] for t in (0, 1))
    assert len(walls) and len(fluid)
    slots = np.array([walls[0], fluid[0]])
    c.state.rhop[o.tmp["index"][slots], 0] = value
    o = po.Oracle(c.json, c.state, np.float32)
    o.search()
    o.boundary("new")
    assert not o.tmp["dofv_grandrho"][slots].any()
    sol = z.Solver.from_case(c)
    if precise:
        sol.set_precision(True, c.state.pos.astype(np.float64))
    sol.neighbor_search("old", "new")
    sol.boundary("new")
    got = sol.download_tmp()["dofv_grandrho"]
    assert np.array_equal(got[slots], np.zeros((2, 4), np.float32))
    assert np.array_equal(np.isfinite(got), np.isfinite(o.tmp["dofv_grandrho"]))
    sol.close()
