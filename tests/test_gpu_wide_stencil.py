"""The 5x5 stencil (grid_size_factor 2: cells of side h) on the GPU: neighbour
lists, the wall, boundary and governing passes and whole steps against the CPU
oracle.  Tolerances: tests/test_gpu_equations.py's, stated there."""
import numpy as np
import pytest

import zsph_b200 as z
from oracle import pyoracle as po
from zsph_b200 import cases
from tests.helpers import condition_walls
from tests.test_gpu_equations import _by_id, _close, _sorted_pair, err_norms

pytestmark = pytest.mark.gpu


def _wide(c):
    """The case with cells of side h."""
    c.json.grid_size_factor = 2.0
    return c


# dam_break(0.02): 105,048 particles, inside the range that takes the six-CTA governing budget
@pytest.mark.parametrize("mk", [lambda: _wide(cases.small(0.06)), lambda: _wide(cases.small(0.04)),
                                lambda: _wide(cases.random_cloud(31, 4, box=(0.2, 0.2, 0.2))),
                                lambda: _wide(cases.random_cloud(2500, 2)), lambda: _wide(cases.config0())],
                         ids=["dam_6k", "dam_20k", "cloud_31", "cloud_2500", "dam_105k"])
def test_passes_match_oracle(mk):
    c = condition_walls(mk())
    sol, o32, o64 = _sorted_pair(c)
    nb_b, nb_g = sol.neighbor_counts("new")
    full = o32.neighbor_count("new", "governing") > 128
    assert np.array_equal(nb_b, np.where(full, -1, o32.neighbor_count("new", "boundary")))
    assert np.array_equal(nb_g, np.where(full, -1, o32.neighbor_count("new", "governing")))
    for o in (o32, o64):
        o.boundary("new", po.WALLS_FIRST)
    sol.boundary("new")
    t, new = sol.download_tmp(), sol.download("new")
    for a in range(4):
        _close(t["dofv_grandrho"][:, a], o32.tmp["dofv_grandrho"][:, a], o64.tmp["dofv_grandrho"][:, a], ("dofv", a))
    for a in range(2):
        _close(new.rhop[:, a], o32.new["rhop"][:, a], o64.new["rhop"][:, a], ("rhop", a))
    sol.governing("new")
    for o in (o32, o64):
        o.governing("new")
    t = sol.download_tmp()
    for a in range(4):
        _close(t["acc_drhodt"][:, a], o32.tmp["acc_drhodt"][:, a], o64.tmp["acc_drhodt"][:, a], ("acc", a))
    assert sol.status() & z.FLAG_NAN == 0
    sol.close()


def test_crowded_lists_are_filtered_again():
    """Lists past their capacity and queues of hit words that fill more than once."""
    c = cases.random_cloud(8000, 5)
    mid, k = c.state.pos.mean(0), 2000
    c.state.pos[:k] = mid + (c.state.pos[:k] - mid) * 0.3
    c.state.tmp_pos[:] = c.state.pos
    sol, o32, o64 = _sorted_pair(condition_walls(_wide(c)))
    nb_b, nb_g = sol.neighbor_counts("new")
    want = o32.neighbor_count("new", "governing")
    assert (want > 128).any() and (want <= 128).any()
    assert np.array_equal(nb_g, np.where(want > 128, -1, want))
    for o in (o32, o64):
        o.boundary("new", po.WALLS_FIRST)
    sol.boundary("new")
    assert sol.status() & z.FLAG_NB_OVERFLOW
    t, new = sol.download_tmp(), sol.download("new")
    _close(t["dofv_grandrho"][:, 3], o32.tmp["dofv_grandrho"][:, 3], o64.tmp["dofv_grandrho"][:, 3], "div v")
    for a in range(2):
        _close(new.rhop[:, a], o32.new["rhop"][:, a], o64.new["rhop"][:, a], ("rhop", a))
    sol.close()


def test_steps_match_fp64_oracle():
    c, nsteps = _wide(cases.small(0.04)), 2
    sol = z.Solver.from_case(c)
    sol.run(nsteps)
    assert sol.status() == 0
    g = sol.download("old")
    sol.close()
    o32, o64 = po.Oracle(c.json, c.state, np.float32), po.Oracle(c.json, c.state, np.float64)
    o32.step(nsteps)
    o64.step(nsteps)
    assert np.array_equal(g.table, o32.old["table"])
    for k, col in (("pos", slice(None)), ("vel", slice(None)), ("rhop", 0)):
        gv, v32, v64 = (_by_id(a, t)[:, col] for a, t in ((getattr(g, k), g.table), (o32.old[k], o32.old["table"]),
                                                          (o64.old[k], o64.old["table"])))
        e_gpu, e_32, scale = err_norms(gv, v64), err_norms(v32, v64), float(np.abs(v64).max())
        for a in range(2):
            assert e_gpu[a] <= 4 * e_32[a] + 1e-6 * scale, (k, e_gpu, e_32)
