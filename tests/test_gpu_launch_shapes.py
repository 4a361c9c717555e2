"""Launch shapes below and above the size up to which the untuned list build
has a form of its own: the shapes that were set are the ones launched, and
every one gives the untuned results bit for bit, crowded lists included."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import zsph_b200 as z
from zsph_b200 import cases

pytestmark = pytest.mark.gpu


def _list_kernels(sol):
    """Names of the list-build kernels of one step."""
    sol.step()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        sol.step()
        torch.cuda.synchronize()
    return {("split" if "k_nblist_split" in e.name else "seq") for e in p.events() if "k_nblist" in e.name}


def _crowded(n, box):
    """A cloud with lists past their capacity and, elsewhere, ordinary ones."""
    c = cases.random_cloud(n, 5, box=box)
    mid, k = c.state.pos.mean(0), n // 8
    c.state.pos[:k] = mid + (c.state.pos[:k] - mid) * 0.25
    c.state.tmp_pos[:] = c.state.pos
    return c


@pytest.mark.parametrize("shapes,want", [((0, 0, 0, 0), "split"), ((2, 0, 0, 0), "seq"), ((0, 0, 0, 4), "seq"),
                                         ((4, 1, 1, 2), "seq"), ((0, 6, 4, 0), "split")])
def test_shapes_that_were_set_are_launched(shapes, want):
    sol = z.Solver.from_case(cases.small(0.04))
    sol.set_launch_shapes(*shapes)
    assert _list_kernels(sol) == {want}
    sol.close()


@pytest.mark.parametrize("mk", [lambda: cases.small(0.04), lambda: cases.dam_break(0.025),
                                lambda: _crowded(20011, (0.9, 0.7, 0.5)), lambda: _crowded(64013, (1.5, 1.0, 0.6))],
                         ids=["dam_20k", "dam_61k", "crowded_20k", "crowded_64k"])
def test_every_shape_gives_the_untuned_counts_and_step(mk):
    c = mk()
    want = want_nb = None
    for cw, sg in ((0, 0), (2, 2), (2, 3), (2, 4), (4, 2), (4, 3), (4, 4)):
        sol = z.Solver.from_case(c)
        sol.set_launch_shapes(cw, 0, 0, sg)
        sol.neighbor_search("old", "new")
        nb = sol.neighbor_counts("new")
        sol.step()
        got = sol.download("old")
        sol.close()
        if want is None:
            want, want_nb = got, nb
            continue
        for a in range(2):
            assert np.array_equal(nb[a], want_nb[a]), (cw, sg)
        for k in ("pos", "vel", "rhop", "type", "table"):
            assert np.array_equal(getattr(got, k), getattr(want, k), equal_nan=k in ("pos", "vel", "rhop")), (cw, sg, k)


def test_tuner_keeps_the_untuned_form_where_it_is_fastest():
    """Of a small case, the untuned list build is the faster one by a quarter:
    the tuner times it, and its result carries no shape that turns it off."""
    sol = z.Solver.from_case(cases.small(0.04))
    r = sol.autotune(20)
    assert r["candidates"] == 36
    assert r["list_cells_per_cta"] == 0 and r["list_segments"] == 0
    assert _list_kernels(sol) == {"split"}
    sol.close()
