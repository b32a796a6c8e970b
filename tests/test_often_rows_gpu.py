"""Rows asked for in every step or every few: the steps then run one by one
within the loop of chains.  They are the steps of single calls, and not much
slower."""
from __future__ import annotations

import numpy as np
import pytest
from test_call_costs_gpu import us_per_step
from test_chains_gpu import _shower

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tree", [False, True])
@pytest.mark.parametrize("kw", [dict(precision="fp64", skin=1e-4), dict(precision="mixed", inner_skin=1e-9),
                                dict(precision="mixed", inner_skin=1e-4), dict(precision="mixed", skin=1e-4)],
                         ids=["fp64-lists", "mixed-every-step", "mixed-some-steps", "mixed-lists"])
def test_steps_that_ask_for_rows_often_are_the_same(kw, tree):
    from gpudem_gb300 import engine
    sc = _shower(900, 13)
    kw = dict(kw, model="hertz_mindlin", bvh_every_step=tree, refresh=0.5 * kw.get("skin", sc.r.max()))
    out = []
    for chain, calls in ((8, [1] * 101), (8, [101]), (1, [101]), (3, [60, 41]), (64, [101])):
        E = engine.Engine(sc, steps_per_graph=chain, **kw)
        for c in calls:
            E.step(c)
        out.append((E.export(history=True), E.stats(), E.lists()))
        E.close()
    a, s, ls = out[0]
    assert s["steps"] == 101 and s["error_word"] == 0 and s["rebuilds"] + s["inner_builds"] > 20
    for b, t, lt in out[1:]:
        for nm in ("steps", "rebuilds", "inner_builds", "n_contacts", "n_nei", "n_inner", "error_word"):
            assert s[nm] == t[nm], nm
        for nm in a:
            assert np.array_equal(a[nm], b[nm]), nm
        for p, q in zip(ls, lt):
            assert np.array_equal(p, q)


@pytest.mark.parametrize("ntri", [300, 50_000])
def test_a_tree_beside_steps_that_pass_is_not_the_cost_of_a_step(ntri):
    """Inner rows that last one step, the mesh tree rebuilt in every step: a call
    of many steps took 3.2 times single calls over 50,000 triangles, 2.0 times over
    300, when the steps behind each request passed with their trees; below 1 now."""
    from gpudem_gb300 import engine, scenes
    sc = (scenes.config3_helical_chute(n=20_000, n_tri=ntri, v_sigma=0.5) if ntri > 1000
          else scenes.config2_tilted_box(n=2000, r0=2e-3))
    E = engine.Engine(sc, precision="mixed", model="hertz_mindlin", inner_skin=1e-9, bvh_every_step=True)
    E.step(40)
    one, many = us_per_step(E, [1] * 80), us_per_step(E, [80])
    E.close()
    assert many < 1.3 * one, (many, one)
