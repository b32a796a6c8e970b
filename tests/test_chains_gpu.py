"""Steps in chains: any chain length and any split of the calls takes the same
steps, with the rows rebuilt at the same ones, as one step at a time."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shower(n=700, seed=3):
    """Fast spheres in a box, so that rows are rebuilt every few steps."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r = rng.uniform(0.9e-3, 1.1e-3, n)
    half = 0.02
    x = scenes.lattice_packing(n, r, np.full(3, -half + 2e-3), np.full(3, half - 2e-3), rng, gap=0.1)
    k = np.full(n, 500.0)
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=k, eta=scenes.eta_const(k, 0.5), mu=0.4, dt=1e-5,
                        tris=scenes.box_mesh_grid(half, 5), inlet_lo=np.full(3, -half), inlet_hi=np.full(3, half),
                        v=rng.normal(0.0, 2.0, (n, 3)), w=np.zeros((n, 3)), E=5e6, nu=0.3, e=0.5)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tree", [False, True])
def test_chains_take_the_same_steps(precision, tree):
    from gpudem_gb300 import engine
    sc = _shower()

    def go(chain, calls):
        E = engine.Engine(sc, precision=precision, model="hertz_mindlin", steps_per_graph=chain, bvh_every_step=tree)
        for c in calls:
            E.step(c)
        st, s, ls = E.export(history=True), E.stats(), E.lists()
        E.close()
        return st, s, ls

    total = 127
    ref, rs, rl = go(8, [1] * total)
    assert rs["steps"] == total and rs["rebuilds"] > 10 and rs["n_contacts"] > 0
    for chain, calls in ((8, [total]), (1, [total]), (3, [2, 0, 5, 1, total - 8]), (40, [7, total - 7]), (8, [8] * 15 + [7])):
        st, s, ls = go(chain, calls)
        for nm in ("steps", "rebuilds", "inner_builds", "n_contacts", "n_nei", "error_word"):
            assert s[nm] == rs[nm], (chain, nm)
        for nm in ref:
            assert np.array_equal(st[nm], ref[nm]), (chain, nm)
        for a, b in zip(ls, rl):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graphs_follow_a_new_import_and_new_materials(precision):
    """An engine that was stepped before takes the same steps after a new import
    (the same grid, another one, per-particle materials) as a new engine."""
    from dataclasses import replace

    from gpudem_gb300 import engine
    a = _shower(600, 5)
    b = replace(a, r=a.r * 0.97, v=-a.v)       # another r_max: another grid and skin
    rng = np.random.default_rng(8)
    mu, e = rng.uniform(0.2, 0.6, a.n), rng.uniform(0.3, 0.8, a.n)

    def run(E, sc, mats):
        E.import_particles(sc)
        if mats:
            E.set_particle_materials(mu, e)
        E.step(29)
        st, s = E.export(history=True), E.stats()
        assert s["error_word"] == 0 and s["steps"] == 29
        return st

    kw = dict(precision=precision, model="hertz_mindlin")
    E = engine.Engine(a, **kw)
    for sc, mats in ((a, False), (a, True), (b, True), (b, False), (a, False)):
        got = run(E, sc, mats)
        F = engine.Engine(sc, **kw)
        want = run(F, sc, mats)
        F.close()
        for nm in want:
            assert np.array_equal(got[nm], want[nm]), (mats, nm)
    E.close()


def test_an_inner_skin_that_widens_changes_no_result():
    """Fast spheres make the inner rows short-lived, so their skin grows; the
    trajectory is that of the list rows."""
    from gpudem_gb300 import engine
    sc = _shower(900, 11)
    out = []
    for skin in (0.0, -1.0):
        E = engine.Engine(sc, precision="mixed", model="hertz_mindlin", inner_skin=skin)
        E.step(150)
        out.append((E.export(history=True), E.stats()))
        E.close()
    (a, s), (b, t) = out
    assert s["error_word"] == 0 and s["n_contacts"] > 0 and s["rebuilds"] == t["rebuilds"]
    assert 0 < s["inner_builds"] < 100
    for nm in a:
        assert np.array_equal(a[nm], b[nm]), nm
