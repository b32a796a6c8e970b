"""List rebuilds where the lane groups meet their edges: particle and cell counts
around a warp and a CTA, sparse and crowded cells, many triangles in a cell, a
periodic x, storage in import order; rows against the oracle, entry by entry."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(n, spread, faces, seed, periodic=False):
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r = 1e-3 * rng.uniform(0.7, 1.3, n)
    side = spread * r.max() * max(2.0, n ** (1.0 / 3.0))
    x = rng.uniform(0.0, side, (n, 3))          # overlaps and empty cells alike: only the rows matter here
    k = np.full(n, 500.0)
    lo, hi = np.zeros(3) - 2e-3, np.full(3, side + 2e-3)
    tris = scenes.box_mesh_grid(0.5 * side, faces, center=(0.5 * side,) * 3)
    kw = {}
    if periodic:
        lo[0], hi[0] = 0.0, side
        kw = dict(box=(lo, hi), periodic_x=True)
        x[:, 0] = np.mod(x[:, 0], side)
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=k, eta=scenes.eta_const(k, 0.5), mu=0.4, dt=1e-7,
                        tris=tris, inlet_lo=lo, inlet_hi=hi, v=np.zeros((n, 3)), w=np.zeros((n, 3)), **kw)


@pytest.mark.parametrize("n,spread,faces", [(1, 2.0, 1), (7, 2.0, 3), (31, 3.0, 2), (33, 1.7, 6), (129, 6.0, 4),
                                            (1000, 1.75, 9), (4099, 1.9, 24), (5000, 8.0, 3)])
@pytest.mark.parametrize("reorder", [True, False])
def test_rows_match_the_oracle(n, spread, faces, reorder):
    _rows(_scene(n, spread, faces, n), reorder)


@pytest.mark.parametrize("n,spread,faces", [(300, 2.2, 5), (3000, 2.0, 9)])
def test_rows_match_the_oracle_periodic(n, spread, faces):
    _rows(_scene(n, spread, faces, n, periodic=True), True)


def _rows(sc, reorder):
    from gpudem_gb300 import engine
    from oracle import port
    O = port.OracleScene(sc)
    O.rebuild()
    want = O.get("neiList").reshape(sc.n, -1), O.get("numNei")
    wall = O.get("neiListWall").reshape(sc.n, -1), O.get("numNeiWall")
    for precision in ("fp64", "mixed"):
        E = engine.Engine(sc, precision=precision, reorder=reorder, nei_capacity=128, wall_capacity=64)
        E.rebuild()
        nn, nl, nw, wl = E.lists()
        s = E.stats()
        E.close()
        assert s["error_word"] == 0
        nl, wl = nl.reshape(sc.n, -1), wl.reshape(sc.n, -1)
        assert np.array_equal(nn, want[1]), precision
        for i in range(sc.n):
            assert np.array_equal(nl[i, :nn[i]], want[0][i, :nn[i]]), (precision, i)
            a, b = wl[i, :nw[i]], wall[0][i, :wall[1][i]]
            if precision == "fp64":
                assert np.array_equal(a, b), (precision, i)
            else:  # the mixed rows may hold a triangle within an FP32 error bound of the cutoff more
                assert np.all(np.diff(a) > 0) and np.isin(b, a).all(), (precision, i)
