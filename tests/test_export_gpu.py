"""Exports: the device gathers against each other where rows are cut short or
slots stay untouched, both precisions."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [1, 33, 3000])
def test_history_rows_are_cut_at_the_stride_and_leave_the_rest(precision, n):
    from gpudem_gb300 import engine, scenes
    rng = np.random.default_rng(n)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    s = np.arange(n)
    x = np.stack([s % k, (s // k) % k, s // (k * k)], 1) * 3.8e-3 + 1.9e-3
    r = np.full(n, 2e-3)
    kk = np.full(n, 2000.0)
    half = 0.5 * k * 3.8e-3
    sc = scenes.Scene(x=x[rng.permutation(n)], r=r, m=scenes.sphere_mass(2500.0, r), k=kk,
                      eta=scenes.eta_const(kk, 0.5), mu=0.4, dt=1e-6,
                      tris=scenes.box_mesh(half, center=(half, half, half)), inlet_lo=np.zeros(3),
                      inlet_hi=np.full(3, 2 * half))
    E = engine.Engine(sc, precision=precision)
    E.step(3)
    full, cut = E.export(hist_stride=100), E.export(hist_stride=2)
    pos = E.export_positions()
    E.close()
    assert np.array_equal(full["x"], pos)
    for nm in ("x", "v", "angv", "r", "m", "k", "etaconst", "isActive", "numCont", "numContWall"):
        assert np.array_equal(full[nm], cut[nm]), nm
    assert np.array_equal(full["r"], r) or precision == "mixed"
    for cnt, rows in (("numCont", ("indHis", "deltHisx", "deltHisy", "deltHisz")),
                      ("numContWall", ("indHisWall", "deltHisxWall", "deltHisyWall", "deltHiszWall"))):
        c = full[cnt]
        assert n < 8 or c.max() > 2
        for nm in rows:
            a, b = full[nm].reshape(n, 100), cut[nm].reshape(n, 2)
            blank = -1 if nm.startswith("ind") else 0.0
            live = np.arange(100)[None] < c[:, None]
            assert np.all(a[~live] == blank)
            assert np.array_equal(b, a[:, :2]), nm
            if nm.startswith("ind"):
                assert np.all(a[live] >= 0)
