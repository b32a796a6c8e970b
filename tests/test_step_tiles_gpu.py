"""The FP64 step at the edges of its tiles: particle counts around the tile and
CTA sizes, dense overlapping beds against walls, and one sphere with dozens of
contacts, against the oracle bit for bit (its sums run in the same row order,
so no rounding may differ)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import compact_rows

pytestmark = pytest.mark.gpu


def _dense(n, seed, mu_roll=0.0):
    """Spheres on a jittered lattice closer than their diameters, in the corner
    of a box of small triangles."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r0 = 2e-3
    r = r0 * rng.uniform(0.9, 1.1, n)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    a = 1.93 * r0
    s = rng.permutation(k ** 3)[:n]
    x = np.stack([s % k, (s // k) % k, s // (k * k)], 1) * a + 0.98 * r0 + rng.uniform(-0.04, 0.04, (n, 3)) * r0
    half = 0.5 * ((k + 1) * a + 4 * r0)
    m = scenes.sphere_mass(2500.0, r)
    kk = np.full(n, 2000.0)
    tris = scenes.box_mesh_grid(half, max(1, int(half / (1.5 * r0))), center=(half, half, half))
    return scenes.Scene(x=x, r=r, m=m, k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4, dt=2e-6, tris=tris,
                        inlet_lo=np.zeros(3) - 0.01, inlet_hi=np.full(3, 2 * half + 0.01),
                        v=rng.normal(0.0, 0.1, (n, 3)), w=rng.normal(0.0, 20.0, (n, 3)), E=5e6, nu=0.3, e=0.5,
                        mu_roll=mu_roll)


def _crowded(seed):
    """A large sphere with some fifty small ones pressed against it, in a corner."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    R, q, m = 8e-3, 1.6e-3, 52
    k = np.arange(m) + 0.5
    th, ph = np.arccos(1 - 2 * k / m), np.pi * (1 + 5 ** 0.5) * k
    c = np.array([R + 3.5 * q] * 3)
    x = c + (R + q) * 0.999 * np.stack([np.cos(ph) * np.sin(th), np.sin(ph) * np.sin(th), np.cos(th)], 1)
    x = np.concatenate([x[:20], [c], x[20:]])
    r = np.full(m + 1, q)
    r[20] = R
    half = 2 * R
    mass = scenes.sphere_mass(2500.0, r)
    kk = np.full(m + 1, 2000.0)
    return scenes.Scene(x=x, r=r, m=mass, k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4, dt=2e-6,
                        tris=scenes.box_mesh_grid(half, 4, center=(half, half, half)), inlet_lo=np.zeros(3) - 0.01,
                        inlet_hi=np.full(3, 2 * half + 0.01), v=rng.normal(0.0, 0.1, (m + 1, 3)),
                        w=rng.normal(0.0, 20.0, (m + 1, 3)), E=5e6, nu=0.3, e=0.5)


def _same(sc, model, steps, **kw):
    from gpudem_gb300 import engine
    from oracle import port
    E = engine.Engine(sc, model=model, store_forces=True, **kw)
    O = port.OracleScene(sc, model=model)
    done = 0
    for c in steps:
        E.step(c - done)
        O.step(c - done)
        done = c
        st = E.export(history=True, forces=True)
        for nm in ("isActive", "numCont", "numContWall", "x", "v", "angv", "f", "mom"):
            assert np.array_equal(st[nm], O.get(nm)), (c, nm)
        nc, ncw = st["numCont"], st["numContWall"]
        for nm, cnt in (("indHis", nc), ("indHisWall", ncw), ("deltHisx", nc), ("deltHisy", nc), ("deltHisz", nc),
                        ("deltHisxWall", ncw), ("deltHisyWall", ncw), ("deltHiszWall", ncw)):
            assert np.array_equal(compact_rows(st[nm], cnt), compact_rows(O.get(nm), cnt)), (c, nm)
    s = E.stats()
    assert s["error_word"] == 0
    E.close()
    return s


@pytest.mark.parametrize("n", [1, 3, 8, 9, 31, 65, 130, 609, 1300, 9_800, 23_000])
@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_fp64_tiles_match_the_oracle(n, model):
    s = _same(_dense(n, 100 + n, 0.05 if n % 2 else 0.0), model, (1, 2, 40))
    if n >= 130:
        assert s["n_contacts"] > n and s["n_wall_contacts"] > 0


@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_fp64_warp_tiles_match_the_oracle(model):
    """Beyond the sizes that take a CTA to a tile."""
    s = _same(_dense(120_001, 21, 0.05), model, (1, 2, 8))
    assert s["n_contacts"] > 120_001 and s["n_wall_contacts"] > 0


@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_fp64_sphere_with_many_contacts_matches_the_oracle(model):
    s = _same(_crowded(7), model, (1, 2, 60), nei_capacity=128, hist_capacity=64, wall_capacity=64)
    assert s["n_contacts"] > 50


def _mixed_state(sc, model, steps, kernel, **kw):
    from gpudem_gb300 import engine
    E = engine.Engine(sc, precision="mixed", model=model, mixed_kernel=kernel, store_forces=True, **kw)
    E.step(steps)
    st = E.export(history=True, forces=True)
    s = E.stats()
    assert s["error_word"] == 0
    E.close()
    return st, s


@pytest.mark.parametrize("n", [1, 7, 9, 33, 130, 2049, 24_400, 49_001])
@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_mixed_tiles_match_one_thread_per_particle(n, model):
    sc = _dense(n, 300 + n, 0.05 if n % 2 else 0.0)
    a, s = _mixed_state(sc, model, 40, 1)
    b, _ = _mixed_state(sc, model, 40, 3)
    # the Hertz-Mindlin law rounds alike in both kernels; the linear law's
    # multiply-adds are contracted differently, a few FP32 ulps (5e-7) of the
    # forces, which move a sphere by some 1e-5 m in these 40 steps: 3e-9 r
    if model == "hertz_mindlin":
        for nm in a:
            assert np.array_equal(a[nm], b[nm]), nm
    else:
        for nm in ("isActive", "numCont", "numContWall", "indHis", "indHisWall"):
            assert np.array_equal(a[nm], b[nm]), nm
        assert np.max(np.abs(a["x"] - b["x"])) <= 1e-7 * sc.r.min()
    if n >= 130:
        assert s["n_contacts"] > n and s["n_wall_contacts"] > 0


@pytest.mark.parametrize("inner_skin", [0.0, -1.0])
def test_mixed_sphere_with_many_contacts(inner_skin):
    sc = _crowded(9)
    kw = dict(nei_capacity=128, hist_capacity=64, wall_capacity=64, inner_skin=inner_skin)
    a, s = _mixed_state(sc, "hertz_mindlin", 30, 1, **kw)
    b, _ = _mixed_state(sc, "hertz_mindlin", 30, 3, **kw)
    for nm in a:
        assert np.array_equal(a[nm], b[nm]), nm
    assert s["n_contacts"] > 50
