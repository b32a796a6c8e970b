"""Every tile width and kernel form of the step at the sizes where the dispatch
changes over, counted in multiprocessors of the device at hand; periodic x in each
of them; and tiles whose pair list does not fit."""
from __future__ import annotations

import numpy as np
import pytest
from test_step_tiles_gpu import _dense, _mixed_state, _same

pytestmark = pytest.mark.gpu


def sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


def _channel(n, seed):
    """A dense slab, periodic in x, between floor, ceiling and side walls, drifting
    along x: a plane of spheres lies on the x faces and passes through them."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r0 = 2e-3
    r = r0 * rng.uniform(0.9, 1.1, n)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    a = 1.93 * r0
    s = rng.permutation(k ** 3)[:n]
    x = np.stack([s % k, (s // k) % k, s // (k * k)], 1) * a + rng.uniform(-0.04, 0.04, (n, 3)) * r0
    x[:, 1:] += 0.98 * r0
    length, width = k * a, (k - 1) * a + 2 * 0.98 * r0
    x[:, 0] %= length
    gx, gw = np.linspace(0.0, length, 9), np.linspace(0.0, width, 9)
    tris = []
    for u0, u1 in zip(gx[:-1], gx[1:]):
        for w0, w1 in zip(gw[:-1], gw[1:]):
            for end in (0.0, width):
                for c in ([(u0, end, w0), (u1, end, w0), (u1, end, w1), (u0, end, w1)],
                          [(u0, w0, end), (u1, w0, end), (u1, w1, end), (u0, w1, end)]):
                    c = np.array(c)
                    tris += [c[[0, 1, 2]], c[[0, 2, 3]]]
    lo, hi = np.array([0.0, -0.01, -0.01]), np.array([length, width + 0.01, width + 0.01])
    kk = np.full(n, 2000.0)
    v = rng.normal(0.0, 0.1, (n, 3)) + np.array([2.0, 0.0, 0.0])
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4,
                        dt=2e-6, tris=np.array(tris), inlet_lo=lo, inlet_hi=hi, v=v,
                        w=rng.normal(0.0, 20.0, (n, 3)), E=5e6, nu=0.3, e=0.5, mu_roll=0.05, box=(lo, hi),
                        periodic_x=True)


def _crossed(sc, x):
    return int((np.abs(x.reshape(-1, 3)[:, 0] - sc.x[:, 0]) > 0.5 * sc.box[1][0]).sum())


def _close_packed(n, seed):
    """Spheres on a face-centred lattice closer than their diameters: twelve
    contacts to each inside."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r0 = 2e-3
    k = int(np.ceil((n / 4) ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    base = np.array([[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]])
    side = 2 ** 0.5 * 1.93 * r0
    x = ((g + base) * side).reshape(-1, 3)
    x = x[np.argsort(x[:, 1], kind="stable")[:n]][rng.permutation(n)] + 0.98 * r0
    r = r0 * rng.uniform(0.98, 1.02, n)
    half = 0.5 * (k * side + 4 * r0)
    kk = np.full(n, 2000.0)
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4,
                        dt=2e-6, tris=scenes.box_mesh_grid(half, 4, center=(half, half, half)),
                        inlet_lo=np.zeros(3) - 0.01, inlet_hi=np.full(3, 2 * half + 0.01),
                        v=rng.normal(0.0, 0.1, (n, 3)), w=rng.normal(0.0, 20.0, (n, 3)), E=5e6, nu=0.3, e=0.5)


# FP64: up to 4 spheres to a tile the law is split over lanes; over 12 rounds of 64
# to a multiprocessor a warp takes a tile
@pytest.mark.parametrize("per_sm, more", [(4, 0), (4, 1), (96, 1), (768, 0), (768, 37)])
def test_fp64_forms_match_the_oracle_where_they_change_over(per_sm, more):
    n = per_sm * sms() + more
    s = _same(_dense(n, 40 + more, 0.05), "hertz_mindlin", (1, 6))
    assert s["n_contacts"] > n


@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_fp64_warp_tiles_match_the_oracle_in_a_periodic_channel(model):
    n = 768 * sms() + 37
    s = _same(_channel(n, 8), model, (1, 12))
    assert s["n_contacts"] > n and s["n_wall_contacts"] > 1000


@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_fp64_tiles_with_too_many_pairs_match_the_oracle(model):
    """Twelve contacts a sphere in tiles of 64: 768 pairs for a list of 448."""
    n = 192 * sms()
    s = _same(_close_packed(n, 9), model, (1, 2, 8))
    assert s["n_contacts"] > 10 * n


def _alike(a, b, r, model):
    """As the cooperative kernel and the one of a thread per particle agree: bit
    for bit with the Hertz-Mindlin law; the linear law's multiply-adds are
    contracted differently (a few FP32 ulps of the forces)."""
    if model == "hertz_mindlin":
        for nm in a:
            assert np.array_equal(a[nm], b[nm]), nm
    else:
        for nm in ("isActive", "numCont", "numContWall", "indHis", "indHisWall"):
            assert np.array_equal(a[nm], b[nm]), nm
        assert np.max(np.abs(a["x"] - b["x"])) <= 1e-7 * r.min()


# mixed: tiles of 8 and 16 up to 8 and 16 spheres to each of 20 warps, 32 beyond
@pytest.mark.parametrize("per_sm, more", [(160, 0), (160, 1), (320, 0), (320, 1)])
@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_mixed_widths_match_one_thread_per_particle_where_they_change_over(per_sm, more, model):
    n = per_sm * sms() + more
    sc = _dense(n, 70 + more, 0.05)
    a, s = _mixed_state(sc, model, 30, 1)
    b, _ = _mixed_state(sc, model, 30, 3)
    assert s["n_contacts"] > n
    _alike(a, b, sc.r, model)


@pytest.mark.parametrize("per_sm", [100, 240, 400], ids=["8-wide", "16-wide", "32-wide"])
@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_mixed_widths_match_one_thread_per_particle_in_a_periodic_channel(per_sm, model):
    n = per_sm * sms() + 3
    sc = _channel(n, 9)
    a, s = _mixed_state(sc, model, 30, 1)
    b, _ = _mixed_state(sc, model, 30, 3)
    assert s["n_contacts"] > n and s["n_wall_contacts"] > 1000 and _crossed(sc, a["x"]) > 100
    _alike(a, b, sc.r, model)
