"""The mixed step without inner rows, on tiles of 32: its entries carry no slot
hints, so it has a kernel of its own.  Results do not depend on the rows that
are scanned, so they equal those with inner rows bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def full_tiles():
    """A count of spheres (odd) that takes tiles of 32: more
    than 16 to each of the 20 resident warps of an SM."""
    torch = pytest.importorskip("torch")
    return 16 * 20 * torch.cuda.get_device_properties(0).multi_processor_count + 37


def dense(n, seed):
    """Spheres on a jittered lattice closer than their diameters, in a box."""
    from gpudem_gb300 import scenes
    rng = np.random.default_rng(seed)
    r0 = 2e-3
    r = r0 * rng.uniform(0.9, 1.1, n)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    a = 1.93 * r0
    s = rng.permutation(k ** 3)[:n]
    x = np.stack([s % k, (s // k) % k, s // (k * k)], 1) * a + 0.98 * r0 + rng.uniform(-0.04, 0.04, (n, 3)) * r0
    half = 0.5 * ((k + 1) * a + 4 * r0)
    kk = np.full(n, 2000.0)
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4,
                        dt=2e-6, tris=scenes.box_mesh_grid(half, 8, center=(half, half, half)),
                        inlet_lo=np.zeros(3) - 0.01, inlet_hi=np.full(3, 2 * half + 0.01),
                        v=rng.normal(0.0, 0.1, (n, 3)), w=rng.normal(0.0, 20.0, (n, 3)), E=5e6, nu=0.3, e=0.5,
                        mu_roll=0.05)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_without_inner_rows_the_step_is_the_same(model, periodic):
    from gpudem_gb300 import engine, scenes
    n = full_tiles()
    sc = (scenes.config5_periodic_channel(n=n, length=0.3, width=0.15, n_tri=2000, v_drift=1.0, dt=5e-6) if periodic
          else dense(n, 5))
    out = []
    for skin in (0.0, -1.0):
        E = engine.Engine(sc, precision="mixed", model=model, inner_skin=skin)
        E.step(400 if periodic else 120)
        out.append((E.export(history=True), E.stats()))
        E.close()
    (a, s), (b, t) = out
    assert s["error_word"] == 0 and t["error_word"] == 0 and t["n_inner"] == 0 < s["n_inner"]
    assert s["n_contacts"] > (1000 if periodic else 3 * n)
    for nm in a:
        assert np.array_equal(a[nm], b[nm]), nm


@pytest.mark.parametrize("model", ["linear", "hertz_mindlin"])
def test_without_inner_rows_the_search_is_not_a_chain(model):
    """The slot search of a contact loads its keys side by side.  Against the
    kernel of one thread per particle, which scans the same rows, the kernel
    takes 0.64 (linear) and 0.60 (Hertz-Mindlin) of the time on this bed with the
    keys read one after another, and 0.52 and 0.50 side by side: the bound lies
    between."""
    from gpudem_gb300 import engine
    sc = dense(300_001, 6)
    ms = {}
    for kernel in (1, 3):
        E = engine.Engine(sc, precision="mixed", model=model, inner_skin=-1.0, mixed_kernel=kernel)
        E.step(40)
        E.profile_step(20)
        ms[kernel] = float(np.median([E.profile_step(40) for _ in range(5)]))
        E.close()
    assert ms[1] < 0.56 * ms[3], ms


@pytest.mark.parametrize("scene", ["lattice", "box"])
def test_spheres_that_do_not_touch_cost_their_state(scene):
    """A step of spheres that do not touch is their state read and
    written.  Against the kernel of one thread per particle the step takes 0.89 of
    the time; with a word of the control block read for every particle it took
    1.17 to 1.20."""
    from gpudem_gb300 import engine, scenes
    sc = (scenes.config3_helical_chute(n=300_000, n_tri=20_000, v_sigma=0.5) if scene == "lattice"
          else scenes.config2_tilted_box(n=300_000, r0=2e-3))
    us = {}
    for kernel in (1, 3):
        E = engine.Engine(sc, precision="mixed", model="hertz_mindlin", mixed_kernel=kernel)
        E.step(11)
        E.profile_step(20)
        us[kernel] = 1e3 * float(np.median([E.profile_step(20) for _ in range(7)]))
        E.close()
    assert us[1] < 1.04 * us[3], us
