"""An export commits the pages that it writes and little more: what the caller's
history arrays hold in memory afterwards, by the kernel's own account."""
from __future__ import annotations

import ctypes as C
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STRIDE = 100
ARRAYS = ("deltHisx", "deltHisy", "deltHisz", "deltHisxWall", "deltHisyWall", "deltHiszWall")


def _lattice(n, spacing):
    from gpudem_gb300 import scenes
    k = int(np.ceil(n ** (1.0 / 3.0)))
    s = np.random.default_rng(4).permutation(n)
    r = np.full(n, 2e-3)
    x = np.stack([s % k, (s // k) % k, s // (k * k)], 1) * spacing * r[0] + 2.5e-3
    kk = np.full(n, 2000.0)
    half = 0.5 * (k * spacing * r[0] + 5e-3)
    return scenes.Scene(x=x, r=r, m=scenes.sphere_mass(2500.0, r), k=kk, eta=scenes.eta_const(kk, 0.5), mu=0.4,
                        dt=1e-6, tris=scenes.box_mesh(half, center=(half, half, half)), inlet_lo=np.zeros(3),
                        inlet_hi=np.full(3, 2 * half))


def _resident(buf, size):
    vec = (C.c_ubyte * -(-size // mmap.PAGESIZE))()
    at = C.addressof(C.c_char.from_buffer(buf))
    assert C.CDLL(None, use_errno=True).mincore(C.c_void_p(at), C.c_size_t(size), vec) == 0
    return sum(b & 1 for b in vec) / len(vec)


def _export(E, forces=False):
    """One export into fresh anonymous maps: (return code, resident share of each history array)."""
    from gpudem_gb300 import _lib
    n = E.n
    cnt = [np.zeros(n, np.int32) for _ in range(2)]
    maps = {nm: mmap.mmap(-1, n * STRIDE * 8) for nm in ARRAYS}
    p = _lib.Particles()
    p.n, p.hist_stride = n, STRIDE
    ip, dp = C.POINTER(C.c_int), C.POINTER(C.c_double)
    p.numCont, p.numContWall = (c.ctypes.data_as(ip) for c in cnt)
    for nm, m in maps.items():
        setattr(p, nm, C.cast(C.addressof(C.c_char.from_buffer(m)), dp))
    if forces:
        f = np.zeros(3 * n)
        p.f = f.ctypes.data_as(dp)
    rc = E.L.gdem_export_particles(E.h, C.byref(p))
    share = {nm: _resident(m, n * STRIDE * 8) for nm, m in maps.items()}
    return rc, cnt[0], share


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_scene_without_contacts_leaves_the_rows_untouched(precision):
    from gpudem_gb300 import engine
    E = engine.Engine(_lattice(20_000, 2.4), precision=precision)
    E.step(2)
    rc, nc, share = _export(E)
    E.close()
    assert rc == 0 and nc.max() == 0
    assert max(share.values()) < 0.01, share


def test_a_refused_export_leaves_the_rows_untouched():
    from gpudem_gb300 import engine
    E = engine.Engine(_lattice(20_000, 1.99), precision="mixed")
    E.step(2)
    assert _export(E)[0] == 0
    rc, _, share = _export(E, forces=True)       # GDEM_ERR_STATE: forces are not stored
    E.close()
    assert rc == 4 and max(share.values()) < 0.01, share


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rows_are_whole_where_every_sphere_has_contacts(precision):
    """The arrays mapped ahead (the second export, after rows were seen) hold the
    same values as those that were not."""
    from gpudem_gb300 import engine
    E = engine.Engine(_lattice(20_000, 1.99), precision=precision)
    E.step(2)
    a, b = E.export(history=True), E.export(history=True)
    rc, nc, share = _export(E)
    E.close()
    assert rc == 0 and nc.min() >= 3
    for nm in a:
        assert np.array_equal(a[nm], b[nm]), nm
    assert min(share[nm] for nm in ARRAYS[:3]) > 0.9
