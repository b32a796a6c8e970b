"""Plain launches (no graphs): every step is followed by the kernels of a rebuild
that returns at once unless asked for.  What they cost grows with their CTAs."""
from __future__ import annotations

import numpy as np
import pytest
from test_call_costs_gpu import us_per_step

pytestmark = pytest.mark.gpu


def test_a_rebuild_that_is_not_asked_for_costs_little_per_sphere(monkeypatch):
    """Per sphere beyond half a million, the gated kernels against the step kernel
    of spheres at rest that do not touch: 0.98 of its time where the cells' walls
    had a CTA to every 16 particles, 0.60 with a bounded number."""
    from gpudem_gb300 import engine, scenes
    monkeypatch.setenv("GDEM_GRAPHS", "0")
    step, gated = {}, {}
    for n in (500_000, 2_000_000):
        E = engine.Engine(scenes.config3_helical_chute(n=n, n_tri=20_000, v_sigma=0.0), precision="mixed",
                          model="hertz_mindlin")
        E.step(10)
        E.profile_step(20)
        step[n] = 1e3 * float(np.median([E.profile_step(20) for _ in range(5)]))
        gated[n] = us_per_step(E, [20]) - step[n]
        assert E.stats()["rebuilds"] == 1
        E.close()
    a, b = sorted(step)
    ratio = (gated[b] - gated[a]) / (step[b] - step[a])
    print(f"gated kernels per sphere over the step kernel: {ratio:.2f}", step, gated)
    assert ratio < 0.8
