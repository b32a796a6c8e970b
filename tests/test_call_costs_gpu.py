"""What calls cost beside one another: forms of the same steps that may not be
much slower than their plain one.  Times by CUDA events on the engine's stream,
medians of repeats; the bounds lie far from both the sound and the faulty time."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def us_per_step(E, calls, repeats=7):
    """Median time per step of the calls (steps of each), on the device."""
    torch = pytest.importorskip("torch")
    stream = torch.cuda.ExternalStream(E.stream())
    out = []
    for _ in range(repeats):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record(stream)
        for c in calls:
            E.step(c)
        b.record(stream)
        b.synchronize()
        out.append(a.elapsed_time(b) * 1e3 / sum(calls))
    return float(np.median(out))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("count", [2, 3])
def test_short_calls_do_not_pay_for_a_long_chain(precision, count):
    """Two or three steps a call with chains of 64: as single steps (1.0 of their
    time), not as a chain whose other kernels pass (2.6 and 1.8)."""
    from gpudem_gb300 import engine, scenes
    E = engine.Engine(scenes.config2_tilted_box(n=2000, r0=2e-3), precision=precision, model="hertz_mindlin",
                      steps_per_graph=64)
    E.step(130)
    one, short = us_per_step(E, [1] * 120), us_per_step(E, [count] * (120 // count))
    E.close()
    assert short < 1.4 * one, (short, one)
