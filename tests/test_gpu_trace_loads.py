"""The trace of one warp a droplet where a load lies outside the range in
which its quotient by the evaporation is formed from a reciprocal (from 2^-500
on, zero aside), down to the subnormals, against the trace of one thread a
droplet, which divides: passes bit for bit the same.  Nothing erodes, so the
loads stay as small as they start and show in the empty sediment they drop
into."""
import numpy as np
import pytest

from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world
from tests.test_gpu_trace_warps import _both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["closed", "shelf"])
@pytest.mark.parametrize("low,high", [(-324, -300), (-200, -149), (-152, -149)])
def test_loads_beyond_the_reciprocals_range(cuda, monkeypatch, kind, low, high):
    arr, params = window_world(kind, N=32)
    ep = params.erosion
    ep.max_steps, ep.erodibility, ep.evap_rate = 70, 0.0, 0.02
    P, rng = 600, np.random.default_rng(-low)
    x, y, dirs = rng.random(P) * 32, rng.random(P) * 32, rng.random(P) * 6.0
    sed = np.power(10.0, low + rng.random(P) * (high - low))
    sed[::7] = 0.0
    made = []

    def make():
        made.append(gpu_window(arr))
        return made[-1]

    s = _both(monkeypatch, make, lambda g: gm.apply_spawns(g, ep, np.zeros(P, np.int64), x, y, sed, dirs, 1.0, wave=256))
    assert s["droplet_steps"] > 0
    a = made[0].to_numpy()
    moved = a["sediment"][a["sediment"] != 0.0]
    assert moved.size > 100 or np.count_nonzero(a["pending"]) > 100
