"""The trace of one warp a droplet (``trace_lanes`` 0, small waves) against
the trace of one thread a droplet (``trace_lanes`` 1, the general path): both
do the same operations in the same order, so passes and steps must come out
bit for bit the same, whatever the list lengths (a warp walks 32 steps ahead,
8 at sea, and looks back 8 active cells), with faces crossed, lakes, parks,
banks, roots, masks and loaded spawns."""
import numpy as np
import pytest
import torch

from pgerosion import maps as gm
from tests.parity_cases import GOLDEN, gpu_window, step_case, window_case, window_world
from tests.test_gpu_lake_parks import _park_window
from tests.test_gpu_parity import _gpu_window_state

pytestmark = pytest.mark.gpu


def _both(monkeypatch, make, run):
    out = []
    make_params = gm.make_params
    for lanes in (1, 0):
        g = make()
        with monkeypatch.context() as m:
            def with_lanes(*a, **k):
                p = make_params(*a, **k)
                p.trace_lanes = lanes
                return p

            m.setattr(gm, "make_params", with_lanes)
            s = run(g)
        extra = {k: getattr(g, k).cpu().numpy() for k in ("lake_load", "lake_room") if getattr(g, k, None) is not None}
        out.append((s, g.to_numpy() | extra))
    (s1, a1), (s0, a0) = out
    for k in s1:
        if k != "seconds":
            assert s1[k] == s0[k], k
    for k in a1:
        if isinstance(a1[k], np.ndarray):
            assert a1[k].tobytes() == a0[k].tobytes(), k
    return s0


def _spawns(P, lo, hi, seed):
    rng = np.random.default_rng(seed)
    x, y = lo + rng.random(P) * (hi - lo), lo + rng.random(P) * (hi - lo)
    sed = np.where(rng.random(P) < 0.5, 0.02 * rng.random(P), 0.0)
    return x, y, sed, rng.random(P) * 6.0


@pytest.mark.parametrize("kind", ["closed", "tilt", "shelf"])
@pytest.mark.parametrize("max_steps", [1, 7, 8, 9, 31, 32, 33, 65, 200])
def test_windows(cuda, monkeypatch, kind, max_steps):
    arr, params = window_world(kind, N=40)
    ep = params.erosion
    ep.max_steps, ep.evap_rate, ep.pit_steps = max_steps, 1e-3, 3 if kind == "tilt" else 1000
    P = 700
    x, y, sed, dirs = _spawns(P, 0.0, 40.0, max_steps)
    s = _both(monkeypatch, lambda: gpu_window(arr),
              lambda g: gm.apply_spawns(g, ep, np.zeros(P, np.int64), x, y, sed, dirs, 1.0, wave=256))
    assert s["droplet_steps"] > 0


@pytest.mark.parametrize("exponent", [0.0, 0.5, 0.7])
@pytest.mark.parametrize("fixture", ["window_trace", "roots_trace", "lateral_trace", "lake_parks"])
def test_fixtures(cuda, monkeypatch, fixture, exponent):
    case = window_case(GOLDEN / f"{fixture}.npz")
    ep, parks = case["params"], fixture == "lake_parks"
    ep.disc_exponent = exponent

    def make():
        g = _park_window(case) if parks else _gpu_window_state(case)
        if "roots" in fixture:
            g.roots = torch.as_tensor(np.random.default_rng(1).random(g.height.shape), dtype=torch.float32, device=g.height.device)
        return g

    P = len(case["sp_face"])
    s = _both(monkeypatch, make,
              lambda g: gm.apply_spawns(g, ep, case["sp_face"], case["sp_x"], case["sp_y"], case["sp_sed"], case["sp_dir"],
                                        case["volume0"], wave=P // 3 + 1, parks=parks))
    assert s["entries"] > s["droplet_steps"] > 0


@pytest.mark.parametrize("fixture", ["step_tiny", "step_lateral", "step_lake"])
def test_sphere_steps(cuda, monkeypatch, fixture):
    c = step_case(GOLDEN / f"{fixture}.npz")

    def make():
        g = gm.ErosionState.from_world(c["world"])
        gm.start_replay(g, c["params"])
        return g

    def run(g):
        for it in range(2):
            s = gm.step(g, c["params"], it, n_particles=c["n_particles"])
        return {k: s[k] for k in ("droplet_steps", "clamped") if k in s}

    _both(monkeypatch, make, run)
