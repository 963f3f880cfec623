"""A map pass on one stream does not wait for other streams' passes: worlds
step together, each on a stream and a host thread of its own, and an exact
pass of many waves keeps its thread in the launches until the GPU has caught
up with them, so nothing a pass calls may wait for the other threads'
launches to end."""
import threading
import time

import numpy as np
import pytest
import torch

from pgerosion import maps as gm
from tests.parity_cases import GOLDEN, gpu_window, step_case, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", ["thermal", "uplift", "datum", "route", "base"])
def test_map_passes_run_beside_exact_passes(cuda, run):
    c = step_case(GOLDEN / "step_tiny.npz")
    g = gm.ErosionState.from_world(c["world"])
    gm.start_replay(g, c["params"])
    passes = {"thermal": lambda: gm.thermal_erosion(g, c["params"]), "uplift": lambda: gm.apply_uplift(g),
              "datum": lambda: gm.hold_datum(g, 0.3), "route": lambda: g.refresh_route(1e-4), "base": lambda: g.refresh_base()}
    P, N = 12000, 40  # as many waves: more launches than a stream's queue holds
    rng, z = np.random.default_rng(1), np.zeros(P)
    spawns = (np.zeros(P, np.int64), rng.random(P) * N, rng.random(P) * N, z, z, 1.0)
    mine = torch.cuda.Stream()

    def exact_pass(w, ep, stream):
        with torch.cuda.stream(stream):
            gm.apply_spawns(w, ep, *spawns, wave=1)

    worlds = []
    for _ in range(4):
        arr, params = window_world("tilt", N=N)
        worlds.append((gpu_window(arr), params.erosion, torch.cuda.Stream()))

    def start():
        threads = [threading.Thread(target=exact_pass, args=w) for w in worlds]
        for t in threads:
            t.start()
        return threads

    for t in start():  # (a first call makes tables and the workspaces)
        t.join()
    with torch.cuda.stream(mine):
        passes[run]()
    torch.cuda.synchronize()
    threads = start()
    time.sleep(0.2)
    t0 = time.perf_counter()
    with torch.cuda.stream(mine):
        for _ in range(3):
            passes[run]()
    mine.synchronize()
    took, running = time.perf_counter() - t0, sum(t.is_alive() for t in threads)
    for t in threads:
        t.join()
    assert running == 4, f"{run}: the exact passes were over before three map passes were ({took:.2f} s)"
