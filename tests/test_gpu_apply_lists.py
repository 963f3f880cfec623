"""The ordered apply at the list lengths and revisits where its on-chip
windows end, against the oracle's trace and serial apply.

The apply reads a droplet's records in chunks of 32 entries, four at a time,
and keeps the net change of the last 128 entries on chip for the droplet's
own revisits.  ``closed`` is a bowl whose droplets, never stopped for
climbing, run down into it and circle its floor: they come back to cells
after any number of entries, and share them with every other droplet of the
wave.  Nothing crosses a face there, so every operation is the oracle's
(IEEE float64, the same order); the bound is the passes' own: heights
identical in 99.9 % of the cells, everything within 1e-5."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_steps", [1, 23, 24, 31, 56, 119, 128, 129, 300, 640])
def test_lists_of_every_chunk_length_match_the_oracle(cuda, max_steps):
    arr, params = window_world("closed", N=40)
    ep = params.erosion
    ep.max_steps, ep.pit_steps, ep.evap_rate, ep.chunk = max_steps, 100000, 1e-4, 64
    g = gpu_window(arr)
    N, H = arr["N"], arr["H"]
    P = 1026  # 16 waves of 64 and one of two droplets
    rng = np.random.default_rng(max_steps)
    f, x, y = np.zeros(P, np.int64), rng.random(P) * N, rng.random(P) * N
    x[:400], y[:400] = 0.5 * N + rng.random(400) * 3, 0.5 * N + rng.random(400) * 3  # crowded on the floor
    zero, v0 = np.zeros(P), 1.0
    h = lambda t: t.detach().cpu().numpy().copy()
    o = orc.OracleState(height=h(g.height), sediment=h(g.sediment), discharge=h(g.discharge), momentum=h(g.momentum),
                        hardness=h(g.hardness), precip=h(g.precip), evap=h(g.evap), uplift=h(g.uplift), mask=arr["mask"],
                        metric=arr["metric"], metric_inv=arr["metric_inv"], N=N, H=H, spherical=False, height_unit_m=arr["cell"],
                        base=h(g.base), deposit_on_exit=True)
    s = gm.apply_spawns(g, ep, f, x, y, zero, zero, v0, wave=64)
    o.pack()
    o.acc[...] = 0.0
    tp = orc.trace_params(o, ep, v0, 64 / (v0 * P))
    ap = orc.apply_params(o, ep, ep.iter_deposit / o.height_unit_m)
    cap = orc.change_list_cap(tp.max_steps)
    clamped, longest, gap = 0, 0, 0
    for c0 in range(0, P, 64):
        sl = slice(c0, c0 + 64)
        cl = orc.trace(o, tp, f[sl], x[sl], y[sl], zero[sl], zero[sl], v0)
        cells, count = np.asarray(cl[0]).reshape(-1, cap), np.asarray(cl[4])
        longest = max(longest, int(count.max()))
        last = {}
        for k, c in enumerate(cells[0, :count[0]].tolist()):
            gap = max(gap, k - last.get(c, k))
            last[c] = k
        clamped += orc.apply(o, ap, cl, cap)[0]
    lib = orc.lib()
    lib.orc_fold(ctypes.c_int64(o.height.size), orc._p(o.height), orc._p(o.sediment), orc._p(o.acc), orc._p(o.mask))
    lib.orc_ema(ctypes.c_int64(o.height.size), orc._p(o.discharge), orc._p(o.momentum), orc._p(o.disch_track), orc._p(o.mom_track),
                orc._p(o.mask), ctypes.c_double(float(ep.ema)))
    a = g.to_numpy()
    for k in ("height", "sediment", "discharge", "momentum", "pending"):
        np.testing.assert_allclose(a[k], getattr(o, k), rtol=1e-5, atol=1e-9, err_msg=k)
    assert np.mean(a["height"] == o.height) >= 0.999
    assert s["clamped"] == clamped
    assert longest >= min(max_steps, 119)  # the lists do reach the lengths the test is for
    if max_steps >= 300:
        assert gap >= 128, gap  # and come back after more entries than are kept on chip
