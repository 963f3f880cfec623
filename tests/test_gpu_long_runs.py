"""The ranks and the per-cell sums where a cell's run of sorted entries is
longer than the windows they are counted in (32 and 64 slots, 128 looked
back): waves whose droplets all stand on a few cells, so that runs of
hundreds to thousands of entries start and end at every place in a window,
against the oracle's serial apply (IEEE float64 in the same order: heights
identical in 99.9 % of the cells, everything within 1e-5, the clamped count
equal)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("droplets,spread", [(7, 1), (31, 1), (33, 1), (64, 1), (129, 1), (257, 2), (512, 1), (1500, 3), (2048, 1)])
def test_crowded_cells_match_the_oracle(cuda, droplets, spread):
    arr, params = window_world("closed", N=24, seed=3)
    ep = params.erosion
    ep.max_steps, ep.pit_steps = 12, 100000
    g = gpu_window(arr)
    N, H, P = arr["N"], arr["H"], droplets
    rng = np.random.default_rng(droplets)
    f = np.zeros(P, np.int64)
    x, y = 11.0 + rng.integers(0, spread, P) + rng.random(P), 12.0 + rng.random(P)
    sed = np.where(rng.random(P) < 0.5, rng.random(P), 0.0)
    dirs = rng.random(P) * 6.0
    h = lambda t: t.detach().cpu().numpy().copy()
    o = orc.OracleState(height=h(g.height), sediment=h(g.sediment), discharge=h(g.discharge), momentum=h(g.momentum),
                        hardness=h(g.hardness), precip=h(g.precip), evap=h(g.evap), uplift=h(g.uplift), mask=arr["mask"],
                        metric=arr["metric"], metric_inv=arr["metric_inv"], N=N, H=H, spherical=False, height_unit_m=arr["cell"],
                        base=h(g.base), deposit_on_exit=True)
    s = gm.apply_spawns(g, ep, f, x, y, sed, dirs, 1.0, wave=P)
    o.pack()
    o.acc[...] = 0.0
    tp = orc.trace_params(o, ep, 1.0, P / (1.0 * P))
    cl = orc.trace(o, tp, f, x, y, sed, dirs, 1.0)
    cells = np.asarray(cl[0]).reshape(P, -1)
    used = np.concatenate([cells[q, :n] for q, n in enumerate(np.asarray(cl[4]))])
    clamped = orc.apply(o, orc.apply_params(o, ep, ep.iter_deposit / o.height_unit_m), cl, orc.change_list_cap(tp.max_steps))[0]
    lib = orc.lib()
    lib.orc_fold(ctypes.c_int64(o.height.size), orc._p(o.height), orc._p(o.sediment), orc._p(o.acc), orc._p(o.mask))
    lib.orc_ema(ctypes.c_int64(o.height.size), orc._p(o.discharge), orc._p(o.momentum), orc._p(o.disch_track), orc._p(o.mom_track),
                orc._p(o.mask), ctypes.c_double(float(ep.ema)))
    assert np.bincount(used).max() >= droplets // spread  # the runs are as long as the test is for
    a = g.to_numpy()
    for k in ("height", "sediment", "discharge", "momentum", "pending"):
        np.testing.assert_allclose(a[k], getattr(o, k), rtol=1e-5, atol=1e-9, err_msg=k)
    assert np.mean(a["height"] == o.height) >= 0.999
    assert s["clamped"] == clamped
