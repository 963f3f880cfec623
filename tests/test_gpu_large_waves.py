"""The ordered apply where a wave has more droplets than the GPU holds at
once (at most 32 one-warp blocks a multiprocessor, 4736 of 148), so that many
of its droplets start only when others have ended, against the oracle's trace and
serial apply (IEEE float64 in the same order: heights identical in 99.9 % of
the cells, everything within 1e-5, the clamped count equal)."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as orc
from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["closed", "tilt"])
@pytest.mark.parametrize("droplets,wave", [(4737, 4737), (9001, 9001), (16001, 8000)])
def test_waves_above_the_resident_droplets_match_the_oracle(cuda, kind, droplets, wave):
    arr, params = window_world(kind, N=40, seed=5)
    ep, P = params.erosion, droplets
    ep.max_steps, ep.chunk = 48, wave
    g = gpu_window(arr)
    N, H = arr["N"], arr["H"]
    rng = np.random.default_rng(droplets)
    f, x, y, zero = np.zeros(P, np.int64), rng.random(P) * N, rng.random(P) * N, np.zeros(P)
    h = lambda t: t.detach().cpu().numpy().copy()
    o = orc.OracleState(height=h(g.height), sediment=h(g.sediment), discharge=h(g.discharge), momentum=h(g.momentum),
                        hardness=h(g.hardness), precip=h(g.precip), evap=h(g.evap), uplift=h(g.uplift), mask=arr["mask"],
                        metric=arr["metric"], metric_inv=arr["metric_inv"], N=N, H=H, spherical=False, height_unit_m=arr["cell"],
                        base=h(g.base), deposit_on_exit=True)
    s = gm.apply_spawns(g, ep, f, x, y, zero, zero, 1.0, wave=wave)
    o.pack()
    o.acc[...] = 0.0
    tp = orc.trace_params(o, ep, 1.0, wave / (1.0 * P))
    ap = orc.apply_params(o, ep, ep.iter_deposit / o.height_unit_m)
    cap = orc.change_list_cap(tp.max_steps)
    clamped = 0
    for c0 in range(0, P, wave):
        sl = slice(c0, c0 + wave)
        clamped += orc.apply(o, ap, orc.trace(o, tp, f[sl], x[sl], y[sl], zero[sl], zero[sl], 1.0), cap)[0]
    lib = orc.lib()
    lib.orc_fold(ctypes.c_int64(o.height.size), orc._p(o.height), orc._p(o.sediment), orc._p(o.acc), orc._p(o.mask))
    lib.orc_ema(ctypes.c_int64(o.height.size), orc._p(o.discharge), orc._p(o.momentum), orc._p(o.disch_track), orc._p(o.mom_track),
                orc._p(o.mask), ctypes.c_double(float(ep.ema)))
    assert s["droplets"] == P
    a = g.to_numpy()
    for k in ("height", "sediment", "discharge", "momentum", "pending"):
        np.testing.assert_allclose(a[k], getattr(o, k), rtol=1e-5, atol=1e-9, err_msg=k)
    assert np.mean(a["height"] == o.height) >= 0.999
    assert s["clamped"] == clamped
