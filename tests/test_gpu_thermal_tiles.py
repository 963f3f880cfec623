"""The thermal pass's 16 x 32 tiles against the oracle's three sweeps, bit for
bit (IEEE float64 in the same order): arrays around whole tiles and smaller
than one, masks with frozen and outside cells across tile edges, seas that
fill up (the inflow's share), the outflow cap, with and without creep."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("creep", [0.0, 0.05])
@pytest.mark.parametrize("N", [4, 11, 12, 13, 27, 28, 29, 44, 61, 92])
def test_thermal_equals_the_oracle(cuda, N, creep):
    arr, params = window_world("tilt", N=N, seed=N)
    ep = params.erosion
    ep.creep_rate, ep.thermal_max = creep, 20.0 if N % 2 else 0.0
    rng = np.random.default_rng(N)
    sh = arr["height"].shape
    arr["height"] = arr["height"] + rng.standard_normal(sh) * 0.6  # steep: every cell moves something
    arr["mask"][0, N // 2, 1:] = 2
    arr["mask"][0, 2:, N // 3] = 0
    g = gpu_window(arr)
    sed = rng.random(sh) * 0.3
    g.sediment.copy_(torch.as_tensor(sed))
    hard = rng.random(sh).astype(np.float32)
    g.hardness.copy_(torch.as_tensor(hard))
    g.base.copy_(torch.as_tensor(np.where(rng.random(sh) < 0.2, 0.3, 0.0)))
    z = np.zeros(sh)
    o = orc.OracleState(height=arr["height"].copy(), sediment=sed.copy(), discharge=z.copy(), momentum=np.zeros(sh + (2,)), hardness=hard,
                        precip=np.ones(sh, np.float32), evap=np.ones(sh, np.float32), uplift=z.copy(), mask=arr["mask"],
                        metric=arr["metric"], metric_inv=arr["metric_inv"], N=N, H=arr["H"], spherical=False, height_unit_m=arr["cell"],
                        base=g.base.cpu().numpy().copy())
    gm.thermal_erosion(g, params)
    orc.thermal_erosion(o, params)
    assert not np.array_equal(o.height + o.sediment, arr["height"] + sed)
    assert np.array_equal(g.height.cpu().numpy(), o.height) and np.array_equal(g.sediment.cpu().numpy(), o.sediment)
