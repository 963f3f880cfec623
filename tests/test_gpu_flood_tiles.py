"""The routing flood's 32 x 32 tiles and the sea mask's unions at sizes where
they can go wrong -- arrays one short of, equal to and one past whole tiles,
single rows of cells left over, faces smaller than a tile -- against the
oracle's heap flood and component labels, bit for bit on the interior (the
fixed point and the lowest id of a component do not depend on the order)."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from pgerosion import maps as gm
from pgerosion import synth
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,land", [(8, 0.5), (9, 0.3), (27, 0.4), (28, 0.15), (29, 0.6), (33, 0.4), (60, 0.05), (61, 0.5), (93, 0.3)])
def test_sphere_floods_equal_the_oracle(cuda, N, land):
    world = synth.earth_world(seed=N, N=N, cell_size_m=9773.0, land_fraction=land)
    params, _ = synth.config_params("earth")
    params.world.N_c = N
    g = gm.ErosionState.from_world(world)
    # rough ground: many small basins, on land and under the sea
    rng = np.random.default_rng(N)
    rough = rng.standard_normal(tuple(g.height.shape)) * 0.05
    g.height += torch.as_tensor(rough, device=g.height.device)
    g.exchange_halos()
    o = orc.OracleState.from_world(world, params)
    o.height[...] = g.height.cpu().numpy()
    eps = 0.05 / g.height_unit_m
    for fraction in (0.02, 0.5):
        assert g.refresh_base(fraction) == orc.refresh_base(o, fraction)
        assert g.base.cpu().numpy().tobytes() == o.base.tobytes()
        assert g.refresh_route(eps) > 0
        orc.refresh_route(o, eps)
        assert torch.equal(g.route[g.interior].cpu(), torch.as_tensor(o.route[o.interior]))


@pytest.mark.parametrize("N", [6, 28, 29, 60, 75])
def test_window_floods_equal_the_oracle(cuda, N):
    arr, _ = window_world("tilt", N=N, seed=N)
    arr["mask"][0, N // 2, 2 + N // 3:] = 0  # a wall outside the window, and frozen cells
    arr["mask"][0, 3:5, 3:] = 2
    g = gpu_window(arr)
    g.refresh_route(0.01)
    H = arr["H"]
    z = arr["height"].copy()
    owner = np.arange(z.size, dtype=np.int64).reshape(z.shape)
    want = orc.priority_flood_eps(z, arr["mask"], owner, H, N, 0.01, np.zeros_like(z))
    assert g.route.cpu().numpy().tobytes() == np.ascontiguousarray(want).tobytes()
