"""The thermal pass over the six faces, unmasked, on either side of the size
(592 tiles a face) from which a block takes its tile of every face in turn,
the distances kept from face to face, against the oracle's three sweeps bit
for bit (IEEE float64 in the same order)."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from pgerosion import maps as gm
from pgerosion.params import ErosionParams, WorldGroup, WorldParams, plain_knobs
from pgerosion.synth import plain_small_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("creep", [0.0, 0.05])
@pytest.mark.parametrize("N", [29, 378, 380, 381, 396, 399])  # 24 x 24 tiles a face up to 380, 25 x 25 from 381 on
def test_six_faces_equal_the_oracle(cuda, N, creep):
    world = plain_small_world(seed=N, N=N)
    ep = ErosionParams(uplift_mode="stack", **plain_knobs())
    ep.creep_rate, ep.thermal_max = creep, 20.0 if N % 2 else 0.0
    params = WorldParams(world=WorldGroup(seed=N, N_c=N, cell_size_m=50.0, land_fraction=0.30, halo=2), erosion=ep)
    g = gm.ErosionState.from_world(world)
    o = orc.OracleState.from_world(world, params)
    rng = np.random.default_rng(N)
    sh = o.height.shape
    o.height = o.height + rng.standard_normal(sh) * 0.6  # steep, and each face of its own: every cell moves something
    o.sediment = rng.random(sh) * 0.3
    o.hardness = rng.random(sh).astype(np.float32)
    o.base = np.where(rng.random(sh) < 0.2, 0.3, 0.0)
    for k in ("height", "sediment", "hardness", "base"):
        getattr(g, k).copy_(torch.as_tensor(getattr(o, k)))
    before = o.height + o.sediment
    gm.thermal_erosion(g, params)
    orc.thermal_erosion(o, params)
    assert all(not np.array_equal((o.height + o.sediment)[f], before[f]) for f in range(6))
    assert np.array_equal(g.height.cpu().numpy(), o.height) and np.array_equal(g.sediment.cpu().numpy(), o.sediment)
