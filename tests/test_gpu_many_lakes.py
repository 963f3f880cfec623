"""The lake parks of one wave over many lakes at once -- lakes of one park,
of a few, and of more than the 32 parks read at a time, side by side in the
sorted parks: the wave's own change lists, counted down on the host in droplet
order, give the rooms and the loads bit for bit (the same float64 operations
in the same order)."""
import numpy as np
import pytest
import torch

from pgerosion import _lib
from pgerosion import maps as gm
from tests.parity_cases import changelist_rows, gpu_window, window_world

pytestmark = pytest.mark.gpu


def lake_blocks(N, cells_a_lake):
    """A coast whose every other 2 x 2 block is a lake's, ``cells_a_lake`` cells of them in a row of the
    array to a lake (0: one lake)."""
    arr, params = window_world("tilt", N=N)
    params.erosion.max_steps, params.erosion.lake_trap = 64, 0.9
    g = gpu_window(arr)
    NE = g.height.shape[1]
    i, j = np.meshgrid(np.arange(NE), np.arange(NE), indexing="ij")
    water = (i % 4 < 2) & (j % 4 < 2)
    ids = np.full((NE, NE), -1, np.int32)
    n = int(water.sum())
    ids[water] = np.arange(n) // cells_a_lake if cells_a_lake else 0
    dev = g.height.device
    g.route = (g.height + g.sediment + torch.as_tensor(np.where(water, 0.01, 0.0), device=dev)[None]).contiguous()
    g.lake_flag = torch.as_tensor(np.where(water, 2, 0).astype(np.uint8)[None], device=dev)
    g.lake_id = torch.as_tensor(ids[None], device=dev)
    g.lake_room = torch.as_tensor(np.random.default_rng(N).random(int(ids.max()) + 1) * 2.0, device=dev)
    g.lake_load = torch.zeros_like(g.height)
    return g, params.erosion


def spawns(P, N):
    rng = np.random.default_rng(P)
    return np.zeros(P, np.int64), rng.random(P) * N, rng.random(P) * N, np.full(P, 1.0), rng.random(P) * 6.0


@pytest.mark.parametrize("cells_a_lake", [1, 4, 37, 500, 0])
@pytest.mark.parametrize("droplets", [3, 700, 2048])
def test_many_lakes(cuda, droplets, cells_a_lake):
    N, P = 96, droplets
    (g, ep), (ref, _) = lake_blocks(N, cells_a_lake), lake_blocks(N, cells_a_lake)
    room, ids = g.lake_room.cpu().numpy().copy(), g.lake_id.cpu().numpy().reshape(-1)
    sp = spawns(P, N)
    res = gm.trace_changelist(ref, ep, *sp, 1.0, 1.0, precision=_lib.PREC_F64, parks=True)
    load, parks = np.zeros(ids.size), np.zeros(len(room), int)
    for cells, delta, vol, _ in changelist_rows(res, len(res["cl_cell"]) // P):
        for c, d in zip(cells[vol == -3.0], delta[vol == -3.0]):
            lk = ids[c]
            if lk >= 0:
                parks[lk] += 1
                take = min(d, room[lk])
                if take > 0.0:
                    load[c] += take
                    room[lk] -= take
    gm.apply_spawns(g, ep, *sp, 1.0, wave=P, parks=True, conc_scale=1.0)
    assert parks.sum() > P // 4  # the parks the test is for, and lakes that run out
    assert droplets < 700 or (room == 0.0).any()
    assert g.lake_room.cpu().numpy().tobytes() == room.tobytes()
    assert g.lake_load.cpu().numpy().reshape(-1).tobytes() == load.tobytes()
