"""The lake parks of one wave where a lake's run is longer than the 32 parks
walked at a time, several on one cell: the wave's own change lists, counted
down on the host in droplet order, give the rooms and the loads bit for bit
(the same float64 operations in the same order)."""
import numpy as np
import pytest

from pgerosion import _lib
from pgerosion import maps as gm
from tests.parity_cases import GOLDEN, changelist_rows, window_case
from tests.test_gpu_lake_parks import _park_window

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,scale", [(1, 1.0), (4, 1.0), (4, 1e6), (12, 3.0), (12, 1e-9)])
def test_long_runs_of_parks(cuda, copies, scale):
    case = window_case(GOLDEN / "lake_parks.npz")
    ep = case["params"]
    spawn = [np.concatenate([np.asarray(case[k])] * copies) for k in ("sp_face", "sp_x", "sp_y", "sp_sed", "sp_dir")]
    P = len(spawn[0])
    g, ref = _park_window(case), _park_window(case)
    for st in (g, ref):
        st.lake_room *= scale
    room, lake_id = g.lake_room.cpu().numpy().copy(), case["lake_id"].reshape(-1)
    res = gm.trace_changelist(ref, ep, *spawn, case["volume0"], case["conc_scale"], precision=_lib.PREC_F64, parks=True)
    load = np.zeros(lake_id.size)
    longest = np.zeros(len(room), int)
    for cells, delta, vol, _ in changelist_rows(res, case["cap"]):
        for c, d in zip(cells[vol == -3.0], delta[vol == -3.0]):
            lk = lake_id[c]
            if 0 <= lk < len(room):
                longest[lk] += 1
                take = min(d, room[lk])
                if take > 0.0:
                    load[c] += take
                    room[lk] -= take
    gm.apply_spawns(g, ep, *spawn, case["volume0"], wave=P, parks=True, conc_scale=case["conc_scale"])
    assert copies < 4 or longest.max() > 64
    assert g.lake_room.cpu().numpy().tobytes() == room.tobytes()
    assert g.lake_load.cpu().numpy().reshape(-1).tobytes() == load.tobytes()
