"""The wave apply's warps at the counts where they wait for one another: lists
are closed and droplets taken once six lanes of a warp wait, or none is left
walking, and final deposits end as soon as nothing is left to place.  A taped
pass applies every deposit, so it must come out bit for bit the same as the
pass without a tape, for waves of a few droplets and of more than a warp's
refills; and the stats count every entry either way."""
import numpy as np
import pytest
import torch

from pgerosion import _lib, adjoint
from pgerosion import maps as gm
from tests.parity_cases import gpu_window, window_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["closed", "tilt", "shelf"])
@pytest.mark.parametrize("droplets,max_steps", [(1, 40), (2, 1), (5, 7), (6, 40), (7, 40), (31, 5), (33, 40), (997, 40), (5000, 3)])
def test_taped_and_plain_passes_are_identical(cuda, kind, droplets, max_steps):
    arr, params = window_world(kind, N=40, seed=droplets)
    ep = params.erosion
    ep.max_steps = max_steps
    rng = np.random.default_rng(droplets)
    x, y = rng.random(droplets) * 40.0, rng.random(droplets) * 40.0
    sed, dirs = np.where(rng.random(droplets) < 0.5, 0.02 * rng.random(droplets), 0.0), rng.random(droplets) * 6.0
    out = []
    for tapes in (None, adjoint.TapeStore(torch.device("cuda"))):
        g = gpu_window(arr)
        s = gm.apply_spawns(g, ep, np.zeros(droplets, np.int64), x, y, sed, dirs, 1.0, wave=max(droplets // 3, 1),
                            apply=_lib.APPLY_WAVE, tape=tapes)
        out.append((s, g.to_numpy()))
    (s0, a0), (s1, a1) = out
    assert s0["droplets"] == droplets
    for k in s0:
        if k != "seconds":
            assert s0[k] == s1[k], k
    for k in a0:
        if isinstance(a0[k], np.ndarray):
            assert a0[k].tobytes() == a1[k].tobytes(), k
