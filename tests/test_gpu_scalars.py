"""The map passes' scalars at the counts where they can go wrong, against
numpy to the bit: the spawn total in numpy's pairwise order (ranges shorter
than eight values, around a leaf of 128, unbalanced halves, several blocks of
nodes) and the datum's order statistic (ties, both zeros, all cells land or
none, digits that all keys share)."""
import numpy as np
import pytest
import torch

from pgerosion import maps as gm
from pgerosion import synth

pytestmark = pytest.mark.gpu


def _state(N, seed=0):
    return gm.ErosionState.from_world(synth.earth_world(seed=seed, N=N, cell_size_m=9773.0))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 127, 128, 129, 135, 136, 137, 255, 256, 257, 264, 1000, 1025, 4097, 9599, 9600])
def test_pairwise_total_equals_numpy(cuda, n):
    g = _state(40)
    rng = np.random.default_rng(n)
    H, N = g.H, g.N
    mask = np.zeros((6, N, N), np.uint8).reshape(-1)
    mask[rng.permutation(mask.size)[:n]] = 1
    w = (10.0 ** rng.uniform(-6, 3, mask.size)).astype(np.float32)
    g.mask = torch.zeros(g.height.shape, dtype=torch.uint8, device="cuda")
    g.mask[g.interior] = torch.as_tensor(mask.reshape(6, N, N), device="cuda")
    g.precip[g.interior] = torch.as_tensor(w.reshape(6, N, N), device="cuda")
    g.height.fill_(1.0)
    r = gm.spawn_rain(g, rng.random(4), rng.random((4, 2)))
    assert r["n_spawnable"] == n
    assert r["total"] == w[mask == 1].astype(np.float64).sum()


def test_pairwise_mean_of_a_larger_field_equals_numpy(cuda):
    g = _state(301)  # 543,606 values: 64 blocks of nodes
    rng = np.random.default_rng(5)
    u = rng.standard_normal(tuple(g.height.shape)) * 10.0 ** rng.uniform(-8, 4, tuple(g.height.shape))
    g.uplift.copy_(torch.as_tensor(u))
    h0 = g.height.cpu().numpy()
    gm.apply_uplift(g)
    want = h0 + (u - u[g.interior].mean())
    assert np.array_equal(g.height.cpu().numpy(), want)


@pytest.mark.parametrize("kind", ["mixed", "ties", "equal", "zeros", "close"])
@pytest.mark.parametrize("fraction", [0.0, 0.29, 0.5, 1.0])
def test_datum_equals_the_order_statistic(cuda, kind, fraction):
    g = _state(37)
    rng = np.random.default_rng(3)
    sh = tuple(g.height.shape)
    z = {"mixed": rng.standard_normal(sh) * 10.0 ** rng.uniform(-9, 9, sh), "ties": np.round(rng.standard_normal(sh)),
         "equal": np.full(sh, -2.5), "zeros": np.where(rng.random(sh) < 0.5, 0.0, -0.0) + np.where(rng.random(sh) < 0.3, 1.0, 0.0),
         "close": 1.0 + rng.integers(0, 50, sh) * 2.0 ** -52}[kind]
    g.height.copy_(torch.as_tensor(z))
    g.sediment.zero_()
    q = gm.hold_datum(g, fraction)
    v = np.sort((z + 0.0)[g.interior].reshape(-1))
    M = v.size
    land = int(np.round(fraction * M))
    want = v[M - 1] + 1.0 if land == 0 else v[M - land]
    assert q == want
    assert np.array_equal(g.height.cpu().numpy(), z - q)
