"""The sea mask's component labels at a size where thousands of unions run at
once (N_c = 512, seas and basins of every size): each cell's label is its
component's lowest cell id, so a label is its own label, and no two cells that
touch have different ones."""
import numpy as np
import pytest
import torch

from pgerosion import maps as gm
from pgerosion import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rough,land", [(0.0, 0.3), (0.3, 0.5), (5.0, 0.45)])
def test_labels_are_roots_and_agree_across_neighbours(cuda, rough, land):
    N = 512
    g = gm.ErosionState.from_world(synth.earth_world(seed=3, N=N, cell_size_m=9773.0, land_fraction=land))
    gen = torch.Generator(device="cuda").manual_seed(1)
    g.height += rough * 0.1 * torch.randn(g.height.shape, dtype=torch.float64, device="cuda", generator=gen)
    g.exchange_halos()
    H, NE = g.H, g.NE
    own = g.grid.owner
    r = own % (NE * NE)
    cell = torch.as_tensor(((own // (NE * NE)) * N + r // NE - H) * N + r % NE - H, device="cuda")
    first = None
    for _ in range(3):
        base, labels = g._sea_base(0.02)
        lab = labels.reshape(-1).long()
        wet = lab >= 0
        assert torch.equal(wet.view(6, N, N), (g.height + g.sediment)[g.interior].float() < 0)
        assert torch.equal(lab[lab[wet]], lab[wet])  # a root's label is itself
        assert bool((lab[wet] <= torch.arange(lab.numel(), device="cuda")[wet]).all())
        for a, b in ((1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1)):
            q = cell[:, H + a:H + a + N, H + b:H + b + N].reshape(-1)
            both = wet & wet[q]
            assert torch.equal(lab[both], lab[q][both])
        if first is not None:
            assert torch.equal(first[0], lab) and torch.equal(first[1], base)
        first = (lab, base)
