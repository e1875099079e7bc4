"""Cells whose neighbours hold no distance yet leave the Eikonal update early:
only where the full update would keep them.  Kept boundary values so large that
the middle neighbour value rounds, with both neighbours along one axis on the boundary;
a negative spacing; spacings up to the initial distance of 2."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import redistance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("h", [1.5, 0.75, 1.9, 0.004, 0.0, -0.25])
@pytest.mark.parametrize("n", [(3, 9, 40), (9, 3, 40), (9, 12, 3), (7, 8, 9)])
def test_cells_without_a_distance(n, h, sign):
    rng = np.random.default_rng(sum(n))
    phi = np.full(n, 3.0, np.float32)
    edge = np.ones(n, bool)
    edge[1:-1, 1:-1, 1:-1] = False
    big = rng.choice(np.float32([2.0 ** 24 + 2, 2.0 ** 25, 2.0 ** 26, 70000.25, 100.3, 2.0, 2.5, 1.0]), size=n)
    phi = (sign * np.where(edge, big, phi)).astype(np.float32)
    ref = O.redistance(phi, h, 0)
    g = torch.from_numpy(phi).cuda()
    redistance(g, h, 0)
    assert np.array_equal(g.cpu().numpy(), ref, equal_nan=True)
