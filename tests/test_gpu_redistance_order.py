"""The chained half-sweeps of a redistance, each launched while the one in front
of it drains, against the same half-sweeps as separate calls with a
synchronisation between them."""
import numpy as np
import pytest
import torch

from flub_gb300 import _init_distance, _sweep, launch, redistance

pytestmark = pytest.mark.gpu

DIRECTIONS = ((1, 1, -1), (-1, 1, -1), (-1, -1, -1), (1, -1, -1), (1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1))


@pytest.mark.parametrize("n", [(24, 20, 16), (96, 65, 127), (128, 64, 256)])
def test_chained_sweeps_match_separate_ones(n):
    i, j, k = np.meshgrid(*(np.arange(s) + 0.5 for s in n), indexing="ij")
    h = 1.0 / max(n)
    r = np.sqrt((i - 0.4 * n[0]) ** 2 + (j - 0.6 * n[1]) ** 2 + (k - 0.5 * n[2]) ** 2)
    phi = ((r - min(n) / 3.1) * h + 0.1 * h * np.random.default_rng(sum(n)).standard_normal(n)).astype(np.float32)
    want = torch.from_numpy(phi).cuda()
    launch(_init_distance, dim=n, inputs=[want, h, 1])
    for _ in range(2):
        for d in DIRECTIONS:
            for odd in (0, 1):
                launch(_sweep, dim=n, inputs=[want, *d, odd, h])
                torch.cuda.synchronize()
    got = [torch.from_numpy(phi).cuda() for _ in range(20)]
    for g in got:
        redistance(g, h, 1, n_rounds=2)
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)
