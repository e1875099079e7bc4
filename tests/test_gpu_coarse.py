"""The one-launch coarse levels (flub_gb300/csrc/coarse.cuh) against the
oracle's V-cycle, bit for bit: rows of every item width (nz / 2 a multiple of
4, of 2, odd), slabs of one to several planes with a short last one, levels
that end inside the cluster and levels that hand over to one block, with and
without clusters."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

# shape, levels
SHAPES = [((16, 16, 16), 1), ((8, 8, 8), 2), ((2, 3, 2), 1), ((6, 10, 12), 2), ((26, 18, 22), 1), ((31, 12, 36), 1),
          ((36, 20, 24), 2), ((40, 24, 52), 2), ((64, 16, 64), 2), ((32, 32, 32), 3), ((48, 40, 32), 3),
          ((52, 36, 44), 2), ((60, 32, 32), 2), ((16, 64, 64), 2), ((104, 72, 88), 3)]


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    x = np.linspace(0, 1, shape[0])[:, None, None]
    tag = np.where(x + 0.1 * rng.standard_normal(shape) < 0.8, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.06] = 2
    r = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    return tag, r


@pytest.mark.parametrize("no_cluster", ["0", "1"])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_coarse_levels_bit_exact(shape, levels, no_cluster, monkeypatch):
    monkeypatch.setenv("FLUB_NO_CLUSTER", no_cluster)
    tag, r = _case(shape, sum(shape))
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    rd = torch.from_numpy(r).cuda()
    tags = O.tag_levels(tag, levels)
    z = mg.apply_preconditioner(rd).cpu().numpy()
    assert np.array_equal(z, O.vcycle(r, tags, np.float32))
    mg.set_schedule(2, 4, 0.5)
    z = mg.apply_preconditioner(rd).cpu().numpy()
    with O.schedule(2, 4, 0.5):
        assert np.array_equal(z, O.vcycle(r, tags, np.float32))


# shape, levels, precision: rows of every item width with and without a halo
# along k, tiles with remainders along every axis, levels just above the coarse
# kernel's, and level 0 itself
BLOCKED = [((48, 40, 44), 2), ((64, 64, 64), 2), ((41, 44, 42), 1), ((42, 44, 52), 2), ((128, 32, 64), 3),
           ((50, 36, 88), 2), ((34, 30, 104), 2), ((128, 64, 128), 4), ((104, 72, 88), 3)]


@pytest.mark.parametrize("nu", [1, 2, 3, 4])
@pytest.mark.parametrize("shape,levels", BLOCKED)
def test_blocked_smoothing_bit_exact(shape, levels, nu):
    """smooth_block.cuh: one and two iterations a launch, odd and even numbers
    of launches a side (the ping-pong of the buffers)."""
    tag, r = _case(shape, sum(shape) + nu)
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    mg.set_schedule(nu, 3, 0.5)
    rd = torch.from_numpy(r).cuda()
    tags = O.tag_levels(tag, levels)
    with O.schedule(nu, 3, 0.5):
        want = O.vcycle(r, tags, np.float32)
    z = torch.full(shape, float("nan"), device="cuda")  # every cell is written
    assert np.array_equal(mg.apply_preconditioner(rd, z).cpu().numpy(), want)
    assert np.array_equal(mg.apply_preconditioner(rd, rd.clone()).cpu().numpy(), want)
