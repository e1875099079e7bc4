"""A caller's r and z of the V-cycle at any 4-byte address, on rows that are not
whole 8-cell groups: level 0 in tiles, in the coarse kernel and in scalar sweeps."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off_r,off_z", [(1, 0), (0, 1), (1, 1), (3, 2), (2, 2)])
@pytest.mark.parametrize("shape,levels", [((42, 44, 52), 2), ((34, 30, 108), 2), ((12, 10, 20), 2), ((50, 36, 90), 1)])
def test_vcycle_arrays_4_byte_aligned(shape, levels, off_r, off_z):
    rng = np.random.default_rng(sum(shape))
    tag = np.where(rng.random(shape) < 0.8, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.05] = 2
    r = torch.from_numpy(np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)).cuda()
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    mg.set_schedule(3, 3, 0.5)
    want = mg.apply_preconditioner(r)
    ro = torch.empty(r.numel() + off_r, device="cuda")[off_r:].view(shape)
    zo = torch.full((r.numel() + off_z,), float("nan"), device="cuda")[off_z:].view(shape)
    ro.copy_(r)
    assert ro.data_ptr() % 16 == 4 * off_r and zo.data_ptr() % 16 == 4 * off_z
    assert torch.equal(mg.apply_preconditioner(ro, zo), want)
    assert torch.equal(mg.apply_preconditioner(r), want)  # and the handle's buffers after it
