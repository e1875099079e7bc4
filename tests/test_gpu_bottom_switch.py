"""Switching the bottom's precision on a handle that has its tags already, at
shapes where the FP64 bottom moves a level out of the coarse kernel: the V-cycle
is that of a handle that had the precision before the tags."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("shape,levels", [((16, 2, 1024), 2), ((32, 4, 2048), 3), ((64, 32, 64), 3)])
def test_bottom_precision_after_tags(shape, levels, precision):
    rng = np.random.default_rng(sum(shape))
    tag = np.where(rng.random(shape) < 0.9, 1, 0).astype(np.int32)
    r = torch.from_numpy(np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)).cuda()
    tag = torch.from_numpy(tag).cuda()

    def z(mg):
        return mg.apply_preconditioner(r)

    want = {}
    for bits in (32, 64):
        mg = MGPCG(3, shape, levels, float, precision=precision)
        mg.set_bottom_precision(bits)
        mg.set_tags(tag)
        want[bits] = z(mg)
        assert bool(torch.isfinite(want[bits]).all()) and float(want[bits].abs().max()) > 0.0
    mg = MGPCG(3, shape, levels, float, precision=precision)
    mg.set_tags(tag)
    for bits in (64, 32, 64):
        mg.set_bottom_precision(bits)
        assert torch.equal(z(mg), want[bits])
