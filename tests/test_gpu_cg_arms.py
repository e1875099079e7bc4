"""FLUB_NO_CLUSTER=1 runs the separate CG kernels at every size, the smallest
included: four kernels between two V-cycles instead of two."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu


# shapes whose V-cycle is one launch with and without clusters
@pytest.mark.parametrize("shape,levels", [((8, 8, 8), 2), ((10, 6, 8), 1), ((16, 16, 8), 1), ((16, 16, 16), 2)])
def test_separate_cg_kernels(shape, levels, monkeypatch):
    rng = np.random.default_rng(sum(shape))
    tag = np.where(rng.random(shape) < 0.8, 1, 0).astype(np.int32)
    r = torch.from_numpy(np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)).cuda()
    tag = torch.from_numpy(tag).cuda()
    iters, kernels = 6, []
    for off in ("0", "1"):
        monkeypatch.setenv("FLUB_NO_CLUSTER", off)
        mg = MGPCG(3, shape, levels, float)
        mg.set_schedule(1, 1, 0.5)  # a V-cycle too weak to converge in these iterations
        mg.set_tags(tag)
        mg.init(r, 1.0)
        mg.mask_interior()
        before = mg.kernels_executed()
        mg.solve(max_iters=iters, eps=1e-12, abs_tol=0.0, rel_tol=0.0, smoother="phases")
        assert mg.info()["iterations"] == iters
        kernels.append(mg.kernels_executed() - before)
    assert kernels[1] - kernels[0] == 2 * iters
