"""The one-launch CG step of small grids (flub_gb300/csrc/cg_small.cuh) against
the four kernels it stands for: one block to sixteen, one and two groups a thread, a
last block that is not full, rows at the cluster's seams, a residual that is not 0
off the fluid, the iteration limit and convergence."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

SHAPES = [((8, 8, 8), 2), ((10, 6, 8), 1), ((16, 16, 16), 2), ((18, 22, 24), 1), ((32, 32, 32), 3), ((40, 32, 48), 2),
          ((16, 64, 64), 3)]


@pytest.mark.parametrize("masked", [True, False])
@pytest.mark.parametrize("max_iters", [2, 60])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_cg_step_matches_the_separate_kernels(shape, levels, max_iters, masked, monkeypatch):
    rng = np.random.default_rng(sum(shape))
    x = np.linspace(0, 1, shape[0])[:, None, None]
    tag = np.where(x + 0.1 * rng.standard_normal(shape) < 0.8, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.06] = 2
    r = rng.standard_normal(shape).astype(np.float32)
    if masked:
        r = np.where(tag == 1, r, 0).astype(np.float32)
    tag, r = torch.from_numpy(tag).cuda(), torch.from_numpy(r).cuda()
    out = []
    for loop in ("0", "1"):
        # the separate kernels: the "fraction" branch aside, only handles without clusters run them
        monkeypatch.setenv("FLUB_NO_CLUSTER", loop)
        mg = MGPCG(3, shape, levels, float)
        mg.set_tags(tag)
        mg.init(r, 1.0)
        if masked:
            mg.mask_interior()
        mg.solve(max_iters=max_iters, eps=1e-12, abs_tol=0.0, rel_tol=1e-10, smoother="phases")
        out.append((mg.info(), mg.x.double().cpu()))
    (a, xa), (b, xb) = out
    assert a["converged"] == b["converged"] and abs(a["iterations"] - b["iterations"]) <= (1 if a["converged"] else 0)
    assert abs(a["rtr0"] - b["rtr0"]) <= 1e-12 * b["rtr0"]
    # the FP64 sums differ in their last bits: the iterates agree to FP32 rounding, carried over the iterations
    assert float((xa - xb).norm()) <= 2e-5 * float(xb.norm())
