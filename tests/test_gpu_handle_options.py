"""What the environment decides about a handle is decided when it is created: a
variable that changes before the solve's graph is captured, or captured again, or
before the bottom's precision is switched, changes nothing."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 32), 3, "fp32"), ((64, 64, 64), 4, "mixed"), ((64, 32, 32), 4, "mixed"), ((128, 64, 128), 4, "mixed")]


@pytest.mark.parametrize("shape,levels,precision", SHAPES)
def test_environment_after_creation(shape, levels, precision, monkeypatch):
    rng = np.random.default_rng(sum(shape))
    tag = np.where(rng.random(shape) < 0.9, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.03] = 2
    r = torch.from_numpy(np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)).cuda()
    tag = torch.from_numpy(tag).cuda()
    out = []
    for change in (False, True):
        for var in ("FLUB_NO_CLUSTER", "FLUB_COARSE_FP16"):
            monkeypatch.delenv(var, raising=False)
        mg = MGPCG(3, shape, levels, float, precision=precision)
        if change:
            monkeypatch.setenv("FLUB_NO_CLUSTER", "1")
            monkeypatch.setenv("FLUB_COARSE_FP16", "0")
        mg.set_tags(tag)
        x = []
        for step in ("reference", 2, 32):
            if step == 32:
                mg.set_bottom_precision(32)
            else:
                mg.set_schedule(step)
            mg.init(r, 1.0)
            mg.mask_interior()
            mg.solve(max_iters=3, eps=1e-12, abs_tol=0.0, rel_tol=0.0, smoother="phases")
            x += [mg.x.clone(), mg.apply_preconditioner(r)]
        out.append(x)
    assert all(bool(torch.isfinite(a).all()) for a in out[0])
    assert all(torch.equal(a, b) for a, b in zip(*out))
