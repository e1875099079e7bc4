"""New tags on a used handle (flub_gb300/csrc/setup_levels.cuh): lists, words
and cleared buffers are those of a fresh handle, on levels of whole 8-cell rows and
not, with one to many blocks a level, in FP32 and FP16."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 32), 3, "fp32"), ((8, 8, 8), 2, "fp32"), ((10, 6, 8), 1, "fp32"), ((104, 72, 88), 3, "fp32"),
          ((48, 40, 44), 2, "fp32"), ((1028, 32, 16), 3, "fp32"), ((128, 160, 128), 4, "fp32"),
          ((64, 64, 64), 3, "mixed"), ((128, 128, 128), 4, "mixed")]


def _case(shape, seed):
    rng = np.random.default_rng(seed)
    tag = np.zeros(shape, np.int32)
    lo = [rng.integers(0, n // 2) for n in shape]
    hi = [rng.integers(l + n // 2, n + 1) for l, n in zip(lo, shape)]
    tag[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = 1
    tag[rng.random(shape) < 0.03] = 2
    r = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    return torch.from_numpy(tag).cuda(), torch.from_numpy(r).cuda()


@pytest.mark.parametrize("shape,levels,precision", SHAPES)
def test_retagged_handle_solves_as_a_fresh_one(shape, levels, precision):
    def solve(mg, tag, r):
        mg.set_tags(tag)
        mg.init(r, 1.0)
        mg.mask_interior()
        mg.solve(max_iters=3, eps=1e-12, abs_tol=0.0, rel_tol=0.0, smoother="phases")
        return mg.x.clone()

    used = MGPCG(3, shape, levels, float, precision=precision)
    for seed in range(3):
        tag, r = _case(shape, seed)
        x = solve(used, tag, r)
        assert torch.equal(x, solve(MGPCG(3, shape, levels, float, precision=precision), tag, r))
        assert bool(torch.isfinite(x).all())
