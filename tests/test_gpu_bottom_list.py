"""The FP64 bottom whose pairs are dealt out from a list (more pairs than threads):
full of fluid, with a part of it, with a single pair and with none, against the
oracle bit for bit."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

# bottoms of 2016, 2048, 1980, 1377, 432, 257 and 256 pairs (the last one is not listed)
SHAPES = [((24, 12, 14), 1), ((32, 32, 32), 2), ((36, 20, 44), 2), ((34, 18, 36), 2), ((96, 48, 48), 4),
          ((257, 1, 2), 1), ((16, 16, 16), 2)]


@pytest.mark.parametrize("fluid", ["full", "part", "one", "none"])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_fp64_bottom_from_list_bit_exact(shape, levels, fluid):
    rng = np.random.default_rng(sum(shape) + levels)
    tag = np.zeros(shape, np.int32)
    if fluid == "full":
        tag[:] = 1
    elif fluid == "part":
        tag[: (shape[0] + 2) // 3, : (shape[1] + 1) // 2] = 1
        tag[rng.random(shape) < 0.1] = 2
        tag[rng.random(shape) < 0.05] = 1
    elif fluid == "one":
        tag[-1:, -1:, -(1 << (levels - 1)):] = 1
    r = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    mg = MGPCG(3, shape, levels, float)
    mg.set_bottom_precision(64)
    mg.set_schedule(2, 3, 0.5)
    mg.set_tags(torch.from_numpy(tag).cuda())
    z = mg.apply_preconditioner(torch.from_numpy(r).cuda()).cpu().numpy()
    with O.schedule(2, 3, 0.5), O.bottom_fp64():
        assert np.array_equal(z, O.vcycle(r, O.tag_levels(tag, levels), np.float32))
