"""A caller's residual that holds NaN and infinities in air cells: the V-cycle
is that of a residual that is 0 there (a coarse cell with an air child is air, so
the restriction sums none of them), with level 0 in tiles, on colour-split rows,
in natural order and in the coarse kernel."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

# tiles with rows of every item width; colour-split; coarse kernel; one level alone
SHAPES = [((64, 64, 64), 2), ((42, 44, 52), 2), ((50, 36, 90), 1), ((34, 30, 104), 2), ((104, 72, 88), 3),
          ((128, 128, 128), 4), ((32, 32, 32), 3), ((16, 16, 16), 1)]


@pytest.mark.parametrize("nu", [1, 2, 3])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_non_finite_residual_in_air(shape, levels, nu):
    rng = np.random.default_rng(sum(shape) + nu)
    x = np.linspace(0, 1, shape[0])[:, None, None]
    tag = np.where(x + 0.1 * rng.standard_normal(shape) < 0.7, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.05] = 2
    clean = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    odd = rng.choice(np.float32([np.nan, np.inf, -np.inf, 1e38, 0.0]), size=shape)
    r = np.where(tag == 0, odd, clean).astype(np.float32)
    with O.schedule(nu, 3, 0.5):
        want = O.vcycle(clean, O.tag_levels(tag, levels), np.float32)
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    mg.set_schedule(nu, 3, 0.5)
    z = torch.full(shape, float("nan"), device="cuda")
    z = mg.apply_preconditioner(torch.from_numpy(r).cuda(), z).cpu().numpy()
    assert np.isfinite(want).all() and np.array_equal(z, want)


@pytest.mark.parametrize("nu", [1, 3])
@pytest.mark.parametrize("shape,levels", [((64, 64, 64), 3), ((32, 32, 32), 3)])
def test_non_finite_residual_in_air_mixed(shape, levels, nu):
    """Mixed precision against itself with 0 in the air (FP16 turns 1e38 into an infinity)."""
    rng = np.random.default_rng(nu)
    tag = np.where(rng.random(shape) < 0.7, 1, 0).astype(np.int32)
    tag[rng.random(shape) < 0.05] = 2
    clean = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    r = np.where(tag == 0, rng.choice(np.float32([np.nan, np.inf, 1e38]), size=shape), clean).astype(np.float32)
    mg = MGPCG(3, shape, levels, float, precision="mixed")
    mg.set_tags(torch.from_numpy(tag).cuda())
    mg.set_schedule(nu, 3, 0.5)
    want = mg.apply_preconditioner(torch.from_numpy(clean).cuda())
    got = mg.apply_preconditioner(torch.from_numpy(r).cuda())
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)
