"""A V-cycle or a sweep enqueued directly behind set_tags, with nothing between
them on the stream: it uses the lists and words of the new tags, on grids whose
first launch is the coarse kernel, a tile launch, a colour-split sweep, a scalar
sweep, or the FP16 copy of the residual."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32, 32), 3), ((64, 64, 64), 4), ((42, 44, 52), 2), ((128, 128, 128), 4), ((128, 160, 128), 4)]


def _tags(shape, seed):
    rng = np.random.default_rng(seed)
    tag = np.zeros(shape, np.int32)
    if seed % 3:  # every third one is full of fluid, so that the lists' lengths differ widely
        lo = [int(rng.integers(0, n // 2)) for n in shape]
        hi = [int(rng.integers(l + n // 4, n + 1)) for l, n in zip(lo, shape)]
        tag[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = 1
    else:
        tag[:] = 1
    tag[rng.random(shape) < 0.03] = 2
    return torch.from_numpy(tag).cuda()


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_vcycle_directly_after_set_tags(shape, levels, precision):
    if precision == "mixed" and shape[2] % 8:
        pytest.skip("mixed precision needs rows of whole 8-cell groups")
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(shape).astype(np.float32)).cuda()
    tags = [_tags(shape, seed) for seed in range(6)]
    want = []
    for tag in tags:
        mg = MGPCG(3, shape, levels, float, precision=precision)
        mg.set_schedule(2, 3, 0.5)
        mg.set_tags(tag)
        torch.cuda.synchronize()
        want.append(mg.apply_preconditioner(r))
        torch.cuda.synchronize()
    assert all(bool(torch.isfinite(w).all()) for w in want)
    used = MGPCG(3, shape, levels, float, precision=precision)
    used.set_schedule(2, 3, 0.5)
    order = np.random.default_rng(2).integers(0, len(tags), 40)
    z = [torch.empty(shape, device="cuda") for _ in order]
    torch.cuda.synchronize()
    for n, q in enumerate(order):
        used.set_tags(tags[q])
        used.apply_preconditioner(r, z[n])
    torch.cuda.synchronize()
    for n, q in enumerate(order):
        assert torch.equal(z[n], want[q]), n


@pytest.mark.parametrize("shape,levels", SHAPES)
def test_sweep_directly_after_set_tags(shape, levels):
    """Half-sweeps of level 0's correction, which set_tags clears, with the residual of init."""
    n = int(np.prod(shape))
    step = (4 * n + 255) // 256 * 256  # the residual, then the correction
    r = torch.from_numpy(np.random.default_rng(3).standard_normal(shape).astype(np.float32)).cuda()
    tags = [_tags(shape, seed) for seed in range(6)]

    def swept(mg, tag, wait):
        mg.set_tags(tag)
        if wait:
            torch.cuda.synchronize()
        mg.smooth(0, 0)
        mg.smooth(0, 1)
        return mg._view(mg.r0.data_ptr() + step, n).clone()

    want = []
    for tag in tags:
        mg = MGPCG(3, shape, levels, float)
        mg.init(r, 1.0)
        want.append(swept(mg, tag, True))
        torch.cuda.synchronize()
        assert float(want[-1].abs().max()) > 0.0
    used = MGPCG(3, shape, levels, float)
    used.init(r, 1.0)
    for q in np.random.default_rng(4).integers(0, len(tags), 20):
        assert torch.equal(swept(used, tags[q], False), want[q])
