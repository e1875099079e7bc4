"""The colour-split half-sweeps (flub_gb300/csrc/smooth_split.cuh) against the
oracle's V-cycle, bit for bit, at level 0 and below: solids, air and walls on every side of a group,
1 to 3 iterations a side, a residual that holds anything off the fluid; and
after a V-cycle that ran in natural order on the same handle."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu

SHAPES = [((104, 72, 88), 3), ((66, 50, 80), 2), ((128, 128, 128), 4), ((34, 258, 16), 2), ((130, 66, 8), 2),
          ((1028, 32, 16), 3), ((256, 192, 80), 3)]


def _case(shape, seed, solids):
    rng = np.random.default_rng(seed)
    x = np.linspace(0, 1, shape[0])[:, None, None]
    tag = np.where(x + 0.05 * rng.standard_normal(shape) < 0.8, 1, 0).astype(np.int32)
    tag[rng.random(shape) < solids] = 2
    r = np.where(tag == 1, rng.standard_normal(shape), 0).astype(np.float32)
    return tag, r


@pytest.mark.parametrize("solids", [0.0, 0.05])
@pytest.mark.parametrize("nu", [1, 2, 3])
@pytest.mark.parametrize("shape,levels", SHAPES)
def test_split_bit_exact(shape, levels, nu, solids):
    tag, r = _case(shape, sum(shape) + nu, solids)
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    mg.set_schedule(nu, 3, 0.5)
    rd = torch.from_numpy(r).cuda()
    with O.schedule(nu, 3, 0.5):
        want = O.vcycle(r, O.tag_levels(tag, levels), np.float32)
    z = torch.full(shape, float("nan"), device="cuda")  # every cell is written
    assert np.array_equal(mg.apply_preconditioner(rd, z).cpu().numpy(), want)
    inplace = rd.clone()  # z the array of r: level 0 in natural order
    mg.apply_preconditioner(inplace, inplace)
    assert np.array_equal(mg.apply_preconditioner(rd).cpu().numpy(), want)


@pytest.mark.parametrize("shape,levels", [((64, 64, 64), 3), ((128, 32, 64), 3), ((128, 128, 128), 4)])
def test_split_mixed_after_natural(shape, levels):
    """A caller's z in mixed precision runs level 0 in natural order; the solve
    after it is the one of a fresh handle."""
    tag, r = _case(shape, sum(shape), 0.05)
    rd = torch.from_numpy(r).cuda()
    x = []
    for natural in (False, True):
        mg = MGPCG(3, shape, levels, float, precision="mixed")
        mg.set_tags(torch.from_numpy(tag).cuda())
        if natural:
            mg.apply_preconditioner(rd)
        mg.init(rd, 1.0)
        mg.solve(max_iters=4, eps=1e-12, abs_tol=1e-12, rel_tol=1e-12, smoother="phases")
        x.append(mg.x.cpu().numpy())
    assert np.isfinite(x[0]).all() and np.array_equal(x[0], x[1])


@pytest.mark.parametrize("nu", [1, 3])
@pytest.mark.parametrize("shape,levels", [((2048, 32, 16), 3), ((256, 256, 128), 4)])
def test_split_mixed_lower_levels(shape, levels, nu, monkeypatch):
    """FP16 levels below level 0: the values stored are those of the natural-order sweeps."""
    tag, r = _case(shape, sum(shape), 0.05)
    rd = torch.from_numpy(r).cuda()
    z = []
    for off in ("1", "0"):
        monkeypatch.setenv("FLUB_NO_SPLIT", off)
        mg = MGPCG(3, shape, levels, float, precision="mixed")
        mg.set_tags(torch.from_numpy(tag).cuda())
        mg.set_schedule(nu, 3, 0.5)
        mg.init(rd, 1.0)
        mg.solve(max_iters=3, eps=1e-12, abs_tol=1e-12, rel_tol=1e-12, smoother="phases")
        z.append((mg.apply_preconditioner(rd).cpu().numpy(), mg.x.cpu().numpy()))
    assert np.isfinite(z[0][1]).all()
    assert np.array_equal(z[0][0], z[1][0]) and np.array_equal(z[0][1], z[1][1])


@pytest.mark.parametrize("solids", [0.0, 0.05])
@pytest.mark.parametrize("shape,levels", [((32, 32, 32), 3), ((10, 6, 8), 1), ((66, 50, 80), 2), ((34, 258, 16), 2)])
def test_solver_matvec_bit_exact(shape, levels, solids):
    """A p of the solve's first iteration: rows read 32 bytes a lane, their ends
    from the neighbouring lanes, a last warp that is not full."""
    tag, r = _case(shape, sum(shape), solids)
    mg = MGPCG(3, shape, levels, float)
    mg.set_tags(torch.from_numpy(tag).cuda())
    rd = torch.from_numpy(r).cuda()
    mg.init(rd, 1.0)
    mg.mask_interior()
    mg.solve(max_iters=1, eps=1e-12, abs_tol=0.0, rel_tol=0.0, smoother="phases")
    n = r.size
    step = (4 * n + 255) // 256 * 256  # x, p, A p lie one after the other
    Ap = mg._view(mg.x.data_ptr() + 2 * step, n)
    assert torch.equal(Ap, mg.matvec(mg.apply_preconditioner(rd)))


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_split_arrays_16_byte_aligned(precision):
    """A caller's r and z at an address that is a multiple of 16 but not of 32."""
    shape, levels = (128, 128, 128), 4
    tag, r = _case(shape, 5, 0.02)
    mg = MGPCG(3, shape, levels, float, precision=precision)
    mg.set_tags(torch.from_numpy(tag).cuda())
    rd = torch.from_numpy(r).cuda()
    ro = torch.empty(r.size + 4, device="cuda")[4:].view(shape)
    zo = torch.empty(r.size + 4, device="cuda")[4:].view(shape)
    ro.copy_(rd)
    assert ro.data_ptr() % 32 == 16 and zo.data_ptr() % 32 == 16
    assert torch.equal(mg.apply_preconditioner(ro, zo), mg.apply_preconditioner(rd))


@pytest.mark.parametrize("nu", [1, 2, 5])
@pytest.mark.parametrize("shape,levels", [((88, 64, 64), 4), ((176, 128, 128), 5), ((48, 48, 64), 3), ((64, 64, 32), 2),
                                          ((40, 64, 128), 3)])
def test_fp16_levels_in_the_coarse_kernel(shape, levels, nu, monkeypatch):
    """Small FP16 levels run in the coarse kernel with every value rounded where
    the level-by-level sweeps store it: the same bits."""
    tag, r = _case(shape, sum(shape), 0.05)
    rd = torch.from_numpy(r).cuda()
    z = []
    for on in ("0", "1"):
        monkeypatch.setenv("FLUB_COARSE_FP16", on)
        mg = MGPCG(3, shape, levels, float, precision="mixed")
        mg.set_tags(torch.from_numpy(tag).cuda())
        mg.set_schedule(nu, 3, 0.5)
        mg.init(rd, 1.0)
        mg.solve(max_iters=3, eps=1e-12, abs_tol=1e-12, rel_tol=1e-12, smoother="phases")
        z.append((mg.apply_preconditioner(rd).cpu().numpy(), mg.x.cpu().numpy()))
    assert np.isfinite(z[0][1]).all()
    assert np.array_equal(z[0][0], z[1][0]) and np.array_equal(z[0][1], z[1][1])
