"""The halo-plane convolution (flub_gb300/csrc/unet_conv.cu) where its march
along x can go wrong: fewer planes than the ring, a last CTA with a rest of
planes, forced planes per CTA, one and two sources of every item count; and the
bias gradient's sums over lanes and warps.  Against float64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 16, 8, 16, 0, 16), (1, 17, 16, 8, 32, 16, 16), (2, 5, 32, 24, 16, 16, 32), (1, 3, 16, 16, 64, 16, 16),
         (1, 18, 16, 8, 32, 0, 64), (1, 2, 16, 40, 64, 32, 16), (1, 37, 32, 16, 16, 0, 32), (1, 7, 16, 8, 64, 0, 16)]


@pytest.mark.parametrize("planes", [0, 1, 3, 16])
@pytest.mark.parametrize("case", CASES)
def test_conv3d_planes_match_float64(case, planes, monkeypatch):
    from flub_gb300 import unet as U
    from oracle import unet_ref as R
    B, X, Y, Z, c0, c1, co = case
    monkeypatch.setenv("FLUB_CONV_XR", str(planes))
    g = torch.Generator().manual_seed(X + planes)
    rand = lambda s, k=1.0: (torch.randn(s, generator=g, dtype=torch.float64) * k).to(torch.bfloat16)
    x0, w0 = rand((B, X, Y, Z, c0)), rand((27, co, c0), 1.0 / math.sqrt(27 * c0))
    x1, w1 = (rand((B, X, Y, Z, c1)), rand((27, co, c1), 1.0 / math.sqrt(27 * c1))) if c1 else (None, None)
    bias = rand((co,), 0.1).float()
    dev = lambda t: None if t is None else t.cuda()
    dbl = lambda t: None if t is None else t.double()
    U.conv_error(reset=True)
    y = U.conv3d(dev(x0), dev(w0), dev(x1), dev(w1), dev(bias), relu=True).double().cpu()
    assert U.conv_error() == 0
    ref = R.conv3d(dbl(x0), dbl(w0), dbl(x1), dbl(w1), bias.double(), relu=True)
    # FP32 accumulation of at most 27 * 96 products, BF16 output: 2^-9 of the value, and of the cancelling terms 2^-16
    assert float(((y - ref).abs() - 2.0 ** -8 * ref.abs()).max()) <= 2.0 ** -10 * float(ref.abs().max())


@pytest.mark.parametrize("case", [(2, 64, 64, 64, 32, 16, 16), (1, 23, 64, 64, 16, 0, 16), (2, 32, 32, 32, 32, 0, 32)])
def test_conv3d_planes_round_as_the_tap_tiles(case, monkeypatch):
    """The same products in the same order per output: not a bit apart."""
    from flub_gb300 import unet as U
    B, X, Y, Z, c0, c1, co = case
    g = torch.Generator(device="cuda").manual_seed(X)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
    args = (rand(B, X, Y, Z, c0), rand(27, co, c0), rand(B, X, Y, Z, c1) if c1 else None,
            rand(27, co, c1) if c1 else None, torch.randn(co, generator=g, device="cuda"))
    y = U.conv3d(*args, relu=False)
    monkeypatch.setenv("FLUB_CONV_HALO", "0")
    assert torch.equal(y, U.conv3d(*args, relu=False))


@pytest.mark.parametrize("co", [16, 32, 64])
@pytest.mark.parametrize("grid", [(1, 1, 2, 64), (1, 3, 8, 16), (2, 33, 32, 32)])
def test_bias_gradient_matches_float64(grid, co):
    from flub_gb300 import unet as U
    g = torch.Generator().manual_seed(co)
    dy = torch.randn(grid + (co,), generator=g).to(torch.bfloat16)
    x = torch.zeros(grid + (16,), dtype=torch.bfloat16, device="cuda")
    dw, db = torch.zeros((27, co, 16), device="cuda"), torch.full((co,), 0.5, device="cuda")
    U.conv3d_wgrad(x, dy.cuda(), dw, db)
    want = 0.5 + dy.double().sum((0, 1, 2, 3))
    n = dy.numel() // co
    # FP32 partial sums: n rounding errors of 2^-24 of sums below sum |dy|
    assert float((db.double().cpu() - want).abs().max()) <= 2.0 ** -20 * n


@pytest.mark.parametrize("grid", [(1, 1, 16, 8), (1, 2, 16, 16), (2, 3, 32, 8), (1, 7, 16, 16), (1, 20, 48, 64)])
@pytest.mark.parametrize("ci,co", [(16, 16), (16, 32), (32, 16), (32, 32)])
def test_wgrad_planes_match_float64(grid, ci, co, monkeypatch):
    """The halo-plane weight gradient: fewer x planes than a segment, rests of
    one and two, more segments than buffers; added to what dW holds."""
    from flub_gb300 import unet as U
    from oracle import unet_ref as R
    monkeypatch.setenv("FLUB_CONV_XR", "1")  # forces the kernel on small grids
    g = torch.Generator().manual_seed(sum(grid) + ci + co)
    x = torch.randn(grid + (ci,), generator=g).to(torch.bfloat16)
    dy = torch.randn(grid + (co,), generator=g).to(torch.bfloat16)
    dw = torch.full((27, co, ci), 0.25, device="cuda")
    U.conv_error(reset=True)
    U.conv3d_wgrad(x.cuda(), dy.cuda(), dw)
    assert U.conv_error() == 0
    w = torch.zeros((27, co, ci), dtype=torch.float64, requires_grad=True)
    (R.conv3d(x.double(), w, bias=torch.zeros(co, dtype=torch.float64), relu=False) * dy.double()).sum().backward()
    want = 0.25 + w.grad
    # exact products of BF16 values, FP32 sums of n of them: n roundings of 2^-24 of sums below n
    n = grid[0] * grid[1] * grid[2] * grid[3]
    assert float((dw.double().cpu() - want).abs().max()) <= 2.0 ** -22 * n + 2.0 ** -20
