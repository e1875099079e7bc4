"""The fused extrapolation of large grids (more than 2^22 cells) at the edges of
its tiles of 8 x 8 x 128 faces, with a last face layer whose flags the caller
set, against the oracle bit for bit; and the grid at the line, which takes the
other kernels."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import extrapolate
from flub_gb300.fields import Field, IntField, MACGrid, MACGridInt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cells", [1, 2])
@pytest.mark.parametrize("shape", [(128, 128, 256), (128, 128, 257), (129, 127, 260), (255, 129, 128), (136, 137, 255),
                                   (1, 4097, 1025), (2049, 17, 127)])
def test_large_extrapolation_bit_exact(shape, n_cells):
    rng = np.random.default_rng(sum(shape) + n_cells)
    phi = rng.standard_normal(shape).astype(np.float32)
    phi[:, : shape[1] // 2] += 3.0  # mostly air: parts without any known face
    faces, flags = [], []
    for d in range(3):
        fs = tuple(n + (a == d) for a, n in enumerate(shape))
        faces.append(rng.standard_normal(fs).astype(np.float32))
        flags.append(rng.integers(0, 3, size=fs).astype(np.int32))
    ref, rflags = [f.copy() for f in faces], [f.copy() for f in flags]
    O.extrapolate(*ref, *rflags, phi, n_cells)
    vel = MACGrid(*(Field(torch.from_numpy(a).cuda(), d=d + 1) for d, a in enumerate(faces)))
    tags = MACGridInt(*(IntField(torch.from_numpy(a).cuda(), d=d + 1) for d, a in enumerate(flags)))
    extrapolate(vel, tags, Field(torch.from_numpy(phi).cuda()), n_cells)
    for a, b in zip((vel.u.f, vel.v.f, vel.w.f, tags.u.f, tags.v.f, tags.w.f), ref + rflags):
        assert np.array_equal(a.cpu().numpy(), b)
