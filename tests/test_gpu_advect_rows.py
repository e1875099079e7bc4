"""Advection on either side of the row length from which samples away from the
array's ends take a path without clamps, bit for bit against the oracle: feet
inside, across both ends, far outside and NaN."""
import numpy as np
import pytest
import torch

import oracle as O
from flub_gb300 import advect_mc, advect_phi, advect_simple_3d, advect_uv_mc, launch
from flub_gb300.fields import Field, MACGrid

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def same(t, ref):
    got = t.cpu().numpy()
    return np.array_equal(got, ref, equal_nan=True)


def _mac(arrs):
    return MACGrid(*(Field(dev(a), stagger=O.STAGGER[d + 1], d=d + 1) for d, a in enumerate(arrs)))


@pytest.mark.parametrize("minmax_h", [None, 1.0])
@pytest.mark.parametrize("n,scale", [((9, 6, 159), 15.0), ((9, 6, 160), 15.0), ((2, 3, 200), 4.0), ((1, 1, 300), 50.0),
                                     ((4, 12, 257), 8.0)])
def test_advection_by_row_length_bit_exact(n, scale, minmax_h):
    rng = np.random.default_rng(sum(n))
    nx, ny, nz = n
    vel = [(scale * rng.standard_normal(s)).astype(np.float32)
           for s in ((nx + 1, ny, nz), (nx, ny + 1, nz), (nx, ny, nz + 1))]
    vel[0][0, 0, nz // 2] = 1e30
    vel[1][0, 0, nz // 3] = -1e7
    vel[2][0, 0, nz // 4] = np.nan
    q = rng.standard_normal(n).astype(np.float32)
    h = 1.0 / nx
    mac = _mac(vel)
    out = Field(torch.zeros(n, device="cuda"))
    advect_mc(mac, Field(dev(q)), out, minmax_h=minmax_h)
    assert same(out.f, O.advect_mc(*vel, q, O.STAGGER[0], 0.01, h, minmax_h=minmax_h))
    new = _mac([np.zeros_like(a) for a in vel])
    advect_uv_mc(mac, new, minmax_h=minmax_h)
    for a, r in zip((new.u.f, new.v.f, new.w.f), O.advect_velocity_mc(*vel, 0.01, h, minmax_h)):
        assert same(a, r)
    launch(advect_phi, dim=n, inputs=[mac, Field(dev(q)), out])
    assert same(out.f, O.advect_phi(*vel, q, 0.01, h))
    launch(advect_simple_3d, dim=n, inputs=[*(dev(a) for a in vel), dev(q), out.f, 0.02, 0.05])
    assert same(out.f, O.advect_simple(*vel, q, 0.02, 0.05))
