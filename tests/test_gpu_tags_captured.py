"""set_tags and the V-cycle behind it in a captured graph, replayed after calls
outside it, and calls outside it behind set_tags while another graph is captured:
always the lists and words of the tags in front."""
import numpy as np
import pytest
import torch

from flub_gb300 import MGPCG

pytestmark = pytest.mark.gpu


def _tags(shape, seed):
    rng = np.random.default_rng(seed)
    tag = np.zeros(shape, np.int32)
    if seed % 2:
        tag[: shape[0] // 4, : shape[1] // 3] = 1
    else:
        tag[:] = 1
    tag[rng.random(shape) < 0.03] = 2
    return torch.from_numpy(tag).cuda()


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("shape,levels", [((32, 32, 32), 3), ((64, 64, 64), 4), ((128, 128, 128), 4)])
def test_tags_and_vcycle_captured(shape, levels, precision):
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(shape).astype(np.float32)).cuda()
    tags = [_tags(shape, seed) for seed in range(4)]
    want = []
    for tag in tags:
        mg = MGPCG(3, shape, levels, float, precision=precision)
        mg.set_schedule(2, 3, 0.5)
        mg.set_tags(tag)
        torch.cuda.synchronize()
        want.append(mg.apply_preconditioner(r))
    torch.cuda.synchronize()
    mg = MGPCG(3, shape, levels, float, precision=precision)
    mg.set_schedule(2, 3, 0.5)
    mg.set_tags(tags[0])
    z = [torch.empty(shape, device="cuda") for _ in range(12)]
    mg.apply_preconditioner(r, z[0])  # outside a capture first: static launch shapes
    cur, zg = tags[1].clone(), torch.empty(shape, device="cuda")
    torch.cuda.synchronize()
    both, one = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(both):
        mg.set_tags(cur)
        mg.apply_preconditioner(r, zg)
    torch.cuda.synchronize()
    order = [1, 2, 3, 1, 0, 3]
    for n, q in enumerate(order):
        cur.copy_(tags[q])
        both.replay()
        z[n].copy_(zg)
        mg.apply_preconditioner(r, z[6 + n])  # the tags of the replay, outside it
    torch.cuda.synchronize()
    for n, q in enumerate(order):
        assert torch.equal(z[n], want[q]), n
        assert torch.equal(z[6 + n], want[q]), n
    mg.set_tags(tags[2])
    with torch.cuda.graph(one):
        mg.apply_preconditioner(r, zg)
    mg.set_tags(tags[3])
    mg.apply_preconditioner(r, z[0])
    one.replay()
    torch.cuda.synchronize()
    assert torch.equal(z[0], want[3]) and torch.equal(zg, want[3])
