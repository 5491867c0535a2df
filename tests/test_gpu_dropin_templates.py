"""GPU tests of the drop-in objects when a program hands over other templates from
call to call: each call renders those that it was given."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import cuda_tile_rasterizer as ctr

pytestmark = pytest.mark.gpu

H, W, N, S = 60, 80, 40, 32


def scene(seed):
    rng = np.random.default_rng(seed)
    cu = lambda a, t=np.float32: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()
    return [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(4, 30, N)), cu(rng.uniform(0, 7, N)),
            cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3)))], cu(rng.integers(0, 2, N), np.int32)


def templates(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(2, S, S, generator=g, device="cuda")


def make(fp16):
    return ctr.TileRasterizer(H, W, 16, num_primitives=N, use_fp16=fp16)


def render(tr, T, batch):
    p, sel = scene(0)
    none, lr = torch.empty(0, device="cuda"), torch.ones(7, device="cuda")
    if batch:
        return tr.forward_batch(*[q.unsqueeze(0) for q in p], none, T, sel, 0.0, lr)[0]
    return tr(*p, none, T, sel, 0.0, lr)[0]


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("fp16", [True, False])
@pytest.mark.parametrize("given", ["float32", "float16", "temporary"])
def test_other_templates_in_the_next_call_gpu(fp16, given, batch):
    """Templates converted inside the call, or made for it, share their address with
    those of the call before."""
    def pick(seed):
        T = templates(seed)
        return T if given == "float32" else T.half() if given == "float16" else (T * 0.5).half().float() * 2
    with torch.no_grad():
        want = [render(make(fp16), pick(k), batch) for k in range(3)]
        tr = make(fp16)
        for k in (0, 1, 2, 0):
            assert torch.equal(render(tr, pick(k), batch), want[k])


@pytest.mark.parametrize("fp16", [True, False])
def test_transposed_templates_in_the_next_call_gpu(fp16):
    with torch.no_grad():
        T = templates(5).half() if fp16 else templates(5)
        want = render(make(fp16), T.transpose(1, 2).contiguous(), False)
        tr = make(fp16)
        render(tr, T, False)
        assert torch.equal(render(tr, T.transpose(1, 2), False), want)
