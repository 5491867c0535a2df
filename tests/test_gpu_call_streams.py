"""GPU tests of the calls' `stream` argument while the current stream is busy: copies
that a call makes, its scratch and its read of the list lengths belong to the given
stream, on which the caller has the inputs ready."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu

H, W, N = 90, 120, 500


def params(seed):
    rng = np.random.default_rng(seed)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(2, 40, N)), cu(rng.uniform(0, 7, N)),
            cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3))), torch.zeros(N, dtype=torch.int32, device="cuda")]


def ups(*lead):
    g = torch.Generator(device="cuda").manual_seed(0)
    return torch.randn(*lead, H, W, 3, generator=g, device="cuda"), torch.randn(*lead, H, W, generator=g, device="cuda")


def gradients_equal(a, b):
    for x, y in zip(a, b):
        assert (x - y).norm() <= 1e-6 * y.norm()


@pytest.mark.parametrize("kind", ["f32", "f16q"])
def test_one_candidate_gpu(kind, monkeypatch):
    monkeypatch.setattr(R, "quads_pay", lambda pixels, N, texels: True)
    atlas, p, (gc, ga) = R.Atlas(torch.rand(2, 20, 24, device="cuda"), kind), params(0), ups()
    c0, a0, st = R.Rasterizer(H, W).forward(*p, atlas)
    g0 = R.Rasterizer(H, W).backward(st, gc, ga, *p[1:5], atlas)
    lists0 = R.Rasterizer(H, W).bin(*p, atlas)[1]
    torch.cuda.synchronize()
    s, rz = torch.cuda.Stream(), R.Rasterizer(H, W)
    rz._hint = 1                                     # the first attempt does not hold the lists
    half = gc.double()                               # converted by the call
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                   # a tenth of a second on the current stream
    c, a, st = rz.forward(*p, atlas, stream=s)
    g = rz.backward(st, half, ga, *p[1:5], atlas, stream=s)
    rz._hint = 1
    lists = rz.bin(*p, atlas, stream=s)[1]
    torch.cuda.synchronize()
    assert torch.equal(c, c0) and torch.equal(a, a0) and lists.length == lists0.length
    assert torch.equal(lists.mapping_tensor(), lists0.mapping_tensor())
    gradients_equal(g, g0)


def test_strided_candidates_gpu():
    B = 3
    atlas, (gc, ga) = R.Atlas(torch.rand(2, 20, 24, device="cuda"), "f16q"), ups(B)
    one = [torch.stack([params(k)[i] for k in range(B)]) for i in range(6)]
    c0, a0, st = R.Rasterizer(H, W).forward_batch(*one, atlas)
    g0 = R.Rasterizer(H, W).backward_batch(st, gc, ga, *one[1:5], atlas)
    strided = [torch.stack([q, q], 1)[:, 1] for q in one]
    assert not strided[0].is_contiguous()
    torch.cuda.synchronize()
    s, rz = torch.cuda.Stream(), R.Rasterizer(H, W)
    torch.cuda._sleep(200_000_000)
    c, a, st = rz.forward_batch(*strided, atlas, stream=s)
    g = rz.backward_batch(st, gc, ga, *one[1:5], atlas, stream=s)
    torch.cuda.synchronize()
    assert torch.equal(c, c0) and torch.equal(a, a0)
    gradients_equal(g, g0)
