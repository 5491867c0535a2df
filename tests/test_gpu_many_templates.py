"""GPU test of atlases with more templates than a grid's second dimension holds."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["f32", "f32q", "f16"])
@pytest.mark.parametrize("P,th,tw", [(65535, 3, 5), (65536, 4, 4), (70001, 6, 5)])
def test_templates_beyond_65535_gpu(kind, P, th, tw, monkeypatch):
    """The used templates alone, in an atlas of their own, give the same image and gradients."""
    monkeypatch.setattr(R, "quads_pay", lambda pixels, N, texels: True, raising=False)
    rng = np.random.default_rng(P)
    H, W, N = 70, 90, 60
    T = torch.rand(P, th, tw, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).round(decimals=1)
    ids = np.concatenate([[0, 65534, P - 1], rng.integers(0, P, N - 3)])
    cu = lambda a, t=np.float32: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()
    d = [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(4, 40, N)), cu(rng.uniform(0, 7, N)),
         cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3)))]
    up = torch.randn(H, W, 3, device="cuda"), torch.randn(H, W, device="cuda")
    res = []
    for templates, sel in ((T, ids), (T[torch.from_numpy(ids).cuda()], np.arange(N))):
        atlas, rz = R.Atlas(templates, kind), R.Rasterizer(H, W)
        c, a, st = rz.forward(*d, cu(sel, np.int32), atlas)
        res.append(([c, a], rz.backward(st, *up, *d[1:], atlas)))
    for x, y in zip(*(r[0] for r in res)):
        assert torch.equal(x, y)
    for x, y in zip(*(r[1] for r in res)):
        assert (x - y).norm() <= 1e-6 * y.norm()
