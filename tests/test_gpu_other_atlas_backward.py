"""GPU tests of a backward that is given other templates than its forward (sharp
forward, blurred backward, say): it tests its footprints on the templates it is
given, as the backward of a state without the forward's masks does."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu

H, W, N = 75, 130, 60


def disks(radius, soft):
    yy, xx = np.mgrid[0:40, 0:40]
    d = np.hypot(xx - 19.5, yy - 19.5)
    t = np.clip((radius - d) / soft + 0.5, 0, 1).astype(np.float32)
    return torch.from_numpy(np.stack([t, t.T ** 2])).cuda()


def setup(kind):
    rng = np.random.default_rng(4)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    p = [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(10, 60, N)), cu(rng.uniform(0, 7, N)),
         cu(rng.normal(-2, 1, N)), cu(rng.normal(0, 1, (N, 3))),
         torch.from_numpy(rng.integers(0, 2, N).astype(np.int32)).cuda()]
    g = torch.Generator(device="cuda").manual_seed(1)
    return p, torch.randn(H, W, 3, generator=g, device="cuda"), torch.randn(H, W, generator=g, device="cuda")


def check(got, want, other):
    for a, b in zip(got, want):
        assert (a - b).norm() <= 1e-6 * b.norm()
    assert (got[0] - other[0]).norm() > 1e-2 * other[0].norm()      # the templates matter


@pytest.mark.parametrize("kind", ["f32", "f32q", "f16q", "bf16"])
@pytest.mark.parametrize("ts", [16, 32])
def test_backward_on_another_atlas_gpu(kind, ts, monkeypatch):
    monkeypatch.setattr(R, "quads_pay", lambda pixels, N, texels: True, raising=False)
    p, gc, ga = setup(kind)
    sharp, soft, rz = R.Atlas(disks(9, 1.0), kind), R.Atlas(disks(12, 14.0), kind), R.Rasterizer(H, W, ts)
    st = rz.forward(*p, sharp)[2]
    own = rz.backward(st, gc, ga, *p[1:5], sharp)
    got = rz.backward(st, gc, ga, *p[1:5], soft)
    st.walk_masks = None
    check(got, rz.backward(st, gc, ga, *p[1:5], soft), own)


@pytest.mark.parametrize("kind", ["f32q", "f16q", "bf16"])
def test_backward_on_a_refilled_atlas_gpu(kind):
    p, gc, ga = setup(kind)
    atlas, rz = R.Atlas(disks(9, 1.0), kind), R.Rasterizer(H, W)
    st = rz.forward(*p, atlas)[2]
    own = rz.backward(st, gc, ga, *p[1:5], atlas)
    atlas.pack(disks(12, 14.0))
    got = rz.backward(st, gc, ga, *p[1:5], atlas)
    st.walk_masks = None
    check(got, rz.backward(st, gc, ga, *p[1:5], atlas), own)
