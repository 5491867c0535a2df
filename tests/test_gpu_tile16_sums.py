"""GPU test of the gradient sums at 16-pixel tiles: FP32 sums end at 8x4 pixels, and
those of the two halves of a warp's 8x8 footprint meet in FP64.  Image gradients of
+-2^24 on the upper halves, which cancel over the footprints, and of 1 on the lower
ones leave the lower ones' sum; a sum over a lane's two pixels in FP32 loses half of
it (2^23 + 0.5 is not an FP32 number).  Every other term here is exact."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["f32", "f32q", "f16q", "bf16"])
@pytest.mark.parametrize("masked", [True, False])
@pytest.mark.parametrize("H,W", [(16, 16), (16, 32)])
def test_halves_of_a_footprint_meet_in_fp64_gpu(kind, masked, H, W):
    T = torch.ones(1, 64, 64, device="cuda")
    d = [torch.tensor([[8.0, 8.0]]).cuda(), torch.tensor([100.0]).cuda(), torch.zeros(1).cuda(),
         torch.zeros(1).cuda(), torch.zeros(1, 3).cuda()]
    atlas, rz = R.Atlas(T, kind), R.Rasterizer(H, W, 16)
    c, a, st = rz.forward(*d, torch.zeros(1, dtype=torch.int32).cuda(), atlas)
    assert torch.equal(a, torch.full((H, W), 0.5, device="cuda"))      # mask 1, opacity 1/2, T = 1
    up = np.zeros((H, W), np.float32)
    for y in range(0, H, 8):
        for x in range(0, W, 8):
            up[y:y + 4, x:x + 8] = 2.0 ** 24 * (1 if (x // 8) % 2 == 0 else -1)
            up[y + 4:y + 8, x:x + 8] = 1.0
    if not masked:
        st.walk_masks = None
    gc = torch.from_numpy(np.repeat(up[..., None], 3, 2).copy()).cuda()
    g = rz.backward(st, gc, None, *d[1:], atlas)
    want = 0.25 * 0.5 * up.astype(np.float64).sum()                    # sigmoid'(0) a sum
    assert torch.equal(g[4].cpu().double(), torch.full((1, 3), want, dtype=torch.float64))
