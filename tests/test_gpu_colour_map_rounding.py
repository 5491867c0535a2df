"""GPU test of the roundings of a blended colour, (1 - b) sigmoid(c) + b map: one of
the two products is rounded and the other enters by an FMA, the map's with 32-pixel
tiles and the logit's with 16-pixel ones.  Texel coordinates here are the pixels
themselves, sigmoid(c) and alpha are 1/2, and the map's values have all their bits,
so that float64 holds every exact sum and one cast to float32 rounds it."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts", [16, 32])
@pytest.mark.parametrize("kind", ["f32", "f32q", "f16q", "bf16"])
def test_blended_colours_round_as_written_gpu(kind, ts):
    S, blend = 64, np.float32(0.4)
    rng = np.random.default_rng(1)
    cmap = rng.uniform(0.5, 1.0, (1, S, S, 3)).astype(np.float32)
    d = [torch.tensor([[31.5, 31.5]]).cuda(), torch.tensor([31.5]).cuda(), torch.zeros(1).cuda(), torch.zeros(1).cuda(),
         torch.zeros(1, 3).cuda(), torch.zeros(1, dtype=torch.int32).cuda()]
    atlas = R.Atlas(torch.ones(1, S, S, device="cuda"), kind)
    color, alpha, _ = R.Rasterizer(S, S, ts).forward(*d, atlas, None, None, torch.from_numpy(cmap).cuda(), float(blend))
    inner = (slice(1, -1), slice(1, -1))
    assert torch.equal(alpha[inner], torch.full((S - 2, S - 2), 0.5, device="cuda"))
    k = np.float32(1) - blend
    product = np.float64(blend) * cmap[0].astype(np.float64)
    if ts == 16:
        product = product.astype(np.float32).astype(np.float64)
    want = (product + np.float64(k) * 0.5).astype(np.float32) * np.float32(0.5)
    assert np.array_equal(color.cpu().numpy()[inner], want[inner])
