"""The rule that has an "f32" atlas packed for a call, at measured points: there, the
walks gained clearly more than the packing took, or clearly less (us, one forward
and backward, B200)."""
import pytest

from diffbmp_b200.rasterizer import quads_pay

MEASURED = [  # H, W, N, P, side, gain, packing
    (64, 64, 60, 1, 64, -4.2, 9.7), (256, 256, 6000, 1, 64, -3.2, 9.7), (384, 384, 600, 1, 64, 0.6, 9.7),
    (768, 768, 600, 1, 64, 18.1, 9.7), (1024, 1024, 6000, 1, 64, 42.2, 9.7),
    (300, 300, 600, 8, 128, 17.8, 23.1), (384, 384, 300, 8, 128, 4.1, 23.1), (512, 500, 600, 8, 128, 40.5, 23.1),
    (768, 768, 300, 8, 128, 36.2, 23.1), (1024, 1024, 60, 8, 128, -0.5, 23.1), (1024, 1024, 100, 8, 128, 7.5, 23.1),
    (384, 384, 600, 16, 256, 29.4, 61.1), (500, 512, 300, 16, 256, 29.3, 61.1), (768, 768, 600, 16, 256, 104.8, 61.1),
    (1024, 1024, 300, 16, 256, 93.3, 61.1), (1024, 1024, 100, 16, 256, 14.3, 61.1), (1500, 1500, 60, 16, 256, 7.3, 61.1),
    (500, 512, 600, 16, 512, 51.8, 97.8), (1500, 1500, 600, 16, 512, 401.5, 97.8)]


@pytest.mark.parametrize("H,W,N,P,side,gain,packing", MEASURED)
def test_an_atlas_is_packed_where_one_call_gains(H, W, N, P, side, gain, packing):
    assert quads_pay(H * W, N, P * side * side) == (gain > packing)
