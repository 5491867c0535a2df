"""GPU test of encode_channel_blocks on a stream of its own while the current one is
busy: its plan is summed and read behind its count pass, and before its write pass."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import psd as P

pytestmark = pytest.mark.gpu


def test_blocks_encoded_on_another_stream_gpu():
    rng = np.random.default_rng(0)
    hs = np.array([[40, 70], [3, 5], [65, 33]])
    sizes = torch.from_numpy(hs.astype(np.int32)).cuda()
    offs = torch.from_numpy(np.concatenate([[0], np.cumsum(4 * hs[:, 0] * hs[:, 1])[:-1]])).cuda()
    buf = torch.from_numpy(rng.integers(0, 3, int((4 * hs[:, 0] * hs[:, 1]).sum()), dtype=np.uint8)).cuda()
    select = lambda alpha: np.nonzero(alpha > 0)[0][::-1]
    want = P.encode_channel_blocks(buf, sizes, offs, hs, P.ORDER_LAYER, select)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    torch.cuda._sleep(200_000_000)                   # a tenth of a second on the current stream
    got = P.encode_channel_blocks(buf, sizes, offs, hs, P.ORDER_LAYER, select, stream=s)
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0])
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
