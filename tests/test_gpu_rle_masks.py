"""GPU test of the PackBits passes at the edges of their work split: rows in
groups of 32 looked at four at a time, chunks of 32 columns with four pixels per
lane, the 32-way search for a group's layer.  Blocks byte-identical to the
oracle's encoder."""
import numpy as np
import pytest
import torch

from oracle import psd_file as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,heights,copies", [
    ((1, 2, 3, 4, 5), (1, 3, 4, 5), 60),                 # 1200 small images: three steps of the search
    ((31, 32, 33, 36, 63, 64, 65), (1, 31, 32, 33, 36), 1),
    ((127, 128, 130, 161, 290), (2, 35, 64, 65), 1),
])
def test_blocks_match_oracle_at_split_edges_gpu(widths, heights, copies):
    from diffbmp_b200.psd import encode_channel_blocks
    rng = np.random.default_rng(sum(widths))
    imgs = []
    for w in widths:
        for h in heights:
            for _ in range(copies):
                im = np.zeros((h, w, 4), np.uint8)
                # runs that start in different columns per channel, single and double pixels, rows alike
                for ch in range(4):
                    run = rng.integers(1, 6 if ch % 2 else 90)
                    im[:, :, ch] = np.repeat(rng.integers(0, 3, (h, w // run + 1)), run, axis=1)[:, :w]
                im[h // 2:] = im[h // 2]
                imgs.append(im)
    order = 0x02010003
    sizes = np.array([[im.shape[1], im.shape[0]] for im in imgs], np.int32)
    offs = np.concatenate([[0], np.cumsum([im.size for im in imgs])[:-1]]).astype(np.int64)
    buf = np.concatenate([im.reshape(-1) for im in imgs])
    flags = []
    blob, blocks, _ = encode_channel_blocks(torch.from_numpy(buf).cuda(), torch.from_numpy(sizes).cuda(),
                                            torch.from_numpy(offs).cuda(), sizes, order,
                                            lambda a: flags.append(a) or np.arange(len(a)))
    exp = [O.channel_block(im[:, :, (order >> (8 * s)) & 3]) for im in imgs for s in range(4)]
    assert blocks.reshape(-1).tolist() == [len(b) for b in exp]
    assert blob.cpu().numpy().tobytes() == b"".join(exp)
    assert [bool(f) for f in flags[0]] == [bool(im[:, :, 3].any()) for im in imgs]
