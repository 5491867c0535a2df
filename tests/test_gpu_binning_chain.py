"""GPU tests of the binning launches at the edges of their work split (tile
groups of 32, chunks of 512 primitives, writing and counting slices, canvases
whose difference arrays leave shared memory): lists bit-exact with the oracle's,
alone and as a batch of candidates, with and without capacity for them."""
import ctypes

import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [  # H, W, tile, N, largest radius
    (1, 1, 16, 1, 5.0),
    (40, 31 * 32 + 1, 32, 511, 300.0),
    (70, 33 * 32, 32, 513, 100.0),
    (2081, 64, 32, 1300, 200.0),
    (64, 65, 32, 40000, 40.0),
    (3713, 3712, 16, 700, 60.0),
    # lists from primitive masks: few primitives per word; more than a buffer of them
    # in a cell; more than a chunk of words in the only slice; just below the rule
    (33 * 32 + 1, 65 * 32, 32, 8200, 30.0),
    (1100, 1050, 32, 26000, 900.0),
    (16 * 790, 16 * 100, 16, 17000, 20.0),
    (1024, 1024, 32, 25088, 40.0),
    (1024, 1024, 32, 25089, 40.0),
]


def params(rng, H, W, N, rmax):
    return (rng.uniform(-20, [W + 20, H + 20], (N, 2)).astype(np.float32), rng.uniform(1, rmax, N).astype(np.float32),
            rng.uniform(0, 7, N).astype(np.float32), rng.normal(0, 1, N).astype(np.float32),
            rng.normal(0, 1, (N, 3)).astype(np.float32))


@pytest.mark.parametrize("H,W,ts,N,rmax", CASES)
def test_lists_match_oracle_alone_and_in_a_batch_gpu(H, W, ts, N, rmax):
    rng = np.random.default_rng(N)
    T = np.zeros((2, 20, 24), np.float32)
    T[0, 3:17, 5:20], T[1, 1:5, 2:23] = 1, 0.5
    sel = rng.integers(0, 2, N).astype(np.int32)
    cands = [params(rng, H, W, N, rmax) for _ in range(3)]
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    atlas = R.Atlas(cu(T), "f16q")
    want = [O.bin_tiles(H, W, ts, *c[:3], sel, O.template_bboxes(T), 20, 24) for c in cands]
    rz = R.Rasterizer(H, W, ts)
    d = [cu(np.stack([c[k] for c in cands])) for k in range(5)]
    prim, offsets, indices = rz.bin_batch(*d, cu(sel), atlas)      # grows from capacity 0
    for b, (wo, wi) in enumerate(want):
        one, lists = rz.bin(*[x[b] for x in d], cu(sel), atlas)
        assert lists.length == len(wi)
        for o, i in ((lists.offsets, lists.indices), (offsets[b], indices[b])):
            assert np.array_equal(o.cpu().numpy(), wo)
            assert np.array_equal(i[:len(wi)].cpu().numpy(), wi)
        assert torch.equal(prim[b * N:(b + 1) * N], one)


def test_overflow_leaves_lists_and_reports_length_gpu():
    rng = np.random.default_rng(1)
    H, W, N = 200, 300, 700
    p = [torch.from_numpy(a).cuda() for a in params(rng, H, W, N, 50.0)] + [torch.zeros(N, dtype=torch.int32).cuda()]
    atlas = R.Atlas(torch.ones(1, 8, 8).cuda(), "f16q")
    rz = R.Rasterizer(H, W)
    L = rz.bin(*p, atlas)[1].length
    cv = rz.canvas(N, atlas)
    rz._ensure(cv, L)
    ws, wsb = rz._ws_ptr()
    prim = torch.empty((N, 16), device="cuda")
    offsets = torch.full((rz.T + 1,), -7, dtype=torch.int32, device="cuda")
    indices = torch.full((L,), -7, dtype=torch.int32, device="cuda")
    flags = torch.zeros(2, dtype=torch.int32, device="cuda")
    pr = R._ptr
    R.call("dbmp_bin", ctypes.byref(cv), *[pr(x) for x in p], pr(atlas.bbox), pr(prim), pr(offsets), pr(indices),
           ctypes.c_longlong(L - 1), pr(flags), ctypes.c_void_p(flags.data_ptr() + 4), ws, ctypes.c_size_t(wsb), R._stream())
    assert flags.tolist() == [L, 1]
    assert int(offsets.max()) == -7 and int(indices.max()) == -7


def test_batch_of_expanded_candidates_gpu():
    """Candidates that share a parameter through a stride of 0."""
    rng = np.random.default_rng(2)
    H, W, N = 100, 90, 40
    p = [torch.from_numpy(a).cuda() for a in params(rng, H, W, N, 30.0)]
    sel = torch.zeros(N, dtype=torch.int32).cuda()
    atlas = R.Atlas(torch.ones(1, 8, 8).cuda(), "f16q")
    rz = R.Rasterizer(H, W)
    c, a, _ = rz.forward_batch(*[x.unsqueeze(0).expand(2, *x.shape) for x in p], sel.unsqueeze(0).expand(2, N), atlas)
    c1, a1, _ = rz.forward(*p, sel, atlas)
    for b in range(2):
        assert torch.equal(c[b], c1) and torch.equal(a[b], a1)
