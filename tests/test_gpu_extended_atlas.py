"""GPU tests of the extended atlas: its solid grid against the definition, and
the walks that use it against the same walks on the plain atlas.  Solid
footprints have mask 1 and mask gradient 0 exactly, so images are identical
bit for bit and gradient sums hold the same terms in the same order per warp
(the FP64 sums over warps are unordered: 1e-6 of the block's norm allows for
their rounding to float32)."""
import ctypes

import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R
from diffbmp_b200._lib import EXTENDED_ATLAS, call

pytestmark = pytest.mark.gpu


def binary_templates(rng, P, Ht, Wt):
    """Rectangles and disks of exact ones with a soft rim, one almost-one texel, one NaN texel."""
    yy, xx = np.mgrid[0:Ht, 0:Wt].astype(np.float64)
    T = np.zeros((P, Ht, Wt), np.float32)
    for p in range(P):
        if p % 2:
            d = np.maximum(np.abs(xx - (Wt - 1) / 2) - 0.38 * Wt, np.abs(yy - (Ht - 1) / 2) - 0.35 * Ht)
        else:
            d = np.hypot((xx - (Wt - 1) / 2) / Wt, (yy - (Ht - 1) / 2) / Ht) * min(Ht, Wt) - 0.42 * min(Ht, Wt)
        T[p] = np.clip(0.5 - d, 0, 1)
    T[0, Ht // 2, Wt // 3] = np.nextafter(np.float32(1), np.float32(0))
    return T


def solid_bruteforce(t, cap=64, max_cells=128):
    """Per cell of the clearance grid: L-infinity distance from its coordinate range to the nearest texel != 1."""
    def shape(n):
        s = 0
        while -(-n // (1 << s)) > max_cells:
            s += 1
        return s, -(-n // (1 << s))
    (Ht, Wt), (sx, gx), (sy, gy) = t.shape, shape(t.shape[1]), shape(t.shape[0])
    ys, xs = np.nonzero(~(t == 1))
    out = np.full((gy, gx), cap, np.int64)
    for iy in range(gy):
        dy = np.maximum(0, np.maximum((iy << sy) - ys, ys - min((iy + 1) << sy, Ht - 1)))
        for ix in range(gx):
            dx = np.maximum(0, np.maximum((ix << sx) - xs, xs - min((ix + 1) << sx, Wt - 1)))
            if len(xs):
                out[iy, ix] = min(cap, int(np.maximum(dx, dy).min()))
    return out


@pytest.mark.parametrize("kind", ["f16", "bf16q"])
@pytest.mark.parametrize("Ht,Wt", [(2, 2), (40, 72), (130, 130), (300, 20)])
def test_solid_grid_matches_definition_gpu(kind, Ht, Wt):
    T = binary_templates(np.random.default_rng(0), 3, Ht, Wt)
    T[1, Ht // 2, Wt // 2] = np.nan
    atlas = R.Atlas(torch.from_numpy(T).cuda(), kind)
    raw = torch.as_strided(atlas.data, (int(R.lib.dbmp_atlas_extended_bytes(3, Ht, Wt, atlas.kind)),), (1,))
    raw = raw.cpu().numpy()
    want = [solid_bruteforce(t) for t in T]
    off = raw.size - sum(w.size for w in want)
    assert off % 256 == 0 and off >= atlas.data.numel()
    for p, w in enumerate(want):
        assert np.array_equal(raw[off + p * w.size: off + (p + 1) * w.size].reshape(w.shape), w), p


def walk(atlas, extended, d, N, H, W, ts, gc, ga):
    """(image, alpha, T_last, last_pos, five gradients) of one binning, with or without the extension."""
    rz = R.Rasterizer(H, W, ts, 0.9)
    prim, lists = rz.bin(*d, atlas)
    cv = rz.canvas(N, atlas)
    assert cv.reserved == EXTENDED_ATLAS
    if not extended:
        cv.reserved = 0
    out = [torch.empty(s, device="cuda", dtype=t) for s, t in
           (((H, W, 3), torch.float32), ((H, W), torch.float32), ((H, W), torch.float32), ((H, W), torch.int32))]
    pr, st = R._ptr, R._stream()
    call("dbmp_forward", ctypes.byref(cv), pr(prim), pr(atlas.data), pr(lists.offsets), pr(lists.indices),
         *[pr(o) for o in out], st)
    acc = torch.empty((N, 8), dtype=torch.float64, device="cuda")
    g = [torch.empty(s, device="cuda") for s in ((N, 2), (N,), (N,), (N,), (N, 3))]
    call("dbmp_backward", ctypes.byref(cv), pr(prim), pr(atlas.data), pr(lists.offsets), pr(lists.indices),
         pr(out[2]), pr(out[3]), pr(gc), pr(ga), pr(d[1]), pr(d[2]), pr(d[3]), pr(d[4]), pr(acc),
         *[pr(x) for x in g], st)
    return out, g


@pytest.mark.parametrize("kind", ["f16q", "f16", "bf16", "f32q"])
@pytest.mark.parametrize("H,W,ts,N,Ht,Wt", [(33, 70, 32, 3, 2, 2), (160, 97, 16, 60, 90, 41), (200, 333, 32, 300, 64, 64)])
@pytest.mark.parametrize("bad", [None, "nan", "inf"])
def test_walks_equal_the_plain_atlas_gpu(kind, H, W, ts, N, Ht, Wt, bad):
    rng = np.random.default_rng(H + N)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    d = [cu(rng.uniform(-10, [W + 10, H + 10], (N, 2))), cu(rng.uniform(4, 90, N)), cu(rng.uniform(0, 7, N)),
         cu(rng.normal(0, 2, N)), cu(rng.normal(0, 1, (N, 3))), torch.from_numpy(rng.integers(0, 3, N).astype(np.int32)).cuda()]
    atlas = R.Atlas(cu(binary_templates(rng, 3, Ht, Wt)), kind)
    gc, ga = cu(rng.normal(0, 1, (H, W, 3))), cu(rng.normal(0, 1, (H, W)))
    if bad:
        gc[H // 2, W // 2, 1] = float(bad)
        ga[H // 3, W // 3] = float(bad)
    (o1, g1), (o0, g0) = (walk(atlas, e, d, N, H, W, ts, gc, ga) for e in (True, False))
    for a, b in zip(o1, o0):
        assert torch.equal(a, b)
    for a, b in zip(g1, g0):
        fin = torch.isfinite(b)
        assert torch.equal(fin, torch.isfinite(a))
        assert (a - b)[fin].norm() <= 1e-6 * b[fin].norm()
