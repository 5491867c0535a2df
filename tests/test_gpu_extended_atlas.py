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


def grid_bruteforce(t, free, cap=64, max_cells=128):
    """Per cell: L-infinity distance from its coordinate range to the nearest texel that is not free, capped."""
    def shape(n):
        s = 0
        while -(-n // (1 << s)) > max_cells:
            s += 1
        return s, -(-n // (1 << s))
    (Ht, Wt), (sx, gx), (sy, gy) = t.shape, shape(t.shape[1]), shape(t.shape[0])
    ys, xs = np.nonzero(~free)
    out = np.full((gy, gx), cap, np.int64)
    for iy in range(gy):
        dy = np.maximum(0, np.maximum((iy << sy) - ys, ys - min((iy + 1) << sy, Ht - 1)))
        for ix in range(gx):
            dx = np.maximum(0, np.maximum((ix << sx) - xs, xs - min((ix + 1) << sx, Wt - 1)))
            if len(xs):
                out[iy, ix] = min(cap, int(np.maximum(dx, dy).min()))
    return out


@pytest.mark.parametrize("kind", ["f16", "bf16q"])
@pytest.mark.parametrize("Ht,Wt", [(2, 2), (40, 72), (130, 130), (300, 20), (33, 1030), (4100, 31), (257, 129)])
def test_solid_grid_matches_definition_gpu(kind, Ht, Wt):
    T = binary_templates(np.random.default_rng(0), 3, Ht, Wt)
    T[1, Ht // 2, Wt // 2] = np.nan
    atlas = R.Atlas(torch.from_numpy(T).cuda(), kind)
    raw = torch.as_strided(atlas.data, (int(R.lib.dbmp_atlas_extended_bytes(3, Ht, Wt, atlas.kind)),), (1,))
    raw = raw.cpu().numpy()
    want = [grid_bruteforce(t, t == 1) for t in T]
    clear = [grid_bruteforce(t, t <= 5e-7) for t in T]
    off = raw.size - sum(w.size for w in want)
    assert off % 256 == 0 and off >= atlas.data.numel()
    for p, w in enumerate(want):
        assert np.array_equal(raw[off + p * w.size: off + (p + 1) * w.size].reshape(w.shape), w), p
        at = atlas.data.numel() + (p - 3) * w.size      # the clearance grid ends the plain atlas
        assert np.array_equal(raw[at: at + w.size].reshape(w.shape), clear[p]), p


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


def test_f32_atlas_follows_its_templates_gpu():
    """An "f32" atlas renders the caller's tensor as it is, also after an in-place change."""
    rng = np.random.default_rng(3)
    T = torch.from_numpy(binary_templates(rng, 2, 48, 48)).cuda()
    d = [torch.tensor([[30.0, 30.0], [50.0, 40.0]]).cuda(), torch.tensor([25.0, 30.0]).cuda(), torch.zeros(2).cuda(),
         torch.zeros(2).cuda(), torch.zeros(2, 3).cuda(), torch.tensor([0, 1], dtype=torch.int32).cuda()]
    rz = R.Rasterizer(64, 80)
    atlas = R.Atlas(T, "f32")
    before = rz.forward(*d, atlas)[0]
    T.mul_(0.5)
    after = rz.forward(*d, atlas)[0]
    assert torch.equal(after, rz.forward(*d, R.Atlas(T, "f32"))[0])
    assert not torch.equal(before, after)


@pytest.mark.parametrize("H,W,ts", [(64, 48, 32), (130, 77, 16)])
def test_f32_quads_equal_the_reference_layout_gpu(H, W, ts, monkeypatch):
    """The walks of an extended "f32" atlas (quads) against those on the plain templates."""
    rng = np.random.default_rng(H)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    N = 80
    d = [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(4, 50, N)), cu(rng.uniform(0, 7, N)),
         cu(rng.normal(0, 2, N)), cu(rng.normal(0, 1, (N, 3))), torch.from_numpy(rng.integers(0, 3, N).astype(np.int32)).cuda()]
    T = cu(binary_templates(rng, 3, 70, 51) * rng.uniform(0.5, 1, (3, 70, 51)))
    gc, ga = cu(rng.normal(0, 1, (H, W, 3))), cu(rng.normal(0, 1, (H, W)))
    res = []
    for limit in (1 << 30, 0):
        monkeypatch.setattr(R, "MAX_F32_QUAD_BYTES", limit)
        atlas, rz = R.Atlas(T, "f32"), R.Rasterizer(H, W, ts)
        assert atlas.extended == (limit > 0)
        c, a, st = rz.forward(*d, atlas)
        res.append(([c, a, st.T_last, st.last_pos], rz.backward(st, gc, ga, *d[1:5], atlas)))
    for a, b in zip(*(r[0] for r in res)):
        assert torch.equal(a, b)
    for a, b in zip(*(r[1] for r in res)):
        assert (a - b).norm() <= 1e-6 * b.norm()
