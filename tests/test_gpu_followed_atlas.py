"""GPU tests of "f32" atlases whose templates are written to after the atlas was
made, by routes that PyTorch's version counter sees and by those that it does not:
every render and backward takes the texels that are in memory when its turn on
its stream comes, as a walk of the plain templates does.  Both walks composite the
same values in the same order: images are equal bit for bit, gradients up to the
unordered FP64 sums over warps (1e-6 of the block's norm)."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import cuda_tile_rasterizer as ctr
from diffbmp_b200 import fitting as F
from diffbmp_b200 import rasterizer as R
from diffbmp_b200.fitting import FitConfig, ImageFitter

pytestmark = pytest.mark.gpu

H, W, N = 75, 130, 90


@pytest.fixture(autouse=True)
def packed_at_any_size(monkeypatch):
    monkeypatch.setattr(R, "quads_pay", lambda pixels, N, texels: True)
    monkeypatch.setattr(F, "fit_quads_pay", lambda pixels, N, texels: True)


def cu(a, dtype=np.float32):
    return torch.from_numpy(np.ascontiguousarray(a, dtype)).cuda()


def templates(seed, P=3, th=33, tw=28):
    """Soft blobs with solid cores and empty corners, so that both grids skip something."""
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:th, 0:tw]
    r = np.hypot((xx - tw / 2) / tw, (yy - th / 2) / th)
    return cu(np.stack([np.clip(rng.uniform(0.1, 0.4) * 8 - 8 * r + rng.uniform(0, 1), 0, 1) for _ in range(P)]))


def params(seed, P=3, n=N, lead=()):
    rng = np.random.default_rng(seed)
    s = (*lead, n)
    return [cu(rng.uniform(0, [W, H], (*s, 2))), cu(rng.uniform(4, 50, s)), cu(rng.uniform(0, 7, s)),
            cu(rng.normal(-1, 1, s)), cu(rng.normal(0, 1, (*s, 3))), cu(rng.integers(0, P, n), np.int32)]


def ups(lead=()):
    g = torch.Generator(device="cuda").manual_seed(1)
    return (torch.randn(*lead, H, W, 3, generator=g, device="cuda"), torch.randn(*lead, H, W, generator=g, device="cuda"))


def plain(T, like, monkeypatch):
    """An atlas of a copy of T whose walks read it in the reference layout, binned as
    `like` (an atlas's content boxes are those of its construction)."""
    with monkeypatch.context() as m:
        m.setattr(R, "MAX_F32_QUAD_BYTES", 0)
        a = R.Atlas(T.clone(), "f32")
    if like is not None:
        a.bbox = like.bbox
    return a


def same(got, want):
    for a, b in zip(got[0], want[0]):
        assert torch.equal(a, b)
    for a, b in zip(got[1], want[1]):
        assert (a - b).norm() <= 1e-6 * b.norm()


class Graph:
    """A captured kernel that writes to a tensor."""

    def __init__(self, T, src):
        self.g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.g):
            T.copy_(src)

    def __call__(self):
        self.g.replay()


def write(how, T, src, atlas):
    if how == "counted":
        T.copy_(src)
    elif how == "data":
        T.data.copy_(src)
    elif how == "one texel":
        src.copy_(T)
        src[-1, 17, 13] = 0.25
        T.data[-1, 17, 13] = 0.25
    elif how == "dlpack":
        torch.from_dlpack(T).copy_(src)
    elif how == "atlas":
        atlas.data.copy_(src)
    elif how == "graph":
        Graph(T, src)()


@pytest.mark.parametrize("how", ["counted", "data", "one texel", "dlpack", "atlas", "graph"])
@pytest.mark.parametrize("ts", [16, 32])
def test_writes_are_rendered_gpu(how, ts, monkeypatch):
    T, src, p, (gc, ga) = templates(0), templates(1), params(2), ups()
    atlas, rz = R.Atlas(T, "f32"), R.Rasterizer(H, W, ts)
    before = rz.forward(*p, atlas)[0]
    write(how, T, src, atlas)
    color, alpha, st = rz.forward(*p, atlas)
    ref = plain(src, atlas, monkeypatch)
    c0, a0, s0 = R.Rasterizer(H, W, ts).forward(*p, ref)
    assert not torch.equal(before, c0)
    same(([color, alpha, st.T_last, st.last_pos], rz.backward(st, gc, ga, *p[1:5], atlas)),
         ([c0, a0, s0.T_last, s0.last_pos], R.Rasterizer(H, W, ts).backward(s0, gc, ga, *p[1:5], ref)))
    # and back again, on the same copy or another
    T.data.copy_(templates(0))
    assert torch.equal(rz.forward(*p, atlas)[0], before)


@pytest.mark.parametrize("ts", [16, 32])
@pytest.mark.parametrize("blend", [0.0, 0.5])
@pytest.mark.parametrize("route", ["one", "batch", "mapping"])
def test_every_walk_takes_the_changed_templates_gpu(ts, blend, route, monkeypatch):
    """A write between forward and backward, too: the backward samples what is there then."""
    T, src = templates(3), templates(4)
    lead = (2,) if route == "batch" else ()
    p, (gc, ga) = params(5, lead=lead), ups(lead)
    maps = cu(np.random.default_rng(6).uniform(0, 1, (N, 33, 28, 3))) if blend else None
    res = []
    first = R.Atlas(T, "f32")
    for made in (lambda: first, lambda: plain(src, first, monkeypatch)):
        T.copy_(templates(3))
        atlas, rz = made(), R.Rasterizer(H, W, ts)
        more = dict(colors_orig=maps, c_blend=blend)
        if route == "mapping":
            more["mapping"] = rz.bin(*p, first)[1].mapping_tensor()
        fwd, bwd = (rz.forward_batch, rz.backward_batch) if route == "batch" else (rz.forward, rz.backward)
        c, a, st = fwd(*p, atlas, **more)
        if atlas.data.data_ptr() == T.data_ptr():
            c1, a1, _ = fwd(*p, atlas, **more)          # on the packed copy
            assert torch.equal(c1, c) and torch.equal(a1, a)
        T.data.copy_(src)
        c, a, st = fwd(*p, atlas, **more)
        late = bwd(st, gc, ga, *p[1:5], atlas)
        if atlas.data.data_ptr() == T.data_ptr():
            T.data.copy_(templates(3))                  # as packed: the walk goes back to the copy
        else:
            atlas.data.copy_(templates(3))
        res.append(([c, a, st.T_last, st.last_pos], late, bwd(st, gc, ga, *p[1:5], atlas)))
    same(res[0][:2], res[1][:2])
    same(([], res[0][2]), ([], res[1][2]))


@pytest.mark.parametrize("offset,th,tw", [(0, 33, 28), (1, 32, 32), (4, 32, 32), (0, 3, 5)])
def test_alignment_of_the_comparison_gpu(offset, th, tw, monkeypatch):
    """The last texel of tensors that 16-byte loads do and do not cover."""
    n = 3 * th * tw
    T = torch.zeros(n + 8, device="cuda")[offset:offset + n].view(3, th, tw)
    T.copy_(templates(0, 3, th, tw))
    p = params(7)
    atlas, rz = R.Atlas(T, "f32"), R.Rasterizer(H, W)
    rz.forward(*p, atlas)
    for k in (0, n // 2, n - 1):
        T.data.view(-1)[k] = 0.75
        c, a, _ = rz.forward(*p, atlas)
        c0, a0, _ = rz.forward(*p, plain(T, atlas, monkeypatch))
        assert torch.equal(c, c0) and torch.equal(a, a0)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("capture", [True, False])
def test_fit_steps_take_the_changed_templates_gpu(fused, capture, monkeypatch):
    T, src, p = templates(0), templates(1), params(8)
    target = torch.rand(H, W, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    jobs = []
    for atlas in (R.Atlas(T, "f32"), plain(T, None, monkeypatch)):
        job = ImageFitter(*p, atlas, target, torch.ones_like(target), FitConfig(fused=fused))
        job.step()
        if capture:
            job.capture()
        atlas.data.data.copy_(src)
        job.step()
        job.sync()
        jobs.append(job)
    got, want = jobs
    assert abs(got.loss() - want.loss()) <= 1e-6 * abs(want.loss())
    # Adam divides by the gradient's own size: its first moments, not the parameters,
    # carry the gradients
    assert (got.adam_m - want.adam_m).norm() <= 1e-5 * want.adam_m.norm()


def test_fp32_drop_in_takes_the_changed_templates_gpu(monkeypatch):
    T, src, p = templates(0), templates(1), params(9)
    tr = ctr.TileRasterizer(H, W, 16, num_primitives=N)
    none = torch.empty(0, device="cuda")
    run = lambda: tr(*p[:5], none, T, p[5], 0.0, torch.ones(7, device="cuda"))[0]
    before = run()
    T.data.copy_(src)
    after = run()
    assert not torch.equal(after, before)
    assert torch.equal(after, R.Rasterizer(H, W, 16, bin_mode=R.BIN_CULL).forward(*p, plain(src, None, monkeypatch))[0])


def test_changed_templates_on_several_streams_gpu(monkeypatch):
    """After each counted write, ordered before both streams, the renders of either
    stream (one through its `stream` argument) and fit steps walk the new texels."""
    T, p = templates(0), params(10)
    atlas, rz = R.Atlas(T, "f32"), R.Rasterizer(H, W)
    sets = [templates(k) for k in range(4)]
    want = [rz.forward(*p, plain(s, atlas, monkeypatch))[0] for s in sets]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for k in (1, 2, 3, 0, 1):
        T.copy_(sets[k])
        got = []
        for i, s in enumerate(streams):
            s.wait_stream(torch.cuda.current_stream())
            if i:
                got.append(rz.forward(*p, atlas, stream=s)[0])
            else:
                with torch.cuda.stream(s):
                    got.append(rz.forward(*p, atlas)[0])
        for s in streams:
            torch.cuda.current_stream().wait_stream(s)
        for g in got:
            assert torch.equal(g, want[k])
        torch.cuda.synchronize()


def test_a_writer_that_is_never_counted_gpu(monkeypatch):
    """Templates that change before every call: each render shows them, from copies
    packed anew after the first few calls that found theirs out of date."""
    T, p, rz = templates(0), params(11), R.Rasterizer(H, W)
    atlas = R.Atlas(T, "f32")
    misses = []
    monkeypatch.setattr(atlas, "_missed", lambda: (misses.append(1), R.Atlas._missed(atlas)))
    for k in range(40):
        T.data.copy_(templates(k % 7))
        ref = plain(T, atlas, monkeypatch)
        c, a, st = rz.forward(*p, atlas)
        c0, a0, _ = R.Rasterizer(H, W).forward(*p, ref)
        assert torch.equal(c, c0) and torch.equal(a, a0)
    assert 1 <= len(misses) <= 6
