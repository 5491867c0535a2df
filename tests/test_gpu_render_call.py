"""GPU tests of the one-call render (binning and forward without the host in
between): growth of the list capacity, several streams in flight, refusal under
graph capture, and the drop-in FP16 conversions."""
import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu


def params(seed, N, W, H, rmax=40.0):
    rng = np.random.default_rng(seed)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(2, rmax, N)), cu(rng.uniform(0, 7, N)),
            cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3))),
            torch.from_numpy(rng.integers(0, 2, N).astype(np.int32)).cuda()]


def atlas():
    rng = np.random.default_rng(0)
    return R.Atlas(torch.from_numpy(rng.uniform(0, 1, (2, 20, 24)).astype(np.float32)).cuda(), "f32")


def two_calls(rz, p, at):
    """The same image from dbmp_bin and dbmp_forward on their own."""
    import ctypes
    prim, lists = rz.bin(*p, at)
    out = [torch.empty(s, device="cuda", dtype=t) for s, t in
           (((rz.H, rz.W, 3), torch.float32), ((rz.H, rz.W), torch.float32), ((rz.H, rz.W), torch.float32),
            ((rz.H, rz.W), torch.int32))]
    cv = rz.canvas(p[1].numel(), at)
    R.call("dbmp_forward", ctypes.byref(cv), R._ptr(prim), R._ptr(at.data), R._ptr(lists.offsets),
           R._ptr(lists.indices), *[R._ptr(o) for o in out], R._stream())
    return out, lists


@pytest.mark.parametrize("N,hint", [(0, None), (1, None), (500, 0), (500, 7), (500, None)])
def test_render_grows_its_lists_gpu(N, hint):
    at, rz = atlas(), R.Rasterizer(130, 170)
    p = params(1, N, 170, 130)
    rz._hint = hint
    c, a, st = rz.forward(*p, at)
    want, lists = two_calls(rz, p, at)
    assert torch.equal(c, want[0]) and torch.equal(a, want[1]) and torch.equal(st.last_pos, want[3])
    assert st.lists.length == lists.length
    assert torch.equal(st.lists.mapping_tensor(), lists.mapping_tensor())


@pytest.mark.parametrize("kind,ts,N,opac,blend", [
    ("f32", 32, 40, 0.0, 0.0), ("f16q", 16, 700, -5.0, 0.0),     # 700 faint layers: beyond the chunks whose masks are kept
    ("bf16", 32, 700, -5.0, 0.0), ("f32", 32, 300, -3.0, 0.5)])
def test_backward_with_the_forwards_masks_gpu(kind, ts, N, opac, blend):
    """The backward that stages from the forward's masks against the one that tests
    again: the same terms in the same order per warp (FP64 sums over warps are
    unordered: 1e-6 of the block's norm)."""
    W, H = 75, 61
    rng = np.random.default_rng(5)
    at = R.Atlas(torch.from_numpy(rng.uniform(0, 1, (2, 20, 24)).astype(np.float32)).cuda(), kind)
    p = params(3, N, W, H, 60.0)
    p[3] += opac
    maps = torch.rand(N, 20, 24, 3, device="cuda") if blend else None
    rz = R.Rasterizer(H, W, ts)
    c, a, st = rz.forward(*p, at, None, None, maps, blend)
    assert int(st.last_pos.max()) >= (8 * 32 if N == 700 else 1)
    gc, ga = torch.randn_like(c), torch.randn_like(a)
    with_masks = rz.backward(st, gc, ga, *p[1:5], at)
    st.walk_masks = None
    for x, y in zip(with_masks, rz.backward(st, gc, ga, *p[1:5], at)):
        assert (x - y).norm() <= 1e-6 * y.norm()


def test_renders_on_several_streams_gpu():
    at, rz = atlas(), R.Rasterizer(300, 500)
    sets = [params(k, 300 + 200 * k, 500, 300) for k in range(3)]
    want = [two_calls(rz, p, at)[0][0] for p in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    got = []
    for _ in range(10):
        for p, s in zip(sets, streams):
            with torch.cuda.stream(s):
                got.append(rz.forward(*p, at)[0])
    torch.cuda.synchronize()
    for k, g in enumerate(got):
        assert torch.equal(g, want[k % 3])


def test_render_refuses_graph_capture_gpu():
    at, rz = atlas(), R.Rasterizer(64, 64)
    p = params(2, 20, 64, 64)
    want = rz.forward(*p, at)[0]
    g = torch.cuda.CUDAGraph()
    with pytest.raises(Exception, match="captur"):
        with torch.cuda.graph(g):
            rz.forward(*p, at)
    torch.cuda.synchronize()
    assert torch.equal(rz.forward(*p, at)[0], want)


def test_half_conversions_equal_torch_gpu():
    from diffbmp_b200.cuda_tile_rasterizer import _ext
    x = torch.cat([torch.randn(999) * 1e3, torch.tensor([0.0, -0.0, 1e-8, 65519.0, 65520.0, float("inf"), float("nan")])]).cuda()
    ts = [x[:k].clone() for k in (0, 1, 255, 257)] + [x] * 5
    for t, h in zip(ts, _ext._halves(ts)):
        assert torch.equal(h.view(torch.int16)[~t.isnan()], t.half().view(torch.int16)[~t.isnan()])
        assert torch.equal(h.isnan(), t.isnan())
    hs = [t.half() for t in ts]
    for h, f in zip(hs, _ext._floats(*hs)):
        assert torch.equal(f.nan_to_num(7.0), h.float().nan_to_num(7.0))
