"""GPU tests of copied and pickled objects after use: they render and fit as the
originals do, from memory of their own."""
import copy
import gc
import pickle

import numpy as np
import pytest
import torch

from diffbmp_b200 import fitting as F
from diffbmp_b200 import rasterizer as R
from diffbmp_b200.pydiffbmp.core.renderer.simple_tile_renderer import SimpleTileRenderer

pytestmark = pytest.mark.gpu

H, W, N = 70, 100, 50
COPIES = {"deepcopy": copy.deepcopy, "pickle": lambda x: pickle.loads(pickle.dumps(x))}


@pytest.fixture(autouse=True)
def packed_at_any_size(monkeypatch):
    monkeypatch.setattr(R, "quads_pay", lambda pixels, N, texels: True)
    monkeypatch.setattr(F, "fit_quads_pay", lambda pixels, N, texels: True)


def params(seed=0):
    rng = np.random.default_rng(seed)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(4, 40, N)), cu(rng.uniform(0, 7, N)),
            cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3))), torch.zeros(N, dtype=torch.int32, device="cuda")]


def overwrite_freed_memory():
    gc.collect()
    torch.cuda.synchronize()
    return [torch.full((n,), float("nan"), device="cuda") for n in (2, 64, 1024, 4096, 8192, 65536) for _ in range(40)]


@pytest.mark.parametrize("how", COPIES)
@pytest.mark.parametrize("kind", ["f32", "f16q"])
def test_rasterizer_and_atlas_gpu(how, kind):
    p, rz, atlas = params(), R.Rasterizer(H, W), R.Atlas(torch.rand(1, 24, 24, device="cuda"), kind)
    c, a, _ = rz.forward(*p, atlas)
    rz2, atlas2 = COPIES[how](rz), COPIES[how](atlas)
    del rz, atlas
    junk = overwrite_freed_memory()
    c2, a2, st = rz2.forward(*p, atlas2)
    assert torch.equal(c2, c) and torch.equal(a2, a) and len(junk)
    rz2.backward(st, torch.randn_like(c), torch.randn_like(a), *p[1:5], atlas2)


@pytest.mark.parametrize("how", COPIES)
@pytest.mark.parametrize("fp16", [False, True])
def test_renderer_gpu(how, fp16):
    m, r, th, v, c, _ = params()
    q = (m[:, 0].contiguous(), m[:, 1].contiguous(), r, th, v, c)
    one = SimpleTileRenderer((H, W), torch.rand(2, 24, 24, device="cuda"), use_fp16=fp16)
    want = one.render_from_params(*q)
    two = COPIES[how](one)
    del one
    junk = overwrite_freed_memory()
    assert torch.equal(two.render_from_params(*q), want) and len(junk)


@pytest.mark.parametrize("kind", ["f32", "f16q"])
@pytest.mark.parametrize("fused", [True, False])
def test_fit_job_gpu(kind, fused):
    target = torch.rand(H, W, 3, device="cuda")
    job = F.ImageFitter(*params(), R.Atlas(torch.rand(1, 24, 24, device="cuda"), kind), target, None,
                        F.FitConfig(fused=fused))
    job.step()
    job.sync()
    other = copy.deepcopy(job)
    job.step()
    job.sync()
    want = job.adam_m.clone()
    del job
    junk = overwrite_freed_memory()
    other.step()
    other.sync()
    assert (other.adam_m - want).norm() <= 1e-5 * want.norm() and len(junk)


def test_backward_in_a_graph_gpu():
    """Captured on another stream than the packed copy's, replayed after a write to
    the templates that PyTorch does not count."""
    p, T, rz = params(), torch.rand(1, 24, 24, device="cuda"), R.Rasterizer(H, W)
    atlas = R.Atlas(T, "f32")
    c, a, st = rz.forward(*p, atlas)
    up = torch.randn_like(c), torch.randn_like(a)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = rz.backward(st, *up, *p[1:5], atlas)
    for change in (False, True):
        if change:
            T.data.mul_(0.9)
        g.replay()
        for x, y in zip(got, rz.backward(st, *up, *p[1:5], atlas)):
            assert (x - y).norm() <= 1e-6 * y.norm()
