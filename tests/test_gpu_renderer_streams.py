"""GPU tests of what a SimpleTileRenderer keeps between calls when these run on
several streams and in inference mode."""
import pytest
import torch

from diffbmp_b200.pydiffbmp.core.renderer.simple_tile_renderer import SimpleTileRenderer

pytestmark = pytest.mark.gpu

N, P = 70001, 3


def renderer():
    return SimpleTileRenderer((64, 64), torch.rand(P, 16, 16, device="cuda"))


def expected():
    return (torch.arange(N, dtype=torch.int32) % P).flip(0)


def test_template_ids_made_on_a_busy_stream_gpu():
    """A call on another stream reads the ids that the first one is still to write."""
    r = renderer()
    renderer()._global_bmp_sel(N).clone()            # (a kernel's first launch may wait for the device)
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        poison = [torch.full((N,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
        a.synchronize()
        del poison                                   # the ids' memory starts as -1
        torch.cuda._sleep(200_000_000)               # a tenth of a second
        r._global_bmp_sel(N)
    with torch.cuda.stream(b):
        got = r._global_bmp_sel(N).clone()
    b.synchronize()
    assert torch.equal(got.cpu(), expected())
    torch.cuda.synchronize()


def test_template_ids_outlive_their_replacement_gpu():
    """Work that another stream enqueued on the ids still reads them after a call of
    another N has replaced them."""
    r = renderer()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        r._global_bmp_sel(N)
    a.synchronize()
    with torch.cuda.stream(b):
        torch.cuda._sleep(200_000_000)
        got = r._global_bmp_sel(N).clone()
    with torch.cuda.stream(a):
        r._global_bmp_sel(N + 1)
        over = [torch.full((N,), -1, dtype=torch.int32, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    assert torch.equal(got.cpu(), expected()) and len(over) == 4


def test_ids_made_in_inference_mode_gpu():
    r = renderer()
    p = [torch.rand(5, device="cuda") * 60, torch.rand(5, device="cuda") * 60, torch.rand(5, device="cuda") * 20 + 4,
         torch.rand(5, device="cuda"), torch.rand(5, device="cuda"), torch.rand(5, 3, device="cuda")]
    with torch.inference_mode():
        want = r.render_from_params(*p)
    q = [x.clone().requires_grad_() for x in p]
    got = r.render_from_params(*q)
    assert torch.equal(got.detach(), want)
    got.sum().backward()
    assert all(torch.isfinite(x.grad).all() for x in q)
