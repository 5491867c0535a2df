"""GPU tests of one Rasterizer called by several host threads."""
import threading

import numpy as np
import pytest
import torch

from diffbmp_b200 import rasterizer as R

pytestmark = pytest.mark.gpu

H, W = 130, 170


def params(seed, N):
    rng = np.random.default_rng(seed)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    return [cu(rng.uniform(0, [W, H], (N, 2))), cu(rng.uniform(2, 40, N)), cu(rng.uniform(0, 7, N)),
            cu(rng.normal(0, 1, N)), cu(rng.normal(0, 1, (N, 3))),
            torch.from_numpy(rng.integers(0, 2, N).astype(np.int32)).cuda()]


class TakenBetween(list):
    """A pool whose last buffer another thread takes between a look and the pop."""

    def __len__(self):
        return 1


def test_a_pool_emptied_by_another_thread_gpu():
    rz, p = R.Rasterizer(H, W), params(0, 50)
    atlas = R.Atlas(torch.rand(2, 20, 24, device="cuda"), "f16q")
    want = rz.forward(*p, atlas)[0]
    rz._pins = TakenBetween()
    assert torch.equal(rz.forward(*p, atlas)[0], want)


@pytest.mark.parametrize("kind", ["f32", "f16q"])
def test_threads_with_other_sizes_and_streams_gpu(kind):
    atlas = R.Atlas(torch.rand(2, 20, 24, device="cuda"), kind)
    shared = R.Rasterizer(H, W)
    sets = [params(k, n) for k, n in enumerate((3, 400, 900, 4000))]
    up = torch.randn(H, W, 3, device="cuda"), torch.randn(H, W, device="cuda")
    want = []
    for p in sets:
        c, _, st = R.Rasterizer(H, W).forward(*p, atlas)
        want.append((c, R.Rasterizer(H, W).backward(st, *up, *p[1:5], atlas)))
    torch.cuda.synchronize()
    errors = []

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for _ in range(40):
                    c, _, st = shared.forward(*sets[k], atlas)
                    g = shared.backward(st, *up, *sets[k][1:5], atlas)
                s.synchronize()
                assert torch.equal(c, want[k][0])
                for a, b in zip(g, want[k][1]):
                    assert (a - b).norm() <= 1e-6 * b.norm()
        except BaseException as e:    # noqa: BLE001 (reported by the test below)
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
