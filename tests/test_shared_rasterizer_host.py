"""CPU tests of what the calls of several threads share in one Rasterizer: each read
of it is made once, so that another thread's call in between cannot mix two sizes."""
import ctypes

import torch

from diffbmp_b200 import rasterizer as R


class Between(R.Rasterizer):
    """A rasterizer whose size memo another thread's call replaces after each read."""

    @property
    def _ws_need(self):
        v = self._memo
        self._memo = ((1, 3), 256)
        return v

    @_ws_need.setter
    def _ws_need(self, v):
        self._memo = v


def test_workspace_size_of_a_call_is_its_own():
    rz = Between(2048, 2048, device="cpu")
    cv = R.Canvas(2048, 2048, 32, 20000, 1, 8, 8, R.ATLAS_F32, R.BIN_CONTENT, 1.0, 1e-6, 0)
    need = int(R.lib.dbmp_bin_batch_workspace_bytes(ctypes.byref(cv), 2))
    assert need > 1024
    for memo in (((2, 20000), (need + 255) & ~255), ((7, 7), 512)):
        rz._memo = memo
        t, nbytes = rz._scratch(cv, 2, 20000, None)
        assert nbytes >= need and t.numel() >= nbytes + 8 * 2 and t.device == torch.device("cpu")


def test_copies_start_without_pinned_buffers():
    """A copied pinned tensor is pageable memory, which the device cannot write to."""
    import copy
    import pickle
    rz = R.Rasterizer(64, 96, device="cpu")
    rz._pins, rz._hint = [torch.zeros(2, dtype=torch.int32)], 77
    for other in (copy.deepcopy(rz), pickle.loads(pickle.dumps(rz)), copy.copy(rz)):
        assert other._pins == [] and other._hint == 77 and (other.H, other.W, other.T) == (64, 96, 6)
    assert len(rz._pins) == 1
