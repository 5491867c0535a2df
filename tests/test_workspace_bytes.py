"""CPU test of the binning workspace: no more than its arrays take."""
import ctypes

import pytest

from diffbmp_b200._lib import ATLAS_F16_QUAD, BIN_CONTENT, Canvas, lib


@pytest.mark.parametrize("H,W,N,parts,slices", [(4096, 4096, 100000, 66, 2), (256, 256, 512, 1, 1)])
@pytest.mark.parametrize("batch", [1, 3])
def test_workspace_holds_its_arrays_once(H, W, N, parts, slices, batch):
    """Rectangles, counts per (tile, counting slice), positions per (tile, writing
    slice), row totals and, on the larger canvas, a bit per primitive and cell of
    32 tiles; each array may be padded to 256 bytes."""
    T, rows, cells = H * W // 1024, H // 32, -(-W // 1024) * H // 32
    masks = cells * -(-N // 512) * 64 if N > 1536 else 0
    need = batch * (16 * N + 4 * T * parts + 8 * (T * slices + 1) + 8 * rows + masks)
    cv = Canvas(H, W, 32, N, 1, 16, 16, ATLAS_F16_QUAD, BIN_CONTENT, 1.0, 1e-6, 0)
    got = lib.dbmp_bin_batch_workspace_bytes(ctypes.byref(cv), batch)
    assert need <= got <= need + 5 * 256
