"""GPU test of the call after a failed one: an error that a launch returned (here
into a stream capture that the host has invalidated) is that call's alone."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
from diffbmp_b200 import rasterizer as R
T = torch.rand(1, 16, 16, device="cuda")
p = [torch.rand(5, 2, device="cuda") * 40, torch.rand(5, device="cuda") * 9 + 2, torch.zeros(5, device="cuda"),
     torch.zeros(5, device="cuda"), torch.zeros(5, 3, device="cuda"), torch.zeros(5, dtype=torch.int32, device="cuda")]
atlas, rz = R.Atlas(T, "f16q"), R.Rasterizer(64, 64)
c, a, st = rz.forward(*p, atlas)
s = torch.cuda.Stream()
g = torch.cuda.CUDAGraph()
failed = None
with torch.cuda.stream(s):
    g.capture_begin()
    try:
        s.synchronize()                  # not allowed: the capture is invalid from here on
    except RuntimeError:
        pass
    try:
        R.call("dbmp_convert_half", 1, (R.ctypes.c_void_p * 1)(c.data_ptr()), (R.ctypes.c_void_p * 1)(a.data_ptr()),
               (R.ctypes.c_longlong * 1)(1), 1, R._stream())
    except R.DbmpError as e:
        failed = str(e)
    try:
        g.capture_end()
    except RuntimeError:
        pass
assert failed and "apture" in failed, failed
R.call("dbmp_template_bboxes", T.data_ptr(), 1, 16, 16, atlas.bbox.data_ptr(), R._stream())
torch.cuda.synchronize()
print("the next call succeeded")
"""


def test_next_call_after_a_failed_launch_gpu():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "the next call succeeded" in r.stdout, r.stdout + r.stderr
