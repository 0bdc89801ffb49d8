"""Calls of the network's kernels that are refused before anything reaches the GPU."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import ctypes
from graptor_gb300 import _lib as L
p = ctypes.c_void_p(256)  # never read: the call is refused
B, D, H, W = {dims}
rc = L.lib().gt_nn_conv3d_wgrad(p, 1, 1, 0, p, 1, 1, 1, 0, B, D, H, W, {k}, 128, p, p, 0, None)
assert rc != 0, rc
print("refused")
"""


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("dims", [(0, 4, 4, 4), (1, 0, 4, 4), (1, 4, 4, 0)])
def test_weight_gradient_of_an_empty_batch_is_refused(dims, k):
    r = subprocess.run([sys.executable, "-c", CODE.format(dims=dims, k=k)], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stderr)
