"""What the C++ host path does with arguments that no kernel should see: an error in Python, never the end of the process. Each in a
process of its own, on the CPU."""
import copy
import ctypes
import importlib
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEAD = "import importlib, torch; xl = importlib.import_module('neural-networks_b200'); ops = xl.ops; t = torch.ones(4)\n"


@pytest.mark.parametrize("code", [
    "ops.rms_norm_forward(torch.ones(2, 4), t, 0, False)",
    "ops.adamw(None, t, t, t, ops.AdamCfg(1e-3, 0.1, t=1), True)",
    "ops.adamw([1.0], t, t, t, ops.AdamCfg(1e-3, 0.1, t=1), True)",
])
def test_a_wrong_argument_is_an_error(code):
    r = subprocess.run([sys.executable, "-c", HEAD + "try:\n    %s\nexcept (xl._lib.XlstmError, TypeError):\n    print('refused')" % code], cwd=ROOT,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stdout[-2000:])


def test_a_copied_shape_points_at_its_own_fields():
    import torch
    ops = importlib.import_module("neural-networks_b200").ops
    st = ops.MlstmShape(1, 2, 3, 64, 64, 64, torch.float32, torch.float32)
    other = copy.deepcopy(st)
    assert other.addr == ctypes.addressof(other.c) != st.addr
