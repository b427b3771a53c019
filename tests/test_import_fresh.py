"""The package and the build entry point in a process that has imported nothing else: a host program need not import torch
before the package, and the tests themselves always have (conftest.py imports it)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("code", [
    "import importlib; importlib.import_module('neural-networks_b200')",
    "import importlib; importlib.import_module('neural-networks_b200._lib')",
    "import __graft_entry__ as g; g.build()",
])
def test_runs_in_a_fresh_process(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:]
