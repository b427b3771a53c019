"""The sLSTM loops when the device has no memory left to give: a host whose runtime holds all of it, as the reference's buffer pool does,
runs them as before the register-resident kernels came, on those that need nothing beyond their arguments. In a process of its own, whose
calls before that are the short ones that do not ask for memory either."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = r"""
import ctypes, glob, importlib, os, sys
sys.path[:0] = [%r, os.path.join(%r, "tests")]
import torch
xl = importlib.import_module("neural-networks_b200")
ops = xl.ops
B, NH, dh = 32, 4, 256
H = NH * dh
g = torch.Generator(device="cuda").manual_seed(1)
wh = torch.randn(NH, dh, 4 * dh, device="cuda", generator=g) / 16
bc = torch.zeros(4 * H, device="cuda")
def buffers(T):
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    e = lambda n: tuple(torch.empty((B, H), device="cuda") for _ in range(n))
    return dict(T=T, g=r(B, T, 4 * H), dy=r(B, T, H), out=torch.empty((B, T, H), device="cuda"), slabs=ops.SlstmSlabs(B, T, H, "cuda"), st=e(4), ds=e(3))
def run(s):
    ops.slstm_fused_time(wh, s["g"], bc, s["st"], s["out"], s["slabs"], nh=NH)
    ops.slstm_fused_time_bwd(wh, s["dy"], s["g"], s["ds"], s["slabs"], nh=NH)
    torch.cuda.synchronize()
    return s["out"].clone(), s["g"].clone()
def reset(s, keep):
    s["g"].copy_(keep)
T = 24
short, full = buffers(4), buffers(T)
keep = full["g"].clone()
room = [torch.empty_like(x) for x in (full["out"], full["g"])]
run(short)
torch.cuda.synchronize()
cudart = ctypes.CDLL(glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*"))[0])
held = []
for size in (1 << 30, 1 << 28, 1 << 25, 1 << 23, 1 << 21, 1 << 20):
    while True:
        p = ctypes.c_void_p()
        if cudart.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)):
            break
        held.append(p)
cudart.cudaGetLastError()
ops.slstm_fused_time(wh, full["g"], bc, full["st"], full["out"], full["slabs"], nh=NH)
ops.slstm_fused_time_bwd(wh, full["dy"], full["g"], full["ds"], full["slabs"], nh=NH)
torch.cuda.synchronize()
room[0].copy_(full["out"]); room[1].copy_(full["g"])
torch.cuda.synchronize()
for p in held:
    cudart.cudaFree(p)
assert xl._lib.lib.xlstm_device_status() == 0
full["g"].copy_(keep)
a = run(full)
for x, y in zip(room, a):
    e = float((x - y).abs().max() / y.abs().max())
    assert e < 1e-4, e
print("same")
"""


def test_loops_run_when_no_memory_can_be_had():
    env = dict(os.environ, CUDA_MODULE_LOADING="EAGER")  # no kernel's code is waiting for memory
    r = subprocess.run([sys.executable, "-c", CODE % (ROOT, ROOT)], cwd=ROOT, env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout[-3000:]
