"""dgtm_fe_forward_noalloc loads the kernels of every D in its first call: a later call
whose D takes another kernel may be the first inside a stream capture, and reserves
nothing.  In a process of its own, where nothing else has loaded them."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = r"""
import importlib, sys
sys.path.insert(0, %r)
import torch
pkg = importlib.import_module("da-gtm_gb300")
lib = pkg.load_library()
g = torch.Generator(device="cuda").manual_seed(1)
cases = {}
for D in (12, 60, 96, 128, 140, 166, 200, 256):  # the eight classes ceil(D / 32)
    cases[D] = (torch.rand((70, D), device="cuda", generator=g), torch.rand((500, D), device="cuda", generator=g),
                torch.zeros((), dtype=torch.float64, device="cuda"))

def call(D, F):
    Y, T, _ = cases[D]
    s = torch.cuda.current_stream().cuda_stream
    assert lib.dgtm_fe_forward_noalloc(Y.data_ptr(), T.data_ptr(), 500, 70, D, 5.0, 1.2, s, F.data_ptr()) == 0

call(12, cases[12][2])
torch.cuda.synchronize()
graphs = {}
free = None
for D in cases:
    graphs[D] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graphs[D]):
        call(D, cases[D][2])
torch.cuda.synchronize()
for D in cases:
    ref = torch.zeros((), dtype=torch.float64, device="cuda")
    graphs[D].replay()
    call(D, ref)
    torch.cuda.synchronize()
    assert torch.isfinite(ref) and ref.item() == cases[D][2].item(), D
free = torch.cuda.mem_get_info()[0]
for D in cases:
    call(D, cases[D][2])
torch.cuda.synchronize()
assert torch.cuda.mem_get_info()[0] == free
print("ok")
"""


def test_every_kernel_is_loaded_by_the_first_call():
    env = dict(os.environ, CUDA_MODULE_LOADING="LAZY")
    r = subprocess.run([sys.executable, "-c", CODE % ROOT], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
