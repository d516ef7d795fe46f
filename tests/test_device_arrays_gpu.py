"""GPU test of fields given and taken as device arrays, whichever allocator made them: one block of
cudaMalloc, memory mapped in pieces (a field then lies in several) and a stream-ordered pool.  Each runs in
its own process, since the allocator is chosen once a process."""
import os
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = pathlib.Path(__file__).resolve().parent

CHILD = r"""
import ctypes as C
import sys
sys.path.insert(0, sys.argv[1])
import torch
from helpers import pkg, small_params
at = lambda t: C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))
g = torch.Generator(device="cuda:0").manual_seed(1)
for n in (12, 176):   # fields of 22 kB and of 45 MB
    with pkg.Solver(small_params(n, n, n)) as s:
        field = pkg._abi.FIELD["prd1"]
        a = torch.randn(tuple(reversed(s.shape("prd1"))), dtype=torch.float64, device="cuda:0", generator=g)
        b = torch.zeros_like(a)
        # twice the field and 8 bytes, so that an offset one still fits
        c = torch.zeros(2 * a.numel() + 1, dtype=torch.float64, device="cuda:0")
        torch.cuda.synchronize()
        s.upload_device("prd1", a)
        for t in (b, c[1:], c[a.numel():]):
            assert s.lib.suli_download(s._h, field, at(t)) == 0, s.lib.suli_last_error(s._h)
            assert torch.equal(t.flatten()[:a.numel()], a.flatten())
"""


@pytest.mark.parametrize("conf", ["expandable_segments:False", "expandable_segments:True", "backend:cudaMallocAsync"])
def test_any_allocator(conf):
    env = dict(os.environ, PYTORCH_CUDA_ALLOC_CONF=conf, PYTORCH_ALLOC_CONF=conf)
    r = subprocess.run([sys.executable, "-c", CHILD, str(HERE)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
