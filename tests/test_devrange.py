"""The host-side check of a caller's device array before a kernel reads or writes it: the address
ranges on the CPU, against a list of allocations, and on a GPU an array that ends before its field."""
import ctypes as C
import os
import pathlib
import shutil
import subprocess

import numpy as np
import pytest

from helpers import small_params

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "suli-openmp_b200" / "csrc"

MAIN = r"""
#include <cstdio>
#include "devrange.h"
int main() {
    // [1000, 1100) [1100, 1150) gap [1200, 1300)
    const std::uintptr_t base[3] = {1000, 1100, 1200};
    const std::size_t size[3] = {100, 50, 100};
    auto lookup = [&](std::uintptr_t p, std::uintptr_t* b, std::size_t* s) {
        for (int n = 0; n < 3; ++n)
            if (p >= base[n] && p < base[n] + size[n]) { *b = base[n]; *s = size[n]; return true; }
        return false;
    };
    unsigned long p, n;
    while (std::scanf("%lu %lu", &p, &n) == 2) std::printf("%d\n", (int)suli::range_kind(p, n, lookup));
}
"""

CASES = [   # address, bytes, kind
    (1000, 100, 1), (1000, 1, 1), (1099, 1, 1), (1200, 100, 1), (1250, 50, 1),
    (1000, 101, 0), (1050, 100, 0), (1099, 2, 0),
    (1000, 151, -1), (1100, 51, -1), (1149, 2, -1), (1250, 51, -1), (1150, 8, -1), (999, 10, -1), (1300, 1, -1),
]


def test_range_kind(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "main"
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Wextra", "-Werror", f"-I{CSRC}", str(tmp_path / "main.cpp"),
                    "-o", str(exe)], check=True)
    got = subprocess.run([str(exe)], input="\n".join(f"{p} {n}" for p, n, _ in CASES), capture_output=True, text=True,
                         check=True).stdout.split()
    assert [int(g) for g in got] == [k for _, _, k in CASES]


@pytest.mark.gpu
def test_short_device_array_is_refused(pkg):
    import torch
    torch.cuda.init()
    rt = C.CDLL("libcudart.so.12")   # torch's, already loaded: an allocation of exactly these bytes
    size = 32 << 20
    mem = C.c_void_p()
    assert rt.cudaMalloc(C.byref(mem), C.c_size_t(size)) == 0
    try:
        assert rt.cudaMemset(mem, 0, C.c_size_t(size)) == 0
        assert rt.cudaDeviceSynchronize() == 0
        p = small_params(96, 96, 96)   # a field of 7 MB
        with pkg.Solver(p) as s:
            at = lambda address: C.cast(C.c_void_p(address), C.POINTER(C.c_double))
            field = pkg._abi.FIELD["prd1"]
            for room in (8, 1 << 20):
                assert s.lib.suli_upload(s._h, field, at(mem.value + size - room)) < 0
            # whole arrays still go through, from either end of the allocation, aligned or not
            n = int(np.prod(s.shape("prd1"))) * 8
            for address in (mem.value, mem.value + size - n, mem.value + 4):
                assert s.lib.suli_upload(s._h, field, at(address)) == 0
                assert s.lib.suli_download(s._h, field, at(address)) == 0
            assert not s.download("prd1").any()
    finally:
        rt.cudaFree(mem)
