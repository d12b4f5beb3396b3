"""dwf_cg_noalloc after its first call: a call with another lattice or operator, which
picks another kernel, loads no code and so takes no device memory. Run in a process
of its own, where nothing else has loaded the kernels."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes as C
import torch
from three_part_dwf_study_b200 import _capi as A
shapes = [(2, 2, 1), (4, 4, 3), (5, 5, 13), (3, 5, 7), (8, 8, 24), (17, 23, 4), (12, 10, 6), (24, 20, 10),
          (40, 40, 8), (31, 16, 24), (6, 6, 2), (33, 9, 6), (16, 16, 16), (64, 64, 16), (20, 20, 12)]
def bufs(Nt, Nx, Ls):
    n = 2 * Nt * Nx * Ls
    return (torch.zeros(2 * Nt * Nx, dtype=torch.float64, device="cuda"),
            torch.randn(n, dtype=torch.complex128, device="cuda"), torch.empty(n, dtype=torch.complex128, device="cuda"))
def solve(s, b, op):
    info, p = A.SolveInfo(), A.DwfParams(*s, 1.0, 0.2, 0.0, 0)
    st = A.lib().dwf_cg_noalloc(C.byref(p), op, *(C.c_void_p(t.data_ptr()) for t in b), 0, 1e-8, 2000, None, C.byref(info))
    assert st == 0 and info.converged, (s, st)
b = [bufs(*s) for s in shapes]
first = bufs(16, 12, 8)
torch.cuda.synchronize()
solve((16, 12, 8), first, 3)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
for s, x in zip(shapes, b):
    for op in (2, 3):
        solve(s, x, op)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free, (s, op, free - torch.cuda.mem_get_info()[0])
"""


def test_later_lattices_load_no_code():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).resolve().parents[1], timeout=240,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
