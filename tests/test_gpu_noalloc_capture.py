"""ehd_poisson_noalloc captured into a graph: after one call outside any capture, a
call on any other depth can be captured, whatever shared memory its z solve takes
(more than 48 KB from NZ = 99 on).  In a process of its own, because a kernel's
attributes belong to the process and other tests set them.
"""
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

CODE = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import ehd, torch
def params(nz):
    return ehd.params_from_groups(16, 12, nz, 16 / (nz - 1), 12 / (nz - 1), T=200, M=10, C=10, Fe=4000)
def solve(p, q, out):
    rc = ehd.lib().ehd_poisson_noalloc(ctypes.byref(p), q.data_ptr(), *[o.data_ptr() for o in out],
                                       torch.cuda.current_stream().cuda_stream)
    assert rc == 0, ehd.lib().ehd_last_error()
def arrays(nz):
    g = torch.Generator(device="cuda").manual_seed(nz)
    q = torch.rand(nz, 12, 16, generator=g, dtype=torch.float64, device="cuda")
    return q, [torch.full_like(q, float("nan")) for _ in range(4)]
p, (q, out) = params(9), arrays(9)
solve(p, q, out)                       # the first call
torch.cuda.synchronize()
for nz in (99, 201, 860):
    p, (q, out) = params(nz), arrays(nz)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve(p, q, out)
    graph.replay()
    torch.cuda.synchronize()
    ref = [torch.empty_like(q) for _ in range(4)]
    solve(p, q, ref)
    torch.cuda.synchronize()
    for a, b in zip(out, ref):
        assert torch.equal(a, b) and bool(torch.isfinite(a).all())
print("captured")
"""


def test_deeper_grids_can_be_captured_after_the_first_call():
    r = subprocess.run([sys.executable, "-c", CODE, str(PKG)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]
