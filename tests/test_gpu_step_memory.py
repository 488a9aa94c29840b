"""The step calls on device arrays need no device memory: where none is left for
the grouping's scratch they run on the particles in the caller's order.  A
process of its own takes the device's free memory but for less than the scratch
of the call (24 bytes a particle) and compares the scatter and the gathers with
the same calls made while there was memory.

Tolerance: FP64 sums in another order, 1e-12 relative as for every step call."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes as C
import sys
import numpy as np
import torch
from se_fast_gridding_b200 import fgg as F, solver

P, M, force = int(sys.argv[1]), 32, sys.argv[2] == "force"
LEFT = 24 << 20
small, N = 1000, int(sys.argv[3])


def setup(n):
    _, p = F.fcn_params(M, P, 1.0, 4.0, solver.default_m(P), n)
    w = F.Work(p, force=force, where="cuda")
    g = torch.Generator("cuda").manual_seed(n)
    x = torch.rand(3 * n, dtype=torch.float64, device="cuda", generator=g)
    q = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    F.call("SE_FGG_base_gaussian", C.byref(w.s), C.byref(p))
    F.call("SE_FGG_expand_all_SSE_force" if force else "SE_FGG_expand_all", C.byref(w.s), C.byref(F.state(x, q)),
           C.byref(p))
    return p, w, x, q, torch.zeros((3 if force else 1) * n, dtype=torch.float64, device="cuda")


def steps(p, w, x, q, out):
    st = F.state(x, q)
    F.call("SE_FGG_grid_split_AVX_dispatch_force" if force else "SE_FGG_grid_split", C.byref(w.s), C.byref(st),
           C.byref(p))
    if force:
        F.call("SE_FGG_int_split_AVX_dispatch_force", F.dptr(out), C.byref(st), C.byref(w.s), C.byref(p))
    else:
        F.call("SE_FGG_int_split", F.dptr(out), C.byref(w.s), C.byref(p))


a, b = setup(small), setup(N)
steps(*a)                      # few particles: every kernel without grouping is loaded
torch.cuda.synchronize()
hold = []
for size in (1 << 30, 64 << 20, 2 << 20):
    while torch.cuda.mem_get_info()[0] > LEFT + size:
        try:
            hold.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            break
assert torch.cuda.mem_get_info()[0] < 16 * N, "the scratch would fit"
steps(*b)                      # no memory for the grouping
H, out = b[1].get("H").copy(), b[4].cpu().numpy()
del hold[:]
torch.cuda.empty_cache()
b[1].arrays["H"].zero_()
b[4].zero_()
steps(*b)                      # grouped
for got, ref in ((H, b[1].get("H")), (out, b[4].cpu().numpy())):
    assert np.linalg.norm(got - ref) < 1e-12 * np.linalg.norm(ref)
print("equal")
"""


@pytest.mark.parametrize("P,N", [(8, 2_600_000)])
@pytest.mark.parametrize("mode", ["potential", "force"])
def test_steps_without_scratch(mode, P, N):
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(P), mode, str(N)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "equal" in r.stdout, r.stdout + r.stderr
