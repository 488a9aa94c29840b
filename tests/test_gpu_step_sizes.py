"""The reference step calls at the sizes where their kernels change: the scatter
straight into the grid by a CTA or a warp per particle (P < 8: the cells in order), or
through shared-memory windows, the gather of P < 8 and P = 9, and the expansion's last 32
particles; against the oracle.

Tolerance: FP64 sums of a few thousand terms in another order, 1e-12 relative
as for every other step call."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def F():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import fgg
    fgg.lib()
    return fgg


def setup(F, N, M, P, clusters, force):
    import oracle as O
    import torch
    x, q = O.synthetic_system(N, 1.0, seed=N + P, charges="uniform", clusters=clusters, sigma=0.01)
    if N == 1:
        q[:] = 1.0
    m = 0.95 * np.sqrt(O.PI * P)
    _, p = F.fcn_params(M, P, 1.0, 4.0, m, N)
    po = O.Setup(M=M, P=P, L=1.0, xi=4.0, m=m, N=N).params()
    w = F.Work(p, force=force, where="cuda")
    xc, qc = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
    F.call("SE_FGG_base_gaussian", C.byref(w.s), C.byref(p))
    return x, q, p, po, w, F.state(xc, qc), (xc, qc)


# a particle per CTA up to 16 P^2, windows from 1e8 stencil cells on (P = 8, 12, 16)
# or 2.5e8 (P = 13 to 15)
@pytest.mark.parametrize("N,M,P,clusters", [
    (1, 9, 1, 0), (16, 9, 1, 0), (17, 9, 1, 0), (33, 12, 2, 0), (64, 12, 2, 0), (65, 12, 2, 0), (145, 20, 3, 0),
    (257, 20, 4, 1), (401, 21, 5, 0), (577, 20, 6, 0), (784, 22, 7, 0), (785, 22, 7, 1), (1024, 24, 8, 0),
    (1025, 24, 8, 0), (1300, 25, 9, 0), (22_000, 30, 9, 1), (4096, 32, 16, 0), (4097, 32, 16, 0), (300, 34, 32, 0), (95, 40, 17, 0),
    (195_312, 32, 8, 0), (195_313, 32, 8, 2), (57_871, 30, 12, 2), (24_415, 33, 16, 0), (24_415, 40, 16, 2),
    (113_792, 28, 13, 0)])
@pytest.mark.parametrize("force", [False, True])
def test_steps_equal_oracle(F, N, M, P, clusters, force):
    import oracle as O
    x, q, p, po, w, st, keep = setup(F, N, M, P, clusters, force)
    zs, ex = O.base_gaussian(po), O.expand_all(po, x, 3, force)
    F.call("SE_FGG_expand_all_SSE_force" if force else "SE_FGG_expand_all", C.byref(w.s), C.byref(st), C.byref(p))
    for name in ("zx", "zy", "zz") + (("zfx", "zfy", "zfz") if force else ()):
        ref = np.asarray(ex[name]).reshape(-1)
        assert np.linalg.norm(w.get(name).reshape(-1)[:N * P] - ref) <= TOL * np.linalg.norm(ref), name
    np.testing.assert_array_equal(w.get("idx").reshape(-1)[:N], np.asarray(ex["idx"]).reshape(-1))
    H_ref = O.grid_split(po, q, zs, ex, force_order=int(force))
    F.call("SE_FGG_grid_split_AVX_dispatch_force" if force else "SE_FGG_grid_split", C.byref(w.s), C.byref(st),
           C.byref(p))
    assert O.rel_rms(w.get("H"), H_ref) < TOL
    if force:
        out = np.zeros(3 * N)
        F.call("SE_FGG_int_split_AVX_dispatch_force", F.dptr(out), C.byref(st), C.byref(w.s), C.byref(p))
        ref = O.int_split_force(po, q, H_ref, zs, ex)
    else:
        out = np.zeros(N)
        F.call("SE_FGG_int_split", F.dptr(out), C.byref(w.s), C.byref(p))
        ref = O.int_split(po, H_ref, zs, ex)
    assert O.rel_rms(out, ref) < TOL


# the expansion in the scatter: a particle per CTA up to 64 P
@pytest.mark.parametrize("N,M,P", [(1, 9, 1), (64, 9, 1), (65, 9, 1), (512, 24, 8), (513, 24, 8), (1024, 33, 16),
                                   (1025, 33, 16), (40, 40, 32)])
def test_vanilla_scatter_equals_split(F, N, M, P):
    import oracle as O
    x, q, p, po, w, st, keep = setup(F, N, M, P, 0, False)
    F.call("SE_FGG_grid", C.byref(w.s), C.byref(st), C.byref(p))
    H_ref = O.grid_split(po, q, O.base_gaussian(po), O.expand_all(po, x, 3, False))
    assert O.rel_rms(w.get("H"), H_ref) < TOL


def test_windows_skip_stencils_outside(F):
    """Stencils that leave the padded grid are skipped by the windows and reported."""
    import oracle as O
    import torch
    from se_fast_gridding_b200._lib import SEError
    N, M, P = 24_500, 32, 16
    x, q, p, po, w, st, keep = setup(F, N, M, P, 0, False)
    F.call("SE_FGG_expand_all", C.byref(w.s), C.byref(st), C.byref(p))
    bad = [0, 17, N - 1]
    w.arrays["idx"][bad] = torch.tensor([-1, 2 ** 30, p.npdims[0] * p.npdims[1] * p.npdims[2] - 1],
                                        dtype=torch.int32, device="cuda")
    with pytest.raises(SEError):
        F.call("SE_FGG_grid_split", C.byref(w.s), C.byref(st), C.byref(p))
    used = np.ones(N)
    used[bad] = 0.0
    H_ref = O.grid_split(po, q * used, O.base_gaussian(po), O.expand_all(po, x, 3, False))
    assert O.rel_rms(w.get("H"), H_ref) < TOL
