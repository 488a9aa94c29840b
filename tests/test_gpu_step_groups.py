"""The reference step calls on particles grouped by bin (from 1.6e7 stencil cells
on): the scatter through shared-memory windows and the gathers in grouped
order against the oracle, at the edges of their dispatch: stencils with and
without a compiled-in P, the largest window, one more than it, a bin of more
particles than one CTA takes, and particles whose stencil leaves the grid.

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


@pytest.mark.parametrize("N,M,P,clusters", [(3906, 32, 16, 0), (3907, 32, 16, 0), (31_251, 20, 8, 0),
                                            (9300, 24, 12, 2), (7300, 27, 13, 0), (1800, 16, 21, 0),
                                            (1600, 18, 22, 1), (600_000, 33, 3, 0), (500, 16, 32, 0)])
@pytest.mark.parametrize("force", [False, True])
def test_grouped_steps_equal_oracle(F, N, M, P, clusters, force):
    import oracle as O
    import torch
    x, q = O.synthetic_system(N, 1.0, seed=N + P, charges="uniform", clusters=clusters, sigma=0.01)
    m = 0.95 * np.sqrt(O.PI * P)
    _, p = F.fcn_params(M, P, 1.0, 4.0, m, N)
    po = O.Setup(M=M, P=P, L=1.0, xi=4.0, m=m, N=N).params()
    zs = O.base_gaussian(po)
    ex = O.expand_all(po, x, 3, force)
    H_ref = O.grid_split(po, q, zs, ex, force_order=int(force))
    w = F.Work(p, force=force, where="cuda")
    xc, qc = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
    st = F.state(xc, qc)
    F.call("SE_FGG_base_gaussian", C.byref(w.s), C.byref(p))
    F.call("SE_FGG_expand_all_SSE_force" if force else "SE_FGG_expand_all", C.byref(w.s), C.byref(st), C.byref(p))
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


def test_grouped_scatter_skips_stencils_outside(F):
    """Stencils that leave the padded grid are skipped and reported, the rest
    is summed, as for a few particles."""
    import oracle as O
    import torch
    from se_fast_gridding_b200._lib import SEError
    N, M, P = 9400, 24, 12
    x, q = O.synthetic_system(N, 1.0, seed=3, charges="uniform")
    m = 0.95 * np.sqrt(O.PI * P)
    _, p = F.fcn_params(M, P, 1.0, 4.0, m, N)
    w = F.Work(p, where="cuda")
    xc, qc = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
    st = F.state(xc, qc)
    F.call("SE_FGG_base_gaussian", C.byref(w.s), C.byref(p))
    F.call("SE_FGG_expand_all", C.byref(w.s), C.byref(st), C.byref(p))
    bad = [0, 17, N - 1]
    w.arrays["idx"][bad] = torch.tensor([-1, 2 ** 30, p.npdims[0] * p.npdims[1] * p.npdims[2] - 1],
                                        dtype=torch.int32, device="cuda")
    with pytest.raises(SEError):
        F.call("SE_FGG_grid_split", C.byref(w.s), C.byref(st), C.byref(p))
    keep = np.ones(N)
    keep[bad] = 0.0
    po = O.Setup(M=M, P=P, L=1.0, xi=4.0, m=m, N=N).params()
    H_ref = O.grid_split(po, q * keep, O.base_gaussian(po), O.expand_all(po, x, 3, False))
    assert O.rel_rms(w.get("H"), H_ref) < TOL
