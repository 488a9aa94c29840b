"""The cell-list real-space kernel (a warp per target, pairs queued 32 at a
time) against the oracle at its edges: a lone particle, fewer and more than 32
pairs, the fewest cells (3 per axis, every neighbour a wrapped one), many
sparse cells, and a box of one crowded cell; potential alone and with force.

Tolerance: FP64 sums of at most a few thousand pairs in another order, 1e-12
relative as for the other real-space tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("N,L,xi,rc,clusters", [(1, 1.0, 9.0, 0.3, 0), (2, 2.0, 4.0, 0.66, 0), (33, 1.0, 9.0, 0.33, 0),
                                                (700, 1.0, 9.0, 0.33, 0), (900, 1.0, 40.0, 0.06, 0),
                                                (1500, 3.0, 3.0, 0.75, 1)])
@pytest.mark.parametrize("force", [False, True])
def test_cell_list_edges(N, L, xi, rc, clusters, force):
    import oracle as O
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import solver
    x, q = O.synthetic_system(N, L, seed=N, charges="uniform", clusters=clusters, sigma=0.02)
    if N == 1:
        q[:] = 1.0
    for layers in (0, 1):
        phi, f = solver.real_space(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda"), L, xi, layers, rc,
                                   want_force=force)
        assert O.rel_rms(phi.cpu().numpy(), O.direct_real(x, q, L, xi, layers, rc)) < TOL
        if force:
            assert O.rel_rms(f.cpu().numpy(), O.direct_real_force(x, q, L, xi, layers, rc)) < TOL
