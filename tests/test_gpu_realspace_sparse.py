"""The cell-list real-space sum with a thread per target (262,144 particles and more of
few neighbours each): the same as a warp per target, which serves one particle fewer
and is held to the oracle, on sparse and crowded cells, and close to a direct sum in
plain torch for some targets.

Tolerance: FP64 sums of at most a few thousand pairs in another order, 1e-12
relative as for the other real-space tests.  The direct sum takes the separations
from positions that are not wrapped into the box, 4e-16 apart where the closest of
the targets' pairs are above 1e-6: 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12
N = 1 << 18


@pytest.mark.parametrize("rc,clusters,sigma", [(0.0045, 0, 0), (0.009, 0, 0), (0.012, 0, 0), (0.016, 0, 0), (0.027, 0, 0),
                                               (0.007, 8, 0.05), (0.004, 3, 0.01)])
@pytest.mark.parametrize("force", [False, True])
def test_thread_equals_warp_per_target(rc, clusters, sigma, force):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle as O
    from se_fast_gridding_b200 import solver
    L, xi, layers = 1.0, 2.5 / rc, 1
    x, q = O.synthetic_system(N, L, seed=4, charges="uniform", clusters=clusters, sigma=sigma)
    x += np.random.default_rng(1).integers(-1, 2, 3 * N)   # positions outside the box too
    q[-1] = 0.0
    xd, qd = torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")
    x1 = xd.view(3, N)[:, :-1].reshape(-1).contiguous()
    phi, f = solver.real_space(xd, qd, L, xi, layers, rc, want_force=force)
    phi1, f1 = solver.real_space(x1, qd[:-1].contiguous(), L, xi, layers, rc, want_force=force)
    assert float((phi[:-1] - phi1).norm() / phi1.norm()) < TOL
    if force:
        g, g1 = f.view(3, N)[:, :-1], f1.view(3, N - 1)
        assert float((g - g1).norm() / g1.norm()) < TOL
    t = torch.arange(0, N, N // 60, device="cuda")
    w = xd.view(3, N)
    ref = torch.zeros(len(t), dtype=torch.float64, device="cuda")
    for p0 in (-1, 0, 1):
        for p1 in (-1, 0, 1):
            for p2 in (-1, 0, 1):
                d = [w[a][t][:, None] - w[a][None, :] + p * L for a, p in enumerate((p0, p1, p2))]
                r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
                r2[torch.arange(len(t)), t] = torch.where(torch.tensor(p0 == p1 == p2 == 0, device="cuda"),
                                                          4 * L * L, r2[torch.arange(len(t)), t])
                r = r2.sqrt()
                ref += torch.where(r2 <= rc * rc, qd[None, :] * torch.erfc(xi * r) / r, 0.0).sum(1)
    assert float((phi[t] - ref).norm()) <= 1e-9 * float(ref.norm())
