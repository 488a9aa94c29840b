"""The interpolation on FP64 matrix instructions (k_interp3) against the
oracle's solve at its edges: every depth of the contraction from P = 1 to 32,
grids smaller than a stencil, odd grids (single-cell loads) and even ones,
whole tiles and others, bins of one particle, of more than one CTA takes, and
launches of few and many bins.  FP64: 1e-12 relative as for every solve.

A grid that holds an infinity: the particles whose own stencil misses it are
finite, as the stencil sum is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import solver
    return torch, solver


@pytest.mark.parametrize("N,M,P,clusters", [(1, 8, 1, 0), (40, 2, 4, 0), (60, 7, 9, 0), (300, 12, 17, 0),
                                            (300, 15, 13, 0), (500, 32, 16, 0), (900, 32, 8, 1), (2000, 48, 12, 1),
                                            (700, 24, 21, 0), (400, 25, 22, 0), (300, 36, 26, 0), (200, 10, 32, 0),
                                            (3000, 80, 6, 0), (2500, 75, 10, 0),
                                            (5000, 128, 16, 1), (3000, 128, 9, 0)])
@pytest.mark.parametrize("mode", ["potential", "force"])
def test_interp3_equals_oracle(env, N, M, P, clusters, mode):
    import oracle as O
    torch, S = env
    L, xi = 1.3, 0.15 * M
    x, q = O.synthetic_system(N, L, seed=M + P, charges="uniform", clusters=clusters, sigma=0.01)
    if N == 1:
        q[:] = 1.0
    ref = O.spectral_ewald(x, q, M, P, S.default_m(P), L, xi, mode)
    se = S.SpectralEwald(M, P, L, xi, mode=mode, precision="fp64", max_particles=N)
    out = se.solve(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda"))
    assert O.rel_rms(out.cpu().numpy(), ref) < TOL
    se.close()


@pytest.mark.parametrize("M,P", [(128, 16), (36, 12), (27, 15)])
def test_interp3_infinite_cell(env, M, P):
    torch, S = env
    N = 4000
    g = torch.Generator("cuda").manual_seed(5)
    x = torch.rand(3 * N, dtype=torch.float64, device="cuda", generator=g)
    q = torch.rand(N, dtype=torch.float64, device="cuda", generator=g)
    grid = torch.rand(M, M, M, dtype=torch.float64, device="cuda", generator=g)
    se = S.SpectralEwald(M, P, 1.0, 0.15 * M, mode="force", precision="fp64", max_particles=N)
    clean, phi = se.interp(x, q, grid), torch.empty(N, dtype=torch.float64, device="cuda")
    cell = (3, M // 2, M - 2)
    grid[cell] = float("inf")
    out = se.interp(x, q, grid, phi_out=phi)
    cells = torch.floor(x.view(3, N) * M + (0.5 if P % 2 else 0.0)).long() - (P - 1) // 2
    hit = torch.ones(N, dtype=torch.bool, device="cuda")
    for a in range(3):
        hit &= torch.remainder(cell[a] - cells[a], M) < P
    assert 0 < int(hit.sum()) < N
    assert torch.isfinite(out.view(3, N)[:, ~hit]).all() and torch.isfinite(phi[~hit]).all()
    assert torch.isinf(phi[hit]).all()
    a, b = out.view(3, N)[:, ~hit], clean.view(3, N)[:, ~hit]
    assert float((a - b).norm() / b.norm()) < TOL
    se.close()
