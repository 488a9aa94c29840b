"""The ways k_interp3's work is cut -- groups shared by a CTA's warps, chunks of 32 and
of 256 particles, a CTA per particle where bins are more than particles -- give
a particle the same sums: bit for bit on a grid of the caller's, whatever other
particles there are, and the oracle's solve at the sizes where they change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import solver
    return torch, solver


# bins: 1 to 4,913, two classes of rows (whole tiles: M = 128, P <= 16), odd and even M
@pytest.mark.parametrize("M,P", [(8, 3), (18, 32), (33, 21), (50, 12), (67, 9), (128, 16), (130, 20)])
@pytest.mark.parametrize("mode", ["potential", "force"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_sums_do_not_depend_on_the_cut(env, M, P, mode, prec):
    torch, S = env
    N = 60_000
    g = torch.Generator("cuda").manual_seed(M)
    x = torch.rand(3, N, dtype=torch.float64, device="cuda", generator=g)
    x[:, ::3] = x[:, ::3] * 0.02 + 0.4   # a third of them crowded
    q = torch.rand(N, dtype=torch.float64, device="cuda", generator=g)
    grid = torch.rand(M, M, M, dtype=torch.float64, device="cuda", generator=g)
    se = S.SpectralEwald(M, P, 1.0, 0.15 * M, mode=mode, precision=prec, max_particles=N)
    w = se.out_width
    ref = se.interp(x.reshape(-1).contiguous(), q, grid).view(w, N)
    for n in (1, 7, 9, 300, 1_100, 4_800, 9_000, 40_000, 40_001):
        out = se.interp(x[:, :n].reshape(-1).contiguous(), q[:n].contiguous(), grid).view(w, n)
        assert torch.equal(out, ref[:, :n]), n
    se.close()


@pytest.mark.parametrize("N,M,P,clusters", [(1066, 19, 32, 0), (1200, 40, 21, 0), (343, 55, 20, 0), (342, 55, 20, 0),
                                            (7000, 75, 24, 3), (40_000, 36, 12, 2), (40_001, 36, 12, 2)])
@pytest.mark.parametrize("mode", ["potential", "force"])
def test_cuts_equal_oracle(env, N, M, P, clusters, mode):
    import oracle as O
    torch, S = env
    L, xi = 1.3, 0.15 * M
    x, q = O.synthetic_system(N, L, seed=M + P, charges="uniform", clusters=clusters, sigma=0.01)
    ref = O.spectral_ewald(x, q, M, P, S.default_m(P), L, xi, mode)
    se = S.SpectralEwald(M, P, L, xi, mode=mode, precision="fp64", max_particles=N)
    out = se.solve(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda"))
    assert O.rel_rms(out.cpu().numpy(), ref) < 1e-12
    se.close()
