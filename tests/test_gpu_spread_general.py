"""The spread of grids not cut into whole tiles, or with P > 16 (k_spread2 on the
P-wide factor rows) against the oracle's grid: last tiles of 1 to 15 cells, last bins of
1 to 7, odd and even rows, every class of stencil width from 1 to 32, grids on which
a tile meets a stencil in two pieces (M < P + 15) down to the smallest (M = P + 7)
and the one below it (which k_spread serves), tiles
crowded enough to be split into parts.  Bounds: FP64 1e-12 of the grid's norm, as
for every solve; FP32 2e-6, a few times the sums' 24-bit rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 2e-6}


@pytest.mark.parametrize("N,M,P,clusters", [(1, 16, 1, 0), (50, 17, 2, 0), (300, 22, 7, 0), (300, 23, 8, 0),
                                            (400, 31, 16, 0), (400, 30, 16, 0), (500, 33, 16, 0), (700, 47, 32, 0),
                                            (700, 46, 32, 0), (900, 48, 24, 0), (600, 49, 17, 0), (800, 57, 12, 0),
                                            (100, 8, 1, 0), (200, 19, 12, 0), (200, 18, 12, 0),
                                            (300, 27, 20, 0), (9000, 32, 21, 1), (5000, 32, 20, 0), (1024, 31, 16, 0),
                                            (1025, 31, 16, 0), (500, 39, 32, 0),
                                            (400, 38, 32, 0), (20000, 41, 4, 0), (30000, 65, 10, 1), (30000, 50, 9, 1),
                                            (30000, 64, 18, 1)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_general_spread_equals_oracle(N, M, P, clusters, prec):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle as O
    from se_fast_gridding_b200 import solver as S
    L, xi = 1.3, 0.15 * M
    x, q = O.synthetic_system(N, L, seed=M + P, charges="uniform", clusters=clusters, sigma=0.003)
    if N == 1:
        q[:] = 1.0
    setup = O.Setup(M=M, P=P, L=L, xi=xi, m=S.default_m(P), N=N)
    p = setup.params()
    ref = O.wrap(p, O.grid_split(p, q, O.base_gaussian(p), O.expand_all(p, x, 3, False)), 3)
    ref = ref.reshape(M, M, M).transpose(2, 1, 0)
    se = S.SpectralEwald(M, P, L, xi, precision=prec, max_particles=N)
    grid = se.spread(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")).cpu().numpy()
    assert np.linalg.norm(grid - ref) < TOL[prec] * np.linalg.norm(ref)
    se.close()
