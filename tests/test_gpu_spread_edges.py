"""The general spread (k_spread2 on P-wide rows) where blocks have no candidates and
groups are short, on odd and even grids that end inside a tile: the oracle's grid for
a few particles, the other cells zero over what was there before, and the fold of
many parts.  Bound: FP64 1e-12 of the grid's norm, as for every solve; FP32 2e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,P,clusters", [(1, 50, 6, 0), (3, 51, 12, 0), (5, 65, 20, 0), (17, 94, 9, 0), (20, 49, 32, 0),
                                            (33, 36, 4, 0), (90_000, 32, 3, 2), (90_000, 49, 5, 2),
                                            (20_000, 32, 20, 1)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_sparse_and_split_blocks(N, M, P, clusters, prec):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle as O
    from se_fast_gridding_b200 import solver as S
    L, xi = 1.3, 0.15 * M
    x, q = O.synthetic_system(N, L, seed=M + P, charges="uniform", clusters=clusters, sigma=0.004)
    q += 0.5
    p = O.Setup(M=M, P=P, L=L, xi=xi, m=S.default_m(P), N=N).params()
    ref = O.wrap(p, O.grid_split(p, q, O.base_gaussian(p), O.expand_all(p, x, 3, False)), 3)
    ref = ref.reshape(M, M, M).transpose(2, 1, 0)
    se = S.SpectralEwald(M, P, L, xi, precision=prec, max_particles=N)
    grid = torch.full((M, M, M), float("nan"), dtype=torch.float64, device="cuda")
    se.spread(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda"), grid)
    got = grid.cpu().numpy()
    assert np.linalg.norm(got - ref) < {"fp64": 1e-12, "fp32": 2e-6}[prec] * np.linalg.norm(ref)
    if N < 100:
        assert not got[ref == 0.0].any()
    se.close()
