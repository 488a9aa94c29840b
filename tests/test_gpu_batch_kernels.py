"""Batches whose systems are served by different interpolation and spread kernels:
each system's result is its single solve's bit for bit, and the interpolation takes
one launch per kernel and stencil."""
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


# Pairs of systems of one stencil and mode on both sides of the choice of the
# interpolation kernel, with bins of more than 256 particles (which further CTAs
# take), the crowded one served by the other kernel; then a general and a
# whole-tile system whose crowded tiles are split into parts.
@pytest.mark.parametrize("systems", [
    [(20, 192, 12, "force", 0), (3000, 128, 12, "force", 2)],
    [(3000, 192, 12, "force", 2), (3000, 128, 12, "force", 2)],
    [(20, 128, 16, "potential", 0), (3000, 64, 16, "potential", 2)],
    [(20, 100, 8, "force", 0), (3000, 36, 8, "force", 2)],
    [(3000, 100, 8, "potential", 1), (3000, 36, 8, "potential", 2)],
    [(20000, 50, 12, "force", 1), (20000, 64, 12, "force", 1), (20000, 32, 21, "force", 1)],
], ids=str)
def test_crowded_bins_of_another_kernel(env, systems):
    import oracle as O
    torch, S = env
    L = 1.3
    sy = [S.System(N, M, P, L, 0.15 * M, None, mode) for N, M, P, mode, _ in systems]
    xs, qs = zip(*[O.synthetic_system(N, L, seed=M + k, charges="uniform", clusters=c, sigma=0.004)
                   for k, (N, M, P, mode, c) in enumerate(systems)])
    b = S.BatchSolver(sy, "fp64")
    x, q = b.pack(xs, qs)
    outs = [o.cpu().numpy() for o in b.split(b.solve(x, q))]
    b.close()
    for (N, M, P, mode, _), xi, qi, out in zip(systems, xs, qs, outs):
        se = S.SpectralEwald(M, P, L, 0.15 * M, mode=mode, precision="fp64", max_particles=N)
        one = se.solve(torch.tensor(xi, device="cuda"), torch.tensor(qi, device="cuda")).cpu().numpy()
        se.close()
        np.testing.assert_array_equal(out, one)


def test_mixed_modes_take_no_more_launches(env):
    """k_interp2 serves potentials and forces of one stencil in one launch."""
    import oracle as O
    torch, S = env
    count = {}
    for modes in (("force", "force"), ("potential", "force")):
        sy = [S.System(500, 64, P, 1.0, 8.0, None, mode) for P in (8, 12, 16) for mode in modes]
        b = S.BatchSolver(sy, "fp32")
        x, q = b.pack(*zip(*[O.synthetic_system(s.N, 1.0, seed=k) for k, s in enumerate(sy)]))
        b.solve(x, q)
        torch.cuda.synchronize()
        count[modes] = b.launches
        b.close()
    assert len(set(count.values())) == 1, count
