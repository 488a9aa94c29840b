"""Slab memory of the spread's split tiles on grids not cut into whole tiles.

CPU: a plan's bytes, which count what the tiles the grid has may need -- not more
than 8 tiles of 64 further parts at M = 32, P = 21, which is 16.8 MB of slabs --
and never shrink as the capacity grows.

GPU: every particle in one cell, the most parts a tile can have, on a plan of larger
capacity that holds fewer particles in smaller parts, against the oracle's grid
(FP64, 1e-12 of its norm as for every solve)."""
import ctypes as C

import numpy as np
import pytest


def plan_bytes(M, P, N):
    import se_fast_gridding_b200 as pkg
    from se_fast_gridding_b200 import _lib
    cfg = _lib.se_config(M=M, P=P, L=1.0, xi=0.15 * M, m=6.66, mode=1, precision=0, max_particles=N)
    return pkg.lib().se_plan_device_bytes(C.byref(cfg))


@pytest.mark.parametrize("M,P,N,parts", [(32, 21, 60_000, 8 * 64), (32, 21, 1_100, 8 * 2), (32, 21, 600_000, 8 * 64),
                                         (40, 32, 5_000, 27 * 9), (47, 32, 40_000, 27 * 64),
                                         # a bin's particles in at most 3 tiles an axis
                                         (250, 12, 2_000_000, 27 * 2_000_000 // 8192), (36, 12, 20_000, 27 * 2)])
def test_slabs_of_the_tiles_there_are(M, P, N, parts):
    tiles = (M + 15) // 16
    particles = 300 + 24 * P   # bytes a particle: inputs, output, records, sort, factors
    grids = 8 * M ** 3 + 4 * 8 * M * M * (M // 2 + 1)
    others = 2 * 8 * tiles ** 3 + 8 * 1024 * ((M + 7) // 8) ** 3   # tables; the sort's bins
    assert plan_bytes(M, P, N) <= particles * N + grids + others + 32768 * (parts + 1) + 65536


@pytest.mark.parametrize("M,P,least", [(32, 21, 512), (47, 32, 512), (36, 12, 8192), (250, 20, 8192)])
def test_bytes_grow_with_the_capacity(M, P, least):
    sizes = sorted({max(1, k * least + d) for k in (1, 2, 3, 63, 64, 65, 511, 512, 513, 600) for d in (-1, 0, 1, 2)} |
                   {1023, 1024, 1025})
    b = [plan_bytes(M, P, n) for n in sizes]
    assert all(x <= y for x, y in zip(b, b[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("M,P", [(32, 21), (27, 20), (47, 32), (36, 12), (64, 18)])
def test_one_crowded_cell(M, P):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle as O
    from se_fast_gridding_b200 import solver as S
    cap, xi = 40_000, 0.15 * M
    se = S.SpectralEwald(M, P, 1.0, xi, precision="fp64", max_particles=cap)
    rng = np.random.default_rng(M)
    for n in (cap, 32_831, 8_193, 1_025, 1_024):
        x = (rng.random(3 * n) * 0.9 + 0.05 + M // 2) / M
        q = rng.standard_normal(n)
        p = O.Setup(M=M, P=P, L=1.0, xi=xi, m=S.default_m(P), N=n).params()
        ref = O.wrap(p, O.grid_split(p, q, O.base_gaussian(p), O.expand_all(p, x, 3, False)), 3)
        ref = ref.reshape(M, M, M).transpose(2, 1, 0)
        grid = se.spread(torch.tensor(x, device="cuda"), torch.tensor(q, device="cuda")).cpu().numpy()
        assert np.linalg.norm(grid - ref) < 1e-12 * np.linalg.norm(ref), n
    se.close()
