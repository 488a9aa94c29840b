"""A tuned plan gets SE_PATH_RUNTIME_P only where the bit changes the kernels: not where
the matrix interpolation serves every path of the configuration."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,P,mode,prec", [(100, 12, "force", "fp64"), (100, 16, "potential", "fp32"),
                                           (25, 6, "force", "fp64"), (128, 24, "potential", "fp64"),
                                           (40, 21, "force", "fp32")])
def test_no_choice_between_equal_kernels(M, P, mode, prec):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import solver as S
    se = S.SpectralEwald(M, P, 1.0, 0.15 * M, mode=mode, precision=prec, max_particles=3000, path="tune")
    assert se.path == 0
    se.close()


def test_matrix_kernel_paths_have_no_runtime_variant():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from se_fast_gridding_b200 import solver as S
    se = S.SpectralEwald(192, 12, 1.0, 24.0, mode="force", precision="fp64", max_particles=5000, path="tune")
    assert se.path in (0, 1, 2, 3)
    se.close()
