"""Tile widths of the prompt projections (q_gemm_prompt_columns) against measured times."""
import pytest

# (residual, M, N, K, us with 256 columns, us with 160), B200 of 148 SMs, weights rotated through more than L2
MEASURED = [
    (1, 257, 2560, 4096, 26.3, 20.3), (1, 1024, 2560, 4096, 27.8, 21.4), (1, 1280, 2560, 4096, 27.8, 34.7),
    (1, 2048, 2560, 4096, 49.6, 40.3), (1, 2816, 2560, 4096, 51.3, 57.1), (1, 8192, 2560, 4096, 142.6, 154.2),
    (1, 600, 2560, 9728, 45.4, 42.2), (1, 1024, 2560, 9728, 54.7, 45.4), (1, 1500, 2560, 9728, 62.2, 85.4),
    (1, 1900, 2560, 9728, 96.1, 100.3), (1, 2048, 2560, 9728, 95.9, 99.1), (1, 2304, 2560, 9728, 112.0, 105.4),
    (1, 3500, 4096, 4096, 101.7, 109.4),
    (0, 600, 2560, 9728, 39.9, 44.1), (0, 1024, 2560, 9728, 51.1, 47.6), (0, 2048, 2560, 9728, 88.0, 101.2),
    (0, 850, 5120, 8704, 72.7, 83.8), (0, 384, 4096, 6144, 39.4, 33.4), (0, 1100, 4096, 6144, 55.7, 62.6),
    (0, 1280, 4096, 6144, 56.3, 62.4), (0, 2816, 4096, 6144, 125.5, 133.3), (0, 4608, 2560, 2048, 40.9, 42.8),
]


@pytest.mark.parametrize("residual,M,N,K,wide,narrow", MEASURED)
def test_the_faster_width(residual, M, N, K, wide, narrow):
    from starter_b200._lib import lib
    assert lib.q_gemm_prompt_columns(M, N, K, residual) == (256 if wide < narrow else 160)


@pytest.mark.parametrize("M,N,K", [(1, 32, 32), (128, 128, 64), (129, 160, 96), (256, 256, 512), (257, 2560, 416), (700, 96, 4096),
                                   (1000, 2560, 9728), (2048, 2560, 9728), (3800, 2560, 8192), (2103, 2560, 4096),
                                   (2305, 4896, 160), (2100, 2592, 96), (130, 576, 9728), (5000, 672, 160)])
def test_both_epilogues_alike(M, N, K):
    """Shapes at which tests/test_prompt_gemm_gpu.py compares the two forms bit for bit: the same tiles."""
    from starter_b200._lib import lib
    assert lib.q_gemm_prompt_columns(M, N, K, 0) == lib.q_gemm_prompt_columns(M, N, K, 1)


def test_refused_shapes():
    from starter_b200._lib import lib
    for M, N, K in ((0, 64, 64), (4, 48, 64), (4, 64, 80), (4, 0, 64)):
        assert lib.q_gemm_prompt_columns(M, N, K, 1) == 0
