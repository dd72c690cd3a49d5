"""Sizes that the launchers refuse on the host, before anything reaches a device (the pointers are never followed)."""
import pytest

from onnxruntime_genai_b200.ops import _lib

A, W, C, LIST = 1 << 20, 2 << 20, 3 << 20, 4 << 20


@pytest.mark.parametrize("half", [0, 16])
@pytest.mark.parametrize("tile", [-32, 0, 8, 17, 31, 33, 40, 48, 96, 255, 257, 288, 512])
def test_packed_experts_refuse_token_tiles_without_a_kernel(tile, half):
    assert _lib.lib().ogb_moe_gemm_fp4(A, 128, W, C, 256, 64, 256, 128, 4, None, half, 0, 0.0, 0.0, LIST, LIST, LIST, LIST, 8, tile, 64, None, None, None) == -5


@pytest.mark.parametrize("M,N,K,splits", [(129, 512, 14336, 8), (512, 512, 14336, 8), (300, 128, 8192, 8), (200, 896, 4864, 8), (257, 896, 4864, 8), (200, 2048, 8192, 4),
                                          (257, 1024, 14336, 4), (64, 4096, 4096, 4)])
def test_long_sums_of_few_tiles_are_cut_in_eight(M, N, K, splits):
    """Of 256-token tiles, as many clusters of eight CTAs as are resident at once."""
    assert _lib.lib().ogb_gemm_auto_splits(M, N, K, 0, 148) == splits
