"""Sizes that the launchers refuse on the host, before anything reaches a device (the pointers are never followed)."""
import pytest

from onnxruntime_genai_b200.ops import _lib

A, W, C, LIST = 1 << 20, 2 << 20, 3 << 20, 4 << 20


@pytest.mark.parametrize("half", [0, 16])
@pytest.mark.parametrize("tile", [-32, 0, 8, 17, 31, 33, 40, 48, 96, 255, 257, 288, 512])
def test_packed_experts_refuse_token_tiles_without_a_kernel(tile, half):
    assert _lib.lib().ogb_moe_gemm_fp4(A, 128, W, C, 256, 64, 256, 128, 4, None, half, 0, 0.0, 0.0, LIST, LIST, LIST, LIST, 8, tile, 64, None, None, None) == -5


@pytest.mark.parametrize("requests,Hv,dk,dv,longest,blocks", [
    (1, 16, 128, 128, 1, False), (1, 16, 128, 128, 5, False), (1, 16, 128, 128, 6, True), (1, 16, 128, 128, 0, True), (8, 16, 128, 128, 8, False),
    (8, 16, 128, 128, 9, True), (1, 8, 64, 64, 4, False), (1, 8, 64, 64, 5, True), (32, 8, 64, 64, 8, False), (1, 4, 257, 64, 3000, False), (1, 4, 256, 64, 3000, True)])
def test_short_portions_of_the_delta_rule_are_walked(requests, Hv, dk, dv, longest, blocks):
    assert (_lib.lib().ogb_gated_delta_scratch_bytes(requests * max(1, longest), requests, Hv // 2, Hv, dk, dv, longest) > 0) == blocks


@pytest.mark.parametrize("M,N,K,splits", [(129, 512, 14336, 8), (512, 512, 14336, 8), (300, 128, 8192, 8), (200, 896, 4864, 8), (257, 896, 4864, 8), (200, 2048, 8192, 4),
                                          (257, 1024, 14336, 4), (64, 4096, 4096, 4)])
def test_long_sums_of_few_tiles_are_cut_in_eight(M, N, K, splits):
    """Of 256-token tiles, as many clusters of eight CTAs as are resident at once."""
    assert _lib.lib().ogb_gemm_auto_splits(M, N, K, 0, 148) == splits


def test_rotation_of_heads_without_columns_does_nothing():
    """A head size of 0 has nothing to rotate or to append: the call returns (where there is no device, with the launch's error)."""
    assert _lib.lib().ogb_rope_kv_append_bits(A, 8, None, None, None, None, None, None, None, None, 1e-6, 1, 2, 1, 0, 0, 0, 1, 16, None, 0, 0, None) in (0, -4)
