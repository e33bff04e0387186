"""Workspace of the dense-layer products: what a split or a skinny product leaves in it,
and no more than the smallest one where K is too short for either."""
import pytest

from inching_b200 import _native

SMALLEST = 256


@pytest.mark.parametrize("M,N,K", [(5_000_000, 8, 100), (300_000, 1, 132), (1, 300_000, 2048), (8, 8, 1),
                                   (132, 128, 2048), (2_000_000_000, 1, 4)])
def test_short_products_ask_for_nothing(M, N, K):
    assert _native.lib().inch_mp_gemm_workspace_size(M, N, K) == SMALLEST


@pytest.mark.parametrize("M,N,K", [(1, 128, 2049), (5_000_000, 8, 2049), (8, 5_000_000, 4096), (136, 64, 300_000)])
def test_long_products_have_room_for_their_parts(M, N, K):
    assert _native.lib().inch_mp_gemm_workspace_size(M, N, K) >= 4 * M * N
