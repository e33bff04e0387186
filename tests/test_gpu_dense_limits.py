"""Dense-layer products with more output tiles in one direction than a grid's second
dimension holds (65,535).  Small whole numbers make every product exact in FP32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(9, 65536 * 64 + 9, 2), (65536 * 64 + 9, 9, 2), (16, 65536 * 128 + 4, 4)])
def test_more_tiles_than_a_grid_dimension(M, N, K):
    from inching_b200 import _native
    g = torch.Generator(device="cuda")
    g.manual_seed(K)
    A = torch.randint(-8, 9, (M, K), generator=g, device="cuda").float()
    B = torch.randint(-8, 9, (K, N), generator=g, device="cuda").float()
    C = torch.full((M, N), float("nan"), device="cuda")
    _native.mp_gemm(A, B, C)
    ref = A[:, :1] * B[:1]
    for k in range(1, K):
        ref += A[:, k:k + 1] * B[k:k + 1]
    assert torch.equal(C, ref)
