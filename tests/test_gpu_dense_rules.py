"""Dense-layer products on both sides of the lines between the general kernel and the
register tiles, and through many staged chunks of the 64-row tiles.  Up to K = 2,048 the
kernels sum in the same order, so aligned operands give the bits of the same numbers in
views that start at an odd element (general kernel), and both are within the a-priori
bound K u / (1 - K u) * |A| |B|, u = 2^-24, of the FP64 product."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(256, 128, 1000), (132, 128, 776), (68, 20, 36), (12800, 64, 256), (12736, 64, 256), (12800, 64, 260),
         (36, 12800, 64), (32, 12800, 64), (6400, 128, 24), (6400, 128, 28), (4300, 132, 16), (20000, 20, 1000),
         (20000, 64, 132), (20000, 68, 132)]


def _view(m, transposed, offset):
    s = m.t() if transposed else m
    flat = torch.empty(s.numel() + offset, device="cuda")
    flat[offset:] = s.reshape(-1)
    v = flat[offset:].view(s.shape)
    return v.t() if transposed else v


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_product_at_rule_lines(M, N, K, ta, tb):
    from inching_b200 import _native
    g = torch.Generator(device="cuda")
    g.manual_seed(M + 3 * N + 7 * K)
    A = torch.randn((M, K), generator=g, device="cuda")
    B = torch.randn((K, N), generator=g, device="cuda")
    got = [_native.mp_gemm(_view(A, ta, o), _view(B, tb, o), torch.full((M, N), float("nan"), device="cuda"))
           for o in (0, 1)]
    assert torch.equal(got[0], got[1])
    ku = (K + 2) * 2.0 ** -24
    size = A.double().abs() @ B.double().abs()
    assert bool(((got[0].double() - A.double() @ B.double()).abs() <= ku / (1 - ku) * size).all())
