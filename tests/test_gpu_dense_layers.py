"""Dense-layer kernels at the sizes where the call changes its tile, its split or its
kernel: one less and one more than a tile, a K that is no multiple of the staged depth,
1 to 8 rows or columns over a long K, rows left over beyond whole tiles.

An unsplit product sums every output in the order of K with one rounding a term,
whichever kernel runs: aligned operands (register tiles) give the bits of the same
numbers in views that start at an odd element (general strides).  A split product (K
above 2048) is within the a-priori bound of a length-K dot product in any order,
K u / (1 - K u) * |A| |B| with u = 2^-24, of the FP64 product."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(127, 128, 132), (129, 132, 17), (40000, 128, 132), (19000, 132, 128), (132, 128, 5000), (136, 64, 2052),
         (1, 128, 2100), (8, 33, 4100), (9, 20, 4100), (5000, 1, 132), (300, 1, 37), (132, 1, 3000), (64, 7, 2500),
         (16, 16, 4)]


def _view(m, transposed, offset):
    """The matrix m in memory as itself or as the transpose of a row-major one, starting
    `offset` elements after an allocation's start."""
    s = m.t() if transposed else m
    flat = torch.empty(s.numel() + offset, device="cuda")
    flat[offset:] = s.reshape(-1)
    v = flat[offset:].view(s.shape)
    return v.t() if transposed else v


@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", SIZES)
def test_product_at_tile_edges(M, N, K, ta, tb):
    from inching_b200 import _native
    g = torch.Generator(device="cuda")
    g.manual_seed(M + 3 * N + 7 * K)
    A = torch.randn((M, K), generator=g, device="cuda")
    B = torch.randn((K, N), generator=g, device="cuda")
    C0 = torch.randn((M, N), generator=g, device="cuda")
    got = []
    for offset in (0, 1):
        C, D = torch.full_like(C0, float("nan")), C0.clone()
        _native.mp_gemm(_view(A, ta, offset), _view(B, tb, offset), C)
        _native.mp_gemm(_view(A, ta, offset), _view(B, tb, offset), D, beta=1.0)
        got.append((C, D))
    if K <= 2048:
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    ku = (K + 2) * 2.0 ** -24
    size = A.double().abs() @ B.double().abs()
    for C, D in got:
        ref = A.double() @ B.double()
        assert bool(((C.double() - ref).abs() <= ku / (1 - ku) * size).all())
        assert bool(((D.double() - ref - C0.double()).abs() <= ku / (1 - ku) * (size + C0.double().abs())).all())
