"""Dense-layer products and gradients that share nothing between streams or calls."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

# split products through the skinny kernel, the register tiles and the general kernel
SIZES = [(4, 128, 30000), (132, 128, 30000), (33, 65, 9001)]


def test_split_products_on_two_streams():
    """Two host threads, a stream each, products of the same sizes and other numbers: the
    bits of the same products one after the other."""
    from inching_b200 import _native
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ops = [[(torch.randn((M, K), generator=g, device="cuda"), torch.randn((K, N), generator=g, device="cuda"))
            for M, N, K in SIZES * 8] for _ in range(2)]

    def products(pairs):
        return [_native.mp_gemm(A, B, torch.empty((A.shape[0], B.shape[1]), device="cuda")) for A, B in pairs]

    ref = [products(p) for p in ops]
    torch.cuda.synchronize()
    got = [None, None]

    def work(k):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            got[k] = products(ops[k])
        s.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(ref, got):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_products_keep_no_memory():
    from inching_b200 import _native
    A, B = torch.randn((100, 50001), device="cuda"), torch.randn((50001, 70), device="cuda")
    C = torch.empty((100, 70), device="cuda")
    before = torch.cuda.memory_allocated()
    _native.mp_gemm(A, B, C)
    assert torch.cuda.memory_allocated() == before
