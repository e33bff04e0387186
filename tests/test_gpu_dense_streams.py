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


def test_gradients_keep_no_memory():
    """A pass over a graph leaves nothing behind once the graph is gone."""
    from inching_b200 import synth
    from inching_b200.learned import BeadGraph, WarmStartMPNN
    model = WarmStartMPNN(seed=1)
    held = []
    for atoms in (800, 1400, 2000):
        G = BeadGraph(torch.from_numpy(synth.globule(atoms, seed=2) / 10.0).cuda())
        gamma, c = model.forward(G)
        model.backward(G, c, torch.ones_like(gamma))
        del G, gamma, c
        held.append(torch.cuda.memory_allocated())
    assert held[0] == held[1] == held[2]
