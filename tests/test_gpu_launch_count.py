"""The launch counter against the kernels that a profiler sees, on every route of the two
calls that choose their kernels from the inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _seen(call):
    """(counted, the package's own kernels by the profiler) of one call."""
    from torch.profiler import ProfilerActivity, profile
    from inching_b200 import _native
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        before = _native.launches
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return _native.launches - before, sum("k_" in n and "cub" not in n for n in names)


# one column, general kernel, register tiles, split tiles, skinny, whole tiles and a rest,
# two launches of the general kernel
@pytest.mark.parametrize("M,N,K,ta,want", [(500, 1, 100, False, 1), (9, 9, 9, False, 1), (256, 128, 128, False, 1),
                                           (256, 128, 4096, False, 2), (4, 128, 4096, False, 2),
                                           (132, 128, 4096, True, 4), (65536 * 64 + 9, 2, 1, False, 2)])
def test_products(M, N, K, ta, want):
    from inching_b200 import _native
    A = torch.ones((K, M), device="cuda").t() if ta else torch.ones((M, K), device="cuda")
    B, C = torch.ones((K, N), device="cuda"), torch.empty((M, N), device="cuda")
    assert _seen(lambda: _native.mp_gemm(A, B, C)) == (want, want)


@pytest.mark.parametrize("kind,scans", [("one", 1), ("two", 2), ("directed", 1)])
def test_orders(kind, scans):
    from inching_b200 import _native
    n = 50
    a = np.arange(n - 1)
    if kind == "two":
        a = a[a != 20]
    e = np.stack([a, a + 1], 1)
    if kind != "directed":
        e = np.concatenate([e, e[:, ::-1]])
    e = np.concatenate([e, np.stack([np.arange(n)] * 2, 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int64)
    degree = np.diff(rowptr).astype(np.int32)
    seeds = np.argsort(degree)[::-1].astype(np.int64)
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (rowptr, e[:, 1].astype(np.int32), degree, seeds)]
    counted, own = _seen(lambda: _native.cuthill_mckee(*d))
    assert counted == own + scans
