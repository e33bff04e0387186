"""Cuthill-McKee over many components and over directed lists, against a sequential walk."""
import numpy as np
import pytest
import torch

from inching_b200 import _native

pytestmark = pytest.mark.gpu


def _walk(rowptr, cols, degree, seeds):
    n = len(degree)
    seen, order, levels = np.zeros(n, bool), [], 0
    for s in seeds:
        if seen[s]:
            continue
        seen[s] = True
        front = [s]
        while front:
            levels += 1
            order += front
            nxt = []
            for q in front:
                run = [j for j in sorted(cols[rowptr[q]:rowptr[q + 1]])[::-1] if not seen[j]]
                seen[run] = True
                nxt += sorted(run, key=lambda j: degree[j])
            front = nxt
    return np.array(order[::-1]), levels


def _lists(kind, n, rng):
    """Rows of a random graph: `chains` many components, `cloud` one, `directed` one way only."""
    if kind == "chains":
        a = np.arange(n - 1)
        a = a[a % 7 != 6]
        e = np.stack([a, a + 1], 1)
    else:
        e = rng.integers(0, n, (3 * n, 2))
        e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], 1), axis=0)
    perm = rng.permutation(n)
    e = perm[e].reshape(-1, 2)
    if kind != "directed":
        e = np.concatenate([e, e[:, ::-1]])
    e = np.concatenate([e, np.stack([np.arange(n)] * 2, 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]).astype(np.int64)
    return rowptr, e[:, 1].astype(np.int32)


@pytest.mark.parametrize("kind", ["chains", "cloud", "directed"])
@pytest.mark.parametrize("n", [1, 2, 33, 1000, 4097])
def test_order_matches_sequential_walk(kind, n):
    rng = np.random.default_rng(n)
    rowptr, cols = _lists(kind, n, rng)
    degree = np.diff(rowptr).astype(np.int32)
    seeds = np.argsort(degree)
    ref, levels = _walk(rowptr, cols, degree, seeds)
    d = [torch.from_numpy(a).cuda() for a in (rowptr, cols, degree, seeds.astype(np.int64))]
    order, undo, got = _native.cuthill_mckee(*d)
    assert np.array_equal(order.cpu().numpy(), ref) and got == levels
    assert np.array_equal(undo.cpu().numpy()[ref], np.arange(n))
