"""Cuthill-McKee at the line where its kernel takes two blocks an SM, and the lists that it
refuses."""
import numpy as np
import pytest
import torch

from inching_b200 import _native
from oracle import graph as og

pytestmark = pytest.mark.gpu


def _order(rowptr, cols, degree, seeds):
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (np.asarray(rowptr, np.int64), np.asarray(cols, np.int32), np.asarray(degree, np.int32),
          np.asarray(seeds, np.int64))]
    return _native.cuthill_mckee(*d)


def _ladder(n, every):
    """Rows i: i - 2 .. i + 2 and itself, cut into pieces of `every` atoms, numbered at random."""
    i = np.arange(n)
    e = np.concatenate([np.stack([i, i], 1)] + [np.stack([i[:-k], i[k:]], 1) for k in (1, 2)])
    e = e[e[:, 0] // every == e[:, 1] // every]
    e = np.concatenate([e, e[e[:, 0] != e[:, 1]][:, ::-1]])
    e = np.random.default_rng(n).permutation(n)[e]
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    return np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))]), e[:, 1].copy()


@pytest.mark.parametrize("n,every", [(10000, 100), (10001, 100), (10001, 20000), (210000, 700)])
def test_order_around_two_blocks_an_sm(n, every):
    rowptr, cols = _ladder(n, every)
    degree = np.diff(rowptr)
    seeds = np.argsort(degree)
    order, undo, _ = _order(rowptr, cols, degree, seeds)
    ref, ref_undo = og.cuthill_mckee_c(rowptr, cols, degree, seeds)
    assert np.array_equal(order.cpu().numpy(), ref) and np.array_equal(undo.cpu().numpy(), ref_undo)


def _broken(rowptr, cols, row, entry):
    """The lists with one more entry in a row."""
    at = rowptr[row + 1]
    r = rowptr.copy()
    r[row + 1:] += 1
    return r, np.insert(cols, at, entry)


@pytest.mark.parametrize("where", ["first", "last"])
def test_row_that_lists_an_atom_twice(where):
    n = 300
    rowptr, cols = _ladder(n, n)
    degree = np.diff(rowptr)
    order, _, _ = _order(rowptr, cols, degree, np.argsort(degree))
    # the parent of an atom found early, or of the last one, lists it twice
    bfs = order.cpu().numpy()[::-1]
    child = bfs[1] if where == "first" else bfs[-1]
    pos = np.empty(n, int)
    pos[bfs] = np.arange(n)
    parent = min((j for j in cols[rowptr[child]:rowptr[child + 1]] if j != child), key=lambda j: pos[j])
    r, c = _broken(rowptr, cols, parent, child)
    with pytest.raises(AssertionError, match="duplicates"):
        _order(r, c, degree, np.argsort(degree))


@pytest.mark.parametrize("entry", [-1, 300, 2 ** 31 - 1])
def test_column_out_of_range(entry):
    rowptr, cols = _ladder(300, 50)
    degree = np.diff(rowptr)
    r, c = _broken(rowptr, cols, 150, entry)
    with pytest.raises(AssertionError, match="column index"):
        _order(r, c, degree, np.argsort(degree))


def test_row_too_long():
    n = _native.MAX_DEGREE + 1
    rowptr = np.concatenate([[0], np.cumsum([n] + [1] * (n - 1))])
    cols = np.concatenate([np.arange(n), np.arange(1, n)])
    degree = np.diff(rowptr)
    with pytest.raises(_native.InchError, match="neighbours"):
        _order(rowptr, cols, degree, np.argsort(degree))


def test_seeds_not_a_permutation():
    rowptr, cols = _ladder(300, 50)
    degree = np.diff(rowptr)
    seeds = np.argsort(degree)
    seeds[7] = seeds[8]
    with pytest.raises(AssertionError, match="permutation"):
        _order(rowptr, cols, degree, seeds)


def test_seed_behind_many_visited_ones():
    """Directed lists: the first seed reaches all atoms but the last one in seed order."""
    n = 5000
    heads = np.concatenate([np.arange(n - 2), [n - 1]])
    tails = np.concatenate([np.arange(1, n - 1), [0]])
    e = np.concatenate([np.stack([heads, tails], 1), np.stack([np.arange(n)] * 2, 1)])
    e = e[np.lexsort((e[:, 1], e[:, 0]))]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(e[:, 0], minlength=n))])
    degree = np.diff(rowptr)
    order, _, levels = _order(rowptr, e[:, 1].copy(), degree, np.arange(n))
    assert np.array_equal(order.cpu().numpy(), np.arange(n)[::-1]) and levels == n


def test_wait_that_runs_out():
    """A bound that no block's wait keeps: the call says so, and the next one is answered."""
    import ctypes
    n = 2000
    rowptr, cols = _ladder(n, n)
    degree = np.diff(rowptr)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (rowptr.astype(np.int64), cols.astype(np.int32), degree.astype(np.int32),
          np.argsort(degree).astype(np.int64))]
    L = _native.lib()
    ws = torch.empty(L.inch_rcm_workspace_size(n), dtype=torch.uint8, device="cuda")
    order, undo = (torch.empty(n, dtype=torch.int64, device="cuda") for _ in range(2))
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def call(polls):
        return L.inch_rcm_bounded(*[p(t) for t in d], n, p(order), p(undo), None, polls, p(ws), ws.numel(),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))

    assert call(0) == _native.INCH_TIMEOUT
    assert call(1 << 24) == _native.INCH_OK
    torch.cuda.synchronize()
    ref, _ = og.cuthill_mckee_c(rowptr, cols, degree, np.argsort(degree))
    assert np.array_equal(order.cpu().numpy(), ref)
