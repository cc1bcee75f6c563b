"""Split, cut and FM passes on bitmaps (bits.cuh) at their edges: rows at and
above the length a block takes, bitmaps in shared memory and in global memory
(more than 1.6M vertices; for the two bitmaps of an FM pass more than 0.8M),
vertex counts off the 32-bit words, selections that end on index bits (all
values equal), on a full last candidate list and with few distinct values.
All results are integers: exact against the oracle or recomputed in numpy."""
import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G
from oracle import bindings as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()


def hubs(n, lens):
    """A ring of n vertices; vertex i also joined to lens[i] others."""
    u = [np.arange(n)]
    v = [(np.arange(n) + 1) % n]
    for i, k in enumerate(lens):
        v.append(len(lens) + np.arange(k) % (n - len(lens)))
        u.append(np.full(k, i))
    u, v = np.concatenate(u), np.concatenate(v)
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return rp, (key % n).astype(np.uint32)


def check_split(partitioner, rp, col, ev):
    p_o, c_o = O.compute_partition(rp, col, ev)
    part, cut = partitioner.split(dev(rp), dev(col), torch.from_numpy(ev).cuda())
    assert cut == c_o
    assert np.array_equal(part.cpu().numpy().view(np.uint32), p_o)


@pytest.mark.parametrize("values", ["normal", "equal", "two", "near", "zeros", "exponents"])
@pytest.mark.parametrize("n", [2, 31, 33, 1024, 1025, 20001])
def test_split_selection(partitioner, n, values):
    rng = np.random.default_rng(n)
    ev = {"normal": lambda: rng.standard_normal(n), "equal": lambda: np.full(n, 0.25),
          "two": lambda: np.where(rng.random(n) < 0.5, -1.0, 1.0),
          "near": lambda: 1.0 + rng.permutation(n) * 2.0 ** -52,          # differ in the last key bits
          "zeros": lambda: np.where(rng.random(n) < 0.7, np.where(rng.random(n) < 0.5, 0.0, -0.0),
                                    rng.standard_normal(n)),
          "exponents": lambda: np.ldexp(rng.choice([-1.0, 1.0], n), rng.integers(-900, 900, n))}[values]()
    rp, col = hubs(n, [])
    check_split(partitioner, rp, col, ev)


@pytest.mark.parametrize("lens", [(1021, 1022, 1023), (1024, 4000, 15000)])
def test_cut_of_long_rows(partitioner, lens):
    rp, col = hubs(20001, lens)
    ev = np.random.default_rng(2).standard_normal(20001)
    check_split(partitioner, rp, col, ev)


@pytest.mark.parametrize("n", [1638400, 1638401])
def test_split_bitmap_limit(partitioner, n):
    """200 KB of bits, and one vertex more (the bitmap stays in global memory)."""
    rp, col = hubs(n, (3000,))
    ev = np.random.default_rng(3).standard_normal(n)
    order = np.lexsort((np.arange(n), ev))
    part, cut = partitioner.split(dev(rp), dev(col), torch.from_numpy(ev).cuda())
    part = part.cpu().numpy()
    k = n // 2
    expect = np.ones(n, np.int64)
    expect[order[:k]] = 0
    if n % 2:   # the sweep vertex takes the side of the smaller cut
        expect[order[k]] = part[order[k]]
    assert np.array_equal(part, expect)
    rows = np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))
    assert cut == int((part[rows] != part[col]).sum()) // 2


@pytest.mark.parametrize("n,lens", [(1003, ()), (9001, (1022, 1023, 5000, 8000)), (819232, (2000,))])
def test_fm_rows_and_bitmaps(partitioner, n, lens):
    rp, col = hubs(n, lens)
    rng = np.random.default_rng(n)
    start = (rng.permutation(n) >= n // 2).astype(np.uint32)
    p_o, c_o, passes_o, moves_o = O.fm_refine(rp, col, None, start.copy(), 6)
    part = dev(start)
    cut, passes, moves = partitioner.fm_refine(dev(rp), dev(col), part, 6)
    assert (cut, passes, moves) == (c_o, passes_o, moves_o)
    assert np.array_equal(part.cpu().numpy().view(np.uint32), p_o)
