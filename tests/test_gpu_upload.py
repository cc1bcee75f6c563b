"""Pageable host arrays of 16 MiB or more go to the device in slots of a pinned
ring (mtx.cu): the level the device holds equals the host's arrays, with the
last slot partly filled, after the ring has grown and when it is larger than
the array asks for."""
import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def circulant(n, k):
    """Vertex i joined to i +- 1 .. i +- k, weights of (|distance|, i + j)."""
    off = np.concatenate([np.arange(-k, 0), np.arange(1, k + 1)])
    col = (np.arange(n)[:, None] + off[None, :]) % n
    w = np.abs(off)[None, :] + (np.arange(n)[:, None] + col) % 97
    order = np.argsort(col, axis=1)
    col, w = np.take_along_axis(col, order, 1), np.take_along_axis(w, order, 1)
    rp = np.arange(0, 2 * k * n + 1, 2 * k, dtype=np.uint32)
    return G.CSR(rp, col.astype(np.uint32).ravel(), w.astype(np.uint32).ravel())


# 16 MiB of destinations less four bytes, exactly, more; several slots' worth; small again
@pytest.mark.parametrize("n,k", [(1048576, 2), (1048575, 2), (524291, 4), (1100003, 10), (524291, 4)])
def test_large_host_arrays(partitioner, n, k):
    g = circulant(n, k)
    h = partitioner.generate_coarse_graphs(g, cutoff=n // 2)
    lv = h.level(0)
    assert np.array_equal(lv["row_ptr"].view(torch.int32).cpu().numpy().view(np.uint32), g.row_ptr)
    assert np.array_equal(lv["col"].view(torch.int32).cpu().numpy().view(np.uint32), g.col)
    assert np.array_equal(lv["w"].view(torch.int32).cpu().numpy().view(np.uint32), g.w)
    h.free()
