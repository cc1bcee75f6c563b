"""Partitions do not depend on the order in which the power iteration adds up.

Row slices and the rows form of the small levels add in another order than the
plain kernels (SGPB_PI_SLICES=0), so their vectors differ by rounding.  A
partition is certified against that (eigen.cu pi_plain, internal.h) and
repeated in the plain order where the certificate fails: the median among
values that are equal in exact arithmetic (leaves of one aggregate), an
iteration that stops within rounding of the tolerance, an iterate that
cancels.  Bit for bit against the plain order."""
import ctypes

import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import _lib as L
from ipdps_2021_graph_coarsening_b200 import graphs as G
from tests.test_gpu_parity import dev_u32

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def of_edges(n, u, v):
    k = np.unique(np.concatenate([u * n + v, v * n + u]))
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.bincount(k // n, minlength=n))
    return G.CSR(rp, (k % n).astype(np.uint32))


def leafy(core, leaves, seed):
    """An Erdos-Renyi core with leaves, most of them on its first vertices."""
    c = G.erdos_renyi(core, 6.0, seed=seed)
    rng = np.random.default_rng(seed)
    u = np.repeat(np.arange(c.n), np.diff(c.row_ptr.astype(np.int64)))
    hub = (c.n * rng.random(leaves) ** 4).astype(np.int64)
    return of_edges(c.n + leaves, np.concatenate([u, hub]),
                    np.concatenate([c.col.astype(np.int64), c.n + np.arange(leaves)]))


# graphs whose parts (leafy, R-MAT 15), iteration counts and cut (R-MAT 14)
# differ between the two orders
GRAPHS = [(lambda s: leafy(8000, 12000, s), (7, 17, 27, 53)), (lambda s: leafy(3000, 30000, s), (13, 17, 51)),
          (lambda s: leafy(8000, 6000, s), (15, 27, 31, 120)),
          (lambda s: G.rmat(15, 4, seed=s), (30, 51)), (lambda s: G.rmat(14, seed=s), (14, 41)),
          (lambda s: G.rmat(13, seed=s), (42,))]


def both(monkeypatch, call):
    monkeypatch.delenv("SGPB_PI_SLICES", raising=False)
    a = call()
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    return a, call()


def same(a, b):
    assert np.array_equal(a.part, b.part)
    assert (a.edgecut, a.part0_size, a.level_iters, a.rng_state) == (b.edgecut, b.part0_size, b.level_iters, b.rng_state)


@pytest.mark.parametrize("make,seed", [(f, s) for f, seeds in GRAPHS for s in seeds])
def test_partitions_are_the_plain_order_s(partitioner, monkeypatch, make, seed):
    g = make(seed)
    same(*both(monkeypatch, lambda: partitioner.partition(g, rng_state=1000 + seed)))


def test_batch_and_4way_are_the_plain_order_s(partitioner, monkeypatch):
    gs = [make(s) for make, seeds in GRAPHS[:2] for s in seeds]
    for a, b in zip(*both(monkeypatch, lambda: partitioner.partition_batch(gs, rng_state=1007))):
        same(a, b)
    # two vertices joined by an edge: r = 0, and what is left is rounding
    tri = of_edges(3, np.array([0, 0, 1]), np.array([1, 2, 2]))
    for g in (tri, gs[0]):
        for seed in range(70, 80):
            a, b = both(monkeypatch, lambda: partitioner.partition_4way(g, rng_state=seed))
            assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


def test_a_batch_of_both_kinds(partitioner, monkeypatch):
    """Graphs that start in the plain order (mostly leaves) beside ones that do
    not, of which some are repeated; waves of one kind first and last."""
    gs = [make(s) for make, seeds in GRAPHS for s in seeds]
    grids = [G.grid2d(200, 150), G.grid2d(40, 30), G.erdos_renyi(40000, 8.0, seed=2), G.rmat(12, seed=3)]
    for batch in (grids + gs, gs, gs[:3] + grids[1:2]):
        for a, b in zip(*both(monkeypatch, lambda: partitioner.partition_batch(batch, rng_state=1007))):
            same(a, b)


@pytest.mark.parametrize("n", [700, 20000])   # one block's rows form, row slices
def test_a_stop_within_rounding_of_the_tolerance(partitioner, monkeypatch, n):
    g = G.erdos_renyi(n, 8.0, seed=3)
    rp, col = dev_u32(g.row_ptr), dev_u32(g.col)
    x = torch.from_numpy(np.random.default_rng(1).random(g.n)).cuda()

    def run(tol):
        y, iters, lam, _ = partitioner.power_iter(rp, col, None, x, tol=tol, residual=False)
        return y.cpu().numpy(), iters

    # the tolerance at which the plain order takes one iteration more
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    k = run(1e-7)[1]
    lo, hi = 1e-8, 1e-7   # more than k, at most k
    assert run(lo)[1] > k
    while hi - lo > 1e-17:
        mid = 0.5 * (lo + hi)
        if run(mid)[1] > k:
            lo = mid
        else:
            hi = mid
    for tol in (lo, hi, lo - 2e-16, hi + 2e-16):
        (a, ia), (b, ib) = both(monkeypatch, lambda: run(tol))
        assert ia == ib and np.array_equal(a, b)


@pytest.mark.parametrize("n", [700, 20000])
def test_tolerances_near_rounding_take_the_plain_order(partitioner, monkeypatch, n):
    g = G.erdos_renyi(n, 8.0, seed=4)
    for tol in (9e-12, 1e-14, 0.0):
        same(*both(monkeypatch, lambda: partitioner.partition(g, tol=tol, iter_cap=400, rng_state=5)))


@pytest.mark.parametrize("n", [700, 20000])
def test_a_few_iterations_do_without_the_layout(partitioner, monkeypatch, n):
    g = G.erdos_renyi(n, 8.0, seed=5)
    rp, col = dev_u32(g.row_ptr), dev_u32(g.col)
    x = torch.from_numpy(np.random.default_rng(2).random(g.n)).cuda()
    a, b = both(monkeypatch, lambda: partitioner.power_iter(rp, col, None, x, iter_cap=4, residual=False))
    assert a[1] == b[1] == 4 and torch.equal(a[0], b[0])


@pytest.mark.parametrize("at", [-5, 0, 5])
def test_a_result_over_the_start_vector(partitioner, monkeypatch, at):
    """x_out may lie over x_in, which is read before the first iteration."""
    g = G.erdos_renyi(20000, 8.0, seed=6)
    rp, col = dev_u32(g.row_ptr), dev_u32(g.col)
    x = np.random.default_rng(3).random(g.n)
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    want = partitioner.power_iter(rp, col, None, torch.from_numpy(x).cuda(), residual=False)
    monkeypatch.delenv("SGPB_PI_SLICES")
    buf = torch.zeros(g.n + 10, dtype=torch.float64, device="cuda")
    buf[5:5 + g.n] = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    iters, lam = ctypes.c_uint64(0), ctypes.c_double(0)
    ptr = buf.data_ptr() + 40
    L.check(L.lib().sgp_b200_power_iter(partitioner._ctx, g.n, rp.data_ptr(), col.data_ptr(), None, 0, ptr, None,
                                        ptr + 8 * at, 1e-10, 0, 0, ctypes.byref(iters), ctypes.byref(lam), None),
            "sgp_b200_power_iter")
    assert iters.value == want[1] and torch.equal(buf[5 + at:5 + at + g.n], want[0])
