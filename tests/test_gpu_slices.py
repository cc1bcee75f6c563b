"""Power iteration on row slices (slices.cu) at the edges of its forms: the
iterate in one block's shared memory (up to 25,600 vertices), its leading part
there (skewed levels of few entries beyond it), column panels (wider levels of
at least five entries per row and panel) and the global gather; rows of every lane split, rows of several chunks and of several layout
items, unit, repeated, 8-, 16-, 32- and 64-bit weights, rows without entries.
Against the oracle after a fixed number of iterations: each iteration rounds
the FP64 iterate to about 1e-16 per operation, so 40 of them stay well within
1e-11 of its norm."""
import time

import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G
from oracle import bindings as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CAP = 40


def dev(a, wide=False):
    t = np.uint64 if wide else np.uint32
    return torch.from_numpy(np.ascontiguousarray(a, t).view(np.int64 if wide else np.int32)).cuda()


def check(partitioner, rp, col, w=None, wide=False, cap=CAP):
    n = rp.shape[0] - 1
    x0 = np.random.default_rng(n).random(n)
    # a negative tolerance: no iterate, converged or not, stops before the cap
    u_o, it_o, lam_o = O.power_iter(rp, col, w, x0, -1.0, cap)
    u, it, lam, _ = partitioner.power_iter(dev(rp), dev(col), None if w is None else dev(w, wide),
                                           torch.from_numpy(x0).cuda(), None, -1.0, cap)
    assert it == it_o == cap
    assert np.linalg.norm(u.cpu().numpy() - u_o) <= 1e-11
    assert abs(lam - lam_o) <= 1e-10 * abs(lam_o)


def csr(n, u, v, w=None):
    """Symmetric CSR of the given pairs (sorted rows, duplicates merged)."""
    keep = u != v
    u, v = u[keep], v[keep]
    key = np.unique(np.concatenate([u.astype(np.int64) * n + v, v.astype(np.int64) * n + u]))
    rows, cols = key // n, key % n
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return rp, cols.astype(np.uint32)


def weights(rp, col, top, seed=1):
    """Symmetric weights in [1, top] with both ends present."""
    n = rp.shape[0] - 1
    rows = np.repeat(np.arange(n, dtype=np.uint64), np.diff(rp).astype(np.int64))
    lo, hi = np.minimum(rows, col), np.maximum(rows, col)
    h = (lo * np.uint64(0x9E3779B97F4A7C15) ^ hi * np.uint64(0xC2B2AE3D27D4EB4F)) >> np.uint64(11)
    w = 1 + h % np.uint64(top)
    e = int(np.flatnonzero((rows == lo) & (col == hi))[0])
    w[(lo == lo[e]) & (hi == hi[e])] = top
    return w


def skewed(n, m, seed):
    """Power-law ends, a hub joined to every fourth vertex, the last vertices
    without entries."""
    rng = np.random.default_rng(seed)
    u = (n * 0.97 * rng.random(m) ** 4).astype(np.int64)
    v = (n * 0.97 * rng.random(m) ** 2).astype(np.int64)
    hub = np.arange(1, int(n * 0.97), 4)
    return csr(n, np.concatenate([u, np.zeros(hub.size, np.int64)]), np.concatenate([v, hub]))


@pytest.mark.parametrize("n,m", [(4001, 30000), (25600, 400000), (25601, 400000), (51203, 1500000), (77000, 200000),
                                 (51201, 6000000)])
@pytest.mark.parametrize("top", [0, 200, 60000, 1 << 31])
def test_forms_and_weights(partitioner, n, m, top):
    """One panel exactly full, one vertex more, three panels' width of few and
    of many entries, and a sparse level, unit weights and every weight width."""
    rp, col = skewed(n, m, n)
    check(partitioner, rp, col, weights(rp, col, top) if top else None)


def test_wide_weights(partitioner):
    for n, m in ((9000, 120000), (60000, 900000), (51201, 6000000)):
        rp, col = skewed(n, m, 3)
        check(partitioner, rp, col, weights(rp, col, (1 << 33) + 5), wide=True)


def test_repeated_weights(partitioner):
    """Panels of a level whose total weight is within 1.25 of its entries:
    entries are repeated (several copies of one destination in a row)."""
    rp, col = skewed(70001, 8000000, 5)
    w = np.ones(col.size, np.uint64)
    rows = np.repeat(np.arange(70001), np.diff(rp).astype(np.int64))
    w[(rows % 64 == 0) & (col % 64 == 0)] = 37
    assert w.sum() <= 1.25 * w.size and w.max() == 37
    check(partitioner, rp, col, w)


def test_one_heavy_entry(partitioner):
    """The same with one weight far above the others: not repeated."""
    rp, col = skewed(70001, 8000000, 5)
    rows = np.repeat(np.arange(70001), np.diff(rp).astype(np.int64))
    e = int(np.flatnonzero(rows < col)[1000])
    w = np.ones(col.size, np.uint64)
    w[((rows == rows[e]) & (col == col[e])) | ((rows == col[e]) & (col == rows[e]))] = 4097
    assert w.sum() <= 1.25 * w.size and w.max() == 4097
    check(partitioner, rp, col, w)


@pytest.mark.parametrize("name", ["coarse", "finest"])
def test_layout_does_not_fit(partitioner, monkeypatch, name):
    """A level whose layout is refused runs on the main kernel: from its start
    vector, and after a finest level's first iterations."""
    monkeypatch.setenv("SGPB_PI_SLICES_MB", "0")
    if name == "coarse":
        rp, col = skewed(30001, 400000, 2)
        check(partitioner, rp, col, weights(rp, col, 200))
        return
    g = G.erdos_renyi(150001, 8.0, seed=9)
    a = partitioner.partition(g, rng_state=5)
    monkeypatch.delenv("SGPB_PI_SLICES_MB")
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    b = partitioner.partition(g, rng_state=5)
    assert a.level_n == b.level_n and a.level_iters[0] > 4
    assert all(abs(x - y) <= 2 for x, y in zip(a.level_iters, b.level_iters))
    assert abs(a.lam - b.lam) <= 1e-9 * abs(b.lam)
    assert abs(a.edgecut - b.edgecut) <= 0.001 * b.edgecut


@pytest.mark.parametrize("n", [9001, 60001])
def test_long_rows(partitioner, n):
    """Two hubs joined to every vertex: rows of several chunks and of several
    layout items, beside rows of a few entries."""
    i = np.arange(2, n)
    rng = np.random.default_rng(n)
    u = np.concatenate([np.zeros(n - 2, np.int64), np.ones(n - 2, np.int64), rng.integers(0, n, 4 * n)])
    v = np.concatenate([i, i, rng.integers(0, n, 4 * n)])
    rp, col = csr(n, u, v)
    assert np.diff(rp).max() >= n - 2
    check(partitioner, rp, col)
    check(partitioner, rp, col, weights(rp, col, 1000))


@pytest.mark.parametrize("name", ["grid", "er", "rgg"])
def test_meshes(partitioner, name):
    g = {"grid": lambda: G.grid2d(300, 211), "er": lambda: G.erdos_renyi(90001, 8.0, seed=3),
         "rgg": lambda: G.rgg3d(30011, seed=2)}[name]()
    check(partitioner, g.row_ptr, g.col)


def test_finest_level_continues_on_slices(partitioner, monkeypatch):
    """A finest level of at least 2^20 entries that does not stop after its
    first iterations goes on from their iterate: the iteration count, the
    value and the partition agree with the run on the main kernel alone."""
    g = G.erdos_renyi(150001, 8.0, seed=9)
    assert g.m_directed >= 1 << 20
    a = partitioner.partition(g, rng_state=5)
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    b = partitioner.partition(g, rng_state=5)
    assert a.level_n == b.level_n and a.level_iters[0] > 4
    assert all(abs(x - y) <= 2 for x, y in zip(a.level_iters, b.level_iters))
    assert abs(a.lam - b.lam) <= 1e-9 * abs(b.lam)
    assert abs(a.edgecut - b.edgecut) <= 0.001 * b.edgecut


@pytest.mark.parametrize("n", [5, 31, 32, 33, 64, 129, 600, 1023, 1025, 1900])
@pytest.mark.parametrize("top", [0, 50])
def test_small_levels(partitioner, n, top):
    """Levels of one block: one warp, several warps, every lane split, more
    rows than threads, with a hub row beside short ones, unit and integer
    weights."""
    rng = np.random.default_rng(n)
    i = np.arange(n - 1)
    hub = np.arange(1, n, 3)
    u = np.concatenate([i, np.zeros(hub.size, np.int64), rng.integers(0, n, 2 * n)])
    v = np.concatenate([i + 1, hub, rng.integers(0, n, 2 * n)])
    rp, col = csr(n, u, v)
    assert rp[-1] + 8 * n <= 32768
    check(partitioner, rp, col, weights(rp, col, top) if top else None)


def test_small_level_dense(partitioner):
    """A small level of long rows: many lanes a row."""
    rng = np.random.default_rng(7)
    rp, col = csr(90, rng.integers(0, 90, 9000), rng.integers(0, 90, 9000))
    check(partitioner, rp, col, weights(rp, col, 1000))
    check(partitioner, rp, col, weights(rp, col, (1 << 33) + 1), wide=True)


def star(n, hubs, extra):
    """Every vertex joined to one of the first few, and random pairs."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    return csr(n, np.concatenate([i % hubs, rng.integers(0, n, extra)]), np.concatenate([i, rng.integers(0, n, extra)]))


# the iterate in shared memory, its leading part there, and gathers from L2 in
# the level's and (a skewed level wider than its panels pay for) its own order;
# one row, or several, far above a block's share of the entries
@pytest.mark.parametrize("n,hubs,extra", [(25001, 1, 0), (25001, 1, 50000), (40000, 1, 80000), (100001, 1, 0),
                                          (100001, 3, 100000), (200001, 2, 1600000)])
@pytest.mark.parametrize("top", [0, 200, 60000, 1 << 31])
def test_rows_above_a_block_s_share(partitioner, n, hubs, extra, top):
    rp, col = star(n, hubs, extra)
    check(partitioner, rp, col, weights(rp, col, top) if top else None)
    if top == 200:
        check(partitioner, rp, col, weights(rp, col, (1 << 33) + 5), wide=True)


@pytest.mark.parametrize("n,hubs,extra", [(100001, 1, 0), (100001, 4, 100000), (300001, 4, 600000)])
def test_long_rows_are_not_slower(partitioner, monkeypatch, n, hubs, extra):
    """300 iterations with few long rows take no longer than on the main kernel
    (1.1 to 1.8 times as long where one block had the whole of such a row)."""
    rp, col = star(n, hubs, extra)
    rp, col = dev(rp), dev(col)
    x = torch.from_numpy(np.random.default_rng(1).random(n)).cuda()

    def best():
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            partitioner.power_iter(rp, col, None, x, tol=-1.0, iter_cap=300, residual=False)
            t.append(time.perf_counter() - t0)
        return min(t)

    fast = best()
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    assert fast <= best()


@pytest.mark.parametrize("n,m", [(9000, 120000), (40000, 200000), (77000, 200000), (51201, 6000000)])
def test_a_barrier_that_gives_up(partitioner, monkeypatch, n, m):
    """The grid barrier's limit runs out in every form: an error, and the
    context goes on."""
    rp, col = skewed(n, m, 4)
    monkeypatch.setenv("SGPB_PI_SPIN", "0")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    with pytest.raises(RuntimeError, match="grid barrier did not complete"):
        partitioner.power_iter(dev(rp), dev(col), None, x, tol=-1.0, iter_cap=CAP)
    monkeypatch.delenv("SGPB_PI_SPIN")
    check(partitioner, rp, col)
