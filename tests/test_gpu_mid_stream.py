"""The planned stream of the cluster kernel (eigen.cu) where it can go wrong:
rows that end inside a lane's four entries, one entry a row (128 rows a tile),
rows of many tiles, entry counts that are no multiple of four, long runs of
rows without entries at both ends and in the middle, every weight width.
Against the oracle after 40 iterations: each rounds the FP64 iterate to about
1e-16 per operation, well within 1e-11 of its norm; with FP32 differences
(mixed) to 6e-8 of an edge's difference, within 1e-5."""
import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G
from oracle import bindings as O
from tests.test_gpu_slices import csr, dev, weights

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def level(name):
    rng = np.random.default_rng(11)
    if name == "matching":
        n = 12002
        i = np.arange(0, n, 2)
        return csr(n, i, i + 1)
    n = 6003
    if name == "ragged":
        return csr(n, np.concatenate([np.arange(n - 1), rng.integers(0, n, 9001)]),
                   np.concatenate([np.arange(1, n), rng.integers(0, n, 9001)]))
    if name == "hubs":
        hub = np.arange(3, n)
        return csr(n, np.concatenate([np.zeros(hub.size, np.int64), np.full(hub[::2].size, 2), np.arange(n - 1)]),
                   np.concatenate([hub, hub[::2], np.arange(1, n)]))
    # vertices with entries: [500, 2500) and [3500, 5600)
    live = np.concatenate([np.arange(500, 2500), np.arange(3500, 5600)])
    u = live[rng.integers(0, live.size, 12000)]
    v = live[rng.integers(0, live.size, 12000)]
    return csr(n, np.concatenate([u, live[:-1]]), np.concatenate([v, live[1:]]))


@pytest.mark.parametrize("name", ["matching", "ragged", "hubs", "gaps"])
@pytest.mark.parametrize("top", [0, 1000, (1 << 33) + 5])
@pytest.mark.parametrize("mixed", [False, True])
def test_mid_stream(partitioner, monkeypatch, name, top, mixed):
    monkeypatch.setenv("SGPB_PI_SLICES", "0")
    rp, col = level(name)
    n = rp.shape[0] - 1
    assert 32768 < int(rp[-1]) + 8 * n <= 1 << 17
    w = weights(rp, col, top) if top else None
    x0 = np.random.default_rng(n).random(n)
    u_o, it_o, lam_o = O.power_iter(rp, col, w, x0, -1.0, 40)
    u, it, lam, _ = partitioner.power_iter(dev(rp), dev(col), None if w is None else dev(w, top >= 1 << 32),
                                           torch.from_numpy(x0).cuda(), None, -1.0, 40, mixed)
    assert it == it_o == 40
    assert np.linalg.norm(u.cpu().numpy() - u_o) <= (1e-5 if mixed else 1e-11)
    # the mean of u'Lu over a unit vector: at most twice the vector's error times the spectrum's bound 2 max d
    d = np.bincount(np.repeat(np.arange(n), np.diff(rp).astype(np.int64)),
                    None if w is None else w.astype(np.float64), n)
    assert abs(lam - lam_o) <= (1e-5 if mixed else 1e-11) * 4 * d.max()


def test_row_plans_of_fewer_clusters(partitioner, monkeypatch):
    """Row plans that do not fit leave fewer clusters at a time: the batch's
    results are the same."""
    gs = G.batch_graphs(24, seed=5, lo=3000, hi=30000)
    a = partitioner.partition_batch(gs, mixed=True)
    monkeypatch.setenv("SGPB_PI_MID_MB", "1")
    b = partitioner.partition_batch(gs, mixed=True)
    monkeypatch.setenv("SGPB_PI_MID_MB", "0")
    c = partitioner.partition_batch(gs, mixed=True)
    for x, y, z in zip(a, b, c):
        assert np.array_equal(x.part, y.part) and np.array_equal(x.part, z.part)
        assert x.lam == y.lam == z.lam and x.level_iters == y.level_iters == z.level_iters
