"""The bitmap dedupe of the coarse build (build.cu) at the edges of its tiers,
of the bitmap's words and of its two ways to read it, and on both sides of the
rule that leaves wide levels to the radix sort: integers, bit for bit against
the oracle's build."""
import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G
from ipdps_2021_graph_coarsening_b200.api import PCG32
from oracle import bindings as O
from tests.test_gpu_parity import dev_u32, host_u32, host_u64

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# entries of a bucket: the edges of the tiers (larger ones are summed densely,
# where an entry of weight 0 alone leaves no coarse entry)
SIZES = [1, 32, 33, 64, 255, 256, 257, 1024, 1025, 2048, 2049, 4095, 4096]
DENSE = [4097]


def level(nc, seed, sizes):
    """Aggregates whose buckets have the sizes above (from one fine row or from
    three), every other vertex one entry; destinations spread over the level,
    among its first ones (full words) and at its ends, with duplicates."""
    rng = np.random.default_rng(seed)

    def dest(size, c):
        kind = rng.integers(3)
        d = rng.integers(0, nc if kind else min(nc, size + 2), size)
        d[rng.random(size) < 0.05] = nc - 1
        d[rng.random(size) < 0.05] = 0
        if kind == 2 and size > 1:
            d[1::2] = d[: size // 2]           # every destination twice
        return np.where(d == c, 1 if c == 0 else 0, d)

    special, extra = {}, []
    for k, c in enumerate(rng.permutation(nc)[:min(len(sizes) * 2, nc)]):
        size = sizes[k % len(sizes)]
        if k < len(sizes):
            special[int(c)] = [dest(size, c)]
        else:
            special[int(c)] = np.split(dest(size, c), sorted(rng.integers(0, size + 1, 2)))
            extra += [(int(c), q) for q in special[int(c)][1:]]
    lens = np.ones(nc + len(extra), np.int64)
    for c, parts in special.items():
        lens[c] = parts[0].size
    for k, (c, q) in enumerate(extra):
        lens[nc + k] = q.size
    rp = np.zeros(lens.size + 1, np.uint32)
    rp[1:] = np.cumsum(lens)
    col = np.zeros(int(rp[-1]), np.uint32)
    ones = np.array([c for c in range(nc) if c not in special], np.int64)
    col[rp[ones]] = (ones + 1) % nc
    for c, parts in special.items():
        col[rp[c]:rp[c + 1]] = parts[0]
    for k, (c, q) in enumerate(extra):
        col[rp[nc + k]:rp[nc + k + 1]] = q
    vc = np.concatenate([np.arange(nc), [c for c, _ in extra]]).astype(np.uint32)
    return rp, col, vc


# words and summary words of one bit more and less; eight words a thread of
# the 64- and 512-thread tiers; the tiers leave for the radix sort at about
# 190,000 (64 threads), 380,000 (128), 560,000 (256) and 1,100,000 (512)
@pytest.mark.parametrize("nc", [2, 31, 32, 33, 1023, 1024, 1025, 5000, 16384, 16385, 131072, 131073, 190000, 230000,
                                300001, 420001, 700001, 1200001])
@pytest.mark.parametrize("width", [0, 4, 8])
def test_bitmap_dedupe(partitioner, nc, width):
    rp, col, vc = level(nc, nc, SIZES if width else SIZES + DENSE)
    w = None
    if width:
        top = 1000 if width == 4 else 1 << 35
        w = np.random.default_rng(1).integers(0, top, col.size).astype(np.uint64)   # zero weights too
    want = O.build_coarse(rp, col, w, vc, nc)
    dw = None if w is None else (dev_u32(w.astype(np.uint32)) if width == 4 else
                                 torch.from_numpy(w.view(np.int64)).cuda())
    crp, ccol, cw = partitioner.build_coarse(dev_u32(rp), dev_u32(col), dw, dev_u32(vc), nc, 8 if width == 8 else 4)
    got = host_u32(crp), host_u32(ccol), (host_u64(cw) if width == 8 else host_u32(cw)).astype(np.uint64)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


# 32-bit weights into 64-bit sums, as a graph whose total needs 64 bits is
# built: weights near 2^32, so that every pair of equal destinations sums to
# more than 32 bits; buckets of every tier, on both sides of the radix rule
@pytest.mark.parametrize("nc", [33, 1025, 16385, 190000, 420001, 1200001])
def test_sums_wider_than_weights(partitioner, nc):
    rp, col, vc = level(nc, nc + 1, SIZES + DENSE)
    w = np.random.default_rng(2).integers((1 << 32) - 1000, 1 << 32, col.size).astype(np.uint64)
    want = O.build_coarse(rp, col, w, vc, nc)
    assert want[2].max() >= 1 << 32
    crp, ccol, cw = partitioner.build_coarse(dev_u32(rp), dev_u32(col), dev_u32(w.astype(np.uint32)), dev_u32(vc), nc,
                                             8)
    for a, b in zip((host_u32(crp), host_u32(ccol), host_u64(cw)), want):
        assert np.array_equal(a, b)


def test_hierarchy_of_a_total_above_32_bits(partitioner):
    g = G.rmat(13, seed=5)
    rows = np.repeat(np.arange(g.n), np.diff(g.row_ptr.astype(np.int64)))
    lo, hi = np.minimum(rows, g.col).astype(np.uint64), np.maximum(rows, g.col).astype(np.uint64)
    w = ((1 << 32) - 1 - (lo * 31 + hi * 17) % 1000).astype(np.uint32)   # symmetric
    seed = 0x853C49E6748FEA9B
    h = partitioner.generate_coarse_graphs(G.CSR(g.row_ptr, g.col, w), 50, PCG32(seed))
    o = O.partition_graph(g.row_ptr, g.col, w, cutoff=50, rng_state=seed)
    assert len(h) == len(o["level_n"]) > 2
    rp, col, cw = g.row_ptr, g.col, w.astype(np.uint64)
    for l in range(1, len(h)):
        vc = host_u32(h.level(l - 1)["vcmap"])
        lv = h.level(l)
        assert lv["n"] == o["level_n"][l] and lv["wbytes"] == 8
        rp, col, cw = O.build_coarse(rp, col, cw, vc, lv["n"])
        assert np.array_equal(host_u32(lv["row_ptr"]), rp) and np.array_equal(host_u32(lv["col"]), col)
        assert np.array_equal(host_u64(lv["w"]), cw)
    h.free()
