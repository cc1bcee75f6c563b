"""Performance cases: calls a user of this framework makes, over the sizes the
framework is used at.

Every case is one pass through a public entry point of
``ipdps_2021_graph_coarsening_b200.api`` on a synthetic graph of a family the
framework is built for: grids with removed vertices, the 256 x 256 grid,
Erdos-Renyi, 3D random geometric, R-MAT and weighted Chung-Lu graphs.  R-MAT
graphs are generated on the GPU here (scale 22 takes about a second); the
others come from the package's own generators.  A case's sizes stay the same
from seed to seed: the seed renumbers the vertices (a random permutation of
the graphs whose ids mean nothing, a rotation of the meshes, which keeps their
locality) and seeds the program's own random state and vectors.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  a user's state before the call
    run(state)           one pass, its outputs
    exact(case, seed)    the outputs in 64 bits where they are computed numbers
    work(case)           bytes one pass cannot do without
"""
import math

import numpy as np
import torch

from ipdps_2021_graph_coarsening_b200 import api
from ipdps_2021_graph_coarsening_b200 import graphs as G

_handle = None


def _partitioner():
    """The context a program keeps for its lifetime."""
    global _handle
    if _handle is None:
        _handle = api.Partitioner(0)
    return _handle


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest call: a mesh of the size of the batch configuration's
        # smallest graphs, host arrays in and out (latency and launches)
        {"name": "partition_mesh_2k", "call": "partition", "graph": "holes", "n": 2000, "cutoff": 50, "mixed": False,
         "host": True},
        # the 2D grid configuration: 256 x 256, coarsened to 32 vertices, FP64
        {"name": "partition_grid256", "call": "partition", "graph": "grid", "n": 65536, "cutoff": 32, "mixed": False,
         "host": True},
        # the drop-in sgpar.h entry point on an ordinary skewed graph
        {"name": "sgpar_rmat16", "call": "sgpar", "graph": "rmat", "scale": 16},
        # recursive bisection of a 3D random geometric graph (mesh-like,
        # device resident): the driver's 4-way mode
        {"name": "fourway_rgg_190k", "call": "fourway", "graph": "rgg", "n": 190001},
        # many graphs of uneven sizes in one call, mixed precision
        {"name": "batch_40_mixed", "call": "batch", "count": 40, "lo": 1000, "hi": 60000, "mixed": True},
        # weighted power-law graph (integer weights in [1, 100]), device resident
        {"name": "partition_chunglu_weighted", "call": "partition", "graph": "chunglu", "n": 262147, "cutoff": 50,
         "mixed": False, "host": False},
        # the benchmark: R-MAT scale 22 resident in HBM, FP64
        {"name": "partition_rmat22", "call": "partition", "graph": "rmat", "scale": 22, "cutoff": 50, "mixed": False,
         "host": False},
        # the hierarchy alone, for programs with a solver of their own
        {"name": "coarsen_rmat20", "call": "coarsen", "graph": "rmat", "scale": 20},
        # one level's power iteration, to convergence, on a coarse level
        # (integer weights) from a prolongated vector, FP64
        {"name": "power_iter_coarse_rmat20", "call": "power_iter", "scale": 20},
        # median split and cut of a vector the program computed itself
        {"name": "split_er_1m", "call": "split", "graph": "er", "n": 1000003},
        # FM refinement of a bisection the program has
        {"name": "fm_rmat18", "call": "fm", "graph": "rmat", "scale": 18},
        # MatrixMarket text to the CSR of its largest component
        {"name": "mtx_rmat17", "call": "mtx", "graph": "rmat", "scale": 17},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | 1


def draw(rng):
    call = rng.choice(["partition", "partition", "sgpar", "fourway", "batch", "coarsen", "power_iter", "split", "fm",
                       "mtx"])
    if call == "partition":
        kind = rng.choice(["holes", "er", "rmat", "chunglu"])
        c = {"call": call, "graph": kind, "cutoff": rng.choice([32, 50]), "mixed": False,
             "host": rng.random() < 0.5}
        if kind == "rmat":
            c["scale"] = rng.randint(14, 21)
            c["cutoff"] = rng.randint(30, 60)
        else:
            c["n"] = _log_uniform(rng, 1000, {"holes": 70000, "er": 250000, "chunglu": 700000}[kind])
        return c
    if call == "sgpar":
        return {"call": call, "graph": "er", "n": _log_uniform(rng, 1000, 250000)}
    if call == "fourway":
        return {"call": call, "graph": "rgg", "n": _log_uniform(rng, 5000, 190000)}
    if call == "batch":
        return {"call": call, "count": rng.randint(8, 48), "lo": 1000, "hi": _log_uniform(rng, 4000, 60000),
                "mixed": True}
    if call == "power_iter":
        return {"call": call, "scale": rng.randint(16, 20), "group": rng.choice([5, 6, 7, 8, 9, 10])}
    if call == "split":
        return {"call": call, "graph": "er", "n": _log_uniform(rng, 1000, 1500000)}
    if call == "mtx":
        return {"call": call, "graph": "er", "n": _log_uniform(rng, 1000, 500000)}
    return {"call": call, "graph": "chunglu", "n": _log_uniform(rng, 4000, 600000)}   # coarsen, fm


# ------------------------------------------------------------------ graphs --
def _csr_of_keys(keys, n):
    """(row_ptr, col) of sorted distinct keys u * n + v."""
    u = torch.div(keys, n, rounding_mode="floor")
    rp = torch.zeros(n + 1, dtype=torch.int64, device=keys.device)
    rp[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
    return rp.to(torch.int32), (keys - u * n).to(torch.int32)


def _rmat(scale, gen):
    """R-MAT (0.57, 0.19, 0.19, 0.05), 16 edges per vertex, symmetrised,
    duplicates merged, self loops dropped, largest component kept, vertices
    permuted by ``gen``: (row_ptr, col) int32 on the GPU."""
    base = torch.Generator(device="cuda")
    base.manual_seed(scale)
    n, m = 1 << scale, 16 << scale
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, generator=base, device="cuda")
        lower = r >= 0.76
        u = 2 * u + lower
        v = 2 * v + (((r >= 0.57) & ~lower) | (r >= 0.95))
    keep = u != v
    u, v = u[keep], v[keep]
    keys = torch.unique(torch.cat([u * n + v, v * n + u]))
    u = torch.div(keys, n, rounding_mode="floor")
    v = keys - u * n
    label = torch.arange(n, device="cuda")
    while True:                                          # smallest id of each component
        new = label.scatter_reduce(0, u, label[v], "amin")
        new = new[new]
        if torch.equal(new, label):
            break
        label = new
    inside = label == torch.bincount(label[u]).argmax()  # the component of most entries
    nc = int(inside.sum())
    ids = torch.empty(n, dtype=torch.int64, device="cuda")
    ids[inside] = torch.randperm(nc, generator=gen, device="cuda")
    keep = inside[u]
    return _csr_of_keys(torch.sort(ids[u[keep]] * nc + ids[v[keep]])[0], nc)


def _renumber(g, new_id):
    """The host graph ``g`` with vertex i called new_id[i], rows sorted."""
    n = g.n
    rows = np.repeat(new_id, np.diff(g.row_ptr.astype(np.int64)))
    cols = new_id[g.col]
    order = np.argsort(rows * n + cols, kind="stable")
    rp = np.zeros(n + 1, dtype=np.uint32)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return G.CSR(rp, cols[order].astype(np.uint32), None if g.w is None else g.w[order])


def _rotated(g, rng):
    """A mesh with its ids rotated: other inputs of the same locality."""
    return _renumber(g, (np.arange(g.n, dtype=np.int64) + int(rng.integers(1, g.n))) % g.n)


def _graph(case, seed):
    """Host CSR or, for R-MAT, device arrays of the case's graph."""
    kind = case["graph"]
    if kind == "rmat":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        return _rmat(case["scale"], gen)
    n = case["n"]
    rng = np.random.default_rng(seed)
    if kind in ("holes", "grid"):
        nx = int(math.sqrt(n))
        ny = max(2, n // nx)
        return _rotated(G.grid2d(nx, ny) if kind == "grid" else G.grid2d_holes(nx, ny, seed=n), rng)
    if kind == "rgg":
        return _rotated(G.rgg3d(n, 12.0, seed=n), rng)
    g = G.erdos_renyi(n, 8.0, seed=n) if kind == "er" else \
        G.chung_lu(n, seed=n, wmax=100 if case["call"] in ("partition", "coarsen") else 0)
    return _renumber(g, rng.permutation(g.n))


def _host(g):
    if isinstance(g, G.CSR):
        return g
    return G.CSR(g[0].cpu().numpy().view(np.uint32), g[1].cpu().numpy().view(np.uint32))


def _device(g):
    if not isinstance(g, G.CSR):
        return {"row_ptr": g[0], "col": g[1]}
    out = {"row_ptr": torch.from_numpy(g.row_ptr.view(np.int32)).cuda(),
           "col": torch.from_numpy(g.col.view(np.int32)).cuda()}
    if g.w is not None:
        out["w"] = torch.from_numpy(g.w.view(np.int32)).cuda()
    return out


def _coarse_level(case, seed):
    """A weighted coarse level of an R-MAT graph: its vertices in random
    groups (8 a group, about what one coarsening step of these graphs keeps),
    parallel edges summed; and the prolongation from a level half its size
    with that level's vector."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rp, col = _rmat(case["scale"], gen)
    n = rp.numel() - 1
    size = case.get("group", 8)
    nc = -(-n // size)
    # the numbering is random already: consecutive ids make random groups
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    gu = torch.div(u, size, rounding_mode="floor")
    gv = torch.div(col.long(), size, rounding_mode="floor")
    keep = gu != gv
    keys, w = torch.unique(gu[keep] * nc + gv[keep], return_counts=True)
    crp, ccol = _csr_of_keys(keys, nc)
    half = -(-nc // 2)
    vcmap = (torch.randperm(nc, generator=gen, device="cuda") % half).to(torch.int32)
    x = torch.rand(half, generator=gen, device="cuda", dtype=torch.float64)
    return {"row_ptr": crp, "col": ccol, "w": w.to(torch.int32), "vcmap": vcmap, "x": x}


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    call = case["call"]
    s = {"call": call, "case": case, "p": _partitioner()}
    if call in ("partition", "fourway"):
        g = _graph(case, seed)
        s["rng"] = 0x853C49E6748FEA9B + 2 * seed          # the program's own seeding
        if case.get("host", False):
            s["g"] = _host(g)
            s["n"] = s["g"].n
        else:
            s["g"] = _device(g)
            s["n"] = s["g"]["row_ptr"].numel() - 1
    elif call == "sgpar":
        s["g"] = _host(_graph(case, seed))
    elif call == "batch":
        rng = np.random.default_rng(seed)
        s["g"] = [_rotated(g, rng) for g in
                  G.batch_graphs(case["count"], seed=case["count"], lo=case["lo"], hi=case["hi"])]
    elif call == "coarsen":
        s["g"] = _host(_graph(case, seed))
        # the program's own store: its levels one after another, with room
        # for hierarchies of up to twice the vertices and three times the
        # entries of the graph
        n, m = s["g"].n, s["g"].m_directed
        for k, size in (("row_ptr", 2 * n), ("vcmap", 2 * n), ("vtx_w", 2 * n), ("col", 3 * m), ("w", 3 * m)):
            s[k] = torch.zeros(size + 1024, dtype=torch.int32, device="cuda")
    elif call == "power_iter":
        s.update(_coarse_level(case, seed))
    elif call == "mtx":
        g = _host(_graph(case, seed))
        s["text"] = np.frombuffer(G.mtx_of(g, seed=seed, dup_frac=0.1, extra_vertices=g.n // 100), dtype=np.uint8)
    else:                                                # split, fm
        s.update(_device(_graph(case, seed)))
        n = s["row_ptr"].numel() - 1
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        if call == "split":
            s["x"] = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
        else:
            s["part"] = torch.randperm(n, generator=gen, device="cuda").lt(n // 2).logical_not().to(torch.int32)
    return s


# --------------------------------------------------------------------- run --
def run(s):
    call, case, p = s["call"], s["case"], s["p"]
    if call == "partition":
        out = None if case["host"] else torch.empty(s["n"], dtype=torch.int32, device="cuda")
        r = p.partition(s["g"], cutoff=case["cutoff"], mixed=case["mixed"], rng_state=s["rng"], part_out=out)
        return {"part": r.part, "edgecut": r.edgecut, "lambda": r.lam}
    if call == "fourway":
        out = torch.empty(s["n"], dtype=torch.int32, device="cuda")
        part4, cut, cut4, _ = p.partition_4way(s["g"], rng_state=s["rng"], part_out=out)
        return {"part4": part4, "cut": cut, "cut4": cut4}
    if call == "sgpar":
        part, cut = api.partition_graph(s["g"], api.Config())
        return {"part": part, "edgecut": cut}
    if call == "batch":
        rs = p.partition_batch(s["g"], mixed=case["mixed"])
        return {"part": np.concatenate([r.part for r in rs]), "edgecut": np.array([r.edgecut for r in rs])}
    if call == "coarsen":
        h = p.generate_coarse_graphs(s["g"])
        at = dict.fromkeys(("row_ptr", "vcmap", "vtx_w", "col", "w"), 0)
        sizes = np.zeros((32, 2), dtype=np.int64)
        for l in range(len(h)):
            lv = h.level(l)
            sizes[l] = lv["n"], lv["m"]
            for k in at:
                if lv[k] is not None:
                    t = lv[k].view(torch.int32)
                    s[k][at[k]:at[k] + t.numel()].copy_(t)
                    at[k] += t.numel()
        h.free()
        return {"levels": sizes, **{k: s[k] for k in at}}
    if call == "power_iter":
        x, iters, lam, _ = p.power_iter(s["row_ptr"], s["col"], s["w"], s["x"], vcmap=s["vcmap"], residual=False)
        return {"iters": iters, "lambda": lam, "x": x}
    if call == "split":
        part, cut = p.split(s["row_ptr"], s["col"], s["x"])
        return {"part": part, "edgecut": cut}
    if call == "fm":
        part = s["part"].clone()                         # refined in place
        cut, passes, moves = p.fm_refine(s["row_ptr"], s["col"], part)
        return {"part": part, "cut": cut, "passes": passes, "moves": moves}
    csr, info = p.mtx_read(s["text"])
    return {"row_ptr": csr.row_ptr, "col": csr.col, "components": info["components"]}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """Power iteration of the level in 64 bits: r = (gb - d) u + A u with
    gb = max(2 max d, 2), deflated against the constant vector and normalised,
    until the dot product of consecutive iterates moves by at most 1e-10; the
    iterate the last step began with and its Rayleigh quotient."""
    if case["call"] != "power_iter":
        return None
    s = _coarse_level(case, seed)
    n = s["row_ptr"].numel() - 1
    a = torch.sparse_csr_tensor(s["row_ptr"].long(), s["col"].long(), s["w"].double(), size=(n, n))
    d = a @ torch.ones(n, dtype=torch.float64, device="cuda")
    gb = max(2.0 * float(d.max()), 2.0)
    v = s["x"][s["vcmap"].long()]
    v = v - v.mean()
    v = v / v.norm()
    dot, last, limit = 0.0, 1.0, 20000
    while abs(dot - last) > 1e-10 and limit:
        u = v
        r = (gb - d) * u + a @ u
        lam = gb - float(u @ r) / float(u @ u)
        v = r - r.mean()
        v = v / v.norm()
        last, dot = dot, float(u @ v)
        limit -= 1
    return {"iters": None, "lambda": lam, "x": u}


# -------------------------------------------------------------------- work --
def _size(case):
    """About how many vertices and directed entries the case's graph has."""
    if case["call"] == "batch":
        lo, hi = case["lo"], case["hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        return n, 6 * n
    if "scale" in case:
        d = case["scale"] - 16
        k = 2.0 ** case["scale"]
        return k * (0.71 - 0.023 * d), k * (27.7 + 0.48 * d)
    n = case["n"]
    return n, n * {"holes": 3.3, "grid": 4, "er": 8, "rgg": 11.7, "chunglu": 24}[case["graph"]]


def work(case):
    """Each input read once and each output written once."""
    n, m = _size(case)
    call = case["call"]
    graph = 4 * n + 4 * m
    if call == "partition" and case["graph"] == "chunglu":
        graph += 4 * m                                   # weights
    if call == "coarsen":
        return {"bytes": graph + graph + 8 * n, "flops": 0}
    if call == "power_iter":
        k = n / case.get("group", 8)
        return {"bytes": 8 * m + 4 * k + 4 * k + 4 * k + 8 * k, "flops": 2 * m}
    if call == "split":
        return {"bytes": graph + 8 * n + 4 * n, "flops": 0}
    if call == "mtx":
        return {"bytes": 1.1 * m / 2 * 14 + graph, "flops": 0}
    return {"bytes": graph + 4 * n, "flops": 0}
