"""Pageable host arrays of 16 MiB or more go to the device in slots of a pinned
ring (mtx.cu): the level the device holds equals the host's arrays, with the
last slot partly filled, after the ring has grown and when it is larger than
the array asks for."""
import os
import subprocess
import sys

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


SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
static int allowed = -1;
void shim_allow(int n) { allowed = n; }
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) {
    static int (*real)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    if (!real) real = dlsym(RTLD_NEXT, "pthread_create");
    if (allowed == 0) return EAGAIN;
    if (allowed > 0) allowed--;
    return real(t, a, f, x);
}
"""

CHILD = """
import ctypes, sys
import numpy as np
from ipdps_2021_graph_coarsening_b200 import api, graphs as G
shim = ctypes.CDLL(sys.argv[1])
n = 1500000
col = np.empty((n, 4), np.uint32)
for k, d in enumerate((-2, -1, 1, 2)):
    col[:, k] = (np.arange(n) + d) % n
g = G.CSR((4 * np.arange(n + 1)).astype(np.uint32), col.reshape(-1))
p = api.Partitioner(0)
small = G.grid2d(20, 20)
p.generate_coarse_graphs(small).free()
shim.shim_allow(int(sys.argv[2]))
h = p.generate_coarse_graphs(g)
shim.shim_allow(-1)
lv = h.level(0)
assert np.array_equal(lv["col"].cpu().numpy().view(np.uint32), g.col)
print("uploaded")
"""


@pytest.mark.parametrize("allowed", [0, 2])
def test_threads_run_out(tmp_path, allowed):
    """No thread, or only some, to be had for the host pool when the first
    large array goes up: the upload goes on with those there are."""
    src, so, child = tmp_path / "shim.c", tmp_path / "shim.so", tmp_path / "child.py"
    src.write_text(SHIM)
    child.write_text(CHILD)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=root)
    r = subprocess.run([sys.executable, str(child), str(so), str(allowed)], env=env, cwd=root, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "uploaded" in r.stdout, r.stdout[-500:] + r.stderr[-1500:]
