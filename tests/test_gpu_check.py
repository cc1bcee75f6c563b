"""The check of an input graph reads every offset (driver.cu k_check_csr)."""
import numpy as np
import pytest

from ipdps_2021_graph_coarsening_b200 import graphs as G

pytestmark = pytest.mark.gpu


# the check's grid has 8 blocks of 256 threads an SM: offsets of its first
# pass, of later ones, and the last
@pytest.mark.parametrize("at", [1, 303103, 303104, 303105, 650000, 699999])
def test_decreasing_offsets_anywhere(partitioner, at):
    n = 700000
    i = np.arange(n)
    col = np.stack([(i - 1) % n, (i + 1) % n], 1).reshape(-1).astype(np.uint32)
    rp = (2 * np.arange(n + 1)).astype(np.uint32)
    rp[at] = rp[at + 1] + 1
    with pytest.raises(RuntimeError, match="decreasing offsets"):
        partitioner.partition(G.CSR(rp, col))
