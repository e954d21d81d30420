"""The cluster solve of ss_solve_block_tridiagonal at the edges of its split, against the oracle's
sequential block LDL^T: one CTA, one node over it, every CTA full, partitions of unequal length."""
import numpy as np
import pytest

from oracle import oracle
from steadyscan_b200 import api
from tests.test_solve_gpu import random_spd_chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 513, 1793, 2047, 2048, 2049, 4095, 4097, 6145])
def test_edges_of_the_cluster_split(n):
    d, c, b = random_spd_chain(n, np.random.default_rng(n))
    ref = oracle.block_tridiag_solve(d, c, b)
    scale = np.abs(ref).max()
    x = api.solve_block_tridiagonal(d, c, b).cpu().numpy()
    np.testing.assert_allclose(x, ref, rtol=0, atol=1e-9 * scale)
    y = api.solve_block_tridiagonal_noalloc(d, c, b).cpu().numpy()
    np.testing.assert_array_equal(x, y)
