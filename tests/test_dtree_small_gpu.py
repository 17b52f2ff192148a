"""The device tree at the edges of the one-CTA sort (2, 4 and 8 bodies a thread; 8,192 bodies,
above which the radix passes take over), with bodies in equal cells (a stable order decides),
and of the eight lanes that share a node's moments: leaves of 1 to 9 and of 40 bodies.  Against
the host builder, as the other sizes (entry for entry; the bound there)."""
import numpy as np
import pytest

from gplum_gb300.disk import make_disk
from tests.test_dtree_sizes_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 1025, 4095, 4096, 8191, 8192, 8193])
def test_sort_edges(gpu, n):
    d = make_disk(n, 1e-9, 0.9, 1.1, seed=n)
    d["pos"][n // 2:n // 2 + 3] = d["pos"][n // 2]
    check(d, 8, 64)


@pytest.mark.parametrize("leaf", [1, 2, 7, 8, 9, 40])
def test_leaves_and_lanes(gpu, leaf):
    d = make_disk(2500, 1e-9, 0.9, 1.1, seed=leaf)
    d["pos"][700:700 + leaf + 5] = d["pos"][700]  # more than a leaf holds, at the deepest level
    d["mass"][::7] = 0.0
    check(d, leaf, 64)
