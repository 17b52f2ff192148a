"""Fragments that outgrow their bundle: a cluster with more fragmenting collisions in a tree
step than its bundle of 128 slots has room for goes on in a wide bundle, alone or from among
others.  The same run in bundles of 256 slots, which hold the first case's fragments whole
and let go of the others' later, is the reference, bit for bit; fragments beyond the wide
bundle's 512 slots are reported."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.p3t import GpuSystem
from tests.test_bundle_sizes_gpu import FIELDS, clumps

pytestmark = pytest.mark.gpu


def _hard(sizes, f, dt_tree, frag, shape):
    g = GpuSystem(P3TParams(dt_tree=dt_tree))
    g.lib.p3t_set_schedule(0)
    try:
        assert g.lib.p3t_set_hard_bundle(*shape) == 0
        g.set_fragmentation(**frag)
        g.load(clumps(sizes, 1.0, f=f, kick=1e-4))
        g.set_r_planet()
        g.startup()
        g.kick()
        g.cluster()
        cols, ed = g.hard(1)
        return dict({k: g.get(k) for k in FIELDS}, cols=cols, ed=ed, cost=g.hard_costs(), id_next=g.id_next())
    finally:
        g.set_fragmentation(0.0)
        g.lib.p3t_set_hard_bundle(128, 3)


@pytest.mark.parametrize("sizes,n_frag,total", [([100], 5, 245), ([100], 10, 402), ([20] * 6, 10, 150),
                                                ([2] * 30 + [60, 30], 5, 205)])
def test_clusters_outgrow_their_bundle(gpu, sizes, n_frag, total):
    frag = dict(a_frag=0.5, n_frag=n_frag, m_min=5e-11 / n_frag, seed=11)
    got, want = (_hard(sizes, 20.0, 2.0**-9, frag, s) for s in ((128, 3), (256, 2)))
    assert len(want["id"]) == total and len(want["cols"]) > 0
    for k, v in want.items():
        assert np.asarray(got[k]).tobytes() == np.asarray(v).tobytes(), k


def test_more_than_the_wide_bundle_holds(gpu):
    with pytest.raises(RuntimeError, match="status bits 16"):
        _hard([100], 80.0, 2.0**-8, dict(a_frag=0.5, n_frag=10, m_min=5e-12, seed=11), (128, 3))
