"""The cutoff correction's pair pass at the sizes where its work changes shape: one pair, a
CTA's list entries and one more, several entries per thread, pairs inside r_out, between it
and r_search and beyond the neighbour test's critical distance, and bodies of different
masses (a pair's two sides share all but the mass).  Against the CPU oracle: neighbour pairs
exactly; FP64 quantities from identical inputs 1e-12 relative (log of the CUDA math library)."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.p3t import GpuSystem
from oracle import harness as H
from tests.common import rel_err
from tests.test_step_gpu import pair_set, sync_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,size", [(2, 1e-3), (12, 2e-3), (13, 2e-3), (129, 4e-3), (700, 8e-3)])
def test_pair_terms(gpu, n, size):
    P = P3TParams()
    rng = np.random.default_rng(n)
    mass = 1e-9 * rng.uniform(0.5, 2.0, n)
    pos = np.array([1.0, 0.0, 0.0]) + size * (rng.random((n, 3)) - 0.5)
    vel = np.array([0.0, 1.0, 0.0]) + 2e-3 * rng.standard_normal((n, 3))
    d = dict(id=np.arange(n, dtype=np.int64), mass=mass, r_planet=1e-7 * np.ones(n), f=np.ones(n), pos=pos, vel=vel)
    orc, g = H.CpuSystem("orc", P), GpuSystem(P)
    lf = H.tree_lists_fn(P)
    for s in (orc, g):
        s.load(d)
        s.prepare()
    sync_state(orc, g, ("r_out", "r_out_inv", "r_search", "v_disp", "r_planet"))
    listed = 0
    for initial in (True, True, False):
        L = lf(orc)
        orc.soft_force(L)
        g.soft_force(L)
        orc.correct(initial)
        g.correct(initial)
        np.testing.assert_array_equal(g.get("number"), orc.get("number"))
        assert pair_set(g) == pair_set(orc)
        listed = max(listed, len(pair_set(g)))
        if initial:
            for k in ("acc_d", "jerk_d", "acc_s", "jerk_s", "dt", "acc0", "phi_d"):
                a, b = g.get(k), orc.get(k)
                assert np.all(np.abs(a - b) <= 1e-12 * np.abs(b).max()), k
            sync_state(orc, g)
    assert listed > 0
