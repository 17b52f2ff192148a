"""The cutoff correction's pair pass where a CTA takes two, three or four list entries a thread
(from 2, 3 and 4 x 1024 entries per SM on) and sorts them in as many turns: whole CTAs of pairs
inside r_out, of pairs between r_out and r_search, and mixed ones.  Against the CPU oracle in the
initial and the later form: neighbour pairs exactly; FP64 quantities from identical inputs 1e-12
relative (log of the CUDA math library)."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import FORCE_DTYPE
from gplum_gb300.p3t import GpuSystem, VP
from gplum_gb300 import _lib
from oracle import harness as H
from tests.test_step_gpu import pair_set, sync_state

pytestmark = pytest.mark.gpu
R_OUT, R_SEARCH, CLUMP = 1e-3, 1.5e-3, 120


def _lattice(n, step, base):
    k = np.arange(n)
    return np.array(base) + step * np.stack([k % 8, k // 8 % 8, k // 64], 1)


def bodies(n_clumps, rng):
    """Clumps whose pairs all lie inside r_out and clumps of pairs on both sides of r_out and
    r_search in turn, then 600 separate pairs between r_out and r_search."""
    width = np.where(np.arange(n_clumps) % 4 < 2, 0.5e-3, 1.6e-3)[:, None, None]
    c = _lattice(n_clumps, 8e-3, [1.0, 0.0, 0.0])[:, None] + width * (rng.random((n_clumps, CLUMP, 3)) - 0.5)
    a = _lattice(600, 6e-3, [1.0, 0.0, 0.2])
    d = rng.standard_normal((600, 3))
    b = a + 1.25e-3 * d / np.linalg.norm(d, axis=1)[:, None]
    pos = np.concatenate([c.reshape(-1, 3), np.stack([a, b], 1).reshape(-1, 3)])
    n = len(pos)
    return dict(id=np.arange(n, dtype=np.int64), mass=1e-11 * rng.uniform(0.5, 2.0, n), r_planet=1e-8 * np.ones(n),
                f=np.ones(n), pos=pos, vel=np.array([0.0, 1.0, 0.0]) + 2e-3 * rng.standard_normal((n, 3)))


@pytest.mark.parametrize("per", [1, 2, 3, 4])
def test_entries_per_thread(gpu, per):
    import torch

    full = 128 * 8 * torch.cuda.get_device_properties(0).multi_processor_count
    # a clump of either kind lists 4/5 of its CLUMP (CLUMP - 1) entries or more
    d = bodies(int((per + 0.3) * full / (0.9 * CLUMP * (CLUMP - 1))), np.random.default_rng(per))
    n, P = len(d["id"]), P3TParams()
    orc, g = H.CpuSystem("orc", P), GpuSystem(P, cand_cap=128)
    lf = H.tree_lists_fn(P)
    for s in (orc, g):
        s.load(d)
        s.prepare()
        for k, v in (("r_out", R_OUT), ("r_out_inv", 1.0 / R_OUT), ("r_search", R_SEARCH)):
            s.set(k, np.full(n, v))
    sync_state(orc, g, ("r_out", "r_out_inv", "r_search", "v_disp", "r_planet"))
    for initial in (True, True, False):
        L = lf(orc)
        orc.soft_force(L)
        g.soft_force(L)
        f = np.zeros(n, FORCE_DTYPE)
        _lib.check(g.lib.p3t_download_forces(f.ctypes.data_as(VP), n), "p3t_download_forces")
        assert min(4, int(f["number"].sum()) // full) == per  # the entries a thread takes
        orc.correct(initial)
        g.correct(initial)
        np.testing.assert_array_equal(g.get("number"), orc.get("number"))
        assert pair_set(g) == pair_set(orc)
        if initial:
            for k in ("acc_d", "jerk_d", "acc_s", "jerk_s", "dt", "acc0", "phi_d"):
                a, b = g.get(k), orc.get(k)
                assert np.all(np.abs(a - b) <= 1e-12 * np.abs(b).max()), k
            sync_state(orc, g)
    assert len(pair_set(g)) > 1000
