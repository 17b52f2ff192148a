"""The bundle form at the edges of its sizes, bit for bit against the
one-cluster-per-team form: clusters of exactly n members around the warp, the
bundle (128 slots), the large bundle (256) and the wide form (512), many of them
at once and one alone; clumps in which every pair is live, whose pair list is
made in parts; a time step that is no power of two (the corrector's general
products); collisions in a clump (the list that a step cannot rely on is made
again, twins and their targets)."""
import ctypes

import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.p3t import GpuSystem

pytestmark = pytest.mark.gpu
FIELDS = ("pos", "vel", "acc_d", "jerk_d", "acc_s", "jerk_s", "phi_d", "phi_s", "mass", "r_planet", "time", "dt", "id",
          "dead", "merged", "n_cluster")


def clumps(sizes, spread, m=1e-10, f=1.0, seed=3, kick=0.0):
    """One clump of n bodies per entry of sizes, 0.3 rad apart on a circular
    orbit, positions within `spread` Hill radii of its centre on each axis
    (clumps of less than 16 within 0.9, so that any two of their bodies are
    closer than the search radius of 3.3: one cluster each)."""
    rng = np.random.default_rng(seed)
    h = (m / 3.0) ** (1.0 / 3.0)
    pos, vel, wide = [], [], spread
    for k, n in enumerate(sizes):
        spread = min(wide, 0.9) if n < 16 else wide
        ang = 0.3 * k + spread * h * rng.uniform(-1, 1, n)
        r = 1.0 + spread * h * rng.uniform(-1, 1, n)
        pos.append(np.stack([r * np.cos(ang), r * np.sin(ang), spread * h * rng.uniform(-1, 1, n)], 1))
        vel.append(np.stack([-np.sin(ang), np.cos(ang), np.zeros(n)], 1) / np.sqrt(r)[:, None]
                   + kick * rng.standard_normal((n, 3)))
    N = int(np.sum(sizes))
    return dict(id=np.arange(N, dtype=np.int64), mass=np.full(N, m), r_planet=np.zeros(N), f=np.full(N, f),
                pos=np.concatenate(pos), vel=np.concatenate(vel))


def both_forms(d, P, shapes=((128, 3, 1), (256, 2, 1), (128, 3, 0))):
    g = GpuSystem(P)
    g.lib.p3t_set_schedule(0)
    g.load(d)
    g.set_r_planet()
    g.startup()
    g.kick()
    g.cluster()
    off, _ = g.cluster_lists()
    nc = len(off) - 1
    assert g.lib.p3t_state_snapshot(0) == 0

    def run(mode):
        g.lib.p3t_set_hard_mode(mode)
        assert g.lib.p3t_state_snapshot(1) == 0
        cols, ed = g.hard(1)
        cost = np.zeros(2 * nc, np.int64)
        assert g.lib.p3t_hard_costs(cost.ctypes.data_as(ctypes.c_void_p), nc) == 0
        return dict({k: g.get(k) for k in FIELDS}, cols=cols, ed=ed, cost=cost)

    try:
        want = run(1)
        for cap, occ, wide in shapes:
            assert g.lib.p3t_set_hard_bundle(cap, occ) == 0 and g.lib.p3t_set_hard_wide(wide) == 0
            got = run(0)
            for k, v in want.items():
                assert got[k].tobytes() == v.tobytes(), (cap, wide, k)
    finally:
        g.lib.p3t_set_hard_mode(0)
        g.lib.p3t_set_hard_wide(1)
        g.lib.p3t_set_hard_bundle(128, 3)
    return np.diff(off), want


@pytest.mark.parametrize("sizes", [[2], [2] * 20, [3, 31, 32, 33, 2, 5], [63, 64, 65], [127, 2], [128], [129, 2], [256],
                                   [257, 4], [512], [513]])
def test_cluster_sizes(gpu, sizes):
    n, _ = both_forms(clumps(sizes, 3.0), P3TParams(dt_tree=2.0**-9))
    assert sorted(n) == sorted(sizes)


def test_every_pair_live(gpu):
    n, w = both_forms(clumps([128, 60, 256], 0.7), P3TParams(dt_tree=2.0**-10))
    assert sorted(n) == [60, 128, 256]


def test_time_step_not_a_power_of_two(gpu):
    # 3 x 2^-10 and its halvings: their sums stay exact, as the block steps need
    both_forms(clumps([2, 9, 40], 2.0), P3TParams(dt_tree=0.75 * 2.0**-8, dt_min=0.75 * 2.0**-30), shapes=((128, 3, 1),))


@pytest.mark.parametrize("sizes,f", [([2] * 12, 150.0), ([40, 90], 30.0), ([200], 20.0)])
def test_collisions(gpu, sizes, f):
    n, w = both_forms(clumps(sizes, 1.0, f=f, kick=1e-4), P3TParams(dt_tree=2.0**-9))
    assert len(w["cols"]) > 0
