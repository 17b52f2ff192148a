"""The hard launch's time where clusters are large or few, against the same launch in another
form on the same box (the states of both are bit-identical, tests/test_bundle_sizes_gpu.py):
a lone cluster of 300 and of 500 bodies with all pairs live, a lone cluster above the wide bundle's
slots, and copies of one cluster, which run side by side where SMs are free."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.p3t import GpuSystem

pytestmark = pytest.mark.gpu


def clump(n, copies=1, spread=3.0, m=1e-10, seed=5):
    """`copies` of one clump of n bodies on a circular orbit, 0.3 rad apart, positions within
    `spread` Hill radii of its centre on each axis."""
    rng = np.random.default_rng(seed)
    h = (m / 3.0) ** (1.0 / 3.0)
    a, r, z = (spread * h * rng.uniform(-1, 1, n) for _ in range(3))
    a = (a[None] + 0.3 * np.arange(copies)[:, None]).reshape(-1)
    r, z = np.tile(1.0 + r, copies), np.tile(z, copies)
    N = n * copies
    return dict(id=np.arange(N, dtype=np.int64), mass=np.full(N, m), r_planet=np.zeros(N), f=np.full(N, 1e-3),
                pos=np.stack([r * np.cos(a), r * np.sin(a), z], 1),
                vel=np.stack([-np.sin(a), np.cos(a), np.zeros(N)], 1) / np.sqrt(r)[:, None])


def hard_ms(d, clusters, mode=0):
    g = GpuSystem(P3TParams(dt_tree=2.0**-9))
    g.lib.p3t_set_schedule(0)
    assert g.lib.p3t_set_hard_bundle(128, 3) == 0 and g.lib.p3t_set_hard_wide(1) == 0
    g.load(d)
    g.set_r_planet()
    g.startup()
    g.kick()
    g.cluster()
    assert len(g.cluster_lists()[0]) - 1 == clusters
    assert g.lib.p3t_state_snapshot(0) == 0
    ms = []
    try:
        g.lib.p3t_set_hard_mode(mode)
        for _ in range(3):
            assert g.lib.p3t_state_snapshot(1) == 0
            g.hard(1)
            ms.append(g.hard_launch_stats()["ms"])
    finally:
        g.lib.p3t_set_hard_mode(0)
    return min(ms)


@pytest.mark.parametrize("n,most", [(300, 0.30), (500, 0.33)])
def test_lone_wide_cluster(gpu, n, most):
    """Against 128 threads a cluster (0.22 and 0.24 of its time; with one target's sums at a
    time 0.38 and 0.47)."""
    d = clump(n)
    assert hard_ms(d, 1) <= most * hard_ms(d, 1, mode=1)


def test_lone_cluster_above_the_wide_bundle(gpu):
    """In 512 threads against 128 (0.84 of their time; in 256, 0.99)."""
    d = clump(600)
    assert hard_ms(d, 1) <= 0.92 * hard_ms(d, 1, mode=1)


def test_copies_run_side_by_side(gpu):
    """Eight copies of a cluster of 100 take as long as one (one after the other: eight times)."""
    assert hard_ms(clump(100, 8), 8) <= 3.0 * hard_ms(clump(100), 1)
