"""The device tree at the edges of its parts, against the host builder entry for
entry: body counts around one leaf, one scan tile and one radix tile (2048);
leaf limits on both sides of the two ways to find a body's levels (16); bodies
at one place (21 levels, a leaf above its limit) and close pairs (deep chains
of small levels).  The bound of the moments: the device adds children's
moments where the host adds bodies, at most n terms of 2^-53 each."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams, make_disk
from gplum_gb300.p3t import GpuSystem
from gplum_gb300.tree import build_lists

pytestmark = pytest.mark.gpu


def check(d, leaf, group):
    P = P3TParams(n_leaf_limit=leaf, n_group_limit=group)
    g = GpuSystem(P)
    g.load(d)
    g.set_r_planet()
    g.prepare()
    D = g.tree_lists(build=True)
    H = build_lists(g.get("pos"), g.get("mass"), g.get("r_search"), P.theta, leaf, group)
    assert D["n_group"] == H["n_group"]
    for k in ("i_off", "i_idx", "j_off", "j_idx", "s_off"):
        np.testing.assert_array_equal(D[k], H[k], err_msg=k)
    ds, hs = D["spj"][D["s_idx"]], H["spj"][H["s_idx"]]
    tol = len(d["mass"]) * 2.0**-53 + 2.0**-50
    np.testing.assert_allclose(ds["mass"], hs["mass"], rtol=tol)
    np.testing.assert_allclose(ds["pos"], hs["pos"], rtol=tol, atol=tol * max(1.0, np.abs(hs["pos"]).max(initial=0.0)))
    return D


@pytest.mark.parametrize("n", [1, 2, 8, 9, 255, 257, 2047, 2048, 2049, 4097, 20011])
def test_body_counts(gpu, n):
    check(make_disk(n, 1e-9, 0.9, 1.1, seed=n), 8, 64)


@pytest.mark.parametrize("leaf,group", [(1, 1), (1, 64), (16, 64), (17, 64), (64, 256), (300, 256)])
def test_leaf_limits(gpu, leaf, group):
    check(make_disk(5003, 1e-9, 0.9, 1.1, seed=31), leaf, group)


@pytest.mark.parametrize("copies,gap", [(3, 0.0), (40, 0.0), (2, 1e-12), (12, 1e-9)])
def test_bodies_at_one_place(gpu, copies, gap):
    d = make_disk(3001, 1e-9, 0.9, 1.1, seed=32)
    rng = np.random.default_rng(33)
    for c in (100, 1700):  # two clumps
        d["pos"][c:c + copies] = d["pos"][c] + gap * rng.uniform(-1, 1, (copies, 3))
    check(d, 8, 64)
