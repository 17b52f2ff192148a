"""The mixed soft force in its forms by number of groups: 512, 256 and 128 threads a group
(one group; one group per SM and one more; three per SM and one more), over group sizes and
list lengths at the edges of the splits (32, 64, 128 bodies) and of the tiles (128, 256, 512
entries).  The pass that emits candidates always takes the 128-thread form, so it is the
reference: the same pair terms in partial sums of 32 or 16, so neighbour fields exactly equal
and forces apart by at most 32 roundings of 2^-24 of each body's sum of term magnitudes."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPJ_DTYPE, SPJ_DTYPE
from gplum_gb300.soft import SoftForce

pytestmark = pytest.mark.gpu
NI = [1, 32, 33, 64, 65, 128, 129, 20]
NJ = [0, 1, 16, 17, 128, 129, 255, 256, 257, 512, 513]
NS = [513, 0, 1, 15, 256, 127, 512, 33, 0]


@pytest.mark.parametrize("per_sm,more", [(0, 1), (1, 0), (1, 1), (3, 0), (3, 1)])
def test_forms_agree(gpu, per_sm, more):
    import torch

    ng = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(ng)
    n, ns = 3000, 700
    epj = np.zeros(n, EPJ_DTYPE)
    epj["pos"] = rng.standard_normal((n, 3)) * 0.02 + [1.0, 0.3, 0.0]
    epj["mass"] = 1e-9 * rng.random(n)
    epj["r_out"], epj["r_search"] = 2e-3, 2e-3 + 2e-3 * rng.random(n)
    epj["id_local"] = np.arange(n)
    spj = np.zeros(ns, SPJ_DTYPE)
    d = rng.standard_normal((ns, 3))
    spj["pos"] = epj["pos"].mean(0) + d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.3, 1.0, (ns, 1))
    spj["mass"] = 1e-8 * rng.random(ns)
    for k in ("xx", "yy", "zz", "xy", "xz", "yz"):
        spj[k] = spj["mass"] * 1e-3 * rng.uniform(-1, 1, ns)
    cnt = [np.array([s[(g + ng) % len(s)] for g in range(ng)], np.int32) for s in (NI, NJ, NS)]
    off = [np.concatenate([[0], np.cumsum(c)]).astype(np.int32) for c in cnt]
    # every group's bodies of its own where the bodies last; results of a body in two groups are not looked at
    i_idx = (np.arange(off[0][-1]) % n).astype(np.int32)
    L = dict(n_group=ng, i_off=off[0], j_off=off[1], s_off=off[2], i_idx=i_idx,
             j_idx=rng.integers(0, n, off[1][-1]).astype(np.int32),
             s_idx=rng.integers(0, ns, off[2][-1]).astype(np.int32), spj=spj)
    keep = min(ng, int(np.searchsorted(off[0], n, side="right")) - 1)
    L["n_group"], L["i_idx"] = ng, i_idx
    sf = SoftForce(P3TParams())
    sf.upload_particles(epj)
    sf.upload_lists(L)
    sf.run(emit_candidates=False)
    got = sf.download().copy()
    sf = SoftForce(P3TParams(), cand_cap=1024)
    sf.upload_particles(epj)
    sf.upload_lists(L)
    sf.run(emit_candidates=True)
    ref = sf.download().copy()
    SoftForce(P3TParams())
    once = np.bincount(i_idx, minlength=n) == 1
    for k in ("number", "rank", "id_max", "id_min"):
        np.testing.assert_array_equal(got[k][once], ref[k][once], err_msg=k)
    for g in range(keep):
        i = i_idx[off[0][g]:off[0][g + 1]]
        i = i[once[i]]
        j, s = L["j_idx"][off[1][g]:off[1][g + 1]], L["s_idx"][off[2][g]:off[2][g + 1]]
        x = epj["pos"][i][:, None]
        r2 = np.maximum(((x - epj["pos"][j][None]) ** 2).sum(-1), 4e-6)
        q2 = ((x - spj["pos"][s][None]) ** 2).sum(-1)
        mag = (epj["mass"][j] / r2).sum(1) + 2.0 * (spj["mass"][s] / q2).sum(1)
        pot = (epj["mass"][j] / np.sqrt(r2)).sum(1) + 2.0 * (spj["mass"][s] / np.sqrt(q2)).sum(1)
        assert np.all(np.abs(got["acc"][i] - ref["acc"][i]) <= 32 * 2.0**-24 * mag[:, None])
        assert np.all(np.abs(got["phi"][i] - ref["phi"][i]) <= 32 * 2.0**-24 * pot)
