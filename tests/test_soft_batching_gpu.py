"""A group's mixed soft force does not depend on the pass it is in: the forms by number of groups
(512, 256 and 128 threads a group) and the passes that emit candidates give the same bits, over
group sizes at the edges of the splits (32, 64, 128 bodies, and more than one turn) and list
lengths at the edges of the partial sums (16, 32), of the sub-blocks' turns (128) and of the
tiles (256, 512).  Exact equality: the same pair terms, summed in the same order."""
import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPJ_DTYPE, FORCE_DTYPE, SPJ_DTYPE
from gplum_gb300.soft import SoftForce

pytestmark = pytest.mark.gpu
NJ = [0, 1, 16, 17, 32, 33, 48, 127, 128, 129, 161, 255, 256, 257, 300, 511, 512, 513, 1040, 97]
NS = [513, 0, 1, 15, 31, 32, 256, 127, 512, 33, 0, 160, 2, 1025, 64, 96, 95, 128, 129, 511]


def _records(n, ns, rng):
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
    return epj, spj


def _run(sf, epj, spj, i, j, s, emit=False):
    """The forces of the groups whose bodies and lists are i[g], j[g], s[g]."""
    off = [np.concatenate([[0], np.cumsum([len(x) for x in l])]).astype(np.int32) for l in (i, j, s)]
    cat = [np.concatenate(l).astype(np.int32) if sum(map(len, l)) else np.zeros(0, np.int32) for l in (i, j, s)]
    sf.upload_particles(epj)
    sf.upload_lists(dict(n_group=len(i), i_off=off[0], j_off=off[1], s_off=off[2], i_idx=cat[0], j_idx=cat[1], s_idx=cat[2],
                         spj=spj))
    sf.run(emit_candidates=emit)
    return sf.download(np.zeros(len(epj), FORCE_DTYPE)).copy()


@pytest.mark.parametrize("ni", [1, 20, 32, 33, 61, 64, 65, 100, 128, 129, 300])
def test_forms_give_the_same_bits(gpu, ni):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(ni)
    epj, spj = _records(ni * len(NJ) + 4 * sms + 600, 700, rng)
    n = len(epj)
    i = [np.arange(ni) + ni * g for g in range(len(NJ))]
    j, s = [rng.integers(0, n, c) for c in NJ], [rng.integers(0, 700, c) for c in NS]
    # groups of one body that fill a pass up
    more = [np.array([k]) for k in range(ni * len(NJ), ni * len(NJ) + 3 * sms + 1)]
    none = [np.zeros(0, np.int64)] * len(more)
    sf = SoftForce(P3TParams())
    got = {}
    for name, k in (("512 threads", 0), ("256 threads", sms), ("128 threads", 3 * sms + 1)):
        got[name] = _run(sf, epj, spj, i + more[:k], j + none[:k], s + none[:k])
    got["alone"] = got["512 threads"].copy()
    for g in (3, 7, 13, 18):
        got["alone"][i[g]] = _run(sf, epj, spj, i[g:g + 1], j[g:g + 1], s[g:g + 1])[i[g]]
    sf = SoftForce(P3TParams(), cand_cap=1024)
    for name, k in (("512 threads, emitting", 0), ("256 threads, emitting", sms), ("128 threads, emitting", 3 * sms + 1)):
        got[name] = _run(sf, epj, spj, i + more[:k], j + none[:k], s + none[:k], emit=True)
    SoftForce(P3TParams())
    want = got.pop("128 threads")
    own = np.concatenate(i)
    assert np.any(want["acc"][own] != 0)
    for name, f in got.items():
        assert f[own].tobytes() == want[own].tobytes(), name
