"""The one-call host form at the size from which it computes groups as their bodies arrive
(524,288 bodies, 4,500 groups) and one body below: the bits of the resident form on the same
lists (the same kernels in another order), for bodies in the groups' order and in a random one
(where most groups need the last part), results in pinned and in pageable memory, both
precisions, and an entry out of range reported."""
import numpy as np
import pytest

from gplum_gb300 import _lib
from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPJ_DTYPE, FORCE_DTYPE, SPJ_DTYPE
from gplum_gb300.soft import SoftForce, configure, soft_force_host

pytestmark = pytest.mark.gpu


def _problem(n, ng, shuffled):
    rng = np.random.default_rng(n)
    epj = np.zeros(n, EPJ_DTYPE)
    epj["pos"] = rng.random((n, 3))
    epj["mass"] = rng.random(n) * 1e-9
    epj["r_out"], epj["r_search"] = 1e-2, 2e-2
    epj["id_local"] = np.arange(n)
    spj = np.zeros(500, SPJ_DTYPE)
    spj["pos"], spj["mass"] = rng.random((500, 3)) + 2.0, 1e-8
    cut = np.linspace(0, n, ng + 1).astype(np.int32)
    nj = rng.integers(0, 80, ng)
    j_off = np.concatenate([[0], np.cumsum(nj)]).astype(np.int32)
    s_off = (np.arange(ng + 1) * 9).astype(np.int32)
    near = np.repeat(cut[:-1], nj) + rng.integers(-300, 300, j_off[-1])
    i_idx, j_idx = np.arange(n), np.clip(near, 0, n - 1)
    if shuffled:
        perm = rng.permutation(n)
        i_idx, j_idx = perm[i_idx], perm[j_idx]
    return epj, dict(n_group=ng, i_off=cut, j_off=j_off, s_off=s_off, i_idx=i_idx.astype(np.int32),
                     j_idx=j_idx.astype(np.int32), s_idx=rng.integers(0, 500, s_off[-1]).astype(np.int32), spj=spj)


@pytest.mark.parametrize("n,ng", [(524288, 4500), (524287, 4500), (524293, 4499), (600001, 9001)])
@pytest.mark.parametrize("shuffled,precision", [(False, 0), (True, 0), (False, 1)])
def test_staged_host_call(gpu, n, ng, shuffled, precision):
    import torch

    P = P3TParams()
    epj, L = _problem(n, ng, shuffled)
    sf = SoftForce(P, precision=precision)
    sf.upload_particles(epj)
    sf.upload_lists(L)
    sf.run()
    want = sf.download().copy()
    for pinned in (True, False):
        out = np.zeros(n, FORCE_DTYPE)
        if pinned:
            out = torch.empty(n * 32, dtype=torch.uint8, pin_memory=True).numpy().view(FORCE_DTYPE)
        got = soft_force_host(P, epj, L, precision=precision, out=out)
        assert got.tobytes() == want.tobytes()
        res = np.zeros(n, FORCE_DTYPE)  # the resident copy
        _lib.check(sf.lib.p3t_download_forces(res.ctypes.data_as(_lib.ctypes.c_void_p), n), "p3t_download_forces")
        assert res.tobytes() == want.tobytes()


def test_entry_out_of_range(gpu):
    epj, L = _problem(524288, 4500, False)
    L["j_idx"][-1] = len(epj)
    with pytest.raises(RuntimeError, match="status 2"):
        soft_force_host(P3TParams(), epj, L)
    configure(P3TParams())
