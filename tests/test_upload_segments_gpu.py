"""List and state uploads as one launch that reads the caller's arrays (16-byte and 4-byte
pieces, tails of every length), and as copies where an array is not aligned to 4 bytes: the same
device state from the same bytes, exactly."""
import ctypes

import numpy as np
import pytest

from gplum_gb300 import _lib
from gplum_gb300.disk import P3TParams, make_disk
from gplum_gb300.layout import FORCE_DTYPE
from gplum_gb300.p3t import GpuSystem
from gplum_gb300.soft import SoftForce
from tests.test_walks_gpu import _at, _problem

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


@pytest.mark.parametrize("shift", [0, 4, 8, 12, 2, 1])
def test_list_upload(gpu, shift):
    epj, L = _problem(9)
    sf = SoftForce(P3TParams())
    sf.upload_particles(epj)
    sf.upload_lists(L)
    sf.run()
    want = sf.download().copy()
    keep = {k: _at(L[k], shift) for k in ("i_off", "i_idx", "j_off", "j_idx", "s_off", "s_idx", "spj")}
    p = {k: VP(v[1]) for k, v in keep.items()}
    _lib.check(sf.lib.p3t_upload_lists(L["n_group"], p["i_off"], p["i_idx"], p["j_off"], p["j_idx"], p["s_off"],
                                       p["s_idx"], p["spj"], len(L["spj"])), "p3t_upload_lists")
    for raw, _ in keep.values():
        raw[:] = 0xFF
    sf.run()
    assert sf.download(np.zeros(len(epj), FORCE_DTYPE)).tobytes() == want.tobytes()


@pytest.mark.parametrize("n", [1, 3, 1021, 70001])
@pytest.mark.parametrize("shift", [0, 8, 4, 1])
def test_state_load(gpu, n, shift):
    d = make_disk(n, 1e-9, 0.9, 1.1, seed=3)
    g = GpuSystem(P3TParams())
    names = (("id", np.int64), ("mass", np.float64), ("r_planet", np.float64), ("f", np.float64), ("pos", np.float64),
             ("vel", np.float64))
    keep = [_at(np.ascontiguousarray(d[k], dtype=t), shift) for k, t in names]
    _lib.check(g.lib.p3t_state_load(n, *(VP(k[1]) for k in keep)), "p3t_state_load")
    for raw, _ in keep:
        raw[:] = 0xFF
    for k, t in names:
        if k != "f":
            assert np.array_equal(g.get(k), np.asarray(d[k], dtype=t)), k
