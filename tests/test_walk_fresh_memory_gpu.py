"""A retrieve into memory that nobody has written yet: the same records as into used memory, and
no slower than a retrieve into used memory and a host copy of as many bytes into fresh memory
together (with half as much again for the spread; a kernel that touches the pages first takes
twice that)."""
import ctypes
import mmap
import time

import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import FORCE_DTYPE
from gplum_gb300.soft import configure
from tests.test_walk_forces_gpu import _dispatch, _problem

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


def test_retrieve_into_fresh_memory(gpu):
    n = 6200
    lib = configure(P3TParams())
    epj, L = _problem(n, 1)
    used = np.zeros(n, FORCE_DTYPE)
    used["phi"] = 1.0
    best, held = dict(used=1.0, fresh=1.0, host=1.0), []
    for _ in range(12):
        for kind in ("used", "fresh"):
            cnt = _dispatch(lib, 0, epj, L)
            lib.p3t_synchronize()
            out = used if kind == "used" else np.frombuffer(mmap.mmap(-1, n * 32), FORCE_DTYPE)
            held.append(out)
            p = (VP * L["n_group"])(*[out.ctypes.data + 32 * int(o) for o in L["i_off"][:-1]])
            c = VP(cnt.ctypes.data)
            t = time.perf_counter()
            st = lib.p3t_soft_retrieve(0, L["n_group"], c, p)
            best[kind] = min(best[kind], time.perf_counter() - t)
            assert st == 0
        assert held[-1].tobytes() == used.tobytes()
        fresh = np.frombuffer(mmap.mmap(-1, n * 32), FORCE_DTYPE)
        held.append(fresh)
        t = time.perf_counter()
        ctypes.memmove(fresh.ctypes.data, used.ctypes.data, n * 32)
        best["host"] = min(best["host"], time.perf_counter() - t)
    assert best["fresh"] <= 1.5 * (best["used"] + best["host"]), best
