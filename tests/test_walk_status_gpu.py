"""Status bits of multiwalk dispatches in flight: each retrieve reports its own dispatch's and no
other's, in either order and whatever is called in between; a dispatch that is never retrieved,
or not in full, leaves nothing to the slot's next one."""
import ctypes

import numpy as np
import pytest

from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import FORCE_DTYPE
from gplum_gb300.soft import configure, epi_records, soft_force_host
from tests.test_walk_forces_gpu import _problem

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


class Walks:
    """Index-form dispatches of one problem, with a list entry out of range or without."""

    def __init__(self, n=700):
        self.lib = configure(P3TParams())
        self.epj, self.L = _problem(n, 4)
        self.ei = np.ascontiguousarray(epi_records(self.epj)[self.L["i_idx"]])
        self.cnt, self.nj = (np.ascontiguousarray(np.diff(self.L[k])) for k in ("i_off", "j_off"))
        self.ng, self.out, self.keep = self.L["n_group"], np.zeros(n + 8, FORCE_DTYPE), []
        assert self.lib.p3t_status() in (0, 2)
        self.first = 1

    def dispatch(self, tag, bad):
        js = self.L["j_idx"].copy()
        if bad:
            js[5] = len(self.epj)
        self.keep.append(js)
        p = [(VP * self.ng)(*[a.ctypes.data + int(o) * a.dtype.itemsize for o in self.L[k][:-1]])
             for a, k in ((self.ei, "i_off"), (js, "j_off"))]
        ns = np.zeros(self.ng, np.int32)
        st = self.lib.p3t_soft_dispatch_index(tag, self.ng, p[0], VP(self.cnt.ctypes.data), p[1], VP(self.nj.ctypes.data),
                                              (VP * self.ng)(), VP(ns.ctypes.data), VP(self.epj.ctypes.data), len(self.epj),
                                              VP(self.L["spj"].ctypes.data), 1, self.first)
        self.first = 0
        assert st == 0

    def retrieve(self, tag, more=0):
        cnt = np.append(self.cnt, more).astype(np.int32) if more else self.cnt
        off = np.concatenate([[0], np.cumsum(cnt)])
        p = (VP * len(cnt))(*[self.out.ctypes.data + 32 * int(o) for o in off[:-1]])
        return self.lib.p3t_soft_retrieve(tag, len(cnt), VP(cnt.ctypes.data), p)


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
@pytest.mark.parametrize("bad", [(True, True), (True, False), (False, True)])
def test_each_retrieve_reports_its_own(gpu, order, bad):
    w = Walks()
    for tag in (0, 1):
        w.dispatch(tag, bad[tag])
    for tag in order:
        assert w.retrieve(tag) == (2 if bad[tag] else 0)
    assert w.lib.p3t_status() == 0


def test_other_calls_leave_the_bits(gpu):
    w = Walks()
    w.dispatch(3, True)
    soft_force_host(P3TParams(), w.epj, w.L)
    f = np.zeros(3, FORCE_DTYPE)
    assert w.lib.p3t_epep(VP(w.ei.ctypes.data), 3, VP(w.epj.ctypes.data), 10, VP(f.ctypes.data)) == 0
    assert w.retrieve(3) == 2
    assert w.lib.p3t_status() == 0


def test_dropped_and_short_retrieves(gpu):
    w = Walks()
    w.dispatch(2, True)  # never retrieved
    w.dispatch(2, False)
    assert w.retrieve(2) == 0
    assert w.lib.p3t_status() == 2 and w.lib.p3t_status() == 0  # the dropped one's bits
    w.dispatch(2, True)
    assert w.retrieve(2, more=8) == 2  # beyond the dispatch
    w.dispatch(2, False)
    assert w.retrieve(2) == 0
    assert w.lib.p3t_status() == 0
