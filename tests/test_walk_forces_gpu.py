"""Forces of a dispatch large enough to stay on the device until the retrieve (192 KB, 6,144
records): written by the device into the caller's arrays, contiguous or apart, or through a
pinned copy where an array is not aligned for it; one record below that size; two dispatches in
flight; a retrieve that asks for more than the dispatch covered.  The bits of the one-call form
on the same lists (the same kernel on the same values)."""
import ctypes

import numpy as np
import pytest

from gplum_gb300 import _lib
from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPJ_DTYPE, FORCE_DTYPE, SPJ_DTYPE
from gplum_gb300.soft import configure, epi_records, soft_force_host

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p


def _problem(n, seed):
    rng = np.random.default_rng(seed)
    epj = np.zeros(n, EPJ_DTYPE)
    epj["pos"] = rng.standard_normal((n, 3)) * 0.05 + [1.0, 0, 0]
    epj["mass"] = rng.random(n) * 1e-9
    epj["r_out"], epj["r_search"] = 1e-3, 2e-3
    epj["id_local"] = np.arange(n)
    cut = np.unique(np.concatenate([[0, 1, n], rng.integers(1, n, 600)])).astype(np.int32)
    ng = len(cut) - 1
    j_off = (np.arange(ng + 1) * 40).astype(np.int32)
    L = dict(n_group=ng, i_off=cut, j_off=j_off, s_off=np.zeros(ng + 1, np.int32), spj=np.zeros(1, SPJ_DTYPE),
             i_idx=np.arange(n, dtype=np.int32), j_idx=rng.integers(0, n, j_off[-1]).astype(np.int32),
             s_idx=np.zeros(0, np.int32))
    return epj, L


def _dispatch(lib, tag, epj, L):
    ng = L["n_group"]
    ei, js = np.ascontiguousarray(epi_records(epj)[L["i_idx"]]), np.ascontiguousarray(epj[L["j_idx"]])
    cnt = [np.ascontiguousarray(np.diff(L[o])) for o in ("i_off", "j_off", "s_off")]
    p = [(VP * ng)(*[a.ctypes.data + int(o) * a.dtype.itemsize for o in L[k][:-1]]) for a, k in ((ei, "i_off"), (js, "j_off"))]
    _lib.check(lib.p3t_soft_dispatch(tag, ng, p[0], VP(cnt[0].ctypes.data), p[1], VP(cnt[1].ctypes.data),
                                     (VP * ng)(), VP(cnt[2].ctypes.data)), "p3t_soft_dispatch")
    return cnt[0]


def _same(got, want):
    for k in ("acc", "phi", "number", "rank", "id_max", "id_min"):
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)


@pytest.mark.parametrize("n", [6143, 6144, 20001])
@pytest.mark.parametrize("gap,shift", [(0, 0), (96, 4), (32, 2)])
def test_forces_reach_the_callers_arrays(gpu, n, gap, shift):
    P = P3TParams()
    lib = configure(P)
    sets = [_problem(n, s) for s in (1, 2)]
    want = [soft_force_host(P, epj, L)[L["i_idx"]] for epj, L in sets]
    lib = configure(P)
    cnt = [_dispatch(lib, t, epj, L) for t, (epj, L) in enumerate(sets)]
    for t, (epj, L) in enumerate(sets):
        ng = L["n_group"]
        at = L["i_off"][:-1].astype(np.int64) * 32 + np.arange(ng) * gap + shift
        raw = np.full(n * 32 + ng * gap + 64, 0x5A, np.uint8)
        st = lib.p3t_soft_retrieve(t, ng, VP(cnt[t].ctypes.data), (VP * ng)(*[raw.ctypes.data + int(o) for o in at]))
        _lib.check(st, "p3t_soft_retrieve")
        mine = np.zeros(len(raw), bool)
        for o, c in zip(at, cnt[t]):
            mine[o:o + 32 * int(c)] = True
        _same(raw[mine].view(FORCE_DTYPE), want[t])
        assert np.all(raw[~mine] == 0x5A)


def test_retrieve_beyond_the_dispatch(gpu):
    lib = configure(P3TParams())
    epj, L = _problem(7000, 3)
    cnt = _dispatch(lib, 5, epj, L)
    out = np.zeros(7000 + 8, FORCE_DTYPE)
    more = np.append(cnt, 8).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(more)])
    st = lib.p3t_soft_retrieve(5, len(more), VP(more.ctypes.data), (VP * len(more))(*[out.ctypes.data + 32 * int(o) for o in off[:-1]]))
    assert st == 2
    assert lib.p3t_soft_retrieve(5, len(cnt), VP(cnt.ctypes.data), (VP * len(cnt))()) == 2  # retrieved already


def test_status_of_dispatches_in_flight(gpu):
    """Two dispatches in flight, the first with an index out of range: its retrieve reports it and the
    other's does not; a status read between dispatch and retrieve reports it too, once."""
    lib = configure(P3TParams())
    epj, L = _problem(700, 4)
    ng = L["n_group"]
    cnt = np.ascontiguousarray(np.diff(L["i_off"]))
    ei = np.ascontiguousarray(epi_records(epj)[L["i_idx"]])
    nj, ns = np.ascontiguousarray(np.diff(L["j_off"])), np.zeros(ng, np.int32)
    out = np.zeros(700, FORCE_DTYPE)
    bad = L["j_idx"].copy()
    bad[5] = len(epj)

    def dispatch(tag, js, send):
        p = [(VP * ng)(*[a.ctypes.data + int(o) * a.dtype.itemsize for o in L[k][:-1]]) for a, k in ((ei, "i_off"), (js, "j_off"))]
        return lib.p3t_soft_dispatch_index(tag, ng, p[0], VP(cnt.ctypes.data), p[1], VP(nj.ctypes.data), (VP * ng)(),
                                           VP(ns.ctypes.data), VP(epj.ctypes.data), len(epj), VP(L["spj"].ctypes.data), 1, send)

    def retrieve(tag):
        return lib.p3t_soft_retrieve(tag, ng, VP(cnt.ctypes.data),
                                     (VP * ng)(*[out.ctypes.data + 32 * int(o) for o in L["i_off"][:-1]]))

    assert dispatch(0, bad, 1) == 0 and dispatch(1, L["j_idx"], 0) == 0
    assert retrieve(0) == 2 and retrieve(1) == 0
    assert dispatch(0, bad, 0) == 0
    assert lib.p3t_status() == 2 and lib.p3t_status() == 0
    assert retrieve(0) == 0
