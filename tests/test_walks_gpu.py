"""The multiwalk and functor calls read the walks' records in the caller's memory, or through
a pinned copy where they are not aligned for the device: both, record and index form, in
both precisions, give the bits of the one-call host form on the same lists (the same kernels
on the same values, so no tolerance).  Walks of 0 to 300 entries cover the tiles' edges."""
import ctypes

import numpy as np
import pytest

from gplum_gb300 import _lib
from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPI_DTYPE, EPJ_DTYPE, FORCE_DTYPE, SPJ_DTYPE
from gplum_gb300.soft import configure, epi_records, soft_force_host

pytestmark = pytest.mark.gpu
VP = ctypes.c_void_p
SIZES = [(1, 0, 0), (1, 1, 1), (0, 5, 5), (127, 128, 129), (128, 129, 0), (130, 0, 127), (2, 300, 257), (33, 256, 255)]


def _problem(seed):
    rng = np.random.default_rng(seed)
    n, ns = 600, 400
    epj = np.zeros(n, EPJ_DTYPE)
    epj["pos"] = rng.standard_normal((n, 3)) * 0.01 + [1.0, 0, 0]
    epj["mass"] = rng.random(n) * 1e-9
    epj["r_out"], epj["r_search"] = 1e-3, 1e-3 + 2e-3 * rng.random(n)
    epj["id_local"], epj["myrank"] = np.arange(n), rng.integers(0, 3, n)
    spj = np.zeros(ns, SPJ_DTYPE)
    spj["pos"] = rng.standard_normal((ns, 3)) + [1.0, 0, 0]
    for k in ("mass", "xx", "yy", "zz", "xy", "xz", "yz"):
        spj[k] = rng.random(ns) * 1e-7
    off = {k: np.concatenate([[0], np.cumsum([s[i] for s in SIZES])]).astype(np.int32)
           for i, k in enumerate(("i_off", "j_off", "s_off"))}
    L = dict(off, n_group=len(SIZES), spj=spj, i_idx=rng.permutation(n)[:off["i_off"][-1]].astype(np.int32),
             j_idx=rng.integers(0, n, off["j_off"][-1]).astype(np.int32),
             s_idx=rng.integers(0, ns, off["s_off"][-1]).astype(np.int32))
    return epj, L


def _at(a, shift):
    """A copy of `a` that starts `shift` bytes past a 16-byte boundary: (owner, address)."""
    raw = np.zeros(a.nbytes + 32, np.uint8)
    o = -raw.ctypes.data % 16 + shift
    raw[o:o + a.nbytes] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    return raw, raw.ctypes.data + o


def _ptrs(base, size, offs):
    return (VP * (len(offs) - 1))(*[base + int(o) * size for o in offs[:-1]])


def _ints(a):
    return a.ctypes.data_as(VP)


def _walks(lib, epj, L, index, shift, send=1, tag=3):
    ei = epi_records(epj)[L["i_idx"]]
    js = L["j_idx"] if index else epj[L["j_idx"]]
    ss = L["s_idx"] if index else L["spj"][L["s_idx"]]
    keep = [_at(a, s) for a, s in ((ei, shift), (js, shift // 2 if index else shift), (ss, shift // 2 if index else shift),
                                   (epj, shift), (L["spj"], shift))]
    p = [_ptrs(k[1], a.dtype.itemsize, L[o]) for k, a, o in zip(keep, (ei, js, ss), ("i_off", "j_off", "s_off"))]
    cnt = [np.ascontiguousarray(np.diff(L[o])) for o in ("i_off", "j_off", "s_off")]
    force = np.zeros(len(ei), FORCE_DTYPE)
    force["phi"] = 7.0
    args = (tag, L["n_group"], p[0], _ints(cnt[0]), p[1], _ints(cnt[1]), p[2], _ints(cnt[2]))
    if index:
        st = lib.p3t_soft_dispatch_index(*args, VP(keep[3][1]), len(epj), VP(keep[4][1]), len(L["spj"]), send)
    else:
        st = lib.p3t_soft_dispatch(*args)
    _lib.check(st, "dispatch")
    for raw, _ in keep:
        raw[:] = 0xFF  # the records are the caller's again
    _lib.check(lib.p3t_soft_retrieve(tag, L["n_group"], _ints(cnt[0]), _ptrs(force.ctypes.data, 32, L["i_off"])), "retrieve")
    return force


def _same(got, want, what):
    for k in ("acc", "phi", "number", "rank", "id_max", "id_min"):
        np.testing.assert_array_equal(got[k], want[k], err_msg="%s %s" % (what, k))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("index", [False, True])
def test_walks_in_place_and_staged(gpu, index, precision):
    P = P3TParams()
    epj, L = _problem(5)
    want = soft_force_host(P, epj, L, precision=precision)[L["i_idx"]]
    lib = configure(P, precision)
    for shift in (0, 8, 4, 1):
        _same(_walks(lib, epj, L, index, shift), want, shift)


def test_index_form_keeps_its_records_over_other_settings(gpu):
    """The records sent once serve dispatches with another softening, trace form and precision."""
    epj, L = _problem(6)
    lib = configure(P3TParams())
    _walks(lib, epj, L, True, 0)
    for P, precision, trace in ((P3TParams(eps2=1e-5), 0, 0), (P3TParams(eps2=1e-5), 0, 1), (P3TParams(), 1, 1), (P3TParams(), 0, 0)):
        want = soft_force_host(P, epj, L, precision=precision, trace_mode=trace)[L["i_idx"]]
        lib = configure(P, precision, trace)
        _same(_walks(lib, epj, L, True, 0, send=0), want, (precision, trace))


@pytest.mark.parametrize("precision", [0, 1])
def test_functors_in_place_and_staged(gpu, precision):
    epj, L = _problem(7)
    lib = configure(P3TParams(), precision)
    epi = epi_records(epj)
    out = []
    for shift in (0, 4):
        f = np.zeros(130, FORCE_DTYPE)
        f["id_max"], f["id_min"] = -1, 2**31 - 1
        (k0, i), (k1, j), (k2, s) = _at(epi[:130], shift), _at(epj[:257], shift), _at(L["spj"][:129], shift)
        _lib.check(lib.p3t_epep(VP(i), 130, VP(j), 257, _ints(f)), "p3t_epep")
        _lib.check(lib.p3t_epsp(VP(i), 130, VP(s), 129, _ints(f)), "p3t_epsp")
        out.append(f)
    _same(out[1], out[0], "staged")
    assert np.any(out[0]["acc"] != 0)


def test_bad_indices_stay_with_their_dispatch(gpu):
    """Two walks in flight, the first with a list entry out of range: its retrieve reports it, the other's does not."""
    epj, L = _problem(8)
    P = P3TParams()
    want = soft_force_host(P, epj, L)[L["i_idx"]]
    lib = configure(P)
    bad = dict(L, j_idx=L["j_idx"].copy())
    bad["j_idx"][-1] = len(epj)
    with pytest.raises(Exception):
        _walks(lib, epj, bad, True, 0)
    _same(_walks(lib, epj, L, True, 0), want, "after")
