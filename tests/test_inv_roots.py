"""The powers of 1 / sqrt(x) that the FP64 soft force takes from integer arithmetic
(csrc/p3t_exact.cuh), within 0.6 units of the last place; the FP64 soft force on
operands outside their range and with softening, against a float64 sum."""
import os
import subprocess

import numpy as np
import pytest

from gplum_gb300 import build
from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPJ_DTYPE, FORCE_DTYPE, SPJ_DTYPE

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cxx", "inv_roots.cpp")


def _run(cmd, exe, n):
    r = subprocess.run(cmd + ["-I", build.CSRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, str(n)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_powers_round_once(tmp_path):
    _run(["g++", "-O2", "-std=c++17", SRC], str(tmp_path / "roots"), 2000000)


@pytest.mark.gpu
def test_powers_round_once_on_the_device(gpu, tmp_path):
    _run([build._nvcc(), *build.ARCH, "-O2", "-std=c++17", "-x", "cu", SRC], str(tmp_path / "roots"), 1)


@pytest.mark.gpu
@pytest.mark.parametrize("ni", [1, 31, 33, 64, 65, 129, 257])
@pytest.mark.parametrize("scale,eps2", [(1.0, 0.0), (1.0, 1e-6), (1e-60, 0.0), (1e60, 0.0)])
def test_fp64_force_sizes_and_scales(gpu, ni, scale, eps2):
    """One group of ni bodies: the split forms of the kernel, tiles of 128 entries and one more, distances whose
    squares leave the integer range (1e-120, 1e120; monopoles only, as the quadrupoles' products overflow there) and coincident bodies held apart by r_out alone.  The results
    are float32 records: 2^-24 of the largest partial sums, for which 2e-6 of each body's sum of magnitudes is room."""
    from gplum_gb300.soft import SoftForce

    rng = np.random.default_rng(ni)
    n, ns = max(ni, 129) + 5, 131
    epj = np.zeros(n, EPJ_DTYPE)
    epj["pos"] = rng.standard_normal((n, 3)) * scale
    epj["pos"][1] = epj["pos"][0]
    epj["mass"] = rng.random(n) * scale * 1e-3 * scale
    epj["r_out"] = 0.05 * scale
    epj["r_search"] = 0.5 * scale * rng.random(n)
    epj["id_local"] = np.arange(n)
    spj = np.zeros(ns, SPJ_DTYPE)
    d = rng.standard_normal((ns, 3))
    spj["pos"] = (d / np.linalg.norm(d, axis=1)[:, None] * 8.0) * scale
    spj["mass"] = rng.random(ns) * 1e-3 * scale * scale
    for k in ("xx", "yy", "zz", "xy", "xz", "yz"):
        spj[k] = spj["mass"] * rng.uniform(-0.1, 0.1, ns) * (scale == 1.0)
    L = dict(n_group=1, i_off=np.array([0, ni], np.int32), j_off=np.array([0, n], np.int32),
             s_off=np.array([0, ns], np.int32), i_idx=np.arange(ni, dtype=np.int32),
             j_idx=np.arange(n, dtype=np.int32), s_idx=np.arange(ns, dtype=np.int32), spj=spj)
    sf = SoftForce(P3TParams(eps2=eps2), precision=1)
    sf.upload_particles(epj)
    sf.upload_lists(L)
    sf.run()
    f = sf.download(np.zeros(n, FORCE_DTYPE))[:ni]
    x = epj["pos"][:ni]
    r = (x[:, None] - epj["pos"][None]) / scale
    r2r = (r * r).sum(-1) + eps2 / scale**2
    r2 = np.maximum(r2r, 0.05**2)
    m = epj["mass"] / scale**2
    acc, phi = -(m / r2**1.5)[..., None] * r, -m / np.sqrt(r2)
    d = (spj["pos"][None] - x[:, None]) / scale
    q2 = (d * d).sum(-1) + eps2 / scale**2
    ms = spj["mass"] / scale**2
    xx, yy, zz, xy, xz, yz = (spj[k] for k in ("xx", "yy", "zz", "xy", "xz", "yz"))
    tr = xx + yy + xx
    Q = np.empty((ns, 3, 3))
    Q[:, 0, 0], Q[:, 1, 1], Q[:, 2, 2] = 3 * xx - tr, 3 * yy - tr, 3 * zz - tr
    Q[:, 0, 1] = Q[:, 1, 0] = 3 * xy
    Q[:, 0, 2] = Q[:, 2, 0] = 3 * xz
    Q[:, 1, 2] = Q[:, 2, 1] = 3 * yz
    qr = np.einsum("sab,isb->isa", Q, d)
    rqr = ((qr * d).sum(-1) - eps2 / scale**2 * tr) / q2**2
    sacc = ((ms + 2.5 * rqr) / q2**1.5)[..., None] * d - qr / (q2**2.5)[..., None]
    sphi = -(ms + 0.5 * rqr) / np.sqrt(q2)
    want, mag = acc.sum(1) + sacc.sum(1), np.abs(acc).sum(1) + np.abs(sacc).sum(1)
    assert np.all(np.abs(f["acc"] - want) <= 2e-6 * mag)
    if scale == 1.0:  # elsewhere the potential leaves the float32 range
        wphi, magp = phi.sum(1) + sphi.sum(1), np.abs(phi).sum(1) + np.abs(sphi).sum(1)
        assert np.all(np.abs(f["phi"] - wphi) <= 2e-6 * magp)
    rs2 = np.maximum(epj["r_search"][:ni, None], epj["r_search"][None]) ** 2 * 1.0201 / scale**2
    hit = (r2r < rs2) & ~np.eye(ni, n, dtype=bool)
    assert np.array_equal(f["number"], hit.sum(1))
