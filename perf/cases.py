"""Workloads of the P3T library, each through the entry points that a program calls.

A program uses the library in two ways.  A GPLUM/FDPS build hands it interaction lists: one group at a
time through the functors, walk by walk through the multiwalk pair (records or indices), a whole pass
from host buffers, or a whole pass on device buffers of its own.  A program that keeps the bodies on the
device calls the start-up and the tree step.  The cases cover both, from one group to two million bodies.

The disks are planetesimal annuli as in gplum_gb300/disk.py (surface density ~ a^-1.5, Rayleigh e and i
in reduced Hill radii, bulk density 2 g/cm^3, dt_tree = 2^-7), sampled on the GPU from the seed.
"""
import ctypes
import math

import numpy as np
import torch

from gplum_gb300 import _lib, autotune, scheduler
from gplum_gb300.disk import P3TParams
from gplum_gb300.layout import EPI_DTYPE, EPJ_DTYPE, FORCE_DTYPE, FPGRAV_DTYPE, SPJ_DTYPE, cleared_forces
from gplum_gb300.p3t import GpuSystem
from gplum_gb300.soft import SoftForce, configure, epi_records, epj_records, soft_force_host
from gplum_gb300.tree import build_lists

VP = ctypes.c_void_p


def listed():
    return [
        # FDPS without the multiwalk dispatch: one i-group's EPJ and SPJ lists through the two functor calls
        dict(name="functor_group", kind="functor", ni=61, nj=345, ns=324),
        # GPLUM's small run (3000 bodies, m = 1e-9, e = 2 h): every group of a soft pass in walks of 64 groups
        dict(name="multiwalk_3k", kind="multiwalk", n=3000, m=1e-9, a_in=0.95, a_out=1.05, ecc=2.0, group=64,
             theta=0.5, walk=64),
        # a mid-size soft pass in FDPS's index form: records travel once, walks name them by index
        dict(name="multiwalk_index_60k", kind="index", n=60001, m=1e-9, a_in=0.5, a_out=1.5, ecc=2.0, group=64,
             theta=0.5, walk=512),
        # the soft-force disk (m = 1e-10, 0.5-1.5 AU, groups of 256), one call from pinned host buffers
        dict(name="soft_host_1m", kind="host", n=1048576, m=1e-10, a_in=0.5, a_out=1.5, ecc=2.0, group=256,
             theta=0.5),
        # a caller with device buffers of its own that cannot allocate: the same pass on them
        dict(name="soft_device_20k", kind="noalloc", n=20011, m=1e-9, a_in=0.8, a_out=1.2, ecc=2.0, group=128,
             theta=0.5),
        # the plain FP64 form, as a check run uses it
        dict(name="soft_fp64_30k", kind="fp64", n=30000, m=1e-9, a_in=0.8, a_out=1.2, ecc=2.0, group=64, theta=0.5),
        # start-up of a run: radii, tree, soft force and first corrections, forces and derivatives read back
        dict(name="startup_300k", kind="startup", n=300007, m=1e-10, a_in=0.5, a_out=1.5, ecc=4.0, group=256,
             theta=0.5),
        # GPLUM's small run continued from its records: the restart pass and eight tree steps
        dict(name="steps_3k", kind="steps", n=3000, m=1e-9, a_in=0.95, a_out=1.05, ecc=2.0, group=64, theta=0.5,
             steps=8),
        # a crowded ring (rms e = 6 h, most bodies in neighbour clusters) of ordinary size, two steps
        dict(name="steps_ring_50k", kind="steps", n=50021, m=7e-11 * (1048576 / 50021) ** 1.5, a_in=0.95, a_out=1.05,
             ecc=6.0, group=256, theta=0.5, steps=2),
        # the crowded ring at a million bodies: the benchmark's disk, records in and out around one step
        dict(name="steps_ring_1m", kind="steps", n=1048576, m=7e-11, a_in=0.95, a_out=1.05, ecc=6.0, group=256,
             theta=0.5, steps=1),
        # planetesimals with four embryos and fragmenting collisions, from the start-up through two steps
        dict(name="embryos_200k", kind="embryos", n=200000, m=5e-10, a_in=0.5, a_out=1.5, ecc=6.0, group=256,
             theta=0.5, steps=2),
        # a wide disk (0.3-3 AU) of two million bodies, one step
        dict(name="steps_wide_2m", kind="steps", n=2097152, m=5e-11, a_in=0.3, a_out=3.0, ecc=4.0, group=256,
             theta=0.5, steps=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("functor", "multiwalk", "index", "host", "noalloc", "fp64", "startup", "steps", "steps",
                       "steps", "embryos"))
    if kind == "functor":
        return dict(kind=kind, ni=rng.randint(1, 256), nj=_log_int(rng, 16, 2048), ns=_log_int(rng, 16, 2048))
    lo, hi = {"multiwalk": (500, 20000), "index": (2000, 200000), "host": (5000, 1000000), "noalloc": (500, 65536),
              "fp64": (1000, 60000), "startup": (2000, 600000), "steps": (1000, 1000000),
              "embryos": (10000, 300000)}[kind]
    n = _log_int(rng, lo, hi)
    c = dict(kind=kind, n=n, ecc=round(rng.uniform(2.0, 6.0), 2), group=rng.choice((64, 128, 256)),
             theta=round(rng.uniform(0.4, 0.7), 2))
    if kind in ("multiwalk", "index"):
        c["walk"] = rng.choice((16, 64, 200, 512))
    if kind == "steps":
        # up to the crowded ring's mass, above which the neighbour graph percolates
        c.update(a_in=0.95, a_out=1.05, m=7e-11 * (1048576 / n) ** 1.5 * math.exp(rng.uniform(math.log(0.02), 0.0)),
                 steps=max(1, min(8, 100000 // n)))
    else:
        # the wide annuli keep the bench's disk mass of 1e-4 at most
        c.update(a_in=0.5, a_out=1.5, m=1e-10 * min(10.0, 1048576 / n))
        if kind == "embryos":
            c.update(m=1e-10 * min(5.0, 1048576 / n), steps=max(1, min(4, 100000 // n)))
    return c


# ---- inputs ------------------------------------------------------------------------------------------
def _sample(n, m, a_in, a_out, ecc, gen, a=None):
    """Positions and velocities of n bodies (gplum_gb300/disk.py make_disk's distributions), on the GPU."""
    def u():
        return torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)

    h = (m / 3.0) ** (1.0 / 3.0)
    a = (math.sqrt(a_in) + u() * (math.sqrt(a_out) - math.sqrt(a_in))) ** 2 if a is None else a
    e = ecc * h * torch.sqrt(-torch.log1p(-u()))
    inc = 0.5 * ecc * h * torch.sqrt(-torch.log1p(-u()))
    l, w, W = (2 * math.pi * u() for _ in range(3))
    E = l + e * torch.sin(l)
    for _ in range(12):
        E = E - (E - e * torch.sin(E) - l) / (1.0 - e * torch.cos(E))
    cw, sw, cW, sW, ci, si = w.cos(), w.sin(), W.cos(), W.sin(), inc.cos(), inc.sin()
    P = torch.stack([cw * cW - sw * sW * ci, cw * sW + sw * cW * ci, sw * si], 1)
    Q = torch.stack([-sw * cW - cw * sW * ci, -sw * sW + cw * cW * ci, cw * si], 1)
    cu, su, q = E.cos()[:, None], E.sin()[:, None], torch.sqrt(1.0 - e * e)[:, None]
    a = a[:, None]
    pos = a * ((cu - e[:, None]) * P + q * su * Q)
    vel = torch.sqrt(a) / pos.norm(dim=1, keepdim=True) * (-su * P + q * cu * Q)
    return pos.cpu().numpy(), vel.cpu().numpy()


def _disk(case, seed):
    """p3t_state_load's arrays; the embryo disk ends with four bodies of 0.1 Earth mass."""
    n, m = case["n"], case["m"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pos, vel = _sample(n, m, case["a_in"], case["a_out"], case["ecc"], gen)
    mass = np.full(n, m)
    if case["kind"] == "embryos":
        a = torch.tensor([0.7, 0.9, 1.1, 1.3], dtype=torch.float64, device="cuda")
        p, v = _sample(4, 3e-7, 0.5, 1.5, 2.0, gen, a)
        pos, vel, mass = np.concatenate([pos, p]), np.concatenate([vel, v]), np.concatenate([mass, np.full(4, 3e-7)])
    n = len(mass)
    r_planet = (0.75 * mass / (math.pi * P3TParams().dens)) ** (1.0 / 3.0)
    return dict(id=np.arange(n, dtype=np.int64), mass=mass, r_planet=r_planet, f=np.ones(n), pos=pos, vel=vel)


def _params(case):
    return P3TParams(n_group_limit=case.get("group", 64), theta=case.get("theta", 0.5))


def _lists_input(case, seed):
    """EPJ records in tree order, as FDPS passes them, and the CSR interaction lists over them."""
    P = _params(case)
    d = _disk(case, seed)
    n, m = case["n"], case["m"]
    h = (m / 3.0) ** (1.0 / 3.0)
    r_out = np.full(n, 3.0 * h)
    r_search = 1.1 * r_out + 6.0 * 0.6 * case["ecc"] * h * P.dt_tree
    L = build_lists(d["pos"], d["mass"], r_search, P.theta, P.n_leaf_limit, P.n_group_limit)
    order = L["i_idx"].copy()  # tree order
    rank = np.empty(n, np.int32)
    rank[order] = np.arange(n, dtype=np.int32)
    L["i_idx"], L["j_idx"] = rank[L["i_idx"]], rank[L["j_idx"]]
    return P, epj_records(d["pos"][order], d["vel"][order], d["mass"][order], r_out, r_search), L


def _pinned(a):
    t = torch.empty(max(1, a.nbytes), dtype=torch.uint8, pin_memory=True).numpy()[:a.nbytes].view(a.dtype)
    t[...] = a.reshape(-1)
    return t.reshape(a.shape)


def _system(case):
    """The library set up as gplum_gb300/run.py does: tuned launch shapes, learned queue order."""
    g = GpuSystem(_params(case))
    autotune.load(g.lib)
    model = scheduler.load(lib=g.lib)
    g.lib.p3t_set_schedule(1 if model is not None else 0)
    g.set_fragmentation(0.5 if case["kind"] == "embryos" else 0.0)
    return g


def _ptrs(a, offs):
    p = a.ctypes.data
    return (VP * (len(offs) - 1))(*[p + int(o) * a.dtype.itemsize for o in offs[:-1]])


def _walks(case, epi, epj, L, force):
    """Each walk's argument arrays of p3t_soft_dispatch[_index] and p3t_soft_retrieve."""
    index = case["kind"] == "index"
    ei = np.ascontiguousarray(epi[L["i_idx"]])
    js = L["j_idx"] if index else np.ascontiguousarray(epj[L["j_idx"]])
    ss = L["s_idx"] if index else np.ascontiguousarray(L["spj"][L["s_idx"]])
    keep, walks = [ei, js, ss], []
    for g0 in range(0, L["n_group"], case["walk"]):
        o = {k: L[k][g0:min(g0 + case["walk"], L["n_group"]) + 1] for k in ("i_off", "j_off", "s_off")}
        cnt = [np.ascontiguousarray(np.diff(o[k])) for k in ("i_off", "j_off", "s_off")]
        walks.append((len(cnt[0]), _ptrs(ei, o["i_off"]), cnt[0], _ptrs(js, o["j_off"]), cnt[1], _ptrs(ss, o["s_off"]),
                      cnt[2], _ptrs(force, o["i_off"])))
    return keep, walks


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("steps", "startup", "embryos"):
        s["g"] = g = _system(case)
        s["disk"] = d = _disk(case, seed)
        if kind == "steps":
            # the records of a run at its start (GPLUM's ParticleSystem<FPGrav> on the host)
            g.load(d)
            g.startup()
            s["records"] = _pinned(g.get_fpgrav())
        # room for the records read back: no more than at the start, but for fragments
        room = 0 if kind == "steps" else 4 + 512
        s["out"] = _pinned(np.zeros(case["n"] + room, FPGRAV_DTYPE))
        return s
    if kind == "functor":
        # one group's records: i-bodies in a cell, near bodies around it, far cells beyond
        rng = np.random.default_rng(seed)
        ni, nj, ns = case["ni"], case["nj"], case["ns"]
        size, h = 0.01, (1e-9 / 3.0) ** (1.0 / 3.0)
        pos = np.array([1.0, 0.2, 0.0]) + size * (rng.random((nj, 3)) * [6, 6, 0.3] - [3, 3, 0.15])
        epj = epj_records(pos, rng.standard_normal((nj, 3)) * 1e-3, np.full(nj, 1e-9), np.full(nj, 3 * h),
                          np.full(nj, 3.6 * h))
        epi = np.zeros(ni, EPI_DTYPE)
        epi[:min(ni, nj)] = epi_records(epj)[:ni]
        epi["id_local"] = np.arange(ni)
        epi["pos"][nj:] = np.array([1.0, 0.2, 0.0]) + size * (rng.random((max(0, ni - nj), 3)) - 0.5)
        epi["r_out"], epi["r_search"] = 3 * h, 3.6 * h
        spj = np.zeros(ns, SPJ_DTYPE)
        ang = rng.uniform(0, 2 * math.pi, ns)
        dist = rng.uniform(0.1, 1.5, ns)
        cell = 0.2 * dist
        spj["mass"] = 1e-9 * rng.integers(4, 400, ns)
        spj["pos"] = np.array([1.0, 0.2, 0.0]) + np.stack([dist * np.cos(ang), dist * np.sin(ang),
                                                            rng.normal(0, 0.003, ns)], 1)
        for k, lo, hi in (("xx", 0.5, 1.0), ("yy", 0.5, 1.0), ("zz", 0.0, 0.01), ("xy", -0.3, 0.3), ("xz", -0.02, 0.02),
                          ("yz", -0.02, 0.02)):
            spj[k] = spj["mass"] * cell**2 / 12 * rng.uniform(lo, hi, ns)
        s.update(lib=configure(P3TParams()), epi=epi, epj=epj, spj=spj, force=cleared_forces(ni), clear=cleared_forces(ni))
        return s
    P, epj, L = _lists_input(case, seed)
    n = len(epj)
    s.update(P=P, n=n, epj=epj, L=L)
    if kind in ("multiwalk", "index"):
        s["lib"] = configure(P)
        s["force"] = np.zeros(len(L["i_idx"]), FORCE_DTYPE)
        s["keep"], s["walks"] = _walks(case, epi_records(epj), epj, L, s["force"])
    elif kind == "host":
        autotune.load(configure(P))
        s["epj"] = _pinned(epj)
        s["L"] = {k: _pinned(v) if isinstance(v, np.ndarray) else v for k, v in L.items()}
        s["force"] = _pinned(np.zeros(n, FORCE_DTYPE))
    elif kind == "fp64":
        s["sf"] = SoftForce(P, precision=1)
        s["force"] = np.zeros(n, FORCE_DTYPE)
    elif kind == "noalloc":
        autotune.load(configure(P))
        s["lib"] = _lib.host_lib()
        s["dev"] = {k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).cuda()
                    for k, v in dict(L, epj=epj).items() if k != "n_group"}
        s["force"] = torch.zeros(n, 8, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------------------------
def _force(f):
    return {k: f[k] for k in ("acc", "phi", "number", "id_max", "id_min")}


def _run_walks(s):
    """Two walks in flight, as FDPS overlaps its dispatches with the retrieves."""
    lib, index = s["lib"], s["case"]["kind"] == "index"

    def ints(a):
        return a.ctypes.data_as(VP)

    def retrieve(k):
        w = s["walks"][k]
        _lib.check(lib.p3t_soft_retrieve(k & 1, w[0], ints(w[2]), w[7]), "p3t_soft_retrieve")

    for k, (m, pi, ni, pj, nj, ps, ns, _) in enumerate(s["walks"]):
        if k >= 2:
            retrieve(k - 2)
        if index:
            epj, spj = s["epj"], s["L"]["spj"]
            st = lib.p3t_soft_dispatch_index(k & 1, m, pi, ints(ni), pj, ints(nj), ps, ints(ns), ints(epj), len(epj),
                                             ints(spj), len(spj), 1 if k == 0 else 0)
        else:
            st = lib.p3t_soft_dispatch(k & 1, m, pi, ints(ni), pj, ints(nj), ps, ints(ns))
        _lib.check(st, "p3t_soft_dispatch")
    for k in range(max(0, len(s["walks"]) - 2), len(s["walks"])):
        retrieve(k)
    return _force(s["force"])


def _run_steps(s):
    g, case = s["g"], s["case"]
    if case["kind"] == "steps":
        # GPLUM's restart (the neighbour lists of the records' state), then the steps
        g.put_fpgrav(s["records"])
        g.tree_soft()
        g.correct(False)
    else:
        g.load(s["disk"])
        g.startup()
    energy, edisp, counts = [], [], []
    for k in range(case["steps"]):
        r = g.tree_step(k + 1)
        energy.append(r["energy"])
        edisp.append(r["edisp"])
        counts += [r["n_col"], r["n_removed"], r["n_body"], r["n_clusters"], r["n_isolated"]]
    out = s["out"]
    out[len(g.get_fpgrav(out)):] = 0  # the places of merged bodies
    return dict({k: out[k] for k in ("pos", "vel", "mass", "r_planet", "time", "id", "id_cluster", "number")},
                energy=np.array(energy), edisp=np.array(edisp), counts=np.array(counts))


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "functor":
        lib, f = s["lib"], s["force"]
        f[...] = s["clear"]
        epi, epj, spj = s["epi"], s["epj"], s["spj"]
        fp = f.ctypes.data_as(VP)
        _lib.check(lib.p3t_epep(epi.ctypes.data_as(VP), len(epi), epj.ctypes.data_as(VP), len(epj), fp), "p3t_epep")
        _lib.check(lib.p3t_epsp(epi.ctypes.data_as(VP), len(epi), spj.ctypes.data_as(VP), len(spj), fp), "p3t_epsp")
        return _force(f)
    if kind in ("multiwalk", "index"):
        return _run_walks(s)
    if kind == "host":
        return _force(soft_force_host(s["P"], s["epj"], s["L"], out=s["force"]))
    if kind == "fp64":
        sf = s["sf"]
        sf.upload_particles(s["epj"])
        sf.upload_lists(s["L"])
        sf.run()
        return _force(sf.download(s["force"]))
    if kind == "noalloc":
        d, L, f = s["dev"], s["L"], s["force"]
        st = s["lib"].p3t_soft_force_noalloc(
            s["n"], VP(d["epj"].data_ptr()), L["n_group"], *(VP(d[k].data_ptr()) for k in
                                                           ("i_off", "i_idx", "j_off", "j_idx", "s_off", "s_idx", "spj")),
            len(L["spj"]), s["P"].eps2, 0, VP(f.data_ptr()), VP(torch.cuda.current_stream().cuda_stream))
        _lib.check(st, "p3t_soft_force_noalloc")
        w = f.view(torch.int32)
        return {"acc": f[:, :3], "phi": f[:, 3], "number": w[:, 4], "id_max": w[:, 6], "id_min": w[:, 7]}
    if kind == "startup":
        g = s["g"]
        g.load(s["disk"])
        e = g.startup()
        f = np.zeros(g.n, FORCE_DTYPE)
        _lib.check(g.lib.p3t_download_forces(f.ctypes.data_as(VP), len(f)), "p3t_download_forces")
        return dict(_force(f), energy=e, **{k: g.get(k) for k in ("acc_d", "jerk_d", "r_out", "r_search")})
    return _run_steps(s)


# ---- what a pass cannot do without ---------------------------------------------------------------------
def _pairs_per_body(case):
    """(EP-EP, EP-SP) pairs a body: the list lengths of these disks (0.5 opening angle: 120 + 44 at 3,000
    bodies and groups of 64, 177 + 205 at 60,000; 375 + 292 at 300,000 and groups of 256, 384 + 332 at 1M)."""
    g = case["group"]
    ep = {64: 170.0, 128: 260.0}.get(g, 380.0)
    sp = max(20.0, 24.0 * math.log(case["n"] / 500.0)) * (0.5 / case["theta"]) ** 2
    return ep * 0.5 / case["theta"], sp


def work(case):
    """Per pass.  EP-EP 32 flops a pair, EP-SP 70; each record, list entry and result once.  A tree step
    of the ring adds the hard part's block steps (about 20 per body of 3 x 77 flops and 145 more)."""
    kind = case["kind"]
    if kind == "functor":
        ni, nj, ns = case["ni"], case["nj"], case["ns"]
        return dict(bytes=2 * ni * (48 + 64) + nj * 112 + ns * 80, flops=ni * (32 * nj + 70 * ns))
    n = case["n"]
    ep, sp = _pairs_per_body(case)
    soft = n * (32 * ep + 70 * sp)
    if kind in ("steps", "embryos", "startup"):
        soft *= 2 if kind == "startup" else 1 + case["steps"]
        hard = 0 if kind == "startup" else case["steps"] * n * 20 * 376
        return dict(bytes=n * (344 * 2 if kind == "steps" else 344 + 88), flops=soft + hard)
    entries = n * (ep + sp) / {64: 30.0, 128: 58.0}.get(case["group"], 118.0)
    if kind == "multiwalk":
        lists = entries * 95 + n * 48
    else:
        lists = entries * 4 + n * (112 + 4 + 0.35 * 80) + (n * 48 if kind == "index" else 0)
    return dict(bytes=lists + n * 32, flops=soft)


# ---- the same in 64 bits -------------------------------------------------------------------------------
def _exact_group(xi, roi, ej, sp):
    """calcForceEPEPWithSearch + calcForceEPSP (the default build's quadrupole trace xx + yy + xx) in FP64."""
    r = xi[:, None] - ej[None, :, :3]
    ro = torch.maximum(roi[:, None], ej[None, :, 3])
    rinv = torch.rsqrt(torch.maximum((r * r).sum(-1), ro * ro))
    p = rinv * ej[None, :, 4]
    acc = -((p * rinv * rinv)[..., None] * r).sum(1)
    phi = -p.sum(1)
    d = sp[None, :, 1:4] - xi[:, None]
    m, xx, yy, zz, xy, xz, yz = (sp[:, k] for k in (0, 4, 5, 6, 7, 8, 9))
    tr = xx + yy + xx
    x, y, z = d.unbind(-1)
    xx, yy, zz, xy, xz, yz = 3 * xx - tr, 3 * yy - tr, 3 * zz - tr, 3 * xy, 3 * xz, 3 * yz
    q = torch.stack([xx * x + xy * y + xz * z, yy * y + yz * z + xy * x, zz * z + xz * x + yz * y], -1)
    r2inv = 1.0 / (d * d).sum(-1)
    rinv = torch.sqrt(r2inv)
    rqr = (q * d).sum(-1) * r2inv * r2inv
    w = (m + 2.5 * rqr) * r2inv * rinv
    acc = acc - ((r2inv * r2inv * rinv)[..., None] * q - w[..., None] * d).sum(1)
    return acc, phi - ((m + 0.5 * rqr) * rinv).sum(1)


def _dev(*cols):
    return torch.from_numpy(np.ascontiguousarray(np.column_stack(cols))).cuda()


def exact(case, seed):
    """Forces and potentials over the same lists; the tree steps and the start-up, which build their own
    tree and integrate, have no short closed form."""
    kind = case["kind"]
    if kind in ("steps", "embryos", "startup"):
        return None
    s = prepare(case, seed)
    epj, spj = s["epj"], s["spj"] if kind == "functor" else s["L"]["spj"]
    ej = _dev(epj["pos"], epj["r_out"], epj["mass"])
    sp = _dev(spj["mass"], spj["pos"], *(spj[k] for k in ("xx", "yy", "zz", "xy", "xz", "yz")))
    if kind == "functor":
        epi = s["epi"]
        acc, phi = _exact_group(_dev(epi["pos"]), torch.from_numpy(epi["r_out"].copy()).cuda(), ej, sp)
    else:
        L = s["L"]
        i, j, c = (torch.from_numpy(np.ascontiguousarray(L[k])).long().cuda() for k in ("i_idx", "j_idx", "s_idx"))
        acc = torch.zeros(len(epj), 3, dtype=torch.float64, device="cuda")
        phi = torch.zeros(len(epj), dtype=torch.float64, device="cuda")
        io, jo, so = (L[k].tolist() for k in ("i_off", "j_off", "s_off"))
        for g in range(L["n_group"]):
            a = i[io[g]:io[g + 1]]
            e = ej[a]
            acc[a], phi[a] = _exact_group(e[:, :3], e[:, 3], ej[j[jo[g]:jo[g + 1]]], sp[c[so[g]:so[g + 1]]])
        if kind in ("multiwalk", "index"):  # results in walk order
            acc, phi = acc[i], phi[i]
    return {"acc": acc, "phi": phi, "number": None, "id_max": None, "id_min": None}
