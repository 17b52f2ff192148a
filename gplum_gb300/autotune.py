"""Autotuner for the launch shapes of the hot path.

Two choices are made by measurement on the live workload instead of fixed in
code:

* the soft kernel's work split by i-group size (p3t_set_soft_tiles: above
  t_s1 members one i-particle per thread, above t_s2 the j lists split two
  ways, else four) and its register budget (p3t_set_soft_occupancy: 4, 5 or
  6 resident CTAs per SM) -- timed on the 1,048,576-body soft-force
  disk (0.5-1.5 AU, m = 1e-10, theta = 0.5, n_group_limit = 256);
* the bundle form's heavy-cluster threshold (p3t_set_hard_heavy: clusters
  whose learned prediction of log2(1 + block steps) reaches it run alone in a
  CTA first) -- the mean hard launch of the first five tree steps and of the
  twenty after them (one restored state misjudges it) on five disks of the
  workloads' kinds (heavy_disks: rings of three sizes, embryos with fragments, a
  wide disk), by the geometric mean in which the benchmark's disk counts as much as
  the four others together (heavy_score);
* the bundle form's member slots and CTAs per SM (p3t_set_hard_bundle) and
  whether its clusters above the slots run in the concurrent wide launch as lone
  bundles of up to 512 slots or in the team form there (p3t_set_hard_wide) --
  timed from one restored state;
* the one-cluster-per-team form's size cutoffs of the hard launch
  (p3t_set_hard_tiers: clusters of >= cta_min members one per CTA, >= warp_min
  one per warp, smaller one per thread) -- timed from one restored state of the
  1,048,576-body hard-part disk.  (The default bundle form has no cutoffs; its
  queue order comes from the learned cost model, gplum_gb300/scheduler.py.)

    python -m gplum_gb300.autotune --out gplum_gb300/tuning.json

Every candidate gives the same neighbour results and forces equal to
rounding (soft) or bit-identical results (hard); only the time differs.
"""
import argparse
import ctypes
import json
import os
import time

import numpy as np

from . import _lib

TUNING = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning.json")
# (t_ipt2, t_s1, t_s2, CTAs per SM); the mixed form always runs one i per thread
SOFT_GRID = [(128, b, c, o) for b in (32, 48, 64) for c in (0, 16, 32) for o in (4, 5, 6) if c <= b]
TIER_GRID = [(w, t) for w in (2, 4, 8, 16) for t in (32, 64, 128, 256)]


def _timed(lib, fn, reps):
    ts = []
    for _ in range(reps):
        lib.p3t_synchronize()
        t0 = time.perf_counter()
        fn()
        lib.p3t_synchronize()
        ts.append(time.perf_counter() - t0)
    return float(np.median(ts))


def keep_incumbent(best, table, incumbent, tol=0.01):
    """The incumbent choice (from the existing tuning file) unless the best
    measured one is more than tol faster: choices within timing noise of each
    other do not flip from one tuning run to the next."""
    if incumbent is not None and incumbent in table and table[incumbent] <= table[best] * (1.0 + tol):
        return incumbent
    return best


def tune_soft(lib, run, grid=SOFT_GRID, reps=5):
    """Times `run` (one soft-force launch on resident lists) for each work
    split; installs the fastest.  Returns (best, {split: ms})."""
    table = {}
    for cfg in grid:
        _lib.check(lib.p3t_set_soft_tiles(*cfg[:3]), "p3t_set_soft_tiles")
        _lib.check(lib.p3t_set_soft_occupancy(cfg[3]), "p3t_set_soft_occupancy")
        run()
        table[cfg] = 1e3 * _timed(lib, run, reps)
    best = min(table, key=table.get)
    _lib.check(lib.p3t_set_soft_tiles(*best[:3]), "p3t_set_soft_tiles")
    _lib.check(lib.p3t_set_soft_occupancy(best[3]), "p3t_set_soft_occupancy")
    return best, table


def tune_tiers(g, istep=1, grid=TIER_GRID):
    """Times the one-cluster-per-team hard launch from one restored state for
    each (warp_min, cta_min); leaves the fastest installed (and the bundle
    form selected).  Returns (best, {cutoffs: ms})."""
    lib = g.lib
    _lib.check(lib.p3t_state_snapshot(0), "p3t_state_snapshot")
    table = {}
    lib.p3t_set_hard_mode(1)
    try:
        for wm, cm in grid:
            _lib.check(lib.p3t_set_hard_tiers(wm, cm), "p3t_set_hard_tiers")
            _lib.check(lib.p3t_state_snapshot(1), "p3t_state_snapshot")
            table[(wm, cm)] = 1e3 * _timed(lib, lambda: g.hard(istep), 1)
    finally:
        lib.p3t_set_hard_mode(0)
        lib.p3t_state_snapshot(1)
    best = min(table, key=table.get)
    _lib.check(lib.p3t_set_hard_tiers(*best), "p3t_set_hard_tiers")
    return best, table


HEAVY_GRID = (5.0, 5.5, 5.75, 6.0, 6.25, 6.5, 6.75, 7.0, 7.5)
HEAVY_WINDOWS = ((1, 5), (6, 25))  # tree steps after start-up, first to last


def heavy_disks():
    """(name, function that makes it, a_frag) of each disk the heavy threshold is
    measured on: the hard-part ring at the benchmark's size and at a quarter and a
    fiftieth of it, 100,000 planetesimals with embryos and fragmenting collisions, and
    a wide disk of a million bodies (the large disk's mass)."""
    from .disk import disk_1m_embryos, disk_1m_hard, make_disk

    return (("ring 1048576", disk_1m_hard, 0.0),
            ("ring 262144", lambda: disk_1m_hard(262144, seed=11), 0.0),
            ("ring 20000", lambda: disk_1m_hard(20000, seed=12), 0.0),
            ("embryos 100000", lambda: disk_1m_embryos(100000, seed=13, m=1e-9), 0.5),
            ("wide 1048576", lambda: make_disk(1048576, 1e-10, 0.3, 3.0, ecc_hill=4.0, inc_hill=2.0, seed=14), 0.0))


def heavy_score(table, bench="ring 1048576"):
    """{threshold: geometric mean of its times against each row's least} of {row:
    {threshold: ms}}; the benchmark's rows weigh half, the others half (low thresholds
    suit small disks, whose launches wait for one chain, and slow down the benchmark's,
    which the bundles' throughput bounds)."""
    def loss(h, rows):
        return np.mean([np.log(r[h] / min(r.values())) for r in rows])

    own = [r for k, r in table.items() if k.startswith(bench)]
    rest = [r for k, r in table.items() if not k.startswith(bench)]
    return {h: float(np.exp(0.5 * (loss(h, own) + loss(h, rest)))) for h in own[0]}


def tune_heavy(g, istep=1, grid=HEAVY_GRID):
    """Times the bundled hard launch with the learned order from one restored
    state for each heavy-cluster threshold; installs the fastest.  Returns
    (best, {threshold: ms})."""
    import ctypes

    lib = g.lib
    _lib.check(lib.p3t_state_snapshot(0), "p3t_state_snapshot")
    table = {}
    for h in grid:
        _lib.check(lib.p3t_set_hard_heavy(ctypes.c_float(h)), "p3t_set_hard_heavy")
        _lib.check(lib.p3t_state_snapshot(1), "p3t_state_snapshot")
        table[h] = 1e3 * _timed(lib, lambda: g.hard(istep), 1)
    lib.p3t_state_snapshot(1)
    best = min(table, key=table.get)
    _lib.check(lib.p3t_set_hard_heavy(ctypes.c_float(best)), "p3t_set_hard_heavy")
    return best, table


def tune_heavy_steps(P, disks=None, grid=HEAVY_GRID, windows=HEAVY_WINDOWS):
    """The heavy-cluster threshold by whole runs with the learned order: for each disk
    and threshold, start-up and the tree steps of the windows, the mean hard launch of
    each window (the distribution of chain lengths changes as a disk evolves, so one
    state misjudges it).  Returns (best by heavy_score, {disk and steps: {threshold:
    ms}})."""
    from . import scheduler
    from .p3t import GpuSystem

    table = {}
    for name, make, a_frag in disks or heavy_disks():
        disk = make()
        for h in grid:
            g = GpuSystem(P)
            load(g.lib)
            scheduler.load(lib=g.lib)
            g.lib.p3t_set_schedule(1)
            _lib.check(g.lib.p3t_set_hard_heavy(ctypes.c_float(h)), "p3t_set_hard_heavy")
            g.set_fragmentation(a_frag)
            g.load(disk)
            g.set_r_planet()
            g.startup()
            hard = []
            for istep in range(1, windows[-1][1] + 1):
                g.tree_step(istep)
                hard.append(g.hard_launch_stats()["ms"])
            g.set_fragmentation(0.0)
            for lo, hi in windows:
                table.setdefault("%s, steps %d-%d" % (name, lo, hi), {})[h] = float(np.mean(hard[lo - 1:hi]))
    score = heavy_score(table)
    return min(score, key=score.get), table


# (member slots, CTAs per SM, clusters above the slots in the wide launch)
BUNDLE_GRID = ((128, 3, 0), (128, 3, 1), (256, 2, 1))


def tune_wide(g, istep=1, reps=2, grid=BUNDLE_GRID):
    """Times the bundled hard launch from one restored state for each bundle
    shape (p3t_set_hard_bundle) and placement of the clusters above it
    (p3t_set_hard_wide); installs the fastest.  Returns (best, {choice: ms})."""
    lib = g.lib
    _lib.check(lib.p3t_state_snapshot(0), "p3t_state_snapshot")
    table = {}
    for cap, occ, w in grid:
        _lib.check(lib.p3t_set_hard_bundle(cap, occ), "p3t_set_hard_bundle")
        _lib.check(lib.p3t_set_hard_wide(w), "p3t_set_hard_wide")
        ts = []
        for _ in range(reps):
            _lib.check(lib.p3t_state_snapshot(1), "p3t_state_snapshot")
            ts.append(1e3 * _timed(lib, lambda: g.hard(istep), 1))
        table[(cap, occ, w)] = float(min(ts))
    lib.p3t_state_snapshot(1)
    best = min(table, key=table.get)
    _lib.check(lib.p3t_set_hard_bundle(best[0], best[1]), "p3t_set_hard_bundle")
    _lib.check(lib.p3t_set_hard_wide(best[2]), "p3t_set_hard_wide")
    return best, table


def load(lib=None, path=TUNING):
    """Installs a tuning file's choices; returns them (None without a file)."""
    if not os.path.exists(path):
        return None
    lib = lib or _lib.host_lib()
    t = json.load(open(path))
    if "soft_tiles" in t:
        _lib.check(lib.p3t_set_soft_tiles(*t["soft_tiles"]), "p3t_set_soft_tiles")
    if "soft_occ" in t:
        _lib.check(lib.p3t_set_soft_occupancy(t["soft_occ"]), "p3t_set_soft_occupancy")
    if "hard_tiers" in t:
        _lib.check(lib.p3t_set_hard_tiers(*t["hard_tiers"]), "p3t_set_hard_tiers")
    if "hard_wide" in t:
        _lib.check(lib.p3t_set_hard_wide(int(t["hard_wide"])), "p3t_set_hard_wide")
    if "hard_bundle" in t:
        _lib.check(lib.p3t_set_hard_bundle(*t["hard_bundle"]), "p3t_set_hard_bundle")
    if "hard_heavy" in t:
        import ctypes

        _lib.check(lib.p3t_set_hard_heavy(ctypes.c_float(t["hard_heavy"])), "p3t_set_hard_heavy")
    return t


def main():
    from .disk import P3TParams, disk_1m_hard, disk_1m_soft
    from .p3t import GpuSystem
    from .radii import cutoff_radii
    from .soft import SoftForce, epj_records
    from .tree import build_lists

    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=TUNING)
    ap.add_argument("--soft-only", action="store_true",
                    help="retune the soft work split only; keep the file's other entries")
    args = ap.parse_args()
    P = P3TParams(n_group_limit=256)
    # soft: resident lists of the soft-force disk, particles in tree order
    d = disk_1m_soft()
    r_out, r_search, _ = cutoff_radii(d["pos"], d["vel"], d["mass"], P)
    perm = build_lists(d["pos"], d["mass"], r_search, P.theta, P.n_leaf_limit, P.n_group_limit)["i_idx"]
    pos, mass, r_out, r_search = d["pos"][perm], d["mass"][perm], r_out[perm], r_search[perm]
    epj = epj_records(pos, d["vel"][perm], mass, r_out, r_search, ids=d["id"][perm])
    L = build_lists(pos, mass, r_search, P.theta, P.n_leaf_limit, P.n_group_limit)
    sf = SoftForce(P, precision=0)
    sf.upload_particles(epj)
    sf.upload_lists(L)
    lib = _lib.host_lib()
    soft_best, soft_table = tune_soft(lib, lambda: sf.run(emit_candidates=True))
    prev = json.load(open(args.out)) if os.path.exists(args.out) else {}
    if "soft_tiles" in prev and "soft_occ" in prev:
        soft_best = keep_incumbent(soft_best, soft_table, tuple(prev["soft_tiles"]) + (prev["soft_occ"],))
    if args.soft_only:
        out = json.load(open(args.out)) if os.path.exists(args.out) else {}
        out["soft_tiles"] = list(soft_best[:3])
        out["soft_occ"] = soft_best[3]
        out["soft_ms"] = {",".join(map(str, k)): v for k, v in soft_table.items()}
        json.dump(out, open(args.out, "w"), indent=1)
        print(json.dumps({"soft_tiles": out["soft_tiles"], "soft_occ": out["soft_occ"],
                          "soft_ms_best": soft_table[soft_best]}))
        return
    # hard: tier cutoffs of the per-team form on the hard-part disk
    d = disk_1m_hard()
    g = GpuSystem(P)
    g.load(d)
    g.set_r_planet()
    g.prepare()
    for _ in range(2):
        g.tree_soft()
        g.correct(True)
    g.kick()
    g.cluster()
    hard_best, hard_table = tune_tiers(g)
    from . import scheduler

    heavy_best, heavy_table = None, {}
    wide_best, wide_table = tune_wide(g)
    if scheduler.load(lib=g.lib) is not None:
        heavy_best, heavy_table = tune_heavy_steps(P)
        heavy_best = keep_incumbent(heavy_best, heavy_score(heavy_table), prev.get("hard_heavy"))
        _lib.check(g.lib.p3t_set_hard_heavy(ctypes.c_float(heavy_best)), "p3t_set_hard_heavy")
    if "hard_bundle" in prev and "hard_wide" in prev:
        wide_best = keep_incumbent(wide_best, wide_table, tuple(prev["hard_bundle"]) + (prev["hard_wide"],))
    if "hard_tiers" in prev:
        hard_best = keep_incumbent(hard_best, hard_table, tuple(prev["hard_tiers"]))
    out = {"soft_tiles": list(soft_best[:3]),
           "soft_occ": soft_best[3],
           "soft_ms": {",".join(map(str, k)): v for k, v in soft_table.items()},
           "hard_tiers": list(hard_best),
           "hard_heavy": heavy_best if heavy_best is not None else 6.5,
           "hard_bundle": list(wide_best[:2]),
           "hard_wide": wide_best[2],
           "hard_bundle_ms": {",".join(map(str, k)): v for k, v in wide_table.items()},
           "hard_heavy_ms": {k: {str(h): round(v, 3) for h, v in r.items()} for k, r in heavy_table.items()},
           "hard_ms": {",".join(map(str, k)): v for k, v in hard_table.items()},
           "workloads": {"soft": "1048576-body disk 0.5-1.5 AU, m=1e-10, theta=0.5, n_group_limit=256, tree order",
                         "hard": "1048576-body hard-part disk 0.95-1.05 AU, m=7e-11, rms e=6h, rms i=3h",
                         "hard_heavy": "mean hard launch (ms) over the named tree steps after start-up, learned order; "
                                       "the disks of gplum_gb300/autotune.py heavy_disks"}}
    json.dump(out, open(args.out, "w"), indent=1)
    print(json.dumps({"soft_tiles": out["soft_tiles"], "soft_ms_best": soft_table[soft_best],
                      "soft_ms_default": soft_table.get((128, 64, 32, 5)), "hard_tiers": out["hard_tiers"],
                      "hard_ms_best": hard_table[hard_best], "hard_ms_default": hard_table.get((8, 64)),
                      "hard_heavy": out["hard_heavy"], "hard_heavy_ms": out["hard_heavy_ms"]}))


if __name__ == "__main__":
    main()
