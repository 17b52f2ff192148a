"""The shipped tuning file says what the autotuner would choose from the times it holds: every
choice was measured, and is within the 1 % of keep_incumbent of the best measured one."""
import json

import pytest

from gplum_gb300 import autotune

T = json.load(open(autotune.TUNING))


@pytest.mark.parametrize("choice,table", [(("soft_tiles", "soft_occ"), "soft_ms"), (("hard_tiers",), "hard_ms"),
                                          (("hard_bundle", "hard_wide"), "hard_bundle_ms")])
def test_choice_follows_its_table(choice, table):
    flat = []
    for k in choice:
        flat += T[k] if isinstance(T[k], list) else [T[k]]
    t = T[table]
    assert t[",".join(map(str, flat))] <= 1.01 * min(t.values())


def test_bundle_shapes_are_those_that_run():
    assert sorted(T["hard_bundle_ms"]) == sorted(",".join(map(str, k)) for k in autotune.BUNDLE_GRID)


def test_heavy_threshold_follows_its_table():
    t = T["hard_heavy_ms"]
    assert sorted({k.split(",")[0] for k in t}) == sorted(name for name, _, _ in autotune.heavy_disks())
    assert all(set(r) == {str(h) for h in autotune.HEAVY_GRID} for r in t.values())
    score = autotune.heavy_score(t)
    best = min(score, key=score.get)
    assert autotune.keep_incumbent(best, score, str(T["hard_heavy"])) == str(T["hard_heavy"])


def test_heavy_score():
    t = {"ring 1048576, steps 1-5": {5.0: 20.0, 6.0: 10.0}, "ring 1048576, steps 6-25": {5.0: 10.0, 6.0: 10.0},
         "a": {5.0: 1.0, 6.0: 4.0}}
    s = autotune.heavy_score(t)  # half of log 2 / 2 against half of log 4
    assert abs(s[5.0] - 2.0 ** 0.25) < 1e-12 and abs(s[6.0] - 2.0) < 1e-12
