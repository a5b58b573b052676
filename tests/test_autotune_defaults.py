"""The tuners time the library's own choice beside the named ones, so that what
they return is never slower than naming nothing."""
import json

import pytest

import stencil3d_gb300 as S
from stencil3d_gb300 import autotune

DEV = {"sm_count": 152, "cc": (10, 3), "total_bytes": 1 << 38}


def test_batch_tuner_times_the_default(tmp_path, monkeypatch):
    """A batch whose large grids run faster by themselves: only ichunk 0 has them do so."""
    seen = []

    def timed(grids, points, cand, dts=None, srcs=None, steps=20, warmup=3):
        seen.append(cand)
        return 1.0 if cand == {"ichunk": 0, "schedule": "graph"} else 1.2

    monkeypatch.setattr(autotune, "measure_batch_device", timed)
    grids = [S.Grid(300, 280, 260, 4, 4, 4), S.Grid(64, 64, 64, 4, 4, 4)]
    best = autotune.tune_batch(grids, [7, 25], cache=str(tmp_path / "t.json"), device=DEV)
    assert best["opts"] == {"ichunk": 0, "schedule": "graph"}
    assert len(seen) == 1 + len(autotune.batch_candidates())


@pytest.mark.parametrize("points,mode,storage", [
    (p, m, st) for st in ("f32", "f64", "f16", "bf16", "f16_hl")
    for m in (("ref", "wave") if st in ("f32", "f64") else ("wave",)) for p in (7, 13, 25)] + [(2, "ref", "f32")])
def test_every_list_has_the_automatic_unit_length(points, mode, storage):
    """Of each kernel that a list names, one candidate leaves the planes per unit to the library."""
    cands = autotune.candidates(points, mode, storage)
    for kernel in {c["kernel"] for c in cands}:
        assert any(c["kernel"] == kernel and c.get("ichunk", 0) == 0 for c in cands), kernel


def test_a_choice_among_older_candidates_is_not_reused(tmp_path):
    """Cache files of before the version stood in the key: the workload is timed again."""
    grid, path = S.Grid(256, 256, 256, 4, 4, 4), tmp_path / "t.json"
    old = "sm152_cc103|25|wave|f32|256x256x256|h4,4,4"
    stale = {"key": old, "opts": {"kernel": "tma", "tile_j": 16, "stages": 4, "ichunk": 0}, "ms_per_step": 9.0}
    batch = "|".join(autotune.batch_key([grid], [7], DEV).split("|")[:4])
    path.write_text(json.dumps({old: stale, batch: {"key": batch, "opts": {"ichunk": 512, "schedule": "persistent"}}}))
    best = autotune.tune(grid, 25, cache=str(path), device=DEV,
                         measure=lambda c: 1.0 if c == {"kernel": "tma"} else 2.0)
    assert best["opts"] == {"kernel": "tma"}
    best = autotune.tune_batch([grid], [7], cache=str(path), device=DEV,
                               measure=lambda c: 1.0 if c["schedule"] == "graph" else 2.0)
    assert best["opts"]["schedule"] == "graph"
    assert old in json.loads(path.read_text())  # left where an older library finds it
