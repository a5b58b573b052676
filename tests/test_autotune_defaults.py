"""The tuners time the library's own choice beside the named ones, so that what
they return is never slower than naming nothing."""
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
