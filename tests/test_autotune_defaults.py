"""The tuners time the library's own choice beside the named ones, so that what
they return is never slower than naming nothing."""
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
