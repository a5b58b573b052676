"""The graph schedule of a batch large enough that some grids leave the shared
queue for multi-step launches of their own.  Bar: bit for bit the sequential
schedule, over calls of the same and of other lengths (replayed graphs, odd
lengths that swap the buffers between them, more steps than one launch takes),
mixed with calls of another schedule and with one grid advanced by itself."""
import numpy as np
import pytest

import stencil3d_gb300 as S

pytestmark = pytest.mark.gpu

SPECS = [((200, 180, 260, 4, 4, 4), 7, (100, 15, 259)), ((150, 187, 300, 4, 4, 4), 13, (3, 100, 100)),
         ((170, 160, 265, 4, 4, 4), 25, (80, 31, 64)), ((20, 18, 30, 4, 4, 4), 25, (10, 9, 8)),
         ((40, 30, 66, 4, 4, 4), 13, (0, 0, 0))]


def _run(calls):
    grids = [S.Grid(*g) for g, _, _ in SPECS]
    pts = [p for _, p, _ in SPECS]
    with S.Batch(grids, pts, dt=[1e-3 if p == 7 else 5e-4 for p in pts], srcs=[s for _, _, s in SPECS]) as b:
        for i in range(len(SPECS)):
            st = b.context(i)
            st.fill(S.FIELD_U, S.FILL_UNIFORM, 3 + i, -1e-3, 1e-3)
            st.fill(S.FIELD_V, S.FILL_UNIFORM, 50 + i, -1e-3, 1e-3)
            st.fill(S.FIELD_S, S.FILL_UNIFORM, 90 + i, -1.0, 1.0)
        for n, schedule in calls:
            if schedule == "one":
                b.context(1).iterate(n)
            else:
                b.iterate(n, schedule)
        b.synchronize()
        out = []
        for i, g in enumerate(grids):
            u, v = g.empty(), g.empty()
            b.context(i).download(v, u)
            out.append((u, v))
        return out, b.info()


def test_split_graph_matches_sequential():
    calls = [(270, "graph"), (21, "graph"), (21, "graph"), (8, "graph"), (3, "one"), (21, "graph"),
             (5, "pipelined"), (8, "graph")]
    got, info = _run(calls)
    assert info.graphs == 3
    want, _ = _run([(n, "one" if s == "one" else "sequential") for n, s in calls])
    for (ua, va), (ub, vb) in zip(got, want):
        np.testing.assert_array_equal(ua, ub)
        np.testing.assert_array_equal(va, vb)
