"""The FP64 wave update where 2u passes the largest double: the sum is infinite
before v is taken from it, as in the oracle's fused flavour.  Bar: its bits, for
u in the top three binades with and without infinities among them, v beside u."""
import numpy as np
import pytest

import stencil3d_gb300 as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRID = (6, 17, 70, 4, 4, 4)


@pytest.mark.parametrize("points", [7, 13, 25])
@pytest.mark.parametrize("infinite", [False, True])
def test_twice_u_overflows_as_a_sum(points, infinite):
    rng = np.random.default_rng(points)
    shape = O.shape(GRID)
    u = rng.choice([-1.0, 1.0], shape) * np.ldexp(rng.uniform(1.0, 2.0, shape), rng.integers(1021, 1024, shape))
    assert np.isfinite(u).all()
    if infinite:
        u[rng.integers(0, 30, shape) == 0] = np.inf
    v = u * rng.choice([1.0, 0.75, -0.5], shape)
    s = np.full(shape, 0.25)
    with np.errstate(all="ignore"), S.Stencil(S.Grid(*GRID), points, "wave", "f64", dt=5e-4, src=None) as st:
        vv, uu = v.copy(), u.copy()
        st.iterate_host(vv, s, uu, 1)
    c0, c1, c2 = O.wave_constants(points, 1500.0, 5e-4, 10.0)
    O.iterate_wave(u, v, s, GRID, points, 1, c0, c1, c2, fma=True)
    np.testing.assert_array_equal(O.interior(uu, GRID), O.interior(u, GRID))
    np.testing.assert_array_equal(O.interior(vv, GRID), O.interior(v, GRID))
